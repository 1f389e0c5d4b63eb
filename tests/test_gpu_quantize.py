"""Bit-exact parity of the CUDA quantizers against the CPU oracle (through the C ABI)."""
import math

import numpy as np
import pytest

from tests.test_oracle_golden import E2M1_VALUES
from tests.util import require_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    require_cuda()
    from eider_b200 import ops
    return ops


def _dev(a, dtype=None):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.to(dtype)


def test_reference_fixture_static_scale(ops, oracle):
    # crates/eider-cuda/src/kernels/non_gemm.rs:19655-19683: K=96, 3 tokens, input_scale=.25
    k, t = 96, 3
    x = (((np.arange(k * t) % 29) - 14) / 32.0).astype(np.float32).reshape(t, k)
    q = ops.quantize_nvfp4(_dev(x), 0.25)
    packed, scales = oracle.quantize_nvfp4(x, 0.25)
    assert np.array_equal(q.packed.cpu().numpy(), packed)
    assert np.array_equal(q.scales.cpu().numpy(), scales)


@pytest.mark.parametrize("tokens,k", [(1, 16), (1, 5120), (7, 544), (130, 2048), (512, 5120)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_static_scale_random(ops, oracle, tokens, k, dtype):
    import torch
    rng = np.random.default_rng(tokens * 1000 + k)
    x = rng.standard_normal((tokens, k)).astype(np.float32) * np.exp(rng.uniform(-3, 3, (tokens, 1))).astype(np.float32)
    if dtype == "bf16":
        x = oracle.bf16_round(x)
    xd = _dev(x, torch.bfloat16 if dtype == "bf16" else None)
    for scale in (1.0, 0.37):
        q = ops.quantize_nvfp4(xd, scale)
        packed, scales = oracle.quantize_nvfp4(x, scale)
        assert np.array_equal(q.packed.cpu().numpy(), packed)
        assert np.array_equal(q.scales.cpu().numpy(), scales)


def test_edge_values(ops, oracle):
    # every tie point / saturation / NaN / signed zero of the reference's E2M1 list, one per block position
    vals = np.array(E2M1_VALUES, np.float32)
    pad = (-len(vals)) % 16
    x = np.concatenate([vals, np.zeros(pad, np.float32)]).reshape(1, -1)
    # block scale 1.0: put a 6.0 in every block so the codes are the raw E2M1 roundings
    x = x.reshape(-1, 16).copy()
    x = np.concatenate([x[:, :15], np.full((x.shape[0], 1), 6.0, np.float32)], axis=1).reshape(1, -1)
    q = ops.quantize_nvfp4(_dev(x), 1.0)
    packed, scales = oracle.quantize_nvfp4(x, 1.0)
    assert np.array_equal(q.packed.cpu().numpy(), packed)
    assert np.array_equal(q.scales.cpu().numpy(), scales)


def test_all_zero_and_nonfinite_rows(ops, oracle):
    x = np.zeros((3, 64), np.float32)
    x[1, 5] = np.inf
    x[1, 6] = 2.0
    x[2, 17] = np.nan
    x[2, 18] = -3.0
    q = ops.quantize_nvfp4(_dev(x), 1.0)
    packed, scales = oracle.quantize_nvfp4(x, 1.0)
    assert np.array_equal(q.packed.cpu().numpy(), packed)
    assert np.array_equal(q.scales.cpu().numpy(), scales)
    qr = ops.quantize_nvfp4_rowscale(_dev(x))
    p2, s2, r2 = oracle.quantize_nvfp4_rowscale(x)
    assert np.array_equal(qr.packed.cpu().numpy(), p2)
    assert np.array_equal(qr.scales.cpu().numpy(), s2)
    assert np.array_equal(qr.row_scales.cpu().numpy(), r2)


# (up to 16384 elements per row: one thread per 16-element block; up to 32768: one thread per 8 elements in up to four
# passes; longer rows: the generic kernel)
@pytest.mark.parametrize("tokens,k", [(1, 5120), (33, 2048), (512, 5120), (130, 13824), (3, 8208), (5, 32768), (2, 32784),
                                      (1300, 13824)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_rowscale(ops, oracle, tokens, k, dtype):
    import torch
    rng = np.random.default_rng(7 + tokens)
    x = rng.standard_normal((tokens, k)).astype(np.float32)
    if dtype == "bf16":
        x = oracle.bf16_round(x)
    q = ops.quantize_nvfp4_rowscale(_dev(x, torch.bfloat16 if dtype == "bf16" else None))
    packed, scales, row = oracle.quantize_nvfp4_rowscale(x)
    assert np.array_equal(q.row_scales.cpu().numpy(), row)
    assert np.array_equal(q.packed.cpu().numpy(), packed)
    assert np.array_equal(q.scales.cpu().numpy(), scales)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_rowscale_with_specials_everywhere(ops, oracle, dtype):
    # signed zeros, infinities of both signs, NaNs, denormals and huge values sprinkled over random rows: blocks with an
    # infinity take the kernel's careful path, all others the short one, and both must give the reference's bytes
    import torch
    rng = np.random.default_rng(11)
    tokens, k = 96, 5120
    x = rng.standard_normal((tokens, k)).astype(np.float32)
    x[rng.random((tokens, k)) < 0.02] = 0.0
    x[rng.random((tokens, k)) < 0.02] = -0.0
    x[rng.random((tokens, k)) < 0.002] = np.inf
    x[rng.random((tokens, k)) < 0.002] = -np.inf
    x[rng.random((tokens, k)) < 0.002] = np.nan
    x[rng.random((tokens, k)) < 0.01] *= 1e-30
    x[5] *= 1e20
    x[6] *= 1e-25
    x[7, :] = 0.0
    x[8, :16] = -0.0
    x[9, 16:32] = [np.inf] * 8 + [-np.inf] * 8
    if dtype == "bf16":
        x = oracle.bf16_round(x)
    q = ops.quantize_nvfp4_rowscale(_dev(x, torch.bfloat16 if dtype == "bf16" else None))
    packed, scales, row = oracle.quantize_nvfp4_rowscale(x)
    assert np.array_equal(q.row_scales.cpu().numpy(), row)
    assert np.array_equal(q.scales.cpu().numpy(), scales)
    assert np.array_equal(q.packed.cpu().numpy(), packed)


def test_weight_quantize_and_repack(ops, oracle):
    rng = np.random.default_rng(3)
    w = (rng.standard_normal((384, 1024)) * 0.02).astype(np.float32)
    wd = ops.ModelOptWeight.quantize(_dev(w))
    packed, scales, g = oracle.quantize_weight(w)
    assert wd.weight_scale_2 == float(g)
    assert np.array_equal(wd.packed.cpu().numpy(), packed)
    assert np.array_equal(wd.scales_row_major.cpu().numpy(), scales)
    assert np.array_equal(wd.scales_tiled.cpu().numpy(), oracle.scales_to_tiled(scales, 384, 1024))


def test_modelopt_k16_known_answer(ops):
    # crates/eider-format/src/modelopt.rs:1281-1294
    row = np.array([[0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0]], np.float32)
    wd = ops.ModelOptWeight.quantize(_dev(row), global_scale=1.0)
    assert wd.scales_row_major.cpu().numpy().tolist() == [[0x38]]
    assert wd.packed.cpu().numpy().tolist() == [[0x10, 0x32, 0x54, 0x76, 0x98, 0xBA, 0xDC, 0xFE]]


def test_invalid_arguments(ops):
    import torch
    x = torch.zeros(2, 32, device="cuda")
    with pytest.raises(ops.ShapeError):
        ops.quantize_nvfp4(x, 0.0)
    from eider_b200 import _lib
    lib = _lib.load()
    assert lib.infer_quantize_nvfp4_col_major_f32_on_stream(None, None, None, 16, 1, 1.0, None) == 1  # cudaErrorInvalidValue
    assert lib.infer_quantize_nvfp4_col_major_f32_on_stream(x.data_ptr(), x.data_ptr(), x.data_ptr(), 0, 1, 1.0, None) == 1
    assert lib.infer_quantize_nvfp4_col_major_f32_on_stream(x.data_ptr(), x.data_ptr(), x.data_ptr(), 16, 1, math.inf, None) == 1


@pytest.mark.parametrize("rows,cols", [(1, 5120), (8, 5120), (64, 1000)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_fp8_dynamic(ops, oracle, rows, cols, dtype):
    import torch
    rng = np.random.default_rng(rows + cols)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    if dtype == "bf16":
        x = oracle.bf16_round(x)
    q, s = ops.quantize_fp8_dynamic(_dev(x, torch.bfloat16 if dtype == "bf16" else None))
    qo, so = oracle.quantize_fp8_dynamic(x)
    assert np.array_equal(s.cpu().numpy(), so)
    assert np.array_equal(q.cpu().numpy(), qo)


def test_fp8_static_and_weight(ops, oracle):
    rng = np.random.default_rng(11)
    x = rng.standard_normal((5, 4100)).astype(np.float32)
    q = ops.quantize_fp8_static(_dev(x), 0.125)
    assert np.array_equal(q.cpu().numpy(), oracle.quantize_fp8_static(x, 0.125))
    w = (rng.standard_normal((96, 512)) * 0.02).astype(np.float32)
    wq, ws = ops.quantize_fp8_weight(_dev(w))
    wqo, wso = oracle.quantize_fp8_weight(w)
    assert np.array_equal(ws.cpu().numpy(), wso)
    assert np.array_equal(wq.cpu().numpy(), wqo)


@pytest.mark.parametrize("tokens,k,scale", [(1, 768, 1.0), (1, 13824, 0.03125), (5, 2048, 1.0), (130, 256, 0.5)])
def test_fused_silu_mul_quantize_matches_oracle(ops, oracle, tokens, k, scale):
    # non_gemm.cu:559-629: value = g * (1 / (1 + expf(-g))) * up / input_scale, then the block quantizer; the device's
    # expf may differ from the host's in the last place, which can move a code across a rounding boundary now and then
    import torch
    rng = np.random.default_rng(tokens + k)
    gu = (rng.standard_normal((tokens, 2 * k)) * 2.0).astype(np.float32)
    gu[0, :16] = 0.0  # an all-zero block: scale byte 0, codes 0
    q = ops.silu_mul_halves_quantize_nvfp4(torch.from_numpy(gu).cuda(), scale)
    torch.cuda.synchronize()
    p_ref, s_ref, act = oracle.silu_mul_halves_quantize_nvfp4(gu, scale, want_act=True)
    got_p, got_s = q.packed.cpu().numpy(), q.scales.cpu().numpy()
    assert np.count_nonzero(got_p != p_ref) / got_p.size < 2e-3
    assert np.count_nonzero(got_s != s_ref) / got_s.size < 2e-3
    deq = oracle.dequantize_tiled(got_p, got_s) * scale
    bmax = np.abs(act).reshape(tokens, -1, 16).max(axis=2).repeat(16, axis=1)
    assert np.all(np.abs(deq - act) <= 0.27 * bmax + 1e-12)
    if tokens == 1:  # the reference's single-token entry point gives the same bytes
        from eider_b200 import _lib
        lib = _lib.load()
        p1 = torch.zeros(k // 2, dtype=torch.uint8, device="cuda")
        s1 = torch.zeros_like(q.scales)
        assert lib.infer_silu_mul_halves_quantize_nvfp4_col_major_f32_on_stream(
            torch.from_numpy(gu).cuda().data_ptr(), p1.data_ptr(), s1.data_ptr(), k, scale, None) == 0
        torch.cuda.synchronize()
        assert np.array_equal(p1.cpu().numpy(), got_p[0]) and np.array_equal(s1.cpu().numpy(), got_s)
        assert lib.infer_silu_mul_halves_quantize_nvfp4_col_major_f32_on_stream(None, p1.data_ptr(), s1.data_ptr(), k, scale, None) == 1


@pytest.mark.parametrize("rows,cols,scale", [(1, 5120, 1.0), (7, 2048, 0.25), (300, 256, 1.0)])
def test_fused_rms_norm_quantize_matches_oracle(ops, oracle, rows, cols, scale):
    # non_gemm.cu:193-288: x * rsqrt(mean(x^2) + eps) * weight / input_scale, then the block quantizer.  The sum of
    # squares has no canonical order (and the device uses rsqrtf), so inverse_rms may differ from the oracle's by an
    # ulp or two, which moves a code across a rounding boundary now and then.
    import torch
    rng = np.random.default_rng(rows + cols)
    x = (rng.standard_normal((rows, cols)) * np.exp(rng.uniform(-1, 1, (rows, 1)))).astype(np.float32)
    w = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    q = ops.rms_norm_quantize_nvfp4(torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), 1e-6, scale)
    torch.cuda.synchronize()
    p_ref, s_ref, norm = oracle.rms_norm_quantize_nvfp4(x, w, 1e-6, scale, want_norm=True)
    got_p, got_s = q.packed.cpu().numpy(), q.scales.cpu().numpy()
    assert np.count_nonzero(got_p != p_ref) / got_p.size < 5e-3
    assert np.count_nonzero(got_s != s_ref) / got_s.size < 5e-3
    deq = oracle.dequantize_tiled(got_p, got_s)
    bmax = np.abs(norm).reshape(rows, -1, 16).max(axis=2).repeat(16, axis=1)
    assert np.all(np.abs(deq - norm) <= 0.27 * bmax + 1e-12)
    from eider_b200 import _lib
    assert _lib.load().infer_rms_norm_quantize_nvfp4_col_major_f32_on_stream(None, None, None, None, rows, cols, 1e-6, scale, None) == 1


@pytest.mark.parametrize("rows,cols", [(1, 5120), (9, 2048), (200, 256)])
def test_fused_add_then_norm_quantize_matches_oracle(ops, oracle, rows, cols):
    # non_gemm.cu:746-870: h = rmsnorm(x) * w0 + residual (stored), then the quantizing RMSNorm of h
    import torch
    rng = np.random.default_rng(rows * 3 + cols)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    res = rng.standard_normal((rows, cols)).astype(np.float32)
    w0 = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    w1 = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda()
    h, q = ops.rms_norm_add_then_rms_norm_quantize_nvfp4(dev(x), dev(w0), dev(res), dev(w1), 1e-6, 1e-5, 0.5)
    torch.cuda.synchronize()
    h_ref, p_ref, s_ref, norm = oracle.rms_norm_add_then_rms_norm_quantize_nvfp4(x, w0, res, w1, 1e-6, 1e-5, 0.5)
    assert np.allclose(h.cpu().numpy(), h_ref, rtol=2e-6, atol=2e-6)
    got_p, got_s = q.packed.cpu().numpy(), q.scales.cpu().numpy()
    assert np.count_nonzero(got_p != p_ref) / got_p.size < 5e-3
    assert np.count_nonzero(got_s != s_ref) / got_s.size < 5e-3
    deq = oracle.dequantize_tiled(got_p, got_s)
    bmax = np.abs(norm).reshape(rows, -1, 16).max(axis=2).repeat(16, axis=1)
    assert np.all(np.abs(deq - norm) <= 0.27 * bmax + 1e-12)


@pytest.mark.parametrize("rows,cols", [(1, 5120), (33, 1024)])
def test_fused_rms_norm_quantize_pair_matches_oracle(ops, oracle, rows, cols):
    # non_gemm.cu:290-419: the second term quantizes what the first left, block by block
    import torch
    from eider_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(rows + cols + 1)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    n_sf = oracle.scale_layout_len(rows, cols)
    p = torch.zeros(rows, cols // 2, dtype=torch.uint8, device="cuda")
    rp = torch.zeros_like(p)
    s_ = torch.zeros(n_sf, dtype=torch.uint8, device="cuda")
    rs = torch.zeros_like(s_)
    assert lib.infer_rms_norm_quantize_nvfp4_pair_col_major_f32_on_stream(xd.data_ptr(), wd.data_ptr(), p.data_ptr(), s_.data_ptr(),
                                                                          rp.data_ptr(), rs.data_ptr(), rows, cols, 1e-6, 1.0, None) == 0
    torch.cuda.synchronize()
    p0, s0, rp0, rs0 = oracle.rms_norm_quantize_nvfp4_pair(x, w, 1e-6, 1.0)
    _, _, norm = oracle.rms_norm_quantize_nvfp4(x, w, 1e-6, 1.0, want_norm=True)
    got = [t.cpu().numpy() for t in (p, s_, rp, rs)]
    for a, b in zip(got, (p0, s0, rp0, rs0)):
        assert np.count_nonzero(a != b) / a.size < 1e-2
    # the first term alone equals the single-term producer bit for bit
    q1 = ops.rms_norm_quantize_nvfp4(xd, wd, 1e-6, 1.0)
    assert torch.equal(q1.packed, p) and torch.equal(q1.scales, s_)
    two = oracle.dequantize_tiled(got[0], got[1]) + oracle.dequantize_tiled(got[2], got[3])
    bmax = np.abs(norm).reshape(rows, -1, 16).max(axis=2).repeat(16, axis=1)
    assert np.all(np.abs(two - norm) <= 0.08 * bmax + 1e-12)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -20, 2.0 ** 40, 0.0075])
def test_every_block_scale_on_rounding_boundaries(ops, oracle, dtype, scale):
    # one block per UE4M3 scale value: its maximum sets the scale, the other elements are the exact rounding boundaries of E2M1
    # times that scale (ties), their neighbours, and both zeros; per-row scales (powers of two) and a given scale
    import torch
    codes = np.arange(1, 127)
    sv = np.array([oracle.e4m3_value(int(c)) for c in codes], np.float64)
    ties = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])
    blocks = np.concatenate([6.0 * np.ones((126, 1)), np.tile(ties, (126, 1)), np.tile(-ties, (126, 1)), np.zeros((126, 1))], 1) * sv[:, None]
    blocks[:, 15] = -0.0
    x = (blocks.reshape(1, -1) * scale).astype(np.float32)
    rows = [x, np.nextafter(x, np.float32(np.inf)), np.nextafter(x, np.float32(-np.inf))]
    if dtype == "bf16":
        rows = [oracle.bf16_round(r) for r in rows]
    x = np.concatenate(rows)
    t = torch.from_numpy(x).cuda()
    t = t.bfloat16() if dtype == "bf16" else t
    p, s, r = oracle.quantize_nvfp4_rowscale(x)
    got = ops.quantize_nvfp4_rowscale(t)
    assert np.array_equal(got.row_scales.cpu().numpy(), r)
    assert np.array_equal(got.packed.cpu().numpy(), p) and np.array_equal(got.scales.cpu().numpy(), s)
    p, s = oracle.quantize_nvfp4(x, scale)
    got = ops.quantize_nvfp4(t, scale)
    assert np.array_equal(got.packed.cpu().numpy(), p) and np.array_equal(got.scales.cpu().numpy(), s)


@pytest.mark.parametrize("rows,k", [(1, 16), (3, 48), (127, 80), (128, 64), (129, 8208), (700, 512), (2, 16384), (5, 16400)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_quantizers_write_their_padding(ops, oracle, rows, k, dtype):
    # storage full of ones: the padding rows of the last 128-row tile and the padding blocks of a row come out as zero; more rows
    # than resident CTAs, specials in the row ahead
    import torch
    rng = np.random.default_rng(rows + k)
    x = rng.standard_normal((rows, k)).astype(np.float32)
    x[rng.random(x.shape) < 1e-3] = np.inf
    x[rng.random(x.shape) < 1e-3] = np.nan
    x[rng.random(x.shape) < 1e-2] = -0.0
    if dtype == "bf16":
        x = oracle.bf16_round(x)
    t = torch.from_numpy(x).cuda()
    t = t.bfloat16() if dtype == "bf16" else t

    def storage():
        m = ops.Nvfp4Matrix.zeros(rows, k, row_scales=True)
        m.packed.fill_(255), m.scales.fill_(255), m.row_scales.fill_(-1)
        return m

    for got, want in ((ops.quantize_nvfp4_rowscale(t, storage()), oracle.quantize_nvfp4_rowscale(x)[:2]),
                      (ops.quantize_nvfp4(t, 0.02, storage()), oracle.quantize_nvfp4(x, 0.02))):
        assert np.array_equal(got.packed.cpu().numpy(), want[0])
        assert np.array_equal(got.scales.cpu().numpy(), want[1])
    q, s = ops.quantize_fp8_dynamic(t)
    wq, ws = oracle.quantize_fp8_dynamic(x)
    assert np.array_equal(s.cpu().numpy(), ws) and np.array_equal(q.cpu().numpy(), wq)


def _scale_writers(lib, x, k, rows, rng):
    """name -> (plain call, padded call or None) of (packed, scales, row_scales) for every operator that writes tiled scales."""
    import torch
    xb = x.bfloat16()
    gate_up = torch.from_numpy(rng.standard_normal((rows, 2 * k)).astype(np.float32)).cuda()
    w, h = torch.rand(k, device="cuda") + 0.5, torch.empty_like(x)
    other_p, other_s = torch.empty(rows * k // 2, dtype=torch.uint8, device="cuda"), torch.empty(lib.eider_b200_nvfp4_scale_layout_len(rows, k), dtype=torch.uint8, device="cuda")
    keep = (x, xb, gate_up, w, h, other_p, other_s)
    xp, bp, gp, wp, hp = (t.data_ptr() for t in keep[:5])
    padded = lib.eider_b200_quantize_nvfp4_padded_on_stream
    calls = {
        "static f32": (lambda p, s, r: lib.infer_quantize_nvfp4_col_major_f32_on_stream(xp, p, s, k, rows, 0.02, None),
                       lambda p, s, r: padded(xp, 0, p, s, None, k, rows, 0.02, None)),
        "static bf16": (lambda p, s, r: lib.eider_b200_quantize_nvfp4_bf16_on_stream(bp, p, s, k, rows, 1.0, None),
                        lambda p, s, r: padded(bp, 1, p, s, None, k, rows, 1.0, None)),
        "row f32": (lambda p, s, r: lib.eider_b200_quantize_nvfp4_rowscale_on_stream(xp, 0, p, s, r, k, rows, None),
                    lambda p, s, r: padded(xp, 0, p, s, r, k, rows, 1.0, None)),
        "row bf16": (lambda p, s, r: lib.eider_b200_quantize_nvfp4_rowscale_on_stream(bp, 1, p, s, r, k, rows, None),
                     lambda p, s, r: padded(bp, 1, p, s, r, k, rows, 1.0, None)),
        "norm": (lambda p, s, r: lib.infer_rms_norm_quantize_nvfp4_col_major_f32_on_stream(xp, wp, p, s, rows, k, 1e-6, 0.02, None),
                 lambda p, s, r: lib.eider_b200_rms_norm_quantize_nvfp4_padded_on_stream(xp, wp, p, s, rows, k, 1e-6, 0.02, None)),
        "norm pair": (lambda p, s, r: lib.infer_rms_norm_quantize_nvfp4_pair_col_major_f32_on_stream(xp, wp, p, s, other_p.data_ptr(), other_s.data_ptr(),
                                                                                                   rows, k, 1e-6, 0.02, None), None),
        "norm pair residual": (lambda p, s, r: lib.infer_rms_norm_quantize_nvfp4_pair_col_major_f32_on_stream(xp, wp, other_p.data_ptr(), other_s.data_ptr(),
                                                                                                            p, s, rows, k, 1e-6, 0.02, None), None),
        "silu": (lambda p, s, r: lib.eider_b200_silu_mul_halves_quantize_nvfp4_batch_on_stream(gp, p, s, rows, k, 0.02, None),
                 lambda p, s, r: lib.eider_b200_silu_mul_halves_quantize_nvfp4_padded_on_stream(gp, p, s, rows, k, 0.02, None)),
    }
    if k <= 12272:
        args = (xp, wp, xp, hp, wp)
        calls["add norm"] = (lambda p, s, r: lib.infer_rms_norm_add_then_rms_norm_quantize_nvfp4_f32_on_stream(*args, p, s, rows, k, 1e-6, 1e-6, 0.02, None),
                             lambda p, s, r: lib.eider_b200_rms_norm_add_then_rms_norm_quantize_nvfp4_padded_on_stream(*args, p, s, rows, k, 1e-6, 1e-6, 0.02, None))
    return keep, calls


@pytest.mark.parametrize("rows,k", [(1, 16), (1, 5120), (3, 48), (31, 80), (32, 2064), (33, 112), (97, 64), (127, 320), (128, 48), (129, 48), (300, 208),
                                    (5, 16400), (2, 32784)])
def test_scales_past_the_rows_belong_to_the_caller(ops, rows, k):
    # the plain entry points write the bytes of their rows and blocks and nothing else; the padded ones what the plain ones leave in
    # a zeroed buffer, in a buffer that was not zeroed, up to its last byte and not past it
    import torch

    from eider_b200 import _lib
    from tests.test_gpu_guard_bands import guarded
    lib = _lib.load()
    rng = np.random.default_rng(rows + k)
    x = torch.from_numpy(rng.standard_normal((rows, k)).astype(np.float32)).cuda()
    r_, b_ = np.meshgrid(np.arange(rows), np.arange(k // 16), indexing="ij")
    padded_blocks = (k // 16 + 3) // 4 * 4
    own = torch.zeros(ops.scale_layout_len(rows, k), dtype=torch.bool)
    own[torch.from_numpy(((b_ // 4) * 4 + (r_ // 128) * padded_blocks) * 128 + (r_ % 32) * 16 + (r_ % 128) // 32 * 4 + b_ % 4).reshape(-1)] = True
    own = own.cuda()
    keep, calls = _scale_writers(lib, x, k, rows, rng)
    for name, (plain, padded) in calls.items():
        row_scales = torch.empty(rows, device="cuda")
        out = []
        for call, fill in ((plain, 0), (plain, 0xAB)) + (((padded, 0xAB),) if padded else ()):
            packed, ok_p = guarded(torch, rows * k // 2, torch.uint8)
            scales, ok_s = guarded(torch, own.numel(), torch.uint8)
            scales.fill_(fill)
            assert call(packed.data_ptr(), scales.data_ptr(), row_scales.data_ptr()) == 0, name
            torch.cuda.synchronize()
            assert ok_p() and ok_s(), name
            out.append((packed, scales))
        zeroed, plain_out = out[0], out[1]
        assert not zeroed[1][~own].any(), name
        assert torch.equal(plain_out[0], zeroed[0]) and torch.equal(plain_out[1][own], zeroed[1][own]), name
        assert bool((plain_out[1][~own] == 0xAB).all()), name
        if padded:
            assert torch.equal(out[2][0], zeroed[0]) and torch.equal(out[2][1], zeroed[1]), name
            scales = torch.empty(own.numel() + 16, dtype=torch.uint8, device="cuda")
            assert padded(out[2][0].data_ptr(), scales.data_ptr() + 4, row_scales.data_ptr()) == 1, name  # (written in 16-byte units)


def test_quantizing_into_a_larger_matrix_keeps_its_other_rows(ops):
    import torch
    x = torch.randn(100, 320, device="cuda")
    for quantize in (lambda v, m: ops.quantize_nvfp4(v, 0.02, m), lambda v, m: ops.quantize_nvfp4(v.bfloat16(), 0.02, m), ops.quantize_nvfp4_rowscale):
        whole = quantize(x, ops.Nvfp4Matrix.zeros(100, 320, row_scales=True))
        again = quantize(x[:40].contiguous(), ops.Nvfp4Matrix(whole.packed.clone(), whole.scales.clone(), 100, 320, whole.row_scales.clone()))
        assert torch.equal(again.packed, whole.packed) and torch.equal(again.scales, whole.scales)

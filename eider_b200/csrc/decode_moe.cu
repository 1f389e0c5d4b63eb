// Decode-side routed MoE (one to a few tokens, top-k slots each): grouped GEMVs over per-expert weight tables, the
// per-slot SiLU * up stage, the weighted accumulation of the slots and the shared-expert / residual finalize, plus the
// fused lm-head GEMV + arg-max.  Everything a decode step of the reference's routed layers calls between the router and
// the residual stream (crates/eider-cuda/native/non_gemm.cu:3396-3960, 13316-13640; crates/eider-cuda/native/
// cutlass_gemv.cu:277-880), under the reference's names.
//
// All of it is HBM-bound streaming: a slot's expert matrix is read exactly once with 128-bit loads, one warp per output
// row, activations staged once per CTA in shared memory, warp-shuffle reduction; the experts of the slots are found
// through device pointer tables, so nothing is gathered or copied first.  Products are exact in f32 (an E2M1 value times
// an f32 activation, or times another E2M1 value) and only the order of the additions differs from the reference.
#include <algorithm>

#include "common.cuh"
#include "eider_b200.h"

namespace eider {
namespace {

constexpr int kWarps = 8;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Shared-memory slot of element e (0..31) of 32-element chunk c: float4 slots XOR-swizzled by the chunk so that lanes
// reading the same slot of consecutive chunks hit distinct banks.
__device__ __forceinline__ uint32_t xs_index(uint32_t c, uint32_t e) { return c * 32 + ((((e >> 2) ^ (c & 7u)) << 2) | (e & 3u)); }

// Two E2M1 codes, two E4M3 bytes -> f32, by the hardware conversion through f16 (exact): three instructions for two codes
// where e2m1_value's bit operations take about eight each, which is what bound these kernels.
__device__ __forceinline__ float2 e2m1_pair(uint32_t byte) {
    const __half2_raw h = __nv_cvt_fp4x2_to_halfraw2(static_cast<__nv_fp4x2_storage_t>(byte), __NV_E2M1);
    return __half22float2(__half2(h));
}
__device__ __forceinline__ float2 e4m3_pair(uint32_t two_bytes) {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(two_bytes), __NV_E4M3);
    return __half22float2(__half2(h));
}
__device__ __forceinline__ void dot8(uint32_t w, const float4& a, const float4& b, float& acc) {
    const float2 w0 = e2m1_pair(w & 0xffu), w1 = e2m1_pair((w >> 8) & 0xffu), w2 = e2m1_pair((w >> 16) & 0xffu), w3 = e2m1_pair(w >> 24);
    acc = fmaf(w0.x, a.x, acc);
    acc = fmaf(w0.y, a.y, acc);
    acc = fmaf(w1.x, a.z, acc);
    acc = fmaf(w1.y, a.w, acc);
    acc = fmaf(w2.x, b.x, acc);
    acc = fmaf(w2.y, b.y, acc);
    acc = fmaf(w3.x, b.z, acc);
    acc = fmaf(w3.y, b.w, acc);
}
__device__ __forceinline__ void dot_word(uint32_t w, const float* xs, uint32_t c, uint32_t e0, float& acc) {
    dot8(w, *reinterpret_cast<const float4*>(xs + xs_index(c, e0)), *reinterpret_cast<const float4*>(xs + xs_index(c, e0 + 4)), acc);
}

enum XMode { kSharedF32 = 0, kTableF32 = 1, kSharedNvfp4 = 2 };

struct GroupedArgs {
    const uint32_t* indices;          // [groups] expert of every slot (null: slot g uses table entry g)
    const void* x;                    // kSharedF32: f32 [k]; kTableF32: const float* const* [groups]; kSharedNvfp4: packed [k/2]
    const uint8_t* x_scales;          // kSharedNvfp4: tiled scales of the one activation row (outer = 0)
    const uint8_t* const* w_table;    // [table_len] packed weights [n][k/2]
    const uint8_t* const* s_table;    // [table_len] weight scales: row-major [n][k/16] or tiled (TILED)
    const float* alpha_table;         // [table_len] per-expert factor (null: alpha)
    float alpha;
    float* const* y_table;            // [groups] outputs [n] (null: y_flat + g * n)
    float* y_flat;
    uint32_t table_len, groups, n, k;
    const uint32_t* route_ids = nullptr;  // kTableF32: when set, slot g reads input (and writes output) route_ids[g] of the tables
};

// grid = (ceil(n / kWarps), groups); k % 32 == 0.
template <int XMODE, bool TILED>
__global__ void __launch_bounds__(kWarps * 32) grouped_gemv_kernel(const GroupedArgs a) {
    extern __shared__ float xs[];  // [k], swizzled
    const uint32_t group = blockIdx.y;
    const uint32_t expert = a.indices ? __ldg(a.indices + group) : group;
    if (expert >= a.table_len) return;  // (the reference skips such slots, non_gemm.cu:13342-13345)
    const uint32_t k = a.k;
    if (XMODE == kSharedNvfp4) {
        const uint8_t* xp = static_cast<const uint8_t*>(a.x);
        for (uint32_t i = threadIdx.x; i < k / 2; i += blockDim.x) {
            const uint32_t byte = __ldg(xp + i);
            const float s = e4m3_value(__ldg(a.x_scales + tiled_scale_offset(0, i / 8, k)));
            const uint32_t e = 2 * i;
            xs[xs_index(e / 32, e % 32)] = __fmul_rn(e2m1_value(byte), s);
            xs[xs_index(e / 32, e % 32 + 1)] = __fmul_rn(e2m1_value(byte >> 4), s);
        }
    } else {
        const uint32_t x_slot = (XMODE == kTableF32 && a.route_ids) ? __ldg(a.route_ids + group) : group;
        const float* x = XMODE == kTableF32 ? static_cast<const float* const*>(a.x)[x_slot] : static_cast<const float*>(a.x);
        for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) xs[xs_index(i / 32, i % 32)] = __ldg(x + i);
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (row >= a.n) return;
    const uint8_t* wrow = a.w_table[expert] + static_cast<size_t>(row) * (k / 2);
    const uint8_t* sbase = a.s_table[expert];
    float acc = 0.0f;
    for (uint32_t c = lane; c < k / 32; c += 32) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(wrow + c * 16));
        uint32_t sc;
        if (TILED) sc = __ldg(reinterpret_cast<const uint16_t*>(sbase + tiled_scale_offset(row, c * 2, k)));  // blocks 2c, 2c + 1 are adjacent
        else sc = __ldg(reinterpret_cast<const uint16_t*>(sbase + static_cast<size_t>(row) * (k / 16) + c * 2));
        float p0 = 0.0f, p1 = 0.0f;
        dot_word(q.x, xs, c, 0, p0);
        dot_word(q.y, xs, c, 8, p0);
        dot_word(q.z, xs, c, 16, p1);
        dot_word(q.w, xs, c, 24, p1);
        const float2 s = e4m3_pair(sc);
        acc = fmaf(s.x, p0, acc);
        acc = fmaf(s.y, p1, acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) {
        const uint32_t y_slot = (XMODE == kTableF32 && a.route_ids) ? __ldg(a.route_ids + group) : group;
        float* y = a.y_table ? a.y_table[y_slot] : a.y_flat + static_cast<size_t>(y_slot) * a.n;
        y[row] = __fmul_rn(acc, a.alpha_table ? __ldg(a.alpha_table + expert) : a.alpha);
    }
}

template <int XMODE, bool TILED>
cudaError_t launch_grouped(const GroupedArgs& a, cudaStream_t stream) {
    if (a.k == 0 || a.k % 32 != 0 || a.n == 0 || a.groups == 0 || a.table_len == 0) return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(a.k) * sizeof(float);
    if (smem > 200 * 1024) return cudaErrorNotSupported;
    if (smem > 48 * 1024) {
        cudaError_t st = cudaFuncSetAttribute(grouped_gemv_kernel<XMODE, TILED>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (st != cudaSuccess) return st;
    }
    const dim3 grid((a.n + kWarps - 1) / kWarps, a.groups);
    grouped_gemv_kernel<XMODE, TILED><<<grid, kWarps * 32, smem, stream>>>(a);
    return cudaGetLastError();
}

// gate * alpha, up * alpha, then gate * sigmoid(gate) * up (non_gemm.cu:3507-3511, 3570-3574)
__device__ __forceinline__ float slot_silu(float g, float u, float alpha) {
    g = __fmul_rn(g, alpha);
    u = __fmul_rn(u, alpha);
    const float sigmoid = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-g)));
    return __fmul_rn(__fmul_rn(g, sigmoid), u);
}

// Per slot: SiLU(gate) * up of the slot's [gate | up] f32 row -> f32 (non_gemm.cu:3558-3576).  grid = (blocks, groups).
__global__ void __launch_bounds__(256) silu_slots_f32_kernel(const uint32_t* __restrict__ indices, const float* const* gate_up_table,
                                                             float* const* output_table, const float* __restrict__ alpha_table,
                                                             uint32_t rows) {
    const uint32_t slot = blockIdx.y;
    const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= rows) return;
    const float alpha = __ldg(alpha_table + __ldg(indices + slot));
    const float* gu = gate_up_table[slot];
    output_table[slot][row] = slot_silu(__ldg(gu + row), __ldg(gu + rows + row), alpha);
}

// Per slot: the same values / input_scale[expert] -> NVFP4 with one scale byte per 16 values in plain order
// (non_gemm.cu:3485-3536).  One thread per 16-value block; grid = (blocks of 128 threads, groups).
__global__ void __launch_bounds__(128) silu_quantize_slots_kernel(const uint32_t* __restrict__ indices, const float* const* gate_up_table,
                                                                  uint8_t* const* packed_table, uint8_t* const* scales_table,
                                                                  const float* __restrict__ input_scale_table,
                                                                  const float* __restrict__ alpha_table, uint32_t rows) {
    const uint32_t slot = blockIdx.y;
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= (rows + 15) / 16) return;
    const uint32_t expert = __ldg(indices + slot);
    const float input_scale = __ldg(input_scale_table + expert);
    if (!(input_scale > 0.0f) || !isfinite(input_scale)) return;  // (as the reference: such a slot is left untouched)
    const float alpha = __ldg(alpha_table + expert);
    const float* gu = gate_up_table[slot];
    const uint32_t valid = min(16u, rows - b * 16);
    const Divisor di = make_divisor(input_scale);
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i)
        v[i] = static_cast<uint32_t>(i) < valid ? div_rn(slot_silu(__ldg(gu + b * 16 + i), __ldg(gu + rows + b * 16 + i), alpha), di) : 0.0f;
    uint2 bytes;
    scales_table[slot][b] = quantize_block16(v, valid, &bytes);
    const uint32_t w[2] = {bytes.x, bytes.y};
    uint8_t* packed = packed_table[slot];
    for (uint32_t i = 0; i < (valid + 1) / 2; ++i) packed[b * 8 + i] = static_cast<uint8_t>(w[i / 4] >> ((i % 4) * 8));
}

// out[row][c] = sum_slot inputs[route][c] * route_weights[route] * alpha[expert(route)], slot order (non_gemm.cu:3595-3639);
// with FINALIZE: + shared_output * sigmoid(shared_gate_logit) + residual, rounded to bf16 precision (non_gemm.cu:3789-3875).
template <bool FINALIZE>
__global__ void __launch_bounds__(256) accumulate_slots_kernel(const uint32_t* __restrict__ indices, const float* __restrict__ route_weights,
                                                               const float* const* inputs, const float* __restrict__ alpha_table,
                                                               const float* __restrict__ shared_gate_logit,
                                                               const float* __restrict__ shared_output, const float* __restrict__ residual,
                                                               float* __restrict__ output, uint32_t rows, uint32_t len, uint32_t groups) {
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<size_t>(rows) * len) return;
    const uint32_t row = static_cast<uint32_t>(idx / len), col = static_cast<uint32_t>(idx % len);
    float sum = 0.0f;
    for (uint32_t slot = 0; slot < groups; ++slot) {
        const uint32_t route = row * groups + slot;
        // inputs * weight * alpha + sum, the last two as one fused multiply-add (what nvcc makes of non_gemm.cu:3609)
        sum = fmaf(__fmul_rn(inputs[route][col], __ldg(route_weights + route)), __ldg(alpha_table + __ldg(indices + route)), sum);
    }
    if (FINALIZE) {
        const float shared_scale = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-__ldg(shared_gate_logit + row))));
        const float ffn = __fadd_rn(sum, __fmul_rn(__ldg(shared_output + idx), shared_scale));
        sum = bf16_bits_to_float(float_to_bf16_bits(__fadd_rn(__ldg(residual + idx), ffn)));
    }
    output[idx] = sum;
}

// ---- one token through a routed-MoE layer in two launches -------------------------------------------------------------------
// Router top-k + gate/up GEMV + SiLU * up, then down GEMV + weighted sum + shared expert + residual.  As five launches (top-k,
// GEMV, SiLU, GEMV, finalize) a layer of 8 x (3 x 2048 x 768) weights, 21 MB or 3.3 us of HBM time, took 45 us: the chain of
// launches that waited for each other, GEMVs whose CTAs staged 8 KB of x for 8 KB of weights, and eight instructions for
// every weight.  Now 17.5 us: 1.7 us
// until the experts are known, 1 us to look up and request, 3.5 us for the weights, 2.5 us to the last CTA's end, and the same
// again in short for the second launch.
//  * One warp of every CTA selects the experts (k rounds of two warp reductions) while the others read x and the tables,
//    instead of waiting for a launch that does.  (Selected by all threads of every CTA, by counting ranks, the same step took
//    3 to 6 us: forty warps an SM repeating it are bound by issue slots.)
//  * Weights become bf16 by bit operations on pairs of codes, are multiplied by their block scale (E2M1 x E4M3 has at most six
//    significant bits: exact) and go through mma.m16n8k16 with the activation as three bf16 terms of eight bits each, which
//    hold an f32 value exactly: about 2.7 instructions a weight against six and a half with f32 FMAs, f32 accumulation.
//    The tensor cores only stand in for the FMAs; a row is still streamed once.
//  * The second launch is a programmatic dependent, released when the first has started, i.e. when all that the first depends on
//    (the logits too) is complete: it selects its experts and requests its weights before it waits for the activations.
//    (Requesting them into L2 from the first launch instead cost 1 us: its own requests queue behind them.)
constexpr uint32_t kStepThreads = 256;
constexpr uint32_t kStepWarps = kStepThreads / 32;
constexpr uint32_t kStepMaxExperts = 512;
constexpr uint32_t kStepMaxTopK = 32;
constexpr uint32_t kStepMaxHidden = 4096;  // (6 bytes of shared memory an element, 33 KB in all; more has not been measured and takes the five calls)
constexpr uint32_t kStepMaxTasks = 6 * kStepWarps;  // down: (two slots, 128 features) tasks of a tile, six a warp

struct MoeStepArgs {
    const float* logits;
    const float* x;
    const uint8_t* const* w_table;
    const uint8_t* const* s_table;
    const float* g_table;
    uint32_t* indices;       // [top_k], written by the first launch
    float* weights;          // [top_k]
    uint16_t* act;           // [3 terms][top_k][inter], elements of eight in the order 0 4 1 5 2 6 3 7
    const float* shared_gate_logit;
    const float* shared_output;
    const float* residual;
    float* out;
    uint32_t experts, top_k, hidden, inter;
};

__device__ __forceinline__ float router_logit(float v) {
    // NaN -> -inf, +inf -> FLT_MAX (non_gemm.cu:1876-1881)
    if (v != v) return -INFINITY;
    return v == INFINITY ? 3.402823466e+38f : v;
}

struct StepRouting {
    const uint8_t* w[kStepMaxExperts];  // the tables
    const uint8_t* s[kStepMaxExperts];
    uint32_t expert[kStepMaxTopK];
    float weight[kStepMaxTopK];
};
// Order-preserving integer form of a logit (-0 is 0).
__device__ __forceinline__ int order_key(float v) {
    const int b = __float_as_int(v + 0.0f);
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float key_value(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// moe_topk_kernel's selection with normalized weights, by one warp: k rounds of the largest logit, the lowest expert on ties.
// Slots that no finite logit fills get expert 0 with weight 0, and a token without any finite logit experts 0, 1, ... with
// weights 1, 0, ..., as there.
template <int PER_LANE>
__device__ __forceinline__ void warp_select(const MoeStepArgs& a, StepRouting& r) {
    const uint32_t lane = threadIdx.x & 31;
    const int lowest = order_key(-INFINITY);
    int key[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) key[i] = lane + 32 * i < a.experts ? order_key(router_logit(__ldg(a.logits + lane + 32 * i))) : lowest;
    uint32_t expert = 0;
    float logit = -INFINITY;
    for (uint32_t slot = 0; slot < a.top_k; ++slot) {
        int best = key[0];
        uint32_t e = lane;
#pragma unroll
        for (int i = 1; i < PER_LANE; ++i)
            if (key[i] > best) {
                best = key[i];
                e = lane + 32 * i;
            }
        const int top = __reduce_max_sync(0xffffffffu, best);
        if (top == lowest) break;
        const uint32_t winner = __reduce_min_sync(0xffffffffu, best == top ? e : 0xffffffffu);
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i)
            if (lane + 32 * i == winner) key[i] = lowest;
        if (lane == slot) {
            expert = winner;
            logit = key_value(top);
        }
    }
    const float first = __shfl_sync(0xffffffffu, logit, 0);
    const bool none = !(first > -INFINITY);
    float w = lane < a.top_k && !none ? expf(logit - first) : 0.0f;
    float sum = 0.0f;
    for (uint32_t i = 0; i < a.top_k; ++i) sum += __shfl_sync(0xffffffffu, w, i);
    if (sum > 0.0f && sum < INFINITY) w = __fdiv_rn(w, sum);
    r.expert[lane] = none ? lane : expert;
    r.weight[lane] = none ? (lane == 0 ? 1.0f : 0.0f) : w;
}
__device__ __forceinline__ void select_experts(const MoeStepArgs& a, StepRouting& r) {
    if (a.experts <= 128) warp_select<4>(a, r);
    else warp_select<16>(a, r);
}
// The expert tables into shared memory, by all but the first warp, which selects.
__device__ __forceinline__ void read_tables(const MoeStepArgs& a, StepRouting& r) {
    for (uint32_t e = threadIdx.x - 32; e < a.experts; e += kStepThreads - 32) {
        r.w[e] = a.w_table[e];
        r.s[e] = a.s_table[e];
    }
}

// Two f32 values as three pairs of bf16 (eight bits each, by truncation: the sum of the three is exact but for what underflows);
// an infinity or NaN goes into the first alone.
__device__ __forceinline__ void bf16_terms(float lo, float hi, uint32_t (&t)[3]) {
    const uint32_t l = __float_as_uint(lo), h = __float_as_uint(hi);
    const float rl = lo - __uint_as_float(l & 0xffff0000u), rh = hi - __uint_as_float(h & 0xffff0000u);
    const uint32_t l1 = __float_as_uint(rl), h1 = __float_as_uint(rh);
    t[0] = __byte_perm(l, h, 0x7632);
    t[1] = __byte_perm(l1, h1, 0x7632);
    t[2] = __byte_perm(__float_as_uint(rl - __uint_as_float(l1 & 0xffff0000u)), __float_as_uint(rh - __uint_as_float(h1 & 0xffff0000u)), 0x7632);
    if (!(fabsf(lo) < INFINITY) || !(fabsf(hi) < INFINITY)) {
        // (a NaN whose upper half is that of an infinity becomes the canonical one; the other value keeps its terms)
        const uint32_t keep = (fabsf(lo) < INFINITY ? 0x0000ffffu : 0u) | (fabsf(hi) < INFINITY ? 0xffff0000u : 0u);
        t[1] &= keep;
        t[2] &= keep;
        if (lo != lo) t[0] |= 0x00007fffu;
        if (hi != hi) t[0] |= 0x7fff0000u;
    }
}
// Place of element i of a term plane: pairs (0, 4) (1, 5) (2, 6) (3, 7) of every eight, the order the codes of a word come out in.
__device__ __forceinline__ uint32_t term_slot(uint32_t i) { return (i & ~7u) | ((i & 3u) << 1) | ((i >> 2) & 1u); }

// Eight E2M1 codes -> four bf16 pairs (codes j and j + 4) of value * 2^-126, exact: sign to bit 15, exponent and mantissa to
// bits 8..6 of each half.
__device__ __forceinline__ void e2m1_bf16(uint32_t w, uint32_t (&p)[4]) {
    p[0] = ((w << 12) & 0x80008000u) | ((w << 6) & 0x01c001c0u);
    p[1] = ((w << 8) & 0x80008000u) | ((w << 2) & 0x01c001c0u);
    p[2] = ((w << 4) & 0x80008000u) | ((w >> 2) & 0x01c001c0u);
    p[3] = (w & 0x80008000u) | ((w >> 6) & 0x01c001c0u);
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// Block scale * 2^119 in both halves (at most 448 * 2^119: in range), so that a weight comes out as its value * 2^-7.
__device__ __forceinline__ uint32_t scale_bf16x2(float s) {
    const uint32_t b = __float_as_uint(s * 6.64613997892457936e35f);
    return __byte_perm(b, b, 0x3232);
}
constexpr float kWeightUnit = 128.0f;
// 16 bytes of shared memory where `load`, else zeros, without a branch.
__device__ __forceinline__ uint4 load_shared_if(uint32_t address, bool load) {
    uint4 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                 "@p ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w)
                 : "r"(address), "r"(static_cast<uint32_t>(load)));
    return v;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t word_of(const uint4& q, int i) { return i == 0 ? q.x : i == 1 ? q.y : i == 2 ? q.z : q.w; }

// 16 rows x 128 elements: this lane's 32 weights of row lane / 4 and of the row eight below (`lo`, `hi`, with their two block
// scales each), `term`: its 32 elements of the activation term that MMA column lane / 4 holds (or zeros), eight a step.
template <typename Term>
__device__ __forceinline__ void mma_block(float (&d)[4], const uint4& lo, const uint4& hi, uint32_t scales_lo, uint32_t scales_hi, Term term) {
    const float2 sl = e4m3_pair(scales_lo), sh = e4m3_pair(scales_hi);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t fl = scale_bf16x2(i < 2 ? sl.x : sl.y), fh = scale_bf16x2(i < 2 ? sh.x : sh.y);
        uint32_t pl[4], ph[4];
        e2m1_bf16(word_of(lo, i), pl);
        e2m1_bf16(word_of(hi, i), ph);
        const uint4 x = term(i);
        mma_bf16(d, mul_bf16x2(pl[0], fl), mul_bf16x2(ph[0], fh), mul_bf16x2(pl[1], fl), mul_bf16x2(ph[1], fh), x.x, x.y);
        mma_bf16(d, mul_bf16x2(pl[2], fl), mul_bf16x2(ph[2], fh), mul_bf16x2(pl[3], fl), mul_bf16x2(ph[3], fh), x.z, x.w);
    }
}
// 16-byte unit i of chunk c (32 elements) of a term plane in shared memory: the four lanes that read one unit of four chunks,
// four chunks apart, and the first two planes fall on different banks.
__device__ __forceinline__ uint32_t term_offset(uint32_t n, uint32_t c, uint32_t i) {
    return (c >> 1) * 128 + (((((c & 1) << 2) | i) ^ (((c >> 2) & 3) | ((n & 1) << 2))) << 4);
}

// Gate/up: a tile is the gate and up rows of 8 features of one slot's expert (rows 0-7 and 8-15 of the MMA); four warps share
// its K in units of 512 elements, 64 contiguous weight bytes and 8 scale bytes of both rows per lane, all requested at once.
// The two tiles of a CTA belong to one slot.  (64 registers: with at most three of these CTAs on an SM there is room for one
// of the next launch beside them.)
__global__ void __launch_bounds__(kStepThreads, 4) moe_step_gate_up_kernel(const MoeStepArgs a) {
    extern __shared__ __align__(128) uint8_t terms[];  // [3][hidden * 2]
    __shared__ __align__(16) StepRouting routing;
    __shared__ float partial[kStepWarps][16];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t plane = a.hidden * 2, chunks = a.hidden / 32;
    if (threadIdx.x < 32) {
        select_experts(a, routing);
    } else {
        for (uint32_t i = threadIdx.x - 32; i < a.hidden / 8; i += kStepThreads - 32) {
            const float4 lo = __ldg(reinterpret_cast<const float4*>(a.x) + 2 * i), hi = __ldg(reinterpret_cast<const float4*>(a.x) + 2 * i + 1);
            uint32_t t[4][3];
            bf16_terms(lo.x, hi.x, t[0]);
            bf16_terms(lo.y, hi.y, t[1]);
            bf16_terms(lo.z, hi.z, t[2]);
            bf16_terms(lo.w, hi.w, t[3]);
#pragma unroll
            for (uint32_t n = 0; n < 3; ++n)
                *reinterpret_cast<uint4*>(terms + n * plane + term_offset(n, i / 4, i & 3)) = make_uint4(t[0][n], t[1][n], t[2][n], t[3][n]);
        }
        read_tables(a, routing);
    }
    __syncthreads();
    const uint32_t ctas_per_slot = a.inter / 16;
    const uint32_t slot = blockIdx.x / ctas_per_slot, part = blockIdx.x - slot * ctas_per_slot;
    const uint32_t e = routing.expert[slot];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const uint32_t feature = part * 16 + (warp >> 2) * 8 + g;
    const uint8_t* w_lo = routing.w[e] + static_cast<size_t>(feature) * (a.hidden / 2);
    const uint8_t* s_lo = routing.s[e] + static_cast<size_t>(feature) * (a.hidden / 16);
    const uint8_t* w_hi = w_lo + static_cast<size_t>(a.inter) * (a.hidden / 2);
    const uint8_t* s_hi = s_lo + static_cast<size_t>(a.inter) * (a.hidden / 16);
    const uint32_t units = (chunks + 15) / 16;
    const uint32_t terms_base = static_cast<uint32_t>(__cvta_generic_to_shared(terms));
    float gate = 0.0f, up = 0.0f;
    for (uint32_t unit = warp & 3; unit < units; unit += 4) {
        const uint32_t c = unit * 16 + q * 4;  // this lane's four chunks (hidden % 128 == 0: all or none of them exist)
        uint4 lo[4], hi[4];
        uint2 sl = make_uint2(0, 0), sh = make_uint2(0, 0);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) lo[j] = hi[j] = make_uint4(0, 0, 0, 0);
        if (c < chunks) {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                lo[j] = __ldg(reinterpret_cast<const uint4*>(w_lo + (c + j) * 16));
                hi[j] = __ldg(reinterpret_cast<const uint4*>(w_hi + (c + j) * 16));
            }
            sl = __ldg(reinterpret_cast<const uint2*>(s_lo + c * 2));
            sh = __ldg(reinterpret_cast<const uint2*>(s_hi + c * 2));
        }
        // The MMA's eight columns: four share the steps of the first term, the two smaller terms (2^-8, 2^-16) have one each.  An MMA
        // truncates what it adds to, so its sums are kept short (eight MMAs a column and unit) and added in f32: the first term in
        // one column over the whole row came to 4.4e-7 of the result at hidden 4096 (five launches with f32 FMAs 2.0e-7), now 1.9e-7.
        const uint32_t plane_index = g < 4 ? 0 : g - 3, plane_terms = terms_base + plane_index * plane;
        const uint32_t step = c >= chunks || g > 5 ? 8 : g < 4 ? g : 4;  // (8: no step, 4: every step)
        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            mma_block(d, lo[j], hi[j], ((j < 2 ? sl.x : sl.y) >> (16 * (j & 1))) & 0xffffu, ((j < 2 ? sh.x : sh.y) >> (16 * (j & 1))) & 0xffffu,
                      [&](int i) { return load_shared_if(plane_terms + term_offset(plane_index, c + j, i), step == static_cast<uint32_t>(i) || step == 4); });
        gate += d[0] + d[1];
        up += d[2] + d[3];
    }
    // sum over the columns
#pragma unroll
    for (int o = 1; o < 4; o *= 2) {
        gate += __shfl_xor_sync(0xffffffffu, gate, o);
        up += __shfl_xor_sync(0xffffffffu, up, o);
    }
    if (q == 0) {
        partial[warp][g] = gate;
        partial[warp][g + 8] = up;
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        const uint32_t row = threadIdx.x & 7, w0 = (threadIdx.x / 8) * 4;
        gate = up = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < 4; ++w) {
            gate += partial[w0 + w][row];
            up += partial[w0 + w][row + 8];
        }
        const float g2 = __ldg(a.g_table + e);
        // (the weights' unit 2^-7 comes off first: a power of two, exact)
        const float v = slot_silu(__fmul_rn(gate * kWeightUnit, g2), __fmul_rn(up * kWeightUnit, g2), 1.0f);
        uint32_t t3[3];
        bf16_terms(v, v, t3);
#pragma unroll
        for (uint32_t n = 0; n < 3; ++n)
            a.act[static_cast<size_t>(n * a.top_k + slot) * a.inter + term_slot(part * 16 + threadIdx.x)] = static_cast<uint16_t>(t3[n]);
    } else if (blockIdx.x == 0 && threadIdx.x >= 32 && threadIdx.x - 32 < a.top_k) {
        a.indices[threadIdx.x - 32] = routing.expert[threadIdx.x - 32];
        a.weights[threadIdx.x - 32] = routing.weight[threadIdx.x - 32];
    }
}

// Down: a tile is 8 output columns (rows of the down matrices) for two slots at a time: rows 0-7 of the MMA are the columns in
// the first slot's matrix, rows 8-15 in the second's, and MMA columns 0-2 and 3-5 their activations' terms (the two cross
// products are not used).  Tasks, 128 features of two slots each, are dealt to the warps and all requested before the
// activations are awaited; then the slots' weighted sum, the shared expert and the residual, rounded to bf16 precision.
// TASKS = tasks per warp.
template <uint32_t TASKS>
__global__ void __launch_bounds__(kStepThreads, TASKS > 3 ? 2 : 4) moe_step_down_kernel(const MoeStepArgs a) {
    __shared__ __align__(16) StepRouting routing;
    __shared__ float partial[kStepWarps][8];
    if (threadIdx.x < 32) select_experts(a, routing);
    else read_tables(a, routing);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const uint32_t row = blockIdx.x * 8 + g;  // (whole tiles)
    const uint32_t chunks = a.inter / 32, blocks = (chunks + 3) / 4, tasks = (a.top_k + 1) / 2 * blocks;
    const size_t w_off = static_cast<size_t>(row) * (a.inter / 2), s_off = static_cast<size_t>(row) * (a.inter / 16);
    uint4 lo[TASKS], hi[TASKS];
    uint16_t sl[TASKS], sh[TASKS];
#pragma unroll
    for (uint32_t j = 0; j < TASKS; ++j) {
        const uint32_t task = warp + j * kStepWarps;
        const uint32_t pair = task / blocks, c = (task - pair * blocks) * 4 + q;
        lo[j] = hi[j] = make_uint4(0, 0, 0, 0);
        sl[j] = sh[j] = 0;
        if (task < tasks && c < chunks) {
            const uint32_t e0 = routing.expert[2 * pair];
            lo[j] = __ldg(reinterpret_cast<const uint4*>(routing.w[e0] + w_off + c * 16));
            sl[j] = __ldg(reinterpret_cast<const uint16_t*>(routing.s[e0] + s_off + c * 2));
            if (2 * pair + 1 < a.top_k) {
                const uint32_t e1 = routing.expert[2 * pair + 1];
                hi[j] = __ldg(reinterpret_cast<const uint4*>(routing.w[e1] + w_off + c * 16));
                sh[j] = __ldg(reinterpret_cast<const uint16_t*>(routing.s[e1] + s_off + c * 2));
            }
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    float total = 0.0f;
#pragma unroll
    for (uint32_t j = 0; j < TASKS; ++j) {
        const uint32_t task = warp + j * kStepWarps;
        if (task >= tasks) break;  // (warp-uniform)
        const uint32_t pair = task / blocks, c = (task - pair * blocks) * 4 + q;
        const uint32_t term = g < 3 ? g : g - 3, slot = 2 * pair + (g < 3 ? 0 : 1);
        const bool ok = g < 6 && slot < a.top_k && c < chunks;
        const uint4* src = reinterpret_cast<const uint4*>(a.act + static_cast<size_t>(term * a.top_k + slot) * a.inter + c * 32);
        uint4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = ok ? __ldcg(src + i) : make_uint4(0, 0, 0, 0);
        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        mma_block(d, lo[j], hi[j], sl[j], sh[j], [&](int i) { return x[i]; });
        const float first = q == 0 ? d[0] + d[1] : q == 1 ? d[0] : 0.0f, second = q == 1 ? d[3] : q == 2 ? d[2] + d[3] : 0.0f;
        total = fmaf(first, __fmul_rn(__ldg(a.g_table + routing.expert[2 * pair]), routing.weight[2 * pair]), total);
        if (2 * pair + 1 < a.top_k)
            total = fmaf(second, __fmul_rn(__ldg(a.g_table + routing.expert[2 * pair + 1]), routing.weight[2 * pair + 1]), total);
    }
#pragma unroll
    for (int o = 1; o < 4; o *= 2) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (q == 0) partial[warp][g] = total;
    __syncthreads();
    if (threadIdx.x < 8) {
        float sum = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < kStepWarps; ++w) sum += partial[w][threadIdx.x];
        const uint32_t col = blockIdx.x * 8 + threadIdx.x;
        const float shared_scale = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-a.shared_gate_logit[0])));
        const float ffn = __fadd_rn(sum * kWeightUnit, __fmul_rn(a.shared_output[col], shared_scale));
        a.out[col] = bf16_bits_to_float(float_to_bf16_bits(__fadd_rn(a.residual[col], ffn)));
    }
}

template <typename Kernel>
cudaError_t launch_step(Kernel kernel, uint32_t grid, size_t smem, const MoeStepArgs& a, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

// Fused lm-head GEMV + arg-max (non_gemm.cu:13423-13640): pass 1 keeps, per CTA, the best (value, row) of its rows; pass 2
// reduces the per-CTA candidates.  The logits are never written.  Ties go to the lower row, NaN never wins.
__global__ void __launch_bounds__(kWarps * 32) top1_pass1_kernel(const float* __restrict__ x, const uint8_t* __restrict__ w,
                                                                 const uint8_t* __restrict__ s, float w2, uint32_t n, uint32_t k,
                                                                 float* __restrict__ block_value, uint32_t* __restrict__ block_row) {
    extern __shared__ float xs[];
    __shared__ float best_v[kWarps];
    __shared__ uint32_t best_r[kWarps];
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) xs[xs_index(i / 32, i % 32)] = __ldg(x + i);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // every warp walks rows warp, warp + kWarps * gridDim.x ... of this CTA's share
    float bv = -INFINITY;
    uint32_t br = 0xffffffffu;
    for (uint32_t row = blockIdx.x * kWarps + warp; row < n; row += gridDim.x * kWarps) {
        const uint8_t* wrow = w + static_cast<size_t>(row) * (k / 2);
        const uint8_t* srow = s + static_cast<size_t>(row) * (k / 16);
        float acc = 0.0f;
        for (uint32_t c = lane; c < k / 32; c += 32) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(wrow + c * 16));
            const uint32_t sc = __ldg(reinterpret_cast<const uint16_t*>(srow + c * 2));
            float p0 = 0.0f, p1 = 0.0f;
            dot_word(q.x, xs, c, 0, p0);
            dot_word(q.y, xs, c, 8, p0);
            dot_word(q.z, xs, c, 16, p1);
            dot_word(q.w, xs, c, 24, p1);
            const float2 sv = e4m3_pair(sc);
            acc = fmaf(sv.x, p0, acc);
            acc = fmaf(sv.y, p1, acc);
        }
        const float v = __fmul_rn(warp_sum(acc), w2);
        if (v > bv || (v == bv && row < br)) {
            bv = v;
            br = row;
        }
    }
    if (lane == 0) {
        best_v[warp] = bv;
        best_r[warp] = br;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < kWarps; ++i)
            if (best_v[i] > bv || (best_v[i] == bv && best_r[i] < br)) {
                bv = best_v[i];
                br = best_r[i];
            }
        block_value[blockIdx.x] = bv;
        block_row[blockIdx.x] = br;
    }
}

__global__ void __launch_bounds__(256) top1_pass2_kernel(const float* __restrict__ block_value, const uint32_t* __restrict__ block_row,
                                                         uint32_t blocks, uint32_t* __restrict__ out_index, float* __restrict__ out_value) {
    __shared__ float sv[256];
    __shared__ uint32_t sr[256];
    float bv = -INFINITY;
    uint32_t br = 0xffffffffu;
    for (uint32_t i = threadIdx.x; i < blocks; i += blockDim.x) {
        const float v = block_value[i];
        const uint32_t r = block_row[i];
        if (v > bv || (v == bv && r < br)) {
            bv = v;
            br = r;
        }
    }
    sv[threadIdx.x] = bv;
    sr[threadIdx.x] = br;
    __syncthreads();
    for (uint32_t o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            const float v = sv[threadIdx.x + o];
            const uint32_t r = sr[threadIdx.x + o];
            if (v > sv[threadIdx.x] || (v == sv[threadIdx.x] && r < sr[threadIdx.x])) {
                sv[threadIdx.x] = v;
                sr[threadIdx.x] = r;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out_index[0] = sr[0] == 0xffffffffu ? 0u : sr[0];  // (all rows NaN: row 0, as an arg-max over nothing better)
        if (out_value) out_value[0] = sv[0];
    }
}

// ---- FP8 W8A8 slots (crates/eider-cuda/native/non_gemm.cu:10156-10350) ------------------------------------------------------
// One warp per output row, the slot's activation codes decoded once per CTA into shared memory, weights streamed with 128-bit
// loads; every product of two E4M3 values is exact in f32.  GATE_UP: rows [0, n) come from the gate table and [n, 2n) from
// the up table, one shared activation; otherwise one activation row per slot and one output vector per slot.
template <bool GATE_UP>
__global__ void __launch_bounds__(kWarps * 32) fp8_slot_gemv_kernel(const uint32_t* __restrict__ indices, const uint8_t* __restrict__ x_codes,
                                                                    const float* __restrict__ x_scales, const uint8_t* const* w_table,
                                                                    const float* const* s_table, const uint8_t* const* w2_table,
                                                                    const float* const* s2_table, float* y_flat, float* const* y_table,
                                                                    uint32_t n, uint32_t k) {
    extern __shared__ float xs[];  // [k], swizzled
    const uint32_t slot = blockIdx.y;
    const uint32_t expert = __ldg(indices + slot);
    const uint8_t* x = GATE_UP ? x_codes : x_codes + static_cast<size_t>(slot) * k;
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) xs[xs_index(i / 32, i % 32)] = e4m3_value(__ldg(x + i));
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kWarps + (threadIdx.x >> 5);
    const uint32_t total = GATE_UP ? 2 * n : n;
    if (row >= total) return;
    const bool second = GATE_UP && row >= n;
    const uint32_t r = second ? row - n : row;
    const uint8_t* wrow = (second ? w2_table[expert] : w_table[expert]) + static_cast<size_t>(r) * k;
    float acc = 0.0f;
    for (uint32_t h = lane; h < k / 16; h += 32) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(wrow + h * 16));
        const uint32_t ww[4] = {q.x, q.y, q.z, q.w};
        const uint32_t c = h / 2, e0 = (h & 1) * 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 a = *reinterpret_cast<const float4*>(xs + xs_index(c, e0 + 4 * j));
            acc = fmaf(e4m3_value(static_cast<uint8_t>(ww[j])), a.x, acc);
            acc = fmaf(e4m3_value(static_cast<uint8_t>(ww[j] >> 8)), a.y, acc);
            acc = fmaf(e4m3_value(static_cast<uint8_t>(ww[j] >> 16)), a.z, acc);
            acc = fmaf(e4m3_value(static_cast<uint8_t>(ww[j] >> 24)), a.w, acc);
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) {
        const float sx = GATE_UP ? __ldg(x_scales) : __ldg(x_scales + slot);
        const float sw = __ldg((second ? s2_table[expert] : s_table[expert]) + r);
        const float v = __fmul_rn(__fmul_rn(acc, sx), sw);
        if (GATE_UP) y_flat[static_cast<size_t>(slot) * 2 * n + row] = v;
        else y_table[slot][row] = v;
    }
}

// Per slot: SiLU(gate) * up of the slot's [gate | up] row, one dynamic scale amax / 448 per slot (1 for an all-zero slot;
// non-finite values do not enter the maximum), E4M3 codes (non_gemm.cu:10241-10270).  One CTA per slot.
__global__ void __launch_bounds__(256) silu_quantize_fp8_slots_kernel(const float* __restrict__ gate_up, uint8_t* __restrict__ quantized,
                                                                      float* __restrict__ scales, uint32_t rows) {
    __shared__ float red[8];
    __shared__ float scale_sh;
    const uint32_t slot = blockIdx.x;
    const float* gate = gate_up + static_cast<size_t>(slot) * rows * 2;
    const float* up = gate + rows;
    float amax = 0.0f;
    for (uint32_t i = threadIdx.x; i < rows; i += 256) {
        const float g = __ldg(gate + i);
        const float v = __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), __ldg(up + i));
        if (isfinite(v)) amax = fmaxf(amax, fabsf(v));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
        const float sc = amax == 0.0f ? 1.0f : __fdiv_rn(amax, 448.0f);
        scales[slot] = sc;
        scale_sh = sc;
    }
    __syncthreads();
    const float sc = scale_sh;
    for (uint32_t i = threadIdx.x; i < rows; i += 256) {
        const float g = __ldg(gate + i);
        const float v = __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), __ldg(up + i));
        quantized[static_cast<size_t>(slot) * rows + i] = e4m3_satfinite(__fdiv_rn(v, sc));
    }
}

template <bool GATE_UP>
cudaError_t launch_fp8_slots(const uint32_t* indices, const uint8_t* x, const float* x_scales, const uint8_t* const* w, const float* const* s,
                             const uint8_t* const* w2, const float* const* s2, float* y_flat, float* const* y_table, uint32_t n, uint32_t k,
                             uint32_t slots, cudaStream_t stream) {
    if (k % 16 != 0) return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>((k + 31) / 32 * 32) * sizeof(float);
    if (smem > 200 * 1024) return cudaErrorNotSupported;
    if (smem > 48 * 1024) {
        cudaError_t st = cudaFuncSetAttribute(fp8_slot_gemv_kernel<GATE_UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (st != cudaSuccess) return st;
    }
    const uint32_t total = GATE_UP ? 2 * n : n;
    fp8_slot_gemv_kernel<GATE_UP><<<dim3((total + kWarps - 1) / kWarps, slots), kWarps * 32, smem, stream>>>(indices, x, x_scales, w, s, w2, s2,
                                                                                                              y_flat, y_table, n, k);
    return cudaGetLastError();
}

}  // namespace
}  // namespace eider

using namespace eider;

extern "C" {

// ---- FP8 W8A8 decode-side MoE slots (crates/eider-cuda/src/ffi.rs:3163-3196) ----------------------------------------------
cudaError_t infer_fp8_moe_grouped_gate_up_f32_on_stream(const uint32_t* indices, const uint8_t* input, const float* input_scale,
                                                        const uint8_t* const* gate_weights, const float* const* gate_scales,
                                                        const uint8_t* const* up_weights, const float* const* up_scales, float* output,
                                                        uint32_t rows, uint32_t cols, uint32_t slots, cudaStream_t stream) {
    if (!indices || !input || !input_scale || !gate_weights || !gate_scales || !up_weights || !up_scales || !output || rows == 0 ||
        cols == 0 || slots == 0)
        return cudaErrorInvalidValue;
    return launch_fp8_slots<true>(indices, input, input_scale, gate_weights, gate_scales, up_weights, up_scales, output, nullptr, rows, cols,
                                  slots, stream);
}

cudaError_t infer_moe_silu_quantize_fp8_slots_f32_on_stream(const float* gate_up, uint8_t* quantized, float* scales, uint32_t rows,
                                                            uint32_t slots, cudaStream_t stream) {
    if (!gate_up || !quantized || !scales || rows == 0 || slots == 0) return cudaErrorInvalidValue;
    silu_quantize_fp8_slots_kernel<<<slots, 256, 0, stream>>>(gate_up, quantized, scales, rows);
    return cudaGetLastError();
}

cudaError_t infer_fp8_moe_grouped_down_f32_on_stream(const uint32_t* indices, const uint8_t* inputs, const float* input_scales,
                                                     const uint8_t* const* weights, const float* const* weight_scales,
                                                     float* const* outputs, uint32_t rows, uint32_t cols, uint32_t slots,
                                                     cudaStream_t stream) {
    if (!indices || !inputs || !input_scales || !weights || !weight_scales || !outputs || rows == 0 || cols == 0 || slots == 0)
        return cudaErrorInvalidValue;
    return launch_fp8_slots<false>(indices, inputs, input_scales, weights, weight_scales, nullptr, nullptr, nullptr, outputs, rows, cols,
                                   slots, stream);
}


cudaError_t infer_nvfp4_w4a16_grouped_matvec_f32_on_stream(const uint32_t* indices, const float* input,
                                                           const uint8_t* const* packed_weight_table,
                                                           const uint8_t* const* weight_scale_table,
                                                           const float* weight_scale_2_table, float* const* output_table,
                                                           uint32_t table_len, uint32_t groups, uint32_t out_features,
                                                           uint32_t in_features, cudaStream_t stream) {
    if (!indices || !input || !packed_weight_table || !weight_scale_table || !weight_scale_2_table || !output_table)
        return cudaErrorInvalidValue;
    GroupedArgs a{indices, input, nullptr, packed_weight_table, weight_scale_table, weight_scale_2_table, 1.0f, output_table, nullptr,
                  table_len, groups, out_features, in_features};
    return launch_grouped<kSharedF32, false>(a, stream);
}

cudaError_t infer_nvfp4_w4a16_grouped_inputs_matvec_f32_on_stream(const uint32_t* indices, const float* const* input_table,
                                                                  const uint8_t* const* packed_weight_table,
                                                                  const uint8_t* const* weight_scale_table,
                                                                  const float* weight_scale_2_table, float* const* output_table,
                                                                  uint32_t table_len, uint32_t groups, uint32_t out_features,
                                                                  uint32_t in_features, cudaStream_t stream) {
    if (!indices || !input_table || !packed_weight_table || !weight_scale_table || !weight_scale_2_table || !output_table)
        return cudaErrorInvalidValue;
    GroupedArgs a{indices, input_table, nullptr, packed_weight_table, weight_scale_table, weight_scale_2_table, 1.0f, output_table,
                  nullptr, table_len, groups, out_features, in_features};
    return launch_grouped<kTableF32, false>(a, stream);
}

// crates/eider-cuda/src/ffi.rs:3333 (kernel non_gemm.cu:13640-13724): routes sorted by expert, every route with its own input
// and output vector found through the tables by its route id.  The reference shares each decoded weight among four routes
// of one expert; here every route's rows stream its expert's matrix with 128-bit loads (consecutive routes of one expert
// find it in L2), the products are the same exact f32 products and only the order of the additions differs.  `offsets` is
// required non-null as in the reference and is not read.
cudaError_t infer_nvfp4_w4a16_reuse_matvec_f32_on_stream(const uint32_t* sorted_routes, const uint32_t* sorted_experts,
                                                         const uint32_t* offsets, const float* const* inputs,
                                                         const uint8_t* const* weights, const uint8_t* const* scales,
                                                         const float* globals, float* const* outputs, uint32_t routes,
                                                         uint32_t experts, uint32_t out_features, uint32_t in_features,
                                                         cudaStream_t stream) {
    if (!sorted_routes || !sorted_experts || !offsets || !inputs || !weights || !scales || !globals || !outputs)
        return cudaErrorInvalidValue;
    GroupedArgs a{sorted_experts, inputs, nullptr, weights, scales, globals, 1.0f, outputs, nullptr, experts, routes, out_features, in_features};
    a.route_ids = sorted_routes;
    return launch_grouped<kTableF32, false>(a, stream);
}

// ---- W4A4 grouped GEMV (crates/eider-cuda/src/ffi.rs:589-642; crates/eider-cuda/native/cutlass_gemv.cu:277-880) ----------
// The plan only records the shape (the reference's holds CUTLASS workspace); it owns no device memory.
struct GroupedGemvPlan {
    uint32_t m, k, groups;
};

int infer_cutlass_fp4_grouped_gemv_f32_supported(uint32_t m, uint32_t k, uint32_t groups) {
    return (m > 0 && k > 0 && groups > 0 && k % 32 == 0 && static_cast<size_t>(k) * 4 <= 200 * 1024) ? 1 : 0;
}

void* infer_cutlass_fp4_grouped_gemv_f32_create(uint32_t m, uint32_t k, uint32_t groups) {
    if (!infer_cutlass_fp4_grouped_gemv_f32_supported(m, k, groups)) return nullptr;
    return new GroupedGemvPlan{m, k, groups};
}

void infer_cutlass_fp4_grouped_gemv_f32_destroy(void* plan) { delete static_cast<GroupedGemvPlan*>(plan); }

cudaError_t infer_cutlass_fp4_grouped_gemv_f32_indexed_a_tiled_scales_on_stream(void* raw, const uint32_t* indices,
                                                                                const uint8_t* const* a_values_table,
                                                                                const uint8_t* const* a_scales_table,
                                                                                const float* alpha_table, uint32_t table_len,
                                                                                const uint8_t* b_values, const uint8_t* b_scales,
                                                                                const float* c, float* const* d, cudaStream_t stream) {
    auto* plan = static_cast<GroupedGemvPlan*>(raw);
    (void)c;  // beta is 0 in the reference's call (cutlass_gemv.cu:640-648)
    if (!plan || !indices || !a_values_table || !a_scales_table || !alpha_table || !b_values || !b_scales || !d) return cudaErrorInvalidValue;
    GroupedArgs a{indices, b_values, b_scales, a_values_table, a_scales_table, alpha_table, 1.0f, d, nullptr, table_len, plan->groups,
                  plan->m, plan->k};
    return launch_grouped<kSharedNvfp4, true>(a, stream);
}

cudaError_t infer_cutlass_fp4_grouped_gemv_f32_indexed_a_on_stream(void* raw, const uint32_t* indices,
                                                                   const uint8_t* const* a_values_table,
                                                                   const uint8_t* const* a_scales_table, uint32_t table_len,
                                                                   const uint8_t* b_values, const uint8_t* b_scales, float* const* d,
                                                                   float alpha, cudaStream_t stream) {
    auto* plan = static_cast<GroupedGemvPlan*>(raw);
    if (!plan || !indices || !a_values_table || !a_scales_table || !b_values || !b_scales || !d) return cudaErrorInvalidValue;
    GroupedArgs a{indices, b_values, b_scales, a_values_table, a_scales_table, nullptr, alpha, d, nullptr, table_len, plan->groups, plan->m,
                  plan->k};
    return launch_grouped<kSharedNvfp4, true>(a, stream);
}

cudaError_t infer_cutlass_fp4_grouped_gemv_f32_contiguous_b_on_stream(void* raw, const uint8_t* const* a_values_table,
                                                                      const uint8_t* const* a_scales_table, const uint8_t* b_values,
                                                                      const uint8_t* b_scales, float* d, float alpha,
                                                                      cudaStream_t stream) {
    auto* plan = static_cast<GroupedGemvPlan*>(raw);
    if (!plan || !a_values_table || !a_scales_table || !b_values || !b_scales || !d) return cudaErrorInvalidValue;
    // group g multiplies table entry g with the shared activation row and writes d[g * m ...]
    GroupedArgs a{nullptr, b_values, b_scales, a_values_table, a_scales_table, nullptr, alpha, nullptr, d, plan->groups, plan->groups,
                  plan->m, plan->k};
    return launch_grouped<kSharedNvfp4, true>(a, stream);
}

cudaError_t infer_moe_silu_slots_f32_on_stream(const uint32_t* indices, const float* const* gate_up_table, float* const* output_table,
                                               const float* gate_up_alpha_table, uint32_t rows, uint32_t groups, cudaStream_t stream) {
    if (!indices || !gate_up_table || !output_table || !gate_up_alpha_table || rows == 0 || groups == 0) return cudaErrorInvalidValue;
    silu_slots_f32_kernel<<<dim3((rows + 255) / 256, groups), 256, 0, stream>>>(indices, gate_up_table, output_table, gate_up_alpha_table,
                                                                                rows);
    return cudaGetLastError();
}

cudaError_t infer_moe_silu_quantize_slots_nvfp4_simple_scales_on_stream(const uint32_t* indices, const float* const* gate_up_table,
                                                                        uint8_t* const* packed_table, uint8_t* const* scales_table,
                                                                        const float* input_scale_table,
                                                                        const float* gate_up_alpha_table, uint32_t rows,
                                                                        uint32_t groups, cudaStream_t stream) {
    if (!indices || !gate_up_table || !packed_table || !scales_table || !input_scale_table || !gate_up_alpha_table || rows == 0 ||
        groups == 0)
        return cudaErrorInvalidValue;
    const uint32_t blocks = (rows + 15) / 16;
    silu_quantize_slots_kernel<<<dim3((blocks + 127) / 128, groups), 128, 0, stream>>>(indices, gate_up_table, packed_table, scales_table,
                                                                                      input_scale_table, gate_up_alpha_table, rows);
    return cudaGetLastError();
}

cudaError_t infer_moe_weighted_accumulate_slots_f32_batch_on_stream(const uint32_t* indices, const float* route_weights,
                                                                    const float* const* inputs, const float* alpha_table,
                                                                    float* output, uint32_t rows, uint32_t len, uint32_t groups,
                                                                    cudaStream_t stream) {
    if (!indices || !route_weights || !inputs || !alpha_table || !output || rows == 0 || len == 0 || groups == 0)
        return cudaErrorInvalidValue;
    const size_t total = static_cast<size_t>(rows) * len;
    accumulate_slots_kernel<false><<<static_cast<uint32_t>((total + 255) / 256), 256, 0, stream>>>(
        indices, route_weights, inputs, alpha_table, nullptr, nullptr, nullptr, output, rows, len, groups);
    return cudaGetLastError();
}

cudaError_t infer_moe_weighted_accumulate_slots_f32_on_stream(const uint32_t* indices, const float* route_weights,
                                                              const float* const* inputs, const float* alpha_table, float* output,
                                                              uint32_t len, uint32_t groups, cudaStream_t stream) {
    return infer_moe_weighted_accumulate_slots_f32_batch_on_stream(indices, route_weights, inputs, alpha_table, output, 1, len, groups,
                                                                   stream);
}

cudaError_t infer_qwen36_ffn_finalize_routed_batch_f32_on_stream(const uint32_t* indices, const float* route_weights,
                                                                 const float* const* routed_outputs, const float* alpha_table,
                                                                 const float* shared_gate_logit, const float* shared_output,
                                                                 const float* residual, float* output, uint32_t rows, uint32_t cols,
                                                                 uint32_t groups_per_row, cudaStream_t stream) {
    if (!indices || !route_weights || !routed_outputs || !alpha_table || !shared_gate_logit || !shared_output || !residual || !output ||
        rows == 0 || cols == 0 || groups_per_row == 0)
        return cudaErrorInvalidValue;
    const size_t total = static_cast<size_t>(rows) * cols;
    accumulate_slots_kernel<true><<<static_cast<uint32_t>((total + 255) / 256), 256, 0, stream>>>(
        indices, route_weights, routed_outputs, alpha_table, shared_gate_logit, shared_output, residual, output, rows, cols, groups_per_row);
    return cudaGetLastError();
}

cudaError_t infer_qwen36_ffn_finalize_routed_f32_on_stream(const uint32_t* indices, const float* route_weights,
                                                           const float* const* routed_outputs, const float* alpha_table,
                                                           const float* shared_gate_logit, const float* shared_output,
                                                           const float* residual, float* output, uint32_t len, uint32_t groups,
                                                           cudaStream_t stream) {
    return infer_qwen36_ffn_finalize_routed_batch_f32_on_stream(indices, route_weights, routed_outputs, alpha_table, shared_gate_logit,
                                                                shared_output, residual, output, 1, len, groups, stream);
}

int eider_b200_moe_decode_step_supported(uint32_t experts, uint32_t top_k, uint32_t hidden, uint32_t inter) {
    return experts > 0 && experts <= kStepMaxExperts && top_k > 0 && top_k <= kStepMaxTopK && top_k <= experts && hidden > 0 &&
                   hidden % 128 == 0 && hidden <= kStepMaxHidden && inter > 0 && inter % 32 == 0 &&
                   (static_cast<uint64_t>(top_k) + 1) / 2 * ((static_cast<uint64_t>(inter) + 127) / 128) <= kStepMaxTasks
               ? 1
               : 0;
}

cudaError_t eider_b200_moe_decode_step_on_stream(const float* logits, const float* x, const uint8_t* const* gate_up_weights,
                                                 const uint8_t* const* gate_up_scales, const float* gate_up_alpha,
                                                 const uint8_t* const* down_weights, const uint8_t* const* down_scales,
                                                 const float* down_alpha, const float* shared_gate_logit, const float* shared_output,
                                                 const float* residual, uint32_t* indices, float* weights, uint16_t* act, float* output,
                                                 uint32_t experts, uint32_t top_k, uint32_t hidden, uint32_t inter, cudaStream_t stream) {
    if (!logits || !x || !gate_up_weights || !gate_up_scales || !gate_up_alpha || !down_weights || !down_scales || !down_alpha ||
        !shared_gate_logit || !shared_output || !residual || !indices || !weights || !act || !output ||
        ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(act)) & 15) != 0)
        return cudaErrorInvalidValue;
    if (!eider_b200_moe_decode_step_supported(experts, top_k, hidden, inter)) return cudaErrorNotSupported;
    MoeStepArgs a{};
    a.logits = logits;
    a.x = x;
    a.w_table = gate_up_weights;
    a.s_table = gate_up_scales;
    a.g_table = gate_up_alpha;
    a.indices = indices;
    a.weights = weights;
    a.act = act;
    a.experts = experts;
    a.top_k = top_k;
    a.hidden = hidden;
    a.inter = inter;
    cudaError_t st = launch_step(moe_step_gate_up_kernel, top_k * (inter / 16), static_cast<size_t>(hidden) * 6, a, stream);  // (at most 24 KB of shared memory beside 9 KB of static)
    if (st != cudaSuccess) return st;
    a.w_table = down_weights;
    a.s_table = down_scales;
    a.g_table = down_alpha;
    a.shared_gate_logit = shared_gate_logit;
    a.shared_output = shared_output;
    a.residual = residual;
    a.out = output;
    const uint32_t tasks = (top_k + 1) / 2 * ((inter + 127) / 128);
    if (tasks <= 3 * kStepWarps) return launch_step(moe_step_down_kernel<3>, hidden / 8, 0, a, stream);
    return launch_step(moe_step_down_kernel<6>, hidden / 8, 0, a, stream);
}

/* crates/eider-cuda/src/ffi.rs:3473 (kernels non_gemm.cu:13423-13482, 8287-8328): arg-max over the lm-head logits without
 * writing them.  scratch_value / scratch_index hold scratch_len per-CTA candidates; any scratch_len >= 1 works here (the
 * CTAs walk the rows), up to 1024 entries are used.  warps_per_block is the reference's launch width and must be one of
 * its values (4, 8, 16, 32); this implementation needs in_features % 32 == 0. */
cudaError_t infer_nvfp4_w4a16_top1_f32_on_stream(const float* input, const uint8_t* packed_weight, const uint8_t* weight_scale,
                                                 float* scratch_value, uint32_t* scratch_index, uint32_t scratch_len,
                                                 uint32_t* out_index, float* out_value, uint32_t out_features, uint32_t in_features,
                                                 float weight_scale_2, uint32_t warps_per_block, cudaStream_t stream) {
    if (!input || !packed_weight || !weight_scale || !scratch_value || !scratch_index || !out_index || !out_value ||
        out_features == 0 || in_features == 0 || in_features % 32 != 0 || !isfinite(weight_scale_2) || scratch_len == 0 ||
        (warps_per_block != 4 && warps_per_block != 8 && warps_per_block != 16 && warps_per_block != 32))
        return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(in_features) * sizeof(float);
    if (smem > 200 * 1024) return cudaErrorNotSupported;
    if (smem > 48 * 1024) {
        cudaError_t st = cudaFuncSetAttribute(top1_pass1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (st != cudaSuccess) return st;
    }
    uint32_t blocks = (out_features + kWarps - 1) / kWarps;
    if (blocks > 1024) blocks = 1024;
    if (blocks > scratch_len) blocks = scratch_len;
    top1_pass1_kernel<<<blocks, kWarps * 32, smem, stream>>>(input, packed_weight, weight_scale, weight_scale_2, out_features, in_features,
                                                             scratch_value, scratch_index);
    cudaError_t st = cudaGetLastError();
    if (st != cudaSuccess) return st;
    top1_pass2_kernel<<<1, 256, 0, stream>>>(scratch_value, scratch_index, blocks, out_index, out_value);
    return cudaGetLastError();
}

}  // extern "C"

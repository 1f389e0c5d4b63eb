// A 16-element block of a row in registers and its quotients: shared by the activation quantizers and the routed-MoE ones.
#pragma once

#include "common.cuh"

namespace eider {
namespace {

// Two quotients at a time, correctly rounded from r = RN(1 / d) when nothing over- or underflows on the way (div_rn), in three
// packed instructions.  The operand is -x and the reciprocal -r, so that the remainder comes out with the sign that keeps
// the sign of a zero: x = -0: q0 = (+0)(-r) = -0, e = (-0) d + (+0) = +0, q = (+0)(-r) + (-0) = -0.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 div2_negated(f32x2 minus_x, f32x2 d, f32x2 minus_r) {  // -> x / d
    const f32x2 q0 = mul2(minus_x, minus_r);
    return fma2(fma2(q0, d, minus_x), minus_r, q0);
}
// The same from x, with the opposite sign: -(x / d) (x = -0: q0 = +0, e = +0, result +0).
__device__ __forceinline__ f32x2 minus_div2(f32x2 x, f32x2 d, f32x2 minus_r) {
    const f32x2 q0 = mul2(x, minus_r);
    return fma2(fma2(q0, d, x), minus_r, q0);
}
__device__ __forceinline__ uint32_t e2m1_byte(f32x2 v) {
    const float2 f = unpack2(v);
    return e2m1x2_code(f.x, f.y);
}
// RN(1 / s) for a positive E4M3 value: a Newton-Raphson step on the approximate reciprocal (every one of the 126 values is
// tested with quotients on the rounding boundaries).
__device__ __forceinline__ float e4m3_reciprocal(float s) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    return fmaf(r, fmaf(-s, r, 1.0f), r);
}
__device__ __forceinline__ float e4m3_to_float(uint8_t code) {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(code), __NV_E4M3);
    return __half2float(__half(__half_raw{h.x}));
}

// Sixteen consecutive elements as they lie in memory.
template <typename T> struct Block16;
template <> struct Block16<uint16_t> {
    uint4 q[2];
    __device__ __forceinline__ void load(const uint16_t* p) {
        q[0] = __ldg(reinterpret_cast<const uint4*>(p));
        q[1] = __ldg(reinterpret_cast<const uint4*>(p) + 1);
    }
    __device__ __forceinline__ uint32_t word(int j) const {
        const uint4& w = q[j / 4];
        return j % 4 == 0 ? w.x : j % 4 == 1 ? w.y : j % 4 == 2 ? w.z : w.w;
    }
    __device__ __forceinline__ float get(int i) const {
        return __uint_as_float(i % 2 == 0 ? word(i / 2) << 16 : word(i / 2) & 0xffff0000u);
    }
    __device__ __forceinline__ f32x2 pair(int j) const { return pack2(get(2 * j), get(2 * j + 1)); }
    __device__ __forceinline__ f32x2 minus_pair(int j) const {
        const uint32_t w = word(j) ^ 0x80008000u;
        return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    }
    // largest absolute value, NaNs dropped (two elements at a time)
    __device__ __forceinline__ float amax() const {
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t a = word(j) & 0x7fff7fffu;
            asm("max.bf16x2 %0, %0, %1;" : "+r"(m) : "r"(a));
        }
        return fmaxf(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u));
    }
};
template <> struct Block16<float> {
    float4 q[4];
    __device__ __forceinline__ void load(const float* p) {
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = __ldg(reinterpret_cast<const float4*>(p) + j);
    }
    __device__ __forceinline__ float get(int i) const {
        const float4& f = q[i / 4];
        return i % 4 == 0 ? f.x : i % 4 == 1 ? f.y : i % 4 == 2 ? f.z : f.w;
    }
    __device__ __forceinline__ f32x2 pair(int j) const { return pack2(get(2 * j), get(2 * j + 1)); }
    __device__ __forceinline__ f32x2 minus_pair(int j) const { return pack2(-get(2 * j), -get(2 * j + 1)); }
    __device__ __forceinline__ float amax() const {
        float m = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(get(i)));
        return m;
    }
};
template <typename T> __device__ __forceinline__ float finite_amax(const Block16<T>& v) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = fmaxf(m, finite_abs(v.get(i)));
    return m;
}

// Eight bytes of codes, 4-byte aligned.
__device__ __forceinline__ void store_codes(uint8_t* out, size_t offset, const uint32_t (&w)[2]) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(out + offset);
    if ((reinterpret_cast<uintptr_t>(out) & 7) == 0) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    } else {
        dst[0] = w[0];
        dst[1] = w[1];
    }
}

// A block without an infinity, as it is (scale 1): codes and scale byte.
template <typename T> __device__ __forceinline__ uint8_t quantize_unit_block(const Block16<T>& v, float amax, uint32_t (&w)[2]) {
    const uint8_t sc = amax == 0.0f ? 0 : ue4m3_code(div6_rn(amax));
    w[0] = w[1] = 0u;
    if (sc != 0) {
        const float sv = e4m3_to_float(sc), r = -e4m3_reciprocal(sv);
        const f32x2 d2 = pack2(sv, sv), r2 = pack2(r, r);
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j / 4] |= e2m1_byte(div2_negated(v.minus_pair(j), d2, r2)) << ((j % 4) * 8);
    }
    return sc;
}

// A kernel that starts with griddepcontrol.wait, launched so that its prologue overlaps the kernel before it.
template <typename Kernel, typename... Args>
cudaError_t launch_dependent(Kernel kernel, dim3 grid, uint32_t threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace
}  // namespace eider

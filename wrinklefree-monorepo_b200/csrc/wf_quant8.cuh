// Per-token int8 quantization of values held in registers eight at a time, as they lie in memory — shared by the
// quantization kernels and the kernels that quantize their own input.
#pragma once

#include "wf_common.cuh"

namespace wf {

// 8 consecutive elements as they lie in memory (zeros when !ok), and their values
template <int DT>
struct Raw8 {
    static constexpr int V = DT == WF_F32 ? 2 : 1;
    uint4 v[V];
};
template <int DT>
__device__ __forceinline__ void load_raw8(const void* base, int64_t elem_off, bool ok, Raw8<DT>& r) {
    const char* p = static_cast<const char*>(base) + elem_off * (DT == WF_F32 ? 4 : 2);
#pragma unroll
    for (int j = 0; j < Raw8<DT>::V; ++j)  // predicated and not branched around: a thread's loads go out back to back
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %5, 0;\n mov.u32 %0, 0;\n mov.u32 %1, 0;\n mov.u32 %2, 0;\n mov.u32 %3, 0;\n"
            " @p ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n}\n"
            : "=&r"(r.v[j].x), "=&r"(r.v[j].y), "=&r"(r.v[j].z), "=&r"(r.v[j].w)
            : "l"(p + 16 * j), "r"(static_cast<int>(ok))
            : "memory");
}
template <int DT>
__device__ __forceinline__ void values8(const Raw8<DT>& r, float (&f)[8]) {
    if constexpr (DT == WF_F32) {
        f[0] = __uint_as_float(r.v[0].x); f[1] = __uint_as_float(r.v[0].y); f[2] = __uint_as_float(r.v[0].z); f[3] = __uint_as_float(r.v[0].w);
        f[4] = __uint_as_float(r.v[1].x); f[5] = __uint_as_float(r.v[1].y); f[6] = __uint_as_float(r.v[1].z); f[7] = __uint_as_float(r.v[1].w);
    } else {
        const uint32_t w[4] = {r.v[0].x, r.v[0].y, r.v[0].z, r.v[0].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if constexpr (DT == WF_BF16) {
                f[2 * i] = __uint_as_float(w[i] << 16);
                f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
            } else {
                const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                f[2 * i] = v.x;
                f[2 * i + 1] = v.y;
            }
        }
    }
}

// ---- the quantization of a row that is held as Raw8, at about four instructions per element (it was fourteen, one of them
// the quarter-rate conversion to int, and bound the kernel at 58 % of the copy bandwidth):
//   * the absolute maximum over bit patterns (non-negative values order like theirs), two 16-bit elements at a time;
//   * the product with the multiplier as one packed multiplication, which rounds once like the fp32 product of two 16-bit
//     values (exact) rounded to the type;
//   * the rounding to an integer as an addition of 1.5 * 2^23 (half to even), whose lowest byte is the int8.  Only the upper
//     bound of the clamp is applied: the multiplier is 127 / max with two roundings of at most 2^-8 each, so |x * s| is below
//     127 * (1 + 2^-8)^2 = 127.995 and its own rounding ends at 128 at most, which is in range with a minus sign.
// That needs a maximum whose reciprocal is a normal number of the type: bf16 reciprocals of more than 2^126 are off by up to
// 1.6 %, x * s reaches -129 there and would wrap to +127.  (fp16 reciprocals of more than 2^14 are off by 2^-9: 127.4.)  Rows
// with such a maximum, an infinity or a NaN, and a multiplier that is not finite, take quantize_one instead.
template <int DT>
__device__ __forceinline__ uint32_t max_bits8(const Raw8<DT>& r, uint32_t mx) {
#pragma unroll
    for (int j = 0; j < Raw8<DT>::V; ++j) {
        const uint32_t w[4] = {r.v[j].x, r.v[j].y, r.v[j].z, r.v[j].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) mx = DT == WF_F32 ? max(mx, w[i] & 0x7fffffffu) : __vmaxu2(mx, w[i] & 0x7fff7fffu);
    }
    return mx;
}
// over the warp, as one bit pattern of the type
template <int DT>
__device__ __forceinline__ uint32_t warp_max_bits(uint32_t mx) {
    if constexpr (DT != WF_F32) mx = max(mx & 0xffffu, mx >> 16);
    return __reduce_max_sync(0xffffffffu, mx);
}
template <int DT>
__device__ __forceinline__ bool fast_bits(uint32_t bits) {  // the absolute maximum is one that quantize8_fast takes
    return bits < (DT == WF_F32 ? 0x7f800000u : (DT == WF_BF16 ? 0x7e81u : 0x7c00u));
}
template <int DT>
__device__ __forceinline__ float bits_value(uint32_t bits) {
    if constexpr (DT == WF_F32) return __uint_as_float(bits);
    if constexpr (DT == WF_BF16) return __uint_as_float(bits << 16);
    return __half2float(__ushort_as_half(static_cast<unsigned short>(bits)));
}
constexpr float RINT_MAGIC = 12582912.0f;  // 1.5 * 2^23
// two values (already rounded products, at most 127) to two bytes in the low half
__device__ __forceinline__ uint32_t two_bytes(float a, float b) {
    return __byte_perm(__float_as_uint(__fadd_rn(a, RINT_MAGIC)), __float_as_uint(__fadd_rn(b, RINT_MAGIC)), 0x0040);
}
template <int DT>
__device__ __forceinline__ uint2 quantize8_fast(const Raw8<DT>& r, float s) {
    uint32_t h[4];  // pairs of bytes
    if constexpr (DT == WF_F32) {
        float f[8];
        values8<DT>(r, f);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = two_bytes(fminf(__fmul_rn(f[2 * i], s), 127.f), fminf(__fmul_rn(f[2 * i + 1], s), 127.f));
    } else {
        const uint32_t w[4] = {r.v[0].x, r.v[0].y, r.v[0].z, r.v[0].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if constexpr (DT == WF_BF16) {
                const __nv_bfloat162 v = __hmin2(__hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&w[i]), __float2bfloat162_rn(s)), __float2bfloat162_rn(127.f));
                const uint32_t u = *reinterpret_cast<const uint32_t*>(&v);
                h[i] = two_bytes(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
            } else {
                const float2 v = __half22float2(__hmin2(__hmul2_rn(*reinterpret_cast<const __half2*>(&w[i]), __float2half2_rn(s)), __float2half2_rn(127.f)));
                h[i] = two_bytes(v.x, v.y);
            }
        }
    }
    return make_uint2(__byte_perm(h[0], h[1], 0x5410), __byte_perm(h[2], h[3], 0x5410));
}
template <int DT>
__device__ __noinline__ uint2 quantize8_any(const Raw8<DT> r, float s) {
    float f[8];
    values8<DT>(r, f);
    uint32_t w[2] = {0, 0};
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e >> 2] |= static_cast<uint32_t>(quantize_one<DT>(f[e], s) & 0xff) << (8 * (e & 3));
    return make_uint2(w[0], w[1]);
}
template <int DT>
__device__ __forceinline__ float max_abs8(const Raw8<DT>& r, float mx) {  // a NaN counts for nothing
    float f[8];
    values8<DT>(r, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) mx = fmaxf(mx, fabsf(f[e]));
    return mx;
}
__device__ __forceinline__ int sum_bytes(uint2 w, int sum) {
    return __dp4a(static_cast<int>(w.x), 0x01010101, __dp4a(static_cast<int>(w.y), 0x01010101, sum));
}

}  // namespace wf

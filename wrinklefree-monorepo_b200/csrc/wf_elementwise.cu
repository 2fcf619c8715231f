// Small fused elementwise kernels around the BitLinear projections of a decoder layer (bf16 tensors):
// residual add + RMSNorm, RoPE + KV-cache write, gate activation x up.  They replace chains of framework
// kernels in the decode step.  With one token per sequence they are pure latency: every tensor is read with
// 16-byte loads that are all in flight at once, rows stay in registers between the reduction and the
// normalisation, and every kernel can be chained to its neighbours with a programmatic dependency (it lets the
// next kernel start at once and itself reads nothing that the previous kernel writes before it has waited).
#include "wf_common.cuh"
#include "wf_rowquant.cuh"

namespace wf {

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_bf(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float round_bf(float v) { return bf(__float2bfloat16_rn(v)); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

constexpr int NORM_THREADS = 512;
constexpr int NORM_CHUNKS = 4;  // 8-element chunks per thread held in registers: rows up to 16384 elements

// h[m, :] += delta[m, :] (when delta != nullptr); y[m, :] = h * rsqrt(mean(h^2) + eps) * w.  One block per row.
// VEC: K % 8 == 0 and K <= NORM_THREADS * NORM_CHUNKS * 8, the row stays in registers; else two passes over global memory.
// With `q` (VEC only) the normalised row is also quantized to int8 per token, with the arithmetic of the stand-alone
// quantization kernel on the bf16 values (absmax, multiplier 127 / max rounded like torch's, round half to even): the
// projections that follow read q and q_scale and no kernel stands between the norm and them; y may then be null.
template <bool VEC>
__global__ void __launch_bounds__(NORM_THREADS) add_rmsnorm_kernel(__nv_bfloat16* __restrict__ h, const __nv_bfloat16* delta,
                                                                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                                   int K, float eps, int8_t* __restrict__ q, float* __restrict__ q_scale,
                                                                   float q_eps) {
    __shared__ float sh[NORM_THREADS / 32];
    pdl_trigger();
    const int64_t m = blockIdx.x;
    const int tid = threadIdx.x;
    float ss = 0.f;
    uint4 hv[NORM_CHUNKS], wv[NORM_CHUNKS];
    if constexpr (VEC) {
        const int chunks = K >> 3;
        // the norm weights do not depend on the previous kernel
#pragma unroll
        for (int c = 0; c < NORM_CHUNKS; ++c) {
            const int i = tid + c * NORM_THREADS;
            if (i < chunks) wv[c] = __ldg(reinterpret_cast<const uint4*>(w) + i);
        }
        pdl_wait();
        uint4 dv[NORM_CHUNKS];
        uint4* hrow = reinterpret_cast<uint4*>(h + m * K);
#pragma unroll
        for (int c = 0; c < NORM_CHUNKS; ++c) {
            const int i = tid + c * NORM_THREADS;
            if (i < chunks) {
                hv[c] = hrow[i];
                if (delta) dv[c] = ld16_chained(delta + m * K + 8 * static_cast<int64_t>(i));
            }
        }
#pragma unroll
        for (int c = 0; c < NORM_CHUNKS; ++c) {
            const int i = tid + c * NORM_THREADS;
            if (i < chunks) {
                uint32_t a[4] = {hv[c].x, hv[c].y, hv[c].z, hv[c].w};
                if (delta) {
                    const uint32_t d[4] = {dv[c].x, dv[c].y, dv[c].z, dv[c].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)  // the residual stream stays bf16
                        a[e] = pack_bf(bf_lo(a[e]) + bf_lo(d[e]), bf_hi(a[e]) + bf_hi(d[e]));
                    hv[c] = make_uint4(a[0], a[1], a[2], a[3]);
                    hrow[i] = hv[c];
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) ss += bf_lo(a[e]) * bf_lo(a[e]) + bf_hi(a[e]) * bf_hi(a[e]);
            }
        }
    } else {
        pdl_wait();
        for (int k = tid * 2; k < K; k += NORM_THREADS * 2) {
            __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(h + m * K + k);
            if (delta) {
                const __nv_bfloat162 d = *reinterpret_cast<const __nv_bfloat162*>(delta + m * K + k);
                a = __floats2bfloat162_rn(bf(a.x) + bf(d.x), bf(a.y) + bf(d.y));
                *reinterpret_cast<__nv_bfloat162*>(h + m * K + k) = a;
            }
            ss += bf(a.x) * bf(a.x) + bf(a.y) * bf(a.y);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) sh[tid >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < NORM_THREADS / 32; ++i) tot += sh[i];
    const float r = rsqrtf(tot / static_cast<float>(K) + eps);
    // normalise in fp32, round to bf16, then scale by the bf16 weight (the order of the unfused operator chain)
    if constexpr (VEC) {
        const int chunks = K >> 3;
        uint4* yrow = y ? reinterpret_cast<uint4*>(y + m * K) : nullptr;
        uint32_t o[NORM_CHUNKS][4];
        float mx = 0.f;
#pragma unroll
        for (int c = 0; c < NORM_CHUNKS; ++c) {
            const int i = tid + c * NORM_THREADS;
            if (i < chunks) {
                const uint32_t a[4] = {hv[c].x, hv[c].y, hv[c].z, hv[c].w};
                const uint32_t g[4] = {wv[c].x, wv[c].y, wv[c].z, wv[c].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    o[c][e] = pack_bf(round_bf(bf_lo(a[e]) * r) * bf_lo(g[e]), round_bf(bf_hi(a[e]) * r) * bf_hi(g[e]));
                    mx = fmaxf(mx, fmaxf(fabsf(bf_lo(o[c][e])), fabsf(bf_hi(o[c][e]))));
                }
                if (y) yrow[i] = make_uint4(o[c][0], o[c][1], o[c][2], o[c][3]);
            }
        }
        if (q) {
            quantize_row_bf16<NORM_THREADS, NORM_CHUNKS>(o, mx, chunks, tid, sh, q + m * K, q_scale + m, q_eps);
        }
    } else {
        for (int k = tid * 2; k < K; k += NORM_THREADS * 2) {
            const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(h + m * K + k);
            const __nv_bfloat162 g = *reinterpret_cast<const __nv_bfloat162*>(w + k);
            *reinterpret_cast<__nv_bfloat162*>(y + m * K + k) =
                __floats2bfloat162_rn(round_bf(bf(a.x) * r) * bf(g.x), round_bf(bf(a.y) * r) * bf(g.y));
        }
    }
}

// Decode-step RoPE + cache write for one new token per sequence.  One block per (sequence, head): query heads are
// rotated in place; key heads are rotated and written to kcache[b, head, slot, :], and the same block copies the
// value head to vcache[b, head, slot, :].  cos/sin [T, D/2] fp32; the position *pos is read on the device
// (the caller keeps it below T; it is reduced modulo T only so that a stray value stays inside the tables).
__global__ void rope_kv_kernel(__nv_bfloat16* __restrict__ q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                               const float* __restrict__ cosv, const float* __restrict__ sinv, const int64_t* pos,
                               __nv_bfloat16* __restrict__ kcache, __nv_bfloat16* __restrict__ vcache, int nq, int nkv, int D, int T) {
    pdl_trigger();
    const int heads = nq + nkv, half = D / 2;
    const int b = blockIdx.x / heads, head = blockIdx.x % heads;
    pdl_wait();
    const int slot = static_cast<int>(*pos % T);
    const float* c = cosv + static_cast<int64_t>(slot) * half;
    const float* s = sinv + static_cast<int64_t>(slot) * half;
    if (head < nq) {
        __nv_bfloat16* p = q + (static_cast<int64_t>(b) * nq + head) * D;
        for (int j = threadIdx.x; j < half; j += blockDim.x) {
            const float x1 = bf(p[j]), x2 = bf(p[j + half]), cj = c[j], sj = s[j];
            p[j] = __float2bfloat16_rn(x1 * cj - x2 * sj);
            p[j + half] = __float2bfloat16_rn(x2 * cj + x1 * sj);
        }
    } else {
        const int hk = head - nq;
        const __nv_bfloat16* p = k + (static_cast<int64_t>(b) * nkv + hk) * D;
        const __nv_bfloat16* pv = v + (static_cast<int64_t>(b) * nkv + hk) * D;
        const int64_t at = ((static_cast<int64_t>(b) * nkv + hk) * T + slot) * D;
        for (int j = threadIdx.x; j < half; j += blockDim.x) {
            const float x1 = bf(p[j]), x2 = bf(p[j + half]), cj = c[j], sj = s[j];
            const __nv_bfloat16 v1 = pv[j], v2 = pv[j + half];
            kcache[at + j] = __float2bfloat16_rn(x1 * cj - x2 * sj);
            kcache[at + j + half] = __float2bfloat16_rn(x2 * cj + x1 * sj);
            vcache[at + j] = v1;
            vcache[at + j + half] = v2;
        }
    }
}

// RoPE + cache write of a whole prompt: token (b, s) at position s.  Query heads are rotated in place, key heads rotated into
// kcache[b, head, s, :], value heads copied to vcache[b, head, s, :].  One thread per 8 + 8 values of a head (the two halves that
// rotate into each other).  Every product and difference is rounded by itself, as the operator chain it stands for does (two
// slices, four products, a difference, a sum, a concatenation, a conversion, for q and for k, and two copies into the
// cache: 20 launches of about 4 us each on the host).
__global__ void __launch_bounds__(256) rope_kv_prompt_kernel(__nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                                                             const float* __restrict__ cosv, const float* __restrict__ sinv,
                                                             __nv_bfloat16* __restrict__ kcache, __nv_bfloat16* __restrict__ vcache, int S, int nq, int nkv,
                                                             int D, int T, int64_t ldq, int64_t ldkv, int64_t total) {
    pdl_trigger();
    pdl_wait();
    const int half = D / 2, parts = half / 8, heads = nq + nkv;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int part = static_cast<int>(i % parts);
        const int64_t hr = i / parts;
        const int head = static_cast<int>(hr % heads);
        const int64_t row = hr / heads;  // b * S + s
        const int s = static_cast<int>(row % S);
        const int64_t b = row / S;
        const bool is_q = head < nq;
        const int hk = head - nq;
        const __nv_bfloat16* src = is_q ? q + row * ldq + head * D : k + row * ldkv + hk * D;
        __nv_bfloat16* dst = is_q ? q + row * ldq + head * D : kcache + ((b * nkv + hk) * T + s) * D;
        const uint4 lo = ld16_chained(src + part * 8), hi = ld16_chained(src + half + part * 8);
        const uint32_t a[4] = {lo.x, lo.y, lo.z, lo.w}, c[4] = {hi.x, hi.y, hi.z, hi.w};
        const float4* cp = reinterpret_cast<const float4*>(cosv + static_cast<int64_t>(s) * half + part * 8);
        const float4* sp = reinterpret_cast<const float4*>(sinv + static_cast<int64_t>(s) * half + part * 8);
        const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), s0 = __ldg(sp), s1 = __ldg(sp + 1);
        const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        uint32_t o0[4], o1[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float r0[2], r1[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float x1 = u ? bf_hi(a[e]) : bf_lo(a[e]), x2 = u ? bf_hi(c[e]) : bf_lo(c[e]);
                r0[u] = __fsub_rn(__fmul_rn(x1, cs[2 * e + u]), __fmul_rn(x2, sn[2 * e + u]));
                r1[u] = __fadd_rn(__fmul_rn(x2, cs[2 * e + u]), __fmul_rn(x1, sn[2 * e + u]));
            }
            o0[e] = pack_bf(r0[0], r0[1]);
            o1[e] = pack_bf(r1[0], r1[1]);
        }
        *reinterpret_cast<uint4*>(dst + part * 8) = make_uint4(o0[0], o0[1], o0[2], o0[3]);
        *reinterpret_cast<uint4*>(dst + half + part * 8) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
        if (!is_q) {
            const __nv_bfloat16* pv = v + row * ldkv + hk * D;
            __nv_bfloat16* dv = vcache + ((b * nkv + hk) * T + s) * D;
            *reinterpret_cast<uint4*>(dv + part * 8) = ld16_chained(pv + part * 8);
            *reinterpret_cast<uint4*>(dv + half + part * 8) = ld16_chained(pv + half + part * 8);
        }
    }
}

// out = act(g) * u, act = SiLU (mode 0) or ReLU^2 (mode 1); intermediate rounded to bf16 like the unfused chain.
__device__ __forceinline__ float act_one(float a, int mode) {
    float t;
    if (mode == 0) {
        t = a / (1.0f + __expf(-a));
    } else {
        const float rl = round_bf(fmaxf(a, 0.f));
        t = rl * rl;
    }
    return round_bf(t);
}
__global__ void __launch_bounds__(256) act_mul_kernel(const __nv_bfloat16* g, const __nv_bfloat16* u,
                                                      __nv_bfloat16* __restrict__ out, int64_t n, int mode) {
    pdl_trigger();
    pdl_wait();
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t n8 = n >> 3;
    for (int64_t i = tid; i < n8; i += stride) {
        const uint4 a = ld16_chained(g + 8 * i), b = ld16_chained(u + 8 * i);
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            o[e] = pack_bf(act_one(bf_lo(av[e]), mode) * bf_lo(bv[e]), act_one(bf_hi(av[e]), mode) * bf_hi(bv[e]));
        reinterpret_cast<uint4*>(out)[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
    for (int64_t i = n8 * 8 + tid; i < n; i += stride)  // the tail of a length that is not a multiple of 8
        out[i] = __float2bfloat16_rn(act_one(bf(g[i]), mode) * bf(u[i]));
}

// act(g) * u of one token row per block, quantized to int8 per token on the way (and written as bf16 when `out` is given):
// the activation in front of down_proj together with the quantization that projection would otherwise run itself.
constexpr int AMQ_THREADS = 512;
constexpr int AMQ_CHUNKS = 4;  // rows up to 16384 elements
__global__ void __launch_bounds__(AMQ_THREADS) act_mul_quant_kernel(const __nv_bfloat16* g, const __nv_bfloat16* u,
                                                                    __nv_bfloat16* __restrict__ out, int8_t* __restrict__ q,
                                                                    float* __restrict__ q_scale, int I, int64_t ldg, int mode, float q_eps) {
    __shared__ float sh[AMQ_THREADS / 32];
    pdl_trigger();
    pdl_wait();
    const int64_t m = blockIdx.x;
    const int tid = threadIdx.x, chunks = I >> 3;
    uint32_t o[AMQ_CHUNKS][4];
    float mx = 0.f;
#pragma unroll
    for (int c = 0; c < AMQ_CHUNKS; ++c) {
        const int i = tid + c * AMQ_THREADS;
        if (i < chunks) {
            const uint4 a = ld16_chained(g + m * ldg + 8 * i), b = ld16_chained(u + m * ldg + 8 * i);
            const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[c][e] = pack_bf(act_one(bf_lo(av[e]), mode) * bf_lo(bv[e]), act_one(bf_hi(av[e]), mode) * bf_hi(bv[e]));
                mx = fmaxf(mx, fmaxf(fabsf(bf_lo(o[c][e])), fabsf(bf_hi(o[c][e]))));
            }
            if (out) reinterpret_cast<uint4*>(out + m * I)[i] = make_uint4(o[c][0], o[c][1], o[c][2], o[c][3]);
        }
    }
    quantize_row_bf16<AMQ_THREADS, AMQ_CHUNKS>(o, mx, chunks, tid, sh, q + m * I, q_scale + m, q_eps);
}

// Greedy choice of a decode step: one block per row, 16 bytes per load, several loads in flight.  A framework reduction of 49152 values
// took 13.6 us, this takes what reading 98 KB through one SM takes.  A value's key orders like the value (bf16 bits made
// monotone, -0 like +0, every NaN above infinity); ties go to the lowest index.
constexpr int AM_THREADS = 1024;
__device__ __forceinline__ uint32_t argmax_key(uint32_t b) {
    if ((b & 0x7fffu) > 0x7f80u) return 0x1ffffu;
    if (b == 0x8000u) b = 0;
    return (b & 0x8000u) ? 0xffffu - b : b + 0x8000u;
}
__global__ void __launch_bounds__(AM_THREADS) argmax_kernel(const __nv_bfloat16* x, int64_t ld, int V, int vec, int64_t* __restrict__ out, int64_t* pos) {
    __shared__ unsigned long long sh[AM_THREADS / 32];
    pdl_trigger();
    pdl_wait();
    const __nv_bfloat16* row = x + static_cast<int64_t>(blockIdx.x) * ld;
    const int tid = threadIdx.x;
    uint32_t key = 0;
    int at = 0x7fffffff;
    auto take = [&](uint32_t bits, int i) {  // indices of a thread ascend: only a larger key replaces
        const uint32_t k = argmax_key(bits);
        if (k > key || at == 0x7fffffff) {
            key = k;
            at = i;
        }
    };
    const int n8 = vec ? V >> 3 : 0;
    constexpr int U = 4;
    for (int i0 = tid; i0 < n8; i0 += U * AM_THREADS) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * AM_THREADS < n8) v[u] = ld16_chained(row + 8 * static_cast<int64_t>(i0 + u * AM_THREADS));
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u * AM_THREADS < n8) {
                const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    take(w[e] & 0xffffu, 8 * (i0 + u * AM_THREADS) + 2 * e);
                    take(w[e] >> 16, 8 * (i0 + u * AM_THREADS) + 2 * e + 1);
                }
            }
        }
    }
    for (int i = 8 * n8 + tid; i < V; i += AM_THREADS) take(*reinterpret_cast<const volatile unsigned short*>(row + i), i);
    unsigned long long best = (static_cast<unsigned long long>(key) << 32) | (0xffffffffu - static_cast<uint32_t>(at));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((tid & 31) == 0) sh[tid >> 5] = best;
    __syncthreads();
    if (tid < 32) {
        best = sh[tid];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
        if (tid == 0) {
            out[blockIdx.x] = static_cast<int64_t>(0xffffffffu - static_cast<uint32_t>(best));
            if (pos && blockIdx.x == 0) *pos += 1;
        }
    }
}

template <typename... KArgs, typename... Args>
static cudaError_t launch(void (*kernel)(KArgs...), unsigned grid, unsigned block, unsigned flags, void* stream, Args... args) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(block);
    lc.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    if (flags & WF_FLAG_PDL) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&lc, kernel, static_cast<KArgs>(args)...);
}

}  // namespace wf

using namespace wf;

extern "C" int wf_add_rmsnorm_bf16(void* h, const void* delta, const void* weight, void* y, int64_t M, int64_t K, float eps,
                                   unsigned flags, void* stream) {
    WF_REQUIRE(h && weight && y, "wf_add_rmsnorm_bf16: null pointer");
    WF_REQUIRE(M > 0 && K > 0 && K % 2 == 0 && M < (1LL << 31) && K < (1LL << 31), "wf_add_rmsnorm_bf16: need M > 0 and an even K");
    if (int rc = require_device()) return rc;
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const bool vec = K % 8 == 0 && K <= static_cast<int64_t>(NORM_THREADS) * NORM_CHUNKS * 8 && al16(h) && al16(weight) && al16(y) &&
                     (!delta || al16(delta));
    WF_CUDA(launch(vec ? add_rmsnorm_kernel<true> : add_rmsnorm_kernel<false>, static_cast<unsigned>(M), NORM_THREADS, flags, stream,
                   static_cast<__nv_bfloat16*>(h), static_cast<const __nv_bfloat16*>(delta), static_cast<const __nv_bfloat16*>(weight),
                   static_cast<__nv_bfloat16*>(y), static_cast<int>(K), eps, static_cast<int8_t*>(nullptr), static_cast<float*>(nullptr), 0.f));
    return WF_OK;
}

extern "C" int wf_add_rmsnorm_quant_bf16(void* h, const void* delta, const void* weight, void* y, int8_t* q, float* q_scale, int64_t M,
                                         int64_t K, float eps, float quant_eps, unsigned flags, void* stream) {
    WF_REQUIRE(h && weight && q && q_scale, "wf_add_rmsnorm_quant_bf16: null pointer");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    WF_REQUIRE(M > 0 && M < (1LL << 31) && K > 0 && K % 8 == 0 && K <= static_cast<int64_t>(NORM_THREADS) * NORM_CHUNKS * 8,
               "wf_add_rmsnorm_quant_bf16: K must be a multiple of 8, at most %d", NORM_THREADS * NORM_CHUNKS * 8);
    WF_REQUIRE(al16(h) && al16(weight) && (!y || al16(y)) && (!delta || al16(delta)) && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
               "wf_add_rmsnorm_quant_bf16: tensors must be 16-byte aligned (q: 8)");
    if (int rc = require_device()) return rc;
    WF_CUDA(launch(add_rmsnorm_kernel<true>, static_cast<unsigned>(M), NORM_THREADS, flags, stream, static_cast<__nv_bfloat16*>(h),
                   static_cast<const __nv_bfloat16*>(delta), static_cast<const __nv_bfloat16*>(weight), static_cast<__nv_bfloat16*>(y),
                   static_cast<int>(K), eps, q, q_scale, quant_eps));
    return WF_OK;
}

extern "C" int wf_act_mul_quant_bf16(const void* gate, const void* up, void* out, int8_t* q, float* q_scale, int64_t M, int64_t I, int mode,
                                     float quant_eps, unsigned flags, void* stream) {
    return wf_act_mul_quant_ld_bf16(gate, up, I, out, q, q_scale, M, I, mode, quant_eps, flags, stream);
}

extern "C" int wf_act_mul_quant_ld_bf16(const void* gate, const void* up, int64_t ld, void* out, int8_t* q, float* q_scale, int64_t M, int64_t I, int mode,
                                        float quant_eps, unsigned flags, void* stream) {
    WF_REQUIRE(gate && up && q && q_scale, "wf_act_mul_quant_bf16: null pointer");
    WF_REQUIRE(M > 0 && M < (1LL << 31) && I > 0 && I % 8 == 0 && I <= static_cast<int64_t>(AMQ_THREADS) * AMQ_CHUNKS * 8 && (mode == 0 || mode == 1),
               "wf_act_mul_quant_bf16: rows of a multiple of 8 elements, at most %d; mode 0 or 1", AMQ_THREADS * AMQ_CHUNKS * 8);
    WF_REQUIRE(ld >= I && ld % 8 == 0, "wf_act_mul_quant_bf16: the row stride must cover the row and be a multiple of 8");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    WF_REQUIRE(al16(gate) && al16(up) && (!out || al16(out)) && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
               "wf_act_mul_quant_bf16: tensors must be 16-byte aligned (q: 8)");
    if (int rc = require_device()) return rc;
    WF_CUDA(launch(act_mul_quant_kernel, static_cast<unsigned>(M), static_cast<unsigned>(AMQ_THREADS), flags, stream,
                   static_cast<const __nv_bfloat16*>(gate), static_cast<const __nv_bfloat16*>(up), static_cast<__nv_bfloat16*>(out), q, q_scale,
                   static_cast<int>(I), ld, mode, quant_eps));
    return WF_OK;
}

extern "C" int wf_rope_kv_bf16(void* q, const void* k, const void* v, const float* cos, const float* sin, const int64_t* pos,
                               void* kcache, void* vcache, int64_t B, int nq, int nkv, int D, int T, unsigned flags, void* stream) {
    WF_REQUIRE(q && k && v && cos && sin && pos && kcache && vcache, "wf_rope_kv_bf16: null pointer");
    WF_REQUIRE(B > 0 && nq > 0 && nkv > 0 && D > 0 && D % 2 == 0 && T > 0 && B * (nq + nkv) < (1LL << 31), "wf_rope_kv_bf16: bad dimensions");
    if (int rc = require_device()) return rc;
    int threads = (D / 2 + 31) / 32 * 32;
    if (threads > 256) threads = 256;
    WF_CUDA(launch(rope_kv_kernel, static_cast<unsigned>(B * (nq + nkv)), static_cast<unsigned>(threads), flags, stream,
                   static_cast<__nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), cos, sin, pos,
                   static_cast<__nv_bfloat16*>(kcache), static_cast<__nv_bfloat16*>(vcache), nq, nkv, D, T));
    return WF_OK;
}

extern "C" int wf_rope_kv_prompt_bf16(void* q, const void* k, const void* v, const float* cos, const float* sin, void* kcache, void* vcache,
                                      int64_t B, int64_t S, int nq, int nkv, int D, int64_t T, unsigned flags, void* stream) {
    return wf_rope_kv_prompt_ld_bf16(q, static_cast<int64_t>(nq) * D, k, v, static_cast<int64_t>(nkv) * D, cos, sin, kcache, vcache, B, S, nq, nkv, D, T, flags, stream);
}

extern "C" int wf_rope_kv_prompt_ld_bf16(void* q, int64_t ldq, const void* k, const void* v, int64_t ldkv, const float* cos, const float* sin, void* kcache,
                                         void* vcache, int64_t B, int64_t S, int nq, int nkv, int D, int64_t T, unsigned flags, void* stream) {
    WF_REQUIRE(q && k && v && cos && sin && kcache && vcache, "wf_rope_kv_prompt_bf16: null pointer");
    WF_REQUIRE(B > 0 && S > 0 && S <= T && T < (1LL << 31) && nq > 0 && nkv > 0 && D > 0 && D % 16 == 0, "wf_rope_kv_prompt_bf16: need S <= T and a head dimension that is a multiple of 16");
    WF_REQUIRE(ldq >= static_cast<int64_t>(nq) * D && ldkv >= static_cast<int64_t>(nkv) * D && ldq % 8 == 0 && ldkv % 8 == 0,
               "wf_rope_kv_prompt_bf16: row strides must cover the heads and be multiples of 8");
    WF_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(cos) |
                 reinterpret_cast<uintptr_t>(sin) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 15) == 0,
               "wf_rope_kv_prompt_bf16: tensors must be 16-byte aligned");
    if (int rc = require_device()) return rc;
    const int64_t total = B * S * (nq + nkv) * (D / 16);
    const int64_t blocks = (total + 255) / 256, most = 16 * static_cast<int64_t>(num_sms());
    WF_CUDA(launch(rope_kv_prompt_kernel, static_cast<unsigned>(blocks < most ? blocks : most), 256, flags, stream, static_cast<__nv_bfloat16*>(q),
                   static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), cos, sin, static_cast<__nv_bfloat16*>(kcache),
                   static_cast<__nv_bfloat16*>(vcache), static_cast<int>(S), nq, nkv, D, static_cast<int>(T), ldq, ldkv, total));
    return WF_OK;
}

extern "C" int wf_act_mul_bf16(const void* gate, const void* up, void* out, int64_t n, int mode, unsigned flags, void* stream) {
    WF_REQUIRE(gate && up && out, "wf_act_mul_bf16: null pointer");
    WF_REQUIRE(n > 0 && (mode == 0 || mode == 1), "wf_act_mul_bf16: need a positive element count and mode 0 or 1");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    WF_REQUIRE(al16(gate) && al16(up) && al16(out), "wf_act_mul_bf16: tensors must be 16-byte aligned");
    if (int rc = require_device()) return rc;
    int64_t blocks = ((n + 7) / 8 + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    WF_CUDA(launch(act_mul_kernel, static_cast<unsigned>(blocks), 256u, flags, stream, static_cast<const __nv_bfloat16*>(gate),
                   static_cast<const __nv_bfloat16*>(up), static_cast<__nv_bfloat16*>(out), n, mode));
    return WF_OK;
}

extern "C" int wf_argmax_bf16(const void* x, int64_t ld, int64_t B, int64_t V, int64_t* out, int64_t* pos, unsigned flags, void* stream) {
    WF_REQUIRE(x && out, "wf_argmax_bf16: null pointer");
    WF_REQUIRE(B > 0 && B < (1LL << 31) && V > 0 && V < (1LL << 31) - 16 * AM_THREADS && (ld >= V || B == 1), "wf_argmax_bf16: empty or oversized rows");
    WF_REQUIRE(reinterpret_cast<uintptr_t>(x) % 2 == 0, "wf_argmax_bf16: x must be 2-byte aligned");
    if (int rc = require_device()) return rc;
    const int vec = reinterpret_cast<uintptr_t>(x) % 16 == 0 && (ld % 8 == 0 || B == 1);
    WF_CUDA(launch(argmax_kernel, static_cast<unsigned>(B), static_cast<unsigned>(AM_THREADS), flags, stream, static_cast<const __nv_bfloat16*>(x), ld,
                   static_cast<int>(V), vec, out, pos));
    return WF_OK;
}

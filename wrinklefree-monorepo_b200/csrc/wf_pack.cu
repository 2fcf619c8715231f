// Weight-side kernels: absmean ternarization + 2-bit packing, layout conversion.
//
// Data layout in HBM.  Packed weights are row-major [N, K/4] bytes holding
// code = w + 1.  In WF16 every 32-bit little-endian word covers 16 consecutive
// weights k0..k0+15: byte b, bit pair j holds weight k0 + 4*j + b, so that
// (word >> 2j) & 0x03030303 is four consecutive weights as four bytes, the
// operand shape of an int8 dot product.  I2S is the 128-weight block layout of
// the reference's CPU kernels.
#include <atomic>

#include "wf_common.cuh"

namespace wf {

constexpr int PACK_THREADS = 256;
constexpr int PACK_WEIGHTS_PER_BLOCK = 16384;  // sizes the grid: weights per block and pass, at least

__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < (blockDim.x >> 5); ++i) t += sh[i];
        sh[0] = t;
    }
    __syncthreads();
    t = sh[0];
    __syncthreads();
    return t;
}

// Ternarization is two passes over the weights, both bound by memory: 14336 x 4096 fp32 weights (235 MB) took 117 us when a
// thread read 64 consecutive weights (256 bytes apart from its neighbour's) and divided each by the scale.  Now a warp reads
// 1024 consecutive weights at a time, eight per lane and load, and compares with a threshold; the second pass walks
// them from the end, where the first one has left the last 100 MB or so in L2: 71 us (first pass 40, 5.9 TB/s).  6912 x 2560:
// 34.8 -> 20.8 us, 1536 x 576: 10.9 -> 7.2.
constexpr int PACK_UNIT = 1024;  // weights per warp and step: four loads of 8 per lane

// 8 consecutive weights
template <int WDT>
struct Weights8 {
    uint4 v[WDT == WF_F32 ? 2 : 1];
};
template <int WDT>
__device__ __forceinline__ void load_weights8(const void* w, int64_t elem, bool ok, Weights8<WDT>& r) {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const char*>(w) + elem * (WDT == WF_F32 ? 4 : 2));
#pragma unroll
    for (int j = 0; j < (WDT == WF_F32 ? 2 : 1); ++j) r.v[j] = ok ? __ldg(p + j) : make_uint4(0, 0, 0, 0);
}
template <int WDT>
__device__ __forceinline__ void weight_values(const Weights8<WDT>& r, float (&f)[8]) {
    const uint32_t w[4] = {r.v[0].x, r.v[0].y, r.v[0].z, r.v[0].w};
    if constexpr (WDT == WF_F32) {
        const uint32_t u[4] = {r.v[1].x, r.v[1].y, r.v[1].z, r.v[1].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[i] = __uint_as_float(w[i]);
            f[4 + i] = __uint_as_float(u[i]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if constexpr (WDT == WF_BF16) {
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

// The matrix as `rows` rows of `len` weights, ldw apart (one row when the matrix is contiguous); units of PACK_UNIT weights.
struct PackShape {
    const void* w;
    int64_t len, ldw;
    int rows;
    int segs;       // units per row
    int64_t units;  // rows * segs
};

// Pass 1: per-block sum of |w| (after the optional cast) in fp64, fixed order.
template <int WDT, int MODE>
__global__ void __launch_bounds__(PACK_THREADS) abs_sum_kernel(const PackShape s, double* __restrict__ partial) {
    __shared__ double sh[PACK_THREADS / 32];
    const int lane = threadIdx.x & 31;
    double sum = 0.0;
    for (int64_t unit = static_cast<int64_t>(blockIdx.x) * (PACK_THREADS / 32) + (threadIdx.x >> 5); unit < s.units;
         unit += static_cast<int64_t>(gridDim.x) * (PACK_THREADS / 32)) {
        const int64_t row = s.rows == 1 ? 0 : unit / s.segs, at = (unit - row * s.segs) * PACK_UNIT + 8 * lane;
        Weights8<WDT> r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) load_weights8<WDT>(s.w, row * s.ldw + at + 256 * u, at + 256 * u < s.len, r[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float f[8];
            weight_values<WDT>(r[u], f);
            double a = 0.0;
#pragma unroll
            for (int i = 0; i < 8; ++i) a += static_cast<double>(fabsf(rnd<MODE>(f[i])));
            sum += a;
        }
    }
    const double t = block_sum(sum, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// Pass 2: every block re-reduces the partials in the same order, derives the scale, ternarizes and packs.
//
// FP32 mode: the code of w is clamp(rint(w / mean), -1, 1) + 1.  The fp32 quotient exceeds 1/2 exactly when w > mean / 2: the
// next float above mean / 2 is at least half an ulp of 1/2 further in the quotient, and the tie itself rounds to zero.
// So two comparisons with mean / 2 stand for the division, wherever mean / 2 is exact: an eps that lets the mean be subnormal or
// zero keeps the division, and so does a matrix with a NaN or an infinity.  Cast
// modes: the same two comparisons on the rounded product; a NaN compares false with both, the code 0 that the clamp gives it.
//
// The comparisons of four weights as masks of four bytes (code = [v > h] + [v >= -h]): six instructions per weight that take
// a predicate, a select and an addition each were what bounded this pass.
// the sign bits of four floats as four bytes of ones or zeros (a selector with its top bit set replicates the byte's sign)
__device__ __forceinline__ uint32_t signs4(float a, float b, float c, float d) {
    uint32_t lo, hi;
    asm("prmt.b32 %0, %1, %2, 0xfbfb;" : "=r"(lo) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
    asm("prmt.b32 %0, %1, %2, 0xfbfb;" : "=r"(hi) : "r"(__float_as_uint(c)), "r"(__float_as_uint(d)));
    return __byte_perm(lo, hi, 0x5410);
}
// codes of the weights 4 g .. 4 g + 3 of a lane's eight as four bytes.  h = mean / 2 (FP32) or 1/2; `by_sign` (FP32 mode): there is
// no NaN and no infinity among the weights and h is exact, so the signs of differences decide.
template <int WDT, int MODE>
__device__ __forceinline__ uint32_t codes4(const Weights8<WDT>& r, int g, float q_mul, float h, bool by_sign) {
    const uint32_t ones = 0x01010101u;
    float f[8];
    weight_values<WDT>(r, f);
    if constexpr (MODE == WF_F32) {
        if (by_sign) {
            const uint32_t above = signs4(h - f[4 * g], h - f[4 * g + 1], h - f[4 * g + 2], h - f[4 * g + 3]);
            const uint32_t below = signs4(f[4 * g] + h, f[4 * g + 1] + h, f[4 * g + 2] + h, f[4 * g + 3] + h);
            return ones + (above & ones) - (below & ones);
        }
        uint32_t c = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            c |= static_cast<uint32_t>(static_cast<int>(fminf(fmaxf(rintf(__fdiv_rn(f[4 * g + i], q_mul)), -1.f), 1.f)) + 1) << (8 * i);
        return c;
    } else if constexpr (MODE == WF_BF16) {
        __nv_bfloat162 v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) v[i] = __hmul2_rn(__floats2bfloat162_rn(f[4 * g + 2 * i], f[4 * g + 2 * i + 1]), __float2bfloat162_rn(q_mul));
        const __nv_bfloat162 hi = __float2bfloat162_rn(0.5f), lo = __float2bfloat162_rn(-0.5f);
        return (__byte_perm(__hgt2_mask(v[0], hi), __hgt2_mask(v[1], hi), 0x6420) & ones) + (__byte_perm(__hge2_mask(v[0], lo), __hge2_mask(v[1], lo), 0x6420) & ones);
    } else {
        __half2 v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) v[i] = __hmul2_rn(__floats2half2_rn(f[4 * g + 2 * i], f[4 * g + 2 * i + 1]), __float2half2_rn(q_mul));
        const __half2 hi = __float2half2_rn(0.5f), lo = __float2half2_rn(-0.5f);
        return (__byte_perm(__hgt2_mask(v[0], hi), __hgt2_mask(v[1], hi), 0x6420) & ones) + (__byte_perm(__hge2_mask(v[0], lo), __hge2_mask(v[1], lo), 0x6420) & ones);
    }
}

template <int WDT, int MODE>
__global__ void __launch_bounds__(PACK_THREADS)
    ternarize_pack_kernel(const PackShape s, int64_t weights, const double* partial, int npartial, float eps, double by_sign_below,
                          uint8_t* __restrict__ codes, float* __restrict__ scale_out) {
    __shared__ double sh[PACK_THREADS / 32];
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the partial sums
    double sum = 0.0;
    for (int i = threadIdx.x; i < npartial; i += PACK_THREADS) sum += *static_cast<const volatile double*>(partial + i);
    // the per-thread strided sums depend only on npartial and the block size: identical in every block
    const double total = block_sum(sum, sh);
    float mean = static_cast<float>(total / static_cast<double>(weights));
    float q_mul, dq;
    if constexpr (MODE == WF_F32) {
        mean = fmaxf(mean, eps);
        q_mul = mean;  // codes = rint(w / mean)
        dq = mean;
    } else {
        mean = rnd<MODE>(fmaxf(rnd<MODE>(mean), eps));
        q_mul = rnd<MODE>(__frcp_rn(mean));  // codes = rint(rnd(w * scale))
        dq = rnd<MODE>(__frcp_rn(q_mul));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        scale_out[0] = dq;
        scale_out[1] = q_mul;
    }
    const float half = MODE == WF_F32 ? 0.5f * q_mul : 0.5f;
    const bool by_sign = total < by_sign_below;  // false for an infinity and a NaN
    const int lane = threadIdx.x & 31;
    const int64_t code_row = s.len / 4;  // bytes
    for (int64_t back = static_cast<int64_t>(blockIdx.x) * (PACK_THREADS / 32) + (threadIdx.x >> 5); back < s.units;
         back += static_cast<int64_t>(gridDim.x) * (PACK_THREADS / 32)) {
        const int64_t unit = s.units - 1 - back;
        const int64_t row = s.rows == 1 ? 0 : unit / s.segs, at = (unit - row * s.segs) * PACK_UNIT + 8 * lane;
        Weights8<WDT> r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) load_weights8<WDT>(s.w, row * s.ldw + at + 256 * u, at + 256 * u < s.len, r[u]);
        uint32_t word[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            // weights 0-3 in bit pair 0 of the four bytes, 4-7 in bit pair 1
            uint32_t c = codes4<WDT, MODE>(r[u], 0, q_mul, half, by_sign) | (codes4<WDT, MODE>(r[u], 1, q_mul, half, by_sign) << 2);
            c <<= 4 * (lane & 1);  // an odd lane holds the upper half of its word: bit pairs 2 and 3
            word[u] = c | __shfl_xor_sync(0xffffffffu, c, 1);
        }
        // lane l of loads 2h and 2h + 1: the even lanes store the words of one, the odd lanes of the other
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t first = (unit - row * s.segs) * PACK_UNIT + 256 * (2 * h + (lane & 1)) + 16 * (lane >> 1);  // its first weight
            if (first < s.len) *reinterpret_cast<uint32_t*>(codes + row * code_row + first / 4) = (lane & 1) ? word[2 * h + 1] : word[2 * h];
        }
    }
}

// ---- layout conversion ----

// code (0..2) of logical weight (n, k) in a packed buffer of the given layout
__device__ __forceinline__ uint32_t fetch_code(const uint8_t* __restrict__ src, int layout, int64_t N, int64_t K, int64_t n,
                                               int64_t k) {
    switch (layout) {
        case WF_LAYOUT_WF16: {
            int r = static_cast<int>(k & 15);
            uint8_t byte = src[n * (K / 4) + (k >> 4) * 4 + (r & 3)];
            return (byte >> (2 * (r >> 2))) & 3u;
        }
        case WF_LAYOUT_I2S: {
            int r = static_cast<int>(k & 127);
            uint8_t byte = src[n * (K / 4) + (k >> 7) * 32 + (r & 31)];
            return (byte >> (6 - 2 * (r >> 5))) & 3u;
        }
        case WF_LAYOUT_SEQ_LSB:
            return (src[n * (K / 4) + (k >> 2)] >> (2 * (k & 3))) & 3u;
        case WF_LAYOUT_SEQ_MSB:
            return (src[n * (K / 4) + (k >> 2)] >> (6 - 2 * (k & 3))) & 3u;
        default: {  // WF_LAYOUT_HF: [N/4, K]
            int64_t q = N / 4;
            return (src[(n % q) * K + k] >> (2 * (n / q))) & 3u;
        }
    }
}

// logical weight (inside its row) stored at (byte, bit pair s) of a row-major destination layout
__device__ __forceinline__ int64_t dst_weight(int layout, int64_t byte, int s) {
    switch (layout) {
        case WF_LAYOUT_WF16: return (byte >> 2) * 16 + 4 * s + (byte & 3);
        case WF_LAYOUT_I2S: return (byte >> 5) * 128 + 32 * (3 - s) + (byte & 31);
        case WF_LAYOUT_SEQ_LSB: return 4 * byte + s;
        default: return 4 * byte + (3 - s);  // WF_LAYOUT_SEQ_MSB
    }
}

// one thread per output byte
__global__ void repack_kernel(const uint8_t* __restrict__ src, int src_layout, uint8_t* __restrict__ dst, int dst_layout,
                              int64_t N, int64_t K, const int8_t* __restrict__ ternary) {
    const int64_t total = N * (K / 4);
    for (int64_t o = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; o < total;
         o += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        int64_t n = o / (K / 4), byte = o % (K / 4);
        uint32_t out = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int64_t k = dst_weight(dst_layout, byte, s);
            uint32_t code = ternary ? static_cast<uint32_t>(ternary[n * K + k] + 1) : fetch_code(src, src_layout, N, K, n, k);
            out |= (code & 3u) << (2 * s);
        }
        dst[o] = static_cast<uint8_t>(out);
    }
}

// ---- the max-abs quantizers of the inference side ----
// absmax over the whole matrix: non-negative floats order like their bit patterns, one atomicMax per block
template <int WDT>
__global__ void abs_max_kernel(const void* __restrict__ w, int64_t N, int64_t K, int64_t ldw, unsigned* __restrict__ maxbits) {
    float mx = 0.f;
    const int64_t total = N * K;
    for (int64_t o = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; o < total;
         o += static_cast<int64_t>(gridDim.x) * blockDim.x)
        mx = fmaxf(mx, fabsf(load1<WDT>(w, (o / K) * ldw + o % K)));
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
    if ((threadIdx.x & 31) == 0) atomicMax(maxbits, __float_as_uint(mx));
}

// one thread per output byte; rule 0: codes by thresholds at +-0.5 of w / max, rule 1: by sign with a 1e-6 dead zone
template <int WDT>
__global__ void maxabs_pack_kernel(const void* __restrict__ w, int64_t N, int64_t K, int64_t ldw, int rule, int dst_layout,
                                   const unsigned* __restrict__ maxbits, uint8_t* __restrict__ dst, float* __restrict__ scale_out) {
    float mx = __uint_as_float(*maxbits);
    if (rule == WF_MAXABS_HALF && mx < 1e-6f) mx = 1.0f;
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = mx;
    const int64_t total = N * (K / 4);
    for (int64_t o = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; o < total;
         o += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t n = o / (K / 4), byte = o % (K / 4);
        uint32_t out = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const float v = load1<WDT>(w, n * ldw + dst_weight(dst_layout, byte, s));
            uint32_t code = 1;
            if (rule == WF_MAXABS_HALF) {
                const float t = __fdiv_rn(v, mx);
                code = t > 0.5f ? 2u : (t < -0.5f ? 0u : 1u);
            } else if (fabs(static_cast<double>(v)) >= 1e-6) {
                code = static_cast<double>(v) * static_cast<double>(mx) > 0.0 ? 2u : 0u;
            }
            out |= code << (2 * s);
        }
        dst[o] = static_cast<uint8_t>(out);
    }
}

__global__ void unpack_kernel(const uint8_t* __restrict__ src, int layout, int8_t* __restrict__ ternary, int64_t N,
                              int64_t K) {
    const int64_t total = N * K;
    for (int64_t o = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; o < total;
         o += static_cast<int64_t>(gridDim.x) * blockDim.x)
        ternary[o] = static_cast<int8_t>(static_cast<int>(fetch_code(src, layout, N, K, o / K, o % K)) - 1);
}

constexpr int PACK_MAX_GRID = 148 * 8;  // blocks of the two packing kernels = partial sums in the scratch

static int pack_grid(int64_t N, int64_t K) {
    int64_t blocks = (N * K + PACK_WEIGHTS_PER_BLOCK - 1) / PACK_WEIGHTS_PER_BLOCK;
    if (blocks < 1) blocks = 1;
    if (blocks > PACK_MAX_GRID) blocks = PACK_MAX_GRID;
    return static_cast<int>(blocks);
}

template <int WDT, int MODE>
static int launch_pack_mode(const PackShape& s, int64_t weights, int grid, float eps, uint8_t* codes, float* scale, double* partial, cudaStream_t st) {
    abs_sum_kernel<WDT, MODE><<<grid, PACK_THREADS, 0, st>>>(s, partial);
    WF_CUDA(cudaGetLastError());
    // Chained, so that its launch is prepared beside the first pass.  That pass triggers nothing before its end: the blocks of this
    // one start when all of its blocks have left, and wait for its sums to be visible.
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(static_cast<unsigned>(grid));
    lc.blockDim = dim3(PACK_THREADS);
    lc.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    // a mean of at least 2^-125 has an exact half; decided here, for a second condition in the kernel cost 0.25 of 19.9 us (4096^2, bf16)
    const double by_sign_below = eps >= 2.3509887e-38f ? 1e300 : -1.0;
    WF_CUDA(cudaLaunchKernelEx(&lc, ternarize_pack_kernel<WDT, MODE>, s, weights, static_cast<const double*>(partial), grid, eps, by_sign_below, codes, scale));
    return WF_OK;
}

template <int WDT>
static int launch_pack(const void* w, int64_t N, int64_t K, int64_t ldw, int mode, float eps, uint8_t* codes, float* scale,
                       double* partial, cudaStream_t st) {
    const int grid = pack_grid(N, K);
    PackShape s;
    s.w = w;
    s.rows = ldw == K ? 1 : static_cast<int>(N);
    s.len = ldw == K ? N * K : K;
    s.ldw = ldw;
    const int64_t segs = (s.len + PACK_UNIT - 1) / PACK_UNIT;
    s.segs = static_cast<int>(segs);
    s.units = s.rows * segs;
    switch (mode) {
        case WF_PACK_FP32: return launch_pack_mode<WDT, WF_F32>(s, N * K, grid, eps, codes, scale, partial, st);
        case WF_PACK_CAST_BF16: return launch_pack_mode<WDT, WF_BF16>(s, N * K, grid, eps, codes, scale, partial, st);
        default: return launch_pack_mode<WDT, WF_F16>(s, N * K, grid, eps, codes, scale, partial, st);
    }
}

}  // namespace wf

using namespace wf;

extern "C" {

size_t wf_pack_scratch_bytes(int64_t N, int64_t K) {
    if (N <= 0 || K <= 0) return 0;
    return static_cast<size_t>(pack_grid(N, K)) * sizeof(double);
}

int wf_pack_ternary(const void* w, int w_dtype, int64_t N, int64_t K, int64_t ldw, int mode, float eps, uint8_t* codes_out,
                    float* scale_out, void* scratch, size_t scratch_bytes, void* stream) {
    WF_REQUIRE(w && codes_out && scale_out && scratch, "wf_pack_ternary: null pointer");
    WF_REQUIRE(N > 0 && K > 0 && K % 64 == 0, "wf_pack_ternary: need N > 0 and K a positive multiple of 64 (N=%lld K=%lld)",
               (long long)N, (long long)K);
    WF_REQUIRE(is_float_dtype(w_dtype), "wf_pack_ternary: unsupported weight dtype %d", w_dtype);
    WF_REQUIRE(mode >= WF_PACK_FP32 && mode <= WF_PACK_CAST_F16, "wf_pack_ternary: unknown mode %d", mode);
    WF_REQUIRE(ldw >= K && (ldw * dtype_size(w_dtype)) % 16 == 0, "wf_pack_ternary: row stride must cover K and keep rows 16-byte aligned");
    WF_REQUIRE(reinterpret_cast<uintptr_t>(w) % 16 == 0 && reinterpret_cast<uintptr_t>(codes_out) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(scratch) % 8 == 0,
               "wf_pack_ternary: w and codes_out must be 16-byte aligned, scratch 8-byte aligned");
    if (scratch_bytes < wf_pack_scratch_bytes(N, K))
        return fail(WF_E_SCRATCH, "wf_pack_ternary: scratch of %zu bytes, need %zu", scratch_bytes, wf_pack_scratch_bytes(N, K));
    if (int rc = require_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double* partial = static_cast<double*>(scratch);
    switch (w_dtype) {
        case WF_F32: return launch_pack<WF_F32>(w, N, K, ldw, mode, eps, codes_out, scale_out, partial, st);
        case WF_BF16: return launch_pack<WF_BF16>(w, N, K, ldw, mode, eps, codes_out, scale_out, partial, st);
        default: return launch_pack<WF_F16>(w, N, K, ldw, mode, eps, codes_out, scale_out, partial, st);
    }
}

static int check_layout_dims(const char* who, int layout, int64_t N, int64_t K) {
    WF_REQUIRE(N > 0 && K > 0, "%s: empty matrix", who);
    switch (layout) {
        case WF_LAYOUT_WF16: WF_REQUIRE(K % 16 == 0, "%s: WF16 needs K %% 16 == 0 (K=%lld)", who, (long long)K); break;
        case WF_LAYOUT_I2S: WF_REQUIRE(K % 128 == 0, "%s: I2_S needs K %% 128 == 0 (K=%lld)", who, (long long)K); break;
        case WF_LAYOUT_SEQ_LSB:
        case WF_LAYOUT_SEQ_MSB: WF_REQUIRE(K % 4 == 0, "%s: sequential layouts need K %% 4 == 0", who); break;
        case WF_LAYOUT_HF: WF_REQUIRE(N % 4 == 0 && K % 4 == 0, "%s: HF layout needs N %% 4 == 0 and K %% 4 == 0", who); break;
        default: return fail(WF_E_ARG, "%s: unknown layout %d", who, layout);
    }
    return WF_OK;
}

static int grid_for(int64_t total) {
    int64_t b = (total + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    return static_cast<int>(b < 1 ? 1 : b);
}

int wf_repack(const uint8_t* src, int src_layout, uint8_t* dst, int dst_layout, int64_t N, int64_t K, void* stream) {
    WF_REQUIRE(src && dst, "wf_repack: null pointer");
    WF_REQUIRE(dst_layout >= WF_LAYOUT_WF16 && dst_layout <= WF_LAYOUT_SEQ_MSB, "wf_repack: destination must be a row-major layout (not HF)");
    if (int rc = check_layout_dims("wf_repack(src)", src_layout, N, K)) return rc;
    if (int rc = check_layout_dims("wf_repack(dst)", dst_layout, N, K)) return rc;
    if (int rc = require_device()) return rc;
    repack_kernel<<<grid_for(N * (K / 4)), 256, 0, static_cast<cudaStream_t>(stream)>>>(src, src_layout, dst, dst_layout, N, K,
                                                                                     nullptr);
    WF_CUDA(cudaGetLastError());
    return WF_OK;
}

int wf_pack_codes(const int8_t* ternary, uint8_t* dst, int layout, int64_t N, int64_t K, void* stream) {
    WF_REQUIRE(ternary && dst, "wf_pack_codes: null pointer");
    WF_REQUIRE(layout >= WF_LAYOUT_WF16 && layout <= WF_LAYOUT_SEQ_MSB, "wf_pack_codes: layout must be row-major (not HF)");
    if (int rc = check_layout_dims("wf_pack_codes", layout, N, K)) return rc;
    if (int rc = require_device()) return rc;
    repack_kernel<<<grid_for(N * (K / 4)), 256, 0, static_cast<cudaStream_t>(stream)>>>(nullptr, 0, dst, layout, N, K, ternary);
    WF_CUDA(cudaGetLastError());
    return WF_OK;
}

int wf_unpack_codes(const uint8_t* src, int layout, int8_t* ternary, int64_t N, int64_t K, void* stream) {
    WF_REQUIRE(src && ternary, "wf_unpack_codes: null pointer");
    if (int rc = check_layout_dims("wf_unpack_codes", layout, N, K)) return rc;
    if (int rc = require_device()) return rc;
    unpack_kernel<<<grid_for(N * K), 256, 0, static_cast<cudaStream_t>(stream)>>>(src, layout, ternary, N, K);
    WF_CUDA(cudaGetLastError());
    return WF_OK;
}

int wf_quantize_maxabs(const void* w, int w_dtype, int64_t N, int64_t K, int64_t ldw, int rule, int dst_layout,
                       uint8_t* codes_out, float* scale_out, void* stream) {
    WF_REQUIRE(w && codes_out && scale_out, "wf_quantize_maxabs: null pointer");
    WF_REQUIRE(is_float_dtype(w_dtype), "wf_quantize_maxabs: unsupported weight dtype %d", w_dtype);
    WF_REQUIRE(rule == WF_MAXABS_HALF || rule == WF_MAXABS_SIGN, "wf_quantize_maxabs: unknown rule %d", rule);
    WF_REQUIRE(dst_layout >= WF_LAYOUT_WF16 && dst_layout <= WF_LAYOUT_SEQ_MSB, "wf_quantize_maxabs: destination must be a row-major layout");
    WF_REQUIRE(ldw >= K, "wf_quantize_maxabs: row stride must cover K");
    if (int rc = check_layout_dims("wf_quantize_maxabs", dst_layout, N, K)) return rc;
    if (int rc = require_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the running maximum lives in the second float of scale_out until the packing kernel has read it
    unsigned* maxbits = reinterpret_cast<unsigned*>(scale_out) + 1;
    WF_CUDA(cudaMemsetAsync(maxbits, 0, sizeof(unsigned), st));
    const int g1 = grid_for(N * K), g2 = grid_for(N * (K / 4));
    switch (w_dtype) {
        case WF_F32:
            abs_max_kernel<WF_F32><<<g1, 256, 0, st>>>(w, N, K, ldw, maxbits);
            maxabs_pack_kernel<WF_F32><<<g2, 256, 0, st>>>(w, N, K, ldw, rule, dst_layout, maxbits, codes_out, scale_out);
            break;
        case WF_BF16:
            abs_max_kernel<WF_BF16><<<g1, 256, 0, st>>>(w, N, K, ldw, maxbits);
            maxabs_pack_kernel<WF_BF16><<<g2, 256, 0, st>>>(w, N, K, ldw, rule, dst_layout, maxbits, codes_out, scale_out);
            break;
        default:
            abs_max_kernel<WF_F16><<<g1, 256, 0, st>>>(w, N, K, ldw, maxbits);
            maxabs_pack_kernel<WF_F16><<<g2, 256, 0, st>>>(w, N, K, ldw, rule, dst_layout, maxbits, codes_out, scale_out);
            break;
    }
    WF_CUDA(cudaGetLastError());
    return WF_OK;
}
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of wf_pack_ternary.
//
// Some hosts of this library may not allocate device memory at the point where they pack weights:
// a serving process whose own pool has claimed the GPU and forbids cudaMalloc inside layer code,
// or a latency-critical thread that cannot afford the implicit device synchronisation of an
// allocation.  wf_pack_ternary needs a small scratch buffer (the per-block partial sums of |w|);
// here that scratch is a fixed array that lives in the library image on every GPU that loads it
// (WF_PACK_NOALLOC_SCRATCH_BYTES, held until the process exits).  Nothing is allocated or freed by
// this entry point, neither through the CUDA runtime nor through any other library.
//
// The first call on a device looks up the device address of the array (the host-side symbol is
// only a handle, not an address a kernel may use); make that first call outside any stream capture.
// All calls on a device share the one array: two calls whose kernels overlap on the GPU (different
// streams) race on it.  Every launch overwrites the part of the array it later reads, so nothing
// has to be cleared between calls.
// ---------------------------------------------------------------------------------------------
namespace wf {

constexpr int NOALLOC_MAX_PARTIALS = PACK_MAX_GRID;  // the largest grid launch_pack ever uses
static __device__ __align__(256) double g_pack_noalloc_scratch[NOALLOC_MAX_PARTIALS];

constexpr int NOALLOC_MAX_DEVICES = 64;
static std::atomic<double*> g_noalloc_ptr[NOALLOC_MAX_DEVICES];  // device address of the array, per device (zero-initialised)

// Set-up, once per device, with that device current.
static int noalloc_scratch(double** out) {
    int dev = -1;
    WF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return fail(WF_E_LIMIT, "wf_pack_ternary_noalloc: device index %d not supported", dev);
    if (!g_noalloc_ptr[dev].load(std::memory_order_acquire)) {
        double* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_pack_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_pack_noalloc_scratch)");
        if (!ptr) return fail(WF_E_DEVICE, "wf_pack_ternary_noalloc: no device address for the scratch array");
        g_noalloc_ptr[dev].store(ptr, std::memory_order_release);
    }
    *out = g_noalloc_ptr[dev].load(std::memory_order_acquire);
    return WF_OK;
}

}  // namespace wf

extern "C" size_t wf_pack_noalloc_scratch_bytes(void) { return sizeof(double) * wf::NOALLOC_MAX_PARTIALS; }

extern "C" int wf_pack_ternary_noalloc(const void* w, int w_dtype, int64_t N, int64_t K, int64_t ldw, int mode, float eps,
                                       uint8_t* codes_out, float* scale_out, void* stream) {
    WF_REQUIRE(w && codes_out && scale_out, "wf_pack_ternary_noalloc: null pointer");
    WF_REQUIRE(N > 0 && K > 0 && K % 64 == 0, "wf_pack_ternary_noalloc: need N > 0 and K a positive multiple of 64 (N=%lld K=%lld)",
               (long long)N, (long long)K);
    if (N > WF_PACK_NOALLOC_MAX_WEIGHTS / K)
        return fail(WF_E_LIMIT, "wf_pack_ternary_noalloc: %lld x %lld weights exceed the maximum of %lld for the allocation-free "
                                "entry point; use wf_pack_ternary with caller scratch",
                    (long long)N, (long long)K, (long long)WF_PACK_NOALLOC_MAX_WEIGHTS);
    WF_REQUIRE(is_float_dtype(w_dtype), "wf_pack_ternary_noalloc: unsupported weight dtype %d", w_dtype);
    WF_REQUIRE(mode >= WF_PACK_FP32 && mode <= WF_PACK_CAST_F16, "wf_pack_ternary_noalloc: unknown mode %d", mode);
    WF_REQUIRE(ldw >= K && (ldw * dtype_size(w_dtype)) % 16 == 0, "wf_pack_ternary_noalloc: row stride must cover K and keep rows 16-byte aligned");
    WF_REQUIRE(reinterpret_cast<uintptr_t>(w) % 16 == 0 && reinterpret_cast<uintptr_t>(codes_out) % 16 == 0,
               "wf_pack_ternary_noalloc: w and codes_out must be 16-byte aligned");
    if (int rc = require_device()) return rc;
    double* partial = nullptr;
    if (int rc = noalloc_scratch(&partial)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (w_dtype) {
        case WF_F32: return launch_pack<WF_F32>(w, N, K, ldw, mode, eps, codes_out, scale_out, partial, st);
        case WF_BF16: return launch_pack<WF_BF16>(w, N, K, ldw, mode, eps, codes_out, scale_out, partial, st);
        default: return launch_pack<WF_F16>(w, N, K, ldw, mode, eps, codes_out, scale_out, partial, st);
    }
}

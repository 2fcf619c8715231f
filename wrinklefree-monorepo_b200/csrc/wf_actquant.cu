// Stand-alone activation quantization to int8 (per token, or per tensor with the
// semantics of the reference's CPU operator).
#include "wf_common.cuh"
#include "wf_quant8.cuh"

namespace wf {

constexpr int AQ_THREADS = 256;

__device__ __forceinline__ float block_max(float v, float* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    float t = sh[0];
#pragma unroll
    for (int i = 1; i < AQ_THREADS / 32; ++i) t = fmaxf(t, sh[i]);
    __syncthreads();
    return t;
}

__device__ __forceinline__ int block_sum_int(int v, int* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int i = 0; i < AQ_THREADS / 32; ++i) t += sh[i];
    __syncthreads();
    return t;
}

// One token quantized by one block; x is read twice.  K % 8 == 0.
template <int DT>
__device__ __forceinline__ void quant_token(const void* x, int64_t m, int64_t K, int64_t ldx, float eps, int8_t* __restrict__ q,
                                            float* __restrict__ scale, int32_t* __restrict__ rowsum, float* shf, int* shi) {
    float mx = 0.f;
    for (int64_t k = threadIdx.x * 8; k < K; k += AQ_THREADS * 8) {
        float f[8];
        load8<DT>(x, m * ldx + k, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fabsf(f[i]));
    }
    mx = block_max(mx, shf);
    const float s = act_scale_from_absmax<DT>(mx, eps);
    int sum = 0;
    for (int64_t k = threadIdx.x * 8; k < K; k += AQ_THREADS * 8) {
        float f[8];
        load8<DT>(x, m * ldx + k, f);
        uint32_t w0 = 0, w1 = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int a = quantize_one<DT>(f[i], s), b = quantize_one<DT>(f[4 + i], s);
            sum += a + b;
            w0 |= static_cast<uint32_t>(a & 0xff) << (8 * i);
            w1 |= static_cast<uint32_t>(b & 0xff) << (8 * i);
        }
        *reinterpret_cast<uint2*>(q + m * K + k) = make_uint2(w0, w1);
    }
    if (rowsum) sum = block_sum_int(sum, shi);
    if (threadIdx.x == 0) {
        scale[m] = s;
        if (rowsum) rowsum[m] = sum;
    }
}

template <int DT>
__global__ void __launch_bounds__(AQ_THREADS)
    act_quant_token_kernel(const void* x, int64_t K, int64_t ldx, float eps, int8_t* __restrict__ q,
                           float* __restrict__ scale, int32_t* __restrict__ rowsum, int x_ready) {
    __shared__ float shf[AQ_THREADS / 32];
    __shared__ int shi[AQ_THREADS / 32];
    // chained with a programmatic dependency: the next kernel may start (the contraction fetches its first weights
    // meanwhile); x may come from the previous kernel and q may still be read by it, so everything else waits for it
    // -- unless the caller states that neither is the case (x_ready): then only the end of the grid waits, so that
    // whoever waits for this grid may still rely on everything ahead of it in the stream
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (!x_ready) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    quant_token<DT>(x, blockIdx.x, K, ldx, eps, q, scale, rowsum, shf, shi);
    // one block stays until the predecessor has completed, so that this grid does not end before it; the others leave
    if (x_ready && blockIdx.x == 0) asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// Per-tensor absmax: pass 1 reduces |x| into a float kept as ordered uint bits.
__global__ void __launch_bounds__(AQ_THREADS)
    tensor_absmax_kernel(const float* __restrict__ x, int64_t M, int64_t K, int64_t ldx, unsigned* __restrict__ maxbits) {
    __shared__ float shf[AQ_THREADS / 32];
    const int64_t total = M * (K / 4);
    float mx = 0.f;
    for (int64_t v = static_cast<int64_t>(blockIdx.x) * AQ_THREADS + threadIdx.x; v < total;
         v += static_cast<int64_t>(gridDim.x) * AQ_THREADS) {
        int64_t row = v / (K / 4), col = (v % (K / 4)) * 4;
        float4 f = __ldg(reinterpret_cast<const float4*>(x + row * ldx + col));
        mx = fmaxf(mx, fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fmaxf(fabsf(f.z), fabsf(f.w))));
    }
    mx = block_max(mx, shf);
    if (threadIdx.x == 0) atomicMax(maxbits, __float_as_uint(mx));
}

// Pass 2: one block per row; scale = max/127, multiplier 127/max (both fp32 divisions), round to nearest even.
__global__ void __launch_bounds__(AQ_THREADS)
    tensor_quant_kernel(const float* __restrict__ x, int64_t K, int64_t ldx, const unsigned* __restrict__ maxbits,
                        int8_t* __restrict__ q, int32_t* __restrict__ rowsum) {
    __shared__ int shi[AQ_THREADS / 32];
    const int64_t m = blockIdx.x;
    float mx = __uint_as_float(*maxbits);
    if (mx < 1e-6f) mx = 1.0f;
    const float inv = __fdiv_rn(127.0f, mx);
    int sum = 0;
    for (int64_t k = threadIdx.x * 4; k < K; k += AQ_THREADS * 4) {
        float4 f = __ldg(reinterpret_cast<const float4*>(x + m * ldx + k));
        int a = quantize_one<WF_F32>(f.x, inv), b = quantize_one<WF_F32>(f.y, inv);
        int c = quantize_one<WF_F32>(f.z, inv), d = quantize_one<WF_F32>(f.w, inv);
        sum += a + b + c + d;
        *reinterpret_cast<uint32_t*>(q + m * K + k) = (a & 0xff) | ((b & 0xff) << 8) | ((c & 0xff) << 16) | ((d & 0xff) << 24);
    }
    sum = block_sum_int(sum, shi);
    if (threadIdx.x == 0 && rowsum) rowsum[m] = sum;
}

// Pass 3: the reduction cell held the absmax while pass 2 read it; turn it into the returned scale.
__global__ void publish_tensor_scale(float* scale) {
    float mx = scale[0];
    if (mx < 1e-6f) mx = 1.0f;
    scale[0] = __fdiv_rn(mx, 127.0f);
}

}  // namespace wf

using namespace wf;

static int act_quant_impl(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, int mode, float eps, int8_t* q, float* scale,
                          int32_t* rowsum, int x_ready, void* stream);

// One token quantized by one block, the row held in registers between the two passes (K <= 8 * AQ_THREADS * CHUNKS): x is
// read once, and all of a thread's loads are in flight together.
template <int DT, int CHUNKS>
__device__ __forceinline__ void quant_token_reg(const void* x, int64_t m, int64_t K, int64_t ldx, float eps, int8_t* __restrict__ q,
                                                float* __restrict__ scale, int32_t* __restrict__ rowsum, float* shf, int* shi) {
    const int chunks = static_cast<int>(K >> 3);
    Raw8<DT> r[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        const int i = threadIdx.x + c * AQ_THREADS;
        load_raw8<DT>(x, m * ldx + 8 * static_cast<int64_t>(i), i < chunks, r[c]);
    }
    uint32_t bits = 0;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) bits = max_bits8<DT>(r[c], bits);
    bits = warp_max_bits<DT>(bits);
    if ((threadIdx.x & 31) == 0) shi[threadIdx.x >> 5] = static_cast<int>(bits);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < AQ_THREADS / 32; ++i) bits = max(bits, static_cast<uint32_t>(shi[i]));
    bool fast = fast_bits<DT>(bits);
    float mx = bits_value<DT>(bits);
    if (!fast) {  // uniform over the block
        mx = 0.f;
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) mx = max_abs8<DT>(r[c], mx);
        mx = block_max(mx, shf);
    }
    const float s = act_scale_from_absmax<DT>(mx, eps);
    fast = fast && s < INFINITY;
    int sum = 0;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        const int i = threadIdx.x + c * AQ_THREADS;
        if (i < chunks) {
            const uint2 w = fast ? quantize8_fast<DT>(r[c], s) : quantize8_any<DT>(r[c], s);
            sum = sum_bytes(w, sum);
            *reinterpret_cast<uint2*>(q + m * K + 8 * static_cast<int64_t>(i)) = w;
        }
    }
    if (rowsum) {
        __syncthreads();  // shi has been read
        sum = block_sum_int(sum, shi);
    }
    if (threadIdx.x == 0) {
        scale[m] = s;
        if (rowsum) rowsum[m] = sum;
    }
}

template <int DT, int CHUNKS>
__global__ void __launch_bounds__(AQ_THREADS)
    act_quant_token_reg_kernel(const void* x, int64_t K, int64_t ldx, float eps, int8_t* __restrict__ q,
                               float* __restrict__ scale, int32_t* __restrict__ rowsum, int x_ready) {
    __shared__ float shf[AQ_THREADS / 32];
    __shared__ int shi[AQ_THREADS / 32];
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (!x_ready) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    quant_token_reg<DT, CHUNKS>(x, blockIdx.x, K, ldx, eps, q, scale, rowsum, shf, shi);
    // one block stays until the predecessor has completed, so that this grid does not end before it; the others leave
    if (x_ready && blockIdx.x == 0) asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// Chunks of 8 per lane where one warp per token is the better split, else 0.  A block per token spends most of a short row on
// its barrier and leaves threads without a chunk; a warp per token has neither, but takes its time for the row serially, so it
// needs enough tokens to fill the chip: the two cross between 300 tokens of 576 values and 3000 of 2560 (8192 tokens: 4.0
// against 11.1 us at K = 576, 8.4 against 13.9 at 2560; 22 against 19 at 4096; 1920 tokens of 2560: 5.0 against 4.4).
static int warp_form_chunks(int64_t M, int64_t K) {
    const int64_t per_lane = ((K >> 3) + 31) / 32;
    return per_lane <= 10 && M >= 32 * per_lane * per_lane ? static_cast<int>(per_lane) : 0;
}

// One token quantized by one warp (K <= 256 * NCH): no barrier between the two passes, and NCH loads of a lane in flight.
template <int DT, int NCH>
__device__ __forceinline__ void quant_token_warp(const void* x, int64_t m, int64_t K, int64_t ldx, float eps, int8_t* __restrict__ q,
                                                 float* __restrict__ scale, int32_t* __restrict__ rowsum) {
    const int chunks = static_cast<int>(K >> 3), lane = threadIdx.x & 31;
    Raw8<DT> r[NCH];
#pragma unroll
    for (int c = 0; c < NCH; ++c) load_raw8<DT>(x, m * ldx + 8 * static_cast<int64_t>(lane + 32 * c), lane + 32 * c < chunks, r[c]);
    uint32_t bits = 0;
#pragma unroll
    for (int c = 0; c < NCH; ++c) bits = max_bits8<DT>(r[c], bits);
    bits = warp_max_bits<DT>(bits);
    bool fast = fast_bits<DT>(bits);
    float mx = bits_value<DT>(bits);
    if (!fast) {  // uniform over the warp
        mx = 0.f;
#pragma unroll
        for (int c = 0; c < NCH; ++c) mx = max_abs8<DT>(r[c], mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const float s = act_scale_from_absmax<DT>(mx, eps);
    fast = fast && s < INFINITY;
    int sum = 0;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        const int i = lane + 32 * c;
        if (i < chunks) {
            const uint2 w = fast ? quantize8_fast<DT>(r[c], s) : quantize8_any<DT>(r[c], s);
            sum = sum_bytes(w, sum);
            *reinterpret_cast<uint2*>(q + m * K + 8 * static_cast<int64_t>(i)) = w;
        }
    }
    if (rowsum) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    if (lane == 0) {
        scale[m] = s;
        if (rowsum) rowsum[m] = sum;
    }
}

template <int DT, int NCH>
__global__ void __launch_bounds__(AQ_THREADS)
    act_quant_warp_kernel(const void* x, int M, int64_t K, int64_t ldx, float eps, int8_t* __restrict__ q, float* __restrict__ scale,
                          int32_t* __restrict__ rowsum, int x_ready) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (!x_ready) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int m = blockIdx.x * (AQ_THREADS / 32) + (threadIdx.x >> 5);
    if (m < M) quant_token_warp<DT, NCH>(x, m, K, ldx, eps, q, scale, rowsum);
    if (x_ready && blockIdx.x == 0) asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// ---- what the contraction for many tokens needs in front of it, in one launch: every weight as one signed byte, and the
// quantized tokens.  Both are bound by memory and neither fills the chip alone for a thousand tokens, so they share it.

// byte-wise code - 1 of four codes: the borrow of a byte never leaves it, its top bit is set first
__device__ __forceinline__ uint32_t codes_to_s8(uint32_t v) { return ((v | 0x80808080u) - 0x01010101u) ^ 0x80808080u; }

// Packed word i (16 codes) of an [N, K/4] matrix to int8 [N, K]; a warp reads 128 bytes and writes 512.
__device__ __forceinline__ void expand_word(uint32_t w, int64_t i, int layout, int8_t* __restrict__ w8) {
    const uint32_t m = 0x03030303u;
    if (layout == WF_LAYOUT_WF16) {  // bit pairs j of the four bytes: weights 16 i + 4 j .. + 3
        *reinterpret_cast<uint4*>(w8 + 16 * i) =
            make_uint4(codes_to_s8(w & m), codes_to_s8((w >> 2) & m), codes_to_s8((w >> 4) & m), codes_to_s8((w >> 6) & m));
    } else {  // I2_S: byte b of a block of 32 holds weights b, b + 32, b + 64, b + 96 at bits 7:6, 5:4, 3:2, 1:0
        int8_t* d = w8 + (i >> 3) * 128 + (i & 7) * 4;
#pragma unroll
        for (int g = 0; g < 4; ++g) *reinterpret_cast<uint32_t*>(d + 32 * g) = codes_to_s8((w >> (6 - 2 * g)) & m);
    }
}

// Blocks 0 .. expand_blocks - 1 expand the weights, the others quantize: one token each, the row in CHUNKS chunks per thread
// or read twice (0), or one token per warp of -CHUNKS chunks per lane.  DT = WF_I8: the tokens are int8 already and every
// block expands.
template <int DT, int CHUNKS>
__global__ void __launch_bounds__(AQ_THREADS)
    quantize_expand_kernel(const void* x, int M, int64_t K, int64_t ldx, float eps, int8_t* __restrict__ q, float* __restrict__ scale,
                           const uint32_t* codes, int layout, int64_t words, int8_t* __restrict__ w8, int expand_blocks) {
    __shared__ float shf[AQ_THREADS / 32];
    __shared__ int shi[AQ_THREADS / 32];
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // x, and the workspace that the previous call may still read
    if (static_cast<int>(blockIdx.x) < expand_blocks) {
        constexpr int U = 4;  // words in flight per thread
        const int64_t stride = static_cast<int64_t>(expand_blocks) * AQ_THREADS;
        for (int64_t i = static_cast<int64_t>(blockIdx.x) * AQ_THREADS + threadIdx.x; i < words; i += U * stride) {
            uint32_t w[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i + u * stride < words) w[u] = codes[i + u * stride];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i + u * stride < words) expand_word(w[u], i + u * stride, layout, w8);
        }
    } else if constexpr (DT != WF_I8) {
        const int64_t m = static_cast<int64_t>(blockIdx.x) - expand_blocks;
        if constexpr (CHUNKS > 0) {
            quant_token_reg<DT, CHUNKS>(x, m, K, ldx, eps, q, scale, nullptr, shf, shi);
        } else if constexpr (CHUNKS < 0) {
            const int64_t tok = m * (AQ_THREADS / 32) + (threadIdx.x >> 5);
            if (tok < M) quant_token_warp<DT, -CHUNKS>(x, tok, K, ldx, eps, q, scale, nullptr);
        } else {
            quant_token<DT>(x, m, K, ldx, eps, q, scale, nullptr, shf, shi);
        }
    }
}

template <int DT>
static cudaError_t launch_token_quant(cudaLaunchConfig_t& lc, const void* x, int64_t M, int64_t K, int64_t ldx, float eps, int8_t* q,
                                      float* scale, int32_t* rowsum, int x_ready) {
    const int per_lane = warp_form_chunks(M, K);
    if (per_lane) {
        lc.gridDim = dim3(static_cast<unsigned>((M + AQ_THREADS / 32 - 1) / (AQ_THREADS / 32)));
        const int mm = static_cast<int>(M);
        if (per_lane <= 3) return cudaLaunchKernelEx(&lc, act_quant_warp_kernel<DT, 3>, x, mm, K, ldx, eps, q, scale, rowsum, x_ready);
        if (per_lane <= 6) return cudaLaunchKernelEx(&lc, act_quant_warp_kernel<DT, 6>, x, mm, K, ldx, eps, q, scale, rowsum, x_ready);
        return cudaLaunchKernelEx(&lc, act_quant_warp_kernel<DT, 10>, x, mm, K, ldx, eps, q, scale, rowsum, x_ready);
    }
    const int64_t per_thread = ((K >> 3) + AQ_THREADS - 1) / AQ_THREADS;
    if (per_thread <= 2) return cudaLaunchKernelEx(&lc, act_quant_token_reg_kernel<DT, 2>, x, K, ldx, eps, q, scale, rowsum, x_ready);
    if (per_thread <= 4) return cudaLaunchKernelEx(&lc, act_quant_token_reg_kernel<DT, 4>, x, K, ldx, eps, q, scale, rowsum, x_ready);
    if (per_thread <= 7) return cudaLaunchKernelEx(&lc, act_quant_token_reg_kernel<DT, 7>, x, K, ldx, eps, q, scale, rowsum, x_ready);
    return cudaLaunchKernelEx(&lc, act_quant_token_kernel<DT>, x, K, ldx, eps, q, scale, rowsum, x_ready);
}

extern "C" int wf_act_quant_i8(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, int mode, float eps, int8_t* q,
                               float* scale, int32_t* rowsum, void* stream) {
    return act_quant_impl(x, x_dtype, M, K, ldx, mode, eps, q, scale, rowsum, 0, stream);
}

// Per-token quantization whose launch neither reads nor overwrites anything the kernels still running ahead of it use
// (x_ready != 0): see wf_prefill_quantize.
int wf_act_quant_token_ready(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, float eps, int8_t* q, float* scale,
                             int32_t* rowsum, int x_ready, void* stream) {
    return act_quant_impl(x, x_dtype, M, K, ldx, WF_ACT_PER_TOKEN, eps, q, scale, rowsum, x_ready, stream);
}

template <int DT>
static cudaError_t launch_quantize_expand(cudaLaunchConfig_t& lc, const void* x, int64_t M, int64_t K, int64_t ldx, float eps, int8_t* q,
                                          float* scale, const uint32_t* codes, int layout, int64_t words, int8_t* w8) {
    // four words per thread and pass; at most eight blocks per SM, so that the first tokens start beside them
    const int64_t most = 8 * static_cast<int64_t>(num_sms()), want = (words + 4 * AQ_THREADS - 1) / (4 * AQ_THREADS);
    const int blocks = static_cast<int>(want < most ? want : most);
    const int mm = static_cast<int>(M);
    lc.gridDim = dim3(static_cast<unsigned>(blocks + (DT == WF_I8 ? 0 : M)));
    if constexpr (DT == WF_I8) {
        return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, 0>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
    } else {
        const int per_lane = warp_form_chunks(M, K);
        if (per_lane) {
            lc.gridDim = dim3(static_cast<unsigned>(blocks + (M + AQ_THREADS / 32 - 1) / (AQ_THREADS / 32)));
            if (per_lane <= 3) return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, -3>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
            if (per_lane <= 6) return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, -6>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
            return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, -10>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
        }
        const int64_t per_thread = ((K >> 3) + AQ_THREADS - 1) / AQ_THREADS;
        if (per_thread <= 2) return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, 2>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
        if (per_thread <= 4) return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, 4>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
        if (per_thread <= 7) return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, 7>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
        return cudaLaunchKernelEx(&lc, quantize_expand_kernel<DT, 0>, x, mm, K, ldx, eps, q, scale, codes, layout, words, w8, blocks);
    }
}

// The launch in front of the contraction for many tokens: w8 [N, K] int8 from the packed weights and, unless x is int8
// already, q [M, K] and scale [M] (the bits of wf_act_quant_i8 per token).  Arguments as checked by wf_bitlinear_prefill.
int wf_quantize_expand(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, float eps, int8_t* q, float* scale, const uint8_t* codes,
                       int layout, int64_t N, int8_t* w8, void* stream) {
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(AQ_THREADS);
    lc.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    const uint32_t* words = reinterpret_cast<const uint32_t*>(codes);
    const int64_t n = N * (K / 16);
    switch (x_dtype) {
        case WF_F32: WF_CUDA(launch_quantize_expand<WF_F32>(lc, x, M, K, ldx, eps, q, scale, words, layout, n, w8)); break;
        case WF_BF16: WF_CUDA(launch_quantize_expand<WF_BF16>(lc, x, M, K, ldx, eps, q, scale, words, layout, n, w8)); break;
        case WF_F16: WF_CUDA(launch_quantize_expand<WF_F16>(lc, x, M, K, ldx, eps, q, scale, words, layout, n, w8)); break;
        default: WF_CUDA(launch_quantize_expand<WF_I8>(lc, x, M, K, ldx, eps, q, scale, words, layout, n, w8)); break;
    }
    return WF_OK;
}

static int act_quant_impl(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, int mode, float eps, int8_t* q, float* scale,
                          int32_t* rowsum, int x_ready, void* stream) {
    WF_REQUIRE(x && q && scale, "wf_act_quant_i8: null pointer");
    WF_REQUIRE(M > 0 && K > 0 && K % 8 == 0, "wf_act_quant_i8: need M > 0 and K a positive multiple of 8 (M=%lld K=%lld)",
               (long long)M, (long long)K);
    WF_REQUIRE(M <= 0x7fffffff, "wf_act_quant_i8: M too large");
    WF_REQUIRE(is_float_dtype(x_dtype), "wf_act_quant_i8: unsupported dtype %d", x_dtype);
    WF_REQUIRE(ldx >= K && (ldx * dtype_size(x_dtype)) % 16 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0,
               "wf_act_quant_i8: rows of x must be 16-byte aligned");
    WF_REQUIRE(reinterpret_cast<uintptr_t>(q) % 8 == 0, "wf_act_quant_i8: q must be 8-byte aligned");
    if (int rc = require_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (mode == WF_ACT_PER_TOKEN) {
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(static_cast<unsigned>(M));
        lc.blockDim = dim3(AQ_THREADS);
        lc.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
        switch (x_dtype) {
            case WF_F32: WF_CUDA(launch_token_quant<WF_F32>(lc, x, M, K, ldx, eps, q, scale, rowsum, x_ready)); break;
            case WF_BF16: WF_CUDA(launch_token_quant<WF_BF16>(lc, x, M, K, ldx, eps, q, scale, rowsum, x_ready)); break;
            default: WF_CUDA(launch_token_quant<WF_F16>(lc, x, M, K, ldx, eps, q, scale, rowsum, x_ready)); break;
        }
    } else if (mode == WF_ACT_PER_TENSOR) {
        WF_REQUIRE(x_dtype == WF_F32, "wf_act_quant_i8: per-tensor mode takes fp32 input (as the operator it replaces)");
        // scale[0] doubles as the reduction cell: 0.0f has all-zero bits, the identity of the unsigned max
        WF_CUDA(cudaMemsetAsync(scale, 0, sizeof(float), st));
        int64_t blocks = (M * (K / 4) + AQ_THREADS - 1) / AQ_THREADS;
        if (blocks > 148 * 8) blocks = 148 * 8;
        tensor_absmax_kernel<<<(unsigned)blocks, AQ_THREADS, 0, st>>>(static_cast<const float*>(x), M, K, ldx,
                                                                     reinterpret_cast<unsigned*>(scale));
        tensor_quant_kernel<<<(unsigned)M, AQ_THREADS, 0, st>>>(static_cast<const float*>(x), K, ldx,
                                                                reinterpret_cast<const unsigned*>(scale), q, rowsum);
        publish_tensor_scale<<<1, 1, 0, st>>>(scale);
    } else {
        return fail(WF_E_ARG, "wf_act_quant_i8: unknown mode %d", mode);
    }
    WF_CUDA(cudaGetLastError());
    return WF_OK;
}

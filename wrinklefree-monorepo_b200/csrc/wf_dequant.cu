// Operands of the straight-through backward pass: the quantized weights and the quantized tokens as the values that the
// reference's fake-quantized tensors hold, in one pass each.  Both are bound by the bytes they write (6912 x 2560 weights
// in bf16: 35 MB); the operator chains they stand for (unpack, convert, scale; convert twice, divide, convert) moved
// three to four times as many.
#include "wf_common.cuh"

namespace wf {

constexpr int DQ_THREADS = 256;

template <int DT>
__device__ __forceinline__ uint32_t pair_bits(float a, float b) {
    if constexpr (DT == WF_BF16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&v);
    } else {
        const __half2 v = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&v);
    }
}
// E values as one 16-byte store
template <int DT, int E>
__device__ __forceinline__ void store16(void* out, int64_t at, const float (&v)[E]) {
    uint4 w;
    if constexpr (DT == WF_F32) {
        w = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
        *reinterpret_cast<uint4*>(static_cast<float*>(out) + at) = w;
    } else {
        w = make_uint4(pair_bits<DT>(v[0], v[1]), pair_bits<DT>(v[2], v[3]), pair_bits<DT>(v[4], v[5]), pair_bits<DT>(v[6], v[7]));
        *reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + at) = w;
    }
}

// One thread per 16 bytes of output (8 or 4 weights of a packed WF16 word): (code - 1) * scale, rounded to the type.
template <int DT>
__global__ void __launch_bounds__(DQ_THREADS) dequant_weights_kernel(const uint32_t* __restrict__ codes, const float* __restrict__ scale,
                                                                     void* __restrict__ out, int64_t words) {
    constexpr int E = DT == WF_F32 ? 4 : 8, PARTS = 16 / E;
    const float s = rnd<DT>(*scale);
    const int64_t total = words * PARTS, stride = static_cast<int64_t>(gridDim.x) * DQ_THREADS;
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * DQ_THREADS + threadIdx.x; t < total; t += stride) {
        const int part = static_cast<int>(t % PARTS);
        const uint32_t w = codes[t / PARTS] >> (2 * (E / 4) * part);  // bit pair j of byte b: weight 4 j + b
        float v[E];
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = __fmul_rn(static_cast<float>(static_cast<int>((w >> (8 * (e & 3) + 2 * (e >> 2))) & 3u) - 1), s);
        store16<DT, E>(out, t * E, v);
    }
}

// One block per token: q / scale rounded to the type of the activations (XDT), stored as DT.  A token has at most 256
// different values, so each thread divides once and the row is looked up (a division per element took 21 us for 4096 tokens
// of 2560 values, 31 MB).
template <int XDT, int DT>
__global__ void __launch_bounds__(DQ_THREADS) dequant_tokens_kernel(const int8_t* __restrict__ q, const float* __restrict__ scale,
                                                                    void* __restrict__ out, int K) {
    constexpr int E = DT == WF_F32 ? 4 : 8;
    __shared__ uint32_t table[256];  // by the byte of q: the bits of the value
    static_assert(DQ_THREADS == 256, "one entry per thread");
    const int64_t row = static_cast<int64_t>(blockIdx.x) * K;
    const float v = rnd<XDT>(__fdiv_rn(static_cast<float>(static_cast<int8_t>(threadIdx.x)), rnd<XDT>(scale[blockIdx.x])));
    table[threadIdx.x] = DT == WF_F32 ? __float_as_uint(v) : (pair_bits<DT == WF_F32 ? WF_BF16 : DT>(v, 0.f) & 0xffffu);
    __syncthreads();
    for (int k = threadIdx.x * E; k < K; k += DQ_THREADS * E) {
        uint4 o;
        if constexpr (E == 8) {
            const uint2 u = *reinterpret_cast<const uint2*>(q + row + k);
            o.x = table[u.x & 0xff] | (table[(u.x >> 8) & 0xff] << 16);
            o.y = table[(u.x >> 16) & 0xff] | (table[u.x >> 24] << 16);
            o.z = table[u.y & 0xff] | (table[(u.y >> 8) & 0xff] << 16);
            o.w = table[(u.y >> 16) & 0xff] | (table[u.y >> 24] << 16);
            *reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + row + k) = o;
        } else {
            const uint32_t u = *reinterpret_cast<const uint32_t*>(q + row + k);
            o = make_uint4(table[u & 0xff], table[(u >> 8) & 0xff], table[(u >> 16) & 0xff], table[u >> 24]);
            *reinterpret_cast<uint4*>(static_cast<float*>(out) + row + k) = o;
        }
    }
}

static unsigned dq_grid(int64_t threads) {
    const int64_t blocks = (threads + DQ_THREADS - 1) / DQ_THREADS, most = 16 * static_cast<int64_t>(num_sms());
    return static_cast<unsigned>(blocks < most ? blocks : most);
}

template <int XDT>
static void launch_tokens(const int8_t* q, const float* scale, void* out, int dtype, int64_t M, int64_t K, cudaStream_t st) {
    const unsigned grid = static_cast<unsigned>(M);
    const int k = static_cast<int>(K);
    if (dtype == WF_F32) dequant_tokens_kernel<XDT, WF_F32><<<grid, DQ_THREADS, 0, st>>>(q, scale, out, k);
    else if (dtype == WF_BF16) dequant_tokens_kernel<XDT, WF_BF16><<<grid, DQ_THREADS, 0, st>>>(q, scale, out, k);
    else dequant_tokens_kernel<XDT, WF_F16><<<grid, DQ_THREADS, 0, st>>>(q, scale, out, k);
}

}  // namespace wf

using namespace wf;

extern "C" int wf_dequant_weights(const uint8_t* codes, const float* scale, void* out, int dtype, int64_t N, int64_t K, void* stream) {
    WF_REQUIRE(codes && scale && out, "wf_dequant_weights: null pointer");
    WF_REQUIRE(N > 0 && K > 0 && K % 16 == 0, "wf_dequant_weights: need N > 0 and K a positive multiple of 16 (N=%lld K=%lld)", (long long)N, (long long)K);
    WF_REQUIRE(is_float_dtype(dtype), "wf_dequant_weights: unsupported dtype %d", dtype);
    WF_REQUIRE((reinterpret_cast<uintptr_t>(out) % 16 | reinterpret_cast<uintptr_t>(codes) % 4) == 0, "wf_dequant_weights: out must be 16-byte, codes 4-byte aligned");
    if (int rc = require_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(codes);
    const int64_t words = N * (K / 16);
    if (dtype == WF_F32) dequant_weights_kernel<WF_F32><<<dq_grid(4 * words), DQ_THREADS, 0, st>>>(w, scale, out, words);
    else if (dtype == WF_BF16) dequant_weights_kernel<WF_BF16><<<dq_grid(2 * words), DQ_THREADS, 0, st>>>(w, scale, out, words);
    else dequant_weights_kernel<WF_F16><<<dq_grid(2 * words), DQ_THREADS, 0, st>>>(w, scale, out, words);
    WF_CUDA(cudaGetLastError());
    return WF_OK;
}

extern "C" int wf_dequant_tokens(const int8_t* q, const float* scale, int x_dtype, void* out, int dtype, int64_t M, int64_t K, void* stream) {
    WF_REQUIRE(q && scale && out, "wf_dequant_tokens: null pointer");
    WF_REQUIRE(M > 0 && M < (1LL << 31) && K > 0 && K % 8 == 0 && K < (1LL << 30), "wf_dequant_tokens: need M > 0 and K a positive multiple of 8 (M=%lld K=%lld)", (long long)M, (long long)K);
    WF_REQUIRE(is_float_dtype(x_dtype) && is_float_dtype(dtype), "wf_dequant_tokens: unsupported dtype %d or %d", x_dtype, dtype);
    WF_REQUIRE((reinterpret_cast<uintptr_t>(out) % 16 | reinterpret_cast<uintptr_t>(q) % 8) == 0, "wf_dequant_tokens: out must be 16-byte, q 8-byte aligned");
    if (int rc = require_device()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (x_dtype == WF_F32) launch_tokens<WF_F32>(q, scale, out, dtype, M, K, st);
    else if (x_dtype == WF_BF16) launch_tokens<WF_BF16>(q, scale, out, dtype, M, K, st);
    else launch_tokens<WF_F16>(q, scale, out, dtype, M, K, st);
    WF_CUDA(cudaGetLastError());
    return WF_OK;
}

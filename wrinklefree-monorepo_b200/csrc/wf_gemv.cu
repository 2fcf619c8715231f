// One or two tokens through one projection, or through up to four that read the same tokens (q/k/v, gate/up): the launches
// of a decode step.
//
// What bounds such a launch is latency: 4096 x 4096 packed weights are 0.6 us of memory traffic.  The kernel for stacks of
// problems (wf_decode.cu: TMA ring, producer warp, legacy tensor cores for up to 8 tokens, two barriers and a shared-memory
// reduction per item) takes 5 to 6 us per launch of a chain.  Here every warp asks for its first rows of weights straight
// into registers before it waits for the previous kernel; what is left behind that wait is: read x, quantize it
// (each CTA for itself), two barriers, dot products on dp4a, a shuffle reduction, the store.
//   * LPR lanes share a row, each takes CH chunks of 16 bytes (64 weights); a warp holds 32 / LPR rows per task, and the
//     chunk just used is replaced at once by that of the warp's next task;
//   * no shifts: the four bit positions of a word are masked in place and go to four accumulators, which carry factors of
//     1, 4, 16 and 64 until the end (exact);
//   * x lies in shared memory in the order in which a word's four bit positions need it, 16 bytes per word, the words of
//     neighbouring chunks side by side (no bank conflicts).
#include "wf_common.cuh"
#include "wf_quant8.cuh"

namespace wf {

constexpr int GV_THREADS = 512, GV_WARPS = GV_THREADS / 32;
constexpr int GV_MAX_P = 4;
constexpr int GV_MAX_TOKENS = 2;
constexpr int GV_MAX_K = 16384;
constexpr int GV_XCH = 4;  // chunks of 8 activations per thread: tokens x K <= 16384 unless x is int8

struct GemvProblem {
    const uint8_t* codes;
    const float* w_scale;
    const void* bias;
    void* y;
    int32_t* acc_out;
    int64_t ldy;
    float w_scale_host;
    int bias_dtype, y_dtype;
    int N, task0;  // rows; first task
};
struct GemvParams {
    const void* x;
    const float* x_scale;
    const void* x2;
    const void* norm_w;
    void* h_out;
    int64_t ldx;
    float eps, norm_eps;
    int x_dtype, x_mode, layout;
    int M, K, chunks;  // chunks of 64 weights per row
    int lpr_log2, segs, tasks, P;
    GemvProblem p[GV_MAX_P];
};

__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Where the four int8 of activations k .. k + 3 go inside a token's K bytes: word w (16 weights) of chunk kc, bit position j.
__device__ __forceinline__ int x_slot(int layout, int chunks, int k) {
    int kc, w, j;
    if (layout == WF_LAYOUT_WF16) {
        kc = k >> 6; w = (k >> 4) & 3; j = (k >> 2) & 3;
    } else {  // I2_S: byte b of a block of 32 holds weights b, b + 32, b + 64, b + 96 at bit positions 3, 2, 1, 0
        const int i = (k & 31) >> 2;
        kc = ((k >> 7) << 1) + (i >> 2); w = i & 3; j = 3 - ((k >> 5) & 3);
    }
    return (w * chunks + kc) * 16 + 4 * j;
}

__device__ __forceinline__ float gv_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float gv_act(float a, int mode) {  // as the stand-alone activation kernel
    if (mode == WF_X_SILU) return gv_round(a / (1.0f + __expf(-a)));
    const float r = gv_round(fmaxf(a, 0.f));
    return gv_round(r * r);
}

__device__ __forceinline__ uint4 pack8_bf16(const float (&a)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a[2 * i], a[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// x -> int8 in shared memory, multipliers and sums.  512 / MT threads per token.  Ends with a barrier.
template <int DT, int MT>
__device__ __forceinline__ void gemv_quantize(const GemvParams& p, uint8_t* s_x, float* s_inv, int* s_sum, uint32_t* s_red, float* s_redf) {
    constexpr int TPT = GV_THREADS / MT, WPT = TPT / 32;  // threads and warps per token
    const int tid = threadIdx.x, tok = tid / TPT, t = tid % TPT, lane = tid & 31, w0 = tok * WPT;
    const bool live = tok < p.M;
    const int chunks8 = p.K >> 3;
    const int64_t base = static_cast<int64_t>(tok) * p.ldx;
    Raw8<DT> r[GV_XCH];
#pragma unroll
    for (int c = 0; c < GV_XCH; ++c)
        load_raw8<DT>(p.x, base + 8 * (t + c * TPT), live && t + c * TPT < chunks8, r[c]);  // zeros where there is nothing
    if constexpr (DT == WF_BF16) {
        if (p.x_mode != WF_X_PLAIN) {
            // the arithmetic of the stand-alone kernels: the same bits for the activations; the norm's mean of squares is summed in
            // another order (square by square, and over other chunks), which may move its last bit and with it single int8 codes
            Raw8<DT> r2[GV_XCH];
#pragma unroll
            for (int c = 0; c < GV_XCH; ++c)
                load_raw8<DT>(p.x2 ? p.x2 : p.x, base + 8 * (t + c * TPT), p.x2 != nullptr && live && t + c * TPT < chunks8, r2[c]);
            float ss = 0.f;
#pragma unroll
            for (int c = 0; c < GV_XCH; ++c) {
                if (c * TPT + (t & ~31) >= chunks8) continue;  // nothing for this warp
                float a[8], b[8];
                values8<DT>(r[c], a);
                values8<DT>(r2[c], b);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    if (p.x_mode == WF_X_NORM) {
                        if (p.x2) a[e] = gv_round(a[e] + b[e]);
                        ss += a[e] * a[e];
                    } else {
                        a[e] = gv_round(gv_act(a[e], p.x_mode) * b[e]);
                    }
                }
                r[c].v[0] = pack8_bf16(a);
            }
            if (p.x_mode == WF_X_NORM) {
                if (p.h_out && blockIdx.x == 0) {  // the updated residual stream, written by one CTA of the launch
#pragma unroll
                    for (int c = 0; c < GV_XCH; ++c)
                        if (live && t + c * TPT < chunks8)
                            *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.h_out) + base + 8 * (t + c * TPT)) = r[c].v[0];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                if (lane == 0) s_redf[tid >> 5] = ss;
                __syncthreads();
                float tot = 0.f;
#pragma unroll
                for (int i = 0; i < WPT; ++i) tot += s_redf[w0 + i];
                const float rn = rsqrtf(tot / static_cast<float>(p.K) + p.norm_eps);
#pragma unroll
                for (int c = 0; c < GV_XCH; ++c) {
                    if (c * TPT + (t & ~31) >= chunks8) continue;
                    Raw8<DT> wv;
                    load_raw8<DT>(p.norm_w, 8 * (t + c * TPT), live && t + c * TPT < chunks8, wv);
                    float a[8], g[8];
                    values8<DT>(r[c], a);
                    values8<DT>(wv, g);
#pragma unroll
                    for (int e = 0; e < 8; ++e) a[e] = gv_round(a[e] * rn) * g[e];
                    r[c].v[0] = pack8_bf16(a);
                }
            }
        }
    }
    uint32_t bits = 0;
#pragma unroll
    for (int c = 0; c < GV_XCH; ++c)
        if (c * TPT < chunks8) bits = max_bits8<DT>(r[c], bits);
    bits = warp_max_bits<DT>(bits);
    if (lane == 0) s_red[tid >> 5] = bits;
    if (tid < MT) s_sum[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < WPT; ++i) bits = max(bits, s_red[w0 + i]);
    float mx = bits_value<DT>(bits);
    bool fast = fast_bits<DT>(bits);
    if (__syncthreads_or(!fast)) {  // an infinity, a NaN or a maximum out of range among the tokens
        mx = 0.f;
#pragma unroll
        for (int c = 0; c < GV_XCH; ++c)
            if (c * TPT < chunks8) mx = max_abs8<DT>(r[c], mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) s_redf[tid >> 5] = mx;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < WPT; ++i) mx = fmaxf(mx, s_redf[w0 + i]);
    }
    const float s = act_scale_from_absmax<DT>(mx, p.eps);
    fast = fast && s < INFINITY;
    int sum = 0;
#pragma unroll
    for (int c = 0; c < GV_XCH; ++c) {
        const int k = 8 * (t + c * TPT);
        if (live && k < p.K) {
            const uint2 q = fast ? quantize8_fast<DT>(r[c], s) : quantize8_any<DT>(r[c], s);
            sum = sum_bytes(q, sum);
            uint8_t* d = s_x + tok * p.K;
            *reinterpret_cast<uint32_t*>(d + x_slot(p.layout, p.chunks, k)) = q.x;
            *reinterpret_cast<uint32_t*>(d + x_slot(p.layout, p.chunks, k + 4)) = q.y;
        }
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0 && live) atomicAdd(&s_sum[tok], sum);
    if (t == 0) s_inv[tok] = __fdiv_rn(1.0f, s);
    __syncthreads();
}

// x is int8 already
template <int MT>
__device__ __forceinline__ void gemv_stage_i8(const GemvParams& p, uint8_t* s_x, float* s_inv, int* s_sum) {
    constexpr int TPT = GV_THREADS / MT;
    const int tid = threadIdx.x, tok = tid / TPT, t = tid % TPT, lane = tid & 31;
    if (tid < MT) s_sum[tid] = 0;
    __syncthreads();
    int sum = 0;
    if (tok < p.M) {
        const int8_t* row = static_cast<const int8_t*>(p.x) + static_cast<int64_t>(tok) * p.ldx;
        uint8_t* d = s_x + tok * p.K;
        for (int k = t * 16; k < p.K; k += TPT * 16) {
            const uint4 v = ld16_chained(row + k);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sum = __dp4a(static_cast<int>(w[i]), 0x01010101, sum);
                *reinterpret_cast<uint32_t*>(d + x_slot(p.layout, p.chunks, k + 4 * i)) = w[i];
            }
        }
        if (t == 0) s_inv[tok] = p.x_scale ? __frcp_rn(*static_cast<const volatile float*>(p.x_scale + tok)) : 1.0f;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0 && tok < p.M) atomicAdd(&s_sum[tok], sum);
    __syncthreads();
}

template <int MT, int CH>
__global__ void __launch_bounds__(GV_THREADS, 2) gemv_kernel(const __grid_constant__ GemvParams p) {
    extern __shared__ __align__(16) uint8_t s_x[];  // [MT][K]
    __shared__ float s_inv[MT], s_redf[GV_WARPS];
    __shared__ int s_sum[MT];
    __shared__ uint32_t s_red[GV_WARPS];
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lpr = 1 << p.lpr_log2, col = lane & (lpr - 1), rows = 32 >> p.lpr_log2, sub = lane >> p.lpr_log2;

    // tasks are dealt to the CTAs first, so that a small projection uses every SM
    int task = warp * gridDim.x + blockIdx.x;
    const int stride = gridDim.x * GV_WARPS;
    uint4 w[CH];
    int pi = 0, row = 0;          // problem and row (of this lane) of the task whose weights are being requested
    const uint8_t* rp = nullptr;  // null: no such row
    auto locate = [&](int tk) {
        pi = 0;
#pragma unroll
        for (int i = 1; i < GV_MAX_P; ++i)
            if (i < p.P && tk >= p.p[i].task0) pi = i;
        row = (tk - p.p[pi].task0) * rows + sub;
        rp = tk < p.tasks && row < p.p[pi].N ? p.p[pi].codes + static_cast<int64_t>(row) * (p.K / 4) : nullptr;
    };
    auto load = [&](int kc) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (rp && kc < p.chunks) v = __ldg(reinterpret_cast<const uint4*>(rp) + kc);
        return v;
    };
    locate(task);
#pragma unroll
    for (int c = 0; c < CH; ++c) w[c] = load(col + c * lpr);  // the weights do not depend on the previous kernel
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    if (p.x_dtype == WF_I8) gemv_stage_i8<MT>(p, s_x, s_inv, s_sum);
    else if (p.x_dtype == WF_BF16) gemv_quantize<WF_BF16, MT>(p, s_x, s_inv, s_sum, s_red, s_redf);
    else if (p.x_dtype == WF_F16) gemv_quantize<WF_F16, MT>(p, s_x, s_inv, s_sum, s_red, s_redf);
    else gemv_quantize<WF_F32, MT>(p, s_x, s_inv, s_sum, s_red, s_redf);

    for (; task < p.tasks; task += stride) {
        const int now = pi, now_row = row;
        int acc[MT][4];
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0;
        for (int seg = 0; seg < p.segs; ++seg) {  // CH chunks of every lane at a time; what is used up is requested anew
            const int kc0 = col + seg * CH * lpr;
            int next = kc0 + CH * lpr;
            if (seg + 1 == p.segs) {
                locate(task + stride);
                next = col;
            }
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const int kc = min(kc0 + c * lpr, p.chunks - 1);  // a chunk past the row holds zeros
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t ww = i == 0 ? w[c].x : (i == 1 ? w[c].y : (i == 2 ? w[c].z : w[c].w));
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const uint4 xv = *reinterpret_cast<const uint4*>(s_x + m * p.K + (i * p.chunks + kc) * 16);
                        acc[m][0] = dp4a_us(ww & 0x03030303u, xv.x, acc[m][0]);
                        acc[m][1] = dp4a_us(ww & 0x0c0c0c0cu, xv.y, acc[m][1]);
                        acc[m][2] = dp4a_us(ww & 0x30303030u, xv.z, acc[m][2]);
                        acc[m][3] = dp4a_us(ww & 0xc0c0c0c0u, xv.w, acc[m][3]);
                    }
                }
                w[c] = load(next + c * lpr);
            }
        }
        const GemvProblem& q = p.p[now];
        int mine = 0;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            int a = acc[m][0] + (acc[m][1] >> 2) + (acc[m][2] >> 4) + (acc[m][3] >> 6);
            for (int o = lpr >> 1; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (col == m) mine = a;  // lane m of the row stores token m
        }
        if (now_row < q.N && col < MT && col < p.M) {
            const int v = mine - s_sum[col];
            float o = rescale(v, s_inv[col], q.w_scale ? __ldg(q.w_scale) : q.w_scale_host);
            if (q.bias) o = __fadd_rn(o, load1_rt(q.bias, q.bias_dtype, now_row));
            store1_rt(q.y, q.y_dtype, col * q.ldy + now_row, o);
            if (q.acc_out) q.acc_out[static_cast<int64_t>(col) * q.N + now_row] = v;
        }
    }
}

template <int MT, int CH>
static cudaError_t launch_gemv(const cudaLaunchConfig_t& lc, const GemvParams& p) {
    static PerDeviceOnce configured;
    const int dev = current_device();
    if (configured.needs(dev)) {
        const cudaError_t e = cudaFuncSetAttribute(gemv_kernel<MT, CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, MT * GV_MAX_K);
        if (e != cudaSuccess) return e;
        configured.mark(dev);
    }
    return cudaLaunchKernelEx(&lc, gemv_kernel<MT, CH>, p);
}
template <int MT>
static cudaError_t launch_gemv_tokens(const cudaLaunchConfig_t& lc, int ch, const GemvParams& p) {
    if (ch == 1) return launch_gemv<MT, 1>(lc, p);
    if (ch == 2) return launch_gemv<MT, 2>(lc, p);
    if (ch == 3) return launch_gemv<MT, 3>(lc, p);
    return launch_gemv<MT, 4>(lc, p);
}

}  // namespace wf

using namespace wf;

// Whether the kernel above is the faster one for `weights` weights in P problems that read the same M tokens.  It wins
// where a launch is latency and loses where its weights are traffic: its loads are not kept in flight while x is read, and two
// tokens cost twice the dot products.  us per launch of a chain of int8 inputs, against the kernel for stacks: one token
// 2.3 / 3.3 (0.3 Mi weights), 2.6 / 4.5 (6.5 Mi), 3.3 / 6.3 (18 Mi), 6.9 / 7.6 (59 Mi); two tokens 3.0 / 4.5 (6.5 Mi),
// 4.0 / 6.4 (18 Mi).  Inside a decoder layer the neighbours hide part of that: 2560 x 6912 wide, one token 50.1 -> 45.3 us
// per layer up to 48 Mi, two tokens 45.1 -> 45.2 up to 12 Mi and 47.3 up to 20; 117 Mi (gate/up of the 8B shape) lost.
static bool gemv_pays(int64_t M, int64_t K, int64_t weights, int P) {
    return P >= 1 && P <= GV_MAX_P && M >= 1 && M <= GV_MAX_TOKENS && K <= GV_MAX_K && weights <= ((M == 1 ? 48LL : 12LL) << 20);
}

// Whether it quantizes floating-point tokens of this size itself (beside that it takes int8 tokens).
static bool gemv_quantizes(int64_t M, int64_t K) { return M * K <= GV_XCH * 8 * GV_THREADS; }

extern "C" int wf_decode_fuses_quant(int64_t M, int64_t K, int64_t weights, int problems) {
    return gemv_pays(M, K, weights, problems) && gemv_quantizes(M, K) ? 1 : 0;
}

// Whether it runs the group: worth it, the same tokens for every problem, nothing of what only the kernel for stacks does
// (an exchange, a prefetch, several residual outputs).
bool wf_gemv_takes(const wf_problem* q, int P) {
    int64_t weights = 0;
    for (int i = 0; i < P && i < GV_MAX_P; ++i) weights += static_cast<int64_t>(q[i].N) * q[i].K;
    if (!gemv_pays(q[0].M, q[0].K, weights, P) || (q[0].x_dtype != WF_I8 && !gemv_quantizes(q[0].M, q[0].K))) return false;
    const void* h_out = nullptr;  // the launch writes one residual stream
    for (int i = 0; i < P; ++i) {
        if (q[i].h_out && h_out && q[i].h_out != h_out) return false;
        if (q[i].h_out) h_out = q[i].h_out;
        if (q[i].xchg || (q[i].prefetch && q[i].prefetch_bytes > 0)) return false;
        if (q[i].M != q[0].M || q[i].K != q[0].K || q[i].layout != q[0].layout || q[i].x != q[0].x || q[i].ldx != q[0].ldx || q[i].x_scale != q[0].x_scale ||
            q[i].eps != q[0].eps || q[i].x_mode != q[0].x_mode || q[i].x2 != q[0].x2 || q[i].norm_w != q[0].norm_w || q[i].norm_eps != q[0].norm_eps)
            return false;
    }
    return true;
}

int wf_gemv_launch(const wf_problem* q, int P, unsigned flags, void* stream) {
    GemvParams p = {};
    p.x = q[0].x; p.x_scale = q[0].x_scale; p.x2 = q[0].x2; p.norm_w = q[0].norm_w; p.ldx = q[0].ldx;
    p.eps = q[0].eps; p.norm_eps = q[0].norm_eps; p.x_dtype = q[0].x_dtype; p.x_mode = q[0].x_mode; p.layout = q[0].layout;
    p.M = q[0].M; p.K = q[0].K; p.chunks = q[0].K / 64; p.P = P;
    const int sms = num_sms();
    // Lanes per row and chunks per lane: the shortest way of a warp through its tasks (in cycles, about: 40 per chunk and
    // token, 30 per token and step of a reduction).
    int best = 0, ch = 1;
    long long best_cost = 0;
    const long long warps = static_cast<long long>(sms) * GV_WARPS;
    for (int l = 2; l <= 5; ++l) {
        const int need = (p.chunks + (1 << l) - 1) >> l, segs = (need + 3) / 4, c = (need + segs - 1) / segs;
        long long tasks = 0;
        for (int i = 0; i < P; ++i) tasks += (q[i].N + (32 >> l) - 1) / (32 >> l);
        const long long cost = (tasks + warps - 1) / warps * (40 * segs * c + 30 * l);
        if (!best || cost < best_cost) {
            best = l; ch = c; p.segs = segs;
            best_cost = cost;
        }
    }
    p.lpr_log2 = best;
    const int rows = 32 >> best;
    for (int i = 0; i < P; ++i) {
        GemvProblem& g = p.p[i];
        g.codes = q[i].codes; g.w_scale = q[i].w_scale; g.bias = q[i].bias; g.y = q[i].y; g.acc_out = q[i].acc_out; g.ldy = q[i].ldy;
        g.w_scale_host = q[i].w_scale_host; g.bias_dtype = q[i].bias_dtype; g.y_dtype = q[i].y_dtype; g.N = q[i].N;
        g.task0 = p.tasks;
        p.tasks += (q[i].N + rows - 1) / rows;
        if (q[i].h_out) p.h_out = q[i].h_out;
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(static_cast<unsigned>(p.tasks < sms ? p.tasks : sms));
    lc.blockDim = dim3(GV_THREADS);
    lc.dynamicSmemBytes = static_cast<size_t>(p.M) * p.K;
    lc.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    if (flags & WF_FLAG_PDL) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
    }
    if (p.M == 1) WF_CUDA(launch_gemv_tokens<1>(lc, ch, p));
    else WF_CUDA(launch_gemv_tokens<2>(lc, ch, p));
    return WF_OK;
}

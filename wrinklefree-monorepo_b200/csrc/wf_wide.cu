// The contraction for many tokens: an int8 GEMM with both operands in shared memory.
//
//   acc[tok, n] = sum_k q[tok, k] * w[n, k]      (s8 x s8, s32 accumulators in tensor memory; w = code - 1)
//   y[tok, n]   = (float(acc) * inv_sx[tok]) * s_w + bias[n]
//
// The packed weights are expanded to one signed byte per weight ONCE per call, by the launch that quantizes the tokens
// (wf_actquant.cu), into the caller's workspace: the form that expands inside the contraction (wf_prefill.cu) does so again
// for every 128 tokens and holds the weights in tensor memory, which leaves room for 128 x 128 accumulators.  Here tensor
// memory holds two accumulators of 256 tokens x 256 weight rows per pair of SMs (cta_group::2) and both operands come by
// TMA: 32 KB per SM and 8.4 M multiply-adds.  What bounds it (8192 tokens, 6912 x 2560): all of it takes 90.5 us = 3.20 POPS, the
// tensor pipe active 84 % of the cycles under ncu; in one-off variants the instructions alone took 68 us = 4.28 POPS of the 4.58
// measured for the instruction and the copies alone 48 us: at the full rate operand reads and copies fill the
// shared-memory port, and every further byte is in their way.
//   * warp 0 (one lane): TMA of this CTA's 128 tokens and of its half of the weight rows, counted on the leader's barrier;
//     stages of two 128-byte atoms: with one atom per stage the barrier round trip and commit (about 220 ns per
//     stage) were the bound of every tile narrower than 256 rows;
//   * warp 1 of the leader (one lane): eight tcgen05.mma (K = 32) per stage and a commit to both CTAs;
//   * warps 2-5: epilogue under the next tile's instructions.
// Whole call from bf16 tokens: 8192 x (6912 x 2560) 137 -> 106 us, 1237 x (2560 x 6912) 34.4 -> 25.6 us.
#include "wf_common.cuh"

namespace wf {
__device__ int g_wide_status = 0;
}
#define WF_STATUS_WORD ::wf::g_wide_status
#include "wf_async.cuh"
#include "wf_tc.cuh"

namespace wf {

constexpr int WD_BM = 256;                // tokens per tile (128 per CTA of the pair)
constexpr int WD_MAX_BN = 256;            // weight rows per tile, at most
constexpr int WD_BK = 128;                // K of one 128-byte swizzle atom of int8
constexpr int WD_ATOMS = 2;               // atoms per stage
constexpr int WD_STAGES = 3;
constexpr int WD_A_BYTES = 128 * WD_BK;   // an atom of this CTA's 128 tokens
constexpr int WD_B_BYTES = WD_MAX_BN / 2 * WD_BK;  // an atom of this CTA's half of the weight rows
constexpr int WD_STAGE_BYTES = WD_ATOMS * (WD_A_BYTES + WD_B_BYTES);
constexpr int WD_OUT_BYTES = 32 * 128;    // one warp's staged output: 32 tokens x 128 bytes
constexpr int WD_THREADS = 6 * 32;
constexpr size_t WD_SMEM = 1024 + WD_STAGES * WD_STAGE_BYTES + 4 * 2 * WD_OUT_BYTES + 256;
static_assert(WD_SMEM <= 227 * 1024, "shared memory");

struct WideParams {
    const float* x_scale;  // [M] per-token multipliers (nullable: 1)
    const float* w_scale;
    const float* row_scale;  // [N] one scale per weight row (nullable; takes the place of w_scale)
    float w_scale_host;
    const void* bias;
    int bias_dtype;
    int M, N, K;
    int bn;                // weight rows per tile: a multiple of 64, at most WD_MAX_BN
    int tiles_m, tiles_n;
    void* y;               // used where rows of y cannot be written by TMA (not 16-byte aligned)
    int64_t ldy;
    int y_tma;
};

// The four MMAs of one 128-byte swizzle atom of K (both operands advance by 32 bytes, 2 in descriptor units)
__device__ __forceinline__ void mma_i8_ss_x4_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate_first) {
    asm volatile(
        "{\n .reg .pred p, q;\n .reg .b64 a1, a2, a3, b1, b2, b3;\n"
        " setp.ne.b32 p, %4, 0;\n setp.eq.b32 q, %5, %5;\n"
        " add.u64 a1, %1, 2;\n add.u64 a2, %1, 4;\n add.u64 a3, %1, 6;\n"
        " add.u64 b1, %2, 2;\n add.u64 b2, %2, 4;\n add.u64 b3, %2, 6;\n"
        " tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n"
        " tcgen05.mma.cta_group::2.kind::i8 [%0], a1, b1, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, q;\n"
        " tcgen05.mma.cta_group::2.kind::i8 [%0], a2, b2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, q;\n"
        " tcgen05.mma.cta_group::2.kind::i8 [%0], a3, b3, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, q;\n}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate_first), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t addr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
        "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
          "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
          "=r"(v[30]), "=r"(v[31])
        : "r"(addr));
}

// YDT: WF_F32 / WF_F16 / WF_BF16, the type of y.  ROWS: a scale per weight row (an instance of its own: asked at run time, it cost the
// others 0.2 of 27.4 us at 1237 x 2560 x 6912).
template <int YDT, bool ROWS>
__global__ void __launch_bounds__(WD_THREADS, 1)
    wide_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_y,
                const WideParams p) {
    constexpr int COLS = YDT == WF_F32 ? 32 : 64;  // weight rows of one staged output box: 128 bytes
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* ring = smem;                                       // [WD_STAGES][WD_ATOMS][A 128 x 128 B], [B bn/2 x 128 B]; 128-byte swizzle
    uint8_t* out_s = ring + WD_STAGES * WD_STAGE_BYTES;         // [4 warps][2][32 x 128 B], 128-byte swizzle
    uint64_t* full = reinterpret_cast<uint64_t*>(out_s + 4 * 2 * WD_OUT_BYTES);  // leader's copy: bytes of both CTAs
    uint64_t* empty = full + WD_STAGES;                         // multicast commit: the stage may be overwritten
    uint64_t* acc_full = empty + WD_STAGES;                     // multicast commit: the accumulator of a tile is complete
    uint64_t* acc_empty = acc_full + 2;                         // leader's copy: the epilogue warps of both CTAs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* poisoned = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();  // 0: leader (issues the MMAs), 1: peer
    const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    const int kstages = (p.K + WD_ATOMS * WD_BK - 1) / (WD_ATOMS * WD_BK);  // what reaches past K is zero-filled on both operands
    const int total_tiles = p.tiles_m * p.tiles_n;  // weight blocks vary fastest: pairs that run side by side share tokens

    if (tid == 0) {
        for (int s = 0; s < WD_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 8);
        }
        *poisoned = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {  // the same warp of both CTAs allocates the pair's tensor memory
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    // both CTAs have initialised their barriers before either signals the other
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // Tokens and expanded weights come from the launch in front.  The dependents go when this wait is over: what is
            // launched behind this grid then starts after everything ahead of it has completed.
            asm volatile("griddepcontrol.wait;\n" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
            const unsigned bytes = WD_ATOMS * (WD_A_BYTES + p.bn / 2 * WD_BK);
            int sit = 0;
            bool live = true;  // a wait that ran out ends this thread's requests
            for (int t = cluster_id; live && t < total_tiles; t += n_clusters) {
                const int row_x = (t / p.tiles_n) * WD_BM + static_cast<int>(rank) * 128;
                const int row_w = (t % p.tiles_n) * p.bn + static_cast<int>(rank) * (p.bn / 2);
                for (int g = 0; g < kstages; ++g, ++sit) {
                    const int s = sit % WD_STAGES;
                    if (sit >= WD_STAGES) live = mbar_wait(&empty[s], ((sit / WD_STAGES) - 1) & 1, poisoned);
                    if (!live) break;
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * bytes);
                    const uint32_t bar = map_to_rank(&full[s], 0);
                    uint8_t* st = ring + s * WD_STAGE_BYTES;
#pragma unroll
                    for (int j = 0; j < WD_ATOMS; ++j) {
                        tma_load_2d_pair(st + j * WD_A_BYTES, &tmap_x, (g * WD_ATOMS + j) * WD_BK, row_x, bar);
                        tma_load_2d_pair(st + WD_ATOMS * WD_A_BYTES + j * WD_B_BYTES, &tmap_w, (g * WD_ATOMS + j) * WD_BK, row_w, bar);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // D = s32, A = B = signed 8-bit, both K-major, N = bn, M = 256 over the pair
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(p.bn >> 3) << 17) | (static_cast<uint32_t>(WD_BM >> 4) << 24);
            const uint64_t desc0 = smem_desc_sw128(smem_u32(ring));
            int s = 0, nt = 0;
            unsigned par = 0;
            bool live = true;
            for (int t = cluster_id; live && t < total_tiles; t += n_clusters, ++nt) {
                const int a = nt & 1;
                if (nt >= 2) live = mbar_wait(&acc_empty[a], ((nt >> 1) - 1) & 1, poisoned);
                if (!live) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + a * WD_MAX_BN;
                for (int g = 0; g < kstages; ++g) {
                    live = mbar_wait(&full[s], par, poisoned);
                    if (!live) break;
                    tc_fence_after();
                    const uint64_t ad = desc0 + static_cast<uint64_t>(s * (WD_STAGE_BYTES >> 4));
#pragma unroll
                    for (int j = 0; j < WD_ATOMS; ++j)
                        mma_i8_ss_x4_pair(d_tmem, ad + j * (WD_A_BYTES >> 4), ad + ((WD_ATOMS * WD_A_BYTES + j * WD_B_BYTES) >> 4), idesc, (g | j) ? 1u : 0u);
                    tc_commit_pair(&empty[s]);
                    if (++s == WD_STAGES) { s = 0; par ^= 1; }
                }
                if (live) tc_commit_pair(&acc_full[a]);
            }
        }
    } else {
        // ---- epilogue of this CTA's 128 tokens: thread = token (tensor-memory lane), registers = weight rows.  Every warp
        // stages 32 tokens x 128 bytes of y in shared memory and stores them with one TMA copy (two buffers per warp).
        const int quarter = warp & 3;  // the tensor-memory lanes this warp may read
        uint8_t* my_out = out_s + (warp - 2) * 2 * WD_OUT_BYTES;
        const uint32_t acc_empty_leader0 = map_to_rank(&acc_empty[0], 0), acc_empty_leader1 = map_to_rank(&acc_empty[1], 0);
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        const float s_w = p.w_scale ? *static_cast<const volatile float*>(p.w_scale) : p.w_scale_host;
        int nt = 0, buf = 0;
        bool live = true;
        for (int t = cluster_id; live && t < total_tiles; t += n_clusters, ++nt) {
            const int a = nt & 1;
            const int tok0 = (t / p.tiles_n) * WD_BM + static_cast<int>(rank) * 128 + quarter * 32;  // this warp's first token
            const int col0 = (t % p.tiles_n) * p.bn;
            const int tok = tok0 + lane;
            float inv = 1.0f;
            if (p.x_scale && tok < p.M) inv = __frcp_rn(p.x_scale[tok]);
            live = mbar_wait(&acc_full[a], (nt >> 1) & 1, poisoned);
            live = __all_sync(0xffffffffu, live);
            if (!live) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * WD_MAX_BN;
            for (int c = 0; c < p.bn; c += COLS) {
                uint32_t v[COLS];
#pragma unroll
                for (int j = 0; j < COLS; j += 32) tmem_ld32_nowait(acc + c + j, v + j);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int j = 0; j < COLS; ++j) asm volatile("" : "+r"(v[j]));  // no use of v moves above the wait
                if (c + COLS >= p.bn) {  // this warp's part of the accumulator is in registers: hand it back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(a ? acc_empty_leader1 : acc_empty_leader0);
                }
                if (tok0 >= p.M || col0 + c >= p.N) continue;  // nothing of this box exists (uniform over the warp)
                float o[COLS];
                if constexpr (ROWS) {
#pragma unroll
                    for (int j = 0; j < COLS; j += 32) {
                        const int n = col0 + c + j + lane;
                        const float sc = n < p.N ? __ldg(p.row_scale + n) : 0.f;
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[j + i] = rescale(static_cast<int>(v[j + i]), inv, __shfl_sync(0xffffffffu, sc, i));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < COLS; ++j) o[j] = rescale(static_cast<int>(v[j]), inv, s_w);
                }
                if (p.bias) {
#pragma unroll
                    for (int j = 0; j < COLS; j += 32) {
                        const int n = col0 + c + j + lane;
                        const float b = n < p.N ? load1_rt(p.bias, p.bias_dtype, n) : 0.f;
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[j + i] = __fadd_rn(o[j + i], __shfl_sync(0xffffffffu, b, i));
                    }
                }
                // the store that last used this buffer has read it
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
                __syncwarp();
                const uint32_t row = smem_u32(my_out + buf * WD_OUT_BYTES) + lane * 128;
#pragma unroll
                for (int ch = 0; ch < 8; ++ch) {  // 16-byte chunk ch of the row lies at ch ^ (row & 7)
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if constexpr (YDT == WF_F32) {
                            w[i] = __float_as_uint(o[4 * ch + i]);
                        } else if constexpr (YDT == WF_BF16) {
                            const __nv_bfloat162 h = __floats2bfloat162_rn(o[8 * ch + 2 * i], o[8 * ch + 2 * i + 1]);
                            w[i] = *reinterpret_cast<const uint32_t*>(&h);
                        } else {
                            const __half2 h = __floats2half2_rn(o[8 * ch + 2 * i], o[8 * ch + 2 * i + 1]);
                            w[i] = *reinterpret_cast<const uint32_t*>(&h);
                        }
                    }
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(row + ((ch ^ (lane & 7)) << 4)), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                                 "r"(w[3])
                                 : "memory");
                }
                if (!p.y_tma) {  // row by row: a warp writes one token's 128 bytes
                    __syncwarp();
                    const int n = col0 + c + lane * (COLS / 32);
                    for (int r = 0; r < 32 && tok0 + r < p.M; ++r) {
                        const uint32_t w = *reinterpret_cast<const uint32_t*>(my_out + buf * WD_OUT_BYTES + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
                        const int64_t at = static_cast<int64_t>(tok0 + r) * p.ldy + n;
                        if constexpr (YDT == WF_F32) {
                            if (n < p.N) static_cast<uint32_t*>(p.y)[at] = w;
                        } else {
                            if (n < p.N) static_cast<uint16_t*>(p.y)[at] = static_cast<uint16_t>(w);
                            if (n + 1 < p.N) static_cast<uint16_t*>(p.y)[at + 1] = static_cast<uint16_t>(w >> 16);
                        }
                    }
                    __syncwarp();
                    continue;
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];\n" ::"l"(reinterpret_cast<uint64_t>(&tmap_y)),
                                 "r"(col0 + c), "r"(tok0), "r"(smem_u32(my_out + buf * WD_OUT_BYTES))
                                 : "memory");
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                }
                buf ^= 1;
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (*poisoned) {
        // A CTA that gave up: copies and MMAs issued before may still be on their way into this pair's shared and tensor
        // memory.  They take microseconds; the CTA keeps both for half a millisecond.
        for (int i = 0; i < 256; ++i) __nanosleep(2000);
        __syncthreads();
    }
    // neither CTA leaves (nor frees the pair's tensor memory) while the other may still signal it
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512));
    }
}

}  // namespace wf

using namespace wf;

extern "C" int wf_wide_status_fetch(int* out) {
    WF_CUDA(cudaMemcpyFromSymbol(out, g_wide_status, sizeof(int)));
    if (*out) {
        int zero = 0;
        WF_CUDA(cudaMemcpyToSymbol(g_wide_status, &zero, sizeof(int)));
    }
    return WF_OK;
}

// Weight rows per tile (256, 192, 128 or 64), or 0 where the form that keeps the weights packed (128 x 128 tiles, one per SM)
// is the faster one.  Both times are estimated in microseconds from what was measured on B200 over M = 128 ... 8192 on seven
// shapes of 0.9 to 59 Mi weights; over these 70 points a pick of this form takes 0.60 to 0.93 of the packed form's time, and the
// pick is 0.4 % slower than the fastest of the five forms on average and 14 % at worst (512 tokens, 6912 x 2560):
//   packed: waves of 148 tiles x (0.88 per 512 of K + 0.4);
//   here: waves of 74 tiles x (0.65 / 0.54 / 0.45 / 0.44 per 256 of K for 256 / 192 / 128 / 64 weight rows + 0.4), and the
//   expansion, 4.2 million weights per microsecond.  (One instruction of K = 32 takes 73 ns at 256 weight rows and still
//   56 ns at 128, so narrow tiles pay only where they save a wave.)
int wf_wide_tile(int64_t M, int64_t N, int64_t K) {
    static const double stage_us[4] = {0.44, 0.45, 0.54, 0.65};
    const int64_t sms = num_sms(), pairs = sms / 2;
    if (M <= 64 || pairs < 1) return 0;
    const auto blocks = [](int64_t v, int64_t b) { return (v + b - 1) / b; };
    double best = static_cast<double>(blocks(blocks(M, 128) * blocks(N, 128), sms)) * (0.88 * static_cast<double>(blocks(K, 512)) + 0.4);
    int bn = 0;
    for (int i = 3; i >= 0; --i) {
        const int64_t waves = blocks(blocks(M, WD_BM) * blocks(N, 64 * (i + 1)), pairs);
        const double us = static_cast<double>(waves) * (stage_us[i] * static_cast<double>(blocks(K, 256)) + 0.4) + static_cast<double>(N * K) / 4.2e6;
        if (us < best) {
            best = us;
            bn = 64 * (i + 1);
        }
    }
    return bn;
}

template <int YDT, bool ROWS>
static int wide_start(const cudaLaunchConfig_t& lc, const CUtensorMap& x, const CUtensorMap& w, const CUtensorMap& y, const WideParams& p) {
    static PerDeviceOnce configured;
    const int dev = current_device();
    if (configured.needs(dev)) {
        WF_CUDA(cudaFuncSetAttribute(wide_kernel<YDT, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(WD_SMEM)));
        configured.mark(dev);
    }
    WF_CUDA(cudaLaunchKernelEx(&lc, wide_kernel<YDT, ROWS>, x, w, y, p));
    return WF_OK;
}

// q [M, K] int8 (row stride ldq), w8 [N, K] int8 contiguous; bn from wf_wide_tile.
int wf_wide_launch(const int8_t* q, int64_t ldq, const float* x_scale, const int8_t* w8, const float* w_scale, float w_scale_host, const float* row_scale, const void* bias,
                   int bias_dtype, void* y, int y_dtype, int64_t ldy, int64_t M, int64_t N, int64_t K, int bn, void* stream) {
    EncodeTiledFn enc = pf_encode_fn();
    if (!enc) return fail(WF_E_DEVICE, "cuTensorMapEncodeTiled is not available in this driver");
    const int pairs = num_sms() / 2;
    WideParams p;
    p.x_scale = x_scale; p.w_scale = w_scale; p.row_scale = row_scale; p.w_scale_host = w_scale_host; p.bias = bias; p.bias_dtype = bias_dtype;
    p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K);
    p.bn = bn;
    p.tiles_m = static_cast<int>((M + WD_BM - 1) / WD_BM);
    p.tiles_n = static_cast<int>((N + p.bn - 1) / p.bn);
    alignas(64) CUtensorMap tmap_x, tmap_w, tmap_y;
    CUresult r = encode_2d_sw128(enc, &tmap_x, CU_TENSOR_MAP_DATA_TYPE_UINT8, q, K, M, ldq, WD_BK, 128);
    if (r == CUDA_SUCCESS) r = encode_2d_sw128(enc, &tmap_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, w8, K, N, K, WD_BK, p.bn / 2);
    const int ysize = static_cast<int>(dtype_size(y_dtype));
    const CUtensorMapDataType ytype = y_dtype == WF_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                                        : (y_dtype == WF_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
    p.y = y; p.ldy = ldy;
    // (N too: a row that ends inside 16 bytes was written to the end of them, over what lies behind it in the caller's tensor)
    p.y_tma = reinterpret_cast<uintptr_t>(y) % 16 == 0 && (ldy * ysize) % 16 == 0 && (N * ysize) % 16 == 0;
    if (!p.y_tma) tmap_y = tmap_x;  // not used
    if (r == CUDA_SUCCESS && p.y_tma) r = encode_2d_sw128(enc, &tmap_y, ytype, y, N, M, ldy * ysize, 128 / ysize, 32);
    if (r != CUDA_SUCCESS) return fail(WF_E_DEVICE, "cuTensorMapEncodeTiled (wide contraction) failed with %d", (int)r);
    const long long tiles = static_cast<long long>(p.tiles_m) * p.tiles_n;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(static_cast<unsigned>(2 * (tiles < pairs ? tiles : pairs)));
    lc.blockDim = dim3(WD_THREADS);
    lc.dynamicSmemBytes = WD_SMEM;
    lc.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 2;
    if (row_scale) {
        if (y_dtype == WF_F32) return wide_start<WF_F32, true>(lc, tmap_x, tmap_w, tmap_y, p);
        if (y_dtype == WF_BF16) return wide_start<WF_BF16, true>(lc, tmap_x, tmap_w, tmap_y, p);
        return wide_start<WF_F16, true>(lc, tmap_x, tmap_w, tmap_y, p);
    }
    if (y_dtype == WF_F32) return wide_start<WF_F32, false>(lc, tmap_x, tmap_w, tmap_y, p);
    if (y_dtype == WF_BF16) return wide_start<WF_BF16, false>(lc, tmap_x, tmap_w, tmap_y, p);
    return wide_start<WF_F16, false>(lc, tmap_x, tmap_w, tmap_y, p);
}

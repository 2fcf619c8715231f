// The layers of a ternary decoder for one new token per sequence, in one launch: a thread-block cluster per sequence.
//
// What bounds a decode step of a small model is not memory (a layer of width 576 has 0.9 MB of packed weights, which stay in L2) but
// the chain of dependent launches: six per layer, 3 to 5 us each, 22 us per layer on B200 although each does well under 1 us of
// work.  Here the 16 (or 8) CTAs of a cluster carry one sequence through all layers:
//   * the residual stream is kept whole in every CTA's shared memory; a CTA computes its share of the rows of a projection and
//     sends the bf16 results into every CTA of the cluster with st.async, which counts the bytes on the receiver's mbarrier.  That
//     count is the only synchronisation between CTAs: five exchanges per layer, no cluster barrier, nothing through L2;
//   * what follows an exchange (residual add, norm, quantization) is repeated by every CTA on the whole row: it is short
//     where this form pays, and cheaper than one more exchange;
//   * packed weights, norm weights and scales do not depend on the step: one producer warp streams them with bulk copies through a
//     ring of shared-memory stages, as far ahead as the ring reaches (a layer of width 576), so that no phase waits for them;
//   * attention: a KV head's positions are split over up to cluster / n_kv CTAs (one until the context is long enough to share);
//     eight or sixteen lanes hold a position, keys and values go from global memory to registers, and the first tile is
//     requested before the CTA waits for q, because older positions do not depend on it.  Partial results are exchanged in fp32.
// Measured, us per layer of a captured step with a head of 512 rows, against the separate launches, context 140: width 576 (MLP 1536) 13.0 / 22.8
// for one sequence and 13.0 / 39.2 for seven; 960 (2560) 17.3 / 29.5 for two; 1024 (4096) 19.0 / 33.2 for four.  Where it does not pay (with
// the whole head): 1536 (4096) 38 / 37 for one, 2560 (6912) 89 / 44.
// Clusters are independent of one another (no grid-wide wait: sequences that do not fit at once run one after another).  Every wait
// is bounded.  Arithmetic: that of the separate kernels, step by step, except the order of fp32 sums (norm, softmax) and
// probabilities that stay fp32.
#include "wf_common.cuh"

namespace wf {
__device__ int g_step_status = 0;
}
#define WF_STATUS_WORD ::wf::g_step_status
#include "wf_async.cuh"

namespace wf {

constexpr int ST_WARPS = 15, ST_CONSUMERS = ST_WARPS * 32, ST_THREADS = ST_CONSUMERS + 32;  // and the producer warp
constexpr int ST_MAX_STAGES = 16;
constexpr int ST_MAX_K = 8192;                          // inputs of a projection
constexpr int ST_MAX_G = 4;                             // query heads per KV head
constexpr int ST_SMEM_MAX = 227 * 1024;

enum { B_QKV, B_ATTN, B_O, B_ACT, B_DOWN, B_COUNT };    // the five exchanges of a layer

struct StepParams {
    const wf_step_layer* layers;
    const __nv_bfloat16* h;       // [B, hidden] the tokens' embeddings
    const __nv_bfloat16* norm_f;  // [hidden]
    __nv_bfloat16* xf;            // [B, hidden] normalised output of the last layer
    const float* cosv;            // [T, D / 2]
    const float* sinv;
    const int64_t* pos;
    int L, hidden, nq, nkv, inter, T;
    int act;                      // 0 SiLU, 1 ReLU^2
    float eps, qeps, scale_log2;
    int splits;                   // most CTAs that share a KV head
    int stage_bytes, stages;
    int lpr_log2[4];              // lanes per row: q/k/v, o, gate/up, down
    // offsets into shared memory, bytes
    int o_h, o_qkv, o_attn_o, o_attn_ml, o_o, o_act, o_down, o_xq, o_val, o_out, o_qr, o_kn, o_red, o_meta, o_rope, o_ring;
    int meta_bytes;
};

__device__ __forceinline__ float st_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float st_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float st_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ uint32_t st_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void st_sync() { asm volatile("bar.sync 1, 480;\n" ::: "memory"); }  // the consumer warps
// ... and whether `v` holds for any of their threads: the same answer for all of them
__device__ __forceinline__ bool st_sync_any(bool v) {
    unsigned r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, 480, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(r)
                 : "r"(static_cast<unsigned>(v))
                 : "memory");
    return r != 0;
}
__device__ __forceinline__ uint32_t st_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t st_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t st_map(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// stores into a CTA of the cluster that add their bytes to that CTA's mbarrier
__device__ __forceinline__ void st_send8(uint32_t addr, uint64_t v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n" ::"r"(addr), "l"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_send16(uint32_t addr, float4 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z),
                 "f"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Bounded wait for data of this CTA's copies or of other CTAs.  Polls: it is at most a microsecond away, and a warp that the blocking form
// has put to sleep wakes late.
__device__ __forceinline__ unsigned st_test(uint32_t bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok;
}
__device__ __noinline__ bool st_wait_long(uint32_t bar, unsigned parity, volatile int* poisoned) {
    unsigned long long t0 = 0;
    for (unsigned it = 1;; ++it) {
        if (st_test(bar, parity)) return true;
        if ((it & 1023) == 0) {
            if (*poisoned) return false;
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(now));
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_LIMIT_NS) break;
        }
    }
    *poisoned = 1;
    atomicExch(&WF_STATUS_WORD, WF_E_LIMIT);
    return false;
}
// False when the phase has not completed within the limit, or another wait of this CTA has given up meanwhile: what it stands for has not
// arrived, and its barrier may not be armed again.  The whole warp calls it and gets one answer.
__device__ __forceinline__ bool st_wait(uint64_t* bar, unsigned parity, volatile int* poisoned) {
    const uint32_t a = smem_u32(bar);
    return __all_sync(0xffffffffu, st_test(a, parity) || st_wait_long(a, parity, poisoned));
}
// Time for what is on its way into this CTA's shared memory to land.
__device__ __noinline__ void st_settle() {
    unsigned long long t0, now;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t0));
    for (int it = 0; it < 1000; ++it) {
        __nanosleep(2000);
        asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(now));
        if (now - t0 > 500000) break;
    }
}

// Rows [r0, r0 + n) of this CTA: whole groups of four rows (8 bytes of results), shared out evenly; never empty (N >= 4 CTAs).
struct RowRange { int r0, n; };
__device__ __forceinline__ RowRange st_rows(int N, int rank, int ctas) {
    const int u = N >> 2, a = u * rank / ctas, b = u * (rank + 1) / ctas;
    return {a * 4, (b - a) * 4};
}
// A phase's rows in ring stages: `per` rows each, `count` stages.
struct StageSplit { int count, per; };
__device__ __forceinline__ StageSplit st_split(int rows, int row_bytes, int stage_bytes) {
    const int fit = stage_bytes / row_bytes, count = (rows + fit - 1) / fit;
    return {count, (rows + count - 1) / count};
}

__device__ __forceinline__ int st_dp4a(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ float st_exp2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float st_act(float a, int mode) {  // as the stand-alone activation kernel
    if (mode == 0) return st_round(a / (1.0f + __expf(-a)));
    const float r = st_round(fmaxf(a, 0.f));
    return st_round(r * r);
}
// the largest magnitudes of four bf16 values, as two bit patterns side by side (a NaN counts for nothing, as with fmaxf)
__device__ __forceinline__ uint32_t st_max4(uint2 v, uint32_t mx) {
    const __nv_bfloat162 a = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    const __nv_bfloat162 m = __hmax2(__hmax2(a, b), *reinterpret_cast<const __nv_bfloat162*>(&mx));
    return *reinterpret_cast<const uint32_t*>(&m);
}
// over the 15 entries that the warps left (the sixteenth is zero)
__device__ __forceinline__ float st_sum16(const float* r) {
    const float4* v = reinterpret_cast<const float4*>(r);
    const float4 a = v[0], b = v[1], c = v[2], d = v[3];
    return ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w)) + (((c.x + c.y) + (c.z + c.w)) + ((d.x + d.y) + (d.z + d.w)));
}
__device__ __forceinline__ int st_sum16(const int* r) {
    const int4* v = reinterpret_cast<const int4*>(r);
    const int4 a = v[0], b = v[1], c = v[2], d = v[3];
    return a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w + c.x + c.y + c.z + c.w + d.x + d.y + d.z + d.w;
}
__device__ __forceinline__ uint32_t st_max16(const uint32_t* r) {
    const uint4* v = reinterpret_cast<const uint4*>(r);
    const uint4 a = v[0], b = v[1], c = v[2], d = v[3];
    return max(max(max(max(a.x, a.y), max(a.z, a.w)), max(max(b.x, b.y), max(b.z, b.w))), max(max(max(c.x, c.y), max(c.z, c.w)), max(max(d.x, d.y), max(d.z, d.w))));
}

template <int D>
__global__ void __launch_bounds__(ST_THREADS, 1) decode_layers_kernel(const __grid_constant__ StepParams p) {
    constexpr int LPR = D / 8, RP = 32 / LPR;  // lanes of a position, positions per load of a warp
    constexpr int TILE = 4 * RP;               // positions of a warp's tile
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[ST_MAX_STAGES], empty[ST_MAX_STAGES], meta_full[2], meta_empty[2], xbar[B_COUNT];
    __shared__ __align__(16) float red_a[16];
    __shared__ __align__(16) uint32_t red_b[16];
    __shared__ __align__(16) int red_c[16];
    __shared__ volatile int poisoned;
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = static_cast<int>(st_size()), rank = static_cast<int>(st_rank()), seq = blockIdx.x / C;
    const int G = p.nq / p.nkv, QD = p.nq * D, KVD = p.nkv * D, hidden = p.hidden, inter = p.inter;
    const int NQKV = QD + 2 * KVD;
    const RowRange r_qkv = st_rows(NQKV, rank, C), r_h = st_rows(hidden, rank, C), r_i = st_rows(inter, rank, C);
    const StageSplit s_qkv = st_split(r_qkv.n, hidden / 4, p.stage_bytes), s_o = st_split(r_h.n, QD / 4, p.stage_bytes),
                     s_gu = st_split(r_i.n, hidden / 2, p.stage_bytes), s_d = st_split(r_h.n, inter / 4, p.stage_bytes);
    uint8_t* ring = smem + p.o_ring;

    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], ST_WARPS);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&meta_full[s], 1);
            mbar_init(&meta_empty[s], ST_WARPS);
        }
        for (int s = 0; s < B_COUNT; ++s) mbar_init(&xbar[s], 1);
        red_a[15] = 0.f;
        red_b[15] = 0;
        red_c[15] = 0;
        poisoned = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    st_cluster_sync();  // nobody sends before every CTA's barriers exist

    if (warp == ST_WARPS) {
        // ---- producer: norm weights and scales of a layer, then its packed rows, stage by stage, as far ahead as there is room
        int s = 0;
        unsigned lap = 0, norms[2] = {0, 0};  // norms: how often either layer's barrier was armed
        constexpr int NPTR = sizeof(wf_step_layer) / 8;
        static_assert(NPTR == 18, "codes, scales, norms, caches");
        const uint64_t* table = reinterpret_cast<const uint64_t*>(p.layers);
        uint64_t ptr = lane < NPTR ? __ldg(table + lane) : 0;  // lane i: pointer i of the layer, requested one layer ahead
        float sc = lane >= 7 && lane < 14 ? __ldg(reinterpret_cast<const float*>(ptr)) : 0.f;
        // rows [a0, a0 + n) of matrix m to `dst` (lane 0)
        auto rows = [&](uint8_t* dst, uint64_t base, int a0, int n, int rb) {
            bulk_copy_g2s(dst, reinterpret_cast<const uint8_t*>(base) + static_cast<int64_t>(a0) * rb, n * rb, &full[s]);
        };
        auto stage = [&](int bytes) -> uint8_t* {  // lane 0: the next stage, armed for `bytes`
            if (lap > 0) mbar_wait(&empty[s], (lap - 1) & 1, &poisoned);
            if (poisoned) return nullptr;
            mbar_expect_tx(&full[s], bytes);
            return ring + static_cast<size_t>(s) * p.stage_bytes;
        };
        auto next = [&]() { if (++s == p.stages) { s = 0; ++lap; } };
        for (int l = 0; l < p.L; ++l) {
            const int ms = l & 1;
            uint8_t* meta = smem + p.o_meta + ms * p.meta_bytes;
            if (l >= 2) mbar_wait(&meta_empty[ms], ((l >> 1) - 1) & 1, &poisoned);
            uint64_t c[7];
#pragma unroll
            for (int m = 0; m < 7; ++m) c[m] = __shfl_sync(0xffffffffu, ptr, m);
            const uint64_t n1 = __shfl_sync(0xffffffffu, ptr, 14), n2 = __shfl_sync(0xffffffffu, ptr, 15);
            if (lane >= 7 && lane < 14) reinterpret_cast<float*>(meta)[lane - 7] = sc;
            if (lane == 16 || lane == 17) reinterpret_cast<uint64_t*>(meta + 32)[lane - 16] = ptr;
            if (l + 1 < p.L) {
                ptr = lane < NPTR ? __ldg(table + static_cast<int64_t>(l + 1) * NPTR + lane) : 0;
                sc = lane >= 7 && lane < 14 ? __ldg(reinterpret_cast<const float*>(ptr)) : 0.f;
            }
            __syncwarp();
            if (lane == 0 && !poisoned) {
                mbar_expect_tx(&meta_full[ms], hidden * 4);
                if (ms) ++norms[1]; else ++norms[0];
                bulk_copy_g2s(meta + 48, reinterpret_cast<const void*>(n1), hidden * 2, &meta_full[ms]);
                bulk_copy_g2s(meta + 48 + hidden * 2, reinterpret_cast<const void*>(n2), hidden * 2, &meta_full[ms]);
                // q/k/v: rows of up to three matrices side by side
                for (int b = 0; b < s_qkv.count; ++b, next()) {
                    const int a0 = r_qkv.r0 + b * s_qkv.per, a1 = min(a0 + s_qkv.per, r_qkv.r0 + r_qkv.n), rb = hidden / 4;
                    uint8_t* st = stage((a1 - a0) * rb);
                    if (!st) break;
                    const int lo[4] = {0, QD, QD + KVD, NQKV};
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        const int f = max(a0, lo[m]), t = min(a1, lo[m + 1]);
                        if (f < t) rows(st + (f - a0) * rb, c[m], f - lo[m], t - f, rb);
                    }
                }
                for (int b = 0; b < s_o.count; ++b, next()) {
                    const int a0 = b * s_o.per, n = min(s_o.per, r_h.n - a0), rb = QD / 4;
                    uint8_t* st = stage(n * rb);
                    if (!st) break;
                    rows(st, c[3], r_h.r0 + a0, n, rb);
                }
                for (int b = 0; b < s_gu.count; ++b, next()) {
                    const int a0 = b * s_gu.per, n = min(s_gu.per, r_i.n - a0), rb = hidden / 4;
                    uint8_t* st = stage(2 * n * rb);
                    if (!st) break;
                    rows(st, c[4], r_i.r0 + a0, n, rb);
                    rows(st + n * rb, c[5], r_i.r0 + a0, n, rb);
                }
                for (int b = 0; b < s_d.count; ++b, next()) {
                    const int a0 = b * s_d.per, n = min(s_d.per, r_h.n - a0), rb = inter / 4;
                    uint8_t* st = stage(n * rb);
                    if (!st) break;
                    rows(st, c[6], r_h.r0 + a0, n, rb);
                }
            }
            __syncwarp();
        }
        if (poisoned && lane == 0) {  // the copies in flight land before the shared memory goes away: the last one of every stage and of both layers' norms
            volatile int drained = 0;
            for (int i = 0; i < p.stages; ++i) {
                const unsigned n = lap + (i < s ? 1 : 0);
                if (n > 0) mbar_wait(&full[i], (n - 1) & 1, &drained);
            }
            for (int i = 0; i < 2; ++i)
                if (norms[i] > 0) mbar_wait(&meta_full[i], (norms[i] - 1) & 1, &drained);
        }
    } else {
        // ---- consumers.  One body of code for the four projections of a layer, loops that are not unrolled: a step runs through all of
        // this once per layer, and what does not stay in the instruction cache costs more than the work (unrolled phases one after
        // another, 23 us per layer of width 576; their times followed their sizes, not their work).
        __nv_bfloat16* h_s = reinterpret_cast<__nv_bfloat16*>(smem + p.o_h);
        __nv_bfloat16* qkv_s = reinterpret_cast<__nv_bfloat16*>(smem + p.o_qkv);
        float* part_o = reinterpret_cast<float*>(smem + p.o_attn_o);    // [nq][splits][D]
        float* part_ml = reinterpret_cast<float*>(smem + p.o_attn_ml);  // [nq][splits][2]
        uint8_t* xq = smem + p.o_xq;
        __nv_bfloat16* val_s = reinterpret_cast<__nv_bfloat16*>(smem + p.o_val);  // the row that is quantized; every thread reads what it wrote
        __nv_bfloat16* out_s = reinterpret_cast<__nv_bfloat16*>(smem + p.o_out);
        float* qr = reinterpret_cast<float*>(smem + p.o_qr);            // [G][D] rotated query heads of this CTA's KV head
        __nv_bfloat16* kn = reinterpret_cast<__nv_bfloat16*>(smem + p.o_kn);  // [D] rotated new key
        float* red_o = reinterpret_cast<float*>(smem + p.o_red);        // [warps][D], then [warps][2]
        float* red_ml = red_o + ST_WARPS * D;
        float* rope = reinterpret_cast<float*>(smem + p.o_rope);        // cos, sin of this position
        const int clog = __ffs(C) - 1;
        int s = 0;
        unsigned lap = 0;

        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // h and the position come from earlier kernels
        int64_t pos;
        asm volatile("ld.global.s64 %0, [%1];\n" : "=l"(pos) : "l"(p.pos) : "memory");
        int slot = static_cast<int>(pos % p.T);  // the caller keeps the position below T; a stray one stays inside the cache
        if (slot < 0) slot += p.T;
        const int n_valid = pos + 1 < p.T ? max(static_cast<int>(pos + 1), 1) : p.T;
        // A warp takes one query head through a tile of positions; a KV head is shared by as many CTAs as it takes for one round of tiles.
        const int tiles = (n_valid + TILE - 1) / TILE, tw = ST_WARPS / G;
        const int S = max(1, min(p.splits, (tiles + tw - 1) / tw));
        const int kvh = rank % p.nkv, split = rank / p.nkv;
        const int g = warp % G, tile0 = warp / G < tw ? (warp / G) * S + split : tiles;
        const int nw = split < S ? min(tw, (tiles - split + S - 1) / S) : 0;  // tile-warps per head that have a tile (at least one: split < tiles)
        const unsigned bytes_attn = static_cast<unsigned>(p.nq) * S * (D * 4 + 8);
        if (tid == 0) {
            mbar_expect_tx(&xbar[B_QKV], NQKV * 2);
            mbar_expect_tx(&xbar[B_ATTN], bytes_attn);
            mbar_expect_tx(&xbar[B_O], hidden * 2);
            mbar_expect_tx(&xbar[B_ACT], inter * 2);
            mbar_expect_tx(&xbar[B_DOWN], hidden * 2);
        }
        for (int i = tid; i < hidden / 8; i += ST_CONSUMERS)
            *reinterpret_cast<uint4*>(h_s + 8 * i) = ld16_chained(p.h + static_cast<int64_t>(seq) * hidden + 8 * i);
        for (int i = tid; i < D; i += ST_CONSUMERS)
            rope[i] = i < D / 2 ? __ldg(p.cosv + static_cast<int64_t>(slot) * (D / 2) + i) : __ldg(p.sinv + static_cast<int64_t>(slot) * (D / 2) + i - D / 2);
        st_sync();

        // A wait that has run out ends the CTA's part: its warps agree on it at the next barrier in front of a send or a cache write and
        // leave, so that nothing goes out that is computed from what has not arrived; the cluster's other CTAs, which wait for it, run
        // out in turn.  A barrier whose phase has not completed is not armed again.
        bool ok = true;
#pragma unroll 1
        for (int l = 0; l <= p.L; ++l) {  // the turn behind the last layer: its residual add and the final norm
            const int ms = l & 1;
            const uint8_t* meta = smem + p.o_meta + ms * p.meta_bytes;
            const float* scale = reinterpret_cast<const float*>(meta);
            if (l < p.L) ok &= st_wait(&meta_full[ms], (l >> 1) & 1, &poisoned);
#pragma unroll 1
            for (int ph = 0; ph < 4; ++ph) {  // q/k/v, o, gate/up, down
                const int K = ph == 1 ? QD : (ph == 3 ? inter : hidden);
                // ---- what it waits for; the barrier is armed again at once for the next layer
                if (l + ph > 0) {
                    const int b = ph == 0 ? B_DOWN : (ph == 1 ? B_ATTN : (ph == 2 ? B_O : B_ACT));
                    const bool here = st_wait(&xbar[b], (ph == 0 ? l - 1 : l) & 1, &poisoned);
                    ok &= here;
                    if (tid == 0 && here) mbar_expect_tx(&xbar[b], ph == 1 ? bytes_attn : (ph == 3 ? inter : hidden) * 2);
                }
                // ---- its input as bf16, this thread's share, and the largest magnitude
                uint32_t mx = 0;
                const __nv_bfloat16* val = val_s;
                if (!(ph & 1)) {  // residual add, norm
                    const __nv_bfloat16* delta = l + ph == 0 ? nullptr : reinterpret_cast<const __nv_bfloat16*>(smem + (ph == 0 ? p.o_down : p.o_o));
                    float ss = 0.f;
#pragma unroll 1
                    for (int k = 4 * tid; k < hidden; k += 4 * ST_CONSUMERS) {
                        uint2 v = *reinterpret_cast<const uint2*>(h_s + k);
                        if (delta) {
                            const uint2 d = *reinterpret_cast<const uint2*>(delta + k);
                            v = make_uint2(st_pack(st_lo(v.x) + st_lo(d.x), st_hi(v.x) + st_hi(d.x)), st_pack(st_lo(v.y) + st_lo(d.y), st_hi(v.y) + st_hi(d.y)));
                            *reinterpret_cast<uint2*>(h_s + k) = v;
                        }
                        ss += st_lo(v.x) * st_lo(v.x) + st_hi(v.x) * st_hi(v.x) + (st_lo(v.y) * st_lo(v.y) + st_hi(v.y) * st_hi(v.y));
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    if (lane == 0) red_a[warp] = ss;
                    st_sync();
                    const float r = rsqrtf(st_sum16(red_a) / static_cast<float>(hidden) + p.eps);
                    const __nv_bfloat16* nw_ = l == p.L ? p.norm_f : reinterpret_cast<const __nv_bfloat16*>(meta + 48) + (ph == 0 ? 0 : hidden);
#pragma unroll 1
                    for (int k = 4 * tid; k < hidden; k += 4 * ST_CONSUMERS) {
                        const uint2 v = *reinterpret_cast<const uint2*>(h_s + k), w = *reinterpret_cast<const uint2*>(nw_ + k);
                        const uint2 y = make_uint2(st_pack(st_round(st_lo(v.x) * r) * st_lo(w.x), st_round(st_hi(v.x) * r) * st_hi(w.x)),
                                                   st_pack(st_round(st_lo(v.y) * r) * st_lo(w.y), st_round(st_hi(v.y) * r) * st_hi(w.y)));
                        if (l == p.L) {
                            if (rank == 0) *reinterpret_cast<uint2*>(p.xf + static_cast<int64_t>(seq) * hidden + k) = y;
                        } else {
                            *reinterpret_cast<uint2*>(val_s + k) = y;
                            mx = st_max4(y, mx);
                        }
                    }
                    if (l == p.L) break;
                } else if (ph == 1) {  // merge the splits of every head
#pragma unroll 1
                    for (int k = 4 * tid; k < QD; k += 4 * ST_CONSUMERS) {
                        const int hd = k / D;
                        const float* ml = part_ml + hd * p.splits * 2;
                        const float* po = part_o + hd * p.splits * D + (k & (D - 1));
                        float top = ml[0];
#pragma unroll 1
                        for (int w = 1; w < S; ++w) top = fmaxf(top, ml[2 * w]);
                        if (top == -INFINITY) top = 0.f;  // no score above -inf: weights of zero, not inf - inf
                        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                        float ls = 0.f;
#pragma unroll 1
                        for (int w = 0; w < S; ++w) {
                            const float2 m = *reinterpret_cast<const float2*>(ml + 2 * w);
                            const float4 v = *reinterpret_cast<const float4*>(po + w * D);
                            const float f = st_exp2(m.x - top);
                            acc.x += v.x * f; acc.y += v.y * f; acc.z += v.z * f; acc.w += v.w * f;
                            ls += m.y * f;
                        }
                        const float inv = __fdividef(1.0f, ls);
                        const uint2 y = make_uint2(st_pack(acc.x * inv, acc.y * inv), st_pack(acc.z * inv, acc.w * inv));
                        *reinterpret_cast<uint2*>(val_s + k) = y;
                        mx = st_max4(y, mx);
                    }
                } else {
                    val = reinterpret_cast<const __nv_bfloat16*>(smem + p.o_act);
#pragma unroll 1
                    for (int k = 4 * tid; k < inter; k += 4 * ST_CONSUMERS) mx = st_max4(*reinterpret_cast<const uint2*>(val + k), mx);
                }
                // ---- quantization, in the order of the weights' bit positions
                mx = __reduce_max_sync(0xffffffffu, max(mx & 0xffff0000u, mx << 16));
                if (lane == 0) red_b[warp] = mx;
                st_sync();
                const float sx = act_scale_from_absmax<WF_BF16>(__uint_as_float(st_max16(red_b)), p.qeps);
                int qsum = 0;
                const int chunks = K >> 6;
#pragma unroll 1
                for (int k = 4 * tid; k < K; k += 4 * ST_CONSUMERS) {
                    const uint2 v = *reinterpret_cast<const uint2*>(val + k);
                    const int q0 = quantize_one<WF_BF16>(st_lo(v.x), sx), q1 = quantize_one<WF_BF16>(st_hi(v.x), sx);
                    const int q2 = quantize_one<WF_BF16>(st_lo(v.y), sx), q3 = quantize_one<WF_BF16>(st_hi(v.y), sx);
                    qsum += (q0 + q1) + (q2 + q3);
                    *reinterpret_cast<uint32_t*>(xq + (((k >> 4) & 3) * chunks + (k >> 6)) * 16 + (k & 12)) =
                        __byte_perm(__byte_perm(q0, q1, 0x0040), __byte_perm(q2, q3, 0x0040), 0x5410);
                }
                qsum = __reduce_add_sync(0xffffffffu, qsum);
                if (lane == 0) red_c[warp] = qsum;
                const float inv = __fdiv_rn(1.0f, sx);
                st_sync();
                qsum = st_sum16(red_c);
                // ---- the projection: lanes of a group take two rows at a time (gate and up of one column, or rows half a stage apart), 16
                // bytes of weights per lane and step, masked in place (the four bit positions carry factors 1, 4, 16, 64 to the end)
                const RowRange r = ph == 0 ? r_qkv : (ph == 2 ? r_i : r_h);
                const StageSplit sp = ph == 0 ? s_qkv : (ph == 1 ? s_o : (ph == 2 ? s_gu : s_d));
                const int ll = p.lpr_log2[ph], lpr = 1 << ll, col = lane & (lpr - 1), sub = lane >> ll, rpw = 32 >> ll;
#pragma unroll 1
                for (int b = 0; b < sp.count; ++b) {
                    if (!st_wait(&full[s], lap & 1, &poisoned)) {
                        ok = false;
                        break;
                    }
                    const uint8_t* st = ring + static_cast<size_t>(s) * p.stage_bytes;
                    const int n = min(sp.per, r.n - b * sp.per), pairs = ph == 2 ? n : (n + 1) >> 1, total = ph == 2 ? 2 * n : n;
#pragma unroll 1
                    for (int r0 = warp * rpw; r0 < pairs; r0 += ST_WARPS * rpw) {
                        const int row = min(r0 + sub, pairs - 1), row1 = min(row + pairs, total - 1);
                        const uint8_t* w0 = st + row * (K / 4);
                        const uint8_t* w1 = st + row1 * (K / 4);
                        int a0 = 0, a1 = 0, a2 = 0, a3 = 0, c0 = 0, c1 = 0, c2 = 0, c3 = 0;
#pragma unroll 1
                        for (int kc = col; kc < chunks; kc += lpr) {
                            const uint4 v = *reinterpret_cast<const uint4*>(w0 + kc * 16), u = *reinterpret_cast<const uint4*>(w1 + kc * 16);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint4 x = *reinterpret_cast<const uint4*>(xq + (i * chunks + kc) * 16);
                                const uint32_t vv = i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)), uu = i == 0 ? u.x : (i == 1 ? u.y : (i == 2 ? u.z : u.w));
                                a0 = st_dp4a(vv & 0x03030303u, x.x, a0); a1 = st_dp4a(vv & 0x0c0c0c0cu, x.y, a1);
                                a2 = st_dp4a(vv & 0x30303030u, x.z, a2); a3 = st_dp4a(vv & 0xc0c0c0c0u, x.w, a3);
                                c0 = st_dp4a(uu & 0x03030303u, x.x, c0); c1 = st_dp4a(uu & 0x0c0c0c0cu, x.y, c1);
                                c2 = st_dp4a(uu & 0x30303030u, x.z, c2); c3 = st_dp4a(uu & 0xc0c0c0c0u, x.w, c3);
                            }
                        }
                        int d0 = a0 + (a1 >> 2) + (a2 >> 4) + (a3 >> 6), d1 = c0 + (c1 >> 2) + (c2 >> 4) + (c3 >> 6);
#pragma unroll 1
                        for (int o = lpr >> 1; o > 0; o >>= 1) {
                            d0 += __shfl_xor_sync(0xffffffffu, d0, o);
                            d1 += __shfl_xor_sync(0xffffffffu, d1, o);
                        }
                        if (col == 0 && r0 + sub < pairs) {
                            const int at = b * sp.per + row, at1 = b * sp.per + row1;
                            auto index = [&](int i) { return ph == 0 ? (r.r0 + i >= QD) + (r.r0 + i >= QD + KVD) : (ph == 1 ? 3 : 6); };
                            const float y0 = rescale(d0 - qsum, inv, scale[ph == 2 ? 4 : index(at)]), y1 = rescale(d1 - qsum, inv, scale[ph == 2 ? 5 : index(at1)]);
                            if (ph == 2) {
                                out_s[at] = __float2bfloat16_rn(st_act(st_round(y0), p.act) * st_round(y1));
                            } else {
                                out_s[at] = __float2bfloat16_rn(y0);
                                out_s[at1] = __float2bfloat16_rn(y1);  // the middle row of an odd stage twice, with the same value
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[s]);
                    if (++s == p.stages) { s = 0; ++lap; }
                }
                if (ph == 3 && lane == 0) mbar_arrive(&meta_empty[ms]);
                if (st_sync_any(!ok)) goto given_up;
                // ---- the results to every CTA, 8 bytes per store
                {
                    uint8_t* dst = smem + (ph == 0 ? p.o_qkv : (ph == 1 ? p.o_o : (ph == 2 ? p.o_act : p.o_down))) + 2 * r.r0;
                    uint64_t* bar = &xbar[ph == 0 ? B_QKV : (ph == 1 ? B_O : (ph == 2 ? B_ACT : B_DOWN))];
#pragma unroll 1
                    for (int i = tid; i < (r.n >> 2) << clog; i += ST_CONSUMERS) {
                        const int w = i >> clog, to = i & (C - 1);
                        st_send8(st_map(smem_u32(dst + 8 * w), to), *reinterpret_cast<const uint64_t*>(out_s + 4 * w), st_map(smem_u32(bar), to));
                    }
                }
                if (ph != 0) continue;

                // ---- attention: the first tile of keys and values is on its way while q is waited for
                const int sb = lane / LPR, dim = (lane % LPR) * 8;
                const int64_t cache_at = (static_cast<int64_t>(seq) * p.nkv + kvh) * p.T * D;
                __nv_bfloat16* kcache = reinterpret_cast<__nv_bfloat16* const*>(meta + 32)[0] + cache_at;
                __nv_bfloat16* vcache = reinterpret_cast<__nv_bfloat16* const*>(meta + 32)[1] + cache_at;
                uint4 kr[4], vr[4];
                auto load_tile = [&](int tile) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int t = tile * TILE + i * RP + sb;
                        kr[i] = vr[i] = make_uint4(0, 0, 0, 0);
                        if (t < n_valid && t != slot) {
                            kr[i] = ld16_chained(kcache + static_cast<int64_t>(t) * D + dim);
                            vr[i] = ld16_chained(vcache + static_cast<int64_t>(t) * D + dim);
                        }
                    }
                };
                if (nw > 0) load_tile(tile0);  // a warp without a tile loads nothing: its positions are not valid
                const bool here = st_wait(&xbar[B_QKV], l & 1, &poisoned);
                ok &= here;
                if (tid == 0 && here) mbar_expect_tx(&xbar[B_QKV], NQKV * 2);
                if (nw == 0) continue;
#pragma unroll 1
                for (int i = tid; i < (G + 1) * (D / 2); i += ST_CONSUMERS) {  // the last "head" is the key
                    const int hh = i / (D / 2), e = i & (D / 2 - 1);
                    const __nv_bfloat16* x = qkv_s + (hh < G ? (kvh * G + hh) * D : QD + kvh * D);
                    const float x1 = __bfloat162float(x[e]), x2 = __bfloat162float(x[e + D / 2]), c = rope[e], sn = rope[D / 2 + e];
                    const __nv_bfloat16 y1 = __float2bfloat16_rn(x1 * c - x2 * sn), y2 = __float2bfloat16_rn(x2 * c + x1 * sn);
                    if (hh < G) {
                        qr[hh * D + e] = __bfloat162float(y1);
                        qr[hh * D + e + D / 2] = __bfloat162float(y2);
                    } else {
                        kn[e] = y1;
                        kn[e + D / 2] = y2;
                    }
                }
                if (st_sync_any(!ok)) goto given_up;
                const __nv_bfloat16* vn = qkv_s + QD + KVD + kvh * D;
                if (split == 0 && tid < D / 4) {  // the new position goes to the caches
                    const bool is_k = tid < D / 8;
                    const int e = (is_k ? tid : tid - D / 8) * 8;
                    *reinterpret_cast<uint4*>((is_k ? kcache : vcache) + static_cast<int64_t>(slot) * D + e) = *reinterpret_cast<const uint4*>((is_k ? kn : vn) + e);
                }
                if (tile0 < tiles) {
                    const float4 q0 = *reinterpret_cast<const float4*>(qr + g * D + dim), q1 = *reinterpret_cast<const float4*>(qr + g * D + dim + 4);
                    float m = -INFINITY, ls = 0.f, o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
                    for (int tile = tile0; tile < tiles; tile += tw * S) {
                        float sc[4];
                        uint4 vv[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int t = tile * TILE + i * RP + sb;
                            uint4 kk = kr[i];
                            vv[i] = vr[i];
                            if (t == slot) {
                                kk = *reinterpret_cast<const uint4*>(kn + dim);
                                vv[i] = *reinterpret_cast<const uint4*>(vn + dim);
                            }
                            sc[i] = st_lo(kk.x) * q0.x + st_hi(kk.x) * q0.y + st_lo(kk.y) * q0.z + st_hi(kk.y) * q0.w +
                                    (st_lo(kk.z) * q1.x + st_hi(kk.z) * q1.y + st_lo(kk.w) * q1.z + st_hi(kk.w) * q1.w);
                        }
                        if (tile + tw * S < tiles) load_tile(tile + tw * S);
#pragma unroll
                        for (int w = LPR / 2; w > 0; w >>= 1)
#pragma unroll
                            for (int i = 0; i < 4; ++i) sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], w);
                        float top = m;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            sc[i] = tile * TILE + i * RP + sb < n_valid ? sc[i] * p.scale_log2 : -INFINITY;
                            top = fmaxf(top, sc[i]);
                        }
                        const float base = top == -INFINITY ? 0.f : top;  // no valid position for these lanes so far
                        const float corr = st_exp2(m - base);
                        m = top;
                        ls *= corr;
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] *= corr;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float pr = st_exp2(sc[i] - base);
                            ls += pr;
                            const uint32_t v[4] = {vv[i].x, vv[i].y, vv[i].z, vv[i].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                o[2 * e] += pr * st_lo(v[e]);
                                o[2 * e + 1] += pr * st_hi(v[e]);
                            }
                        }
                    }
                    // merge the position groups of the warp
#pragma unroll 1
                    for (int w = LPR; w < 32; w <<= 1) {
                        const float m2 = __shfl_xor_sync(0xffffffffu, m, w), l2 = __shfl_xor_sync(0xffffffffu, ls, w);
                        const float top = fmaxf(m, m2), base = top == -INFINITY ? 0.f : top;
                        const float f1 = st_exp2(m - base), f2 = st_exp2(m2 - base);
                        m = top;
                        ls = ls * f1 + l2 * f2;
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] = o[e] * f1 + __shfl_xor_sync(0xffffffffu, o[e], w) * f2;
                    }
                    if (sb == 0) {
                        float* ro = red_o + warp * D + dim;
                        *reinterpret_cast<float4*>(ro) = make_float4(o[0], o[1], o[2], o[3]);
                        *reinterpret_cast<float4*>(ro + 4) = make_float4(o[4], o[5], o[6], o[7]);
                        if (dim == 0) *reinterpret_cast<float2*>(red_ml + warp * 2) = make_float2(m, ls);
                    }
                }
                st_sync();
                // merge the tile-warps of each head and send: every piece of four outputs by a few threads, each to its share of the CTAs
                {
                    const int pieces = G * (D / 4), shares = ST_CONSUMERS / pieces >= 8 ? 8 : (ST_CONSUMERS / pieces >= 4 ? 4 : 2);
#pragma unroll 1
                    for (int i = tid; i < pieces * shares; i += ST_CONSUMERS) {
                        const int sh = i / pieces, j = i - sh * pieces, gg = j / (D / 4), e = (j & (D / 4 - 1)) * 4;
                        float top = red_ml[gg * 2];
#pragma unroll 1
                        for (int w = 1; w < nw; ++w) top = fmaxf(top, red_ml[(w * G + gg) * 2]);
                        const float base = top == -INFINITY ? 0.f : top;  // of a split whose scores are all -inf: it counts for nothing in the other splits' sum
                        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                        float lsum = 0.f;
#pragma unroll 1
                        for (int w = 0; w < nw; ++w) {
                            const float2 ml = *reinterpret_cast<const float2*>(red_ml + (w * G + gg) * 2);
                            const float4 v = *reinterpret_cast<const float4*>(red_o + (w * G + gg) * D + e);
                            const float f = st_exp2(ml.x - base);
                            acc.x += v.x * f; acc.y += v.y * f; acc.z += v.z * f; acc.w += v.w * f;
                            lsum += ml.y * f;
                        }
                        const int at = (kvh * G + gg) * p.splits + split;
                        const uint32_t dst = smem_u32(part_o + at * D + e), dst_ml = smem_u32(part_ml + at * 2), bar = smem_u32(&xbar[B_ATTN]);
                        const uint64_t ml = static_cast<uint64_t>(__float_as_uint(top)) | (static_cast<uint64_t>(__float_as_uint(lsum)) << 32);
#pragma unroll 1
                        for (int to = sh; to < C; to += shares) {
                            st_send16(st_map(dst, to), acc, st_map(bar, to));
                            if (e == 0) st_send8(st_map(dst_ml, to), ml, st_map(bar, to));
                        }
                    }
                }
            }
        }
    given_up:;
    }
    __syncwarp();
    st_cluster_sync();  // no CTA leaves while another may still send to it
    if (poisoned) st_settle();  // what was sent to a CTA that has stopped waiting for it
}

static int st_align(int v, int a) { return (v + a - 1) / a * a; }

// Lanes per pair of rows for `pairs` pairs of `chunks` 16-byte pieces: the shortest way of a warp through them, about 340 cycles per
// piece for the four warps of a scheduler and 60 per step of the reduction.
static int st_lanes(int pairs, int chunks) {
    int best = 0;
    long long cost = 0;
    for (int l = 0; l <= 5; ++l) {
        const int per = ST_WARPS * (32 >> l), passes = (pairs + per - 1) / per, steps = (chunks + (1 << l) - 1) >> l;
        const long long c = static_cast<long long>(passes) * (steps * 340 + 60 * l + 80);
        if (l == 0 || c < cost) {
            best = l;
            cost = c;
        }
    }
    return best;
}

// Shared-memory plan for a cluster of C CTAs; false when it does not fit.
static bool st_plan(StepParams& p, int C, int D) {
    const int G = p.nq / p.nkv, QD = p.nq * D, KVD = p.nkv * D, NQKV = QD + 2 * KVD;
    int rows[4] = {NQKV, p.hidden, p.inter, p.hidden}, ks[4] = {p.hidden, QD, p.hidden, p.inter};
    int most = 0, kmax = 0;
    for (int i = 0; i < 4; ++i) {
        rows[i] = (rows[i] / 4 + C - 1) / C * 4;
        if (rows[i] > most) most = rows[i];
        if (ks[i] > kmax) kmax = ks[i];
    }
    p.splits = C / p.nkv;
    int o = 0;
    auto take = [&](int bytes) { const int at = o; o += st_align(bytes, 128); return at; };
    p.o_h = take(p.hidden * 2); p.o_qkv = take(NQKV * 2); p.o_attn_o = take(p.nq * p.splits * D * 4); p.o_attn_ml = take(p.nq * p.splits * 8);
    p.o_o = take(p.hidden * 2); p.o_act = take(p.inter * 2); p.o_down = take(p.hidden * 2); p.o_xq = take(kmax); p.o_val = take(kmax * 2); p.o_out = take(most * 2);
    p.o_qr = take(G * D * 4); p.o_kn = take(D * 2); p.o_red = take(ST_WARPS * (D + 2) * 4);
    p.meta_bytes = st_align(48 + p.hidden * 4, 128);
    p.o_meta = take(2 * p.meta_bytes); p.o_rope = take(D * 4);
    p.o_ring = o;
    const int room = ST_SMEM_MAX - 1024 - o;  // the static part
    p.stage_bytes = room >= 5 * 32768 ? 32768 : 16384;
    p.stages = room / p.stage_bytes;
    if (p.stages > ST_MAX_STAGES) p.stages = ST_MAX_STAGES;
    if (p.stages < 3) return false;
    for (int i = 0; i < 4; ++i) {
        const int rb = ks[i] / 4 * (i == 2 ? 2 : 1), fit = p.stage_bytes / rb;
        if (fit < 1) return false;
        const int count = (rows[i] + fit - 1) / fit, per = (rows[i] + count - 1) / count;
        p.lpr_log2[i] = st_lanes(i == 2 ? per : (per + 1) / 2, ks[i] / 64);
    }
    return true;
}

static bool st_shapes_ok(int64_t B, int hidden, int nq, int nkv, int D, int inter, int64_t T) {
    return B > 0 && B <= 4096 && nq > 0 && nkv > 0 && nq % nkv == 0 && nq / nkv <= ST_MAX_G && nkv <= 16 && (D == 64 || D == 128) && T > 0 && T < (1 << 30) &&
           hidden >= 64 && hidden % 64 == 0 && hidden <= ST_MAX_K && inter >= 64 && inter % 64 == 0 && inter <= ST_MAX_K && nq * D <= ST_MAX_K;
}

template <int D>
static int st_configure(cudaLaunchConfig_t& lc, cudaLaunchAttribute* attr, int C, int64_t B, size_t smem) {
    static PerDeviceOnce configured;
    const int dev = current_device();
    if (configured.needs(dev)) {
        WF_CUDA(cudaFuncSetAttribute(decode_layers_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM_MAX - 1024));
        WF_CUDA(cudaFuncSetAttribute(decode_layers_kernel<D>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        configured.mark(dev);
    }
    lc.gridDim = dim3(static_cast<unsigned>(B * C));
    lc.blockDim = dim3(ST_THREADS);
    lc.dynamicSmemBytes = smem;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(C);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return WF_OK;
}

// How many clusters of this plan the device holds at once (0: none).
template <int D>
static int st_clusters(const StepParams& p, int C) {
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (st_configure<D>(lc, attr, C, 1, static_cast<size_t>(p.o_ring) + static_cast<size_t>(p.stages) * p.stage_bytes) != WF_OK) return 0;
    if (cudaOccupancyMaxActiveClusters(&n, decode_layers_kernel<D>, &lc) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace wf

using namespace wf;

// Where it pays, in us per layer: 11 for the chain of a layer, 1.1 per 2^20 weights and 3.8 per 2^20 of context x query width with 16 CTAs,
// twice that with 8 (within 4 of what was measured for widths of 256 to 4096 and contexts of 140 to 10000, up to 45).  The separate launches take,
// for one or two sequences, 21 to 32 at context 140 and 28 to 35 at the longest context that the rule takes; for three and more 33 to 44
// and 37 to 54.  It is the slower one nowhere among the 210 shapes measured (widths of 256 to 1280, one to twelve sequences, at the end of the cache); at the line,
// this kernel / the separate launches: width 512, context 8900, one sequence 28.8 / 29.5, two 32.2 / 32.1; 576, 7300, 29.8 / 32.0 and 29.6 /
// 35.1; 1024, 600, one 20.7 / 29.2; four, 2300, 28.9 / 38.4; 576, 10000, seven 35.2 / 53.6.
// T is the length of the cache: one captured step serves every position.  The kernel reads the valid positions only, so that a short context in
// a long cache would gain more than the rule assumes, and a cache longer than it allows gets none of it.
static bool st_pays(int64_t B, int hidden, int nq, int nkv, int D, int inter, int64_t T, int C) {
    const double mi = 1.0 / (1 << 20), weights = mi * hidden * (2.0 * nq * D + 2.0 * nkv * D + 3.0 * inter), context = mi * nq * D * static_cast<double>(T);
    return 11 + (1.1 * weights + 3.8 * context) * 16 / C <= (B <= 2 ? 30 : 36);
}

extern "C" int wf_decode_layers_cluster(int64_t B, int hidden, int nq, int nkv, int D, int inter, int64_t T) {
    if (!st_shapes_ok(B, hidden, nq, nkv, D, inter, T) || require_device() != WF_OK) return 0;
    for (int C = 16; C >= 8; C /= 2) {
        StepParams p = {};
        p.hidden = hidden; p.nq = nq; p.nkv = nkv; p.inter = inter;
        if (nkv > C || !st_pays(B, hidden, nq, nkv, D, inter, T, C) || !st_plan(p, C, D)) continue;
        const int n = D == 64 ? st_clusters<64>(p, C) : st_clusters<128>(p, C);
        if (n >= B) return C;
    }
    return 0;
}

extern "C" int wf_decode_layers_bf16(const wf_step_layer* layers, int L, const void* h, const void* norm_f, void* xf, const float* cos, const float* sin,
                                     const int64_t* pos, int64_t B, int hidden, int nq, int nkv, int D, int inter, int64_t T, int act, float eps,
                                     float quant_eps, float scale, int cluster, unsigned flags, void* stream) {
    WF_REQUIRE(layers && h && norm_f && xf && cos && sin && pos, "wf_decode_layers_bf16: null pointer");
    WF_REQUIRE(L > 0 && st_shapes_ok(B, hidden, nq, nkv, D, inter, T) && (act == 0 || act == 1), "wf_decode_layers_bf16: shape not supported");
    WF_REQUIRE(cluster == 8 || cluster == 16, "wf_decode_layers_bf16: clusters of 8 or 16 CTAs");
    WF_REQUIRE(((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(norm_f) | reinterpret_cast<uintptr_t>(xf)) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(layers) & 7) == 0,
               "wf_decode_layers_bf16: tensors must be 16-byte aligned");
    if (int rc = require_device()) return rc;
    StepParams p = {};
    p.layers = layers;
    p.h = static_cast<const __nv_bfloat16*>(h); p.norm_f = static_cast<const __nv_bfloat16*>(norm_f); p.xf = static_cast<__nv_bfloat16*>(xf);
    p.cosv = cos; p.sinv = sin; p.pos = pos;
    p.L = L; p.hidden = hidden; p.nq = nq; p.nkv = nkv; p.inter = inter; p.T = static_cast<int>(T);
    p.act = act; p.eps = eps; p.qeps = quant_eps; p.scale_log2 = scale * 1.4426950408889634f;
    if (nkv > cluster || !st_plan(p, cluster, D)) return fail(WF_E_LIMIT, "wf_decode_layers_bf16: the model does not fit a cluster of %d CTAs", cluster);
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute attr[2];
    const size_t smem = static_cast<size_t>(p.o_ring) + static_cast<size_t>(p.stages) * p.stage_bytes;
    if (int rc = D == 64 ? st_configure<64>(lc, attr, cluster, B, smem) : st_configure<128>(lc, attr, cluster, B, smem)) return rc;
    lc.stream = static_cast<cudaStream_t>(stream);
    if (flags & WF_FLAG_PDL) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        lc.numAttrs = 2;
    }
    if (D == 64) WF_CUDA(cudaLaunchKernelEx(&lc, decode_layers_kernel<64>, p));
    else WF_CUDA(cudaLaunchKernelEx(&lc, decode_layers_kernel<128>, p));
    return WF_OK;
}

// read-out for wf_device_status: the status word of this file's kernel (cleared when set)
extern "C" int wf_step_status_fetch(int* out) {
    WF_CUDA(cudaMemcpyFromSymbol(out, g_step_status, sizeof(int)));
    if (*out) {
        int zero = 0;
        WF_CUDA(cudaMemcpyToSymbol(g_step_status, &zero, sizeof(int)));
    }
    return WF_OK;
}

// Split-K flash-decode GQA for sm_100a: 16 query heads over 4 kv heads, head_dim 256.
//
// Math (reference: src/attention.cu:4): score_t = (q_h . K[t][h>>2]) / 16, softmax over
// the cached tokens, out_h = sum_t p_t V[t][h>>2]; cache layout [token][4][256].
//
// The reference runs one CTA per query head, keeps every score in shared memory
// (which fails past ~12K tokens) and re-reads each kv head's cache four times.
// Here a CTA owns (kv head, token range): it streams its slab of K and V exactly
// once for the four query heads that share the kv head, keeps an online softmax
// per warp, and hands (max, denominator, weighted V) to the CTAs of its cluster
// (and, where one cluster is not enough, through scratch to the other clusters);
// partials are folded in split order, so results do not depend on scheduling.  The fused entry also does the per-head RMSNorm,
// partial RoPE and the cache write of the current token (src/ops.cu:9,
// src/qwen_kernels.cu:15,31) so one launch replaces five.
//
// bf16 cache, long contexts: the scalar loop is bound by instruction issue (half the bytes, the same instructions),
// so from kMmaMinTokens cached rows on the warps score and accumulate on the tensor cores instead (mma.sync
// m16n8k16 bf16, fp32 accumulation): 16 cached rows per step per warp, fetched into the warp's own shared-memory
// tiles by one cp.async.bulk per row (keys and values on an mbarrier each, the next tile of one requested while the other is
// worked on; bounded waits); the fp32 query goes in
// as two bf16 pieces (hi + lo) in the eight N columns (4 heads x 2 pieces), the softmax weights likewise for P.V, so
// products keep ~16 bits of the fp32 operands and the cache values are exact.
#include "attention_body.cuh"
#include "host_util.h"
#include "umma_common.cuh"

#include <algorithm>
#include <mutex>

namespace insg {

constexpr int kAtThreads = 256;
constexpr int kAtWarps = 8;
constexpr int kGroup = 4;                    // tokens a warp scores at once
constexpr int kBlock = kAtWarps * kGroup;    // rows the warps of a CTA score at once
constexpr int kMinChunk = kBlock;            // tokens per split at least
constexpr int kMmaMinTokens = 2048;          // bf16 cache: cached rows from which the tensor-core loop is used
constexpr int kTileRow = 528;                // a staged row: 512 bytes of bf16 + 16 of padding (conflict-free ldmatrix)
constexpr int kTileBytes = 16 * kTileRow;    // 16 rows
constexpr size_t kMmaSmem = size_t(kAtWarps) * 2 * kTileBytes; // per warp: a key tile and a value tile

constexpr float kNan = __builtin_nanf("");
__device__ __forceinline__ float warp_max_redux(float v) // maximum over the warp, as fmaxf takes it
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ uint32_t bf16_piece_pair(float a, float b, int piece)
{
    // piece 0: the bf16 roundings of a and b; piece 1: the bf16 roundings of what those left over
    __nv_bfloat16 ha = __float2bfloat16_rn(a), hb = __float2bfloat16_rn(b);
    if (piece) {
        ha = __float2bfloat16_rn(a - __bfloat162float(ha));
        hb = __float2bfloat16_rn(b - __bfloat162float(hb));
    }
    return uint32_t(__bfloat16_as_ushort(ha)) | (uint32_t(__bfloat16_as_ushort(hb)) << 16);
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One warp's share of a split on the tensor cores: rows t0 + 16 (warp + 8 n) .. of [t0, t1), bf16 cache.  Leaves the
// warp's (max, denominator, weighted values) in s_m_w / s_l_w / s_acc_w like the scalar loop does.
__device__ __forceinline__ void attn_mma_warp(const void *kc, const void *vc, int kvh, int t0, int t1, int warp, int lane,
                                              const float (*s_q)[256], uint8_t *tiles, uint64_t *bar, volatile int *abort_flag,
                                              float *s_m_w, float *s_l_w, float (*s_acc_w)[256])
{
    const int g = lane >> 2, t = lane & 3;
    uint8_t *tile_k = tiles + size_t(warp) * 2 * kTileBytes, *tile_v = tile_k + kTileBytes;
    if (lane == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.global;" ::: "memory"); // earlier launches wrote the rows by ordinary stores, the bulk copies read them through the async proxy
    __syncwarp();
    // Keys and values have a barrier each: a tile of keys is requested as soon as the one before has been scored, a tile of values
    // as soon as the one before has been added, so that one of the two is on its way whatever the warp does.
    auto request = [&](const void *cache, uint8_t *tile, uint64_t *b, int tb) {
        __syncwarp();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the tile was read by ordinary loads; the copies below overwrite it
        if (lane == 0) mbar_expect_tx(b, 16 * 512);
        __syncwarp();
        if (lane < 16) {
            const int tok = min(tb + lane, t1 - 1); // rows past the split repeat its last row: masked below
            bulk_load(tile + lane * kTileRow, static_cast<const uint8_t *>(cache) + (size_t(tok) * 4 + kvh) * 512, 512, b);
        }
    };
    const int first = t0 + 16 * warp;
    if (first < t1) {
        request(kc, tile_k, bar, first);
        request(vc, tile_v, bar + 1, first);
    }
    // the query as the B operand: column g = (head g >> 1, piece g & 1), k rows 2t, 2t+1 and 2t+8, 2t+9 of every 16 dims
    uint32_t qb[16][2];
    {
        const float *qh = s_q[g >> 1];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int d = 16 * i + 2 * t;
            qb[i][0] = bf16_piece_pair(qh[d] * 0.0625f, qh[d + 1] * 0.0625f, g & 1);
            qb[i][1] = bf16_piece_pair(qh[d + 8] * 0.0625f, qh[d + 9] * 0.0625f, g & 1);
        }
    }
    float m_run = -3.0e38f, l_run = 0.f; // of head t (the same in the eight lanes that share t, l_run as a partial sum)
    float acc[16][4];                    // [16 dims each][dim g: (hi, lo) of head t | dim g + 8: (hi, lo)]
#pragma unroll
    for (int j = 0; j < 16; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    uint32_t phase = 0;
    const uint32_t lm_row = uint32_t(lane & 7), lm_id = uint32_t(lane >> 3);
    const uint32_t k_addr = smem_u32(tile_k) + ((lm_id & 1) * 8 + lm_row) * kTileRow + (lm_id >> 1) * 16; // + 32 i: rows of K as m, dims as k
    const uint32_t v_addr = smem_u32(tile_v) + ((lm_id >> 1) * 8 + lm_row) * kTileRow + (lm_id & 1) * 16; // + 32 j: transposed: dims as m, rows as k
    for (int tb = t0 + 16 * warp; tb < t1; tb += 16 * kAtWarps) {
        const int tn = tb + 16 * kAtWarps;
        if (!mbar_wait(bar, phase, abort_flag)) {
            mbar_wait(bar + 1, phase, abort_flag); // the values' copy, before the tile's memory is given up
            break;
        }
        // ---- scores: S[16 rows][8 columns] = K tile . q pieces ----
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 16; i++) {
            uint32_t a0, a1, a2, a3;
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3) : "r"(k_addr + 32 * i));
            mma_bf16(c, a0, a1, a2, a3, qb[i][0], qb[i][1]);
        }
        if (tn < t1) request(kc, tile_k, bar, tn);
        const bool v0 = tb + g < t1, v1 = tb + g + 8 < t1;
        const float s0 = v0 ? c[0] + c[1] : -3.0e38f, s1 = v1 ? c[2] + c[3] : -3.0e38f; // rows tb + g and tb + g + 8, head t
        float mx = fmaxf(s0, s1);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float m_new = fmaxf(m_run, mx), corr = __expf(m_run - m_new);
        const float p0 = v0 ? __expf(s0 - m_new) : 0.f, p1 = v1 ? __expf(s1 - m_new) : 0.f;
        l_run = fmaf(l_run, corr, p0 + p1);
        m_run = m_new;
#pragma unroll
        for (int j = 0; j < 16; j++) { acc[j][0] *= corr; acc[j][1] *= corr; acc[j][2] *= corr; acc[j][3] *= corr; }
        // ---- the weights as the B operand of P.V: column g = (head g >> 1, piece g & 1), k rows = cached rows ----
        const int src_a = 8 * t + (g >> 1), src_b = src_a + 4; // lanes that hold rows 2t and 2t + 1 (and + 8) of that head
        const float x0 = __shfl_sync(0xffffffffu, p0, src_a), x1 = __shfl_sync(0xffffffffu, p0, src_b);
        const float y0 = __shfl_sync(0xffffffffu, p1, src_a), y1 = __shfl_sync(0xffffffffu, p1, src_b);
        const uint32_t pb0 = bf16_piece_pair(x0, x1, g & 1), pb1 = bf16_piece_pair(y0, y1, g & 1);
        if (!mbar_wait(bar + 1, phase, abort_flag)) {
            if (tn < t1) mbar_wait(bar, phase ^ 1u, abort_flag); // the next keys' copy
            break;
        }
        phase ^= 1u;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            uint32_t a0, a1, a2, a3;
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3) : "r"(v_addr + 32 * j));
            mma_bf16(acc[j], a0, a1, a2, a3, pb0, pb1);
        }
        if (tn < t1) request(vc, tile_v, bar + 1, tn);
    }
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 4);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 8);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 16);
    if (g == 0) { s_m_w[t] = m_run; s_l_w[t] = l_run; }
#pragma unroll
    for (int j = 0; j < 16; j++) {
        s_acc_w[t][16 * j + g] = acc[j][0] + acc[j][1];
        s_acc_w[t][16 * j + g + 8] = acc[j][2] + acc[j][3];
    }
}

// Clusters: a kv head's cache is cut over clusters of CL CTAs.  The CTAs of a cluster exchange their partial results through
// distributed shared memory, each finishing its share of the output dims: a context that one cluster holds needs no global
// scratch, fence or ticket.  Longer ones use up to `clusters` clusters per head; their results go to scratch and the last one
// to arrive (a ticket per CTA rank) folds them in order.  For one launch's clusters the cut depends on the row count alone; the
// clusters on the cache's type and capacity and, in a batch, on how many sequences share the device (launch_attn).
// Measured as graph replays (fp32 cache, one step; in brackets with one CTA per split and a ticket): 40 rows 4.9 us (7.1), 1024
// rows 8.8 (10.3), 8 x 600 rows 14.2 (38.5), 8 x 5000 rows 58.6 (119.5), which is 5.6 TB/s, 86 % of the copy peak.
//
// A block more costs a CTA 1.5 us (bf16 1.1), the exchange between clusters 2.4 us: one cluster up to two blocks a CTA (three in a batch, whose
// sequences share the device, and with the bf16 cache); then, with the fp32 cache, clusters of one block a CTA up to four blocks a CTA of one
// cluster; beyond that clusters of two.  fp32 cache, one cluster / one block a CTA / two: 400 rows 6.8 / 7.4 / -, 600 rows 8.3 / 7.7 / 8.5, 800 rows
// 9.9 / 8.4 / 8.8, 1500 rows 13.4 / 10.2 / 9.4 us; two sequences of 600 rows 8.4 / 9.2 / 10.4; bf16 cache, 600 rows 7.3 / 7.8 / 8.6.
constexpr int kMaxClusters = 8; // per kv head
struct AttnRule {
    int one, some; // rows up to which one cluster takes them, up to which several take a block a CTA
};
__host__ __device__ inline AttnRule attn_rule(bool bf16, bool batch, int unit) // unit: CTAs of a cluster
{
    return AttnRule{(bf16 || batch ? 3 : 2) * kBlock * unit, bf16 ? 0 : 4 * kBlock * unit};
}
__host__ __device__ inline int attn_clusters(const AttnRule &r, int rows, int unit)
{
    const int per = (rows <= r.some ? kBlock : 2 * kBlock) * unit;
    return rows <= r.one ? 1 : (rows + per - 1) / per;
}

struct AttnCut {
    int active, chunk; // clusters at work, rows per CTA
};
// HALVES: two clusters of four in place of one of eight, with the same bits: when both have rows, the last to arrive folds the
// eight CTAs' results as the cluster of eight does.
template <int CL, bool HALVES> __device__ __forceinline__ AttnCut attn_cut(int rows, int clusters, const AttnRule &rule)
{
    constexpr int kUnit = HALVES ? 2 * CL : CL; // CTAs
    AttnCut c;
    c.active = min(HALVES ? clusters / 2 : clusters, attn_clusters(rule, rows, kUnit));
    const int ctas = c.active * kUnit;
    c.chunk = max(kMinChunk, (rows + ctas - 1) / ctas);
    if (HALVES) c.active = (rows + c.chunk * CL - 1) / (c.chunk * CL); // a half without rows has nothing to do
    return c;
}

template <bool BF16, bool FUSED, int CL, bool HALVES>
__global__ void __launch_bounds__(kAtThreads, 2) attn_splitk_kernel(const __grid_constant__ AttnParams p, int clusters)
{
    using Row = KvRow<BF16>;
    constexpr bool kMma = BF16 && CL == 4 && !HALVES; // the bf16 launches of long contexts
    constexpr bool kQuarters = !BF16 || kMma; // the loop over blocks of rows (below)
    constexpr int kParts = HALVES ? CL : 1; // partial results of a cluster in scratch
    constexpr int kMine = 1024 / CL; // output dims this CTA finishes
    __shared__ __align__(16) float s_q[4][256];
    __shared__ __align__(16) float s_knew[256], s_vnew[256];
    __shared__ float s_m[kAtWarps][4], s_l[kAtWarps][4];
    __shared__ __align__(16) float s_acc[kQuarters && !kMma ? 4 : kAtWarps][4][256]; // the quarters' or the warps' sums
    __shared__ __align__(16) float4 s_score[2][kQuarters ? kBlock : 1];     // [row] scores of the four heads
    __shared__ __align__(16) float4 s_p[kAtWarps][kQuarters ? kBlock : 1];  // a warp's copy of the weights
    __shared__ __align__(16) float s_in[CL][kMine]; // the cluster's partial sums of this CTA's dims
    __shared__ __align__(8) float2 s_ml[CL];        // and their maxima and denominators
    __shared__ __align__(8) uint64_t s_there;       // all of them have come
    __shared__ int s_last;
    __shared__ __align__(8) uint64_t s_bar[2 * kAtWarps];
    __shared__ int s_abort, s_lost; // a wait of the tensor-core loop, or of the exchange, ran out
    __shared__ uint8_t s_lut[84];
    extern __shared__ __align__(128) uint8_t s_tiles[]; // bf16 cache only: per warp a key tile and a value tile

    const int rank = int(blockIdx.x) % CL, cluster = int(blockIdx.x) / CL % clusters, kvh = int(blockIdx.x) / (CL * clusters);
    const int split = cluster * CL + rank;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // token of a chunk (plain form) or sequence of a batch (fused form); a single launch has blockIdx.y == 0 and zero strides
    const int bt = blockIdx.y;
    const float *q_in = p.q + size_t(bt) * p.q_stride;
    float *out_base = p.out + size_t(bt) * p.out_stride;
    unsigned *counters = reinterpret_cast<unsigned *>(reinterpret_cast<uint8_t *>(p.counters) + size_t(bt) * p.scratch_stride);
    float *partials = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(p.partials) + size_t(bt) * p.scratch_stride);
    void *kc = static_cast<uint8_t *>(p.kc) + size_t(bt) * p.cache_stride, *vc = static_cast<uint8_t *>(p.vc) + size_t(bt) * p.cache_stride;
    const float *k_raw = p.k_raw + size_t(bt) * p.kvin_stride, *v_new = p.v_new + size_t(bt) * p.kvin_stride;

    if (tid == 0) {
        s_abort = s_lost = 0;
        mbar_init(&s_there, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory"); // the peers have started, with their barriers, when this completes
    // Launches that may not read ahead start as early and wait here; what follows them may start when they have waited, as if they had been launched then
    // (calls one behind the other: 32768 bf16 rows 30.9 -> 28.5 us, 8 x 5000 fp32 rows 62.8 -> 61.0; a speculative pass, two such launches a layer, 1301 -> 1287).
    if (p.wait_first) pdl_wait();
    pdl_launch_dependents();

    // Geometry from the position as it is visible now.  Cache rows of earlier tokens never change
    // again, so the first token group of every warp is fetched while the producer of q still runs;
    // the position is read again after the wait and the fetch repeated if it moved.
    int pos = -1, tokens = p.tokens;
    if constexpr (FUSED) {
        pos = __ldcg(p.position) + p.position_offset;
        tokens = pos + 1;
    } else if (p.position) { // chunk: the rows were written by the launch before this one (plain stream order)
        tokens = __ldcg(p.position) + p.position_offset + bt + 1;
    }
    tokens = max(1, min(tokens, p.max_context)); // host checks; never index past the cache
    const AttnRule rule = attn_rule(BF16, p.batch != 0, HALVES ? 2 * CL : CL);
    AttnCut cut = attn_cut<CL, HALVES>(tokens, clusters, rule);
    int t0 = split * cut.chunk, t1 = min(tokens, t0 + cut.chunk);
    int fresh = tokens - 1; // the row the producer (or this kernel) is still writing

    if (p.image && tid < 81) s_lut[tid] = digit_pair_code(tid); // read behind the barriers below
    bool use_mma = kMma && tokens >= kMmaMinTokens; // long bf16 contexts: the tensor-core loop (reads every row from the cache)
    // The rows that come next: a warp's four rows of keys are replaced by the following ones as soon as they are scored, its values (of the same rows, or
    // half of the dims of a quarter of the block's rows) as soon as they are added.  (Two groups or blocks would take a CTA's registers past
    // what fits beside the products' launches, and the launch could start only when its predecessor had left the SM.)
    GroupRaw<BF16, kGroup> ga;
    const int quarter = warp >> 1, dim0 = (warp & 1) * 128 + lane * 4;
    typename Row::Quad vr[kQuarters ? kBlock / 4 : 1];
    auto load_quad = [&](const void *cache, int t) { return Row::load_quad(cache, (size_t(t) * 4 + kvh) * 256 + dim0); };
    auto fetch_keys = [&](int tb, int tend) {
#pragma unroll
        for (int g = 0; g < kGroup; g++) {
            const int t = tb + warp * kGroup + g;
            ga.k[g] = t < tend ? Row::load_raw(kc, (size_t(t) * 4 + kvh) * 256, lane) : Row::zero();
        }
    };
    auto fetch_values = [&](int tb, int tend) {
#pragma unroll
        for (int g = 0; g < kBlock / 4; g++) {
            const int t = tb + quarter * (kBlock / 4) + g;
            vr[g] = t < tend ? load_quad(vc, t) : Row::zero_quad();
        }
    };
    auto fetch = [&] {
        if constexpr (kQuarters) {
            if (use_mma) return;
            fetch_keys(t0, min(t1, fresh));
            fetch_values(t0, min(t1, fresh));
        } else if (!use_mma) load_group<BF16, kGroup>(kc, vc, kvh, t0 + warp * kGroup, min(t1, fresh), lane, ga);
    };
    fetch();
    uint4 norm_wv = make_uint4(0u, 0u, 0u, 0u);
    float rope_c[8], rope_s[8];
    if constexpr (FUSED) {
        if (warp < 5) {
            norm_wv = reinterpret_cast<const uint4 *>(warp < 4 ? p.q_w : p.k_w)[lane];
            if (lane < 8) rope_table(pos, lane, p.fast_trig != 0, rope_c, rope_s);
        }
    }

    pdl_wait();

    float raw[8]; // warps 0-3: a query head, 4: the new key, 5: the new value; asked for together with the position
    if constexpr (FUSED) {
        if (warp < 6) {
            const float *src = warp < 4 ? q_in + size_t(kvh * 4 + warp) * 512 : (warp == 4 ? k_raw : v_new) + kvh * 256;
            const float4 a = __ldcg(reinterpret_cast<const float4 *>(src + lane * 8)), b = __ldcg(reinterpret_cast<const float4 *>(src + lane * 8 + 4));
            raw[0] = a.x; raw[1] = a.y; raw[2] = a.z; raw[3] = a.w; raw[4] = b.x; raw[5] = b.y; raw[6] = b.z; raw[7] = b.w;
        }
        const int now = __ldcg(p.position) + p.position_offset;
        if (now != pos) {
            pos = now;
            tokens = max(1, min(pos + 1, p.max_context));
            cut = attn_cut<CL, HALVES>(tokens, clusters, rule);
            t0 = split * cut.chunk;
            t1 = min(tokens, t0 + cut.chunk);
            fresh = tokens - 1;
            use_mma = kMma && tokens >= kMmaMinTokens;
            fetch();
            if (warp < 5 && lane < 8) rope_table(pos, lane, p.fast_trig != 0, rope_c, rope_s);
        }
    }
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    if (cluster >= cut.active) return; // the whole cluster
    const bool has_work = t0 < tokens;
    // the gate of the output this CTA will finish (image only), fetched ahead
    const int my_head = kvh * 4 + rank * kMine / 256, my_dim = rank * kMine % 256 + tid; // of thread tid < kMine
    float gv = 0.f;
    if (p.image && tid < kMine) gv = __ldcg(p.gate + size_t(bt) * 8192 + my_head * 512 + 256 + (p.gate_elementwise ? my_dim : 0));

    if (has_work) {
        // ---- query (and current key) preparation --------------------------------
        if constexpr (FUSED) {
            if (warp < 4) {
                norm_rope_256(raw, norm_wv, lane, pos, rope_c, rope_s);
                reinterpret_cast<float4 *>(s_q[warp])[lane * 2] = make_float4(raw[0], raw[1], raw[2], raw[3]);
                reinterpret_cast<float4 *>(s_q[warp])[lane * 2 + 1] = make_float4(raw[4], raw[5], raw[6], raw[7]);
            } else if (warp == 4 && pos >= t0 && pos < t1) {
                norm_rope_256(raw, norm_wv, lane, pos, rope_c, rope_s);
                const size_t row = (size_t(pos) * 4 + kvh) * 256 + lane * 8;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    s_knew[lane * 8 + j] = Row::round(raw[j]);
                    if (use_mma) Row::store(kc, row + j, raw[j]);
                }
                if (use_mma) asm volatile("fence.proxy.async.global;" ::: "memory"); // the tensor-core loop fetches this row by bulk copy
            } else if (warp == 5 && pos >= t0 && pos < t1) {
                const size_t row = (size_t(pos) * 4 + kvh) * 256 + lane * 8;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    s_vnew[lane * 8 + j] = Row::round(raw[j]);
                    if (use_mma) Row::store(vc, row + j, raw[j]);
                }
                if (use_mma) asm volatile("fence.proxy.async.global;" ::: "memory");
            }
        } else {
            for (int i = tid; i < 1024; i += kAtThreads) s_q[i >> 8][i & 255] = __ldcg(q_in + size_t(kvh) * 1024 + i);
        }
    }
    __syncthreads();

    bool mma_done = false;
    if constexpr (kMma) {
        if (has_work && use_mma) {
            attn_mma_warp(kc, vc, kvh, t0, t1, warp, lane, s_q, s_tiles, &s_bar[2 * warp], &s_abort, s_m[warp], s_l[warp], s_acc[warp]);
            mma_done = true;
        }
    }
    float m0 = -3.0e38f, l0 = 0.f; // of head warp >> 1: the CTA's maximum and denominator
    if constexpr (kQuarters) {
    if (!mma_done) {
        // ---- fp32 cache (and the few rows of a long bf16 cache): blocks of 32 rows.  The CTA's warps score four rows each, then every warp has the weights of all rows and adds its part of the
        // values, so that the warps share their maxima and nothing is left to be rescaled between them.  With a loop as below 40 rows took 5.3 us
        // instead of 4.9, 8192 rows 19.7 instead of 18.1, 8 x 5000 rows the same 58.7; the bf16 cache, with half the bytes to wait for, is better off without
        // the barrier (8 x 2000 rows 24.1 like this, 21.1 as below).
        float m[4], l[4], acc[4][4]; // per head; l: this lane's rows
#pragma unroll
        for (int h = 0; h < 4; h++) {
            m[h] = -3.0e38f;
            l[h] = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) acc[h][j] = 0.f;
        }
        const int tend = min(t1, fresh);
        int buf = 0;
#pragma unroll 1
        for (int tb = t0; tb < t1; tb += kBlock, buf ^= 1) {
            const int gk = fresh < t1 ? fresh - tb - warp * kGroup : -1, gv_row = fresh < t1 ? fresh - tb - quarter * (kBlock / 4) : -1; // the newest row's place
            if (gk >= 0 && gk < kGroup) { // from shared memory or, now that the wait is over, from the cache
                const typename Row::Raw x = FUSED ? Row::pack(s_knew + lane * 8) : Row::load_raw(kc, (size_t(fresh) * 4 + kvh) * 256, lane);
#pragma unroll
                for (int g = 0; g < kGroup; g++)
                    if (g == gk) ga.k[g] = x;
            }
            if (gv_row >= 0 && gv_row < kBlock / 4) {
                const typename Row::Quad x = FUSED ? Row::pack_quad(s_vnew + dim0) : load_quad(vc, fresh);
#pragma unroll
                for (int g = 0; g < kBlock / 4; g++)
                    if (g == gv_row) vr[g] = x;
            }
            float s[16];
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float4 qa = *reinterpret_cast<const float4 *>(&s_q[h][lane * 8]), qb = *reinterpret_cast<const float4 *>(&s_q[h][lane * 8 + 4]);
#pragma unroll
                for (int g = 0; g < kGroup; g++) {
                    float kk[8];
                    Row::unpack(ga.k[g], kk);
                    float z = qa.x * kk[0];
                    z = fmaf(qa.y, kk[1], z); z = fmaf(qa.z, kk[2], z); z = fmaf(qa.w, kk[3], z);
                    z = fmaf(qb.x, kk[4], z); z = fmaf(qb.y, kk[5], z); z = fmaf(qb.z, kk[6], z); z = fmaf(qb.w, kk[7], z);
                    s[g * 4 + h] = z;
                }
            }
            if (tb + kBlock < t1) fetch_keys(tb + kBlock, tend);
            // sums over the lanes, halving the values a lane carries at every step: 16 shuffles where summing each takes 80
#pragma unroll
            for (int n = 8, mk = 16; n; n >>= 1, mk >>= 1) {
                const bool up = (lane & mk) != 0;
#pragma unroll
                for (int i = 0; i < n; i++) {
                    const float keep = up ? s[i + n] : s[i], send = up ? s[i] : s[i + n];
                    s[i] = keep + __shfl_xor_sync(0xffffffffu, send, mk);
                }
            }
            const float score = (s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1)) * 0.0625f; // row lane >> 3, head (lane >> 1) & 3
            if (!(lane & 1)) reinterpret_cast<float *>(&s_score[buf][warp * kGroup + (lane >> 3)])[(lane >> 1) & 3] = score;
            __syncthreads();
            const float4 own = s_score[buf][lane]; // row `lane` of the block
            const float sc[4] = {own.x, own.y, own.z, own.w};
            const bool on = tb + lane < t1;
            float pr[4], corr[4];
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float mn = fmaxf(m[h], warp_max_redux(on ? sc[h] : -3.0e38f));
                corr[h] = __expf(m[h] - mn);
                pr[h] = on ? __expf(sc[h] - mn) : 0.f;
                m[h] = mn;
                l[h] = fmaf(l[h], corr[h], pr[h]);
            }
            s_p[warp][lane] = make_float4(pr[0], pr[1], pr[2], pr[3]);
            __syncwarp();
            float part[4][4]; // of this block
#pragma unroll
            for (int g = 0; g < kBlock / 4; g++) {
                const float4 w = s_p[warp][quarter * (kBlock / 4) + g];
                float vv[4];
                Row::unpack_quad(vr[g], vv);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    part[0][j] = g ? fmaf(w.x, vv[j], part[0][j]) : w.x * vv[j];
                    part[1][j] = g ? fmaf(w.y, vv[j], part[1][j]) : w.y * vv[j];
                    part[2][j] = g ? fmaf(w.z, vv[j], part[2][j]) : w.z * vv[j];
                    part[3][j] = g ? fmaf(w.w, vv[j], part[3][j]) : w.w * vv[j];
                }
            }
            if (tb + kBlock < t1) fetch_values(tb + kBlock, tend);
#pragma unroll
            for (int h = 0; h < 4; h++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[h][j] = fmaf(acc[h][j], corr[h], part[h][j]);
            __syncwarp(); // the weights have been read
        }
        if (has_work) {
#pragma unroll
            for (int h = 0; h < 4; h++) *reinterpret_cast<float4 *>(&s_acc[quarter][h][dim0]) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
            const int h = warp >> 1; // the head this thread hands on below
            m0 = h == 0 ? m[0] : h == 1 ? m[1] : h == 2 ? m[2] : m[3];
            l0 = warp_sum(h == 0 ? l[0] : h == 1 ? l[1] : h == 2 ? l[2] : l[3]);
        }
    }
    } else if (!mma_done) {
        // Of the sixteen scores of a group (four rows x four heads) lane L keeps number L >> 1: row L >> 3, head (L >> 1) & 3.
        // The maximum is that head's, the denominator this lane's own share of it.
        float m = -3.0e38f, l = 0.f, acc[4][8];
#pragma unroll
        for (int h = 0; h < 4; h++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[h][j] = 0.f;
        const int my_row = lane >> 3;
        const int tend = min(t1, fresh);
        for (int tb = has_work ? t0 + warp * kGroup : t1; tb < t1; tb += kAtWarps * kGroup) {
            const bool has_fresh = fresh >= tb && fresh < tb + kGroup && fresh < t1; // warp-uniform
            if (has_fresh) { // the newest row: from shared memory or, now that the wait is over, from the cache
#pragma unroll
                for (int g = 0; g < kGroup; g++) {
                    if (tb + g != fresh) continue;
                    if constexpr (FUSED) {
                        ga.k[g] = Row::pack(s_knew + lane * 8);
                        ga.v[g] = Row::pack(s_vnew + lane * 8);
                    } else {
                        const size_t row = (size_t(fresh) * 4 + kvh) * 256;
                        ga.k[g] = Row::load_raw(kc, row, lane);
                        ga.v[g] = Row::load_raw(vc, row, lane);
                    }
                }
            }
            float s[16];
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float4 qa = *reinterpret_cast<const float4 *>(&s_q[h][lane * 8]), qb = *reinterpret_cast<const float4 *>(&s_q[h][lane * 8 + 4]);
#pragma unroll
                for (int g = 0; g < kGroup; g++) {
                    float kk[8];
                    Row::unpack(ga.k[g], kk);
                    float z = qa.x * kk[0];
                    z = fmaf(qa.y, kk[1], z); z = fmaf(qa.z, kk[2], z); z = fmaf(qa.w, kk[3], z);
                    z = fmaf(qb.x, kk[4], z); z = fmaf(qb.y, kk[5], z); z = fmaf(qb.z, kk[6], z); z = fmaf(qb.w, kk[7], z);
                    s[g * 4 + h] = z;
                }
            }
            const int tn = tb + kAtWarps * kGroup; // the warp's next group
            load_keys<BF16, kGroup>(kc, kvh, tn, tend, lane, ga);
            // sums over the lanes, halving the values a lane carries at every step: 16 shuffles where summing each takes 80
#pragma unroll
            for (int n = 8, mk = 16; n; n >>= 1, mk >>= 1) {
                const bool up = (lane & mk) != 0;
#pragma unroll
                for (int i = 0; i < n; i++) {
                    const float keep = up ? s[i + n] : s[i], send = up ? s[i] : s[i + n];
                    s[i] = keep + __shfl_xor_sync(0xffffffffu, send, mk);
                }
            }
            const float score = (s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1)) * 0.0625f;
            const bool on = tb + my_row < t1;
            float mx = on ? score : -3.0e38f;
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            const float mn = fmaxf(m, mx), corr = __expf(m - mn), pr = on ? __expf(score - mn) : 0.f;
            m = mn;
            l = fmaf(l, corr, pr);
            if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const float c = __shfl_sync(0xffffffffu, corr, 2 * h);
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[h][j] *= c;
                }
            }
#pragma unroll
            for (int g = 0; g < kGroup; g++) {
                float vv[8];
                Row::unpack(ga.v[g], vv);
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const float w = __shfl_sync(0xffffffffu, pr, (g * 4 + h) * 2);
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[h][j] = fmaf(w, vv[j], acc[h][j]);
                }
            }
            load_values<BF16, kGroup>(vc, kvh, tn, tend, lane, ga);
        }
        l += __shfl_xor_sync(0xffffffffu, l, 8);
        l += __shfl_xor_sync(0xffffffffu, l, 16);
        if (lane < 8 && !(lane & 1)) { s_m[warp][lane >> 1] = m; s_l[warp][lane >> 1] = l; }
#pragma unroll
        for (int h = 0; h < 4; h++)
#pragma unroll
            for (int j = 0; j < 8; j += 4)
                *reinterpret_cast<float4 *>(&s_acc[warp][h][lane * 8 + j]) = make_float4(acc[h][j], acc[h][j + 1], acc[h][j + 2], acc[h][j + 3]);
    }
    __syncthreads();
    // ---- add up the CTA's sums, four dims of a head a thread, and hand them to the CTA of the cluster that finishes them ----------------
    const int working = max(0, min(CL, (tokens - t0 + rank * cut.chunk + cut.chunk - 1) / cut.chunk)); // CTAs of the cluster with rows: the first ones
    if (tid == 0) mbar_expect_tx(&s_there, uint32_t(working) * (kMine * 4 + 8));
    if (has_work) {
        const int h = warp >> 1, dim = (tid & 63) * 4, at = h * 256 + dim, owner = at / kMine;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kQuarters && !mma_done) {
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = *reinterpret_cast<const float4 *>(&s_acc[i][h][dim]);
            a = make_float4((x[0].x + x[1].x) + (x[2].x + x[3].x), (x[0].y + x[1].y) + (x[2].y + x[3].y), (x[0].z + x[1].z) + (x[2].z + x[3].z),
                            (x[0].w + x[1].w) + (x[2].w + x[3].w));
        } else {
            m0 = s_m[0][h];
#pragma unroll
            for (int w = 1; w < kAtWarps; w++) m0 = fmaxf(m0, s_m[w][h]);
#pragma unroll
            for (int w = 0; w < kAtWarps; w++) {
                const float e = __expf(s_m[w][h] - m0); // warps without rows carry m = -3e38, l = 0, acc = 0
                const float4 x = *reinterpret_cast<const float4 *>(&s_acc[w][h][dim]);
                l0 = fmaf(s_l[w][h], e, l0);
                a.x = fmaf(x.x, e, a.x); a.y = fmaf(x.y, e, a.y); a.z = fmaf(x.z, e, a.z); a.w = fmaf(x.w, e, a.w);
            }
            if (kMma && s_abort) l0 = kNan; // rows are missing
        }
        const uint32_t bar = map_to_rank(smem_u32(&s_there), owner);
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                     ::"r"(map_to_rank(smem_u32(&s_in[rank][at % kMine]), owner)), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "r"(bar) : "memory");
        if (at % kMine == 0) // the head's maximum and denominator to the owner of these dims
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];"
                         ::"r"(map_to_rank(smem_u32(&s_ml[rank]), owner)), "f"(m0), "f"(l0), "r"(bar) : "memory");
    }
    // the new row goes to the cache while the others' parts come in
    if constexpr (FUSED)
        if (!use_mma && pos >= t0 && pos < t1) {
            const size_t row = (size_t(pos) * 4 + kvh) * 256 + tid;
            Row::store(kc, row, s_knew[tid]);
            Row::store(vc, row, s_vnew[tid]);
        }
    // (s_lost: a wait of the tensor-core loop that ran out does not cut this one short)
    if (!mbar_wait_cluster(&s_there, 0, &s_lost)) { // what has not come counts as NaN, with an error flag or without
#pragma unroll 1
        for (int c = 0; c < CL; c++) {
            if (tid < kMine) s_in[c][tid] = kNan;
            s_ml[c] = make_float2(-3.0e38f, kNan);
        }
    }
    float mg = -3.0e38f, lg = 0.f, a = 0.f;
#pragma unroll
    for (int c = 0; c < CL; c++)
        if (c < working) mg = fmaxf(mg, s_ml[c].x);
#pragma unroll
    for (int c = 0; c < CL; c++)
        if (c < working) {
            const float2 ml = s_ml[c];
            const float e = __expf(ml.x - mg);
            lg = fmaf(ml.y, e, lg);
            if (tid < kMine) a = fmaf(s_in[c][tid], e, a);
        }
    auto leave = [&] {
        const bool lost = *static_cast<volatile int *>(&s_lost) != 0;
        if ((lost || (tid == 0 && s_abort)) && p.error_flag) *p.error_flag = 1;
        // Nobody leaves while a peer may still write into its shared memory.  Ordinarily all of it has come.  After a wait that ran out the peers
        // have sent when they have left or stand here too, and what they sent gets the time of another wait to come in.
        if (p.leave_together || lost) asm volatile("barrier.cluster.arrive.relaxed;\nbarrier.cluster.wait;" ::: "memory");
        if (lost) mbar_wait_cluster(&s_there, 0, &s_lost);
    };
    if (cut.active > 1) { // several clusters: partial results to scratch, the last one folds them in order
        float *part = partials + size_t(kvh * kSplits + cluster * kParts) * kPartFloats;
#pragma unroll
        for (int c = 0; c < kParts; c++, part += kPartFloats) {
            if (tid < kMine) part[8 + rank * kMine + tid] = !HALVES ? a : c < working ? s_in[c][tid] : 0.f;
            if (tid == 0) { // CTAs that share a head write the same values
                part[my_head & 3] = !HALVES ? mg : c < working ? s_ml[c].x : -3.0e38f;
                part[4 + (my_head & 3)] = !HALVES ? lg : c < working ? s_ml[c].y : 0.f;
            }
        }
        __threadfence();
        __syncthreads();
        const int ticket = kvh * CL + rank, shift = (ticket & 3) * 8; // four 8-bit counts per word
        if (tid == 0) {
            const unsigned old = atomicAdd(counters + (ticket >> 2), 1u << shift);
            s_last = int((old >> shift) & 255u) == cut.active - 1;
        }
        __syncthreads();
        if (!s_last) {
            leave();
            return;
        }
        __threadfence();
        const float *pp = partials + size_t(kvh * kSplits) * kPartFloats;
        const int nparts = cut.active * kParts;
        float ms[kMaxClusters];
        mg = -3.0e38f;
#pragma unroll
        for (int c = 0; c < kMaxClusters; c++) {
            ms[c] = c < nparts ? __ldcg(pp + size_t(c) * kPartFloats + (my_head & 3)) : -3.0e38f;
            mg = fmaxf(mg, ms[c]);
        }
        lg = 0.f;
        a = 0.f;
#pragma unroll
        for (int c = 0; c < kMaxClusters; c++)
            if (c < nparts) {
                const float e = __expf(ms[c] - mg);
                lg = fmaf(__ldcg(pp + size_t(c) * kPartFloats + 4 + (my_head & 3)), e, lg);
                if (tid < kMine) a = fmaf(__ldcg(pp + size_t(c) * kPartFloats + 8 + rank * kMine + tid), e, a);
            }
        if (tid == 0) atomicSub(counters + (ticket >> 2), unsigned(cut.active) << shift);
    }
    if (tid < kMine) {
        a *= 1.0f / lg;
        out_base[size_t(my_head) * 256 + my_dim] = a;
        if (p.image) group_digits(a * fast_sigmoid(gv), p.slots, bt, p.image, my_head * 8 + (my_dim >> 5), s_lut, lane);
    }
    leave();
}

template <bool BF16, bool FUSED, int CL, bool HALVES = false> static int launch_clusters(AttnParams p, cudaStream_t st, int along, int rows, int clusters)
{
    size_t smem = 0;
    if constexpr (BF16 && CL == 4 && !HALVES) { // the tensor-core loop's tiles: more than 48 KB of dynamic shared memory is a per-device opt-in
        static std::mutex mu;
        static bool done[64] = {false};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
        if (dev < 0 || dev >= 64) return fail(INSG_E_LIMIT, "attention: device ordinal beyond 63");
        std::lock_guard<std::mutex> lock(mu);
        if (!done[dev]) {
            e = cudaFuncSetAttribute(attn_splitk_kernel<BF16, FUSED, CL, HALVES>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kMmaSmem));
            if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(attention)");
            done[dev] = true;
        }
        if (p.max_context >= kMmaMinTokens) smem = kMmaSmem; // else no launch of these operands gets to the tensor-core loop
    }
    const int most = rows > 0 ? std::min(rows, p.max_context) : p.max_context;
    if (!HALVES) { // as many as some row count up to `most` has at work: clusters without rows cost a launch of two sequences 3 us of 11.  A plain launch's
                   // count is known (1500 rows, called again and again, with three clusters 8.5 us, with a fourth that has no rows 10.7)
        const AttnRule rule = attn_rule(BF16, p.batch != 0, CL);
        const bool known = !FUSED && !p.position;
        const int at_work = std::max(attn_clusters(rule, known ? p.tokens : most, CL), known ? 1 : attn_clusters(rule, std::min(most, rule.some), CL));
        clusters = std::max(1, std::min({clusters, kMaxClusters, at_work}));
    }
    // A launch that started beside this one takes its places as they come free, a cluster of eight at a time.  Where several clusters share a head, those of a
    // cluster's CTAs that arrive last fold and end later than the others: the next launch's clusters then found places for 28 to 31 of 32 and the rest
    // began when the first had ended (8545 rows, called again and again: a call in two took 30 us instead of 20).  Ending as one costs them nothing.
    // Replayed, CTAs ending one by one / as one / launches that start when the one before has ended: 3600 rows 14.6 / 11.9 / 12.6 us, 6000 rows 18.0 / 14.5 /
    // 15.4, 2 x 6000 26.4 / 22.4 / 22.8, 4 x 2047 18.7 / 16.8 / 16.9.  Not where the grid is more than the device holds, whose own later CTAs take the places
    // (eight tokens at 4096 rows 83.7 / 84.9), and not with clusters of four, which find places (three sequences of 4096 rows 24.7 / 24.8).
    if (CL == 8 && p.wait_first && clusters > 1 && 4 * clusters * CL * along <= 2 * sm_count()) p.leave_together = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(4 * clusters * CL, along);
    cfg.blockDim = dim3(kAtThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2; // without pdl the launch starts as early, and waits before it reads
    const cudaError_t e = cudaLaunchKernelEx(&cfg, attn_splitk_kernel<BF16, FUSED, CL, HALVES>, p, clusters);
    return e == cudaSuccess ? INSG_OK : cuda_fail(e, "attention launch");
}

// `along`: tokens of a chunk or sequences of a batch (grid rows); rows: an upper bound of the rows attended, when known.
//
// The tokens of a chunk (the plain form) are cut as single steps are, whatever travels along, so that they have their bits: a
// verify pass must not draw another token than plain decode.  CTAs beyond those that run at once take their turn; clusters without
// rows cost a two-token verify pass on a 2560-row cache 13 us of 1690.
//
// The sequences of a batch share as many clusters as the device runs at once: 33 of eight CTAs at two per SM, or 33 of four at
// one (with the tensor-core loop's tiles).  Where that leaves SMs idle (three sequences or more, not a power of two) and the
// contexts can be long, the fp32 cache goes to clusters of four too.  Where contexts are short and the
// CTAs more than one and a half per SM (seven sequences or more), a second CTA finds no registers beside the products' launches
// before and after: clusters of four find a place sooner than those of eight, and up to 128 rows one of the two has nothing to
// do.  A step of eight sequences 1803 -> 1755 us at 20 rows and 1885 -> 1818 at 450 (alone the launch is 1.5 us slower there);
// five sequences win at 20 rows and lose 12 us from 130 on.  A chunk takes the pairs while one cluster holds its rows.
constexpr int kLongContext = 2048;
static_assert(kLongContext <= kMmaMinTokens, "short contexts never get to the tensor-core loop");
template <bool BF16, bool FUSED> int launch_attn(AttnParams p, cudaStream_t st, bool pdl, int along = 1, int rows = 0)
{
    p.batch = FUSED && along > 1;
    p.wait_first = !pdl;
    const int clusters = FUSED ? kMaxClusters / along : kMaxClusters;
    if (p.max_context < kLongContext) {
        const bool one_cluster = rows > 0 && rows <= attn_rule(BF16, false, 8).one;
        if ((FUSED || one_cluster) && along > kMaxClusters / 2 && 2 * along * 4 * 8 > 3 * sm_count()) return launch_clusters<BF16, FUSED, 4, true>(p, st, along, rows, 2);
        return launch_clusters<BF16, FUSED, 8>(p, st, along, rows, clusters);
    }
    if constexpr (BF16) {
        return launch_clusters<true, FUSED, 4>(p, st, along, rows, clusters);
    } else {
        if (FUSED && along > 2 && (along & (along - 1))) return launch_clusters<false, FUSED, 4>(p, st, along, rows, 17 / along);
        return launch_clusters<false, FUSED, 8>(p, st, along, rows, clusters);
    }
}

// A chunk of consecutive tokens, step one: per token m (one CTA each) the per-head RMSNorm + partial RoPE of the 16 query
// heads (into qn[m][16][256]) and of the 4 key heads, and the token's key and value rows written to the cache at row
// position + offset + m.  Warp tasks 0..15 = query heads, 16..19 = key heads, 20..23 = value heads.  Without qn: the rows alone.
// (reference: split_q_gate + qwen35_qk_norm_rope_gate + store_kv, src/qwen_kernels.cu:15,31 and src/ops.cu:9, once per token)
template <bool BF16> __global__ void __launch_bounds__(kAtThreads) attn_chunk_prepare_kernel(const __grid_constant__ AttnParams p, float *qn)
{
    using Row = KvRow<BF16>;
    const int m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    // What follows a chunk's rows waits before it reads them.  What follows the rows alone may be a step that fetches them ahead of its wait.
    if (qn) pdl_launch_dependents();
    const int pos = __ldcg(p.position) + p.position_offset + m;
    if (pos < 0 || pos >= p.max_context) return; // host checks; never index past the cache
    float rope_c[8], rope_s[8];
    if (lane < 8) rope_table(pos, lane, p.fast_trig != 0, rope_c, rope_s);
    for (int task = qn ? warp : 16 + warp; task < 24; task += kAtWarps) {
        if (task < 20) {
            const bool is_q = task < 16;
            const int h = is_q ? task : task - 16;
            const float *src = is_q ? p.q + size_t(m) * 8192 + size_t(h) * 512 + lane * 8 : p.k_raw + size_t(m) * 1024 + h * 256 + lane * 8;
            const float4 a = __ldcg(reinterpret_cast<const float4 *>(src)), b = __ldcg(reinterpret_cast<const float4 *>(src) + 1);
            float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            norm_rope_256(v, reinterpret_cast<const uint4 *>(is_q ? p.q_w : p.k_w)[lane], lane, pos, rope_c, rope_s);
            if (is_q) {
                float4 *dst = reinterpret_cast<float4 *>(qn + size_t(m) * 4096 + h * 256 + lane * 8);
                dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                dst[1] = make_float4(v[4], v[5], v[6], v[7]);
            } else {
                const size_t row = (size_t(pos) * 4 + h) * 256 + lane * 8;
#pragma unroll
                for (int j = 0; j < 8; j++) Row::store(p.kc, row + j, v[j]);
            }
        } else {
            const int h = task - 20;
            const size_t row = (size_t(pos) * 4 + h) * 256 + lane * 8;
#pragma unroll
            for (int j = 0; j < 8; j++) Row::store(p.vc, row + j, __ldcg(p.v_new + size_t(m) * 1024 + h * 256 + lane * 8 + j));
        }
    }
}

// The optional digit image of the gated output (see insg_attn_op.image).
static void set_image(AttnParams &p, const insg_attn_op *op, int tokens)
{
    p.image = static_cast<uint8_t *>(op->image);
    p.gate = op->qraw;
    p.gate_elementwise = op->gate_elementwise;
    p.slots = op->image ? image_slots(tokens) : 0;
}

size_t attn_scratch_bytes() { return 64 + size_t(4) * kSplits * kPartFloats * sizeof(float); }

int attn_tile_launch(const AttnParams &p, const float *qn, int tokens, bool bf16, cudaStream_t st, bool pdl);
constexpr int kTileFromTokens = 32;

int attn_plain_launch(const float *q, const void *kc, const void *vc, float *out, int tokens, int kv_dtype, void *scratch,
                      cudaStream_t st)
{
    AttnParams p = {};
    p.q = q; p.kc = const_cast<void *>(kc); p.vc = const_cast<void *>(vc); p.out = out;
    p.tokens = tokens; p.max_context = tokens;
    p.counters = static_cast<unsigned *>(scratch);
    p.partials = reinterpret_cast<float *>(static_cast<uint8_t *>(scratch) + 64);
    return kv_dtype == INSG_KV_BF16 ? launch_attn<true, false>(p, st, false) : launch_attn<false, false>(p, st, false);
}

// ---- allocation-free variant -----------------------------------------------------
// Scratch for insg_gqa_decode_noalloc: lives in the library image, one copy per GPU that loads it
// (about 600 KB, held until the process exits).  In host code the symbol name is only a handle, so
// the device address is looked up once per device with cudaGetSymbolAddress and handed to the kernel.
constexpr int kNoAllocMaxTokens = 262144; // the model's longest context
constexpr size_t kNoAllocScratchBytes = 64 + size_t(4) * kSplits * kPartFloats * sizeof(float);
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of the static scratch on the current device.  Looked up on every call: the lookup allocates nothing,
// and an address cached across calls would dangle after the application resets the device or its primary context.
static int noalloc_scratch(void **out)
{
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(static attention scratch)");
    *out = p;
    return INSG_OK;
}

} // namespace insg

using namespace insg;

extern "C" {

int insg_gqa_decode_noalloc(const float *q, const void *k_cache, const void *v_cache, float *out, int tokens, int kv_dtype,
                            insg_stream_t stream)
{
    if (tokens <= 0) return INSG_OK;
    if (tokens > kNoAllocMaxTokens) return fail(INSG_E_LIMIT, "gqa_decode_noalloc: more than 262144 cached tokens");
    if (!q || !k_cache || !v_cache || !out) return fail(INSG_E_ARG, "gqa_decode_noalloc: null pointer");
    if (kv_dtype != INSG_KV_F32 && kv_dtype != INSG_KV_BF16) return fail(INSG_E_ARG, "gqa_decode_noalloc: bad kv dtype");
    void *scratch = nullptr;
    const int rc = noalloc_scratch(&scratch);
    if (rc != INSG_OK) return rc;
    // the per-kv-head arrival counters must start at zero; an earlier call that was cut short could have left them set
    cudaError_t e = cudaMemsetAsync(scratch, 0, 64, stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(static attention scratch)");
    return attn_plain_launch(q, k_cache, v_cache, out, tokens, kv_dtype, scratch, stream);
}

size_t insg_gqa_scratch_bytes(int tokens)
{
    (void)tokens; // the split count is fixed, so the scratch does not grow with the context
    return attn_scratch_bytes();
}

int insg_gqa_decode(const float *q, const void *k_cache, const void *v_cache, float *out, int tokens, int kv_dtype,
                    void *scratch, size_t scratch_bytes, insg_stream_t stream)
{
    if (tokens <= 0) return INSG_OK; // src/attention.cu:5 returns silently
    if (!q || !k_cache || !v_cache || !out || !scratch) return fail(INSG_E_ARG, "gqa_decode: null pointer");
    if (kv_dtype != INSG_KV_F32 && kv_dtype != INSG_KV_BF16) return fail(INSG_E_ARG, "gqa_decode: bad kv dtype");
    if (scratch_bytes < attn_scratch_bytes()) return fail(INSG_E_SHAPE, "gqa_decode: scratch too small");
    return attn_plain_launch(q, k_cache, v_cache, out, tokens, kv_dtype, scratch, stream);
}

int insg_attention_rows(const insg_attn_op *op, int tokens, insg_stream_t stream)
{
    if (!op || !op->k_raw || !op->v || !op->k_norm_w || !op->k_cache || !op->v_cache || !op->position) return fail(INSG_E_ARG, "attention_rows: null pointer");
    if (tokens < 1 || tokens > 65535 || op->max_context <= 0) return fail(INSG_E_SHAPE, "attention_rows: 1 <= tokens <= 65535, max_context > 0");
    AttnParams p = {};
    p.k_raw = op->k_raw; p.v_new = op->v; p.k_w = op->k_norm_w; p.kc = op->k_cache; p.vc = op->v_cache;
    p.position = op->position; p.position_offset = op->position_offset; p.max_context = op->max_context; p.fast_trig = op->fast_trig;
    auto kernel = op->kv_dtype == INSG_KV_BF16 ? attn_chunk_prepare_kernel<true> : attn_chunk_prepare_kernel<false>;
    return launch(kernel, dim3(tokens), dim3(kAtThreads), 0, stream, true, p, static_cast<float *>(nullptr));
}

int insg_attention_chunk(const insg_attn_op *op, int tokens, float *q_scratch, int rows_hint, insg_stream_t stream)
{
    if (!op || !op->qraw || !op->k_raw || !op->v || !op->q_norm_w || !op->k_norm_w || !op->k_cache || !op->v_cache ||
        !op->out || !op->position || !op->scratch || !q_scratch)
        return fail(INSG_E_ARG, "attention_chunk: null pointer");
    if (tokens < 1 || tokens > 65535) return fail(INSG_E_SHAPE, "attention_chunk: 1 <= tokens <= 65535");
    if (tokens <= kTileFromTokens && op->scratch_bytes < size_t(tokens) * attn_scratch_bytes()) return fail(INSG_E_SHAPE, "attention_chunk: scratch too small");
    if (op->max_context <= 0) return fail(INSG_E_SHAPE, "attention_chunk: max_context");
    if (op->image && tokens > 8) return fail(INSG_E_SHAPE, "attention_chunk: a digit image holds up to 8 tokens");
    AttnParams p = {};
    p.q = op->qraw; p.k_raw = op->k_raw; p.v_new = op->v; p.q_w = op->q_norm_w; p.k_w = op->k_norm_w;
    p.kc = op->k_cache; p.vc = op->v_cache; p.out = op->out;
    p.position = op->position; p.position_offset = op->position_offset;
    p.max_context = op->max_context; p.fast_trig = op->fast_trig; p.error_flag = op->error_flag;
    const bool bf16 = op->kv_dtype == INSG_KV_BF16;
    int rc = bf16 ? launch(attn_chunk_prepare_kernel<true>, dim3(tokens), dim3(kAtThreads), 0, stream, true, p, q_scratch)
                  : launch(attn_chunk_prepare_kernel<false>, dim3(tokens), dim3(kAtThreads), 0, stream, true, p, q_scratch);
    if (rc != INSG_OK) return rc;
    // More than 32 tokens: query tiles on the tensor cores.  Fewer: the token-by-token form below, whose results are those of
    // single steps bit for bit (at 33 tokens the tile kernel still has only twelve CTAs; the two take the same time near 24).
    if (tokens > kTileFromTokens) return attn_tile_launch(p, q_scratch, tokens, bf16, stream, false);
    set_image(p, op, tokens);
    // step two: every (kv head, split, token) CTA is the plain split-K decode of its token over the rows up to its own
    p.q = q_scratch; p.q_stride = 4096; p.out_stride = 4096; p.scratch_stride = attn_scratch_bytes();
    p.counters = static_cast<unsigned *>(op->scratch);
    p.partials = reinterpret_cast<float *>(static_cast<uint8_t *>(op->scratch) + 64);
    return bf16 ? launch_attn<true, false>(p, stream, false, tokens, rows_hint) : launch_attn<false, false>(p, stream, false, tokens, rows_hint);
}

int insg_attention_batch(const insg_attn_op *op, int sequences, size_t cache_stride_bytes, insg_stream_t stream)
{
    if (!op || !op->qraw || !op->k_raw || !op->v || !op->q_norm_w || !op->k_norm_w || !op->k_cache || !op->v_cache ||
        !op->out || !op->position || !op->scratch)
        return fail(INSG_E_ARG, "attention_batch: null pointer");
    if (sequences < 1 || sequences > 65535) return fail(INSG_E_SHAPE, "attention_batch: 1 <= sequences <= 65535");
    if (op->scratch_bytes < size_t(sequences) * attn_scratch_bytes()) return fail(INSG_E_SHAPE, "attention_batch: scratch too small");
    if (op->max_context <= 0) return fail(INSG_E_SHAPE, "attention_batch: max_context");
    if (sequences > 1 && (cache_stride_bytes == 0 || (cache_stride_bytes & 15))) return fail(INSG_E_ARG, "attention_batch: cache stride must be a positive multiple of 16 bytes");
    AttnParams p = {};
    p.q = op->qraw; p.k_raw = op->k_raw; p.v_new = op->v; p.q_w = op->q_norm_w; p.k_w = op->k_norm_w;
    p.kc = op->k_cache; p.vc = op->v_cache; p.out = op->out;
    p.position = op->position; p.position_offset = op->position_offset;
    p.max_context = op->max_context; p.fast_trig = op->fast_trig; p.error_flag = op->error_flag;
    p.counters = static_cast<unsigned *>(op->scratch);
    p.partials = reinterpret_cast<float *>(static_cast<uint8_t *>(op->scratch) + 64);
    p.q_stride = 8192; p.out_stride = 4096; p.kvin_stride = 1024; p.scratch_stride = attn_scratch_bytes(); p.cache_stride = cache_stride_bytes;
    if (op->image && sequences > 8) return fail(INSG_E_SHAPE, "attention_batch: a digit image holds up to 8 sequences");
    set_image(p, op, sequences);
    const bool pdl = op->pdl != 0;
    return op->kv_dtype == INSG_KV_BF16 ? launch_attn<true, true>(p, stream, pdl, sequences) : launch_attn<false, true>(p, stream, pdl, sequences);
}

int insg_attention_step(const insg_attn_op *op, insg_stream_t stream)
{
    if (!op || !op->qraw || !op->k_raw || !op->v || !op->q_norm_w || !op->k_norm_w || !op->k_cache || !op->v_cache ||
        !op->out || !op->position || !op->scratch)
        return fail(INSG_E_ARG, "attention_step: null pointer");
    if (op->scratch_bytes < attn_scratch_bytes()) return fail(INSG_E_SHAPE, "attention_step: scratch too small");
    if (op->max_context <= 0) return fail(INSG_E_SHAPE, "attention_step: max_context");
    AttnParams p = {};
    p.q = op->qraw; p.k_raw = op->k_raw; p.v_new = op->v; p.q_w = op->q_norm_w; p.k_w = op->k_norm_w;
    p.kc = op->k_cache; p.vc = op->v_cache; p.out = op->out;
    p.position = op->position; p.position_offset = op->position_offset;
    p.max_context = op->max_context; p.fast_trig = op->fast_trig; p.error_flag = op->error_flag;
    p.counters = static_cast<unsigned *>(op->scratch);
    p.partials = reinterpret_cast<float *>(static_cast<uint8_t *>(op->scratch) + 64);
    set_image(p, op, 1);
    const bool pdl = op->pdl != 0;
    return op->kv_dtype == INSG_KV_BF16 ? launch_attn<true, true>(p, stream, pdl) : launch_attn<false, true>(p, stream, pdl);
}

} // extern "C"

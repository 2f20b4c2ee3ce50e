// MXFP4 weights x one to eight tokens on the 5th-generation tensor cores (tcgen05, sm_100a): the decode-step matrix product.
//
// y[m][r] = sum_k e2m1(code(r,k)) * 2^(s(r,k/32)-127) * x[m][k]                 (reference: src/mxfp4.cu:41-66)
//
// What bounds it: the weight stream (17 bytes per 32 weights, each read once), and, because a token is a chain of some
// 160 of these products, everything between two streams.  The kernel is built so that neither costs instruction slots:
//   * weights go HBM -> shared memory by cp.async.bulk (17 KB per copy: 8.7 KB copies stream at 4.7 TB/s from one issuing
//     thread, 17 KB ones at 6.3) and from there straight into tcgen05.mma.kind::mxf4.block_scale as the A operand, in
//     their packed form; nothing is dequantised in registers;
//   * the activation is the B operand.  kind::mxf4 wants E2M1 there too, so each fp32 value is written as a 25-bit signed
//     fixed-point number relative to the largest of its 32-element group (the group's UE8M0 scale) in balanced base 9:
//     eight digits -4..4, each exact in E2M1.  Column j of a token holds digit j; the epilogue adds 9^j D_j in fp32;
//   * a cluster of four CTAs shares a 128-row tile, each multiplying a quarter of K: a CTA converts only a quarter of the
//     activation, 4096 rows still occupy 128 SMs, and the four partial sums meet through distributed shared memory
//     (st.async with mbarrier completion), added in rank order by the CTA that owns those 32 rows -- no ticket, no
//     global-memory exchange, and the same bits whatever the timing;
//   * a CTA keeps its ring within half an SM's shared memory, so the next launch of the chain (programmatic dependent
//     launch) is resident and has its first ~100 KB of weights per SM on the way while this one finishes.
//
// CTA roles (320 threads): warps 0-7 run the activation prologue (fused RMSNorm / gates, digits); then warps 0-3 read the
// accumulators (tcgen05.ld, tensor-memory lane = row) and send the partial sums to the rows' owners, warps 4-7 add the
// four parts and run the fused epilogue; warp 8 issues tcgen05.cp / tcgen05.mma, warp 9 the bulk copies
// (for packed records four more warps copy cells in its place).  In a launch with a DeltaNet step warps 0-7 make it at the end.  Every wait is
// bounded: on expiry a flag is raised in global memory and all roles drain.
//
// Layout of the weights (insg_mxfp4_repack_umma): rows in tiles of 128, K in blocks of 128; one (tile, block) record is 8704
// contiguous bytes = the shared-memory image the MMA reads: 2 K-steps of 64 x [16 row groups][2 k cores][8 rows][16 bytes]
// (canonical K-major, no swizzle: leading byte offset 128, stride byte offset 256), then the 512-byte scale block
// [32 rows][4 row quarters][4 groups] that tcgen05.cp.32x128b.warpx4 expects.
#include "gemv_prologue.cuh"
#include "umma_common.cuh"
#include "host_util.h"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace insg {

constexpr int kDCl = 4;                    // CTAs per cluster = parts K is cut into = 32-row blocks of a tile
constexpr int kDThreads = 320;
constexpr int kDLoaders = 4;               // warps that fetch packed records (kDRecords), two row tiles each
constexpr int kDStage = 2 * kURec;         // one ring stage: two consecutive k-blocks of a tile
constexpr int kDMaxStages = 8;
constexpr int kDMaxKb = 24;                // k-blocks per CTA: 12288 / 128 / 4
constexpr int kDDigits = 8;                // digits per activation = N columns per token
constexpr uint32_t kDSfaCol = 128, kDSfbCol = 160, kDTmemCols = 256; // accumulators [0,128), weight scales [128,160), digit scales [160,256)
// A CTA takes at most this much dynamic shared memory unless its operands need more: two of them (this launch and the next)
// then fit an SM's 228 KB with their static part (at most 1 KB, which is why eight tokens' sums of squares are not in it) and
// the 1 KB the hardware keeps per CTA.
constexpr int kDHalfSm = 112 * 1024;
// The next launch may start when at most this many ring stages of a CTA are still to be requested, and asks L2 for a few beyond its
// own ring.  Its requests share the SM's copy engine and the memory with this launch's: made while this launch still streams they delay
// the stages it waits for, made at the very end its ring cannot fill in time.  Microseconds a step by (stages left, stages asked of L2), with weights
// that leave L2 first (where they stay, asking for more than three or, from three tokens on, any gains nothing):
//   one token (4, 3) 969, (6, 2) 973, (6, 3) 959, (6, 4) 965, (6, 10) 968, (8, 3) 1025; a speculative pass (5, 4) 1306, (5, 5) 1302,
//   (5, 6) 1301, (6, 3) 1311, (7, 3) 1331, two sequences 1063, 1063, 1070, 1065, -
//   three sequences (3, 6) 1100, (4, 0) 1096, (4, 3) 1074, (4, 6) 1063, (4, 8) 1085, (5, 6) 1074, (6, 0) 1113
//   eight sequences (2, 6) 1250, (2, 8) 1287, (3, 4) 1254, (3, 6) 1246, (3, 10) 1268, (4, 0) 1265, (4, 6) 1250, (6, 3) 1291
// All threads execute the trigger where the CTA sets out: left to the producer warp, with the L2 code in every variant, a launch that stands
// alone took 0.1-0.3 us more (4096 x 4096, one, two, eight tokens 6.85, 8.11, 12.25 us; like this 6.78, 7.98, 12.10).
template <int T> constexpr int kDTriggerStages = T == 1 ? 6 : T == 2 ? 5 : T == 4 ? 4 : 3;
template <int T> constexpr int kDAheadStages = T == 1 ? 3 : T == 2 ? 5 : 6;

struct DSeg {
    const uint8_t *packed, *packed2;
    float *out;
    float *conv_state;
    const uint16_t *conv_w;
    const float *A_log;
    const uint16_t *dt_bias;
    long long conv_stride; // 0: the tokens are one sequence (history carried through them in order), else token m's history at + m * stride
    uint8_t *prep;         // optional: digit image of the output (times prep_w) for a later launch with a prepared input
    const uint16_t *prep_w;
    float *prep_partials;  // with it, [token][rows / 32] sums of squares of the output
    int tile_begin, epilogue, rows;
};

// The DeltaNet step a launch makes beside the product its output is gated with (kDDelta).
struct DDelta {
    float *state;
    const float *q, *k, *v, *g, *beta;
    float *out;
    const uint16_t *norm_w;
    uint8_t *image;
};

struct DParams {
    const float *in, *aux;
    const uint16_t *norm_w;
    float *x_out;
    const float *prep_partials; // prepared input: the producer's sums of squares, or null
    int cols, nkb, prologue, nseg, units, nmat, tokens, stages;
    int ahead; // stages beyond the ring to ask L2 for
    int wait_first; // nothing may be read before the launch before this one has ended
    int late;  // the next launch reads what was there before this one: it may start when this launch's own wait is over
    DDelta delta;
    DSeg seg[4];
    float2 *argmax_partial;
    unsigned *argmax_ticket;
    int *token_out, *token_feedback, *token_log, *position_inout, *host_result;
    int *error_flag;
    int token_log_capacity;
};

// ---- cluster helpers -----------------------------------------------------------------------------------------------------
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// The closing barrier only keeps CTAs from leaving early.  A release there would wait until the epilogue's global stores have been
// acknowledged, which a stream of weights makes slow (one token 1214 -> 1189 us, lm_head with four tokens 145 -> 87 us).
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
// T floats to another CTA's shared memory; their bytes complete on that CTA's barrier.
template <int T> __device__ __forceinline__ void send_floats(uint32_t dst, const float (&v)[T], uint32_t bar)
{
    if constexpr (T == 1) {
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(dst), "f"(v[0]), "r"(bar) : "memory");
    } else if constexpr (T == 2) {
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(dst), "f"(v[0]), "f"(v[1]), "r"(bar) : "memory");
    } else {
#pragma unroll
        for (int t = 0; t < T; t += 4)
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                         ::"r"(dst + 4 * t), "f"(v[t]), "f"(v[t + 1]), "f"(v[t + 2]), "f"(v[t + 3]), "r"(bar) : "memory");
    }
}
__device__ __forceinline__ int dseg_of(const DParams &p, int unit)
{
    int s = 0;
#pragma unroll
    for (int i = 1; i < 4; i++)
        if (i < p.nseg && unit >= p.seg[i].tile_begin) s = i;
    return s;
}

// One output row per lane into the digit image a later launch takes as its prepared input (the layout of store_digits): the
// warp's 32 rows are one 32-element group of that launch's K.  Costs the producer some 50 instructions per token; converting
// in the consumer would be done by every cluster again (eight tokens: 6 us per launch at 4096 columns, 17 at 12288).
template <int T> __device__ __forceinline__ void leave_digits(const DSeg &s, float v, float w, int row, int m, const uint8_t *lut, int lane)
{
    const int grp = row >> 5;
    group_digits(v * w, T, m, s.prep, grp, lut, lane);
    if (s.prep_partials) {
        const float ss = warp_sum(v * v);
        if (lane == 0) s.prep_partials[m * (s.rows >> 5) + grp] = ss;
    }
}

// One accumulator: the eight digit columns of each token, digits combined.
template <int T> __device__ __forceinline__ void load_partial(uint32_t taddr, float (&y)[T])
{
    uint32_t d[8 * T];
    if constexpr (T == 1) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]) : "r"(taddr));
    } else {
#pragma unroll
        for (int h = 0; h < T / 2; h++)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                         : "=r"(d[16 * h]), "=r"(d[16 * h + 1]), "=r"(d[16 * h + 2]), "=r"(d[16 * h + 3]), "=r"(d[16 * h + 4]), "=r"(d[16 * h + 5]),
                           "=r"(d[16 * h + 6]), "=r"(d[16 * h + 7]), "=r"(d[16 * h + 8]), "=r"(d[16 * h + 9]), "=r"(d[16 * h + 10]), "=r"(d[16 * h + 11]),
                           "=r"(d[16 * h + 12]), "=r"(d[16 * h + 13]), "=r"(d[16 * h + 14]), "=r"(d[16 * h + 15])
                         : "r"(taddr + 16 * h));
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int t = 0; t < T; t++) y[t] = combine_digits(d + 8 * t);
}

// Units whose exchange slots exist at once.  Eight tokens: two matrices leave room for one unit's if the launch is to stay within
// half an SM (24576 x 4096 as SwiGLU 14.3 -> 13.3 us in the chain); one matrix keeps two (one: 9.7 -> 10.7 us at 12352 x 4096).
template <int T> __host__ __device__ constexpr int unit_slots(int nmat) { return T == 1 ? 4 : T == 8 ? 3 - nmat : 2; }

// What a variant of the kernel has beside its tokens: a prepared input in place of the prologue; the logits' arg-max; two matrices (SwiGLU); one
// segment that adds into the residual stream, one unit per cluster (kDResidual; with digits that come with the weights kDStreamed, behind the
// gated norm kDGated); epilogues that add nothing and leave nothing prepared (kDPlain); a DeltaNet step beside the product that gates its output
// (kDDelta); weights that come as the packed records of insg_mxfp4_repack (kDRecords).  A launch that fits none takes the general ones.
// A token is 152 of these launches, five to six microseconds each (129 when these figures were taken, the gates' products in the in-projections), and instructions that a launch runs through for the first time come from L2 behind the
// stream of weights.  Microseconds of a device-fed token (a host-fed decode_token gained half of it), a step of three sequences, of eight, and a
// speculative pass (a process is now and then 2 % off for all of its life), and the code of a launch (the last line: of the special variants; what
// takes a general one runs up to 82 KB):
//   one kernel with everything in it                                                  1084 1308 1503 1500   96-125 KB
//   variants prepared and arg-max, the waits' loops not unrolled, one store and one
//   copy of the digits' code behind all epilogues                                     1057 1208 1412 1428   41-66
//   and two matrices, the gated norm, residual                                        1057 1170 1348 1387   28-48
//   and plain; no later runs, last odd block or slot reuse where there are none       1031 1156 1330 1365   20-37
// (20 KB more in the issuer's loop, never run, cost a token 80 us.)
constexpr int kDPrepared = 1, kDLogits = 2, kDStreamed = 4, kDGated = 8, kDTwo = 16, kDResidual = 32, kDPlain = 64, kDDelta = 128, kDRecords = 256;
constexpr int kRec = 1088;                 // a packed record: 16 rows x 128 k (insg_mxfp4_repack)
constexpr int kDLoadAhead = 5;             // stages a loading thread has on their way; fewer than the ring has, or all there are (4 to 6 the same, 7 a third slower)

__device__ __forceinline__ void copy16(void *dst, const void *src) // to shared memory, past L1
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// One DeltaNet step of 32 columns of a head by the first eight warps of a CTA, whose cluster has the head: the arithmetic, and the order of every
// sum, of deltanet_step_kernel and of the gated prologue, so that their bits are the same.  cell: rows kr + 32 j of the state, four columns.
// The step waits for the in-projection, a chain of latencies that leaves the memory and the tensor cores idle, and its gate z is not wanted before
// its end: z's rows of the in-projection (a tile a head, so that a cluster's four CTAs have their columns' gates at hand) are multiplied here,
// from the input that the launch before the in-projection left.  The in-projection then has two units a cluster and not three, and the out
// projection takes digits and not the gated norm: a device-fed token 1010 -> 994 us.
// One token only: eight warps have one state's 32 columns in registers.  Several sequences have several states, and a verify pass leaves two; their products
// keep z in the in-projection, and their step (from three sequences on with the digits) is a launch of its own in deltanet.cu.  The gated norm ahead of an out
// projection (kDGated) is left to them (one and two sequences, verify passes) and, with one token, to the first block, whose input does not come prepared.
struct DeltaShared {
    float qk[8][2][128]; // per warp: its own copy of the normalised q and k
    float part[2][8][32];
    float squares[32];   // of the head's output, four columns each
    float z[32];         // what gates this CTA's columns
};
__device__ __forceinline__ void delta_step(const DDelta &d, float4 (&cell)[4], DeltaShared &sh, int head, int slice, uint64_t *bar, volatile int *abort_flag, const uint8_t *lut,
                                           int tid)
{
    const int lane = tid & 31, warp = tid >> 5, kh = head >> 1, vq = tid & 7, kr = tid >> 3, v0 = slice * 32 + vq * 4;
    const float gw = warp == 0 ? bf16_bits_to_float(d.norm_w[slice * 32 + lane]) : 0.f;
    pdl_wait();
    const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(d.q + kh * 128) + lane);
    const float4 k4 = __ldcg(reinterpret_cast<const float4 *>(d.k + kh * 128) + lane);
    const float4 v4 = __ldcg(reinterpret_cast<const float4 *>(d.v + head * 128 + slice * 32) + vq);
    const float g_in = __ldcg(d.g + head), beta = __ldcg(d.beta + head);
    const float qn = warp_sum(fmaf(q4.x, q4.x, fmaf(q4.y, q4.y, fmaf(q4.z, q4.z, q4.w * q4.w))));
    const float kn = warp_sum(fmaf(k4.x, k4.x, fmaf(k4.y, k4.y, fmaf(k4.z, k4.z, k4.w * k4.w))));
    const float qs = rsqrtf(qn + 1e-6f) * 0.08838834764831845f, ks = rsqrtf(kn + 1e-6f);
    reinterpret_cast<float4 *>(sh.qk[warp][0])[lane] = make_float4(q4.x * qs, q4.y * qs, q4.z * qs, q4.w * qs);
    reinterpret_cast<float4 *>(sh.qk[warp][1])[lane] = make_float4(k4.x * ks, k4.y * ks, k4.z * ks, k4.w * ks);
    __syncwarp();
    float qq[4], kk[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        qq[j] = sh.qk[warp][0][kr + 32 * j];
        kk[j] = sh.qk[warp][1][kr + 32 * j];
    }
    const float decay = expf(g_in);
    float4 pm = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        pm.x = fmaf(cell[j].x, kk[j], pm.x);
        pm.y = fmaf(cell[j].y, kk[j], pm.y);
        pm.z = fmaf(cell[j].z, kk[j], pm.z);
        pm.w = fmaf(cell[j].w, kk[j], pm.w);
    }
#pragma unroll
    for (int m = 16; m >= 8; m >>= 1) {
        pm.x += __shfl_xor_sync(0xffffffffu, pm.x, m);
        pm.y += __shfl_xor_sync(0xffffffffu, pm.y, m);
        pm.z += __shfl_xor_sync(0xffffffffu, pm.z, m);
        pm.w += __shfl_xor_sync(0xffffffffu, pm.w, m);
    }
    if (lane < 8) *reinterpret_cast<float4 *>(&sh.part[0][warp][lane * 4]) = pm;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    float4 t[8];
#pragma unroll
    for (int w = 0; w < 8; w++) t[w] = *reinterpret_cast<const float4 *>(&sh.part[0][w][vq * 4]);
#pragma unroll
    for (int n = 1; n < 8; n <<= 1) // pairs of warps, then of pairs
#pragma unroll
        for (int w = 0; w < 8; w += 2 * n) { t[w].x += t[w + n].x; t[w].y += t[w + n].y; t[w].z += t[w + n].z; t[w].w += t[w + n].w; }
    const float4 dl = make_float4(fmaf(-t[0].x, decay, v4.x) * beta, fmaf(-t[0].y, decay, v4.y) * beta, fmaf(-t[0].z, decay, v4.z) * beta,
                                  fmaf(-t[0].w, decay, v4.w) * beta);
    float *S = d.state + size_t(head) * 128 * 128;
    float4 po = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        cell[j].x = fmaf(kk[j], dl.x, cell[j].x * decay);
        cell[j].y = fmaf(kk[j], dl.y, cell[j].y * decay);
        cell[j].z = fmaf(kk[j], dl.z, cell[j].z * decay);
        cell[j].w = fmaf(kk[j], dl.w, cell[j].w * decay);
        po.x = fmaf(cell[j].x, qq[j], po.x);
        po.y = fmaf(cell[j].y, qq[j], po.y);
        po.z = fmaf(cell[j].z, qq[j], po.z);
        po.w = fmaf(cell[j].w, qq[j], po.w);
        *reinterpret_cast<float4 *>(S + size_t(kr + 32 * j) * 128 + v0) = cell[j];
    }
#pragma unroll
    for (int m = 16; m >= 8; m >>= 1) {
        po.x += __shfl_xor_sync(0xffffffffu, po.x, m);
        po.y += __shfl_xor_sync(0xffffffffu, po.y, m);
        po.z += __shfl_xor_sync(0xffffffffu, po.z, m);
        po.w += __shfl_xor_sync(0xffffffffu, po.w, m);
    }
    if (lane < 8) *reinterpret_cast<float4 *>(&sh.part[1][warp][lane * 4]) = po;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (warp != 0) return;
    float w8[8];
#pragma unroll
    for (int w = 0; w < 8; w++) w8[w] = sh.part[1][w][lane];
    const float o = ((w8[0] + w8[1]) + (w8[2] + w8[3])) + ((w8[4] + w8[5]) + (w8[6] + w8[7]));
    // The head's sum of squares: four columns a term, the terms of the four slices exchanged, then the sum over the 32 lanes that the prologue takes.
    float ss[1];
    {
        const float x = __shfl_sync(0xffffffffu, o, (lane & 7) * 4), y = __shfl_sync(0xffffffffu, o, (lane & 7) * 4 + 1);
        const float u = __shfl_sync(0xffffffffu, o, (lane & 7) * 4 + 2), v = __shfl_sync(0xffffffffu, o, (lane & 7) * 4 + 3);
        ss[0] = fmaf(x, x, fmaf(y, y, fmaf(u, u, v * v)));
    }
    send_floats<1>(map_to_rank(smem_u32(&sh.squares[slice * 8 + (lane & 7)]), uint32_t(lane >> 3)), ss, map_to_rank(smem_u32(bar), uint32_t(lane >> 3)));
    d.out[head * 128 + slice * 32 + lane] = o;
    __all_sync(0xffffffffu, mbar_wait_cluster(bar, 0, abort_flag));
    const float inv = rsqrtf(warp_sum(sh.squares[lane]) / 128.f + 1e-6f);
    group_digits(o * inv * gw * fast_silu(sh.z[lane]), 1, 0, d.image, head * 4 + slice, lut, lane);
}

// Plain products on packed records take any activation and any scale byte, as on mma.sync.  Digits alone do not: below 2^-103 a group's largest element has
// fewer than 24 bits, and with scale bytes below 24 the digit columns are subnormal in tensor memory.  So the digits are those of 2^64 x (kDLift), and
// the sums are taken back by 2^-64: the same bits, and zeros stay exact.  What leaves the range at its other end (elements from 2^64 on, sums that overflow),
// the scale byte 255 (infinity, in digits NaN) and sums of groups with the scale byte 0 (nothing, in digits 2^-127: at most 2^-110 of the token's largest
// element, 12288 of them) are told by a sum that is not finite or below kDFewBits of that element, and its row is added up once more in fp32, each group's
// factor, weights' and token's, applied to its finished sum.  A warp takes four rows of its 32 (in `mask`) at a time, a lane a group of 32 columns; 32 rows of
// 4096 columns take it 80 us.  Ordinary products: 4096 x 4096 with one to four tokens, replayed, 4.9, 5.5, 6.5, 6.6 us without all this, 4.6, 5.2, 6.2, 6.3 like this.
constexpr float kDLift = 18446744073709551616.f;        // 2^64
constexpr float kDFewBits = 5.16987882845642297e-26f;   // 2^-84
__device__ __noinline__ float rows_again(const uint8_t *packed, const float *x, int nkb, int row0, uint32_t mask, uint32_t top, float y, int lane)
{
    const int eb = min(max(int(top >> 23), 1), 253);
    const float alpha = __uint_as_float(uint32_t(254 - eb) << 23); // the largest element to [1, 4), a subnormal one to 2^-23 at least
#pragma unroll 1
    while (mask) {
        int r[4];
        const uint8_t *cells[4];
        float acc[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            r[i] = mask ? __ffs(mask) - 1 : r[0];
            mask &= mask - 1u;
            const int row = row0 + r[i];
            cells[i] = packed + size_t(row >> 4) * nkb * kRec;
            acc[i] = 0.f;
        }
#pragma unroll 1
        for (int g = lane; g < nkb * 4; g += 32) {
            const size_t rec = size_t(g >> 2) * kRec;
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
            for (int j = 0; j < 4; j++) { // eight columns
                const float4 a = __ldcg(reinterpret_cast<const float4 *>(x + g * 32 + j * 8)), b = __ldcg(reinterpret_cast<const float4 *>(x + g * 32 + j * 8 + 4));
                const float v[8] = {a.x * alpha, a.y * alpha, a.z * alpha, a.w * alpha, b.x * alpha, b.y * alpha, b.z * alpha, b.w * alpha};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t q = *reinterpret_cast<const uint32_t *>(cells[i] + rec + ((row0 + r[i]) & 15) * 64 + (g & 3) * 16 + j * 4);
#pragma unroll
                    for (int k = 0; k < 8; k++) part[i] = fmaf(e2m1_to_float(q >> (4 * k)), v[k], part[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int tile_row = (row0 + r[i]) & 15, sc = cells[i][rec + 1024 + (tile_row & 7) * 8 + (g & 3) * 2 + (tile_row >> 3)];
                if (sc) acc[i] += sc == 255 ? part[i] * __int_as_float(0x7f800000) : ldexpf(part[i], sc + eb - 254);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float sum = warp_sum(acc[i]);
            if (lane == r[i]) y = sum;
        }
    }
    return y;
}

template <int T, int F>
__global__ void __cluster_dims__(kDCl, 1, 1) __launch_bounds__(kDThreads + ((F & kDRecords) != 0 ? 32 * kDLoaders : 0), (F & kDRecords) != 0 ? 1 : 2) umma_gemv_kernel(const __grid_constant__ DParams p)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int kBKb = 512 * T;       // digit bytes per k-block
    constexpr int kImg = kBKb + 512;    // a k-block of the image: digits, then their scale block
    constexpr bool prepared = (F & kDPrepared) != 0, logits = (F & kDLogits) != 0, streamed = (F & kDStreamed) != 0;
    constexpr bool records = (F & kDRecords) != 0; // the weights come as packed records; a plain vector, one segment that is stored
    const int pro = (F & kDGated) != 0 ? int(INSG_PRO_GATED_RMSNORM) : records ? int(INSG_PRO_PLAIN) : p.prologue;
    constexpr int kStage = kDStage + (streamed ? 2 * kImg : 0) + (records ? 1024 : 0); // streamed: one unit a cluster, so that its digits come with the weights they multiply
    static_assert(!streamed || prepared, "a streamed image is a prepared one");
    constexpr int N = kDDigits * T;
    constexpr int kSlot = kDCl * 32 * T; // floats of one exchange slot: [source rank][32 rows][T]
    // The four owner warps: with several tokens they split the tokens of a unit among them (TN each), else they take units in turn.
    constexpr int TW = T < 4 ? T : 4, TN = T / TW, kGroups = 4 / TW;
    __shared__ __align__(8) uint64_t full[kDMaxStages], empty[kDMaxStages], dfull[2], dempty[2], xfull[8], xempty[8], ssfull, image[kDMaxKb / 8];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort, s_last;
    __shared__ float s_ssq_static[T < 8 ? T * kDMaxKb : 1], s_rss[kDCl * T], s_scale[T], s_best[4];
    __shared__ int s_bidx[4];
    __shared__ uint8_t s_lut[84];

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    constexpr bool residual = (F & (kDResidual | kDStreamed | kDGated)) != 0; // one segment, added into the residual stream, one unit per cluster
    constexpr bool delta = (F & kDDelta) != 0, single = residual || delta;   // one segment, one unit per cluster
    static_assert(!delta || (prepared && T == 1), "the step's product takes one token's prepared input");
    constexpr bool plain = (F & (kDPlain | kDRecords)) != 0;                       // nothing is left prepared
    constexpr bool even = single || (F & kDPlain) != 0 || (F & kDTwo) != 0;     // every CTA has an even number of k-blocks
    const int rank = int(blockIdx.x) & (kDCl - 1), cl = int(blockIdx.x) / kDCl, C = int(gridDim.x) / kDCl;
    const int nkb = p.nkb, S = p.stages, nmat = (F & kDTwo) != 0 ? 2 : (F & (kDResidual | kDStreamed | kDGated | kDPlain | kDDelta | kDRecords)) != 0 ? 1 : p.nmat, XU = unit_slots<T>(nmat);
    const int kb0 = (nkb * rank) >> 2, len = ((nkb * (rank + 1)) >> 2) - kb0; // this CTA's k-blocks
    const int spt = (len + 1) >> 1;                                            // ring stages per (tile, matrix)
    const int nun = single ? 1 : cl < p.units ? (p.units - cl + C - 1) / C : 0;             // units of this cluster: cl, cl + C, ...
    const int nruns = nun * nmat, nstages = nruns * spt;
    uint8_t *ring = smem;                                // S stages
    uint8_t *bimg = ring + size_t(S) * kStage; // len x kImg bytes, unless streamed
    float *xslot = reinterpret_cast<float *>(bimg + (streamed ? 0 : size_t((nkb + 3) >> 2) * kImg)); // XU * nmat exchange slots
    float *s_ssq = T < 8 ? s_ssq_static : xslot + XU * nmat * kSlot; // [token][k-block], unless the input is prepared

    DeltaShared &s_delta = *reinterpret_cast<DeltaShared *>(xslot + XU * nmat * kSlot); // of a launch with a step

    auto seg_of = [&](int unit) -> const DSeg & { return p.seg[single ? 0 : dseg_of(p, unit)]; };
    // ---- the weight stream starts first: it depends on nothing ----------------------------------------------------------
    auto run_src = [&](int run) -> const uint8_t * { // this CTA's records of the run (tile, matrix)
        const int unit = cl + (nmat == 2 ? run >> 1 : run) * C;
        const DSeg &s = seg_of(unit);
        return (nmat == 2 && (run & 1) ? s.packed2 : s.packed) + (size_t(unit - s.tile_begin) * nkb + kb0) * kURec;
    };
    const uint64_t once = once_policy();
    auto load_stage = [&](int slot, const uint8_t *src, int st) { // stage st of a run: two records, or the last one of an odd count
        const uint32_t records = uint32_t(min(2, len - 2 * st));
        mbar_expect_tx(&full[slot], records * (kURec + (streamed ? kImg : 0)));
        bulk_load_hint(ring + size_t(slot) * kStage, src + size_t(st) * kDStage, records * kURec, &full[slot], once);
    };
    auto load_digits = [&](int slot, int st) { // streamed: behind the weights of the only run's stage st
        bulk_load(ring + size_t(slot) * kStage + kDStage, reinterpret_cast<const uint8_t *>(p.in) + size_t(kb0 + 2 * st) * kImg, uint32_t(min(2, len - 2 * st)) * kImg, &full[slot]);
    };
    // Launches that may not read ahead (no pdl) start as early as the others and wait here, ahead of taking tensor memory that the launch before may still
    // want; what follows them may start when they have waited, as if they had been launched then.  Calls one behind the other gain what a launch takes:
    // 12352 x 4096 on packed records, three tokens 11.3 -> 9.2 us, 4096 x 4096, one 8.2 -> 7.5.
    if (p.wait_first) pdl_wait();
    if (warp == 9) {
        if (lane < S) { // one lane per stage: its barriers and the first ring's copy into it
            mbar_init(&full[lane], records ? kDLoaders : 1);
            mbar_init(&empty[lane], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!records && lane < S && lane < nstages) {
            const int run = single ? 0 : lane / spt;
            load_stage(lane, run_src(run), lane - run * spt);
        }
    } else if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(kDTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    } else if (warp == 0) { // the other barriers, one per lane
        if (lane < 2) mbar_init(&dfull[lane], 1);
        else if (lane < 4) mbar_init(&dempty[lane - 2], 4);
        else if (lane < 12) mbar_init(&xfull[lane - 4], 1);
        else if (lane < 20) mbar_init(&xempty[lane - 12], kDCl * TW);
        else if (lane < 20 + kDMaxKb / 8) // one arrival per (token, k-block), or the copy's
            mbar_init(&image[lane - 20], prepared ? 1u : uint32_t(T * max(1, min(8, len - 8 * (lane - 20)))));
        else if (lane == 31) {
            mbar_init(&ssfull, 1);
            s_abort = 0;
            mbar_expect_tx(&ssfull, delta ? kDCl * 8 * 4 : kDCl * T * 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    } else if (tid >= 128 && tid < 128 + 81) {
        s_lut[tid - 128] = digit_pair_code(tid - 128);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // (late: the next launch reads the input of this one ahead of its own wait.  It may start when this launch has seen that input, in the producer.)
    // The next launch may become resident from here on, not earlier: were it to take tensor memory before every CTA here has its own,
    // a CTA could wait for memory held by a CTA that waits for this grid.
    const bool at_once = nstages - kDTriggerStages<T> <= S;
    if (records || (at_once && !(prepared && p.late))) pdl_launch_dependents();
    // The peers' barriers exist when this completes.  Their initialisation is published by the fences above; a release here waited for
    // whatever the SM still had under way, up to 2 us in a launch that could not start beside its predecessor (eight tokens 1540 -> 1503 us
    // a step, one token 1098 -> 1084).
    cluster_arrive_relaxed();
    cluster_wait();
    const uint32_t tmem = s_tmem;
    volatile int *abort_flag = &s_abort;
    bool arrived = false; // at the closing cluster barrier

    float4 cell[delta ? 4 : 1]; // this thread's part of the state, last written a token ago
    if constexpr (delta) {
        if (warp < 8) {
            const float *S = p.delta.state + size_t(cl) * 128 * 128 + size_t(tid >> 3) * 128 + rank * 32 + (tid & 7) * 4;
#pragma unroll
            for (int j = 0; j < 4; j++) cell[j] = __ldcg(reinterpret_cast<const float4 *>(S + size_t(32 * j) * 128));
        }
    }
    if constexpr (prepared) {
        if (!delta && warp >= 4 && warp < 8) pdl_wait(); // they read what earlier launches wrote
    } else if (warp < 8) {
        // ---- activation prologue: this CTA's quarter of the columns ---------------------------------------------------------
        constexpr int kBatch = (F & kDGated) != 0 ? 1 : 3;
        const int items = len * T; // (token, k-block) pairs, dealt to the eight warps
        const bool rms = pro == INSG_PRO_RMSNORM;
        float4 x[kBatch], a[kBatch];
        uint2 w[kBatch];
        auto place = [&](int it, int &m, int &kb) { m = T == 1 ? 0 : it / len; kb = T == 1 ? it : it - m * len; };
        auto load_weights = [&](int b0) {
#pragma unroll
            for (int j = 0; j < kBatch; j++) {
                int m, kb;
                place(b0 + 8 * j, m, kb);
                w[j] = make_uint2(0u, 0u);
                if (b0 + 8 * j < items) {
                    if (rms) w[j] = reinterpret_cast<const uint2 *>(p.norm_w)[(kb0 + kb) * 32 + lane];
                    else if (pro == INSG_PRO_GATED_RMSNORM) w[j] = reinterpret_cast<const uint2 *>(p.norm_w)[lane];
                }
            }
        };
        load_weights(warp); // parameters: may be read before the producer of the activation is done
        pdl_wait();
        for (int b0 = warp; b0 < items; b0 += 8 * kBatch) {
            if (b0 != warp) load_weights(b0);
#pragma unroll
            for (int j = 0; j < kBatch; j++) { // all loads of the batch in flight together; through L2 (see gemv_prologue.cuh)
                int m, kb;
                place(b0 + 8 * j, m, kb);
                x[j] = a[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (b0 + 8 * j < items && m < p.tokens) {
                    const int k = (kb0 + kb) * 128 + lane * 4;
                    x[j] = __ldcg(reinterpret_cast<const float4 *>(p.in + size_t(m) * p.cols + k));
                    switch (pro) {
                    case INSG_PRO_GATED_RMSNORM:
                    case INSG_PRO_SIGMOID_GATE: a[j] = __ldcg(reinterpret_cast<const float4 *>(p.aux + size_t(m) * p.cols + k)); break;
                    case INSG_PRO_SIGMOID_GATE_HEAD0: a[j].x = __ldcg(p.aux + size_t(m) * 2 * p.cols + (k >> 8) * 512 + 256); break;
                    case INSG_PRO_SIGMOID_GATE_QPROJ:
                        a[j] = __ldcg(reinterpret_cast<const float4 *>(p.aux + size_t(m) * 2 * p.cols + (k >> 8) * 512 + 256 + (k & 255)));
                        break;
                    default: break;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < kBatch; j++) {
                if (b0 + 8 * j >= items) break; // warp-uniform
                int m, kb;
                place(b0 + 8 * j, m, kb);
                float4 v = x[j];
                switch (pro) {
                case INSG_PRO_RMSNORM: { // the factor 1/rms is one number per token: the epilogue applies it
                    const float ss = warp_sum(fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w))));
                    if (lane == 0) s_ssq[m * kDMaxKb + kb] = ss;
                    v.x *= bf16_bits_to_float(w[j].x & 0xffff);
                    v.y *= bf16_bits_to_float(w[j].x >> 16);
                    v.z *= bf16_bits_to_float(w[j].y & 0xffff);
                    v.w *= bf16_bits_to_float(w[j].y >> 16);
                    break;
                }
                case INSG_PRO_GATED_RMSNORM: { // a head is one k-block
                    const float hs = warp_sum(fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w))));
                    const float inv = rsqrtf(hs / 128.f + 1e-6f);
                    v.x = v.x * inv * bf16_bits_to_float(w[j].x & 0xffff) * fast_silu(a[j].x);
                    v.y = v.y * inv * bf16_bits_to_float(w[j].x >> 16) * fast_silu(a[j].y);
                    v.z = v.z * inv * bf16_bits_to_float(w[j].y & 0xffff) * fast_silu(a[j].z);
                    v.w = v.w * inv * bf16_bits_to_float(w[j].y >> 16) * fast_silu(a[j].w);
                    break;
                }
                case INSG_PRO_SIGMOID_GATE:
                case INSG_PRO_SIGMOID_GATE_QPROJ:
                    v.x *= fast_sigmoid(a[j].x); v.y *= fast_sigmoid(a[j].y); v.z *= fast_sigmoid(a[j].z); v.w *= fast_sigmoid(a[j].w);
                    break;
                case INSG_PRO_SIGMOID_GATE_HEAD0: {
                    const float g = fast_sigmoid(a[j].x);
                    v.x *= g; v.y *= g; v.z *= g; v.w *= g;
                    break;
                }
                default: break;
                }
                if (!(F & kDGated) && p.x_out && cl == 0 && !rms && m < p.tokens)
                    reinterpret_cast<float4 *>(p.x_out + size_t(m) * p.cols)[(kb0 + kb) * 32 + lane] = v;
                if constexpr (records) { // the k-block's largest magnitude (rows_again)
                    const uint32_t bx = __float_as_uint(fabsf(v.x)), by = __float_as_uint(fabsf(v.y)), bz = __float_as_uint(fabsf(v.z)), bw = __float_as_uint(fabsf(v.w));
                    const uint32_t top = __reduce_max_sync(0xffffffffu, max(max(bx, by), max(bz, bw)));
                    if (lane == 0) s_ssq[m * kDMaxKb + kb] = __uint_as_float(top);
                }
                if constexpr (records) { v.x *= kDLift; v.y *= kDLift; v.z *= kDLift; v.w *= kDLift; }
                store_digits(v, T, m, bimg + size_t(kb) * kImg, s_lut, lane);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the tensor core reads the image through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(&image[kb >> 3]);
            }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (warp == 4 && lane < kDCl * T) { // this quarter's sum of squares of each token to the four CTAs
            const int dst = lane / T, m = lane - dst * T;
            float ss[1] = {0.f};
            if (rms)
#pragma unroll 4
                for (int kb = 0; kb < len; kb++) ss[0] += s_ssq[m * kDMaxKb + kb];
            if (records) // (and its largest magnitude, as bits)
#pragma unroll 4
                for (int kb = 0; kb < len; kb++) ss[0] = __uint_as_float(max(__float_as_uint(ss[0]), __float_as_uint(s_ssq[m * kDMaxKb + kb])));
            send_floats<1>(map_to_rank(smem_u32(&s_rss[rank * T + m]), uint32_t(dst)), ss, map_to_rank(smem_u32(&ssfull), uint32_t(dst)));
        }
    }

    if constexpr (records) {
        if (warp >= 10) {
            // ---- loaders: packed records into what the tensor core reads -------------------------------------------------
            // For plain products on packed records the kernel of gemv_fused.cu dequantises in registers, which bounds it by its ALU pipe; here nothing is
            // computed on a weight.  Replayed, that kernel -> this one (weights beyond L2): 4096 x 4096, one to four tokens 7.0, 7.7, 8.5, 8.9 -> 4.6, 5.2, 6.2,
            // 6.3 us; 12352 x 4096 11.3, 12.3, 13.0, 13.3 -> 7.2, 7.4, 8.4, 8.6; 4096 x 12288 12.3, 15.0, 17.3, 19.0 -> 7.2, 8.8, 11.6, 11.8; 248320 x 4096, queued, one
            // and three 104, 119 -> 81, 87.  With the unswizzled image, whose cells of a row lie 128 and 4096 bytes apart, 191.
            // A record holds its rows' 64 bytes one after the other: K-major rows as the tensor core takes them with the 64-byte swizzle, which
            // moves 16-byte cells about within a row.  So every cell goes straight to its place, 512 consecutive bytes of either side a warp.
            // The scale bytes of rows g and g + 8 lie side by side: they come as they are, and the lane that asked for them sorts them when they are there.
            const int w = warp - 10, g = lane & 7, t = lane >> 3;
            const uint8_t *cells = p.seg[0].packed + lane * 16, *scales = p.seg[0].packed + 1024 + g * 8;
            const int cell = (lane >> 2) * 64 + (((lane & 3) ^ ((lane >> 3) & 3)) << 4);
            constexpr int kTiles = 8 / kDLoaders;
            const int mine = kTiles * w + (t >> 1), raw = w * (128 * kTiles) + lane * 8, tiles = p.seg[0].rows >> 4; // the record whose scales this lane sorts
            const bool sorts = lane < 16 * kTiles;
            bool ok = true;
            int slot = 0, done = 0, st = 0, unit = cl;
            uint32_t phase = 1;
#pragma unroll 1
            for (int i = 0; i < nstages + kDLoadAhead && ok; i++) {
                if (i < nstages) {
                    if (i >= S) ok = mbar_wait(&empty[slot], phase, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    uint8_t *dst = ring + size_t(slot) * kStage;
                    const int blocks = min(2, len - 2 * st);
#pragma unroll
                    for (int h = 0; h < kTiles; h++) { // this warp's tiles of the eight
                        const int tile = unit * 8 + kTiles * w + h;
                        const size_t rec = (size_t(tile) * nkb + kb0 + 2 * st) * kRec;
#pragma unroll
                        for (int b = 0; b < 2; b++)
                            if (tile < tiles && b < blocks) {
                                copy16(dst + b * kURec + cell + (2 * (kTiles * w + h)) * 512, cells + rec + b * kRec);
                                copy16(dst + b * kURec + cell + (2 * (kTiles * w + h) + 1) * 512, cells + rec + b * kRec + 512);
                            }
                    }
                    const int tile = unit * 8 + mine;
                    if (sorts && tile < tiles && (t & 1) < blocks) copy8(dst + kDStage + raw, scales + (size_t(tile) * nkb + kb0 + 2 * st + (t & 1)) * kRec);
                    if (++slot == S) { slot = 0; phase ^= 1; }
                    if (++st == spt) { st = 0; unit += C; }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (i < kDLoadAhead) continue;
                asm volatile("cp.async.wait_group %0;" ::"n"(kDLoadAhead) : "memory");
                uint8_t *dst = ring + size_t(done) * kStage;
                if (sorts) {
                    const uint2 sc = *reinterpret_cast<const uint2 *>(dst + kDStage + raw); // row g: bytes 0, 2, 4, 6; row g + 8: 1, 3, 5, 7
                    const int r = mine * 16 + g;
                    uint8_t *block = dst + (t & 1) * kURec + 8192;
                    *reinterpret_cast<uint32_t *>(block + (r & 31) * 16 + (r >> 5) * 4) = __byte_perm(sc.x, sc.y, 0x6420);
                    *reinterpret_cast<uint32_t *>(block + ((r + 8) & 31) * 16 + (r >> 5) * 4) = __byte_perm(sc.x, sc.y, 0x7531);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[done]);
                if (++done == S) done = 0;
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
    }
    if (warp == 9 && !records) {
        // ---- producer ----------------------------------------------------------------------------------------------------------
        {
            const bool one = elect_one();
            for (int i = S + lane; i < min(nstages, S + p.ahead); i += 32) {
                const int run = single ? 0 : i / spt, st = i - run * spt;
                bulk_prefetch_hint(run_src(run) + size_t(st) * kDStage, uint32_t(min(2, len - 2 * st)) * kURec, once);
            }
            __syncwarp();
            if constexpr (prepared) { // the digits come ready: eight k-blocks per copy, so that the multiplies can start behind the first
                if (!delta) pdl_wait(); // (delta: they were there when the launch before this one let it start)
                if (at_once && p.late) pdl_launch_dependents();
                asm volatile("fence.proxy.async.global;" ::: "memory"); // written by ordinary stores of an earlier launch
                if constexpr (streamed) {
                    if (lane < S && lane < nstages) load_digits(lane, lane);
                    __syncwarp();
                } else
#pragma unroll 1
                for (int kb = 0; kb < len; kb += 8)
                    if (one) {
                        const uint32_t bytes = uint32_t(min(8, len - kb)) * kImg;
                        mbar_expect_tx(&image[kb >> 3], bytes);
                        bulk_load(bimg + size_t(kb) * kImg, reinterpret_cast<const uint8_t *>(p.in) + size_t(kb0 + kb) * kImg, bytes, &image[kb >> 3]);
                    }
            }
            int i = 0, slot = 0;
            uint32_t phase = 1; // of the empty barriers: slot reuse n waits for the n-th release
            bool ok = true;
#pragma unroll 1
            for (int run = 0; run < nruns && ok; run++) {
                const uint8_t *src = run_src(run);
#pragma unroll 1
                for (int st = 0; st < spt; st++, i++) {
                    if (i >= S) {
                        ok = mbar_wait(&empty[slot], phase, abort_flag);
                        if (!ok) break;
                        if (one) {
                            load_stage(slot, src, st);
                            if (streamed) load_digits(slot, st);
                        }
                        if (i == nstages - 1 - kDTriggerStages<T>) pdl_launch_dependents();
                    }
                    if (++slot == S) { slot = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 8) {
        // ---- MMA issuer --------------------------------------------------------------------------------------------------------
        // The whole warp walks the loop and one elected lane issues: every operand is then warp-uniform and lives in uniform
        // registers.  A loop of one lane costs twice as much per instruction (measured per stage: 258 cycles against 594),
        // which is more than a stage of weights takes to arrive.  Descriptors advance by adding to their address field, and
        // the next stage's barrier is polled before this stage's multiplies are issued.
        if (len > 0 && nruns > 0) {
            const uint32_t one = elect_one();
            // E2M1 x E2M1, UE8M0 scales, N columns, M = 128; K-step s of a block uses scale bytes 2s, 2s+1 of both operands
            constexpr uint32_t idesc0 = (1u << 7) | (1u << 10) | ((uint32_t(N) >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24);
            constexpr uint32_t idesc1 = idesc0 | (2u << 29) | (2u << 4);
            constexpr int kHalf = records ? 2 : 256; // from K-step to K-step of a block: 32 bytes of a row, or half of the image
            const uint64_t da0 = records ? umma_desc(smem_u32(ring), 16, 512) | (uint64_t(4) << 61) : umma_desc(smem_u32(ring), 128, 256), dsf0 = umma_desc(smem_u32(ring) + 8192, 16, 128), db0 = umma_desc(smem_u32(streamed ? ring + kDStage : bimg), 128, 256);
            const uint64_t dsb0 = umma_desc(smem_u32(streamed ? ring + kDStage : bimg) + kBKb, 16, 128);
            bool ok = true;
            int st = 0, sfa = 0;
            uint32_t phase = 0;
            bool here = mbar_test(&full[0], 0), room = true;
#pragma unroll 1
            for (int run = 0; run < nruns && ok; run++) {
                const int buf = run & 1;
                const uint32_t dcol = tmem + uint32_t(64 * buf);
                if (!room) ok = mbar_wait(&dempty[buf], ((run >> 1) & 1) ^ 1, abort_flag); // first use of each buffer passes at once
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint64_t db = db0;
                uint32_t sb = tmem + kDSfbCol;
                // Branches among the issued instructions cost more than the instructions: the first run, which also brings the
                // digits' scales, and the single last block of an odd count have loops of their own.
                auto stage = [&](int kb, auto is_first, auto has_two) -> bool {
                    constexpr bool first = decltype(is_first)::value, two = decltype(has_two)::value;
                    if (!here && !mbar_wait(&full[st], phase, abort_flag)) return false;
                    if (!streamed && first && (kb & 7) == 0 && !mbar_wait(&image[kb >> 3], 0, abort_flag)) return false; // the digits of eight k-blocks
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t off = uint64_t(uint32_t(st) * uint32_t(kStage >> 4)), da = da0 + off, dsf = dsf0 + off;
                    if (streamed) db = db0 + off;
                    const uint64_t dsb = streamed ? dsb0 + off : dsb0 + uint64_t(kb * (kImg >> 4));
                    const uint32_t sa = tmem + kDSfaCol + 8 * sfa;
                    const int cur = st;
                    if (++st == S) { st = 0; phase ^= 1; }
                    here = mbar_test(&full[st], phase);
                    if (kb + 2 >= len) room = mbar_test(&dempty[buf ^ 1], (((run + 1) >> 1) & 1) ^ 1);
                    if (first) { // the digits' scales stay in tensor memory for all tiles
                        copy_scales_if(one, sb, dsb);
                        if (two) copy_scales_if(one, sb + 4, dsb + (kImg >> 4));
                    }
                    copy_scales_if(one, sa, dsf);
                    if (two) copy_scales_if(one, sa + 4, dsf + (kURec >> 4));
                    mma_step_if(one, dcol, da, db, idesc0, kb > 0, sa, sb);
                    mma_step_if(one, dcol, da + kHalf, db + (kBKb >> 5), idesc1, true, sa, sb);
                    if (two) {
                        mma_step_if(one, dcol, da + (kURec >> 4), db + (kImg >> 4), idesc0, true, sa + 4, sb + 4);
                        mma_step_if(one, dcol, da + (kURec >> 4) + kHalf, db + (kImg >> 4) + (kBKb >> 5), idesc1, true, sa + 4, sb + 4);
                    }
                    commit_if(one, &empty[cur]);
                    if (!streamed) db += 2 * (kImg >> 4);
                    sb += 8;
                    sfa = (sfa + 1) & 3;
                    return true;
                };
                constexpr std::true_type yes{};
                constexpr std::false_type no{};
                const int evens = len & ~1;
                if (single || run == 0) {
#pragma unroll 1
                    for (int kb = 0; kb < evens && ok; kb += 2) ok = stage(kb, yes, yes);
                } else {
#pragma unroll 1
                    for (int kb = 0; kb < evens && ok; kb += 2) ok = stage(kb, no, yes);
                }
                if constexpr (!even)
                    if (ok && evens < len) ok = stage(evens, yes, no); // the digits' scales once more: no copy of the code for a rare case
                if (ok) commit_if(one, &dfull[buf]);
            }
        }
    } else if (warp < 4) {
        // ---- accumulators -> partial sums -> the CTA that owns these 32 rows (rank = warp) ------------------------------------
        const uint32_t dst = map_to_rank(smem_u32(xslot) + uint32_t((rank * 32 + lane) * T * 4), uint32_t(warp));
        const uint32_t dbar = map_to_rank(smem_u32(xfull), uint32_t(warp));
        const int nslots = XU * nmat;
        bool ok = true;
#pragma unroll 1
        for (int run = 0; run < nruns && ok; run++) {
            const int buf = run & 1;
            float y[T];
#pragma unroll
            for (int t = 0; t < T; t++) y[t] = 0.f;
            if (len > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait(&dfull[buf], (run >> 1) & 1, abort_flag));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                load_partial<T>(tmem + uint32_t(64 * buf) + (uint32_t(warp * 32) << 16), y);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&dempty[buf]);
            }
            const int slot = run % nslots;
            if (!single && run >= nslots) { // the slot's previous content must have been added up by its owner
                ok = __all_sync(0xffffffffu, mbar_wait_cluster(&xempty[slot], ((run / nslots) - 1) & 1, abort_flag));
                if (!ok) break;
            }
            send_floats<T>(dst + uint32_t(slot * kSlot * 4), y, dbar + uint32_t(slot * 8));
        }
    } else if (warp < 8) {
        // ---- owner of 32 rows of every tile: add the four parts in rank order, fused epilogue ----------------------------------
        const int fw = warp - 4, group = fw / TW, t0 = (fw % TW) * TN;
        float best = -3.402823466e38f;
        int best_idx = 0x7fffffff;
        bool ok = true;
        // The quarters' sums of squares arrive while the weights are still being multiplied.  Every CTA waits for all four
        // (also where they are not needed), so that nobody leaves while a peer still writes into its shared memory.
        if constexpr (!prepared) ok = __all_sync(0xffffffffu, mbar_wait_cluster(&ssfull, 0, abort_flag));
#pragma unroll
        for (int u = 0; u < TN; u++) {
            const int t = t0 + u;
            float sc = records ? 1.f / kDLift : 1.f;
            if (prepared && p.prep_partials) {
                const int groups = p.cols >> 5;
                float ss = 0.f;
                if (t < p.tokens)
#pragma unroll 4
                    for (int i = lane; i < groups; i += 32) ss += __ldcg(p.prep_partials + t * groups + i);
                sc = rsqrtf(warp_sum(ss) / float(p.cols) + 1e-6f);
            } else if (pro == INSG_PRO_RMSNORM) {
                sc = rsqrtf((s_rss[t] + s_rss[T + t] + s_rss[2 * T + t] + s_rss[3 * T + t]) / float(p.cols) + 1e-6f);
            }
            if (lane == 0) s_scale[t] = sc;
        }
        asm volatile("bar.sync 3, 128;" ::: "memory");
        if (!prepared && ok && p.x_out && cl == 0 && pro == INSG_PRO_RMSNORM)
#pragma unroll 1
            for (int m = 0; m < p.tokens; m++)
#pragma unroll 1
                for (int k = kb0 * 128 + fw * 32 + lane; k < (kb0 + len) * 128; k += 128)
                    p.x_out[size_t(m) * p.cols + k] = __ldcg(p.in + size_t(m) * p.cols + k) * s_scale[m] * bf16_bits_to_float(p.norm_w[k]);
        // What the epilogue of a unit needs besides the sums: asked for before the wait for them; where one warp has two tokens of
        // every unit, a unit ahead (eight sequences, in-projection: 10.5 -> 9.7 us; with fewer tokens it costs 0.2 us).
        constexpr bool kAhead = TN > 1;
        struct Fetched {
            float h[TN][3]; // per token: the residual, or the convolution's history; decay: bias and rate
            uint2 w;        // the convolution's weights
        } next;
        auto fetch = [&](int i) {
            const int unit = cl + i * C;
            const DSeg &s = seg_of(unit);
            const int row = (unit - s.tile_begin) * 128 + rank * 32 + lane;
            if ((F & kDTwo) != 0 || delta || row >= s.rows) return;
            if (!residual && s.epilogue == INSG_EPI_CONV_SILU) next.w = reinterpret_cast<const uint2 *>(s.conv_w)[row];
#pragma unroll
            for (int u = 0; u < TN; u++) {
                const int t = t0 + u;
                if (t >= p.tokens) break;
                if (residual || (!plain && s.epilogue == INSG_EPI_RESIDUAL)) {
                    next.h[u][0] = __ldcg(s.out + row + t * size_t(s.rows));
                } else if (s.epilogue == INSG_EPI_CONV_SILU) {
                    const float *hist = s.conv_state + t * s.conv_stride + size_t(row) * 3;
#pragma unroll
                    for (int j = 0; j < 3; j++) next.h[u][j] = __ldcg(hist + j);
                } else if (s.epilogue == INSG_EPI_DECAY && u == 0) {
                    next.h[0][0] = bf16_bits_to_float(s.dt_bias[row]);
                    next.h[0][1] = -__expf(s.A_log[row]);
                }
            }
        };
        if (kAhead && ok && group < nun) fetch(group);
        int i = group;
#pragma unroll 1
        for (; i < nun && ok; i += kGroups) {
            const int unit = cl + i * C;
            const DSeg &s = seg_of(unit);
            const int row = (unit - s.tile_begin) * 128 + rank * 32 + lane;
            const bool on = row < s.rows;
            const size_t ld = size_t(s.rows);
            float *out = s.out + row;
            if (!kAhead) fetch(i);
            const Fetched f = next;
            if (kAhead && i + kGroups < nun) fetch(i + kGroups);
            const float pw = !plain && s.prep_w ? bf16_bits_to_float(s.prep_w[row]) : 1.f; // rows % 128 == 0 where it is set
            const float cw0 = bf16_bits_to_float(f.w.x & 0xffff), cw1 = bf16_bits_to_float(f.w.x >> 16);
            const float cw2 = bf16_bits_to_float(f.w.y & 0xffff), cw3 = bf16_bits_to_float(f.w.y >> 16);
            const bool one_history = s.conv_stride == 0; // consecutive tokens of one sequence
            float y[2][TN];
#pragma unroll
            for (int mat = 0; mat < 2; mat++) {
                if (mat >= nmat) break;
                const int slot = (i % XU) * nmat + mat;
                if (lane == 0 && t0 == 0) mbar_expect_tx(&xfull[slot], kSlot * 4);
                ok = __all_sync(0xffffffffu, mbar_wait_cluster(&xfull[slot], (i / XU) & 1, abort_flag));
                if (!ok) break;
                const float *src = xslot + size_t(slot) * kSlot + lane * T;
                auto sum = [&](int t) { // the four parts in rank order
                    float z = src[t];
#pragma unroll
                    for (int r = 1; r < kDCl; r++) z += src[r * 32 * T + t];
                    return z * s_scale[t];
                };
#pragma unroll
                for (int u = 0; u < TN; u++) y[mat][u] = sum(t0 + u);
                if (T > 1 && !(F & kDTwo) && !residual && one_history && s.epilogue == INSG_EPI_CONV_SILU) { // the history runs through the tokens: one warp takes them in order
                    if (t0 == 0 && on) {
                        float h0 = f.h[0][0], h1 = f.h[0][1], h2 = f.h[0][2];
#pragma unroll 1
                        for (int t = 0; t < p.tokens; t++) {
                            const float raw = sum(t);
                            out[t * ld] = fast_silu(fmaf(h0, cw0, fmaf(h1, cw1, fmaf(h2, cw2, raw * cw3))));
                            h0 = h1; h1 = h2; h2 = raw;
                        }
                        float *hist = s.conv_state + size_t(row) * 3;
                        hist[0] = h0; hist[1] = h1; hist[2] = h2;
                    }
                }
                if (!single && i + XU < nun) { // the slot will be used again: tell the four senders, whose next st.async must come after these reads
                    __syncwarp();
                    if (lane < kDCl) remote_arrive(map_to_rank(smem_u32(&xempty[slot]), uint32_t(lane)));
                }
            }
            if (!ok) break;
            if (!delta && i + kGroups >= nun) { // nothing more comes in for this warp: the peers need not wait for its epilogue
                cluster_arrive_relaxed();
                arrived = true;
            }
            if constexpr (records) {
#pragma unroll
                for (int u = 0; u < TN; u++) {
                    const int t = t0 + u;
                    const uint32_t top = max(max(__float_as_uint(s_rss[t]), __float_as_uint(s_rss[T + t])), max(__float_as_uint(s_rss[2 * T + t]), __float_as_uint(s_rss[3 * T + t])));
                    const float a = fabsf(y[0][u]);
                    const uint32_t again = __ballot_sync(0xffffffffu, on && t < p.tokens && (!(a <= 3.402823466e38f) || (a > 0.f && a < kDFewBits * __uint_as_float(top))));
                    if (again && top < 0x7f800000u) // (a token with an infinity or NaN is NaN)
                        y[0][u] = rows_again(s.packed, p.in + size_t(t) * p.cols, nkb, row - lane, again, top, y[0][u], lane);
                }
            }
            if (!on) continue;
            if constexpr (delta) {
                out[0] = y[0][0];
                s_delta.z[lane] = y[0][0];
            } else if constexpr (logits) {
                out[0] = y[0][0];
                if (y[0][0] > best || (y[0][0] == best && row < best_idx)) { best = y[0][0]; best_idx = row; }
            } else {
                // Each epilogue leaves its value in v; one store and one copy of the digits' code serve them all.
                float v[TN];
                if (T > 1 && !(F & kDTwo) && !residual && one_history && s.epilogue == INSG_EPI_CONV_SILU) continue; // done above
#pragma unroll
                for (int u = 0; u < TN; u++) v[u] = y[0][u];
                if constexpr ((F & kDTwo) != 0) {
#pragma unroll
                    for (int u = 0; u < TN; u++) v[u] = fast_silu(y[0][u]) * y[1][u];
                } else if constexpr (residual) {
#pragma unroll
                    for (int u = 0; u < TN; u++) v[u] = f.h[u][0] + y[0][u];
                } else {
                switch (s.epilogue) {
                case INSG_EPI_STORE: break;
                case INSG_EPI_RESIDUAL:
                    if constexpr (!plain) {
#pragma unroll
                        for (int u = 0; u < TN; u++) v[u] = f.h[u][0] + y[0][u];
                    }
                    break;
                case INSG_EPI_CONV_SILU:
#pragma unroll
                    for (int u = 0; u < TN; u++) {
                        if (t0 + u < p.tokens) {
                            float *hist = s.conv_state + (t0 + u) * s.conv_stride + size_t(row) * 3; // independent sequences: each token has its own
                            v[u] = fast_silu(fmaf(f.h[u][0], cw0, fmaf(f.h[u][1], cw1, fmaf(f.h[u][2], cw2, y[0][u] * cw3))));
                            hist[0] = f.h[u][1]; hist[1] = f.h[u][2]; hist[2] = y[0][u];
                        }
                    }
                    break;
                case INSG_EPI_BETA:
#pragma unroll
                    for (int u = 0; u < TN; u++) v[u] = fast_sigmoid(y[0][u]);
                    break;
                case INSG_EPI_DECAY:
#pragma unroll
                    for (int u = 0; u < TN; u++) {
                        const float z = y[0][u] + f.h[0][0];
                        v[u] = f.h[0][1] * (z > 20.f ? z : log1pf(__expf(z)));
                    }
                    break;
                case INSG_EPI_SWIGLU:
                    if constexpr (!plain) {
#pragma unroll
                        for (int u = 0; u < TN; u++) v[u] = fast_silu(y[0][u]) * y[1][u];
                    }
                    break;
                default: continue; // no such epilogue: nothing is stored
                }
                }
#pragma unroll
                for (int u = 0; u < TN; u++) {
                    if (t0 + u >= p.tokens) break;
                    out[(t0 + u) * ld] = v[u];
                    if (!plain && s.prep) leave_digits<T>(s, v[u], pw, row, t0 + u, s_lut, lane);
                }
            }
        }
        if constexpr (records) // after a wait that ran out: a plain product has no error flag, so what it leaves out must not pass for a result
            if (!ok)
#pragma unroll 1
                for (; i < nun; i += kGroups) {
                    const int row = (cl + i * C) * 128 + rank * 32 + lane;
                    for (int t = t0; t < min(t0 + TN, p.tokens); t++)
                        if (row < p.seg[0].rows) p.seg[0].out[t * size_t(p.seg[0].rows) + row] = __int_as_float(0x7fc00000);
                }
        if constexpr (logits) {
            // per-CTA arg-max, then the last CTA of the grid folds the CTAs' (lowest index on ties)
            auto fold = [&] {
#pragma unroll
                for (int mk = 16; mk; mk >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, best, mk);
                    const int oi = __shfl_xor_sync(0xffffffffu, best_idx, mk);
                    if (ov > best || (ov == best && oi < best_idx)) { best = ov; best_idx = oi; }
                }
            };
            __syncwarp();
            fold();
            if (lane == 0) { s_best[fw] = best; s_bidx[fw] = best_idx; }
            asm volatile("bar.sync 2, 128;" ::: "memory");
            if (fw == 0) {
                if (lane == 0) {
#pragma unroll 1
                    for (int w = 1; w < 4; w++)
                        if (s_best[w] > best || (s_best[w] == best && s_bidx[w] < best_idx)) { best = s_best[w]; best_idx = s_bidx[w]; }
                    p.argmax_partial[blockIdx.x] = make_float2(best, __int_as_float(best_idx));
                    if (*abort_flag && p.error_flag) *p.error_flag = 1; // ahead of the ticket: the last CTA reports for all of them
                    __threadfence();
                    s_last = atomicAdd(p.argmax_ticket, 1u) == gridDim.x - 1;
                }
                __syncwarp();
                if (s_last) {
                    __threadfence();
                    best = -3.402823466e38f;
                    best_idx = 0x7fffffff;
#pragma unroll 1
                    for (int i = lane; i < int(gridDim.x); i += 32) {
                        const float2 e = __ldcg(p.argmax_partial + i);
                        const int idx = __float_as_int(e.y);
                        if (e.x > best || (e.x == best && idx < best_idx)) { best = e.x; best_idx = idx; }
                    }
                    fold();
                    if (lane == 0) {
                        *p.token_out = best_idx;
                        if (p.token_feedback) *p.token_feedback = best_idx;
                        if (p.host_result) { // a host that waits for the stream needs no copy behind it
                            p.host_result[0] = best_idx;
                            p.host_result[1] = p.error_flag ? __ldcg(p.error_flag) : 0;
                        }
                        if (p.position_inout) {
                            const int pos = __ldcg(p.position_inout);
                            if (p.token_log && pos >= 0 && pos < p.token_log_capacity) p.token_log[pos] = best_idx;
                            *p.position_inout = pos + 1;
                        }
                        *p.argmax_ticket = 0u;
                    }
                }
            }
        }
    }
    if constexpr (delta)
        if (warp < 8) delta_step(p.delta, cell, s_delta, cl, rank, &ssfull, abort_flag, s_lut, tid);
    // Nobody leaves while a peer may still write into its shared memory (after an expired wait too).
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!arrived) cluster_arrive_relaxed();
    cluster_wait();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kDTmemCols));
    if (tid == 0 && s_abort && p.error_flag) *p.error_flag = 1;
}

// ---- repack: MLX layout -> shared-memory images ----------------------------------------------------
// One thread per (row of a tile, k-block): copies the row's 64 bytes into the four 16-byte cells of the
// record and its four scale bytes into the scale block.  Rows beyond `rows` are zero weights with scale 1.
__global__ void repack_umma_kernel(const uint32_t *__restrict__ w, const uint8_t *__restrict__ s, uint8_t *__restrict__ out, int rows,
                                   int cols)
{
    const int nkb = cols >> 7;
    const size_t idx = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t ntiles = (size_t(rows) + 127) >> 7;
    if (idx >= ntiles * nkb * 128) return;
    const int r = int(idx & 127);
    const size_t rec_id = idx >> 7;
    const int kb = int(rec_id % nkb);
    const size_t tile = rec_id / nkb;
    const size_t row = tile * 128 + r;
    uint8_t *rec = out + rec_id * kURec;
    uint4 q[4] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
    uint32_t sc = 0x7F7F7F7Fu;
    if (row < size_t(rows)) {
        const uint4 *src = reinterpret_cast<const uint4 *>(w + row * (cols >> 3) + kb * 16);
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = src[i];
        sc = *reinterpret_cast<const uint32_t *>(s + row * (cols >> 5) + kb * 4);
    }
    // 64 bytes of the row = 2 K-steps x 2 k-cores of 16 bytes
#pragma unroll
    for (int i = 0; i < 4; i++) *reinterpret_cast<uint4 *>(rec + (i >> 1) * 4096 + (r >> 3) * 256 + (i & 1) * 128 + (r & 7) * 16) = q[i];
    *reinterpret_cast<uint32_t *>(rec + 8192 + (r & 31) * 16 + (r >> 5) * 4) = sc;
}

namespace {
// The variants there are, for T token slots: the launch chooses among them and the attributes are set for them by the same list.
using DKernel = void (*)(DParams);
template <int T, int... F> DKernel variant_of(int f)
{
    DKernel k = nullptr;
    ((f == F ? void(k = umma_gemv_kernel<T, F>) : void()), ...);
    return k;
}
DKernel gemv_kernel(int slots, int f)
{
    constexpr int kP = kDPrepared;
    switch (slots) {
    case 1: return variant_of<1, 0, kP, kP | kDTwo, kP | kDResidual, kP | kDPlain, kDLogits, kP | kDLogits, kDGated, kP | kDDelta, kDRecords>(f);
    case 2: return variant_of<2, 0, kP, kP | kDTwo, kP | kDResidual, kP | kDPlain, kDGated, kDRecords>(f);
    case 4: return variant_of<4, 0, kP, kP | kDTwo, kP | kDResidual, kP | kDPlain, kP | kDStreamed, kDRecords>(f);
    default: return variant_of<8, 0, kP, kP | kDTwo, kP | kDResidual, kP | kDPlain, kP | kDStreamed>(f);
    }
}

std::mutex g_attr_mutex;
int g_max_clusters[64] = {0}; // per device: clusters that run at once with one CTA per SM (0 = not asked yet)

// The shared-memory opt-in is a per-device function attribute; the cluster count is a property of the device's layout.
int device_clusters(int *out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= 64) return fail(INSG_E_LIMIT, "gemv: device ordinal beyond 63");
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    if (!g_max_clusters[dev]) {
        for (int slots : {1, 2, 4, 8})
            for (int f = 0; f < 2 * kDRecords; f++)
                if (const DKernel k = gemv_kernel(slots, f)) {
                    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
                    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(umma gemv)");
                }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kDCl);
        cfg.blockDim = dim3(kDThreads);
        cfg.dynamicSmemBytes = 200 * 1024;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kDCl;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        e = cudaOccupancyMaxActiveClusters(&n, umma_gemv_kernel<1, 0>, &cfg);
        if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveClusters");
        g_max_clusters[dev] = std::max(1, std::min(n, 128)); // 128 clusters: the arg-max partials are sized for 512 CTAs
    }
    *out = g_max_clusters[dev];
    return INSG_OK;
}
} // namespace

// What the gated-norm prologue makes of a step's output, as a launch of its own: the digits of one token, a warp per head, with its order of every sum.
constexpr int kDigitHeads = 4;
__global__ void __launch_bounds__(32 * kDigitHeads) gated_digits_kernel(const float *core, const float *z, const uint16_t *norm_w, uint8_t *image)
{
    __shared__ uint8_t s_lut[84];
    const int tid = threadIdx.x, lane = tid & 31, head = blockIdx.x * kDigitHeads + (tid >> 5);
    if (tid < 81) s_lut[tid] = digit_pair_code(tid);
    __syncthreads();
    const uint2 w = reinterpret_cast<const uint2 *>(norm_w)[lane];
    pdl_wait();
    float4 v = __ldcg(reinterpret_cast<const float4 *>(core) + head * 32 + lane);
    const float4 g = __ldcg(reinterpret_cast<const float4 *>(z) + head * 32 + lane);
    const float inv = rsqrtf(warp_sum(fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w)))) / 128.f + 1e-6f);
    v.x = v.x * inv * bf16_bits_to_float(w.x & 0xffff) * fast_silu(g.x);
    v.y = v.y * inv * bf16_bits_to_float(w.x >> 16) * fast_silu(g.y);
    v.z = v.z * inv * bf16_bits_to_float(w.y & 0xffff) * fast_silu(g.z);
    v.w = v.w * inv * bf16_bits_to_float(w.y >> 16) * fast_silu(g.w);
    store_digits(v, 1, 0, image + size_t(head) * 1024, s_lut, lane);
}

static int check_gated_step(const insg_gemv_op *gate, const insg_delta_op *step)
{
    if (!gate || !step || !step->state || !step->q16 || !step->k16 || !step->v32 || !step->g32 || !step->beta32 || !step->out32 || !step->norm_w || !step->image)
        return fail(INSG_E_ARG, "deltanet: null pointer");
    if (gate->layout != 1) return fail(INSG_E_SHAPE, "deltanet: the gate's product takes the tcgen05 layout");
    if (gate->prologue != INSG_PRO_PREPARED || gate->tokens > 1 || gate->n_segments != 1 || gate->seg[0].epilogue != INSG_EPI_STORE || gate->seg[0].rows != 4096 ||
        gate->cols <= 0 || gate->cols % 1024)
        return fail(INSG_E_SHAPE, "deltanet: the gate's product takes one token, a prepared input of a multiple of 1024 columns and one stored segment of 4096 rows");
    return INSG_OK;
}

int gemv_umma_launch(const insg_gemv_op *op, cudaStream_t st, const insg_delta_op *step)
{
    const bool records = op && op->layout == 0; // one plain product of up to four tokens (insg_mxfp4_gemv_packed)
    if (!op || !op->in) return fail(INSG_E_ARG, "gemv: null operand");
    const int tokens = op->tokens > 1 ? op->tokens : 1;
    if (tokens > 8) return fail(INSG_E_SHAPE, "gemv: 1..8 tokens");
    if (op->cols <= 0 || (op->cols & 127) || op->cols > kDMaxKb * kDCl * 128) return fail(INSG_E_SHAPE, "gemv: cols must be a multiple of 128, <= 12288");
    if (op->n_segments < 1 || op->n_segments > 4) return fail(INSG_E_SHAPE, "gemv: 1..4 segments");
    if (op->prologue < 0 || op->prologue > INSG_PRO_PREPARED) return fail(INSG_E_ARG, "gemv: unknown prologue");
    if ((op->prologue == INSG_PRO_RMSNORM || op->prologue == INSG_PRO_GATED_RMSNORM) && !op->norm_w) return fail(INSG_E_ARG, "gemv: norm weight missing");
    if (op->prologue >= INSG_PRO_GATED_RMSNORM && op->prologue != INSG_PRO_PREPARED && !op->aux) return fail(INSG_E_ARG, "gemv: prologue operand missing");
    DParams p = {};
    p.in = op->in; p.aux = op->aux; p.norm_w = op->norm_w; p.x_out = op->x_out;
    p.cols = op->cols; p.prologue = op->prologue;
    if (op->prologue == INSG_PRO_PREPARED) {
        if (op->prep_rms && !op->prep_partials) return fail(INSG_E_ARG, "gemv: the RMS factor of a prepared input needs the producer's sums");
        p.x_out = nullptr;
        p.prep_partials = op->prep_rms ? op->prep_partials : nullptr;
    }
    p.nkb = op->cols >> 7;
    p.nseg = op->n_segments;
    p.tokens = tokens;
    bool logits = false;
    for (int i = 0; i < op->n_segments; i++) {
        const insg_gemv_segment &s = op->seg[i];
        if (!s.packed || !s.out || s.rows <= 0) return fail(INSG_E_SHAPE, "gemv: bad segment");
        if (s.epilogue == INSG_EPI_SWIGLU && !s.packed2) return fail(INSG_E_ARG, "gemv: SwiGLU needs two matrices");
        if (s.epilogue == INSG_EPI_CONV_SILU && (!s.conv_state || !s.conv_w)) return fail(INSG_E_ARG, "gemv: conv operands missing");
        if (s.epilogue == INSG_EPI_DECAY && (!s.A_log || !s.dt_bias)) return fail(INSG_E_ARG, "gemv: decay operands missing");
        DSeg &d = p.seg[i];
        d.packed = static_cast<const uint8_t *>(s.packed);
        d.packed2 = static_cast<const uint8_t *>(s.packed2);
        d.out = s.out; d.conv_state = s.conv_state; d.conv_w = s.conv_w; d.A_log = s.A_log; d.dt_bias = s.dt_bias;
        d.conv_stride = s.conv_token_stride;
        if (s.prep) {
            if (s.epilogue != INSG_EPI_RESIDUAL && s.epilogue != INSG_EPI_SWIGLU) return fail(INSG_E_ARG, "gemv: prepared output needs the residual or SwiGLU epilogue");
            if (s.rows & 127) return fail(INSG_E_SHAPE, "gemv: a prepared output needs rows % 128 == 0");
            d.prep = static_cast<uint8_t *>(s.prep);
            d.prep_w = s.prep_w;
            d.prep_partials = s.prep_partials;
        }
        const int nmat = s.epilogue == INSG_EPI_SWIGLU ? 2 : 1;
        if (p.nmat && p.nmat != nmat) return fail(INSG_E_SHAPE, "gemv: SwiGLU segments cannot be mixed with others");
        p.nmat = nmat;
        d.tile_begin = p.units; p.units += (s.rows + 127) >> 7; d.epilogue = s.epilogue; d.rows = s.rows;
        logits |= s.epilogue == INSG_EPI_LOGITS;
    }
    if (logits) {
        if (op->n_segments != 1) return fail(INSG_E_SHAPE, "gemv: the logits epilogue takes one segment");
        if (tokens != 1) return fail(INSG_E_SHAPE, "gemv: the logits epilogue takes one token");
        if (!op->argmax_scratch || !op->token_out) return fail(INSG_E_ARG, "gemv: arg-max scratch/token missing");
        p.argmax_ticket = static_cast<unsigned *>(op->argmax_scratch);
        p.argmax_partial = reinterpret_cast<float2 *>(static_cast<uint8_t *>(op->argmax_scratch) + 64);
        p.token_out = op->token_out; p.token_feedback = op->token_feedback; p.token_log = op->token_log; p.position_inout = op->position_inout;
        p.host_result = op->host_result;
        p.token_log_capacity = op->token_log_capacity;
        if (op->token_log && op->token_log_capacity <= 0) return fail(INSG_E_ARG, "gemv: token_log needs its capacity");
    }
    p.error_flag = static_cast<int *>(op->error_flag);
    p.late = op->pdl == 2;
    p.wait_first = !op->pdl;
    int max_clusters = 0;
    const int rc = device_clusters(&max_clusters);
    if (rc != INSG_OK) return rc;
    const int clusters = std::min(p.units, max_clusters);
    const int T = tokens == 1 ? 1 : tokens == 2 ? 2 : tokens <= 4 ? 4 : 8;
    const int kbq = (p.nkb + 3) >> 2;
    const int slots = (T == 1 ? unit_slots<1>(p.nmat) : T == 8 ? unit_slots<8>(p.nmat) : unit_slots<2>(p.nmat)) * p.nmat;
    const size_t exchange = size_t(slots) * kDCl * 32 * T * sizeof(float), kblock = 512 * T + 512;
    // Digits that only one unit per cluster reads need not lie in shared memory as a whole: with the weights they multiply, two k-blocks a
    // stage, they leave the launch within half an SM where the image (61 KB for three tokens of 12288 columns, 111 for eight) would not,
    // so that it starts beside its predecessor and the next launch beside it: a step of three sequences 1208 -> 1204 us, of eight 1412 -> 1402.
    const bool prep = op->prologue == INSG_PRO_PREPARED;
    const bool whole = (p.nkb & 7) == 0, resid = whole && p.nseg == 1 && p.seg[0].epilogue == INSG_EPI_RESIDUAL && p.units <= clusters;
    bool plain = whole; // epilogues that add nothing and leave nothing prepared
    for (int i = 0; i < p.nseg; i++) plain &= p.seg[i].epilogue != INSG_EPI_RESIDUAL && p.seg[i].epilogue != INSG_EPI_SWIGLU && p.seg[i].epilogue != INSG_EPI_LOGITS;
    const bool streamed = prep && T >= 4 && resid && kbq * kblock + exchange + 4 * kDStage > size_t(kDHalfSm);
    const size_t stage_bytes = kDStage + (streamed ? 2 * kblock : 0) + (records ? 1024 : 0);
    const size_t fixed = exchange + (step ? sizeof(DeltaShared) : 0) + (streamed ? 0 : kbq * kblock) + (T == 8 && !prep ? size_t(8) * kDMaxKb * sizeof(float) : 0);
    // ring: no more stages than the launch has, within half an SM when that leaves at least four, else whatever fits.  Four are too
    // few to stream at full rate, so a launch of many units (the head: 55 per cluster, eight tokens 97 us against 91) takes the
    // whole SM; one of a few gains more from starting beside its predecessor.
    const int need = ((p.units + clusters - 1) / clusters) * p.nmat * ((kbq + 1) / 2);
    int stages = fixed < size_t(kDHalfSm) ? int((kDHalfSm - fixed) / stage_bytes) : 0;
    if (records || stages < 4 || (stages == 4 && need > 96)) stages = int((size_t(222) * 1024 - fixed) / stage_bytes);
    p.stages = std::max(1, std::min({stages, need, kDMaxStages}));
    p.ahead = !op->pdl ? 0 : T == 1 ? kDAheadStages<1> : T == 2 ? kDAheadStages<2> : kDAheadStages<4>; // a launch that waits for its predecessor anyway streams at once
    const size_t smem = fixed + size_t(p.stages) * stage_bytes;

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(clusters * kDCl));
    cfg.blockDim = dim3(kDThreads + (records ? 32 * kDLoaders : 0));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1]; // the cluster's shape is part of the kernel
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1; // without pdl the launch starts as early, and waits before it reads
    if (step) {
        p.delta = DDelta{step->state, step->q16, step->k16, step->v32, step->g32, step->beta32, step->out32, step->norm_w, static_cast<uint8_t *>(step->image)};
    }
    const bool gated = op->prologue == INSG_PRO_GATED_RMSNORM && !op->x_out && resid && T <= 2;
    const int special = step ? kDDelta : logits ? kDLogits : streamed ? kDStreamed : prep && whole && p.nmat == 2 ? kDTwo : prep && resid ? kDResidual : prep && plain ? kDPlain : gated ? kDGated : 0;
    const DKernel kernel = records ? gemv_kernel(T, kDRecords) : gemv_kernel(T, special | (prep ? kDPrepared : 0));
    if (!kernel) return fail(INSG_E_ARG, "gemv: no such variant");
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
    return e == cudaSuccess ? INSG_OK : cuda_fail(e, "umma gemv launch");
}

} // namespace insg

using namespace insg;

extern "C" {

int insg_deltanet_gated_step(const insg_gemv_op *gate, const insg_delta_op *step, insg_stream_t stream)
{
    int clusters = 0, rc = check_gated_step(gate, step);
    if (rc == INSG_OK) rc = device_clusters(&clusters);
    if (rc != INSG_OK) return rc;
    return clusters >= 32 ? gemv_umma_launch(gate, stream, step) : insg_deltanet_gated_step_apart(gate, step, stream);
}

int insg_deltanet_gated_step_apart(const insg_gemv_op *gate, const insg_delta_op *step, insg_stream_t stream)
{
    int rc = check_gated_step(gate, step);
    if (rc == INSG_OK) rc = gemv_umma_launch(gate, stream, nullptr);
    if (rc == INSG_OK) rc = insg_deltanet_decode(step->state, step->q16, step->k16, step->v32, step->g32, step->beta32, step->out32, gate->pdl, stream);
    if (rc == INSG_OK) rc = launch(gated_digits_kernel, dim3(32 / kDigitHeads), dim3(32 * kDigitHeads), 0, stream, true, step->out32, gate->seg[0].out, step->norm_w, static_cast<uint8_t *>(step->image));
    return rc;
}

size_t insg_mxfp4_digit_image_bytes(int cols, int tokens)
{
    if (cols <= 0 || (cols & 127) || tokens < 1 || tokens > 8) return 0;
    const int T = tokens == 1 ? 1 : tokens == 2 ? 2 : tokens <= 4 ? 4 : 8;
    return size_t(cols >> 7) * (512 * T + 512);
}

size_t insg_mxfp4_packed_umma_bytes(int rows, int cols)
{
    if (rows <= 0 || cols <= 0 || (cols & 127)) return 0;
    return size_t((rows + 127) >> 7) * (cols >> 7) * kURec;
}

int insg_mxfp4_repack_umma(const uint32_t *weight, const uint8_t *scales, void *packed, int rows, int cols, insg_stream_t stream)
{
    if (!weight || !scales || !packed) return fail(INSG_E_ARG, "repack_umma: null pointer");
    if (rows <= 0 || cols <= 0 || (cols & 127)) return fail(INSG_E_SHAPE, "repack_umma: cols % 128 must be 0");
    const size_t n = size_t((rows + 127) >> 7) * (cols >> 7) * 128;
    repack_umma_kernel<<<unsigned((n + 255) / 256), 256, 0, stream>>>(weight, scales, static_cast<uint8_t *>(packed), rows, cols);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? INSG_OK : cuda_fail(e, "repack_umma launch");
}

} // extern "C"

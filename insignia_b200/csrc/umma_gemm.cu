// MXFP4 weights x many tokens on the 5th-generation tensor cores (tcgen05, sm_100a): prompt passes of more than eight tokens.
//
// y[m][r] = sum_k e2m1(code(r,k)) * 2^(s(r,k/32)-127) * x[m][k]                 (reference: src/mxfp4.cu:41-66, M times)
//
// tcgen05.mma.kind::mxf4.block_scale, weights as the A operand in their native packed E2M1 + UE8M0 form (the tile layout of
// insg_mxfp4_repack_umma, nothing dequantised), accumulators in tensor memory.  The activations are the B operand.
// kind::mxf4 wants E2M1 there too, so each fp32 activation is written as a signed fixed-point number of at least 25 bits (relative to
// the largest element of its group of 32, whose power of two is the group's UE8M0 scale) in base 13 with the digits 0, +-1..+-4, +-6 and
// +-8, every one exact in E2M1: seven digits, where umma_gemv.cu's balanced base 9 takes eight.  Column j * tokens + t of a group holds
// digit j of its token t; the epilogue combines the seven as sum_j 13^j D_j in fp32, which gives the product to ~7e-8 (4096 columns,
// normal inputs; base 9: 8e-8).  A token takes 7 columns of N.
//
// What bounds it: the tensor pipe, and filling shared memory beside it.  A stage multiplies two 128-row weight records (17.4 KB) a CTA with
// the digits of a group of tokens.  Thirty-two tokens (N = 224) fill tensor memory (448 of 512 columns, beside the scale factors) and
// make the most of the weights' bytes; two CTAs then work on four records with one set of digits, of which each fetches and holds half
// (cta_group::2).  24576 x 4096 at 512 tokens, digitize launch included: one CTA a unit 126 us; pairs 121; without the multiplies 83,
// without the copies 106 (332 stages of 448 cycles on the tensor pipe are 78).
//
// Kernels:
//   umma_digitize_kernel  one CTA or more per token: the fused activation prologue (RMSNorm, gates, ...), then the digit
//                         image of the token in global memory, laid out as the shared-memory image the MMA reads
//                         ([k-block][group of tokens][448 bytes x tokens per group, scale blocks], canonical K-major, no swizzle);
//   umma_gemm_kernel      one CTA per SM; with groups of 32 tokens (tokens_per_group) two work together.  The work is the sequence of all (pair of records, token group, k-block) stages;
//                         every CTA takes an equal contiguous share of it (stream-K), so SMs are busy whatever the number
//                         of tiles.  The pair is two row tiles, or the gate and the up tile of the same rows for SwiGLU
//                         (whose epilogue then has both at hand); two CTAs take twice as many tiles, each with its own
//                         rows' sums and epilogue, and the first one issues for both.  A ring of stages, fetched by cp.async.bulk with mbarrier
//                         completion (local, no multicast); one warp issues the scale copies and the MMAs; four epilogue
//                         warps (tensor memory lane = output row) take a run's sums out before the next one multiplies,
//                         while the ring refills.  A unit (pair, group) that lies inside one CTA's share goes straight
//                         through the fused epilogue; one that is cut by a share boundary leaves per-CTA partial sums in
//                         scratch, and the CTA that arrives last (a ticket per cut unit) adds them in share order -- the
//                         result does not depend on which CTA that is -- and runs the epilogue.  Every wait is bounded:
//                         on expiry an error flag is raised and all roles drain.
//   conv_tokens_kernel    the causal convolution + SiLU over consecutive tokens of one sequence (the history runs
//                         through the tokens in order, so it cannot live in a per-unit epilogue).
#include "gemv_prologue.cuh"
#include "host_util.h"
#include "umma_common.cuh"

#include <algorithm>
#include <mutex>

namespace insg {

constexpr int kDigThreads = 256;           // digitize kernel
constexpr int kGemmThreads = 224;          // GEMM kernel: four epilogue warps, the MMA issuer, the producers of weights and of digits
constexpr int kDigits = 7;                 // base-13 digits per activation = N columns per token
constexpr int kGSfaBufs = 4;               // scale-factor column sets cycled by stage (a power of two)
constexpr int kGTmemCols = 512;            // two accumulators of up to 224 columns, weight scale factors [448,480), digit scale factors [480,512)
constexpr int kGMaxStages = 16;
constexpr int kGMaxGrid = 256;             // partial-sum slots and tickets are sized for this many CTAs
constexpr int kSlotFloats = 128 * 32;      // one partial: 128 rows x up to 32 tokens
// A k-block of a token group in the digit image: the digits (kDigits columns x 64 bytes per token; column = digit * tpg + token), then a
// 512-byte scale block per 128 columns.
__host__ __device__ constexpr int digit_bytes(int tpg) { return 64 * kDigits * tpg; }
__host__ __device__ constexpr int digit_block(int tpg) { return digit_bytes(tpg) + (kDigits * tpg + 127) / 128 * 512; }
// CTAs that work on a unit together.  Groups of 32 tokens: two, whose tensor cores each multiply their own rows with all columns and
// read half of the digits each from either one's shared memory; the digits then lie [half of the columns][K-step].
__host__ __device__ constexpr int group_ctas(int tpg) { return tpg == 32 ? 2 : 1; }

// ---- seven digits of an activation -----------------------------------------------------------------------------------------------
// E2M1 holds 0, 1, 2, 3, 4, 6, 8 and 12 halves of either sign.  Of these, {0, +-1, +-2, +-3, +-4, +-6, +-8} has every residue modulo 13
// once (5 = -8, 7 = -6, 9..12 = -4..-1), so every integer has base-13 digits in it, and seven of them hold all |v| <= 4 1/3 * 13^6 =
// 2^24.3: what is left for the seventh is -4..4.  Balanced base 9 takes eight digits for 2^24: an eighth more to multiply and to move.
// Two digits at a time come from a table, with the carry that the negative ones leave to the next two; the halves go into the
// group's scale.
constexpr int kPair = 169, kSixDigits = kPair * kPair * kPair; // 13^2, 13^6
__device__ __forceinline__ uint16_t digit_pair13(int n) // table entry: the codes of the two digits, least significant first, the carry in bit 8
{
    uint32_t r = 0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int m = n % 13;
        const int d = m <= 4 || m == 6 || m == 8 ? m : m - 13, mag = d < 0 ? -d : d;
        r |= uint32_t((mag <= 4 ? mag : mag == 6 ? 5 : 6) | (d < 0 ? 8 : 0)) << (4 * i);
        n = (n - d) / 13;
    }
    return uint16_t(r | uint32_t(n) << 8);
}
// Seven codes of round(x * alpha) (|.| <= 4 1/3 * 13^6), digit j in nibble j.
__device__ __forceinline__ uint32_t digit_codes13(float x, float alpha, const uint16_t *table)
{
    const int v = max(-20916000, min(__float2int_rn(x * alpha), 20916000));
    const uint32_t u = uint32_t(v + 5 * kSixDigits); // a multiple of 13^6: only the seventh digit sees it
    uint32_t q = u / uint32_t(kPair);
    const uint32_t t0 = table[u - uint32_t(kPair) * q], u1 = q + (t0 >> 8);
    q = u1 / uint32_t(kPair);
    const uint32_t t1 = table[u1 - uint32_t(kPair) * q], u2 = q + (t1 >> 8);
    q = u2 / uint32_t(kPair);
    const uint32_t t2 = table[u2 - uint32_t(kPair) * q];
    // what is left + 5 = 1..9 -> codes of -4..4
    const uint32_t last = uint32_t(0x43210'9ABC0ull >> (4 * (q + (t2 >> 8)))) & 15u;
    return (t0 & 0xFFu) | (t1 & 0xFFu) << 8 | (t2 & 0xFFu) << 16 | last << 24;
}
// A group's exponent (umma_common.cuh), one less where its largest magnitude leaves room for a bit more: 2^24 * 1.2422 fits.
__device__ __forceinline__ int group_exponent13(uint32_t max_bits)
{
    const int eb = group_exponent(max_bits);
    return eb - int(eb != 255 && int(max_bits >> 23) == eb && (max_bits & 0x7FFFFFu) < 0x1F0000u);
}
__device__ __forceinline__ uint8_t digit_scale(int eb) { return uint8_t(eb == 255 ? 255 : eb - 22); } // group_scale, times two for the halves

// The digits of one 128-element k-block of token `t` of a group (four elements per lane) and their scales into the block at `blk`.
template <int TPG> __device__ __forceinline__ void store_digits13(float4 x, int t, uint8_t *blk, const uint16_t *table, int lane)
{
    float mx = fmax_nan(fmax_nan(fabsf(x.x), fabsf(x.y)), fmax_nan(fabsf(x.z), fabsf(x.w)));
    mx = fmax_nan(mx, __shfl_xor_sync(0xffffffffu, mx, 1)); // a group of 32 elements = 8 lanes
    mx = fmax_nan(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    mx = fmax_nan(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    const int eb = group_exponent13(__float_as_uint(mx));
    const float alpha = group_alpha(eb);
    const uint32_t c0 = digit_codes13(x.x, alpha, table), c1 = digit_codes13(x.y, alpha, table);
    const uint32_t c2 = digit_codes13(x.z, alpha, table), c3 = digit_codes13(x.w, alpha, table);
    // columns 0, 2, 4, 6 sit in the low nibbles of the four bytes, 1, 3, 5 in the high ones
    const uint32_t e01 = (c0 & 0x0F0F0F0Fu) | ((c1 & 0x0F0F0F0Fu) << 4), e23 = (c2 & 0x0F0F0F0Fu) | ((c3 & 0x0F0F0F0Fu) << 4);
    const uint32_t o01 = ((c0 >> 4) & 0x0F0F0F0Fu) | (c1 & 0xF0F0F0F0u), o23 = ((c2 >> 4) & 0x0F0F0F0Fu) | (c3 & 0xF0F0F0F0u);
    // columns in groups of eight: [half of the groups][K-step][group][k core][column][16 bytes]
    constexpr int kHalves = group_ctas(TPG), kGroups = kDigits * TPG / 8 / kHalves;
    uint8_t *dst = blk + (lane >> 4) * (kGroups * 256) + ((lane >> 3) & 1) * 128 + (t & 7) * 16 + (lane & 7) * 2;
    auto column = [&](int j) { // of digit j
        const int g = j * (TPG / 8) + (t >> 3);
        return dst + g * 256 + (g >= kGroups ? kGroups * 256 : 0);
    };
#pragma unroll
    for (int j = 0; j < 4; j++) {
        *reinterpret_cast<uint16_t *>(column(2 * j)) = uint16_t(__byte_perm(e01, e23, j | ((4 + j) << 4)));
        if (j < 3) *reinterpret_cast<uint16_t *>(column(2 * j + 1)) = uint16_t(__byte_perm(o01, o23, j | ((4 + j) << 4)));
    }
    // scale block: row = column mod 32, then the column quarter, byte = group; a token's columns share the four bytes
    const uint32_t sc = digit_scale(eb);
    const uint32_t w = __shfl_sync(0xffffffffu, sc, 0) | __shfl_sync(0xffffffffu, sc, 8) << 8 | __shfl_sync(0xffffffffu, sc, 16) << 16 | __shfl_sync(0xffffffffu, sc, 24) << 24;
    if (lane < 2) // 16 tokens: columns of even and odd digits are rows t and 16 + t; 32: digits 0..3 and 4..6 are two blocks
        *reinterpret_cast<uint4 *>(blk + digit_bytes(TPG) + (TPG == 16 ? (16 * lane + t) * 16 : 512 * lane + t * 16)) = make_uint4(w, w, w, w);
}

struct GSeg {
    const uint8_t *packed, *packed2;
    float *out;
    float *conv_state;
    const uint16_t *conv_w;
    const float *A_log;
    const uint16_t *dt_bias;
    long long conv_stride; // 0: one sequence (the epilogue stores the raw product, conv_tokens_kernel follows); else token m's history at conv_state + m * stride
    int tile_begin, epilogue, rows;
};

struct GParams {
    const uint8_t *bimg;    // [nkb][ngroups][digit_block(tpg)]
    float *partials;        // [grid][2 cut units][2 records of the pair][tpg / 4][128 rows][4 tokens], a record's part in kSlotFloats
    int *tickets;           // [grid], zero between launches
    int nkb, nseg, total_tiles, stages, ngroups, tokens;
    int total_stages, share, share_rem; // CTA c owns stages [share * c + share_rem * c / G, ...): all products stay in 32 bits
    GSeg seg[4];
    int *error_flag;
};

struct DigitizeParams {
    ProIn pro;
    uint8_t *bimg;
    int *tickets;
    int tokens, ngroups, parts; // a token's digits are written by `parts` CTAs, each a slice of the columns
    int wait_first;             // nothing may be read, and the GEMM may not start, before the launch before this one has ended
};

// `parts` CTAs of eight warps per token slot, each a slice of the k-blocks (slots beyond `tokens` are written as zeros so that their columns
// contribute nothing).  A warp takes a k-block at a time, two on their way at once; everything but the RMSNorm's sum stays inside the warp
// (a head of the gated norm is one k-block), and that sum is the one barrier.  With few tokens a CTA's chain, load to last store, is the
// time, so the CTAs are small enough for four an SM, 592 at once.  With many it is short of no single thing: issue and ALU are some 60 %
// busy, 512 tokens of 12288 columns take 13 % less without the stores and 32 % less without the digits' arithmetic.  Replayed
// alone, sixteen-warp CTAs of a token with eight base-9 digits -> this with four k-blocks on their way -> with two (less code to run through):
//   4096 columns, 16 tokens 2.63 -> 2.64 -> 2.43 us (gated norm 3.93 -> 2.92 -> 2.74), 128: 4.12 -> 4.46 -> 4.30, 512: 10.3 -> 9.7 -> 9.2
//   12288 columns, 16 tokens 3.43 -> 3.20 -> 3.01 us, 128: 7.67 -> 7.96 -> 7.64, 512: 21.0 -> 23.8 -> 22.0
template <int TPG, int PRO>
__global__ void __launch_bounds__(kDigThreads, 4) umma_digitize_kernel(const __grid_constant__ DigitizeParams p)
{
    constexpr int kBatch = 2, kWarps = kDigThreads / 32;
    __shared__ float scratch[kWarps];
    __shared__ uint16_t table[kPair];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < kPair) table[tid] = digit_pair13(tid);
    if (p.wait_first) pdl_wait(); // (calls one behind the other: 24576 x 4096 with 61 tokens 29.6 -> 27.3 us)
    pdl_launch_dependents(); // the GEMM may set itself up and fetch weights meanwhile
    const int m = blockIdx.x / p.parts, part = blockIdx.x - m * p.parts, grp = m / TPG, ms = m - grp * TPG;
    const ProIn &o = p.pro;
    const int nkb = o.cols >> 7, per = (nkb + p.parts - 1) / p.parts, kb0 = part * per, kb1 = min(nkb, kb0 + per);
    const bool live = m < p.tokens, rms = PRO == INSG_PRO_RMSNORM;
    const float *in = o.in + size_t(m) * o.cols + lane * 4;
    uint2 w[kBatch]; // the norm's weights are parameters: asked for before the wait
    auto load_weights = [&](int b0) {
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const int kb = b0 + j * kWarps;
            if (rms && kb < kb1) w[j] = *reinterpret_cast<const uint2 *>(o.norm_w + kb * 128 + lane * 4);
            else if (PRO == INSG_PRO_GATED_RMSNORM) w[j] = *reinterpret_cast<const uint2 *>(o.norm_w + lane * 4);
        }
    };
    load_weights(kb0 + warp);
    pdl_wait();
    if (blockIdx.x == 0)
        for (int i = tid; i < kGMaxGrid; i += kDigThreads) p.tickets[i] = 0;
    float4 x[kBatch], a[kBatch]; // values and what gates them
    auto load = [&](int b0) { // through L2 (see gemv_prologue.cuh)
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const int kb = b0 + j * kWarps, k = kb * 128 + lane * 4;
            x[j] = a[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!live || kb >= kb1) continue;
            x[j] = __ldcg(reinterpret_cast<const float4 *>(in + size_t(kb) * 128));
            const float *gate = o.aux + size_t(m) * 2 * o.cols + (k >> 8) * 512 + 256; // interleaved [head][query 256 | gate 256]
            switch (PRO) {
            case INSG_PRO_GATED_RMSNORM:
            case INSG_PRO_SIGMOID_GATE: a[j] = __ldcg(reinterpret_cast<const float4 *>(o.aux + size_t(m) * o.cols + k)); break;
            case INSG_PRO_SIGMOID_GATE_HEAD0: a[j].x = __ldcg(gate); break;
            case INSG_PRO_SIGMOID_GATE_QPROJ: a[j] = __ldcg(reinterpret_cast<const float4 *>(gate + (k & 255))); break;
            default: break;
            }
        }
    };
    load(kb0 + warp);
    float inv_rms = 1.f;
    if (rms) {
        float ss = 0.f;
        if (p.parts == 1 && nkb <= kBatch * kWarps) { // the row is in the CTA's registers
#pragma unroll
            for (int j = 0; j < kBatch; j++) ss = fmaf(x[j].x, x[j].x, fmaf(x[j].y, x[j].y, fmaf(x[j].z, x[j].z, fmaf(x[j].w, x[j].w, ss))));
        } else if (live) {
#pragma unroll 4
            for (int kb = warp; kb < nkb; kb += kWarps) {
                const float4 v = __ldcg(reinterpret_cast<const float4 *>(in + size_t(kb) * 128));
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            }
        }
        ss = warp_sum(ss);
        if (lane == 0) scratch[warp] = ss;
        __syncthreads(); // and the table
        float tot = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) tot += scratch[w];
        inv_rms = rsqrtf(tot / float(o.cols) + 1e-6f);
    } else {
        __syncthreads(); // the table
    }
    for (int b0 = kb0 + warp; b0 < kb1; b0 += kBatch * kWarps) {
        if (b0 != kb0 + warp) {
            load_weights(b0);
            load(b0);
        }
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const int kb = b0 + j * kWarps;
            if (kb >= kb1) break; // warp-uniform
            float4 v = x[j];
            if (live) {
                auto weigh = [&](float f) {
                    v.x = v.x * f * bf16_bits_to_float(w[j].x & 0xffff);
                    v.y = v.y * f * bf16_bits_to_float(w[j].x >> 16);
                    v.z = v.z * f * bf16_bits_to_float(w[j].y & 0xffff);
                    v.w = v.w * f * bf16_bits_to_float(w[j].y >> 16);
                };
                switch (PRO) {
                case INSG_PRO_RMSNORM: weigh(inv_rms); break;
                case INSG_PRO_GATED_RMSNORM: { // a head is one k-block
                    const float hs = warp_sum(fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w))));
                    weigh(rsqrtf(hs / 128.f + 1e-6f));
                    v.x *= fast_silu(a[j].x); v.y *= fast_silu(a[j].y); v.z *= fast_silu(a[j].z); v.w *= fast_silu(a[j].w);
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
            }
            store_digits13<TPG>(v, ms, p.bimg + (size_t(kb) * p.ngroups + grp) * digit_block(TPG), table, lane);
        }
    }
}

// Causal convolution (kernel 4) + SiLU over `tokens` consecutive tokens of one sequence, in place: io[m][c] holds the raw
// projection on entry and the activation on return; the three-value history per channel is read and left updated.
// (reference: src/qwen_kernels.cu:31, once per token)  The filter is not recursive (out[m] needs raw[m-3..m] only): a CTA
// takes eight channels (one 32-byte sector per row) and 256 tokens at a time, a thread one channel and eight tokens; all
// raw values are in registers before the first result is stored.  1024 CTAs at 8192 channels: 27 -> 6 us at 256 tokens
// against one thread per channel walking the tokens.
constexpr int kConvCh = 8, kConvTok = 8, kConvBlocks = 32;
__global__ void __launch_bounds__(kConvCh * kConvBlocks) conv_tokens_kernel(float *io, float *conv_state, const uint16_t *conv_w, int channels, int tokens)
{
    __shared__ float hist[2][3][kConvCh];
    const int ch = threadIdx.x & (kConvCh - 1), blk = threadIdx.x / kConvCh, c = blockIdx.x * kConvCh + ch;
    const bool on = c < channels;
    pdl_launch_dependents();
    float w0 = 0.f, w1 = 0.f, w2 = 0.f, w3 = 0.f;
    if (on) {
        const uint2 wv = reinterpret_cast<const uint2 *>(conv_w)[c];
        w0 = bf16_bits_to_float(wv.x & 0xffff); w1 = bf16_bits_to_float(wv.x >> 16);
        w2 = bf16_bits_to_float(wv.y & 0xffff); w3 = bf16_bits_to_float(wv.y >> 16);
    }
    pdl_wait();
    if (blk < 3) hist[0][blk][ch] = on ? __ldcg(conv_state + size_t(c) * 3 + blk) : 0.f;
    __syncthreads();
    int cur = 0;
    for (int m0 = 0; m0 < tokens; m0 += kConvTok * kConvBlocks, cur ^= 1) {
        const int first = m0 + blk * kConvTok, end = min(tokens, m0 + kConvTok * kConvBlocks);
        float x[kConvTok + 3]; // raw[first - 3 ..]
#pragma unroll
        for (int j = 0; j < kConvTok + 3; j++) {
            const int m = first + j - 3;
            x[j] = m < m0 ? hist[cur][m - m0 + 3][ch] : (on && m < end) ? __ldcg(io + size_t(m) * channels + c) : 0.f;
        }
        // the chunk's last three raw values (older ones when it is shorter than three) are the next history
#pragma unroll
        for (int j = 0; j < kConvTok + 3; j++) {
            const int m = first + j - 3, i = m - (end - 3);
            if (i >= 0 && i < 3 && (j >= 3 || blk == 0)) hist[cur ^ 1][i][ch] = x[j];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kConvTok; j++)
            if (on && first + j < end) io[size_t(first + j) * channels + c] = fast_silu(fmaf(x[j], w0, fmaf(x[j + 1], w1, fmaf(x[j + 2], w2, x[j + 3] * w3))));
    }
    if (on && blk < 3) conv_state[size_t(c) * 3 + blk] = hist[cur][blk][ch];
}

__device__ __forceinline__ int gseg_of(const GParams &p, int tile)
{
    int s = 0;
#pragma unroll
    for (int i = 1; i < 4; i++)
        if (i < p.nseg && tile >= p.seg[i].tile_begin) s = i;
    return s;
}

// ---- the stream-K schedule ----------------------------------------------------------------------------------------------
// Stage g of the launch: unit = g / nkb = pair * ngroups + group, k-block = g % nkb.  CTA c owns stages [share_begin(c),
// share_begin(c + 1)).  A run = the part of one unit inside one share.
__device__ __forceinline__ int share_begin(const GParams &p, int c, int G) { return p.share * c + (p.share_rem * c) / G; }
__device__ __forceinline__ int cta_of_stage(const GParams &p, int g, int G)
{
    int c = min(G - 1, g / p.share); // share >= 1; the remainder term moves the answer down by a few at most
    while (share_begin(p, c, G) > g) c--;
    while (c + 1 < G && share_begin(p, c + 1, G) <= g) c++;
    return c;
}

struct GRun {
    int len;       // stages
    int unit, kb0;
};
__device__ __forceinline__ GRun run_at(const GParams &p, int g, int end)
{
    GRun r;
    r.unit = g / p.nkb;
    r.len = min((r.unit + 1) * p.nkb, end) - g;
    r.kb0 = g - r.unit * p.nkb;
    return r;
}

// The fused epilogue of one row for the tokens of one group; y[] are finished sums.
// Everything stays in registers (fully unrolled, predicated): with nearly all of the SM's memory configured as shared
// memory, the little L1 that is left cannot hold a stack frame per thread, and spilled arrays would go to L2 and back.
// The switch sits outside the token loops so that a launch runs through one short straight-line piece only.
template <int TPG, bool SWIGLU>
__device__ __forceinline__ void finish_row(const GParams &p, const GSeg &s, int row, int grp, const float (&y)[TPG], const float (&gate)[TPG])
{
    const int m0 = grp * TPG, live = min(TPG, p.tokens - m0);
    float *out = s.out + size_t(m0) * s.rows + row;
    const size_t ld = size_t(s.rows);
    if constexpr (SWIGLU) {
#pragma unroll
        for (int t = 0; t < TPG; t++)
            if (t < live) out[t * ld] = fast_silu(gate[t]) * y[t];
        return;
    }
    switch (s.epilogue) {
    case INSG_EPI_RESIDUAL: {
        float r[TPG];
#pragma unroll
        for (int t = 0; t < TPG; t++) r[t] = t < live ? __ldcg(out + t * ld) : 0.f;
#pragma unroll
        for (int t = 0; t < TPG; t++)
            if (t < live) out[t * ld] = r[t] + y[t];
        break;
    }
    case INSG_EPI_CONV_SILU:
        if (s.conv_stride != 0) { // independent sequences: each token has its own history
            const uint2 wv = reinterpret_cast<const uint2 *>(s.conv_w)[row];
            const float cw0 = bf16_bits_to_float(wv.x & 0xffff), cw1 = bf16_bits_to_float(wv.x >> 16);
            const float cw2 = bf16_bits_to_float(wv.y & 0xffff), cw3 = bf16_bits_to_float(wv.y >> 16);
#pragma unroll
            for (int t = 0; t < TPG; t++) {
                if (t < live) {
                    float *st = s.conv_state + size_t(m0 + t) * s.conv_stride + size_t(row) * 3;
                    const float h0 = __ldcg(st), h1 = __ldcg(st + 1), h2 = __ldcg(st + 2), yv = y[t];
                    st[0] = h1; st[1] = h2; st[2] = yv;
                    out[t * ld] = fast_silu(fmaf(h0, cw0, fmaf(h1, cw1, fmaf(h2, cw2, yv * cw3))));
                }
            }
            break;
        }
        // one sequence: the raw product is stored, the convolution over the tokens follows as its own kernel
        [[fallthrough]];
    case INSG_EPI_STORE:
#pragma unroll
        for (int t = 0; t < TPG; t++)
            if (t < live) out[t * ld] = y[t];
        break;
    case INSG_EPI_BETA:
#pragma unroll
        for (int t = 0; t < TPG; t++)
            if (t < live) out[t * ld] = fast_sigmoid(y[t]);
        break;
    case INSG_EPI_DECAY: {
        const float bias = bf16_bits_to_float(s.dt_bias[row]), a = -__expf(s.A_log[row]);
#pragma unroll
        for (int t = 0; t < TPG; t++) {
            const float z = y[t] + bias;
            if (t < live) out[t * ld] = a * (z > 20.f ? z : log1pf(__expf(z)));
        }
        break;
    }
    default: break;
    }
}

// The sums of the TPG tokens of one accumulator (TMEM lane = row, column = digit * TPG + token), digits combined: least significant
// first, 13^j is exact in fp32.
template <int TPG> __device__ __forceinline__ void load_column_block(uint32_t taddr, uint32_t (&d)[TPG])
{
    static_assert(TPG == 16 || TPG == 32, "columns per load");
    if constexpr (TPG == 32)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                     "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]),
                       "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]),
                       "=r"(d[16]), "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]), "=r"(d[21]), "=r"(d[22]), "=r"(d[23]),
                       "=r"(d[24]), "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]), "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
                     : "r"(taddr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]),
                       "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
                     : "r"(taddr));
}
template <int TPG> __device__ __forceinline__ void load_sums(uint32_t taddr, float (&y)[TPG])
{
    constexpr float kPower[kDigits] = {1.f, 13.f, 169.f, 2197.f, 28561.f, 371293.f, 4826809.f};
#pragma unroll
    for (int t = 0; t < TPG; t++) y[t] = 0.f;
#pragma unroll
    for (int j = 0; j < kDigits; j += 2) { // two digits per wait
        uint32_t d0[TPG], d1[TPG];
        load_column_block<TPG>(taddr + j * TPG, d0);
        if (j + 1 < kDigits) load_column_block<TPG>(taddr + (j + 1) * TPG, d1);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int t = 0; t < TPG; t++) {
            y[t] = fmaf(__uint_as_float(d0[t]), kPower[j], y[t]);
            if (j + 1 < kDigits) y[t] = fmaf(__uint_as_float(d1[t]), kPower[j + 1 < kDigits ? j + 1 : j], y[t]);
        }
    }
}

// The two weight records CTA `rank` of CL multiplies for a unit: row tiles 2 CL u + h CL + rank (h = 0, 1), or the gate and the up tile of
// rows CL u + rank.  Beyond the last tile a CTA of a pair multiplies that one again and leaves no result.
struct PairSrc {
    const uint8_t *a[2];
    int tile[2];
    bool live[2]; // has results
    bool two;     // the unit has a second record (for all of its CTAs)
};
template <int CL, bool SWIGLU> __device__ __forceinline__ PairSrc pair_src(const GParams &p, int u, int rank, int kb)
{
    PairSrc q;
    q.two = SWIGLU || 2 * CL * u + CL < p.total_tiles;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int want = SWIGLU ? CL * u + rank : 2 * CL * u + h * CL + rank;
        q.live[h] = want < p.total_tiles;
        q.tile[h] = min(want, p.total_tiles - 1);
        const GSeg &s = p.seg[gseg_of(p, q.tile[h])];
        q.a[h] = (SWIGLU && h == 1 ? s.packed2 : s.packed) + (size_t(q.tile[h] - s.tile_begin) * p.nkb + kb) * kURec;
    }
    return q;
}

// ---- tcgen05 instructions of one CTA or of a pair (issued by its first CTA) ------------------------------------------------------
template <int CL> __device__ __forceinline__ void g_copy_scales(uint32_t on, uint32_t taddr, uint64_t desc) // CL == 2: in both CTAs, each from its own shared memory
{
    if constexpr (CL == 1) copy_scales_if(on, taddr, desc);
    else asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %2, 0;\n@q tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;\n}" ::"r"(taddr), "l"(desc), "r"(on) : "memory");
}
template <int CL> __device__ __forceinline__ void g_mma(uint32_t on, uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate, uint32_t sa, uint32_t sb)
{
    if constexpr (CL == 1) mma_step_if(on, d, da, db, idesc, accumulate, sa, sb);
    else
        asm volatile("{\n.reg .pred q, r;\nsetp.ne.b32 q, %4, 0;\nsetp.ne.b32 r, %7, 0;\n"
                     "@r tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], q;\n}"
                     ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(uint32_t(accumulate)), "r"(sa), "r"(sb), "r"(on) : "memory");
}
template <int CL> __device__ __forceinline__ void g_commit(uint32_t on, uint64_t *bar) // CL == 2: arrives at both CTAs' barrier
{
    if constexpr (CL == 1) commit_if(on, bar);
    else
        asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %2, 0;\n@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}"
                     ::"r"(smem_u32(bar)), "h"(uint16_t(3)), "r"(on) : "memory");
}
// Arrival at a barrier of the pair's first CTA: what this CTA's copies brought, or that its sums have been taken out of tensor memory.  A
// release of everything, global memory included, waited some 800 cycles a stage; restricted to shared memory, with the issuer's waits acquiring
// at cluster scope, a product takes as long as without any order (24576 x 4096, 512 tokens: 119.4 us either way).
__device__ __forceinline__ void first_arrive(uint64_t *bar) { remote_arrive(map_to_rank(smem_u32(bar), 0)); }
// The issuer's looks at its barriers; with CL == 2 the other CTA arrives there, too.
template <int CL> __device__ __forceinline__ bool g_test(uint64_t *bar, uint32_t parity) { return CL == 1 ? mbar_test(bar, parity) : mbar_test_cluster(bar, parity); }
template <int CL> __device__ __forceinline__ bool g_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag)
{
    return CL == 1 ? mbar_wait(bar, parity, abort_flag) : mbar_wait_cluster(bar, parity, abort_flag);
}

template <int TPG, bool SWIGLU>
__global__ void __launch_bounds__(kGemmThreads, 1) umma_gemm_kernel(const __grid_constant__ GParams p)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int CL = group_ctas(TPG);
    constexpr int kBBlock = digit_block(TPG);                 // the group's digits of one k-block, 7 * TPG columns x 128 k x 4 bit, and their scales
    constexpr int kBDig = digit_bytes(TPG) / CL, kBScales = kBBlock - digit_bytes(TPG); // this CTA's columns; every CTA has all scales
    constexpr int kGStage = 2 * kURec + kBDig + kBScales;     // one ring stage: the CTA's two weight records + the digits both multiply
    constexpr int N = kDigits * TPG;
    constexpr uint32_t kD1Col = TPG == 32 ? 224 : 128, kSfaCol = 448, kSfbCol = 480;
    static_assert(N <= int(kD1Col) && kD1Col + N <= int(kSfaCol) && 8 * kGSfaBufs == int(kSfbCol - kSfaCol) && kSfbCol + 8 * kGSfaBufs == uint32_t(kGTmemCols), "tensor memory");
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nkb = p.nkb, S = p.stages;
    uint8_t *ring = smem;                          // S stages of kGStage bytes
    __shared__ __align__(8) uint64_t full[kGMaxStages], empty[kGMaxStages], dfull, dempty;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort, s_last, s_early[2];

    const int G = int(gridDim.x) / CL, c = int(blockIdx.x) / CL, rank = int(blockIdx.x) % CL;
    const int begin = share_begin(p, c, G), end = share_begin(p, c + 1, G);

    if (tid == 0) {
        for (int i = 0; i < S; i++) {
            mbar_init(&full[i], CL == 2 && rank == 0 ? 3 : 2); // the two producers; in the first CTA of a pair the second one's word for its part, too
            mbar_init(&empty[i], 1);
        }
        mbar_init(&dfull, 1);
        mbar_init(&dempty, 4 * CL);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        if constexpr (CL == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(kGTmemCols));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(kGTmemCols));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (CL == 2) { // the other CTA's barriers and tensor memory
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    pdl_launch_dependents(); // this CTA holds its tensor memory: whatever follows may take an SM as it becomes free
    const uint32_t tmem = s_tmem;
    volatile int *abort_flag = &s_abort;

    if (warp == 5) {
        // ---- producer of the weights: two records per stage ----------------------------------------------------------
        // They do not depend on the launch before this one (the digits do): the first ring is requested at once, by one lane per
        // stage (a bulk copy takes the issuing thread a few hundred cycles).
        // One group of tokens reads a record once.  (Several read it one after the other: with the hint for the last of them 24576 x 4096 with 23
        // tokens takes 21.9 us instead of 20.0.)
        const bool once = TPG == 16 && p.ngroups == 1;
        const uint64_t policy = once_policy();
        auto load_record = [&](uint8_t *dst, const uint8_t *src, uint64_t *bar) {
            if (once) bulk_load_hint(dst, src, kURec, bar, policy);
            else bulk_load(dst, src, kURec, bar);
        };
        const int first = min(S, end - begin);
        if (lane < first) {
            const GRun r = run_at(p, begin + lane, end);
            const PairSrc q = pair_src<CL, SWIGLU>(p, r.unit / p.ngroups, rank, r.kb0);
            uint8_t *dst = ring + size_t(lane) * kGStage;
            mbar_expect_tx(&full[lane], (q.two ? 2 : 1) * kURec);
            load_record(dst, q.a[0], &full[lane]);
            if (q.two) load_record(dst + kURec, q.a[1], &full[lane]);
        }
        __syncwarp();
        // from here on the whole warp walks the loop and one elected lane issues: warp-uniform operands issue twice as fast
        const bool one = elect_one();
        int g = begin + first, st = first == S ? 0 : first;
        uint32_t phase = 0; // of the empty barriers
        bool ok = true, room = g < end && mbar_test(&empty[st], phase);
        while (g < end && ok) {
            const GRun r = run_at(p, g, end);
            const PairSrc q = pair_src<CL, SWIGLU>(p, r.unit / p.ngroups, rank, r.kb0);
            const uint8_t *a0 = q.a[0], *a1 = q.a[1];
            for (int k = 0; k < r.len; k++, a0 += kURec, a1 += kURec) {
                if (!room && !mbar_wait(&empty[st], phase, abort_flag)) { ok = false; break; }
                const int cur = st;
                if (++st == S) { st = 0; phase ^= 1; }
                room = mbar_test(&empty[st], phase);
                if (one) {
                    uint8_t *dst = ring + size_t(cur) * kGStage;
                    mbar_expect_tx(&full[cur], (q.two ? 2 : 1) * kURec);
                    load_record(dst, a0, &full[cur]);
                    if (q.two) load_record(dst + kURec, a1, &full[cur]);
                }
            }
            g += r.len;
        }
    } else if (warp == 6) {
        // ---- producer of the digits: this CTA's columns and all scales -----------------------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("fence.proxy.async.global;" ::: "memory"); // the digits were written by ordinary stores, the bulk copies read them through the async proxy
        auto load = [&](uint8_t *dst, const uint8_t *b, uint64_t *bar) {
            mbar_expect_tx(bar, kBDig + kBScales);
            if constexpr (CL == 1) bulk_load(dst, b, kBBlock, bar);
            else {
                bulk_load(dst, b + rank * kBDig, kBDig, bar);
                bulk_load(dst + kBDig, b + digit_bytes(TPG), kBScales, bar);
            }
        };
        const int first = min(S, end - begin);
        if (lane < first) {
            const GRun r = run_at(p, begin + lane, end);
            const int grp = r.unit % p.ngroups;
            load(ring + size_t(lane) * kGStage + 2 * kURec, p.bimg + (size_t(r.kb0) * p.ngroups + grp) * kBBlock, &full[lane]);
        }
        __syncwarp();
        const bool one = elect_one();
        int g = begin + first, st = first == S ? 0 : first;
        uint32_t phase = 0;
        bool ok = true, room = g < end && mbar_test(&empty[st], phase);
        while (g < end && ok) {
            const GRun r = run_at(p, g, end);
            const uint8_t *b = p.bimg + (size_t(r.kb0) * p.ngroups + r.unit % p.ngroups) * kBBlock;
            const size_t bstep = size_t(p.ngroups) * kBBlock;
            for (int k = 0; k < r.len; k++, b += bstep) {
                if (!room && !mbar_wait(&empty[st], phase, abort_flag)) { ok = false; break; }
                const int cur = st;
                if (++st == S) { st = 0; phase ^= 1; }
                room = mbar_test(&empty[st], phase);
                if (one) load(ring + size_t(cur) * kGStage + 2 * kURec, b, &full[cur]);
            }
            g += r.len;
        }
    } else if (warp == 4 && rank == 1) {
        // ---- the second CTA of a pair tells the first one which of its stages are there ------------------------------
        int st = 0;
        uint32_t phase = 0;
        for (int g = begin; g < end; g++) {
            if (!__all_sync(0xffffffffu, mbar_wait(&full[st], phase, abort_flag))) break; // together: the lanes meet again below
            if (lane == 0) first_arrive(&full[st]);
            __syncwarp();
            if (++st == S) { st = 0; phase ^= 1; }
        }
    } else if (warp == 4) {
        // ---- MMA issuer --------------------------------------------------------------------------------------------------
        // The whole warp walks the loop and one elected lane issues (see umma_gemv.cu: operands in uniform registers); the next
        // stage's barriers are polled before this stage's multiplies go out.
        const uint32_t one = elect_one();
        // E2M1 x E2M1, UE8M0 scales, N columns, M = 128 rows a CTA; K-step s of a block uses scale bytes 2s, 2s+1 of both operands
        constexpr uint32_t idesc0 = (1u << 7) | (1u << 10) | ((uint32_t(N) >> 3) << 17) | (1u << 23) | (uint32_t(128 * CL >> 4) << 24);
        constexpr uint32_t idesc1 = idesc0 | (2u << 29) | (2u << 4);
        const uint64_t da0 = umma_desc(smem_u32(ring), 128, 256), dsf0 = umma_desc(smem_u32(ring) + 8192, 16, 128);
        const uint32_t d0 = tmem, d1 = tmem + kD1Col;
        int st = 0, sfa = 0;
        uint32_t phase = 0;
        bool ok = true, here = g_test<CL>(&full[0], 0);
        int g = begin;
        for (int run = 0; g < end && ok; run++) {
            const GRun r = run_at(p, g, end);
            const bool two = SWIGLU || 2 * CL * (r.unit / p.ngroups) + CL < p.total_tiles;
            // a wait that runs out ends the loop for all lanes: they vote again at the next stage
            ok = __all_sync(0xffffffffu, g_wait<CL>(&dempty, (run & 1) ^ 1, abort_flag)); // the first run passes at once
            if (!ok) break;
#pragma unroll 1
            for (int k = 0; k < r.len; k++) {
                // (Two or four stages behind one look at their barriers, in straight-line code: no faster.  Without the early look at the next stage's
                // 40 tokens of 24576 x 4096 take 24.3 us instead of 23.5, 61 of 12352 x 4096 20.9 instead of 20.1; large products the same.)
                if (!__all_sync(0xffffffffu, here) && !__all_sync(0xffffffffu, g_wait<CL>(&full[st], phase, abort_flag))) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t off = uint64_t(uint32_t(st) * uint32_t(kGStage >> 4));
                const uint64_t da = da0 + off, dsf = dsf0 + off, db = da + uint64_t((2 * kURec) >> 4);
                const uint32_t sa = tmem + kSfaCol + 8 * sfa, sb = tmem + kSfbCol + 8 * sfa;
                uint64_t *back = &empty[st];
                if (++st == S) { st = 0; phase ^= 1; }
                here = g_test<CL>(&full[st], phase);
                const uint32_t second = two ? one : 0u;
                g_copy_scales<CL>(one, sa, dsf);
                g_copy_scales<CL>(second, sa + 4, dsf + (kURec >> 4));
                const uint64_t dsb = dsf + uint64_t((2 * kURec - 8192 + kBDig) >> 4); // 128 columns' scales per copy
                g_copy_scales<CL>(one, sb, dsb);
                if (N > 128) g_copy_scales<CL>(one, sb + 4, dsb + 32);
                g_mma<CL>(one, d0, da, db, idesc0, k > 0, sa, sb); // the run's first MMA overwrites
                g_mma<CL>(second, d1, da + (kURec >> 4), db, idesc0, k > 0, sa + 4, sb);
                g_mma<CL>(one, d0, da + 256, db + (kBDig >> 5), idesc1, true, sa, sb);
                g_mma<CL>(second, d1, da + (kURec >> 4) + 256, db + (kBDig >> 5), idesc1, true, sa + 4, sb);
                g_commit<CL>(one, back);
                sfa = (sfa + 1) & (kGSfaBufs - 1);
            }
            if (ok) g_commit<CL>(one, &dfull);
            g += r.len;
        }
    } else if (warp < 4) {
        // ---- epilogue: tensor-memory lane = row of the tile; digit j of the group's token t = column j * TPG + t ------------
        asm volatile("griddepcontrol.wait;" ::: "memory"); // residual inputs and tickets come from earlier launches
        bool ok = true;
        int g = begin;
        for (int run = 0; g < end && ok; run++) {
            const GRun r = run_at(p, g, end);
            g += r.len;
            const int u = r.unit / p.ngroups, grp = r.unit - u * p.ngroups;
            const int ubegin = r.unit * nkb, uend = ubegin + nkb;
            const bool cut = begin > ubegin || uend > end;
            const int c_first = cut ? cta_of_stage(p, ubegin, G) : c, c_last = cut ? cta_of_stage(p, uend - 1, G) : c;
            // A unit of two parts whose other one is already there (the usual case of a share's last unit, with nothing behind it to hide
            // the trips to L2): this CTA adds it to its own, which it need not store.
            if (tid == 0) {
                int seen = 0;
                if (c_last == c_first + 1) asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.tickets + CL * c_first + rank) : "memory");
                s_early[run & 1] = seen;
            }
            ok = mbar_wait(&dfull, run & 1, abort_flag);
            {   // the 128 epilogue threads go on or give up together (they meet at named barriers below)
                uint32_t all;
                asm volatile("{\n.reg .pred q, r;\nsetp.ne.b32 q, %1, 0;\nbar.red.and.pred r, 1, 128, q;\nselp.u32 %0, 1, 0, r;\n}"
                             : "=r"(all) : "r"(uint32_t(ok)) : "memory");
                ok = all != 0;
            }
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const PairSrc q0 = pair_src<CL, SWIGLU>(p, u, rank, 0);
            const bool has1 = q0.two;
            float y[2][TPG];
            load_sums<TPG>(tmem + (uint32_t(warp * 32) << 16), y[0]);
            if (has1) load_sums<TPG>(tmem + kD1Col + (uint32_t(warp * 32) << 16), y[1]);
            else {
#pragma unroll
                for (int t = 0; t < TPG; t++) y[1][t] = 0.f;
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) { // the issuer sits in the first CTA
                if constexpr (CL == 2) first_arrive(&dempty);
                else mbar_arrive(&dempty);
            }

            auto fetch = [&](int cc, float4 (&q)[2][TPG / 4]) { // a CTA's part of this unit
                const float4 *slot = reinterpret_cast<const float4 *>(p.partials + (size_t(CL * cc + rank) * 2 + (share_begin(p, cc, G) > ubegin ? 0 : 1)) * 2 * kSlotFloats) + tid;
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int t = 0; t < TPG / 4; t++)
                        q[h][t] = h == 0 || has1 ? __ldcg(slot + h * (kSlotFloats / 4) + t * 128) : make_float4(0.f, 0.f, 0.f, 0.f);
            };
            if (cut && s_early[run & 1]) {
                float4 q[2][TPG / 4];
                fetch(c_first + c_last - c, q);
                if (tid == 0) p.tickets[CL * c_first + rank] = 0; // ready for the next launch
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int t = 0; t < TPG / 4; t++) {
                        const float part[4] = {q[h][t].x, q[h][t].y, q[h][t].z, q[h][t].w};
#pragma unroll
                        for (int i = 0; i < 4; i++) y[h][4 * t + i] = (y[h][4 * t + i] + 0.f) + part[i]; // from zero, as below (the sign of a zero)
                    }
            } else if (cut) {
                // ---- a unit cut by a share boundary: leave the partial sums; the CTA that arrives last adds them up ----
                // (A warp's rows lie side by side for each four tokens: with a row's tokens side by side instead every access touches
                // 32 sectors, and 4096 x 4096 with 61 tokens took 35 us instead of 22.)
                const int which = (begin > ubegin) ? 0 : 1; // the unit that contains this share's first stage, or a later one
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (h == 1 && !has1) break;
                    float4 *slot = reinterpret_cast<float4 *>(p.partials + ((size_t(CL * c + rank) * 2 + which) * 2 + h) * kSlotFloats) + tid; // [four tokens][row]
#pragma unroll
                    for (int t = 0; t < TPG / 4; t++)
                        __stcg(slot + t * 128, make_float4(y[h][4 * t], y[h][4 * t + 1], y[h][4 * t + 2], y[h][4 * t + 3]));
                }
                // The barrier makes the 128 threads' partial stores visible to thread 0; its release at GPU scope is cumulative
                // over them, and the last arriver's acquire + the next barrier hand the other CTAs' stores to its 128 readers.
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (tid == 0) {
                    int seen;
                    asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(seen) : "l"(p.tickets + CL * c_first + rank) : "memory");
                    s_last = seen == c_last - c_first;
                    if (s_last) p.tickets[CL * c_first + rank] = 0; // ready for the next launch
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                const bool last = s_last != 0;
                asm volatile("bar.sync 1, 128;" ::: "memory"); // s_last may be rewritten by the next cut unit
                if (!last) continue;
                // the last arriver: add the parts in share order (the sum does not depend on who arrived last), both records
                // of a part at once, so that a part costs one trip to L2
#pragma unroll
                for (int t = 0; t < TPG; t++) y[0][t] = y[1][t] = 0.f;
                float4 q[2][TPG / 4];
                fetch(c_first, q);
                for (int cc = c_first; cc <= c_last; cc++) {
                    float4 nq[2][TPG / 4]; // the next part is on its way while this one is added
                    fetch(min(cc + 1, c_last), nq);
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int t = 0; t < TPG / 4; t++) {
                            y[h][4 * t] += q[h][t].x; y[h][4 * t + 1] += q[h][t].y; y[h][4 * t + 2] += q[h][t].z; y[h][4 * t + 3] += q[h][t].w;
                            q[h][t] = nq[h][t];
                        }
                }
            }
            if constexpr (SWIGLU) {
                const GSeg &s = p.seg[gseg_of(p, q0.tile[0])];
                const int row = (q0.tile[0] - s.tile_begin) * 128 + tid;
                if (q0.live[0] && row < s.rows) finish_row<TPG, SWIGLU>(p, s, row, grp, y[1], y[0]);
            } else {
#pragma unroll 1
                for (int h = 0; h < 2; h++) { // one copy of the code for both records
                    const int tile = h ? q0.tile[1] : q0.tile[0];
                    const GSeg &s = p.seg[gseg_of(p, tile)];
                    const int row = (tile - s.tile_begin) * 128 + tid;
                    if ((h ? q0.live[1] : q0.live[0]) && row < s.rows) finish_row<TPG, SWIGLU>(p, s, row, grp, y[0], y[0]);
#pragma unroll
                    for (int t = 0; t < TPG; t++) y[0][t] = y[1][t];
                }
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (CL == 2) { // nobody leaves while the other CTA may still read its shared memory or arrive at its barriers
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) {
        if constexpr (CL == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kGTmemCols));
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kGTmemCols));
    }
    if (tid == 0 && s_abort && p.error_flag) *p.error_flag = 1;
}

// ---- host side --------------------------------------------------------------------------------------------------------
namespace {
std::mutex g_gemm_attr_mutex;
bool g_gemm_attr_done[64] = {false}; // the shared-memory opt-in is a per-device function attribute

// Tokens per group, 32 of them on pairs of CTAs.  32 take fewer bytes into shared memory for every count beyond 48, the last group's padding
// included.  Where an SM has few stages, every CTA works on parts of cut units and what these cost is the time: 16 tokens make them half as
// large, and up to 48 tokens the weights bound it.  Microseconds replayed with 16 / 32 a group, in brackets the stages an SM has with 16:
//                  24576 x 4096      4096 x 12288      12352 x 4096      10240 x 4096      8192 x 4096       4096 x 4096
//   49..64 tokens  32.7 / 26.4 (83)  24.6 / 24.8 (42)  22.4 / 22.6 (42)  19.1 / 20.7 (35)  18.7 / 19.4 (28)  15.9 / 19.9 (14)
//   65..80         38.1 / 31.3 (104) 27.7 / 26.5 (52)  25.1 / 21.6 (53)  21.3 / 23.1 (43)  19.1 / 20.8 (35)  16.6 / 17.6 (17)
//   96                                                                   24.1 / 23.1 (52)  21.0 / 21.1 (42)  17.5 / 18.4 (21)
//   128                                                                  28.5 / 23.7 (69)  24.7 / 23.2 (55)  19.8 / 19.8 (28)
//   192                                                                                                      22.0 / 22.2 (42)
//   256                                                                                                      25.7 / 24.2 (55)
// With few k-blocks that many stages are whole units, of which only the first and the last are cut: then 32 again, from 2.5 units an SM on
// (16 / 32, in brackets the units): 4096 x 1024, 256 tokens 14.4 / 15.0 (1.7), 12352 x 2048, 100 tokens 19.2 / 18.8 (2.3), 8192 x 2048, 192 tokens
// 21.1 / 19.2 (2.6), 8192 x 1024, 256 tokens 18.2 / 17.4 (3.5), 12352 x 1024, 256 tokens 22.4 / 20.2 (5.3), 24576 x 256, 512 tokens 40.7 / 36.0 (21).
constexpr int kFewStages = 44;
int tokens_per_group(int tokens, long long stages16, int nkb)
{
    return tokens <= 48 || (stages16 <= (long long)kFewStages * sm_count() && 2 * stages16 <= 5ll * nkb * sm_count()) ? 16 : 32;
}
size_t image_bytes(int cols, int tokens) // room for either: groups of 32 take as many bytes as groups of 16 or more
{
    const int tpg = tokens <= 48 ? 16 : 32;
    const size_t groups = size_t(tokens + tpg - 1) / tpg;
    return size_t(cols >> 7) * groups * digit_block(tpg);
}
static_assert(2 * digit_block(16) <= digit_block(32), "a group of 32 has room for two of 16");
// One kernel per prologue: a launch of some ten microseconds runs through little code.
template <int TPG> auto digitize_kernel(int prologue)
{
    switch (prologue) {
    case INSG_PRO_RMSNORM: return umma_digitize_kernel<TPG, INSG_PRO_RMSNORM>;
    case INSG_PRO_GATED_RMSNORM: return umma_digitize_kernel<TPG, INSG_PRO_GATED_RMSNORM>;
    case INSG_PRO_SIGMOID_GATE: return umma_digitize_kernel<TPG, INSG_PRO_SIGMOID_GATE>;
    case INSG_PRO_SIGMOID_GATE_HEAD0: return umma_digitize_kernel<TPG, INSG_PRO_SIGMOID_GATE_HEAD0>;
    case INSG_PRO_SIGMOID_GATE_QPROJ: return umma_digitize_kernel<TPG, INSG_PRO_SIGMOID_GATE_QPROJ>;
    default: return umma_digitize_kernel<TPG, INSG_PRO_PLAIN>;
    }
}
constexpr size_t kPartialBytes = size_t(kGMaxGrid) * 2 * 2 * kSlotFloats * sizeof(float); // [CTA][cut unit][record of the pair]
} // namespace


// digit image | partial sums of cut units | tickets
size_t umma_gemm_scratch(int cols, int tokens)
{
    if (cols <= 0 || (cols & 127) || tokens <= 0) return 0;
    return image_bytes(cols, tokens) + kPartialBytes + kGMaxGrid * sizeof(int);
}

int gemv_umma_launch(const insg_gemv_op *op, cudaStream_t st, const insg_delta_op *step); // 1..8 tokens (umma_gemv.cu)

int gemm_umma_launch(const insg_gemv_op *op, cudaStream_t st)
{
    if (!op || !op->in) return fail(INSG_E_ARG, "gemm: null operand");
    const int tokens = op->tokens;
    if (tokens < 1 || tokens > 4096) return fail(INSG_E_SHAPE, "gemm: 1 <= tokens <= 4096");
    if (op->cols <= 0 || (op->cols & 127) || op->cols > kMaxVec * kProThreads * 4) return fail(INSG_E_SHAPE, "gemm: cols must be a multiple of 128, <= 12288");
    if (op->n_segments < 1 || op->n_segments > 4) return fail(INSG_E_SHAPE, "gemm: 1..4 segments");
    if (op->prologue < 0 || op->prologue >= INSG_PRO_PREPARED) return fail(INSG_E_ARG, "gemm: prologue not available for several tokens");
    if ((op->prologue == INSG_PRO_RMSNORM || op->prologue == INSG_PRO_GATED_RMSNORM) && !op->norm_w) return fail(INSG_E_ARG, "gemm: norm weight missing");
    if (op->prologue >= INSG_PRO_GATED_RMSNORM && !op->aux) return fail(INSG_E_ARG, "gemm: prologue operand missing");
    const size_t need = umma_gemm_scratch(op->cols, tokens);
    if (!op->umma_scratch || op->umma_scratch_bytes < need) return fail(INSG_E_ARG, "gemm: scratch missing or too small (insg_umma_gemm_scratch_bytes)");
    if (reinterpret_cast<uintptr_t>(op->umma_scratch) & 255) return fail(INSG_E_ARG, "gemm: scratch must be 256-byte aligned");
    GParams p = {};
    int tiles = 0, nmat_all = 0;
    for (int i = 0; i < op->n_segments; i++) {
        const insg_gemv_segment &s = op->seg[i];
        if (!s.packed || !s.out || s.rows <= 0) return fail(INSG_E_SHAPE, "gemm: bad segment");
        if (s.epilogue == INSG_EPI_LOGITS) return fail(INSG_E_SHAPE, "gemm: the logits epilogue takes one token");
        if (s.prep) return fail(INSG_E_SHAPE, "gemm: a prepared output carries one token");
        if (s.epilogue == INSG_EPI_SWIGLU && !s.packed2) return fail(INSG_E_ARG, "gemm: SwiGLU needs two matrices");
        if (s.epilogue == INSG_EPI_CONV_SILU && (!s.conv_state || !s.conv_w)) return fail(INSG_E_ARG, "gemm: conv operands missing");
        if (s.epilogue == INSG_EPI_DECAY && (!s.A_log || !s.dt_bias)) return fail(INSG_E_ARG, "gemm: decay operands missing");
        GSeg &g = p.seg[i];
        g.packed = static_cast<const uint8_t *>(s.packed);
        g.packed2 = static_cast<const uint8_t *>(s.packed2);
        g.out = s.out; g.conv_state = s.conv_state; g.conv_w = s.conv_w; g.A_log = s.A_log; g.dt_bias = s.dt_bias;
        g.conv_stride = s.conv_token_stride;
        const int nmat = s.epilogue == INSG_EPI_SWIGLU ? 2 : 1;
        if (nmat_all && nmat_all != nmat) return fail(INSG_E_SHAPE, "gemm: SwiGLU segments cannot be mixed with others");
        nmat_all = nmat;
        g.tile_begin = tiles; tiles += (s.rows + 127) >> 7; g.epilogue = s.epilogue; g.rows = s.rows;
    }
    const int nkb = op->cols >> 7;
    const int tpg = tokens_per_group(tokens, (long long)(nmat_all == 2 ? tiles : (tiles + 1) / 2) * ((tokens + 15) / 16) * nkb, nkb);
    const int ngroups = (tokens + tpg - 1) / tpg;

    DigitizeParams d = {};
    d.pro = ProIn{op->in, op->aux, op->norm_w, nullptr, op->cols, op->prologue};
    d.bimg = static_cast<uint8_t *>(op->umma_scratch);
    d.tokens = tokens;
    d.ngroups = ngroups;
    d.wait_first = !op->pdl;
    // up to four CTAs per SM, a k-block for every warp of theirs at least
    d.parts = std::max(1, std::min(nkb / (kDigThreads / 32), 4 * sm_count() / (ngroups * tpg)));

    p.bimg = d.bimg;
    p.partials = reinterpret_cast<float *>(d.bimg + image_bytes(op->cols, tokens));
    p.tickets = reinterpret_cast<int *>(reinterpret_cast<uint8_t *>(p.partials) + kPartialBytes);
    d.tickets = p.tickets;
    p.nkb = nkb;
    p.nseg = op->n_segments;
    p.ngroups = ngroups;
    p.tokens = tokens;
    p.total_tiles = tiles;
    const int cl = group_ctas(tpg), per_unit = (nmat_all == 2 ? 1 : 2) * cl; // a unit = (row tiles of cl CTAs, token group)
    const long long total = (long long)((tiles + per_unit - 1) / per_unit) * ngroups * nkb;
    if (total > (1ll << 30)) return fail(INSG_E_LIMIT, "gemm: more than 2^30 (tile, group, k-block) stages");
    p.total_stages = int(total);
    p.error_flag = op->error_flag;
    const int stage_bytes = 2 * kURec + digit_block(tpg) - digit_bytes(tpg) + digit_bytes(tpg) / cl;
    p.stages = std::min(kGMaxStages, 224 * 1024 / stage_bytes);
    const size_t smem = size_t(p.stages) * stage_bytes;
    auto kernel = tpg == 16 ? (nmat_all == 2 ? umma_gemm_kernel<16, true> : umma_gemm_kernel<16, false>)
                            : (nmat_all == 2 ? umma_gemm_kernel<32, true> : umma_gemm_kernel<32, false>);
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
        if (dev < 0 || dev >= 64) return fail(INSG_E_LIMIT, "gemm: device ordinal beyond 63");
        std::lock_guard<std::mutex> lock(g_gemm_attr_mutex);
        if (!g_gemm_attr_done[dev]) {
            for (auto k : {umma_gemm_kernel<16, false>, umma_gemm_kernel<16, true>, umma_gemm_kernel<32, false>, umma_gemm_kernel<32, true>})
                if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
            if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(umma gemm)");
            g_gemm_attr_done[dev] = true;
        }
    }
    // the GEMM is the digitize kernel's programmatic dependent: it allocates tensor memory and requests its first weight
    // records while the digits are being written
    int rc = launch(tpg == 16 ? digitize_kernel<16>(op->prologue) : digitize_kernel<32>(op->prologue), dim3(ngroups * tpg * d.parts), dim3(kDigThreads), 0, st, true, d);
    if (rc != INSG_OK) return rc;
    // Every part of a cut unit costs the CTA that adds them a trip to L2, about what a stage takes: few stages go to fewer CTAs,
    // so that a unit is cut into about sqrt(nkb) parts of sqrt(nkb) stages at most.
    int least = 1;
    while (least * least < nkb) least++;
    const int grid = std::max(1, std::min({sm_count() / cl, kGMaxGrid / cl, p.total_stages, std::max(1, p.total_stages / least)})); // of cl CTAs
    p.share = p.total_stages / grid;
    p.share_rem = p.total_stages % grid;
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(unsigned(grid * cl));
        cfg.blockDim = dim3(kGemmThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; // may start while the digits are being written
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = unsigned(cl);
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = cl > 1 ? 2 : 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
        if (e != cudaSuccess) return cuda_fail(e, "umma gemm launch");
    }
    for (int i = 0; i < op->n_segments; i++) {
        const insg_gemv_segment &s = op->seg[i];
        if (s.epilogue == INSG_EPI_CONV_SILU && s.conv_token_stride == 0) { // one sequence: the history runs through the tokens
            rc = launch(conv_tokens_kernel, dim3((s.rows + kConvCh - 1) / kConvCh), dim3(kConvCh * kConvBlocks), 0, st, op->pdl != 0, s.out, s.conv_state, s.conv_w, s.rows, tokens);
            if (rc != INSG_OK) return rc;
        }
    }
    return INSG_OK;
}

} // namespace insg

using namespace insg;

extern "C" {


size_t insg_umma_gemm_scratch_bytes(int cols, int tokens) { return umma_gemm_scratch(cols, tokens); }

int insg_mxfp4_gemm_umma(const void *packed_umma, const float *x, float *y, int rows, int cols, int M, void *scratch, size_t scratch_bytes,
                         insg_stream_t stream)
{
    insg_gemv_op op = {};
    op.in = x;
    op.cols = cols;
    op.prologue = INSG_PRO_PLAIN;
    op.n_segments = 1;
    op.seg[0].packed = packed_umma;
    op.seg[0].out = y;
    op.seg[0].rows = rows;
    op.seg[0].epilogue = INSG_EPI_STORE;
    op.tokens = M;
    op.layout = 1;
    op.umma_scratch = scratch;
    op.umma_scratch_bytes = scratch_bytes;
    if (M < 1) return fail(INSG_E_SHAPE, "gemm: 1 <= tokens <= 4096");
    return M <= 8 ? gemv_umma_launch(&op, stream, nullptr) : gemm_umma_launch(&op, stream);
}

} // extern "C"

// Gated DeltaNet single-token step for sm_100a.
//
// Recurrence (reference: src/deltanet.cu:4-13), per value head h with key head kh = h>>1:
//   qh = q * rsqrt(sum q^2 + 1e-6) / sqrt(128),  kh_ = k * rsqrt(sum k^2 + 1e-6),  d = exp(g_h)
//   mem_v  = sum_i S[i][v] * d * kh_[i]
//   dl_v   = (v_v - mem_v) * beta_h
//   S[i][v] = S[i][v] * d + kh_[i] * dl_v
//   out_v  = sum_i S[i][v] * qh[i]
// State layout fp32 [head][k=128][v=128], v contiguous.
//
// The reference reads the 64 KiB head state twice and writes it once from global
// memory with 32 CTAs.  Columns v are independent, so here each head is cut into
// 4 slices of 32 columns (128 CTAs); a CTA pulls its 16 KiB slice into registers
// once (coalesced 128-byte row segments, issued before the dependent-launch wait
// because the state was last written a whole token ago), does both reductions
// over k on chip, and writes the slice back once: 2 x 2 MiB of traffic per layer.
// The step is a latency chain, so it is kept short: all inputs are requested
// together, every warp normalises q and k for itself, and only the two sums over
// the eight warps cross a CTA barrier.
#include "common.cuh"
#include "host_util.h"
#include "umma_common.cuh"

namespace insg {

constexpr int kDnThreads = 256;
constexpr int kSlices = 4; // 32 columns each

// `tokens` consecutive steps of the sequence in one launch: the slice stays in registers from step to step and is
// written back once; q/k/v of step m are at + m * qkv_stride, g/beta at + m * 32, the output at + m * 4096.
// For one step the chain from the inputs to the stored state counts, not the arithmetic: eight warps hold rows kr + 32 j of
// 32 columns (whole 128-byte row segments), and the sums cross the warps through shared memory: 2.5 us against 2.9 with the
// warp-local columns of the kernel below, whose 8-byte accesses to the state cost a decoded token 1316 us instead of 1214.
// Sums are taken in that kernel's order: over j, the rows 4 kq + 0..3 as (0 + 2) + (1 + 3), then the eight kq (here the warps)
// in a tree.
__global__ void __launch_bounds__(kDnThreads) deltanet_step_kernel(float *__restrict__ state, const float *__restrict__ q16,
                                                                   const float *__restrict__ k16, const float *__restrict__ v32,
                                                                   const float *__restrict__ g32, const float *__restrict__ beta32,
                                                                   float *__restrict__ out32, int tokens, int qkv_stride, long long state_stride,
                                                                   float *__restrict__ state_first, float *__restrict__ state_last, int wait_first)
{
    __shared__ __align__(16) float s_qk[8][2][128]; // per warp: its own copy of the normalised q and k (no block barrier)
    __shared__ __align__(16) float s_part[2][8][32]; // per-warp partial sums over k: [0] memory read-out, [1] output

    const int head = blockIdx.x / kSlices, slice = blockIdx.x % kSlices, kh = head >> 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int vq = tid & 7, kr = tid >> 3; // float4 column group, k row (rows kr, kr+32, kr+64, kr+96)
    const int v0 = slice * 32 + vq * 4;

    if (wait_first) pdl_wait(); // the launch before this one may have written the state; what follows may start when this one has waited
    pdl_launch_dependents();

    // blockIdx.y: independent sequence of a decode batch (its own state, its own inputs and outputs)
    const int seq = blockIdx.y;
    q16 += size_t(seq) * qkv_stride; k16 += size_t(seq) * qkv_stride; v32 += size_t(seq) * qkv_stride;
    g32 += seq * 32; beta32 += seq * 32; out32 += size_t(seq) * 4096;
    float *S = state + size_t(seq) * state_stride + size_t(head) * 128 * 128;
    float4 cell[4];
#pragma unroll
    for (int j = 0; j < 4; j++) cell[j] = __ldcg(reinterpret_cast<const float4 *>(S + size_t(kr + 32 * j) * 128 + v0));

    pdl_wait();

    // Every dependent input of a step is requested at once; with several steps the next step's inputs are requested
    // before this step's arithmetic (they do not depend on it), so only the first step waits for a load.
    // Each warp reads the whole q and k of the key head (four values per lane) and normalises them itself: L2 norms
    // over 128 with eps added to the sum, as the reference.
    float4 nq4 = __ldcg(reinterpret_cast<const float4 *>(q16 + kh * 128) + lane);
    float4 nk4 = __ldcg(reinterpret_cast<const float4 *>(k16 + kh * 128) + lane);
    float4 nv4 = __ldcg(reinterpret_cast<const float4 *>(v32 + head * 128 + slice * 32) + vq); // this thread's columns
    float ng = __ldcg(g32 + head), nbeta = __ldcg(beta32 + head);
    for (int step = 0; step < tokens; step++, q16 += qkv_stride, k16 += qkv_stride, v32 += qkv_stride, g32 += 32, beta32 += 32, out32 += 4096) {
        __syncwarp(); // the previous step's reads of this warp's q/k copy are done
        const float4 q4 = nq4, k4 = nk4, v4 = nv4;
        const float g_in = ng, beta = nbeta;
        if (step + 1 < tokens) {
            nq4 = __ldcg(reinterpret_cast<const float4 *>(q16 + qkv_stride + kh * 128) + lane);
            nk4 = __ldcg(reinterpret_cast<const float4 *>(k16 + qkv_stride + kh * 128) + lane);
            nv4 = __ldcg(reinterpret_cast<const float4 *>(v32 + qkv_stride + head * 128 + slice * 32) + vq);
            ng = __ldcg(g32 + 32 + head);
            nbeta = __ldcg(beta32 + 32 + head);
        }
        const float qn = warp_sum(fmaf(q4.x, q4.x, fmaf(q4.y, q4.y, fmaf(q4.z, q4.z, q4.w * q4.w))));
        const float kn = warp_sum(fmaf(k4.x, k4.x, fmaf(k4.y, k4.y, fmaf(k4.z, k4.z, k4.w * k4.w))));
        const float qs = rsqrtf(qn + 1e-6f) * 0.08838834764831845f, ks = rsqrtf(kn + 1e-6f);
        reinterpret_cast<float4 *>(s_qk[warp][0])[lane] = make_float4(q4.x * qs, q4.y * qs, q4.z * qs, q4.w * qs);
        reinterpret_cast<float4 *>(s_qk[warp][1])[lane] = make_float4(k4.x * ks, k4.y * ks, k4.z * ks, k4.w * ks);
        __syncwarp();
        float qq[4], kk[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            qq[j] = s_qk[warp][0][kr + 32 * j];
            kk[j] = s_qk[warp][1][kr + 32 * j];
        }
        const float decay = expf(g_in);

        // mem_v = sum_i S * k (times d below)
        float4 pm = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            pm.x = fmaf(cell[j].x, kk[j], pm.x);
            pm.y = fmaf(cell[j].y, kk[j], pm.y);
            pm.z = fmaf(cell[j].z, kk[j], pm.z);
            pm.w = fmaf(cell[j].w, kk[j], pm.w);
        }
        // a warp holds 4 k-rows (lane>>3) x 8 column groups: fold the rows, then every thread folds the 8 warps itself
#pragma unroll
        for (int m = 16; m >= 8; m >>= 1) {
            pm.x += __shfl_xor_sync(0xffffffffu, pm.x, m);
            pm.y += __shfl_xor_sync(0xffffffffu, pm.y, m);
            pm.z += __shfl_xor_sync(0xffffffffu, pm.z, m);
            pm.w += __shfl_xor_sync(0xffffffffu, pm.w, m);
        }
        if (lane < 8) *reinterpret_cast<float4 *>(&s_part[0][warp][lane * 4]) = pm;
        __syncthreads();
        float4 t[8];
#pragma unroll
        for (int w = 0; w < 8; w++) t[w] = *reinterpret_cast<const float4 *>(&s_part[0][w][vq * 4]);
#pragma unroll
        for (int n = 1; n < 8; n <<= 1) // pairs of warps, then of pairs
#pragma unroll
            for (int w = 0; w < 8; w += 2 * n) { t[w].x += t[w + n].x; t[w].y += t[w + n].y; t[w].z += t[w + n].z; t[w].w += t[w + n].w; }
        const float4 mem = t[0];
        const float4 dl = make_float4(fmaf(-mem.x, decay, v4.x) * beta, fmaf(-mem.y, decay, v4.y) * beta, fmaf(-mem.z, decay, v4.z) * beta,
                                      fmaf(-mem.w, decay, v4.w) * beta);

        // S = S*d + k*delta ; out_v = sum_i S * q
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
            // the state after the last step goes to state_last (default: in place); a speculative verify pass also keeps the
            // state after its first step (state_first), which is the one to continue from when the second token is rejected
            if (step == tokens - 1) *reinterpret_cast<float4 *>((state_last ? state_last + size_t(head) * 128 * 128 : S) + size_t(kr + 32 * j) * 128 + v0) = cell[j];
            else if (step == 0 && state_first) *reinterpret_cast<float4 *>(state_first + size_t(head) * 128 * 128 + size_t(kr + 32 * j) * 128 + v0) = cell[j];
        }
#pragma unroll
        for (int m = 16; m >= 8; m >>= 1) {
            po.x += __shfl_xor_sync(0xffffffffu, po.x, m);
            po.y += __shfl_xor_sync(0xffffffffu, po.y, m);
            po.z += __shfl_xor_sync(0xffffffffu, po.z, m);
            po.w += __shfl_xor_sync(0xffffffffu, po.w, m);
        }
        if (lane < 8) *reinterpret_cast<float4 *>(&s_part[1][warp][lane * 4]) = po;
        __syncthreads();
        if (tid < 32) {
            float o[8];
#pragma unroll
            for (int w = 0; w < 8; w++) o[w] = s_part[1][w][tid];
            out32[head * 128 + slice * 32 + tid] = ((o[0] + o[1]) + (o[2] + o[3])) + ((o[4] + o[5]) + (o[6] + o[7]));
        }
    }
}

// ---- the same arithmetic inside a warp, for many steps ------------------------------------------------------------------------
// A warp owns eight columns: lane = (k part kq = lane & 7) x (column pair lane >> 3), 16 rows (32 j + 4 kq + 0..3) of two columns
// per lane.  Rows go in pairs through the packed fp32 instructions of sm_100 (two lanes of arithmetic per issue), so that a
// step of a warp is 16 packed multiply-adds three times over; a sum over k is three shuffles, and nothing crosses a warp.
// (Four columns and eight warps: 107 us for 512 steps against 97.)
struct DnCells {
    unsigned long long c[2][8]; // [column of the pair][row pair 2 j + h]
};
__device__ __forceinline__ void dn_load(DnCells &s, const float *S, int lane) // S: the warp's first column
{
    const float *base = S + size_t((lane & 7) * 4) * 128 + (lane >> 3) * 2;
    float2 x[16];
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = __ldcg(reinterpret_cast<const float2 *>(base + size_t((i >> 2) * 32 + (i & 3)) * 128));
#pragma unroll
    for (int i = 0; i < 8; i++) {
        s.c[0][i] = pack2(x[2 * i].x, x[2 * i + 1].x);
        s.c[1][i] = pack2(x[2 * i].y, x[2 * i + 1].y);
    }
}
__device__ __forceinline__ void dn_store(const DnCells &s, float *S, int lane)
{
    float *base = S + size_t((lane & 7) * 4) * 128 + (lane >> 3) * 2;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float2 a = unpack2(s.c[0][i]), b = unpack2(s.c[1][i]);
        float *p = base + size_t((i >> 1) * 32 + (i & 1) * 2) * 128;
        *reinterpret_cast<float2 *>(p) = make_float2(a.x, b.x);
        *reinterpret_cast<float2 *>(p + 128) = make_float2(a.y, b.y);
    }
}
// A lane's 16 values of a 128-vector in shared memory, as row pairs.
__device__ __forceinline__ void dn_vector(unsigned long long (&v)[8], const float *s, int lane)
{
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(s + 32 * j + (lane & 7) * 4);
        v[2 * j] = u.x;
        v[2 * j + 1] = u.y;
    }
}
// This lane's part of sum_k cells * w for its two columns.
__device__ __forceinline__ float2 dn_products(const DnCells &s, const unsigned long long (&w)[8])
{
    float r[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        unsigned long long a = mul2(s.c[c][0], w[0]), b = mul2(s.c[c][1], w[1]);
#pragma unroll
        for (int i = 2; i < 8; i += 2) {
            a = fma2(s.c[c][i], w[i], a);
            b = fma2(s.c[c][i + 1], w[i + 1], b);
        }
        const float2 t = unpack2(add2(a, b));
        r[c] = t.x + t.y;
    }
    return make_float2(r[0], r[1]);
}
// The whole sum of this lane's own column (column lane & 1 of its pair).
__device__ __forceinline__ float dn_fold(float2 p, int lane)
{
    const bool odd = lane & 1;
    float x = (odd ? p.y : p.x) + __shfl_xor_sync(0xffffffffu, odd ? p.x : p.y, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    return x;
}
// S = S d + k (v - d S k) beta; v, and the result of dn_products(s, k) folded, are those of the lane's own column.
__device__ __forceinline__ void dn_update(DnCells &s, const unsigned long long (&k)[8], float mem, float v, float decay, float beta, int lane)
{
    const float own = fmaf(-mem, decay, v) * beta, other = __shfl_xor_sync(0xffffffffu, own, 1);
    const float d0 = (lane & 1) ? other : own, d1 = (lane & 1) ? own : other;
    const unsigned long long dd = pack2(decay, decay), e0 = pack2(d0, d0), e1 = pack2(d1, d1);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        s.c[0][i] = fma2(k[i], e0, mul2(s.c[0][i], dd));
        s.c[1][i] = fma2(k[i], e1, mul2(s.c[1][i], dd));
    }
}

// The recurrence over many consecutive steps (a prompt pass), bit-identical to single steps: the state stays in the registers of four warps, which find
// everything that does not depend on it in shared memory: four more warps normalise q and k and fetch v, beta and exp(g) for
// the next kDnBlock steps meanwhile.  A step is a latency chain (products, three shuffles, update) of some 370 cycles (512 steps 97 us) with no
// barrier in it; the fold of step t's output runs beside step t + 1's.  (With the k sum cut over eight warps and a CTA barrier
// in every step, and the inputs prepared between the blocks: 0.61 us a step.)
constexpr int kDnBlock = 16;
struct DnInputs {
    float q[kDnBlock][128], k[kDnBlock][128], v[kDnBlock][32], decay[kDnBlock], beta[kDnBlock];
};

__global__ void __launch_bounds__(kDnThreads, 1) deltanet_steps_kernel(float *__restrict__ state, const float *__restrict__ q16,
                                                                           const float *__restrict__ k16, const float *__restrict__ v32,
                                                                           const float *__restrict__ g32, const float *__restrict__ beta32,
                                                                           float *__restrict__ out32, int tokens, int qkv_stride, int wait_first)
{
    __shared__ __align__(16) DnInputs s_in[2];
    const int head = blockIdx.x / kSlices, slice = blockIdx.x % kSlices, kh = head >> 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

    if (wait_first) pdl_wait(); // (64 steps a call, one behind the other: 16.4 -> 15.1 us)
    pdl_launch_dependents();
    const int col = slice * 32 + (warp & 3) * 8, in = (warp & 3) * 8 + (lane >> 3) * 2 + (lane & 1);
    float *S = state + size_t(head) * 128 * 128 + col;
    DnCells cells;
    if (warp < 4) dn_load(cells, S, lane);
    pdl_wait();

    constexpr int kEach = kDnBlock / 4; // steps per preparing warp
    auto prepare = [&](int base, DnInputs &d) {
        float4 q4[kEach], k4[kEach], x4[kEach];
        float gs[kEach];
#pragma unroll
        for (int i = 0; i < kEach; i++) {
            const int s = (warp & 3) + 4 * i;
            q4[i] = k4[i] = x4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            gs[i] = 0.f;
            if (base + s < tokens) {
                const size_t off = size_t(base + s) * qkv_stride;
                q4[i] = __ldcg(reinterpret_cast<const float4 *>(q16 + off + kh * 128) + lane);
                k4[i] = __ldcg(reinterpret_cast<const float4 *>(k16 + off + kh * 128) + lane);
                if (lane < 8) x4[i] = __ldcg(reinterpret_cast<const float4 *>(v32 + off + head * 128 + slice * 32) + lane);
                else if (lane == 8) gs[i] = __ldcg(g32 + size_t(base + s) * 32 + head);
                else if (lane == 9) gs[i] = __ldcg(beta32 + size_t(base + s) * 32 + head);
            }
        }
#pragma unroll
        for (int i = 0; i < kEach; i++) {
            const int s = (warp & 3) + 4 * i;
            const float qn = warp_sum(fmaf(q4[i].x, q4[i].x, fmaf(q4[i].y, q4[i].y, fmaf(q4[i].z, q4[i].z, q4[i].w * q4[i].w))));
            const float kn = warp_sum(fmaf(k4[i].x, k4[i].x, fmaf(k4[i].y, k4[i].y, fmaf(k4[i].z, k4[i].z, k4[i].w * k4[i].w))));
            const float qs = rsqrtf(qn + 1e-6f) * 0.08838834764831845f, ks = rsqrtf(kn + 1e-6f);
            reinterpret_cast<float4 *>(d.q[s])[lane] = make_float4(q4[i].x * qs, q4[i].y * qs, q4[i].z * qs, q4[i].w * qs);
            reinterpret_cast<float4 *>(d.k[s])[lane] = make_float4(k4[i].x * ks, k4[i].y * ks, k4[i].z * ks, k4[i].w * ks);
            if (lane < 8) reinterpret_cast<float4 *>(d.v[s])[lane] = x4[i];
            else if (lane == 8) d.decay[s] = expf(gs[i]);
            else if (lane == 9) d.beta[s] = gs[i];
        }
    };
    if (warp >= 4) prepare(0, s_in[0]);
    __syncthreads();
    float *out = out32 + head * 128 + slice * 32 + in;
    float2 po = make_float2(0.f, 0.f);
    for (int base = 0, b = 0; base < tokens; base += kDnBlock, b ^= 1) {
        if (warp >= 4) {
            if (base + kDnBlock < tokens) prepare(base + kDnBlock, s_in[b ^ 1]);
        } else {
            const DnInputs &d = s_in[b];
            const int n = min(kDnBlock, tokens - base);
            unsigned long long q[8], k[8];
            dn_vector(k, d.k[0], lane);
            float v = d.v[0][in], decay = d.decay[0], beta = d.beta[0];
#pragma unroll 4
            for (int s = 0; s < n; s++) {
                const int next = min(s + 1, kDnBlock - 1); // what the next step needs is requested a step ahead
                unsigned long long nk[8];
                dn_vector(nk, d.k[next], lane);
                const float nv = d.v[next][in], ndecay = d.decay[next], nbeta = d.beta[next];
                dn_vector(q, d.q[s], lane);
                const float2 pm = dn_products(cells, k);
                const float mem = dn_fold(pm, lane), o = dn_fold(po, lane); // po: the previous step's output
                if (base + s > 0 && (lane & 7) < 2) out[size_t(base + s - 1) * 4096] = o;
                dn_update(cells, k, mem, v, decay, beta, lane);
                po = dn_products(cells, q);
#pragma unroll
                for (int i = 0; i < 8; i++) k[i] = nk[i];
                v = nv; decay = ndecay; beta = nbeta;
            }
        }
        __syncthreads();
    }
    if (warp < 4) {
        const float o = dn_fold(po, lane);
        if ((lane & 7) < 2) out[size_t(tokens - 1) * 4096] = o;
        dn_store(cells, S, lane);
    }
}

// One step of several sequences (a decode batch), which also leaves the out projection's input: the gated RMSNorm over the head
// (src/qwen_kernels.cu:5) as the digit image of the tcgen05 kernel.  With three sequences or more there are enough heads to
// fill the device without slicing them, and a CTA that holds a whole head normalises its output without asking anybody (four
// slices exchanging their sums through a cluster took 16 us at eight sequences, this form 6; the out projection's own
// conversion, done again by each of its clusters, 6 us more than taking the image).  A warp holds 16 rows of the state, a lane four columns: the
// sums over k need no shuffles, only one pass over the eight warps' partials.
struct DnGate {
    const float *z;          // [sequences][4096]
    const uint16_t *norm_w;  // bf16 [128]
    uint8_t *image;
    int slots;
};
__global__ void __launch_bounds__(kDnThreads, 2) deltanet_heads_kernel(float *__restrict__ state, long long state_stride, const float *__restrict__ q16,
                                                                       const float *__restrict__ k16, const float *__restrict__ v32,
                                                                       const float *__restrict__ g32, const float *__restrict__ beta32,
                                                                       float *__restrict__ out32, int qkv_stride, const DnGate gate)
{
    __shared__ __align__(16) float s_qk[8][2][128];
    __shared__ __align__(16) float4 s_part[2][8][32];
    __shared__ float s_ss[4];
    __shared__ uint8_t s_lut[84];
    const int head = blockIdx.x, seq = blockIdx.y, kh = head >> 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    pdl_launch_dependents();
    float *S = state + size_t(seq) * state_stride + size_t(head) * 128 * 128 + lane * 4;
    float4 cell[16]; // rows warp + 8 j
#pragma unroll
    for (int j = 0; j < 16; j++) cell[j] = __ldcg(reinterpret_cast<const float4 *>(S + size_t(warp + 8 * j) * 128));
    if (tid < 81) s_lut[tid] = digit_pair_code(tid);
    const float gw = tid < 128 ? bf16_bits_to_float(gate.norm_w[tid]) : 0.f;
    pdl_wait();
    const size_t in = size_t(seq) * qkv_stride;
    const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(q16 + in + kh * 128) + lane);
    const float4 k4 = __ldcg(reinterpret_cast<const float4 *>(k16 + in + kh * 128) + lane);
    const float4 v4 = __ldcg(reinterpret_cast<const float4 *>(v32 + in + head * 128) + lane);
    const float g_in = __ldcg(g32 + seq * 32 + head), beta = __ldcg(beta32 + seq * 32 + head);
    const float zv = tid < 128 ? __ldcg(gate.z + size_t(seq) * 4096 + head * 128 + tid) : 0.f;
    const float qn = warp_sum(fmaf(q4.x, q4.x, fmaf(q4.y, q4.y, fmaf(q4.z, q4.z, q4.w * q4.w))));
    const float kn = warp_sum(fmaf(k4.x, k4.x, fmaf(k4.y, k4.y, fmaf(k4.z, k4.z, k4.w * k4.w))));
    const float qs = rsqrtf(qn + 1e-6f) * 0.08838834764831845f, ks = rsqrtf(kn + 1e-6f);
    reinterpret_cast<float4 *>(s_qk[warp][0])[lane] = make_float4(q4.x * qs, q4.y * qs, q4.z * qs, q4.w * qs);
    reinterpret_cast<float4 *>(s_qk[warp][1])[lane] = make_float4(k4.x * ks, k4.y * ks, k4.z * ks, k4.w * ks);
    __syncwarp();
    const float decay = expf(g_in);
    float4 pm = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 16; j++) { // mem_v = sum_i (S*d) * k
        const float kk = s_qk[warp][1][warp + 8 * j];
        cell[j].x *= decay; cell[j].y *= decay; cell[j].z *= decay; cell[j].w *= decay;
        pm.x = fmaf(cell[j].x, kk, pm.x);
        pm.y = fmaf(cell[j].y, kk, pm.y);
        pm.z = fmaf(cell[j].z, kk, pm.z);
        pm.w = fmaf(cell[j].w, kk, pm.w);
    }
    s_part[0][warp][lane] = pm;
    __syncthreads();
    float4 mem = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < 8; w++) {
        const float4 t = s_part[0][w][lane];
        mem.x += t.x; mem.y += t.y; mem.z += t.z; mem.w += t.w;
    }
    const float4 dl = make_float4((v4.x - mem.x) * beta, (v4.y - mem.y) * beta, (v4.z - mem.z) * beta, (v4.w - mem.w) * beta);
    float4 po = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 16; j++) { // S = S*d + k*delta ; out_v = sum_i S * q
        const float kk = s_qk[warp][1][warp + 8 * j], qq = s_qk[warp][0][warp + 8 * j];
        cell[j].x = fmaf(kk, dl.x, cell[j].x);
        cell[j].y = fmaf(kk, dl.y, cell[j].y);
        cell[j].z = fmaf(kk, dl.z, cell[j].z);
        cell[j].w = fmaf(kk, dl.w, cell[j].w);
        po.x = fmaf(cell[j].x, qq, po.x);
        po.y = fmaf(cell[j].y, qq, po.y);
        po.z = fmaf(cell[j].z, qq, po.z);
        po.w = fmaf(cell[j].w, qq, po.w);
        *reinterpret_cast<float4 *>(S + size_t(warp + 8 * j) * 128) = cell[j];
    }
    s_part[1][warp][lane] = po;
    __syncthreads();
    float o = 0.f;
    if (tid < 128) { // column tid of the head
        const float *part = reinterpret_cast<const float *>(s_part[1]);
#pragma unroll
        for (int w = 0; w < 8; w++) o += part[w * 128 + tid];
        out32[size_t(seq) * 4096 + head * 128 + tid] = o;
        const float ss = warp_sum(o * o);
        if (lane == 0) s_ss[warp] = ss;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const float inv = rsqrtf((s_ss[0] + s_ss[1] + s_ss[2] + s_ss[3]) / 128.f + 1e-6f);
        group_digits(o * inv * gw * fast_silu(zv), gate.slots, seq, gate.image, head * 4 + warp, s_lut, lane);
    }
}

} // namespace insg

using namespace insg;

extern "C" int insg_deltanet_decode(float *state, const float *q16, const float *k16, const float *v32, const float *g32,
                                    const float *beta32, float *out32, int pdl, insg_stream_t stream)
{
    if (!state || !q16 || !k16 || !v32 || !g32 || !beta32 || !out32) return fail(INSG_E_ARG, "deltanet: null pointer");
    return launch(deltanet_step_kernel, dim3(32 * kSlices), dim3(kDnThreads), 0, stream, true, state, q16, k16, v32, g32,
                  beta32, out32, 1, 0, 0ll, nullptr, nullptr, pdl == 0);
}

extern "C" int insg_deltanet_decode_tokens(float *state, const float *q16, const float *k16, const float *v32, const float *g32,
                                           const float *beta32, float *out32, int tokens, int qkv_stride, int pdl,
                                           insg_stream_t stream)
{
    if (!state || !q16 || !k16 || !v32 || !g32 || !beta32 || !out32) return fail(INSG_E_ARG, "deltanet: null pointer");
    if (tokens < 1 || tokens > INSG_DELTANET_MAX_TOKENS || qkv_stride < 0) return fail(INSG_E_SHAPE, "deltanet: 1..1024 tokens per launch");
    if (tokens == 1)
        return launch(deltanet_step_kernel, dim3(32 * kSlices), dim3(kDnThreads), 0, stream, true, state, q16, k16, v32, g32, beta32,
                      out32, 1, qkv_stride, 0ll, nullptr, nullptr, pdl == 0);
    return launch(deltanet_steps_kernel, dim3(32 * kSlices), dim3(kDnThreads), 0, stream, true, state, q16, k16, v32, g32, beta32,
                  out32, tokens, qkv_stride, pdl == 0);
}

extern "C" int insg_deltanet_decode_verify(const float *state, float *state_first, float *state_second, const float *q16, const float *k16,
                                           const float *v32, const float *g32, const float *beta32, float *out32, int qkv_stride, int pdl,
                                           insg_stream_t stream)
{
    if (!state || !state_first || !state_second || !q16 || !k16 || !v32 || !g32 || !beta32 || !out32) return fail(INSG_E_ARG, "deltanet: null pointer");
    if (qkv_stride < 0 || state_second == state) return fail(INSG_E_SHAPE, "deltanet: the second state needs a buffer of its own");
    return launch(deltanet_step_kernel, dim3(32 * kSlices), dim3(kDnThreads), 0, stream, true, const_cast<float *>(state), q16, k16, v32, g32,
                  beta32, out32, 2, qkv_stride, 0ll, state_first, state_second, pdl == 0);
}

extern "C" int insg_deltanet_decode_batch(float *state, long long state_stride, const float *q16, const float *k16, const float *v32,
                                          const float *g32, const float *beta32, float *out32, int sequences, int qkv_stride, int pdl,
                                          insg_stream_t stream)
{
    if (!state || !q16 || !k16 || !v32 || !g32 || !beta32 || !out32) return fail(INSG_E_ARG, "deltanet: null pointer");
    if (sequences < 1 || sequences > 64 || qkv_stride < 0 || state_stride < 32 * 128 * 128) return fail(INSG_E_SHAPE, "deltanet: 1..64 sequences");
    return launch(deltanet_step_kernel, dim3(32 * kSlices, sequences), dim3(kDnThreads), 0, stream, true, state, q16, k16, v32, g32,
                  beta32, out32, 1, qkv_stride, state_stride, nullptr, nullptr, pdl == 0);
}

extern "C" int insg_deltanet_decode_gated(float *state, long long state_stride, const float *q16, const float *k16, const float *v32, const float *g32,
                                          const float *beta32, float *out32, int sequences, int qkv_stride, const float *z, const uint16_t *norm_w,
                                          void *image, int pdl, insg_stream_t stream)
{
    if (!state || !q16 || !k16 || !v32 || !g32 || !beta32 || !out32 || !z || !norm_w || !image) return fail(INSG_E_ARG, "deltanet: null pointer");
    if (sequences < 1 || sequences > 8 || qkv_stride < 0 || state_stride < 32 * 128 * 128) return fail(INSG_E_SHAPE, "deltanet: 1..8 sequences");
    return launch(deltanet_heads_kernel, dim3(32, sequences), dim3(kDnThreads), 0, stream, pdl != 0, state, state_stride, q16, k16, v32, g32, beta32,
                  out32, qkv_stride, DnGate{z, norm_w, static_cast<uint8_t *>(image), image_slots(sequences)});
}

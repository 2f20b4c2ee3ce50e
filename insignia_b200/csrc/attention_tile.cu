// Attention of a prompt pass on the tensor cores: tiles of query tokens against tiles of cached rows (sm_100a).
//
// Math (reference: src/attention.cu:4, once per token): score_t = (q_h . K[t][h>>2]) / 16 over the rows up to the token's own,
// softmax, out_h = sum_t p_t V[t][h>>2].  The split-K decode kernel (attention.cu) streams the whole cache once per token; a
// pass of hundreds of tokens reads the same rows hundreds of times (2048 tokens: 79 ms of a 192 ms prompt).  Here a CTA takes
// one kv head and 16 consecutive tokens = 64 query rows (row = token * 4 + query head of the group), walks the cached rows
// in tiles of 32 and keeps an online softmax: every row fetched serves 64 query rows.
//
// Precision: the products run on mma.sync.m16n8k16 (fp16 in, fp32 accumulate).  Every fp32 operand is scaled by a power of two
// that puts the largest element of its tile in [2^12, 2^13) and cut into two fp16 pieces hi + lo, which together round it to
// 23 bits or better; all four products of pieces are accumulated.  A bf16 cache needs one piece (8 significant bits fit fp16
// exactly).  The value tiles share one running scale, so that the output accumulators are rescaled (with the softmax correction,
// by a power of two) when a tile brings a larger element.
// The instruction rounds its accumulator toward zero every time, and a sum kept in it through a whole row is off by some 1e-6.
// So it only adds the products with a lo piece, 2^-11 of the rest, to a running sum; 16 products hi * hi start from zero and
// are added outside, compensated, and so are the outputs.  Distance from float64 (2-norm, 512 tokens behind 512 rows):
// 1.6e-7 (fp32 cache), 1.4e-7 (bf16), the split-K kernel's 1.8e-7; with everything left to the accumulator 2.4e-6 and 1.6e-6,
// at 155 and 118 us instead of 220 and 156 (226 and 163 without the packed additions).
//
// Eight warps: warp & 3 = 16 of the query rows, warp >> 2 = which half of the 32 keys a warp scores and which half of the 256
// dims it sums; the two warps of a row exchange maxima and weights through shared memory.  Per tile of 32 keys a warp issues
// 128 + 128 MMAs (fp32 cache) between the conversion of the tile and three barriers: the tensor pipe is busy a third of the time,
// the issue slots half of it (two warps a scheduler; sixteen warps of half the keys and dims read the query twice as often and
// take the same time).  Rows of 528 bytes keep ldmatrix free of bank conflicts.
#include "attention_body.cuh"
#include "host_util.h"

#include <mutex>

namespace insg {

constexpr int kTileTokens = 16, kTileRows = 4 * kTileTokens, kTileKeys = 32;
constexpr int kTThreads = 256;
constexpr int kPitch = 528; // bytes per row of fp16 pieces: 512 + 16

template <bool BF16> struct TileSmem {
    static constexpr int pieces = BF16 ? 1 : 2;                                // of keys and values
    static constexpr int raw_row = BF16 ? 512 : 1024;                          // bytes of a cached row of one kv head
    static constexpr int q = 0;                                                // [2][64] rows
    static constexpr int k = q + 2 * kTileRows * kPitch;                       // [pieces][32] rows
    static constexpr int v = k + pieces * kTileKeys * kPitch;                  // [pieces][32] rows
    static constexpr int raw = v + pieces * kTileKeys * kPitch;                // [K, V][32] rows as cached
    static constexpr int bytes = raw + 2 * kTileKeys * raw_row;
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) // no sum to add to
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// sum + rest += x, rest being what the additions have rounded off.
__device__ __forceinline__ void add_compensated(float &sum, float &rest, float x)
{
    const float y = x + rest, z = sum + y;
    rest = y - (z - sum);
    sum = z;
}
// The same for two numbers in the packed fp32 instructions.
__device__ __forceinline__ void add_compensated(unsigned long long &sum, unsigned long long &rest, float x0, float x1)
{
    const unsigned long long y = add2(pack2(x0, x1), rest), z = add2(sum, y), minus = pack2(-1.f, -1.f);
    rest = fma2(fma2(sum, minus, z), minus, y);
    sum = z;
}
// hi and lo fp16 pieces of two scaled values
__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo)
{
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
// Biased exponent of a tile's largest magnitude, kept where both 2^(12 - e) and its inverse are normal numbers.
constexpr int kMaxExponent = 230; // tiles beyond it are not multiplied
__device__ __forceinline__ int tile_exponent(uint32_t max_bits) { return max(int(max_bits >> 23), 24); }
__device__ __forceinline__ float scale_up(int e) { return __uint_as_float(uint32_t(127 + 12 + 127 - e) << 23); }   // 2^(12 - (e - 127))
__device__ __forceinline__ float scale_down(int e) { return __uint_as_float(uint32_t(e - 12) << 23); }             // its inverse

// One token's four query heads over its first `rows` cached rows in fp32, by a warp (the loop of attn_splitk_kernel): for what the
// fp16 pieces cannot hold, infinities, NaN and values beyond 2^104, which must reach the tokens that see them and no others.
// (For short contexts too it would be slower, 64 tokens from an empty cache 50 us against 30, and no closer to float64.)
template <bool BF16> __device__ __noinline__ void attn_token(const AttnParams &p, const float *qn, int tok, int rows, int kvh)
{
    using Row = KvRow<BF16>;
    const int lane = threadIdx.x & 31, my_row = lane >> 3;
    float q[4][8], acc[4][8], m = -3.0e38f, l = 0.f;
#pragma unroll
    for (int h = 0; h < 4; h++) {
        const float4 *src = reinterpret_cast<const float4 *>(qn + (size_t(tok) * 16 + kvh * 4 + h) * 256 + lane * 8);
        const float4 a = __ldcg(src), b = __ldcg(src + 1);
        q[h][0] = a.x; q[h][1] = a.y; q[h][2] = a.z; q[h][3] = a.w; q[h][4] = b.x; q[h][5] = b.y; q[h][6] = b.z; q[h][7] = b.w;
#pragma unroll
        for (int j = 0; j < 8; j++) acc[h][j] = 0.f;
    }
    GroupRaw<BF16, 4> kv;
    load_group<BF16, 4>(p.kc, p.vc, kvh, 0, rows, lane, kv);
    for (int tb = 0; tb < rows; tb += 4) {
        float s[16]; // [row of the group][head]
#pragma unroll
        for (int g = 0; g < 4; g++) {
            float k[8];
            Row::unpack(kv.k[g], k);
#pragma unroll
            for (int h = 0; h < 4; h++) {
                s[g * 4 + h] = q[h][0] * k[0];
#pragma unroll
                for (int j = 1; j < 8; j++) s[g * 4 + h] = fmaf(q[h][j], k[j], s[g * 4 + h]);
            }
        }
        load_keys<BF16, 4>(p.kc, kvh, tb + 4, rows, lane, kv);
#pragma unroll
        for (int n = 8, mk = 16; n; n >>= 1, mk >>= 1) { // lane L is left with number L >> 1: row L >> 3, head (L >> 1) & 3
            const bool up = (lane & mk) != 0;
#pragma unroll
            for (int i = 0; i < n; i++) {
                const float keep = up ? s[i + n] : s[i], send = up ? s[i] : s[i + n];
                s[i] = keep + __shfl_xor_sync(0xffffffffu, send, mk);
            }
        }
        const float score = (s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1)) * 0.0625f;
        const bool on = tb + my_row < rows;
        float mx = on ? score : -3.0e38f;
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float mn = fmaxf(m, mx), corr = expf(m - mn), pr = on ? expf(score - mn) : 0.f;
        m = mn;
        l = fmaf(l, corr, pr);
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const float c = __shfl_sync(0xffffffffu, corr, 2 * h);
#pragma unroll
            for (int j = 0; j < 8; j++) acc[h][j] *= c;
        }
#pragma unroll
        for (int g = 0; g < 4; g++) {
            float v[8];
            Row::unpack(kv.v[g], v);
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float w = __shfl_sync(0xffffffffu, pr, (g * 4 + h) * 2);
#pragma unroll
                for (int j = 0; j < 8; j++) acc[h][j] = fmaf(w, v[j], acc[h][j]);
            }
        }
        load_values<BF16, 4>(p.vc, kvh, tb + 4, rows, lane, kv);
    }
    l += __shfl_xor_sync(0xffffffffu, l, 8);
    l += __shfl_xor_sync(0xffffffffu, l, 16);
#pragma unroll
    for (int h = 0; h < 4; h++) {
        const float lh = __shfl_sync(0xffffffffu, l, 2 * h);
        float4 *dst = reinterpret_cast<float4 *>(p.out + (size_t(tok) * 16 + kvh * 4 + h) * 256 + lane * 8);
        dst[0] = make_float4(acc[h][0] / lh, acc[h][1] / lh, acc[h][2] / lh, acc[h][3] / lh);
        dst[1] = make_float4(acc[h][4] / lh, acc[h][5] / lh, acc[h][6] / lh, acc[h][7] / lh);
    }
}

template <bool BF16>
__global__ void __launch_bounds__(kTThreads, 1) attn_tile_kernel(const __grid_constant__ AttnParams p, const float *__restrict__ qn, int tokens)
{
    using L = TileSmem<BF16>;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ uint32_t s_max[3][2]; // largest magnitude bits of [tile buffer][K, V]; [2][0]: the query rows
    __shared__ float s_mx[4][2][16], s_l[4][2][16]; // [16 query rows][key half][row]
    __shared__ uint32_t s_p[4][2][8][32];            // the weights' pieces as the A operand: [16 query rows][key half][register][lane]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = blockIdx.x, q0 = (int(gridDim.y) - 1 - int(blockIdx.y)) * kTileTokens; // the longest rows first
    const int rg = warp & 3, kg = warp >> 2, g = lane >> 2, t = lane & 3;

    pdl_launch_dependents();
    if (tid < 6) s_max[tid >> 1][tid & 1] = 0u;
    pdl_wait();
    __syncthreads();
    const int pos0 = __ldcg(p.position) + p.position_offset;
    // only tokens with a place in the cache (the prepare kernel stores no others): first .. last - 1
    const int first = max(q0, -pos0), last = min(min(q0 + kTileTokens, tokens), p.max_context - pos0); // of this tile
    if (first >= last) return;
    const int nkeys = pos0 + last; // rows the tile's last token attends
    auto live = [&](int tok) { return tok >= first && tok < last; };
    const int ntiles = (nkeys + kTileKeys - 1) / kTileKeys;

    auto fetch = [&](int tile) { // both raw tiles of 32 cached rows by 16-byte asynchronous copies; rows past the end repeat the last
        constexpr int per_row = L::raw_row / 16;
        for (int i = tid; i < 2 * kTileKeys * per_row; i += kTThreads) {
            const int kv = i / (kTileKeys * per_row), r = (i / per_row) % kTileKeys, c = i % per_row;
            const int row = min(tile * kTileKeys + r, nkeys - 1);
            const uint8_t *src = static_cast<const uint8_t *>(kv ? p.vc : p.kc) + (size_t(row) * 4 + kvh) * L::raw_row + c * 16;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(sm + L::raw + (kv * kTileKeys + r) * L::raw_row + c * 16)), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto plain = [&] { // every token by a warp in fp32
        for (int tok = first + warp; tok < last; tok += kTThreads / 32) attn_token<BF16>(p, qn, tok, pos0 + tok + 1, kvh);
    };
    fetch(0);

    // ---- query rows: scaled by 1/16 and the tile's power of two, two pieces ----
    float invq;
    {
        uint32_t mx = 0;
        for (int i = tid; i < kTileRows * 64; i += kTThreads) {
            const int r = i >> 6, c = i & 63, tok = q0 + (r >> 2);
            if (live(tok)) {
                const float4 x = __ldcg(reinterpret_cast<const float4 *>(qn + (size_t(tok) * 16 + kvh * 4 + (r & 3)) * 256) + c);
                mx = max(max(mx, max(__float_as_uint(fabsf(x.x)), __float_as_uint(fabsf(x.y)))), max(__float_as_uint(fabsf(x.z)), __float_as_uint(fabsf(x.w))));
            }
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) atomicMax(&s_max[2][0], mx);
        __syncthreads();
        const int e = tile_exponent(s_max[2][0]);
        if (e > kMaxExponent) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            plain();
            return;
        }
        const float up = scale_up(e);
        invq = scale_down(e) * 0.0625f;
        for (int i = tid; i < kTileRows * 64; i += kTThreads) {
            const int r = i >> 6, c = i & 63, tok = q0 + (r >> 2);
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live(tok)) x = __ldcg(reinterpret_cast<const float4 *>(qn + (size_t(tok) * 16 + kvh * 4 + (r & 3)) * 256) + c);
            uint2 hi, lo;
            split2(x.x * up, x.y * up, hi.x, lo.x);
            split2(x.z * up, x.w * up, hi.y, lo.y);
            *reinterpret_cast<uint2 *>(sm + L::q + r * kPitch + c * 8) = hi;
            *reinterpret_cast<uint2 *>(sm + L::q + (kTileRows + r) * kPitch + c * 8) = lo;
        }
    }

    unsigned long long o[16][2], oc[16][2]; // [8 dims each][rows g, g + 8]: dims 2t, 2t+1; the sum is o + oc
#pragma unroll
    for (int j = 0; j < 16; j++) o[j][0] = o[j][1] = oc[j][0] = oc[j][1] = 0ull;
    float m_run[2] = {-3.0e38f, -3.0e38f}, l_run[2] = {0.f, 0.f}, l_rest[2] = {0.f, 0.f}; // rows g and g + 8 (l: this thread's share of its keys)
    int ev = 24;                                                  // exponent of the running value scale
    const int limit0 = pos0 + q0 + ((rg * 16 + g) >> 2), limit1 = pos0 + q0 + ((rg * 16 + g + 8) >> 2); // last row each query row sees
    const uint32_t qaddr = smem_u32(sm + L::q) + (rg * 16 + (lane & 15)) * kPitch + (lane >> 4) * 16;
    const uint32_t kaddr = smem_u32(sm + L::k) + (kg * 16 + ((lane >> 4) & 1) * 8 + (lane & 7)) * kPitch + ((lane >> 3) & 1) * 16;
    const uint32_t vaddr = smem_u32(sm + L::v) + (((lane >> 3) & 1) * 8 + (lane & 7)) * kPitch + ((lane >> 4) & 1) * 16 + kg * 256;
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + rg) : "memory"); }; // the two warps of 16 query rows

    for (int tile = 0; tile < ntiles; tile++) {
        const int buf = tile & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads(); // the raw tile is complete; everybody is done with the previous tile's pieces and maxima
        // ---- largest magnitudes of the two raw tiles ----
        if (tid < 2) s_max[buf ^ 1][tid] = 0u;
        constexpr int per = 2 * kTileKeys * L::raw_row / 16 / kTThreads; // 16-byte cells per thread, the first half keys
        uint4 cell[per];
#pragma unroll
        for (int i = 0; i < per; i++) cell[i] = *reinterpret_cast<const uint4 *>(sm + L::raw + (tid + i * kTThreads) * 16);
#pragma unroll
        for (int kv = 0; kv < 2; kv++) {
            uint32_t mx = 0;
#pragma unroll
            for (int i = kv * per / 2; i < (kv + 1) * per / 2; i++) {
                const uint32_t w[4] = {cell[i].x, cell[i].y, cell[i].z, cell[i].w};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (BF16) mx = max(mx, max((w[q] << 16) & 0x7fffffffu, w[q] & 0x7fff0000u));
                    else mx = max(mx, w[q] & 0x7fffffffu);
                }
            }
            mx = __reduce_max_sync(0xffffffffu, mx);
            if (lane == 0) atomicMax(&s_max[buf][kv], mx);
        }
        __syncthreads(); // maxima complete, the raw tile is in registers
        const int ek = tile_exponent(s_max[buf][0]), ev_new = max(ev, tile_exponent(s_max[buf][1]));
        if (max(ek, ev_new) > kMaxExponent) { // all threads; nothing is in flight
            plain();
            return;
        }
        if (tile + 1 < ntiles) fetch(tile + 1);
        const float fv = __uint_as_float(uint32_t(max(127 + ev - ev_new, 0)) << 23); // rescales what was accumulated so far
        ev = ev_new;
        {
            const float up[2] = {scale_up(ek), scale_up(ev)};
#pragma unroll
            for (int i = 0; i < per; i++) {
                const int at = tid + i * kTThreads, kv = i >= per / 2;
                if (BF16) { // eight values of one row
                    const int r = (at >> 5) & 31, c = at & 31;
                    const uint32_t w[4] = {cell[i].x, cell[i].y, cell[i].z, cell[i].w};
                    uint32_t h[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const __half2 x = __floats2half2_rn(__uint_as_float(w[q] << 16) * up[kv], __uint_as_float(w[q] & 0xffff0000u) * up[kv]);
                        h[q] = *reinterpret_cast<const uint32_t *>(&x);
                    }
                    *reinterpret_cast<uint4 *>(sm + (kv ? L::v : L::k) + r * kPitch + c * 16) = make_uint4(h[0], h[1], h[2], h[3]);
                } else { // four values of one row
                    const int r = (at >> 6) & 31, c = at & 63;
                    uint2 hi, lo;
                    split2(__uint_as_float(cell[i].x) * up[kv], __uint_as_float(cell[i].y) * up[kv], hi.x, lo.x);
                    split2(__uint_as_float(cell[i].z) * up[kv], __uint_as_float(cell[i].w) * up[kv], hi.y, lo.y);
                    uint8_t *dst = sm + (kv ? L::v : L::k) + r * kPitch + c * 8;
                    *reinterpret_cast<uint2 *>(dst) = hi;
                    *reinterpret_cast<uint2 *>(dst + kTileKeys * kPitch) = lo;
                }
            }
        }
        __syncthreads(); // the pieces are complete
        const int key0 = tile * kTileKeys + kg * 16 + 2 * t; // this thread's first key of four
        // ---- scores of 16 rows x 16 keys ----
        float s[2][4], low[2][4]; // sums with a lo piece
        unsigned long long high[2][2], rest[2][2]; // sums of hi*hi (rows g and g + 8), what their additions rounded off
#pragma unroll
        for (int n = 0; n < 2; n++) {
            high[n][0] = high[n][1] = rest[n][0] = rest[n][1] = 0ull;
#pragma unroll
            for (int c = 0; c < 4; c++) low[n][c] = 0.f;
        }
#pragma unroll 4
        for (int i = 0; i < 16; i++) {
            uint32_t qh[4], ql[4], kh[4], kl[4];
            float part[2][4];
            ldsm4(qh, qaddr + 32 * i);
            ldsm4(ql, qaddr + kTileRows * kPitch + 32 * i);
            ldsm4(kh, kaddr + 32 * i);
            if (!BF16) ldsm4(kl, kaddr + kTileKeys * kPitch + 32 * i);
#pragma unroll
            for (int n = 0; n < 2; n++) {
                mma_f16_first(part[n], qh, kh[2 * n], kh[2 * n + 1]);
                if (!BF16) mma_f16(low[n], ql, kl[2 * n], kl[2 * n + 1]);
                if (!BF16) mma_f16(low[n], qh, kl[2 * n], kl[2 * n + 1]);
                mma_f16(low[n], ql, kh[2 * n], kh[2 * n + 1]);
            }
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int h = 0; h < 2; h++) add_compensated(high[n][h], rest[n][h], part[n][2 * h], part[n][2 * h + 1]);
        }
        // ---- online softmax (rows g and g + 8; a row's 32 keys sit in the quads of two warps) ----
        const float sc = invq * scale_down(ek);
        bool on[2][4]; // the row sees the key
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float2 a = unpack2(high[n][c >> 1]), b = unpack2(rest[n][c >> 1]);
                s[n][c] = (c & 1) ? (a.y + (low[n][c] + b.y)) * sc : (a.x + (low[n][c] + b.x)) * sc;
                on[n][c] = key0 + n * 8 + (c & 1) <= (c < 2 ? limit0 : limit1);
            }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float mx = -3.0e38f;
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int c = 2 * h; c < 2 * h + 2; c++) mx = on[n][c] ? fmaxf(mx, s[n][c]) : mx;
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            if (t == 0) s_mx[rg][kg][g + 8 * h] = mx;
        }
        pair_sync();
        float corr[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float m_new = fmaxf(m_run[h], fmaxf(s_mx[rg][0][g + 8 * h], s_mx[rg][1][g + 8 * h]));
            corr[h] = expf(m_run[h] - m_new);
            m_run[h] = m_new;
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 2; n++) {
#pragma unroll
                for (int c = 2 * h; c < 2 * h + 2; c++) {
                    s[n][c] = on[n][c] ? expf(s[n][c] - m_new) : 0.f;
                    sum += s[n][c];
                }
                uint32_t hi, lo;
                split2(s[n][2 * h] * 4096.f, s[n][2 * h + 1] * 4096.f, hi, lo);
                s_p[rg][kg][2 * n + h][lane] = hi;
                s_p[rg][kg][4 + 2 * n + h][lane] = lo;
            }
            l_run[h] *= corr[h];
            l_rest[h] *= corr[h];
            add_compensated(l_run[h], l_rest[h], sum);
        }
        pair_sync();
        uint32_t w[2][2][4]; // the weights as the A operand: [key half][hi, lo]
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int i = 0; i < 8; i++) w[k][i >> 2][i & 3] = s_p[rg][k][i][lane];
        const float c0 = corr[0] * fv, c1 = corr[1] * fv;
        if (__any_sync(0xffffffffu, c0 != 1.f || c1 != 1.f)) {
            const unsigned long long f0 = pack2(c0, c0), f1 = pack2(c1, c1);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                o[j][0] = mul2(o[j][0], f0); o[j][1] = mul2(o[j][1], f1);
                oc[j][0] = mul2(oc[j][0], f0); oc[j][1] = mul2(oc[j][1], f1);
            }
        }
        // ---- values: 128 of the 256 dims, 16 keys and 16 dims at a time; the small products first, one rounding of the large one ----
#pragma unroll
        for (int j = 0; j < 8; j++) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                uint32_t vh[4], vl[4];
                float part[2][4];
                ldsm4t(vh, vaddr + k * 16 * kPitch + 32 * j);
                if (!BF16) ldsm4t(vl, vaddr + (kTileKeys + k * 16) * kPitch + 32 * j);
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    if (BF16) {
                        mma_f16_first(part[n], w[k][1], vh[2 * n], vh[2 * n + 1]);
                    } else {
                        mma_f16_first(part[n], w[k][1], vl[2 * n], vl[2 * n + 1]);
                        mma_f16(part[n], w[k][1], vh[2 * n], vh[2 * n + 1]);
                        mma_f16(part[n], w[k][0], vl[2 * n], vl[2 * n + 1]);
                    }
                    mma_f16(part[n], w[k][0], vh[2 * n], vh[2 * n + 1]);
                }
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int h = 0; h < 2; h++) add_compensated(o[2 * j + n][h], oc[2 * j + n][h], part[n][2 * h], part[n][2 * h + 1]);
            }
        }
    }
    // ---- the denominator from both key halves; write the rows ----
#pragma unroll
    for (int h = 0; h < 2; h++) {
        l_run[h] += l_rest[h];
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
        if (t == 0) s_l[rg][kg][g + 8 * h] = l_run[h];
    }
    pair_sync();
    const float up_v = scale_down(ev) * (1.f / 4096.f); // undoes the values' and the weights' powers of two
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int r = rg * 16 + g + 8 * h, tok = q0 + (r >> 2);
        const float l = s_l[rg][0][g + 8 * h] + s_l[rg][1][g + 8 * h], inv = 1.f / l, off = fmaf(-l, inv, 1.f);
        auto quotient = [&](float a, float b) { // (a + b) / l with one rounding
            const float q = a * inv;
            return (q + fmaf(q, off, fmaf(a, inv, -q) + b * inv)) * up_v;
        };
        if (live(tok)) {
            float *dst = p.out + (size_t(tok) * 16 + kvh * 4 + (r & 3)) * 256 + kg * 128 + 2 * t;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float2 a = unpack2(o[j][h]), b = unpack2(oc[j][h]);
                *reinterpret_cast<float2 *>(dst + 8 * j) = make_float2(quotient(a.x, b.x), quotient(a.y, b.y));
            }
        }
    }
}

template <bool BF16> static int launch_tile(const AttnParams &p, const float *qn, int tokens, cudaStream_t st, bool pdl)
{
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= 64) return fail(INSG_E_LIMIT, "attention: device ordinal beyond 63");
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!done[dev]) {
            e = cudaFuncSetAttribute(attn_tile_kernel<BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, TileSmem<BF16>::bytes);
            if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(attention tiles)");
            done[dev] = true;
        }
    }
    return launch(attn_tile_kernel<BF16>, dim3(4, (tokens + kTileTokens - 1) / kTileTokens), dim3(kTThreads), TileSmem<BF16>::bytes, st, pdl, p, qn, tokens);
}

// p: the caches, the device position and the output rows; qn [tokens][16][256]: the normalised, rotated queries.
int attn_tile_launch(const AttnParams &p, const float *qn, int tokens, bool bf16, cudaStream_t st, bool pdl)
{
    return bf16 ? launch_tile<true>(p, qn, tokens, st, pdl) : launch_tile<false>(p, qn, tokens, st, pdl);
}

} // namespace insg

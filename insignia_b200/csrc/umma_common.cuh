// Helpers shared by the tcgen05 kernels (umma_gemv.cu: one to eight tokens, activation image resident in shared memory;
// umma_gemm.cu: more tokens, activation image streamed): shared-memory descriptors, mbarrier waits with a bound,
// bulk copies, the tcgen05 instructions, and the split of an fp32 activation into exact E2M1 digits.
#pragma once
#include "common.cuh"

namespace insg {

constexpr int kURec = 8704;          // bytes per (128-row tile, 128-k block) weight record: 8192 of codes + 512 of scales
constexpr uint32_t kSpinLimit = 1u << 22;

// shared-memory matrix descriptor: no swizzle, version 1 (sm_100); offsets in bytes
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return uint64_t((saddr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) | (uint64_t((sbo >> 4) & 0x3FFF) << 32) | (uint64_t(1) << 46);
}

__device__ __forceinline__ void mbar_init(uint64_t *b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// Bounded wait on a phase parity; false when the limit ran out or another role raised the abort flag.
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity, volatile int *abort_flag)
{
#pragma unroll 1
    for (uint32_t it = 0; it < kSpinLimit; it++) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(smem_u32(b)), "r"(parity) : "memory");
        if (done) return true;
        if ((it & 1023u) == 1023u && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}

// A wait on data other CTAs of the cluster send (acquire at cluster scope).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *b, uint32_t parity, volatile int *abort_flag)
{
#pragma unroll 1
    for (uint32_t it = 0; it < kSpinLimit; it++) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(smem_u32(b)), "r"(parity) : "memory");
        if (done) return true;
        if ((it & 1023u) == 1023u && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}

// An arrival at another CTA's barrier that hands over what this thread did or saw in its own shared memory: a release at cluster scope,
// restricted to shared memory, so that it waits for no store to global memory.
__device__ __forceinline__ void remote_arrive(uint32_t bar)
{
    asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n"
                 "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// A poll that never suspends the thread.
__device__ __forceinline__ bool mbar_test(uint64_t *b, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done) : "r"(smem_u32(b)), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_test_cluster(uint64_t *b, uint32_t parity) // of what other CTAs of the cluster arrive at
{
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done) : "r"(smem_u32(b)), "r"(parity) : "memory");
    return done != 0;
}
// One lane of a converged warp (the same one every time).
__device__ __forceinline__ bool elect_one()
{
    uint32_t e;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(e));
    return e != 0;
}

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Weights that a launch reads once leave L2 first: what else a token touches (states, caches, digits, and the kernels' code, which would come from memory
// behind the weights) stays there.  A device-fed token 981 -> 960 us, a step of three sequences 1122 -> 1100, of eight 1300 -> 1267, a speculative pass
// 1332 -> 1320, a prompt of 12 tokens 2.80 -> 2.72 ms.
__device__ __forceinline__ uint64_t once_policy()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void bulk_load_hint(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint64_t policy)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy) : "memory");
}
__device__ __forceinline__ void bulk_prefetch_hint(const void *src, uint32_t bytes, uint64_t policy) // to L2
{
    asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(src), "r"(bytes), "l"(policy) : "memory");
}

// ---- tcgen05 instructions as the kernels issue them ----
// A warp walks the issuing loop together and one lane (on != 0) issues, by a predicate.  Behind a branch the same instructions cost a decoded
// token 1029 us instead of 1010, a speculative pass 1366 instead of 1343, eight sequences 1330 instead of 1320, and 40 tokens of 24576 x 4096 25.6
// instead of 24.3.
__device__ __forceinline__ void copy_scales_if(uint32_t on, uint32_t taddr, uint64_t desc)
{
    asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %2, 0;\n@q tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;\n}" ::"r"(taddr), "l"(desc), "r"(on) : "memory");
}
__device__ __forceinline__ void mma_step_if(uint32_t on, uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate, uint32_t sa, uint32_t sb)
{
    asm volatile("{\n.reg .pred q, r;\nsetp.ne.b32 q, %4, 0;\nsetp.ne.b32 r, %7, 0;\n"
                 "@r tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], q;\n}"
                 ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(uint32_t(accumulate)), "r"(sa), "r"(sb), "r"(on) : "memory");
}
__device__ __forceinline__ void commit_if(uint32_t on, uint64_t *bar)
{
    asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %1, 0;\n@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(smem_u32(bar)), "r"(on) : "memory");
}

// Eight balanced base-9 digits of round(x * alpha) (|.| < 2^24) as E2M1 codes, digit j in nibble j.  u = v + 4 * (9^8 - 1) / 8
// has plain base-9 digits 0..8 (the balanced digit + 4); they are taken in pairs (base 81) through an 81-byte table, which
// costs a third of the instructions of eight divisions by 9.
__device__ __forceinline__ uint32_t digit_codes81(float x, float alpha, const uint8_t *lut)
{
    const int v = max(-0xFFFFFF, min(__float2int_rn(x * alpha), 0xFFFFFF));
    const uint32_t u = uint32_t(v + 21523360);
    const uint32_t hi = u / 6561u, lo = u - 6561u * hi;
    const uint32_t h1 = (hi * 6473u) >> 19, h0 = hi - 81u * h1; // n / 81 for n < 6562 (6473 / 2^19 = 1/81 + 1.7e-7)
    const uint32_t l1 = (lo * 6473u) >> 19, l0 = lo - 81u * l1;
    return uint32_t(lut[l0]) | (uint32_t(lut[l1]) << 8) | (uint32_t(lut[h0]) << 16) | (uint32_t(lut[h1]) << 24);
}
__device__ __forceinline__ uint8_t digit_pair_code(int n) // table entry: digits n % 9 - 4 (low nibble) and n / 9 - 4 (high nibble)
{
    uint32_t r = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int d = (h ? n / 9 : n % 9) - 4, mag = d < 0 ? -d : d; // 0..4 -> E2M1 codes 0, 2, 4, 5, 6
        r |= uint32_t((mag < 3 ? 2 * mag : mag + 2) | (d < 0 ? 8 : 0)) << (4 * h);
    }
    return uint8_t(r);
}

// The digits of four consecutive elements: two bytes in each of the eight digit columns (16 bytes apart) from `base` on.
__device__ __forceinline__ void pack_digits(float4 x, float alpha, const uint8_t *lut, uint8_t *base)
{
    const uint32_t c0 = digit_codes81(x.x, alpha, lut), c1 = digit_codes81(x.y, alpha, lut);
    const uint32_t c2 = digit_codes81(x.z, alpha, lut), c3 = digit_codes81(x.w, alpha, lut);
    // columns 0, 2, 4, 6 sit in the low nibbles of the four bytes, 1, 3, 5, 7 in the high ones
    const uint32_t e01 = (c0 & 0x0F0F0F0Fu) | ((c1 & 0x0F0F0F0Fu) << 4), e23 = (c2 & 0x0F0F0F0Fu) | ((c3 & 0x0F0F0F0Fu) << 4);
    const uint32_t o01 = ((c0 >> 4) & 0x0F0F0F0Fu) | (c1 & 0xF0F0F0F0u), o23 = ((c2 >> 4) & 0x0F0F0F0Fu) | (c3 & 0xF0F0F0F0u);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        *reinterpret_cast<uint16_t *>(base + (2 * j) * 16) = uint16_t(__byte_perm(e01, e23, j | ((4 + j) << 4)));
        *reinterpret_cast<uint16_t *>(base + (2 * j + 1) * 16) = uint16_t(__byte_perm(o01, o23, j | ((4 + j) << 4)));
    }
}

// A token's eight digit columns of an accumulator: the sum they stand for (least significant first; 9^j is exact in fp32).
__device__ __forceinline__ float combine_digits(const uint32_t *d)
{
    float y = __uint_as_float(d[0]);
    y = fmaf(__uint_as_float(d[1]), 9.f, y);
    y = fmaf(__uint_as_float(d[2]), 81.f, y);
    y = fmaf(__uint_as_float(d[3]), 729.f, y);
    y = fmaf(__uint_as_float(d[4]), 6561.f, y);
    y = fmaf(__uint_as_float(d[5]), 59049.f, y);
    y = fmaf(__uint_as_float(d[6]), 531441.f, y);
    return fmaf(__uint_as_float(d[7]), 4782969.f, y);
}

// ---- a group of 32 elements: its scale from its largest magnitude -------------------------------------------------------------
// Infinities and NaN have no digits: the scale byte 255 is the format's NaN, and makes every product with the group NaN.
__device__ __forceinline__ float fmax_nan(float a, float b) // NaN where either is
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ int group_exponent(uint32_t max_bits) { return max(int(max_bits >> 23), 24); } // bits of |.|: 255 = not finite
__device__ __forceinline__ float group_alpha(int eb) { return __uint_as_float(uint32_t(277 - eb) << 23); }  // largest element * alpha in [2^23, 2^24)
__device__ __forceinline__ uint8_t group_scale(int eb) { return uint8_t(eb == 255 ? 255 : eb - 23); }

// ---- digit image of activation vectors: [k-block of 128][digits of T token slots: 512 T bytes | scale block: 512 bytes] ----
// The digits of one 128-element k-block of one token (four elements per lane) into the B image, and their group scales.
// Image of a k-block: [2 K-steps][T column groups][2 k cores][8 columns][16 B]; a token's eight digit columns are one group.
__device__ __forceinline__ void store_digits(float4 x, int T, int m, uint8_t *bkb, const uint8_t *lut, int lane)
{
    float mx = fmax_nan(fmax_nan(fabsf(x.x), fabsf(x.y)), fmax_nan(fabsf(x.z), fabsf(x.w)));
    mx = fmax_nan(mx, __shfl_xor_sync(0xffffffffu, mx, 1)); // a group of 32 elements = 8 lanes
    mx = fmax_nan(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    mx = fmax_nan(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    const int eb = group_exponent(__float_as_uint(mx));
    pack_digits(x, group_alpha(eb), lut, bkb + (lane >> 4) * (256 * T) + m * 256 + ((lane >> 3) & 1) * 128 + (lane & 7) * 2);
    const int n = 8 * m + (lane & 7); // scale block: row = column n of B (32 rows, then the next quarter), byte = group
    bkb[512 * T + (n & 31) * 16 + (n >> 5) * 4 + (lane >> 3)] = group_scale(eb);
}

// One element per lane: the warp's 32 lanes are the 32-element group `grp` of token slot m's vector.
__device__ __forceinline__ void group_digits(float x, int T, int m, uint8_t *image, int grp, const uint8_t *lut, int lane)
{
    const int eb = group_exponent(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(x))));
    const uint32_t c = digit_codes81(x, group_alpha(eb), lut), o = __shfl_xor_sync(0xffffffffu, c, 1);
    // a pair of lanes holds two neighbouring k = one byte per column: the even lane stores columns 0, 2, 4, 6, the odd one the others
    const uint32_t b = (lane & 1) ? ((o >> 4) & 0x0F0F0F0Fu) | (c & 0xF0F0F0F0u) : (c & 0x0F0F0F0Fu) | ((o & 0x0F0F0F0Fu) << 4);
    const int g = grp & 3;
    uint8_t *kb = image + size_t(grp >> 2) * (512 * T + 512), *dst = kb + (g >> 1) * (256 * T) + m * 256 + (g & 1) * 128 + (lane & 1) * 16 + (lane >> 1);
#pragma unroll
    for (int j = 0; j < 4; j++) dst[32 * j] = uint8_t(b >> (8 * j));
    const int n = 8 * m + (lane & 7);
    if (lane < 8) kb[512 * T + (n & 31) * 16 + (n >> 5) * 4 + g] = group_scale(eb);
}
// Token slots of an image of `tokens` (1..8) vectors.
__host__ __device__ inline int image_slots(int tokens) { return tokens == 1 ? 1 : tokens == 2 ? 2 : tokens <= 4 ? 4 : 8; }

} // namespace insg

/*
 * philox.h -- Philox4x32-10 keep-mask shared by host and device code.
 *
 * The reference forward kernel takes dropout as a caller-materialised dense
 * float tensor dropout_mask[B*nh, T, T] that it multiplies into exp(s - m)
 * (kernels/attention/fused_attn_forward_kernel_tc_sm89.cu:21-22,321-324); it
 * has no generator.  This header defines the generator the sm_100a kernels
 * evaluate in registers, and the host evaluates to materialise that same dense
 * mask, so the two agree bit for bit (integer arithmetic only).
 *
 * Element (bh, qi, kj) -- qi and kj are GLOBAL sequence positions -- draws from
 *   counter = { kj >> 3, qi, bh, lo32(offset) }
 *   key     = { lo32(seed), hi32(seed) ^ hi32(offset) }
 * and uses 16-bit half number (kj & 7) of the 128 output bits (half h of word
 * (kj & 7) >> 1, low half first), so one Philox call covers eight consecutive
 * keys of a query row.  keep <=> half >= floor(p * 2^16): the drop probability
 * is p rounded down to a multiple of 2^-16.
 */
#ifndef HK_PHILOX_H_
#define HK_PHILOX_H_

#include <stdint.h>

#if defined(__CUDACC__)
#define HK_HD __host__ __device__ __forceinline__
#else
#define HK_HD static inline
#endif

#define HK_PHILOX_M0 0xD2511F53u
#define HK_PHILOX_M1 0xCD9E8D57u
#define HK_PHILOX_W0 0x9E3779B9u
#define HK_PHILOX_W1 0xBB67AE85u

typedef struct { uint32_t v[4]; } hk_philox4_t;

HK_HD void hk_mulhilo32(uint32_t a, uint32_t b, uint32_t* hi, uint32_t* lo) {
#if defined(__CUDA_ARCH__)
    *lo = a * b;
    *hi = __umulhi(a, b);
#else
    uint64_t p = (uint64_t)a * (uint64_t)b;
    *lo = (uint32_t)p;
    *hi = (uint32_t)(p >> 32);
#endif
}

HK_HD hk_philox4_t hk_philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0, uint32_t k1) {
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0, lo0, hi1, lo1;
        hk_mulhilo32(HK_PHILOX_M0, c0, &hi0, &lo0);
        hk_mulhilo32(HK_PHILOX_M1, c2, &hi1, &lo1);
        uint32_t n0 = hi1 ^ c1 ^ k0;
        uint32_t n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += HK_PHILOX_W0;
        k1 += HK_PHILOX_W1;
    }
    hk_philox4_t out;
    out.v[0] = c0; out.v[1] = c1; out.v[2] = c2; out.v[3] = c3;
    return out;
}

/* The key of every round, which the kernels take from their argument block: 20 additions per call less. */
typedef struct { uint32_t k0[10], k1[10]; } hk_philox_keys_t;
HK_HD hk_philox_keys_t hk_philox_keys(uint64_t seed, uint64_t offset) {
    hk_philox_keys_t k;
    for (int r = 0; r < 10; ++r) {
        k.k0[r] = (uint32_t)seed + (uint32_t)r * HK_PHILOX_W0;
        k.k1[r] = ((uint32_t)(seed >> 32) ^ (uint32_t)(offset >> 32)) + (uint32_t)r * HK_PHILOX_W1;
    }
    return k;
}
#if defined(__CUDACC__)
__device__ __forceinline__ hk_philox4_t hk_philox_row8_keys(const hk_philox_keys_t& k, uint32_t offset, uint32_t bh, uint32_t qi,
                                                            uint32_t kj8) {
    uint32_t c0 = kj8, c1 = qi, c2 = bh, c3 = offset;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0, lo0, hi1, lo1;
        hk_mulhilo32(HK_PHILOX_M0, c0, &hi0, &lo0);
        hk_mulhilo32(HK_PHILOX_M1, c2, &hi1, &lo1);
        const uint32_t n0 = hi1 ^ c1 ^ k.k0[r], n2 = hi0 ^ c3 ^ k.k1[r];
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    }
    hk_philox4_t out;
    out.v[0] = c0; out.v[1] = c1; out.v[2] = c2; out.v[3] = c3;
    return out;
}

/* Both halves of a product by one instruction.  With the calls in parts (below) this is faster than the two of hk_mulhilo32,
 * with whole calls it is not. */
__device__ __forceinline__ void hk_mulwide32(uint32_t a, uint32_t b, uint32_t* hi, uint32_t* lo) {
    unsigned long long p;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(p) : "r"(a), "r"(b));
    *lo = (uint32_t)p;
    *hi = (uint32_t)(p >> 32);
}
/* The same call in parts.  Of the first two and a half rounds every product has a factor that depends on the query row alone
 * or on the keys alone (the other words enter by exclusive or): 5 of the 20 wide products of a call. */
__device__ __forceinline__ uint4 hk_philox_key_part(const hk_philox_keys_t& k, uint32_t offset, uint32_t bh, uint32_t kj8) {
    uint32_t hi, lo0, lo1, hi2, lo2;
    hk_mulwide32(HK_PHILOX_M0, kj8, &hi, &lo0);
    hk_mulwide32(HK_PHILOX_M1, hi ^ offset ^ k.k1[0], &hi, &lo1);
    hk_mulwide32(HK_PHILOX_M0, hi ^ (HK_PHILOX_M1 * bh) ^ k.k0[1], &hi2, &lo2);
    return make_uint4(lo0 ^ k.k1[1], lo1 ^ k.k0[2], hi2 ^ k.k1[2], lo2);
}
__device__ __forceinline__ uint2 hk_philox_row_part(const hk_philox_keys_t& k, uint32_t bh, uint32_t qi) {
    uint32_t hi, lo;
    hk_mulwide32(HK_PHILOX_M0, __umulhi(HK_PHILOX_M1, bh) ^ qi ^ k.k0[0], &hi, &lo);
    return make_uint2(hi, lo);
}
__device__ __forceinline__ hk_philox4_t hk_philox_join(const hk_philox_keys_t& k, const uint4& key, const uint2& row) {
    uint32_t hi0, lo0, hi1, lo1;
    hk_mulwide32(HK_PHILOX_M1, row.x ^ key.x, &hi1, &lo1);
    uint32_t c0 = hi1 ^ key.y, c1 = lo1, c2 = key.z ^ row.y, c3 = key.w;
#pragma unroll
    for (int r = 3; r < 10; ++r) {
        hk_mulwide32(HK_PHILOX_M0, c0, &hi0, &lo0);
        hk_mulwide32(HK_PHILOX_M1, c2, &hi1, &lo1);
        const uint32_t n0 = hi1 ^ c1 ^ k.k0[r], n2 = hi0 ^ c3 ^ k.k1[r];
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    }
    hk_philox4_t out;
    out.v[0] = c0; out.v[1] = c1; out.v[2] = c2; out.v[3] = c3;
    return out;
}
#endif

/* floor(p * 2^16), in [0, 65535]; p in [0,1). */
HK_HD uint32_t hk_philox_threshold(float p) {
    double t = (double)p * 65536.0;
    if (t <= 0.0) return 0u;
    if (t >= 65535.0) return 65535u;
    return (uint32_t)t;
}

/* The 128 random bits for keys 8*kj8 .. 8*kj8+7 of query row qi. */
HK_HD hk_philox4_t hk_philox_row8(uint64_t seed, uint64_t offset, uint32_t bh, uint32_t qi, uint32_t kj8) {
    return hk_philox4x32_10(kj8, qi, bh, (uint32_t)offset, (uint32_t)seed,
                            (uint32_t)(seed >> 32) ^ (uint32_t)(offset >> 32));
}

/* Is key u (0..7) of one Philox call kept?  half >= thr, compared in the upper 16 bits (thr < 2^16). */
HK_HD int hk_philox_keep1(hk_philox4_t r, int u, uint32_t thr) {
    return ((u & 1) ? r.v[u >> 1] : r.v[u >> 1] << 16) >= (thr << 16);
}

/* Keep bits of the eight keys of one Philox call: bit u <=> key 8*kj8+u is kept. */
HK_HD uint32_t hk_philox_keep8(hk_philox4_t r, uint32_t thr) {
    uint32_t m = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int u = 0; u < 8; ++u) m |= hk_philox_keep1(r, u, thr) ? 1u << u : 0u;
    return m;
}

HK_HD int hk_philox_keep(uint64_t seed, uint64_t offset, uint32_t bh, uint32_t qi, uint32_t kj, uint32_t thr) {
    hk_philox4_t r = hk_philox_row8(seed, offset, bh, qi, kj >> 3);
    return (int)((hk_philox_keep8(r, thr) >> (kj & 7u)) & 1u);
}

#endif /* HK_PHILOX_H_ */

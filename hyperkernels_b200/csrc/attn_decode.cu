// attn_decode.cu -- the forward for a few query rows against many keys (a decoding step against a key/value cache).
//
// Same function as attn_fwd_sm100.cu without dropout and without a starting state; fp32 arithmetic throughout.  Such a
// call reads K and V once and does next to nothing with them, so it is bound by HBM: what counts is that every SM has
// enough loads in flight.  The tensor-core kernel works on 128 query rows whatever the call has and one CTA fills an SM,
// so 192 (batch, head) slices on 148 SMs take two rounds.  Here a slice is cut into runs of keys, one CTA each, many CTAs
// per SM.
//   A half-warp reads one row of K and V (16 lanes x float4); lanes keep four of the 64 output columns.  A warp issues the
// loads of 2 * UNROLL rows before it uses the first.  Scores are reduced over the 16 lanes with shuffles; the running
// maximum is raised once per batch of rows.  The partial (m, l, O) of the warps are merged in shared memory, those of the
// CTAs of a slice (a cluster) through distributed shared memory.
//   B16 H12, one query, 2 047 keys (201 MB, 31 us at the copy bandwidth): 33 us, 55 with the tensor-core kernel.
#include <algorithm>

#include "attn_kernels.cuh"

namespace hk {

namespace dec {

constexpr int UNROLL = 4;

struct Partial {  // of one warp, then (warp 0's) of the CTA
    float m[DECODE_MAX_Q], l[DECODE_MAX_Q];
    float o[DECODE_MAX_Q][HEAD_DIM];
};

// fold (m2, l2, o2) into (m, l, o); a side that saw no key has m = -inf, l = 0, o = 0
__device__ __forceinline__ void fold(float& m, float& l, float4& o, float m2, float l2, float4 o2) {
    const float mn = fmaxf(m, m2);
    const float a = m == -INFINITY ? 0.f : ex2_approx(m - mn), c = m2 == -INFINITY ? 0.f : ex2_approx(m2 - mn);
    l = l * a + l2 * c;
    o.x = o.x * a + o2.x * c; o.y = o.y * a + o2.y * c; o.z = o.z * a + o2.z * c; o.w = o.w * a + o2.w * c;
    m = mn;
}

}  // namespace dec

template <int NQ, int WARPS>  // registers for 24 warps per SM with one query, 16 with two
__global__ void __launch_bounds__(WARPS * 32, (NQ == 1 ? 24 : 16) / WARPS) attn_decode_kernel(const DecodeArgs a) {
    using namespace dec;
    extern __shared__ __align__(16) uint8_t dsmem[];
    Partial* part = reinterpret_cast<Partial*>(dsmem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4, sub = lane & 15;
    constexpr int n_warps = WARPS;
    const int ns = a.n_splits, split = ns > 1 ? (int)cluster_ctarank() : 0;
    const int bh = blockIdx.x / ns, b = bh / a.H, h = bh - b * a.H;

    pdl_wait();
    pdl_trigger();
    // keys any row of the call may see, and this CTA's run of them
    long long n_ll = a.Tk;
    if (a.causal) n_ll = max(0ll, min(n_ll, (long long)a.q_pos0 + a.Tq - a.k_pos0));
    const int n = (int)n_ll, per = (n + ns - 1) / ns;
    const int begin = min(n, split * per), end = min(n, begin + per);

    const float4* Kp = reinterpret_cast<const float4*>(a.K.ptr + (int64_t)b * a.K.sB + (int64_t)h * a.K.sH) + sub;
    const float4* Vp = reinterpret_cast<const float4*>(a.V.ptr + (int64_t)b * a.V.sB + (int64_t)h * a.V.sH) + sub;
    const int64_t kM = a.K.sM >> 2, vM = a.V.sM >> 2;
    float4 q[NQ], o[NQ];
    float m[NQ], l[NQ];
    int lim[NQ];  // last key the row may see
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        const int row = min(i, a.Tq - 1);
        q[i] = __ldg(reinterpret_cast<const float4*>(a.Q.ptr + (int64_t)b * a.Q.sB + (int64_t)h * a.Q.sH + row * a.Q.sM) + sub);
        q[i].x *= a.scale_log2e; q[i].y *= a.scale_log2e; q[i].z *= a.scale_log2e; q[i].w *= a.scale_log2e;
        o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        m[i] = -INFINITY;
        l[i] = 0.f;
        lim[i] = a.causal ? (int)max(-1ll, min((long long)end - 1, (long long)a.q_pos0 + row - a.k_pos0)) : end - 1;
    }
    const int stride = n_warps * 2 * UNROLL;
    float4 kn[UNROLL], vn[UNROLL];  // the batch after the one at work: its loads run under the arithmetic
    auto load = [&](int k0) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) kn[u] = __ldcs(Kp + (int64_t)min(k0 + 2 * u, end - 1) * kM);
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) vn[u] = __ldcs(Vp + (int64_t)min(k0 + 2 * u, end - 1) * vM);
    };
    int k0 = begin + warp * 2 * UNROLL + half;
    if (k0 - half < end) load(k0);
    for (; k0 - half < end; k0 += stride) {
        float4 k[UNROLL], v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            k[u] = kn[u];
            v[u] = vn[u];
        }
        if (k0 - half + stride < end) load(k0 + stride);
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            float s[UNROLL], mx = -INFINITY;
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) s[u] = q[i].x * k[u].x + q[i].y * k[u].y + q[i].z * k[u].z + q[i].w * k[u].w;
#pragma unroll
            for (int off = 8; off > 0; off >>= 1)
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                if (k0 + 2 * u > lim[i]) s[u] = -INFINITY;
                mx = fmaxf(mx, s[u]);
            }
            const float mn = fmaxf(m[i], mx), ref = mn == -INFINITY ? 0.f : mn;
            const float alpha = ex2_approx(m[i] - ref);  // 0 while m is -inf
            o[i].x *= alpha; o[i].y *= alpha; o[i].z *= alpha; o[i].w *= alpha;
            l[i] *= alpha;
            m[i] = mn;
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const float p = ex2_approx(s[u] - ref);
                l[i] += p;
                o[i].x += p * v[u].x; o[i].y += p * v[u].y; o[i].z += p * v[u].z; o[i].w += p * v[u].w;
            }
        }
    }
    // the two half-warps, then the warps of the CTA
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        float4 o2;
        o2.x = __shfl_xor_sync(0xffffffffu, o[i].x, 16); o2.y = __shfl_xor_sync(0xffffffffu, o[i].y, 16);
        o2.z = __shfl_xor_sync(0xffffffffu, o[i].z, 16); o2.w = __shfl_xor_sync(0xffffffffu, o[i].w, 16);
        fold(m[i], l[i], o[i], __shfl_xor_sync(0xffffffffu, m[i], 16), __shfl_xor_sync(0xffffffffu, l[i], 16), o2);
        if (half == 0) {
            reinterpret_cast<float4*>(part[warp].o[i])[sub] = o[i];
            if (sub == 0) {
                part[warp].m[i] = m[i];
                part[warp].l[i] = l[i];
            }
        }
    }
    __syncthreads();
    const int qi = threadIdx.x >> 4;  // 16 threads per query row
    const bool mine = qi < NQ && qi < a.Tq;
    float M = -INFINITY, L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mine)
        for (int w = 0; w < n_warps; ++w)
            fold(M, L, acc, part[w].m[qi], part[w].l[qi], reinterpret_cast<const float4*>(part[w].o[qi])[sub]);
    if (ns > 1) {
        __syncthreads();
        if (mine) {
            reinterpret_cast<float4*>(part[0].o[qi])[sub] = acc;
            if (sub == 0) {
                part[0].m[qi] = M;
                part[0].l[qi] = L;
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (split == 0 && mine)
            for (int s = 1; s < ns; ++s)
                fold(M, L, acc, ld_cluster_f(mapa(&part[0].m[qi], s)), ld_cluster_f(mapa(&part[0].l[qi], s)),
                     ld_cluster_f4(mapa(reinterpret_cast<const float4*>(part[0].o[qi]) + sub, s)));
    }
    if (split == 0 && mine) {
        const float f = L > 0.f ? 1.f / L : 0.f;
        reinterpret_cast<float4*>(a.O + (int64_t)b * a.o_sB + (int64_t)h * a.o_sH + qi * a.o_sM)[sub] =
            make_float4(acc.x * f, acc.y * f, acc.z * f, acc.w * f);
        if (sub == 0) a.LSE[(int64_t)b * a.lse_sB + (int64_t)h * a.lse_sH + qi] = L > 0.f ? (M + log2f(L)) * LN2 : -INFINITY;
    }
    if (ns > 1) {  // the partial results of the other CTAs have been read
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
}

// Warps of a CTA and CTAs of a slice (a cluster of up to eight, the portable size): as many warps per slice as should all be
// resident at once by the estimate below, each with at least one batch of rows.  A second wave finds a chip that the first is leaving a CTA at a
// time.  B4 H8, 8 191 keys: 25.0 us with 14 warps per SM, 37.7 with 28 wanted and 24 that fit; B16 H12, 2 047 keys: 33.0 with 21, 37.1
// with 42, 36.6 with 10; B64 H16, 511 keys: 45.3 one CTA per slice, 48 - 63 with more.  Slices that do not fit at all take
// one CTA each.
// Of equal numbers the order decides.  One CTA of sixteen warps is faster than two of eight (120 slices of 2 056 keys 22.1 and
// 24.8 us); two of sixteen than four of eight only where these no longer get an SM each (68 slices 15.5 and 16.2; 4 slices of
// 359 keys 4.9 and 4.3; two query rows: 64 slices 15.9 and 15.6).
// What fits is an estimate.  The device is asked how many clusters of the forward kernel, one CTA per SM, it holds
// (attn_fwd_slots); here an SM holds two to six CTAs by the kernels' launch bounds, and the number of clusters is taken to grow
// with that.  Clusters of eight pack better than this two and three to an SM: with 15 of them at one CTA per SM, 48 slices
// still run at once at three (12.7 us), 52 do not (19.0), hence 0.87 of the places.  That share is measured on a chip of 148
// SMs; elsewhere, and where the estimate is off, a call takes a wave more or leaves places empty, nothing else.
DecodePlan plan_attn_decode(int BH, int Tq, int Tk, const int slots[4]) {
    static const DecodePlan order[2][9] = {{{8, 4}, {16, 1}, {16, 2}, {8, 2}, {8, 1}, {16, 8}, {16, 4}, {8, 8}, {4, 1}},
                                           {{16, 2}, {16, 1}, {8, 4}, {8, 2}, {8, 1}, {16, 8}, {16, 4}, {8, 8}, {4, 1}}};
    DecodePlan best{Tq == 1 ? 8 : 4, 1};
    int most = 0;
    for (const DecodePlan& p : order[Tq == 1 && 2 * BH > 3 * slots[2]]) {
        const int per_sm = (Tq == 1 ? 24 : 16) / p.warps;  // by the kernels' launch bounds
        int fit = per_sm * slots[p.n_splits == 8 ? 3 : p.n_splits == 4 ? 2 : p.n_splits == 2 ? 1 : 0];
        if (p.n_splits == 8 && per_sm > 1) fit = std::max(fit, (int)(0.87 * slots[0] * per_sm / 8));
        const int n = p.warps * p.n_splits;
        if (BH <= fit && (long long)n * 2 * dec::UNROLL <= Tk && n > most) {
            most = n;
            best = p;
        }
    }
    return best;
}

int launch_attn_decode(DecodeArgs a, cudaStream_t stream) {
    typedef void (*Kernel)(DecodeArgs);
    static const Kernel kernels[2][3] = {{attn_decode_kernel<1, 4>, attn_decode_kernel<1, 8>, attn_decode_kernel<1, 16>},
                                         {attn_decode_kernel<2, 4>, attn_decode_kernel<2, 8>, attn_decode_kernel<2, 16>}};
    const int* slots = nullptr;
    const int slots_rc = attn_fwd_slots(&slots);
    if (slots_rc != HK_OK) return slots_rc;
    const DecodePlan plan = plan_attn_decode(a.BH, a.Tq, a.Tk, slots);
    const int warps = plan.warps;
    const Kernel k = kernels[a.Tq - 1][warps == 4 ? 0 : warps == 8 ? 1 : 2];
    a.n_splits = plan.n_splits;
    const long long blocks = (long long)a.BH * a.n_splits;
    if (blocks > 0x7fffffffLL) return HK_ERR_BAD_SHAPE;
    LaunchConfig lc((unsigned)blocks, warps * 32, warps * sizeof(dec::Partial), stream, a.n_splits, true);
    timing_mark(TIMED_FWD, true, stream);
    const cudaError_t rc = cudaLaunchKernelEx(&lc.cfg, k, a);
    timing_mark(TIMED_FWD, false, stream);
    count_launch();
    return rc == cudaSuccess ? HK_OK : check_launch();
}

}  // namespace hk

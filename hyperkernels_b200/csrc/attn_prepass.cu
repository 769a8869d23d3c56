// attn_prepass.cu -- the HBM-bound helper kernels around the two tensor-core
// kernels: TF32 operand rounding, D = rowsum(dO * O), dQ zeroing and the
// softmax merge of two partial forward results.
#include "attn_prepass.cuh"

#include <algorithm>

namespace hk {

// ---------------------------------------------------------------------------
// TF32 rounding of contiguous rows (hk_attn_round_tf32).  The reference adds 0x1000 to the bit pattern of every MMA
// operand as it loads it from shared memory (fused_attn_forward_kernel_tc_sm89.cu:197,209-210,219;
// mem_efficient_bwd_unified_kernel_exp12.cu:118,127,136), i.e. round to nearest, ties away.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) round_tf32_kernel(const float* src, float* dst_, long long nvec) {
    uint4* dst = reinterpret_cast<uint4*>(dst_);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec;
         i += (long long)gridDim.x * blockDim.x) {
        // plain load: dst may be src, which rules the read-only path out
        const uint4 x = reinterpret_cast<const uint4*>(src)[i];
        dst[i] = make_uint4(tf32_round_bits(x.x), tf32_round_bits(x.y), tf32_round_bits(x.z), tf32_round_bits(x.w));
    }
}

int launch_round_tf32(const float* src, float* dst, int64_t rows, cudaStream_t stream) {
    const long long nvec = (long long)rows * 16;  // 16 float4 per 64-float row
    if (nvec == 0) return HK_OK;
    const int blocks = (int)std::min<long long>((nvec + 255) / 256, sm_count() * 8);
    round_tf32_kernel<<<blocks, 256, 0, stream>>>(src, dst, nvec);
    count_launch();
    return check_launch();
}

// ---------------------------------------------------------------------------
// Row bookkeeping of the kernels below: row -> (b, h, r) with 32-bit divisions (a 64-bit one costs more instructions than
// the rest of a row's work).  The launchers cut anything of 2^31 rows or more into runs of batches.
// ---------------------------------------------------------------------------
struct RowPos {
    int b, h, r;
};
__device__ __forceinline__ RowPos row_pos(uint32_t row, uint32_t T, uint32_t H) {
    const uint32_t bh = row / T, b = bh / H;
    return {(int)b, (int)(bh - b * H), (int)(row - bh * T)};
}
__device__ __forceinline__ int64_t row_off(const RowPos& p, int64_t sB, int64_t sM, int64_t sH) {
    return (int64_t)p.b * sB + (int64_t)p.h * sH + (int64_t)p.r * sM;
}
// batches that fit one launch
static int batches_per_launch(int B, int H, int T) {
    const long long per = (long long)H * T;
    return (int)std::max<long long>(1, std::min<long long>(B, ((1LL << 31) - 1) / per));
}

constexpr int ROWS_PER_BLOCK = 64;  // 256 threads: 16 lanes per row, four rows per lane

// ---------------------------------------------------------------------------
// D[b,h,i] = sum_k dO[i,k] * O[i,k]  (mem_efficient_bwd_precompute_D_sm89.cu:45-91),
// 16 lanes per row, one float4 of each operand per lane.  Optionally also
// zeroes the matching rows of dQ (the reference leaves that to its caller,
// kernels_test.cu:562).  HBM-bound: a lane issues the eight loads of its four rows before it uses the first.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) precompute_D_kernel(const DJob j, uint32_t nrows) {
    pdl_wait();     // O comes from the forward
    pdl_trigger();  // the backward sets itself up and loads its first tiles meanwhile
    const int sub = threadIdx.x & 15;
    const uint32_t row0 = blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 4);
    float4 g[4], o[4];
    RowPos p[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const uint32_t row = min(row0 + 16 * u, nrows - 1);  // rows past the end are computed and not stored
        p[u] = row_pos(row, j.T, j.H);
        g[u] = __ldg(reinterpret_cast<const float4*>(j.dO.ptr + row_off(p[u], j.dO.sB, j.dO.sM, j.dO.sH)) + sub);
        o[u] = __ldg(reinterpret_cast<const float4*>(j.O.ptr + row_off(p[u], j.O.sB, j.O.sM, j.O.sH)) + sub);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const bool valid = row0 + 16 * u < nrows;
        if (j.dQ_zero && valid)
            reinterpret_cast<float4*>(j.dQ_zero + row_off(p[u], j.dq_sB, j.dq_sM, j.dq_sH))[sub] = make_float4(0.f, 0.f, 0.f, 0.f);
        float s = g[u].x * o[u].x + g[u].y * o[u].y + g[u].z * o[u].z + g[u].w * o[u].w;
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (sub == 0 && valid) j.D[(int64_t)p[u].b * j.d_sB + (int64_t)p[u].h * j.d_sH + p[u].r] = s;
    }
}

int launch_precompute_D(const DJob& job, cudaStream_t stream) {
    const int B = job.BH / job.H, step = batches_per_launch(B, job.H, job.T);
    for (int b = 0; b < B; b += step) {
        DJob j = job;
        j.dO.ptr += b * j.dO.sB;
        j.O.ptr += b * j.O.sB;
        j.D += b * j.d_sB;
        if (j.dQ_zero) j.dQ_zero += b * j.dq_sB;
        const uint32_t nrows = (uint32_t)std::min(step, B - b) * j.H * j.T;
        LaunchConfig lc((nrows + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK, 256, 0, stream, 1, true);
        if (cudaLaunchKernelEx(&lc.cfg, precompute_D_kernel, j, nrows) != cudaSuccess) return check_launch();
        count_launch();
    }
    return check_launch();
}

// ---------------------------------------------------------------------------
// The same row sum for the other head dimensions the reference instantiates
// (mem_efficient_bwd_precompute_D_sm89.cu:93-102: 16, 32, 48, 64, 80, 96, 128,
// 160, 192, 256).  A row of HD floats is HD/4 float4; LANES lanes (a power of
// two, at most a warp) share a row and each takes every LANES-th float4, so
// the dimensions that are not powers of two leave some lanes idle in the last
// round; shuffle reduction within the group.
// ---------------------------------------------------------------------------
template <int HD>
__global__ void __launch_bounds__(256) precompute_D_hd_kernel(const DJob j) {
    constexpr int NV = HD / 4;                                        // float4 per row
    constexpr int LANES = NV >= 32 ? 32 : NV >= 16 ? 16 : NV >= 8 ? 8 : 4;  // lanes that share a row
    constexpr int ROUNDS = (NV + LANES - 1) / LANES;
    const long long nrows = (long long)j.BH * j.T;
    const int sub = threadIdx.x % LANES;
    const long long stride = ((long long)gridDim.x * blockDim.x) / LANES;
    const long long rows_pad = (nrows + 32 / LANES - 1) / (32 / LANES) * (32 / LANES);  // whole warps iterate together
    for (long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES; row < rows_pad; row += stride) {
        float s = 0.f;
        int b = 0, h = 0, r = 0;
        if (row < nrows) {
            const int bh = (int)(row / j.T);
            r = (int)(row - (long long)bh * j.T);
            b = bh / j.H;
            h = bh - b * j.H;
            const float4* g4 = reinterpret_cast<const float4*>(j.dO.ptr + (int64_t)b * j.dO.sB + (int64_t)h * j.dO.sH +
                                                               (int64_t)r * j.dO.sM);
            const float4* o4 = reinterpret_cast<const float4*>(j.O.ptr + (int64_t)b * j.O.sB + (int64_t)h * j.O.sH +
                                                               (int64_t)r * j.O.sM);
#pragma unroll
            for (int v = 0; v < ROUNDS; ++v) {
                const int c = sub + v * LANES;
                if (NV % LANES == 0 || c < NV) {
                    const float4 g = __ldg(g4 + c), o = __ldg(o4 + c);
                    s += g.x * o.x + g.y * o.y + g.z * o.z + g.w * o.w;
                }
            }
        }
#pragma unroll
        for (int off = LANES / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (row < nrows && sub == 0) j.D[(int64_t)b * j.d_sB + (int64_t)h * j.d_sH + r] = s;
    }
}

template <int HD>
static void launch_D_hd(const DJob& j, cudaStream_t stream) {
    constexpr int NV = HD / 4;
    constexpr int LANES = NV >= 32 ? 32 : NV >= 16 ? 16 : NV >= 8 ? 8 : 4;
    const long long nrows = (long long)j.BH * j.T;
    const int blocks = (int)std::min<long long>((nrows * LANES + 255) / 256, sm_count() * 8);
    precompute_D_hd_kernel<HD><<<blocks, 256, 0, stream>>>(j);
}

int launch_precompute_D_hd(const DJob& j, int head_dim, cudaStream_t stream) {
    const long long nrows = (long long)j.BH * j.T;
    if (nrows == 0) return HK_OK;
    switch (head_dim) {
        case 16: launch_D_hd<16>(j, stream); break;
        case 32: launch_D_hd<32>(j, stream); break;
        case 48: launch_D_hd<48>(j, stream); break;
        case 64: launch_D_hd<64>(j, stream); break;
        case 80: launch_D_hd<80>(j, stream); break;
        case 96: launch_D_hd<96>(j, stream); break;
        case 128: launch_D_hd<128>(j, stream); break;
        case 160: launch_D_hd<160>(j, stream); break;
        case 192: launch_D_hd<192>(j, stream); break;
        case 256: launch_D_hd<256>(j, stream); break;
        default: return HK_ERR_UNSUPPORTED;
    }
    count_launch();
    return check_launch();
}

// ---------------------------------------------------------------------------
// zero a strided [B, H, T, 64] tensor (dQ is accumulated with atomics; the
// reference leaves this to its caller, kernels_test.cu:562)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) zero_rows_kernel(float* ptr, int64_t sB, int64_t sM, int64_t sH, int H, int T,
                                                        uint32_t nrows) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const uint32_t row = blockIdx.x * ROWS_PER_BLOCK + 16 * u + (threadIdx.x >> 4);
        if (row < nrows)
            reinterpret_cast<float4*>(ptr + row_off(row_pos(row, T, H), sB, sM, sH))[threadIdx.x & 15] =
                make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

int launch_zero_rows(float* ptr, int64_t sB, int64_t sM, int64_t sH, int B, int H, int T, cudaStream_t stream) {
    const int step = batches_per_launch(B, H, T);
    for (int b = 0; b < B; b += step) {
        const uint32_t nrows = (uint32_t)std::min(step, B - b) * H * T;
        zero_rows_kernel<<<(nrows + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK, 256, 0, stream>>>(ptr + b * sB, sB, sM, sH, H, T, nrows);
        count_launch();
    }
    return check_launch();
}

// ---------------------------------------------------------------------------
// Deterministic dQ: add the per-KV-tile slabs in KV-tile order.  A query tile is in the slab of KV tile kt only if
// the backward CTA of kt visited it (attn_bwd_sm100.cu computes the same bound).  HBM-bound: the slabs are read four at
// a time, all loads before the first addition.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) reduce_dq_slabs_kernel(DqReduceJob j, uint32_t nrows) {
    const uint32_t row = blockIdx.x * 16u + (threadIdx.x >> 4);
    if (row >= nrows) return;
    const int sub = threadIdx.x & 15;
    const RowPos p = row_pos(row, j.T, j.H);
    // KV tiles 0 .. n-1 visited this row's query tile: under the causal mask those whose first key is not past its end
    int n = j.n_kvtiles;
    if (j.causal) {
        const long long end = (long long)(p.r / TILE + 1) * TILE + j.q_pos0 - j.k_pos0;
        n = (int)max(0ll, min((long long)n, (end + TILE - 1) / TILE));
    }
    float4* out = reinterpret_cast<float4*>(j.dQ + row_off(p, j.dq_sB, j.dq_sM, j.dq_sH)) + sub;
    float4 acc = j.accumulate ? *out : make_float4(0.f, 0.f, 0.f, 0.f);
    const int64_t slab = (int64_t)j.slab_rows * 16;  // float4 per slab
    const float4* src = reinterpret_cast<const float4*>(j.slabs) + (int64_t)row * 16 + sub;
    for (int kt = 0; kt < n; kt += 4) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            v[u] = kt + u < n ? __ldcs(src + (kt + u) * slab) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w;
        }
    }
    *out = acc;
}

int launch_reduce_dq_slabs(const DqReduceJob& job, cudaStream_t stream) {
    const int step = batches_per_launch(job.B, job.H, job.T);
    for (int b = 0; b < job.B; b += step) {
        DqReduceJob j = job;
        j.slab_rows = (int64_t)job.B * j.H * j.T;
        j.slabs += (int64_t)b * j.H * j.T * 64;
        j.dQ += b * j.dq_sB;
        const uint32_t nrows = (uint32_t)std::min(step, job.B - b) * j.H * j.T;
        reduce_dq_slabs_kernel<<<(nrows + 15) / 16, 256, 0, stream>>>(j, nrows);
        count_launch();
    }
    return check_launch();
}

// ---------------------------------------------------------------------------
// (O_acc, LSE_acc) <- merge with (O_part, LSE_part): both are normalised
// softmax outputs over disjoint key sets, so
//   LSE = log(exp(LSE_a) + exp(LSE_p)),  O = O_a * exp(LSE_a - LSE) + O_p * exp(LSE_p - LSE).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) merge_partial_kernel(float* O_acc, float* LSE_acc, const float* O_part,
                                                            const float* LSE_part, long long rows) {
    const int sub = threadIdx.x & 15;
    // both half-warps of a warp run the same number of iterations (bound rounded up to even)
    for (long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4; row < ((rows + 1) & ~1ll);
         row += ((long long)gridDim.x * blockDim.x) >> 4) {
        const bool valid = row < rows;
        float wa = 0.f, wp = 0.f, lse = -INFINITY;
        if (valid) {
            const float la = LSE_acc[row], lp = LSE_part[row];
            const float mx = fmaxf(la, lp);
            if (mx > -INFINITY) {
                const float ea = expf(la - mx), ep = expf(lp - mx);
                const float inv = 1.f / (ea + ep);
                wa = ea * inv;
                wp = ep * inv;
                lse = mx + logf(ea + ep);
            }
            float4 x = reinterpret_cast<float4*>(O_acc)[row * 16 + sub];
            const float4 y = __ldg(reinterpret_cast<const float4*>(O_part) + row * 16 + sub);
            x.x = x.x * wa + y.x * wp;
            x.y = x.y * wa + y.y * wp;
            x.z = x.z * wa + y.z * wp;
            x.w = x.w * wa + y.w * wp;
            reinterpret_cast<float4*>(O_acc)[row * 16 + sub] = x;
        }
        __syncwarp();  // every lane has read LSE_acc[row] before lane 0 overwrites it
        if (valid && sub == 0) LSE_acc[row] = lse;
    }
}

int launch_merge_partial(float* O_acc, float* LSE_acc, const float* O_part, const float* LSE_part, long long rows,
                         cudaStream_t stream) {
    if (rows == 0) return HK_OK;
    const int blocks = (int)std::min<long long>((rows * 16 + 255) / 256, sm_count() * 8);
    merge_partial_kernel<<<blocks, 256, 0, stream>>>(O_acc, LSE_acc, O_part, LSE_part, rows);
    count_launch();
    return check_launch();
}

}  // namespace hk

// hk_api.cu -- the extern "C" boundary declared in include/hk_attention.h:
// argument validation, workspace carving, tensor-map construction and the
// launch sequence of each entry point.  No device memory is allocated here.
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "attn_kernels.cuh"
#include "attn_prepass.cuh"
#include "philox.h"

// The leading bytes of both argument blocks must be the reference's by-value
// structs (fused_attn_forward_kernel_tc_sm89.cu:8-29, 192 bytes;
// mem_efficient_bwd_unified_kernel_exp12.cu:11-38, 328 bytes).
static_assert(offsetof(hk_attn_fwd_params, Q) == 0 && offsetof(hk_attn_fwd_params, LSE) == 32, "fwd head");
static_assert(offsetof(hk_attn_fwd_params, B) == 40 && offsetof(hk_attn_fwd_params, nh) == 44, "fwd head");
static_assert(offsetof(hk_attn_fwd_params, T) == 48 && offsetof(hk_attn_fwd_params, scale) == 56, "fwd head");
static_assert(offsetof(hk_attn_fwd_params, is_causal) == 60 && offsetof(hk_attn_fwd_params, dropout_p) == 64, "fwd head");
static_assert(offsetof(hk_attn_fwd_params, dropout_mask) == 72 && offsetof(hk_attn_fwd_params, q_strideB) == 80, "fwd head");
static_assert(offsetof(hk_attn_fwd_params, lse_strideH) == 184 && offsetof(hk_attn_fwd_params, dropout_seed) == 192, "fwd head");
static_assert(offsetof(hk_attn_bwd_params, D) == 48 && offsetof(hk_attn_bwd_params, dV) == 72, "bwd head");
static_assert(offsetof(hk_attn_bwd_params, B) == 80 && offsetof(hk_attn_bwd_params, T) == 88, "bwd head");
static_assert(offsetof(hk_attn_bwd_params, scale) == 92 && offsetof(hk_attn_bwd_params, is_causal) == 96, "bwd head");
static_assert(offsetof(hk_attn_bwd_params, q_strideB) == 104 && offsetof(hk_attn_bwd_params, d_strideH) == 320, "bwd head");
static_assert(sizeof(hk_attn_fwd_params) == 256 && sizeof(hk_attn_bwd_params) == 408, "block sizes");
static_assert(offsetof(hk_attn_bwd_params, dropout_p) == 328, "bwd tail starts after the 328-byte reference block");

namespace hk {


// ---- process-wide state ------------------------------------------------------
static std::atomic<uint64_t> g_launches{0};
void count_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }

int sm_count() {
    static std::atomic<int> cache[HK_MAX_DEVICES];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= HK_MAX_DEVICES) return 148;
    if ((n = cache[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

// ---- optional kernel timing -----------------------------------------------------
static std::atomic<int> g_timing_on{0};
static std::mutex g_timing_mu;
struct EventPair { cudaEvent_t a, b; };
static std::vector<EventPair> g_events[TIMED_KINDS];

void timing_mark(int kind, bool begin, cudaStream_t stream) {
    if (!g_timing_on.load(std::memory_order_relaxed)) return;
    std::lock_guard<std::mutex> lock(g_timing_mu);
    if (begin) {
        EventPair e{};
        if (cudaEventCreate(&e.a) != cudaSuccess || cudaEventCreate(&e.b) != cudaSuccess) return;
        cudaEventRecord(e.a, stream);
        g_events[kind].push_back(e);
    } else if (!g_events[kind].empty()) {
        cudaEventRecord(g_events[kind].back().b, stream);
    }
}

int check_launch() {
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return HK_OK;
    fprintf(stderr, "libhk_attention: kernel launch failed: %s\n", cudaGetErrorString(e));
    return HK_ERR_CUDA;
}

__device__ DeviceStatus g_device_status;  // one instance per device that loads the module

DeviceStatus* device_status_ptr() {
    static DeviceStatus* cache[HK_MAX_DEVICES] = {};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= HK_MAX_DEVICES) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!cache[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_device_status) != cudaSuccess) return nullptr;
        cache[dev] = static_cast<DeviceStatus*>(p);
    }
    return cache[dev];
}

EncodeTiledFn get_encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

int make_tile_map(CUtensorMap* map, const float* ptr, int inner, int B, int H, int64_t T, int64_t sB, int64_t sM,
                  int64_t sH, int box_rows, bool mn_major, bool operand) {
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return HK_ERR_CUDA;
    // A size-1 dimension may carry any stride; give it a harmless valid one.
    if (H == 1) sH = sM * T;
    if (B == 1) sB = (sH * H > sM * T) ? sH * H : sM * T;
    const int boxes = inner / HALF_D;  // a row's 128-byte pieces are a dimension of their own: one copy takes them all
    cuuint64_t dims[5] = {(cuuint64_t)HALF_D, (cuuint64_t)T, (cuuint64_t)boxes, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[4] = {(cuuint64_t)sM * 4, (cuuint64_t)HALF_D * 4, (cuuint64_t)sH * 4, (cuuint64_t)sB * 4};
    cuuint32_t box[5] = {(cuuint32_t)HALF_D, (cuuint32_t)box_rows, (cuuint32_t)boxes, 1, 1};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = enc(map, operand ? CU_TENSOR_MAP_DATA_TYPE_TFLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE,
                     mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? HK_OK : HK_ERR_CUDA;
}

// ---- validation helpers -------------------------------------------------------
static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
static inline bool stride_ok(int64_t s) { return s >= 0 && (s % 4) == 0; }
// A stride of 0 would broadcast one slice over batches or heads; the TMA tensor maps cannot express that.
static inline bool broadcast_stride(int n, int64_t s) { return n > 1 && s == 0; }
static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// The scratch the boundary asks for.  The operands are rounded to TF32 by the copies that bring them into shared memory
// (make_tile_map), so neither call touches it any more, except for the slabs of the deterministic dQ; the sizes and the
// calls that must bring it are part of the C ABI and stay as callers know them.
static bool scratch_optional(uint32_t flags, int64_t Tq, bool causal) {
    if (flags & (HK_FLAG_OPERANDS_PREROUNDED | HK_FLAG_ROUND_IN_HBM)) return false;
    return Tq >= 512 && Tq * (causal ? 1 : 2) <= 2048;
}

static bool scratch_ok(const void* ws, size_t have, size_t need) {
    return need == 0 || (ws && have >= need && !(reinterpret_cast<uintptr_t>(ws) & 255u));
}

// bytes at the head of the backward's workspace in front of the slabs (one tensor each for Q, K, V, dO)
static size_t bwd_head_bytes(const hk_attn_bwd_params* p) {
    if (p->flags & HK_FLAG_OPERANDS_PREROUNDED) return 0;
    const int64_t Tk = p->kv_len > 0 ? p->kv_len : p->T;
    const size_t bh = (size_t)p->B * p->nh;
    return 2 * align_up(bh * p->T * 256, 256) + 2 * align_up(bh * Tk * 256, 256);
}

// 1/(1-p) of the inverted-dropout option, with p as the kernels apply it: the Philox mask drops with
// probability floor(p * 65536) / 65536, a caller's dense mask is taken to have been drawn with p itself.
static float keep_scale_of(float p, int mode, uint32_t flags) {
    if (!(flags & HK_FLAG_DROPOUT_SCALED) || mode == 0) return 1.f;
    const double pe = (mode == 2) ? (double)hk_philox_threshold(p) / 65536.0 : (double)p;
    return (float)(1.0 / (1.0 - pe));
}

static int validate_dropout(float p, const float* mask, uint32_t flags, int64_t k_pos0, int* mode) {
    *mode = 0;
    if (!(p >= 0.f && p < 1.f)) return HK_ERR_BAD_DROPOUT;
    const bool philox = (flags & HK_FLAG_PHILOX_DROPOUT) != 0;
    if (philox && mask) return HK_ERR_BAD_DROPOUT;
    if (p > 0.f) {
        if (philox) {
            if (k_pos0 % 8 != 0) return HK_ERR_UNSUPPORTED;  // one Philox call covers keys 8n .. 8n+7
            *mode = 2;
        } else if (mask) {
            *mode = 1;  // reference semantics: active only when p > 0 and mask != nullptr
        }
    }
    return HK_OK;
}

// A few query rows: the tensor-core kernel would work on 128 rows whatever there are, the decode kernel is bound by reading
// K and V.  Up to two rows: its arithmetic per key grows with them (B8 H12, 2 047 keys: four rows 31 us, eight 54, 29 with
// the tensor cores); below 128 keys there is nothing to split.
static bool decodes(int64_t Tq, int64_t Tk, int dropout_mode, uint32_t flags) {
    return Tq <= DECODE_MAX_Q && Tk >= 128 && dropout_mode == 0 && !(flags & HK_FLAG_CONTINUE_SOFTMAX_STATE);
}

int attn_forward(const hk_attn_fwd_params& pr, cudaStream_t stream, bool check_scratch) {
    const hk_attn_fwd_params* p = &pr;
    if (!p->Q || !p->K || !p->V || !p->O || !p->LSE) return HK_ERR_NULL_POINTER;
    const int64_t Tq = p->T, Tk = p->kv_len > 0 ? p->kv_len : p->T;
    if (p->B <= 0 || p->nh <= 0 || Tq <= 0 || p->kv_len < 0) return HK_ERR_BAD_SHAPE;
    if (Tq > (1 << 30) || Tk > (1 << 30) || (int64_t)p->B * p->nh > (1 << 24)) return HK_ERR_BAD_SHAPE;
    if (p->q_pos0 < 0 || p->k_pos0 < 0 || p->q_pos0 + Tq > (1LL << 31) - 1 || p->k_pos0 + Tk > (1LL << 31) - 1)
        return HK_ERR_BAD_SHAPE;
    if (!aligned16(p->Q) || !aligned16(p->K) || !aligned16(p->V) || !aligned16(p->O)) return HK_ERR_MISALIGNED;
    const int64_t st[] = {p->q_strideB, p->q_strideM, p->q_strideH, p->k_strideB, p->k_strideM, p->k_strideH,
                          p->v_strideB, p->v_strideM, p->v_strideH, p->o_strideB, p->o_strideM, p->o_strideH};
    for (int64_t s : st)
        if (!stride_ok(s)) return HK_ERR_MISALIGNED;
    if (p->q_strideM < HEAD_DIM || p->k_strideM < HEAD_DIM || p->v_strideM < HEAD_DIM || p->o_strideM < HEAD_DIM)
        return HK_ERR_BAD_SHAPE;
    {
        const int64_t sb[] = {p->q_strideB, p->k_strideB, p->v_strideB, p->o_strideB};
        const int64_t sh[] = {p->q_strideH, p->k_strideH, p->v_strideH, p->o_strideH};
        for (int i = 0; i < 4; ++i)
            if (broadcast_stride(p->B, sb[i]) || broadcast_stride(p->nh, sh[i])) return HK_ERR_UNSUPPORTED;
    }
    if (!std::isfinite(p->scale) || p->scale == 0.f) return HK_ERR_BAD_SHAPE;  // masking multiplies -inf by the scale
    int mode = 0;
    int rc = validate_dropout(p->dropout_p, p->dropout_mask, p->flags, p->k_pos0, &mode);
    if (rc != HK_OK) return rc;

    if (check_scratch && !scratch_ok(p->workspace, p->workspace_bytes, hk_attn_fwd_workspace_bytes(p))) return HK_ERR_WORKSPACE;

    const int B = p->B, H = p->nh, BH = B * H;
    if (decodes(Tq, Tk, mode, p->flags)) {
        DecodeArgs d{};
        d.Q = View4{p->Q, p->q_strideB, p->q_strideM, p->q_strideH};
        d.K = View4{p->K, p->k_strideB, p->k_strideM, p->k_strideH};
        d.V = View4{p->V, p->v_strideB, p->v_strideM, p->v_strideH};
        d.O = p->O; d.LSE = p->LSE;
        d.o_sB = p->o_strideB; d.o_sM = p->o_strideM; d.o_sH = p->o_strideH;
        d.lse_sB = p->lse_strideB; d.lse_sH = p->lse_strideH;
        d.H = H; d.BH = BH; d.Tq = (int)Tq; d.Tk = (int)Tk;
        d.q_pos0 = (int)p->q_pos0; d.k_pos0 = (int)p->k_pos0;
        d.scale_log2e = p->scale * LOG2E;
        d.causal = p->is_causal ? 1 : 0;
        return launch_attn_decode(d, stream);
    }
    CUtensorMap mq, mk, mv;
    if ((rc = make_tile_map(&mq, p->Q, HEAD_DIM, B, H, Tq, p->q_strideB, p->q_strideM, p->q_strideH, TILE, false, true))) return rc;
    if ((rc = make_tile_map(&mk, p->K, HEAD_DIM, B, H, Tk, p->k_strideB, p->k_strideM, p->k_strideH, TILE, false, true))) return rc;
    if ((rc = make_tile_map(&mv, p->V, HEAD_DIM, B, H, Tk, p->v_strideB, p->v_strideM, p->v_strideH, TILE, true, true))) return rc;

    FwdArgs a{};
    a.O = p->O; a.LSE = p->LSE;
    a.mask = (mode == 1) ? p->dropout_mask : nullptr;
    a.o_sB = p->o_strideB; a.o_sM = p->o_strideM; a.o_sH = p->o_strideH;
    a.lse_sB = p->lse_strideB; a.lse_sH = p->lse_strideH;
    a.H = H; a.BH = BH; a.Tq = (int)Tq; a.Tk = (int)Tk;
    a.q_pos0 = (int)p->q_pos0; a.k_pos0 = (int)p->k_pos0;
    a.scale_log2e = p->scale * LOG2E;
    a.causal = p->is_causal ? 1 : 0;
    a.dropout_mode = mode;
    a.keep_scale = keep_scale_of(p->dropout_p, mode, p->flags);
    a.drop_scaled = (mode != 0 && (p->flags & HK_FLAG_DROPOUT_SCALED)) ? 1 : 0;
    a.continue_state = (p->flags & HK_FLAG_CONTINUE_SOFTMAX_STATE) ? 1 : 0;
    if (a.continue_state && a.drop_scaled) return HK_ERR_UNSUPPORTED;
    a.drop_thr = hk_philox_threshold(p->dropout_p);
    a.philox_keys = hk_philox_keys(p->dropout_seed, p->dropout_offset);
    a.philox_offset = (uint32_t)p->dropout_offset;
    a.bh_pos0 = p->bh_pos0;
    a.status = device_status_ptr();
    if (!a.status) return HK_ERR_CUDA;
    CUtensorMap mo;
    if ((rc = make_tile_map(&mo, p->O, HEAD_DIM, B, H, Tq, p->o_strideB, p->o_strideM, p->o_strideH, TILE))) return rc;
    return launch_attn_fwd(mq, mk, mv, mo, a, stream);
}

int attn_backward(const hk_attn_bwd_params& pr, cudaStream_t stream, bool check_scratch) {
    const hk_attn_bwd_params* p = &pr;
    if (!p->Q || !p->K || !p->V || !p->dO || !p->LSE || !p->D || !p->dQ || !p->dK || !p->dV) return HK_ERR_NULL_POINTER;
    const bool d_given = (p->flags & HK_FLAG_D_PRECOMPUTED) != 0;
    if (!d_given && !p->O) return HK_ERR_NULL_POINTER;
    const int64_t Tq = p->T, Tk = p->kv_len > 0 ? p->kv_len : p->T;
    if (p->B <= 0 || p->nh <= 0 || Tq <= 0 || p->kv_len < 0) return HK_ERR_BAD_SHAPE;
    if (Tk > (1 << 30) || (int64_t)p->B * p->nh > (1 << 24)) return HK_ERR_BAD_SHAPE;
    if (p->q_pos0 < 0 || p->k_pos0 < 0 || p->q_pos0 + Tq > (1LL << 31) - 1 || p->k_pos0 + Tk > (1LL << 31) - 1)
        return HK_ERR_BAD_SHAPE;
    const void* ptrs[] = {p->Q, p->K, p->V, p->dO, p->dQ, p->dK, p->dV};
    for (const void* q : ptrs)
        if (!aligned16(q)) return HK_ERR_MISALIGNED;
    if (!d_given && !aligned16(p->O)) return HK_ERR_MISALIGNED;
    const int64_t st[] = {p->q_strideB,  p->q_strideM,  p->q_strideH,  p->k_strideB,  p->k_strideM,  p->k_strideH,
                          p->v_strideB,  p->v_strideM,  p->v_strideH,  p->o_strideB,  p->o_strideM,  p->o_strideH,
                          p->do_strideB, p->do_strideM, p->do_strideH, p->dq_strideB, p->dq_strideM, p->dq_strideH,
                          p->dk_strideB, p->dk_strideM, p->dk_strideH, p->dv_strideB, p->dv_strideM, p->dv_strideH};
    for (int64_t s : st)
        if (!stride_ok(s)) return HK_ERR_MISALIGNED;
    if (p->q_strideM < HEAD_DIM || p->k_strideM < HEAD_DIM || p->v_strideM < HEAD_DIM || p->do_strideM < HEAD_DIM ||
        p->dq_strideM < HEAD_DIM || p->dk_strideM < HEAD_DIM || p->dv_strideM < HEAD_DIM)
        return HK_ERR_BAD_SHAPE;
    {
        const int64_t sb[] = {p->q_strideB, p->k_strideB, p->v_strideB, p->do_strideB, p->dq_strideB, p->dk_strideB, p->dv_strideB};
        const int64_t sh[] = {p->q_strideH, p->k_strideH, p->v_strideH, p->do_strideH, p->dq_strideH, p->dk_strideH, p->dv_strideH};
        for (int i = 0; i < 7; ++i)
            if (broadcast_stride(p->B, sb[i]) || broadcast_stride(p->nh, sh[i])) return HK_ERR_UNSUPPORTED;
    }
    if (!std::isfinite(p->scale) || p->scale == 0.f) return HK_ERR_BAD_SHAPE;  // as in the forward
    int mode = 0;
    int rc = validate_dropout(p->dropout_p, p->dropout_mask, p->flags, p->k_pos0, &mode);
    if (rc != HK_OK) return rc;

    const int B = p->B, H = p->nh, BH = B * H;
    if (check_scratch && !scratch_ok(p->workspace, p->workspace_bytes, hk_attn_bwd_workspace_bytes(p))) return HK_ERR_WORKSPACE;
    const bool det_dq = (p->flags & HK_FLAG_DETERMINISTIC_DQ) != 0;
    const int n_kvtiles = (int)((Tk + TILE - 1) / TILE);
    float* dq_slabs = nullptr;
    if (det_dq) {
        if ((int64_t)n_kvtiles * B > (1 << 24)) return HK_ERR_BAD_SHAPE;
        if (!p->workspace) return HK_ERR_WORKSPACE;
        dq_slabs = reinterpret_cast<float*>(static_cast<uint8_t*>(p->workspace) + (check_scratch ? bwd_head_bytes(p) : 0));
    }
    BwdMaps m;
    auto operand = [&](CUtensorMap* map, const float* ptr, int64_t T, int64_t sB, int64_t sM, int64_t sH, bool mn) {
        return make_tile_map(map, ptr, HEAD_DIM, B, H, T, sB, sM, sH, TILE, mn, true);
    };
    if ((rc = operand(&m.q, p->Q, Tq, p->q_strideB, p->q_strideM, p->q_strideH, false))) return rc;
    if ((rc = operand(&m.k, p->K, Tk, p->k_strideB, p->k_strideM, p->k_strideH, false))) return rc;
    if ((rc = operand(&m.v, p->V, Tk, p->v_strideB, p->v_strideM, p->v_strideH, false))) return rc;
    if ((rc = operand(&m.dO, p->dO, Tq, p->do_strideB, p->do_strideM, p->do_strideH, false))) return rc;
    if ((rc = operand(&m.q_mn, p->Q, Tq, p->q_strideB, p->q_strideM, p->q_strideH, true))) return rc;
    if ((rc = operand(&m.k_mn, p->K, Tk, p->k_strideB, p->k_strideM, p->k_strideH, true))) return rc;
    if ((rc = operand(&m.dO_mn, p->dO, Tq, p->do_strideB, p->do_strideM, p->do_strideH, true))) return rc;
    if (det_dq) {
        // the slabs as one tensor [n_kvtiles * B, H, Tq, 64]: KV tile kt of batch b is "batch" kt * B + b
        if ((rc = make_tile_map(&m.dQ, dq_slabs, HEAD_DIM, n_kvtiles * B, H, Tq, (int64_t)H * Tq * 64, 64, Tq * 64, TILE, false)))
            return rc;
    } else if ((rc = make_tile_map(&m.dQ, p->dQ, HEAD_DIM, B, H, Tq, p->dq_strideB, p->dq_strideM, p->dq_strideH, TILE, false)))
        return rc;
    if ((rc = make_tile_map(&m.dK, p->dK, HEAD_DIM, B, H, Tk, p->dk_strideB, p->dk_strideM, p->dk_strideH, TILE, false)))
        return rc;
    if ((rc = make_tile_map(&m.dV, p->dV, HEAD_DIM, B, H, Tk, p->dv_strideB, p->dv_strideM, p->dv_strideH, TILE, false)))
        return rc;
    if (!d_given) {
        DJob j{};
        j.dO = View4{p->dO, p->do_strideB, p->do_strideM, p->do_strideH};
        j.O = View4{p->O, p->o_strideB, p->o_strideM, p->o_strideH};
        j.D = p->D; j.d_sB = p->d_strideB; j.d_sH = p->d_strideH;
        if (!(p->flags & HK_FLAG_ACCUM_DQ) && !det_dq) {  // the slab reduction overwrites dQ
            j.dQ_zero = p->dQ; j.dq_sB = p->dq_strideB; j.dq_sM = p->dq_strideM; j.dq_sH = p->dq_strideH;
        }
        j.H = H; j.BH = BH; j.T = (int)Tq;
        if ((rc = launch_precompute_D(j, stream))) return rc;
    } else if (!(p->flags & HK_FLAG_ACCUM_DQ) && !det_dq) {
        if ((rc = launch_zero_rows(p->dQ, p->dq_strideB, p->dq_strideM, p->dq_strideH, B, H, (int)Tq, stream))) return rc;
    }

    BwdArgs a{};
    a.LSE = p->LSE; a.D = p->D; a.dQ = p->dQ; a.dK = p->dK; a.dV = p->dV;
    a.mask = (mode == 1) ? p->dropout_mask : nullptr;
    a.lse_sB = p->lse_strideB; a.lse_sH = p->lse_strideH; a.d_sB = p->d_strideB; a.d_sH = p->d_strideH;
    a.dq_sB = p->dq_strideB; a.dq_sM = p->dq_strideM; a.dq_sH = p->dq_strideH;
    a.dk_sB = p->dk_strideB; a.dk_sM = p->dk_strideM; a.dk_sH = p->dk_strideH;
    a.dv_sB = p->dv_strideB; a.dv_sM = p->dv_strideM; a.dv_sH = p->dv_strideH;
    a.H = H; a.BH = BH; a.Tq = (int)Tq; a.Tk = (int)Tk;
    a.det_dq = det_dq ? 1 : 0;
    a.B = B;
    a.q_pos0 = (int)p->q_pos0; a.k_pos0 = (int)p->k_pos0;
    a.scale = p->scale; a.scale_log2e = p->scale * LOG2E;
    a.causal = p->is_causal ? 1 : 0;
    a.accum_dkdv = (p->flags & HK_FLAG_ACCUM_DKDV) ? 1 : 0;
    a.dropout_mode = mode;
    a.drop_scaled = (mode != 0 && (p->flags & HK_FLAG_DROPOUT_SCALED)) ? 1 : 0;
    a.dv_scale = keep_scale_of(p->dropout_p, mode, p->flags);
    a.dp_scale = p->scale * a.dv_scale;
    a.drop_thr = hk_philox_threshold(p->dropout_p);
    a.philox_keys = hk_philox_keys(p->dropout_seed, p->dropout_offset);
    a.philox_offset = (uint32_t)p->dropout_offset;
    a.bh_pos0 = p->bh_pos0;
    a.status = device_status_ptr();
    if (!a.status) return HK_ERR_CUDA;
    if ((rc = launch_attn_bwd(m, a, !d_given, stream))) return rc;
    if (det_dq) {
        DqReduceJob r{};
        r.slabs = dq_slabs; r.dQ = p->dQ;
        r.dq_sB = p->dq_strideB; r.dq_sM = p->dq_strideM; r.dq_sH = p->dq_strideH;
        r.B = B; r.H = H; r.T = (int)Tq; r.n_kvtiles = n_kvtiles;
        r.causal = a.causal; r.q_pos0 = a.q_pos0; r.k_pos0 = a.k_pos0;
        r.accumulate = (p->flags & HK_FLAG_ACCUM_DQ) ? 1 : 0;
        return launch_reduce_dq_slabs(r, stream);
    }
    return HK_OK;
}

}  // namespace hk

using namespace hk;

extern "C" {

const char* hk_status_string(int s) {
    switch (s) {
        case HK_OK: return "ok";
        case HK_ERR_NULL_POINTER: return "null pointer";
        case HK_ERR_BAD_SHAPE: return "bad shape";
        case HK_ERR_MISALIGNED: return "pointer or stride not 16-byte aligned";
        case HK_ERR_BAD_DROPOUT: return "bad dropout arguments";
        case HK_ERR_WORKSPACE: return "workspace missing or too small";
        case HK_ERR_UNSUPPORTED: return "unsupported combination";
        case HK_ERR_CUDA: return "CUDA error";
        case HK_ERR_DEVICE_TIMEOUT: return "a bounded wait inside a kernel gave up";
        case HK_ERR_STATIC_SCRATCH:
            return "problem needs more scratch than the 24 MiB built into the library; use hk_attn_forward with a workspace";
        default: return "unknown status";
    }
}

void hk_attn_kernel_timing_enable(int on) { g_timing_on.store(on ? 1 : 0); }

int hk_attn_kernel_timing_read(int kind, double* total_ms, int* launches) {
    if (kind < 0 || kind >= TIMED_KINDS || !total_ms || !launches) return HK_ERR_BAD_SHAPE;
    std::lock_guard<std::mutex> lock(g_timing_mu);
    double tot = 0;
    int n = 0;
    for (EventPair& e : g_events[kind]) {
        float ms = 0.f;
        if (cudaEventSynchronize(e.b) == cudaSuccess && cudaEventElapsedTime(&ms, e.a, e.b) == cudaSuccess) {
            tot += ms;
            ++n;
        }
        cudaEventDestroy(e.a);
        cudaEventDestroy(e.b);
    }
    g_events[kind].clear();
    *total_ms = tot;
    *launches = n;
    return HK_OK;
}

uint64_t hk_attn_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

int hk_attn_last_device_status(void) {
    DeviceStatus* d = device_status_ptr();
    if (!d) return HK_ERR_CUDA;
    if (cudaDeviceSynchronize() != cudaSuccess) return HK_ERR_CUDA;
    DeviceStatus h;
    if (cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return HK_ERR_CUDA;
    if (h.code != 0) {
        DeviceStatus z = {0, 0, 0, 0};
        cudaMemcpy(d, &z, sizeof(z), cudaMemcpyHostToDevice);
        return HK_ERR_DEVICE_TIMEOUT;
    }
    return HK_OK;
}

int hk_attn_dropout_mask(float* mask, int BH, int64_t Tq, int64_t Tk, float p, uint64_t seed, uint64_t offset,
                         int64_t q_pos0, int64_t k_pos0) {
    return hk_attn_dropout_mask_slices(mask, 0u, BH, Tq, Tk, p, seed, offset, q_pos0, k_pos0);
}

int hk_attn_dropout_mask_slices(float* mask, uint32_t bh_pos0, int BH, int64_t Tq, int64_t Tk, float p, uint64_t seed,
                                uint64_t offset, int64_t q_pos0, int64_t k_pos0) {
    if (!mask) return HK_ERR_NULL_POINTER;
    if (!(p >= 0.f && p < 1.f)) return HK_ERR_BAD_DROPOUT;
    if (BH < 0 || Tq < 0 || Tk < 0) return HK_ERR_BAD_SHAPE;
    const uint32_t thr = hk_philox_threshold(p);
    for (int bh = 0; bh < BH; ++bh)
        for (int64_t i = 0; i < Tq; ++i) {
            float* row = mask + ((size_t)bh * Tq + i) * Tk;
            for (int64_t j = 0; j < Tk; ++j)
                row[j] = hk_philox_keep(seed, offset, bh_pos0 + (uint32_t)bh, (uint32_t)(q_pos0 + i), (uint32_t)(k_pos0 + j), thr)
                             ? 1.0f
                             : 0.0f;
        }
    return HK_OK;
}

size_t hk_attn_fwd_workspace_bytes(const hk_attn_fwd_params* p) {
    if (!p || (p->flags & HK_FLAG_OPERANDS_PREROUNDED)) return 0;
    if (p->B <= 0 || p->nh <= 0 || p->T <= 0) return 0;
    if (scratch_optional(p->flags, p->T, p->is_causal != 0)) return 0;
    const int64_t Tk = p->kv_len > 0 ? p->kv_len : p->T;
    const size_t bh = (size_t)p->B * p->nh;
    return align_up(bh * p->T * 256, 256) + 2 * align_up(bh * Tk * 256, 256);
}

size_t hk_attn_bwd_workspace_bytes(const hk_attn_bwd_params* p) {
    if (!p || p->B <= 0 || p->nh <= 0 || p->T <= 0) return 0;
    size_t n = bwd_head_bytes(p);
    if (p->flags & HK_FLAG_DETERMINISTIC_DQ) {  // one slab of partial dQ per KV tile
        const int64_t Tk = p->kv_len > 0 ? p->kv_len : p->T;
        n += (size_t)((Tk + TILE - 1) / TILE) * align_up((size_t)p->B * p->nh * p->T * 256, 256);
    }
    return n;
}

int hk_attn_forward(const hk_attn_fwd_params* p, void* stream) {
    if (!p) return HK_ERR_NULL_POINTER;
    return attn_forward(*p, static_cast<cudaStream_t>(stream), true);
}

int hk_attn_backward(const hk_attn_bwd_params* p, void* stream) {
    if (!p) return HK_ERR_NULL_POINTER;
    return attn_backward(*p, static_cast<cudaStream_t>(stream), true);
}

int hk_attn_forward_noscratch(const hk_attn_fwd_params* p, void* stream) {
    return attn_forward(*p, static_cast<cudaStream_t>(stream), false);
}

int hk_attn_backward_noscratch(const hk_attn_bwd_params* p, void* stream) {
    return attn_backward(*p, static_cast<cudaStream_t>(stream), false);
}

int hk_attn_forward_plan(const hk_attn_fwd_params* p, const int* slots, int* plan) {
    const int64_t Tk = p->kv_len > 0 ? p->kv_len : p->T;
    int mode = 0, rc = validate_dropout(p->dropout_p, p->dropout_mask, p->flags, p->k_pos0, &mode);
    if (rc != HK_OK) return rc;
    if (!slots && (rc = attn_fwd_slots(&slots))) return rc;
    if (decodes(p->T, Tk, mode, p->flags)) {
        const DecodePlan d = plan_attn_decode(p->B * p->nh, (int)p->T, (int)Tk, slots);
        plan[0] = -1; plan[1] = d.n_splits; plan[2] = d.warps;
        return HK_OK;
    }
    const FwdPlan f = plan_attn_fwd(p->B * p->nh, (int)p->T, (int)Tk, p->is_causal, (int)p->q_pos0, (int)p->k_pos0, mode != 0, slots);
    plan[0] = f.mode; plan[1] = f.n_splits; plan[2] = f.job;
    return HK_OK;
}

int hk_attn_backward_plan(const hk_attn_bwd_params* p, const int* slots, int* plan) {
    const int64_t Tk = p->kv_len > 0 ? p->kv_len : p->T;
    int rc = HK_OK;
    if (!slots && (rc = attn_bwd_slots(&slots))) return rc;
    const BwdPlan b = plan_attn_bwd(p->B * p->nh, p->T, (int)Tk, p->is_causal, (int)p->q_pos0, (int)p->k_pos0, slots);
    plan[0] = b.n_splits; plan[1] = b.job;
    return HK_OK;
}

void hk_attn_item_order(int all, int n, double slice_bytes, int* pairs) {
    for (int i = 0; i < all * n; ++i) take_in_groups(i, all, n, slices_in_l2(all, slice_bytes), pairs[2 * i], pairs[2 * i + 1]);
}

int hk_attn_forward_run(const hk_attn_fwd_params* p, const int* slots, int* slices) {
    const int BH = p->B * p->nh, Tq = (int)p->T, Tk = (int)(p->kv_len > 0 ? p->kv_len : p->T);
    int mode = 0, rc = validate_dropout(p->dropout_p, p->dropout_mask, p->flags, p->k_pos0, &mode);
    if (rc != HK_OK) return rc;
    if (!slots && (rc = attn_fwd_slots(&slots))) return rc;
    const FwdPlan f = plan_attn_fwd(BH, Tq, Tk, p->is_causal, (int)p->q_pos0, (int)p->k_pos0, mode != 0, slots);
    *slices = fwd_run(f, BH, Tq, Tk, p->is_causal, (int)p->q_pos0, (int)p->k_pos0, mode);
    return HK_OK;
}

int hk_attn_backward_run(const hk_attn_bwd_params* p, const int* slots, int* slices) {
    const int BH = p->B * p->nh, Tk = (int)(p->kv_len > 0 ? p->kv_len : p->T);
    int mode = 0, rc = validate_dropout(p->dropout_p, p->dropout_mask, p->flags, p->k_pos0, &mode);
    if (rc != HK_OK) return rc;
    if (!slots && (rc = attn_bwd_slots(&slots))) return rc;
    const BwdPlan b = plan_attn_bwd(BH, p->T, Tk, p->is_causal, (int)p->q_pos0, (int)p->k_pos0, slots);
    *slices = bwd_run(b, BH, p->T, Tk, mode);
    return HK_OK;
}

int hk_attn_zero_dq(const hk_attn_bwd_params* p, void* stream) {
    if (!p || !p->dQ) return HK_ERR_NULL_POINTER;
    if (p->B <= 0 || p->nh <= 0 || p->T <= 0) return HK_ERR_BAD_SHAPE;
    // the rows are written 16 bytes at a time; the stride of a dimension of one is not used
    if (!aligned16(p->dQ) || (p->B > 1 && !stride_ok(p->dq_strideB)) || (p->nh > 1 && !stride_ok(p->dq_strideH)) ||
        (p->T > 1 && !stride_ok(p->dq_strideM)))
        return HK_ERR_MISALIGNED;
    return launch_zero_rows(p->dQ, p->dq_strideB, p->dq_strideM, p->dq_strideH, p->B, p->nh, p->T, static_cast<cudaStream_t>(stream));
}

int hk_attn_bwd_precompute_D(const hk_attn_bwd_params* p, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!p) return HK_ERR_NULL_POINTER;
    if (!p->dO || !p->O || !p->D) return HK_ERR_NULL_POINTER;
    if (p->B <= 0 || p->nh <= 0 || p->T <= 0) return HK_ERR_BAD_SHAPE;
    if (!aligned16(p->dO) || !aligned16(p->O)) return HK_ERR_MISALIGNED;
    const int64_t st[] = {p->o_strideB, p->o_strideM, p->o_strideH, p->do_strideB, p->do_strideM, p->do_strideH};
    for (int64_t s : st)
        if (!stride_ok(s)) return HK_ERR_MISALIGNED;
    if (p->o_strideM < HEAD_DIM || p->do_strideM < HEAD_DIM) return HK_ERR_BAD_SHAPE;
    DJob j{};
    j.dO = View4{p->dO, p->do_strideB, p->do_strideM, p->do_strideH};
    j.O = View4{p->O, p->o_strideB, p->o_strideM, p->o_strideH};
    j.D = p->D; j.d_sB = p->d_strideB; j.d_sH = p->d_strideH;
    j.dQ_zero = nullptr;
    j.H = p->nh; j.BH = p->B * p->nh; j.T = p->T;
    return launch_precompute_D(j, stream);
}

int hk_attn_bwd_precompute_D_hd(const hk_attn_bwd_params* p, int head_dim, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!p) return HK_ERR_NULL_POINTER;
    if (!p->dO || !p->O || !p->D) return HK_ERR_NULL_POINTER;
    if (p->B <= 0 || p->nh <= 0 || p->T <= 0) return HK_ERR_BAD_SHAPE;
    {
        // the ten instantiations of mem_efficient_bwd_precompute_D_sm89.cu:93-102
        static const int dims[] = {16, 32, 48, 64, 80, 96, 128, 160, 192, 256};
        bool known = false;
        for (int d : dims) known = known || d == head_dim;
        if (!known) return HK_ERR_UNSUPPORTED;
    }
    if (!aligned16(p->dO) || !aligned16(p->O)) return HK_ERR_MISALIGNED;
    const int64_t st[] = {p->o_strideB, p->o_strideM, p->o_strideH, p->do_strideB, p->do_strideM, p->do_strideH};
    for (int64_t s : st)
        if (!stride_ok(s)) return HK_ERR_MISALIGNED;
    if (p->o_strideM < head_dim || p->do_strideM < head_dim) return HK_ERR_BAD_SHAPE;
    DJob j{};
    j.dO = View4{p->dO, p->do_strideB, p->do_strideM, p->do_strideH};
    j.O = View4{p->O, p->o_strideB, p->o_strideM, p->o_strideH};
    j.D = p->D; j.d_sB = p->d_strideB; j.d_sH = p->d_strideH;
    j.H = p->nh; j.BH = p->B * p->nh; j.T = p->T;
    return launch_precompute_D_hd(j, head_dim, stream);
}

int hk_attn_merge_partial(float* O_acc, float* LSE_acc, const float* O_part, const float* LSE_part, int64_t rows,
                          void* stream_) {
    if (!O_acc || !LSE_acc || !O_part || !LSE_part) return HK_ERR_NULL_POINTER;
    if (rows < 0) return HK_ERR_BAD_SHAPE;
    if (!aligned16(O_acc) || !aligned16(O_part)) return HK_ERR_MISALIGNED;
    return launch_merge_partial(O_acc, LSE_acc, O_part, LSE_part, rows, static_cast<cudaStream_t>(stream_));
}

int hk_attn_selftest(int which, const float* A, const float* B, float* out, void* stream_) {
    return run_umma_selftest(which, A, B, out, static_cast<cudaStream_t>(stream_));
}

int hk_attn_round_tf32(const float* src, float* dst, int64_t rows, void* stream_) {
    if (!src || !dst) return HK_ERR_NULL_POINTER;
    if (rows < 0 || rows > (1LL << 31) - 1) return HK_ERR_BAD_SHAPE;
    if (!aligned16(src) || !aligned16(dst)) return HK_ERR_MISALIGNED;
    return launch_round_tf32(src, dst, rows, static_cast<cudaStream_t>(stream_));
}

}  // extern "C"

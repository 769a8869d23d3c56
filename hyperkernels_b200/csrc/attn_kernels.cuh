// attn_kernels.cuh -- argument blocks and launchers of the two tensor-core kernels.
#pragma once
#include <algorithm>

#include "attn_common.cuh"
#include "philox.h"

namespace hk {

// Order of work items: slice `bh` (batch x head) and part `part` of it (a KV tile or a block of rows, 0 the longest) of item
// `item`, where the `n` parts of each of `all` slices are handed out part by part inside runs of `group` slices.  With all slices
// in one run a slice's second part came up when its tensors had long left the L2 again, and every part fetched them (the
// backward's dQ both ways) from memory.  One run -> runs whose tensors take half of the L2 (slices_in_l2), kernels alone, ten launches
// after a pause of 50 ms, 1 965 MHz: backward B32 H25 T1024 780 -> 634 us, B16 H16 T2048 without a mask 1 637 -> 1 258, H32 T32768
// 20 565 -> 18 551; forward 266 -> 254, 495 -> 441, 6 526 -> 5 945.  From memory at B16 H20 T1024: the backward 1 736 -> 631 MB, the
// forward 553 -> 314.  A run also has to be long enough for the CTAs to finish together (longest parts first, and the last run takes
// what is left over): with 8 MB per run the backward of B2 H16 T2000 took 1.24 times as long as with 64 MB or more.  24 to 96 MB are
// within 4 % of each other for most shapes.  How many runs there have to be: fwd_run, bwd_run.
__host__ __device__ __forceinline__ void take_in_groups(int item, int all, int n, int group, int& bh, int& part) {
    int first = 0, size = all;
    if (group < all) {  // with one run the divisions before the first load would cost the smallest calls 1 %
        const int run = item / (n * group), last = all / group - 1;
        first = (run < last ? run : last) * group;
        size = run < last ? group : all - first;
        item -= first * n;
    }
    part = item / size;
    bh = first + (item - part * size);
}

// Slices in a run: the number whose tensors come closest to 64 MB, about half of the 126 MB of L2 of the one chip this is built for,
// and at least one; all, if that leaves one run.  So a run of two slices may be of 85 MB, and one slice of any size; the last run
// holds up to twice the number, which its balance needs more than its loads need the L2.  The slabs of a reproducible dQ and a dense
// mask, which go through once, are not counted, nor is it that a causal mask leaves half of the loads.
inline int slices_in_l2(int all, double slice_bytes) {
    const int group = std::max(1, (int)std::min((double)all, 67108864.0 / slice_bytes + 0.5));
    return all < 2 * group ? all : group;
}

// what the two streams of a forward CTA are (attn_fwd_sm100.cu)
enum FwdMode { FWD_ROWS = 0, FWD_ROW = 1, FWD_KEYS = 2 };

struct FwdArgs {
    float* O;
    float* LSE;
    const float* mask;  // dense dropout mask [BH, Tq, Tk] or nullptr
    int64_t o_sB, o_sM, o_sH, lse_sB, lse_sH;
    int H, BH;
    int Tq, Tk;
    int n_qblocks, n_splits, mode;  // how the work is cut: set by launch_attn_fwd, as is
    int group;                      // slices whose blocks of rows come before those of others (take_in_groups)
    int q_pos0, k_pos0;
    float scale_log2e;
    int causal;
    int dropout_mode;  // 0 none, 1 dense mask, 2 Philox
    int drop_scaled;   // 1: inverted dropout (normaliser over all visible keys, kept terms times keep_scale)
    int continue_state;  // 1: O, LSE hold the result over earlier keys and are the starting state
    float keep_scale;  // 1/(1-p) when drop_scaled, else 1
    uint32_t drop_thr;
    uint32_t bh_pos0;  // added to the local (batch, head) index in the Philox counter
    hk_philox_keys_t philox_keys;
    uint32_t philox_offset;
    DeviceStatus* status;
    uint64_t unused[6];  // up to a size that launches fast: FWD_PARAM_BYTES
};
// The smallest forwards are bound by how fast the host launches them, and that depends on the bytes of parameters, four maps and this
// block: 24 or 32 beyond a multiple of 64 take 2.1 us per launch of an empty kernel, any other number 2.4 to 2.5 (640 to 808 and
// 1 536 to 1 656 bytes in steps of 8).  B2 H25 T68 with 736 or 792 bytes 5.95 us per call, with 744 6.3.
constexpr size_t FWD_PARAM_BYTES = 4 * sizeof(CUtensorMap) + sizeof(FwdArgs);
static_assert(FWD_PARAM_BYTES % 64 == 24 || FWD_PARAM_BYTES % 64 == 32, "a forward's launch would take 0.3 us longer");

// How a forward's work is cut, from sizes and the resident clusters of 1, 2, 4, 8 CTAs (slots) alone.
struct FwdPlan {
    int mode, n_splits, n_qblocks;
    int job;  // FwdJob (attn_fwd_sm100.cu): the kernel that runs it
};
FwdPlan plan_attn_fwd(int BH, int Tq, int Tk, int causal, int q_pos0, int k_pos0, bool drop, const int slots[4]);
int attn_fwd_slots(const int** slots);  // of the current device; status
// slices in a run of its work items, BH where they come in one
int fwd_run(const FwdPlan& plan, int BH, int Tq, int Tk, int causal, int q_pos0, int k_pos0, int dropout_mode);

// mq, mk, mv: TMA maps of the operands (rounded to TF32 by the copy); mo: map of O, the destination of the kernel's bulk stores.
int launch_attn_fwd(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mo,
                    FwdArgs a, cudaStream_t stream);

// A few query rows against many keys (attn_decode.cu): no dropout, no starting state.
constexpr int DECODE_MAX_Q = 2;
struct DecodeArgs {
    View4 Q, K, V;
    float* O;
    float* LSE;
    int64_t o_sB, o_sM, o_sH, lse_sB, lse_sH;
    int H, BH;
    int Tq, Tk;
    int q_pos0, k_pos0;
    float scale_log2e;
    int causal;
    int n_splits;  // set by launch_attn_decode
};
struct DecodePlan {
    int warps, n_splits;
};
DecodePlan plan_attn_decode(int BH, int Tq, int Tk, const int slots[4]);  // slots: as attn_fwd_slots gives them
int launch_attn_decode(DecodeArgs a, cudaStream_t stream);

struct BwdArgs {
    const float* LSE;
    const float* D;
    float* dQ;
    float* dK;
    float* dV;
    const float* mask;
    int64_t lse_sB, lse_sH, d_sB, d_sH;
    int64_t dq_sB, dq_sM, dq_sH, dk_sB, dk_sM, dk_sH, dv_sB, dv_sM, dv_sH;
    int H, BH;
    int Tq, Tk;
    int n_splits;      // CTAs (a cluster) that share the query tiles of a KV tile; this and the next two set by launch_attn_bwd
    int live;          // KV tiles of a slice in the grid
    int group;         // slices whose KV tiles come before those of others (take_in_groups)
    int q_pos0, k_pos0;
    float scale, scale_log2e;
    int causal;
    int accum_dkdv;
    int det_dq;        // 1: dQ tiles are stored (map dQ = the slabs [n_kvtiles * B, H, Tq, 64]) instead of added; B below
    int B;
    int dropout_mode;
    int drop_scaled;   // 1: inverted dropout; p below is then the softmax over all visible keys
    float dp_scale;    // factor of dP inside dS: scale, times 1/(1-p) when drop_scaled
    float dv_scale;    // factor of the dV accumulator: 1/(1-p) when drop_scaled, else 1
    uint32_t drop_thr;
    uint32_t bh_pos0;  // added to the local (batch, head) index in the Philox counter
    hk_philox_keys_t philox_keys;
    uint32_t philox_offset;
    DeviceStatus* status;
};

// K-major maps (16-byte-chunk swizzle) of Q, K, V, dO and MN-major maps
// (32-byte-chunk swizzle) of Q, K, dO over the same memory; dQ, dK, dV are
// the destinations of the kernel's bulk reductions and stores (16-byte-chunk
// swizzle).
struct BwdMaps {
    CUtensorMap q, k, v, dO, q_mn, k_mn, dO_mn, dQ, dK, dV;
};

// How a backward's work is cut, from the same.
struct BwdPlan {
    int n_splits;  // CTAs that share the query tiles of a KV tile
    int live;      // KV tiles that a query tile sees: the others are not in the grid
    int job;       // BwdJob (attn_bwd_sm100.cu): the kernel that runs it
};
BwdPlan plan_attn_bwd(int BH, int Tq, int Tk, int causal, int q_pos0, int k_pos0, const int slots[4]);
int attn_bwd_slots(const int** slots);
int bwd_run(const BwdPlan& plan, int BH, int Tq, int Tk, int dropout_mode);

// after_prepass: the launch before it in the stream is this call's D pre-pass, the only kernel whose results it waits for
// itself (Q, K, V and dO are complete when the pre-pass lets it start)
int launch_attn_bwd(const BwdMaps& m, BwdArgs a, bool after_prepass, cudaStream_t stream);

// What hk_attn_forward / hk_attn_backward run.  check_scratch: ask for the workspace the C ABI documents; without it the
// forward takes none and `workspace` of a deterministic backward holds the slabs of partial dQ alone.
int attn_forward(const hk_attn_fwd_params& p, cudaStream_t stream, bool check_scratch);
int attn_backward(const hk_attn_bwd_params& p, cudaStream_t stream, bool check_scratch);
// the same for callers in this package, by name (dlsym)
extern "C" int hk_attn_forward_noscratch(const hk_attn_fwd_params* p, void* stream);
extern "C" int hk_attn_backward_noscratch(const hk_attn_bwd_params* p, void* stream);
// How the call of this block would be cut, for tests: nothing is launched and no pointer is read.  slots: resident clusters
// of 1, 2, 4, 8 CTAs, or null for those of the current device.  Forward: plan = {FwdMode, or -1 for the decode kernel; CTAs
// that share a block of rows (decode: a slice); FwdJob (decode: warps of a CTA)}.  Backward: plan = {CTAs that share a KV tile;
// BwdJob}.
extern "C" int hk_attn_forward_plan(const hk_attn_fwd_params* p, const int* slots, int* plan);
extern "C" int hk_attn_backward_plan(const hk_attn_bwd_params* p, const int* slots, int* plan);
// The order of the work items (take_in_groups) of `all` slices of `slice_bytes` and `n` parts each, for tests: all * n pairs
// {slice, part}.
extern "C" void hk_attn_item_order(int all, int n, double slice_bytes, int* pairs);
// Slices in a run of the call of this block, all of them where it has one run; for tests, as the plans above.
extern "C" int hk_attn_forward_run(const hk_attn_fwd_params* p, const int* slots, int* slices);
extern "C" int hk_attn_backward_run(const hk_attn_bwd_params* p, const int* slots, int* slices);
// zeroes dQ (fields dQ, dq_stride*, B, nh, T), for a caller that runs the backward with HK_FLAG_ACCUM_DQ
extern "C" int hk_attn_zero_dq(const hk_attn_bwd_params* p, void* stream);

int run_umma_selftest(int which, const float* A, const float* B, float* out, cudaStream_t stream);

}  // namespace hk

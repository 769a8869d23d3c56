// attn_fwd_static.cu -- hk_attn_forward_static_scratch: the forward for callers
// that have no workspace to give: an operator plugged into a host framework that
// owns every byte of device memory through its own pool, a latency-critical
// serving loop in which cudaMalloc/cudaFree would synchronise the whole device,
// or code that runs where the allocator simply is not reachable.
//
// The forward needs no scratch (its operands are rounded to TF32 by the copies
// that load them), so the call only lifts the workspace requirement.  The size
// limit of the entry point, B*nh*(T + 2*kv_len)*256 bytes <= 24 MiB, stays.
#include "attn_kernels.cuh"

extern "C" int hk_attn_forward_static_scratch(const hk_attn_fwd_params* p, void* stream) {
    if (!p) return HK_ERR_NULL_POINTER;
    hk_attn_fwd_params q = *p;  // the caller's block is left untouched
    q.workspace = nullptr;
    q.workspace_bytes = 0;
    q.flags |= HK_FLAG_ROUND_IN_HBM;  // the size the limit is stated for
    if (hk_attn_fwd_workspace_bytes(&q) > HK_STATIC_SCRATCH_BYTES) return HK_ERR_STATIC_SCRATCH;
    return hk::attn_forward(q, static_cast<cudaStream_t>(stream), false);
}

// attn_bwd_sm100.cu -- fused attention backward for sm_100a.
//
// Computes what mem_efficient_bwd_unified_kernel_exp12<64,Causal> computes
// (kernels/attention/mem_efficient_bwd_unified_kernel_exp12.cu:54-329 of the
// reference), a KV tile at a time, looping over the query tiles that can see it:
//   S = Q K^T, dP = dO V^T                    (:186-212)
//   p = exp2(log2e * (S*scale - LSE)), 0 outside bounds / above the diagonal   (:224-227)
//   dS = p * (dP - D) * scale                 (:228)
//   dQ_i += dS K_j   (accumulated into global memory with atomics, :239-282)
//   dK_j += dS^T Q_i (:261-274)     dV_j += P^T dO_i (:285-299)
// plus the dropout keep-mask (p is multiplied by it), which the reference
// backward lacks but its forward implies.
//
// Blackwell structure (a CTA works on one 128-row KV tile at a time, 128-row query tiles):
// the transposed products S^T = K Q^T and dP^T = V dO^T put key rows on the 128
// tensor-memory lanes, so P^T and dS^T -- written back over S^T and dP^T by the
// compute warps -- are directly the tensor-memory A operands of dV += P^T dO and
// dK += dS^T Q.  dS is also staged once through shared memory (MN-major) as the
// A operand of dQ = dS K.  dV, dK (64 columns each) stay in tensor memory for
// the whole KV tile; dQ (64 columns) is drained per query tile; V (64 columns) is
// copied into tensor memory once and is the A operand of dP^T, which frees its
// 32 KiB of shared memory for dS.  Everything the kernel writes leaves through
// shared memory and the TMA unit: dQ tiles are added to global memory with bulk
// reductions (per-thread atomics stall the tensor-core instruction issue of the
// same SM), dV and dK are stored with bulk copies at the end (a thread-per-row
// store touches 32 lines per instruction).
//
// Q, dO and K each feed one product that contracts over d (K-major operand,
// 16-byte-chunk swizzle) and one that contracts over the sequence (MN-major
// operand, which for TF32 must use the 32-byte-chunk swizzle; the tensor core
// refuses the 32-byte-chunk swizzle for a K-major operand), so TMA brings each
// of them into shared memory twice, once per swizzle.
//
// Tensor-pipe order per query tile i:
//     dV(i) | S^T(i+1) | dK(i) | dQ(i) | dP^T(i+1)
// dV(i) starts as soon as P^T(i) is in tensor memory, i.e. before the compute
// warps have formed dS(i); dK(i) follows when dS^T(i) is there, dQ(i) when dS(i)
// is staged in shared memory.
// S^T(i+1) only needs the P^T columns back, i.e. dV(i); issuing it before dK(i)
// lets the compute warps start the exponentials of tile i+1 -- the longest
// stretch of scalar work -- while dK(i), dQ(i) and dP^T(i+1) execute.  Two of the
// four 32-column boxes of dS(i) go over the MN-major dO tile as soon as dV(i) has
// consumed it, so that tile can be loaded for i+1 only when dQ(i) is done, and
// dV(i+1) waits for it: with dQ(i) in front of dP^T(i+1) half of that load is
// hidden (B4 H16 T2048 433 -> 388 us, H32 T8192 1 670 -> 1 500, against dQ last).
// Measured tensor-pipe time of the 72 instructions of a tile: about 3 050 cycles
// (M128 N128 K8: 74 cycles, M128 N64 K8: 36 from tensor memory, 52 from shared
// memory).
//
// Splits: where few KV tiles have many query tiles (cross-attention of a long sequence to a short one), a cluster of 2, 4
// or 8 CTAs shares the query tiles of a KV tile; at the end each adds up a slice of the rows of dV and dK from the partial
// sums the others left in their shared memory (plan_attn_bwd picks the number).  B1 H4, 5 000 queries,
// 200 keys: 107 -> 25 us; B1 H1, 16 384 and 4 096: 330 -> 100.
//
// Where there are more KV tiles than SMs, a CTA that is through with one takes over another of a CTA not started yet (cluster
// launch control, BwdJob::TAKE_OVER): loads and S^T of the next KV tile run under the last products of this one.  B8 H12 T1024
// 108 -> 94 us.  All roles run different code at the same time, so it is kept short: at 194 KiB of text (waits unrolled) the
// first tile of a CTA took 11 000 cycles more than the others, at 108 KiB the loop over the items was 13 - 30 % slower per
// tile than one item per CTA, at 60 KiB no slower.
//
//   warps 0-15  compute: four threads per key row (tensor-memory lane), each
//               owning 32 of the 128 query columns, all held in registers so
//               that S^T and dP^T are read from tensor memory exactly once
//   warp 16     TMA loads (K, V per KV tile; Q and dO per query tile, each in two layouts)
//   warp 17     MMA issuer (the whole warp runs the issuing code, one elected lane
//               issues)
//   warp 18     TMA reductions of dQ (per query tile) and stores of dK, dV (per KV tile)
//   warp 19     LSE and D of the query rows into shared memory
#include <algorithm>
#include <cmath>
#include <mutex>

#include "attn_kernels.cuh"
#include "attn_prepass.cuh"
#include "philox.h"

namespace hk {

namespace bwd {

constexpr int NUM_COMPUTE = 512;
constexpr int NUM_THREADS = NUM_COMPUTE + 128;  // 16 compute warps, 4 control warps
constexpr int W_LOAD = 16, W_MMA = 17, W_STORE = 18, W_ROWS = 19;
constexpr int TMEM_COLS = 512;
constexpr int COL_S = 0;     // S^T, then P^T
constexpr int COL_DP = 128;  // dP^T, then dS^T
constexpr int COL_DV = 256;
constexpr int COL_DK = 320;
constexpr int COL_DQ = 384;
constexpr int COL_V = 448;   // V of this KV tile, A operand of dP^T

// The KV tile of a work item and the query tiles it loops over.
struct Item {
    int b, h, bh, kt;
    int it0, n_it;  // first query tile (with splits: of this CTA) and number of them, 0 with splits alone; -1: there is no item
    int live;       // splits that have query tiles
    int pad;
    __device__ __forceinline__ int kv0() const { return kt * TILE; }
};

// Work items beyond the first that may be known at a time: the load warp can be two items ahead of the store warp and asks
// for one more, into a buffer that every warp has read.
constexpr int ITEMS = 4;

struct __align__(16) Shared {
    float lse[TILE];   // -LSE * log2e of the query tile; -inf for a row that saw no key or is past the end
    float dsum[TILE];  // -D * scale of the query tile
    uint64_t k_full, v_full, km_full, q_full, do_full, qm_full, dom_full;  // TMA loads
    uint64_t v_ready;       // V is in tensor memory (and its landing buffer is free)
    uint64_t qk_free, dok_free;  // S^T(i) / dP^T(i) complete: the K-major Q / dO tile may be refilled
    uint64_t s_full;        // S^T is complete and the query tile's LSE and D are staged
    uint64_t dp_full;
    // One barrier for all four column groups: with one each (so that a group's slices could go as soon as it was in) the
    // issuing warp spent more on the six extra waits per tile than the early start gained (4 - 8 % of the kernel).
    uint64_t pt_ready;      // P^T is in tensor memory: dV += P^T dO may go
    uint64_t p_ready;       // dS^T is in tensor memory: dK += dS^T Q may go
    uint64_t dv_done, dk_done;   // dV(i) / dK(i) complete: the MN-major dO / Q tile is free
    uint64_t ds_ready, dq_full, dq_empty;
    uint64_t dv_staged, dk_staged;  // dV / dK of the CTA is staged for the bulk store
    uint64_t dq_staged;     // dQ of a query tile is staged (in the K-major dO tile) for the bulk reduction
    uint64_t dq_out;        // the bulk reduction has read the staged dQ tile: the K-major dO tile may be refilled
    uint64_t dv_out, dk_out;  // the bulk store has read the staged dV / dK: the MN-major K / Q tile may be refilled
    uint64_t item_full[ITEMS], item_empty[ITEMS];
    Item item[ITEMS];       // the items taken over, decoded
    uint4 answer;           // to a request for one
    uint64_t answered;
    uint32_t tmem_base;
    Abort abort;
};

constexpr int OFF_KK = 0;                // K, K-major swizzle   (S^T = K Q^T)
constexpr int OFF_KM = TILE_BYTES;       // K, MN-major swizzle  (dQ = dS K); staging of dV between items
constexpr int OFF_QK = 2 * TILE_BYTES;   // Q, K-major           (S^T); staging of the last dV
constexpr int OFF_DOK = 3 * TILE_BYTES;  // dO, K-major          (dP^T); staging of dQ
constexpr int OFF_QM = 4 * TILE_BYTES;   // Q, MN-major          (dK += dS^T Q); staging of dK
constexpr int OFF_DS = 5 * TILE_BYTES;   // dS boxes 0, 1 ([128 kv][32 q] each); first of all the landing buffer of V
constexpr int OFF_DOM = 6 * TILE_BYTES;  // dO, MN-major         (dV += P^T dO); dS boxes 2, 3 once dV is done
static_assert(OFF_DOM == OFF_DS + 2 * BOX_BYTES, "the four dS boxes are one descriptor: equally spaced");
constexpr int OFF_SH = 7 * TILE_BYTES;
// no slack for re-aligning the dynamic shared-memory base: it is declared 1024-byte aligned
// and the kernel checks that it is (the 128-byte swizzles need it)
constexpr int SMEM_BYTES = OFF_SH + sizeof(Shared);
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KiB a CTA may opt in to");

enum WaitId {
    W_KVFULL = 201, W_QKFULL, W_QKEMPTY, W_QMFULL, W_QMFREE, W_SFULL, W_PREADY, W_BDONE, W_DSREADY, W_DQFULL, W_DQEMPTY,
    W_ROWSFREE, W_DQSTAGED, W_ACCSTAGED, W_ACCOUT, W_VREADY, W_DVDONE, W_DQOUT, W_ITEM
};

}  // namespace bwd

namespace bwd {
// RUNS: the items may come in runs of slices (take_in_groups), which the kernels that take over decide as they run: kernels of their
// own for one run, as the forward has them, gain nothing here (B16 H12 T256 22.54 us either way).
template <bool RUNS>
__device__ __forceinline__ Item make_item(const BwdArgs& a, int item, int split, int ns) {
    Item x;
    // early KV tiles first: under the causal mask they see the most query tiles
    take_in_groups(item, a.BH, a.live, RUNS ? a.group : a.BH, x.bh, x.kt);
    x.b = x.bh / a.H;
    x.h = x.bh - x.b * a.H;
    const int n_qtiles = (a.Tq + TILE - 1) / TILE;
    // first query tile with a row at or below the diagonal of this KV tile
    x.it0 = 0;
    if (a.causal) {
        const long long first_q = (long long)x.kv0() + a.k_pos0 - a.q_pos0;  // smallest local q that sees key kv0
        if (first_q > 0) x.it0 = (int)min((long long)n_qtiles, first_q / TILE);
    }
    x.n_it = n_qtiles - x.it0;
    x.live = 1;
    if (ns > 1) {  // each CTA of the cluster takes a contiguous run of the query tiles
        const int run = (x.n_it + ns - 1) / ns, n_all = x.n_it;
        x.it0 += split * run;
        x.n_it = max(0, min(run, n_all - split * run));
        x.live = (n_all + run - 1) / max(run, 1);
    }
    return x;
}
}  // namespace bwd

// DROP: 0 none, 1 dense mask, 2 Philox.  JOB: what a CTA does with its items.  SPLIT_ITEM: a cluster shares the query tiles of
// a KV tile (the set-up and the registers it needs cost the plain kernel 1 - 3 %).  A kernel that contains cluster launch
// control is not started under the tail of the one before it, programmatic dependent launch or not, so grids that fit the
// device use one without.
enum BwdJob { ONE_ITEM = 0, TAKE_OVER = 1, SPLIT_ITEM = 2 };
template <int DROP, int JOB>
__global__ void __launch_bounds__(bwd::NUM_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapdO,
                const __grid_constant__ CUtensorMap mapQm, const __grid_constant__ CUtensorMap mapKm,
                const __grid_constant__ CUtensorMap mapdOm, const __grid_constant__ CUtensorMap mapdQ,
                const __grid_constant__ CUtensorMap mapdK, const __grid_constant__ CUtensorMap mapdV,
                const __grid_constant__ BwdArgs a) {
    using namespace bwd;
    constexpr bool SPLIT = JOB == SPLIT_ITEM, TAKES_OVER = JOB == TAKE_OVER;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0) {  // never expected; refuse to run on a misplaced buffer
        if (threadIdx.x == 0 && atomicCAS(&a.status->code, 0, 299) == 0) a.status->block = blockIdx.x;
        return;
    }
    uint8_t* sK = smem + OFF_KK;
    uint8_t* sKm = smem + OFF_KM;
    uint8_t* sV = smem + OFF_DS;  // landing buffer of V, read once into tensor memory
    uint8_t* sQ = smem + OFF_QK;
    uint8_t* sdO = smem + OFF_DOK;
    uint8_t* sQm = smem + OFF_QM;
    uint8_t* sdOm = smem + OFF_DOM;
    uint8_t* sdS = smem + OFF_DS;  // box b at sdS + b * BOX_BYTES
    Shared& sh = *reinterpret_cast<Shared*>(smem + OFF_SH);

    const int warp = (int)uniform(threadIdx.x >> 5);  // uniform for the compiler too: see uniform()
    const int lane = threadIdx.x & 31;

    const int ns = SPLIT ? a.n_splits : 1;  // cluster size
    const int split = SPLIT ? (int)cluster_ctarank() : 0;
    const Item first = make_item<TAKES_OVER>(a, (int)blockIdx.x / ns, split, ns);

    auto load_tile = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int row, const Item& x) {
        mbar_arrive_expect_tx(bar, TILE_BYTES);
        tma_load_tile(dst, map, bar, row, x.h, x.b);
    };
    // everything an item starts with, in the order its first products need it: K, Q (S^T), V, dO (dP^T), MN-major dO (dV),
    // Q (dK), K (dQ)
    auto load_all = [&](const Item& x) {
        load_tile(sK, &mapK, &sh.k_full, x.kv0(), x);
        load_tile(sQ, &mapQ, &sh.q_full, x.it0 * TILE, x);
        load_tile(sV, &mapV, &sh.v_full, x.kv0(), x);
        load_tile(sdO, &mapdO, &sh.do_full, x.it0 * TILE, x);
        load_tile(sdOm, &mapdOm, &sh.dom_full, x.it0 * TILE, x);
        load_tile(sQm, &mapQm, &sh.qm_full, x.it0 * TILE, x);
        load_tile(sKm, &mapKm, &sh.km_full, x.kv0(), x);
    };

    // The load warp initialises the barriers its copies complete on and issues the loads of the first tile at once:
    // the other warps meet those barriers only after the __syncthreads below, and ~1 000 cycles of set-up (the other
    // barriers, the tensor-memory allocation) run under the latency of the first loads instead of before it.
    if (warp == W_LOAD && lane == 0) {
        mbar_init(&sh.k_full, 1);
        mbar_init(&sh.v_full, 1);
        mbar_init(&sh.km_full, 1);
        mbar_init(&sh.q_full, 1);
        mbar_init(&sh.do_full, 1);
        mbar_init(&sh.qm_full, 1);
        mbar_init(&sh.dom_full, 1);
        for (int i = 0; i < ITEMS; ++i) {
            mbar_init(&sh.item_full[i], 1);
            mbar_init(&sh.item_empty[i], NUM_THREADS / 32 - 1);  // every warp but the load warp
        }
        mbar_init(&sh.answered, 1);
        fence_mbar_init();
        if (first.n_it > 0) load_all(first);
    }
    if (threadIdx.x == 0) {
        // compute-warp barriers count one arrival per warp
        mbar_init(&sh.v_ready, 8);    // column groups 2, 3 copy V
        mbar_init(&sh.qk_free, 1);
        mbar_init(&sh.dok_free, 1);
        mbar_init(&sh.s_full, 2);     // the commit of S^T and the warp that stages LSE and D
        mbar_init(&sh.dp_full, 1);
        mbar_init(&sh.pt_ready, NUM_COMPUTE / 32);
        mbar_init(&sh.p_ready, NUM_COMPUTE / 32);
        mbar_init(&sh.dv_done, 1);
        mbar_init(&sh.dk_done, 1);
        mbar_init(&sh.ds_ready, NUM_COMPUTE / 32);
        mbar_init(&sh.dq_full, 1);
        mbar_init(&sh.dq_empty, NUM_COMPUTE / 32);
        mbar_init(&sh.dq_staged, NUM_COMPUTE / 32);
        mbar_init(&sh.dq_out, 1);
        mbar_init(&sh.dv_staged, 8);  // column groups 0, 1
        mbar_init(&sh.dk_staged, 8);  // column groups 2, 3
        mbar_init(&sh.dv_out, 1);
        mbar_init(&sh.dk_out, 1);
        sh.abort.id = 0;
        fence_mbar_init();
    }
    if (warp == W_MMA) {
        tmem_alloc(&sh.tmem_base, TMEM_COLS);
        tmem_relinquish();
        tc_fence_before_sync();
    }
    __syncthreads();
    tc_fence_after_sync();
    // The CTA holds all 512 columns of tensor memory, so its allocation starts at address 0: with the base a constant, so is
    // every operand of the MMAs, and none has to be moved to a uniform register.
    constexpr uint32_t tmem = 0;
    if (sh.tmem_base != tmem) {  // never expected
        sh.abort.id = 298;
    }
    WaitNote wc{&sh.abort};

    // Work items.  A CTA starts with the one of its blockIdx and then, until none is left, takes over those of CTAs that have
    // not started yet (cluster launch control), so that the loads and the first S^T of the next KV tile run under the last
    // products and the stores of this one.  One CTA per item spent ~13 000 cycles on set-up, first loads, first tile and last
    // stores beside ~5 000 per query tile; B8 H12 T1024 (768 items of 1 .. 8 tiles) 104 -> 93 us, B32 H25 T1024 995 -> 895.
    // The load warp asks, decodes the answer and puts the item into a ring that every warp reads in its own time.
    struct Items {
        Item x;    // the current one
        int n;     // items read from the ring
    };
    // Goes on to the next item; false if there is none (or a wait gave up).  All lanes of a warp, or one thread alone (`solo`).
    auto next_item = [&](Items& s, bool solo) -> bool {
        if (!TAKES_OVER) return false;
        const int buf = s.n % ITEMS;
        bool ok = mbar_wait(wc, &sh.item_full[buf], (s.n / ITEMS) & 1, W_ITEM, s.n);
        if (!solo) ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        s.x = sh.item[buf];
        ++s.n;
        if (!solo) __syncwarp();
        if (solo || lane == 0) mbar_arrive(&sh.item_empty[buf]);
        return s.x.n_it >= 0;
    };
    if (warp == W_LOAD) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0 && first.n_it > 0) {
            Item cur = first;
            int published = 0;
            int items = 0;  // whose accumulators have left
            bool tok = true, more = TAKES_OVER;
            // on to the next item: publishes what the request brought
            auto next = [&]() -> bool {
                const int buf = published % ITEMS;
                if (!more || !(tok = mbar_wait(wc, &sh.answered, published & 1, W_ITEM, published))) return false;
                const int id = clc_read(&sh.answer);
                fence_proxy_async_smem();  // the answer's buffer is next written by the async proxy
                if (published >= ITEMS && !(tok = mbar_wait(wc, &sh.item_empty[buf], (published / ITEMS - 1) & 1, W_ITEM, 1000 + published)))
                    return false;
                more = id >= 0;
                if (more) {
                    cur = make_item<true>(a, id, 0, 1);
                    sh.item[buf] = cur;
                } else {
                    sh.item[buf].n_it = -1;
                }
                mbar_arrive(&sh.item_full[buf]);
                ++published;
                return more;
            };
            // The query tiles of all items in a row: iteration n of the loop loads K-major Q (and K) of tile n and the rest of
            // tile n - 1, each as soon as its buffer is free, in the order in which that happens.  The K-major Q tile is
            // free first (S^T runs a tile ahead); behind the others its load came late for S^T.
            struct Tile {
                Item x;
                int it;
            } t1, t2{first, -1};  // tile n - 1, tile n
            for (int n = 0;; ++n) {
                t1 = t2;
                if (++t2.it >= cur.n_it && next()) t2.it = 0;
                if (!tok) break;
                t2.x = cur;
                const bool have = t2.it < cur.n_it;
                // Asked for a tile before it is needed: at the start of a long item it would be taken from a CTA that is
                // through sooner (training step at B2 H16 T2000, reproducible: 190 instead of 183 us).
                if (TAKES_OVER && t2.it + 1 == cur.n_it) {
                    mbar_arrive_expect_tx(&sh.answered, sizeof(uint4));
                    clc_try_cancel(&sh.answer, &sh.answered);
                }
                if (have && n > 0) {  // (tile 0: issued before the set-up barrier)
                    // free as soon as S^T(n - 1) is done
                    if (!(tok = mbar_wait(wc, &sh.qk_free, (n - 1) & 1, W_QKEMPTY, n))) break;
                    if (t2.it == 0) load_tile(sK, &mapK, &sh.k_full, t2.x.kv0(), t2.x);
                    load_tile(sQ, &mapQ, &sh.q_full, (t2.x.it0 + t2.it) * TILE, t2.x);
                }
                const int g = n - 2;  // the tile before tile n - 1
                const int q1 = (t1.x.it0 + t1.it) * TILE;
                if (n > 1) {
                    auto free = [&](uint64_t* bar, int phase, int id) { return tok = mbar_wait(wc, bar, phase & 1, id, n); };
                    // K-major dO: dQ(g-1) passes through the tile once dP^T(g) is done; free when the reduction has read it
                    if (!(g == 0 ? free(&sh.dok_free, 0, W_QKEMPTY) : free(&sh.dq_out, g - 1, W_DQOUT))) break;
                    load_tile(sdO, &mapdO, &sh.do_full, q1, t1.x);
                    if (t1.it > 0) {
                        // MN-major Q: free once dK(g) is done
                        if (!free(&sh.dk_done, g, W_QMFREE)) break;
                        load_tile(sQm, &mapQm, &sh.qm_full, q1, t1.x);
                    }
                    // MN-major dO doubles as staging area of two dS boxes: free once dQ(g) is done; so is that of the other
                    // two, where V of the next item lands
                    if (!free(&sh.dq_full, g, W_QMFREE)) break;
                    if (t1.it == 0) load_tile(sV, &mapV, &sh.v_full, t1.x.kv0(), t1.x);
                    load_tile(sdOm, &mapdOm, &sh.dom_full, q1, t1.x);
                    if (t1.it == 0) {
                        // dK leaves through the MN-major Q tile, dV through the MN-major K tile
                        if (!free(&sh.dk_out, items, W_ACCOUT)) break;
                        load_tile(sQm, &mapQm, &sh.qm_full, q1, t1.x);
                        if (!free(&sh.dv_out, items, W_ACCOUT)) break;
                        load_tile(sKm, &mapKm, &sh.km_full, t1.x.kv0(), t1.x);
                        ++items;
                    }
                }
                if (!have) break;
            }
        }
    } else if (warp == W_MMA) {
        // ------------------------------ MMA issuer ------------------------------
        // The whole warp runs this code with uniform control flow; only the tcgen05 instructions are predicated on
        // the elected lane (see umma_ss_tf32_lead).
        const uint32_t leader = elect_one_sync();
        auto wait = [&](uint64_t* bar, uint32_t parity, int id, int aux) -> bool {
            return __all_sync(0xffffffffu, mbar_wait(wc, bar, parity, id, aux));
        };
        constexpr uint32_t IDESC_ST = make_idesc_tf32(TILE, TILE, false, false);     // K-major x K-major, N = 128
        constexpr uint32_t IDESC_TS = make_idesc_tf32(TILE, HEAD_DIM, false, true);  // tmem A, MN-major B, N = 64
        constexpr uint32_t IDESC_DQ = make_idesc_tf32(TILE, HEAD_DIM, true, true);   // MN-major A and B, N = 64
        const Desc k_desc = kmajor_desc(smem_u32(sK), 0, BOX_BYTES), q_desc = kmajor_desc(smem_u32(sQ), 0, BOX_BYTES),
                       do_desc = kmajor_desc(smem_u32(sdO), 0, BOX_BYTES), qm_desc = mnmajor_desc(smem_u32(sQm), 0, BOX_BYTES),
                       dom_desc = mnmajor_desc(smem_u32(sdOm), 0, BOX_BYTES), km_desc = mnmajor_desc(smem_u32(sKm), 0, BOX_BYTES),
                       ds_desc = mnmajor_desc(smem_u32(sdS), 0, BOX_BYTES);
        // S^T of query tile `g` as soon as K (of item `item`, at its first tile) and Q have landed; the exponentials need
        // nothing else
        auto issue_st = [&](int g, bool first_tile, int item) -> bool {
            if (first_tile && !wait(&sh.k_full, item & 1, W_KVFULL, 0)) return false;
            if (!wait(&sh.q_full, g & 1, W_QKFULL, g)) return false;
            tc_fence_after_sync();
#pragma unroll 1
            for (uint32_t o = 0; o < 2; ++o)  // S^T = K Q^T
                umma_ss4<KMAJOR_STEP, KMAJOR_STEP>(leader, tmem + COL_S, k_desc + o * BOX_BYTES, q_desc + o * BOX_BYTES, IDESC_ST, o);
            umma_commit_lead(leader, &sh.s_full);
            umma_commit_lead(leader, &sh.qk_free);
            return true;
        };
        // dP^T = V dO^T, V from tensor memory
        auto issue_dp = [&](int g, bool first_tile, int item) -> bool {
            if (first_tile && !wait(&sh.v_ready, item & 1, W_VREADY, 0)) return false;
            if (!wait(&sh.do_full, g & 1, W_QKFULL, 1000 + g)) return false;
            tc_fence_after_sync();
#pragma unroll 1
            for (uint32_t o = 0; o < 2; ++o)
                umma_ts4<KMAJOR_STEP>(leader, tmem + COL_DP, tmem + COL_V + o * 32, do_desc + o * BOX_BYTES, IDESC_ST, o);
            umma_commit_lead(leader, &sh.dp_full);
            umma_commit_lead(leader, &sh.dok_free);
            return true;
        };
        Items s{first, 0};
        int n_it = first.n_it;
        bool ok = n_it > 0 && issue_st(0, true, 0) && issue_dp(0, true, 0);
        int it = 0, item = 0;  // query tile of the item, item
        for (int g = 0; ok; ++g) {
            const uint32_t par = g & 1;
            if (!(ok = wait(&sh.dom_full, par, W_QMFULL, g))) break;
            // dV += P^T dO
            if (!(ok = wait(&sh.pt_ready, par, W_PREADY, g))) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (uint32_t o = 0; o < 4; ++o)
                umma_ts4<MNMAJOR_STEP>(leader, tmem + COL_DV, tmem + COL_S + o * 32, dom_desc + o * 4096, IDESC_TS, (it > 0 || o > 0) ? 1u : 0u);
            umma_commit_lead(leader, &sh.dv_done);  // MN-major dO consumed: two of the dS boxes may be staged over it
            // next tile's S^T: P^T of this tile was consumed by the MMAs just issued
            const bool last = it + 1 == n_it;
            const bool more = !last || next_item(s, false);
            if (more && !(ok = issue_st(g + 1, last, item + 1))) break;
            if (!(ok = wait(&sh.qm_full, par, W_QMFULL, 1000 + g))) break;
            // dK += dS^T Q
            if (!(ok = wait(&sh.p_ready, par, W_PREADY, 1000 + g))) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (uint32_t o = 0; o < 4; ++o)
                umma_ts4<MNMAJOR_STEP>(leader, tmem + COL_DK, tmem + COL_DP + o * 32, qm_desc + o * 4096, IDESC_TS, (it > 0 || o > 0) ? 1u : 0u);
            umma_commit_lead(leader, &sh.dk_done);  // MN-major Q consumed
            // dQ = dS K once dS is staged (shortly after dS^T was stored) and the previous dQ has left tensor memory
            if (!(ok = wait(&sh.ds_ready, par, W_DSREADY, g))) break;
            if (g > 0 && !(ok = wait(&sh.dq_empty, (g - 1) & 1, W_DQEMPTY, g))) break;
            if (it == 0 && !(ok = wait(&sh.km_full, item & 1, W_KVFULL, 2))) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (uint32_t o = 0; o < 4; ++o)
                umma_ss4<MNMAJOR_STEP, MNMAJOR_STEP>(leader, tmem + COL_DQ, ds_desc + o * 4096, km_desc + o * 4096, IDESC_DQ, o);
            umma_commit_lead(leader, &sh.dq_full);  // also: the dS staging area is free again
            if (!more) break;
            // next tile's dP^T: dS^T of this tile was consumed by the MMAs just issued
            if (!(ok = issue_dp(g + 1, last, item + 1))) break;
            ++it;
            if (last) {
                it = 0;
                ++item;
                n_it = (int)uniform(s.x.n_it);
            }
        }
    } else if (warp == W_STORE) {
        // ------------------------------ store warp ------------------------------
        // Everything that leaves the CTA: the staged dQ tiles (bulk reductions) and, at the end of an item, dK and dV (bulk
        // stores).  A thread of its own, so that a reduction is issued the moment its tile is staged.
        if constexpr (SPLIT) cluster_arrive();
        if (lane == 0) {
            pdl_wait();
            tma_prefetch_desc(&mapdK);
            tma_prefetch_desc(&mapdV);
            tma_prefetch_desc(&mapdQ);
            Items s{first, 0};
            int g = 0, items = 0;
            bool tok = first.n_it > 0;
            // dQ of the next query tile, staged in the K-major dO tile: add it to global memory; once the reduction has read
            // the tile, hand it back to the load warp
            auto reduce_dq = [&](int it) -> bool {
                if (!mbar_wait(wc, &sh.dq_staged, g & 1, W_DQSTAGED, g)) return false;
                const int q = (s.x.it0 + it) * TILE;
                if (a.det_dq) {  // this KV tile's slab of partial dQ; reduce_dq_slabs adds the slabs in a fixed order
                    tma_store_tile(&mapdQ, sdO, q, s.x.h, s.x.kt * a.B + s.x.b);
                } else {
                    tma_reduce_add_tile(&mapdQ, sdO, q, s.x.h, s.x.b);
                }
                bulk_commit_group();
                bulk_wait_group_read_all();
                mbar_arrive(&sh.dq_out);
                ++g;
                return true;
            };
            // dK and dV, staged by the compute warps (see there): stored -- added, if the caller accumulates -- with bulk
            // copies, each as soon as it is staged; a thread-per-row store would be 32 lines per instruction.  Over a cluster
            // they are added up below.
            auto store_acc = [&](bool v, bool more) -> bool {
                if (!mbar_wait(wc, v ? &sh.dv_staged : &sh.dk_staged, items & 1, W_ACCSTAGED, items)) return false;
                if (SPLIT) return true;
                const CUtensorMap* map = v ? &mapdV : &mapdK;
                const uint8_t* src = !v ? sQm : more ? sKm : sQ;
                if (a.accum_dkdv)
                    tma_reduce_add_tile(map, src, s.x.kv0(), s.x.h, s.x.b);
                else
                    tma_store_tile(map, src, s.x.kv0(), s.x.h, s.x.b);
                bulk_commit_group();
                if (more) {  // the load warp waits for the tile
                    bulk_wait_group_read_all();
                    mbar_arrive(v ? &sh.dv_out : &sh.dk_out);
                }
                return true;
            };
            while (tok) {
                for (int it = 0; tok && it + 1 < s.x.n_it; ++it) tok = reduce_dq(it);  // the last tile's dQ follows dK and dV
                if (!tok) break;
                Items nx = s;
                const bool more = next_item(nx, true);
                tok = store_acc(!more, more) && store_acc(more, more) && reduce_dq(s.x.n_it - 1);
                ++items;
                if (!more) break;
                s = nx;
            }
            // the copies have read their shared-memory sources; they complete on their own
            bulk_wait_group_read_all();
        }
    } else if (warp == W_ROWS) {
        // ------------------------------ LSE and D of the query rows ------------------------------
        // A lane takes rows lane, lane + 32, .. of each query tile; they are fetched a tile ahead and written, negated and
        // scaled so that both enter the arithmetic as FMA addends, once the compute warps are through with the previous
        // tile's (they are when dS^T is stored).  A warp of its own: eight compute warps that did this beside their work,
        // and sixteen that waited for it, were ~400 cycles per tile longer at it.
        Items s{first, 0};
        if (first.n_it > 0) {
            float l[TILE / 32], d[TILE / 32];
            auto fetch = [&](int it) {
                const float* lse_bh = a.LSE + (int64_t)s.x.b * a.lse_sB + (int64_t)s.x.h * a.lse_sH;
                const float* d_bh = a.D + (int64_t)s.x.b * a.d_sB + (int64_t)s.x.h * a.d_sH;
#pragma unroll
                for (int u = 0; u < TILE / 32; ++u) {
                    const int q = (s.x.it0 + it) * TILE + 32 * u + lane;
                    l[u] = q < a.Tq ? __ldg(lse_bh + q) : -INFINITY;
                    d[u] = q < a.Tq ? __ldg(d_bh + q) : 0.f;
                }
            };
            pdl_wait();  // D
            fetch(0);
            int it = 0;
            for (int g = 0;; ++g) {
                if (g > 0 && !__all_sync(0xffffffffu, mbar_wait(wc, &sh.p_ready, (g - 1) & 1, W_ROWSFREE, g))) break;
#pragma unroll
                for (int u = 0; u < TILE / 32; ++u) {
                    sh.lse[32 * u + lane] = (l[u] == -INFINITY) ? -INFINITY : -l[u] * LOG2E;
                    sh.dsum[32 * u + lane] = -d[u] * a.scale;
                }
                mbar_arrive_warp(&sh.s_full, lane);
                if (++it == s.x.n_it) {
                    if (!next_item(s, false)) break;
                    it = 0;
                }
                fetch(it);
            }
        }
    } else {
        // ------------------------------ compute ------------------------------
        const int quarter = warp & 3;
        const int part = warp >> 2;             // which 32 of the 128 query columns this thread owns
        const int row = quarter * 32 + lane;    // key row inside the tile = tensor-memory lane
        const int c0 = part * 32;
        const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
        bool ok = true;
        uint32_t rs[32], rp[32];

        // dQ of query tile j out of tensor memory into the K-major dO tile (this thread's query row `row`, 16 of the 64
        // columns), in the layout of a 128-byte-swizzled TMA box: 16-byte chunk c of row r at
        // position c ^ (r & 7).  Done in the middle of the NEXT tile, in two parts: read while dP^T of that tile is still
        // being computed, stored when it is done: its operand, the K-major dO tile, is then dead until the tile after it
        // is prefetched, long enough for the bulk reduction, which keeps its source for ~1 600 cycles.
        auto read_dq = [&](int j, uint32_t* v) -> bool {
            if (!__all_sync(0xffffffffu, mbar_wait(wc, &sh.dq_full, j & 1, W_DQFULL, j))) return false;
            tc_fence_after_sync();
            tmem_ld16(trow + COL_DQ + 16 * part, v);
            tmem_wait_ld();
            tc_fence_before_sync();
            mbar_arrive_warp(&sh.dq_empty, lane);  // dQ is in registers: the next dQ = dS K may overwrite tensor memory
            return true;
        };
        auto stage_dq = [&](const uint32_t* v) {
            uint8_t* srow = sdO + (part >> 1) * BOX_BYTES + row * 128;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(srow + (((4 * (part & 1) + c) ^ (row & 7)) << 4)) =
                    make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
            fence_proxy_async_smem();
            mbar_arrive_warp(&sh.dq_staged, lane);
        };

        // V of an item's KV tile into tensor memory (A operand of dP^T = V dO^T), by column groups 2 and 3, which are there
        // first: this thread's key row, 32 of the 64 columns, read from the 128-byte-swizzled landing buffer (16-byte chunk
        // c of row r at position c ^ (r & 7))
        auto copy_v = [&](int item, uint32_t (&v)[32]) -> bool {
            if (!__all_sync(0xffffffffu, mbar_wait(wc, &sh.v_full, item & 1, W_KVFULL, 3))) return false;
            const uint8_t* vrow = sV + (part & 1) * BOX_BYTES + row * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint4 x = *reinterpret_cast<const uint4*>(vrow + ((c ^ (row & 7)) << 4));
                v[4 * c] = x.x; v[4 * c + 1] = x.y; v[4 * c + 2] = x.z; v[4 * c + 3] = x.w;
            }
            tmem_st32(trow + COL_V + 32 * (part & 1), v);
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive_warp(&sh.v_ready, lane);
            return true;
        };

        int g = 0, item = 0;  // query tiles, items done with
        Items s{first, 0};
        for (;;) {
            const int kv0 = s.x.kv0(), bh = s.x.bh, it0 = s.x.it0, n_it = s.x.n_it;
            const int kvrow = kv0 + row;
            const bool kv_ok = kvrow < a.Tk;
            if (SPLIT && n_it == 0) pdl_wait();  // the rows written at the end; with query tiles the barriers order everything
            for (int it = 0; it < n_it; ++it, ++g) {
                const int q0 = (it0 + it) * TILE;
                // V lands before the first S^T of the CTA is complete; that of later items while their first P^T is computed
                if (g == 0 && part >= 2 && !(ok = copy_v(0, rp))) break;
                ok = __all_sync(0xffffffffu, mbar_wait(wc, &sh.s_full, g & 1, W_SFULL, g));
                if (!ok) break;
                tc_fence_after_sync();

                tmem_ld32(trow + COL_S + c0, rs);

                // first query column (local to the tile) this key row is visible to
                int cmin = 0;
                if (a.causal) {
                    const long long c = (long long)a.k_pos0 + kvrow - a.q_pos0 - q0;
                    cmin = (int)max(0ll, min((long long)TILE, c));
                }
                if (!kv_ok) cmin = TILE;

                // dropout keep bits of this thread's 32 (query, key) pairs
                uint32_t keep = 0xffffffffu;
                if constexpr (DROP == 2) {
                    // One Philox call covers the eight keys kpos & ~7 .. of one query row, i.e. the key rows of eight
                    // adjacent lanes (k_pos0 and kv0 are multiples of 8, so row & 7 == lane & 7).  Lane j of such a
                    // group evaluates the query columns 8m + j (m = 0..3) and keeps 8 bits per call; the group then
                    // swaps them with shuffles, so every lane does 4 calls for its 32 columns instead of 32.
                    const int j8 = lane & 7;
                    const uint32_t kgrp = (uint32_t)(a.k_pos0 + kvrow) >> 3;
                    uint32_t mine = 0u;  // bit 8m + u: query column c0 + 8m + j8, key row (row & ~7) + u
#pragma unroll
                    for (int mI = 0; mI < 4; ++mI) {
                        const hk_philox4_t w = hk_philox_row8_keys(a.philox_keys, a.philox_offset, a.bh_pos0 + (uint32_t)bh,
                                                              (uint32_t)(a.q_pos0 + q0 + c0 + 8 * mI + j8), kgrp);
                        mine |= hk_philox_keep8(w, a.drop_thr) << (8 * mI);
                    }
                    keep = 0u;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t other = __shfl_sync(0xffffffffu, mine, (lane & ~7) | j);  // lane j's columns 8m + j
                        keep |= ((other >> j8) & 0x01010101u) << j;                              // its bit for MY key row
                    }
                } else if constexpr (DROP == 1) {
                    keep = 0u;
                    if (kv_ok) {
#pragma unroll 4
                        for (int i = 0; i < 32; ++i) {
                            const int q = q0 + c0 + i;
                            if (q < a.Tq && __ldg(a.mask + ((size_t)bh * a.Tq + q) * (size_t)a.Tk + kvrow) != 0.f)
                                keep |= 1u << i;
                        }
                    }
                }
                // fold the causal / tail mask into the keep bits: column cc is visible iff cc >= cmin
                uint32_t vis = 0xffffffffu;
                {
                    const int lo = cmin - c0;  // first visible local index, may be <= 0 or >= 32
                    if (lo > 0) vis = (lo >= 32) ? 0u : (0xffffffffu << lo);
                    keep &= vis;
                }
                // pairs whose p is zero: hidden ones, and dropped ones unless the dropout is the inverted kind
                const uint32_t live = DROP != 0 && a.drop_scaled ? vis : keep;
                tmem_wait_ld();

                // p = exp2(s*scale*log2e - LSE*log2e) needs S^T only: dP^T is still being computed.  Two scores per
                // packed FMA (fma.rn.f32x2 gives the same bits as two scalar FMAs).
                {
                    const float4* lse4 = reinterpret_cast<const float4*>(sh.lse + c0);
                    const float2 c2 = make_float2(a.scale_log2e, a.scale_log2e);
#pragma unroll
                    for (int f = 0; f < 8; ++f) {
                        const float4 L = lse4[f];
                        const float2 x01 = __ffma2_rn(make_float2(__uint_as_float(rs[4 * f]), __uint_as_float(rs[4 * f + 1])), c2,
                                                      make_float2(L.x, L.y));
                        const float2 x23 = __ffma2_rn(make_float2(__uint_as_float(rs[4 * f + 2]), __uint_as_float(rs[4 * f + 3])), c2,
                                                      make_float2(L.z, L.w));
                        rs[4 * f] = __float_as_uint(ex2_approx(x01.x));
                        rs[4 * f + 1] = __float_as_uint(ex2_approx(x01.y));
                        rs[4 * f + 2] = __float_as_uint(ex2_approx(x23.x));
                        rs[4 * f + 3] = __float_as_uint(ex2_approx(x23.y));
                    }
                    if (live != 0xffffffffu) {  // tiles on the diagonal, the ragged end, dropout
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (!((live >> i) & 1u)) rs[i] = 0u;
                    }
                }
                // P^T goes to tensor memory at once (rounded; a pair dropped by inverted dropout counts as zero in dV but
                // keeps its p for dS below): dV += P^T dO and, behind it, the next tile's S^T run while dS is computed,
                // and the store has drained by the time its first reader starts.  rp is free until dP^T is loaded.
                {
                    const bool dropped_some = DROP != 0 && a.drop_scaled && keep != 0xffffffffu;
#pragma unroll
                    for (int i = 0; i < 32; ++i) rp[i] = tf32_round_bits_mma(rs[i]);
                    if (dropped_some) {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (!((keep >> i) & 1u)) rp[i] = 0u;
                    }
                    tmem_st32(trow + COL_S + c0, rp);
                    tmem_wait_st();
                    tc_fence_before_sync();
                    mbar_arrive_warp(&sh.pt_ready, lane);
                }
                if (g > 0) {  // rp is free until dP^T is loaded
                    if (it == 0 && part >= 2 && !(ok = copy_v(item, rp))) break;
                    if (!(ok = read_dq(g - 1, rp))) break;
                }
                ok = __all_sync(0xffffffffu, mbar_wait(wc, &sh.dp_full, g & 1, W_SFULL, 1000 + g));
                if (!ok) break;
                tc_fence_after_sync();
                if (g > 0) stage_dq(rp);
                tmem_ld32(trow + COL_DP + c0, rp);
                tmem_wait_ld();

                // dS = p * (dP*scale - D*scale), two elements per packed instruction
                {
                    const float4* ds4 = reinterpret_cast<const float4*>(sh.dsum + c0);
                    const bool dropped_some = DROP != 0 && a.drop_scaled && keep != 0xffffffffu;
                    if (dropped_some) {
                        // inverted dropout: a dropped pair keeps the -D term of dS but contributes neither dP (zeroed
                        // here) nor to dV (its P^T entry was stored as zero above)
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (!((keep >> i) & 1u)) rp[i] = 0u;
                    }
                    const float2 dps2 = make_float2(a.dp_scale, a.dp_scale);
#pragma unroll
                    for (int f = 0; f < 8; ++f) {
                        const float4 Dv = ds4[f];  // -D * scale
#pragma unroll
                        for (int h2 = 0; h2 < 2; ++h2) {
                            const int i = 4 * f + 2 * h2;
                            const float2 nd = h2 ? make_float2(Dv.z, Dv.w) : make_float2(Dv.x, Dv.y);
                            const float2 t = __ffma2_rn(make_float2(__uint_as_float(rp[i]), __uint_as_float(rp[i + 1])), dps2, nd);
                            const float2 ds = __fmul2_rn(make_float2(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), t);
                            rp[i] = tf32_round_bits_mma(__float_as_uint(ds.x));
                            rp[i + 1] = tf32_round_bits_mma(__float_as_uint(ds.y));
                        }
                    }
                }
                tmem_st32(trow + COL_DP + c0, rp);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive_warp(&sh.p_ready, lane);

                // dS into shared memory, the MN-major A operand of dQ = dS K: box `part` holds query columns
                // 32*part..32*part+31, one 128-byte row per key row, 32-byte chunks XOR-swizzled with (row & 3).  Boxes 0, 1
                // have a buffer of their own, free once dQ of the previous tile is done -- and, at the first tile of an item, V
                // has left it --: dP^T of this tile, complete here, was issued behind either.  Boxes 2, 3 go over the MN-major dO
                // tile as soon as dV of this tile is done.
                if (part >= 2) {
                    ok = __all_sync(0xffffffffu, mbar_wait(wc, &sh.dv_done, g & 1, W_DVDONE, g));
                    if (!ok) break;
                }
                {
                    // Rows r and r + 4 share a 32-byte chunk position, so two of the eight lanes of a quarter-warp meet in a
                    // 16-byte bank group.  Storing the two halves in opposite order avoids that, but the 32 selects that it
                    // takes cost what it gains (B8 H12 T1024 87.6 us with them, 88.0 without; ten launches after a pause, 1 965
                    // MHz), and more where the warps have keep bits to draw too (with dropout 101.5 -> 99.9, B32 H25 T1024 736 -> 723).
                    uint8_t* drow = sdS + part * BOX_BYTES + row * 128;
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        *reinterpret_cast<uint4*>(drow + (((u >> 1) ^ (row & 3)) << 5) + ((u & 1) << 4)) =
                            make_uint4(rp[4 * u], rp[4 * u + 1], rp[4 * u + 2], rp[4 * u + 3]);
                }
                fence_proxy_async_smem();
                mbar_arrive_warp(&sh.ds_ready, lane);
            }

            if (!ok) break;
            Items nx = s;
            const bool more = next_item(nx, false);
            // The accumulators, as the boxes of a 128-byte-swizzled TMA tile (16-byte chunk c of row r at position c ^ (r & 7)):
            // column groups 2, 3 put dK into the MN-major Q tile, dead with the last dK; groups 0, 1 put dV (times 1/(1-p) for
            // inverted dropout) into the MN-major K tile, dead with the last dQ, or, if no item follows, at once into the
            // K-major Q tile.  They are in registers when this warp hands over its next P^T, which the first dV of the next item
            // waits for.
            if (n_it > 0)
                ok = __all_sync(0xffffffffu, mbar_wait(wc, (part >= 2) ? &sh.dk_done : more ? &sh.dq_full : &sh.dv_done, (g - 1) & 1, W_BDONE, g));
            if (!ok) break;
            if (n_it > 0) {
                tc_fence_after_sync();
                tmem_ld32(trow + ((part < 2) ? COL_DV + part * 32 : COL_DK + (part - 2) * 32), rs);
                tmem_wait_ld();
                tc_fence_before_sync();
                const float f = (part < 2) ? a.dv_scale : 1.f;
                uint8_t* srow = ((part >= 2) ? sQm : more ? sKm : sQ) + (part & 1) * BOX_BYTES + row * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<float4*>(srow + ((c ^ (row & 7)) << 4)) =
                        make_float4(__uint_as_float(rs[4 * c]) * f, __uint_as_float(rs[4 * c + 1]) * f,
                                    __uint_as_float(rs[4 * c + 2]) * f, __uint_as_float(rs[4 * c + 3]) * f);
                fence_proxy_async_smem();
                mbar_arrive_warp((part < 2) ? &sh.dv_staged : &sh.dk_staged, lane);
            }
            if (!more) break;
            s = nx;
            ++item;
        }  // items

        if constexpr (SPLIT) {
            __syncwarp();
            cluster_arrive();
        }

        // dQ of the last query tile takes the same way out as the others: staged in the K-major dO tile (dead: its
        // last reader was dP^T of this tile) once the reduction of the previous tile has read that buffer, then
        // added to global memory by the store warp.  (From registers with red.global.add it took ~2 500 cycles per
        // CTA and held up the bulk stores of dV and dK behind it.)
        if (ok && g > 0) {
            if (g > 1) ok = __all_sync(0xffffffffu, mbar_wait(wc, &sh.dq_out, (g - 2) & 1, W_DQOUT, g - 2));
            if (ok) ok = read_dq(g - 1, rs);
            if (ok) stage_dq(rs);
        }

    }

    if constexpr (SPLIT) {
        // dV and dK of the KV tile: the sum over the splits, always in the same order, from what each left in its shared
        // memory; each CTA adds up an equal slice of the rows, 32 threads per row (16 for dV, 16 for dK).  The compute warps
        // have arrived once their dV and dK were staged, the store warp at its start: no CTA waits for another's last dQ, and
        // the sums are stored while the others leave (24.7 -> 22.7 us for B=4 H=6, 777 queries, 333 keys).
        __syncwarp();
        if (warp >= W_LOAD && warp != W_STORE) cluster_arrive();
        cluster_wait();
        if (warp < W_LOAD) {
            // (rows of this thread) x (splits) = 8: all loads first, their latency is that of the other SM's memory
            const int ch = lane & 15;
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int row = split * (TILE / ns) + warp + NUM_COMPUTE / 32 * (u / ns);
                const uint8_t* src = (lane < 16 ? sQ : sQm) + (ch >> 3) * BOX_BYTES + row * 128 + (((ch & 7) ^ (row & 7)) << 4);
                v[u] = u % ns < first.live ? ld_cluster_f4(mapa(src, u % ns)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w;
                if (u == 7) {  // every v is in: the others may leave
                    __syncwarp();
                    cluster_arrive();
                }
                if ((u + 1) % ns != 0) continue;
                const int64_t kvrow = first.kv0() + split * (TILE / ns) + warp + NUM_COMPUTE / 32 * (u / ns);
                if (kvrow < a.Tk) {
                    float* dst = lane < 16 ? a.dV + (int64_t)first.b * a.dv_sB + (int64_t)first.h * a.dv_sH + kvrow * a.dv_sM
                                           : a.dK + (int64_t)first.b * a.dk_sB + (int64_t)first.h * a.dk_sH + kvrow * a.dk_sM;
                    float4* out = reinterpret_cast<float4*>(dst) + ch;
                    if (a.accum_dkdv) {
                        const float4 old = *out;
                        acc.x += old.x; acc.y += old.y; acc.z += old.z; acc.w += old.w;
                    }
                    *out = acc;
                }
                acc = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        __syncwarp();
        if (warp >= W_LOAD) cluster_arrive();
        cluster_wait();  // the others have read this CTA's shared memory
    }

    // ------------------------------ teardown ------------------------------
    tc_fence_before_sync();
    __syncthreads();
    // A CTA that gave up does not leave while copies into its shared memory may be in flight (otherwise every copy was waited
    // for by what it was for).
    if (sh.abort.id)
        for (const unsigned long long t0 = globaltimer_ns(); globaltimer_ns() - t0 < 100000ull;) {}
    if (warp == W_MMA) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem, TMEM_COLS);
        if (lane == 0) report_abort(sh.abort, a.status);
    }
}

// Per-device launch data: the large shared-memory opt-in and how many clusters of each size run at once.
namespace {
struct BwdDevice {
    std::once_flag once;
    cudaError_t rc = cudaSuccess;
    int slots[4] = {148, 74, 33, 15};  // resident clusters of 1, 2, 4, 8 CTAs; the device is asked
};
typedef void (*BwdKernel)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap,
                          CUtensorMap, CUtensorMap, BwdArgs);
const BwdKernel bwd_kernels[9] = {attn_bwd_kernel<0, ONE_ITEM>,   attn_bwd_kernel<1, ONE_ITEM>,   attn_bwd_kernel<2, ONE_ITEM>,
                                  attn_bwd_kernel<0, TAKE_OVER>,  attn_bwd_kernel<1, TAKE_OVER>,  attn_bwd_kernel<2, TAKE_OVER>,
                                  attn_bwd_kernel<0, SPLIT_ITEM>, attn_bwd_kernel<1, SPLIT_ITEM>, attn_bwd_kernel<2, SPLIT_ITEM>};

// of the current device; set up by the first call on it
int bwd_device(BwdDevice** out) {
    static BwdDevice devices[HK_MAX_DEVICES];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return HK_ERR_CUDA;
    if (dev < 0 || dev >= HK_MAX_DEVICES) return HK_ERR_UNSUPPORTED;
    BwdDevice& d = devices[dev];
    std::call_once(d.once, [&d] {
        d.slots[0] = sm_count();
        for (BwdKernel k : bwd_kernels)
            if (d.rc == cudaSuccess)
                d.rc = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd::SMEM_BYTES);
        for (int i = 1; i < 4 && d.rc == cudaSuccess; ++i) {
            LaunchConfig lc(8u << i, bwd::NUM_THREADS, bwd::SMEM_BYTES, nullptr, 1 << i, false);
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, bwd_kernels[6], &lc.cfg) == cudaSuccess && n > 0) d.slots[i] = n;
        }
    });
    if (d.rc != cudaSuccess) return HK_ERR_CUDA;
    *out = &d;
    return HK_OK;
}

}  // namespace

int attn_bwd_slots(const int** slots) {
    BwdDevice* d = nullptr;
    const int rc = bwd_device(&d);
    if (rc == HK_OK) *slots = d->slots;
    return rc;
}

BwdPlan plan_attn_bwd(int BH, int Tq, int Tk, int causal, int q_pos0, int k_pos0, const int slots[4]) {
    // KV tiles that a query tile sees.  (The grid has no others: the store warp could not read past a run of items without
    // query tiles, since it hands over the last dQ of an item beside the first tile of the next.)
    const int n_kvtiles = (Tk + TILE - 1) / TILE;
    BwdPlan plan{1, n_kvtiles, ONE_ITEM};
    if (causal) {
        const long long last_q = (long long)(Tq + TILE - 1) / TILE * TILE - 1 + q_pos0 - k_pos0;  // in key positions
        plan.live = (int)std::max(0ll, std::min((long long)n_kvtiles, last_q < 0 ? 0 : last_q / TILE + 1));
    }
    // Splits by an estimate of the makespan: whole waves of CTAs that cost ~7 us and ~2.5 us per query tile, ~2.5 - 3 us more
    // where they add dV and dK up over a cluster.  They pay where few KV tiles have many query tiles (cross-attention of a
    // long sequence to a short one).  Over 110 such shapes the number is 0.2 % from the best one on average; with half a wave
    // for what the last one leaves over it was 1.3 % (B2 H2, 9 851 queries, 2 554 keys took two CTAs per tile, 80 clusters in
    // 74 slots, 208 us; four take 173).  Of 500 further shapes 36 are cut differently, 1.10 times as fast on average, one of
    // them 2 % slower.  The sum is taken in another order and the choice depends on batch x heads, so sequences of training
    // length do without: a batch cut into calls gives the bits of the single call.
    if (Tq >= 2 * (long long)Tk) {
        const double n_q = (Tq + TILE - 1) / TILE;
        double best_cost = 0;
        for (int i = 0; i < 4; ++i) {
            const double one = 7.0 + (i ? 2.2 + 0.3 * i : 0.0) + 2.5 * std::ceil(n_q / (1 << i));
            const double cost = one * std::ceil((double)n_kvtiles * BH / slots[i]);
            if (i == 0 || cost < 0.95 * best_cost) {
                best_cost = cost;
                plan.n_splits = 1 << i;
            }
        }
    }
    plan.job = plan.n_splits > 1 ? SPLIT_ITEM : (long long)plan.live * BH > slots[0] ? TAKE_OVER : ONE_ITEM;
    return plan;
}

// As in the forward, several runs cost balance at the end of the grid, the more the more KV tiles a slice has.  us, one run ->
// several, at 2.2 times the slices of a run: T512 55.8 -> 54.9, T768 69.0 -> 66.7, T1024 78.2 -> 78.0, without a causal mask 129.3 ->
// 130.4, with Philox 89.1 -> 90.2; T2048 123.6 -> 124.7, T3000 170.8 -> 173.9, T4096 213.6 -> 216.5; at 2.7 times T1024 94.6 -> 92.9,
// T2048 146.7 -> 143.9, T4096 255.3 -> 254.8.  With a dense mask T1024 377 -> 386 and 469 -> 463; T2048 at 2.6, 3.3 and 4.1 times
// 808 -> 819, 1 010 -> 1 012, 1 261 -> 1 239; T4096 at 2.6, 3.5 and 5 times 1 547 -> 1 562, 2 043 -> 2 061, 2 924 -> 2 895.  With
// Philox T4096 at 3.5 times 404.9 -> 401.6, T5067 at 3.2 and 5.4 times 463 -> 474, 762 -> 751, T8192 at 3.5 and 5.2 times 754 -> 768,
// 1 118 -> 1 105.  Without dropout T8192 at 3.5 times 631 -> 630, but T16384 at 2.6, 3.5 and 7 times 912 -> 921, 1 209 -> 1 212,
// 2 467 -> 2 382 and T24000 at 3.2 and 5.1 times 1 596 -> 1 619, 2 574 -> 2 544: runs of one or two slices.
int bwd_run(const BwdPlan& plan, int BH, int Tq, int Tk, int dropout_mode) {
    const int group = slices_in_l2(BH, 256.0 * (3.0 * Tq + 4.0 * Tk));  // Q, dO, dQ; K, V, dK, dV
    if (plan.job != TAKE_OVER || plan.live == 1) return BH;
    const bool many = dropout_mode == 1 ? plan.live >= 16 : dropout_mode == 2 ? plan.live > 32 : group <= 2;
    const double least = plan.live < 8 ? 2.0 : many ? 4.0 : 2.5;  // in runs
    return BH < least * group ? BH : group;
}

int launch_attn_bwd(const BwdMaps& m, BwdArgs a, bool after_prepass, cudaStream_t stream) {
    BwdDevice* d = nullptr;
    const int device_rc = bwd_device(&d);
    if (device_rc != HK_OK) return device_rc;
    const BwdPlan plan = plan_attn_bwd(a.BH, a.Tq, a.Tk, a.causal, a.q_pos0, a.k_pos0, d->slots);
    const int live = plan.live;
    a.n_splits = plan.n_splits;
    a.live = live;
    a.group = bwd_run(plan, a.BH, a.Tq, a.Tk, a.dropout_mode);
    const long long nblocks = (long long)live * a.BH * a.n_splits;
    if (nblocks > 0x7fffffffLL) return HK_ERR_BAD_SHAPE;
    if (nblocks > 0) {
        timing_mark(TIMED_BWD, true, stream);
        LaunchConfig lc((unsigned)nblocks, bwd::NUM_THREADS, bwd::SMEM_BYTES, stream, a.n_splits, after_prepass);
        const cudaError_t rc = cudaLaunchKernelEx(&lc.cfg, bwd_kernels[a.dropout_mode + 3 * plan.job], m.q, m.k, m.v, m.dO, m.q_mn, m.k_mn,
                                                  m.dO_mn, m.dQ, m.dK, m.dV, a);
        timing_mark(TIMED_BWD, false, stream);
        count_launch();
        if (rc != cudaSuccess) return check_launch();
    }
    // the rows of the other KV tiles are zero
    const int rows = a.Tk - live * TILE;
    if (rows > 0 && !a.accum_dkdv) {
        int rc = launch_zero_rows(a.dK + (int64_t)live * TILE * a.dk_sM, a.dk_sB, a.dk_sM, a.dk_sH, a.BH / a.H, a.H, rows, stream);
        if (rc == HK_OK) rc = launch_zero_rows(a.dV + (int64_t)live * TILE * a.dv_sM, a.dv_sB, a.dv_sM, a.dv_sH, a.BH / a.H, a.H, rows, stream);
        return rc;
    }
    return HK_OK;
}

}  // namespace hk

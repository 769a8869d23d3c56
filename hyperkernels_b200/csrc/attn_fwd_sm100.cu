// attn_fwd_sm100.cu -- fused attention forward for sm_100a.
//
// Computes what fused_attn_forward_kernel_tc_sm89<64,64,64,1> computes
// (kernels/attention/fused_attn_forward_kernel_tc_sm89.cu:72-426 of the
// reference): S = Q K^T on TF32 tensor cores, v = S*scale, causal mask,
// running max m and alpha = exp(m_old - m_new), e = exp(v - m_new), dropout
// mask multiplied into e BEFORE the row sum, l = alpha*l + sum(e),
// O = alpha*O + P V with P rounded to TF32, finally O /= l (0 if l == 0) and
// LSE = m + log l (-inf if l == 0).
//
// Blackwell structure: a CTA runs two streams of "products", 128 query rows against 128 keys each, which take turns on
// the tensor pipe, so that the softmax of one runs while the MMAs of the other execute.  The streams are
//   rows mode     two adjacent blocks of 128 query rows against the same key tiles (256 rows per CTA),
//   row mode      one block of 128 rows, the second stream idle, or
//   keys mode     the even and the odd key tiles of one block of 128 rows, merged at the end.
// The last two have twice the CTAs, each shorter, and twice the loads: for problems whose row blocks are few.
//   warp 0        TMA producer: Q once, then K and V tiles through one ring of five slots in the order the products
//                 use them up, K0 K1 V0 K2 V1 ... (128-byte-swizzled boxes of 128 rows x 32 floats, mbarrier tx; V
//                 with the 32-byte-chunk swizzle an MN-major TF32 operand needs).  Two stages of K and V each,
//                 the previous layout, waited for the copy of the tile they had just released (9 % at 8 192 keys).
//   warp 1        MMA issuer (the whole warp runs the issuing code, one elected lane issues).
//                 S = Q K^T is 8 tcgen05.mma (M128 N128 K8, operands from shared memory), O_t += P V is 16
//                 (M128 N64 K8, A = P from tensor memory, B = V MN-major from shared memory).  Product q keeps
//                 its S, then its P, in score buffer q mod 3, and the issue order is S(0) S(1) S(2) | P V(0) S(3) |
//                 P V(1) S(4) | ...: the scores of a stream's NEXT step are computed while its softmax works on the
//                 current one (the tensor pipe executes in issue order, so S(q+3) cannot overtake the P V(q) that
//                 reads the same buffer).
//   warp 2        where further blocks of rows follow: O of a finished one to global memory, by TMA
//   warps 4-7     softmax of stream 0, warps 8-11 softmax of stream 1: thread r owns query row r (tensor-memory lane
//                 r), holds the 128 scores of a step in registers (one tensor-memory read per score) and writes P back
//                 over S.  (Two threads per row, sixteen warps: the exchange of the row maximum alone takes 300 cycles
//                 of a step.)  The running output is rescaled only when the running maximum grew by more than 2^8 (the
//                 final O/l and LSE use the same maximum, so the result is the same function).
// Tensor memory: three score buffers (128 columns each), O_0, O_1 (64 columns each): 512 of 512 columns.
// Warps 0-3 give most of their registers to the softmax warps (setmaxnreg 72 / 216).
//
// Where there are more blocks of rows than SMs and they are short, a CTA that is through with one takes over another of a CTA
// not started yet (cluster launch control, FwdJob::TAKE_OVER): its loads, scores and first softmax run under the last products
// of the block before it.
//
// Key splits: a cluster of NS CTAs shares one block of query rows; split s takes a contiguous run of its key tiles, and at
// the end every CTA combines a slice of the rows from the partial (O, m, l) the others left in their shared memory (keys
// mode merges its two streams with the same code).  The host picks mode and splits (plan_attn_fwd).
// CTA pairs (cta_group::2, half of every K and V tile per CTA) were built and measured: the MMAs and copies alone run at
// 2 360 instead of 3 100 cycles per step, the whole kernel 4 % faster at H32 T8192, but every CTA spends ~4 000 cycles
// more on set-up and hand-over between the two, 57 against 45 us at B8 H12 T1024.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "attn_kernels.cuh"
#include "philox.h"

namespace hk {

namespace fwd {

constexpr int NUM_SOFTMAX = 256;
constexpr int NUM_THREADS = 128 + NUM_SOFTMAX;
constexpr int TMEM_COLS = 512;
constexpr int COL_O0 = 256;  // O_t at COL_O0 + 64 t
// score buffer b of three: columns 0, 128, 384
__device__ __forceinline__ uint32_t score_col(int b) { return b == 2 ? 384u : (uint32_t)b * 128u; }
constexpr int SLOTS = 5;                    // K / V ring
constexpr float RESCALE_THRESHOLD = 8.f;    // log2 units

// What a CTA works on: one or two blocks of 128 query rows and the key tiles it takes them through.
struct Item {
    int b, h, bh, q0;  // q0: first query row
    int n0, n1;        // steps of the streams; n0 < 0: there is no item
    int nk, jb;        // key tiles loaded, the first of them (with splits: of this CTA's run)
    int all0, all1;    // key tiles that the rows of the streams see, over all splits
    __device__ __forceinline__ int steps(int t) const { return t == 0 ? n0 : n1; }
};
constexpr int ITEMS = 8;  // items that may be known beyond the one that the slowest warp is at

struct __align__(16) Shared {
    float m[2][TILE], l[2][TILE];  // [stream]: row maxima and sums for the combination
    uint64_t q_full[2], q_empty[2], kv_full[SLOTS], kv_empty[SLOTS], s_full[3], p_full[3], o_full[3];
    uint64_t o_staged[2];          // O of stream t is in its slot of the ring
    uint64_t o_taken[2];           // the store warp knows: the stream may stage the next one
    uint64_t item_full[ITEMS], item_empty[ITEMS], answered;
    uint4 answer;                  // to a request for another item
    Item item[ITEMS];              // the items taken over, decoded
    uint32_t tmem_base;
    Abort abort;
};

constexpr int OFF_Q = 0;                          // two tiles
constexpr int OFF_KV = 2 * TILE_BYTES;            // ring
constexpr int OFF_SH = OFF_KV + SLOTS * TILE_BYTES;
constexpr int SMEM_BYTES = OFF_SH + sizeof(Shared);
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KiB a CTA may opt in to");

enum WaitId { W_QFULL = 101, W_KFULL, W_KVEMPTY, W_VFULL, W_SFULL, W_PFULL, W_OFULL, W_QEMPTY, W_ITEM, W_OSLOT, W_OSTAGED };

// 384 threads x 168 registers at launch = 128 x 72 + 256 x 216 after the hand-over (setmaxnreg.inc can only take what
// the launch-time pool of the CTA holds)
static_assert(128 * 72 + NUM_SOFTMAX * 216 <= NUM_THREADS * 168, "register hand-over exceeds the CTA's pool");
__device__ __forceinline__ void reg_release() { asm volatile("setmaxnreg.dec.sync.aligned.u32 72;\n"); }
__device__ __forceinline__ void reg_acquire() { asm volatile("setmaxnreg.inc.sync.aligned.u32 216;\n"); }

// Ring sequence of an item of n key tiles: K0 K1 V0 K2 V1 .. K(n-1) V(n-2) - V(n-1): K(0) is entry 0, K(j) entry 2 j - 1, V(j)
// entry 2 j + 2, so the entry before the last V is skipped.  Where other items follow (FOLLOWED) it is not, the last V is
// entry 2 n - 1, and then comes one entry per stream that has rows: a slot through which its O leaves.
template <bool FOLLOWED>
__device__ __forceinline__ int ring_v(int j, int n) {
    return FOLLOWED ? min(2 * j + 2, 2 * n - 1) : 2 * j + 2;
}
struct RingPos {
    uint32_t slot, phase;
    __device__ __forceinline__ RingPos(uint32_t entry) : slot(entry % SLOTS), phase((entry / SLOTS) & 1u) {}
    __device__ __forceinline__ void advance(uint32_t by) {
        slot += by;
        if (slot >= SLOTS) {
            slot -= SLOTS;
            phase ^= 1u;
        }
    }
};

// number of key tiles the query rows q0 .. q0 + TILE - 1 attend to
__host__ __device__ inline int kv_tiles_for(int q0, int Tq, int Tk, int causal, int q_pos0, int k_pos0) {
    if (q0 >= Tq) return 0;
    long long kv_end = Tk;
    if (causal) {
        const int last_row = (q0 + TILE < Tq ? q0 + TILE : Tq) - 1;
        const long long lim = (long long)q_pos0 + last_row - k_pos0 + 1;
        kv_end = lim < 0 ? 0 : lim < kv_end ? lim : kv_end;
    }
    return (int)((kv_end + TILE - 1) / TILE);
}

// RUNS: the items come in runs of slices (take_in_groups)
template <bool RUNS>
__device__ __forceinline__ Item make_item(const FwdArgs& a, int work, int split, int ns) {
    Item x;
    // heavy (late) query blocks first: under the causal mask they have the most key tiles
    int qb;
    take_in_groups(work, a.BH, a.n_qblocks, RUNS ? a.group : a.BH, x.bh, qb);
    qb = a.n_qblocks - 1 - qb;
    x.b = x.bh / a.H;
    x.h = x.bh - x.b * a.H;
    // rows mode: stream t = query rows q0 + 128 t ..; keys mode: both streams = rows q0 .., stream t = key tiles 2 j + t.
    const bool keys = a.mode == FWD_KEYS;
    x.q0 = qb * (a.mode == FWD_ROWS ? 2 * TILE : TILE);
    x.all0 = kv_tiles_for(x.q0, a.Tq, a.Tk, a.causal, a.q_pos0, a.k_pos0);
    x.all1 = keys ? x.all0 : a.mode == FWD_ROW ? 0 : kv_tiles_for(x.q0 + TILE, a.Tq, a.Tk, a.causal, a.q_pos0, a.k_pos0);
    const int all = max(x.all0, x.all1);
    const int per = (all + ns - 1) / ns;  // split 0 is never empty while any key is seen
    const int je = min(all, min(all, split * per) + per);
    x.jb = min(all, split * per);
    x.nk = je - x.jb;  // one per step (rows) or per product (keys)
    x.n0 = keys ? (x.nk + 1) / 2 : max(0, min(je, x.all0) - x.jb);
    x.n1 = keys ? x.nk / 2 : max(0, min(je, x.all1) - x.jb);
    return x;
}

}  // namespace fwd

// DROP: 0 none, 1 dense mask, 2 Philox.  JOB: what a CTA does with its items.  A kernel that contains cluster launch control is
// not started under the tail of the one before it, programmatic dependent launch or not, so grids that fit the device use one
// without (B1 H12 T512: 8.5 us, with it 9.5).
enum FwdJob { ONE_ITEM = 0, TAKE_OVER = 1, COMBINE_ITEM = 2 };  // COMBINE_ITEM: keys mode or key splits, merged at the end
// RUNS: the blocks come in runs of slices (take_in_groups).  A kernel without them is 1 % faster where there is one run (B8 H12
// T1024 39.3 -> 38.9 us), so there are both.
template <int DROP, int JOB, bool RUNS>
__global__ void __launch_bounds__(fwd::NUM_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapO, const __grid_constant__ FwdArgs a) {
    using namespace fwd;
    constexpr bool COMBINE = JOB == COMBINE_ITEM, TAKES_OVER = JOB == TAKE_OVER;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem + OFF_Q;
    uint8_t* sKV = smem + OFF_KV;
    Shared& sh = *reinterpret_cast<Shared*>(smem + OFF_SH);

    const int warp = (int)uniform(threadIdx.x >> 5);  // uniform for the compiler too: the issuing warp depends on it
    const int lane = threadIdx.x & 31;
    const int ns = COMBINE ? a.n_splits : 1;  // cluster size
    const int split = COMBINE && ns > 1 ? (int)cluster_ctarank() : 0;
    const bool keys = COMBINE && a.mode == FWD_KEYS;
    const int block_rows = a.mode == FWD_ROWS ? 2 * TILE : TILE;
    const Item first = make_item<RUNS>(a, blockIdx.x / ns, split, ns);

    auto end_of = [&](const Item& x) { return min(a.Tq, x.q0 + block_rows); };             // of the block's rows
    auto row0_of = [&](const Item& x, int t) { return x.q0 + (keys ? 0 : t * TILE); };      // first row of stream t
    // streams that have rows, whose O leaves through a slot of the ring
    auto o_slots = [&](const Item& x) { return !TAKES_OVER ? 0 : row0_of(x, 1) < end_of(x) ? 2 : 1; };
    auto load_q = [&](const Item& x, int t) {
        mbar_arrive_expect_tx(&sh.q_full[t], TILE_BYTES);
        tma_load_tile(sQ + t * TILE_BYTES, &mapQ, &sh.q_full[t], row0_of(x, t), x.h, x.b);
    };
    auto ring_end = [&](const Item& x) { return TAKES_OVER || x.nk == 0 ? 2 * x.nk : 2 * x.nk + 1; };
    auto in_ring = [&](const Item& x, int i) { return TAKES_OVER || i != 2 * x.nk - 1; };
    auto load_kv = [&](const Item& x, int i, uint32_t s) {  // entry i of the item's ring sequence, into slot s
        const bool last = TAKES_OVER && i == 2 * x.nk - 1;
        const bool v = i > 0 && ((i & 1) == 0 || last);
        const int tile = x.jb + (last ? x.nk - 1 : v ? (i - 2) / 2 : (i + 1) / 2);
        mbar_arrive_expect_tx(&sh.kv_full[s], TILE_BYTES);
        tma_load_tile(sKV + s * TILE_BYTES, v ? &mapV : &mapK, &sh.kv_full[s], tile * TILE, x.h, x.b);
    };

    // The producer initialises the barriers its copies complete on and issues the first loads at once (they wait for no
    // consumer): the rest of the set-up -- the other barriers, the tensor-memory allocation -- runs under their latency.
    // The other warps meet these barriers only after the __syncthreads below.
    if (warp == 0 && lane == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&sh.q_full[i], 1);
        for (int s = 0; s < SLOTS; ++s) mbar_init(&sh.kv_full[s], 1);
        fence_mbar_init();
        pdl_wait();  // whatever made Q, K, V
        pdl_trigger();
        if (first.nk > 0) {
            if (first.n0 > 0) load_q(first, 0);
            load_kv(first, 0, 0);
            if (first.n1 > 0 && !keys) load_q(first, 1);
#pragma unroll 1
            for (int i = 1; i < min(SLOTS, ring_end(first)); ++i)
                if (in_ring(first, i)) load_kv(first, i, i);
        }
    }
    if (threadIdx.x == 64) {  // another warp takes the rest of the barriers
        for (int s = 0; s < SLOTS; ++s) mbar_init(&sh.kv_empty[s], 1);
        // The score barriers belong to the score BUFFER, not to the stream: the warps of a stream may be a whole step
        // apart (the scores of the next step are there before the slowest warp has finished this one), and a
        // buffer is only refilled after every warp has handed over the P it held.
        // A wait by parity needs to know that the phase before it is complete: whoever waits for s_full of product q, that
        // S(q - 3) is.  A stream with a product among the last three has seen it.  One that sat out the item before (the last
        // block of a slice may be of one row tile, without stream 1) has not: with two key tiles its next product is number
        // three, and on the fresh barrier of buffer 0 the wait would pass before S(0).  An item is therefore made known
        // only when every score of such a one before it is complete (q_empty[0], in the producer).
        for (int bf = 0; bf < 3; ++bf) {
            mbar_init(&sh.s_full[bf], 1);
            mbar_init(&sh.p_full[bf], 4);  // one arrival per softmax warp of the stream
            mbar_init(&sh.o_full[bf], 1);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(&sh.q_empty[t], 1);
            mbar_init(&sh.o_staged[t], 4);
            mbar_init(&sh.o_taken[t], 1);
        }
        for (int i = 0; i < ITEMS; ++i) {
            mbar_init(&sh.item_full[i], 1);
            mbar_init(&sh.item_empty[i], 10);  // the issuing, the storing and the softmax warps
        }
        mbar_init(&sh.answered, 1);
        sh.abort.id = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(&sh.tmem_base, TMEM_COLS);
        tmem_relinquish();
        tc_fence_before_sync();
    }
    __syncthreads();
    tc_fence_after_sync();
    // The CTA holds all 512 columns of tensor memory, so its allocation starts at address 0.
    constexpr uint32_t tmem = 0;
    if (sh.tmem_base != tmem) sh.abort.id = 198;  // never expected
    WaitNote wc{&sh.abort};
    // all threads of the cluster (of the CTA, when it is alone)
    auto barrier_all = [&] {
        if (COMBINE && ns > 1) {
            __syncwarp();
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
    };

    // Work items.  A CTA that takes over starts with the item of its blockIdx and then, until none is left, takes over
    // those of CTAs that have not started yet (cluster launch control): Q and the first keys of the next item are loaded, and
    // its first scores computed, under the last steps of this one, and O leaves under the next one.  The producer asks, decodes
    // the answer and puts the item into a ring that every warp reads in its own time: item r > 0 in entry r - 1.
    auto read_item = [&](Item& x, int r, bool solo, bool release) -> bool {
        if (!TAKES_OVER) return false;
        const int buf = (r - 1) % ITEMS;
        bool ok = mbar_wait(wc, &sh.item_full[buf], ((r - 1) / ITEMS) & 1, W_ITEM, r);
        if (!solo) ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        x = sh.item[buf];
        if (!solo) __syncwarp();
        if (release && (solo || lane == 0)) mbar_arrive(&sh.item_empty[buf]);
        return x.n0 >= 0;
    };

    if (warp < 4) {
        reg_release();
        if (warp == 0) {
            // ------------------------------ TMA producer ------------------------------
            if (lane == 0) {
                Item x = first;
                int q0_uses = first.n0 > 0 ? 1 : 0, q1_uses = first.n1 > 0 ? 1 : 0;  // loads of the streams' Q tiles
                bool tok = true;
                // entry e of the ring: free when what it held SLOTS entries ago has been used up
                auto free_slot = [&](int e) -> bool {
                    return e < SLOTS || (tok = mbar_wait(wc, &sh.kv_empty[e % SLOTS], (e / SLOTS - 1) & 1, W_KVEMPTY, e));
                };
                for (int r = 0, base = 0;; ++r) {
                    for (int i = r == 0 ? min(SLOTS, ring_end(x)) : 0; i < ring_end(x); ++i) {
                        if (!in_ring(x, i)) continue;
                        if (!free_slot(base + i)) break;
                        load_kv(x, i, (base + i) % SLOTS);
                        if (i == 0 && x.n1 > 0) {  // Q of the second stream behind the first keys
                            if (q1_uses > 0 && !(tok = mbar_wait(wc, &sh.q_empty[1], (q1_uses - 1) & 1, W_QEMPTY, r))) break;
                            load_q(x, 1);
                            ++q1_uses;
                        }
                    }
                    if (!TAKES_OVER || !tok) break;
                    base += 2 * x.nk;
                    // asked for here, a step or two before this CTA is through
                    mbar_arrive_expect_tx(&sh.answered, sizeof(uint4));
                    clc_try_cancel(&sh.answer, &sh.answered);
                    const int n_o = o_slots(x);
                    for (int t = 0; tok && t < n_o; ++t, ++base)
                        if (free_slot(base)) mbar_arrive(&sh.kv_full[base % SLOTS]);
                    if (!tok || !(tok = mbar_wait(wc, &sh.answered, r & 1, W_ITEM, r))) break;
                    const int id = clc_read(&sh.answer);
                    fence_proxy_async_smem();  // the answer's buffer is next written by the async proxy
                    const int buf = r % ITEMS;
                    if (r >= ITEMS && !(tok = mbar_wait(wc, &sh.item_empty[buf], (r / ITEMS - 1) & 1, W_ITEM, 1000 + r))) break;
                    if (id >= 0) {
                        // The next item is made known behind the last score of stream 0 in this one: see s_full.  Q and K of the
                        // next item wait for it anyway.
                        if (q0_uses > 0 && !(tok = mbar_wait(wc, &sh.q_empty[0], (q0_uses - 1) & 1, W_QEMPTY, r))) break;
                        x = make_item<RUNS>(a, id, 0, 1);
                        sh.item[buf] = x;
                    } else {
                        sh.item[buf].n0 = -1;
                    }
                    mbar_arrive(&sh.item_full[buf]);
                    if (id < 0) break;
                    if (x.n0 > 0) {
                        load_q(x, 0);
                        ++q0_uses;
                    }
                }
                // Every copy has landed once the softmax warps have seen the last product complete (they wait for it, and
                // the barrier below waits for them).  Only a CTA that gave up may have some in flight still: give them
                // time to land before it leaves.
                if (!tok)
                    for (const unsigned long long t0 = globaltimer_ns(); globaltimer_ns() - t0 < 100000ull;) {}
            }
        } else if (warp == 1) {
            // ------------------------------ MMA issuer ------------------------------
            // The whole warp runs this code with uniform control flow; only the tcgen05 instructions are predicated
            // on the elected lane (see umma_ss_tf32_lead).
            //
            // The tensor pipe takes instructions about as fast as it executes them and queues next to none, so every
            // cycle this warp spends on something else than issuing leaves the pipe idle.  A wait costs some 150 cycles
            // even when the barrier completed long ago; each barrier is therefore looked at (test_wait) while the MMAs
            // before it are still being issued, and waited for only if that look came too early.
            const uint32_t leader = elect_one_sync();
            auto wait = [&](bool seen, uint64_t* bar, uint32_t parity, int id, int aux) -> bool {
                if (__all_sync(0xffffffffu, seen)) return true;
                return __all_sync(0xffffffffu, mbar_wait(wc, bar, parity, id, aux));
            };
            constexpr uint32_t IDESC_S = make_idesc_tf32(TILE, TILE, false, false);
            constexpr uint32_t IDESC_O = make_idesc_tf32(TILE, HEAD_DIM, false, true);
            // products in issue order: step by step, stream 0 before stream 1 (a stream takes part while j < n_t), item by item
            struct Product {
                int n0, n1, nk, left;  // of the item: steps of the streams, key tiles, products from this one on
                int j, t, idx;         // step, stream, number of its key tile
                int buf;               // score buffer
                uint32_t par;          // parity of the score buffer's barriers
                int ke, ve;            // ring entries of its key and value tile
                RingPos k, v;          // the same as slots
                int base, r;           // ring entry behind the item, the item's number
            };
            auto start = [&](Product& p, const Item& x) {  // at the first product of an item
                auto u = [](int v) { return TAKES_OVER ? (int)uniform(v) : v; };
                p.n0 = u(x.n0), p.n1 = u(x.n1), p.nk = u(x.nk);
                p.left = p.n0 + p.n1;
                p.j = p.idx = 0;
                p.t = p.n0 > 0 ? 0 : 1;
                p.ke = p.base, p.ve = p.base + ring_v<TAKES_OVER>(0, p.nk);
                p.k = RingPos(p.ke), p.v = RingPos(p.ve);
                p.base += 2 * p.nk + u(o_slots(x));
            };
            auto step = [&](Product& p) {  // past a product, inside the item
                if (++p.buf == 3) {
                    p.buf = 0;
                    p.par ^= 1u;
                }
                --p.left;
                const bool next_step = p.t == 1 || p.j >= p.n1;
                if (next_step) ++p.j;
                p.t = (next_step && p.j < p.n0) ? 0 : 1;
                if (next_step || keys) {
                    ++p.idx;
                    const int dk = p.idx == 1 ? 1 : 2, dv = TAKES_OVER && p.idx == p.nk - 1 ? 1 : 2;
                    if (TAKES_OVER) p.ke += dk, p.ve += dv;
                    p.k.advance(dk), p.v.advance(dv);
                }
            };
            // first and last product that reads its K / V tile
            auto new_kv = [&](const Product& p) { return keys || p.t == 0 || p.j >= p.n0; };
            auto last_kv = [&](const Product& p) { return keys || p.t == 1 || p.j >= p.n1; };
            const Desc q_desc = kmajor_desc(smem_u32(sQ), 0, BOX_BYTES), k_desc = kmajor_desc(smem_u32(sKV), 0, BOX_BYTES),
                       v_desc = mnmajor_desc(smem_u32(sKV), 0, BOX_BYTES);
            auto issue_qk = [&](const Product& p, int box) {  // 32 of the 64 d's
                umma_ss4<KMAJOR_STEP, KMAJOR_STEP>(leader, tmem + score_col(p.buf),
                                                   q_desc + ((keys ? 0 : p.t * TILE_BYTES) + box * BOX_BYTES),
                                                   k_desc + (p.k.slot * TILE_BYTES + box * BOX_BYTES), IDESC_S, box);
            };
            const bool state_in = a.continue_state && split == 0;
            Product pq{0, 0, 0, 0, 0, 0, 0, 0, 0u, 0, 0, RingPos(0u), RingPos(0u), 0, 0};  // the next S = Q K^T to issue
            start(pq, first);
            Product pv = pq;               // the next P V to issue
            uint32_t q_par = 0u;           // bit t: parity of stream t's Q tile
            int ahead = 0, released = 0;   // products between the two; items handed back
            bool done = !TAKES_OVER, ok = true, seen_k = false, seen_v = false, seen_p = false;
            auto release_to = [&](int r) {
#pragma unroll 1
                for (; released < r; ++released)
                    if (lane == 0) mbar_arrive(&sh.item_empty[released % ITEMS]);
            };
            while (ok) {
                // Scores are computed up to three products ahead, into the next item if that is known already.  Neither it nor a
                // key tile is waited for while that may take a P V that is not issued yet: the ring entry five in front of
                // the key tile's must have been used up by those that are.
                if (TAKES_OVER && pq.left == 0 && !done && (ahead == 0 || __all_sync(0xffffffffu, mbar_test_wait(&sh.item_full[pq.r % ITEMS], (pq.r / ITEMS) & 1)))) {
                    Item x;
                    done = !__all_sync(0xffffffffu, read_item(x, ++pq.r, false, false));
                    if (!done) start(pq, x);
                    continue;
                }
                if (pq.left > 0 && ahead < 3 && (!TAKES_OVER || ahead == 0 || pq.ke < pv.ve + SLOTS)) {
                    if (TAKES_OVER && ahead == 0) pv = pq;
                    if (pq.j == 0) {
                        if (!(ok = wait(false, &sh.q_full[keys ? 0 : pq.t], (q_par >> pq.t) & 1u, W_QFULL, pq.t))) break;
                        if (!keys) q_par ^= 1u << pq.t;
                    }
                    if (new_kv(pq) && !(ok = wait(seen_k, &sh.kv_full[pq.k.slot], pq.k.phase, W_KFULL, pq.j))) break;
                    tc_fence_after_sync();
                    issue_qk(pq, 0);
                    seen_v = mbar_test_wait(&sh.kv_full[pv.v.slot], pv.v.phase);
                    seen_p = mbar_test_wait(&sh.p_full[pv.buf], pv.par);
                    // on to the next product between the MMAs, whose issue hides it (2 % at 512 queries against 8 192 keys); with
                    // items to take over the copies cost more than that
                    Product next = pq;
                    if (!TAKES_OVER) step(next);
                    issue_qk(pq, 1);
                    umma_commit_lead(leader, &sh.s_full[pq.buf]);
                    if (last_kv(pq)) umma_commit_lead(leader, &sh.kv_empty[pq.k.slot]);
                    if (TAKES_OVER && pq.j + 1 == (pq.t == 0 ? pq.n0 : pq.n1)) umma_commit_lead(leader, &sh.q_empty[pq.t]);
                    if (TAKES_OVER) step(next);
                    pq = next;
                    seen_k = false;
                    if (++ahead < 3) continue;
                }
                if (ahead == 0) {
                    if (!TAKES_OVER || done) break;
                    continue;
                }
#pragma unroll 1
                while (TAKES_OVER && pv.left == 0) {  // on to the item the scores went on to before
                    Item x;
                    if (!(ok = __all_sync(0xffffffffu, read_item(x, ++pv.r, false, false)))) break;
                    start(pv, x);
                    seen_v = false;  // that look was at another entry
                }
                if (!ok) break;
                if (TAKES_OVER) release_to(pv.r);
                if (new_kv(pv) && !(ok = wait(seen_v, &sh.kv_full[pv.v.slot], pv.v.phase, W_VFULL, pv.j))) break;
                if (!(ok = wait(seen_p, &sh.p_full[pv.buf], pv.par, W_PFULL, pv.j))) break;
                tc_fence_after_sync();
                if (pq.left > 0) seen_k = mbar_test_wait(&sh.kv_full[pq.k.slot], pq.k.phase);
                Product next = pv;
                {  // O_t += P V, P in the product's score buffer
                    const uint32_t pc = tmem + score_col(pv.buf), d = tmem + COL_O0 + pv.t * HEAD_DIM;
                    const Desc vd = v_desc + pv.v.slot * TILE_BYTES;
                    umma_ts4<MNMAJOR_STEP>(leader, d, pc, vd, IDESC_O, (pv.j > 0 || (state_in && !(keys && pv.t == 1))) ? 1u : 0u);
                    umma_ts4<MNMAJOR_STEP>(leader, d, pc + 32, vd + 4096, IDESC_O, 1u);
                    if (!TAKES_OVER) step(next);
#pragma unroll
                    for (int g = 2; g < 4; ++g) umma_ts4<MNMAJOR_STEP>(leader, d, pc + 32 * g, vd + 4096 * g, IDESC_O, 1u);
                    umma_commit_lead(leader, &sh.o_full[pv.buf]);
                    if (last_kv(pv)) umma_commit_lead(leader, &sh.kv_empty[pv.v.slot]);
                }
                if (TAKES_OVER) step(next);
                pv = next;
                --ahead;
                seen_v = seen_p = false;
            }
        } else if (TAKES_OVER && warp == 2) {
            // ------------------------------ store warp ------------------------------
            if (lane == 0) {
                pdl_wait();
                Item x = first;
                uint32_t par = 0u;  // bit t: parity of stream t's barrier
                bool tok = true;
                for (int r = 0, base = 0; tok; ) {
                    base += 2 * x.nk;
                    const int n_o = o_slots(x);
                    for (int t = 0; t < n_o; ++t, ++base) {
                        if (!(tok = mbar_wait(wc, &sh.o_staged[t], (par >> t) & 1u, W_OSTAGED, r))) break;
                        par ^= 1u << t;
                        mbar_arrive(&sh.o_taken[t]);
                        // rows past the end of the sequence are clipped by the copy
                        tma_store_tile(&mapO, sKV + base % SLOTS * TILE_BYTES, row0_of(x, t), x.h, x.b);
                        bulk_commit_group();
                        bulk_wait_group_read_all();  // the copy has read its source; it completes on its own
                        mbar_arrive(&sh.kv_empty[base % SLOTS]);
                    }
                    if (!tok || !read_item(x, ++r, true, true)) break;
                }
            }
        }
        // teardown of the control warps (kept inside this branch: the two register regimes never
        // share code after the hand-over)
        if (COMBINE) barrier_all();  // partial results staged
        tc_fence_before_sync();
        barrier_all();
        if (warp == 1) {
            tc_fence_after_sync();
            tmem_dealloc(tmem, TMEM_COLS);
            if (lane == 0) report_abort(sh.abort, a.status);
        }
    } else {
        // ------------------------------ softmax ------------------------------
        reg_acquire();
        pdl_wait();  // these warps write the outputs, which an earlier kernel may still be using
        const int t = (warp - 4) >> 2;                   // stream
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;             // row inside the product = tensor-memory lane
        const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
        const uint32_t tO = trow + COL_O0 + t * HEAD_DIM;
        const float cs = a.scale_log2e;
        const float worst = (cs >= 0.f) ? -INFINITY : INFINITY;  // raw score that can never win the max
        const bool scaled = a.drop_scaled != 0;
        bool ok = true;
        uint32_t r[128];

        Item x = first;
        int base = 0, q_base = 0, uses = 0;  // ring entries, products of the items before; items in which this stream had rows
        for (int item = 0; ok;) {
            const int n0 = x.n0, n1 = x.n1, b = x.b, h = x.h, bh = x.bh, q_end = end_of(x);
            const int nt = x.steps(t);
            const int qrow = row0_of(x, t) + row;               // row inside this (b,h)
            const bool row_ok = qrow < q_end;
            const bool warp_live = row0_of(x, t) + quarter * 32 < q_end;  // any row of this warp exists
            // last key index (local to this call's K) this row may see
            long long lim_ll = a.Tk - 1;
            if (a.causal) lim_ll = min(lim_ll, (long long)a.q_pos0 + qrow - a.k_pos0);
            const int kv_lim = row_ok ? (int)max(-1ll, lim_ll) : -1;
            const bool state_in = a.continue_state && split == 0 && !(keys && t == 1);

            const uint2 row_part = DROP == 2 ? hk_philox_row_part(a.philox_keys, a.bh_pos0 + (uint32_t)bh, (uint32_t)(a.q_pos0 + qrow)) : make_uint2(0u, 0u);
            float m = -INFINITY;  // running max actually used as exponent reference, log2 units
            float l = 0.f;
            if (state_in && nt > 0) {
                // The result over the keys seen so far is the starting state: reference LSE, normaliser 1 and the running
                // output O itself (a row that has seen no key starts from nothing).  The output accumulator is written
                // before this warp's first arrival on p_full, which the first P V of the stream waits for.
                const float lse0 = row_ok ? a.LSE[(int64_t)b * a.lse_sB + (int64_t)h * a.lse_sH + qrow] : -INFINITY;
                const bool have = lse0 > -INFINITY;
                m = have ? lse0 * LOG2E : -INFINITY;
                l = have ? 1.f : 0.f;
                const float4* orow = reinterpret_cast<const float4*>(a.O + (int64_t)b * a.o_sB + (int64_t)h * a.o_sH +
                                                                     (int64_t)(row_ok ? qrow : 0) * a.o_sM);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float4 v = have ? orow[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                    r[4 * i] = __float_as_uint(v.x); r[4 * i + 1] = __float_as_uint(v.y);
                    r[4 * i + 2] = __float_as_uint(v.z); r[4 * i + 3] = __float_as_uint(v.w);
                }
                tmem_st32p(tO, r);
                tmem_st32p(tO + 32, r + 32);
                tmem_wait_st();
            }

            // a product's number in the issue order picks its score buffer
            auto product = [&](int j) { return q_base + min(j, n0) + min(j, n1) + ((t == 1 && j < n0) ? 1 : 0); };
            int q_prev = 0;  // number of this stream's previous product
            for (int j = 0; j < nt; ++j) {
                const int q = product(j);
                const int buf = q % 3;
                const uint32_t tS = trow + score_col(buf);
                // the vote keeps the warp converged for the .sync.aligned tensor-memory accesses below
                ok = __all_sync(0xffffffffu, mbar_wait(wc, &sh.s_full[buf], (q / 3) & 1, W_SFULL, j));
                if (!ok) break;
                if (warp_live) {
                    tc_fence_after_sync();
                    tmem_ld32p(tS, r);
                    tmem_ld32p(tS + 32, r + 32);
                    tmem_ld32p(tS + 64, r + 64);
                    tmem_ld32p(tS + 96, r + 96);
                    const int kv0 = (x.jb + (keys ? 2 * j + t : j)) * TILE;
                    const int lim_local = kv_lim - kv0;  // columns 0..lim_local are visible
                    tmem_wait_ld();
                    if (lim_local < TILE - 1) {
#pragma unroll
                        for (int i = 0; i < 128; ++i)
                            if (i > lim_local) r[i] = __float_as_uint(worst);
                    }
                    // row max of the raw scores (min if the scale is negative), four chains
                    float mx0 = __uint_as_float(r[0]), mx1 = __uint_as_float(r[1]), mx2 = __uint_as_float(r[2]),
                          mx3 = __uint_as_float(r[3]);
                    if (cs >= 0.f) {
#pragma unroll
                        for (int i = 4; i < 124; i += 8) {
                            mx0 = fmax3(mx0, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                            mx1 = fmax3(mx1, __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
                            mx2 = fmax3(mx2, __uint_as_float(r[i + 4]), __uint_as_float(r[i + 5]));
                            mx3 = fmax3(mx3, __uint_as_float(r[i + 6]), __uint_as_float(r[i + 7]));
                        }
                        mx0 = fmax3(mx0, __uint_as_float(r[124]), __uint_as_float(r[125]));
                        mx1 = fmax3(mx1, __uint_as_float(r[126]), __uint_as_float(r[127]));
                        mx0 = fmax3(fmaxf(mx0, mx1), mx2, mx3);
                    } else {
#pragma unroll
                        for (int i = 4; i < 128; i += 4) {
                            mx0 = fminf(mx0, __uint_as_float(r[i]));
                            mx1 = fminf(mx1, __uint_as_float(r[i + 1]));
                            mx2 = fminf(mx2, __uint_as_float(r[i + 2]));
                            mx3 = fminf(mx3, __uint_as_float(r[i + 3]));
                        }
                        mx0 = fminf(fminf(mx0, mx1), fminf(mx2, mx3));
                    }
                    const float m_cand = mx0 * cs;  // -inf when nothing is visible
                    // raise the reference only when it pays: a stale m makes p at most 2^8 larger, which fp32 absorbs
                    const bool raise = (m == -INFINITY) ? (m_cand > -INFINITY) : (m_cand > m + RESCALE_THRESHOLD);
                    const float m_new = raise ? m_cand : m;
                    const float alpha = raise ? ((m == -INFINITY) ? 0.f : ex2_approx(m - m_cand)) : 1.f;
                    if ((j > 0 || state_in) && __any_sync(0xffffffffu, raise)) {
                        // rescale the running output, once the P V of the previous step has completed
                        if (j > 0) {
                            ok = __all_sync(0xffffffffu, mbar_wait(wc, &sh.o_full[q_prev % 3], (q_prev / 3) & 1, W_OFULL, j));
                            if (!ok) break;
                            tc_fence_after_sync();
                        }
#pragma unroll 1
                        for (int cc = 0; cc < 2; ++cc) {
                            uint32_t o[32];
                            tmem_ld32(tO + cc * 32, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st32(tO + cc * 32, o);
                        }
                    }
                    const float neg_m = (m_new == -INFINITY) ? 0.f : -m_new;
                    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
                    if constexpr (DROP == 0) {
                        // two scores per FMA and per add (fma.rn.f32x2 / add.rn.f32x2: the same roundings as the scalar forms)
                        const float2 c2 = make_float2(cs, cs), nm2 = make_float2(neg_m, neg_m);
                        float2 s01 = make_float2(0.f, 0.f), s23 = make_float2(0.f, 0.f);
#pragma unroll
                        for (int i = 0; i < 128; i += 4) {
                            const float2 t01 = __ffma2_rn(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), c2, nm2);
                            const float2 t23 = __ffma2_rn(make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), c2, nm2);
                            const float2 p01 = make_float2(ex2_approx(t01.x), ex2_approx(t01.y));
                            const float2 p23 = make_float2(ex2_approx(t23.x), ex2_approx(t23.y));
                            s01 = __fadd2_rn(s01, p01);
                            s23 = __fadd2_rn(s23, p23);
                            r[i] = tf32_round_bits_mma(__float_as_uint(p01.x));
                            r[i + 1] = tf32_round_bits_mma(__float_as_uint(p01.y));
                            r[i + 2] = tf32_round_bits_mma(__float_as_uint(p23.x));
                            r[i + 3] = tf32_round_bits_mma(__float_as_uint(p23.y));
                        }
                        s0 = s01.x; s1 = s01.y; s2 = s23.x; s3 = s23.y;
                    } else if constexpr (DROP == 2) {
                        // One Philox call per eight keys of this row.  32 keys at a time, read from tensor memory once more, in a
                        // rolled loop: the integer arithmetic is what dropout costs, and unrolled over the 128 registers
                        // its code does not stay in the instruction cache.  None for 32 keys that no row of the warp
                        // sees (on the diagonal three in eight).
                        const float2 c2 = make_float2(cs, cs), nm2 = make_float2(neg_m, neg_m);
                        float2 sk = make_float2(0.f, 0.f), sa = make_float2(0.f, 0.f);  // kept terms, all terms
                        const int warp_lim = __reduce_max_sync(0xffffffffu, lim_local);
                        // The part of the 16 calls that depends on the keys alone is the same for all rows: a lane works out one,
                        // and the others read it from where the warp's m and l go at the end.  The integer products are what
                        // dropout costs: 15 instead of 20 per call, each by one wide multiplication, took B16 H16 T2048 without
                        // a mask from 846 to 809 us, B8 H12 T1024 from 58.7 to 56.8 (ten launches after a pause, 1 965 MHz).
                        uint4 *keys0 = reinterpret_cast<uint4*>(&sh.m[t][quarter * 32]), *keys8 = reinterpret_cast<uint4*>(&sh.l[t][quarter * 32]);
                        if (lane < 16)
                            (lane < 8 ? keys0 : keys8)[lane & 7] = hk_philox_key_part(a.philox_keys, a.philox_offset, a.bh_pos0 + (uint32_t)bh,
                                                                                      ((uint32_t)(a.k_pos0 + kv0) >> 3) + lane);
                        __syncwarp();
#pragma unroll 1
                        for (int c = 0; c < 128; c += 32) {
                            if (c > warp_lim) {
#pragma unroll
                                for (int u = 0; u < 32; ++u) r[u] = 0u;
                            } else {
                                tmem_ld32p(tS + c, r);
                                hk_philox4_t w[4];
#pragma unroll
                                for (int g = 0; g < 4; ++g)
                                    w[g] = hk_philox_join(a.philox_keys, (c < 64 ? keys0 : keys8)[(c & 63) / 8 + g], row_part);
                                tmem_wait_ld();
                                if (lim_local < c + 31) {
#pragma unroll
                                    for (int i = 0; i < 32; ++i)
                                        if (c + i > lim_local) r[i] = __float_as_uint(worst);
                                }
#pragma unroll
                                for (int i = 0; i < 32; i += 2) {
                                    const float2 t01 = __ffma2_rn(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), c2, nm2);
                                    float2 p = make_float2(ex2_approx(t01.x), ex2_approx(t01.y));
                                    if (scaled) sa = __fadd2_rn(sa, p);  // the normaliser ignores the mask
                                    if (!hk_philox_keep1(w[i >> 3], i & 7, a.drop_thr)) p.x = 0.f;
                                    if (!hk_philox_keep1(w[i >> 3], (i & 7) + 1, a.drop_thr)) p.y = 0.f;
                                    sk = __fadd2_rn(sk, p);
                                    r[i] = tf32_round_bits_mma(__float_as_uint(p.x));
                                    r[i + 1] = tf32_round_bits_mma(__float_as_uint(p.y));
                                }
                            }
                            tmem_st32p(tS + c, r);
                        }
                        __syncwarp();  // the next step's parts go to the same place
                        s0 = sk.x; s1 = sk.y; s2 = sa.x; s3 = sa.y;
                    } else {
                        const float* mrow = a.mask + ((size_t)bh * a.Tq + (row_ok ? qrow : 0)) * (size_t)a.Tk + kv0;
#pragma unroll
                        for (int i = 0; i < 128; ++i) {
                            float p = ex2_approx(fmaf(__uint_as_float(r[i]), cs, neg_m));
                            if (scaled) s2 += (i <= lim_local) ? p : 0.f;
                            p = (i <= lim_local) ? p * __ldg(mrow + i) : 0.f;
                            s0 += p;
                            r[i] = tf32_round_bits_mma(__float_as_uint(p));
                        }
                    }
                    if constexpr (DROP != 2) {
                        tmem_st32p(tS, r);
                        tmem_st32p(tS + 32, r + 32);
                        tmem_st32p(tS + 64, r + 64);
                        tmem_st32p(tS + 96, r + 96);
                    }
                    // inverted dropout: s2, s3 hold the sums over all visible keys, s0, s1 the kept ones
                    l = l * alpha + ((scaled && DROP != 0) ? (s2 + s3) : ((s0 + s1) + (s2 + s3)));
                    m = m_new;
                    tmem_wait_st();
                    tc_fence_before_sync();
                }
                mbar_arrive_warp(&sh.p_full[buf], lane);
                q_prev = q;
            }

            // epilogue: O / l and LSE
            if (ok && nt > 0) ok = __all_sync(0xffffffffu, mbar_wait(wc, &sh.o_full[q_prev % 3], (q_prev / 3) & 1, W_OFULL, nt));
            tc_fence_after_sync();
            const float inv_l = COMBINE ? 1.f : (l > 0.f) ? a.keep_scale / l : 0.f;
            if (ok && nt > 0) {
                tmem_ld32p(tO, r);
                tmem_ld32p(tO + 32, r + 32);
                tmem_wait_ld();
                tc_fence_before_sync();  // the next item's first P V overwrites it
            } else {
#pragma unroll
                for (int i = 0; i < 64; ++i) r[i] = 0u;
            }
            // O leaves through shared memory (a thread-per-row store would touch 32 lines per instruction): a slot of the ring or, with
            // one item, the stream's own Q buffer, which is dead -- o_full covered its last S = Q K^T, and in keys mode,
            // where the streams share Q, every S: the last one is issued before the last two P V.  Either way as the two
            // 32-column boxes of a 128-byte-swizzled TMA tile: 16-byte chunk i of row r at position i ^ (r & 7).
            auto stage = [&](uint8_t* dst) {
                uint8_t* srow = dst + row * 128;
#pragma unroll
                for (int ch = 0; ch < 16; ++ch)
                    *reinterpret_cast<float4*>(srow + (ch >> 3) * BOX_BYTES + (((ch & 7) ^ (row & 7)) << 4)) =
                        make_float4(__uint_as_float(r[4 * ch]) * inv_l, __uint_as_float(r[4 * ch + 1]) * inv_l,
                                    __uint_as_float(r[4 * ch + 2]) * inv_l, __uint_as_float(r[4 * ch + 3]) * inv_l);
            };
            if constexpr (TAKES_OVER) {
                const int n_o = o_slots(x);
                if (ok && t < n_o) {
                    const int e = base + 2 * x.nk + t;
                    ok = (uses == 0 || mbar_wait(wc, &sh.o_taken[t], (uses - 1) & 1, W_OSLOT, 1000 + item)) &&
                         mbar_wait(wc, &sh.kv_full[e % SLOTS], (e / SLOTS) & 1, W_OSLOT, item);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    ++uses;
                    stage(sKV + e % SLOTS * TILE_BYTES);
                    fence_proxy_async_smem();
                    mbar_arrive_warp(&sh.o_staged[t], lane);
                    if (row_ok)
                        a.LSE[(int64_t)b * a.lse_sB + (int64_t)h * a.lse_sH + qrow] = (l > 0.f) ? (m + log2f(l)) * LN2 : -INFINITY;
                }
                base += 2 * x.nk + n_o;
                q_base += n0 + n1;
                if (!ok || !read_item(x, ++item, false, true)) break;
            } else if constexpr (!COMBINE) {
                stage(sQ + t * TILE_BYTES);
                fence_proxy_async_smem();
                // a block none of whose rows sees a key of this call leaves a continued result untouched
                const bool keep_old = a.continue_state && nt == 0;
                if (row_ok && !keep_old)
                    a.LSE[(int64_t)b * a.lse_sB + (int64_t)h * a.lse_sH + qrow] = (l > 0.f) ? (m + log2f(l)) * LN2 : -INFINITY;
                // the 128 threads of this stream (every one gets here, whatever `ok` is), then one of them stores
                asm volatile("bar.sync %0, 128;" ::"r"(1 + t) : "memory");
                if (row == 0 && row_ok && !keep_old) {
                    tma_store_tile(&mapO, sQ + t * TILE_BYTES, qrow, h, b);
                    bulk_commit_group();
                    bulk_wait_group_read_all();  // the copy has read its source; it completes on its own
                }
                break;
            } else {
                const int all0 = x.all0, all1 = x.all1;
                stage(sQ + t * TILE_BYTES);
                // Combine: O = sum_s O_s 2^(m_s - M) / sum_s l_s 2^(m_s - M) over the splits and, in keys mode, the two
                // streams.  Each CTA takes an equal slice of the rows it shares with its counterparts, 16 threads per row.
                sh.m[t][row] = m;
                sh.l[t][row] = l;
                barrier_all();
                const int rows = block_rows / ns, streams = keys ? 2 : 1;
#pragma unroll 1
                for (int i = threadIdx.x - 128; i < rows * 16; i += NUM_SOFTMAX) {
                    const int rr = split * rows + (i >> 4), ch = i & 15;
                    const int tt = rr / TILE, r1 = rr % TILE;
                    const int qr = row0_of(x, tt) + r1;
                    if (qr >= q_end || (a.continue_state && (tt == 0 ? all0 : all1) == 0)) continue;
                    const uint8_t* src = sQ + tt * TILE_BYTES + (ch >> 3) * BOX_BYTES + r1 * 128 + (((ch & 7) ^ (r1 & 7)) << 4);
                    float M = -INFINITY, L = 0.f;
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    auto fold = [&](float ms, float ls, const float4& v) {
                        const float Mn = fmaxf(M, ms);
                        const float wa = M == -INFINITY ? 0.f : ex2_approx(M - Mn), w = ms == -INFINITY ? 0.f : ex2_approx(ms - Mn);
                        L = L * wa + w * ls;
                        acc.x = acc.x * wa + w * v.x; acc.y = acc.y * wa + w * v.y;
                        acc.z = acc.z * wa + w * v.z; acc.w = acc.w * wa + w * v.w;
                        M = Mn;
                    };
                    for (int u = 0; u < streams; ++u) {
                        if (ns == 1) {
                            fold(sh.m[tt + u][r1], sh.l[tt + u][r1], *reinterpret_cast<const float4*>(src + u * TILE_BYTES));
                        } else {
                            for (int s0 = 0; s0 < ns; s0 += 2) {
                                float ms[2], ls[2];
                                float4 v[2];
#pragma unroll
                                for (int s = 0; s < 2; ++s) {
                                    ms[s] = ld_cluster_f(mapa(&sh.m[tt + u][r1], s0 + s));
                                    ls[s] = ld_cluster_f(mapa(&sh.l[tt + u][r1], s0 + s));
                                    v[s] = ld_cluster_f4(mapa(src + u * TILE_BYTES, s0 + s));
                                }
                                fold(ms[0], ls[0], v[0]);
                                fold(ms[1], ls[1], v[1]);
                            }
                        }
                    }
                    const float f = (L > 0.f) ? a.keep_scale / L : 0.f;
                    reinterpret_cast<float4*>(a.O + (int64_t)b * a.o_sB + (int64_t)h * a.o_sH + (int64_t)qr * a.o_sM)[ch] =
                        make_float4(acc.x * f, acc.y * f, acc.z * f, acc.w * f);
                    if (ch == 0)
                        a.LSE[(int64_t)b * a.lse_sB + (int64_t)h * a.lse_sH + qr] = (L > 0.f) ? (M + log2f(L)) * LN2 : -INFINITY;
                }
                break;
            }
        }  // items
        tc_fence_before_sync();
        barrier_all();  // pairs with the control warps' barrier before tensor memory is freed
    }
}

// Per-device launch data: the large shared-memory opt-in and how many clusters of each size run at once.
namespace {
struct FwdDevice {
    std::once_flag once;
    cudaError_t rc = cudaSuccess;
    int slots[4] = {148, 74, 33, 15};  // resident clusters of 1, 2, 4, 8 CTAs; the device is asked
};
typedef void (*FwdKernel)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, FwdArgs);
const FwdKernel fwd_kernels[15] = {
    attn_fwd_kernel<0, ONE_ITEM, false>,     attn_fwd_kernel<1, ONE_ITEM, false>,     attn_fwd_kernel<2, ONE_ITEM, false>,
    attn_fwd_kernel<0, TAKE_OVER, false>,    attn_fwd_kernel<1, TAKE_OVER, false>,    attn_fwd_kernel<2, TAKE_OVER, false>,
    attn_fwd_kernel<0, COMBINE_ITEM, false>, attn_fwd_kernel<1, COMBINE_ITEM, false>, attn_fwd_kernel<2, COMBINE_ITEM, false>,
    attn_fwd_kernel<0, ONE_ITEM, true>,      attn_fwd_kernel<1, ONE_ITEM, true>,      attn_fwd_kernel<2, ONE_ITEM, true>,
    attn_fwd_kernel<0, TAKE_OVER, true>,     attn_fwd_kernel<1, TAKE_OVER, true>,     attn_fwd_kernel<2, TAKE_OVER, true>};

// of the current device; set up by the first call on it
int fwd_device(FwdDevice** out) {
    static FwdDevice devices[HK_MAX_DEVICES];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return HK_ERR_CUDA;
    if (dev < 0 || dev >= HK_MAX_DEVICES) return HK_ERR_UNSUPPORTED;
    FwdDevice& d = devices[dev];
    std::call_once(d.once, [&d] {
        d.slots[0] = sm_count();
        for (FwdKernel k : fwd_kernels)
            if (d.rc == cudaSuccess)
                d.rc = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd::SMEM_BYTES);
        for (int i = 1; i < 4 && d.rc == cudaSuccess; ++i) {
            LaunchConfig lc(8u << i, fwd::NUM_THREADS, fwd::SMEM_BYTES, nullptr, 1 << i, false);
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, fwd_kernels[6], &lc.cfg) == cudaSuccess && n > 0) d.slots[i] = n;
        }
    });
    if (d.rc != cudaSuccess) return HK_ERR_CUDA;
    *out = &d;
    return HK_OK;
}

}  // namespace

int attn_fwd_slots(const int** slots) {
    FwdDevice* d = nullptr;
    const int rc = fwd_device(&d);
    if (rc == HK_OK) *slots = d->slots;
    return rc;
}

FwdPlan plan_attn_fwd(int BH, int Tq, int Tk, int causal, int q_pos0, int k_pos0, bool drop, const int slots[4]) {
    // Mode and splits by estimates of the makespan.  Rows mode loads a key tile once for two products and is the fastest
    // where it fills the chip; row mode where it does not; keys mode and splits when even those leave most SMs idle (512
    // queries of 32 heads against 8 192 keys: 64 CTAs of 64 steps on 148 SMs).  Those two sum in another order, and the choice
    // depends on batch x heads: they are left out for sequences of training length, so that a batch cut into calls gives the
    // bits of the single call.
    //
    // Two estimates.  The coarse one takes the mean load of a slot plus half of the longest cluster, but at least that
    // cluster, whether or not one wave holds all of them; a CTA costs ~3.5 us and ~2.1 us per step of two products (1.5 with
    // one stream, 2.3 in keys mode), ~2 us more when it merges streams and ~3 us more when it combines splits.  The fine one
    // tells one wave from several and is fitted to kernel times of every cut of 330 shapes, with dropout and without (1 - 400
    // slices, 16 - 12 000 queries, 64 - 18 000 keys).  It is off by 9 % on average, so it replaces the coarse one's cut only
    // where it expects a gain of 15 % (13 % between rows and row mode): a quarter of those shapes, chosen close to the lines
    // between the cuts.  Of 1 000 further ones 103 are cut differently, 1.23 times as fast on average; three of them are 3 - 4 %
    // slower and one 10 %.  (By itself the fine estimate slows 7 % of the fitted shapes, by up to 25 %.)  H16, 512 queries, 4 096
    // keys 27.7 -> 21.4 us; H32, 128 queries, 2 048 keys 16.0 -> 12.2; H24 T525 without a mask, with dropout 19.3 -> 16.2.
    const bool may_split = Tk > 4096 || Tk >= 2 * (long long)Tq;
    // Where eight key tiles or fewer may be split, 2 us are at stake between the cuts, and the coarse estimate stays alone.  (The
    // tests of every cut use such shapes: they hold on to the cuts that it gives.)
    const bool refine = !may_split || Tk > 8 * TILE;
    const int n_kvtiles = (Tk + TILE - 1) / TILE;
    // CTAs take over further items where the grid is larger than the device and items are short: what overlaps at their ends is
    // then more than the bookkeeping costs per step (about 2 %, of which some may be registers: the kernels that take over spill
    // 76 to 160 bytes per thread, those for one item none).  (With a dense mask the latter spill 172 bytes and are the faster for it:
    // in another schedule of the same code with 88, H36 T512 took 87.1 instead of 62.5 us, H8 T4096 815 instead of 548.)
    // Steps per item on average, one item per CTA -> taken over: 1.5 (H384 T256) 26.9 -> 23.9 us, 5 (H96 T1024) 41.3 -> 39.8, 9 (H96 T2048) 128 -> 124.5, 16 (the same
    // without a mask) 224 -> 225, 17 (H48 T4096) 206 -> 208, 33 (H32 T8192) 494 -> 505.
    // Every block sees a key then (q_pos0 >= k_pos0 under the mask): the hand-over between the streams, the issuing and the
    // storing warp counts on a product in every item.
    const bool sees_keys = !causal || q_pos0 >= k_pos0;
    auto taken_over = [&](int nb, double mean_steps) { return (long long)nb * BH > slots[0] && mean_steps <= 12.0 && sees_keys; };
    FwdPlan plan{}, fine_plan{};
    double coarse_cost = 0, cost_of_plan = 0, fine_cost = 0;  // cost_of_plan: of the coarse one's cut, by the fine one
    for (int mode = FWD_ROWS; mode <= (may_split ? FWD_KEYS : FWD_ROW); ++mode) {
        const int rows = mode == FWD_ROWS ? 2 * TILE : TILE;
        const int nb = (Tq + rows - 1) / rows;
        // steps of one (batch, head) slice, of its longest block, of its last, of the shortest of the others
        double sum = 0, longest = 0, last_block = 0, shortest = 1e30;
        const int sampled = std::min(nb, 64);  // the work per block is linear in its position: long sequences are sampled
        for (int i = 0; i < sampled; ++i) {
            const long long blk = sampled == nb ? i : (long long)i * (nb - 1) / (sampled - 1);
            const int last = (int)(std::min<long long>(Tq, (blk + 1) * rows) - 1);  // its tile sees the most keys of the block
            const int tiles = fwd::kv_tiles_for(last / TILE * TILE, Tq, Tk, causal, q_pos0, k_pos0);
            if (i > 0) shortest = std::min(shortest, last_block);
            last_block = mode == FWD_KEYS ? 0.5 * tiles : tiles;
            sum += last_block;
            longest = std::max(longest, last_block);
        }
        sum *= (double)nb / sampled;
        // in rows mode the last block may be of a single row tile: its steps are those of row mode
        const bool single = mode == FWD_ROWS && (Tq + TILE - 1) / TILE % 2 == 1;
        for (int i = 0; i < (may_split ? 4 : 1); ++i) {
            const int ns = 1 << i;
            const FwdPlan cut = {mode, ns, nb, mode == FWD_KEYS || ns > 1 ? COMBINE_ITEM : taken_over(nb, sum / nb) ? TAKE_OVER : ONE_ITEM};
            double fine = 1e30;
            if (refine && (mode != FWD_KEYS || n_kvtiles >= 2 * ns)) {
                // A CTA, adding up a cluster, a step (with dropout), how much longer a step is on a full device; a key tile's
                // share of the L2's bandwidth (keys mode loads two per step) and, once per slice, of the memory's.  All in us.
                static const double CTA[3] = {3.7, 3.4, 3.9}, CLUSTER[3] = {5.3, 2.4, 2.3}, BUSY[3] = {0.07, 0.04, 0.16};
                static const double STEP[2][3] = {{1.5, 1.3, 1.7}, {3.0, 2.5, 2.9}};
                const double L2_TILE = 0.007, HBM_TILE = 0.0024, TAKING_OVER = 0.6;
                const double n = (double)BH * nb, busy = std::min(1.0, n / slots[i]), waves = std::ceil(n / slots[i]);
                const double fixed = CTA[mode] + (i ? CLUSTER[mode] : 0.0);
                const double step = STEP[drop][mode] * (1.0 + BUSY[mode] * busy);
                const double last_step = single ? STEP[drop][FWD_ROW] * (1.0 + BUSY[FWD_ROW] * busy) : step;
                const double loads = BH * (L2_TILE * sum * (mode == FWD_KEYS ? 2 : 1) + HBM_TILE * n_kvtiles);
                fine = fixed + std::max(loads, (nb == 1 ? last_step : step) * std::ceil(longest / ns));
                if (waves > 1) {  // longest first: about a third of the shortest CTA is left over
                    const double least = fixed + std::min(nb == 1 ? 1e30 : step * std::ceil(shortest / ns), last_step * std::ceil(last_block / ns));
                    const double mean = (n * fixed + BH * (step * (sum - last_block) + last_step * last_block) / ns) / slots[i];
                    fine = std::max(fine, std::max(mean + 0.3 * least, waves * least));
                    if (mode != FWD_KEYS && i == 0) fine += TAKING_OVER;
                }
                if (fine_plan.n_splits == 0 || fine < fine_cost) {
                    fine_cost = fine;
                    fine_plan = cut;
                }
            }
            const double fixed = 3.5 + (mode == FWD_KEYS ? 2.0 : 0.0) + (i ? 3.0 : 0.0);
            const double step = mode == FWD_ROWS ? 2.1 : mode == FWD_ROW ? 1.5 : 2.3;
            const double one = fixed + step * std::ceil(longest / ns);
            const double mean = BH * (nb * fixed + step * sum / ns) / slots[i];
            const double cost = std::max(one, mean + 0.5 * one);
            if ((mode == FWD_ROWS && i == 0) || cost < 0.95 * coarse_cost) {
                coarse_cost = cost;
                cost_of_plan = fine;
                plan = cut;
            }
        }
    }
    return refine && fine_cost < (may_split ? 0.85 : 0.87) * cost_of_plan ? fine_plan : plan;
}

// Runs save loads from memory, and what they cost is the balance at the end of the grid: where a causal mask makes blocks of very
// different lengths, the short ones of the last run alone even it out less than those of all slices.  us, one run -> several, at
// 2, 3.2 and 4.3 times the slices of a run: T512 37.7 -> 39.1, 55.4 -> 55.9, 70.4 -> 71.0; T768 3.2 times 63.3 -> 64.5, 4.3 times 82.6 ->
// 82.0; T1024 48.4 -> 51.4, 71.2 -> 72.7, 95.1 -> 93.0.  Of more than four blocks they pay earlier, at 2.6, 2.9, 3.5 and 3.8 times: T1100
// 73.7 -> 72.1, 80.4 -> 79.4, 95.6 -> 93.6, 101.8 -> 100.4; T1536 75.0 -> 77.7, 83.5 -> 84.5, 100.1 -> 98.9, 107.9 -> 106.2; T2048 90.7 ->
// 93.0, 100.6 -> 100.8, 121.5 -> 119.4, 132.5 -> 128.1.  Without a causal mask, at 2, 3.2 and 4.3 times, T512 47.4 -> 46.4, 67.7 -> 65.7,
// 86.3 -> 84.0; T1024 73.2 -> 73.1, 109.7 -> 106.4, 145.9 -> 137.3; T2048 129.0 -> 130.0, 195.5 -> 190.0, 268.9 -> 249.5; with one,
// but keys in front of the queries, 512 of 2 048 at 2.5 times 62.8 -> 60.9, 1 024 of 1 400 at 2.3 and 3.1 times 69.4 -> 65.8, 90.0 ->
// 87.7.  Blocks that are alone in their slice come in one order either way, and the kernels without runs take less to decode
// them: T256 45.7 -> 47.2.
// A dense mask goes through the L2 as well, and its kernels for runs are the faster ones whatever the order: T512 301 -> 287,
// T1024 514 -> 455, T2048 984 -> 869 at twice the slices, blocks alone in their slice (T256) 260 -> 247.
int fwd_run(const FwdPlan& plan, int BH, int Tq, int Tk, int causal, int q_pos0, int k_pos0, int dropout_mode) {
    const int group = slices_in_l2(BH, 256.0 * (2.0 * Tq + 2.0 * Tk));  // Q, O; K, V
    if (plan.job == COMBINE_ITEM) return BH;
    const bool uneven = causal && q_pos0 <= k_pos0;
    const int least = !uneven ? 2 : plan.n_qblocks <= 4 ? 4 : 3;  // in runs
    if (dropout_mode != 1 && (plan.n_qblocks == 1 || BH < least * (long long)group)) return BH;
    return group;
}

int launch_attn_fwd(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mo,
                    FwdArgs a, cudaStream_t stream) {
    FwdDevice* d = nullptr;
    const int device_rc = fwd_device(&d);
    if (device_rc != HK_OK) return device_rc;
    const FwdPlan plan = plan_attn_fwd(a.BH, a.Tq, a.Tk, a.causal, a.q_pos0, a.k_pos0, a.dropout_mode != 0, d->slots);
    a.mode = plan.mode;
    a.n_splits = plan.n_splits;
    a.n_qblocks = plan.n_qblocks;
    a.group = fwd_run(plan, a.BH, a.Tq, a.Tk, a.causal, a.q_pos0, a.k_pos0, a.dropout_mode);
    const long long nblocks = (long long)a.n_qblocks * a.BH * a.n_splits;
    if (nblocks <= 0 || nblocks > 0x7fffffffLL) return HK_ERR_BAD_SHAPE;
    timing_mark(TIMED_FWD, true, stream);
    LaunchConfig lc((unsigned)nblocks, fwd::NUM_THREADS, fwd::SMEM_BYTES, stream, a.n_splits, true);
    const bool runs = a.group < a.BH;
    const cudaError_t rc = cudaLaunchKernelEx(&lc.cfg, fwd_kernels[a.dropout_mode + 3 * plan.job + (runs ? 9 : 0)], mq, mk, mv, mo, a);
    timing_mark(TIMED_FWD, false, stream);
    count_launch();
    return rc == cudaSuccess ? HK_OK : check_launch();
}

}  // namespace hk

// Parallax training backward on the Blackwell tensor cores (tcgen05.mma, TMEM
// accumulators, TMA-staged tiles): one kernel template, two modes.
//
//   DQR: CTA = 128 query rows of one (batch, q head); streams key tiles of 64.
//        S1 = Q K^T, S2 = R K^T, A = dO V^T  ->  gl, gu  ->  dQ += gl K, dR += gu K
//   DKV: CTA = 128 keys of one (batch, kv head); streams 64-row tiles of q, r, dO
//        (and their row statistics) of every q head of the group.
//        S1^T = K Q^T, S2^T = K R^T, A^T = V dO^T  ->  gl^T, gu^T, W^T
//        ->  dK += gl^T Q + gu^T R, dV += W^T dO   (the tile holds -W^T, the accumulator -dV until it is written)
//
// Formulas (parallax/triton/parallax_train.py:561-573 and :765-792 of the reference):
//   w = 2^(S1*c2 - m), p = w / d1, delta = A - b, cs = bart - S2
//   gl = p (A - t + cs delta), gu = -p delta, W = p (1 + cs); dQ and the gl part of dK carry qk_scale.
// Evaluated as W = p (1 + bart - S2), gl = W delta + p (b - t) with 1/d1 folded into the exponent.
//
// The kernel is persistent: at most one CTA per SM, each walking its share of the work items.
// Pipeline per CTA (12 warps):
//   warp 0      TMA producer (resident tiles once per item, streamed tiles through an NS-deep ring)
//   warp 1      TMEM allocation + the lane that issues the score products
//   warp 2      the lane that issues the output products
//   warp 3      dk/dv: the row statistics of the streamed tiles
//   warps 4-11  element-wise: warp 4 + w works on TMEM lane quarter w % 4.  At head_dim 128 on column
//               group w / 4 (32 of the 64 streamed columns, one row per thread): a thread reads its columns of the three
//               score tiles from TMEM, releases them at once (so the next tile's scores are computed while it works),
//               writes gl / gu / -W as 16-bit values into shared memory in the 128-byte-swizzled K-major
//               layout, and the MMA lane consumes them as the A operand of the output products.  (At 64: see Plan.)
//               The arithmetic of a tile is ONE basic block (tiles that need a mask run a second copy
//               of the loop): measured with every MMA removed, the element-wise chain (TMEM load ->
//               arithmetic -> shared-memory store -> hand-over), not the tensor pipe, sets the pace,
//               and the independent column pairs of a thread must be free to interleave.
//
// TMEM columns at head_dim 128: acc0 [0,128) (dQ | dK), acc1 [128,256) (dR | dV), S1 [256,320), S2 [320,384), A [384,448),
// and at [448,512) the M-side tile that is the A operand of score products: k in DKV mode (S1^T, S2^T), dO in DQR mode (A).
// At 64: acc0 [0,64), acc1 [64,128), the two score buffers at 128 and 320.
#include <cuda.h>

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "plx_common.cuh"
#include "plx_launch.h"
#include "plx_sm100.cuh"
#include "plx_tma_host.h"

namespace plx {

using namespace sm100;

namespace {

constexpr int kModeDQR = 0, kModeDKV = 1;
constexpr int kEwWarps = 8;                    // element-wise warps per CTA: two per lane quarter of tensor memory
constexpr int kBM = 128, kBN = 64;
constexpr uint32_t kResPanel = kBM * 128;      // one 64-channel panel of a resident tile: [128][128 B]
constexpr uint32_t kStrPanel = kBN * 128;      // one 64-channel panel of a streamed tile: [64][128 B]
constexpr uint32_t kGBytes = kBM * kBN * 2;    // 16 KB gl / gu / W tile: [128][128 B]
constexpr uint32_t kTmemCols = 512;

template <typename T>
struct Fmt;
template <>
struct Fmt<__nv_bfloat16> {
    static constexpr int kUmma = 1;
    static constexpr CUtensorMapDataType kTma = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
};
template <>
struct Fmt<__half> {
    static constexpr int kUmma = 0;
    static constexpr CUtensorMapDataType kTma = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
};

constexpr uint32_t kStatBytes = kBN * 16;      // four planes of 64 floats: -mL, -(1 + bart), b, (b - t) * scale

// How a kernel is laid out, by head_dim.
//
// 128: the accumulators take half of the tensor memory, which leaves room for one score buffer {S1, S2, A} and for the
// M-side tile that is the A operand of two (DKV: k) or one (DQR: dO) of the score products (kMTile); that frees the
// shared memory for another stage of streamed tiles.  All element-wise warps work on every tile, 32 columns per thread,
// and leave gl / gu / -W as 16-bit tiles in shared memory.
//
// 64 (kTwo): two score buffers, and two groups of four element-wise warps that take the streamed tiles in turn, so that
// one group's arithmetic runs under the waits and the hand-overs of the other.  gl / gu / -W go IN PLACE over the scores they
// came from (16-bit pairs, the first 32 of 64 columns), as A operands from tensor memory: a buffer is free for the
// scores of tile g + 2 when the output products of tile g have completed.
// Bound by the latency of the element-wise warps, two per scheduler.  B=8, H=16, L=4096, fp16, us: dk/dv 1330 -> 1066,
// dq/dr 875 -> 755.  Two groups alone, with the tiles in shared memory: 1354 and 750, and 32768 tokens in sequences of 1 to
// 256 dq/dr 205 against 191 (before 223).  Two groups at 128 (one score buffer, S1 and S2 of a whole tile read at once into
// 224 registers a thread) changed nothing, 1498 -> 1494: a tile then lives 7700 clocks and the ring has three stages;
// short sequences were slower (dk/dv 239 -> 260).
//
// SHORT (dq/dr at 128): dO is a resident tile in shared memory like q and r, which costs a stage of the ring.  On the way into
// tensor memory it passes through the registers of the element-wise warps at the start of an item, 2500 of the 11300 clocks
// that an item of 2.3 streamed tiles took.  See short_items.
template <int D, int MODE, bool SHORT>
struct Plan {
    static constexpr bool kTwo = D == 64, kMTile = D == 128 && !SHORT;
    static constexpr int kGroups = kTwo ? 2 : 1;                            // of element-wise warps, = score buffers
    static constexpr int kStatStages = kTwo ? 4 : 2;                        // tiles' row statistics (DKV): what is left at head_dim 128
    // stages of streamed tiles: what the shared memory allows at 128; six at 64 (four: dq/dr 4 %, dk/dv 1 % slower, measured
    // before the two groups)
    static constexpr int NS = kTwo ? 6 : MODE == kModeDQR && !SHORT ? 4 : 3;
};

// D = head dim (64 or 128): tiles are D / 64 panels.
template <int D, int MODE, bool SHORT>
struct Smem {
    using P = Plan<D, MODE, SHORT>;
    static constexpr int NS = P::NS, kStatStages = P::kStatStages;
    static constexpr int kPanels = D / 64;
    static constexpr uint32_t kResBytes = kPanels * kResPanel;   // resident tile (128 rows)
    static constexpr uint32_t kStrBytes = kPanels * kStrPanel;   // streamed tile (64 rows)
    static constexpr int kNRes = (MODE == kModeDQR ? 2 : 1) + (P::kMTile ? 0 : 1);   // DQR: q, r (, dO); DKV: v (, k)
    static constexpr int kNStr = MODE == kModeDQR ? 2 : 3;
    static constexpr int kNG = P::kTwo ? 0 : MODE == kModeDQR ? 2 : 3;
    static constexpr uint32_t kRes = 0;
    static constexpr uint32_t kStr = kNRes * kResBytes;
    // A stage.  DQR: k, v.  DKV: the panels of q and r in turn (q0 r0 q1 r1: a panel pair is the B operand of ONE score
    // product of 128 columns, 64 rows of q beside 64 of r), then dO.
    static constexpr uint32_t kStage = kNStr * kStrBytes;
    static constexpr uint32_t kG = kStr + NS * kStage;
    static constexpr uint32_t kStats = kG + kNG * kGBytes;
    static constexpr uint32_t kBars = kStats + (MODE == kModeDKV ? kStatStages * kStatBytes : 0);
    // per streamed tile: NFull / NEmpty (ring), SFull / SFree (score columns), GFull / GFree (G tiles), the latter four in
    // pairs for even and odd tiles where two groups take them in turn (a group waits for every second tile, so a phase has to
    // be as long as two), StatFull / StatEmpty (DKV); per work item: XFull / XEmpty (resident tiles), KReady (M-side tile in tensor memory),
    // AccDone / AccFree
    static constexpr int kXFull = 0, kXEmpty = 1, kNFull = 2, kNEmpty = 2 + NS, kSFull = 2 + 2 * NS, kSFree = kSFull + 2,
                         kGFull = kSFull + 4, kGFree = kSFull + 6, kAccDone = kSFull + 8, kAccFree = kSFull + 9,
                         kKReady = kSFull + 10, kStatFull = kSFull + 11, kStatEmpty = kStatFull + kStatStages,
                         kItemFull = kStatEmpty + kStatStages, kItemEmpty = kItemFull + kItemSlots,
                         kClcFull = kItemEmpty + kItemSlots, kNumBars = kClcFull + 1;
    static constexpr uint32_t kItems = (kBars + 8 * kNumBars + 15u) & ~15u;      // item ring, then the launch-control answer
    static constexpr uint32_t kClc = kItems + 4 * kItemWords * kItemSlots;
    static constexpr uint32_t kTmemSlot = kClc + 16;
    static constexpr uint32_t kAbort = kTmemSlot + 8;
    static constexpr uint32_t kBytes = kTmemSlot + 16;   // the dynamic shared memory must start 1024-byte aligned
    static_assert(kBytes <= 227 * 1024, "more than a CTA may have");
    static constexpr uint32_t kStageTx = kStage;
};

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// One unit of work: 128 query rows of one (batch, q head) (DQR) or 128 keys of one (batch, kv head) (DKV),
// and the range of 64-wide tiles of the other side that it streams.
struct Item {
    int bos, nq, nk, m0, b, hy, hk, off, t_lo, n_t, n_iter;   // streamed tiles t_lo .. t_lo + n_t - 1, per q head
    int valid;
};

// Work item `idx` of the launch.  Items are (batch, head)-major, so that CTAs running at the same time
// share their streamed tiles in L2; inside a (batch, head) the 128-wide tiles alternate last, first,
// last - 1, second, ...: under the causal mask any two neighbours add up to the same work.
// With one item per CTA, and handed out by the hardware (group > 0), the longest items come first instead (see
// longest_first): the CTAs of dq/dr take over the SMs that dk/dv leaves one by one.
template <bool DQR>
__device__ __forceinline__ Item get_item(const TrainArgs &a, int idx, int n_mt, int group) {
    Item it;
    int bh = idx / n_mt, k = idx % n_mt;
    int tile_id = (k & 1) ? (k >> 1) : n_mt - 1 - (k >> 1);
    if (group > 0) {
        longest_first(idx, n_mt, a.batch * (DQR ? a.heads_q : a.heads_kv), group, bh, k);
        tile_id = DQR ? n_mt - 1 - k : k;
    }
    Seq s;
    int tis = 0;
    it.valid = locate_tile(a, tile_id, kBM, s, tis);
    it.bos = s.bos;
    it.nq = s.nq;
    it.nk = s.nk;
    it.m0 = tis * kBM;
    if (it.valid && it.m0 >= (DQR ? it.nq : it.nk)) it.valid = false;
    const int heads_y = DQR ? a.heads_q : a.heads_kv;
    it.b = bh / heads_y;
    it.hy = bh % heads_y;
    it.hk = DQR ? it.hy / a.n_rep : it.hy;
    it.off = it.nk - it.nq;
    int n_t = 0;
    if (DQR) {
        // keys [lo_col, hi_col) are visible to some row of the tile (a sliding window drops whole key tiles)
        const int hi_col = min(it.nk, it.m0 + kBM + it.off);
        const int lo_col = a.window < 0 ? 0 : max(0, it.m0 + it.off - a.window + 1);
        it.t_lo = lo_col / kBN;
        n_t = hi_col > lo_col ? (hi_col + kBN - 1) / kBN - it.t_lo : 0;
    } else {
        // rows [i_lo, i_hi) see some key of the tile: key m is seen by rows m - off .. m - off + window - 1
        const int i_lo = max(0, it.m0 - it.off);
        const int i_hi = a.window < 0 ? it.nq : min(it.nq, it.m0 + kBM - 1 - it.off + a.window);
        it.t_lo = i_lo / kBN;
        n_t = i_hi > i_lo ? (i_hi + kBN - 1) / kBN - it.t_lo : 0;
    }
    it.n_t = it.valid ? n_t : 0;
    it.n_iter = DQR ? it.n_t : it.n_t * a.n_rep;
    return it;
}

// n-th item of this CTA: CTAs take chunks of 2^chunk_shift neighbouring items, round robin.  (chunk_shift < 0: the
// hardware hands the items out one by one.)
__device__ __forceinline__ int item_index(int n, int chunk_shift) {
    return ((blockIdx.x + gridDim.x * (n >> chunk_shift)) << chunk_shift) + (n & ((1 << chunk_shift) - 1));
}

// Persistent kernel: gridDim.x CTAs (at most one per SM) walk the item list.  The streamed-tile pipeline
// (TMA ring -> score products -> element-wise -> G tiles -> output products) runs as ONE sequence of
// tiles across items; what an item adds is its resident tiles, its M-side tile in tensor memory and its
// accumulators, and the hand-overs for those are arranged so that the loads, the tensor-memory tile and
// the first score products of the next item are under way while the element-wise warps write out the
// accumulators of the current one.  TMEM allocation, barrier set-up and launch latency are paid once.
template <typename T, int D, int MODE, bool SHORT>
__global__ void __launch_bounds__((4 + kEwWarps) * 32, 1)
bwd_sm100_kernel(const TrainArgs a, int n_tok, const __grid_constant__ CUtensorMap tm_q,
                 const __grid_constant__ CUtensorMap tm_r, const __grid_constant__ CUtensorMap tm_go,
                 const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const ErrSink sink,
                 int n_mt, int n_items, int chunk_shift, int group) {
    using P = Plan<D, MODE, SHORT>;
    using L = Smem<D, MODE, SHORT>;
    constexpr int NS = P::NS, kStatStages = P::kStatStages;
    constexpr bool DQR = MODE == kModeDQR, kMTile = P::kMTile;
    constexpr uint32_t kResBytes = L::kResBytes, kStrBytes = L::kStrBytes;
    constexpr int GR = P::kGroups, CH = 32;      // columns of a tile that a thread holds at once
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const uint32_t base = smem_u32(smem_raw);
    auto res = [&](int i) -> uint32_t { return base + L::kRes + i * kResBytes; };
    // streamed tile i of stage s (see Smem)
    auto str = [&](int s, int i) -> uint32_t { return base + L::kStr + s * L::kStage + (DQR || i == 2 ? i * kStrBytes : i * kStrPanel); };
    auto str_panel = [](int i) -> uint32_t { return DQR || i == 2 ? kStrPanel : 2 * kStrPanel; };   // distance of its panels
    auto gt = [&](int i) -> uint32_t { return base + L::kG + i * kGBytes; };
    auto bar = [&](int i) -> uint32_t { return base + L::kBars + 8u * i; };
    // barrier and phase of tile g where there is one per group
    auto tile_bar = [&](int i, int g) -> uint32_t { return bar(i + (GR == 2 ? g & 1 : 0)); };
    auto tile_phase = [](int g) -> uint32_t { return (GR == 2 ? g >> 1 : g) & 1; };
    const uint32_t tmem_slot = base + L::kTmemSlot;
    const WaitCtx err{sink, base + L::kAbort};

    if (threadIdx.x == 0) {
        asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(err.abort_flag), "r"(0u) : "memory");
        for (int i = 0; i < L::kNumBars; ++i) {
            // arrivals from the element-wise threads: of the tile's group, or all
            const bool group_ew = i == L::kSFree || i == L::kSFree + 1 || i == L::kGFull || i == L::kGFull + 1 ||
                                  (i >= L::kStatEmpty && i < L::kStatEmpty + kStatStages);
            const bool stat_full = i >= L::kStatFull && i < L::kStatFull + kStatStages;      // from the statistics warp
            const bool all_ew = i == L::kKReady || i == L::kAccFree;
            // every role that reads the items: two MMA issuers, the element-wise warps and (DKV) the statistics warp
            const bool item_empty = i >= L::kItemEmpty && i < L::kItemEmpty + kItemSlots;
            mbar_init(bar(i), group_ew ? 32 * kEwWarps / GR : all_ew ? 32 * kEwWarps : stat_full ? 32 : item_empty ? 2 + kEwWarps + (DQR ? 0 : 1) : 1);
        }
        fence_barrier_init();
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_r);
        prefetch_tensormap(&tm_go);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
        if ((base & 1023u) != 0) cta_abort(err, (12 << 8) | kErrWaitTimeout);   // the swizzled tiles need a 1024-byte aligned base
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
    const uint32_t tAcc0 = tmem_base, tAcc1 = tmem_base + D;
    auto tS = [&](int sb) -> uint32_t { return tmem_base + 2 * D + 192 * sb; };       // S1, S2, A at + 0 / 64 / 128
    const uint32_t tK = tmem_base + 448;                                              // kMTile: the M-side tile as an A operand
    const bool misaligned = cta_aborted(err);
    // Set-up may run under the end of the kernel before.  dk/dv waits here for the row statistics, then lets dq/dr
    // start; dq/dr waits for dk/dv at its end, so that whatever follows on the stream follows both.
    // What dq/dr reads of the statistics it reads without a wait of its own: they were complete and visible to dk/dv
    // (its wait), dk/dv passes them on (fence) before any CTA of dq/dr can exist, and dq/dr takes them up (fence).  For
    // both kernels the statistics are written while the kernel may already be resident, so they are read at the
    // L2 (ld.global.cg), never by the non-coherent path or from a line of L1.
    if (!DQR) {
        grid_wait();
        __threadfence();
        launch_dependents();
    } else {
        __threadfence();
    }

    // Items: the producer finds them (`valid` = 0: no more) ...
    const ItemRing ring{base + L::kItems, bar(L::kItemFull), bar(L::kItemEmpty)};
    struct Source {
        int taken, asked;
    };
    auto find_item = [&](Source &src, Item &it) -> bool {
        for (;;) {
            int idx = -1;
            if (chunk_shift >= 0) {
                idx = item_index(src.taken, chunk_shift);
                if (idx >= n_items) idx = -1;
            } else if (src.taken == 0) {
                idx = blockIdx.x;
            } else {
                if (!mbar_wait(bar(L::kClcFull), (src.taken - 1) & 1, err, 19)) return false;
                idx = clc_answer(base + L::kClc);
            }
            ++src.taken;
            if (idx < 0) {
                it.valid = 0;
                return true;
            }
            if (chunk_shift < 0) {
                clc_ask(base + L::kClc, bar(L::kClcFull));
                src.asked = src.taken;
            }
            it = get_item<DQR>(a, idx, n_mt, group);
            if (it.valid) return true;
        }
    };
    // ... and lets no answer of the hardware arrive in shared memory that is no longer its own
    auto leave_source = [&](const Source &src) {
        if (src.asked == src.taken && src.asked > 0) mbar_wait_quiet(bar(L::kClcFull), (src.asked - 1) & 1);
    };

    if (misaligned) {
        // nothing was started: fall through to the common exit
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int g = 0, n = 0, s = 0;      // streamed tiles and items so far, ring stage of tile g
            uint32_t ph = 0;              // phase of the ring
            bool ok = true;
            int x_issued = 0;             // resident-tile loads started
            Source src{0, 0};
            for (int i = 0; ok; ++i) {
                Item it;
                ok = find_item(src, it) && ring.publish(i, it, err, 20);
                if (!ok || !it.valid) break;
                if (it.n_iter == 0) continue;
                // short items: what they wait for is the first touch of their own tiles, so have those on the way into
                // L2 while the tiles of the item before still occupy the shared (and tensor) memory
                if (chunk_shift < 0 && n > 0)
                    for (int pn = 0; pn < L::kPanels; ++pn) {
                        if (DQR) {
                            tma_prefetch_4d(&tm_q, 64 * pn, it.bos + it.m0, it.hy, it.b);
                            tma_prefetch_4d(&tm_r, 64 * pn, it.bos + it.m0, it.hy, it.b);
                            tma_prefetch_4d(&tm_go, 64 * pn, it.bos + it.m0, it.hy, it.b);
                        } else {
                            tma_prefetch_4d(&tm_k, 64 * pn, it.bos + it.m0, it.hk, it.b);
                            tma_prefetch_4d(&tm_v, 64 * pn, it.bos + it.m0, it.hk, it.b);
                        }
                    }
                // the resident tiles of the previous item are free once its last score product has completed
                if (n > 0) {
                    ok = mbar_wait(bar(L::kXEmpty), (n - 1) & 1, err, 1);
                    if (!ok) break;
                }
                mbar_expect_tx(bar(L::kXFull), L::kNRes * kResBytes);
                ++x_issued;
                if (DQR) {
                    const CUtensorMap *maps[3] = {&tm_q, &tm_r, &tm_go};
                    for (int j = 0; j < L::kNRes; ++j)
                        for (int pn = 0; pn < L::kPanels; ++pn)
                            tma_load_4d(res(j) + pn * kResPanel, maps[j], bar(L::kXFull), 64 * pn, it.bos + it.m0, it.hy, it.b);
                } else {
                    const CUtensorMap *maps[2] = {&tm_v, &tm_k};
                    for (int j = 0; j < L::kNRes; ++j)
                        for (int pn = 0; pn < L::kPanels; ++pn)
                            tma_load_4d(res(j) + pn * kResPanel, maps[j], bar(L::kXFull), 64 * pn, it.bos + it.m0, it.hk, it.b);
                }
                // streamed tile t of the item -> stage s (DQR: k, v of key tile t; DKV: q, r, dO of a 64-row tile of one q head)
                int hq = it.hk * a.n_rep, tt = 0;
                for (int t = 0; t < it.n_iter; ++t, ++g) {
                    if (g >= NS) {
                        ok = mbar_wait(bar(L::kNEmpty + s), ph ^ 1, err, 2);
                        if (!ok) break;
                    }
                    mbar_expect_tx(bar(L::kNFull + s), L::kStageTx);
                    const int row0 = it.bos + (it.t_lo + tt) * kBN;
                    if (DQR) {
                        const CUtensorMap *maps[2] = {&tm_k, &tm_v};
                        for (int j = 0; j < 2; ++j)
                            for (int pn = 0; pn < L::kPanels; ++pn)
                                tma_load_4d(str(s, j) + pn * kStrPanel, maps[j], bar(L::kNFull + s), 64 * pn, row0, it.hk, it.b);
                    } else {
                        const CUtensorMap *maps[3] = {&tm_q, &tm_r, &tm_go};
                        for (int j = 0; j < 3; ++j)
                            for (int pn = 0; pn < L::kPanels; ++pn)
                                tma_load_4d(str(s, j) + pn * str_panel(j), maps[j], bar(L::kNFull + s), 64 * pn, row0, hq, it.b);
                    }
                    if (++tt == it.n_t) {
                        tt = 0;
                        ++hq;
                    }
                    if (++s == NS) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                ++n;
            }
            if (!ok) {
                // unwinding: let the copies already in flight land before the CTA (and its shared memory) goes away
                for (int j = 0; j < min(g, NS); ++j) {
                    if (--s < 0) {
                        s = NS - 1;
                        ph ^= 1;
                    }
                    mbar_wait_quiet(bar(L::kNFull + s), ph);
                }
                if (x_issued > 0) mbar_wait_quiet(bar(L::kXFull), (x_issued - 1) & 1);
                leave_source(src);
            }
        }
    } else if (warp == 1 || warp == 2) {
        // ------------------------------------------------------------------ MMA issuers
        // Two threads in two warps issue the MMAs (warp 1: the score products, warp 2: the output
        // products): one thread's instruction stream, not the tensor pipe, is what bounds a single issuer.
        // The whole warp runs the loop (so that its values stay warp-uniform); one elected lane issues.
        // This path is kept to a few instructions per MMA: descriptor low words are "base + immediate",
        // high words and flags are compile-time constants.
        constexpr uint32_t idesc_s = umma_idesc(Fmt<T>::kUmma, 0, 0, kBM, kBN);
        constexpr uint32_t idesc_s2 = umma_idesc(Fmt<T>::kUmma, 0, 0, kBM, 2 * kBN);
        constexpr uint32_t idesc_o = umma_idesc(Fmt<T>::kUmma, 0, 1, kBM, D);
        constexpr uint32_t hi = umma_desc_hi(1024);
        // DQR: q, r and dO; DKV: v and k (the last of them in tensor memory where kMTile)
        const uint32_t res_lo0 = umma_desc_lo(res(0), 16), res_lo1 = umma_desc_lo(res(kMTile && !DQR ? 0 : 1), 16),
                       res_lo2 = umma_desc_lo(res(DQR && !kMTile ? 2 : 0), 16);
        const uint32_t g_lo0 = umma_desc_lo(gt(0), 16), g_lo1 = umma_desc_lo(gt(1), 16), g_lo2 = umma_desc_lo(gt(DQR ? 1 : 2), 16);
        const uint32_t strk_lo0 = umma_desc_lo(str(0, 0), 16);          // streamed tiles as K-major B (scores)
        const uint32_t strm_lo0 = umma_desc_lo(str(0, 0), str_panel(0));   // streamed tiles as MN-major B (outputs)
        const uint32_t strm_lo2 = umma_desc_lo(str(0, DQR ? 0 : 2), kStrPanel);
        // scores: S1, S2, A into tS + 0 / 64 / 128
        auto issue_scores = [&](int s, int sb) {
            const uint32_t b0 = strk_lo0 + s * (L::kStage >> 4), d = tS(sb);
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                const uint32_t aoff = ((ks >> 2) * kResPanel + (ks & 3) * 32) >> 4;
                const uint32_t boff = ((ks >> 2) * kStrPanel + (ks & 3) * 32) >> 4, qoff = ((ks >> 2) * str_panel(0) + (ks & 3) * 32) >> 4;
                auto products = [&](auto acc) {
                    constexpr bool kAcc = decltype(acc)::value;
                    if (DQR) {     // (Q, K) (R, K) (dO, V)
                        const uint32_t b3 = b0 + (kStrBytes >> 4) + boff;
                        umma_ss_lean<kAcc>(d, res_lo0 + aoff, hi, b0 + boff, hi, idesc_s);
                        umma_ss_lean<kAcc>(d + 64, res_lo1 + aoff, hi, b0 + boff, hi, idesc_s);
                        if (kMTile) umma_ts_lean<kAcc>(d + 128, tK + ks * 8, b3, hi, idesc_s);    // 16 channels = 8 columns per step
                        else umma_ss_lean<kAcc>(d + 128, res_lo2 + aoff, hi, b3, hi, idesc_s);
                    } else {       // (K, Q | R) (V, dO)
                        if (kMTile) umma_ts_lean<kAcc>(d, tK + ks * 8, b0 + qoff, hi, idesc_s2);
                        else umma_ss_lean<kAcc>(d, res_lo1 + aoff, hi, b0 + qoff, hi, idesc_s2);
                        umma_ss_lean<kAcc>(d + 128, res_lo0 + aoff, hi, b0 + 2 * (kStrBytes >> 4) + boff, hi, idesc_s);
                    }
                };
                if (ks == 0) products(std::false_type{});
                else products(std::true_type{});
            }
        };
        // outputs: A = G tile (K-major, 64 wide), B = streamed tile as MN-major [64 rows][128 channels]
        //   DQR: acc0 += G0 K, acc1 += G1 K;   DKV: acc0 += G0 Q + G1 R, acc1 += G2 dO
        auto issue_out = [&](int s, int g, bool first) {
            const uint32_t bq = strm_lo0 + s * (L::kStage >> 4), br = bq + (DQR ? 0 : (kStrPanel >> 4)), bg = strm_lo2 + s * (L::kStage >> 4);
            const uint32_t gtm = tS(g % GR);
            auto product = [&](auto acc, uint32_t d, int i, int kk, uint32_t b) {     // G tile i, rows 16 kk .. 16 kk + 15 of b
                constexpr bool kAcc = decltype(acc)::value;
                if (P::kTwo) umma_ts_lean<kAcc>(d, gtm + 64 * i + 8 * kk, b + kk * (2048 >> 4), hi, idesc_o);
                else umma_ss_lean<kAcc>(d, (i == 0 ? g_lo0 : i == 1 ? g_lo1 : g_lo2) + kk * (32 >> 4), hi, b + kk * (2048 >> 4), hi, idesc_o);
            };
            using yes = std::true_type;
            using no = std::false_type;
            if (first) {
                product(no{}, tAcc0, 0, 0, bq);
                product(no{}, tAcc1, DQR ? 1 : 2, 0, DQR ? br : bg);
            } else {
                product(yes{}, tAcc0, 0, 0, bq);
                product(yes{}, tAcc1, DQR ? 1 : 2, 0, DQR ? br : bg);
            }
            if (!DQR) product(yes{}, tAcc0, 1, 0, br);
#pragma unroll
            for (int kk = 1; kk < kBN / 16; ++kk) {
                product(yes{}, tAcc0, 0, kk, bq);
                product(yes{}, tAcc1, DQR ? 1 : 2, kk, DQR ? br : bg);
                if (!DQR) product(yes{}, tAcc0, 1, kk, br);
            }
        };
        int g = 0, n = 0, s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int i = 0; ok; ++i) {
            Item it;
            ok = ring.read(i, it, true, err, 21);
            if (!ok || !it.valid) break;
            if (it.n_iter == 0) continue;
            if (warp == 1) {
                ok = mbar_wait(bar(L::kXFull), n & 1, err, 4);
                if (kMTile && ok) ok = mbar_wait(bar(L::kKReady), n & 1, err, 14);
                ok = __all_sync(0xffffffffu, ok);
                for (int t = 0; t < it.n_iter && ok; ++t, ++g) {
                    ok = mbar_wait(bar(L::kNFull + s), ph, err, 6);
                    // the score columns are free once the element-wise warps have read the tile before in them, or (G in
                    // place) its output products have completed
                    if (ok && g >= GR) ok = mbar_wait(tile_bar(P::kTwo ? L::kGFree : L::kSFree, g - GR), tile_phase(g - GR), err, 7);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one_sync()) {
                        issue_scores(s, g % GR);
                        umma_commit(tile_bar(L::kSFull, g));
                        if (t == it.n_iter - 1) umma_commit(bar(L::kXEmpty));   // resident tiles and the TMEM tile may be replaced
                    }
                    __syncwarp();
                    if (++s == NS) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            } else {
                for (int t = 0; t < it.n_iter && ok; ++t, ++g) {
                    ok = mbar_wait(tile_bar(L::kGFull, g), tile_phase(g), err, 8);
                    // the first product of an item overwrites the accumulators: the previous item's epilogue must have read them
                    if (ok && t == 0 && n > 0) ok = mbar_wait(bar(L::kAccFree), (n - 1) & 1, err, 13);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one_sync()) {
                        issue_out(s, g, t == 0);
                        umma_commit(tile_bar(L::kGFree, g));
                        umma_commit(bar(L::kNEmpty + s));
                        if (t == it.n_iter - 1) umma_commit(bar(L::kAccDone));
                    }
                    __syncwarp();
                    if (++s == NS) s = 0;
                }
            }
            ++n;
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ row statistics (DKV)
        // The per-row statistics of a streamed tile are per-COLUMN constants of the element-wise warps.  This warp
        // fetches them ({b, mL, 1 + bart, (b - t) * scale}, 16 bytes a row, two rows a lane, a tile ahead) and lays them
        // out in shared memory as four planes of 64 floats (with mL and 1 + bart negated, the latter also times scale), so
        // that a thread reads the constants of adjacent columns as aligned pairs for the packed two-wide arithmetic.
        if constexpr (!DQR) {
            bool ok = true;
            int g = 0;
            for (int i = 0; ok; ++i) {
                Item it;
                ok = ring.read(i, it, true, err, 22);
                if (!ok || !it.valid) break;
                int hq = it.hk * a.n_rep, tt = 0;
                float4 x[2];
                auto fetch = [&]() {
                    const int row0 = it.bos + (it.t_lo + tt) * kBN;
                    const float4 *src = reinterpret_cast<const float4 *>(a.cst) + (static_cast<int64_t>(it.b) * a.heads_q + hq) * n_tok + row0;
                    // (rows past the sequence: those of the next one or of the next head, masked; the records end with 64 spare ones)
                    x[0] = __ldcg(src + lane);
                    x[1] = __ldcg(src + 32 + lane);
                    if (++tt == it.n_t) {
                        tt = 0;
                        ++hq;
                    }
                };
                if (it.n_iter > 0) fetch();
                for (int t = 0; t < it.n_iter; ++t, ++g) {
                    const int st = g % kStatStages;
                    if (g >= kStatStages) {
                        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kStatEmpty + st), (g / kStatStages - 1) & 1, err, 15));
                        if (!ok) break;
                    }
                    float *dst = reinterpret_cast<float *>(smem_raw + L::kStats + st * kStatBytes) + lane;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        dst[32 * h] = -x[h].y;
                        dst[kBN + 32 * h] = -x[h].z * a.scale;
                        dst[2 * kBN + 32 * h] = x[h].x;
                        dst[3 * kBN + 32 * h] = x[h].w;
                    }
                    mbar_arrive(bar(L::kStatFull + st));
                    if (t + 1 < it.n_iter) fetch();
                }
            }
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------------ element-wise + epilogue
        // warp 4 + w: TMEM lane quarter w % 4 (a warp may only touch the lanes of its own quarter); `sel` = w / 4 is its
        // group (GR = 2: the tiles g with g % 2 = sel, GR = 1: columns 32 * sel .. of every tile) and its accumulator
        const int quarter = warp & 3, sel = (warp - 4) >> 2;
        const int ml = quarter * 32 + lane;                 // lane of the M tile: query row (DQR) / key (DKV)
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        const float2 c2v = make_float2(a.c2, a.c2), scale2 = make_float2(a.scale, a.scale);
        bool ok = true;
        int g0 = 0, n = 0, i_next = 0;                      // streamed tiles before this item, items, items looked at

        // With mL = m + log2(d1), c1 = 1 + bart, ct = b - t:
        //   p = 2^(S1*c2 - mL), un = S2 - c1, dn = b - A   =>   W = -p un, gu = p dn, gl = (p un) dn + p ct
        // DQR: the constants of this thread's row
        float r_ml = INFINITY, r_c1 = 0.f, r_ct = 0.f, r_b = 0.f;

        Item cur;
        // next item of this CTA that has tiles to stream; items without any (no visible key / no row
        // that sees the keys) get their zero outputs here
        auto next_item = [&]() -> bool {
            for (;;) {
                ok = ring.read(i_next++, cur, true, err, 21);
                if (!ok || !cur.valid) return false;
                if (cur.n_iter > 0) return true;
                const int row = cur.m0 + ml;
                if (row < (DQR ? cur.nq : cur.nk)) {
                    T *dst = DQR ? static_cast<T *>(sel == 0 ? a.dq : a.dr) + cur.b * a.q_sb + cur.hy * a.q_sh + static_cast<int64_t>(cur.bos + row) * a.q_st
                                 : static_cast<T *>(sel == 0 ? a.dk : a.dv) + cur.b * a.kv_sb + cur.hy * a.kv_sh + static_cast<int64_t>(cur.bos + row) * a.kv_st;
#pragma unroll
                    for (int c = 0; c < D / 8; ++c) *reinterpret_cast<uint4 *>(dst + 8 * c) = make_uint4(0u, 0u, 0u, 0u);
                }
            }
        };
        // Start of an item (nn-th with tiles of this CTA): the row's constants (DQR), and where kMTile the tile of the M side
        // that is the A operand of score products goes to the 64 spare TMEM columns instead of shared memory, where MMA
        // operand reads are the scarce resource: this thread's half of row mg, two 16-bit channels per column.
        auto prologue = [&](int nn) -> bool {
            const int mg = cur.m0 + ml;
            uint32_t kw[D / 4];
            if (kMTile) {
                const T *krow = DQR ? static_cast<const T *>(a.go) + cur.b * a.q_sb + cur.hy * a.q_sh + static_cast<int64_t>(cur.bos + mg) * a.q_st + sel * (D / 2)
                                    : static_cast<const T *>(a.k) + cur.b * a.kv_sb + cur.hk * a.kv_sh + static_cast<int64_t>(cur.bos + mg) * a.kv_st + sel * (D / 2);
#pragma unroll
                for (int c = 0; c < D / 16; ++c) {
                    uint4 x = make_uint4(0u, 0u, 0u, 0u);
                    if (mg < (DQR ? cur.nq : cur.nk)) x = *reinterpret_cast<const uint4 *>(krow + 8 * c);
                    kw[4 * c] = x.x; kw[4 * c + 1] = x.y; kw[4 * c + 2] = x.z; kw[4 * c + 3] = x.w;
                }
            }
            if (DQR) {
                r_ml = INFINITY;
                r_c1 = r_ct = r_b = 0.f;
                if (mg < cur.nq) {
                    const float4 hi4 = __ldcg(reinterpret_cast<const float4 *>(
                        a.cst + ((static_cast<int64_t>(cur.b) * a.heads_q + cur.hy) * n_tok + cur.bos + mg) * 4));   // b, mL, 1 + bart, (b - t) * scale
                    r_b = hi4.x;
                    r_ml = hi4.y;
                    r_c1 = hi4.z;
                    r_ct = hi4.w / a.scale;
                }
            }
            if (kMTile) {
                // the previous item's score products (the readers of the TMEM tile) must have completed
                if (nn > 0 && !__all_sync(0xffffffffu, mbar_wait(bar(L::kXEmpty), (nn - 1) & 1, err, 16))) return false;
                tc_fence_after();
                tmem_st_cols(tK + lane_base + sel * (D / 4), kw);
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(bar(L::kKReady));
            }
            return true;
        };

        bool have = next_item();
        if (have && ok) ok = prologue(0);
        while (have && ok) {
            const int m0 = cur.m0, nq = cur.nq, nk = cur.nk, off = cur.off, mg = m0 + ml;
            for (int it = GR == 2 ? (g0 ^ sel) & 1 : 0; it < cur.n_iter; it += GR) {
                const int g = g0 + it;
                ok = __all_sync(0xffffffffu, mbar_wait(tile_bar(L::kSFull, g), tile_phase(g), err, 9));
                if (!ok) break;
                tc_fence_after();

                const int tile0 = (cur.t_lo + (DQR ? it : it % cur.n_t)) * kBN;   // first streamed index of the tile
                const int win = a.window;
                // tile-uniform: every element of the tile is visible
                const bool full = DQR ? (tile0 + kBN - 1 <= m0 + off && tile0 + kBN <= nk && m0 + kBM <= nq &&
                                         (win < 0 || tile0 >= m0 + kBM + off - win))
                                      : (tile0 >= m0 + kBM - 1 - off && tile0 + kBN <= nq && m0 + kBM <= nk &&
                                         (win < 0 || tile0 + kBN - 1 <= m0 - off + win - 1));
                const float *stats = reinterpret_cast<const float *>(smem_raw + L::kStats + (g % kStatStages) * kStatBytes);
                // One pair of adjacent columns: constants nml = -mL, nc1 = -(1 + bart), bb = b, ct = b - t (DKV: times
                // scale; DKV: nc1 times scale too).  The third tile carries -W * scale = p un scale (DKV
                // only): the dV accumulator is multiplied by -1 / scale when it is written out, which saves a
                // negation and a multiplication per element here.  `masked` is a compile-time tag:
                // tiles that are visible as a whole (all but the ones on the diagonal or at a window edge) run
                // the loop without any mask arithmetic AND as one basic block, so that the independent pairs
                // interleave; a branch per pair would keep them apart.  Else columns lo .. hi are visible.
                auto element_pair = [&](auto masked, int lo, int hi, int col, uint32_t s1a, uint32_t s1b, uint32_t s2a, uint32_t s2b, uint32_t aa,
                                        uint32_t ab, const float2 &nml, const float2 &nc1, const float2 &bb, const float2 &ct, uint32_t &w0,
                                        uint32_t &w1, uint32_t &w2) {
                    const float2 s1 = make_float2(__uint_as_float(s1a), __uint_as_float(s1b));
                    const float2 s2 = make_float2(__uint_as_float(s2a), __uint_as_float(s2b));
                    const float2 av = make_float2(__uint_as_float(aa), __uint_as_float(ab));
                    const float2 arg = __ffma2_rn(s1, c2v, nml);
                    const float2 p = make_float2(fast_exp2(arg.x), fast_exp2(arg.y));
                    // DKV carries qk_scale on gl = (p un scale) dn + p ct scale: nc1 and ct come scaled from the
                    // statistics planes, so wn = -W scale there (1 / scale goes on dV when it is written out)
                    const float2 un = DQR ? __fadd2_rn(s2, nc1) : __ffma2_rn(s2, scale2, nc1);
                    const float2 dn = __ffma2_rn(av, make_float2(-1.f, -1.f), bb);
                    const float2 pc = __fmul2_rn(p, ct);
                    float2 wn = __fmul2_rn(p, un);                            // -W (DKV: times scale)
                    float2 gu = __fmul2_rn(p, dn);
                    float2 gl = __ffma2_rn(wn, dn, pc);
                    if (decltype(masked)::value) {
                        const bool v0 = col >= lo && col <= hi, v1 = col + 1 >= lo && col + 1 <= hi;
                        gl = make_float2(v0 ? gl.x : 0.f, v1 ? gl.y : 0.f);
                        gu = make_float2(v0 ? gu.x : 0.f, v1 ? gu.y : 0.f);
                        wn = make_float2(v0 ? wn.x : 0.f, v1 ? wn.y : 0.f);
                    }
                    w0 = Elem<T>::pack(gl.x, gl.y);
                    w1 = Elem<T>::pack(gu.x, gu.y);
                    if (!DQR) w2 = Elem<T>::pack(wn.x, wn.y);
                };
                auto stats_ready = [&]() -> bool {
                    return __all_sync(0xffffffffu, mbar_wait(bar(L::kStatFull + g % kStatStages), (g / kStatStages) & 1, err, 15));
                };
                const uint32_t tsg = tS(g % GR) + lane_base;
                if constexpr (P::kTwo && !DQR) {
                    // The fragment arrangement: in each half h of the warp's 32 lanes (keys), this thread has the keys
                    // 16 h + lane / 4 and + 8 and the columns 8 k + 2 (lane % 4), + 1 -- so it needs the constants of 16
                    // columns for 32 elements.  (With one key and 32 columns a thread, every thread of a warp reads every constant.)
                    const int gq = lane >> 2, t2 = 2 * (lane & 3);
                    const float *st2 = stats + t2;
                    auto constant = [&](int plane, int k) { return *reinterpret_cast<const float2 *>(st2 + plane * kBN + 8 * k); };
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t at = tsg + (16u * h << 16);
                        uint32_t x1[32], x2[32], x3[32], w0[16], w1[16], w2[16];
                        tmem_ld_16x256b_x8(at, x1);
                        tmem_ld_16x256b_x8(at + 64, x2);
                        tmem_ld_16x256b_x8(at + 128, x3);
                        tmem_wait_ld();
                        if (h == 0) {
                            ok = stats_ready();
                            if (!ok) break;
                        }
                        auto math = [&](auto masked) {
                            int lo[2], hi[2];                  // visible rows of the two keys
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                const int key = m0 + quarter * 32 + 16 * h + 8 * j + gq;
                                lo[j] = max(key - off, 0);
                                hi[j] = key < nk ? (win < 0 ? nq - 1 : min(nq - 1, key - off + win - 1)) : -1;
                            }
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const float2 nml = constant(0, k), nc1 = constant(1, k), bb = constant(2, k), ct = constant(3, k);
#pragma unroll
                                for (int j = 0; j < 2; ++j) {
                                    const int e = 4 * k + 2 * j;
                                    element_pair(masked, lo[j], hi[j], tile0 + 8 * k + t2, x1[e], x1[e + 1], x2[e], x2[e + 1], x3[e], x3[e + 1], nml,
                                                 nc1, bb, ct, w0[2 * k + j], w1[2 * k + j], w2[2 * k + j]);
                                }
                            }
                        };
                        if (full) math(std::false_type{});
                        else math(std::true_type{});
                        tmem_st_16x128b_x8(at, w0);
                        tmem_st_16x128b_x8(at + 64, w1);
                        tmem_st_16x128b_x8(at + 128, w2);
                    }
                    if (!ok) break;
                    mbar_arrive(bar(L::kStatEmpty + g % kStatStages));
                } else {
                    // one row (DQR) or key (DKV) a thread, CH columns at a time
                    const int lo = DQR ? (win < 0 ? INT_MIN : mg + off - win + 1) : max(mg - off, 0);      // visible columns
                    const int hi = DQR ? (mg < nq ? min(mg + off, nk - 1) : -1)
                                       : (mg < nk ? (win < 0 ? nq - 1 : min(nq - 1, mg - off + win - 1)) : -1);
#pragma unroll 1
                    for (int ch = 0; ch < GR; ++ch) {
                        const int col0 = (GR == 2 ? ch : sel) * CH;
                        uint32_t x1[CH], x2[CH], x3[CH], w0[CH / 2], w1[CH / 2], w2[CH / 2];
                        tmem_ld_cols(tsg + col0, x1);
                        tmem_ld_cols(tsg + 64 + col0, x2);
                        tmem_ld_cols(tsg + 128 + col0, x3);
                        tmem_wait_ld();
                        if constexpr (!P::kTwo) {
                            tc_fence_before();
                            mbar_arrive(tile_bar(L::kSFree, g));
                        }
                        if constexpr (!DQR) {
                            ok = stats_ready();
                            if (!ok) break;
                        }
                        auto math = [&](auto masked) {
#pragma unroll
                            for (int c = 0; c < CH; c += 4) {
                                float4 st[4];
                                const float row[4] = {-r_ml, -r_c1, r_b, r_ct};
#pragma unroll
                                for (int i = 0; i < 4; ++i)
                                    st[i] = DQR ? make_float4(row[i], row[i], row[i], row[i]) : *reinterpret_cast<const float4 *>(stats + i * kBN + col0 + c);
#pragma unroll
                                for (int e = c; e < c + 4; e += 2) {
                                    auto half = [&](int i) { return e == c ? make_float2(st[i].x, st[i].y) : make_float2(st[i].z, st[i].w); };
                                    element_pair(masked, lo, hi, tile0 + col0 + e, x1[e], x1[e + 1], x2[e], x2[e + 1], x3[e], x3[e + 1], half(0), half(1),
                                                 half(2), half(3), w0[e / 2], w1[e / 2], w2[e / 2]);
                                }
                            }
                        };
                        if (full) math(std::false_type{});
                        else math(std::true_type{});
                        if constexpr (!DQR) mbar_arrive(bar(L::kStatEmpty + g % kStatStages));
                        if constexpr (P::kTwo) {
                            // (the second half of the columns is still to be read: the first half of G goes over the first)
                            tmem_st_cols(tsg + col0 / 2, w0);
                            tmem_st_cols(tsg + 64 + col0 / 2, w1);
                        } else {
                            // the G tiles are free once the output products of the tile before have completed
                            if (g > 0) {
                                ok = __all_sync(0xffffffffu, mbar_wait(tile_bar(L::kGFree, g - 1), tile_phase(g - 1), err, 10));
                                if (!ok) break;
                            }
                            // row ml of each G tile: 128 bytes, 16-byte chunk i stored at position i ^ (ml & 7)
#pragma unroll
                            for (int c = 0; c < CH / 8; ++c) {
                                const uint32_t o = static_cast<uint32_t>(ml) * 128u + static_cast<uint32_t>(((col0 / 8 + c) ^ (ml & 7)) * 16);
                                st_shared_v4(gt(0) + o, w0[4 * c], w0[4 * c + 1], w0[4 * c + 2], w0[4 * c + 3]);
                                st_shared_v4(gt(1) + o, w1[4 * c], w1[4 * c + 1], w1[4 * c + 2], w1[4 * c + 3]);
                                if (!DQR) st_shared_v4(gt(2) + o, w2[4 * c], w2[4 * c + 1], w2[4 * c + 2], w2[4 * c + 3]);
                            }
                        }
                    }
                    if (!ok) break;
                }
                if constexpr (P::kTwo) {
                    tmem_wait_st();
                    tc_fence_before();
                } else {
                    fence_proxy_async();
                }
                mbar_arrive(tile_bar(L::kGFull, g));
            }
            if (!ok) break;

            // ---- what the epilogue of this item needs, then the start of the next item: its TMEM tile and
            // first score products are under way while the accumulators of this one are written out
            // dQ carries qk_scale; the dV accumulator holds -dV * qk_scale (the W tile is stored as -W * qk_scale)
            g0 += cur.n_iter;
            const float mul = DQR ? (sel == 0 ? a.scale : 1.f) : (sel == 0 ? 1.f : -1.f / a.scale);
            const int rows_left = (DQR ? nq : nk) - m0;
            T *dst0;
            int64_t row_stride;
            if (DQR) {
                dst0 = static_cast<T *>(sel == 0 ? a.dq : a.dr) + cur.b * a.q_sb + cur.hy * a.q_sh + static_cast<int64_t>(cur.bos + m0) * a.q_st;
                row_stride = a.q_st;
            } else {
                dst0 = static_cast<T *>(sel == 0 ? a.dk : a.dv) + cur.b * a.kv_sb + cur.hy * a.kv_sh + static_cast<int64_t>(cur.bos + m0) * a.kv_st;
                row_stride = a.kv_st;
            }
            have = next_item();
            if (have) ok = prologue(n + 1);
            if (!ok) break;

            // epilogue: half of the element-wise warps write acc0 (dQ | dK), the other half acc1 (dR | dV); an
            // accumulator is 2 x D / 64 units of 16 rows x 64 columns per lane quarter.  The accumulators are read in the fragment arrangement (a row is spread
            // over the four lanes of a quad); a 4 x 4 word transpose inside the quad gives every thread 16
            // contiguous bytes, so a warp store covers 64 contiguous bytes of 8 rows.
            ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kAccDone), n & 1, err, 11));
            if (!ok) break;
            tc_fence_after();
            const int gq = lane >> 2, t = lane & 3;
            const uint32_t acc = sel == 0 ? tAcc0 : tAcc1;
            constexpr int kUnits = 2 * (D / 64);
#pragma unroll 1
            for (int u = 0; u < kUnits; ++u) {
                const int rh = u / (D / 64), cc = u % (D / 64);
                const int rl = quarter * 32 + rh * 16 + gq;     // local rows of this thread: rl and rl + 8
                uint32_t x[32];
                tmem_ld_16x256b_x8(acc + (static_cast<uint32_t>(quarter * 32 + rh * 16) << 16) + 64 * cc, x);
                tmem_wait_ld();
                if (u == kUnits - 1) {
                    // this thread's share of the accumulators is in registers: the next item may overwrite them
                    tc_fence_before();
                    mbar_arrive(bar(L::kAccFree));
                }
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                    for (int grp = 0; grp < 2; ++grp) {
                        uint32_t w[4];
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            const int e = 4 * (4 * grp + kk) + 2 * hh;
                            w[kk] = Elem<T>::pack(__uint_as_float(x[e]) * mul, __uint_as_float(x[e + 1]) * mul);
                        }
                        quad_transpose(w, t);
                        const int row = rl + 8 * hh;
                        if (row < rows_left)
                            *reinterpret_cast<uint4 *>(dst0 + static_cast<int64_t>(row) * row_stride + 64 * cc + 32 * grp + 8 * t) =
                                make_uint4(w[0], w[1], w[2], w[3]);
                    }
            }
            ++n;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
    if (DQR) grid_wait();
}

// ------------------------------------------------------------------------- //
// host side
// ------------------------------------------------------------------------- //
template <typename T, int D, int MODE, bool SHORT>
int launch_mode(const TrainArgs &a, int n_tok, const ErrSink &sink, bool overlap, cudaStream_t stream) {
    using L = Smem<D, MODE, SHORT>;
    constexpr bool DQR = MODE == kModeDQR;
    const int q_rows = DQR ? kBM : kBN, kv_rows = DQR ? kBN : kBM;
    CUtensorMap tq, tr, tg, tk, tv;
    const CUtensorMapDataType dt = Fmt<T>::kTma;
    if (!tma::make_map(&tq, dt, a.q, D, a.len_q, a.heads_q, a.batch, a.q_st, a.q_sh, a.q_sb, q_rows) ||
        !tma::make_map(&tr, dt, a.r, D, a.len_q, a.heads_q, a.batch, a.q_st, a.q_sh, a.q_sb, q_rows) ||
        !tma::make_map(&tg, dt, a.go, D, a.len_q, a.heads_q, a.batch, a.q_st, a.q_sh, a.q_sb, q_rows) ||
        !tma::make_map(&tk, dt, a.k, D, a.len_k, a.heads_kv, a.batch, a.kv_st, a.kv_sh, a.kv_sb, kv_rows) ||
        !tma::make_map(&tv, dt, a.v, D, a.len_k, a.heads_kv, a.batch, a.kv_st, a.kv_sh, a.kv_sb, kv_rows))
        return PLX_ERR_LAUNCH;
    auto kern = bwd_sm100_kernel<T, D, MODE, SHORT>;
    static std::mutex attr_mu;
    static bool attr_done[tma::kMaxDevices] = {};
    if (!tma::opt_in_smem(kern, static_cast<int>(L::kBytes), attr_done, attr_mu)) return PLX_ERR_LAUNCH;
    const int len = DQR ? a.len_q : a.len_k;
    const int tiles = a.cu ? (len + kBM - 1) / kBM + a.n_seqs : (len + kBM - 1) / kBM;
    const int n_items = tiles * a.batch * (DQR ? a.heads_q : a.heads_kv), sms = tma::sm_count();
    if (sms <= 0) return PLX_ERR_LAUNCH;
    // with plenty of items a CTA takes them in neighbouring pairs (a heavy and a light tile)
    const bool dynamic = items_by_hardware(n_items, sms, a.cu != nullptr);
    const int chunk_shift = dynamic ? -1 : n_items >= 2 * sms ? 1 : 0;
    const int units = dynamic ? n_items : (n_items + (1 << chunk_shift) - 1) >> chunk_shift;
    const int group = !dynamic && n_items > sms ? 0 : dynamic && a.cu ? 1 : item_group(a.batch * (DQR ? a.heads_q : a.heads_kv), tiles, sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(dynamic || units < sms ? units : sms);
    cfg.blockDim = dim3((4 + kEwWarps) * 32);
    cfg.dynamicSmemBytes = L::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    const cudaError_t st = cudaLaunchKernelEx(&cfg, kern, a, n_tok, tq, tr, tg, tk, tv, sink, tiles, n_items, chunk_shift, group);
    count_launch();
    return st == cudaSuccess && cudaGetLastError() == cudaSuccess ? PLX_OK : PLX_ERR_LAUNCH;
}

// SHORT pays where an item streams few tiles and costs a stage of the ring where it streams many: what counts is the keys that
// the mean item of 128 rows sees, len_k - len_q / 2 + 64 in a dense problem (rows are the last ones of the keys) and at
// most the window and the item's own rows.  Lengths of packed sequences are on the device; for lengths spread evenly from 1 up
// to twice their mean the mean item sees 2 / 3 of the mean and 64.
// dq/dr alone, us, tile in tensor memory against shared memory.  By keys: dense, B=16, H=16, 128 tokens (128 keys) 20.5 / 16.5, 512
// (320) 80.9 / 73.9, 1024 (576) 203 / 193; B=8, 1536 (832) 198.7 / 196.2, 2048 (1088) 325 / 317 to 334; B=4, 2048 165.6 / 166.6;
// 128 rows against 512 keys (512) 43 / 40, 1024 (1024) 58.1 / 57.5, 2048 (2048) 87.9 / 94.4, 4096 (4096) 75.8 / 82.9; 512 against
// 1024 (832) 80.4 / 78.8, 1536 (1344) 114.6 / 116.6, 2048 (1856) 151 / 156; 4096 tokens, window 64 (192) 138 / 111, 256 (384) 167 / 149, 512
// (640) 216 / 211, 768 (896) 274 / 262, 1024 (1152) 326 / 317, 2048 506 / 505.  Packed, 1 to 256 tokens, 16 : 4 heads (149) 324 / 298,
// 256 to 1024 (490) 378 / 374, 256 to 1700 (704) 463 / 463, 15 of 2048 625 / 623, 64 to 8192 2770 / 2786.  A few long sequences among very many
// short ones are on the wrong side of it: one of 16384 and 256 of 64 2445 / 2568, two of 8192 and 200 of 64 1257 / 1272.
bool short_items(const TrainArgs &a) {
    int64_t keys = a.cu ? 2ll * a.len_q / (3ll * a.n_seqs) + kBM / 2 : a.len_k - a.len_q / 2 + std::min(a.len_q, kBM) / 2;
    if (a.window > 0) keys = std::min<int64_t>(keys, a.window + kBM);
    return keys <= 14 * kBN;
}

}  // namespace

bool train_bwd_sm100_supported(const TrainArgs &a, int head_dim) {
    if ((head_dim != 64 && head_dim != 128) || a.window == 0 || !(a.c2 > 0.f)) return false;
    const char *env = std::getenv("PLX_BWD_KERNEL");
    if (env && env[0] == 'm') return false;  // "mma": force the warp-level kernels
    return tma::encode_fn() != nullptr;
}

int launch_train_bwd_sm100(const TrainArgs &a, int dtype, int head_dim, int stage, bool overlap, cudaStream_t stream) {
    const ErrorWords ew = sm100_error_words();
    if (!ew.word) return PLX_ERR_LAUNCH;
    const ErrSink err{ew.word, ew.mirror};
    const int n_tok = a.len_q;
    const bool dqr = stage == PLX_BWD_DQR;
    if (dtype == PLX_BF16) {
        if (head_dim == 64)
            return dqr ? launch_mode<__nv_bfloat16, 64, kModeDQR, false>(a, n_tok, err, overlap, stream)
                       : launch_mode<__nv_bfloat16, 64, kModeDKV, false>(a, n_tok, err, overlap, stream);
        return dqr ? (short_items(a) ? launch_mode<__nv_bfloat16, 128, kModeDQR, true>(a, n_tok, err, overlap, stream)
                                     : launch_mode<__nv_bfloat16, 128, kModeDQR, false>(a, n_tok, err, overlap, stream))
                   : launch_mode<__nv_bfloat16, 128, kModeDKV, false>(a, n_tok, err, overlap, stream);
    }
    if (dtype == PLX_FP16) {
        if (head_dim == 64)
            return dqr ? launch_mode<__half, 64, kModeDQR, false>(a, n_tok, err, overlap, stream)
                       : launch_mode<__half, 64, kModeDKV, false>(a, n_tok, err, overlap, stream);
        return dqr ? (short_items(a) ? launch_mode<__half, 128, kModeDQR, true>(a, n_tok, err, overlap, stream)
                                     : launch_mode<__half, 128, kModeDQR, false>(a, n_tok, err, overlap, stream))
                   : launch_mode<__half, 128, kModeDKV, false>(a, n_tok, err, overlap, stream);
    }
    return PLX_ERR_UNSUPPORTED;
}

}  // namespace plx

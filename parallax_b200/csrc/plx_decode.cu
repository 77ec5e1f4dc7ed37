// Parallax single-token decode: an HBM-bound split-KV sweep over the cache.
//
// (Grouped-query shapes run the tensor-core kernel further down; this is the kernel
// of the one-q-head-per-kv-head case.)
// One warp per (split, q head, batch row); a CTA groups the warps of adjacent q
// heads.  Inside a warp the key range is dealt out to independent "streams" of D/8
// lanes: every lane owns 8 of the D channels and fetches them with one 128-bit
// load per key, so a stream reads a whole K (or V) row per load instruction and a
// warp keeps 32/(D/8) * 8 rows of K and as many of V in flight (two register buffers).  Each stream runs
// its own online softmax (m, d1, d2, O1, O2); streams are merged by shuffles,
// splits by the last warp to arrive (wait-free: an atomic counter, no spinning).
//
// Math: parallax/triton/parallax_decode.py:43-97 (per-key update and final
// out = O1/d1 * (1 + d2/d1) - O2/d1); partial-state merge:
// parallax/cute/parallax_decode.py:1107-1136.
#include <atomic>
#include <mutex>
#include <type_traits>

#include "plx_common.cuh"
#include "plx_decode.h"
#include "plx_launch.h"
#include "plx_sm100.cuh"

namespace plx {

__device__ __forceinline__ uint4 ld_stream16(const void *p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

template <typename T>
__device__ __forceinline__ void unpack8(const uint4 &x, float (&f)[8]) {
    float2 a = Elem<T>::unpack(x.x), b = Elem<T>::unpack(x.y), c = Elem<T>::unpack(x.z), d = Elem<T>::unpack(x.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
    f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}

// Combine `n` partial records (record s at rec0 + s * stride floats; layout
// m, d1, d2, pad, O1[D], O2[D]) for channel `d`.  Returns the merged
// un-normalised state of that channel.
template <int D, bool VOLATILE_READ>
__device__ __forceinline__ void merge_records(const float *rec0, int n, int64_t stride, int d, float &m_out,
                                              float &d1, float &d2, float &o1, float &o2) {
    auto rd = [](const float *p) -> float { return VOLATILE_READ ? __ldcg(p) : *p; };
    float big = -INFINITY;
    for (int s = 0; s < n; ++s) big = fmaxf(big, rd(rec0 + s * stride));
    const float safe = big == -INFINITY ? 0.f : big;
    d1 = d2 = o1 = o2 = 0.f;
    for (int s = 0; s < n; ++s) {
        const float *rec = rec0 + s * stride;
        const float w = fast_exp2(rd(rec) - safe);
        d1 += w * rd(rec + 1);
        d2 += w * rd(rec + 2);
        o1 += w * rd(rec + 4 + d);
        o2 += w * rd(rec + 4 + D + d);
    }
    m_out = big;
}

// thread-block cluster: size and rank along x, the address of a shared-memory word of another CTA of the
// cluster, a store through it, and the cluster-wide barrier
__device__ __forceinline__ uint32_t cluster_size_x() {
    uint32_t v;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;\n" : "=r"(v));
    return v;
}
__device__ __forceinline__ uint32_t cluster_rank_x() {
    uint32_t v;
    asm volatile("mov.u32 %0, %%cluster_ctaid.x;\n" : "=r"(v));
    return v;
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t smem_addr, uint32_t rank) {
    uint32_t v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(v) : "r"(smem_addr), "r"(rank));
    return v;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float x) {
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(addr), "f"(x) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// Paged cache: element offset of key kj of batch row b inside k / v (head and channel offsets not
// included).  Dense caches are addressed by strides directly at the call sites.
__device__ __forceinline__ uint32_t paged_key_page(const DecodeArgs &a, int b, int kj) {
    // page numbers are kept inside the pool: a row length that the caller is yet to find out of range may lead here
    return min(static_cast<uint32_t>(a.page_table[static_cast<int64_t>(b) * a.pages_per_seq + (kj >> a.page_shift)]), a.last_page);
}
__device__ __forceinline__ int64_t paged_key_offset(const DecodeArgs &a, int b, int kj) {
    return static_cast<int64_t>(paged_key_page(a, b, kj)) * a.kv_sb + static_cast<int64_t>(kj & a.page_mask) * a.kv_st;
}

__device__ __forceinline__ float finalize(float d1, float d2, float o1, float o2) {
    const float inv = d1 > 0.f ? 1.f / d1 : 0.f;
    return o1 * inv * (1.f + d2 * inv) - o2 * inv;
}

template <typename T>
__device__ __forceinline__ void store_elem(void *out, int64_t idx, float x);
template <>
__device__ __forceinline__ void store_elem<__nv_bfloat16>(void *out, int64_t idx, float x) {
    static_cast<__nv_bfloat16 *>(out)[idx] = __float2bfloat16_rn(x);
}
template <>
__device__ __forceinline__ void store_elem<__half>(void *out, int64_t idx, float x) {
    static_cast<__half *>(out)[idx] = __float2half_rn(x);
}

// Merge of n <= 32 partial records (stride REC floats) by one warp.  On return every lane holds the
// maximum, the two sums, and the D / 32 channels lane * (D / 32) .. of O1 and O2, all relative to
// the common maximum.  Bound by round trips to the L2: the channels of the first N records are requested together
// with the headers of all.  SKIP: of those that there are (grouped heads: a warp may be the only one of its CTA to merge all rows of
// a kv head, and with N records read for each whatever n, calls of 4 rows of 1000 keys went from 27 to 35 us at 16 : 1 heads, from
// 16.5 to 20.4 at 64 : 8).  Without it where a warp merges one row: there the condition costs more than the reads (25 rows of 14518
// down to 5000 keys, 8 : 8 heads, 166.9 us against 165.7).
template <int D, int N = 8, bool SKIP = false>
__device__ __forceinline__ void warp_merge(const float *rec0, int n, int lane, float &big, float &D1, float &D2,
                                           float (&O1)[D / 32], float (&O2)[D / 32]) {
    constexpr int CH = D / 32, REC = 2 * D + 4;
    float4 h = make_float4(-INFINITY, 0.f, 0.f, 0.f);
    if (lane < n) h = __ldcg(reinterpret_cast<const float4 *>(rec0 + static_cast<int64_t>(lane) * REC));
    const float *col = rec0 + 4 + lane * CH;
    float x[N][CH], y[N][CH];
    auto load = [&](int j0) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (SKIP && j0 + j >= n) {
#pragma unroll
                for (int e = 0; e < CH; ++e) x[j][e] = y[j][e] = 0.f;
                continue;
            }
            const float *pr = col + static_cast<int64_t>(SKIP ? j0 + j : min(j0 + j, n - 1)) * REC;   // weight 0 past the end
            if (CH == 4) {
                const float4 u = __ldcg(reinterpret_cast<const float4 *>(pr)), v = __ldcg(reinterpret_cast<const float4 *>(pr + D));
                x[j][0] = u.x; x[j][1] = u.y; x[j][CH - 2] = u.z; x[j][CH - 1] = u.w;
                y[j][0] = v.x; y[j][1] = v.y; y[j][CH - 2] = v.z; y[j][CH - 1] = v.w;
            } else {
                const float2 u = __ldcg(reinterpret_cast<const float2 *>(pr)), v = __ldcg(reinterpret_cast<const float2 *>(pr + D));
                x[j][0] = u.x; x[j][1] = u.y;
                y[j][0] = v.x; y[j][1] = v.y;
            }
        }
    };
    load(0);
    big = h.x;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, off));
    const float safe = big == -INFINITY ? 0.f : big;
    const float wl = fast_exp2(h.x - safe);   // weight of record `lane` (0 beyond n: m = -inf there)
    D1 = wl * h.y;
    D2 = wl * h.z;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        D1 += __shfl_xor_sync(0xffffffffu, D1, off);
        D2 += __shfl_xor_sync(0xffffffffu, D2, off);
    }
#pragma unroll
    for (int e = 0; e < CH; ++e) O1[e] = O2[e] = 0.f;
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += N) {
        if (j0 >= n) break;
        if (j0 > 0) load(j0);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float w = __shfl_sync(0xffffffffu, wl, j0 + j);
#pragma unroll
            for (int e = 0; e < CH; ++e) {
                O1[e] = fmaf(w, x[j][e], O1[e]);
                O2[e] = fmaf(w, y[j][e], O2[e]);
            }
        }
    }
}

__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t));
    return t;
}

// Inbox layout of the peer-memory exchange (see decode_exchange_merge_kernel below): record slots
// [2 parities][world][n_records], then as many 32-bit stamps, then [n_records] step counters.
struct InboxView {
    int world, n_records, rec;      // rec = floats per record
    __device__ __forceinline__ size_t rec_floats() const { return static_cast<size_t>(2) * world * n_records * rec; }
    __device__ __forceinline__ float *slot(float *inbox, uint32_t parity, int src, int64_t i) const {
        return inbox + ((static_cast<size_t>(parity) * world + src) * n_records + i) * rec;
    }
    __device__ __forceinline__ uint32_t *stamp(float *inbox, uint32_t parity, int src, int64_t i) const {
        return reinterpret_cast<uint32_t *>(inbox + rec_floats()) + (static_cast<size_t>(parity) * world + src) * n_records + i;
    }
    __device__ __forceinline__ uint32_t *epoch(float *inbox, int64_t i) const {
        return reinterpret_cast<uint32_t *>(inbox + rec_floats()) + static_cast<size_t>(2) * world * n_records + i;
    }
};

// Sweep and exchange in ONE kernel.  The warp that holds the merged state of (batch, head) `bh` -- every
// lane the maximum, the two sums and D / 32 channels of O1 and O2 -- pushes it as record bh into every
// rank's inbox (plain stores over NVLink, then a release-stamp per peer), waits, bounded, for the stamps
// of record bh from the other ranks, merges the `world` records and writes row bh of `out`.  The protocol
// is that of decode_exchange_merge_kernel, and the merge is the same per-channel arithmetic, so the
// result is bit-identical to partial sweep + that kernel.  The waiting warp keeps its CTA resident; it
// waits only for warps of OTHER GPUs, which wait for nothing of this GPU's launch.
template <typename T, int D>
__device__ __forceinline__ void exchange_merge_warp(const DecodeArgs &a, int64_t bh, int lane, float big, float D1, float D2,
                                                    const float (&O1)[D / 32], const float (&O2)[D / 32]) {
    constexpr int REC = 2 * D + 4, CH = D / 32;
    const ExchangeArgs &x = a.xch;
    const InboxView iv{x.world, x.n_records, REC};
    uint32_t epoch = 0;
    if (lane == 0) epoch = *iv.epoch(x.inbox[x.rank], bh);
    epoch = __shfl_sync(0xffffffffu, epoch, 0);
    const uint32_t parity = epoch & 1u, stamp = epoch + 1u;
    // (1) push this rank's record to every rank (own inbox included)
    for (int p = 0; p < x.world; ++p) {
        float *dst = iv.slot(x.inbox[p], parity, x.rank, bh);
        if (lane == 0) *reinterpret_cast<float4 *>(dst) = make_float4(big, D1, D2, 0.f);
#pragma unroll
        for (int e = 0; e < CH; ++e) {
            dst[4 + lane * CH + e] = O1[e];
            dst[4 + D + lane * CH + e] = O2[e];
        }
    }
    __threadfence_system();
    __syncwarp();
    if (lane < x.world && lane != x.rank) {
        uint32_t *f = iv.stamp(x.inbox[lane], parity, x.rank, bh);
        asm volatile("st.release.sys.global.u32 [%0], %1;\n" ::"l"(f), "r"(stamp) : "memory");
    }
    // (2) wait for record bh of every other rank
    int bad = 0;
    if (lane < x.world && lane != x.rank) {
        const uint32_t *f = iv.stamp(x.inbox[x.rank], parity, lane, bh);
        const uint64_t t0 = global_timer_ns(), limit = static_cast<uint64_t>(x.wait_ms) * 1000000ull;
        uint32_t seen;
        for (;;) {
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(f) : "memory");
            if (seen == stamp) break;
            if (global_timer_ns() - t0 > limit) {
                sm100::report_error(sm100::ErrSink{x.err_word, x.err_mirror}, ((40 + lane) << 8) | 1);   // source rank never delivered
                if (x.status) atomicOr(x.status, 1 << lane);
                bad = 1;
                break;
            }
        }
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) *iv.epoch(x.inbox[x.rank], bh) = epoch + 1u;   // also after a time-out: the ranks stay in step
    // (3) merge and finalise this lane's channels (NaN when a record is missing)
    const float *rec0 = iv.slot(x.inbox[x.rank], parity, 0, bh);
#pragma unroll
    for (int e = 0; e < CH; ++e) {
        float M, S1, S2, A1, A2, y = __int_as_float(0x7fc00000);
        if (!bad) {
            merge_records<D, true>(rec0, x.world, static_cast<int64_t>(x.n_records) * REC, lane * CH + e, M, S1, S2, A1, A2);
            y = finalize(S1, S2, A1, A2);
        }
        store_elem<T>(a.out, bh * D + lane * CH + e, y);
    }
}

// Active key range [lo, hi) of a batch row, as indices into this buffer.
__device__ __forceinline__ void row_range(const DecodeArgs &a, int b, int &lo, int &hi) {
    int hi_g = a.total_len;
    if (a.n_lens) hi_g = min(max(a.lens[b], 1), a.total_len);
    else if (a.seqused) hi_g = min(max(a.seqused[b], 1), a.total_len);
    int lo_g = a.cache_start ? max(a.cache_start[b], 0) : 0;
    if (a.window >= 0) lo_g = max(lo_g, hi_g - a.window);
    lo = min(max(lo_g - a.kv_offset, 0), a.cache_len);
    hi = min(max(hi_g - a.kv_offset, 0), a.cache_len);
}

// What one of the batch * n_splits slots of a launch (per head) sweeps: part `part` of the `n_parts` into
// which the keys of row `b` are cut.  The records of (b, head) start at record first + head * n_parts.
struct SplitPlan {
    int b, part, n_parts, lo, hi;
    int64_t first;
};

// Part `part` of n_splits equal ones of the keys [lo, hi) of row b.  G: keys come in multiples of G.
template <int G>
__device__ __forceinline__ SplitPlan even_part(const DecodeArgs &a, int b, int part, int lo, int hi) {
    int chunk = (max(hi - lo, 0) + a.n_splits - 1) / a.n_splits;
    chunk = (chunk + G - 1) / G * G;
    const int my_lo = min(lo + part * chunk, hi);
    return SplitPlan{b, part, a.n_splits, my_lo, min(my_lo + chunk, hi), static_cast<int64_t>(b) * a.n_splits * a.heads_q};
}
template <int G>
__device__ __forceinline__ SplitPlan plan_even(const DecodeArgs &a, int b, int part) {
    int lo, hi;
    row_range(a, b, lo, hi);
    return even_part<G>(a, b, part, lo, hi);
}

// Slot -> plan, computed by a whole warp.
// Rows of one length get n_splits parts each.  With lengths of their own (seqused / cache_start) that makes the
// longest row set the time while the warps of the others idle.  There the slots are dealt out by length: the
// smallest part size for which the parts of all rows still fit into the slots.  Lane l looks after rows l, l + 32,
// ..: up to kBalancedRows rows.  `cap`: the most parts of a row that the merge takes.
// Not so where the longest row is within a.balanced sixteenths of the mean (see balance_from): dealing out costs the
// search and leaves parts and rows that no longer fall together with CTAs.
template <int G>
__device__ __forceinline__ SplitPlan plan_slot(const DecodeArgs &a, int slot, int lane, int cap) {
    SplitPlan p{-1, 0, 1, 0, 0, 0};
    constexpr int kRows = kBalancedRows / 32;
    int start[kRows], n[kRows], units[kRows], sum = 0, most = 0;   // units: multiples of G keys
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        start[i] = n[i] = units[i] = 0;
        if (lane + 32 * i < a.batch) {
            int hi;
            row_range(a, lane + 32 * i, start[i], hi);
            n[i] = max(hi - start[i], 0);
            units[i] = (n[i] + G - 1) / G;
        }
        sum += units[i];
        most = max(most, units[i]);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    most = __reduce_max_sync(0xffffffffu, most);
    if (16 * static_cast<int64_t>(most) * a.batch <= static_cast<int64_t>(a.balanced) * sum) {
        p.b = slot / a.n_splits;
        int lo = 0, len = 0;
#pragma unroll
        for (int i = 0; i < kRows; ++i)
            if (p.b >> 5 == i) {
                lo = __shfl_sync(0xffffffffu, start[i], p.b & 31);
                len = __shfl_sync(0xffffffffu, n[i], p.b & 31);
            }
        return even_part<G>(a, p.b, slot - p.b * a.n_splits, lo, lo + len);
    }
    const int slots = a.batch * a.n_splits;
    // part size in units: `good` fits (every row has at most n_splits parts), below `bad` none can
    // (A row of u units has fewer than u / m + 1 parts of m units, so m = sum / (slots - batch) fits as well.)  Four steps
    // between the two come within a sixteenth of the best; a step is a division per row and a reduction, in series.
    int bad = max(max((sum + slots - 1) / slots, (most + cap - 1) / cap), 1);
    int good = max(min((most + a.n_splits - 1) / a.n_splits, (sum + slots - a.batch - 1) / (slots - a.batch)), bad);
    for (int step = 0; step < 4 && bad < good; ++step) {
        const int mid = (bad + good) >> 1;
        int parts = 0;
#pragma unroll
        for (int i = 0; i < kRows; ++i)
            if (lane + 32 * i < a.batch) parts += max((units[i] + mid - 1) / mid, 1);
        if (static_cast<int>(__reduce_add_sync(0xffffffffu, parts)) <= slots) good = mid;
        else bad = mid + 1;
    }
    // the row that owns this slot
    int before = 0;       // parts of the rows of earlier i
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        if (32 * i >= a.batch || p.b >= 0) continue;
        const int mine = lane + 32 * i < a.batch ? max((units[i] + good - 1) / good, 1) : 0;
        int incl = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += x;
        }
        const unsigned owner = __ballot_sync(0xffffffffu, slot >= before + incl - mine && slot < before + incl);
        if (owner) {
            const int l = __ffs(owner) - 1;
            p.b = l + 32 * i;
            const int head = before + __shfl_sync(0xffffffffu, incl - mine, l);
            p.n_parts = __shfl_sync(0xffffffffu, mine, l);
            p.part = slot - head;
            p.first = static_cast<int64_t>(head) * a.heads_q;
            const int lo = __shfl_sync(0xffffffffu, start[i], l), hi = lo + __shfl_sync(0xffffffffu, n[i], l);
            p.lo = min(lo + p.part * good * G, hi);
            p.hi = min(p.lo + good * G, hi);
        }
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    return p;             // p.b < 0: a slot that no row needs
}

// Decode kernels are launched without waiting for the kernel before them to be over and done with (launch_overlapped): their
// CTAs come as soon as its last one has left, and wait (grid_wait, before anything touches global memory) for its writes.
// What they read may have been written while they were already resident, so no load takes the non-coherent path.
// Calls one after the other, us: 8 : 8 heads, B = 1, 4096 keys 12.2 -> 9.9, B = 32, 1024 keys 30.6 -> 28.5, B = 16, 8192 keys 92 -> 90.  Letting the next launch in earlier
// (griddepcontrol.launch_dependents, at the start or after the sweep) was slower: its CTAs then go where SMs are free first
// instead of evenly over the chip.  B = 64, 4096 keys, 32 : 8 heads, 128 CTAs: 164 us at the end, 180 after the sweep.
template <typename... Params, typename... Args>
static cudaError_t launch_overlapped(void (*kern)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// One WARP per (split, q head, batch row); a CTA is HG warps working on HG adjacent q
// heads of the same key range, so that together they sweep contiguous memory (all heads
// of a key are adjacent in the cache layout).  One q head per kv head.  Streams are merged by
// shuffles, splits by the last warp to arrive.
//
// SG ("split group") is the arrangement for launches with few (batch, head) pairs, which are bound by
// latency, not bandwidth: a CTA is the HG = 8 warps of eight ADJACENT SPLITS of one q head.  Every
// warp still sweeps its own keys, but the eight partial states meet in shared memory, so only one
// record per CTA goes through global memory, and the CTA that arrives last merges the (at most 32) CTA
// records with all 256 threads at once -- one round trip to L2 where a single merging warp needs one
// per eight records.  That allows splits of ~16 keys, whose loads are all in flight together.
//
// DEAL: the slots may be dealt out by length (a.balanced > 0).  A kernel of its own: with the plan of either kind in one,
// launches without lengths were 0.3 to 0.6 us longer (32 rows of 300 down to 100 keys, 8 : 8 heads, 12.4 -> 13.0).
template <typename T, int D, int HG, int U, bool SG, bool DEAL>
__global__ void __launch_bounds__(HG * 32, U > 4 ? 1 : 512 / (HG * 32)) decode_kernel(const DecodeArgs a) {
    grid_wait();
    constexpr int LPK = D / 8;      // lanes per key row
    constexpr int NS = 32 / LPK;    // streams per warp
    constexpr int REC = 2 * D + 4;  // floats per partial record
    constexpr int CH = D / 32;      // channels per lane in the merge

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hq = SG ? blockIdx.y : blockIdx.y * HG + warp;
    const int sid = lane / LPK, sl = lane % LPK;

    // the part of a batch row's keys that this warp sweeps
    SplitPlan plan;
    if constexpr (!DEAL) {
        plan = plan_even<NS>(a, blockIdx.z, SG ? blockIdx.x * HG + warp : blockIdx.x);
    } else {
        // the warps of a CTA have one slot: one of them plans (all eight, they queued for the divisions)
        __shared__ SplitPlan s_plan;
        if (warp == 0) {
            plan = plan_slot<NS>(a, blockIdx.z * a.n_splits + blockIdx.x, lane, a.n_groups ? 32 * a.n_groups : 32);
            if (lane == 0) s_plan = plan;
        }
        __syncthreads();
        plan = s_plan;
        if (plan.b < 0) return;
    }
    const int b = plan.b, my_lo = plan.lo, my_hi = plan.hi;
    const int n_iter = (my_hi - my_lo + NS * U - 1) / (NS * U);

    // this lane's 8 channels of q and r
    float qf[8], rf[8];
    {
        const int64_t qi = (static_cast<int64_t>(b) * a.heads_q + hq) * D + sl * 8;
        const uint4 qv = *reinterpret_cast<const uint4 *>(static_cast<const T *>(a.q) + qi), rv = *reinterpret_cast<const uint4 *>(static_cast<const T *>(a.r) + qi);
        unpack8<T>(qv, qf);
        unpack8<T>(rv, rf);
        if (plan.part == 0 && sid == 0) {
            if (a.q_copy) *reinterpret_cast<uint4 *>(static_cast<T *>(a.q_copy) + qi) = qv;
            if (a.r_copy) *reinterpret_cast<uint4 *>(static_cast<T *>(a.r_copy) + qi) = rv;
            if (a.lens_copy && hq == 0 && sl == 0) a.lens_copy[b] = a.lens[b];
        }
    }
    const bool paged = a.page_table != nullptr;      // uniform over the launch
    const int64_t row0 = (paged ? 0 : b * a.kv_sb) + hq * a.kv_sh + sl * 8;
    const T *kp = static_cast<const T *>(a.k) + row0;
    const T *vp = static_cast<const T *>(a.v) + row0;

    float m = -INFINITY, d1 = 0.f, d2 = 0.f, o1[8], o2[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) o1[e] = o2[e] = 0.f;

    // rows of iteration `it` -> registers (keys past the range read nothing and count as masked)
    // (the first argument is a compile-time tag: std::true_type for a paged cache.  The dense sweep must
    // not carry the page-table branch inside its unrolled loads -- that cost 4 to 12 % of the bandwidth.)
    auto load = [&](auto paged_tag, int it, uint4 (&kr)[U], uint4 (&vr)[U]) {
        const int base = my_lo + it * NS * U + sid;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kj = base + u * NS;
            if (kj < my_hi) {
                const int64_t at = decltype(paged_tag)::value ? paged_key_offset(a, b, kj) : static_cast<int64_t>(kj) * a.kv_st;
                const T *pk = kp + at, *pv = vp + at;
                kr[u] = ld_stream16(pk);
                vr[u] = ld_stream16(pv);
            } else {
                kr[u] = make_uint4(0u, 0u, 0u, 0u);
                vr[u] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    auto compute = [&](int it, const uint4 (&kr)[U], const uint4 (&vr)[U]) {
        const int base = my_lo + it * NS * U + sid;
        float s1[U], s2[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float kf[8];
            unpack8<T>(kr[u], kf);
            float x = 0.f, y = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                x = fmaf(qf[e], kf[e], x);
                y = fmaf(rf[e], kf[e], y);
            }
            s1[u] = x;
            s2[u] = y;
        }
#pragma unroll
        for (int off = LPK / 2; off > 0; off >>= 1)
#pragma unroll
            for (int u = 0; u < U; ++u) {
                s1[u] += __shfl_xor_sync(0xffffffffu, s1[u], off);
                s2[u] += __shfl_xor_sync(0xffffffffu, s2[u], off);
            }
        float cmax = -INFINITY;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            s1[u] = (base + u * NS < my_hi) ? s1[u] * a.c2 : -INFINITY;
            cmax = fmaxf(cmax, s1[u]);
        }
        const float m_new = fmaxf(m, cmax);
        const float m_safe = m_new == -INFINITY ? 0.f : m_new;
        const float alpha = fast_exp2(m - m_safe);
        m = m_new;
        d1 *= alpha;
        d2 *= alpha;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            o1[e] *= alpha;
            o2[e] *= alpha;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float p1 = fast_exp2(s1[u] - m_safe);
            const float p2 = p1 * s2[u];
            d1 += p1;
            d2 += p2;
            float vf[8];
            unpack8<T>(vr[u], vf);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                o1[e] = fmaf(p1, vf[e], o1[e]);
                o2[e] = fmaf(p2, vf[e], o2[e]);
            }
        }
    };
    // two register buffers: the rows of the next iteration are in flight while this one is reduced
    auto sweep = [&](auto paged_tag) {
        uint4 ka[U], va[U], kb[U], vb[U];
        if (n_iter > 0) load(paged_tag, 0, ka, va);
        for (int it = 0; it < n_iter; it += 2) {
            if (it + 1 < n_iter) load(paged_tag, it + 1, kb, vb);
            compute(it, ka, va);
            if (it + 1 < n_iter) {
                if (it + 2 < n_iter) load(paged_tag, it + 2, ka, va);
                compute(it + 1, kb, vb);
            }
        }
    };
    if (paged) sweep(std::true_type{});
    else sweep(std::false_type{});

    // merge the warp's streams (lanes that differ in bits >= log2(LPK) hold the same channels)
#pragma unroll
    for (int off = LPK; off < 32; off <<= 1) {
        const float m_o = __shfl_xor_sync(0xffffffffu, m, off);
        const float big = fmaxf(m, m_o);
        const float safe = big == -INFINITY ? 0.f : big;
        const float wa = fast_exp2(m - safe), wb = fast_exp2(m_o - safe);
        d1 = wa * d1 + wb * __shfl_xor_sync(0xffffffffu, d1, off);
        d2 = wa * d2 + wb * __shfl_xor_sync(0xffffffffu, d2, off);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            o1[e] = wa * o1[e] + wb * __shfl_xor_sync(0xffffffffu, o1[e], off);
            o2[e] = wa * o2[e] + wb * __shfl_xor_sync(0xffffffffu, o2[e], off);
        }
        m = big;
    }
    // every lane now holds the warp's state for channels sl * 8 .. sl * 8 + 7; lanes < LPK write
    const int64_t bh = static_cast<int64_t>(b) * a.heads_q + hq;
    const bool writer = lane < LPK;

    auto emit = [&](float M, float D1, float D2, const float (&O1)[8], const float (&O2)[8]) {
        if (!writer) return;
        if (a.part_out) {
            float *rec = a.part_out + bh * REC;
            if (lane == 0) {
                rec[0] = M;
                rec[1] = D1;
                rec[2] = D2;
                rec[3] = 0.f;
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                rec[4 + sl * 8 + e] = O1[e];
                rec[4 + D + sl * 8 + e] = O2[e];
            }
        } else {
            uint32_t pk[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                pk[e] = Elem<T>::pack(finalize(D1, D2, O1[2 * e], O2[2 * e]), finalize(D1, D2, O1[2 * e + 1], O2[2 * e + 1]));
            *reinterpret_cast<uint4 *>(static_cast<T *>(a.out) + bh * D + sl * 8) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
    };

    if constexpr (SG) {
        // ---- the eight splits of this CTA meet in shared memory
        static_assert(HG == 8, "a split group is eight warps");
        __shared__ __align__(16) float s_rec[HG][REC];
        __shared__ int s_last;
        if (writer) {
            if (lane == 0) *reinterpret_cast<float4 *>(&s_rec[warp][0]) = make_float4(m, d1, d2, 0.f);
#pragma unroll
            for (int e = 0; e < 8; e += 4) {
                *reinterpret_cast<float4 *>(&s_rec[warp][4 + sl * 8 + e]) = make_float4(o1[e], o1[e + 1], o1[e + 2], o1[e + 3]);
                *reinterpret_cast<float4 *>(&s_rec[warp][4 + D + sl * 8 + e]) = make_float4(o2[e], o2[e + 1], o2[e + 2], o2[e + 3]);
            }
        }
        __syncthreads();
        // thread c < 2 D owns element c of the concatenated [O1 | O2] from here on
        const int c = threadIdx.x;
        const bool active = c < 2 * D;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < HG; ++w) M = fmaxf(M, s_rec[w][0]);
        const float safe = M == -INFINITY ? 0.f : M;
        float S1 = 0.f, S2 = 0.f, A = 0.f;
#pragma unroll
        for (int w = 0; w < HG; ++w) {
            const float wt = fast_exp2(s_rec[w][0] - safe);
            S1 = fmaf(wt, s_rec[w][1], S1);
            S2 = fmaf(wt, s_rec[w][2], S2);
            if (active) A = fmaf(wt, s_rec[w][4 + c], A);
        }
        const int n_cta = gridDim.x;
        if (n_cta > 1 && cluster_size_x() == static_cast<uint32_t>(n_cta)) {
            // All CTAs of this (batch, head) form one thread-block cluster: the CTA records meet in the
            // shared memory of the cluster's first CTA (stores through distributed shared memory, one
            // cluster barrier) and never touch global memory -- no publish / fence / atomic / re-read.
            __shared__ __align__(16) float s_crec[8][REC];
            const uint32_t rank = cluster_rank_x();
            const uint32_t dst = cluster_map(smem_u32(&s_crec[rank][0]), 0);
            if (c == 0) {
                st_cluster_f32(dst, M);
                st_cluster_f32(dst + 4, S1);
                st_cluster_f32(dst + 8, S2);
            }
            if (active) st_cluster_f32(dst + 4u * (4 + c), A);
            cluster_sync();
            if (rank != 0) return;
            M = -INFINITY;
            for (int j = 0; j < n_cta; ++j) M = fmaxf(M, s_crec[j][0]);
            const float safe2 = M == -INFINITY ? 0.f : M;
            S1 = S2 = A = 0.f;
            for (int j = 0; j < n_cta; ++j) {
                const float wt = fast_exp2(s_crec[j][0] - safe2);
                S1 = fmaf(wt, s_crec[j][1], S1);
                S2 = fmaf(wt, s_crec[j][2], S2);
                if (active) A = fmaf(wt, s_crec[j][4 + c], A);
            }
        } else if (n_cta > 1) {
            // one record per CTA through global memory; the last CTA of the (batch, head) merges them
            float *rec = a.ws_parts + (bh * n_cta + blockIdx.x) * REC;
            if (c == 0) __stcg(reinterpret_cast<float4 *>(rec), make_float4(M, S1, S2, 0.f));
            if (active) __stcg(rec + 4 + c, A);
            __threadfence();
            __syncthreads();
            if (c == 0) s_last = atomicAdd(a.ws_counters + bh, 1) == n_cta - 1;
            __syncthreads();
            if (!s_last) return;
            __threadfence();
            const float *rec0 = a.ws_parts + bh * n_cta * REC;
            // all loads of all records in flight at once (n_cta <= 32): thread c its element of every
            // record, thread j < n_cta the header of record j, which then goes round through shared memory
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = (j < n_cta && active) ? __ldcg(rec0 + static_cast<int64_t>(j) * REC + 4 + c) : 0.f;
            float4 *s_head = reinterpret_cast<float4 *>(&s_rec[0][0]);     // the CTA's own records are spent
            if (c < 32)
                s_head[c] = c < n_cta ? __ldcg(reinterpret_cast<const float4 *>(rec0 + static_cast<int64_t>(c) * REC))
                                      : make_float4(-INFINITY, 0.f, 0.f, 0.f);
            __syncthreads();
            M = -INFINITY;
#pragma unroll
            for (int j = 0; j < 32; ++j) M = fmaxf(M, s_head[j].x);
            const float safe2 = M == -INFINITY ? 0.f : M;
            S1 = S2 = A = 0.f;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float4 h = s_head[j];
                const float wt = fast_exp2(h.x - safe2);
                S1 = fmaf(wt, h.y, S1);
                S2 = fmaf(wt, h.z, S2);
                A = fmaf(wt, x[j], A);
            }
            if (c == 0) a.ws_counters[bh] = 0;  // ready for the next launch on this workspace
        }
        if (a.part_out) {
            float *rec = a.part_out + bh * REC;
            if (c == 0) *reinterpret_cast<float4 *>(rec) = make_float4(M, S1, S2, 0.f);
            if (active) rec[4 + c] = A;
        } else {
            // O1 and O2 of a channel sit in two threads: pair them up through shared memory
            float *s_out = &s_rec[2][0];
            __syncthreads();                 // everybody has read the headers / the CTA's records
            if (active) s_out[c] = A;
            __syncthreads();
            if (c < D) store_elem<T>(a.out, bh * D + c, finalize(S1, S2, s_out[c], s_out[D + c]));
        }
        return;
    }

    if (plan.n_parts == 1) {
        emit(m, d1, d2, o1, o2);
        return;
    }

    // publish this split's state; the last warp of the (batch, head) to arrive merges all splits
    float *recs = a.ws_parts + (plan.first + static_cast<int64_t>(hq) * plan.n_parts) * REC;   // of this (batch, head)
    float *ws = recs + static_cast<int64_t>(plan.part) * REC;
    if (writer) {
        if (lane == 0) __stcg(reinterpret_cast<float4 *>(ws), make_float4(m, d1, d2, 0.f));
        __stcg(reinterpret_cast<float4 *>(ws + 4 + sl * 8), make_float4(o1[0], o1[1], o1[2], o1[3]));
        __stcg(reinterpret_cast<float4 *>(ws + 4 + sl * 8 + 4), make_float4(o1[4], o1[5], o1[6], o1[7]));
        __stcg(reinterpret_cast<float4 *>(ws + 4 + D + sl * 8), make_float4(o2[0], o2[1], o2[2], o2[3]));
        __stcg(reinterpret_cast<float4 *>(ws + 4 + D + sl * 8 + 4), make_float4(o2[4], o2[5], o2[6], o2[7]));
    }
    __threadfence();
    __syncwarp();

    // The merge is a chain of dependent L2 round trips if done record by record, and for small
    // batches it is most of the launch.  So the 32 lanes read the {m, d1, d2} headers of up to 32
    // records at once and reduce the maximum and the two sums with shuffles; for the O1 / O2 rows
    // every lane owns D / 32 channels and the loads of eight records are in flight together.  More
    // than 32 splits are merged in two levels, so that no warp walks more than 16 records.
    float big, D1, D2, O1[CH], O2[CH];
    auto arrive_last = [&](int *counter, int expected) -> bool {
        int last = 0;
        if (lane == 0) last = (atomicAdd(counter, 1) == expected - 1);
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) __threadfence();
        return last != 0;
    };
    if (plan.n_parts <= 32) {
        if (!arrive_last(a.ws_counters + bh, plan.n_parts)) return;
        warp_merge<D>(recs, plan.n_parts, lane, big, D1, D2, O1, O2);
    } else {
        const int gsize = max(PLX_DECODE_GROUP, (plan.n_parts + a.n_groups - 1) / a.n_groups), n_groups = (plan.n_parts + gsize - 1) / gsize;
        const int group = plan.part / gsize;
        const int first = group * gsize, size = min(gsize, plan.n_parts - first);
        int *gc = a.ws_gcounters + bh * a.n_groups + group;
        if (!arrive_last(gc, size)) return;
        warp_merge<D>(recs + static_cast<int64_t>(first) * REC, size, lane, big, D1, D2, O1, O2);
        float *grec = a.ws_gparts + (bh * a.n_groups + group) * REC;
        if (lane == 0) {
            __stcg(reinterpret_cast<float4 *>(grec), make_float4(big, D1, D2, 0.f));
            *gc = 0;   // ready for the next launch on this workspace
        }
#pragma unroll
        for (int e = 0; e < CH; ++e) {
            __stcg(grec + 4 + lane * CH + e, O1[e]);
            __stcg(grec + 4 + D + lane * CH + e, O2[e]);
        }
        __threadfence();
        __syncwarp();
        if (!arrive_last(a.ws_counters + bh, n_groups)) return;
        warp_merge<D>(a.ws_gparts + bh * a.n_groups * REC, n_groups, lane, big, D1, D2, O1, O2);
    }
    if (a.xch.world > 0) {
        exchange_merge_warp<T, D>(a, bh, lane, big, D1, D2, O1, O2);
    } else if (a.part_out) {
        float *rec = a.part_out + bh * REC;
        if (lane == 0) *reinterpret_cast<float4 *>(rec) = make_float4(big, D1, D2, 0.f);
#pragma unroll
        for (int e = 0; e < CH; ++e) {
            rec[4 + lane * CH + e] = O1[e];
            rec[4 + D + lane * CH + e] = O2[e];
        }
    } else {
        T *dst = static_cast<T *>(a.out) + bh * D + lane * CH;
        const uint32_t p0 = Elem<T>::pack(finalize(D1, D2, O1[0], O2[0]), finalize(D1, D2, O1[1], O2[1]));
        if (CH == 4) {
            const uint32_t p1 = Elem<T>::pack(finalize(D1, D2, O1[CH - 2], O2[CH - 2]), finalize(D1, D2, O1[CH - 1], O2[CH - 1]));
            *reinterpret_cast<uint2 *>(dst) = make_uint2(p0, p1);
        } else {
            *reinterpret_cast<uint32_t *>(dst) = p0;
        }
    }
    if (lane == 0) a.ws_counters[bh] = 0;  // ready for the next launch on this workspace
}

// n_parts arrays of n_records records each -> out
template <typename T, int D>
__global__ void __launch_bounds__(D) decode_merge_kernel(const float *parts, int n_parts, int n_records, void *out) {
    constexpr int REC = 2 * D + 4;
    const int i = blockIdx.x, d = threadIdx.x;
    float M, D1, D2, O1, O2;
    merge_records<D, false>(parts + static_cast<int64_t>(i) * REC, n_parts, static_cast<int64_t>(n_records) * REC, d, M,
                            D1, D2, O1, O2);
    store_elem<T>(out, static_cast<int64_t>(i) * D + d, finalize(D1, D2, O1, O2));
}

// ========================================================================= //
// Exchange + merge of the per-rank partial states of a KV-sharded decode, in one kernel over peer
// memory (NVLink loads / stores; no TMA, no multicast): instead of an all-gather followed by a
// merge kernel.
//
// Every rank owns an "inbox" that all ranks have mapped: [2 parities][world][n_records] records,
// then [2][world][n_records] 32-bit stamps, then [n_records] step counters (read only by their owner).  CTA i of rank g (1) stores record i of its partial
// array into slot (parity, g, i) of EVERY rank's inbox and then, after a system-wide fence, the
// stamp (step + 1) beside it; (2) waits -- bounded -- until its own inbox holds the stamps of record i
// from every other rank, and merges the `world` records into out[i].  A CTA waits only for CTAs of the
// same index on OTHER GPUs, which depend on nothing, so no CTA of a grid ever waits for another CTA
// of the same grid.  Two parities: a rank cannot start step e + 2 before every peer has finished
// merging step e (it needs their records of step e + 1, which they send after that merge).
//
// The wait is bounded (x.wait_ms).  A CTA whose wait runs out sets bit `src` of the caller's status
// word, reports (40 + src) through the error words, and writes NaN into its row of `out`, so that a
// result built on a missing record cannot pass for a number; the step counter advances all the same,
// which keeps the ranks in step for the next call.
// ========================================================================= //

template <typename T, int D>
__global__ void __launch_bounds__(D) decode_exchange_merge_kernel(const ExchangeArgs x, const float *part, void *out,
                                                                  const sm100::ErrSink err) {
    constexpr int REC = 2 * D + 4;
    const int i = blockIdx.x, d = threadIdx.x;
    const size_t rec_floats = static_cast<size_t>(2) * x.world * x.n_records * REC;
    // the step counter of record i lives beside this rank's stamps (so a captured launch can be replayed)
    uint32_t *my_epoch = reinterpret_cast<uint32_t *>(x.inbox[x.rank] + rec_floats) + static_cast<size_t>(2) * x.world * x.n_records + i;
    const uint32_t epoch = *my_epoch;
    const uint32_t parity = epoch & 1u, stamp = epoch + 1u;
    auto slot = [&](float *inbox, int src) -> float * {
        return inbox + ((static_cast<size_t>(parity) * x.world + src) * x.n_records + i) * REC;
    };
    auto stamp_of = [&](float *inbox, int src) -> uint32_t * {
        return reinterpret_cast<uint32_t *>(inbox + rec_floats) + (static_cast<size_t>(parity) * x.world + src) * x.n_records + i;
    };
    // (1) push record i to every rank (own inbox included)
    const float *mine = part + static_cast<size_t>(i) * REC;
    for (int p = 0; p < x.world; ++p) {
        float *dst = slot(x.inbox[p], x.rank);
        for (int c = d; c < REC; c += D) dst[c] = mine[c];
    }
    __threadfence_system();
    __syncthreads();
    if (d < x.world && d != x.rank) {
        uint32_t *f = stamp_of(x.inbox[d], x.rank);
        asm volatile("st.release.sys.global.u32 [%0], %1;\n" ::"l"(f), "r"(stamp) : "memory");
    }
    // (2) wait for record i of every other rank, then merge
    __shared__ int s_bad;
    if (d == 0) s_bad = 0;
    __syncthreads();
    if (d < x.world && d != x.rank) {
        const uint32_t *f = stamp_of(x.inbox[x.rank], d);
        const uint64_t t0 = global_timer_ns(), limit = static_cast<uint64_t>(x.wait_ms) * 1000000ull;
        uint32_t seen;
        for (;;) {
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(f) : "memory");
            if (seen == stamp) break;
            if (global_timer_ns() - t0 > limit) {
                sm100::report_error(err, ((40 + d) << 8) | 1);   // source rank d never delivered
                if (x.status) atomicOr(x.status, 1 << d);
                s_bad = 1;
                break;
            }
        }
    }
    __syncthreads();
    if (d == 0) *my_epoch = epoch + 1u;   // also after a time-out: the ranks stay in step
    if (s_bad) {
        store_elem<T>(out, static_cast<int64_t>(i) * D + d, __int_as_float(0x7fc00000));   // NaN: this row has no answer
        return;
    }
    float M, D1, D2, O1, O2;
    merge_records<D, true>(slot(x.inbox[x.rank], 0), x.world, static_cast<int64_t>(x.n_records) * REC, d, M, D1, D2, O1, O2);
    store_elem<T>(out, static_cast<int64_t>(i) * D + d, finalize(D1, D2, O1, O2));
}

template <typename T, int D>
static int launch_exchange_t(const ExchangeArgs &x, const float *part, void *out, const ErrorWords &ew, cudaStream_t stream) {
    decode_exchange_merge_kernel<T, D><<<x.n_records, D, 0, stream>>>(x, part, out, sm100::ErrSink{ew.word, ew.mirror});
    count_launch();
    return cudaGetLastError() == cudaSuccess ? PLX_OK : PLX_ERR_LAUNCH;
}

int launch_decode_exchange_merge(const ExchangeArgs &x, const float *part, int head_dim, int dtype, void *out,
                                 const ErrorWords &err, cudaStream_t stream) {
    if (dtype == PLX_BF16) {
        if (head_dim == 128) return launch_exchange_t<__nv_bfloat16, 128>(x, part, out, err, stream);
        if (head_dim == 64) return launch_exchange_t<__nv_bfloat16, 64>(x, part, out, err, stream);
    } else if (dtype == PLX_FP16) {
        if (head_dim == 128) return launch_exchange_t<__half, 128>(x, part, out, err, stream);
        if (head_dim == 64) return launch_exchange_t<__half, 64>(x, part, out, err, stream);
    }
    return PLX_ERR_UNSUPPORTED;
}

// ========================================================================= //
// Grouped-query decode on the warp-level tensor cores.
//
// With n_rep q heads per kv head, the per-key arithmetic of the kernel above grows n_rep-fold
// while the bytes stay the same: from n_rep = 4 on it is bound by the FMA pipe, not by HBM.  Here
// the q heads of a group are the M dimension of m16n8k16 MMAs (up to 16 rows, zero-padded), so
// K and V are read once per group and the arithmetic moves to the tensor cores.
//
// One warp per (split, kv head [x 16-row head group], batch row).  The warp stages 16-key tiles of
// K and V in its own shared memory (16-byte cp.async, kGqaStages deep, rows padded to D + 8
// elements; one bulk copy per row measured 1.6x slower: 32 small copies per tile queue up),
// forms S1 = Q_g K^T and S2 = R_g K^T, runs the online softmax per row in the accumulator
// fragments, and accumulates O1 += P1 V, O2 += P2 V with the P fragments as the A operand.  The eight
// warps of a CTA are adjacent splits of one kv head; they meet in shared memory at the end.
//
// Short launches are bound by latency, long ones by HBM and by what the warps have in flight: three tiles each from the
// start (q and r go straight to registers instead of through the last stage), the next one as soon as a stage is free.
// Calls one after the other, us, this, the overlapped launches (above) and the transposed products (below) together: 32 : 8 heads, B = 1,
// 1000 keys 16.5 -> 12.2, 8192 keys 16.4 -> 11.8, 32768 keys 31.7 -> 28.1, B = 64, 4096 keys 163.6 -> 157.2 (6.8 TB/s); 16 : 2 heads, B = 3,
// 3000 keys 18.6 -> 13.8; 16 : 1 heads, B = 8, 8192 keys 22.8 -> 19.0.
// ========================================================================= //
// a lane's channels of a record, 16 or 8 bytes
__device__ __forceinline__ void load_channels(const float *p, float (&x)[4]) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void load_channels(const float *p, float (&x)[2]) {
    const float2 v = *reinterpret_cast<const float2 *>(p);
    x[0] = v.x; x[1] = v.y;
}
__device__ __forceinline__ void store_channels(float *p, const float (&x)[4]) {
    __stcg(reinterpret_cast<float4 *>(p), make_float4(x[0], x[1], x[2], x[3]));
}
__device__ __forceinline__ void store_channels(float *p, const float (&x)[2]) {
    __stcg(reinterpret_cast<float2 *>(p), make_float2(x[0], x[1]));
}

// transpose of an 8 x 8 block of 16-bit elements (lane 4 g + t holds elements 2 t, + 1 of row g)
__device__ __forceinline__ uint32_t movmatrix_t(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
    return y;
}

constexpr int kGqaTile = 16;     // keys per staged tile
constexpr int kGqaStages = 3;
constexpr int kGqaWarps = kDecodeGqaWarps;   // warps (independent splits) per CTA

template <int D>
struct GqaSmem {
    static constexpr int kPerWarp = kGqaStages * 2 * kGqaTile * (D + 8) * 2;   // K and V tiles, 16-bit elements
};

// PAGED: a kernel of its own, so that the dense sweep carries neither the page numbers nor the choice in its loop.  (In
// one kernel, with a register spilled: B = 64, 8192 keys, 32 q / 8 kv heads 348 us against 329, B = 8, 32768 keys 182 against 175.)
//
// FEW: at most 8 q heads per kv head, the usual case.  Then the products are transposed -- keys are the M dimension of the
// scores (S^T = K Q_g^T), channels that of the outputs (O^T += V^T P^T), and the heads the 8 columns -- which takes half the
// MMAs, with none of them on rows of zeros, and half the registers for accumulators and fragments (in all 190 to 201 at
// head_dim 128, where the other form fills 255); a movmatrix per 8 x 8 block turns P^T around.
// B = 16, 1024 keys, 32 : 8 heads 16.7 -> 16.0 us, B = 8, 4000 keys, rows of different lengths 40.8 -> 34.0.
template <typename T, int D, bool PAGED, bool FEW>
__global__ void __launch_bounds__(kGqaWarps * 32, 1) decode_gqa_kernel(const DecodeArgs a, int n_hgroups) {
    grid_wait();
    constexpr int LD = D + 8;                       // padded row: ldmatrix without bank conflicts
    constexpr int REC = 2 * D + 4, CH = D / 32;
    constexpr int KS = D / 16;                      // k-steps of the score products
    constexpr uint32_t kTileBytes = kGqaTile * LD * 2;
    constexpr int CPR = D / 8;                      // 16-byte chunks per row
    static_assert(16 * REC * 4 <= GqaSmem<D>::kPerWarp, "a warp's records fit where its tiles were");
    extern __shared__ __align__(16) unsigned char gqa_smem[];
    __shared__ int s_row[kGqaWarps], s_arrived[kGqaWarps];   // batch row of each warp (-1: none); arrival order of its segment

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // A CTA is eight adjacent slots of one (kv head, head group); heads are fastest over the grid, so CTAs that run
    // together read neighbouring memory.
    const int n_hunits = a.heads_kv * n_hgroups, n_slots = a.batch * a.n_splits;
    const int hunit = blockIdx.x % n_hunits, cta = blockIdx.x / n_hunits, slot = cta * kGqaWarps + warp;
    const int hk = hunit / n_hgroups, hgrp = hunit % n_hgroups;
    SplitPlan plan{-1, 0, 0, 0, 0, 0};
    if (slot < n_slots) plan = a.balanced ? plan_slot<kGqaTile>(a, slot, lane, n_slots) : plan_even<kGqaTile>(a, slot / a.n_splits, slot % a.n_splits);
    const int b = max(plan.b, 0), my_lo = plan.lo, my_hi = plan.b < 0 ? plan.lo : plan.hi;
    const int n_tiles = (my_hi - my_lo + kGqaTile - 1) / kGqaTile;
    const int hq0 = hk * a.n_rep + hgrp * 16;       // first q head of this CTA's rows
    const int n_rows = min(16, a.n_rep - hgrp * 16);
    const uint32_t sbase = smem_u32(gqa_smem) + warp * GqaSmem<D>::kPerWarp;
    auto sK = [&](int st) -> uint32_t { return sbase + st * 2 * kTileBytes; };
    auto sV = [&](int st) -> uint32_t { return sbase + st * 2 * kTileBytes + kTileBytes; };
    if (lane == 0) s_row[warp] = plan.b;

    // Tile i of this warp -> stage i % kGqaStages.  A lane copies the same 16-byte column of every
    // (32 / CPR)-th row, so its source and destination advance by constants; rows past my_hi (last tile
    // only) are zero-filled.  In a paged cache a tile lies in one page when pages hold at least a tile and the
    // range starts on a tile boundary (it does but for windows and cache_start): one page number per tile then,
    // read ahead.
    constexpr int RPI = 32 / CPR;                                  // rows covered by one instruction of the warp
    const int my_row = lane / CPR, my_col = lane % CPR;
    const bool page_per_tile = PAGED && a.page_mask + 1 >= kGqaTile && my_lo % kGqaTile == 0;
    const T *kp = static_cast<const T *>(a.k) + (PAGED ? 0 : b * a.kv_sb) + hk * a.kv_sh + my_col * 8;
    const T *vp = static_cast<const T *>(a.v) + (PAGED ? 0 : b * a.kv_sb) + hk * a.kv_sh + my_col * 8;
    const uint32_t my_dst = (my_row * LD + my_col * 8) * 2;
    // Pages of the next tiles to be loaded: as many as there are stages, so that no load waits for the page number of another;
    // two where registers are short (B = 64, 4096 keys, 16 : 1 heads, pages, 34.0 us, three 35.8).
    constexpr int kPages = FEW ? kGqaStages : 2;
    uint32_t next_page[kPages];
    auto page_of_tile = [&](int i) -> uint32_t { return page_per_tile && i < n_tiles ? paged_key_page(a, b, my_lo + i * kGqaTile) : 0u; };
    if (PAGED)
#pragma unroll
        for (int i = 0; i < kPages; ++i) next_page[i] = page_of_tile(i);
    auto load_tile = [&](int i) {
        if (i < n_tiles) {
            const int st = i % kGqaStages, tile0 = my_lo + i * kGqaTile, key0 = tile0 + my_row;
            const uint32_t dk = sK(st) + my_dst, dv = sV(st) + my_dst;
            const bool whole = tile0 + kGqaTile <= my_hi;
            if (!PAGED || page_per_tile) {
                const int64_t step = static_cast<int64_t>(RPI) * a.kv_st;
                const int64_t at = page_per_tile ? static_cast<int64_t>(next_page[0]) * a.kv_sb + static_cast<int64_t>(key0 & a.page_mask) * a.kv_st
                                                 : static_cast<int64_t>(key0) * a.kv_st;
                if (PAGED) {
#pragma unroll
                    for (int n = 1; n < kPages; ++n) next_page[n - 1] = next_page[n];
                    next_page[kPages - 1] = page_of_tile(i + kPages);
                }
                if (whole) {
#pragma unroll
                    for (int j = 0; j < kGqaTile / RPI; ++j) {
                        cp_async16(dk + j * RPI * LD * 2, kp + at + j * step, 16);
                        cp_async16(dv + j * RPI * LD * 2, vp + at + j * step, 16);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < kGqaTile / RPI; ++j) {
                        const bool in = key0 + j * RPI < my_hi;
                        cp_async16(dk + j * RPI * LD * 2, kp + (in ? at + j * step : 0), in ? 16 : 0);
                        cp_async16(dv + j * RPI * LD * 2, vp + (in ? at + j * step : 0), in ? 16 : 0);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < kGqaTile / RPI; ++j) {
                    const bool in = whole || key0 + j * RPI < my_hi;
                    const int64_t at = in ? paged_key_offset(a, b, key0 + j * RPI) : 0;
                    cp_async16(dk + j * RPI * LD * 2, kp + at, in ? 16 : 0);
                    cp_async16(dv + j * RPI * LD * 2, vp + at, in ? 16 : 0);
                }
            }
        }
        cp_async_commit();             // always: keeps the group count uniform
    };
    // q and r of the group as A fragments (FEW: as B fragments, of 8 rows), rows past the group as zeros, straight from global
    // memory, so that all stages are free for the first tiles; requested behind the first tile, with which they are needed.
    // Beyond 4 rows a lane takes 16 bytes of every fourth chunk of its rows and the quad trades words, else a word of the fragment
    // per load, which is a line per row each time.  (Words against 16 bytes: 4 rows of 1000 keys, 16 : 1 heads 28.7 / 24.8 us, 64 : 8
    // 16.8 / 13.1; one row of 400 keys, 32 : 8 heads 8.75 / 8.9.)
    constexpr int QF = FEW ? 2 : 4, QC = D / 32;
    const bool words = FEW && n_rows <= 4;
    uint32_t qa[KS][QF], ra[KS][QF];
    uint4 qx[QF / 2][QC], rx[QF / 2][QC];
    load_tile(0);
    {
        const int64_t at = (static_cast<int64_t>(b) * a.heads_q + hq0) * D;
        const T *qg = static_cast<const T *>(a.q) + at, *rg = static_cast<const T *>(a.r) + at;
        if (words) {
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int x = g * D + ks * 16 + 8 * e + 2 * t;
                    qa[ks][e] = g < n_rows ? *reinterpret_cast<const uint32_t *>(qg + x) : 0u;
                    ra[ks][e] = g < n_rows ? *reinterpret_cast<const uint32_t *>(rg + x) : 0u;
                }
        } else {
#pragma unroll
            for (int h = 0; h < QF / 2; ++h)
#pragma unroll
                for (int j = 0; j < QC; ++j) {
                    const int row = g + 8 * h, x = row * D + 32 * j + 8 * t;
                    qx[h][j] = row < n_rows ? *reinterpret_cast<const uint4 *>(qg + x) : make_uint4(0u, 0u, 0u, 0u);
                    rx[h][j] = row < n_rows ? *reinterpret_cast<const uint4 *>(rg + x) : make_uint4(0u, 0u, 0u, 0u);
                }
        }
    }
#pragma unroll
    for (int i = 1; i < kGqaStages; ++i) load_tile(i);
    if (!words) {
#pragma unroll
        for (int h = 0; h < QF / 2; ++h)
#pragma unroll
            for (int j = 0; j < QC; ++j) {
                auto trade = [&](const uint4 &x, uint32_t (&f)[KS][QF]) {
                    uint32_t w[4] = {x.x, x.y, x.z, x.w};
                    sm100::quad_transpose(w, t);               // w[i]: channels 2 t, + 1 of chunk 4 j + i
#pragma unroll
                    for (int i = 0; i < 4; ++i) f[2 * j + (i >> 1)][FEW ? i & 1 : h + 2 * (i & 1)] = w[i];
                };
                trade(qx[h][j], qa);
                trade(rx[h][j], ra);
            }
    }

    // State of two rows of the group, g and g + 8 (FEW: 2 t and 2 t + 1); d1 / d2 are this thread's share until the end.
    // Accumulators: channels 8 i + 2 t, + 1 of the two rows (FEW: channels 16 i + g and + 8).
    constexpr int NO = FEW ? D / 16 : D / 8;
    float m[2] = {-INFINITY, -INFINITY}, d1[2] = {0.f, 0.f}, d2[2] = {0.f, 0.f};
    float o1[NO][4], o2[NO][4];
#pragma unroll
    for (int i = 0; i < NO; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o1[i][e] = o2[i][e] = 0.f;

    for (int i = 0; i < n_tiles; ++i) {
        const int st = i % kGqaStages, key0 = my_lo + i * kGqaTile;
        cp_async_wait<kGqaStages - 1>();
        __syncwarp();                    // tile i has landed for every lane

        if constexpr (FEW) {
            // S1^T, S2^T: 16 keys x 8 rows; this thread has keys g and g + 8 of its two rows
            float s1[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                uint32_t ka[4];
                ldsm_x4(ka, a_addr<LD>(sK(st), 0, ks * 16, lane));
                Elem<T>::mma(s1, ka, qa[ks][0], qa[ks][1]);
                Elem<T>::mma(s2, ka, ra[ks][0], ra[ks][1]);
            }
            uint32_t pb1[2], pb2[2];
            float alpha[2], m_safe[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                s1[e] = key0 + g < my_hi ? s1[e] * a.c2 : -INFINITY;
                s1[2 + e] = key0 + g + 8 < my_hi ? s1[2 + e] * a.c2 : -INFINITY;
                float mx = fmaxf(s1[e], s1[2 + e]);
#pragma unroll
                for (int off = 4; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
                const float m_new = fmaxf(m[e], mx);
                m_safe[e] = m_new == -INFINITY ? 0.f : m_new;
                alpha[e] = fast_exp2(m[e] - m_safe[e]);
                m[e] = m_new;
            }
            if (alpha[0] != 1.f || alpha[1] != 1.f) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    d1[e] *= alpha[e];
                    d2[e] *= alpha[e];
                }
#pragma unroll
                for (int i2 = 0; i2 < NO; ++i2)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        o1[i2][e] *= alpha[e & 1];
                        o2[i2][e] *= alpha[e & 1];
                    }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float p0 = fast_exp2(s1[2 * h] - m_safe[0]), p1 = fast_exp2(s1[2 * h + 1] - m_safe[1]);
                const uint32_t u = Elem<T>::pack(p0, p1), w = Elem<T>::pack(p0 * s2[2 * h], p1 * s2[2 * h + 1]);
                // (the sums are those of the ROUNDED weights, see below)
                const float2 pr = Elem<T>::unpack(u), qr = Elem<T>::unpack(w);
                d1[0] += pr.x;
                d1[1] += pr.y;
                d2[0] += qr.x;
                d2[1] += qr.y;
                pb1[h] = movmatrix_t(u);
                pb2[h] = movmatrix_t(w);
            }
#pragma unroll
            for (int cb = 0; cb < NO; ++cb) {
                uint32_t vb[4];
                ldsm_x4_t(vb, bt_addr<LD>(sV(st), 0, cb * 16, lane));
                const uint32_t va[4] = {vb[0], vb[2], vb[1], vb[3]};
                Elem<T>::mma(o1[cb], va, pb1[0], pb1[1]);
                Elem<T>::mma(o2[cb], va, pb2[0], pb2[1]);
            }
        } else {
        // S1, S2: 16 rows x 16 keys (two 8-key blocks)
        float s1[2][4], s2[2][4];
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int e = 0; e < 4; ++e) s1[nb][e] = s2[nb][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            uint32_t kb[4];
            ldsm_x4(kb, bn_addr<LD>(sK(st), 0, ks * 16, lane));
            Elem<T>::mma(s1[0], qa[ks], kb[0], kb[1]);
            Elem<T>::mma(s1[1], qa[ks], kb[2], kb[3]);
            Elem<T>::mma(s2[0], ra[ks], kb[0], kb[1]);
            Elem<T>::mma(s2[1], ra[ks], kb[2], kb[3]);
        }
        // scale, mask the keys past the range, row maxima (a row lives in the four lanes of a quad)
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = key0 + nb * 8 + 2 * t + (e & 1);
                s1[nb][e] = key < my_hi ? s1[nb][e] * a.c2 : -INFINITY;
                mx[e >> 1] = fmaxf(mx[e >> 1], s1[nb][e]);
            }
        uint32_t pa1[4], pa2[4];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            mx[hh] = fmaxf(mx[hh], __shfl_xor_sync(0xffffffffu, mx[hh], 1));
            mx[hh] = fmaxf(mx[hh], __shfl_xor_sync(0xffffffffu, mx[hh], 2));
            const float m_new = fmaxf(m[hh], mx[hh]);
            const float m_safe = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = fast_exp2(m[hh] - m_safe);
            m[hh] = m_new;
            if (alpha != 1.f) {
                d1[hh] *= alpha;
                d2[hh] *= alpha;
#pragma unroll
                for (int i2 = 0; i2 < D / 8; ++i2) {
                    o1[i2][2 * hh] *= alpha;
                    o1[i2][2 * hh + 1] *= alpha;
                    o2[i2][2 * hh] *= alpha;
                    o2[i2][2 * hh + 1] *= alpha;
                }
            }
#pragma unroll
            for (int nb = 0; nb < 2; ++nb) {
                const float p0 = fast_exp2(s1[nb][2 * hh] - m_safe), p1 = fast_exp2(s1[nb][2 * hh + 1] - m_safe);
                const float q0 = p0 * s2[nb][2 * hh], q1 = p1 * s2[nb][2 * hh + 1];
                // A fragment of the output products: {row g, keys 2t..}, {row g + 8, ..}, {row g, keys 8 + 2t..}, {row g + 8, ..}
                pa1[2 * nb + hh] = Elem<T>::pack(p0, p1);
                pa2[2 * nb + hh] = Elem<T>::pack(q0, q1);
                // The sums are those of the ROUNDED weights that multiply V: the output then cancels as in
                // exact arithmetic when a row sees few keys (one key returns v exactly).
                const float2 pr = Elem<T>::unpack(pa1[2 * nb + hh]), qr = Elem<T>::unpack(pa2[2 * nb + hh]);
                d1[hh] += pr.x + pr.y;
                d2[hh] += qr.x + qr.y;
            }
        }
        // O1 += P1 V, O2 += P2 V: 16 channels per step
#pragma unroll
        for (int db = 0; db < D / 16; ++db) {
            uint32_t vb[4];
            ldsm_x4_t(vb, bt_addr<LD>(sV(st), 0, db * 16, lane));
            Elem<T>::mma(o1[2 * db], pa1, vb[0], vb[1]);
            Elem<T>::mma(o1[2 * db + 1], pa1, vb[2], vb[3]);
            Elem<T>::mma(o2[2 * db], pa2, vb[0], vb[1]);
            Elem<T>::mma(o2[2 * db + 1], pa2, vb[2], vb[3]);
        }
        }
        __syncwarp();                    // every lane has left tile i
        load_tile(i + kGqaStages);       // into its stage
    }
    cp_async_wait<0>();
    if (plan.b >= 0 && plan.part == 0) {
        const int64_t at = (static_cast<int64_t>(b) * a.heads_q + hq0) * D;
        for (int c = lane; c < n_rows * CPR; c += 32) {
            if (a.q_copy) reinterpret_cast<uint4 *>(static_cast<T *>(a.q_copy) + at)[c] = reinterpret_cast<const uint4 *>(static_cast<const T *>(a.q) + at)[c];
            if (a.r_copy) reinterpret_cast<uint4 *>(static_cast<T *>(a.r_copy) + at)[c] = reinterpret_cast<const uint4 *>(static_cast<const T *>(a.r) + at)[c];
        }
        if (a.lens_copy && hunit == 0 && lane == 0) a.lens_copy[b] = a.lens[b];
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int off = FEW ? 4 : 1; off < (FEW ? 32 : 4); off <<= 1) {     // the lanes that share a row
            d1[hh] += __shfl_xor_sync(0xffffffffu, d1[hh], off);
            d2[hh] += __shfl_xor_sync(0xffffffffu, d2[hh], off);
        }

    // ---- merge.  Every warp leaves its state in its own shared memory, where its tiles were: one record per row of
    // the group.  The warps of a batch row are neighbours (a segment).  The rows of all segments are dealt out to the
    // warps; a segment that is all of its (batch row, head) writes the result, any other one record per row to
    // global memory, and the CTA whose segment arrives last there merges those.
    // (Through global memory warp by warp, in two levels beyond 32 splits, the merge was most of a short launch, which is
    // bound by latency: B = 1, 8192 keys, 32 q / 8 kv heads 29.5 -> 16.5 us.)
    float *own = reinterpret_cast<float *>(gqa_smem + warp * GqaSmem<D>::kPerWarp);
    __syncwarp();                        // every lane has left the last tile
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int row = FEW ? 2 * t + hh : g + 8 * hh;
        if (row >= n_rows) continue;
        float *rec = own + row * REC;
        if ((FEW ? g : t) == 0) *reinterpret_cast<float4 *>(rec) = make_float4(m[hh], d1[hh], d2[hh], 0.f);
#pragma unroll
        for (int i = 0; i < NO; ++i) {
            if constexpr (FEW) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    rec[4 + 16 * i + 8 * c + g] = o1[i][2 * c + hh];
                    rec[4 + D + 16 * i + 8 * c + g] = o2[i][2 * c + hh];
                }
            } else {
                *reinterpret_cast<float2 *>(rec + 4 + 8 * i + 2 * t) = make_float2(o1[i][2 * hh], o1[i][2 * hh + 1]);
                *reinterpret_cast<float2 *>(rec + 4 + D + 8 * i + 2 * t) = make_float2(o2[i][2 * hh], o2[i][2 * hh + 1]);
            }
        }
    }
    // segment of this warp: warps w0 .. w0 + n_seg - 1; where its (batch row, head) begins among the slots
    __syncthreads();
    int w0 = warp, n_seg = 0;
    while (w0 > 0 && s_row[w0 - 1] == plan.b) --w0;
    while (w0 + n_seg < kGqaWarps && s_row[w0 + n_seg] == plan.b) ++n_seg;
    const int head_slot = slot - plan.part, first_cta = head_slot / kGqaWarps;
    const int n_ctas = plan.b < 0 ? 0 : (head_slot + plan.n_parts - 1) / kGqaWarps - first_cta + 1;
    const bool alone = n_ctas == 1;
    auto bh_of = [&](int row) -> int64_t { return static_cast<int64_t>(b) * a.heads_q + hq0 + row; };
    auto recs_of = [&](int row) -> float * { return a.ws_parts + (plan.first + static_cast<int64_t>(hq0 + row) * plan.n_parts) * REC; };

    float big = -INFINITY, D1 = 0.f, D2 = 0.f, O1[CH], O2[CH];
    auto emit = [&](int64_t bh) {
        if (a.part_out) {
            float *rec = a.part_out + bh * REC;
            if (lane == 0) *reinterpret_cast<float4 *>(rec) = make_float4(big, D1, D2, 0.f);
#pragma unroll
            for (int e = 0; e < CH; ++e) {
                rec[4 + lane * CH + e] = O1[e];
                rec[4 + D + lane * CH + e] = O2[e];
            }
        } else {
            T *dst = static_cast<T *>(a.out) + bh * D + lane * CH;
            const uint32_t p0 = Elem<T>::pack(finalize(D1, D2, O1[0], O2[0]), finalize(D1, D2, O1[1], O2[1]));
            if (CH == 4) {
                const uint32_t p1 = Elem<T>::pack(finalize(D1, D2, O1[CH - 2], O2[CH - 2]), finalize(D1, D2, O1[CH - 1], O2[CH - 1]));
                *reinterpret_cast<uint2 *>(dst) = make_uint2(p0, p1);
            } else {
                *reinterpret_cast<uint32_t *>(dst) = p0;
            }
        }
    };
    // the warps of a segment share its rows
    if (plan.b >= 0) {
        for (int row = warp - w0; row < n_rows; row += n_seg) {
            const float *rec0 = reinterpret_cast<const float *>(gqa_smem + w0 * GqaSmem<D>::kPerWarp) + row * REC;
            constexpr int kStride = GqaSmem<D>::kPerWarp / 4;
            big = -INFINITY;
            for (int w = 0; w < n_seg; ++w) big = fmaxf(big, rec0[w * kStride]);
            const float safe = big == -INFINITY ? 0.f : big;
            D1 = D2 = 0.f;
#pragma unroll
            for (int e = 0; e < CH; ++e) O1[e] = O2[e] = 0.f;
            for (int w = 0; w < n_seg; ++w) {
                const float *rec = rec0 + w * kStride;
                const float wt = fast_exp2(rec[0] - safe);
                D1 = fmaf(wt, rec[1], D1);
                D2 = fmaf(wt, rec[2], D2);
                float x[CH], y[CH];
                load_channels(rec + 4 + lane * CH, x);
                load_channels(rec + 4 + D + lane * CH, y);
#pragma unroll
                for (int e = 0; e < CH; ++e) {
                    O1[e] = fmaf(wt, x[e], O1[e]);
                    O2[e] = fmaf(wt, y[e], O2[e]);
                }
            }
            if (alone) {
                emit(bh_of(row));
            } else {
                float *dst = recs_of(row) + static_cast<int64_t>(cta - first_cta) * REC;
                if (lane == 0) __stcg(reinterpret_cast<float4 *>(dst), make_float4(big, D1, D2, 0.f));
                store_channels(dst + 4 + lane * CH, O1);
                store_channels(dst + 4 + D + lane * CH, O2);
            }
        }
    }
    __threadfence();
    __syncthreads();
    if (plan.b >= 0 && !alone && warp == w0 && lane == 0) s_arrived[warp] = atomicAdd(a.ws_counters + bh_of(0), 1);
    __syncthreads();
    if (plan.b < 0 || alone || s_arrived[w0] != n_ctas - 1) return;
    __threadfence();
    // last: merge the n_ctas records of every row, 32 at a time
    constexpr int kAhead = FEW ? 16 : 8;
    for (int row = warp - w0; row < n_rows; row += n_seg) {
        const float *recs = recs_of(row);
        warp_merge<D, kAhead, true>(recs, min(n_ctas, 32), lane, big, D1, D2, O1, O2);
        for (int j = 32; j < n_ctas; j += 32) {
            float big2, E1, E2, P1[CH], P2[CH];
            warp_merge<D, kAhead, true>(recs + static_cast<int64_t>(j) * REC, min(n_ctas - j, 32), lane, big2, E1, E2, P1, P2);
            const float top = fmaxf(big, big2), safe = top == -INFINITY ? 0.f : top;
            const float wa = fast_exp2(big - safe), wb = fast_exp2(big2 - safe);
            big = top;
            D1 = wa * D1 + wb * E1;
            D2 = wa * D2 + wb * E2;
#pragma unroll
            for (int e = 0; e < CH; ++e) {
                O1[e] = wa * O1[e] + wb * P1[e];
                O2[e] = wa * O2[e] + wb * P2[e];
            }
        }
        emit(bh_of(row));
    }
    if (warp == w0 && lane == 0) a.ws_counters[bh_of(0)] = 0;   // ready for the next launch on this workspace
}

template <typename T, int D, bool PAGED, bool FEW>
static int launch_decode_gqa(const DecodeArgs &a, cudaStream_t stream) {
    const int n_hgroups = (a.n_rep + 15) / 16;
    constexpr int kSmem = kGqaWarps * GqaSmem<D>::kPerWarp;
    auto kern = decode_gqa_kernel<T, D, PAGED, FEW>;
    {   // the shared-memory opt-in is a per-device function attribute: set it once per device
        constexpr int kMaxDevices = 64;
        static std::mutex mu;
        static bool done[kMaxDevices] = {};
        int dev = -1;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return PLX_ERR_DEVICE;
        std::lock_guard<std::mutex> lock(mu);
        if (!done[dev]) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) {
                (void)cudaGetLastError();
                return PLX_ERR_LAUNCH;
            }
            done[dev] = true;
        }
    }
    const int64_t ctas = (static_cast<int64_t>(a.batch) * a.n_splits + kGqaWarps - 1) / kGqaWarps * a.heads_kv * n_hgroups;
    const cudaError_t st = launch_overlapped(kern, dim3(static_cast<unsigned>(ctas)), kGqaWarps * 32, kSmem, stream, a, n_hgroups);
    count_launch();
    return st == cudaSuccess && cudaGetLastError() == cudaSuccess ? PLX_OK : PLX_ERR_LAUNCH;
}

template <typename T, int D, int HG>
static int launch_decode_hg(const DecodeArgs &a, cudaStream_t stream) {
    constexpr int U = 4;  // key rows per stream and register buffer (two buffers: 8 rows of K and of V in flight)
    dim3 grid(a.n_splits, a.heads_q / HG, a.batch);
    auto kern = a.balanced ? decode_kernel<T, D, HG, U, false, true> : decode_kernel<T, D, HG, U, false, false>;
    const cudaError_t st = launch_overlapped(kern, grid, HG * 32, 0, stream, a);
    count_launch();
    return st == cudaSuccess && cudaGetLastError() == cudaSuccess ? PLX_OK : PLX_ERR_LAUNCH;
}

// number of SMs of the current device (cached per device; 0 on failure)
static int tma_free_sm_count() {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static int cached[kMaxDevices] = {};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    std::lock_guard<std::mutex> lock(mu);
    if (!cached[dev] && cudaDeviceGetAttribute(&cached[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        cached[dev] = 0;
    }
    return cached[dev];
}

// Few (batch, head) pairs, not many keys (the shapes that are bound by latency: the same test as in
// plx_decode_choose_splits) and a split count that is a multiple of eight, at most 256: split groups
// (see decode_kernel).  Both arrangements are correct for any problem; long sweeps stay with one warp per
// split, whose CTAs read contiguous memory.
static bool decode_split_groups(const DecodeArgs &a) {
    const int64_t bh = static_cast<int64_t>(a.batch) * a.heads_q;
    const int64_t n_keys = a.window >= 0 && a.window < a.cache_len ? a.window : a.cache_len;
    return a.n_rep == 1 && a.n_splits >= 8 && a.n_splits % 8 == 0 && a.n_splits <= 256 &&
           bh <= PLX_DECODE_SPLIT_GROUP_MAX_BH && bh * n_keys <= (static_cast<int64_t>(1) << 19);
}

template <typename T, int D>
static int launch_decode_sg(const DecodeArgs &a, cudaStream_t stream) {
    const int n_cta = a.n_splits / 8;
    dim3 grid(n_cta, a.heads_q, a.batch);
    // Up to eight CTAs per (batch, head): one thread-block cluster, merged through distributed shared memory.
    // (Sixteen, beyond the portable size, was measured too: 12.5 us against 10.8 at B = 1, H = 8, 4096 keys.)
    const bool cluster = n_cta == 2 || n_cta == 4 || n_cta == 8;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(n_cta);
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    // When every CTA gets an SM of its own, a warp keeps 16 rows of K and of V in flight per buffer
    // (U = 8, more registers, one CTA per SM); otherwise 8 rows and two CTAs per SM.  The CTAs of a
    // cluster must sit in one GPC, so fewer clusters than (SM count / cluster size) are resident at
    // once: the occupancy calculator gives the number, asked once per device and cluster size.
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return PLX_ERR_DEVICE;
    const int64_t units = static_cast<int64_t>(a.heads_q) * a.batch;
    bool roomy = units * n_cta <= tma_free_sm_count();
    if (cluster) {
        // resident clusters of the U = 8 kernel: 0 = not asked yet, -1 = none / the query failed
        static std::atomic<int> resident[64][4] = {};
        const int slot = n_cta == 2 ? 1 : n_cta == 4 ? 2 : 3;
        int n = resident[dev][slot].load(std::memory_order_acquire);
        if (n == 0) {
            cfg.numAttrs = 2;
            if (cudaOccupancyMaxActiveClusters(&n, decode_kernel<T, D, 8, 8, true, false>, &cfg) != cudaSuccess || n < 1) {
                (void)cudaGetLastError();
                n = -1;
            }
            resident[dev][slot].store(n, std::memory_order_release);
        }
        roomy = roomy && units <= n;
    }
    auto kern = roomy ? decode_kernel<T, D, 8, 8, true, false> : decode_kernel<T, D, 8, 4, true, false>;
    cfg.numAttrs = cluster ? 2 : 1;
    cudaError_t st = cudaLaunchKernelEx(&cfg, kern, a);
    count_launch();
    return st == cudaSuccess && cudaGetLastError() == cudaSuccess ? PLX_OK : PLX_ERR_LAUNCH;
}

template <typename T, int D>
static int launch_decode_t(const DecodeArgs &a, cudaStream_t stream) {
    if (a.n_rep > 8)    // grouped heads: tensor-core kernel
        return a.page_table ? launch_decode_gqa<T, D, true, false>(a, stream) : launch_decode_gqa<T, D, false, false>(a, stream);
    if (a.n_rep >= 2)
        return a.page_table ? launch_decode_gqa<T, D, true, true>(a, stream) : launch_decode_gqa<T, D, false, true>(a, stream);
    if (decode_split_groups(a)) return launch_decode_sg<T, D>(a, stream);
    // adjacent q heads share a CTA (one warp each): the largest group that divides the head count
    if (a.heads_q % 8 == 0) return launch_decode_hg<T, D, 8>(a, stream);
    if (a.heads_q % 4 == 0) return launch_decode_hg<T, D, 4>(a, stream);
    if (a.heads_q % 2 == 0) return launch_decode_hg<T, D, 2>(a, stream);
    return launch_decode_hg<T, D, 1>(a, stream);
}

// The fused sweep + exchange exists in the one-warp-per-split arrangement with at least two splits.
bool decode_fused_exchange_supported(const DecodeArgs &a) {
    return a.n_rep == 1 && a.n_splits >= 2 && !decode_split_groups(a);
}

// From which ratio of the longest row to the mean, in sixteenths, the splits are dealt out by length; 0: never.
// Not for split groups, whose CTAs belong to one row, and not for a key-sharded launch, whose fused and two-launch forms
// have to cut the keys alike.
// Where the parts are large and the launch is bound by HBM, dealing out pays from a small skew on (17): rows from T down
// to T / 3 keys (a skew of 1.5), even parts against dealt out: 32 rows of 4000, 8 : 8 heads, 76 -> 70 us; 16 rows of 8192,
// 32 : 8 heads, 94 -> 76; two rows of 29184 and 19456 (1.2), 64 -> 55.  Elsewhere only from a skew of 2 on (32), since it costs the plan and, with grouped heads, the
// merge inside a CTA: 64 rows of 512, 16 : 2 heads, 11.6 -> 21.0 us; 128 rows of 1000, 8 : 8 heads, 80 -> 87; but where one
// row is ten times the others, those 128 rows took 71 us in even parts against 27.
// `part`, the keys of an even part times head_dim: the lines lie between 250 and 512 keys at head_dim 128 (512 and 1024 at
// 64) with grouped heads, else between 75 and 111; below 64 the wait for the plan is all there is to see (12 rows of 900, 13.5 ->
// 14.7 us).  Also against an even cut of grouped heads: rows that end inside a CTA of another row (3 rows of 1000 keys in 15
// parts, 16 : 2 heads, 20.0 us even, 15.0 dealt out).
static int balance_from(const DecodeArgs &a, int head_dim) {
    if ((!a.seqused && !a.n_lens && !a.cache_start) || a.batch < 2 || a.batch > kBalancedRows || a.n_splits < 2 || a.part_out || a.xch.world != 0 ||
        decode_split_groups(a))
        return 0;
    const int64_t n_keys = a.window >= 0 && a.window < a.cache_len ? a.window : a.cache_len, part = n_keys / a.n_splits * head_dim;
    if (a.n_rep > 1) {
        const bool rows_end_with_ctas = a.n_splits % kGqaWarps == 0 || kGqaWarps % a.n_splits == 0;
        return part < 384 * 128 && rows_end_with_ctas ? 32 : 17;
    }
    if (part < 64 * 128) return 0;
    const bool one_wave = static_cast<int64_t>(a.batch) * a.heads_q * a.n_splits <= 16 * static_cast<int64_t>(tma_free_sm_count());
    return part < 100 * 128 || a.n_splits < 4 || !one_wave ? 32 : 17;
}

int launch_decode(const DecodeArgs &problem, int dtype, int head_dim, cudaStream_t stream) {
    DecodeArgs a = problem;
    a.balanced = balance_from(a, head_dim);
    if (dtype == PLX_BF16) {
        if (head_dim == 128) return launch_decode_t<__nv_bfloat16, 128>(a, stream);
        if (head_dim == 64) return launch_decode_t<__nv_bfloat16, 64>(a, stream);
    } else if (dtype == PLX_FP16) {
        if (head_dim == 128) return launch_decode_t<__half, 128>(a, stream);
        if (head_dim == 64) return launch_decode_t<__half, 64>(a, stream);
    }
    return PLX_ERR_UNSUPPORTED;
}

// The inputs of a captured step into its buffers: q and r by 16-byte copies, the lengths out of the launch
// parameters.  Bound by its launch.  One of these in place of two device copies, a host tensor and its synchronising
// copy: a GraphedDecode call of 4 rows of up to 4096 keys 31.9 -> 21.8 us.
struct StageLens {
    int32_t n[PLX_DECODE_STAGE_LENS];
};
__global__ void __launch_bounds__(256) decode_stage_kernel(uint4 *q, const uint4 *q_src, uint4 *r, const uint4 *r_src, int64_t n16, int32_t *lens,
                                                           const __grid_constant__ StageLens src, int n) {
    grid_wait();
    const int64_t i0 = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x, step = static_cast<int64_t>(gridDim.x) * 256;
    for (int64_t i = i0; i < n16; i += step) {
        if (q_src) q[i] = q_src[i];
        if (r_src) r[i] = r_src[i];
    }
    for (int64_t i = i0; i < n; i += step) lens[i] = src.n[i];
}

int launch_decode_stage(void *q, const void *q_src, void *r, const void *r_src, size_t bytes, int32_t *lens, const int32_t *lens_src, int n,
                        cudaStream_t stream) {
    StageLens src{};
    if (!lens_src) n = 0;
    for (int i = 0; i < n; ++i) src.n[i] = lens_src[i];
    const int64_t n16 = q_src || r_src ? static_cast<int64_t>(bytes / 16) : 0, items = n16 > n ? n16 : n;
    if (items == 0) return PLX_OK;
    const int64_t blocks = (items + 255) / 256;
    const cudaError_t st = launch_overlapped(decode_stage_kernel, dim3(static_cast<unsigned>(blocks < 1024 ? blocks : 1024)), 256, 0, stream,
                                             static_cast<uint4 *>(q), static_cast<const uint4 *>(q_src), static_cast<uint4 *>(r),
                                             static_cast<const uint4 *>(r_src), n16, lens, src, n);
    count_launch();
    return st == cudaSuccess && cudaGetLastError() == cudaSuccess ? PLX_OK : PLX_ERR_LAUNCH;
}

template <typename T, int D>
static int launch_merge_t(const float *parts, int n_parts, int n_records, void *out, cudaStream_t stream) {
    decode_merge_kernel<T, D><<<n_records, D, 0, stream>>>(parts, n_parts, n_records, out);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? PLX_OK : PLX_ERR_LAUNCH;
}

int launch_decode_merge(const float *parts, int n_parts, int n_records, int head_dim, int dtype, void *out,
                        cudaStream_t stream) {
    if (dtype == PLX_BF16) {
        if (head_dim == 128) return launch_merge_t<__nv_bfloat16, 128>(parts, n_parts, n_records, out, stream);
        if (head_dim == 64) return launch_merge_t<__nv_bfloat16, 64>(parts, n_parts, n_records, out, stream);
    } else if (dtype == PLX_FP16) {
        if (head_dim == 128) return launch_merge_t<__half, 128>(parts, n_parts, n_records, out, stream);
        if (head_dim == 64) return launch_merge_t<__half, 64>(parts, n_parts, n_records, out, stream);
    }
    return PLX_ERR_UNSUPPORTED;
}

}  // namespace plx

// ========================================================================= //
// plx_decode_static: decode with the split-KV scratch built into the library,
// for callers that cannot allocate device memory.
// ========================================================================= //
// The scratch of all such calls on a device.  In HOST code this name is only a
// stand-in for the symbol -- it is not a device address and must never be handed
// to a kernel; the address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_decode_static_scratch[PLX_DECODE_STATIC_SCRATCH_BYTES];

// Device address of the array on the CURRENT device, looked up once per device.
static int decode_static_scratch(void **ptr) {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static void *cached[kMaxDevices] = {};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return PLX_ERR_DEVICE;
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] == nullptr) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_decode_static_scratch) != cudaSuccess || p == nullptr) {
            (void)cudaGetLastError();
            return PLX_ERR_DEVICE;
        }
        cached[dev] = p;
    }
    *ptr = cached[dev];
    return PLX_OK;
}

// argument and device checks of plx_decode (defined beside it)
extern "C" int plx_decode_check_args(const plx_decode_problem *p, const void *q, const void *r, const void *k, const void *v,
                                     const void *out);

extern "C" int plx_decode_static(const plx_decode_problem *p, const void *q, const void *r, const void *k,
                                 const void *v, void *out, const int32_t *seqused_k, const int32_t *cache_start,
                                 plx_stream_t stream) {
    size_t need = 0;
    int st = plx_decode_workspace_bytes(p, &need);  // also validates the problem
    if (st != PLX_OK) return st;
    if (p->n_splits == 1)  // a single split publishes nothing: no scratch involved at all
        return plx_decode(p, q, r, k, v, out, seqused_k, cache_start, nullptr, 0, stream);
    if (need > PLX_DECODE_STATIC_SCRATCH_BYTES) return PLX_ERR_STATIC_SCRATCH;
    // everything plx_decode would refuse is refused here, before anything is enqueued on the stream
    if ((st = plx_decode_check_args(p, q, r, k, v, out)) != PLX_OK) return st;
    void *scratch = nullptr;
    if ((st = decode_static_scratch(&scratch)) != PLX_OK) return st;
    // The array keeps whatever the previous call (possibly of another shape) left in it.  Partial
    // records are fully rewritten before they are read; the arrival counters must start at zero.
    const size_t counter_bytes =
        static_cast<size_t>(p->batch) * p->heads_q * (1 + PLX_DECODE_GROUPS(p->n_splits)) * sizeof(int);
    if (cudaMemsetAsync(static_cast<unsigned char *>(scratch) + (need - counter_bytes), 0, counter_bytes,
                        reinterpret_cast<cudaStream_t>(stream)) != cudaSuccess) {
        (void)cudaGetLastError();
        return PLX_ERR_LAUNCH;
    }
    return plx_decode(p, q, r, k, v, out, seqused_k, cache_start, scratch, PLX_DECODE_STATIC_SCRATCH_BYTES, stream);
}

// Blackwell (sm_100a) primitives used by the tcgen05 kernels: mbarrier, TMA
// (cp.async.bulk.tensor), tensor memory (tcgen05.alloc / ld / st), UMMA
// descriptors and tcgen05.mma / commit.  All spin-waits are bounded.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace plx {
namespace sm100 {

// ------------------------------------------------------------------------- //
// error reporting: a kernel that gives up a bounded wait records where.
//
// The record goes to two places: a word in device memory (first error since it was last cleared) and
// its mirror in mapped pinned host memory, which the host can read without synchronising.  Kernels
// never READ either word, so an error left behind by one launch cannot change what a later launch
// does; inside a CTA the roles tell each other to unwind through a flag in shared memory.
// ------------------------------------------------------------------------- //
enum : int { kErrNone = 0, kErrWaitTimeout = 1 };

struct ErrSink {
    int *word;     // device memory
    int *mirror;   // mapped pinned host memory (may be null)
};

__device__ __forceinline__ void report_error(const ErrSink &e, int code) {
    atomicCAS(e.word, 0, code);
    if (e.mirror) {
        *reinterpret_cast<volatile int *>(e.mirror) = code;
        __threadfence_system();
    }
}

// What a bounded wait needs: where to report, and the CTA's abort flag (a 32-bit word in shared memory,
// zero-initialised by the kernel before its roles start).
struct WaitCtx {
    ErrSink sink;
    uint32_t abort_flag;   // shared-memory address
};

__device__ __forceinline__ bool cta_aborted(const WaitCtx &w) {
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(w.abort_flag) : "memory");
    return v != 0;
}
__device__ __forceinline__ void cta_abort(const WaitCtx &w, int code) {
    asm volatile("st.volatile.shared.u32 [%0], %1;\n" ::"r"(w.abort_flag), "r"(1u) : "memory");
    report_error(w.sink, code);
}

// ------------------------------------------------------------------------- //
// mbarrier
// ------------------------------------------------------------------------- //
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::); }

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait.  Returns false when the limit is hit (the error is then recorded and the CTA's abort
// flag raised) or another role of this CTA has already given up; the caller must unwind.
constexpr uint32_t kWaitLimit = 1u << 22;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const WaitCtx &w, int where) {
    // not unrolled: the compiler otherwise makes sixteen copies of the body at each of the ~25 wait sites of a
    // kernel (a fifth of its code size, for no measured difference in time)
#pragma unroll 1
    for (uint32_t it = 0; it < kWaitLimit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 1023u) == 1023u && cta_aborted(w)) return false;
    }
    cta_abort(w, (where << 8) | kErrWaitTimeout);
    return false;
}

// Bounded wait without error reporting (used while unwinding after an error).
__device__ __forceinline__ bool mbar_wait_quiet(uint32_t bar, uint32_t parity) {
#pragma unroll 1
    for (uint32_t it = 0; it < kWaitLimit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// ------------------------------------------------------------------------- //
// TMA: 4-d tiled load global -> shared, completion on an mbarrier (no multicast)
// ------------------------------------------------------------------------- //
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
// the same box into L2 only
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap *map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];\n" ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(map) : "memory");
}

// ------------------------------------------------------------------------- //
// Work items.  One thread of a CTA (the TMA producer) finds the next item and passes it to the other roles through a
// ring in shared memory, so that finding it (a search in cu_seqlens for packed sequences) happens once and ahead of
// time.  Where the work per item is uneven the hardware hands the items out (cluster launch control): the grid has
// one CTA per item, and a running CTA asks for one that has not started ("try_cancel") and does its work.
// ------------------------------------------------------------------------- //
constexpr int kItemSlots = 4, kItemWords = 12;
struct ItemRing {
    uint32_t slots, full, empty;   // shared-memory addresses: kItemSlots records of 48 bytes, and as many barriers each
    // item n, by one thread; false if the ring did not drain in time
    template <typename Item>
    __device__ __forceinline__ bool publish(int n, const Item &it, const WaitCtx &w, int where) const {
        static_assert(sizeof(Item) == 4 * kItemWords, "an item is twelve words");
        const int s = n % kItemSlots;
        if (n >= kItemSlots && !mbar_wait(empty + 8u * s, (n / kItemSlots - 1) & 1, w, where)) return false;
        const uint32_t *x = reinterpret_cast<const uint32_t *>(&it);
#pragma unroll
        for (int i = 0; i < kItemWords; i += 4)
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(slots + 48u * s + 4u * i), "r"(x[i]), "r"(x[i + 1]), "r"(x[i + 2]),
                         "r"(x[i + 3])
                         : "memory");
        mbar_arrive(full + 8u * s);
        return true;
    }
    // item n, by every lane of a warp (whole) or one thread; each reading role arrives once on the slot's `empty`
    template <typename Item>
    __device__ __forceinline__ bool read(int n, Item &it, bool whole, const WaitCtx &w, int where) const {
        const int s = n % kItemSlots;
        bool ok = mbar_wait(full + 8u * s, (n / kItemSlots) & 1, w, where);
        if (whole) ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        uint32_t *x = reinterpret_cast<uint32_t *>(&it);
#pragma unroll
        for (int i = 0; i < kItemWords; i += 4)
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n"
                         : "=r"(x[i]), "=r"(x[i + 1]), "=r"(x[i + 2]), "=r"(x[i + 3])
                         : "r"(slots + 48u * s + 4u * i)
                         : "memory");
        if (whole) __syncwarp();
        if (!whole || (threadIdx.x & 31) == 0) mbar_arrive(empty + 8u * s);
        return true;
    }
};

// Place of item `idx` among n_bh (batch, head) pairs of n_tiles items each, the k-th longest of its pair: inside groups
// of `group` pairs the longest items of all of them come first, so that the last ones to start are short, while the
// CTAs that run together still share a few heads in L2.
__device__ __forceinline__ void longest_first(int idx, int n_tiles, int n_bh, int group, int &bh, int &k) {
    const int first = idx / (group * n_tiles) * group, in = idx - first * n_tiles, n = min(group, n_bh - first);
    bh = first + in % n;
    k = in / n;
}

// Asks for another item; the answer (16 bytes) is there when `bar` has completed its next phase.  One thread, one
// question at a time.
__device__ __forceinline__ void clc_ask(uint32_t answer, uint32_t bar) {
    mbar_expect_tx(bar, 16);
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n" ::"r"(answer), "r"(bar)
                 : "memory");
}
// The block index of the item, or -1 when no more are to be had.
__device__ __forceinline__ int clc_answer(uint32_t answer) {
    uint32_t got, x;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b128 r;\n"
        "mov.u32 %1, 0;\n"
        "ld.shared.b128 r, [%2];\n"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n"
        "}\n"
        : "=r"(got), "=&r"(x)
        : "r"(answer)
        : "memory");
    fence_proxy_async();           // the next answer is written by the async proxy
    return got ? static_cast<int>(x) : -1;
}

// ------------------------------------------------------------------------- //
// tensor memory
// ------------------------------------------------------------------------- //
__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot_smem), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// 32 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// overloads by register count, so that code templated on the number of columns per thread reads the same
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]);
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[32]);
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }
__device__ __forceinline__ void tmem_st_cols(uint32_t taddr, const uint32_t (&r)[8]) { tmem_st8(taddr, r); }
__device__ __forceinline__ void tmem_st_cols(uint32_t taddr, const uint32_t (&r)[16]) { tmem_st16(taddr, r); }
__device__ __forceinline__ void tmem_st_cols(uint32_t taddr, const uint32_t (&r)[32]) { tmem_st32(taddr, r); }

// 16 lanes x 64 columns (32-bit) in the accumulator-fragment arrangement: with g = lane / 4,
// t = lane % 4, register 4k + 2j + e holds TMEM lane (base lane + g + 8j), column 8k + 2t + e.
__device__ __forceinline__ void tmem_ld_16x256b_x8(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_16x256b_x8(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x8.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
// 16 lanes x 32 columns: register 2k + j holds TMEM lane (base lane + g + 8j), column 4k + t.
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// 4 x 4 transpose of 32-bit words inside a quad of lanes (t = lane & 3): on return w[i] holds what
// lane i of the quad had in w[t].
__device__ __forceinline__ void quad_transpose(uint32_t (&w)[4], int t) {
    const bool p = t & 1, q = t & 2;
    // with lane ^ 1: keep the words whose index has the parity of t, trade the other two
    const uint32_t own_lo = p ? w[1] : w[0], own_hi = p ? w[3] : w[2];
    const uint32_t got_lo = __shfl_xor_sync(0xffffffffu, p ? w[0] : w[1], 1);
    const uint32_t got_hi = __shfl_xor_sync(0xffffffffu, p ? w[2] : w[3], 1);
    // with lane ^ 2: keep the pair of index t, trade the other pair
    const uint32_t keep_a = q ? own_hi : own_lo, keep_b = q ? got_hi : got_lo;   // from lanes t, t ^ 1
    const uint32_t far_a = __shfl_xor_sync(0xffffffffu, q ? own_lo : own_hi, 2);  // from lane t ^ 2
    const uint32_t far_b = __shfl_xor_sync(0xffffffffu, q ? got_lo : got_hi, 2);  // from lane t ^ 3
    const uint32_t u0 = p ? keep_b : keep_a, u1 = p ? keep_a : keep_b;
    const uint32_t v0 = p ? far_b : far_a, v1 = p ? far_a : far_b;
    w[0] = q ? v0 : u0;
    w[1] = q ? v1 : u1;
    w[2] = q ? u0 : v0;
    w[3] = q ? u1 : v1;
}

// named barrier for a subset of the CTA's warps
__device__ __forceinline__ void named_barrier_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// ------------------------------------------------------------------------- //
// UMMA descriptors (128-byte swizzle, tiles as TMA writes them: panels of
// [rows][128 B], 8-row groups 1024 B apart, tile base 1024-byte aligned)
// ------------------------------------------------------------------------- //
// 64-bit shared-memory matrix descriptor:
//   [0,14)  start address >> 4        [16,30) leading byte offset >> 4
//   [32,46) stride byte offset >> 4   [46,48) version = 1 (Blackwell)
//   [61,64) layout type: 2 = 128-byte swizzle
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3fffu);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3fffu) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3fffu) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

// 32-bit instruction descriptor for kind::f16 with fp32 accumulation:
//   [4,6) D format 1 = f32   [7,10) A format   [10,13) B format (0 = f16, 1 = bf16)
//   [15] A major, [16] B major (0 = K-major, 1 = MN-major)   [17,23) N >> 3   [24,29) M >> 4
__host__ __device__ constexpr uint32_t umma_idesc(int ab_format, int a_mn_major, int b_mn_major, int m, int n) {
    return (1u << 4) | (static_cast<uint32_t>(ab_format) << 7) | (static_cast<uint32_t>(ab_format) << 10) |
           (static_cast<uint32_t>(a_mn_major) << 15) | (static_cast<uint32_t>(b_mn_major) << 16) |
           (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
        : "memory");
}
// --- lean issue path -------------------------------------------------------
// ONE thread issues every MMA of a CTA, so its instruction count per MMA bounds the
// tensor throughput: a descriptor is kept as two 32-bit halves (the high half is a
// compile-time constant, the low half = address field + immediate offset) and the
// accumulate flag is a template parameter.
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
    return ((smem_addr >> 4) & 0x3fffu) | ((lbo_bytes >> 4) << 16);
}
__host__ __device__ constexpr uint32_t umma_desc_hi(uint32_t sbo_bytes) {
    return ((sbo_bytes >> 4) & 0x3fffu) | (1u << 14) | (2u << 29);   // SBO | version 1 | 128-byte swizzle
}
template <bool ACC>
__device__ __forceinline__ void umma_ss_lean(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                             uint32_t idesc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "setp.ne.b32 p, %6, 0;\n"
        "mov.b64 da, {%1, %2};\n"
        "mov.b64 db, {%3, %4};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(ACC ? 1 : 0)
        : "memory");
}
template <bool ACC>
__device__ __forceinline__ void umma_ts_lean(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 db;\n"
        "setp.ne.b32 p, %5, 0;\n"
        "mov.b64 db, {%2, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(ACC ? 1 : 0)
        : "memory");
}

// True in exactly one lane of a converged warp.  A warp whose lanes all run the issuing loop and
// elect one lane for the MMAs themselves keeps the loop's addresses and descriptors warp-uniform,
// which is what the tcgen05 instructions take their operands from.
__device__ __forceinline__ bool elect_one_sync() {
    uint32_t pred = 0;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "@p mov.s32 %0, 1;\n"
        "}\n"
        : "+r"(pred));
    return pred != 0;
}

// the mbarrier gets one arrival when every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

}  // namespace sm100
}  // namespace plx

// Internal launch interface between the C ABI (plx_abi.cu) and the kernel files.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace plx {

struct TrainArgs;
struct DecodeArgs;
struct ExchangeArgs;

// Are the items of a tcgen05 kernel handed out by the hardware (see ItemRing in plx_sm100.cuh) or dealt out in advance,
// in pairs of a heavy and a light one?  `uneven`: packed sequences and rows of a cache, whose items take as long as the
// lengths say, always by the hardware (32768 tokens in 270 sequences of 1 to 256: fwd 334 -> 269, dk/dv 320 -> 250, dq/dr
// 390 -> 293 us; the fullest CTA of dk/dv had 1.48 times the average work).  Dense problems, where every pair is the same
// work, when the last round of pairs is so empty that it costs more than 4 %.  Measured, dealt out against by hardware:
// waste 23 % (720 items, B = 9, H = 16, L = 548) fwd 63 -> 50, bwd 171 -> 134 us; 16 % (512 items, B = 1, H = 16, L = 4096)
// fwd 142 -> 130, bwd 390 -> 356; 6 % (1536 items, B = 4, H = 16, L = 3000) fwd 316 -> 281, bwd 891 -> 786; at 1.2 % (4096
// items, L = 4096) pairs were 2.7 % faster.
inline bool items_by_hardware(int64_t n_items, int sms, bool uneven) {
    if (n_items <= sms) return false;                      // one item per CTA
    if (uneven) return true;
    const int64_t units = n_items >= 2 * sms ? (n_items + 1) / 2 : n_items, rounds = (units + sms - 1) / sms;
    return 100 * rounds * sms > 104 * units;
}

// Pairs of (batch, head) whose items are interleaved, the longest first (see longest_first): groups of about equal size
// with at least four items per SM, which is enough for the items that end a group to be short.  (One pair at a time left
// the longest items of the last pairs to the end: forward at B = 1, H = 16, L = 4096 145 us dealt out in pairs, 176 so.)
inline int item_group(int n_bh, int n_tiles, int sms) {
    const int64_t groups = static_cast<int64_t>(n_bh) * n_tiles / (4 * static_cast<int64_t>(sms));
    return groups <= 1 ? n_bh : static_cast<int>((n_bh + groups - 1) / groups);
}

// Every kernel launch of this library goes through count_launch() so that
// plx_kernel_launch_count() can report how many ran.
void count_launch();

int launch_train_fwd_mma(const TrainArgs &a, int dtype, int head_dim, cudaStream_t stream);
int launch_train_bwd_mma(const TrainArgs &a, int dtype, int head_dim, int stages, cudaStream_t stream);

// tcgen05 + TMEM + TMA forward; `supported` decides per problem
bool train_fwd_sm100_supported(const TrainArgs &a, int head_dim);
int launch_train_fwd_sm100(const TrainArgs &a, int dtype, int head_dim, cudaStream_t stream);
// the same kernel for several query rows per sequence against a dense or paged KV cache (writes `o` only)
bool train_extend_sm100_supported(const TrainArgs &a, int head_dim);
int launch_train_extend_sm100(const TrainArgs &a, int dtype, int head_dim, cudaStream_t stream);
// Error words of the current device (see sm100::ErrSink): `word` in device memory, `mirror` in mapped
// pinned host memory.  Both null on failure.  The first call on a device allocates the mirror.
struct ErrorWords {
    int *word, *mirror;
};
ErrorWords sm100_error_words();
int sm100_error_word(int *value, bool clear);   // synchronises the device
int sm100_error_peek(int *value, bool clear);   // reads (and optionally clears) the host mirror only: no synchronisation
// tcgen05 backward: stage is PLX_BWD_DQR or PLX_BWD_DKV (the row statistics must already be in a.bst)
bool train_bwd_sm100_supported(const TrainArgs &a, int head_dim);
// `overlap`: the kernel launched just before on this stream is the row statistics (dk/dv) or dk/dv (dq/dr) of the
// same call, and this one may start under its end
int launch_train_bwd_sm100(const TrainArgs &a, int dtype, int head_dim, int stage, bool overlap, cudaStream_t stream);

constexpr int kDecodeGqaWarps = 8;   // warps (independent splits) per CTA of the grouped-query decode kernel
int launch_decode(const DecodeArgs &a, int dtype, int head_dim, cudaStream_t stream);
bool decode_fused_exchange_supported(const DecodeArgs &a);   // see exchange_merge_warp in plx_decode.cu
int launch_decode_exchange_merge(const ExchangeArgs &x, const float *part, int head_dim, int dtype, void *out,
                                 const ErrorWords &err, cudaStream_t stream);
int launch_decode_stage(void *q, const void *q_src, void *r, const void *r_src, size_t bytes, int32_t *lens, const int32_t *lens_src, int n,
                        cudaStream_t stream);
int launch_decode_merge(const float *parts, int n_parts, int n_records, int head_dim, int dtype, void *out,
                        cudaStream_t stream);

}  // namespace plx

// sort.cuh — interface of the in-house stable radix sort (sort.cu).
#pragma once
#include <cstdint>
#include <string>
#include <cuda_runtime.h>

namespace dfsph {

struct SortBuffers {
    uint32_t* keys_a = nullptr;
    uint32_t* vals_a = nullptr;
    uint32_t* keys_b = nullptr;
    uint32_t* vals_b = nullptr;
    uint32_t* workspace = nullptr;  // radix_sort_workspace_words(n_max, 4) words
};

// Workspace: the digit histograms of the passes (256 words each), then what a sort needs cleared.
constexpr uint32_t kSortDigits = 256;
constexpr uint32_t kSortHistWords = 4 * kSortDigits;
size_t radix_sort_workspace_words(uint32_t n_max, int passes);
inline uint32_t* sort_histograms(const SortBuffers& b) { return b.workspace; }
inline uint32_t* sort_clear_begin(const SortBuffers& b) { return b.workspace + kSortHistWords; }
inline size_t sort_clear_words(uint32_t n, int passes) { return radix_sort_workspace_words(n, passes) - kSortHistWords; }

// Message slot of dfsph_last_error(NULL): errors of calls that have no context (dfsph_create and
// the allocation-free entry points). Thread-local.
void set_global_error(const std::string& msg);
// withheld_tile: a tile id whose look-back flags are never published (failure-detection tests: its
// successors' bounded waits run out and set DFSPH_ST_SORT_TIMEOUT; the output is then unspecified
// but every write stays in range). kNoWithheldTile in normal use.
constexpr uint32_t kNoWithheldTile = 0xFFFFFFFFu;
// The key pass has counted the digits into sort_histograms and zeroed sort_clear_words(n, passes) words
// from sort_clear_begin on this stream; the caller zeroes the histograms again after the sort.
void radix_sort_pairs(SortBuffers& b, uint32_t n, int passes, bool iota_values, cudaStream_t stream,
                      uint32_t* status_word, uint64_t* launch_counter, uint32_t** keys_out, uint32_t** vals_out,
                      uint32_t withheld_tile = kNoWithheldTile);

}  // namespace dfsph

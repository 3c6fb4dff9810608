// Launch interface of the sm_100a PairHMM kernels (kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include "program.h"

namespace fgkl {

// Arithmetic of one kernel instantiation.
enum class Kind : int {
  kShortF32 = 0,   // one read of at most 248 bases, FP32, rows-per-lane 1..8
  kOneF32 = 1,     // one read, FP32, rows-per-lane 10..20 (even)
  kOneF64 = 2,     // one read, FP64, priors from a table, rows-per-lane 1..8 and 10..20 (even)
  kOneF32Pd = 3,   // PD-HMM, one read, FP32, rows-per-lane 1..8 and 10..20 (even)
  kOneF64Pd = 4,   // PD-HMM, one read, FP64, same rows
  kPackedF32Pd = 5,  // PD-HMM, two reads per lane set in FP32x2, rows-per-lane 1..8
  // Reads longer than kMaxBlockRead bases: one read against one distinct haplotype, unshared, the
  // rows strip-mined over blocks of 32 * R rows (rows-per-lane R from long_rows).
  kLongF32 = 6,
  kLongF64 = 7,
  kLongF32Pd = 8,
  kLongF64Pd = 9,
  // PD-HMM regions whose reads hold more read bytes than the class bit sets cover: every pair as in
  // the long kinds, with the prior decided by comparing bytes (any read length).
  kGenericF32Pd = 10,
  kGenericF64Pd = 11,
  kQuadF32 = 12,   // up to four reads, two on each half of the lanes in FP32x2, rows-per-lane 2..14 (even)
  kOneF64Codes = 13,  // as kOneF64, priors by comparing haplotype codes (bytes other than A, C, G, T and N)
  kPairF64 = 14,   // up to two reads, one on each half of the lanes in FP64, priors from a table, the quad form's rows
  kPackedF32 = 15,  // two reads of at most 248 bases on all lanes in FP32x2, rows-per-lane 1..8
};
constexpr int kNumKinds = 16;
// Lanes that hold two reads (FP32x2) or one (FP64) in the quad form, reads a warp in FP32x2, its largest
// rows-per-lane and its longest read (the first row of the first lane is padding).
constexpr int kQuadLanes = 16, kQuadReads = 4;
constexpr int kQuadMaxRows = 14;
constexpr int kQuadMaxRead = kQuadLanes * kQuadMaxRows - 1;
// Rows per lane of a read of `len` bases: even values only. Each value is a launch of its own, which ends
// with the GPU partly idle; the padding of the odd ones' reads costs less.
__host__ __device__ constexpr int quad_rows(int len) { return (len / kQuadLanes + 2) / 2 * 2; }

// Longest read a single 32 * R-row block holds (lane 0 is padding: 31 rows per lane x 20).
constexpr int kMaxBlockRead = 620;
// Rows-per-lane values of the strip-mined kinds: 8, 10, 12 and 16 for plain FP32 (kLongF32); 4, 6
// and 8 for the others, whose per-row state (FP64 values, PD branch values) takes more registers.
constexpr int kNumLongRows = 4;
__host__ __device__ constexpr int long_rows_value(int i, bool wide) {
  return wide ? (i == 0 ? 8 : (i == 1 ? 10 : (i == 2 ? 12 : 16))) : (i == 0 ? 4 : (i == 1 ? 6 : 8));
}
__host__ __device__ constexpr int long_rows_count(bool wide) { return wide ? 4 : 3; }
// Rows per lane of a strip-mined read of `len` bases: the value whose blocks waste the fewest
// padding rows (ties: the smaller). Blocks = ceil(len / (32 * R)). `wide`: the plain FP32 kind.
__host__ __device__ inline int long_rows(int len, bool wide) {
  int best = 8;
  unsigned best_rows = 0;
#pragma unroll
  for (int i = 0; i < kNumLongRows; ++i) {
    if (i >= long_rows_count(wide)) break;
    const unsigned r = static_cast<unsigned>(long_rows_value(i, wide));
    const unsigned rows = (static_cast<unsigned>(len) + 32 * r - 1) / (32 * r) * (32 * r);
    if (best_rows == 0 || rows < best_rows) {
      best_rows = rows;
      best = static_cast<int>(r);
    }
  }
  return best;
}
__host__ __device__ inline int long_blocks(int len, int rows) { return (len + 32 * rows - 1) / (32 * rows); }
// Warps a block of the strip-mined kernels at most: one a row block up to kLongWarps; more row blocks run in
// rounds of about equal size.
constexpr int kLongWarps = 8;
inline int long_warps(int row_blocks) {
  const int rounds = (row_blocks + kLongWarps - 1) / kLongWarps;
  return rounds > 0 ? (row_blocks + rounds - 1) / rounds : 1;
}

// Recomputation queue bins, by group and rows-per-lane: reads whose rows one warp holds (0), strip-mined on
// one or two warps a pair (1; 2 for the pairs of byte-compared PD regions), and strip-mined on a warp a row
// block, for the runs that lose few pairs (3, and 4 byte-compared).
constexpr int kRowBins = 21;
constexpr int kQueueGroups = 5;
constexpr int kQueueBins = kQueueGroups * kRowBins;
__host__ __device__ inline int queue_bin(int len, bool generic) {
  if (generic) return 2 * kRowBins + long_rows(len, false);
  if (len > kMaxBlockRead) return kRowBins + long_rows(len, false);
  int rows = (len + 30) / 31;
  if (rows > 8) rows = (rows + 1) & ~1;
  return rows;
}
__host__ __device__ inline int queue_bin_rows(int bin) { return bin % kRowBins; }
__host__ __device__ inline int queue_bin_group(int bin) { return bin / kRowBins; }
// The bin of a single lost pair of a read (a read's whole-program tasks are queue_bin's). `few`: the run lost few
// pairs of reads above 248 bases (few_pairs), so that a pair's row blocks have warps to run side by side on;
// else the warps are worth more on pairs of their own (32 pairs of 540 bases 0.27 against 0.39 ms, 1,000 pairs
// 1.05 against 0.87). In a single block 10 to 14 rows a lane of the plain FP64 form are the faster even then
// (16 pairs of 350 bases: 0.17 against 0.18 ms); those of the PD form spill registers, and reads of 12 and
// more, or that two strip-mined blocks hold with hardly any padding, go strip-mined even when many are lost
// (1,000 pairs of 480 bases: 1.15 against 2.01 ms; 9,134 of 250 bases 3.2 against 4.5; but 5,977 of 300 bases,
// padded to 384 rows, 3.2 against 3.0).
__host__ __device__ inline int queue_pair_bin(int len, bool generic, bool pd, bool few) {
  const int bin = queue_bin(len, generic);
  const int group = queue_bin_group(bin);
  if (group == 0 && bin <= 8) return bin;
  if (few && (group > 0 || bin >= (pd ? 10 : 16))) return (group == 2 ? 4 : 3) * kRowBins + long_rows(len, false);
  return group == 0 && pd && (bin >= 12 || len <= 256) ? kRowBins + long_rows(len, false) : bin;
}
// Lost pairs of reads above 248 bases up to which they are few for a read of this many strip-mined row blocks:
// with more, several warps a pair no longer pay (148 SMs: pairs of 700 bases 0.43 ms at six warps a pair and
// 0.93 at one with 148 pairs, 0.69 and 0.94 with 200, 0.98 and 0.96 with 300; PD pairs of 250 bases at two
// warps 0.29 against 0.37 at one with 400 pairs, 0.58 against 0.47 with 1,000).
__host__ __device__ inline int few_pairs(int sms, int row_blocks) { return row_blocks <= 2 ? 4 * sms : sms + sms / 2; }
// The most pairs that a bin of several warps a pair holds.
inline int few_pairs_most(int sms) { return few_pairs(sms, 1); }

inline bool is_long(Kind k) { return k >= Kind::kLongF32 && k <= Kind::kGenericF64Pd; }
inline bool is_quad(Kind k) { return k == Kind::kQuadF32 || k == Kind::kPairF64; }
inline bool is_pd(Kind k) {
  return k == Kind::kOneF32Pd || k == Kind::kOneF64Pd || k == Kind::kPackedF32Pd || k == Kind::kLongF32Pd ||
         k == Kind::kLongF64Pd || k == Kind::kGenericF32Pd || k == Kind::kGenericF64Pd;
}

// The PD instantiation a PD kind selects.
enum class PdForm : int { kOneF32 = 0, kOneF64 = 1, kPackedF32 = 2 };
inline PdForm pd_form(Kind k) {
  return k == Kind::kOneF64Pd ? PdForm::kOneF64 : (k == Kind::kPackedF32Pd ? PdForm::kPackedF32 : PdForm::kOneF32);
}

struct LaunchArgs {
  BatchView v;
  const Task* tasks;     // this launch's tasks
  int n_tasks;           // host-known count, or the capacity when `count` is set
  const int* count;      // device-side task count (recomputation queues), or nullptr
  int* task_counter;     // zeroed before the launch
  char* scratch;
  size_t scratch_stride; // bytes per warp, strip-mined per block
  int min_accept_plain;  // 1: results below the single-precision threshold are lost
  int only_lost;         // recomputation: a whole-program task writes only pairs whose result is NaN
};

// The pass between the first pass and the recomputation: queues lost pairs.
struct CollectArgs {
  BatchView v;
  Task* queue;           // recomputation queue: (read, distinct haplotype) FP64 tasks, and dense reads
  const int* queue_off;  // per rows-per-lane bin: first queue index (one past the last bin at the end)
  int* queue_tail;       // per bin: tasks queued
  int dense;             // 1 after an FP32 pass: a read lost against a third of its haplotypes or more
                         // is queued once, as a whole-program FP64 task (fgkl lib.rs:495-520)
  int pd;                // 1 in a PD-HMM batch
  int sms;               // of the device (few_pairs)
};

// Rows per lane the instantiations cover.
int max_rows(Kind k);
// Bytes of per-warp scratch one task of this instantiation needs.
size_t scratch_bytes(Kind k, int rows, int max_slots, int max_nodes, int max_segs);
// Resident blocks per SM and threads per block of an instantiation.
void occupancy(Kind k, int rows, int* blocks_per_sm, int* threads_per_block, int warps_per_block = 4);
// Launches one persistent grid of `blocks` blocks.
cudaError_t launch(Kind k, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps_per_block = 4);
// The quad form (quad.cpp): one warp a block, or two for any more.
size_t quad_scratch_bytes(Kind k, int rows, int max_slots, int max_nodes, int max_segs);
void quad_occupancy(Kind k, int rows, int* blocks_per_sm, int* threads_per_block, int warps_per_block);
cudaError_t quad_launch(Kind k, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps_per_block);
// PD-HMM instantiations (pd_kernels.cu).
size_t pd_scratch_bytes(PdForm form, int rows, int max_slots, int max_segs);
void pd_occupancy(PdForm form, int rows, int* blocks_per_sm, int* threads_per_block, int warps_per_block = 4);
cudaError_t pd_launch(PdForm form, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps_per_block = 4);
// Strip-mined kinds (is_long): per-warp scratch for haplotypes of at most `max_hap_len` bases (the
// bottom row a block hands to the next, plus the pair's result), occupancy and launch. The plain
// ones live in kernels.cu, the PD ones in pd_kernels.cu.
size_t long_scratch_bytes(Kind k, int rows, int max_hap_len);
void long_occupancy(Kind k, int rows, int* blocks_per_sm, int* threads_per_block, int warps_per_block);
cudaError_t long_launch(Kind k, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps_per_block);
size_t pd_long_scratch_bytes(Kind k, int rows, int max_hap_len);
void pd_long_occupancy(Kind k, int rows, int* blocks_per_sm, int* threads_per_block, int warps_per_block);
cudaError_t pd_long_launch(Kind k, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps_per_block);

// Launches the lost-pair collection over `n_regions` regions.
cudaError_t launch_collect(const CollectArgs& args, int n_regions, cudaStream_t stream);

// ---- allocation-free entry (file-scope device scratch; see capi.cpp) ----
constexpr size_t kMaxQualTable = 255;  // error-probability entries
constexpr size_t kM2MTable = 32640;    // match-to-match entries

// Per-device state of the allocation-free entry, filled once by noalloc_setup.
struct NoAllocDevice {
  bool ready = false;
  char* scratch = nullptr;  // the file-scope scratch array: header (pair counter), then per-warp slots
  double* err = nullptr;
  double* m2m = nullptr;
  uint8_t* codes = nullptr;
  size_t scratch_bytes = 0, header_bytes = 0, per_warp_bytes = 0;
  int blocks_per_sm[21] = {};
  int sms = 0;
};

// One call's caller-owned device arrays.
struct NoAllocCall {
  const uint8_t *bases, *quals, *ins, *del, *gcp;
  const int64_t* read_off;
  const uint8_t* hap_bases;
  const int64_t* hap_off;
  int n_reads, n_haps;
  double* out;
};

// Rows per lane for reads of at most `max_read_len` bases.
int noalloc_rows(int max_read_len);
// The current device's address of the file-scope scratch array (changes when the device's primary
// context is reset and recreated).
cudaError_t noalloc_scratch_address(char** scratch);
// Resolves the file-scope arrays of the current device and uploads the tables (synchronous).
cudaError_t noalloc_setup(NoAllocDevice* d, const double* err, size_t n_err, const double* m2m, size_t n_m2m,
                          const uint8_t codes[256]);
// Zeroes the pair counter and launches `blocks` blocks on `stream`; allocates nothing.
cudaError_t noalloc_launch(const NoAllocDevice& d, const NoAllocCall& c, int rows, int blocks, cudaStream_t stream);

}  // namespace fgkl

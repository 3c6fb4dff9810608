// sm_100a PairHMM launches: the plain kernel's instantiations of one read a warp and their dispatch, the
// lost-pair collection, the strip-mined form for long reads, and the allocation-free entry. The recurrence
// itself is in plain_kernel.cuh.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "kernels.cuh"
#include "plain_kernel.cuh"

namespace fgkl {

namespace {

// Queues a lost pair in a bin; whether the bin had room.
__device__ __forceinline__ bool queue_pair(const CollectArgs& a, int bin, int read, int hap, int prog) {
  const int slot = atomicAdd(a.queue_tail + bin, 1);
  if (slot >= a.queue_off[bin + 1] - a.queue_off[bin]) return false;
  a.queue[a.queue_off[bin] + slot] = Task{static_cast<int32_t>(blockIdx.x), {read, -1, -1, -1}, queue_bin_rows(bin), hap, prog};
  return true;
}

// Queues what the first pass lost for FP64 recomputation, in the queue bin of the read's form and
// rows-per-lane (queue_bin, queue_pair_bin), one warp per read. After an FP32 pass, a read of a shared program lost
// against at least a third of its haplotypes (duplicates counted, fgkl lib.rs:495-505) is queued once,
// as a whole-program task that fills in every lost pair of the read with one shared sweep, when that
// sweep is the cheaper one; any other lost pair is queued as (read, distinct sorted haplotype), swept
// unshared. Both are FP64 sweeps of fgkl's recurrence and agree to rounding. One block per region;
// nothing to do (one load per block) when no pair was lost.
__global__ void __launch_bounds__(256) collect_kernel(CollectArgs a) {
  if (a.v.counters->lost_pairs == 0) return;
  const Region region = a.v.regions[blockIdx.x];
  const bool generic = (region.flags & kRegionGeneric) != 0;
  const unsigned long long lost_wide = a.v.counters->lost_wide;
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < region.n_reads; r += blockDim.x >> 5) {
    const double* row = a.v.out + region.out_off + static_cast<int64_t>(r) * region.n_haps;
    int lost_all = 0, lost_distinct = 0, lost_steps = 0;
    for (int k = lane; k < region.n_haps; k += 32) {
      const HapInfo info = a.v.haps[region.hap_off + k];
      const bool lost = isnan(row[info.order]);
      lost_all += lost;
      lost_distinct += lost && info.src == k;
      lost_steps += (lost && info.src == k) ? info.len + 32 : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lost_all += __shfl_xor_sync(kFull, lost_all, o);
      lost_distinct += __shfl_xor_sync(kFull, lost_distinct, o);
      lost_steps += __shfl_xor_sync(kFull, lost_steps, o);
    }
    if (lost_all == 0) continue;
    const int read = region.read_off + r;
    const int len = static_cast<int>(a.v.read_off[read + 1] - a.v.read_off[read]);
    const int bin = queue_bin(len, generic);
    const int rows = queue_bin_rows(bin);
    const int cap = a.queue_off[bin + 1] - a.queue_off[bin];
    // The shared sweep must also cost at most two thirds of the unshared ones in wavefront steps:
    // a program that shares little (most PD regions) runs slower whole, in one warp, than its pairs
    // spread over many.
    if (a.dense && bin < kRowBins && 3 * lost_all >= region.n_haps && 3 * region.whole_steps <= 2 * lost_steps) {
      // One task for each of the region's programs; there are no more of them than distinct haplotypes.
      for (int p = lane; p < region.n_progs; p += 32) {
        const int slot = atomicAdd(a.queue_tail + bin, 1);
        if (slot < cap)
          a.queue[a.queue_off[bin] + slot] = Task{static_cast<int32_t>(blockIdx.x), {read, -1, -1, -1}, rows, -1, region.prog + p};
      }
      if (lane == 0) atomicAdd(&a.v.counters->rescue_reads, static_cast<unsigned long long>(lost_distinct));
      continue;
    }
    // Where many are lost, the longest reads' pairs go to several warps each all the same, as many as those
    // bins hold: on one warp such a pair runs on by itself when the others are done.
    const int wide_bin = queue_pair_bin(len, generic, a.pd != 0, true);
    const bool grouped = queue_bin_group(wide_bin) >= 3;
    const int row_blocks = long_blocks(len, queue_bin_rows(wide_bin));
    const bool few = lost_wide <= static_cast<unsigned long long>(few_pairs(a.sms, row_blocks));
    const bool longest = !few && grouped && row_blocks > kLongWarps;
    const int pair_bin = few || !grouped ? wide_bin : queue_pair_bin(len, generic, a.pd != 0, false);
    for (int k = lane; k < region.n_haps; k += 32) {
      const HapInfo info = a.v.haps[region.hap_off + k];
      if (info.src != k || !isnan(row[info.order])) continue;
      bool queued = longest && queue_pair(a, wide_bin, read, k, region.prog);
      if (!queued) queued = queue_pair(a, pair_bin, read, k, region.prog);
      if (queued) atomicAdd(&a.v.counters->rescue_reads, 1ull);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Strip-mined reads (longer than 620 bases; fgkl sizes its row tables by the batch's longest read,
// kernel.rs:485-577, so any length is accepted): one read against one distinct haplotype, unshared,
// from a stream synthesised from the haplotype's codes (the recomputation form above), with the read's
// rows cut into B = ceil(len / 32R) blocks of 32R rows, the padding rows at the top of the first.
//
// A block of W warps runs W consecutive row blocks of a pair as a pipeline: warp w takes what its top row
// needs from the bottom row of warp w - 1's, column by column, from a ring in shared memory, kDelay
// supersteps of kChunk columns behind it; a barrier ends each superstep, so nothing waits on a flag. A
// pair's latency is then n + 64 (W - 1) + 32 steps instead of W (n + 32). More row blocks than warps run
// as several rounds, the last warp's bottom row going through the block's scratch to the first warp of
// the next round. (One warp a pair, its row blocks one after another, left 288 reads of about 1,000 bases
// against 6 haplotypes at 2.6 ms in FP32 and 5.8 ms for the 72 pairs recomputed in FP64, most of the GPU
// idle.)
// ---------------------------------------------------------------------------------------------

template <class P, int R>
constexpr size_t long_smem_per_warp() {
  using L = Layout<P, R>;
  return static_cast<size_t>(L::kPriorCodes) * L::kRp * 32 * sizeof(typename P::V) + kRing * sizeof(Carry<P>);
}

// One superstep of a warp: columns' steps t0 .. t0 + kChunk - 1. kInner: every lane is strictly inside the
// haplotype throughout, so no events and no bounds.
template <class P, int R, bool kInner>
__device__ __forceinline__ void long_superstep(const LaunchArgs& a, const ReadRef* rd, int lane, const FwdRows<P, R, 32>& fr,
                                               typename P::V an, Scratch<P, R>& sc, FwdState<P, R>& st, const uint8_t* seq, int n,
                                               int t0, const Carry<P>* in, Carry<P>* out, int out_mask) {
  const Program prog{};  // unused: the stream is synthesised
#pragma unroll 4
  for (int i = 0; i < kChunk; ++i) {
    const int t = t0 + i;
    const uint32_t e = kInner ? __ldg(seq + t - lane) : synth_entry(seq, n, t - lane);
    const Carry<P> c = in[t & (kRing - 1)];
    st.cX = c.x;
    st.cT = c.t;
    forward_step<P, R, 32, !kInner, true>(a, prog, rd, lane, fr, an, sc, st, n, e);
    const int p = t - 31;  // lane 31's column
    if (lane == 31 && out && (kInner || (p >= 0 && p < n))) out[p & out_mask] = Carry<P>{st.xs, st.ts};
  }
}

template <class P, int R>
__global__ void __launch_bounds__(kLongWarps * 32, (P::kDouble || R > 12 ? 1 : 2)) long_kernel(LaunchArgs a) {
  using V = typename P::V;
  using S = typename P::S;
  using C = Consts<P::kDouble>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_task;
  __shared__ double s_raw[kLongWarps][kMaxReads];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  Carry<P>* const rings = reinterpret_cast<Carry<P>*>(smem_raw);  // [warp][kRing]: what the warp's top row takes
  V* const priors = reinterpret_cast<V*>(rings + warps * kRing) +
                    static_cast<size_t>(w) * ((long_smem_per_warp<P, R>() - kRing * sizeof(Carry<P>)) / sizeof(V));
  Carry<P>* const ring = rings + w * kRing;
  const int count = a.count ? min(*a.count, a.n_tasks) : a.n_tasks;
  // The block's scratch: one carry entry a column, from the last warp of a round to the first of the next.
  Carry<P>* const carry = reinterpret_cast<Carry<P>*>(a.scratch + static_cast<size_t>(blockIdx.x) * a.scratch_stride);
  Scratch<P, R> sc(nullptr, priors, 0, 0, 0);
  sc.priors = priors;
  sc.seg_raw = s_raw[w];
  for (;;) {
    if (threadIdx.x == 0) s_task = atomicAdd(a.task_counter, 1);
    __syncthreads();
    const int task_i = s_task;
    if (task_i >= count) break;
    const Task task = a.tasks[task_i];
    const Region region = a.v.regions[task.region];
    const HapInfo info = a.v.haps[region.hap_off + task.hap];
    const uint8_t* seq = a.v.hap_codes + region.seq_off + info.seq;
    const int n = info.len;
    ReadRef rd[1];
    rd[0].off = a.v.read_off[task.read[0]];
    rd[0].len = static_cast<int>(a.v.read_off[task.read[0] + 1] - rd[0].off);
    const int blocks = long_blocks(rd[0].len, R);
    const int pad0 = 32 * R * blocks - rd[0].len;
    const uint8_t* codes = a.v.code_of_byte + region.code_off;
    // X factor of the read's last row: the accumulated result is the sum of M + mi_n * X^.
    const V an = static_cast<S>(P::kTransformed ? err_prob(a.v, a.v.ins[rd[0].off + rd[0].len - 1]) : 1.0);
    for (int b0 = 0; b0 < blocks; b0 += warps) {
      const int in_round = min(warps, blocks - b0), b = b0 + w;
      const bool on = w < in_round;
      FwdRows<P, R, 32> fr;
      FwdState<P, R> st;
      st.clear();
      Carry<P> next{S(0), S(0)};  // the first warp's input for column t0 + kChunk + lane
      if (on) {
        rd[0].pad = pad0 - 32 * R * b;
        fr.load(a.v, rd, lane, codes, priors);
        if (b == 0) {
          // GATK's row 0 above the first block: M = X = 0, Y = INITIAL / hap_len. Below a padding row
          // nothing reads it.
          if (pad0 == 0) {
            const BracketFactors<P> k(row_model(a.v, rd[0], 0, codes));
            next.t = cell_match<P>(S(0), S(0), static_cast<S>(C::kInitial / n), k.k0, k.k1, k.k2);
          }
        } else if (w == 0 && lane < n) {
          next = carry[lane];
        }
        __syncwarp();
      }
      // The last row block hands nothing on; a round's last warp hands on through the scratch.
      const bool through_ring = w + 1 < in_round;
      Carry<P>* const out = !on || b == blocks - 1 ? nullptr : (through_ring ? ring + kRing : carry);
      const int out_mask = through_ring ? kRing - 1 : -1;
      const int supersteps = (n + 32 + kChunk - 1) / kChunk + (in_round - 1) * kDelay;
      for (int s = 0; s < supersteps; ++s) {
        const int t0 = (s - w * kDelay) * kChunk;
        if (on && t0 >= 0 && t0 < n + 32) {
          if (w == 0) {
            ring[(t0 + lane) & (kRing - 1)] = next;
            const int col = t0 + kChunk + lane;
            if (b > 0 && col < n) next = carry[col];
            __syncwarp();
          }
          if (t0 >= 32 && t0 + kChunk <= n)
            long_superstep<P, R, true>(a, rd, lane, fr, an, sc, st, seq, n, t0, ring, out, out_mask);
          else
            long_superstep<P, R, false>(a, rd, lane, fr, an, sc, st, seq, n, t0, ring, out, out_mask);
        }
        __syncthreads();
      }
    }
    if (w == 0) {
      // Thresholds of an unshared pair (fgkl kernel.rs:897-914): FP32 results below 1e-28 or not finite
      // go to the FP64 recomputation.
      const double raw = s_raw[(blocks - 1) % warps][0];
      bool lost = a.min_accept_plain ? !(raw >= C::kMinAccepted) : (raw != raw);
      if (!P::kDouble) lost |= isinf(raw);
      const double result = lost ? __longlong_as_double(0x7ff8000000000000ll) : log10(raw) - C::kLog10Initial;
      const int read_local = task.read[0] - region.read_off;
      unsigned long long lost_count = 0;
      for (int k = lane; k < region.n_haps; k += 32) {
        const HapInfo h = a.v.haps[region.hap_off + k];
        if (h.src != task.hap) continue;
        a.v.out[region.out_off + static_cast<int64_t>(read_local) * region.n_haps + h.order] = result;
        lost_count += lost;
      }
      if (lost_count) {
        atomicAdd(&a.v.counters->lost_pairs, lost_count);
        atomicAdd(&a.v.counters->lost_wide, lost_count);
      }
    }
    __syncthreads();
  }
}

template <class P, int R>
void occ(int* blocks, int* threads, int warps) {
  *threads = warps * 32;
  static std::atomic<int> cache[3][kMaxDevices];
  *blocks = resident_blocks(pairhmm_kernel<P, R, 32>, warps * Layout<P, R>::kSmemPerWarp, warps * 32, cache[warps_index(warps)],
                            kWarpsPerBlock * Layout<P, R>::kSmemPerWarp);
}

template <class P, int R>
cudaError_t go(int blocks, const LaunchArgs& a, cudaStream_t s, int warps) {
  const size_t smem = warps * Layout<P, R>::kSmemPerWarp;
  pairhmm_kernel<P, R, 32><<<blocks, warps * 32, smem, s>>>(a);
  return cudaGetLastError();
}

template <class P, int R>
struct OccF {
  static int run(int* b, int* t, int warps) {
    occ<P, R>(b, t, warps);
    return 0;
  }
};
template <class P, int R>
struct GoF {
  static cudaError_t run(int blocks, const LaunchArgs& a, cudaStream_t s, int warps) { return go<P, R>(blocks, a, s, warps); }
};
template <class P, int R>
struct SizeF {
  static size_t run(int slots, int nodes, int segs) { return scratch_size<P, R>(slots, nodes, segs); }
};

// Rows-per-lane dispatch over the instantiated values of each kind: FP32 covers the short reads (1..8)
// and the longer ones (10..20 rows, even), FP64 both.
template <template <class, int> class F, class... Args>
auto dispatch(Kind k, int rows, Args&&... args) -> decltype(F<OneF32, 1>::run(args...)) {
  using Ret = decltype(F<OneF32, 1>::run(args...));
#define FGKL_CASE(P, N) \
  case N:               \
    return F<P, N>::run(args...);
  switch (k) {
    case Kind::kShortF32:
      switch (rows) {
        FGKL_CASE(OneF32, 1)
        FGKL_CASE(OneF32, 2)
        FGKL_CASE(OneF32, 3)
        FGKL_CASE(OneF32, 4)
        FGKL_CASE(OneF32, 5)
        FGKL_CASE(OneF32, 6)
        FGKL_CASE(OneF32, 7)
        FGKL_CASE(OneF32, 8)
        default:
          break;
      }
      break;
    case Kind::kPackedF32:
      switch (rows) {
        FGKL_CASE(PackedF32, 1)
        FGKL_CASE(PackedF32, 2)
        FGKL_CASE(PackedF32, 3)
        FGKL_CASE(PackedF32, 4)
        FGKL_CASE(PackedF32, 5)
        FGKL_CASE(PackedF32, 6)
        FGKL_CASE(PackedF32, 7)
        FGKL_CASE(PackedF32, 8)
        default:
          break;
      }
      break;
    case Kind::kOneF32:
      switch (rows) {
        FGKL_CASE(OneF32, 10)
        FGKL_CASE(OneF32, 12)
        FGKL_CASE(OneF32, 14)
        FGKL_CASE(OneF32, 16)
        FGKL_CASE(OneF32, 18)
        FGKL_CASE(OneF32, 20)
        default:
          break;
      }
      break;
    case Kind::kOneF64:
      switch (rows) {
        FGKL_CASE(OneF64Table, 1)
        FGKL_CASE(OneF64Table, 2)
        FGKL_CASE(OneF64Table, 3)
        FGKL_CASE(OneF64Table, 4)
        FGKL_CASE(OneF64Table, 5)
        FGKL_CASE(OneF64Table, 6)
        FGKL_CASE(OneF64Table, 7)
        FGKL_CASE(OneF64Table, 8)
        FGKL_CASE(OneF64Table, 10)
        FGKL_CASE(OneF64Table, 12)
        FGKL_CASE(OneF64Table, 14)
        FGKL_CASE(OneF64Table, 16)
        FGKL_CASE(OneF64Table, 18)
        FGKL_CASE(OneF64Table, 20)
        default:
          break;
      }
      break;
    case Kind::kOneF64Codes:
      switch (rows) {
        FGKL_CASE(OneF64, 1)
        FGKL_CASE(OneF64, 2)
        FGKL_CASE(OneF64, 3)
        FGKL_CASE(OneF64, 4)
        FGKL_CASE(OneF64, 5)
        FGKL_CASE(OneF64, 6)
        FGKL_CASE(OneF64, 7)
        FGKL_CASE(OneF64, 8)
        FGKL_CASE(OneF64, 10)
        FGKL_CASE(OneF64, 12)
        FGKL_CASE(OneF64, 14)
        FGKL_CASE(OneF64, 16)
        FGKL_CASE(OneF64, 18)
        FGKL_CASE(OneF64, 20)
        default:
          break;
      }
      break;
    default:
      break;
  }
#undef FGKL_CASE
  return Ret{};
}

bool valid_long_rows(Kind k, int rows) {
  const bool wide = k == Kind::kLongF32;
  for (int i = 0; i < long_rows_count(wide); ++i)
    if (long_rows_value(i, wide) == rows) return true;
  return false;
}

bool valid_rows(Kind k, int rows) {
  if (is_long(k)) return valid_long_rows(k, rows);
  switch (k) {
    case Kind::kShortF32:
    case Kind::kPackedF32:
      return rows >= 1 && rows <= 8;
    case Kind::kQuadF32:
    case Kind::kPairF64:
      return rows >= 2 && rows <= kQuadMaxRows && rows % 2 == 0;
    case Kind::kOneF32:
      return rows >= 10 && rows <= 20 && rows % 2 == 0;
    case Kind::kOneF64:
    case Kind::kOneF64Codes:
    case Kind::kOneF32Pd:
    case Kind::kOneF64Pd:
      return (rows >= 1 && rows <= 8) || (rows >= 10 && rows <= 20 && rows % 2 == 0);
    case Kind::kPackedF32Pd:
      return rows >= 1 && rows <= 8;
    default:
      break;
  }
  return false;
}

// Strip-mined plain kinds over the rows-per-lane values of long_rows: 8..16 in FP32, 4..8 in FP64.
template <class F>
auto long_rows_narrow(int rows, F&& f) {
  switch (rows) {
    case 4: return f(std::integral_constant<int, 4>{});
    case 6: return f(std::integral_constant<int, 6>{});
    default: return f(std::integral_constant<int, 8>{});
  }
}
template <class F>
auto long_rows_wide(int rows, F&& f) {
  switch (rows) {
    case 8: return f(std::integral_constant<int, 8>{});
    case 10: return f(std::integral_constant<int, 10>{});
    case 12: return f(std::integral_constant<int, 12>{});
    default: return f(std::integral_constant<int, 16>{});
  }
}

template <class P, int R>
void long_occ(int* blocks, int warps) {
  static std::atomic<int> cache[kLongWarps + 1][kMaxDevices];
  *blocks = resident_blocks(long_kernel<P, R>, warps * long_smem_per_warp<P, R>(), warps * 32, cache[warps],
                            kLongWarps * long_smem_per_warp<P, R>());
}

template <class P, int R>
cudaError_t long_go(int blocks, const LaunchArgs& a, cudaStream_t s, int warps) {
  long_kernel<P, R><<<blocks, warps * 32, warps * long_smem_per_warp<P, R>(), s>>>(a);
  return cudaGetLastError();
}

}  // namespace

int max_rows(Kind) { return 20; }

size_t long_scratch_bytes(Kind k, int rows, int max_hap_len) {
  if (!is_long(k) || !valid_long_rows(k, rows)) return 0;
  if (is_pd(k)) return pd_long_scratch_bytes(k, rows, max_hap_len);
  return k == Kind::kLongF64 ? long_scratch_size<OneF64>(max_hap_len) : long_scratch_size<OneF32>(max_hap_len);
}

void long_occupancy(Kind k, int rows, int* blocks, int* threads, int warps) {
  *blocks = 0;
  *threads = warps * 32;
  if (!is_long(k) || !valid_long_rows(k, rows) || warps < 1 || warps > kLongWarps) return;
  if (is_pd(k)) return pd_long_occupancy(k, rows, blocks, threads, warps);
  if (k == Kind::kLongF64)
    long_rows_narrow(rows, [&](auto r) {
      long_occ<OneF64, decltype(r)::value>(blocks, warps);
      return 0;
    });
  else
    long_rows_wide(rows, [&](auto r) {
      long_occ<OneF32, decltype(r)::value>(blocks, warps);
      return 0;
    });
}

cudaError_t long_launch(Kind k, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps) {
  if (!is_long(k) || !valid_long_rows(k, rows) || warps < 1 || warps > kLongWarps) return cudaErrorInvalidValue;
  if (is_pd(k)) return pd_long_launch(k, rows, blocks, args, stream, warps);
  if (k == Kind::kLongF64)
    return long_rows_narrow(rows, [&](auto r) { return long_go<OneF64, decltype(r)::value>(blocks, args, stream, warps); });
  return long_rows_wide(rows, [&](auto r) { return long_go<OneF32, decltype(r)::value>(blocks, args, stream, warps); });
}

size_t scratch_bytes(Kind k, int rows, int max_slots, int max_nodes, int max_segs) {
  if (is_long(k) || !valid_rows(k, rows)) return 0;
  if (is_pd(k)) return pd_scratch_bytes(pd_form(k), rows, max_slots, max_segs);
  if (is_quad(k)) return quad_scratch_bytes(k, rows, max_slots, max_nodes, max_segs);
  return dispatch<SizeF>(k, rows, max_slots, max_nodes, max_segs);
}

void occupancy(Kind k, int rows, int* blocks, int* threads, int warps) {
  *blocks = 0;
  *threads = kWarpsPerBlock * 32;
  if (is_long(k)) return long_occupancy(k, rows, blocks, threads, warps);
  if (!valid_rows(k, rows) || (warps != 1 && warps != 2 && warps != 4)) return;
  if (is_pd(k)) return pd_occupancy(pd_form(k), rows, blocks, threads, warps);
  if (is_quad(k)) return quad_occupancy(k, rows, blocks, threads, warps);
  dispatch<OccF>(k, rows, blocks, threads, warps);
}

cudaError_t launch_collect(const CollectArgs& args, int n_regions, cudaStream_t stream) {
  if (n_regions <= 0) return cudaSuccess;
  collect_kernel<<<n_regions, 256, 0, stream>>>(args);
  return cudaGetLastError();
}

cudaError_t launch(Kind k, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps) {
  if (is_long(k)) return long_launch(k, rows, blocks, args, stream, warps);
  if (!valid_rows(k, rows) || (warps != 1 && warps != 2 && warps != 4)) return cudaErrorInvalidValue;
  if (is_pd(k)) return pd_launch(pd_form(k), rows, blocks, args, stream, warps);
  if (is_quad(k)) return quad_launch(k, rows, blocks, args, stream, warps);
  return dispatch<GoF>(k, rows, blocks, args, stream, warps);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free entry: one region's (read, haplotype) pairs from caller-owned device arrays, each
// pair computed by one warp in FP64 without sharing (the recomputation form of the kernel above),
// with the per-warp scratch -- the segment result the last lane hands to lane 0 -- in a file-scope
// device array instead of an allocated buffer.
// ---------------------------------------------------------------------------------------------

namespace {

constexpr size_t kNoAllocScratchBytes = size_t{2} << 20;  // 2 MiB (FGKL_NOALLOC_SCRATCH_BYTES): header + 8191 warps
constexpr size_t kNoAllocHeader = 256;                    // the 64-bit pair counter (must be 0 at launch)
constexpr size_t kNoAllocPerWarp = 256;                   // one warp's segment result, 256-aligned

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
static __device__ double g_noalloc_err[kMaxQualTable];
static __device__ double g_noalloc_m2m[kM2MTable];
static __device__ uint8_t g_noalloc_codes[256];
static __device__ uint8_t g_noalloc_acgt[256];  // read byte -> acgtn_code, kNoCode for the others

struct NoAllocArgs {
  BatchView v;  // read arrays and offsets, tables, read byte -> code table
  const uint8_t* hap_bases;
  const int64_t* hap_off;
  int n_reads, n_haps;
  unsigned long long* counter;  // pairs claimed so far (64-bit: every warp claims one past the last pair)
  char* scratch;  // kNoAllocPerWarp bytes per warp
  double* out;    // n_reads x n_haps, row-major
};

// Prior code of a haplotype byte: the byte itself, with 'N' and byte kCodeN swapped so that N is
// code kCodeN (matches every read base) and the mapping stays one-to-one. The read table holds the
// same permutation, so a read base matches exactly the haplotype bytes equal to it.
__device__ __forceinline__ uint32_t byte_code(uint32_t b) { return b == 'N' ? kCodeN : (b == kCodeN ? 'N' : b); }

// Prior codes of the bytes A, C, T, G and N for the table form: 0 to 3 by two bits of the letter, N as
// kCodeN.
__device__ __forceinline__ uint32_t acgtn_code(uint32_t b) { return b == 'N' ? kCodeN : (b >> 1) & 3u; }
__device__ __forceinline__ bool is_acgtn(uint32_t b) { return b == 'A' || b == 'C' || b == 'G' || b == 'T' || b == 'N'; }

// One unshared sweep: P is OneF64Table for a haplotype of A, C, G, T and N only (priors from the warp's
// table, read codes from g_noalloc_acgt), else OneF64 (priors by comparing bytes).
template <class P, int R>
__device__ __forceinline__ void forward_unshared(const LaunchArgs& a, const ReadRef* rd, int lane, char* scratch, double* priors,
                                                 const uint8_t* hap, int n) {
  auto code = [](uint32_t b) { return P::kTable ? acgtn_code(b) : byte_code(b); };
  auto entry = [&](int p) -> uint32_t {
    if (p < 0 || p > n) return 0u;
    return (p < n ? code(__ldg(hap + p)) : 0u) | (p == 0 ? EV_BEGIN : 0u) | (p == n ? EV_END : 0u);
  };
  Scratch<P, R> sc(scratch, nullptr, 0, 0, 0);
  sc.priors = priors;
  FwdRows<P, R, 32> fr;
  fr.load(a.v, rd, lane, P::kTable ? g_noalloc_acgt : a.v.code_of_byte, sc.priors);
  __syncwarp();
  const double an = 1.0;  // the plain recurrence: the result is the sum of the last row's M and X
  FwdState<P, R> st;
  st.clear();
  const Program prog{};  // unused: the stream is synthesised from the haplotype bytes
  int t = 0;
  for (; t < 32; ++t) forward_step<P, R, 32>(a, prog, rd, lane, fr, an, sc, st, n, entry(t - lane));
  // Every lane strictly inside the haplotype: no events.
  const uint8_t* seq = hap - lane;
  for (; t + 4 <= n; t += 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) forward_step<P, R, 32, false>(a, prog, rd, lane, fr, an, sc, st, n, code(__ldg(seq + t + i)));
  }
  for (; t < n + 32; ++t) forward_step<P, R, 32>(a, prog, rd, lane, fr, an, sc, st, n, entry(t - lane));
  __syncwarp();
}

template <int R>
constexpr size_t noalloc_smem_per_warp() {
  using L = Layout<OneF64Table, R>;
  return static_cast<size_t>(L::kPriorCodes) * L::kRp * 32 * sizeof(double);
}

template <int R>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, f64_min_blocks(R, false)) noalloc_kernel(NoAllocArgs na) {
  extern __shared__ __align__(16) unsigned char smem_raw[];  // a prior table a warp
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  LaunchArgs a{};
  a.v = na.v;
  const long long pairs = static_cast<long long>(na.n_reads) * na.n_haps;
  for (;;) {
    unsigned long long claimed = 0;
    if (lane == 0) claimed = atomicAdd(na.counter, 1ull);
    const long long t = static_cast<long long>(__shfl_sync(kFull, claimed, 0));
    if (t >= pairs) break;
    const int r = static_cast<int>(t / na.n_haps), h = static_cast<int>(t % na.n_haps);
    ReadRef rd[1];
    rd[0].off = na.v.read_off[r];
    const int64_t read_len = na.v.read_off[r + 1] - rd[0].off;
    const int64_t hap_lo = na.hap_off[h], hap_len = na.hap_off[h + 1] - hap_lo;
    if (read_len <= 0 || read_len > 31 * R || hap_len <= 0 || hap_len > (int64_t{1} << 30)) {
      // Lengths the call's bounds exclude: the pair has no result.
      if (lane == 0) na.out[t] = __longlong_as_double(0x7ff8000000000000ll);
      continue;
    }
    rd[0].len = static_cast<int>(read_len);
    rd[0].pad = 32 * R - rd[0].len;
    char* const scratch = na.scratch + static_cast<size_t>(warp) * kNoAllocPerWarp;
    double* const priors = reinterpret_cast<double*>(smem_raw + (threadIdx.x >> 5) * noalloc_smem_per_warp<R>());
    const uint8_t* const hap = na.hap_bases + hap_lo;
    const int n = static_cast<int>(hap_len);
    bool plain = true;
    for (int i = lane; i < n; i += 32) plain &= is_acgtn(__ldg(hap + i));
    if (__all_sync(kFull, plain))
      forward_unshared<OneF64Table, R>(a, rd, lane, scratch, priors, hap, n);
    else
      forward_unshared<OneF64, R>(a, rd, lane, scratch, priors, hap, n);
    if (lane == 0) na.out[t] = log10(*reinterpret_cast<const double*>(scratch)) - Consts<true>::kLog10Initial;
    __syncwarp();
  }
}

template <int R>
cudaError_t noalloc_go(int blocks, const NoAllocArgs& na, cudaStream_t s) {
  noalloc_kernel<R><<<blocks, kWarpsPerBlock * 32, kWarpsPerBlock * noalloc_smem_per_warp<R>(), s>>>(na);
  return cudaGetLastError();
}

template <int R>
int noalloc_occupancy() {
  int b = 0;
  constexpr size_t smem = kWarpsPerBlock * noalloc_smem_per_warp<R>();
  if (cudaFuncSetAttribute(noalloc_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, noalloc_kernel<R>, kWarpsPerBlock * 32, smem) != cudaSuccess)
    return 0;
  return b;
}

template <class F>
auto noalloc_dispatch(int rows, F&& f) {
  switch (rows) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 5: return f(std::integral_constant<int, 5>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 7: return f(std::integral_constant<int, 7>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 10: return f(std::integral_constant<int, 10>{});
    case 12: return f(std::integral_constant<int, 12>{});
    case 14: return f(std::integral_constant<int, 14>{});
    case 16: return f(std::integral_constant<int, 16>{});
    case 18: return f(std::integral_constant<int, 18>{});
    default: return f(std::integral_constant<int, 20>{});
  }
}

}  // namespace

int noalloc_rows(int max_read_len) {
  int rows = (max_read_len + 30) / 31;
  if (rows > 8) rows = (rows + 1) & ~1;
  return rows;
}

cudaError_t noalloc_scratch_address(char** scratch) {
  return cudaGetSymbolAddress(reinterpret_cast<void**>(scratch), g_noalloc_scratch);
}

cudaError_t noalloc_setup(NoAllocDevice* d, const double* err, size_t n_err, const double* m2m, size_t n_m2m,
                          const uint8_t codes[256]) {
  cudaError_t e;
  if (n_err != kMaxQualTable || n_m2m != kM2MTable) return cudaErrorInvalidValue;
  if ((e = cudaGetSymbolAddress(reinterpret_cast<void**>(&d->scratch), g_noalloc_scratch)) != cudaSuccess) return e;
  if ((e = cudaGetSymbolAddress(reinterpret_cast<void**>(&d->err), g_noalloc_err)) != cudaSuccess) return e;
  if ((e = cudaGetSymbolAddress(reinterpret_cast<void**>(&d->m2m), g_noalloc_m2m)) != cudaSuccess) return e;
  if ((e = cudaGetSymbolAddress(reinterpret_cast<void**>(&d->codes), g_noalloc_codes)) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(g_noalloc_err, err, n_err * sizeof(double))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(g_noalloc_m2m, m2m, n_m2m * sizeof(double))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(g_noalloc_codes, codes, 256)) != cudaSuccess) return e;
  uint8_t acgt[256];
  for (uint8_t& c : acgt) c = kNoCode;
  for (const char b : {'A', 'C', 'T', 'G'}) acgt[static_cast<uint8_t>(b)] = static_cast<uint8_t>((b >> 1) & 3);
  if ((e = cudaMemcpyToSymbol(g_noalloc_acgt, acgt, 256)) != cudaSuccess) return e;
  for (int rows = 1; rows <= 20; ++rows) {
    if (rows > 8 && rows % 2) continue;
    d->blocks_per_sm[rows] = noalloc_dispatch(rows, [](auto r) { return noalloc_occupancy<decltype(r)::value>(); });
    if (d->blocks_per_sm[rows] <= 0) return cudaErrorInvalidDeviceFunction;
  }
  d->scratch_bytes = kNoAllocScratchBytes;
  d->header_bytes = kNoAllocHeader;
  d->per_warp_bytes = kNoAllocPerWarp;
  return cudaSuccess;
}

cudaError_t noalloc_launch(const NoAllocDevice& d, const NoAllocCall& c, int rows, int blocks, cudaStream_t stream) {
  NoAllocArgs na{};
  na.v.bases = c.bases;
  na.v.quals = c.quals;
  na.v.ins = c.ins;
  na.v.del = c.del;
  na.v.gcp = c.gcp;
  na.v.read_off = c.read_off;
  na.v.code_of_byte = d.codes;
  na.v.err_prob = d.err;
  na.v.m2m = d.m2m;
  na.hap_bases = c.hap_bases;
  na.hap_off = c.hap_off;
  na.n_reads = c.n_reads;
  na.n_haps = c.n_haps;
  na.counter = reinterpret_cast<unsigned long long*>(d.scratch);
  na.scratch = d.scratch + d.header_bytes;
  na.out = c.out;
  cudaError_t e = cudaMemsetAsync(d.scratch, 0, sizeof(unsigned long long), stream);  // the pair counter starts at zero
  if (e != cudaSuccess) return e;
  return noalloc_dispatch(rows, [&](auto r) { return noalloc_go<decltype(r)::value>(blocks, na, stream); });
}

}  // namespace fgkl

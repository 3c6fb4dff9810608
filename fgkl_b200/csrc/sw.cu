// sm_100a Smith-Waterman: GATK's SmithWatermanJavaAligner (fgkl crates/smithwaterman/src/reference.rs,
// lib.rs) over a batch of (reference, alternate) pairs, one warp per pair, or several where the pairs are few.
//
// Rows are reference positions, on lanes: lane l holds rows l*R+1 .. l*R+R of a 32*R-row block (R = 4, 8 or
// 16 by the batch's lengths), and a longer reference runs as consecutive blocks. Columns are alternate
// positions, walked as an anti-diagonal wavefront: at step t lane l is at column t - l + 1, and the row
// above arrives from lane l - 1 by shuffle (lane 0 takes GATK's row 0, or, below the first block, the bottom
// row the block above stored per column). Per cell (reference.rs:69-110), in integers:
//   diag  = H(i-1, j-1) + (ref[i] == alt[j] ? match : mismatch)
//   F(i, j) = max over the vertical gap: F(i-1, j) + extend, or H(i-1, j) + open when that is larger
//   E(i, j) = the same along the row from (i, j-1)
//   H = diag when diag >= F and diag >= E, else E when E >= F, else F; never below -1e8.
// Each cell keeps one traceback byte: the direction (diagonal, horizontal, vertical) and whether its
// vertical and its horizontal gap extend the neighbour's (not opened here), from which the traceback
// recovers GATK's gap lengths. The bytes are stored anti-diagonal-major ([block][step][lane][R rows]), so
// each step's stores are one contiguous run. After the fill, the warp picks the end cell from the last
// column and last row with GATK's tie rules and walks back (reference.rs:113-203). For the SoftClip and
// Ignore strategies an alternate that occurs exactly in the reference short-circuits to one match
// (lib.rs:602-607, the last occurrence), found first by the warp testing 32 start positions at a time.
//
// The integer ALU pipe bounds the fill (85% active; 80% in the plain form). Measured on 16,384 pairs of 500 x
// 500 bases: 25 ALU operations a cell, 8 rows a lane 6.31 ms; tagged cells (below) and the traceback by the
// warp 5.14 ms; steps inside the matrix without edge cases, the end cell's row and column kept only where a
// strategy looks there 4.43 ms; 16 rows a lane, so that 500 rows are one block and a step's overhead is shared
// by twice the cells, 3.7 ms (1,100 G cells/s).
#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "dp_common.cuh"
#include "sw.cuh"

namespace fgkl {

namespace {

constexpr int kCutoff = -100000000;  // GATK's MATRIX_MIN_CUTOFF
constexpr int kLowInit = INT_MIN / 2;  // GATK's lowInitValue

// The two cell forms. Plain: GATK's scores as they are, floored at -1e8. Tagged (scores small enough, see
// sw_tagged): a score s is held as 16 s, and the low bits say how it came about, so that the maximum
// that takes the better score also takes GATK's choice among equal ones and its traceback bits:
//   F (vertical gap)   bit 0 set: extends the gap above        (a tie extends)
//   E (horizontal gap) bit 1 set: extends the gap to the left  (a tie extends)
//   H                  8 + .. diagonal, 4 + .. horizontal, else vertical (ties in that order)
// A cell is then five add-and-maximum operations, a base comparison with its select and six bit
// operations instead of 25 compares, selects and adds on the integer ALU pipe, which bounds the kernel.
constexpr int kTagLow = -1200000000;  // below any tagged score, and so that adding a penalty does not overflow
template <bool kTagged>
struct Cell {
  static constexpr int kLow = kTagged ? kTagLow : kLowInit;
  static constexpr uint32_t kExtV = kTagged ? 1 : 4, kExtH = kTagged ? 2 : 8;
  // A traceback byte's direction: 0 diagonal, 1 horizontal, 2 vertical.
  __device__ static uint32_t dir(uint32_t byte) { return kTagged ? 2u - ((byte >> 2) & 3u) : byte & 3u; }

  // The launch's scores, in the form's scale. Tagged scores are held with the penalty of opening a gap from
  // them already added, which both gaps take.
  int open, extend, bias, match, mismatch;
  bool edge;
  __device__ explicit Cell(const SwArgs& a) {
    constexpr int kScale = kTagged ? 16 : 1;
    open = kScale * a.open;
    extend = kScale * a.extend;
    bias = kTagged ? open : 0;
    match = kScale * a.match - bias + (kTagged ? 8 : 0);
    mismatch = kScale * a.mismatch - bias + (kTagged ? 8 : 0);
    edge = a.strategy == kSwIndel || a.strategy == kSwLeadingIndel;
  }
  // H of row 0 at column x, and of column 0 at row x (reference.rs:50-62).
  __device__ int edge_val(int x) const { return bias + ((edge && x >= 1) ? open + (x - 1) * extend : 0); }

  // One column of a lane's rows: rb the reference bases, H and E the rows' values at the column before
  // (updated), ab the alternate's base, dg the diagonal above the top row, (upH, upF) the row above at this
  // column (replaced by the bottom row); the traceback bytes go to `words`.
  template <int kRows>
  __device__ __forceinline__ void column(const int (&rb)[kRows], int (&H)[kRows], int (&E)[kRows], int ab, int dg, int& upH, int& upF,
                                         uint32_t (&words)[kRows / 4]) const {
    uint32_t bytes[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      if constexpr (kTagged) {
        const int F = __viaddmax_s32(upF | 1, extend, upH);
        E[r] = __viaddmax_s32(E[r] | 2, extend, H[r]);
        const int h = __viaddmax_s32(dg, rb[r] == ab ? match : mismatch, __viaddmax_s32(E[r], 4, F));
        // The direction from H, the horizontal flag from E, the vertical one from F; the bits above
        // are not read.
        bytes[r] = (static_cast<uint32_t>(h) & 12u) | (static_cast<uint32_t>(E[r]) & ~12u);
        bytes[r] = (bytes[r] & ~1u) | (static_cast<uint32_t>(F) & 1u);
        dg = H[r];
        H[r] = (h & ~15) + open;
        upH = H[r];
        upF = F;
      } else {
        const int sd = dg + (rb[r] == ab ? match : mismatch);
        // A gap extends the neighbour's unless opening here scores strictly more. H is the largest
        // of the three: the diagonal when it is at least both gaps, else the horizontal gap when it
        // is at least the vertical one (so max(sd, max(E, F)) and one compare decide it).
        const int fe = upF + extend, fo = upH + open;
        const int F = max(fe, fo);
        const int ee = E[r] + extend, eo = H[r] + open;
        E[r] = max(ee, eo);
        const int gap = max(E[r], F);
        const uint32_t dir = sd >= gap ? 0u : (E[r] >= F ? 1u : 2u);
        int h = max(sd, gap);
        h = h > kCutoff ? h : kCutoff;
        bytes[r] = dir | (fe >= fo ? kExtV : 0u) | (ee >= eo ? kExtH : 0u);
        dg = H[r];
        H[r] = h;
        upH = h;
        upF = F;
      }
    }
#pragma unroll
    for (int q = 0; q < kRows / 4; ++q)
      words[q] = __byte_perm(__byte_perm(bytes[4 * q], bytes[4 * q + 1], 0x0040),
                             __byte_perm(bytes[4 * q + 2], bytes[4 * q + 3], 0x0040), 0x5410);
  }
};

__host__ __device__ inline size_t sw_align256(size_t x) { return (x + 255) / 256 * 256; }

// A pair's per-warp scratch, at kRows reference rows a lane.
template <int kRows>
struct SwScratch {
  static constexpr int kBlockRows = 32 * kRows;
  uint8_t* tb;         // [block][step][lane][kRows]
  int32_t* last_col;   // H(i, m), i = 1..n
  int32_t* last_row;   // H(n, j), j = 1..m
  int2* carry;         // bottom row of a block: (H, F) per column
  int m;

  __host__ __device__ static size_t tb_bytes(int64_t n, int64_t m) {
    return sw_align256(static_cast<size_t>((n + kBlockRows - 1) / kBlockRows) * static_cast<size_t>(m + 31) * kBlockRows);
  }
  __host__ __device__ static size_t bytes(int64_t n, int64_t m) {
    return tb_bytes(n, m) + sw_align256(4 * static_cast<size_t>(n)) + sw_align256(4 * static_cast<size_t>(m)) +
           sw_align256(8 * static_cast<size_t>(m));
  }
  __device__ SwScratch(char* base, int n, int m_) : m(m_) {
    tb = reinterpret_cast<uint8_t*>(base);
    last_col = reinterpret_cast<int32_t*>(base + tb_bytes(n, m_));
    last_row = reinterpret_cast<int32_t*>(base + tb_bytes(n, m_) + sw_align256(4 * static_cast<size_t>(n)));
    carry = reinterpret_cast<int2*>(base + tb_bytes(n, m_) + sw_align256(4 * static_cast<size_t>(n)) +
                                    sw_align256(4 * static_cast<size_t>(m_)));
  }
  // Traceback byte of cell (i, j), 1 <= i <= n, 1 <= j <= m.
  __device__ uint32_t at(int i, int j) const {
    const int b = (i - 1) / kBlockRows, rl = (i - 1) - b * kBlockRows, ln = rl / kRows, r = rl % kRows;
    const size_t t = static_cast<size_t>(j - 1) + ln;
    return tb[((static_cast<size_t>(b) * (m + 31) + t) * 32 + ln) * kRows + r];
  }
};

// A lane's traceback bytes of a step, one store.
__device__ __forceinline__ void store_words(uint8_t* dst, const uint32_t (&w)[1]) { *reinterpret_cast<uint32_t*>(dst) = w[0]; }
__device__ __forceinline__ void store_words(uint8_t* dst, const uint32_t (&w)[2]) {
  *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
}
__device__ __forceinline__ void store_words(uint8_t* dst, const uint32_t (&w)[4]) {
  *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}

// The end cell, the traceback and the CIGAR of pair k, by one warp, once the fill's stores are visible to it.
template <bool kTagged, int kRows>
__device__ __forceinline__ void sw_finish(const SwArgs& a, int k, const SwScratch<kRows>& sc, int n, int m, int lane) {
  using C = Cell<kTagged>;
  uint32_t* cig = a.cigar + a.cigar_slot[k];
  // End cell (reference.rs:113-143), by the warp: the best of the last column, ties to the lowest
  // row (the scan runs down the column and keeps the last of equal values), then, unless the
  // strategy is LeadingIndel, the last row's cells, each taking over when higher, or equal and
  // nearer the diagonal (|n - j| below the current |p1 - p2|, ties to the earlier column). Each
  // lane scans a strided share; the shares combine in the scan's order.
  int p1 = 0, p2 = m, seg = 0;
  if (a.strategy == kSwIndel) {
    p1 = n;
  } else {
    int cv = INT_MIN, ci = 0;
    for (int i = lane + 1; i <= n; i += 32) {
      const int cur = sc.last_col[i - 1];
      if (cur >= cv) {
        cv = cur;
        ci = i;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const int ov = __shfl_xor_sync(kFull, cv, o), oi = __shfl_xor_sync(kFull, ci, o);
      if (ov > cv || (ov == cv && oi > ci)) {
        cv = ov;
        ci = oi;
      }
    }
    p1 = ci;
    if (a.strategy != kSwLeadingIndel) {
      int rv = INT_MIN, rj = 0, rd = INT_MAX;
      for (int j = lane + 1; j <= m; j += 32) {
        const int cur = sc.last_row[j - 1], d = abs(n - j);
        if (cur > rv || (cur == rv && d < rd)) {
          rv = cur;
          rj = j;
          rd = d;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const int ov = __shfl_xor_sync(kFull, rv, o), oj = __shfl_xor_sync(kFull, rj, o), od = __shfl_xor_sync(kFull, rd, o);
        if (ov > rv || (ov == rv && (od < rd || (od == rd && oj < rj)))) {
          rv = ov;
          rj = oj;
          rd = od;
        }
      }
      if (rv > cv || (rv == cv && rd < abs(ci - m))) {
        p1 = n;
        p2 = rj;
        seg = m - rj;
      }
    }
  }

  // Traceback (reference.rs:144-203), by the warp: 32 cells of a diagonal run, or of a gap, at a time (one
  // lane following one cell after another waited on a load for each). Elements last to first, reversed at
  // the end; lane 0 writes them.
  int e = 0;
  auto put = [&](int len, uint32_t op) {
    if (lane == 0) cig[e] = (static_cast<uint32_t>(len) << 4) | op;
    ++e;
  };
  if (seg > 0 && a.strategy == kSwSoftClip) {
    put(seg, kSwOpS);
    seg = 0;
  }
  uint32_t state = kSwOpM;
  do {
    // The diagonal from (p1, p2): lane l looks at the l-th cell up it.
    const int i = p1 - lane, j = p2 - lane;
    const bool in = i > 0 && j > 0;
    const uint32_t dir = in ? C::dir(sc.at(i, j)) : 3u;
    const uint32_t here = __shfl_sync(kFull, dir, 0);
    uint32_t next;
    int step = 0;
    if (here == 0) {
      next = kSwOpM;
      const unsigned off_diagonal = __ballot_sync(kFull, dir != 0);
      step = off_diagonal ? __ffs(off_diagonal) - 1 : 32;
      p1 -= step;
      p2 -= step;
    } else {
      // GATK's gap length: one more than the run of extending cells before this one (the first row or
      // column always opens).
      const bool vertical = here == 2;
      next = vertical ? kSwOpD : kSwOpI;
      const int from = vertical ? p1 : p2;
      unsigned opens = 0;
      while (!opens) {
        const int q = from - step - lane;
        const bool extends = q > 1 && (sc.at(vertical ? q : p1, vertical ? p2 : q) & (vertical ? C::kExtV : C::kExtH)) != 0;
        opens = __ballot_sync(kFull, !extends);
        step += opens ? __ffs(opens) - 1 : 32;
      }
      ++step;
      if (vertical)
        p1 -= step;
      else
        p2 -= step;
    }
    if (next == state) {
      seg += step;
    } else {
      if (seg > 0) put(seg, state);
      seg = step;
      state = next;
    }
  } while (p1 > 0 && p2 > 0);
  int off = 0;
  if (a.strategy == kSwSoftClip) {
    put(seg, state);
    if (p2 > 0) put(p2, kSwOpS);
    off = p1;
  } else if (a.strategy == kSwIgnore) {
    put(seg + p2, state);
    off = p1 - p2;
  } else {
    put(seg, state);
    if (p1 > 0)
      put(p1, kSwOpD);
    else if (p2 > 0)
      put(p2, kSwOpI);
  }
  if (lane == 0) {
    for (int x = 0, y = e - 1; x < y; ++x, --y) {
      const uint32_t tmp = cig[x];
      cig[x] = cig[y];
      cig[y] = tmp;
    }
    a.count[k] = e;
    a.offset[k] = off;
  }
}

// The exact-substring shortcut of SoftClip and Ignore (reference.rs:15-23): the last occurrence of the
// alternate. Whether pair k is done with it.
__device__ __forceinline__ bool sw_substring(const SwArgs& a, int k, const uint8_t* ref, const uint8_t* alt, int n, int m, int lane) {
  if (!((a.strategy == kSwSoftClip || a.strategy == kSwIgnore) && m <= n)) return false;
  for (int start = n - m; start >= 0; start -= 32) {
    const int s = start - lane;
    bool ok = s >= 0;
    for (int q = 0; ok && q < m; ++q) ok = __ldg(ref + s + q) == __ldg(alt + q);
    const unsigned hits = __ballot_sync(kFull, ok);
    if (hits) {
      if (lane == 0) {
        a.cigar[a.cigar_slot[k]] = (static_cast<uint32_t>(m) << 4) | kSwOpM;
        a.count[k] = 1;
        a.offset[k] = start - (__ffs(hits) - 1);
      }
      __syncwarp();
      return true;
    }
  }
  return false;
}

// Resident blocks of four warps per SM: what the registers of kRows rows leave room for.
constexpr int sw_min_blocks(int rows) { return rows <= 8 ? 8 : 5; }

template <bool kTagged, int kRows>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, sw_min_blocks(kRows)) sw_kernel(SwArgs a) {
  using C = Cell<kTagged>;
  constexpr int kBlockRows = 32 * kRows;
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  char* const base = a.scratch + static_cast<size_t>(warp) * a.stride;
  const C p(a);
  // The end cell is looked for in the last column (not for Indel) and the last row (SoftClip and Ignore).
  const bool keep_col = a.strategy != kSwIndel, keep_row = a.strategy == kSwSoftClip || a.strategy == kSwIgnore;
  for (;;) {
    int task = 0;
    if (lane == 0) task = atomicAdd(a.counter, 1);
    task = __shfl_sync(kFull, task, 0);
    if (task >= a.n_pairs) break;
    const int k = a.order ? a.order[task] : task;
    const uint8_t* ref = a.ref + a.ref_off[k];
    const uint8_t* alt = a.alt + a.alt_off[k];
    const int n = static_cast<int>(a.ref_off[k + 1] - a.ref_off[k]);
    const int m = static_cast<int>(a.alt_off[k + 1] - a.alt_off[k]);

    if (sw_substring(a, k, ref, alt, n, m, lane)) continue;

    // The fill, one row block after another.
    SwScratch<kRows> sc(base, n, m);
    const int blocks = (n + kBlockRows - 1) / kBlockRows;
    const int last_r = (n - 1) % kRows;  // row n among its lane's rows
    for (int b = 0; b < blocks; ++b) {
      const int top = b * kBlockRows + lane * kRows + 1;  // the lane's first row (1-based)
      int rb[kRows], H[kRows], E[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        rb[r] = top + r <= n ? static_cast<int>(__ldg(ref + top + r - 1)) : -1;
        H[r] = 0;
        E[r] = C::kLow;
      }
      const bool row_here = keep_row && n >= top && n < top + kRows;
      int dH = 0;                  // H of the row above at the previous column (the top row's diagonal)
      int bH = 0, bF = C::kLow;    // this lane's bottom row at its last column, for the lane below
      uint8_t* tbb = sc.tb + (static_cast<size_t>(b) * (m + 31) * 32 + lane) * kRows;
      // Lane 0's row above and every lane's base, loaded a step ahead.
      int2 above = make_int2(p.edge_val(1), C::kLow);
      if (b > 0 && lane == 0) above = sc.carry[0];
      int base_next = lane == 0 ? static_cast<int>(__ldg(alt)) : 0;
      // One step. kInner: every lane is past column 1 and before column m.
      auto step = [&](auto inner, int t) {
        constexpr bool kInner = decltype(inner)::value;
        const int j = t - lane + 1;
        int uH = __shfl_up_sync(kFull, bH, 1), uF = __shfl_up_sync(kFull, bF, 1);
        const bool active = kInner || (j >= 1 && j <= m);
        const int ab = base_next;
        if (kInner || (j >= 0 && j < m)) base_next = static_cast<int>(__ldg(alt + j));
        if (lane == 0) {
          uH = above.x;
          uF = above.y;
          if (b == 0)
            above.x = p.edge_val(j + 1);
          else if (j < m)
            above = sc.carry[j];
        }
        if (!kInner && j == 1) {
          // Column 0: GATK's edge values, no horizontal gap yet.
#pragma unroll
          for (int r = 0; r < kRows; ++r) {
            H[r] = p.edge_val(top + r);
            E[r] = C::kLow;
          }
          dH = p.edge_val(top - 1);
        }
        uint32_t words[kRows / 4] = {};
        if (active) {
          int upH = uH, upF = uF;
          p.template column<kRows>(rb, H, E, ab, dH, upH, upF, words);
          bH = upH;
          bF = upF;
          // The last row and the last column, for the end cell: the lane holding the reference's last
          // row stores its H at every column, and each lane stores its rows once, at the last column.
          if (row_here) {
            // H[last_r], halving the candidates by a bit of last_r at a time (the same in every lane).
            int v[kRows];
#pragma unroll
            for (int r = 0; r < kRows; ++r) v[r] = H[r];
#pragma unroll
            for (int half = kRows / 2; half > 0; half /= 2)
#pragma unroll
              for (int r = 0; r < half; ++r) v[r] = (last_r & half) ? v[r + half] : v[r];
            sc.last_row[j - 1] = v[0];
          }
          if (!kInner && keep_col && j == m) {
#pragma unroll
            for (int r = 0; r < kRows; ++r)
              if (top + r <= n) sc.last_col[top + r - 1] = H[r];
          }
          if (lane == 31 && b + 1 < blocks) sc.carry[j - 1] = make_int2(bH, bF);
        }
        dH = uH;
        store_words(tbb + static_cast<size_t>(t) * kBlockRows, words);
      };
      // Steps 32 .. m - 2 are inside in every lane.
      int t = 0;
      for (; t < min(32, m + 31); ++t) step(std::false_type{}, t);
#pragma unroll 2
      for (; t <= m - 2; ++t) step(std::true_type{}, t);
      for (; t < m + 31; ++t) step(std::false_type{}, t);
      __syncwarp();
    }
    __threadfence_block();
    __syncwarp();
    sw_finish<kTagged, kRows>(a, k, sc, n, m, lane);
    __syncwarp();
  }
}

// The same fill with a pair's row blocks on the warps of a block, for batches of few pairs: a lone warp is
// bound by its scheduler's ALU pipe (0.4 us a step of 16 rows), and the other three are idle. Warp w runs row
// block w of a round, kPipeDelay supersteps of 32 columns behind the one above, whose bottom row it takes
// from a ring in shared memory; a barrier ends each superstep. At superstep s a warp reads ring entries up
// to (s - kPipeDelay w) 32 + 31, of which the warp above wrote all up to 32 (s - kPipeDelay (w - 1)) - 32
// before, and writes meanwhile at most 96 entries past the oldest one needed. Rounds hand on through the
// pair's carry row.
constexpr int kPipeRows = 4, kPipeWarps = 8, kPipeDelay = 2, kPipeRing = 128;

template <bool kTagged>
__global__ void __launch_bounds__(kPipeWarps * 32, 2) sw_pipe_kernel(SwArgs a) {
  using C = Cell<kTagged>;
  constexpr int kRows = kPipeRows, kBlockRows = 32 * kRows;
  __shared__ int2 rings[kPipeWarps][kPipeRing];
  __shared__ int s_task, s_done;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  char* const base = a.scratch + static_cast<size_t>(blockIdx.x) * a.stride;
  const C p(a);
  const bool keep_col = a.strategy != kSwIndel, keep_row = a.strategy == kSwSoftClip || a.strategy == kSwIgnore;
  for (;;) {
    if (threadIdx.x == 0) s_task = atomicAdd(a.counter, 1);
    __syncthreads();
    const int task = s_task;
    if (task >= a.n_pairs) break;
    const int k = a.order ? a.order[task] : task;
    const uint8_t* ref = a.ref + a.ref_off[k];
    const uint8_t* alt = a.alt + a.alt_off[k];
    const int n = static_cast<int>(a.ref_off[k + 1] - a.ref_off[k]);
    const int m = static_cast<int>(a.alt_off[k + 1] - a.alt_off[k]);
    if (w == 0) {
      const bool done = sw_substring(a, k, ref, alt, n, m, lane);
      if (lane == 0) s_done = done;
    }
    __syncthreads();
    if (s_done) {
      __syncthreads();  // before the next pair's s_task and s_done
      continue;
    }
    SwScratch<kRows> sc(base, n, m);
    const int blocks = (n + kBlockRows - 1) / kBlockRows;
    const int last_r = (n - 1) % kRows;
    for (int b0 = 0; b0 < blocks; b0 += warps) {
      const int in_round = min(warps, blocks - b0), b = b0 + w;
      const bool on = w < in_round, hands_on = on && b + 1 < blocks, through_ring = w + 1 < in_round;
      const int top = b * kBlockRows + lane * kRows + 1;
      int rb[kRows], H[kRows], E[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        rb[r] = top + r <= n ? static_cast<int>(__ldg(ref + top + r - 1)) : -1;
        H[r] = 0;
        E[r] = C::kLow;
      }
      const bool row_here = keep_row && n >= top && n < top + kRows;
      int dH = 0, bH = 0, bF = C::kLow;
      uint8_t* const tbb = sc.tb + (static_cast<size_t>(b) * (m + 31) * 32 + lane) * kRows;
      const int supersteps = (m + 31 + 31) / 32 + (in_round - 1) * kPipeDelay;
      for (int s = 0; s < supersteps; ++s) {
        const int t0 = (s - w * kPipeDelay) * 32;
        if (on && t0 >= 0 && t0 < m + 31) {
          if (w == 0) {
            // The row above for columns t0 + 1 .. t0 + 32: GATK's row 0, or the round above's bottom row.
            const int c = t0 + lane;
            int2 above = make_int2(p.edge_val(c + 1), C::kLow);
            if (b > 0 && c < m) above = sc.carry[c];
            rings[0][c & (kPipeRing - 1)] = above;
            __syncwarp();
          }
          const int t1 = min(t0 + 32, m + 31);
          for (int t = t0; t < t1; ++t) {
            const int j = t - lane + 1;
            int uH = __shfl_up_sync(kFull, bH, 1), uF = __shfl_up_sync(kFull, bF, 1);
            const int2 above = rings[w][t & (kPipeRing - 1)];
            if (lane == 0) {
              uH = above.x;
              uF = above.y;
            }
            if (j == 1) {
              // Column 0: GATK's edge values, no horizontal gap yet.
#pragma unroll
              for (int r = 0; r < kRows; ++r) {
                H[r] = p.edge_val(top + r);
                E[r] = C::kLow;
              }
              dH = p.edge_val(top - 1);
            }
            uint32_t words[kRows / 4] = {};
            if (j >= 1 && j <= m) {
              int upH = uH, upF = uF;
              p.template column<kRows>(rb, H, E, static_cast<int>(__ldg(alt + j - 1)), dH, upH, upF, words);
              bH = upH;
              bF = upF;
              if (row_here) sc.last_row[j - 1] = last_r == 0 ? H[0] : last_r == 1 ? H[1] : last_r == 2 ? H[2] : H[3];
              if (keep_col && j == m) {
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                  if (top + r <= n) sc.last_col[top + r - 1] = H[r];
              }
              if (lane == 31 && hands_on) {
                if (through_ring)
                  rings[w + 1][(j - 1) & (kPipeRing - 1)] = make_int2(bH, bF);
                else
                  sc.carry[j - 1] = make_int2(bH, bF);
              }
            }
            dH = uH;
            store_words(tbb + static_cast<size_t>(t) * kBlockRows, words);
          }
        }
        __syncthreads();
      }
    }
    if (w == 0) sw_finish<kTagged, kRows>(a, k, sc, n, m, lane);
    __syncthreads();
  }
}

// Packs every pair's CIGAR elements (counts[k] of them from cigar_slot[k]) into one dense run,
// pair after pair, so the host downloads only the elements the batch produced rather than every
// slot's capacity. One block: each thread sums a contiguous share of the counts, the block scans the
// 1024 sums, each thread then copies its share's pairs.
constexpr int kCompactThreads = 1024;
__global__ void __launch_bounds__(kCompactThreads) sw_compact_kernel(const uint32_t* cigar, const int64_t* slot, const int32_t* count,
                                                                     int n_pairs, uint32_t* packed) {
  __shared__ int64_t warp_sum[kCompactThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t share = (static_cast<int64_t>(n_pairs) + kCompactThreads - 1) / kCompactThreads;
  const int64_t lo = min(static_cast<int64_t>(n_pairs), tid * share), hi = min(static_cast<int64_t>(n_pairs), lo + share);
  int64_t own = 0;
  for (int64_t k = lo; k < hi; ++k) own += count[k];
  // Exclusive scan of the per-thread sums: within each warp, then over the warps.
  int64_t incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t v = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[w] = incl;
  __syncthreads();
  if (w == 0) {
    int64_t ws = warp_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t v = __shfl_up_sync(kFull, ws, o);
      if (lane >= o) ws += v;
    }
    warp_sum[lane] = ws;  // inclusive over the warps
  }
  __syncthreads();
  int64_t pos = (w > 0 ? warp_sum[w - 1] : 0) + incl - own;
  for (int64_t k = lo; k < hi; ++k) {
    const uint32_t* src = cigar + slot[k];
    for (int i = 0; i < count[k]; ++i) packed[pos + i] = src[i];
    pos += count[k];
  }
}

}  // namespace

bool sw_tagged(int64_t longest, int match, int mismatch, int open, int extend) {
  int64_t most = 0;
  for (const int64_t v : {int64_t{match}, int64_t{mismatch}, int64_t{open}, int64_t{extend}}) most = std::max(most, v < 0 ? -v : v);
  // No score or gap is further from zero than `most` a row and column; 16 times that and a further penalty
  // must stay above kTagLow, and above the plain form's floor, so that the floor is never met.
  return most * (longest + 2) <= 50000000;
}

namespace {
template <class F>
auto sw_at(int rows, F&& f) {
  switch (rows) {
    case 4: return f(std::integral_constant<int, 4>{});
    case 8: return f(std::integral_constant<int, 8>{});
    default: return f(std::integral_constant<int, 16>{});
  }
}
}  // namespace

size_t sw_scratch_bytes(int rows, int64_t ref_len, int64_t alt_len) {
  return sw_at(rows, [&](auto r) { return SwScratch<decltype(r)::value>::bytes(ref_len, alt_len); });
}

cudaError_t sw_compact(const uint32_t* cigar, const int64_t* slot, const int32_t* count, int n_pairs, uint32_t* packed,
                       cudaStream_t stream) {
  if (n_pairs <= 0) return cudaSuccess;
  sw_compact_kernel<<<1, kCompactThreads, 0, stream>>>(cigar, slot, count, n_pairs, packed);
  return cudaGetLastError();
}

void sw_occupancy(int rows, bool tagged, int* blocks_per_sm, int* threads_per_block) {
  *threads_per_block = kWarpsPerBlock * 32;
  sw_at(rows, [&](auto r) {
    constexpr int R = decltype(r)::value;
    static std::atomic<int> cache[2][kMaxDevices];
    *blocks_per_sm = tagged ? resident_blocks(sw_kernel<true, R>, 0, kWarpsPerBlock * 32, cache[1])
                            : resident_blocks(sw_kernel<false, R>, 0, kWarpsPerBlock * 32, cache[0]);
    return 0;
  });
}

cudaError_t sw_launch(int rows, int blocks, const SwArgs& a, cudaStream_t stream) {
  sw_at(rows, [&](auto r) {
    constexpr int R = decltype(r)::value;
    if (a.tagged)
      sw_kernel<true, R><<<blocks, kWarpsPerBlock * 32, 0, stream>>>(a);
    else
      sw_kernel<false, R><<<blocks, kWarpsPerBlock * 32, 0, stream>>>(a);
    return 0;
  });
  return cudaGetLastError();
}

void sw_pipe_occupancy(bool tagged, int warps, int* blocks_per_sm) {
  static std::atomic<int> cache[2][kPipeWarps + 1][kMaxDevices];
  *blocks_per_sm = tagged ? resident_blocks(sw_pipe_kernel<true>, 0, warps * 32, cache[1][warps])
                          : resident_blocks(sw_pipe_kernel<false>, 0, warps * 32, cache[0][warps]);
}

int sw_pipe_warps(int64_t longest_ref) {
  const int64_t row_blocks = (longest_ref + 32 * kPipeRows - 1) / (32 * kPipeRows);
  const int64_t rounds = (row_blocks + kPipeWarps - 1) / kPipeWarps;
  return static_cast<int>((row_blocks + rounds - 1) / rounds);
}

size_t sw_pipe_scratch_bytes(int64_t ref_len, int64_t alt_len) { return SwScratch<kPipeRows>::bytes(ref_len, alt_len); }

cudaError_t sw_pipe_launch(int warps, int blocks, const SwArgs& a, cudaStream_t stream) {
  if (a.tagged)
    sw_pipe_kernel<true><<<blocks, warps * 32, 0, stream>>>(a);
  else
    sw_pipe_kernel<false><<<blocks, warps * 32, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace fgkl

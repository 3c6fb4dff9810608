#pragma once
// The sm_100a plain PairHMM kernel: a warp per task of one to four reads of a region, read rows on lanes,
// the program's column stream walked as an anti-diagonal wavefront.
//
// Rows. A group of G lanes holds a read (two in FP32x2). Lane l of the group holds rows l*R .. l*R+R-1 of
// a G*R-row block whose LAST row is the read's last row; at least the block's first row is padding.
// Padding rows have zero transitions and priors and a deletion chain of 1: they keep M = X = 0 and
// Y = INITIAL / hap_len, i.e. they reproduce row 0 of GATK's matrix, and the row just above the read
// plays row 0. At loop step t lane l is at stream position t - l (forward) or t - (G - 1 - l) (backward).
//
// What crosses lanes. The lane above computes what the lane below needs of its bottom row: the new
// insertion value of the lane's top row, and the bracket of that row's match value for the next column
// (two shuffles a step instead of the bottom row's M, X and Y, and no above-row state to keep, store in
// snapshots or reload).
//
// Three forms. One read on all 32 lanes (G = 32) has the shortest steps and serves small batches, long reads
// and the recomputation. Four reads on two groups of 16 lanes in FP32x2 (the quad form) have half the steps that an
// event spans and half the shuffles, selects and loop overhead a cell; at R = 10 they need 255 registers
// and 21 KB of shared memory a warp, 8 warps an SM. Measured on 54,000 reads of 151 bases (1,024 uneven
// regions): 20.5 ms, 2,750 G cells/s (the FP32 pipe 58% active without events, where it reaches 4,080);
// two reads on 32 lanes in FP32x2 26.6 ms; two on 16 lanes in scalar FP32 at 16 warps an SM 23.2 ms; four
// on 8 lanes in scalar FP32 23.3 ms. Two reads on 32 lanes serve full batches where the quad form does not
// fit: regions whose reads leave its slots empty, and reads of 224 to 248 bases (512 regions of 54 reads of
// 236 bases: 9.8 ms, one a warp 10.4).
// In FP64 the same form holds two reads, one on each half of the lanes.
//
// Forward recurrence per cell (GATK LoglessPairHMM, fgkl kernel.rs:1011-1013):
//   M = prior * (mm*M(i-1,j-1) + im*(X(i-1,j-1) + Y(i-1,j-1)))
//   X = mi*M(i-1,j) + ii*X(i-1,j)          Y = md*M(i,j-1) + dd*Y(i,j-1)
// The FP32 kernels carry X/mi and Y/md (per-row constants) instead of X and Y: every term stays
// positive, the X and Y updates become one FMA each. They also fold each row's mm into its priors
// (M = (prior*mm) * (M(i-1,j-1) + k1*X^ + k2*Y^)), 5 FP32 operations per cell instead of 8. An
// overflow this could cause for extreme gap-open ratios surfaces as a non-finite result, which is
// recomputed in FP64 with the plain recurrence.
//
// Backward recurrence (suffix sharing, fgkl kernel.rs:1080-1088), row i from row i+1:
//   into = prior(i+1,j+1) * BM(i+1,j+1);  BX = ii'*BX(i+1,j) + im'*into
//   BY = dd*BY(i,j+1) + im'*into;         BM = md*BY(i,j+1) + mi'*BX(i+1,j) + mm'*into
// (primed: transitions of row i+1), plus BACKWARD_SCALE at the read's last row. The padding row
// above the read accumulates fgkl's row-0 start mass `s` in its BY (dd = 1 there).
//
// Events. A lane handles all events of a step in one divergent branch: the stores for the previous
// column (SNAP, END, NODE) and then the loads for its own (BEGIN, SWEEP). Start states come from a
// per-warp staging buffer in shared memory, one record per lane: the previous segment writes it
// directly when it is the snapshot's last writer, otherwise the state is prefetched from global
// scratch with cp.async at the previous segment's BEGIN, after that BEGIN has read the record. Joins only
// store their forward column; the products with the backward node are summed after the sweep, warp-wide, in
// an order fixed by the read row.
#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "dp_common.cuh"
#include "kernels.cuh"

namespace fgkl {

namespace {

// Per-lane field counts of the scratch records, rounded so every record starts on 16 bytes.
template <class P, int R>
struct Layout {
  using V = typename P::V;
  static constexpr int kRound = 16 / static_cast<int>(sizeof(V)) > 1 ? 16 / static_cast<int>(sizeof(V)) : 1;
  static constexpr int up(int x) { return (x + kRound - 1) / kRound * kRound; }
  static constexpr int kSnap = up(3 * R + 1);  // M, X, Y rows; accumulated result
  static constexpr int kNode = up(2 * R + 1);  // BM, BY rows; below-row BM
  static constexpr int kJoin = up(2 * R);      // cut column M and Y rows
  static constexpr int kStage = kSnap > kNode ? kSnap : kNode;
  // Priors are looked up in a per-lane table indexed by haplotype code (A, C, G, T, N); regions holding
  // other haplotype bytes run on the FP64 form that compares codes instead.
  static constexpr int kPriorCodes = P::kTable ? 5 : 0;
  // A lane's priors for one code: its rows padded to whole 16-byte chunks, kPer16 rows a chunk.
  static constexpr int kPer16 = kRound;
  static constexpr int kRp = up(R);
  static constexpr int kChunks = kRp / kPer16;
  static constexpr size_t kStageBytes = 32ull * kStage * sizeof(V);
  static constexpr size_t kSmemPerWarp = kStageBytes + static_cast<size_t>(kPriorCodes) * kRp * 32 * sizeof(V);
  // Element of row r's prior for `code` in the table, [code][chunk][lane][row in chunk]: each chunk of
  // the warp is 512 contiguous bytes, so a step's chunk loads are conflict-free 16-byte loads.
  __device__ static int prior_at(int code, int r, int lane) {
    return ((code * kChunks + r / kPer16) * 32 + lane) * kPer16 + r % kPer16;
  }
};

// Priors of the lane's rows for every haplotype code, in shared memory (Layout::prior_at), times the
// row's match-to-match factor in the FP32 form (cell_match).
template <class P, int R>
__device__ __forceinline__ void put_priors(typename P::V* table, int lane, int r, int c, const RowModel& m) {
  using S = typename P::S;
  const double fold = (P::kTransformed && m.read) ? m.mm : 1.0;
  for (int code = 0; code < Layout<P, R>::kPriorCodes; ++code) {
    const bool match = code == m.oc || code == kCodeN;
    P::put(table[Layout<P, R>::prior_at(code, r, lane)], c, static_cast<S>((match ? m.pm : m.px) * fold));
  }
}

// The lane's priors of every row for `code`, one 16-byte shared-memory load per chunk.
template <class P, int R>
__device__ __forceinline__ void load_priors(const typename P::V* table, int code, int lane,
                                            typename P::V (&pri)[Layout<P, R>::kRp]) {
  using L = Layout<P, R>;
  const uint4* src = reinterpret_cast<const uint4*>(table);
#pragma unroll
  for (int k = 0; k < L::kChunks; ++k) reinterpret_cast<uint4*>(pri)[k] = src[(code * L::kChunks + k) * 32 + lane];
}

// Forward coefficients of the lane's rows. What row r + 1 takes from row r is held with row r (k0..k3
// at index r are row r + 1's), because the lane computes both values that its bottom row hands to the
// lane below: the bracket of that lane's top match value and its new insertion value.
template <class P, int R, int G>
struct FwdRows {
  using V = typename P::V;
  using S = typename P::S;
  // Row r + 1: k0 mm (FP64 form), k1 and k2 the X and Y factors of the bracket, k3 the insertion chain's
  // factor, k5 mi (FP64 form). Row r: k4 the deletion chain's factor, k6 md (FP64 form).
  V k0[R], k1[R], k2[R], k3[R], k4[R], k5[R], k6[R];
  V pm[R], px[R];
  int oc[P::NC][R];
  const V* table;  // prior table (policies with kTable)

  __device__ V prior(int code, bool isN, int r) const {
    const bool m0 = (code == oc[0][r]) | isN;
    const bool m1 = (code == oc[P::NC - 1][r]) | isN;
    return P::sel(m0, m1, pm[r], px[r]);
  }

  // FP32 form: X^ = M_up + (gc*mi'/mi)*X^_up; Y^ = M_left + gc*Y^_left.
  __device__ void load(const BatchView& v, const ReadRef* rd, int lane, const uint8_t* codes, V* ptable) {
    table = ptable;
    const int top = (lane % G) * R;
#pragma unroll
    for (int r = 0; r <= R; ++r) {
#pragma unroll
      for (int c = 0; c < P::NC; ++c) {
        const RowModel m = row_model(v, rd[c], top + r - rd[c].pad, codes);
        if (r > 0) {
          const BracketFactors<P> b(m);
          P::put(k0[r - 1], c, b.k0);
          P::put(k1[r - 1], c, b.k1);
          P::put(k2[r - 1], c, b.k2);
          P::put(k3[r - 1], c, static_cast<S>(!P::kTransformed ? (m.read ? m.gc : 1.0) : (m.read ? m.gc * m.mi_prev / m.mi : 0.0)));
          P::put(k5[r - 1], c, static_cast<S>(m.mi));
        }
        if (r < R) {
          P::put(k4[r], c, static_cast<S>(m.read ? m.gc : 1.0));
          P::put(k6[r], c, static_cast<S>(m.md));
          P::put(pm[r], c, static_cast<S>(m.pm));
          P::put(px[r], c, static_cast<S>(m.px));
          oc[c][r] = m.oc;
          put_priors<P, R>(ptable, lane, r, c, m);
        }
      }
    }
  }

  // What row r + 1's match value is, before its prior, from row r.
  __device__ V bracket(const V& M, const V& X, const V& Y, int r) const {
    return cell_match<P>(M, X, Y, k0[r], k1[r], k2[r]);
  }
  // Row r + 1's insertion value from row r's.
  __device__ V insertion(const V& M, const V& X, int r) const {
    return P::kTransformed ? P::fma(X, k3[r], M) : P::fma(X, k3[r], P::mul(M, k5[r]));
  }
  __device__ V deletion(const V& M, const V& Y, int r) const {
    return P::kTransformed ? P::fma(Y, k4[r], M) : P::fma(Y, k4[r], P::mul(M, k6[r]));
  }
};

// Backward coefficients: each row's own deletion transitions and the transitions and priors of the
// row below it (rows l*R+1 .. l*R+R; the last comes from the next lane's top row). In the FP32 form
// the row below's match-to-match factor sits in its prior table (put_priors), so `into` carries it
// and im holds im/mm of the row below.
template <class P, int R, int G>
struct BwdRows {
  using V = typename P::V;
  using S = typename P::S;
  V md[R], dd[R], mm[R], im[R], mi[R], ii[R], pm[R], px[R];
  int oc[P::NC][R];
  const V* table;  // prior table of the rows below (policies with kTable)

  __device__ V prior(int code, bool isN, int r, int lane) const {
    if (Layout<P, R>::kPriorCodes) return table[Layout<P, R>::prior_at(code, r, lane)];
    const bool m0 = (code == oc[0][r]) | isN;
    const bool m1 = (code == oc[P::NC - 1][r]) | isN;
    return P::sel(m0, m1, pm[r], px[r]);
  }

  __device__ void load(const BatchView& v, const ReadRef* rd, int lane, const uint8_t* codes, V* ptable) {
    table = ptable;
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int c = 0; c < P::NC; ++c) {
        const int g = (lane % G) * R + r;
        const RowModel self = row_model(v, rd[c], g - rd[c].pad, codes);
        const RowModel below = row_model(v, rd[c], g + 1 - rd[c].pad, codes);
        P::put(md[r], c, static_cast<S>(self.read ? self.md : 0.0));
        P::put(dd[r], c, static_cast<S>(self.read ? self.gc : 1.0));
        P::put(mm[r], c, static_cast<S>(below.mm));
        P::put(im[r], c, static_cast<S>(P::kTransformed ? (below.read ? below.im / below.mm : 0.0) : below.im));
        P::put(mi[r], c, static_cast<S>(below.mi));
        P::put(ii[r], c, static_cast<S>(below.gc));
        P::put(pm[r], c, static_cast<S>(below.pm));
        P::put(px[r], c, static_cast<S>(below.px));
        oc[c][r] = below.oc;
        put_priors<P, R>(ptable, lane, r, c, below);
      }
    }
  }
};

// ---------------------------------------------------------------------------------------------
// Scratch: global per-warp records and the shared-memory staging buffers.
// ---------------------------------------------------------------------------------------------

template <class P, int R>
struct Scratch {
  using V = typename P::V;
  using L = Layout<P, R>;
  V* slots;         // [slot][lane][kSnap]
  V* nodes;         // [node][lane][kNode]
  V* joins;         // [seg][lane][kJoin]
  double* seg_raw;  // [seg][read slot]
  V* stage;         // shared: [buf][lane][kStage]
  V* priors;        // shared: [code][row][lane]

  __device__ Scratch(char* base, V* smem, int n_slots, int n_nodes, int n_segs) {
    slots = reinterpret_cast<V*>(base);
    nodes = slots + static_cast<size_t>(n_slots) * 32 * L::kSnap;
    joins = nodes + static_cast<size_t>(n_nodes) * 32 * L::kNode;
    seg_raw = reinterpret_cast<double*>(joins + static_cast<size_t>(n_segs) * 32 * L::kJoin);
    stage = smem;
    priors = reinterpret_cast<V*>(reinterpret_cast<char*>(smem) + L::kStageBytes);
  }
  __device__ V* slot(int s, int lane) { return slots + (static_cast<size_t>(s) * 32 + lane) * L::kSnap; }
  __device__ V* node(int n, int lane) { return nodes + (static_cast<size_t>(n) * 32 + lane) * L::kNode; }
  // The result of a segment for one of the warp's reads, before its factor.
  __device__ double& raw(int seg, int slot) { return seg_raw[seg * kMaxReads + slot]; }
  __device__ V* join(int seg, int lane) { return joins + (static_cast<size_t>(seg) * 32 + lane) * L::kJoin; }
  // One staging record per lane serves every segment (sweep): a lane writes or prefetches the next
  // segment's start into it only after loading the current segment's start at its BEGIN (SWEEP), and
  // each lane touches its own record alone.
  __device__ V* staged(int, int lane) { return stage + static_cast<size_t>(lane) * L::kStage; }
};

template <class P, int R>
__host__ __device__ constexpr size_t scratch_size(int n_slots, int n_nodes, int n_segs) {
  using V = typename P::V;
  using L = Layout<P, R>;
  return (static_cast<size_t>(n_slots) * 32 * L::kSnap + static_cast<size_t>(n_nodes) * 32 * L::kNode +
          static_cast<size_t>(n_segs) * 32 * L::kJoin) * sizeof(V) + static_cast<size_t>(n_segs) * kMaxReads * sizeof(double);
}

// Warps per block: two in the quad form; the others' is a tuning axis, at most kWarpsPerBlock.
template <int G>
constexpr int block_warps() {
  return G == 32 ? kWarpsPerBlock : 2;
}

// Resident blocks per SM each instantiation is compiled for: in the quad form what registers (seven values
// a row and component, and about 42 for the rest) and shared memory leave room for; one read a warp at 16
// warps an SM up to 8 rows.
// FP64: three blocks of four warps while their registers hold the rows (128 regions in FP64, 5 rows: 7.8 ms,
// against 8.3 at the 8 warps an SM of one block's full budget; four blocks 7.9); priors from the table
// instead of by comparison 6.4 ms, and at 6 rows three blocks fit then. Two reads on 16 lanes each take the
// registers of 8 warps an SM (238 at 10 rows): 128 uneven regions 8.6 -> 7.5 ms, 128 of 128 SNP haplotypes
// 35.1 -> 28.6 ms.
constexpr int f64_min_blocks(int rows, bool table) { return rows <= (table ? 6 : 5) ? 3 : 1; }
// Two FP32 reads on 32 lanes: four blocks up to 4 rows, three up to 7, two at 8.
template <class P, int R, int G>
struct MinBlocks {
  static constexpr int kRegs = (7 * R * P::NC + 42) > 255 ? 255 : 7 * R * P::NC + 42;
  static constexpr int kBySmem = static_cast<int>(228 * 1024 / (2 * Layout<P, R>::kSmemPerWarp + 1024));
  // A quarter of the SM's registers serves a quarter of its warps.
  static constexpr int kByRegs = 2 * (512 / ((kRegs + 7) / 8 * 8));
  static constexpr int kQuad = kByRegs < kBySmem ? kByRegs : kBySmem;
  static constexpr int kPair = R <= 4 ? 4 : (R <= 7 ? 3 : 2);
  static constexpr int value = G < 32 ? (P::kDouble ? 4 : (kQuad > 12 ? 12 : kQuad)) : (P::kDouble ? f64_min_blocks(R, P::kTable) : P::NC == 2 ? kPair : (R <= 8 ? 4 : 2));
};

// ---------------------------------------------------------------------------------------------
// Backward pass: every suffix sweep of the program, writing backward nodes.
// ---------------------------------------------------------------------------------------------

template <class P, int R, int G>
__device__ __forceinline__ void backward_pass(const LaunchArgs& a, const Program& prog, const ReadRef* rd, const uint8_t* codes, int lane,
                              Scratch<P, R>& sc) {
  using V = typename P::V;
  using L = Layout<P, R>;
  BwdRows<P, R, G> bp;
  const int gl = lane % G;
  bp.load(a.v, rd, lane, codes, sc.priors);
  const V sink = P::splat(gl == G - 1 ? static_cast<typename P::S>(Consts<P::kDouble>::kBackwardScale) : 0);
  V BM[R], BY[R];
#pragma unroll
  for (int r = 0; r < R; ++r) BM[r] = BY[r] = P::zero();
  V dBM = P::zero(), topBM = P::zero(), topBX = P::zero();
  const int n = prog.bwd_len;
  const uint32_t* stream = a.v.stream + prog.bwd_off - (G - 1 - gl);  // entry of this lane's position at t
  int sweep = -1;
  uint32_t ev_next = __ldg(stream);
  for (int t = 0; t < n + G; ++t) {
    const uint32_t ev = ev_next;
    ev_next = __ldg(stream + t + 1);
    const V rBM = P::template down<G>(topBM), rBX = P::template down<G>(topBX);
    if (ev & kEvMask) {
      if (ev & EV_NODE) {
        V rec[L::kNode];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          rec[r] = BM[r];
          rec[R + r] = BY[r];
        }
        rec[2 * R] = dBM;
#pragma unroll
        for (int i = 2 * R + 1; i < L::kNode; ++i) rec[i] = P::zero();
        store_record(sc.node(static_cast<int>(ev >> kPayloadShift), lane), rec);
        if (ev & EV_NSTAGE) store_record(sc.staged(sweep + 1, lane), rec);
      }
      if (ev & EV_SWEEP) {
        ++sweep;
        const Sweep cur = a.v.sweeps[prog.sweep_off + sweep];
        if (sweep + 1 < prog.n_sweeps) prefetch_l1(a.v.sweeps + prog.sweep_off + sweep + 1);
        if (cur.staged) {
          __pipeline_wait_prior(0);
          V rec[L::kNode];
          load_record(rec, sc.staged(sweep, lane));
#pragma unroll
          for (int r = 0; r < R; ++r) {
            BM[r] = rec[r];
            BY[r] = rec[R + r];
          }
          dBM = rec[2 * R];
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) BM[r] = BY[r] = P::zero();
          dBM = P::zero();
        }
        if (cur.next_node >= 0) prefetch(sc.staged(sweep + 1, lane), sc.node(cur.next_node, lane), L::kNode);
      }
    }
    const int code = ev & kCodeMask;
    const bool isN = code == kCodeN;
    V pri[L::kRp];
    if (L::kPriorCodes) load_priors<P, R>(bp.table, code, lane, pri);
    V belowX = rBX, diagM = dBM;
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const V into = P::mul(L::kPriorCodes ? pri[r] : bp.prior(code, isN, r, lane), diagM);
      const V itm = P::mul(into, bp.im[r]);
      V bx = P::fma(belowX, bp.ii[r], itm);
      const V by = P::fma(BY[r], bp.dd[r], itm);
      V bm = P::fma(BY[r], bp.md[r], P::fma(belowX, bp.mi[r], P::kTransformed ? into : P::mul(into, bp.mm[r])));
      if (r == R - 1) {
        bm = P::add(bm, sink);
        bx = P::add(bx, sink);
      }
      diagM = BM[r];
      BM[r] = bm;
      BY[r] = by;
      belowX = bx;
    }
    topBM = BM[0];
    topBX = belowX;
    dBM = rBM;
  }
  __pipeline_wait_prior(0);
}

// ---------------------------------------------------------------------------------------------
// Forward pass.
// ---------------------------------------------------------------------------------------------

// Loop-carried state of the forward sweep of one lane.
template <class P, int R>
struct FwdState {
  using V = typename P::V;
  using S = typename P::S;
  V M[R], X[R], Y[R];
  // For the lane below's top row, at the column the lane has just computed: its new insertion value,
  // and the bracket of its match value (from the column before).
  V xs, ts;
  V acc;
  int seg_i;
  // The next segment's record, loaded a segment ahead so a BEGIN never waits on memory.
  int nx_staged, nx_slot;
  S nx_init;
  // Strip-mined reads: what lane 0's top row takes from the row above for this step's column. Read only
  // by forward_step<..., kCarry = true>.
  V cX, cT;

  __device__ void clear() {
#pragma unroll
    for (int r = 0; r < R; ++r) M[r] = X[r] = Y[r] = P::zero();
    xs = ts = acc = P::zero();
    seg_i = -1;
    nx_staged = 0;
    nx_slot = -1;
    nx_init = S(0);
  }

  __device__ void load_next(const BatchView& v, const Program& prog, int seg) {
    if (seg < prog.n_segs) {
      const Segment* rec = v.segs + prog.seg_off + seg;
      nx_staged = rec->staged;
      nx_slot = rec->next_slot;
      nx_init = P::kDouble ? static_cast<S>(rec->init_d) : static_cast<S>(rec->init_f);
    } else {
      nx_staged = 0;
      nx_slot = -1;
      nx_init = S(0);
    }
  }
};

// One forward step: events, then the column. kEv = false compiles the event code out, for steps where
// no lane of the warp has an event. kCarry = true gives lane 0 the row above from the state's carry
// values (strip-mined reads); otherwise a group's first lane starts with a padding row, for which the
// row above is zero.
template <class P, int R, int G, bool kEv = true, bool kCarry = false>
__device__ __forceinline__ void forward_step(const LaunchArgs& a, const Program& prog, const ReadRef* rd, int lane,
                                             const FwdRows<P, R, G>& fr, const typename P::V& an, Scratch<P, R>& sc,
                                             FwdState<P, R>& st, int synth_len, uint32_t ev) {
  using V = typename P::V;
  using S = typename P::S;
  using L = Layout<P, R>;
  const int gl = lane % G;
  V qX = P::template up<G>(st.xs), T = P::template up<G>(st.ts);
  if (gl == 0) {
    qX = kCarry ? st.cX : P::zero();
    T = kCarry ? st.cT : P::zero();
  }
  // END and ACC act in the group's last lane alone (the read's last row); the other lanes pass them by
  // without entering the event code, which every lane otherwise reaches at its own step.
  if (kEv && (ev & (gl == G - 1 ? kEvMask : (kEvMask & ~(EV_END | EV_ACC))))) {
    const int slot0 = lane / G * P::NC;  // the group's first read slot
    if (ev & EV_SNAP) {
      const uint32_t slot = ev >> kPayloadShift;
      V* dst[2] = {slot != kPayloadNone ? sc.slot(static_cast<int>(slot), lane) : nullptr,
                   (ev & EV_STAGE) ? sc.staged(st.seg_i + 1, lane) : nullptr};
      V rec[L::kSnap];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        rec[r] = st.M[r];
        rec[R + r] = st.X[r];
        rec[2 * R + r] = st.Y[r];
      }
      rec[3 * R] = st.acc;
#pragma unroll
      for (int i = 3 * R + 1; i < L::kSnap; ++i) rec[i] = P::zero();
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (dst[k]) store_record(dst[k], rec);
    }
    if ((ev & EV_END) && gl == G - 1) {
#pragma unroll
      for (int c = 0; c < P::NC; ++c) sc.raw(st.seg_i, slot0 + c) = static_cast<double>(P::get(st.acc, c));
    }
    if (ev & EV_JOIN) {
      // The cut column's match and deletion rows, joined with the backward node after the sweep
      // (fgkl kernel.rs:744-755).
      V rec[L::kJoin];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        rec[r] = st.M[r];
        rec[R + r] = st.Y[r];
      }
#pragma unroll
      for (int i = 2 * R; i < L::kJoin; ++i) rec[i] = P::zero();
      store_record(sc.join(st.seg_i, lane), rec);
    }
    if (ev & EV_BEGIN) {
      ++st.seg_i;
      // A recomputation stream (FP64 only) has one unshared segment from the origin and no record.
      const bool synth = synth_len > 0;
      const int next_slot = synth ? -1 : st.nx_slot;
      const bool staged = !synth && st.nx_staged;
      const S init = st.nx_init;
      if (!synth) st.load_next(a.v, prog, st.seg_i + 1);
      if (staged) {
        __pipeline_wait_prior(0);
        V s[L::kSnap];
        load_record(s, sc.staged(st.seg_i, lane));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          st.M[r] = s[r];
          st.X[r] = s[R + r];
          st.Y[r] = s[2 * R + r];
        }
        st.acc = s[3 * R];
      } else {
        // The origin: nothing but the row-0 constant, in the padding rows.
        const S in_s = synth ? static_cast<S>(Consts<P::kDouble>::kInitial / synth_len) : init;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          st.M[r] = st.X[r] = P::zero();
#pragma unroll
          for (int c = 0; c < P::NC; ++c) P::put(st.Y[r], c, gl * R + r < rd[c].pad ? in_s : S(0));
        }
        st.acc = P::zero();
      }
      if (next_slot >= 0) prefetch(sc.staged(st.seg_i + 1, lane), sc.slot(next_slot, lane), L::kSnap);
    }
    if ((ev & EV_ACC) && gl == G - 1) {
#pragma unroll
      for (int c = 0; c < P::NC; ++c) sc.raw(st.seg_i, slot0 + c) = static_cast<double>(P::get(st.acc, c));
    }
  }
  const int code = ev & kCodeMask;
  const bool isN = code == kCodeN;
  V pri[L::kRp];
  if (L::kPriorCodes) load_priors<P, R>(fr.table, code, lane, pri);
  // Rows from the top down, in place: row r hands its old values to row r + 1 as the bracket Tn. Row 0,
  // which waits for the lane above, comes after the others, and the insertion chain, the only serial one,
  // last (1.5% faster than the chain row by row with the others).
  V Tn = fr.bracket(st.M[0], st.X[0], st.Y[0], 0);
#pragma unroll
  for (int r = 1; r < R; ++r) {
    const V prior = L::kPriorCodes ? pri[r] : fr.prior(code, isN, r);
    const V below = fr.bracket(st.M[r], st.X[r], st.Y[r], r);
    st.Y[r] = fr.deletion(st.M[r], st.Y[r], r);
    st.M[r] = P::mul(prior, Tn);
    Tn = below;
  }
  st.Y[0] = fr.deletion(st.M[0], st.Y[0], 0);
  st.M[0] = P::mul(L::kPriorCodes ? pri[0] : fr.prior(code, isN, 0), T);
  T = Tn;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    st.X[r] = qX;
    qX = fr.insertion(st.M[r], qX, r);
  }
  st.xs = qX;
  st.ts = T;
  st.acc = P::fma(st.X[R - 1], an, P::add(st.acc, st.M[R - 1]));
}

// Entry p of a recomputation stream: the haplotype's codes, BEGIN on the first column and END after
// the last.
__device__ __forceinline__ uint32_t synth_entry(const uint8_t* seq, int len, int p) {
  if (p < 0 || p > len) return 0u;
  uint32_t e = p < len ? __ldg(seq + p) : 0u;
  if (p == 0) e |= EV_BEGIN;
  if (p == len) e |= EV_END;
  return e;
}

template <class P, int R, int G>
__device__ __forceinline__ void forward_pass(const LaunchArgs& a, const Program& prog, const ReadRef* rd, const uint8_t* codes, int lane,
                             Scratch<P, R>& sc, const uint8_t* synth_seq, int synth_len) {
  using V = typename P::V;
  using S = typename P::S;
  const int gl = lane % G;
  FwdRows<P, R, G> fr;
  fr.load(a.v, rd, lane, codes, sc.priors);
  // X factor of the read's last row (the group's last lane): the accumulated result is Σ M + mi_n * X^.
  V an;
#pragma unroll
  for (int c = 0; c < P::NC; ++c)
    P::put(an, c, static_cast<S>((P::kTransformed && rd[c].len > 0) ? err_prob(a.v, a.v.ins[rd[c].off + rd[c].len - 1]) : 1.0));

  FwdState<P, R> st;
  st.clear();
  st.load_next(a.v, prog, synth_len > 0 ? prog.n_segs : 0);
  if (P::kDouble && synth_len > 0) {
    const int n = synth_len;
    int t = 0;
    for (; t < G; ++t) forward_step<P, R, G>(a, prog, rd, lane, fr, an, sc, st, n, synth_entry(synth_seq, n, t - gl));
    // Every lane strictly inside the haplotype: no events.
    const uint8_t* seq = synth_seq - gl;
    for (; t + 4 <= n; t += 4) {
#pragma unroll
      for (int i = 0; i < 4; ++i) forward_step<P, R, G, false>(a, prog, rd, lane, fr, an, sc, st, n, __ldg(seq + t + i));
    }
    for (; t < n + G; ++t) forward_step<P, R, G>(a, prog, rd, lane, fr, an, sc, st, n, synth_entry(synth_seq, n, t - gl));
  } else {
    const int n = prog.fwd_len;
    const uint32_t* stream = a.v.stream + prog.fwd_off - gl;
    // Four steps an iteration, their stream entries loaded one iteration ahead (the stream carries
    // kStreamPad zero entries past its end, so the last iteration's look-ahead and the steps past
    // n + G - 1 read no events). An iteration where no lane has an event runs a body without event
    // code, which the compiler schedules across the steps (two steps an iteration: 10% slower without
    // events); in the others one copy of the step with event code runs four times (four copies: 11%
    // slower on uneven regions, for their size).
    constexpr int kSteps = 4;
    const uint32_t keep = gl == G - 1 ? kEvMask : (kEvMask & ~(EV_END | EV_ACC));
    uint32_t next[kSteps];
#pragma unroll
    for (int i = 0; i < kSteps; ++i) next[i] = __ldg(stream + i);
    for (int t = 0; t < n + G; t += kSteps) {
      uint32_t e[kSteps], any = 0;
#pragma unroll
      for (int i = 0; i < kSteps; ++i) {
        e[i] = next[i];
        any |= e[i];
        next[i] = __ldg(stream + t + kSteps + i);
      }
      if (__any_sync(kFull, any & keep)) {
#pragma unroll 1
        for (int i = 0; i < kSteps; ++i) {
          const uint32_t ev = e[0];
#pragma unroll
          for (int k = 0; k + 1 < kSteps; ++k) e[k] = e[k + 1];
          forward_step<P, R, G>(a, prog, rd, lane, fr, an, sc, st, 0, ev);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) forward_step<P, R, G, false>(a, prog, rd, lane, fr, an, sc, st, 0, e[i]);
      }
    }
  }
  __pipeline_wait_prior(0);
}

// ---------------------------------------------------------------------------------------------
// Finalisation: joins, thresholds, log10, and the caller's layout.
// ---------------------------------------------------------------------------------------------

template <class P, int R, int G>
__device__ __forceinline__ void finalize(const LaunchArgs& a, const Task& task, const Region& region, const Program& prog, const ReadRef* rd,
                         int lane, Scratch<P, R>& sc) {
  using C = Consts<P::kDouble>;
  constexpr int kReads = 32 / G * P::NC;  // read slots of the warp
  double* red = reinterpret_cast<double*>(sc.stage);  // [slot][row q], the staging buffers are free now
  constexpr int max_rows = G * R;
  const int slot0 = lane / G * P::NC, top = (lane % G) * R;
  const int n_join_segs = (P::kDouble && G == 32 && task.hap >= 0) ? 0 : prog.n_segs;
  // Joins (fgkl kernel.rs:767-791): raw = acc + (Σ_rows F_M*B_M + F_Y*B_Y + init*s) / BACKWARD_SCALE,
  // with the row sum taken in an order fixed by the read row so it does not depend on R or G.
  double yfac[R][P::NC];
  bool any_join = false;
  for (int seg = 0; seg < n_join_segs; ++seg) {
    const int node = a.v.segs[prog.seg_off + seg].node;
    if (node < 0) continue;
    if (!any_join) {
      any_join = true;
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < P::NC; ++c) {
          const int q = top + r - rd[c].pad;
          yfac[r][c] = (P::kTransformed && rd[c].len > 0 && q >= 0) ? err_prob(a.v, a.v.del[rd[c].off + q]) : 1.0;
        }
    }
    const typename P::V* f = sc.join(seg, lane);
    const typename P::V* b = sc.node(node, lane);
    double row0[P::NC];
#pragma unroll
    for (int c = 0; c < P::NC; ++c) row0[c] = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const typename P::V fM = f[r], fY = f[R + r], bM = b[r], bY = b[R + r];
#pragma unroll
      for (int c = 0; c < P::NC; ++c) {
        const int q = top + r - rd[c].pad;
        const double fy = __dmul_rn(yfac[r][c], static_cast<double>(P::get(fY, c)));
        const double prod = __dadd_rn(__dmul_rn(static_cast<double>(P::get(fM, c)), static_cast<double>(P::get(bM, c))),
                                      __dmul_rn(fy, static_cast<double>(P::get(bY, c))));
        if (q >= 0) red[(slot0 + c) * max_rows + q] = prod;
        if (q == -1) row0[c] = prod;
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kReads; ++k) {
      const int c = k % P::NC, first = k / P::NC * G;  // the slot's component and its group's first lane
      const int len = __shfl_sync(kFull, rd[c].len, first), pad = max_rows - len;
      double s = 0.0;
      for (int q = lane; q < len; q += 32) s = __dadd_rn(s, red[k * max_rows + q]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(kFull, s, o));
      // Row 0's start mass lives in one lane.
      const double r0 = __shfl_sync(kFull, row0[c], first + (pad - 1) / R);
      if (lane == 0 && task.read[k] >= 0)
        sc.raw(seg, k) = __dadd_rn(sc.raw(seg, k), __ddiv_rn(__dadd_rn(s, r0), C::kBackwardScale));
    }
    __syncwarp();
  }
  __syncwarp();
  if (P::kDouble && G == 32 && task.hap >= 0) {
    // A recomputation task: its one segment's result goes to the haplotype and its duplicates.
    const double raw = sc.raw(0, 0);
    const bool lost = raw != raw;
    const double result = lost ? __longlong_as_double(0x7ff8000000000000ll) : log10(raw) - C::kLog10Initial;
    const int read_local = task.read[0] - region.read_off;
    for (int k = lane; k < region.n_haps; k += 32) {
      const HapInfo info = a.v.haps[region.hap_off + k];
      if (info.src == task.hap) a.v.out[region.out_off + static_cast<int64_t>(read_local) * region.n_haps + info.order] = result;
    }
    return;
  }
  // A dense read's recomputation (only_lost) fills in only the pairs the first pass lost and counts
  // nothing: the pairs it loses again stay NaN for the unshared sweep that follows it.
  const bool dense = a.only_lost != 0;
  unsigned long long lost_count = 0;
  for (int i = lane; i < region.n_haps; i += 32) {
    const HapInfo info = a.v.haps[region.hap_off + i];
    const int own = info.seg - prog.seg_first;  // another task's, outside the program's segments
    if (own < 0 || own >= prog.n_segs) continue;
    const Segment* seg = a.v.segs + prog.seg_off + own;
    const bool joined = seg->node >= 0;
    const double factor = seg->factor;
#pragma unroll
    for (int k = 0; k < kReads; ++k) {
      if (task.read[k] < 0) continue;
      const int read_local = task.read[k] - region.read_off;
      double* dst = a.v.out + region.out_off + static_cast<int64_t>(read_local) * region.n_haps + info.order;
      if (dense && !isnan(*dst)) continue;
      const double raw = __dmul_rn(sc.raw(own, k), factor);
      bool lost;
      if (joined)
        lost = !(raw >= C::kMinAcceptedJoined);
      else
        lost = a.min_accept_plain ? !(raw >= C::kMinAccepted) : (raw != raw);
      if (!P::kDouble) lost |= isinf(raw);
      const double result = lost ? __longlong_as_double(0x7ff8000000000000ll) : log10(raw) - C::kLog10Initial;
      *dst = result;
      lost_count += lost;
    }
  }
  if (lost_count && !dense) {
    atomicAdd(&a.v.counters->lost_pairs, lost_count);
    if (G == 32 && R > 8) atomicAdd(&a.v.counters->lost_wide, lost_count);
  }
}

// One task at its R rows per lane.
template <class P, int R, int G>
__device__ __forceinline__ void run_task(const LaunchArgs& a, const Task& task, int lane, char* scratch, typename P::V* smem) {
  const Region region = a.v.regions[task.region];
  const Program prog = a.v.progs[task.prog];
  ReadRef rd[P::NC];
#pragma unroll
  for (int c = 0; c < P::NC; ++c) {
    const int id = task.read[lane / G * P::NC + c];
    if (id >= 0) {
      rd[c].off = a.v.read_off[id];
      rd[c].len = static_cast<int>(a.v.read_off[id + 1] - rd[c].off);
    } else {
      rd[c].off = 0;
      rd[c].len = 0;
    }
    rd[c].pad = G * R - rd[c].len;
  }
  const uint8_t* codes = a.v.code_of_byte + region.code_off;
  if (P::kDouble && G == 32 && task.hap >= 0) {
    const HapInfo info = a.v.haps[region.hap_off + task.hap];
    Scratch<P, R> sc(scratch, smem, 0, 0, 1);
    forward_pass<P, R, G>(a, prog, rd, codes, lane, sc, a.v.hap_codes + region.seq_off + info.seq, info.len);
    __syncwarp();
    finalize<P, R, G>(a, task, region, prog, rd, lane, sc);
  } else {
    Scratch<P, R> sc(scratch, smem, prog.n_slots, prog.n_nodes, prog.n_segs);
    if (prog.bwd_len > 0) backward_pass<P, R, G>(a, prog, rd, codes, lane, sc);
    __syncwarp();
    forward_pass<P, R, G>(a, prog, rd, codes, lane, sc, nullptr, 0);
    __syncwarp();
    finalize<P, R, G>(a, task, region, prog, rd, lane, sc);
    if (P::kDouble && G == 32 && a.only_lost) {
      // A dense read's shared FP64 sweep can lose a pair again (a joined result below the backward
      // range): each such distinct haplotype is swept once more here without sharing, which
      // cannot lose it (fgkl lib.rs:476-486).
      __syncwarp();
      const double* row = a.v.out + region.out_off + static_cast<int64_t>(task.read[0] - region.read_off) * region.n_haps;
      for (int base = 0; base < region.n_haps; base += 32) {
        const int k = base + lane;
        bool again = false;
        if (k < region.n_haps) {
          const HapInfo info = a.v.haps[region.hap_off + k];
          const int own = info.seg - prog.seg_first;
          again = info.src == k && own >= 0 && own < prog.n_segs && isnan(row[info.order]);
        }
        unsigned mask = __ballot_sync(kFull, again);
        while (mask) {
          Task one = task;
          one.hap = base + __ffs(mask) - 1;
          mask &= mask - 1;
          const HapInfo info = a.v.haps[region.hap_off + one.hap];
          Scratch<P, R> s1(scratch, smem, 0, 0, 1);
          forward_pass<P, R, G>(a, prog, rd, codes, lane, s1, a.v.hap_codes + region.seq_off + info.seq, info.len);
          __syncwarp();
          finalize<P, R, G>(a, one, region, prog, rd, lane, s1);
          __syncwarp();
        }
      }
    }
  }
}

template <class P, int R, int G>
__global__ void __launch_bounds__(block_warps<G>() * 32, (MinBlocks<P, R, G>::value)) pairhmm_kernel(LaunchArgs a) {
  using V = typename P::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int warp_in_block = threadIdx.x >> 5;
  const int warp = blockIdx.x * static_cast<int>(blockDim.x >> 5) + warp_in_block;
  V* smem = reinterpret_cast<V*>(smem_raw + warp_in_block * Layout<P, R>::kSmemPerWarp);
  char* scratch = a.scratch + static_cast<size_t>(warp) * a.scratch_stride;
  const int count = a.count ? min(*a.count, a.n_tasks) : a.n_tasks;
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(a.task_counter, 1);
    t = __shfl_sync(kFull, t, 0);
    if (t >= count) break;
    run_task<P, R, G>(a, a.tasks[t], lane, scratch, smem);
    __syncwarp();
  }
}

}  // namespace

}  // namespace fgkl

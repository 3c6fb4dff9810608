// sm_100a PD-HMM kernels (GATK LoglessPDPairHMM for DRAGEN concordance mode; fgkl pd_kernel.rs and
// pd_reference.rs:29-118): the plain kernels' warp wavefront over a prefix-shared column stream,
// with GATK's branch matrices.
//
// Per cell (row i, column j in deletion state s; left = (i, j-1), up = (i-1, j), diag = (i-1, j-1);
// B = branch values, V = (M, X, Y)):
//   B(i,j) = V(left)                 s = NORMAL
//          = B(left)                 s = INSIDE_DEL
//          = max(B(left), V(left))   s = AFTER_DEL
//   M = prior * (mm*D.M + im*(D.X + D.Y)),  D = max(B(diag), V(diag)) after a deletion, else V(diag)
//   Y = md*W.M + dd*W.Y,                    W = max(B(left), V(left)) after a deletion, else V(left)
//   X = mi*U.M + ii*U.X,                    U = max(B(up), V(up)) on a DEL_END column, else V(up)
// The state of a column depends only on the flags and on the state the row started in: NORMAL for
// the read's first row, the state the previous row ended in for the others. The host resolves both
// per column into the stream entry (program.h), with the column's prior code (a match set: its base
// and, on a SNP column, the flagged alternates).
//
// A column right after DEL_END is AFTER_DEL in every row (the state machine sets it from the
// DEL_END flag alone), and there the diagonal and the left cell enter only as max(B, V). So a lane
// takes that max once, at the DEL_END column itself: after computing the column, each row's M, X
// and Y become max(B, V) (row by row down the insertion sweep, so the next row's X reads U =
// max(B(up), V(up)) as GATK's DEL_END rule asks, and the last row after the result has taken its
// unmerged values). Every later reader of those values is a max reader, and the max is idempotent,
// so the AFTER_DEL column itself needs no branch values at all. Branch values are then only the
// lane's own rows: set to V(left) on a column carrying DEL_START or DEL_END (held inside a
// deletion), read on DEL_END columns, stale elsewhere where nothing reads them; the lane above's
// never cross. Columns carrying neither flag (the vast majority) run the plain recurrence.
//
// Priors. A PD region maps its reads' distinct bytes to classes 0..30; each match-set code carries
// the bit set of classes it accepts, so a row's prior is pm or px by one bit test.
//
// FP32 kernels carry X/mi and Y/md per row like the plain kernels; max() commutes with the positive
// per-row scale, so the branch values are kept in the same scale.
#include "dp_common.cuh"
#include "kernels.cuh"

namespace fgkl {

namespace {

template <class P, int R>
struct PdLayout {
  using V = typename P::V;
  static constexpr int kRound = 16 / static_cast<int>(sizeof(V)) > 1 ? 16 / static_cast<int>(sizeof(V)) : 1;
  static constexpr int up(int x) { return (x + kRound - 1) / kRound * kRound; }
  // M, X, Y rows; branch M, X, Y rows; accumulated result.
  static constexpr int kSnap = up(6 * R + 1);
  static constexpr size_t kStageBytes = 32ull * kSnap * sizeof(V);
  static constexpr size_t kSmemPerWarp = kStageBytes;
};

template <class P, int R>
struct PdScratch {
  using V = typename P::V;
  using L = PdLayout<P, R>;
  V* slots;         // [slot][lane][kSnap]
  double* seg_raw;  // [seg][read slot]
  V* stage;         // shared: [buf][lane][kSnap]

  __device__ PdScratch(char* base, V* smem, int n_slots) {
    slots = reinterpret_cast<V*>(base);
    seg_raw = reinterpret_cast<double*>(slots + static_cast<size_t>(n_slots) * 32 * L::kSnap);
    stage = smem;
  }
  __device__ V* slot(int s, int lane) { return slots + (static_cast<size_t>(s) * 32 + lane) * L::kSnap; }
  // The result of a segment for one of the warp's reads, before its factor.
  __device__ double& raw(int seg, int slot) { return seg_raw[seg * kMaxReads + slot]; }
  // One staging record per lane serves every segment: a lane writes or prefetches the next
  // segment's start into it only after loading the current one at its BEGIN.
  __device__ V* staged(int, int lane) { return stage + static_cast<size_t>(lane) * L::kSnap; }
};

template <class P, int R>
constexpr size_t pd_scratch_size(int n_slots, int n_segs) {
  return static_cast<size_t>(n_slots) * 32 * PdLayout<P, R>::kSnap * sizeof(typename P::V) +
         static_cast<size_t>(n_segs) * kMaxReads * sizeof(double);
}

// Forward coefficients of the lane's rows and each row's read class. As in the plain kernel, what row r + 1
// takes from row r is held with row r (k0..k3, k5), because the lane computes both values that its bottom
// row hands to the lane below.
template <class P, int R>
struct PdRows {
  using V = typename P::V;
  using S = typename P::S;
  V k0[R], k1[R], k2[R], k3[R], k4[R], k5[R], k6[R], pm[R], px[R];
  uint32_t cls[P::NC][R];  // bit of the row's read class; 0 for a padding row (no code accepts it)

  __device__ V prior(uint32_t sig, int r) const {
    return P::sel((sig & cls[0][r]) != 0u, (sig & cls[P::NC - 1][r]) != 0u, pm[r], px[r]);
  }
  // What row r + 1's match value is, before its prior, from row r.
  __device__ V bracket(const V& M, const V& X, const V& Y, int r) const { return cell_match<P>(M, X, Y, k0[r], k1[r], k2[r]); }
  // Row r + 1's insertion value from row r's.
  __device__ V insertion(const V& M, const V& X, int r) const {
    return P::kTransformed ? P::fma(X, k3[r], M) : P::fma(X, k3[r], P::mul(M, k5[r]));
  }
  __device__ V deletion(const V& M, const V& Y, int r) const {
    return P::kTransformed ? P::fma(Y, k4[r], M) : P::fma(Y, k4[r], P::mul(M, k6[r]));
  }

  // Regions whose reads hold more distinct bytes than the class bits cover compare bytes instead:
  // after load_generic, cls holds the row's read byte (bits 0-7), whether it is N (bit 8) and the ALT
  // bit it answers to (bits 9-12), and a stream entry carries the column's haplotype byte (bits 0-7)
  // and its ALT bits (kPdPayloadShift up), so the column accepts the row's base exactly when
  // MatchSet::accepts would (fgkl pd_kernel.rs:196-214).
  __device__ V prior_generic(uint32_t ev, int r) const {
    const uint32_t base = ev & kCodeMask, alts = (ev >> kPdPayloadShift) & 0xFu, c = cls[0][r];
    const bool match = c != 0u && (((c & 0xFFu) == base) || base == 'N' || ((c >> 8) & 1u) || (((c >> 9) & alts) != 0u));
    return match ? pm[r] : px[r];
  }

  __device__ void load(const BatchView& v, const ReadRef* rd, int lane, const uint8_t* classes) {
    const int top = lane * R;
#pragma unroll
    for (int r = 0; r <= R; ++r) {
#pragma unroll
      for (int c = 0; c < P::NC; ++c) {
        const RowModel m = row_model(v, rd[c], top + r - rd[c].pad, classes);
        if (r > 0) {
          const BracketFactors<P> b(m);
          P::put(k0[r - 1], c, b.k0);
          P::put(k1[r - 1], c, b.k1);
          P::put(k2[r - 1], c, b.k2);
          P::put(k3[r - 1], c, static_cast<S>(!P::kTransformed ? (m.read ? m.gc : 1.0) : (m.read ? m.gc * m.mi_prev / m.mi : 0.0)));
          P::put(k5[r - 1], c, static_cast<S>(m.mi));
        }
        if (r < R) {
          // The match-to-match factor moves into the priors in the FP32 form (cell_match).
          const double fold = (P::kTransformed && m.read) ? m.mm : 1.0;
          P::put(k4[r], c, static_cast<S>(m.read ? m.gc : 1.0));
          P::put(k6[r], c, static_cast<S>(m.md));
          P::put(pm[r], c, static_cast<S>(m.pm * fold));
          P::put(px[r], c, static_cast<S>(m.px * fold));
          cls[c][r] = m.read ? (1u << (m.oc & 31)) : 0u;
        }
      }
    }
  }

  // As load, with the byte-comparison row descriptors of prior_generic in cls (one read).
  __device__ void load_generic(const BatchView& v, const ReadRef* rd, int lane, const uint8_t* classes) {
    load(v, rd, lane, classes);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q = lane * R + r - rd[0].pad;
      uint32_t d = 0;
      if (rd[0].len > 0 && q >= 0 && q < rd[0].len) {
        const uint32_t b = v.bases[rd[0].off + q];
        const uint32_t alt = (b == 'A' || b == 'a') ? 1u : (b == 'C' || b == 'c') ? 2u : (b == 'G' || b == 'g') ? 4u : (b == 'T' || b == 't') ? 8u : 0u;
        d = b | (b == 'N' ? 1u << 8 : 0u) | (alt << 9) | (1u << 13);  // bit 13: a read row (never 0)
      }
      cls[0][r] = d;
    }
  }
};

template <class P, int R>
struct PdState {
  using V = typename P::V;
  V M[R], X[R], Y[R];
  V BM[R], BX[R], BY[R];
  // For the lane below's top row, at the column the lane has just computed: its new insertion value (from
  // the merged bottom row on a DEL_END column), and the bracket of its match value (from the column before).
  V xs, ts;
  V acc;
  int seg_i;
  // Strip-mined reads: what lane 0's top row takes from the row above for this step's column (read only by
  // pd_step<..., kCarry = true>).
  V cX, cT;

  __device__ void clear() {
#pragma unroll
    for (int r = 0; r < R; ++r) M[r] = X[r] = Y[r] = BM[r] = BX[r] = BY[r] = P::zero();
    xs = ts = acc = P::zero();
    seg_i = -1;
  }
};

// The rows of one column. kSlow: some lane's column carries DEL_START or DEL_END; the branch-value path is
// exact for every column, so the whole warp takes it. keep(r): what to do with the branch values of row r
// before its column; de: the lane's column carries DEL_END, and each row's values take the max with its
// branch values once its X is computed, so that the next row's X reads U = max(B(up), V(up)).
template <class P, int R, bool kSlow, class Prior, class Keep>
__device__ __forceinline__ void pd_rows_down(const PdRows<P, R>& pr, PdState<P, R>& st, const typename P::V& an, typename P::V qX,
                                             typename P::V T, bool de, Prior&& prior, Keep&& keep) {
  using V = typename P::V;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const V below = pr.bracket(st.M[r], st.X[r], st.Y[r], r);
    if (kSlow) keep(r);
    st.Y[r] = pr.deletion(st.M[r], st.Y[r], r);
    st.M[r] = P::mul(prior(r), T);
    T = below;
    st.X[r] = qX;
    if (r == R - 1) st.acc = P::fma(qX, an, P::add(st.acc, st.M[r]));  // the result takes the unmerged values
    if (kSlow && de) {
      st.M[r] = P::max(st.BM[r], st.M[r]);
      st.X[r] = P::max(st.BX[r], st.X[r]);
      st.Y[r] = P::max(st.BY[r], st.Y[r]);
    }
    qX = pr.insertion(st.M[r], st.X[r], r);
  }
  st.xs = qX;
  st.ts = T;
}

// One PD forward step: events, then the column. kEv = false compiles the event code out, for steps where no
// lane of the warp has an event. kCarry = true gives lane 0 the row above from the state's carry values
// (strip-mined reads); otherwise lane 0 starts with a padding row, for which the row above is
// zero. kGeneric = true decides priors by comparing bytes (PdRows::prior_generic) instead of by class bits.
template <class P, int R, bool kEv = true, bool kCarry = false, bool kGeneric = false>
__device__ __forceinline__ void pd_step(const LaunchArgs& a, const Program& prog, const ReadRef* rd, int lane,
                                        const PdRows<P, R>& pr, const typename P::V& an, PdScratch<P, R>& sc,
                                        PdState<P, R>& st, int synth_len, uint32_t ev, uint32_t sig) {
  using V = typename P::V;
  using S = typename P::S;
  using L = PdLayout<P, R>;
  V qX = P::up(st.xs), T = P::up(st.ts);
  if (lane == 0) {
    qX = kCarry ? st.cX : P::zero();
    T = kCarry ? st.cT : P::zero();
  }
  // END and ACC act in the last lane alone (the read's last row); the other lanes pass them by
  // without entering the event code, which every lane otherwise reaches at its own step.
  if (kEv && (ev & (lane == 31 ? kEvMask : (kEvMask & ~(EV_END | EV_ACC))))) {
    if (ev & EV_SNAP) {
      const uint32_t slot = ev >> kPdPayloadShift;
      V* dst[2] = {slot != kPdPayloadNone ? sc.slot(static_cast<int>(slot), lane) : nullptr,
                   (ev & EV_STAGE) ? sc.staged(st.seg_i + 1, lane) : nullptr};
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        V* o = dst[k];
        if (!o) continue;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          o[r] = st.M[r];
          o[R + r] = st.X[r];
          o[2 * R + r] = st.Y[r];
          o[3 * R + r] = st.BM[r];
          o[4 * R + r] = st.BX[r];
          o[5 * R + r] = st.BY[r];
        }
        o[6 * R] = st.acc;
      }
    }
    if ((ev & EV_END) && lane == 31) {
#pragma unroll
      for (int c = 0; c < P::NC; ++c) sc.raw(st.seg_i, c) = static_cast<double>(P::get(st.acc, c));
    }
    if (ev & EV_BEGIN) {
      ++st.seg_i;
      // A recomputation stream (FP64 only) has one unshared segment from the origin and no record.
      const bool synth = synth_len > 0;
      const Segment* rec = a.v.segs + prog.seg_off + st.seg_i;
      if (!synth && st.seg_i + 1 < prog.n_segs) prefetch_l1(rec + 1);
      const int next_slot = synth ? -1 : rec->next_slot;
      if (!synth && rec->staged) {
        __pipeline_wait_prior(0);
        const V* s = sc.staged(st.seg_i, lane);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          st.M[r] = s[r];
          st.X[r] = s[R + r];
          st.Y[r] = s[2 * R + r];
          st.BM[r] = s[3 * R + r];
          st.BX[r] = s[4 * R + r];
          st.BY[r] = s[5 * R + r];
        }
        st.acc = s[6 * R];
      } else {
        // The origin: the row-0 constant in the padding rows, zero branch values (GATK never writes
        // branch column zero).
        const S in_s = synth ? static_cast<S>(Consts<P::kDouble>::kInitial / synth_len)
                             : (P::kDouble ? static_cast<S>(rec->init_d) : static_cast<S>(rec->init_f));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          st.M[r] = st.X[r] = st.BM[r] = st.BX[r] = st.BY[r] = P::zero();
#pragma unroll
          for (int c = 0; c < P::NC; ++c) P::put(st.Y[r], c, lane * R + r < rd[c].pad ? in_s : S(0));
        }
        st.acc = P::zero();
      }
      if (next_slot >= 0) prefetch(sc.staged(st.seg_i + 1, lane), sc.slot(next_slot, lane), L::kSnap);
    }
  }
  auto prior = [&](int r) { return kGeneric ? pr.prior_generic(ev, r) : pr.prior(sig, r); };
  if (__any_sync(kFull, (ev & kPdSlowMask) != 0)) {
    const bool de = (ev & PD_DE) != 0, mat = (ev & PD_MAT) != 0;
    const uint32_t s_first = (ev >> kPdFirstShift) & 3u, s_later = (ev >> kPdLaterShift) & 3u;
    if (__all_sync(kFull, s_first == s_later)) {
      // Every row of each lane in one deletion state (the read's first row starts NORMAL, the later
      // rows in the state the row above ended in; the two differ only when a deletion runs to the
      // haplotype's end): a column carrying either flag keeps V(left) as the branch values unless
      // inside a deletion, one predicate a lane.
      const bool keep = mat && s_later != kPdInsideDel;
      pd_rows_down<P, R, true>(pr, st, an, qX, T, de, prior, [&](int r) {
        if (keep) {
          st.BM[r] = st.M[r];
          st.BX[r] = st.X[r];
          st.BY[r] = st.Y[r];
        }
      });
    } else {
      // Some lane's first read row is in another state than its later rows.
      pd_rows_down<P, R, true>(pr, st, an, qX, T, de, prior, [&](int r) {
        bool inside[P::NC];
#pragma unroll
        for (int c = 0; c < P::NC; ++c) inside[c] = ((lane * R + r == rd[c].pad) ? s_first : s_later) == kPdInsideDel;
        if (mat) {
          st.BM[r] = P::sel(inside[0], inside[P::NC - 1], st.BM[r], st.M[r]);
          st.BX[r] = P::sel(inside[0], inside[P::NC - 1], st.BX[r], st.X[r]);
          st.BY[r] = P::sel(inside[0], inside[P::NC - 1], st.BY[r], st.Y[r]);
        }
      });
    }
  } else {
    pd_rows_down<P, R, false>(pr, st, an, qX, T, false, prior, [](int) {});
  }
}

// Entry p of a recomputation stream: the haplotype's forward entries (code and deletion bits),
// BEGIN on the first column and END after the last.
__device__ __forceinline__ uint32_t pd_synth_entry(const uint32_t* seq, int len, int p) {
  if (p < 0 || p > len) return 0u;
  uint32_t e = p < len ? __ldg(seq + p) : 0u;
  if (p == 0) e |= EV_BEGIN;
  if (p == len) e |= EV_END;
  return e;
}

template <class P, int R>
__device__ __forceinline__ void pd_forward_pass(const LaunchArgs& a, const Program& prog, const ReadRef* rd, const uint8_t* classes,
                                                const uint32_t* sigs, int lane, PdScratch<P, R>& sc, const uint32_t* synth_seq,
                                                int synth_len) {
  using V = typename P::V;
  using S = typename P::S;
  PdRows<P, R> pr;
  pr.load(a.v, rd, lane, classes);
  V an;
#pragma unroll
  for (int c = 0; c < P::NC; ++c)
    P::put(an, c, static_cast<S>((P::kTransformed && rd[c].len > 0) ? err_prob(a.v, a.v.ins[rd[c].off + rd[c].len - 1]) : 1.0));

  PdState<P, R> st;
  st.clear();
  if (P::kDouble && synth_len > 0) {
    const int n = synth_len;
    auto at = [&](int t) {
      const uint32_t e = pd_synth_entry(synth_seq, n, t - lane);
      pd_step<P, R>(a, prog, rd, lane, pr, an, sc, st, synth_len, e, __ldg(sigs + (e & kCodeMask)));
    };
    int t = 0;
    for (; t < 32; ++t) at(t);
    // Every lane strictly inside the haplotype: no events. An entry is loaded two steps ahead and its
    // signature one, so neither load waits on the other.
    const uint32_t* seq = synth_seq - lane;
    if (t < n) {
      auto entry = [&](int i) { return i < n ? __ldg(seq + i) : 0u; };
      uint32_t e0 = entry(t), e1 = entry(t + 1), g0 = __ldg(sigs + (e0 & kCodeMask));
#pragma unroll 2
      for (; t < n; ++t) {
        const uint32_t e2 = entry(t + 2), g1 = __ldg(sigs + (e1 & kCodeMask));
        pd_step<P, R, false>(a, prog, rd, lane, pr, an, sc, st, synth_len, e0, g0);
        e0 = e1;
        e1 = e2;
        g0 = g1;
      }
    }
    for (; t < n + 32; ++t) at(t);
  } else {
    const int n = prog.fwd_len;
    const uint32_t* stream = a.v.stream + prog.fwd_off - lane;
    // Two steps an iteration; one where no lane has an event runs a body without event code.
    const uint32_t keep = lane == 31 ? kEvMask : (kEvMask & ~(EV_END | EV_ACC));
    uint32_t n0 = __ldg(stream), n1 = __ldg(stream + 1);
    uint32_t g0 = __ldg(sigs + (n0 & kCodeMask)), g1 = __ldg(sigs + (n1 & kCodeMask));
    for (int t = 0; t < n + 32; t += 2) {
      const uint32_t e0 = n0, e1 = n1, s0 = g0, s1 = g1;
      n0 = __ldg(stream + t + 2);
      n1 = __ldg(stream + t + 3);
      g0 = __ldg(sigs + (n0 & kCodeMask));
      g1 = __ldg(sigs + (n1 & kCodeMask));
      if (__any_sync(kFull, (e0 | e1) & keep)) {
        pd_step<P, R>(a, prog, rd, lane, pr, an, sc, st, 0, e0, s0);
        pd_step<P, R>(a, prog, rd, lane, pr, an, sc, st, 0, e1, s1);
      } else {
        pd_step<P, R, false>(a, prog, rd, lane, pr, an, sc, st, 0, e0, s0);
        pd_step<P, R, false>(a, prog, rd, lane, pr, an, sc, st, 0, e1, s1);
      }
    }
  }
  __pipeline_wait_prior(0);
}

// Thresholds, log10 and the caller's layout (fgkl kernel.rs:897-914 via pd_kernel.rs:262-270).
template <class P, int R>
__device__ __forceinline__ void pd_finalize(const LaunchArgs& a, const Task& task, const Region& region, const Program& prog, int lane,
                            PdScratch<P, R>& sc) {
  using C = Consts<P::kDouble>;
  __syncwarp();
  if (P::kDouble && task.hap >= 0) {
    const double raw = sc.raw(0, 0);
    const double result = raw != raw ? __longlong_as_double(0x7ff8000000000000ll) : log10(raw) - C::kLog10Initial;
    const int read_local = task.read[0] - region.read_off;
    for (int k = lane; k < region.n_haps; k += 32) {
      const HapInfo info = a.v.haps[region.hap_off + k];
      if (info.src == task.hap) a.v.out[region.out_off + static_cast<int64_t>(read_local) * region.n_haps + info.order] = result;
    }
    return;
  }
  // A dense read's recomputation (only_lost) fills in only the pairs the first pass lost; a PD program
  // has no joins, so in FP64 it loses none.
  const bool dense = a.only_lost != 0;
  unsigned long long lost_count = 0;
  for (int k = lane; k < region.n_haps; k += 32) {
    const HapInfo info = a.v.haps[region.hap_off + k];
    const int own = info.seg - prog.seg_first;  // another task's, outside the program's segments
    if (own < 0 || own >= prog.n_segs) continue;
    const double factor = a.v.segs[prog.seg_off + own].factor;
#pragma unroll
    for (int c = 0; c < P::NC; ++c) {
      if (task.read[c] < 0) continue;
      const int read_local = task.read[c] - region.read_off;
      double* dst = a.v.out + region.out_off + static_cast<int64_t>(read_local) * region.n_haps + info.order;
      if (dense && !isnan(*dst)) continue;
      const double raw = __dmul_rn(sc.raw(own, c), factor);
      bool lost = a.min_accept_plain ? !(raw >= C::kMinAccepted) : (raw != raw);
      if (!P::kDouble) lost |= isinf(raw);
      const double result = lost ? __longlong_as_double(0x7ff8000000000000ll) : log10(raw) - C::kLog10Initial;
      *dst = result;
      lost_count += lost;
    }
  }
  if (lost_count && !dense) {
    atomicAdd(&a.v.counters->lost_pairs, lost_count);
    if (R > 8) atomicAdd(&a.v.counters->lost_wide, lost_count);
  }
}

// Resident blocks of 4 warps the register budget is cut for. Two reads a warp at 5 rows: three (168
// registers, a few spilled values; 256 regions of 64 reads x 16 haplotypes 8.8 ms, 9.8 at two); one read
// a warp: four up to 6 rows and fewer above, where four spill (41 reads of 342 bases, 12 rows: 2.75 ms at
// two, 6.3 at four); FP64 three up to 5 rows. Two reads on 16 lanes each in scalar FP32 at 10 rows measured
// the same as two on 32 lanes in FP32x2 (8.8 ms).
template <class P, int R>
struct PdMinBlocks {
  static constexpr int value = P::kDouble ? (R <= 5 ? 3 : 1) : (P::NC == 2 ? (R <= 5 ? 3 : 2) : (R <= 6 ? 4 : R <= 9 ? 3 : 2));
};

template <class P, int R>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, (PdMinBlocks<P, R>::value)) pd_kernel(LaunchArgs a) {
  using V = typename P::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int warp_in_block = threadIdx.x >> 5;
  const int warp = blockIdx.x * static_cast<int>(blockDim.x >> 5) + warp_in_block;
  V* smem = reinterpret_cast<V*>(smem_raw + warp_in_block * PdLayout<P, R>::kSmemPerWarp);
  const int count = a.count ? min(*a.count, a.n_tasks) : a.n_tasks;
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(a.task_counter, 1);
    t = __shfl_sync(kFull, t, 0);
    if (t >= count) break;
    const Task task = a.tasks[t];
    const Region region = a.v.regions[task.region];
    const Program prog = a.v.progs[task.prog];
    ReadRef rd[P::NC];
#pragma unroll
    for (int c = 0; c < P::NC; ++c) {
      const int id = task.read[c];
      if (id >= 0) {
        rd[c].off = a.v.read_off[id];
        rd[c].len = static_cast<int>(a.v.read_off[id + 1] - rd[c].off);
      } else {
        rd[c].off = 0;
        rd[c].len = 0;
      }
      rd[c].pad = 32 * R - rd[c].len;
    }
    const uint8_t* classes = a.v.code_of_byte + region.code_off;
    const uint32_t* sigs = a.v.pd_sigs + region.sig_off;
    char* scratch = a.scratch + static_cast<size_t>(warp) * a.scratch_stride;
    if (P::kDouble && task.hap >= 0) {
      const HapInfo info = a.v.haps[region.hap_off + task.hap];
      PdScratch<P, R> sc(scratch, smem, 0);
      pd_forward_pass<P, R>(a, prog, rd, classes, sigs, lane, sc, a.v.pd_entries + region.seq_off + info.seq, info.len);
      pd_finalize<P, R>(a, task, region, prog, lane, sc);
    } else {
      PdScratch<P, R> sc(scratch, smem, prog.n_slots);
      pd_forward_pass<P, R>(a, prog, rd, classes, sigs, lane, sc, nullptr, 0);
      pd_finalize<P, R>(a, task, region, prog, lane, sc);
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// Strip-mined PD pairs (reads longer than 620 bases), every pair of a region whose reads hold more distinct
// bytes than the class bits cover (kGeneric), and the FP64 recomputation of reads above 248 bases, whose
// rows in one block would not fit the registers: one read against one distinct haplotype, unshared, over
// the haplotype's forward entries, the rows cut into blocks of 32 R rows that the warps of a block run as a
// pipeline (the plain strip-mined kernel's scheme, kernels.cu). The first block's row above is GATK's row 0
// (M = X = 0, Y = INITIAL / hap_len). The state a block's top row starts in is the previous row's, which
// the entries' later-row state carries; only the read's first row (in the first block) takes the first-row
// state.
// ---------------------------------------------------------------------------------------------

template <class P>
constexpr size_t pd_long_scratch_size(int max_hap_len) {
  return static_cast<size_t>(max_hap_len) * sizeof(Carry<P>);
}

template <class P>
constexpr size_t pd_long_smem_per_warp() {
  return kRing * sizeof(Carry<P>);
}

// One superstep of a warp: steps t0 .. t0 + kChunk - 1. kInner: every lane is strictly inside the haplotype
// throughout, so no events and no bounds.
template <class P, int R, bool kGeneric, bool kInner>
__device__ __forceinline__ void pd_long_superstep(const LaunchArgs& a, const ReadRef* rd, int lane, const PdRows<P, R>& pr,
                                                  typename P::V an, PdScratch<P, R>& sc, PdState<P, R>& st, const uint32_t* seq,
                                                  const uint32_t* sigs, int n, int t0, const Carry<P>* in, Carry<P>* out,
                                                  int out_mask) {
  const Program prog{};
  // An entry is loaded two steps ahead and its signature one.
  auto entry = [&](int i) { return kInner ? (i < kChunk ? __ldg(seq + t0 + i - lane) : 0u) : pd_synth_entry(seq, n, t0 + i - lane); };
  auto signature = [&](uint32_t e) { return kGeneric ? 0u : __ldg(sigs + (e & kCodeMask)); };
  uint32_t e0 = entry(0), e1 = entry(1), g0 = signature(e0);
#pragma unroll 2
  for (int i = 0; i < kChunk; ++i) {
    const int t = t0 + i;
    const uint32_t e = e0, sig = g0;
    e0 = e1;
    g0 = signature(e0);
    e1 = entry(i + 2);
    const Carry<P> c = in[t & (kRing - 1)];
    st.cX = c.x;
    st.cT = c.t;
    pd_step<P, R, !kInner, true, kGeneric>(a, prog, rd, lane, pr, an, sc, st, n, e, sig);
    const int p = t - 31;  // lane 31's column
    if (lane == 31 && out && (kInner || (p >= 0 && p < n))) out[p & out_mask] = Carry<P>{st.xs, st.ts};
  }
}

template <class P, int R, bool kGeneric>
__global__ void __launch_bounds__(kLongWarps * 32, 1) pd_long_kernel(LaunchArgs a) {
  using V = typename P::V;
  using S = typename P::S;
  using C = Consts<P::kDouble>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_task;
  __shared__ double s_raw[kLongWarps][kMaxReads];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  Carry<P>* const ring = reinterpret_cast<Carry<P>*>(smem_raw) + w * kRing;  // what the warp's top row takes
  const int count = a.count ? min(*a.count, a.n_tasks) : a.n_tasks;
  // The block's scratch: one carry entry a column, from the last warp of a round to the first of the next.
  Carry<P>* const carry = reinterpret_cast<Carry<P>*>(a.scratch + static_cast<size_t>(blockIdx.x) * a.scratch_stride);
  PdScratch<P, R> sc(nullptr, nullptr, 0);
  sc.seg_raw = s_raw[w];
  for (;;) {
    if (threadIdx.x == 0) s_task = atomicAdd(a.task_counter, 1);
    __syncthreads();
    const int task_i = s_task;
    if (task_i >= count) break;
    const Task task = a.tasks[task_i];
    const Region region = a.v.regions[task.region];
    const HapInfo info = a.v.haps[region.hap_off + task.hap];
    const uint32_t* seq = a.v.pd_entries + region.seq_off + info.seq;
    const uint32_t* sigs = a.v.pd_sigs + region.sig_off;
    const uint8_t* classes = a.v.code_of_byte + region.code_off;
    const int n = info.len;
    ReadRef rd[1];
    rd[0].off = a.v.read_off[task.read[0]];
    rd[0].len = static_cast<int>(a.v.read_off[task.read[0] + 1] - rd[0].off);
    const int blocks = long_blocks(rd[0].len, R);
    const int pad0 = 32 * R * blocks - rd[0].len;
    const V an = static_cast<S>(P::kTransformed ? err_prob(a.v, a.v.ins[rd[0].off + rd[0].len - 1]) : 1.0);
    for (int b0 = 0; b0 < blocks; b0 += warps) {
      const int in_round = min(warps, blocks - b0), b = b0 + w;
      const bool on = w < in_round;
      PdRows<P, R> pr;
      PdState<P, R> st;
      st.clear();
      Carry<P> next{S(0), S(0)};  // the first warp's input for column t0 + kChunk + lane
      if (on) {
        rd[0].pad = pad0 - 32 * R * b;
        if (kGeneric)
          pr.load_generic(a.v, rd, lane, classes);
        else
          pr.load(a.v, rd, lane, classes);
        if (b == 0) {
          // GATK's row 0 above the first block. Below a padding row nothing reads it.
          if (pad0 == 0) {
            const BracketFactors<P> k(row_model(a.v, rd[0], 0, classes));
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
            pd_long_superstep<P, R, kGeneric, true>(a, rd, lane, pr, an, sc, st, seq, sigs, n, t0, ring, out, out_mask);
          else
            pd_long_superstep<P, R, kGeneric, false>(a, rd, lane, pr, an, sc, st, seq, sigs, n, t0, ring, out, out_mask);
        }
        __syncthreads();
      }
    }
    if (w == 0) {
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
void pd_occ(int* blocks, int warps) {
  static std::atomic<int> cache[3][kMaxDevices];
  *blocks = resident_blocks(pd_kernel<P, R>, warps * PdLayout<P, R>::kSmemPerWarp, warps * 32, cache[warps_index(warps)],
                            kWarpsPerBlock * PdLayout<P, R>::kSmemPerWarp);
}

template <class P, int R>
cudaError_t pd_go(int blocks, const LaunchArgs& a, cudaStream_t s, int warps) {
  const size_t smem = warps * PdLayout<P, R>::kSmemPerWarp;
  pd_kernel<P, R><<<blocks, warps * 32, smem, s>>>(a);
  return cudaGetLastError();
}

// Rows-per-lane dispatch over 1..8 and 10..20 (even), FP32 or FP64.
template <class P, class F>
auto pd_rows(int rows, F&& f) {
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


// Rows 1..8 only (the packed two-read form).
template <class F>
auto pd_rows8(int rows, F&& f) {
  switch (rows) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 5: return f(std::integral_constant<int, 5>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 7: return f(std::integral_constant<int, 7>{});
    default: return f(std::integral_constant<int, 8>{});
  }
}

template <class F>
auto pd_long_rows(int rows, F&& f) {
  switch (rows) {
    case 4: return f(std::integral_constant<int, 4>{});
    case 6: return f(std::integral_constant<int, 6>{});
    default: return f(std::integral_constant<int, 8>{});
  }
}

template <class P, int R, bool kGeneric>
void pd_long_occ(int* blocks, int warps) {
  static std::atomic<int> cache[kLongWarps + 1][kMaxDevices];
  *blocks = resident_blocks(pd_long_kernel<P, R, kGeneric>, warps * pd_long_smem_per_warp<P>(), warps * 32, cache[warps],
                            kLongWarps * pd_long_smem_per_warp<P>());
}

template <class P, int R, bool kGeneric>
void pd_long_go(int blocks, const LaunchArgs& a, cudaStream_t s, int warps) {
  pd_long_kernel<P, R, kGeneric><<<blocks, warps * 32, warps * pd_long_smem_per_warp<P>(), s>>>(a);
}

}  // namespace

size_t pd_long_scratch_bytes(Kind k, int, int max_hap_len) {
  const bool dbl = k == Kind::kLongF64Pd || k == Kind::kGenericF64Pd;
  return dbl ? pd_long_scratch_size<OneF64>(max_hap_len) : pd_long_scratch_size<OneF32>(max_hap_len);
}

void pd_long_occupancy(Kind k, int rows, int* blocks, int* threads, int warps) {
  *threads = warps * 32;
  *blocks = 0;
  pd_long_rows(rows, [&](auto r) {
    constexpr int R = decltype(r)::value;
    switch (k) {
      case Kind::kLongF32Pd: pd_long_occ<OneF32, R, false>(blocks, warps); break;
      case Kind::kLongF64Pd: pd_long_occ<OneF64, R, false>(blocks, warps); break;
      case Kind::kGenericF32Pd: pd_long_occ<OneF32, R, true>(blocks, warps); break;
      case Kind::kGenericF64Pd: pd_long_occ<OneF64, R, true>(blocks, warps); break;
      default: break;
    }
    return 0;
  });
}

cudaError_t pd_long_launch(Kind k, int rows, int blocks, const LaunchArgs& a, cudaStream_t s, int warps) {
  return pd_long_rows(rows, [&](auto r) -> cudaError_t {
    constexpr int R = decltype(r)::value;
    switch (k) {
      case Kind::kLongF32Pd: pd_long_go<OneF32, R, false>(blocks, a, s, warps); break;
      case Kind::kLongF64Pd: pd_long_go<OneF64, R, false>(blocks, a, s, warps); break;
      case Kind::kGenericF32Pd: pd_long_go<OneF32, R, true>(blocks, a, s, warps); break;
      case Kind::kGenericF64Pd: pd_long_go<OneF64, R, true>(blocks, a, s, warps); break;
      default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
  });
}

size_t pd_scratch_bytes(PdForm form, int rows, int max_slots, int max_segs) {
  switch (form) {
    case PdForm::kOneF64:
      return pd_rows<OneF64>(rows, [&](auto r) { return pd_scratch_size<OneF64, decltype(r)::value>(max_slots, max_segs); });
    case PdForm::kPackedF32:
      return pd_rows8(rows, [&](auto r) { return pd_scratch_size<PackedF32, decltype(r)::value>(max_slots, max_segs); });
    default:
      return pd_rows<OneF32>(rows, [&](auto r) { return pd_scratch_size<OneF32, decltype(r)::value>(max_slots, max_segs); });
  }
}

void pd_occupancy(PdForm form, int rows, int* blocks, int* threads, int warps) {
  *threads = warps * 32;
  *blocks = 0;
  switch (form) {
    case PdForm::kOneF64:
      pd_rows<OneF64>(rows, [&](auto r) {
        pd_occ<OneF64, decltype(r)::value>(blocks, warps);
        return 0;
      });
      break;
    case PdForm::kPackedF32:
      pd_rows8(rows, [&](auto r) {
        pd_occ<PackedF32, decltype(r)::value>(blocks, warps);
        return 0;
      });
      break;
    default:
      pd_rows<OneF32>(rows, [&](auto r) {
        pd_occ<OneF32, decltype(r)::value>(blocks, warps);
        return 0;
      });
  }
}

cudaError_t pd_launch(PdForm form, int rows, int blocks, const LaunchArgs& a, cudaStream_t s, int warps) {
  switch (form) {
    case PdForm::kOneF64:
      return pd_rows<OneF64>(rows, [&](auto r) { return pd_go<OneF64, decltype(r)::value>(blocks, a, s, warps); });
    case PdForm::kPackedF32:
      return pd_rows8(rows, [&](auto r) { return pd_go<PackedF32, decltype(r)::value>(blocks, a, s, warps); });
    default:
      return pd_rows<OneF32>(rows, [&](auto r) { return pd_go<OneF32, decltype(r)::value>(blocks, a, s, warps); });
  }
}

}  // namespace fgkl

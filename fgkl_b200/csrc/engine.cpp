#include "engine.h"

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstddef>
#include <cstring>
#include <deque>
#include <exception>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <thread>

#include "../../include/fgkl_b200.h"
#include "planner.h"
#include "tables.h"

namespace fgkl {

namespace {
std::atomic<int64_t> g_allocation_limit{0};
}  // namespace

int64_t allocation_limit() { return g_allocation_limit.load(std::memory_order_relaxed); }
int64_t set_allocation_limit(int64_t bytes) { return g_allocation_limit.exchange(bytes); }

bool over_allocation_limit(size_t bytes) {
  const int64_t lim = allocation_limit();
  return lim > 0 && bytes > static_cast<size_t>(lim);
}

cudaError_t device_alloc(void** p, size_t bytes) {
  const int64_t lim = allocation_limit();
  if (lim > 0 && bytes > static_cast<size_t>(lim)) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaMalloc(p, bytes);
}

cudaError_t pinned_alloc(void** p, size_t bytes) {
  const int64_t lim = allocation_limit();
  if (lim > 0 && bytes > static_cast<size_t>(lim)) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaMallocHost(p, bytes);
}

namespace {

constexpr int kWarpsPerBlock = 4;

// Rows per lane: lane 0 holds only padding rows, so 31 * rows >= len.
int packed_rows(int len) { return (len + 30) / 31; }

size_t align_up(size_t x, size_t a = 256) { return (x + a - 1) / a * a; }

// Rows per lane for one read on the single-read kinds: 31 * rows >= len, even above 8.
int single_rows(int len) {
  int rows = packed_rows(len);
  if (rows > 8) rows = (rows + 1) & ~1;
  return rows;
}

}  // namespace

struct RegionPlan {
  std::unique_ptr<SortedHaps> set;  // until its programs are emitted, as fwd.segs
  ForwardPlan fwd;
  std::vector<ProgramBuild> progs;
  std::vector<HapInfo> haps;
  std::vector<uint8_t> seq;        // prior codes of the distinct sorted haplotypes, concatenated
  std::vector<uint32_t> pd_seq;    // PD: their forward entries (code and deletion bits)
  std::vector<uint32_t> pd_sigs;   // PD: per match-set code, the read classes it accepts
  std::string error;               // a region the kernels cannot take
  uint8_t codes[256];
  SharedColumns cols;
  uint64_t read_bases = 0, hap_bases = 0;
  int n_distinct = 0;
  bool extra_codes = false;  // a haplotype byte outside ACGTN: the region runs on the FP64 kernel
  bool generic = false;      // PD: more read bytes than class bits, or more than 256 match sets
};

namespace {

// PD regions: the reads' distinct bytes become classes 0..30 (first-seen order) and each match-set
// code the bit set of classes it accepts, so the kernel's prior is one bit test per row.
bool pd_read_classes(const BatchInput& in, int64_t first_read, int n_reads, const SortedHaps& s, RegionPlan& out) {
  std::memset(out.codes, kNoCode, 256);
  std::vector<uint8_t> bytes;
  for (int r = 0; r < n_reads; ++r)
    for (int64_t o = in.read_off[first_read + r]; o < in.read_off[first_read + r + 1]; ++o) {
      const uint8_t b = in.bases[o];
      if (out.codes[b] != kNoCode) continue;
      if (static_cast<int>(bytes.size()) >= kPdMaxReadClasses) return false;
      out.codes[b] = static_cast<uint8_t>(bytes.size());
      bytes.push_back(b);
    }
  out.pd_sigs.assign(s.match_sets.size(), 0u);
  for (size_t code = 0; code < s.match_sets.size(); ++code)
    for (size_t c = 0; c < bytes.size(); ++c)
      if (s.match_sets[code].accepts(bytes[c])) out.pd_sigs[code] |= 1u << c;
  return true;
}

// Emits a planned region's programs: its segments in `chunks` runs at most. Gives the sorted set back.
void emit_region(RegionPlan& plan, int chunks) {
  const std::vector<int32_t> bounds = split_segments(plan.fwd, chunks);
  plan.progs.resize(bounds.size() - 1);
  try {
    for (size_t c = 0; c + 1 < bounds.size(); ++c) emit_program(*plan.set, plan.fwd, bounds[c], bounds[c + 1], plan.progs[c]);
  } catch (const std::exception& e) {
    plan.error = e.what();
  }
  plan.set.reset();
  plan.fwd.segs = {};
}

// `whole`: the region's one program is emitted here too and the sorted set, most of a plan's memory, given
// back; else emit_region follows.
void plan_region(const BatchInput& in, int g, int64_t first_read, int64_t first_hap, bool share, bool whole, RegionPlan& out) {
  const int n_haps = in.region_haps[g], n_reads = in.region_reads[g];
  std::vector<HapView> views(static_cast<size_t>(n_haps));
  std::vector<const uint8_t*> flags(in.hap_flags ? static_cast<size_t>(n_haps) : 0);
  for (int h = 0; h < n_haps; ++h) {
    const int64_t lo = in.hap_off[first_hap + h], hi = in.hap_off[first_hap + h + 1];
    views[h] = HapView{in.hap_bases + lo, static_cast<int32_t>(hi - lo)};
    if (in.hap_flags) flags[h] = in.hap_flags + lo;
    out.hap_bases += static_cast<uint64_t>(hi - lo);
  }
  for (int r = 0; r < n_reads; ++r)
    out.read_bases += static_cast<uint64_t>(in.read_off[first_read + r + 1] - in.read_off[first_read + r]);
  if (n_haps == 0 || n_reads == 0) return;
  const bool pd = in.hap_flags != nullptr;
  out.set = std::make_unique<SortedHaps>();
  SortedHaps& s = *out.set;
  try {
    s = pd ? SortedHaps::make_pd(views, flags) : SortedHaps::make(views, share);
    out.fwd = forward_plan(s, share && !pd);
  } catch (const std::exception& e) {
    out.error = e.what();
    return;
  }
  if (pd) {
    // Regions the class bits cannot describe compare bytes in the kernel instead (every pair then
    // runs unshared, as fgkl's answer for them does not depend on sharing).
    out.generic = s.too_many_sets || !pd_read_classes(in, first_read, n_reads, s, out);
    if (out.generic) out.pd_sigs.clear();
  } else {
    code_table(s, out.codes);
    out.extra_codes = s.num_codes() > 5;
  }
  out.cols = s.columns();
  out.haps.resize(static_cast<size_t>(n_haps));
  int seg = -1, src = 0;
  for (int k = 0; k < n_haps; ++k) {
    if (!s.dup[k]) {
      ++seg;
      src = k;
      if (pd) {
        out.haps[k].seq = static_cast<int32_t>(out.pd_seq.size());
        for (int32_t j = 0; j < s.bases[k].len; ++j) {
          if (out.generic) {
            // The column's own byte and ALT bits (shifted to bit 0) in place of a match-set code.
            const MatchSet set = MatchSet::of(s.bases[k].bases[j], s.flags[k][j]);
            out.pd_seq.push_back(set.base | (static_cast<uint32_t>(set.alts >> 3) << kPdPayloadShift) | s.pd_bits[k][j]);
          } else {
            out.pd_seq.push_back(s.codes[k][j] | s.pd_bits[k][j]);
          }
        }
      } else {
        out.haps[k].seq = static_cast<int32_t>(out.seq.size());
        out.seq.insert(out.seq.end(), s.codes[k].begin(), s.codes[k].end());
      }
      ++out.n_distinct;
    } else {
      out.haps[k].seq = out.haps[src].seq;
    }
    HapInfo& h = out.haps[k];
    h.order = s.order[k];
    h.seg = seg;
    h.src = src;
    h.len = s.bases[k].len;
    h.pad_[0] = h.pad_[1] = h.pad_[2] = 0;
  }
  if (whole) emit_region(out, 1);
}

// The process's helper threads. They are started when a loop asks for them, wait for the next one, and
// end after two idle seconds (starting a loop's threads anew took 10-20 us each, 100-200 us of the
// planning of a batch of a few regions). They run host code only and make no CUDA call. Never destroyed:
// a helper that waits when the process exits holds nothing. Loops of several callers share the helpers;
// a caller works on its own loop beside them and never waits for one that has not begun on it, so a
// process that cannot start any runs its loops by itself.
class Helpers {
 public:
  // The process's own. A forked child has none of its parent's threads, but copies of the lock and the
  // condition variables that they may have held or waited on, which must not be used again: it gets
  // helpers of its own.
  static Helpers& get() {
    static std::atomic<Helpers*> current{nullptr};
    const pid_t self = getpid();
    Helpers* h = current.load(std::memory_order_acquire);
    while (!h || h->owner_ != self) {
      Helpers* const fresh = new Helpers(self);
      if (current.compare_exchange_strong(h, fresh, std::memory_order_acq_rel)) return *fresh;
      delete fresh;  // another thread was first; no helper has been started on this one
    }
    return *h;
  }

  // Runs work() on the calling thread and on up to `more` helpers at once; returns when all are done. An
  // exception of any of them is thrown here, after the others have ended.
  void run(int more, const std::function<void()>& work) {
    Job job{&work, 0, nullptr};
    {
      std::lock_guard<std::mutex> lock(m_);
      try {
        for (int i = 0; i < more; ++i) tickets_.push_back(&job);
        const int wanted = std::min(static_cast<int>(tickets_.size()), kMost);
        while (idle_ + starting_ < wanted && total_ < kMost) {
          std::thread([this] { help(); }).detach();
          ++total_;
          ++starting_;
        }
      } catch (const std::exception&) {
        // Fewer helpers than asked for: the caller does what they would have done.
      }
    }
    wake_.notify_all();
    do_work(job);
    std::unique_lock<std::mutex> lock(m_);
    tickets_.erase(std::remove(tickets_.begin(), tickets_.end(), &job), tickets_.end());
    done_.wait(lock, [&] { return job.active == 0; });
    if (job.error) std::rethrow_exception(job.error);
  }

 private:
  struct Job {
    const std::function<void()>* work;
    int active;
    std::exception_ptr error;
  };
  static constexpr int kMost = 64;

  explicit Helpers(pid_t owner) : owner_(owner) {}

  void do_work(Job& job) {
    try {
      (*job.work)();
    } catch (...) {
      std::lock_guard<std::mutex> lock(m_);
      if (!job.error) job.error = std::current_exception();
    }
  }

  void help() {
    std::unique_lock<std::mutex> lock(m_);
    --starting_;
    for (;;) {
      ++idle_;
      const bool some = wake_.wait_for(lock, std::chrono::seconds(2), [&] { return !tickets_.empty(); });
      --idle_;
      if (!some) break;
      Job* const job = tickets_.front();
      tickets_.pop_front();
      ++job->active;
      lock.unlock();
      do_work(*job);
      lock.lock();
      if (--job->active == 0) done_.notify_all();
    }
    --total_;
  }

  const pid_t owner_;  // the process whose threads these are
  std::mutex m_;
  std::condition_variable wake_, done_;
  std::deque<Job*> tickets_;
  int idle_ = 0, starting_ = 0, total_ = 0;
};

// Runs fn(i) for i in [0, n) on up to `threads` threads, the calling thread among them. Each thread
// takes the next item when it finishes one, so uneven items (regions of 8 to 256 reads) balance.
template <class F>
void parallel_for(int64_t n, int threads, F&& fn) {
  threads = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(threads, n)));
  if (threads == 1) {
    for (int64_t i = 0; i < n; ++i) fn(i);
    return;
  }
  std::atomic<int64_t> next{0};
  Helpers::get().run(threads - 1, [&] {
    for (int64_t i = next.fetch_add(1, std::memory_order_relaxed); i < n; i = next.fetch_add(1, std::memory_order_relaxed))
      fn(i);
  });
}

int host_threads() { return std::max(1, static_cast<int>(std::thread::hardware_concurrency())); }

// The pairs of a strip-mined launch, by their numbers of row blocks.
struct LongPairs {
  struct Of {  // the pairs of one number of row blocks
    double pairs = 0, columns = 0, longest = 0;
  };
  std::vector<Of> by_blocks;
  void add(int blocks, int columns) {
    const size_t at = static_cast<size_t>(std::min(blocks, 4095));  // beyond it all the same
    if (at >= by_blocks.size()) by_blocks.resize(at + 1);
    Of& o = by_blocks[at];
    o.pairs += 1;
    o.columns += columns;
    o.longest = std::max(o.longest, static_cast<double>(columns));
  }
};

// Warps a block of a strip-mined launch of these pairs, on `sms` SMs. A pair's row blocks on W warps take
// ceil(blocks / W) rounds of n + 32 + 64 (W - 1) steps: more warps shorten a pair, fewer waste no steps on
// starting one behind another, nor on rounds that they do not fill. The W with the smallest estimate -- the larger
// of the warps' steps in all at the rate of a busy GPU and the longest pair --, the fewest among equals; a busy
// SM's rate is that of 8 warps (in FP64 of 4.5, one a scheduler and a little). Passes over 6 haplotypes a
// region, 8 warps a block or a read's row blocks, and as chosen: 32 regions of 48 reads of 1,000 bases, PD, the
// FP32 pass 28.9 -> 12.2 ms; 64 regions, plain, 10.3 -> 8.8; 64 regions of reads of 640 bases beside one of
// 3,200, both passes, 8.7 -> 6.4.
int choose_long_warps(Kind kind, int rows, int sms, const LongPairs& of) {
  const int blocks = static_cast<int>(of.by_blocks.size()) - 1, most = blocks > kLongWarps ? kLongWarps : std::max(1, blocks);
  const bool f64 = kind == Kind::kLongF64 || kind == Kind::kLongF64Pd || kind == Kind::kGenericF64Pd;
  const double kBusy = f64 ? 4.5 : 8.0;
  int best = 1;
  double least = -1;
  for (int w = 1; w <= most; ++w) {
    int per_sm = 0, threads = 0;
    long_occupancy(kind, rows, &per_sm, &threads, w);
    if (per_sm <= 0) continue;
    double sum = 0, longest = 0;
    for (int b = 1; b <= blocks; ++b) {
      const LongPairs::Of& o = of.by_blocks[static_cast<size_t>(b)];
      if (o.pairs == 0) continue;
      const double rounds = (b + w - 1) / w, fill = 32 + 64 * (std::min(w, b) - 1);
      sum += rounds * (o.columns + o.pairs * fill) * w;
      longest = std::max(longest, rounds * (o.longest + fill));
    }
    const double time = std::max(sum / (sms * std::min(kBusy, static_cast<double>(per_sm * w))), longest);
    if (least < 0 || time < least) {
      least = time;
      best = w;
    }
  }
  return best;
}

// Copies `bytes` bytes in `chunks` pieces on several threads.
void parallel_copy(uint8_t* dst, const uint8_t* src, size_t bytes) {
  constexpr size_t kChunk = size_t{4} << 20;
  const int64_t chunks = static_cast<int64_t>((bytes + kChunk - 1) / kChunk);
  parallel_for(chunks, std::min(host_threads(), 16), [&](int64_t c) {
    const size_t lo = static_cast<size_t>(c) * kChunk, n = std::min(kChunk, bytes - lo);
    std::memcpy(dst + lo, src + lo, n);
  });
}

}  // namespace

Engine::Engine(int device, cudaStream_t stream) : device_(device), stream_(stream) {
  DeviceGuard device_guard(device_);
  cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, device_);
  if (!stream_) {
    cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking);
    own_stream_ = true;
  }
  const Tables& t = tables();
  cudaMalloc(&d_err_, sizeof(double) * t.error_prob.size());
  cudaMalloc(&d_m2m_, sizeof(double) * t.m2m.size());
  cudaMemcpy(d_err_, t.error_prob.data(), sizeof(double) * t.error_prob.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(d_m2m_, t.m2m.data(), sizeof(double) * t.m2m.size(), cudaMemcpyHostToDevice);
  for (int i = 0; i < kAuxStreams; ++i) {
    cudaStreamCreateWithFlags(&aux_[i], cudaStreamNonBlocking);
    cudaEventCreateWithFlags(&join_[i], cudaEventDisableTiming);
  }
  cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming);
  cudaStreamCreateWithFlags(&copy_, cudaStreamNonBlocking);
  cudaEventCreateWithFlags(&uploaded_, cudaEventDisableTiming);
  cudaEventCreateWithFlags(&computed_, cudaEventDisableTiming);
  cudaEventCreateWithFlags(&fetched_, cudaEventDisableTiming);
}

Engine::~Engine() {
  DeviceGuard device_guard(device_);
  if (stream_) cudaStreamSynchronize(stream_);
  if (copy_) cudaStreamSynchronize(copy_);
  cudaFree(d_reads_);
  cudaFree(d_in_);
  cudaFree(d_queue_);
  cudaFree(d_out_);
  cudaFree(d_scratch_);
  cudaFree(d_err_);
  cudaFree(d_m2m_);
  if (h_stage_) cudaFreeHost(h_stage_);
  if (h_reads_) cudaFreeHost(h_reads_);
  for (int i = 0; i < kAuxStreams; ++i) {
    cudaStreamDestroy(aux_[i]);
    cudaEventDestroy(join_[i]);
  }
  cudaEventDestroy(fork_);
  cudaEventDestroy(uploaded_);
  cudaEventDestroy(computed_);
  cudaEventDestroy(fetched_);
  if (copy_) cudaStreamDestroy(copy_);
  for (cudaEvent_t e : ev_) cudaEventDestroy(e);
  if (own_stream_) cudaStreamDestroy(stream_);
}

int Engine::fail(int code, const std::string& msg) {
  error_ = msg;
  return code;
}

int Engine::check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return FGKL_OK;
  return fail(FGKL_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

template <class T>
T* Engine::grow(T*& ptr, size_t& cap, size_t n) {
  const size_t bytes = std::max<size_t>(n * sizeof(T), 256);
  if (over_allocation_limit(bytes)) return nullptr;  // the buffer held so far is kept
  if (bytes > cap) {
    // Half as much again as the old size: a caller whose batches vary in size stops reallocating
    // after a few calls (cudaFree waits for the whole device, other callers' streams included).
    // The first size gets an eighth more, so that the next batches of its kind fit.
    const size_t want = cap > 0 ? std::max(bytes, cap + cap / 2) : bytes + bytes / 8;
    cudaFree(ptr);
    ptr = nullptr;
    if (device_alloc(reinterpret_cast<void**>(&ptr), want) == cudaSuccess) {
      cap = want;
    } else if (want > bytes && (cudaGetLastError(), device_alloc(reinterpret_cast<void**>(&ptr), bytes) == cudaSuccess)) {
      cap = bytes;
    } else {
      cudaGetLastError();
      cap = 0;
      ptr = nullptr;
      return nullptr;
    }
  }
  return ptr;
}

namespace {
double ms_since(std::chrono::steady_clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}
}  // namespace

namespace {
// Whether [p, p + bytes) lies in one page-locked host allocation (cudaMallocHost, cudaHostAlloc or
// cudaHostRegister): both ends are host memory the device maps, at device addresses `bytes - 1`
// apart. Pageable memory answers false.
bool host_pinned(const void* p, size_t bytes) {
  if (!p || bytes == 0) return false;
  cudaPointerAttributes lo{}, hi{};
  if (cudaPointerGetAttributes(&lo, p) != cudaSuccess ||
      cudaPointerGetAttributes(&hi, static_cast<const uint8_t*>(p) + bytes - 1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (lo.type != cudaMemoryTypeHost || hi.type != cudaMemoryTypeHost || !lo.devicePointer || !hi.devicePointer) return false;
  return static_cast<const uint8_t*>(hi.devicePointer) - static_cast<const uint8_t*>(lo.devicePointer) ==
         static_cast<std::ptrdiff_t>(bytes - 1);
}

// Grows a pinned host buffer to at least `bytes`, by half again at least (cudaFreeHost waits for the
// whole device); false when the allocation fails.
bool grow_pinned(uint8_t*& p, size_t& cap, size_t bytes) {
  if (over_allocation_limit(bytes)) return false;
  if (bytes <= cap) return true;
  const size_t want = cap > 0 ? std::max(bytes, cap + cap / 2) : bytes;
  if (p) cudaFreeHost(p);
  p = nullptr;
  if (pinned_alloc(reinterpret_cast<void**>(&p), want) == cudaSuccess) {
    cap = want;
    return true;
  }
  cudaGetLastError();
  if (want > bytes && pinned_alloc(reinterpret_cast<void**>(&p), bytes) == cudaSuccess) {
    cap = bytes;
    return true;
  }
  cudaGetLastError();
  p = nullptr;
  cap = 0;
  return false;
}

// Runs a callable on a helper thread and joins it when it goes out of scope, so an early return
// from prepare() never leaves the copy running.
class Helper {
 public:
  template <class F>
  explicit Helper(bool on, F&& f) {
    if (on) th_ = std::thread(std::forward<F>(f));
    else f();
  }
  ~Helper() { join(); }
  void join() {
    if (th_.joinable()) th_.join();
  }

 private:
  std::thread th_;
};
}  // namespace

int plan_region_cells(const BatchInput& in, const EngineConfig& cfg, uint64_t* cells, std::string* error) {
  const int N = in.num_regions;
  if (N < 0) return (*error = "negative region count", FGKL_E_INVALID_ARGUMENT);
  std::vector<int64_t> first_read(N + 1, 0), first_hap(N + 1, 0);
  for (int g = 0; g < N; ++g) {
    if (in.region_reads[g] < 0 || in.region_haps[g] < 0) return (*error = "negative region size", FGKL_E_INVALID_ARGUMENT);
    first_read[g + 1] = first_read[g] + in.region_reads[g];
    first_hap[g + 1] = first_hap[g] + in.region_haps[g];
  }
  for (int64_t h = 0; h < first_hap[N]; ++h)
    if (in.hap_off[h + 1] - in.hap_off[h] <= 0) return (*error = "haplotype " + std::to_string(h) + " has no bases", FGKL_E_EMPTY_HAPLOTYPE);
  for (int64_t r = 0; r < first_read[N]; ++r)
    if (in.read_off[r + 1] - in.read_off[r] <= 0) return (*error = "read " + std::to_string(r) + " has no bases", FGKL_E_EMPTY_READ);
  // The cells each region's tasks compute (the counts prepare() gives the launches): reads of one
  // block walk the region's program (forward and backward columns); strip-mined reads and the reads
  // of byte-compared PD regions run each distinct haplotype unshared.
  parallel_for(N, host_threads(), [&](int64_t gi) {
    const int g = static_cast<int>(gi);
    RegionPlan rp;
    plan_region(in, g, first_read[g], first_hap[g], cfg.share_suffixes, false, rp);
    uint64_t distinct_len = 0;
    for (int k = 0; k < static_cast<int>(rp.haps.size()); ++k)
      if (rp.haps[k].src == k) distinct_len += static_cast<uint64_t>(rp.haps[k].len);
    uint64_t c = 0;
    for (int64_t r = first_read[g]; r < first_read[g + 1]; ++r) {
      const uint64_t len = static_cast<uint64_t>(in.read_off[r + 1] - in.read_off[r]);
      if (rp.generic || len > static_cast<uint64_t>(kMaxBlockRead))
        c += len * distinct_len;
      else
        c += len * (rp.fwd.fwd_columns + rp.fwd.bwd_columns);
    }
    cells[g] = rp.error.empty() ? c : 0;
  });
  return FGKL_OK;
}

// How a batch's first pass is spread: see choose_split.
int Engine::SplitRule::chunks(const ForwardPlan& p) const {
  const uint64_t steps = p.steps(), n = static_cast<uint64_t>(p.n_segs);
  if (steps <= limit || n < 2) return 1;
  return static_cast<int>(std::min<uint64_t>(n, (steps + limit - 1) / limit));
}

// Chooses the forms and the split of the first pass. A task's wavefront steps are serial, so a batch with
// few tasks leaves most of the GPU idle while the longest run: there the reads go one to a warp and each
// region's segments are spread over several programs, at the cost of the prefixes that these recompute
// (one region of 64 reads x 16 PD haplotypes: 1.38 -> 0.30 ms with a haplotype a program). A batch with
// tasks enough for every resident warp keeps one program a region and the form that takes its regions'
// reads in the least time: four a warp where the regions have many (1,024 uneven regions: 29.6 ms; one a
// warp 41.2), two or one where they have few (6,000 regions of 1, 2, 3 and 6 reads: one a warp 1.59, 2.94,
// 4.26 and 8.31 ms, two 2.49, 2.53, 4.73 and 7.05, four 3.89, 3.99, 4.01 and 7.72). In between, the step limit
// is the one that makes the estimate -- the larger of the mean steps a warp gets and the longest program --
// smallest (16 uneven regions: 1,400 steps and 0.78 ms; 600 steps 1.11 ms, 3,000 steps 0.98 ms).
Engine::SplitRule Engine::choose_split(const BatchInput& in, const EngineConfig& cfg, const std::vector<int64_t>& first_read,
                                       const std::vector<RegionPlan>& plans) const {
  const int N = in.num_regions;
  const double warps = 8.0 * sms_;
  const bool pd = in.hap_flags != nullptr;
  SplitRule rule;
  struct Work {
    double steps, segs, prefix;
    int short_reads, mid_reads, rest;  // of at most kQuadMaxRead bases, of more that fit 8 rows per lane, longer
    double tasks;
  };
  std::vector<Work> work;
  work.reserve(static_cast<size_t>(N));
  bool extra_codes = false;  // a batch of FP64 reads takes one form
  for (int g = 0; g < N; ++g) {
    const RegionPlan& rp = plans[g];
    if (rp.fwd.n_segs == 0) continue;
    Work w{static_cast<double>(rp.fwd.steps()), static_cast<double>(rp.fwd.n_segs),
           static_cast<double>(rp.fwd.prefixes) / static_cast<double>(rp.fwd.n_segs), 0, 0, 0, 0};
    for (int64_t r = first_read[g]; r < first_read[g + 1]; ++r) {
      const int64_t len = in.read_off[r + 1] - in.read_off[r];
      const bool apart = rp.generic || len > 8 * 31 || (rp.extra_codes && !cfg.double_precision);
      ++(apart ? w.rest : len > kQuadMaxRead ? w.mid_reads : w.short_reads);
    }
    extra_codes |= rp.extra_codes;
    work.push_back(w);
  }
  // A region's tasks with `reads` a warp, and the time they take for each step, in steps of one read's: only
  // reads of one region share a warp, and only those that the form holds.
  struct Count {
    double tasks, time;
  };
  auto count = [&](const Work& w, int reads) -> Count {
    const int fit = w.short_reads + w.mid_reads;
    if (reads == 1) return {static_cast<double>(fit + w.rest), static_cast<double>(fit + w.rest)};
    if (reads == kQuadReads) {
      // The reads too long for the form go one to a warp or, where they are many, two, an odd one of a region
      // with a shorter read.
      const int apart = rule.mid_pairs ? (w.mid_reads + 1) / 2 : w.mid_reads;
      const int quads = (std::max(0, w.short_reads - (rule.mid_pairs ? w.mid_reads % 2 : 0)) + kQuadReads - 1) / kQuadReads;
      return {static_cast<double>(w.rest + apart + quads), w.rest + apart * (rule.mid_pairs ? kPairCost : 1.0) + quads * kQuadCost};
    }
    const int alone = w.rest + (cfg.double_precision ? w.mid_reads : 0);
    const int pairs = (fit + w.rest - alone + 1) / 2;
    return {static_cast<double>(alone + pairs), alone + pairs * (cfg.double_precision ? kF64PairCost : pd ? kPdPairCost : kPairCost)};
  };
  double mid_pairs = 0;
  for (const Work& w : work) mid_pairs += (w.mid_reads + 1) / 2;
  rule.mid_pairs = mid_pairs >= kPairTasks * warps;
  // The form whose tasks take the least time in all, among those that give every resident warp work.
  auto choose = [&](std::initializer_list<int> forms) {
    int chosen = 1;
    double least = -1;
    for (const int reads : forms) {
      double steps = 0, tasks = 0, time = 0;
      for (const Work& w : work) {
        const Count c = count(w, reads);
        tasks += c.tasks;
        steps += w.steps * c.tasks;
        time += w.steps * c.time;
      }
      if (reads > 1 && steps < kFullSteps * warps) continue;
      if (reads == 2 && !pd && tasks < (cfg.double_precision ? kF64PairTasks : kPairTasks) * warps) continue;
      if (least < 0 || time < least) {
        least = time;
        chosen = reads;
      }
    }
    return chosen;
  };
  if (pd && !cfg.double_precision) {
    if (tuning_.reads_per_warp == 2) rule.reads = choose({1, 2});
  } else if (!pd && cfg.double_precision) {
    if (!extra_codes) rule.reads = choose({1, 2});
  } else if (!pd) {
    rule.reads = choose({1, 2, kQuadReads});
  }
  for (Work& w : work) w.tasks = count(w, rule.reads).tasks;
  double total = 0, best = -1;
  for (const Work& w : work) total += w.steps * w.tasks;
  for (const double part : {16.0, 4.0, 2.0, 1.4, 1.0, 0.7, 0.5, 0.25, 0.1, 0.02}) {
    const double limit = std::max(32.0, total / warps * part);
    double sum = 0, longest = 0;
    for (const Work& w : work) {
      const double k = std::min(w.segs, std::max(1.0, std::ceil(w.steps / limit)));
      const double each = w.steps / k + (k > 1 ? w.prefix + 32 : 0);
      sum += each * k * w.tasks;
      longest = std::max(longest, each);
    }
    const double time = std::max(sum / warps, longest);
    if (best < 0 || time < 0.97 * best) {
      best = time;
      rule.limit = static_cast<uint64_t>(limit);
    }
  }
  return rule;
}

int Engine::prepare(const BatchInput& in, const EngineConfig& cfg) {
  DeviceGuard device_guard(device_);
  const auto t_start = std::chrono::steady_clock::now();
  cfg_ = cfg;
  pd_ = in.hap_flags != nullptr;
  error_.clear();
  planned_ = BatchStats{};
  bins_.clear();
  rescue_bins_.clear();
  const int N = in.num_regions;
  if (N < 0) return fail(FGKL_E_INVALID_ARGUMENT, "negative region count");

  // Region starts and validation (lib.rs:278-290).
  std::vector<int64_t> first_read(N + 1, 0), first_hap(N + 1, 0), out_off(N + 1, 0);
  for (int g = 0; g < N; ++g) {
    if (in.region_reads[g] < 0 || in.region_haps[g] < 0) return fail(FGKL_E_INVALID_ARGUMENT, "negative region size");
    first_read[g + 1] = first_read[g] + in.region_reads[g];
    first_hap[g + 1] = first_hap[g] + in.region_haps[g];
    out_off[g + 1] = out_off[g] + static_cast<int64_t>(in.region_reads[g]) * in.region_haps[g];
  }
  const int64_t total_reads = first_read[N], total_haps = first_hap[N];
  out_len_ = out_off[N];
  n_regions_ = N;
  for (int g = 0; g < N; ++g) {
    for (int64_t r = first_read[g]; r < first_read[g + 1]; ++r) {
      const int64_t len = in.read_off[r + 1] - in.read_off[r];
      if (len <= 0) return fail(FGKL_E_EMPTY_READ, "read " + std::to_string(r - first_read[g]) + " has no bases");
      if (len > INT32_MAX) return fail(FGKL_E_INVALID_ARGUMENT, "read " + std::to_string(r - first_read[g]) + " is longer than 2^31 - 1 bases");
    }
    for (int64_t h = first_hap[g]; h < first_hap[g + 1]; ++h)
      if (in.hap_off[h + 1] - in.hap_off[h] <= 0)
        return fail(FGKL_E_EMPTY_HAPLOTYPE, "haplotype " + std::to_string(h - first_hap[g]) + " has no bases");
  }

  // This engine's previous batch: its kernels may still read the device inputs about to be
  // overwritten, and its copies may still read or fill the staging buffers. Events recorded before
  // anything was enqueued complete at once.
  int rc0;
  if ((rc0 = check(cudaEventSynchronize(computed_), "previous batch"))) return rc0;
  if ((rc0 = check(cudaEventSynchronize(uploaded_), "previous upload"))) return rc0;
  if ((rc0 = check(cudaEventSynchronize(fetched_), "previous download"))) return rc0;

  // The five read arrays: uploaded from where they lie when the caller holds them in page-locked
  // memory; otherwise copied to pinned staging first, on a helper thread while the regions are
  // planned (large batches only; a small call copies them in line).
  const int64_t read_bytes = total_reads > 0 ? in.read_off[total_reads] : 0;
  const uint8_t* const read_arrays[5] = {in.bases, in.quals, in.ins, in.del, in.gcp};
  bool direct_reads = read_bytes > 0;
  for (int a = 0; a < 5 && direct_reads; ++a) direct_reads = host_pinned(read_arrays[a], static_cast<size_t>(read_bytes));
  // A small call's reads travel with its plan, in one copy.
  const bool reads_with_plan = !direct_reads && read_bytes <= (int64_t{1} << 18);
  if (!direct_reads && !reads_with_plan && !grow_pinned(h_reads_, cap_h_reads_, static_cast<size_t>(read_bytes) * 5 + 16))
    return fail(FGKL_E_OUT_OF_MEMORY, "pinned host allocation failed");
  Helper read_copy(!direct_reads && read_bytes >= (int64_t{8} << 20), [this, &read_arrays, read_bytes, direct_reads, reads_with_plan] {
    if (direct_reads || reads_with_plan) return;
    for (int a = 0; a < 5; ++a)
      if (read_bytes) parallel_copy(h_reads_ + static_cast<size_t>(a) * read_bytes, read_arrays[a], static_cast<size_t>(read_bytes));
  });
  // Page-locked reads start uploading now, under the planning. Any return from here on waits for
  // these copies first: they read the caller's memory.
  struct UploadGuard {
    cudaStream_t s = nullptr;
    ~UploadGuard() {
      if (s) cudaStreamSynchronize(s);
    }
  } upload_guard;
  if (direct_reads) {
    if (!grow(d_reads_, cap_reads_, static_cast<size_t>(read_bytes) * 5 + 16)) return fail(FGKL_E_OUT_OF_MEMORY, "device allocation failed");
    upload_guard.s = copy_;
    for (int a = 0; a < 5; ++a)
      if ((rc0 = check(cudaMemcpyAsync(d_reads_ + static_cast<size_t>(a) * read_bytes, read_arrays[a], static_cast<size_t>(read_bytes),
                                       cudaMemcpyHostToDevice, copy_),
                       "upload reads")))
        return rc0;
  }

  // Plan the regions in parallel, one region a thread for small batches (a region takes about
  // 75 us to plan; a combined batch of per-call requests holds a few).
  std::vector<RegionPlan> plans(static_cast<size_t>(N));
  const bool share = cfg.share_suffixes;
  // A batch of many reads keeps one program a region (choose_split), so they are emitted while their
  // regions are planned, and the few regions to split, if any, are planned again: sorted sets kept for all
  // regions until the split is known cost host time: planning 6,000 regions of 2 reads x 16
  // haplotypes of 350 bases took 44 ms on 8 cores that way, and takes 30.
  const bool whole = total_reads >= kWholeReads * 8 * sms_ || N >= kWholeRegions * 8 * sms_;
  parallel_for(N, host_threads(),
               [&](int64_t g) { plan_region(in, static_cast<int>(g), first_read[g], first_hap[g], share, whole, plans[g]); });

  const bool pd = in.hap_flags != nullptr;
  const SplitRule split = choose_split(in, cfg, first_read, plans);
  const auto emit = [&](int64_t g) {
    RegionPlan& rp = plans[g];
    if (!rp.error.empty() || rp.haps.empty()) return;
    const int chunks = split.chunks(rp.fwd);
    if (whole && chunks == 1) return;
    if (whole) {
      rp = RegionPlan();
      plan_region(in, static_cast<int>(g), first_read[g], first_hap[g], share, false, rp);
    }
    emit_region(rp, chunks);
  };
  parallel_for(N, host_threads(), emit);

  for (int g = 0; g < N; ++g)
    if (!plans[g].error.empty()) return fail(FGKL_E_UNSUPPORTED, "region " + std::to_string(g) + ": " + plans[g].error);

  planned_.host_plan_ms = ms_since(t_start);
  const auto t_pack = std::chrono::steady_clock::now();
  // Section offsets. Each stream gets kStreamPad zero entries on both sides.
  std::vector<Region> regions(static_cast<size_t>(N));
  std::vector<Program> progs;
  int64_t n_haps = 0, n_stream = kStreamPad, n_segs = 0, n_sweeps = 0, n_seq = 0, n_pd_seq = 0, n_sigs = 0;
  int max_slots = 1, max_nodes = 1, max_segs = 1;
  std::vector<int64_t> queue_cap(kQueueBins, 0);
  std::vector<int64_t> many_cap(kQueueBins, 0);  // pairs of the bins that only a run losing many fills
  std::vector<int> queue_len(kQueueBins, 1);     // the longest read of each bin
  int64_t wide_pairs = 0;                        // what Counters::lost_wide counts, if all were lost
  int max_hap_len = 1;  // scratch of the strip-mined kinds: one carry column per haplotype base
  for (int g = 0; g < N; ++g) {
    const RegionPlan& rp = plans[g];
    Region& R = regions[g];
    std::memset(&R, 0, sizeof R);
    R.prog = static_cast<int32_t>(progs.size());
    R.n_progs = static_cast<int32_t>(rp.progs.size());
    R.whole_steps = static_cast<int32_t>(std::min<uint64_t>(rp.fwd.steps(), INT32_MAX / 4));
    auto put_stream = [&](const std::vector<uint32_t>& v, int32_t& off, int32_t& len) {
      off = static_cast<int32_t>(n_stream);
      len = v.empty() ? 0 : static_cast<int32_t>(v.size()) - 1;  // the last entry only carries post events
      n_stream += static_cast<int64_t>(v.size()) + kStreamPad;
    };
    for (const ProgramBuild& pb : rp.progs) {
      Program p{};
      put_stream(pb.fwd, p.fwd_off, p.fwd_len);
      put_stream(pb.bwd, p.bwd_off, p.bwd_len);
      p.seg_off = static_cast<int32_t>(n_segs);
      p.n_segs = static_cast<int32_t>(pb.segs.size());
      n_segs += p.n_segs;
      p.sweep_off = static_cast<int32_t>(n_sweeps);
      p.n_sweeps = static_cast<int32_t>(pb.sweeps.size());
      n_sweeps += p.n_sweeps;
      p.n_slots = pb.n_slots;
      p.n_nodes = pb.n_nodes;
      p.seg_first = pb.seg_first;
      max_slots = std::max(max_slots, pb.n_slots);
      max_nodes = std::max(max_nodes, pb.n_nodes);
      max_segs = std::max(max_segs, p.n_segs);
      progs.push_back(p);
    }
    R.hap_off = static_cast<int32_t>(n_haps);
    R.n_haps = in.region_haps[g];
    n_haps += static_cast<int64_t>(rp.haps.size());
    R.read_off = static_cast<int32_t>(first_read[g]);
    R.n_reads = in.region_reads[g];
    R.out_off = out_off[g];
    R.code_off = g * 256;
    R.seq_off = static_cast<int32_t>(pd ? n_pd_seq : n_seq);
    n_seq += static_cast<int64_t>(rp.seq.size());
    n_pd_seq += static_cast<int64_t>(rp.pd_seq.size());
    R.sig_off = static_cast<int32_t>(n_sigs);
    R.flags = rp.generic ? kRegionGeneric : 0;
    n_sigs += static_cast<int64_t>(rp.pd_sigs.size());
    planned_.nominal_cells += rp.read_bases * rp.hap_bases;
    planned_.prefix_only_cells += rp.read_bases * rp.cols.prefix_only;
    for (const HapInfo& h : rp.haps) max_hap_len = std::max(max_hap_len, static_cast<int>(h.len));
    if (rp.n_distinct > 0)
      for (int64_t r = first_read[g]; r < first_read[g + 1]; ++r) {
        const int len = static_cast<int>(in.read_off[r + 1] - in.read_off[r]);
        const int bin = queue_bin(len, rp.generic);
        if (bin <= 8) {
          queue_cap[bin] += rp.n_distinct;
          continue;
        }
        const int few = queue_pair_bin(len, rp.generic, pd, true), many = queue_pair_bin(len, rp.generic, pd, false);
        queue_cap[few] += rp.n_distinct;
        if (few != many) {
          many_cap[many] += rp.n_distinct;
          if (queue_bin_group(bin) == 0) queue_cap[bin] += static_cast<int64_t>(rp.progs.size());  // whole-program tasks
        }
        for (const int q : {few, many}) queue_len[q] = std::max(queue_len[q], len);
        wide_pairs += R.n_haps;
      }
  }
  // A batch that cannot lose more than a few pairs has no use for the other bins.
  if (wide_pairs > few_pairs(sms_, kLongWarps))
    for (int q = 0; q < kQueueBins; ++q) queue_cap[q] += many_cap[q];
  for (int q = 3 * kRowBins; q < kQueueBins; ++q) queue_cap[q] = std::min<int64_t>(queue_cap[q], few_pairs_most(sms_));
  if (n_stream > INT32_MAX || n_seq > INT32_MAX || n_pd_seq > INT32_MAX || n_haps > INT32_MAX)
    return fail(FGKL_E_INVALID_ARGUMENT, "batch too large for 32-bit plan offsets; split it");

  // Tasks: a region's reads sorted longest first and packed in that order by the batch's form. A task costs
  // its region's stream length times its rows, so within a bin (one rows value) the costliest
  // regions' tasks come first: regions are visited in that order (ties by index), which lists each
  // bin's tasks longest first without sorting them.
  constexpr int kKinds = kNumKinds;
  constexpr int kBinRows = kQuadMaxRows + 1 > kRowBins ? kQuadMaxRows + 1 : kRowBins;  // rows-per-lane values of any kind
  struct BinList {
    std::vector<std::pair<uint64_t, Task>> list;
    uint64_t fwd_cells = 0, bwd_cells = 0;  // forward, backward DP cells
    LongPairs pairs;                        // strip-mined
  };
  std::vector<BinList> by_bin(static_cast<size_t>(kKinds) * kBinRows);
  auto bin_at = [&](Kind kind, int rows) -> BinList& { return by_bin[static_cast<size_t>(kind) * kBinRows + rows]; };
  std::vector<int> region_order(static_cast<size_t>(N));
  for (int g = 0; g < N; ++g) region_order[g] = g;
  auto cost_of = [&](int g) {
    uint64_t most = 0;
    for (const ProgramBuild& pb : plans[g].progs) most = std::max(most, pb.steps());
    return most;
  };
  std::vector<uint64_t> region_cost(static_cast<size_t>(N));
  for (int g = 0; g < N; ++g) region_cost[g] = cost_of(g);
  std::stable_sort(region_order.begin(), region_order.end(), [&](int a, int b) { return region_cost[a] > region_cost[b]; });
  // Each region's tasks, built in parallel (its reads sorted longest first, then packed), then
  // appended to the bins serially in region order.
  struct RegionTask {
    Kind kind;
    int rows;
    int len;  // read bases of the task, for the bin's cell counts
    Task task;
    uint64_t cost;  // strip-mined pairs: steps x rows; 0 for the region's program tasks
  };
  // One FP64 form a batch: the one that compares codes when a region needs it (the bits are the same).
  bool extra_codes = false;
  for (const RegionPlan& rp : plans) extra_codes |= rp.extra_codes;
  const Kind f64 = extra_codes ? Kind::kOneF64Codes : Kind::kOneF64;
  std::vector<std::vector<RegionTask>> region_tasks(static_cast<size_t>(N));
  parallel_for(N, std::min(host_threads(), (N + 63) / 64), [&](int64_t gi) {
    const int g = static_cast<int>(gi);
    const int n_reads = in.region_reads[g];
    if (n_reads == 0 || in.region_haps[g] == 0) return;
    std::vector<int> order(static_cast<size_t>(n_reads));
    for (int r = 0; r < n_reads; ++r) order[r] = r;
    auto len_of = [&](int r) { return static_cast<int>(in.read_off[first_read[g] + r + 1] - in.read_off[first_read[g] + r]); };
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return len_of(a) > len_of(b); });
    std::vector<RegionTask>& out = region_tasks[g];
    out.reserve(static_cast<size_t>(n_reads));
    auto one = [&](Kind kind, int rows, size_t i) {
      out.push_back({kind, rows, len_of(order[i]), Task{g, {static_cast<int32_t>(first_read[g] + order[i]), -1, -1, -1}, rows, -1, 0}, 0});
    };
    auto two = [&](Kind kind, int rows, size_t i) {
      const int32_t a = static_cast<int32_t>(first_read[g] + order[i]);
      const int32_t b = i + 1 < order.size() ? static_cast<int32_t>(first_read[g] + order[i + 1]) : -1;
      out.push_back({kind, rows, len_of(order[i]) + (i + 1 < order.size() ? len_of(order[i + 1]) : 0), Task{g, {a, b, -1, -1}, rows, -1, 0}, 0});
    };
    auto quad = [&](Kind kind, size_t i, size_t reads) {
      const int rows = quad_rows(len_of(order[i]));
      Task t{g, {-1, -1, -1, -1}, kind == Kind::kQuadF32 && tuning_.rows_extra != 0 && rows < kQuadMaxRows ? rows + 2 : rows, -1, 0};
      int len = 0;
      for (size_t k = 0; k < reads && i + k < order.size(); ++k) {
        t.read[k] = static_cast<int32_t>(first_read[g] + order[i + k]);
        len += len_of(order[i + k]);
      }
      out.push_back({kind, t.rows, len, t, 0});
    };
    // One task per distinct sorted haplotype of read order[i], strip-mined over row blocks.
    const RegionPlan& rp = plans[g];
    auto pairs = [&](Kind kind, size_t i) {
      const int len = len_of(order[i]);
      const int rows = long_rows(len, kind == Kind::kLongF32);
      const uint64_t blocks = static_cast<uint64_t>(long_blocks(len, rows));
      for (int k = 0; k < static_cast<int>(rp.haps.size()); ++k)
        if (rp.haps[k].src == k)
          out.push_back({kind, rows, len, Task{g, {static_cast<int32_t>(first_read[g] + order[i]), -1, -1, -1}, rows, k, 0},
                         (static_cast<uint64_t>(rp.haps[k].len) + 32) * blocks * static_cast<uint64_t>(rows)});
    };
    size_t i = 0;
    const bool dbl = cfg.double_precision;
    if (rp.generic) {
      for (; i < order.size(); ++i) pairs(dbl ? Kind::kGenericF64Pd : Kind::kGenericF32Pd, i);
      return;
    }
    const Kind long_kind = pd ? (dbl ? Kind::kLongF64Pd : Kind::kLongF32Pd) : ((dbl || rp.extra_codes) ? Kind::kLongF64 : Kind::kLongF32);
    for (; i < order.size() && len_of(order[i]) > kMaxBlockRead; ++i) pairs(long_kind, i);
    if (pd && cfg.double_precision) {
      // PD in FP64: one read per warp.
      for (; i < order.size(); ++i) one(Kind::kOneF64Pd, single_rows(len_of(order[i])), i);
    } else if (pd) {
      // PD in FP32: reads above 248 bases one per warp, the others by the batch's form, one or two (FP32x2).
      for (; i < order.size() && (packed_rows(len_of(order[i])) > 8 || split.reads == 1); ++i)
        one(Kind::kOneF32Pd, single_rows(len_of(order[i])), i);
      for (; i < order.size(); i += 2) two(Kind::kPackedF32Pd, packed_rows(len_of(order[i])), i);
    } else if (cfg.double_precision || plans[g].extra_codes) {
      const bool pairs_fit = cfg.double_precision && split.reads == 2;
      for (; i < order.size() && !(pairs_fit && len_of(order[i]) <= kQuadMaxRead); ++i) one(f64, single_rows(len_of(order[i])), i);
      for (; i < order.size(); i += 2) quad(Kind::kPairF64, i, 2);
    } else {
      // The tile-shape axis: rows_extra moves each read to the next instantiated rows-per-lane
      // (more padding rows, other registers and occupancy; the same bits).
      const bool up = tuning_.rows_extra != 0;
      auto single_up = [&](int rows) { return up && rows + 2 <= max_rows(Kind::kOneF32) ? rows + 2 : rows; };  // even, 10..20
      auto short_up = [&](int rows) { return up && rows < 8 ? rows + 1 : rows; };
      for (; i < order.size() && packed_rows(len_of(order[i])) > 8; ++i) one(Kind::kOneF32, single_up(single_rows(len_of(order[i]))), i);
      // Shorter ones by the batch's form, in a batch of quads those too long for it in pairs or alone.
      const auto fits = [&](size_t k) { return split.reads == kQuadReads && len_of(order[k]) <= kQuadMaxRead; };
      const bool pairs = split.reads == 2 || (split.reads == kQuadReads && split.mid_pairs);
      while (i < order.size() && !fits(i)) {
        if (pairs)
          two(Kind::kPackedF32, short_up(packed_rows(len_of(order[i]))), i);
        else
          one(Kind::kShortF32, short_up(packed_rows(len_of(order[i]))), i);
        i += pairs ? 2 : 1;
      }
      for (; i < order.size(); i += kQuadReads) quad(Kind::kQuadF32, i, kQuadReads);
    }
  });
  {
    std::vector<size_t> bin_size(by_bin.size(), 0);
    for (const auto& v : region_tasks)
      for (const RegionTask& t : v)
        bin_size[static_cast<size_t>(t.kind) * kBinRows + t.rows] += t.task.hap >= 0 ? 1 : plans[t.task.region].progs.size();
    for (size_t k = 0; k < by_bin.size(); ++k) by_bin[k].list.reserve(bin_size[k]);
  }
  for (const int g : region_order) {
    const RegionPlan& rp = plans[g];
    for (RegionTask& t : region_tasks[g]) {
      BinList& bl = bin_at(t.kind, t.rows);
      if (t.task.hap >= 0) {
        // An unshared strip-mined pair: read length x haplotype length forward cells.
        bl.list.push_back({t.cost, t.task});
        bl.pairs.add(long_blocks(t.len, t.rows), static_cast<int>(rp.haps[t.task.hap].len));
        bl.fwd_cells += static_cast<uint64_t>(rp.haps[t.task.hap].len) * static_cast<uint64_t>(t.len);
        continue;
      }
      for (size_t c = 0; c < rp.progs.size(); ++c) {
        t.task.prog = regions[g].prog + static_cast<int32_t>(c);
        bl.list.push_back({rp.progs[c].steps() * static_cast<uint64_t>(t.task.rows), t.task});
      }
      // The cells of the plan; prefixes that several programs compute count once.
      bl.fwd_cells += rp.fwd.fwd_columns * static_cast<uint64_t>(t.len);
      bl.bwd_cells += rp.fwd.bwd_columns * static_cast<uint64_t>(t.len);
    }
  }
  for (const BinList& bl : by_bin) {
    planned_.forward_cells += bl.fwd_cells;
    planned_.backward_cells += bl.bwd_cells;
  }
  planned_.computed_cells = planned_.forward_cells + planned_.backward_cells;
  std::vector<Task> tasks;
  std::vector<std::pair<uint64_t, Bin>> first;
  size_t n_tasks_all = 0;
  for (const BinList& bl : by_bin) n_tasks_all += bl.list.size();
  tasks.reserve(n_tasks_all);
  for (int kind = 0; kind < kKinds; ++kind)
    for (int rows = 0; rows < kBinRows; ++rows) {
      const BinList& bl = by_bin[static_cast<size_t>(kind) * kBinRows + rows];
      const auto& list = bl.list;
      if (list.empty()) continue;
      Bin b{static_cast<Kind>(kind), rows, static_cast<int>(tasks.size()), static_cast<int>(list.size()), 0, 0, 0};
      b.fwd_cells = bl.fwd_cells;
      b.bwd_cells = bl.bwd_cells;
      uint64_t cost = 0;
      for (auto& e : list) {
        tasks.push_back(e.second);
        cost += e.first;
      }
      const bool fp32 = b.kind == Kind::kShortF32 || b.kind == Kind::kPackedF32 || b.kind == Kind::kQuadF32 ||
                        b.kind == Kind::kOneF32 || b.kind == Kind::kPackedF32Pd || b.kind == Kind::kOneF32Pd;
      const bool pipelined = is_long(b.kind);
      b.warps = pipelined ? choose_long_warps(b.kind, b.rows, sms_, bl.pairs) : (fp32 ? tuning_.warps_per_block : kWarpsPerBlock);
      int per_sm = 0, threads = 0;
      occupancy(b.kind, b.rows, &per_sm, &threads, b.warps);
      b.warps = threads / 32;
      if (per_sm <= 0) return fail(FGKL_E_CUDA, "kernel instantiation unavailable on this device");
      const int grid = std::max(sms_, per_sm * sms_ * tuning_.grid_percent / 100);
      b.blocks = std::max(1, std::min(pipelined ? b.n_tasks : (b.n_tasks + b.warps - 1) / b.warps, grid));
      first.push_back({cost, b});
    }
  // The launch with the most work comes last: its many tasks fill the SMs that the others' last ones leave
  // (before them, their few and as long tasks ran at the end, by themselves). The launches run one after
  // another all the same: a grid of each at a time, in proportion to its work, took twice as long (62
  // against 30 ms for 1,024 uneven regions), as warps of several kernels on an SM share its instruction
  // caches.
  std::stable_sort(first.begin(), first.end(), [](const auto& x, const auto& y) { return x.first < y.first; });
  for (auto& f : first) bins_.push_back(f.second);
  // Recomputation queues: room for every (read, distinct haplotype) pair of each rows-per-lane bin.
  // Pairs either pass loses (an FP32 underflow, or a joined FP64 result below the backward range)
  // are recomputed in FP64 (lib.rs:461-520): after an FP32 pass, a read lost against a third of its
  // haplotypes or more once with its region's shared program, any pair that sweep loses again and
  // every other lost pair without sharing, which cannot lose a pair.
  const bool queue_on = cfg.double_fallback;
  std::vector<int> queue_off(kQueueBins + 1, 0);
  {
    int64_t acc = 0;
    for (int r = 0; r < kQueueBins; ++r) {
      queue_off[r] = static_cast<int>(acc);
      if (queue_on) acc += queue_cap[r];
    }
    if (acc > INT32_MAX) return fail(FGKL_E_INVALID_ARGUMENT, "batch too large for the recomputation queue; split it");
    queue_off[kQueueBins] = static_cast<int>(acc);
  }
  if (queue_on) {
    // The bins of several warps a pair first: their pairs take the longest.
    for (int i = 0; i < kQueueBins; ++i) {
      const int q = (i + 3 * kRowBins) % kQueueBins;
      const int cap = queue_off[q + 1] - queue_off[q];
      if (cap == 0) continue;
      // Queue bin -> the FP64 form of the pairs it holds (queue_bin).
      const int r = queue_bin_rows(q);
      const int group = queue_bin_group(q);
      const Kind kind = group == 0 ? (pd ? Kind::kOneF64Pd : f64)
                                   : (group == 2 || group == 4 ? Kind::kGenericF64Pd : (pd ? Kind::kLongF64Pd : Kind::kLongF64));
      int per_sm = 0, threads = 0;
      const bool pipelined = is_long(kind);
      Bin b{kind, r, queue_off[q], cap, 0, 0, 0};
      // Many pairs: two warps a pair, so that the longest does not run on alone for long (1,000 pairs of 700
      // bases 1.62 ms against 1.45 at one, 300 of 1,200 bases 1.86 against 2.25), one for short ones.
      const int row_blocks = pipelined ? long_blocks(queue_len[q], r) : 0;
      if (pipelined) b.warps = group >= 3 ? long_warps(row_blocks) : (row_blocks > (group == 1 ? 2 : 4) ? 2 : 1);
      occupancy(kind, r, &per_sm, &threads, b.warps);
      if (per_sm <= 0) return fail(FGKL_E_CUDA, "recomputation kernel unavailable on this device");
      b.queue_bin = q;
      b.blocks = std::max(1, std::min(pipelined ? cap : (cap + kWarpsPerBlock - 1) / kWarpsPerBlock, per_sm * sms_));
      rescue_bins_.push_back(b);
    }
  }
  // Bins of one pass run concurrently, so each owns a slice of the scratch.
  size_t scratch_total = 256;
  for (auto* list : {&bins_, &rescue_bins_}) {
    const bool rescue = list == &rescue_bins_;
    size_t off = 0;
    for (Bin& b : *list) {
      // Short-read recomputation bins also run dense reads' whole programs after an FP32 pass.
      const bool whole = !rescue || !cfg.double_precision;
      b.stride = align_up(is_long(b.kind) ? long_scratch_bytes(b.kind, b.rows, max_hap_len)
                          : whole         ? scratch_bytes(b.kind, b.rows, max_slots, max_nodes, max_segs)
                                          : scratch_bytes(b.kind, b.rows, 0, 0, 1));
      b.scratch_off = off;
      // A block of a strip-mined launch has one carry column (allocated in fours: calls of a few pairs more or
      // less fit one buffer), the others' warps a record set each.
      off += (is_long(b.kind) ? align_up(static_cast<size_t>(b.blocks), 4) : static_cast<size_t>(b.blocks) * b.warps) * b.stride;
    }
    scratch_total = std::max(scratch_total, off);
  }

  // Plan blob: regions | programs | haps | stream | segs | sweeps | code tables | haplotype codes | PD entries | PD signatures.
  size_t o_regions, o_progs, o_haps, o_stream, o_segs, o_sweeps, o_codes, o_seq, o_pd_seq, o_sigs, blob_bytes = 0;
  auto section = [&](size_t bytes, size_t& off) {
    off = align_up(blob_bytes, 16);
    blob_bytes = off + bytes;
  };
  section(regions.size() * sizeof(Region), o_regions);
  section(progs.size() * sizeof(Program), o_progs);
  section(static_cast<size_t>(n_haps) * sizeof(HapInfo), o_haps);
  section(static_cast<size_t>(n_stream) * sizeof(uint32_t), o_stream);
  section(static_cast<size_t>(n_segs) * sizeof(Segment), o_segs);
  section(static_cast<size_t>(n_sweeps) * sizeof(Sweep), o_sweeps);
  section(static_cast<size_t>(N) * 256, o_codes);
  section(static_cast<size_t>(n_seq) + 16, o_seq);
  section(static_cast<size_t>(n_pd_seq) * sizeof(uint32_t) + 16, o_pd_seq);
  section(static_cast<size_t>(n_sigs) * sizeof(uint32_t) + 16, o_sigs);

  // One upload: read offsets | plan | tasks | queue offsets | a small call's reads. The pinned staging holds
  // it, and after it the results and counters that come back. On the device the results are followed by what
  // every run zeroes: the counters, then a task counter for each launch and the queues' tails.
  const size_t s_read_off = 0;
  const size_t s_blob = s_read_off + align_up((total_reads + 1) * sizeof(int64_t));
  const size_t s_tasks = s_blob + align_up(blob_bytes);
  const size_t s_qoff = s_tasks + align_up(tasks.size() * sizeof(Task));
  const size_t s_reads = s_qoff + align_up((kQueueBins + 1) * sizeof(int));
  const size_t s_out = s_reads + (reads_with_plan ? align_up(static_cast<size_t>(read_bytes) * 5) : 0);
  const size_t stage_bytes = s_out + align_up(static_cast<size_t>(out_len_) * sizeof(double) + sizeof(Counters));
  zero_bytes_ = sizeof(Counters) + (bins_.size() + rescue_bins_.size() + kQueueBins) * sizeof(int);
  if ((!reads_with_plan && !grow(d_reads_, cap_reads_, static_cast<size_t>(read_bytes) * 5 + 16)) || !grow(d_in_, cap_in_, s_out + 16) ||
      !grow(d_queue_, cap_queue_, static_cast<size_t>(queue_off[kQueueBins]) + 1) ||
      !grow(d_out_, cap_out_, static_cast<size_t>(out_len_) + (zero_bytes_ + 7) / 8) || !grow(d_scratch_, cap_scratch_, scratch_total))
    return fail(FGKL_E_OUT_OF_MEMORY, "device allocation failed");
  if (over_allocation_limit(stage_bytes)) return fail(FGKL_E_OUT_OF_MEMORY, "pinned host allocation failed");
  if (stage_bytes > cap_stage_) {
    // Grown by half again at least, as the device buffers are (cudaFreeHost waits for the device).
    const size_t want = cap_stage_ > 0 ? std::max(stage_bytes, cap_stage_ + cap_stage_ / 2) : stage_bytes;
    if (h_stage_) cudaFreeHost(h_stage_);
    h_stage_ = nullptr;
    if (pinned_alloc(reinterpret_cast<void**>(&h_stage_), want) == cudaSuccess) {
      cap_stage_ = want;
    } else if (want > stage_bytes && (cudaGetLastError(), pinned_alloc(reinterpret_cast<void**>(&h_stage_), stage_bytes) == cudaSuccess)) {
      cap_stage_ = stage_bytes;
    } else {
      cudaGetLastError();
      cap_stage_ = 0;
      h_stage_ = nullptr;
      return fail(FGKL_E_OUT_OF_MEMORY, "pinned host allocation failed");
    }
  }
  out_stage_ = s_out;
  uint8_t* const st = h_stage_;
  std::memcpy(st + s_read_off, in.read_off, (total_reads + 1) * sizeof(int64_t));
  {
    uint8_t* blob = st + s_blob;
    std::memcpy(blob + o_regions, regions.data(), regions.size() * sizeof(Region));
    if (!progs.empty()) std::memcpy(blob + o_progs, progs.data(), progs.size() * sizeof(Program));
    uint32_t* stream = reinterpret_cast<uint32_t*>(blob + o_stream);
    std::memset(stream, 0, kStreamPad * sizeof(uint32_t));
    std::memset(blob + o_seq + n_seq, 0, 16);
    std::memset(blob + o_pd_seq + n_pd_seq * sizeof(uint32_t), 0, 16);
    std::memset(blob + o_sigs + n_sigs * sizeof(uint32_t), 0, 16);
    parallel_for(N, std::min(host_threads(), (N + 31) / 32), [&](int64_t g) {
      const RegionPlan& rp = plans[g];
      const Region& R = regions[g];
      if (!rp.haps.empty()) std::memcpy(blob + o_haps + static_cast<size_t>(R.hap_off) * sizeof(HapInfo), rp.haps.data(), rp.haps.size() * sizeof(HapInfo));
      auto put = [&](const std::vector<uint32_t>& v, int32_t off) {
        if (!v.empty()) std::memcpy(stream + off, v.data(), v.size() * sizeof(uint32_t));
        std::memset(stream + off + v.size(), 0, kStreamPad * sizeof(uint32_t));
      };
      for (size_t c = 0; c < rp.progs.size(); ++c) {
        const ProgramBuild& pb = rp.progs[c];
        const Program& p = progs[static_cast<size_t>(R.prog) + c];
        put(pb.fwd, p.fwd_off);
        put(pb.bwd, p.bwd_off);
        if (!pb.segs.empty())
          std::memcpy(blob + o_segs + static_cast<size_t>(p.seg_off) * sizeof(Segment), pb.segs.data(), pb.segs.size() * sizeof(Segment));
        if (!pb.sweeps.empty())
          std::memcpy(blob + o_sweeps + static_cast<size_t>(p.sweep_off) * sizeof(Sweep), pb.sweeps.data(), pb.sweeps.size() * sizeof(Sweep));
      }
      if (!rp.haps.empty()) std::memcpy(blob + o_codes + static_cast<size_t>(g) * 256, rp.codes, 256);
      else std::memset(blob + o_codes + static_cast<size_t>(g) * 256, 0, 256);
      if (!rp.seq.empty()) std::memcpy(blob + o_seq + R.seq_off, rp.seq.data(), rp.seq.size());
      if (!rp.pd_seq.empty())
        std::memcpy(blob + o_pd_seq + static_cast<size_t>(R.seq_off) * sizeof(uint32_t), rp.pd_seq.data(), rp.pd_seq.size() * sizeof(uint32_t));
      if (!rp.pd_sigs.empty())
        std::memcpy(blob + o_sigs + static_cast<size_t>(R.sig_off) * sizeof(uint32_t), rp.pd_sigs.data(), rp.pd_sigs.size() * sizeof(uint32_t));
    });
  }
  if (!tasks.empty()) std::memcpy(st + s_tasks, tasks.data(), tasks.size() * sizeof(Task));
  std::memcpy(st + s_qoff, queue_off.data(), (kQueueBins + 1) * sizeof(int));
  if (reads_with_plan)
    for (int a = 0; a < 5; ++a)
      if (read_bytes) std::memcpy(st + s_reads + static_cast<size_t>(a) * read_bytes, read_arrays[a], static_cast<size_t>(read_bytes));

  read_copy.join();
  planned_.host_pack_ms = ms_since(t_pack);
  const auto t_up = std::chrono::steady_clock::now();
  int rc;
  if (!direct_reads && !reads_with_plan &&
      (rc = check(cudaMemcpyAsync(d_reads_, h_reads_, static_cast<size_t>(read_bytes) * 5, cudaMemcpyHostToDevice, copy_), "upload reads")))
    return rc;
  if ((rc = check(cudaMemcpyAsync(d_in_, st, s_out, cudaMemcpyHostToDevice, copy_), "upload plan"))) return rc;
  if ((rc = check(cudaEventRecord(uploaded_, copy_), "upload event"))) return rc;
  // The plans of many regions are freed by several threads, while the copies run.
  if (N >= 512) parallel_for(N, std::min(host_threads(), 16), [&](int64_t g) { plans[g] = RegionPlan(); });
  // Uploaded from the caller's own memory: done before returning, so the caller may reuse it.
  if (direct_reads) {
    upload_guard.s = nullptr;
    if ((rc = check(cudaEventSynchronize(uploaded_), "upload reads"))) return rc;
  }

  planned_.host_upload_ms = ms_since(t_up);
  const uint8_t* const reads = reads_with_plan ? d_in_ + s_reads : d_reads_;
  const uint8_t* const plan = d_in_ + s_blob;
  tasks_ = reinterpret_cast<const Task*>(d_in_ + s_tasks);
  queue_off_ = reinterpret_cast<const int*>(d_in_ + s_qoff);
  view_.bases = reads;
  view_.quals = reads + read_bytes;
  view_.ins = reads + 2 * read_bytes;
  view_.del = reads + 3 * read_bytes;
  view_.gcp = reads + 4 * read_bytes;
  view_.read_off = reinterpret_cast<const int64_t*>(d_in_ + s_read_off);
  view_.regions = reinterpret_cast<const Region*>(plan + o_regions);
  view_.progs = reinterpret_cast<const Program*>(plan + o_progs);
  view_.haps = reinterpret_cast<const HapInfo*>(plan + o_haps);
  view_.stream = reinterpret_cast<const uint32_t*>(plan + o_stream);
  view_.segs = reinterpret_cast<const Segment*>(plan + o_segs);
  view_.sweeps = reinterpret_cast<const Sweep*>(plan + o_sweeps);
  view_.code_of_byte = plan + o_codes;
  view_.hap_codes = plan + o_seq;
  view_.pd_entries = reinterpret_cast<const uint32_t*>(plan + o_pd_seq);
  view_.pd_sigs = reinterpret_cast<const uint32_t*>(plan + o_sigs);
  view_.err_prob = d_err_;
  view_.m2m = d_m2m_;
  view_.out = d_out_;
  view_.counters = reinterpret_cast<Counters*>(d_out_ + out_len_);
  (void)total_haps;
  return FGKL_OK;
}

int Engine::begin_run() {
  DeviceGuard device_guard(device_);
  return check(cudaStreamWaitEvent(stream_, uploaded_, 0), "wait for the uploads");
}

int Engine::end_run() {
  DeviceGuard device_guard(device_);
  return check(cudaEventRecord(computed_, stream_), "kernels event");
}

int Engine::run() {
  DeviceGuard device_guard(device_);
  int rc;
  const size_t n_launch = bins_.size() + rescue_bins_.size();
  int* counters = reinterpret_cast<int*>(view_.counters + 1);  // one per launch
  int* queue_tail = counters + n_launch;
  if ((rc = check(cudaMemsetAsync(view_.counters, 0, zero_bytes_, stream_), "reset counters"))) return rc;
  planned_.kernel_launches = 0;
  int i = 0;
  if (profile_) {
    const size_t need = 2 * (bins_.size() + rescue_bins_.size() + 1);
    while (ev_.size() < need) {
      cudaEvent_t e;
      if ((rc = check(cudaEventCreate(&e), "profiling event"))) return rc;
      ev_.push_back(e);
    }
  }
  // Each pass forks its bins onto the auxiliary streams and joins them back.
  auto pass = [&](const std::vector<Bin>& list, bool rescue) -> int {
    if (list.empty()) return FGKL_OK;
    // A pass of one launch stays on the main stream.
    const bool fork = !profile_ && list.size() > 1;
    if (fork && (rc = check(cudaEventRecord(fork_, stream_), "fork"))) return rc;
    for (size_t b = 0; b < list.size(); ++b) {
      const Bin& bin = list[b];
      // Profiled runs serialise the launches on the main stream so each one's events time it alone.
      const int lanes = std::max(1, std::min(tuning_.streams, kAuxStreams));
      cudaStream_t s = fork ? aux_[b % lanes] : stream_;
      if (fork && (rc = check(cudaStreamWaitEvent(s, fork_, 0), "fork wait"))) return rc;
      LaunchArgs a{};
      a.v = view_;
      a.tasks = (rescue ? d_queue_ : tasks_) + bin.task_off;
      a.n_tasks = bin.n_tasks;
      a.count = rescue ? queue_tail + bin.queue_bin : nullptr;
      a.task_counter = counters + i++;
      a.scratch = d_scratch_ + bin.scratch_off;
      a.scratch_stride = bin.stride;
      a.min_accept_plain = (!rescue && !cfg_.double_precision) ? 1 : 0;
      a.only_lost = rescue ? 1 : 0;
      const int li = i - 1;  // this launch's index, for profiling events
      if (profile_ && (rc = check(cudaEventRecord(ev_[2 * li], s), "profiling event"))) return rc;
      if ((rc = check(launch(bin.kind, bin.rows, bin.blocks, a, s, bin.warps), rescue ? "recomputation launch" : "first-pass launch")))
        return rc;
      if (profile_ && (rc = check(cudaEventRecord(ev_[2 * li + 1], s), "profiling event"))) return rc;
      planned_.kernel_launches++;
      if (fork && (rc = check(cudaEventRecord(join_[b % lanes], s), "join"))) return rc;
    }
    if (!fork) return FGKL_OK;
    const size_t used = std::min<size_t>(list.size(), static_cast<size_t>(std::max(1, std::min(tuning_.streams, kAuxStreams))));
    for (size_t b = 0; b < used; ++b)
      if ((rc = check(cudaStreamWaitEvent(stream_, join_[b], 0), "join wait"))) return rc;
    return FGKL_OK;
  };
  if ((rc = pass(bins_, false))) return rc;
  if (!rescue_bins_.empty()) {
    CollectArgs c{view_, d_queue_, queue_off_, queue_tail, cfg_.double_precision ? 0 : 1, pd_ ? 1 : 0, sms_};
    if ((rc = check(launch_collect(c, n_regions_, stream_), "lost-pair collection"))) return rc;
    planned_.kernel_launches++;
  }
  if ((rc = pass(rescue_bins_, true))) return rc;
  return FGKL_OK;
}

void Engine::set_tuning(const Tuning& t) {
  tuning_.streams = std::max(1, std::min(t.streams, kAuxStreams));
  tuning_.grid_percent = std::max(10, std::min(t.grid_percent, 100));
  tuning_.reads_per_warp = t.reads_per_warp == 1 ? 1 : 2;
  tuning_.rows_extra = t.rows_extra ? 1 : 0;
  tuning_.warps_per_block = (t.warps_per_block == 1 || t.warps_per_block == 2) ? t.warps_per_block : kWarpsPerBlock;
}

std::vector<std::array<int, 4>> Engine::first_pass() const {
  std::vector<std::array<int, 4>> out;
  for (const Bin& b : bins_) out.push_back({static_cast<int>(b.kind), b.rows, b.blocks, b.warps});
  return out;
}

int Engine::time_run(int repeats, double* ms) {
  DeviceGuard device_guard(device_);
  if (repeats < 1) repeats = 1;
  int rc;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if ((rc = check(cudaEventCreate(&e0), "timing event")) || (rc = check(cudaEventCreate(&e1), "timing event"))) return rc;
  std::vector<double> t;
  for (int i = 0; i <= repeats && rc == FGKL_OK; ++i) {
    if ((rc = begin_run())) break;
    if ((rc = check(cudaEventRecord(e0, stream_), "timing event"))) break;
    if ((rc = run())) break;
    if ((rc = check(cudaEventRecord(e1, stream_), "timing event"))) break;
    if ((rc = end_run())) break;
    if ((rc = check(cudaEventSynchronize(e1), "timed run"))) break;
    float f = 0.f;
    cudaEventElapsedTime(&f, e0, e1);
    if (i > 0) t.push_back(f);  // the first run is a warm-up
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  std::sort(t.begin(), t.end());
  *ms = t[t.size() / 2];
  return FGKL_OK;
}

int Engine::bin_profile(std::vector<BinProfile>* out) {
  DeviceGuard device_guard(device_);
  out->clear();
  if (!profile_) return fail(FGKL_E_INVALID_ARGUMENT, "profiling is off");
  int rc;
  if ((rc = check(cudaStreamSynchronize(stream_), "profiled run"))) return rc;
  int i = 0;
  for (int pass = 0; pass < 2; ++pass)
    for (const Bin& b : pass == 0 ? bins_ : rescue_bins_) {
      float ms = 0.f;
      if (2 * i + 1 < static_cast<int>(ev_.size())) cudaEventElapsedTime(&ms, ev_[2 * i], ev_[2 * i + 1]);
      out->push_back(BinProfile{static_cast<int>(b.kind), b.rows, b.n_tasks, b.blocks, pass, b.fwd_cells, b.bwd_cells, ms});
      ++i;
    }
  return FGKL_OK;
}

int Engine::fetch(double* out, int64_t out_len, BatchStats* stats) {
  DeviceGuard device_guard(device_);
  const auto t_fetch = std::chrono::steady_clock::now();
  if (out_len != out_len_)
    return fail(FGKL_E_OUTPUT_LENGTH, "output has " + std::to_string(out_len) + " elements but reads x haplotypes is " +
                                          std::to_string(out_len_));
  int rc;
  double* h_out = reinterpret_cast<double*>(h_stage_ + out_stage_);
  Counters* h_cnt = reinterpret_cast<Counters*>(h_out + out_len_);
  if ((rc = check(cudaStreamWaitEvent(copy_, computed_, 0), "wait for the kernels"))) return rc;
  // Results go straight into a page-locked output array, else through pinned staging.
  const size_t out_bytes = static_cast<size_t>(out_len_) * sizeof(double);
  const bool direct_out = out_len_ > 0 && host_pinned(out, out_bytes);
  // The counters follow the results on the device and in the staging.
  if (direct_out) {
    if ((rc = check(cudaMemcpyAsync(out, d_out_, out_bytes, cudaMemcpyDeviceToHost, copy_), "download results")) ||
        (rc = check(cudaMemcpyAsync(h_cnt, view_.counters, sizeof(Counters), cudaMemcpyDeviceToHost, copy_), "download counters")))
      return rc;
  } else if ((rc = check(cudaMemcpyAsync(h_out, d_out_, out_bytes + sizeof(Counters), cudaMemcpyDeviceToHost, copy_), "download results"))) {
    return rc;
  }
  if ((rc = check(cudaEventRecord(fetched_, copy_), "download event"))) return rc;
  if ((rc = check(cudaEventSynchronize(fetched_), "kernel execution"))) return rc;
  if (out_len_ > 0 && !direct_out) parallel_copy(reinterpret_cast<uint8_t*>(out), reinterpret_cast<const uint8_t*>(h_out), out_bytes);
  planned_.host_fetch_ms = ms_since(t_fetch);
  if (stats) {
    *stats = planned_;
    stats->fallback_pairs = h_cnt->lost_pairs;
    stats->rescue_reads = h_cnt->rescue_reads;
  }
  return FGKL_OK;
}

int Engine::compute(const BatchInput& in, const EngineConfig& cfg, double* out, int64_t out_len, BatchStats* stats) {
  int rc = prepare(in, cfg);
  if (rc) return rc;
  if (out_len != out_len_)
    return fail(FGKL_E_OUTPUT_LENGTH, "output has " + std::to_string(out_len) + " elements but reads x haplotypes is " +
                                          std::to_string(out_len_));
  if (out_len_ == 0) {
    if (stats) *stats = planned_;
    return FGKL_OK;
  }
  if ((rc = begin_run()) || (rc = run()) || (rc = end_run())) return rc;
  return fetch(out, out_len, stats);
}

}  // namespace fgkl

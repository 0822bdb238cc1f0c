// Batched, tick-driven correction engine.
//
// Every job (one field) runs the reference GPU driver's control flow
// (src/ExtreM_cuda.cu main() :5508-5997) as a state machine on the host: one
// state per phase of that flow (c_loops detection and rounds, r_loops, a
// manifold round with the wrong-neighbour arbitration, s_loops, saddle_loops,
// their join variants, the third block's detection, the final join pass).
// A tick runs, in program order, every phase that any job is in: one launch
// per kernel serves all jobs in that phase (kernels take the device array of
// job descriptors and a selection), and a job moves on through phases whose
// successor does not depend on a counter within the same tick.  At the end of
// a tick its last kernel publishes the counter blocks of all jobs to the host
// (k_tick_end; a copy brings them where it cannot) and every job that stopped at a
// branch takes it, with the reference's rules.
//
// The branches read exactly the counters the reference reads at the same
// points, so a job's sequence of kernel launches, and its result, do not
// depend on what else is in the batch.  The plain entry points run a batch of
// one job; the batch and serving entry points admit many.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <functional>
#include <string>
#include <unordered_map>
#include <vector>

#include "extremz_encode.cuh"
#include "extremz_kernels.cuh"
#include "extremz_topo.cuh"

namespace extremz {

// Trace phases (the same records as the oracle's trace).
enum Phase : int {
  PH_CLOOP_DETECT = 1, PH_WRONG_NBR = 2, PH_SLOOPS = 3, PH_SADDLE = 4, PH_DETECT3 = 5,
  PH_SLOOPS_JOIN = 6, PH_SADDLE_JOIN = 7, PH_OUTER = 8, PH_CHECKSUM = 9
};

// Kernel classes for the optional per-class timing (extremz_report.prof_*).
enum KClass : int {
  K_SETUP = 0, K_DETECT, K_DIRECTION, K_JUMP, K_PROPOSE, K_APPLY, K_ROWS, K_WRONG_NBR,
  K_FIXPATH, K_OTHER, K_DIRECTION_FIRST, K_JUMP_FIRST, K_NUM
};

// Program counter of a job, in the order phases run within a tick.
enum Pc : int {
  PC_SETUP_A = 0,   // classify f, f's manifolds, CP counts          -> sync
  PC_SETUP_B,       // CP lists, rows, per-extremum saddles             -> CL_DETECT
  PC_CL_DETECT,     // c_loops entry: detection                         -> sync
  PC_CL_ROUND,      // c_loops round: proposals, apply, detection       -> sync
  PC_RLOOPS,        // r_loops (fixpath)                                -> MANIFOLD
  PC_MANIFOLD,      // manifolds, rows, wrong neighbours                -> sync
  PC_SLOOPS,        // s_loops                                          -> sync
  PC_SADDLE,        // saddle_loops
  PC_SLOOPS_J,      // s_loops_join                                     -> sync
  PC_SADDLE_J,      // saddle_loops_join (inside the loop)
  PC_PRE_END,       // counters re-read before the loop (:5589-5599)    -> sync
  PC_DET3,          // third block: wrong max / saddle detection
  PC_DET3J,         // third block: join detection
  PC_FINAL_DETECT,  // end of an outer iteration: detection             -> sync
  PC_FINAL_JOIN,    // unconditional saddle_loops_join (:5997)          -> sync
  PC_DONE,
  PC_COUNT = PC_DONE
};

// The branch of a phase.  A job that passes through several phases in one tick
// stays in one branch: setup to detection, r_loops to the manifold round,
// saddle_loops to the join variants, the third block to its detection.
constexpr int kBranches = 6;
constexpr int branch_of(int pc) {
  return pc <= PC_CL_DETECT                       ? 0
         : pc == PC_CL_ROUND                      ? 1
         : pc == PC_RLOOPS || pc == PC_MANIFOLD   ? 2
         : pc == PC_SLOOPS                        ? 3
         : pc <= PC_PRE_END || pc == PC_FINAL_JOIN ? 4
                                                  : 5;
}

template <class T>
__global__ void k_checksum(const T* __restrict__ a, int N, unsigned long long* out) {
  unsigned long long acc = 0;
  const int stride = gridDim.x * blockDim.x;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < N; v += stride) {
    unsigned long long bits = 0;
    if (sizeof(T) == 8) bits = (unsigned long long)__double_as_longlong((double)a[v]);
    else bits = (unsigned long long)__float_as_uint((float)a[v]);
    unsigned long long z = bits + 0x9e3779b97f4a7c15ull * (unsigned long long)(v + 1);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    acc += z ^ (z >> 31);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, acc);
}

// Workspace of one job of n voxels, in two parts: the per-voxel arrays, taken
// at admission, and the per-critical-point arrays, taken once the counts are
// known (ns2 2-saddles, ns1 1-saddles, nmax maxima, nmin minima).  ksz is the
// size of an order-preserving key (4 or 8).
constexpr long long arr_bytes(long long count, long long sz) { return (count * sz + 255) & ~255ll; }

// Internal job flag (outside the public EXTREMZ_FLAG_* bits): keep a copy of
// the incoming decompressed field for the edit stream.
constexpr int kFlagKeepInput = 1 << 30;
// Internal job flag: analysis only -- classification, labels and critical-point
// lists of the field (admitted as the original), no correction.
constexpr int kFlagAnalysis = 1 << 29;
// Internal job flag: keep the bitset of voxels whose value changed (Job::edited)
// so that only those travel back to a host buffer.
constexpr int kFlagTrackEdits = 1 << 28;
// Internal job flag: mismatch census -- the loop test's eleven counters
// evaluated once on the decompressed field (detection, one manifold round
// with the wrong-neighbour arbitration, and the wrong-extremum / wrong-saddle
// detection of both trees), no edit.
constexpr int kFlagCensus = 1 << 27;
// Internal job flag, with kFlagAnalysis: the analysis ends with the types and
// labels (no critical-point lists).
constexpr int kFlagLabels = 1 << 26;
constexpr int kInternalFlags =
    kFlagKeepInput | kFlagAnalysis | kFlagTrackEdits | kFlagCensus | kFlagLabels;

constexpr long long job_bytes_voxels(long long n, long long ksz) {
  return arr_bytes(n, 1) + arr_bytes(n, 2)                          // otype, olm
         + 5 * arr_bytes(n, 4)                                      // ds, as, dds, das, ext
         + arr_bytes(n, ksz) + 3 * arr_bytes(n, 4)                  // delta, counter, touched, mm
         + 3 * arr_bytes(n, 4)                                      // mm_next, dirty lists
         + arr_bytes(n, 8)                                          // claim
         + 4 * arr_bytes(n, 4)                                      // cand(_next), flagged(1)
         + arr_bytes(n, 4) + arr_bytes(n, 1)                        // cand_j, mis
         + 2 * arr_bytes(n, 4)                                      // pdd, pda
         + arr_bytes((n + 31) / 32, 4) + arr_bytes(n, 1)            // change bitset, dirtyv
         + 8 * arr_bytes((n + 31) / 32, 4)  // wrong-saddle change, touched roots, dirty, taken
         + 2 * arr_bytes((n + kCpBlock - 1) / kCpBlock, 4)  // bdirty, seed count per block
         + arr_bytes(6 * ((n + kCpBlock - 1) / kCpBlock), 4)        // CP block counts
         + arr_bytes(6 * ((n + kCpBlock - 1) / kCpBlock / 1024 + 1), 4)  // and their chunk sums
         + 4096;
}

constexpr long long job_bytes_cps(long long ns2, long long ns1, long long nmax, long long nmin,
                                  long long e2, long long e1, long long ksz) {
  return arr_bytes(ns2, 4) + arr_bytes(ns1, 4) + arr_bytes(nmax, 4) + arr_bytes(nmin, 4)
         + arr_bytes(ns2, 2)                                        // smask2
         + arr_bytes(ns2 * kRowStride, 4) + arr_bytes(ns2 * 2, 4) + arr_bytes(ns2, 1)
         + arr_bytes(ns1 * kRowStride, 4) + arr_bytes(ns1 * 2, 4) + arr_bytes(ns1, 1)
         + 2 * arr_bytes(ns2, 16) + 2 * arr_bytes(ns1, 16)  // compact rows (orm, oend)
         + 2 * arr_bytes(ns2, 1) + 2 * arr_bytes(ns1, 1)            // seed bits, wrong-row bits
         + 4 * arr_bytes(nmax, 4) + 4 * arr_bytes(nmin, 4)
         + arr_bytes(nmax > nmin ? nmax : nmin, ksz) + arr_bytes(nmax > nmin ? nmax : nmin, 4)
         + arr_bytes(8, 8)
         // per-extremum row-entry lists: offsets, entries, stamps; queue, chunk sums
         + arr_bytes(nmax + 1, 4) + arr_bytes(e2, 4) + arr_bytes(nmax, 4)
         + arr_bytes(nmin + 1, 4) + arr_bytes(e1, 4) + arr_bytes(nmin, 4)
         + 2 * arr_bytes(nmax > nmin ? nmax : nmin, 4)
         + arr_bytes((nmax > nmin ? nmax : nmin) / 1024 + 2, 4) + 4096;
}

// An analysis job (kFlagAnalysis) takes the original field's types, masks and
// labels, the extremum index and the CP block counts; then the CP lists.
constexpr long long job_bytes_analysis(long long n) {
  return arr_bytes(n, 1) + arr_bytes(n, 2) + 3 * arr_bytes(n, 4)
         + arr_bytes(6 * ((n + kCpBlock - 1) / kCpBlock), 4)
         + arr_bytes(6 * ((n + kCpBlock - 1) / kCpBlock / 1024 + 1), 4) + 4096;
}
constexpr long long job_bytes_lists(long long ns2, long long ns1, long long nmax, long long nmin) {
  return arr_bytes(ns2, 4) + arr_bytes(ns1, 4) + arr_bytes(nmax, 4) + arr_bytes(nmin, 4) + 4096;
}

// Per tile: change mark, jump stamp and queue entry.
constexpr long long job_bytes_tiles(long long nt) { return 2 * arr_bytes(nt, 4) + arr_bytes(nt, 8); }

// Worst case (every voxel a critical point of every kind; a voxel's upper and
// lower neighbours, at most 14, give the row entries of both sides; a tile for
// every four voxels and one more, as a 1 x 1 x n column has).
static_assert(TZ == 4 && TY >= 4 && TX >= 4, "the worst case's tiles");
constexpr long long job_bytes_sz(long long n, long long ksz) {
  return job_bytes_voxels(n, ksz) + job_bytes_tiles(n / 4 + 1) +
         job_bytes_cps(n, n, n, n, 7 * n, 7 * n, ksz);
}
template <class T>
constexpr long long job_bytes(long long n) {
  return job_bytes_sz(n, sizeof(typename KeyOf<T>::K));
}
constexpr long long job_bytes_max(long long n) { return job_bytes_sz(n, 8); }

// What a field of n voxels is charged against a server's budget and reported as
// its footprint: a published number, so it does not follow every change of the
// workspace.  It stands for the arrays below (count x bytes each) and must cover
// the worst case; the 64 KiB are for alignment, which only fields of some thousand
// voxels notice.
constexpr long long job_charge(long long n) {
  const long long words = (n + 31) / 32, blocks = (n + kCpBlock - 1) / kCpBlock;
  return 9 * arr_bytes(n, 1) + arr_bytes(n, 2) + 38 * arr_bytes(n, 4) + 5 * arr_bytes(n, 8) +
         4 * arr_bytes(n, 16) + 2 * arr_bytes(7 * n, 4) + 2 * arr_bytes(n * kRowStride, 4) +
         2 * arr_bytes(n + 1, 4) + 5 * arr_bytes(words, 4) + 2 * arr_bytes(blocks, 4) +
         arr_bytes(6 * blocks, 4) + arr_bytes(6 * (blocks / 1024 + 1), 4) +
         arr_bytes(n / 1024 + 2, 4) + arr_bytes(8, 8) + 2 * 4096;
}
static_assert(job_charge(1) + (64 << 10) >= job_bytes_max(1) &&
                  job_charge(1 << 12) >= job_bytes_max(1 << 12) &&
                  job_charge(1ll << 28) >= job_bytes_max(1ll << 28),
              "a field's charge covers its worst case");

// One job's host-side state.
template <class T>
struct JobHost {
  using K = typename KeyOf<T>::K;
  bool used = false;
  int pc = PC_DONE;
  int block = 0;          // 0 = before the loop, 1..3 = block of an outer iteration
  bool waiting = false;   // stopped at a branch that needs this tick's counters
  cudaEvent_t input_ready = nullptr;  // the decompressed field is still arriving until this event
  int outer = 0, rounds = 0, cloop_total = 0, manifold_rounds = 0;
  bool wim_seen = false, wis_seen = false;  // the split side's scans ran since the last
                                            // computed manifold round
  int reused = 0;         // manifold rounds that launched nothing: no value had changed
  int nfc = 0, nfc1 = 0;
  int c[11] = {0};        // loop-test counters (:5603-5605)
  bool dense_done = false;
  int status = EXTREMZ_OK;
  extremz_params p{};
  Job<T> J{};
  Arena arena, arena2;  // per-voxel part, per-critical-point part
  bool own_arena = false, own_arena2 = false;
  int ntiles = 0, nb = 0;
  int* bcount = nullptr;
  int* chunk = nullptr;  // chunk sums of the CP block counts
  unsigned long long* checksum = nullptr;
  int32_t* trace = nullptr;
  int trace_cap = 0, trace_len = 0;
  std::vector<int> pending;  // trace phases to emit once the tick's counters are back
  int blocks_per_sm = 4;      // grid-stride kernels' blocks per SM (tuning knob)
  long long applied_tick = -1;  // last tick that issued edits for this job
  long long tag = 0;

  void emit(int phase, int a = 0, int b = 0, int c3 = 0) {
    if (!trace || trace_len + 4 > trace_cap) return;
    trace[trace_len++] = phase;
    trace[trace_len++] = a;
    trace[trace_len++] = b;
    trace[trace_len++] = c3;
  }
};

// Where an analysis job writes its types and labels when the caller's buffers
// can be written in place (null: into the workspace).
struct LabelOut {
  int8_t* type = nullptr;
  int* ds = nullptr;
  int* as = nullptr;
};

template <class T>
class BatchEngine {
 public:
  using K = typename KeyOf<T>::K;

  explicit BatchEngine(cudaStream_t st) : st_(st) {}
  ~BatchEngine() { release_all(); }

  int init(const DeviceTables* preset_tables, Arena* fixed_storage) {
    wait_known_ = false;
    if (ready_) return EXTREMZ_OK;
    int dev = 0;
    EZ_CHECK(cudaGetDevice(&dev));
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    sms_ = sms;
    grid_ = sms * 8;
    if (preset_tables) tb_ = *preset_tables;
    else if (int rc = device_tables(&tb_)) return rc;
    const size_t desc_bytes = sizeof(Job<T>) * kMaxSel;
    const size_t ctr_bytes = sizeof(int) * C_COUNT * kMaxSel;
    if (fixed_storage) {  // borrowed: carve the engine's arrays from it
      jobs_dev_ = fixed_storage->template take<Job<T>>(kMaxSel);
      ctr_dev_ = fixed_storage->template take<int>(C_COUNT * kMaxSel);
      if (!jobs_dev_ || !ctr_dev_) return EXTREMZ_OOM;
      borrowed_ = true;
      ctr_host_ = static_ctr_host_;
    } else {
      if (cudaMalloc(&jobs_dev_, desc_bytes) != cudaSuccess ||
          cudaMalloc(&ctr_dev_, ctr_bytes + sizeof(unsigned)) != cudaSuccess ||
          cudaMemset(ctr_dev_, 0, ctr_bytes + sizeof(unsigned)) != cudaSuccess ||
          cudaMallocHost(&ctr_host_, 3 * ctr_bytes) != cudaSuccess) {
        cudaGetLastError();
        return EXTREMZ_OOM;
      }
      std::memset(ctr_host_, 0, 3 * ctr_bytes);
      seq_dev_ = reinterpret_cast<unsigned*>(ctr_dev_ + C_COUNT * kMaxSel);
      static_assert(C_COUNT * kMaxSel % 2 == 0, "the published counters are 8-byte aligned");
      pub_host_ = reinterpret_cast<volatile unsigned long long*>(ctr_host_ + C_COUNT * kMaxSel);
    }
    slots_.assign(kMaxSel, JobHost<T>());
    ready_ = true;
    return EXTREMZ_OK;
  }

  void release_all() {
    drop_graphs();
    for (auto& j : slots_) free_job(j);
    if (!borrowed_) {
      if (jobs_dev_) cudaFree(jobs_dev_);
      if (ctr_dev_) cudaFree(ctr_dev_);
      if (ctr_host_) cudaFreeHost(ctr_host_);
    }
    jobs_dev_ = nullptr;
    ctr_dev_ = nullptr;
    ctr_host_ = nullptr;
    ready_ = false;
  }

  int free_slots() const {
    int n = 0;
    for (const auto& j : slots_) n += !j.used;
    return n;
  }
  int active() const {
    int n = 0;
    for (const auto& j : slots_) n += j.used && j.pc != PC_DONE;
    return n;
  }
  long long launches() const { return launches_; }
  long long graph_replays() const { return graph_replays_; }
  long long graph_captures() const { return graph_captures_; }
  void set_graphs(bool on) {
    graphs_on_ = on;
    if (!on) drop_graphs();
  }
  void set_stream(cudaStream_t st) { st_ = st; }
  cudaStream_t stream() const { return st_; }
  // Stream-ordered pool the job workspaces come from (nullptr: the device's
  // default pool).
  void set_pool(cudaMemPool_t pool) { pool_mem_ = pool; }
  void set_profile(bool on, int mask) {
    profile_ = on;
    profile_mask_ = mask;
  }

  // Admits a job.  storage: borrowed workspace (nullptr = allocate).
  int admit(const T* f, T* g, int W, int H, int D, const extremz_params& p, int32_t* trace,
            int trace_cap, Arena* storage, long long tag, int* slot_out,
            const LabelOut& out = LabelOut()) {
    int slot = -1;
    for (int i = 0; i < kMaxSel; ++i)
      if (!slots_[i].used) {
        slot = i;
        break;
      }
    if (slot < 0) return EXTREMZ_OOM;
    JobHost<T>& jh = slots_[slot];
    jh = JobHost<T>();
    jh.used = true;
    jh.p = p;
    jh.tag = tag;
    jh.trace = trace;
    jh.trace_cap = trace_cap;
    Job<T>& J = jh.J;
    std::memset(&J, 0, sizeof(J));
    J.dim = Dims{W, H, D, W * H * D};
    J.f = f;
    J.g = g;
    J.bound = (T)p.bound;
    J.thr = (T)p.thr;
    J.sentinel = T(-4.0) * J.bound;  // init_delta (:2572)
    J.sentinel_key = KeyOf<T>::enc(J.sentinel);
    J.q = p.q;
    J.edit_type = p.edit_type;
    J.iter_cap = p.device_iter_cap > 0 ? p.device_iter_cap : J.dim.N + 1;
    J.pass_chunk = p.tune_pass_chunk > 0 ? p.tune_pass_chunk : 4;
    J.wn_lockstep = (p.flags & EXTREMZ_FLAG_WN_ASCENDING) == 0;
    J.join_rows = p.preserve_join || (p.flags & kFlagCensus);
    jh.blocks_per_sm = p.tune_blocks_per_sm > 0 ? p.tune_blocks_per_sm : 4;
    J.tb = tb_;
    J.ctr = ctr_dev_ + (size_t)slot * C_COUNT;
    const int N = J.dim.N;
    // Borrowed storage holds both parts; an allocation holds the first (and a
    // copy of the incoming field when an edit stream will be encoded).
    const bool keep_input = (p.flags & kFlagKeepInput) != 0;
    const bool track_edits = (p.flags & kFlagTrackEdits) != 0;
    const bool analysis = (p.flags & kFlagAnalysis) != 0;
    const long long ntiles = (long long)((W + TX - 1) / TX) * ((H + TY - 1) / TY) * ((D + TZ - 1) / TZ);
    const long long need = (storage    ? job_bytes<T>(N)
                            : analysis ? job_bytes_analysis(N)
                                       : job_bytes_voxels(N, sizeof(K)) + job_bytes_tiles(ntiles)) +
                           (keep_input ? arr_bytes(N, sizeof(T)) : 0) +
                           (track_edits ? arr_bytes((N + 31) / 32, 4) : 0);
    if (storage) {
      jh.arena = *storage;
      jh.arena.used = 0;
      if ((long long)jh.arena.cap < need) {
        jh.used = false;
        return EXTREMZ_OOM;
      }
    } else {
      void* base = nullptr;
      const cudaError_t e = pool_mem_ ? cudaMallocFromPoolAsync(&base, (size_t)need, pool_mem_, st_)
                                      : cudaMallocAsync(&base, (size_t)need, st_);
      if (e != cudaSuccess) {
        cudaGetLastError();
        jh.used = false;
        return EXTREMZ_OOM;
      }
      jh.arena.base = static_cast<char*>(base);
      jh.arena.cap = (size_t)need;
      jh.arena.fixed = true;
      jh.own_arena = true;
    }
    Arena& A = jh.arena;
    J.otype = out.type ? out.type : A.take<int8_t>(N);
    J.olm = A.take<uint16_t>(N);
    J.ds = out.ds ? out.ds : A.take<int>(N);
    J.as = out.as ? out.as : A.take<int>(N);
    J.ext = A.take<int>(N);
    jh.nb = (N + kCpBlock - 1) / kCpBlock;
    jh.bcount = A.take<int>(6ll * jh.nb);
    jh.chunk = A.take<int>(6ll * ((jh.nb + 1023) / 1024));
    J.cpoff = jh.bcount;
    jh.ntiles = ((W + TX - 1) / TX) * ((H + TY - 1) / TY) * ((D + TZ - 1) / TZ);
    if (!jh.chunk) {
      free_job(jh);
      return EXTREMZ_OOM;
    }
    // An analysis reads and writes nothing else.
    if (!analysis) {
      J.dds = A.take<int>(N);
      J.das = A.take<int>(N);
      J.delta = A.take<K>(N);
      J.counter = A.take<int>(N);
      J.touched = A.take<int>(N);
      J.mm = A.take<int>(N);
      J.mm_next = A.take<int>(N);
      J.dirty = A.take<int>(N);
      J.dirty1 = A.take<int>(N);
      J.claim = A.take<unsigned long long>(N);
      J.cand = A.take<int>(N);
      J.cand_next = A.take<int>(N);
      J.flagged = A.take<int>(N);
      J.flagged1 = A.take<int>(N);
      J.cand_j = A.take<int>(N);
      J.mis = A.take<uint8_t>(N);
      J.pdd = A.take<int>(N);
      J.pda = A.take<int>(N);
      J.vchg = A.take<unsigned>((N + 31) / 32);
      J.rtouch2 = A.take<unsigned>((N + 31) / 32);
      J.rtouch1 = A.take<unsigned>((N + 31) / 32);
      J.wchg2 = A.take<unsigned>((N + 31) / 32);
      J.wchg1 = A.take<unsigned>((N + 31) / 32);
      J.dbits = A.take<unsigned>((N + 31) / 32);
      J.dbits1 = A.take<unsigned>((N + 31) / 32);
      J.taken = A.take<unsigned>((N + 31) / 32);
      J.taken1 = A.take<unsigned>((N + 31) / 32);
      J.dirtyv = A.take<uint8_t>(N);
      J.bdirty = A.take<int>(jh.nb);
      J.hcnt = A.take<int>(jh.nb);
      J.tseen = A.take<int>(jh.ntiles);
      J.tqueue = A.take<unsigned long long>(jh.ntiles);
      J.tdirty = A.take<int>(jh.ntiles);
      J.g0 = keep_input ? A.take<T>(N) : nullptr;
      J.edited = track_edits ? A.take<unsigned>((N + 31) / 32) : nullptr;
    }
    if ((!analysis && !J.tdirty) || (keep_input && !J.g0) || (track_edits && !J.edited)) {
      free_job(jh);
      return EXTREMZ_OOM;
    }
    if (track_edits)
      EZ_CHECK(cudaMemsetAsync(J.edited, 0, (size_t)((N + 31) / 32) * 4, st_));
    if (keep_input)
      EZ_CHECK(cudaMemcpyAsync(J.g0, g, (size_t)N * sizeof(T), cudaMemcpyDeviceToDevice, st_));
    // Tile maps of both fields (TMA when the stride allows).
    const bool tma_ok = (p.flags & EXTREMZ_FLAG_NO_TMA) == 0;
    J.tma_f = tma_ok && make_tile_map(&J.map_f, f, J.dim);
    J.tma_g = tma_ok && make_tile_map(&J.map_g, (const T*)g, J.dim);
    EZ_CHECK(cudaMemsetAsync(J.ctr, 0, C_COUNT * sizeof(int), st_));
    EZ_CHECK(cudaMemcpyAsync(jobs_dev_ + slot, &J, sizeof(J), cudaMemcpyHostToDevice, st_));
    jh.pc = PC_SETUP_A;
    if (slot_out) *slot_out = slot;
    return EXTREMZ_OK;
  }

  const JobHost<T>& job(int slot) const { return slots_[slot]; }

  void fill_report(int slot, extremz_report* r) const {
    const JobHost<T>& j = slots_[slot];
    if (!r) return;
    r->status = j.status;
    r->outer_iters = j.outer;
    r->cloop_rounds = j.cloop_total;
    r->manifold_rounds = j.manifold_rounds;
    std::memcpy(r->counters, j.c, sizeof(j.c));
    r->error_bits = ctr_host_ ? ctr_host_[(size_t)slot * C_COUNT + C_ERROR] : 0;
    r->manifold_reused = j.reused + (ctr_host_ ? ctr_host_[(size_t)slot * C_COUNT + C_MFREUSED] : 0);
    for (int k = 0; k < 4; ++k)
      r->cp_counts[k] = ctr_host_ ? ctr_host_[(size_t)slot * C_COUNT + C_NS2 + k] : 0;
  }

  // Edit stream of a finished job admitted with kFlagKeepInput, into the
  // caller's device buffers es->index / es->edits (see extremz_encode.cuh).
  // Synchronises the stream.  BAD_ARG when a buffer is too small (the sizes
  // needed are filled in) or a counter does not fit three bits.
  int encode(int slot, extremz_edit_stream* es) {
    JobHost<T>& jh = slots_[slot];
    const Job<T>& J = jh.J;
    if (!J.g0 || !es) return EXTREMZ_BAD_ARG;
    const int N = J.dim.N, nb = jh.nb, et = jh.p.edit_type, q = jh.p.q;
    if (et == 0 && q > 7) return EXTREMZ_BAD_ARG;  // counters up to q: three bits
    unsigned long long* acc = jh.checksum;         // 8 words of scratch
    unsigned long long init[8] = {0, 0, KeyOf<double>::enc((double)INFINITY),
                                  KeyOf<double>::enc(-(double)INFINITY), 0, 0, 0, 0};
    EZ_CHECK(cudaMemcpyAsync(acc, init, sizeof(init), cudaMemcpyHostToDevice, st_));
    int* bc = jh.bcount;  // 4 x nb ints, free once the correction is over
    launch(K_OTHER, k_enc_count<T>, nb, kCpBlock, (const T*)J.g0, (const T*)J.g,
           (const int*)J.counter, N, q, et, bc);
    launch(K_OTHER, k_scan_lists, 2, 1024, bc, nb, reinterpret_cast<int*>(acc + 4), (int*)nullptr);
    launch(K_OTHER, k_enc_stats<T>, grid_, 256, J.f, (const T*)J.g0, (const T*)J.g, N, acc);
    unsigned long long h[8];
    EZ_CHECK(cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, st_));
    EZ_CHECK(cudaStreamSynchronize(st_));
    int tot[2];
    std::memcpy(tot, &h[4], sizeof(tot));
    const long long index_bytes = et == 0 ? (3ll * N + 7) / 8 : 4ll * tot[0];
    const long long edit_bytes = (long long)tot[1] * (long long)sizeof(T);
    es->edited = tot[0];
    es->n_edits = tot[1];
    es->index_bytes = index_bytes;
    es->edit_bytes = edit_bytes;
    double s0, s1;
    std::memcpy(&s0, &h[0], 8);
    std::memcpy(&s1, &h[1], 8);
    const double range = KeyOf<double>::dec(h[3]) - KeyOf<double>::dec(h[2]);
    auto psnr = [&](double sse) {
      const double mse = sse / (double)N;
      return mse == 0 ? (double)INFINITY : -20.0 * std::log10(std::sqrt(mse) / range);
    };
    es->psnr_before = psnr(s0);
    es->psnr_after = psnr(s1);
    if (index_bytes > es->index_cap || edit_bytes > es->edits_cap ||
        (index_bytes && !es->index) || (edit_bytes && !es->edits))
      return EXTREMZ_BAD_ARG;
    launch(K_OTHER, k_enc_write<T>, nb, kCpBlock, J.f, (const T*)J.g0, (const T*)J.g,
           (const int*)J.counter, N, J.bound, q, et, (const int*)bc, J.touched,
           static_cast<T*>(es->edits));
    if (et == 1) {
      launch(K_OTHER, k_enc_diff, grid_, 256, (const int*)J.touched, tot[0],
             static_cast<int*>(es->index));
    } else {
      launch(K_OTHER, k_enc_pack3<T>, grid_, 256, (const T*)J.g0, (const T*)J.g,
             (const int*)J.counter, (long long)N, static_cast<uint8_t*>(es->index), index_bytes,
             acc + 5);
    }
    unsigned long long bad = 0;
    EZ_CHECK(cudaMemcpyAsync(&bad, acc + 5, 8, cudaMemcpyDeviceToHost, st_));
    EZ_CHECK(cudaStreamSynchronize(st_));
    return bad ? EXTREMZ_BAD_ARG : EXTREMZ_OK;
  }

  // Voxels of a finished job admitted with kFlagTrackEdits whose value
  // changed: ids (ascending) into the job's `touched` array and their
  // corrected values into its proposal buffer, both free once the correction
  // is over.  Returns the count; edited_ids / edited_vals give the arrays.
  int edited_list(int slot, int* count) {
    JobHost<T>& jh = slots_[slot];
    const Job<T>& J = jh.J;
    static_assert(sizeof(K) == sizeof(T), "values are written over the proposal keys");
    if (!J.edited) return EXTREMZ_BAD_ARG;
    const int N = J.dim.N, nb = jh.nb;
    int* tot = reinterpret_cast<int*>(jh.checksum);
    launch(K_OTHER, k_edit_count, nb, 32, (const unsigned*)J.edited, N, jh.bcount);
    launch(K_OTHER, k_scan_lists, 1, 1024, jh.bcount, nb, tot, (int*)nullptr);
    launch(K_OTHER, k_edit_write<T>, nb, 32, (const unsigned*)J.edited, (const T*)J.g, N,
           (const int*)jh.bcount, J.touched, reinterpret_cast<T*>(J.delta));
    EZ_CHECK(cudaMemcpyAsync(count, tot, sizeof(int), cudaMemcpyDeviceToHost, st_));
    EZ_CHECK(cudaStreamSynchronize(st_));
    return EXTREMZ_OK;
  }
  const int* edited_ids(int slot) const { return slots_[slot].J.touched; }
  const T* edited_vals(int slot) const { return reinterpret_cast<const T*>(slots_[slot].J.delta); }

  // Stream-ordered scratch from the engine's pool (or the device's default).
  void* scratch(size_t bytes) {
    void* p = nullptr;
    const cudaError_t e = pool_mem_ ? cudaMallocFromPoolAsync(&p, bytes, pool_mem_, st_)
                                    : cudaMallocAsync(&p, bytes, st_);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    return p;
  }

  // Merge-tree persistence pairs of a finished analysis job (see
  // extremz_topo.cuh): split tree into max_pairs (2 ints per maximum), join
  // tree into min_pairs (2 per minimum), device buffers of the caller.
  // counts (host) receives the numbers of maxima and minima.  Synchronises.
  int persistence(int slot, int* max_pairs, long long max_cap, int* min_pairs, long long min_cap,
                  long long* counts, int* max_parent = nullptr, int* min_parent = nullptr) {
    JobHost<T>& jh = slots_[slot];
    const Job<T>& J = jh.J;
    const int ne[2] = {h(slot, C_NMAX), h(slot, C_NMIN)};
    counts[0] = ne[0];
    counts[1] = ne[1];
    if (2ll * ne[0] > max_cap || 2ll * ne[1] > min_cap || (ne[0] && !max_pairs) ||
        (ne[1] && !min_pairs))
      return EXTREMZ_BAD_ARG;
    // Merge vertices of both trees, ascending id (the job's CP-block scratch
    // is free once the analysis is done).
    const int N = J.dim.N;
    // The two lists, then the component table and the membership words.
    const size_t cand_bytes = ((size_t)2 * N * sizeof(int) + 255) & ~size_t(255);
    const size_t member_words = (size_t)2 * jh.nb * (kCpBlock / 32);
    int* cand = static_cast<int*>(scratch(cand_bytes + (kMergeWords + member_words) * 4));
    if (!cand) return EXTREMZ_OOM;
    unsigned* table = reinterpret_cast<unsigned*>(reinterpret_cast<char*>(cand) + cand_bytes);
    unsigned* member = table + kMergeWords;
    int* ctot = J.ctr + C_CAND;  // two free counter slots of the finished job
    launch(K_OTHER, k_pp_merge_table, kMergeWords * 32 / 256, 256, tb_, table);
    launch(K_OTHER, k_pp_cand_count<T>, jh.nb, kCpBlock, J.f, J.dim, (const unsigned*)table, member,
           jh.bcount);
    launch(K_OTHER, k_scan_lists, 2, 1024, jh.bcount, jh.nb, ctot, (int*)nullptr);
    launch(K_OTHER, k_pp_cand_write, dim3((jh.nb + 7) / 8, 2), 256, (const unsigned*)member, jh.nb,
           (const int*)jh.bcount, cand, cand + N);
    int ns[2];
    EZ_CHECK(cudaMemcpyAsync(ns, ctot, sizeof(ns), cudaMemcpyDeviceToHost, st_));
    EZ_CHECK(cudaStreamSynchronize(st_));
    const int nmaxall = std::max(std::max(ns[0], ns[1]), std::max(ne[0], ne[1])) + 1;
    // Scratch: sort keys and values (in and out), ranks, rows and counts,
    // largest / pointer / pair per extremum, sorted list indices of both
    // sides' extrema, and the round flag.
    size_t cub_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, (unsigned long long*)nullptr,
                                    (unsigned long long*)nullptr, (int*)nullptr, (int*)nullptr,
                                    nmaxall, 0, 64, st_);
    const size_t a = ((size_t)nmaxall * 8 + 255) & ~size_t(255);
    const size_t b = ((size_t)nmaxall * 4 + 255) & ~size_t(255);
    const size_t rows_bytes = (((size_t)std::max(ns[0], ns[1]) + 1) * kPpRow * 4 + 255) & ~size_t(255);
    const size_t total = 2 * a + 10 * b + rows_bytes + ((cub_bytes + 255) & ~size_t(255)) + 256;
    char* base = static_cast<char*>(scratch(total));
    if (!base) {
      cudaFreeAsync(cand, st_);
      return EXTREMZ_OOM;
    }
    char* q = base;
    auto take = [&](size_t n) { char* r = q; q += n; return r; };
    auto* kin = reinterpret_cast<unsigned long long*>(take(a));
    auto* kout = reinterpret_cast<unsigned long long*>(take(a));
    int* vin = reinterpret_cast<int*>(take(b));
    int* ext_li[2] = {reinterpret_cast<int*>(take(b)), reinterpret_cast<int*>(take(b))};
    int* sad_li = reinterpret_cast<int*>(take(b));
    int* erank = reinterpret_cast<int*>(take(b));
    int* largest = reinterpret_cast<int*>(take(b));
    int* ptr = reinterpret_cast<int*>(take(b));
    int* pair = reinterpret_cast<int*>(take(b));
    int* lmax = reinterpret_cast<int*>(take(b));
    int* cnt = reinterpret_cast<int*>(take(b));
    int* rows = reinterpret_cast<int*>(take(rows_bytes));
    void* cub_tmp = take((cub_bytes + 255) & ~size_t(255));
    int* flag = reinterpret_cast<int*>(take(256));  // [0] round paired, [1] jump limit hit
    EZ_CHECK(cudaMemsetAsync(flag, 0, 8, st_));
    const int* elist[2] = {J.maxima, J.minima};
    const int* slist[2] = {cand, cand + N};
    int rc = EXTREMZ_OK;
    auto sort = [&](const int* list, int n, bool reverse, bool complement, int* out_li) {
      launch(K_OTHER, k_pp_keys<T>, grid_, 256, J.f, list, n, reverse, complement, kin, vin);
      size_t tb = cub_bytes;
      // A float's key has 32 bits (complemented, the others are all ones).
      if (cub::DeviceRadixSort::SortPairs(cub_tmp, tb, kin, kout, vin, out_li, n, 0,
                                          8 * (int)sizeof(K), st_) !=
          cudaSuccess)
        rc = EXTREMZ_CUDA_ERR;
    };
    // Extrema ascending in each tree's order: maxima by (value, id), minima by
    // the reverse of it.
    if (ne[0]) sort(elist[0], ne[0], false, false, ext_li[0]);
    if (ne[1]) sort(elist[1], ne[1], true, true, ext_li[1]);
    int glob[2] = {-1, -1};  // global maximum, global minimum (vertex ids)
    if (ne[0] && ne[1] && rc == EXTREMZ_OK) {
      int li[2];
      EZ_CHECK(cudaMemcpyAsync(&li[0], ext_li[0] + ne[0] - 1, 4, cudaMemcpyDeviceToHost, st_));
      EZ_CHECK(cudaMemcpyAsync(&li[1], ext_li[1] + ne[1] - 1, 4, cudaMemcpyDeviceToHost, st_));
      EZ_CHECK(cudaStreamSynchronize(st_));
      EZ_CHECK(cudaMemcpyAsync(&glob[0], elist[0] + li[0], 4, cudaMemcpyDeviceToHost, st_));
      EZ_CHECK(cudaMemcpyAsync(&glob[1], elist[1] + li[1], 4, cudaMemcpyDeviceToHost, st_));
      EZ_CHECK(cudaStreamSynchronize(st_));
    }
    for (int side = 0; side < 2 && rc == EXTREMZ_OK; ++side) {
      const bool kmax = side == 0;
      const int n_e = ne[side], n_s = ns[side];
      if (n_e == 0) continue;
      launch(K_OTHER, k_pp_rank, grid_, 256, (const int*)ext_li[side], n_e, erank);
      // Saddles descending in the tree's order.
      if (n_s) sort(slist[side], n_s, kmax, kmax, sad_li);
      if (kmax)
        launch(K_OTHER, k_pp_rows<T, true>, grid_, 256, J.f, (const uint16_t*)J.olm,
               (const int*)J.ctr, J.dim, slist[0],
               (const int*)sad_li, n_s, (const int*)J.ds, (const int*)J.ext, (const int*)erank, rows,
               cnt);
      else
        launch(K_OTHER, k_pp_rows<T, false>, grid_, 256, J.f, (const uint16_t*)J.olm,
               (const int*)J.ctr, J.dim, slist[1],
               (const int*)sad_li, n_s, (const int*)J.as, (const int*)J.ext, (const int*)erank, rows,
               cnt);
      launch(K_OTHER, k_fill<int>, grid_, 256, largest, kInf, (long long)n_e);
      launch(K_OTHER, k_fill<int>, grid_, 256, pair, -1, (long long)n_e);
      launch(K_OTHER, k_iota, grid_, 256, ptr, n_e);
      // Every round but the last pairs one; a round that pairs none changes
      // nothing, so the host asks only after every fourth.
      for (int round = 0; round <= n_e; ++round) {
        if (round % 4 == 0) EZ_CHECK(cudaMemsetAsync(flag, 0, 4, st_));
        if (n_s) launch(K_OTHER, k_pp_largest, grid_, 256, (const int*)rows, (const int*)cnt, n_s,
                        n_e - 1, largest);
        launch(K_OTHER, k_pp_pair, grid_, 256, (const int*)rows, (const int*)cnt, n_e, n_s,
               largest, ptr, pair, lmax, flag);
        if (round % 4 == 3) {
          int changed = 0;
          EZ_CHECK(cudaMemcpyAsync(&changed, flag, 4, cudaMemcpyDeviceToHost, st_));
          EZ_CHECK(cudaStreamSynchronize(st_));
          if (!changed) break;
        }
        launch(K_OTHER, k_pp_jump, grid_, 256, ptr, n_e, n_e + 1, flag + 1);
        if (n_s) launch(K_OTHER, k_pp_remap, grid_, 256, rows, cnt, n_s, (const int*)ptr);
      }
      launch(K_OTHER, k_pp_out, grid_, 256, (const int*)pair, n_e, (const int*)ext_li[side],
             elist[side], (const int*)sad_li, slist[side], glob[1 - side],
             kmax ? max_pairs : min_pairs, (const int*)lmax, kmax ? max_parent : min_parent);
    }
    int jump_err = 0;
    cudaMemcpyAsync(&jump_err, flag + 1, 4, cudaMemcpyDeviceToHost, st_);
    cudaFreeAsync(base, st_);
    cudaFreeAsync(cand, st_);
    EZ_CHECK(cudaStreamSynchronize(st_));
    if (rc == EXTREMZ_OK && jump_err) rc = EXTREMZ_DEVICE_TIMEOUT;
    return rc;
  }

  // Releases a finished job's slot and (stream-ordered) its workspace.
  void release(int slot) {
    slots_[slot].input_ready = nullptr;
    free_job(slots_[slot]);
  }
  // The job's decompressed field is still being copied in until `ev` (on
  // another stream): setup, which reads only the original field, runs
  // meanwhile, and the first tick that reads the decompressed field waits.
  void set_input_event(int slot, cudaEvent_t ev) { slots_[slot].input_ready = ev; }
  // Releases every job (after an error that ends a batch).
  void release_jobs() {
    for (auto& j : slots_) free_job(j);
  }

  // One tick: every phase any job is in, in program order; then all counter
  // blocks and the branches.  Returns a status (the jobs keep their own
  // statuses).
  int tick() {
    EZ_RUN(tick_issue());
    return tick_complete();
  }

  // First half of a tick: the launches, the last of which publishes the counters
  // the host branches on.  Engines on different streams issue, then complete, so
  // their ticks overlap on the device.
  int tick_issue() {
    issued_ = false;
    ++tick_id_;
    const long long launches0 = launches_;
    if (!seq_known_) {  // an earlier tick ended in an error: take up its number
      EZ_CHECK(cudaStreamSynchronize(st_));
      EZ_CHECK(cudaMemcpy(&seq_next_, seq_dev_, sizeof(unsigned), cudaMemcpyDeviceToHost));
      seq_known_ = true;
    }
    // A tick whose launches repeat an earlier tick's exactly (kernels, launch
    // shapes and arguments; per-job state is read from device memory) runs as
    // one CUDA graph: recorded, captured the third time its signature is
    // seen, replayed from then on.  Ticks that allocate (setup) launch
    // directly.  Timed launches (EXTREMZ_FLAG_PROFILE) keep their events
    // inside the graph; a tick with timed launches runs its branches one after the
    // other, and a profiled correction's counters come by a copy, so that the times
    // by class are not those of overlapped ticks.
    bool graph = graphs_on_;
    for (const auto& j : slots_)
      if (j.used && !j.waiting && j.pc == PC_SETUP_B) graph = false;
    if (graph) {
      recording_ = true;
      sig_.clear();
      pending_.clear();
      pending_timed_.clear();
      sig_append(profile_ ? profile_mask_ | (1 << 30) : 0);
    }
    int rc = EXTREMZ_OK;
    for (int ph = 0; ph < PC_COUNT && rc == EXTREMZ_OK; ++ph) {
      std::vector<int> sel;
      for (int i = 0; i < kMaxSel; ++i)
        if (slots_[i].used && !slots_[i].waiting && slots_[i].pc == ph) sel.push_back(i);
      if (sel.empty()) continue;
      issued_ = true;
      // A job can reach its first phase that reads the decompressed field in
      // the same tick as its setup, so the wait goes right before that phase.
      if (ph >= PC_CL_DETECT)
        for (int i : sel)
          if (slots_[i].input_ready) {
            EZ_CHECK(cudaStreamWaitEvent(st_, slots_[i].input_ready, 0));
            slots_[i].input_ready = nullptr;
          }
      branch_ = branch_of(ph);
      rc = run_phase(ph, sel);
    }
    branch_ = -1;
    // A tick that launched nothing (a manifold round over an unchanged field, a
    // re-read of the counters) leaves the host's copy as it is.
    launched_ = rc == EXTREMZ_OK && launches_ != launches0;
    int hi = 0;  // the counter blocks up to the last slot in use (the host reads no other)
    for (int i = 0; i < kMaxSel; ++i)
      if (slots_[i].used) hi = i + 1;
    pub_n_ = launched_ && pub_host_ && !profile_ && !capturing_stream() ? C_COUNT * hi : 0;
    if (launched_)
      launch(K_OTHER, k_tick_end<T>, 1, 256, jobs_dev_, ctr_dev_, hi, seq_dev_,
             pub_n_ ? pub_host_ : (volatile unsigned long long*)nullptr);
    if (pub_n_) {
      ++seq_next_;
      seq_known_ = false;
    }
    recording_ = false;
    if (rc != EXTREMZ_OK) return rc;
    if (graph && !pending_.empty()) EZ_RUN(run_recorded());
    if (!launched_) return EXTREMZ_OK;
    EZ_CHECK(cudaGetLastError());
    if (!pub_n_)
      EZ_CHECK(cudaMemcpyAsync(ctr_host_, ctr_dev_, sizeof(int) * C_COUNT * (size_t)hi,
                               cudaMemcpyDeviceToHost, st_));
    return EXTREMZ_OK;
  }

  // Second half: wait for the counters, then every job's branches.
  int tick_complete() {
    if (!issued_) return EXTREMZ_OK;
    issued_ = false;
    if (launched_) {
      if (pub_n_) EZ_RUN(await_published());
      else EZ_CHECK(cudaStreamSynchronize(st_));
      fold_timings();
    }
    for (int i = 0; i < kMaxSel; ++i) {
      JobHost<T>& j = slots_[i];
      if (!j.used || j.pc == PC_DONE) continue;
      flush_pending(i);
      if (h(i, C_ERROR)) {
        finish(i, EXTREMZ_DEVICE_TIMEOUT);
        continue;
      }
      if (j.waiting) {
        j.waiting = false;
        EZ_RUN(decide(i));
      }
    }
    return EXTREMZ_OK;
  }

  bool capturing_stream() const {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st_, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone)
      return false;
    cudaGetLastError();
    return true;
  }

  // Takes over the published counters as they arrive.  The stream is asked now
  // and then: an error ends the wait, and once all its work is done they are
  // there.  A process that asked for blocking or yielding waits gets them: there
  // the counters are read once the stream is done.
  int await_published() {
    bool all_done = false;
    if (!wait_known_) {  // asked at the first wait of a call, while the device works
      unsigned flags = 0;
      if (cudaGetDeviceFlags(&flags) != cudaSuccess) cudaGetLastError();
      flags &= cudaDeviceScheduleMask;
      spin_ = flags != cudaDeviceScheduleBlockingSync && flags != cudaDeviceScheduleYield;
      wait_known_ = true;
    }
    if (!spin_) {
      EZ_CHECK(cudaStreamSynchronize(st_));
      all_done = true;
    }
    for (int i = 0, spins = 0; i < pub_n_;) {
      const unsigned long long p = pub_host_[i];
      if ((unsigned)(p >> 32) == seq_next_) {
        ctr_host_[i++] = (int)(unsigned)p;
        continue;
      }
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
      if (++spins < 4000) continue;
      spins = 0;
      if (all_done) {
        last_cuda_error() = cudaErrorUnknown;
        return EXTREMZ_CUDA_ERR;
      }
      const cudaError_t e = cudaStreamQuery(st_);
      if (e == cudaErrorNotReady) continue;
      EZ_CHECK(e);
      EZ_CHECK(cudaStreamSynchronize(st_));
      all_done = true;
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    seq_known_ = true;
    return EXTREMZ_OK;
  }

  // Per-class timing of the launches since set_profile(true, ...).
  void collect_profile(extremz_report* rep) {
    if (!recs_.empty()) {
      cudaStreamSynchronize(st_);
      fold_timings();
    }
    if (rep)
      for (int c = 0; c < K_NUM; ++c) {
        rep->prof_ms[c] += prof_ms_[c];
        rep->prof_launches[c] += prof_n_[c];
      }
    reset_timings();
  }
  void drop_profile_events() {
    for (const Rec& r : recs_)
      if (r.owned) {
        pool_.push_back(r.a);
        pool_.push_back(r.b);
      }
    recs_.clear();
    reset_timings();
    for (cudaEvent_t e : pool_) cudaEventDestroy(e);
    pool_.clear();
  }

 private:
  cudaStream_t st_;
  struct Rec { int cls; cudaEvent_t a, b; bool owned; };
  // Tick graphs (see tick_issue).
  bool graphs_on_ = true, recording_ = false, capturing_ = false;
  std::string sig_;
  // A recorded launch and its branch: the phases of a tick work on different
  // jobs, so those of different branches run side by side (branch_of), each
  // branch on a stream of its own between a fork and a join; -1 comes after the
  // join.
  struct Launch {
    int branch;
    std::function<void(cudaStream_t)> go;
  };
  std::vector<Launch> pending_;
  int branch_ = 0;
  // Timed launches of the tick being recorded: class, and the event pair the
  // launch records around itself (filled in just before the launches run).
  std::vector<Rec> pending_timed_;
  struct GraphEntry {
    cudaGraphExec_t exec = nullptr;
    unsigned long long last = 0;
    std::vector<Rec> timed;  // events recorded by the graph's timed launches
  };
  std::unordered_map<std::string, GraphEntry> graphs_;
  std::unordered_map<std::string, int> seen_;
  unsigned long long graph_clock_ = 0;
  long long graph_replays_ = 0, graph_captures_ = 0;
  static constexpr size_t kMaxGraphs = 256;
  static constexpr unsigned long long kGraphRest = 8192;  // ticks
  // A signature is captured at its third sighting: ticks of a single
  // correction repeat many times, while a batch's changing selections often
  // repeat once or twice, where a capture would not pay for itself.
  static constexpr int kCaptureAt = 3;
  cudaStream_t cap_ = nullptr;  // capture stream
  cudaStream_t side_[kBranches] = {};
  cudaEvent_t fork_ = nullptr, join_[kBranches] = {};
  bool branches_ok_ = false;
  cudaMemPool_t pool_mem_ = nullptr;
  bool ready_ = false, borrowed_ = false, issued_ = false, launched_ = false;
  long long tick_id_ = 0;
  int grid_ = 1184;  // grid of the grid-stride kernels for the phase being issued
  int sms_ = 148;
  DeviceTables tb_{};
  Job<T>* jobs_dev_ = nullptr;
  int* ctr_dev_ = nullptr;
  int* ctr_host_ = nullptr;
  // Published counters (k_tick_end): the mapped host copy, a counter in the low
  // half and its tick's number in the high half of each entry; the number of the
  // last tick on the device, and of the one the host waits for.  The borrowed
  // engine, whose host copy is not mapped, copies instead.
  volatile unsigned long long* pub_host_ = nullptr;
  unsigned* seq_dev_ = nullptr;
  unsigned seq_next_ = 0;
  bool seq_known_ = true;
  bool wait_known_ = false, spin_ = true;  // wait for the published counters by reading them
  int pub_n_ = 0;           // counters published by this tick; 0: copied
  int static_ctr_host_[C_COUNT * kMaxSel];
  std::vector<JobHost<T>> slots_;
  long long launches_ = 0;
  bool profile_ = false;
  int profile_mask_ = 0;
  // A timed launch: events around it.  Events of a launch inside a captured
  // tick graph belong to the graph (recorded again at every replay, read after
  // the tick's synchronisation); the others return to the pool.
  std::vector<Rec> recs_;
  float prof_ms_[K_NUM] = {};
  int prof_n_[K_NUM] = {};
  void fold_timings() {
    for (const Rec& r : recs_) {
      float ms = 0.f;
      if (cudaEventElapsedTime(&ms, r.a, r.b) != cudaSuccess) {
        cudaGetLastError();
        ms = 0.f;
      }
      prof_ms_[r.cls] += ms;
      prof_n_[r.cls] += 1;
      if (r.owned) {
        pool_.push_back(r.a);
        pool_.push_back(r.b);
      }
    }
    recs_.clear();
  }
  void reset_timings() {
    for (int c = 0; c < K_NUM; ++c) {
      prof_ms_[c] = 0.f;
      prof_n_[c] = 0;
    }
  }
  std::vector<cudaEvent_t> pool_;

  int h(int slot, int c) const { return ctr_host_[(size_t)slot * C_COUNT + c]; }

  cudaEvent_t event() {
    if (!pool_.empty()) {
      cudaEvent_t e = pool_.back();
      pool_.pop_back();
      return e;
    }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
  }

  template <class A>
  void sig_append(const A& a) {
    sig_.append(reinterpret_cast<const char*>(&a), sizeof(A));
  }
  // A job selection by its used part (kernels read no entry past n): the
  // signature of a one-job tick stays a few hundred bytes to hash.
  void sig_append(const Sel& s) {
    sig_.append(reinterpret_cast<const char*>(&s.n), sizeof(int));
    sig_.append(reinterpret_cast<const char*>(s.idx), sizeof(int) * (size_t)s.n);
    sig_.append(reinterpret_cast<const char*>(s.off), sizeof(int) * (size_t)(s.n + 1));
  }

  template <class... KArgs, class... Args>
  void launch(int cls, void (*kern)(KArgs...), dim3 grid, dim3 block, Args... args) {
    const bool timed = profile_ && (profile_mask_ == 0 || (profile_mask_ >> cls & 1));
    if (recording_) {  // tick graphs: record, launch later as one graph
      sig_append(reinterpret_cast<const void*>(kern));
      sig_append(grid);
      sig_append(block);
      sig_append(branch_);
      (sig_append(args), ...);
      if (timed) {
        const size_t k = pending_timed_.size();
        pending_timed_.push_back({cls, nullptr, nullptr, false});
        pending_.push_back({branch_, [=](cudaStream_t s) {
          // In a capture the events become event-record nodes of the graph.
          const Rec& r = pending_timed_[k];
          const unsigned fl = capturing_ ? cudaEventRecordExternal : cudaEventRecordDefault;
          if (r.a) cudaEventRecordWithFlags(r.a, s, fl);
          kern<<<grid, block, 0, s>>>(args...);
          if (r.b) cudaEventRecordWithFlags(r.b, s, fl);
        }});
      } else {
        pending_.push_back({branch_, [=](cudaStream_t s) { kern<<<grid, block, 0, s>>>(args...); }});
      }
      ++launches_;
      return;
    }
    cudaEvent_t a = nullptr, b = nullptr;
    if (timed) {
      a = event();
      b = event();
      cudaEventRecord(a, st_);
    }
    kern<<<grid, block, 0, st_>>>(args...);
    ++launches_;
    if (timed) {
      cudaEventRecord(b, st_);
      recs_.push_back({cls, a, b, true});
    }
  }

  // Event pairs for the recorded tick's timed launches, from the pool.
  void arm_timed() {
    for (Rec& r : pending_timed_) {
      r.a = event();
      r.b = event();
      r.owned = true;
    }
  }

  // The recorded launches on stream `main`: its branches side by side when there
  // are several (fork), else in order.
  void run_pending(cudaStream_t main, bool fork) {
    int used = 0, first = -1;
    for (const Launch& l : pending_)
      if (l.branch >= 0 && !(used >> l.branch & 1)) {
        used |= 1 << l.branch;
        if (first < 0) first = l.branch;
      }
    cudaStream_t on[kBranches];
    for (int b = 0; b < kBranches; ++b) on[b] = main;
    const int rest = used & ~(1 << std::max(first, 0));
    fork = fork && rest && ensure_branches() && cudaEventRecord(fork_, main) == cudaSuccess;
    if (fork)
      for (int b = 0; b < kBranches; ++b)
        if (rest >> b & 1) {
          on[b] = side_[b];
          cudaStreamWaitEvent(side_[b], fork_, 0);
        }
    for (const Launch& l : pending_)
      if (l.branch >= 0) l.go(on[l.branch]);
    if (fork)
      for (int b = 0; b < kBranches; ++b)
        if (rest >> b & 1) {
          cudaEventRecord(join_[b], side_[b]);
          cudaStreamWaitEvent(main, join_[b], 0);
        }
    for (const Launch& l : pending_)
      if (l.branch < 0) l.go(main);
  }

  // The branches' streams (of the engine stream's priority) and events, made
  // when a tick first has two branches.
  bool ensure_branches() {
    if (fork_) return branches_ok_;
    int prio = 0;
    branches_ok_ = cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming) == cudaSuccess &&
                   cudaStreamGetPriority(st_, &prio) == cudaSuccess;
    for (int b = 0; b < kBranches && branches_ok_; ++b)
      branches_ok_ =
          cudaStreamCreateWithPriority(&side_[b], cudaStreamNonBlocking, prio) == cudaSuccess &&
          cudaEventCreateWithFlags(&join_[b], cudaEventDisableTiming) == cudaSuccess;
    if (!branches_ok_) cudaGetLastError();
    return branches_ok_;
  }

  void run_direct(bool timing = true) {
    if (timing) arm_timed();
    run_pending(st_, timing && pending_timed_.empty());
    pending_.clear();
    for (const Rec& r : pending_timed_)
      if (r.a) recs_.push_back(r);
    pending_timed_.clear();
  }

  // (cudaEventDestroy of an event still pending releases it once it completes.)
  static void release_graph_events(GraphEntry& e) {
    for (const Rec& r : e.timed) {
      cudaEventDestroy(r.a);
      cudaEventDestroy(r.b);
    }
    e.timed.clear();
  }

  void drop_graphs() {
    for (auto& kv : graphs_) {
      if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
      release_graph_events(kv.second);
    }
    graphs_.clear();
    seen_.clear();
    if (cap_) cudaStreamDestroy(cap_);
    cap_ = nullptr;
    for (int b = 0; b < kBranches; ++b) {
      if (side_[b]) cudaStreamDestroy(side_[b]);
      if (join_[b]) cudaEventDestroy(join_[b]);
      side_[b] = nullptr;
      join_[b] = nullptr;
    }
    if (fork_) cudaEventDestroy(fork_);
    fork_ = nullptr;
  }

  // Launches the recorded tick: replays its graph, captures it on the third
  // sighting of its signature, or launches directly.
  int run_recorded() {
    ++graph_clock_;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st_, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
      cudaGetLastError();  // the caller is capturing this stream: launch into it directly
      run_direct(false);   // (untimed: the events would not have run when read)
      return EXTREMZ_OK;
    }
    auto it = graphs_.find(sig_);
    if (it != graphs_.end()) {
      it->second.last = graph_clock_;
      pending_.clear();
      pending_timed_.clear();
      ++graph_replays_;
      EZ_CHECK(cudaGraphLaunch(it->second.exec, st_));
      for (Rec r : it->second.timed) {
        r.owned = false;
        recs_.push_back(r);
      }
      return EXTREMZ_OK;
    }
    if (seen_.size() > 4 * kMaxGraphs) seen_.clear();
    if (++seen_[sig_] < kCaptureAt) {
      run_direct();
      return EXTREMZ_OK;
    }
    if (graphs_.size() >= kMaxGraphs) {
      // The least recently used one makes room only once it has rested for a
      // while: a batch of many fields has more distinct ticks than the cache
      // holds, and a pass over them would capture each in place of one that the
      // next pass wants.
      auto old = graphs_.begin();
      for (auto g = graphs_.begin(); g != graphs_.end(); ++g)
        if (g->second.last < old->second.last) old = g;
      if (graph_clock_ - old->second.last < kGraphRest) {
        run_direct();
        return EXTREMZ_OK;
      }
      cudaGraphExecDestroy(old->second.exec);
      release_graph_events(old->second);
      graphs_.erase(old);
    }
    // Captured on a private stream (the caller's may be the legacy stream,
    // which cannot be captured), launched on the caller's.
    if (!cap_ && cudaStreamCreateWithFlags(&cap_, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      graphs_on_ = false;
      run_direct();
      return EXTREMZ_OK;
    }
    cudaGraph_t g = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (cudaStreamBeginCapture(cap_, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      cudaGetLastError();
      graphs_on_ = false;
      run_direct();
      return EXTREMZ_OK;
    }
    arm_timed();
    capturing_ = true;
    run_pending(cap_, pending_timed_.empty());
    capturing_ = false;
    const cudaError_t ec = cudaStreamEndCapture(cap_, &g);
    if (ec != cudaSuccess || !g || cudaGraphInstantiate(&exec, g, 0) != cudaSuccess) {
      cudaGetLastError();
      if (g) cudaGraphDestroy(g);
      graphs_on_ = false;  // capture unavailable here: launch directly from now on
      for (const Rec& r : pending_timed_) {
        pool_.push_back(r.a);
        pool_.push_back(r.b);
      }
      run_direct();
      return EXTREMZ_OK;
    }
    cudaGraphDestroy(g);
    pending_.clear();
    GraphEntry ge{exec, graph_clock_};
    ge.timed = pending_timed_;
    pending_timed_.clear();
    ++graph_captures_;
    EZ_CHECK(cudaGraphLaunch(exec, st_));
    for (Rec r : ge.timed) {
      r.owned = false;
      recs_.push_back(r);
    }
    graphs_[sig_] = std::move(ge);
    return EXTREMZ_OK;
  }

  void free_job(JobHost<T>& j) {
    if (j.used && j.own_arena && j.arena.base) cudaFreeAsync(j.arena.base, st_);
    if (j.used && j.own_arena2 && j.arena2.base) cudaFreeAsync(j.arena2.base, st_);
    j = JobHost<T>();
  }

  // The per-critical-point part of a job's workspace: exact size from the
  // counts, or the rest of borrowed storage.
  int take_cp_storage(JobHost<T>& jh, int ns2, int ns1, int nmax, int nmin, int e2, int e1) {
    if (!jh.own_arena) return EXTREMZ_OK;  // borrowed: carve from the same arena
    const long long need = (jh.p.flags & kFlagAnalysis)
                               ? job_bytes_lists(ns2, ns1, nmax, nmin)
                               : job_bytes_cps(ns2, ns1, nmax, nmin, e2, e1, sizeof(K));
    void* base = nullptr;
    const cudaError_t e = pool_mem_ ? cudaMallocFromPoolAsync(&base, (size_t)need, pool_mem_, st_)
                                    : cudaMallocAsync(&base, (size_t)need, st_);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return EXTREMZ_OOM;
    }
    jh.arena2.base = static_cast<char*>(base);
    jh.arena2.cap = (size_t)need;
    jh.arena2.used = 0;
    jh.arena2.fixed = true;
    jh.own_arena2 = true;
    return EXTREMZ_OK;
  }

  Sel make_sel(const std::vector<int>& slots, bool tiles) const {
    Sel s;
    std::memset(&s, 0, sizeof(s));
    s.n = (int)slots.size();
    int off = 0;
    for (int k = 0; k < s.n; ++k) {
      s.idx[k] = slots[k];
      s.off[k] = off;
      if (tiles) off += slots_[slots[k]].ntiles;
    }
    s.off[s.n] = off;
    return s;
  }

  // Block spans for the grid-stride kernels: a block per 1024 voxels of each
  // job, scaled down to the grid of the phase (the SMs times the blocks-per-SM
  // knob; twice that when several jobs share it), at least one block each.
  Sel make_span(const std::vector<int>& slots) const {
    Sel s;
    std::memset(&s, 0, sizeof(s));
    s.n = (int)slots.size();
    const long long budget = s.n > 1 ? 2ll * grid_ : grid_;
    long long want = 0;
    for (int i : slots) want += slots_[i].nb;
    int off = 0;
    for (int k = 0; k < s.n; ++k) {
      const long long nb = slots_[slots[k]].nb;
      s.idx[k] = slots[k];
      s.off[k] = off;
      off += (int)std::max(1ll, want <= budget ? nb : nb * budget / want);
    }
    s.off[s.n] = off;
    return s;
  }
  static int blocks(const Sel& s) { return s.off[s.n]; }

  // ------------------------------------------------------------- phases --
  int run_phase(int ph, const std::vector<int>& sel) {
    int bps = 1;  // jobs share launches: the largest knob of the selection
    for (int i : sel) bps = std::max(bps, slots_[i].blocks_per_sm);
    grid_ = sms_ * bps;
    if (ph == PC_CL_ROUND || ph == PC_RLOOPS || ph == PC_SLOOPS_J || ph == PC_SADDLE_J ||
        ph == PC_FINAL_JOIN)
      for (int i : sel) edits(i);  // phases that apply edits
    const Sel s = make_span(sel);
    const int nb = blocks(s);
    const Job<T>* jobs = jobs_dev_;
    switch (ph) {
      case PC_SETUP_A: {
        const Sel st = make_sel(sel, true);
        launch(K_SETUP, k_direction<T, false>, st.off[st.n], 256, jobs, st);
        launch(K_SETUP, k_jump2<T, false>, nb, 256, jobs, s);
        for (int i : sel) {
          JobHost<T>& j = slots_[i];
          j.waiting = true;
          if (j.p.flags & kFlagLabels) continue;
          launch(K_OTHER, k_cp_count, (j.nb + kCpWarps - 1) / kCpWarps, 32 * kCpWarps,
                 (const int8_t*)j.J.otype, (const uint16_t*)j.J.olm, j.J.dim, j.nb, j.bcount);
          EZ_RUN(scan_counts(j.bcount, j.nb, 6, j.J.ctr + C_NS2, j.chunk));
        }
        return EXTREMZ_OK;
      }
      case PC_SETUP_B:
        for (int i : sel) {
          const int rc = setup_b(i);
          if (rc == EXTREMZ_OOM) {  // this job ends; the others go on
            finish(i, EXTREMZ_OOM);
            continue;
          }
          if (rc != EXTREMZ_OK) return rc;
          if (slots_[i].p.flags & kFlagAnalysis) finish(i, EXTREMZ_OK);
          else slots_[i].pc = PC_CL_DETECT;
        }
        return EXTREMZ_OK;
      case PC_CL_DETECT:
      case PC_FINAL_DETECT: {
        // No value changed since the last detection: its list and counts stand.
        std::vector<int> busy;
        for (int i : sel) {
          const JobHost<T>& j = slots_[i];
          if (!j.dense_done || j.applied_tick == tick_id_ || h(i, C_DIRTY) > 0) busy.push_back(i);
        }
        detect(busy);
        for (int i : sel) slots_[i].waiting = true;
        return EXTREMZ_OK;
      }
      case PC_CL_ROUND:
        launch(K_PROPOSE, k_propose_cp<T>, nb, 256, jobs, s);
        launch(K_APPLY, k_apply<T>, nb, 256, jobs, s);
        detect(sel);
        for (int i : sel) slots_[i].waiting = true;
        return EXTREMZ_OK;
      case PC_RLOOPS:
        launch(K_FIXPATH, k_fixpath<T>, nb, 256, jobs, s);
        launch(K_APPLY, k_apply<T>, nb, 256, jobs, s);
        for (int i : sel) slots_[i].pc = PC_MANIFOLD;
        return EXTREMZ_OK;
      case PC_MANIFOLD: {
        // Jobs known on the host to have no value change since their last
        // manifold round began (no edit in the counters of the last tick, none
        // issued in this one) launch nothing; their kernels would return at
        // once.  The others run the round (whose kernels check again on the
        // device).
        std::vector<int> busy;
        for (int i : sel) {
          JobHost<T>& j = slots_[i];
          const bool known_clean =
              j.manifold_rounds > 0 && j.applied_tick != tick_id_ && h(i, C_CHANGED) == 0;
          if (known_clean) {
            j.reused += 1;
          } else {
            busy.push_back(i);
            j.wim_seen = j.wis_seen = false;
          }
        }
        if (!busy.empty()) {
          // Steepest pointers: every tile in a job's first round, one block
          // per tile; in later rounds the tiles that changed, as k_apply
          // listed them, taken by a fixed grid (a launch of one block per tile
          // of the field costs more than the few changed tiles).
          std::vector<int> fresh, later;
          for (int i : busy) (slots_[i].manifold_rounds == 0 ? fresh : later).push_back(i);
          if (!fresh.empty()) {
            const Sel ft = make_sel(fresh, true);
            launch(K_DIRECTION_FIRST, k_direction<T, true>, ft.off[ft.n], 256, jobs, ft);
          }
          if (!later.empty()) {
            const Sel lt = tile_span(later);
            launch(K_DIRECTION, k_direction_list<T>, blocks(lt), 256, jobs, lt);
            std::vector<int> large;
            for (int i : later)
              if (slots_[i].J.dim.N >= kTouchMin) large.push_back(i);
            if (!large.empty()) {
              const Sel qt = tile_span(large);
              launch(K_JUMP, k_touched_tiles<T>, blocks(qt), 256, jobs, qt);
            }
          }
          if (!fresh.empty()) {
            const Sel fs = make_span(fresh);
            launch(K_JUMP_FIRST, k_jump2<T, true, false>, blocks(fs), 256, jobs, fs);
          }
          if (!later.empty()) {
            const Sel ls = make_span(later);
            launch(K_JUMP, k_jump2<T, true, true>, blocks(ls), 256, jobs, ls);
          }
          // The first round of a correction runs right after a detection without
          // mismatch; a census's may not.
          std::vector<int> first, other;
          for (int i : busy)
            (slots_[i].manifold_rounds == 0 && !(slots_[i].p.flags & kFlagCensus) && !h(i, C_NAN)
                 ? first
                 : other)
                .push_back(i);
          if (!first.empty()) {
            const Sel fs = make_span(first);
            launch(K_ROWS, k_saddle_first<T>, blocks(fs), 256, jobs, fs);
          }
          if (!other.empty()) {
            const Sel os = make_span(other);
            launch(K_ROWS, k_saddle_pass<T>, blocks(os), 256, jobs, os);
          }
          // Lockstep jobs: the fourteen steps in one cluster per job when the
          // job's previous round had short candidate lists (the counts of
          // that round are still in the host copy of its counters), or before
          // its first round when it has few saddles, else one grid launch per
          // step.  Either is exact for any list length.
          std::vector<int> vote, lock_small, lock_large;
          for (int i : busy) {
            if (!slots_[i].J.wn_lockstep) {
              vote.push_back(i);
              continue;
            }
            const bool small = slots_[i].manifold_rounds > 0
                                   ? h(i, C_CAND) + h(i, C_CANDJ) <= kWnClusterMax
                                   : h(i, C_NS2) + h(i, C_NS1) <= kWnClusterFirst;
            (small ? lock_small : lock_large).push_back(i);
          }
          if (!vote.empty()) {
            const Sel vs = make_span(vote);
            wn_rounds<true>(vs);  // its completion brings in the join side's list
            wn_rounds<false>(vs);
          }
          if (!lock_small.empty()) {
            const Sel ss = make_sel(lock_small, false);
            launch(K_WRONG_NBR, k_wn_steps_block<T>, ss.n * kWnCluster, 1024, jobs, ss);
          }
          if (!lock_large.empty()) {
            const Sel sl = make_span(lock_large);
            for (int d = 0; d < kNumDirs; ++d)
              launch(K_WRONG_NBR, k_wn_step<T>, blocks(sl), 256, jobs, sl, d);
          }
        }
        for (int i : sel) {
          slots_[i].manifold_rounds++;
          slots_[i].waiting = true;
        }
        return EXTREMZ_OK;
      }
      case PC_SLOOPS: {
        // A scan of this very state that found nothing proposes nothing again.
        std::vector<int> busy;
        for (int i : sel)
          if (!(still(i, slots_[i].wim_seen) && h(i, C_WMC) == 0 && h(i, C_WMC2) == 0))
            busy.push_back(i);
        if (!busy.empty()) {
          const Sel bs = make_span(busy);
          launch(K_OTHER, k_wim_scan<T, true>, blocks(bs), 256, jobs, bs);
          launch(K_OTHER, k_wim_collect<T, true>, blocks(bs), 256, jobs, bs, 1);
          launch(K_APPLY, k_apply<T>, blocks(bs), 256, jobs, bs);
        }
        for (int i : busy) edits(i).wim_seen = true;
        for (int i : sel) slots_[i].waiting = true;
        return EXTREMZ_OK;
      }
      case PC_SADDLE: {
        std::vector<int> busy;
        for (int i : sel)
          if (!(still(i, slots_[i].wis_seen) && h(i, C_WSC) == 0)) busy.push_back(i);
        if (!busy.empty()) {
          const Sel bs = make_span(busy);
          wis_scan<true>(bs, 1);
          launch(K_APPLY, k_apply<T>, blocks(bs), 256, jobs, bs);
        }
        for (int i : busy) edits(i).wis_seen = true;
        for (int i : sel) {
          slots_[i].pending.push_back(PH_SADDLE);
          slots_[i].pc = joinb(slots_[i]);
        }
        return EXTREMZ_OK;
      }
      case PC_SLOOPS_J:
        launch(K_OTHER, k_wim_scan<T, false>, nb, 256, jobs, s);
        launch(K_OTHER, k_wim_collect<T, false>, nb, 256, jobs, s, 1);
        launch(K_OTHER, k_wim_min2_scan<T>, nb, 256, jobs, s);
        launch(K_OTHER, k_wim_min2_collect<T>, nb, 256, jobs, s);
        launch(K_APPLY, k_apply<T>, nb, 256, jobs, s);
        for (int i : sel) slots_[i].waiting = true;
        return EXTREMZ_OK;
      case PC_SADDLE_J:
      case PC_FINAL_JOIN: {
        std::vector<int> lists, once;
        for (int i : sel) (slots_[i].J.join_rows ? lists : once).push_back(i);
        if (!lists.empty()) wis_scan<false>(make_span(lists), 1);
        if (!once.empty()) {
          const Sel os = make_span(once);
          launch(K_OTHER, k_join_keys<T>, blocks(os), 256, jobs, os);
          launch(K_OTHER, k_join_ids<T>, blocks(os), 256, jobs, os);
          launch(K_OTHER, k_join_scan<T>, blocks(os), 256, jobs, os);
          launch(K_OTHER, k_wis_collect<T, false>, blocks(os), 256, jobs, os, 1);
        }
        launch(K_APPLY, k_apply<T>, nb, 256, jobs, s);
        for (int i : sel) {
          slots_[i].pending.push_back(PH_SADDLE_JOIN);
          if (ph == PC_SADDLE_J) slots_[i].pc = endb(slots_[i]);
          else slots_[i].waiting = true;
        }
        return EXTREMZ_OK;
      }
      case PC_PRE_END:
        for (int i : sel) slots_[i].waiting = true;
        return EXTREMZ_OK;
      case PC_DET3: {
        std::vector<int> busy;
        for (int i : sel)
          if (!still(i, slots_[i].wim_seen && slots_[i].wis_seen)) busy.push_back(i);
        if (!busy.empty()) {
          const Sel bs = make_span(busy);
          launch(K_OTHER, k_wim_scan<T, true>, blocks(bs), 256, jobs, bs);
          launch(K_OTHER, k_wim_collect<T, true>, blocks(bs), 256, jobs, bs, 0);
          wis_scan<true>(bs, 0);
        }
        for (int i : busy) slots_[i].wim_seen = slots_[i].wis_seen = true;
        for (int i : sel) {
          slots_[i].pending.push_back(PH_DETECT3);
          slots_[i].pc = (slots_[i].p.flags & kFlagCensus) ? PC_DET3J : join3(slots_[i]);
        }
        return EXTREMZ_OK;
      }
      case PC_DET3J:
        launch(K_OTHER, k_wim_scan<T, false>, nb, 256, jobs, s);
        launch(K_OTHER, k_wim_collect<T, false>, nb, 256, jobs, s, 0);
        wis_scan<false>(s, 0);
        for (int i : sel) slots_[i].pc = PC_FINAL_DETECT;
        return EXTREMZ_OK;
      default:
        return EXTREMZ_OK;
    }
  }

  JobHost<T>& edits(int i) {
    slots_[i].applied_tick = tick_id_;
    return slots_[i];
  }
  // seen: a scan ran since job i's last computed manifold round.  True when no
  // value has changed since that round, so that the scan's counts, which are in
  // the host's copy, are those of the present field.
  bool still(int i, bool seen) const {
    return seen && slots_[i].applied_tick != tick_id_ && h(i, C_CHANGED) == 0;
  }

  // Blocks over a selection's listed tiles: a job's share of four per SM goes
  // by its tiles.
  Sel tile_span(const std::vector<int>& slots) const {
    Sel s = make_sel(slots, true);
    const long long total = s.off[s.n], budget = 4ll * sms_;
    int off = 0;
    for (int k = 0; k < s.n; ++k) {
      const long long nt = slots_[s.idx[k]].ntiles;
      s.off[k] = off;
      off += (int)std::max(1ll, total <= budget ? nt : nt * budget / total);
    }
    s.off[s.n] = off;
    return s;
  }

  // The incremental wrong-saddle scan of one side; fix: with its proposals.
  template <bool kMax>
  void wis_scan(const Sel& s, int fix) {
    const Job<T>* jobs = jobs_dev_;
    launch(K_OTHER, k_wis_mark<T, kMax>, blocks(s), 256, jobs, s);
    launch(K_OTHER, k_wis_update<T, kMax>, blocks(s), 256, jobs, s);
    launch(K_OTHER, k_wis_long<T, kMax>, blocks(s), 256, jobs, s);
    launch(K_OTHER, k_wis_collect<T, kMax>, blocks(s), 256, jobs, s, fix);
  }

  // Mismatch detection: dense the first time a job detects, then incremental
  // over the neighbourhoods of the vertices changed since.
  void detect(const std::vector<int>& sel) {
    if (sel.empty()) return;
    std::vector<int> dense, incr;
    for (int i : sel) (slots_[i].dense_done ? incr : dense).push_back(i);
    if (!dense.empty()) {
      const Sel st = make_sel(dense, true);
      launch(K_DETECT, k_classify<T>, st.off[st.n], 256, (const Job<T>*)jobs_dev_, st);
      for (int i : dense) slots_[i].dense_done = true;
    }
    if (!incr.empty()) {
      const Sel s = make_span(incr);
      launch(K_DETECT, k_redetect<T>, blocks(s), 256, (const Job<T>*)jobs_dev_, s);
    }
  }

  // Three grid-wide arbitration rounds and the per-job completion rounds of
  // the candidate list being resolved (one side).
  template <bool kSplit>
  void wn_rounds(const Sel& s) {
    const Job<T>* jobs = jobs_dev_;
    for (int r = 0; r < kWnGridRounds; ++r) {
      launch(K_WRONG_NBR, k_wn_vote<T, kSplit>, blocks(s), 256, jobs, s, r);
      launch(K_WRONG_NBR, k_wn_commit<T, kSplit>, blocks(s), 256, jobs, s, r);
    }
    launch(K_WRONG_NBR, k_wn_resolve<T, kSplit>, s.n, 1024, jobs_dev_, s);
  }

  // Exclusive scan of nl lists of n counts each (list l at c + l * n), the
  // list totals into totals[0 .. nl), a second copy of the (one) scanned list
  // into cursor; chunk holds nl * ceil(n / 1024) sums.  Up to one pass of a
  // block (32 Ki counts) a block per list does it all.
  int scan_counts(int* c, int n, int nl, int* totals, int* chunk, int* cursor = nullptr) {
    if (n <= 32 * 1024) {
      launch(K_OTHER, k_scan_lists, nl, 1024, c, n, totals, cursor);
      return EXTREMZ_OK;
    }
    const int nc = (n + 1023) / 1024;
    launch(K_OTHER, k_chunk_sums, dim3(nc, nl), 1024, (const int*)c, n, chunk);
    launch(K_OTHER, k_scan_lists, nl, 1024, chunk, nc, totals, (int*)nullptr);
    launch(K_OTHER, k_chunk_scan, dim3(nc, nl), 1024, c, n, (const int*)chunk, cursor);
    return EXTREMZ_OK;
  }

  // Arrays to fill before a job's first round, in one launch (k_fill_many).
  struct Fills {
    FillList f{};
    template <class P>
    void add(P* at, long long count, unsigned long long value) {
      if (count <= 0) return;
      const long long pieces = (count * (long long)sizeof(P) + 15) / 16;
      f.at[f.n] = reinterpret_cast<ulonglong2*>(at);
      f.end[f.n] = (f.n ? f.end[f.n - 1] : 0) + pieces;
      f.value[f.n++] = value;
    }
  };
  void fill(const Fills& fl) {
    if (fl.f.n == 0) return;
    const long long pieces = fl.f.end[fl.f.n - 1];
    launch(K_OTHER, k_fill_many, (int)std::min<long long>(grid_, (pieces + 255) / 256), 256, fl.f);
  }
  // A 4-byte value in both halves of the pattern.
  static constexpr unsigned long long twice(unsigned v) {
    return (unsigned long long)v << 32 | v;
  }
  static constexpr unsigned long long key_pattern(K k) {
    return sizeof(K) == 8 ? (unsigned long long)k : twice((unsigned)k);
  }

  int setup_b(int slot) {
    JobHost<T>& jh = slots_[slot];
    Job<T>& J = jh.J;
    const int N = J.dim.N;
    const int ns2 = h(slot, C_NS2), ns1 = h(slot, C_NS1), nmax = h(slot, C_NMAX),
              nmin = h(slot, C_NMIN), e2 = h(slot, C_E2), e1 = h(slot, C_E1);
    EZ_RUN(take_cp_storage(jh, ns2, ns1, nmax, nmin, e2, e1));
    Arena& A = jh.own_arena2 ? jh.arena2 : jh.arena;
    J.sad2 = A.take<int>(ns2);
    J.sad1 = A.take<int>(ns1);
    J.maxima = A.take<int>(nmax);
    J.minima = A.take<int>(nmin);
    if (!J.minima) return EXTREMZ_OOM;
    // Without NaNs every path ends at an extremum, so only their entries are read.
    if (h(slot, C_NAN)) launch(K_OTHER, k_fill<int>, grid_, 256, J.ext, 0, (long long)N);
    launch(K_OTHER, k_cp_write, (jh.nb + kCpWarps - 1) / kCpWarps, 32 * kCpWarps,
           (const int8_t*)J.otype, N, jh.nb, (const int*)jh.bcount,
           J.sad2, J.sad1, J.maxima, J.minima, J.ext);
    // The lists and the extremum index are all that an analysis needs.
    if (jh.p.flags & kFlagAnalysis) return EXTREMZ_OK;
    J.smask2 = A.take<uint16_t>(ns2);
    J.orow2 = A.take<int>((long long)ns2 * kRowStride);
    J.orm2 = A.take<int4>(ns2);
    J.oend2 = A.take<int4>(ns2);
    J.drow2 = A.take<int>((long long)ns2 * 2);
    J.ocnt2 = A.take<uint8_t>(ns2);
    J.orow1 = A.take<int>((long long)ns1 * kRowStride);
    J.orm1 = A.take<int4>(ns1);
    J.oend1 = A.take<int4>(ns1);
    J.drow1 = A.take<int>((long long)ns1 * 2);
    J.ocnt1 = A.take<uint8_t>(ns1);
    J.has2 = A.take<uint8_t>(ns2);
    J.has1 = A.take<uint8_t>(ns1);
    J.bad2 = A.take<uint8_t>(ns2);
    J.bad1 = A.take<uint8_t>(ns1);
    J.largest = A.take<int>(nmax);
    J.first1 = A.take<int>(nmax);
    J.flag2 = A.take<int>(nmax);
    J.first_s = A.take<int>(nmax);
    J.smallest = A.take<int>(nmin);
    J.first_min1 = A.take<int>(nmin);
    J.flag_min2 = A.take<int>(nmin);
    J.first_sj = A.take<int>(nmin);
    const int ne = std::max(nmax, nmin);
    J.ext_key = A.take<K>(ne);
    J.ext_id = A.take<int>(ne);
    jh.checksum = A.take<unsigned long long>(8);
    J.moff2 = A.take<int>(nmax + 1);
    J.ment2 = A.take<int>(e2);
    J.wstamp2 = A.take<int>(nmax);
    J.moff1 = A.take<int>(nmin + 1);
    J.ment1 = A.take<int>(e1);
    J.wstamp1 = A.take<int>(nmin);
    J.aff = A.take<int>(ne);
    J.wlong = A.take<int>(ne);
    int* chunk = A.take<int>(ne / 1024 + 2);
    if (!jh.checksum || !J.ext_id || !J.ocnt1 || !J.first_sj || !chunk) return EXTREMZ_OOM;
    const long long words = (N + 31) / 32;
    const bool join_side = J.join_rows || jh.p.final_join;
    Fills fl;
    // The maxima's selection scratch, entry counts, arbitration slots and
    // wrong-saddle results.
    fl.add(J.ext_key, nmax, 0);
    fl.add(J.largest, nmax, ~0ull);
    fl.add(J.moff2, nmax + 1, 0);
    fl.add(J.wstamp2, nmax, 0);
    fl.add(J.first1, nmax, twice(kInf));
    fl.add(J.first_s, nmax, twice(kInf));
    fl.add(J.flag2, nmax, 0);
    // The minima's; without join_rows only what the final join pass uses.
    if (join_side) {
      fl.add(J.smallest, nmin, twice(kInf));
      fl.add(J.first_sj, nmin, twice(kInf));
    }
    if (J.join_rows) {
      fl.add(J.moff1, nmin + 1, 0);
      fl.add(J.wstamp1, nmin, 0);
      fl.add(J.first_min1, nmin, twice(kInf));
      fl.add(J.flag_min2, nmin, 0);
      fl.add(J.ext_id, nmin, twice(kInf));
      fl.add(J.drow1, ns1 * 2ll, 0);
    }
    // Decompressed row slots start at zero: the reference's rows are fresh
    // cudaMalloc memory read before first written (:5338-5341, :3128-3130).
    fl.add(J.drow2, ns2 * 2ll, 0);
    fl.add(J.bad2, ns2, 0);
    if (J.join_rows) fl.add(J.bad1, ns1, 0);
    // Every tile's pointers are computed in the first manifold round, block
    // stamps start below its stamp, no root is touched, every value counts as
    // changed for it and none for the wrong-saddle scans and detections.
    fl.add(J.tdirty, jh.ntiles, ~0ull);
    fl.add(J.tseen, jh.ntiles, 0);
    fl.add(J.tqueue, jh.ntiles, 0);
    fl.add(J.bdirty, jh.nb, 0);
    fl.add(J.hcnt, jh.nb, 0);
    fl.add(J.rtouch2, words, 0);
    fl.add(J.rtouch1, words, 0);
    fl.add(J.vchg, words, ~0ull);
    fl.add(J.wchg2, words, 0);
    if (J.join_rows) fl.add(J.wchg1, words, 0);
    fl.add(J.dbits, words, 0);
    fl.add(J.dbits1, words, 0);
    fill(fl);
    // Proposal buffer at the sentinel; edit counters, which only edit_type 0
    // reads, at -1 (:5082); arbitration votes, which only the ascending order
    // reads, at 0.
    Fills fv;
    fv.add(J.delta, N, key_pattern(J.sentinel_key));
    if (J.edit_type == 0) fv.add(J.counter, N, ~0ull);
    if (!J.wn_lockstep) fv.add(J.claim, N, 0);
    fill(fv);
    // Per side: the rows (with their compact copies, each named extremum's
    // extreme saddle key and entry count), the entry lists' offsets, then the
    // extreme saddle ids and the entries.  The sides share the selection
    // scratch (ext_key) and the fill cursors (aff), so they go one after the
    // other.  Rows name only extrema, so a side with rows has extrema.  Without
    // join_rows the minima's side waits for the final join pass (k_join_*).
    if (h(slot, C_NAN)) launch(K_SETUP, k_rows<T, true, true>, grid_, 256, J);
    else launch(K_SETUP, k_rows<T, true>, grid_, 256, J);
    if (nmax) {
      EZ_RUN(scan_counts(J.moff2, nmax, 1, J.moff2 + nmax, chunk, J.aff));
      launch(K_OTHER, k_extreme_saddle<T, true>, grid_, 256, J);
    }
    if (join_side) {
      Fills fk;
      fk.add(J.ext_key, nmin, ~0ull);
      fill(fk);
    }
    if (J.join_rows) {
      launch(K_SETUP, k_rows<T, false>, grid_, 256, J);
      if (nmin) {
        EZ_RUN(scan_counts(J.moff1, nmin, 1, J.moff1 + nmin, chunk, J.aff));
        launch(K_OTHER, k_extreme_saddle<T, false>, grid_, 256, J);
      }
    }
    EZ_CHECK(cudaMemcpyAsync(jobs_dev_ + slot, &J, sizeof(J), cudaMemcpyHostToDevice, st_));
    return EXTREMZ_OK;
  }

  // ----------------------------------------------------------- branches --
  // Immediate successors (no counter needed).
  int after_cl(JobHost<T>& j) {
    if (j.block == 1) return PC_RLOOPS;
    return PC_MANIFOLD;
  }
  int joinb(JobHost<T>& j) {
    if (j.nfc1 == 0 && j.p.preserve_join) return PC_SLOOPS_J;
    return endb(j);
  }
  int endb(JobHost<T>& j) {
    if (j.block == 0) return PC_PRE_END;
    j.block += 1;  // block 1 -> 2, 2 -> 3
    j.rounds = 0;
    return PC_CL_DETECT;
  }
  int join3(JobHost<T>& j) {
    if (j.nfc1 == 0 && j.p.preserve_join) return PC_DET3J;
    return PC_FINAL_DETECT;
  }

  void finish(int slot, int status) {
    JobHost<T>& j = slots_[slot];
    j.status = status;
    j.pc = PC_DONE;
  }

  void flush_pending(int slot) {
    JobHost<T>& j = slots_[slot];
    for (int ph : j.pending) {
      if (ph == PH_SADDLE) j.emit(PH_SADDLE, h(slot, C_WSC));
      else if (ph == PH_SADDLE_JOIN) j.emit(PH_SADDLE_JOIN, h(slot, C_WSCJ));
      else if (ph == PH_DETECT3) j.emit(PH_DETECT3, h(slot, C_WSC), h(slot, C_WMC), h(slot, C_WMC2));
    }
    j.pending.clear();
  }

  void snapshot(int slot) {
    JobHost<T>& j = slots_[slot];
    const int v[11] = {j.nfc, j.nfc1, h(slot, C_CMAX), h(slot, C_CMIN), h(slot, C_CSAD),
                       h(slot, C_WMC), h(slot, C_WMC2), h(slot, C_WSC), h(slot, C_WMIN),
                       h(slot, C_WMIN2), h(slot, C_WSCJ)};
    std::memcpy(j.c, v, sizeof(v));
  }

  int loop_test(int slot) {
    JobHost<T>& j = slots_[slot];
    bool any = false;
    for (int i = 0; i < 11; ++i) any |= j.c[i] > 0;
    if (!any) {
      if (j.p.final_join) j.pc = PC_FINAL_JOIN;
      else finish(slot, EXTREMZ_OK);
      return EXTREMZ_OK;
    }
    if (j.outer >= j.p.max_outer) {
      finish(slot, EXTREMZ_ROUND_CAP);
      return EXTREMZ_OK;
    }
    j.outer += 1;
    j.block = 1;
    j.rounds = 0;
    j.pc = PC_CL_DETECT;
    return EXTREMZ_OK;
  }

  int checksum_emit(int slot) {
    JobHost<T>& j = slots_[slot];
    if (!j.trace) return EXTREMZ_OK;
    EZ_CHECK(cudaMemsetAsync(j.checksum, 0, 8, st_));
    launch(K_OTHER, k_checksum<T>, grid_, 256, (const T*)j.J.g, j.J.dim.N, j.checksum);
    unsigned long long hsum = 0;
    EZ_CHECK(cudaMemcpyAsync(&hsum, j.checksum, 8, cudaMemcpyDeviceToHost, st_));
    EZ_CHECK(cudaStreamSynchronize(st_));
    j.emit(PH_CHECKSUM, (int)(hsum & 0x7fffffff), (int)((hsum >> 31) & 0x7fffffff));
    return EXTREMZ_OK;
  }

  // Branch of a job that stopped at a counter-dependent point.
  int decide(int slot) {
    JobHost<T>& j = slots_[slot];
    switch (j.pc) {
      case PC_SETUP_A:
        if (j.p.flags & kFlagLabels) finish(slot, EXTREMZ_OK);
        else j.pc = PC_SETUP_B;
        return EXTREMZ_OK;
      case PC_CL_DETECT:
      case PC_CL_ROUND:
        j.emit(PH_CLOOP_DETECT, h(slot, C_CMAX), h(slot, C_CMIN), h(slot, C_CSAD));
        if (j.p.flags & kFlagCensus) {  // no edit: on to the third block's checks
          j.block = 3;
          j.pc = PC_MANIFOLD;
          return EXTREMZ_OK;
        }
        if (h(slot, C_MM) > 0) {
          if (j.rounds >= j.p.max_cloop_rounds) {
            finish(slot, EXTREMZ_ROUND_CAP);
            return EXTREMZ_OK;
          }
          j.rounds += 1;
          j.cloop_total += 1;
          j.pc = PC_CL_ROUND;
        } else {
          j.pc = after_cl(j);
        }
        return EXTREMZ_OK;
      case PC_MANIFOLD:
        j.nfc = h(slot, C_NFC);
        j.nfc1 = h(slot, C_NFC1);
        j.emit(PH_WRONG_NBR, j.nfc, j.nfc1);
        if (j.p.flags & kFlagCensus) j.pc = PC_DET3;
        else if (j.block == 3) j.pc = j.nfc == 0 ? PC_DET3 : join3(j);
        else j.pc = j.nfc == 0 ? PC_SLOOPS : joinb(j);
        return EXTREMZ_OK;
      case PC_SLOOPS:
        // s_loops refreshes the file-scope host copies (:3473-3476).
        j.emit(PH_SLOOPS, h(slot, C_WMC), h(slot, C_WMC2));
        j.pc = h(slot, C_WMC) == 0 ? PC_SADDLE : joinb(j);
        return EXTREMZ_OK;
      case PC_SLOOPS_J:
        j.emit(PH_SLOOPS_JOIN, h(slot, C_WMIN), h(slot, C_WMIN2));
        j.pc = h(slot, C_WMIN) == 0 ? PC_SADDLE_J : endb(j);
        return EXTREMZ_OK;
      case PC_PRE_END:  // :5589-5599
        snapshot(slot);
        return loop_test(slot);
      case PC_FINAL_DETECT:
        j.emit(PH_CLOOP_DETECT, h(slot, C_CMAX), h(slot, C_CMIN), h(slot, C_CSAD));
        snapshot(slot);
        if (j.p.flags & kFlagCensus) {
          finish(slot, EXTREMZ_OK);
          return EXTREMZ_OK;
        }
        j.emit(PH_OUTER, j.outer);
        EZ_RUN(checksum_emit(slot));
        return loop_test(slot);
      case PC_FINAL_JOIN:
        finish(slot, EXTREMZ_OK);
        return EXTREMZ_OK;
      default:
        return EXTREMZ_OK;
    }
  }
};

}  // namespace extremz

// ExtreM correction kernels for sm_100a.
//
// Each kernel replaces one or more kernels of the reference GPU path
// (src/ExtreM_cuda.cu); the comment on each names them.  Integer, label and
// comparison work is exact; floating-point updates repeat the reference's
// operations in the field type T (build with -fmad=false).
#pragma once

#include <type_traits>

#include "extremz_common.cuh"
#include "extremz_queue.h"

namespace extremz {

// ---------------------------------------------------------------------------
// Per-job device state passed by value to every kernel.
// ---------------------------------------------------------------------------
template <class T>
struct Job {
  using K = typename KeyOf<T>::K;
  Dims dim;
  const T* f;  // original field
  T* g;        // decompressed field, corrected in place
  T* g0;       // copy of the decompressed field as it came in (edit streams only)
  T bound, thr, sentinel;
  K sentinel_key;
  int q, edit_type;

  int8_t* otype;      // original vertex type (-1, 0..5)
  uint16_t* olm;      // original lower-star direction mask
  uint16_t* smask2;   // per 2-saddle row: its upper-neighbour directions in the original field
                      // (a 1-saddle's lower ones are olm)
  uint8_t* ocnt2; uint8_t* ocnt1;  // original row counts (compact copy of row[14])
  int* ds; int* as;   // original steepest ascent / descent roots
  int* dds; int* das; // decompressed roots
  int* ext;           // vertex -> index in the maxima / minima list

  K* delta;           // proposal buffer (order-preserving keys), sentinel between phases
  int* counter;       // delta_counter of the reference (starts at -1)
  int* touched;       // vertices whose delta left the sentinel in this phase
  int* mm;            // mismatch list: v | cat << 29
  int* mm_next;       // the list being rebuilt by the incremental detection
  int* dirty; int* dirty1;  // vertices whose value changed since the last detection, and since
                            // the one before it (they change roles at each detection)
  unsigned* dbits; unsigned* dbits1;  // their membership bitsets
  unsigned long long* claim;  // wrong-neighbour arbitration in ascending saddle order,
                              // (round << 32) | ~saddle
  unsigned* taken; unsigned* taken1;  // bitsets: neighbours flagged in this manifold round
  int* cand; int* cand_next;  // wrong-neighbour candidate saddles (side being resolved)
  int* cand_j;        // join-side candidates, produced with the split side's
  int* flagged; int* flagged1;  // flagged neighbours (split / join)
  uint8_t* mis;       // per vertex: 1 if dds != ds, 2 if das != as
  unsigned* vchg;     // bitset: vertices whose value changed since the last computed round
  unsigned* edited;   // bitset: vertices whose value changed in this correction (or null)
  uint8_t* dirtyv;    // per vertex: the round's byte (mf_byte) when an input of its saddle
                      // rows changed in that round, else 0 or an earlier round's
  int* bdirty;        // per 1024-id block: the round stamp when some dirtyv byte in it was
                      // set
  uint8_t* has2; uint8_t* has1;  // per saddle row: its wrong-neighbour seed bit
  uint8_t* bad2; uint8_t* bad1;  // per saddle row: 1 if its first row slot differs from the
                                 // original row's first entry, 2 if its second from the last
  int* hcnt;          // per saddle-pass chunk: seed bits set in it
  int* cpoff;         // per list (2-saddles, 1-saddles, maxima, minima) and
                      // 1024-id block: offset of the block's first entry
  int* pdd; int* pda; // decompressed steepest pointers, tile-compressed (k_direction): the
                      // path's root with kRootFlag, or the vertex where it leaves the tile
  int* tdirty;        // per tile: a value in the tile or its halo changed since the tile's
                      // pointers were computed (k_apply lists the tile in cand_next then)
  int* tseen;         // per tile: the stamp of the round that last listed it in tqueue
  unsigned long long* tqueue;  // tiles a light round's jump goes over, stamp << 32 | tile
  unsigned* rtouch2; unsigned* rtouch1;  // bitsets: labels (of dds / das) of the vertices of
                                         // the tiles whose pointers this round recomputes

  int* sad2; int* sad1; int* maxima; int* minima;
  int* orow2; int* orow1;  // original rows of kRowStride ints: entries 4 .. count-1 as
                           // extremum indices, -1 for a repeated label (the first four
                           // are in orm2 / orm1)
  int4* orm2; int4* orm1;  // per row: its first four entries as extremum indices (-1 past the
                           // count and for a repeated label; rows are in direction order)
  int4* oend2; int4* oend1;  // per row: first and last entry, then both as extremum indices
  int* drow2; int* drow1;  // decompressed rows: 2 persistent slots per row, see k_saddle_pass
  int* largest; int* smallest;  // per maximum / minimum
  int* first1; int* flag2;      // per maximum: wrong_index_max arbitration
  int* first_min1; int* flag_min2;
  int* first_s; int* first_sj;  // per extremum: its first wrong saddle-row entry (kept across scans)
  int* moff2; int* ment2;       // per maximum: the row entries (i * kRowStride + p) that name it
  int* moff1; int* ment1;       // per minimum: the same over the 1-saddles' rows
  int* wstamp2; int* wstamp1;   // per extremum: the wrong-saddle epoch that last queued it
  int* aff;                     // extrema queued for the wrong-saddle update
  int* wlong;                   // of those, the ones with long entry lists
  unsigned* wchg2; unsigned* wchg1;  // bitsets: values changed since the last wrong-saddle scan
  K* ext_key;                   // largest / smallest saddle selection scratch
  int* ext_id;                  // lowest-row arbitration of get_wrong_index_min (kInf)

  int* ctr;  // device counters, see Ctr
  DeviceTables tb;
  CUtensorMap map_f, map_g;  // tile maps of f and g (when tma_f / tma_g); the kernels that load
                             // tiles read the descriptor in device memory
  int tma_f, tma_g;
  int iter_cap;  // device-side limit of pointer jumping and path walks
  int join_rows;  // the 1-saddles' rows are read during the correction (preserve_join, or a
                  // census); else only the final join pass looks at them (k_join_*)
  int pass_chunk; // 1024-id blocks per saddle-pass work item (a tuning knob)
  int wn_lockstep; // wrong neighbours by the lockstep resolution (k_wn_step, the
                   // default), else in ascending saddle order (k_wn_vote / commit / resolve)
};

// Jobs served by one launch.  Every per-round kernel takes the device array of
// job descriptors and a selection: indices into that array and the exclusive
// prefix of the selected jobs' block counts (for tile kernels their tile
// counts); a block's flat index picks its job by binary search.  A block works
// on one job, so the jobs of a launch run side by side: when every block went
// through all jobs in turn, a launch over 32 small jobs took 32 times the
// latency of one.  A plain correction is a selection of one job.
constexpr int kMaxSel = 64;
struct Sel {
  int n;
  int idx[kMaxSel];
  int off[kMaxSel + 1];
};

// Job of a grid-stride kernel's block, the block's index among the job's blocks
// and their number.
template <class J>
__device__ __forceinline__ J& span_job(J* __restrict__ jobs, const Sel& sel, int& blk, int& nblk) {
  int lo = 0, hi = sel.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (sel.off[mid] <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  blk = (int)blockIdx.x - sel.off[lo];
  nblk = sel.off[lo + 1] - sel.off[lo];
  return jobs[sel.idx[lo]];
}

// Indices into the device counter block.
enum Ctr : int {
  C_MM = 0, C_CMAX, C_CMIN, C_CSAD, C_TOUCHED, C_NFC, C_NFC1, C_CAND, C_CAND_NEXT,
  C_WMC, C_WMC2, C_WSC, C_WMIN, C_WMIN2, C_WSCJ, C_NS2, C_NS1, C_NMAX, C_NMIN,
  C_E2, C_E1,  // row entries of the 2-saddles' / 1-saddles' original rows (upper bound)
  C_NAN,       // the original field holds a NaN
  C_ERROR,
  C_CHANGED,   // some value changed since the last computed manifold round began
  C_DIRTY, C_MM_NEXT, C_CANDJ,
  C_MFDONE,    // a manifold round has run
  C_MFREUSED,  // manifold rounds whose kernels found nothing changed
  // Per-job epochs and stamps, so that one launch can serve jobs at different
  // points of their correction.  There are no launches for bookkeeping: a
  // counter is reset by a kernel that does not use it, or at the end of the tick
  // (k_tick_end).
  C_DEPOCH,    // detections so far; its parity picks dirty / dirty1
  C_DIRTYP,    // entries of the dirty list of the detection before
  C_AMAX, C_AMIN, C_ASAD,  // mismatch counts of the detection under way
  C_WNSTAMP,   // computed manifold rounds so far; a round's stamp is this + 1
  C_WNROUND,   // wrong-neighbour arbitration round (vote high word)
  C_WNSMALL,   // this side's candidate list is small: the block completion does it all
  C_TLIST,     // tiles listed for the next manifold round's steepest pointers (k_apply)
  C_WEP2, C_WEP1,  // wrong-saddle scans so far (maxima, minima); the first computes every extremum
  C_WLIST2, C_WLIST1,  // extrema named by a wrong row in this tick's scan (k_wim_scan)
  C_AFF,       // extrema queued for the current wrong-saddle update
  C_WLONG,     // of those, the ones with long entry lists (wlong)
  C_DETECTED, C_MFRUN,  // a detection, a manifold round ran in this tick
  C_NAFF,      // tiles that hold a vertex whose label may change this round (k_touched_tiles)
  C_QHEAD, C_QDONE,  // of those, taken up and searched
  C_JDENSE,    // they are not listed: the jump goes over every vertex
  C_COUNT
};

// A manifold round's outputs (labels, row slots, flagged neighbours and their
// counts) are functions of the decompressed field alone, so when no value
// changed since the last computed round began they are still in place and the
// round's kernels return at once.
__device__ __forceinline__ bool mf_skip(const int* ctr) {
  return ctr[C_MFDONE] && !ctr[C_CHANGED];
}
__device__ __forceinline__ int mf_stamp(const int* ctr) { return ctr[C_WNSTAMP] + 1; }
// A round's stamp as a byte (dirtyv), never the zero of an unchanged vertex: with
// the stamp's low byte, every 256th round's changes read as no change and their
// blocks were not flagged.
__device__ __forceinline__ unsigned mf_byte(int stamp) { return 1u + (unsigned)stamp % 255u; }
// A light round's jump goes over the tiles that k_touched_tiles finds only in
// fields of at least this many vertices: a pass over every vertex costs about
// 2.2 us per million, the search 50-100 us whatever the field.  Corrections of noisy
// fields (512 Gaussians per 256^3 and noise, bound 1e-5) without the search and with
// it: 3.90 and 4.04 ms at 272^3, 4.74 and 4.75 at 300^3, 6.66 and 6.58 at 340^3, 10.55
// and 10.35 at 400^3, 21.3 and 20.1 at 512^3.  A smooth field, whose few labels lie in
// more than a quarter of the tiles, pays the search for nothing (4.77 and 5.15 ms at
// 400^3).
constexpr int kTouchMin = 1 << 25;
// Start of a round, in its first kernel (which uses none of these).
__device__ __forceinline__ void mf_begin(int* ctr, int n) {
  ctr[C_MFRUN] = 1;
  if (mf_skip(ctr)) return;
  ctr[C_NFC] = ctr[C_NFC1] = 0;
  ctr[C_CAND] = ctr[C_CANDJ] = ctr[C_CAND_NEXT] = 0;
  ctr[C_NAFF] = ctr[C_TLIST];  // the recomputed tiles come first
  ctr[C_QHEAD] = ctr[C_QDONE] = 0;
  ctr[C_JDENSE] = n < kTouchMin;
}
// End of a round.
__device__ __forceinline__ void mf_end(int* ctr) {
  if (mf_skip(ctr)) {
    ctr[C_MFREUSED] += 1;
    return;
  }
  ctr[C_CHANGED] = 0;
  ctr[C_MFDONE] = 1;
  ctr[C_WNSTAMP] += 1;
}
// Error bits in ctr[C_ERROR].
constexpr int kErrJump = 1, kErrPath = 2, kErrTile = 4, kErrResolve = 8;
// Ids per changed-input flag of the jump (the CP-list block size, kCpBlock).
constexpr int kCpBlockJ = 1024;

template <class T>
__device__ __forceinline__ T tabs(T v) { return v < T(0) ? -v : v; }

// Direction components packed two bits per direction (component + 1), so a
// runtime direction index decodes with a shift and a mask.
__host__ __device__ constexpr unsigned pack_dir(int axis) {
  unsigned p = 0;
  for (int d = 0; d < kNumDirs; ++d)
    p |= (unsigned)((axis == 0 ? dir_x(d) : axis == 1 ? dir_y(d) : dir_z(d)) + 1) << (2 * d);
  return p;
}
__device__ __forceinline__ int ddx(int d) { return (int)((pack_dir(0) >> (2 * d)) & 3u) - 1; }
__device__ __forceinline__ int ddy(int d) { return (int)((pack_dir(1) >> (2 * d)) & 3u) - 1; }
__device__ __forceinline__ int ddz(int d) { return (int)((pack_dir(2) >> (2 * d)) & 3u) - 1; }

// ---------------------------------------------------------------------------
// Classification over a shared-memory halo tile.
//
// Replaces classifyVertex_CUDA (:3720-3911): the original field's types and
// lower-star masks (type=0 call, :5289) come from the direction pass over it;
// k_classify is the fused mismatch detection of the type=1 call (:3856-3910),
// appending each mismatching vertex once with its categories (max, min, saddle).
// ---------------------------------------------------------------------------
constexpr int TX = 32, TY = 8, TZ = 4;
// Tile kernels run 256 threads, one per (x, y) column of the tile.
static_assert(TX * TY == 256, "tile kernels map one thread to each (x, y) column of a tile");
// Shared tile rows start 4 elements left of the tile origin so that the TMA
// box origin x = bx - 4 is 16-byte aligned; the tile's x = 0 sits at kXOff.
constexpr int SX = TX + 8, SY = TY + 2, SZ = TZ + 2, kXOff = 4;

template <class T>
struct alignas(128) Tile {
  T v[SZ][SY][SX];
};

// Job and tile origin of a tile kernel's block.
template <class T>
__device__ __forceinline__ const Job<T>& tile_job(const Job<T>* __restrict__ jobs, const Sel& sel,
                                                  int& bx, int& by, int& bz, int* tile = nullptr) {
  const int t = blockIdx.x;
  int lo = 0, hi = sel.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (sel.off[mid] <= t) lo = mid;
    else hi = mid - 1;
  }
  const Job<T>& J = jobs[sel.idx[lo]];
  const int lt = t - sel.off[lo];
  const int ntx = (J.dim.W + TX - 1) / TX, nty = (J.dim.H + TY - 1) / TY;
  bx = (lt % ntx) * TX;
  by = ((lt / ntx) % nty) * TY;
  bz = (lt / (ntx * nty)) * TZ;
  if (tile) *tile = lt;
  return J;
}

// Lists the tiles whose halo tile contains vertex (x, y, z), those holding one
// of its 26 neighbours or itself, unless they are listed already (or not yet
// computed: every mark is set before a job's first round).  The marks of the (at
// most eight) tiles are read together.  All lanes of a warp call it, those with
// `any`, to list theirs with one atomic per warp.
__device__ __forceinline__ void mark_tiles(int* tdirty, int* list, int* count, const Dims& g, int x,
                                           int y, int z, bool any) {
  const int ntx = (g.W + TX - 1) / TX, nty = (g.H + TY - 1) / TY;
  const int x0 = max(x - 1, 0) / TX, x1 = min(x + 1, g.W - 1) / TX;
  const int y0 = max(y - 1, 0) / TY, y1 = min(y + 1, g.H - 1) / TY;
  const int z0 = max(z - 1, 0) / TZ, z1 = min(z + 1, g.D - 1) / TZ;
  int t[8];
  unsigned need = 0u;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const bool own = any && (!(k & 1) || x1 != x0) && (!(k & 2) || y1 != y0) && (!(k & 4) || z1 != z0);
    t[k] = ((k & 4 ? z1 : z0) * nty + (k & 2 ? y1 : y0)) * ntx + (k & 1 ? x1 : x0);
    if (own && tdirty[t[k]] == 0) need |= 1u << k;
  }
  if (!__any_sync(0xffffffffu, need != 0u)) return;
  unsigned mine = 0u;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if ((need >> k & 1u) && atomicExch(tdirty + t[k], 1) == 0) mine |= 1u << k;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int slot = warp_append(count, mine >> k & 1u, 0xffffffffu);
    if (slot >= 0) list[slot] = t[k];
  }
}

// Halo tile: TMA box (one bulk tensor copy, zero fill outside the grid) when
// the field's row stride allows it, else plain loads with every thread's loads
// issued before its first shared store, and zeros outside the grid too.
// A block that loads several tiles initialises the barrier once (init) and
// waits on alternating phases (parity = loads issued before this one, mod 2).
// tile_issue starts the bulk copy; between it and load_tile, which waits for it,
// the block may do other work.
template <class T>
__device__ __forceinline__ void tile_issue(Tile<T>& s, uint64_t* bar, const CUtensorMap* map, int bx,
                                           int by, int bz, bool init) {
  if (threadIdx.x == 0) {
    tma_map_acquire(map);
    if (init) mbar_init(bar, 1);
    mbar_expect_tx(bar, (unsigned)sizeof(Tile<T>));
    tma_load_3d(&s.v[0][0][0], map, bx - kXOff, by - 1, bz - 1, bar);
  }
}

template <class T>
__device__ __forceinline__ bool load_tile(Tile<T>& s, uint64_t* bar, bool tma,
                                          const T* __restrict__ a, const Dims& g, int bx, int by,
                                          int bz, unsigned parity = 0) {
  if (tma) {
    __syncthreads();
    return mbar_wait(bar, parity, 1ll << 26);
  }
  constexpr int HX = TX + 2;
  constexpr int kTotal = HX * SY * SZ;
  constexpr int kPer = (kTotal + 255) / 256;
  T v[kPer];
  int off[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = threadIdx.x + k * 256;
    const int lx = i % HX, t = i / HX, ly = t % SY, lz = t / SY;
    const int gx = bx + lx - 1, gy = by + ly - 1, gz = bz + lz - 1;
    const bool ok = i < kTotal && gx >= 0 && gx < g.W && gy >= 0 && gy < g.H && gz >= 0 && gz < g.D;
    off[k] = i < kTotal ? (lz * SY + ly) * SX + lx + kXOff - 1 : -1;
    v[k] = ok ? __ldg(a + gx + (long long)gy * g.W + (long long)gz * g.W * g.H) : T(0);
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k)
    if (off[k] >= 0) (&s.v[0][0][0])[off[k]] = v[k];
  constexpr int kPad = SX - HX;  // the tile rows' unused columns
  for (int i = threadIdx.x; i < kPad * SY * SZ; i += 256) {
    const int c = i % kPad;
    (&s.v[0][0][0])[(i / kPad) * SX + (c < kXOff - 1 ? c : HX + c)] = T(0);
  }
  __syncthreads();
  return true;
}

// Lower-star direction mask and upper mask of the tile voxel at tile
// coordinates (tx, ty, tz).  A tie goes to the lower side exactly when the
// neighbour's id is smaller, i.e. for odd directions.
template <class T>
__device__ __forceinline__ void tile_masks(const Tile<T>& s, int tx, int ty, int tz, int valid,
                                           int& lm, int& um) {
  const T c = s.v[tz + 1][ty + 1][tx + kXOff];
  lm = 0;
#pragma unroll
  for (int d = 0; d < kNumDirs; ++d) {
    const T nv = s.v[tz + 1 + dir_z(d)][ty + 1 + dir_y(d)][tx + kXOff + dir_x(d)];
    const bool lower = dir_neighbour_is_before(d) ? (nv <= c) : (nv < c);
    lm |= (int)lower << d;
  }
  // Values and ids order the vertices totally: a valid neighbour is upper
  // exactly when it is not lower.
  lm &= valid;
  um = valid & ~lm;
}

// Vertex type from the masks (classifyVertex_CUDA :3835-3853): maximum when no
// upper neighbour, minimum when no lower one, else the LUT entry of the
// boundary configuration, or -1 for a configuration the LUT has no key for.
__device__ __forceinline__ int type_from_masks(int lm, int um, int valid, int bc,
                                               const DeviceTables& tb) {
  if (um == 0) return 4;
  if (lm == 0) return 0;
  const int off = tb.key_offset[bc];
  if (off < 0) return -1;
  int idx = um;
  if (bc != 0) {  // index bits follow the valid neighbours' order
    idx = 0;
    int k = 0;
#pragma unroll
    for (int d = 0; d < kNumDirs; ++d) {
      if (valid >> d & 1) {
        idx |= (um >> d & 1) << k;
        ++k;
      }
    }
  }
  return __ldg(tb.lut + off + idx);
}

// Type of an interior vertex from its lower mask and the packed table in shared
// memory.  (From global memory, the 32 lanes' bytes lie in up to 32 lines of the
// 16 KB table: a third of the original field's direction pass.)
__device__ __forceinline__ int interior_type(int lm, const unsigned* types) {
  constexpr int kAll = (1 << kNumDirs) - 1;
  const int um = kAll & ~lm;
  const int code = (int)(types[um >> 4] >> (2 * (um & 15)) & 3u);
  return um == 0 ? 4 : lm == 0 ? 0 : code ? code : 5;
}

__device__ __forceinline__ int mismatch_cats(int t, int o, int lm, int olm) {
  int cat = 0;
  if (t != o) {
    if ((t == 4) != (o == 4)) cat |= kCatMax;
    if ((t == 0) != (o == 0)) cat |= kCatMin;
    if ((t == 2) != (o == 2) || (t == 1) != (o == 1) || (t == 3) != (o == 3)) cat |= kCatSaddle;
  } else if ((t == 1 || t == 2 || t == 3) && lm != olm) {
    cat |= kCatSaddle;  // areVectorsDifferent_local (:909-921) on direction masks
  }
  return cat;
}

// Per-category counts of mismatching vertices, one atomic per warp and category.
__device__ __forceinline__ void count_cats(int* ctr, int cat) {
  const unsigned bm = __ballot_sync(0xffffffffu, cat & kCatMax);
  const unsigned bn = __ballot_sync(0xffffffffu, cat & kCatMin);
  const unsigned bs = __ballot_sync(0xffffffffu, cat & kCatSaddle);
  if (lane_id() == 0) {
    if (bm) atomicAdd(ctr + C_AMAX, __popc(bm));
    if (bn) atomicAdd(ctr + C_AMIN, __popc(bn));
    if (bs) atomicAdd(ctr + C_ASAD, __popc(bs));
  }
}

// Vertex-id offsets of the 14 directions, for loops over the set bits of a
// direction mask (threads 0..13 fill it; the caller synchronises).
__device__ __forceinline__ void fill_offsets(int* off, const Dims& g) {
  if (threadIdx.x < kNumDirs) {
    const int d = threadIdx.x;
    off[d] = ddx(d) + ddy(d) * g.W + ddz(d) * g.W * g.H;
  }
}

// The upper neighbours of a vertex are the valid ones that are not lower, except a
// NaN, which is neither (only fields with C_NAN look): side without its NaNs.
template <class T>
__device__ __forceinline__ unsigned drop_nans(const T* __restrict__ a, const int* off, int s,
                                              unsigned side) {
  for (unsigned rest = side; rest; rest &= rest - 1u) {
    const int d = __ffs((int)rest) - 1;
    const T v = a[s + off[d]];
    if (v != v) side &= ~(1u << d);
  }
  return side;
}

// A tile-compressed pointer that is its path's root.
constexpr int kRootFlag = (int)0x80000000u;
// At the jump's limit: the end u of a chain that names itself is a root after all
// (the look at a root is not a hop of its own in the limit's count).
__device__ __forceinline__ int root_at_limit(const int* a, int u) {
  return u >= 0 && (a[u] & ~kRootFlag) == u ? u | kRootFlag : u;
}

// In-tile positions of the path following: p = x + 64 y + 1024 z, with one bit
// free above each coordinate's range.  A step adds the direction's offset in the
// same measure (step_of); the result left the tile exactly when one of the free
// bits is set (a borrow below zero sets the bits above), so no coordinate is
// compared.
constexpr int kPosY = 64, kPosZ = 1024, kPosOut = 1 << 5 | 1 << 9 | 1 << 12;
constexpr int kPosCount = kPosZ * (TZ - 1) + kPosY * (TY - 1) + TX;
static_assert(TX == 32 && TY == 8 && TZ == 4, "the free bits of the in-tile positions");
__host__ __device__ constexpr int step_of(int dx, int dy, int dz) {
  return dx + kPosY * dy + kPosZ * dz;
}
// Steps are ordered as the vertex ids they lead to.
static_assert(step_of(1, -1, 0) < step_of(-1, 0, 0) && step_of(1, 0, -1) < step_of(0, -1, 0),
              "in-tile steps order as (z, y, x)");

// Running best of (value, id) over star members; st is the step to it.
template <class T>
struct Best {
  T v;
  int st;
};
// Offers a member with a larger id than all before: it replaces the best when it
// is at least as large (maximum), when it is smaller (minimum), or by force.
template <bool kMax, class T>
__device__ __forceinline__ void offer(Best<T>& b, const Best<T>& m, bool ok = true,
                                      bool force = false) {
  const bool take = force || (ok && (kMax ? m.v >= b.v : m.v < b.v));
  b.v = take ? m.v : b.v;
  b.st = take ? m.st : b.st;
}
// Of two bests in no id order, the one that comes first by (value, id).
template <bool kMax, class T>
__device__ __forceinline__ Best<T> merge(const Best<T>& a, const Best<T>& m) {
  const bool take = kMax ? m.v > a.v || (m.v == a.v && m.st > a.st)
                         : m.v < a.v || (m.v == a.v && m.st < a.st);
  return Best<T>{take ? m.v : a.v, take ? m.st : a.st};
}

// Which neighbours of a tile column exist (kEdge tiles; all do elsewhere).
struct ColumnEdges {
  bool xm, xp, dn, up;
  int z0, z1;  // tile planes -1 .. TZ that are in the grid: z0 .. z1
};

// The seven values of a column's voxel and its in-plane neighbours.
template <class T>
struct Plane {
  T c, xm, xp, up, upm, dn, dnp;
};

// One side's part of a plane: `lo` the best of the four members that the voxel
// above sees of this plane, `hi` of the four that the voxel below sees (in-plane
// steps).  Together they are the voxel's own plane.
template <bool kMax, bool kEdge, class T>
__device__ __forceinline__ void plane_best(const Plane<T>& q, const ColumnEdges& e, Best<T>& lo,
                                           Best<T>& hi) {
  Best<T> bc{q.c, 0};
  offer<kMax>(bc, Best<T>{q.xp, step_of(1, 0, 0)}, !kEdge || e.xp);
  lo = Best<T>{q.dn, step_of(0, -1, 0)};
  offer<kMax>(lo, Best<T>{q.dnp, step_of(1, -1, 0)}, !kEdge || e.xp);
  offer<kMax>(lo, bc, true, kEdge && !e.dn);
  hi = Best<T>{q.xm, step_of(-1, 0, 0)};
  offer<kMax>(hi, Best<T>{q.c, 0}, true, kEdge && !e.xm);
  Best<T> aup{q.upm, step_of(-1, 1, 0)};
  offer<kMax>(aup, Best<T>{q.up, step_of(0, 1, 0)}, true, kEdge && !e.xm);
  offer<kMax>(hi, aup, !kEdge || e.up);
}

// One tile column (x, y) upwards: for each of its TZ voxels, kSteps, the step to
// its steepest-ascent and steepest-descent neighbour (0 at a root), and, kMasks,
// its lower-star direction mask before the validity mask.  The closed star of v is
// v + C and v - C for C = {0, 1}^3 in (-x, y, z), so a plane's values serve three
// voxels of the column: 7 loads and 11 two-way choices a voxel and side, where
// each voxel by itself takes 15 of both.  The steps want finite values (the caller
// checks).
template <class T, bool kEdge, bool kSteps, bool kMasks>
__device__ __forceinline__ void column_steps(const Tile<T>& s, int tx, int ty, const ColumnEdges& e,
                                             int* up_st, int* dn_st, int* lm) {
  const T(*row)[SY][SX] = s.v;
  const int x = tx + kXOff, y = ty + 1;
  Best<T> plo[2], part[2];  // the plane below: its lo; the voxel below: its best so far
  T cprev = T(0);
#pragma unroll
  for (int pz = 0; pz < SZ; ++pz) {  // tile plane pz - 1
    Plane<T> q;
    q.c = row[pz][y][x];
    if (pz > 0) {
      q.xm = row[pz][y][x - 1];
      q.up = row[pz][y + 1][x];
      q.upm = row[pz][y + 1][x - 1];
    } else {
      q.xm = q.up = q.upm = q.c;
    }
    if (pz < SZ - 1) {
      q.xp = row[pz][y][x + 1];
      q.dn = row[pz][y - 1][x];
      q.dnp = row[pz][y - 1][x + 1];
    } else {
      q.xp = q.dn = q.dnp = q.c;
    }
    if (kMasks) {
      // A tie goes to the lower side exactly when the neighbour's id is smaller
      // (odd directions).
      if (pz >= 2) {
        int& m = lm[pz - 2];
        m |= (int)(q.c < cprev) << 4 | (int)(q.xm < cprev) << 10 | (int)(q.up < cprev) << 8 |
             (int)(q.upm < cprev) << 12;
      }
      if (pz >= 1 && pz < SZ - 1) {
        int& m = lm[pz - 1];
        m |= (int)(q.xp < q.c) << 0 | (int)(q.xm <= q.c) << 1 | (int)(q.up < q.c) << 2 |
             (int)(q.dn <= q.c) << 3 | (int)(q.upm < q.c) << 6 | (int)(q.dnp <= q.c) << 7;
      }
      if (pz < SZ - 2) {
        const T cn = row[pz + 1][y][x];
        lm[pz] = (int)(q.c <= cn) << 5 | (int)(q.xp <= cn) << 11 | (int)(q.dn <= cn) << 9 |
                 (int)(q.dnp <= cn) << 13;
      }
      cprev = q.c;
    }
    auto side = [&](auto kmax, int k, int* st) {
      constexpr bool kMax = decltype(kmax)::value;
      Best<T> lo, hi;
      plane_best<kMax, kEdge>(q, e, lo, hi);
      if (pz >= 2) {  // the voxel below is complete
        offer<kMax>(part[k], Best<T>{hi.v, hi.st + kPosZ}, !kEdge || pz - 1 <= e.z1);
        st[pz - 2] = part[k].st;
      }
      if (pz >= 1 && pz < SZ - 1) {
        part[k] = Best<T>{plo[k].v, plo[k].st - kPosZ};
        offer<kMax>(part[k], merge<kMax>(lo, hi), true, kEdge && pz - 2 < e.z0);
      }
      plo[k] = lo;
    };
    if constexpr (kSteps) {
      side(std::true_type{}, 0, up_st);
      side(std::false_type{}, 1, dn_st);
    }
  }
}

// The first detection of a job: the whole decompressed field.
template <class T>
__global__ void __launch_bounds__(256, 8) k_classify(const Job<T>* __restrict__ jobs,
                                                  const __grid_constant__ Sel sel) {
  __shared__ Tile<T> s;
  __shared__ uint64_t bar;
  int bx, by, bz;
  const Job<T>& J = tile_job(jobs, sel, bx, by, bz);
  const Dims g = J.dim;
  // The block decides together: its threads meet at barriers further on.
  if (J.tma_g) tile_issue<T>(s, &bar, &J.map_g, bx, by, bz, true);
  if (!__syncthreads_and(load_tile<T>(s, &bar, J.tma_g, J.g, g, bx, by, bz))) {
    if (threadIdx.x == 0) atomicOr(J.ctr + C_ERROR, kErrTile);
    return;
  }
  // Detection: the tile's mismatching vertices are gathered in shared memory
  // and appended with one global atomic per block (per warp, the appends of a
  // dense pass all queue on the same counter).
  __shared__ int s_list[TZ * TY * TX];
  __shared__ int s_n, s_base, s_cat[3];
  if (threadIdx.x == 0) {
    s_n = 0;
    s_cat[0] = s_cat[1] = s_cat[2] = 0;
  }
  __syncthreads();
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  // A tile off the field's faces has every direction valid at every voxel.
  const bool interior = bx > 0 && by > 0 && bz > 0 && bx + TX < g.W && by + TY < g.H &&
                        bz + TZ < g.D;
  int mask[TZ];
  column_steps<T, false, false, true>(s, tx, ty, ColumnEdges{}, nullptr, nullptr, mask);
#pragma unroll
  for (int tz = 0; tz < TZ; ++tz) {
    const int x = bx + tx, y = by + ty, z = bz + tz;
    const bool in = x < g.W && y < g.H && z < g.D;
    if (in) {
      const int v = x + y * g.W + z * g.W * g.H;
      const int bc = interior ? 0 : boundary_code(x, y, z, g.W, g.H, g.D);
      const int valid = interior ? (1 << kNumDirs) - 1 : valid_mask(bc);
      const int lm = mask[tz] & valid, om = J.olm[v];
      // The type follows from the mask: with the original's mask nothing differs.
      const int cat = lm == om ? 0
                               : mismatch_cats(type_from_masks(lm, valid & ~lm, valid, bc, J.tb),
                                               J.otype[v], lm, om);
      if (cat) {
        s_list[atomicAdd(&s_n, 1)] = v | (cat << kCatShift);
        if (cat & kCatMax) atomicAdd(&s_cat[0], 1);
        if (cat & kCatMin) atomicAdd(&s_cat[1], 1);
        if (cat & kCatSaddle) atomicAdd(&s_cat[2], 1);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_n) {
    s_base = atomicAdd(J.ctr + C_MM, s_n);
    if (s_cat[0]) atomicAdd(J.ctr + C_CMAX, s_cat[0]);
    if (s_cat[1]) atomicAdd(J.ctr + C_CMIN, s_cat[1]);
    if (s_cat[2]) atomicAdd(J.ctr + C_CSAD, s_cat[2]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < s_n; k += blockDim.x) J.mm[s_base + k] = s_list[k];
}

// ---------------------------------------------------------------------------
// Incremental mismatch detection.
//
// The type of v depends only on the values of v and its 14 neighbours, so after
// the first dense detection only the closed neighbourhoods of vertices whose
// value changed can change status.  k_redetect re-evaluates them, once each: a
// vertex belongs to the first changed vertex of its closed neighbourhood, in
// direction order with itself first, found from the membership bitset of the
// changed vertices.  Beside that it carries over the entries of the previous
// list that have no changed vertex in their neighbourhood.  The resulting set
// equals a dense re-detection (the lists are unordered; every consumer merges by
// atomic max).  The end of the tick publishes the counts and swaps the lists
// (detect_end), so a detection is one launch (four with a stamp per vertex, a
// second kernel for the carried entries and two for the bookkeeping).
// ---------------------------------------------------------------------------
// Mismatch categories of vertex v on the decompressed field.
template <class T>
__device__ __forceinline__ int vertex_cats(const Job<T>& J, int v) {
  const Dims g = J.dim;
  int x, y, z;
  coords(v, g, x, y, z);
  const int bc = boundary_code(x, y, z, g.W, g.H, g.D);
  const int valid = valid_mask(bc);
  const int om = J.olm[v];
  const T c = J.g[v];
  int lm = 0;
#pragma unroll
  for (int d = 0; d < kNumDirs; ++d) {
    if (!(valid >> d & 1)) continue;
    const T nv = J.g[v + dir_x(d) + dir_y(d) * g.W + dir_z(d) * g.W * g.H];
    if (dir_neighbour_is_before(d) ? nv <= c : nv < c) lm |= 1 << d;
  }
  // The type follows from the mask: with the original's mask nothing differs.
  return lm == om ? 0
                  : mismatch_cats(type_from_masks(lm, valid & ~lm, valid, bc, J.tb), J.otype[v], lm, om);
}

__device__ __forceinline__ bool bit_of(const unsigned* bits, int v) {
  return bits[v >> 5] >> (v & 31) & 1u;
}

template <class T>
__device__ __forceinline__ void detect_end(Job<T>& J) {
  int* c = J.ctr;
  int* t = J.mm;
  J.mm = J.mm_next;
  J.mm_next = t;
  c[C_MM] = c[C_MM_NEXT];
  c[C_MM_NEXT] = 0;
  c[C_CMAX] = c[C_AMAX];
  c[C_CMIN] = c[C_AMIN];
  c[C_CSAD] = c[C_ASAD];
  c[C_AMAX] = c[C_AMIN] = c[C_ASAD] = 0;
  c[C_DIRTYP] = c[C_DIRTY];
  c[C_DIRTY] = 0;
  c[C_DEPOCH] += 1;
}

// Changed vertices (one in this many) from which k_redetect goes by the bitset.
constexpr int kRedetectMany = 64;

template <class T>
__global__ void __launch_bounds__(256) k_redetect(const Job<T>* __restrict__ jobs,
                                                  const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const Dims g = J.dim;
  const bool odd = J.ctr[C_DEPOCH] & 1;
  const int* __restrict__ dirty = odd ? J.dirty1 : J.dirty;
  const unsigned* __restrict__ bits = odd ? J.dbits1 : J.dbits;
  const int n = J.ctr[C_DIRTY], nmm = J.ctr[C_MM];
  // Many changed vertices: their dilated bitset, a word (32 vertices) per lane,
  // then word by word a vertex per lane, instead of fifteen candidates per changed
  // vertex and a search for each one's owner.  Across the ends of rows the
  // dilation is too wide, which evaluates a vertex that need not be; the carried
  // entries are tested against the same set.  (By the list, the first detection
  // after the first edits took 0.16 ms at 256^3.)
  const bool many = n > g.N / kRedetectMany;
  __shared__ int off[kNumDirs];
  fill_offsets(off, g);
  __syncthreads();
  const int nw = (g.N + 31) >> 5;
  if (many) {
    for (int w0 = (blk * 8 + (int)(threadIdx.x >> 5)) * 32; w0 < nw; w0 += nblk * 256) {
      const int w = w0 + (int)lane_id();
      unsigned near = 0u;
      if (w < nw) {
        near = bits[w];
#pragma unroll
        for (int k = 0; k < kNumDirs; ++k) {
          const int at = 32 * w + off[k], i = at >> 5;
          const unsigned lo = (unsigned)i < (unsigned)nw ? bits[i] : 0u;
          const unsigned hi = (unsigned)(i + 1) < (unsigned)nw ? bits[i + 1] : 0u;
          near |= __funnelshift_r(lo, hi, at & 31);
        }
      }
      for (int j = 0; j < 32; ++j) {
        const unsigned word = __shfl_sync(0xffffffffu, near, j);
        if (!word) continue;
        const int v = 32 * (w0 + j) + (int)lane_id();
        const int cat = (word >> lane_id() & 1u) && v < g.N ? vertex_cats(J, v) : 0;
        const int slot = warp_append(J.ctr + C_MM_NEXT, cat != 0, 0xffffffffu);
        if (slot >= 0) J.mm_next[slot] = v | (cat << kCatShift);
        count_cats(J.ctr, cat);
      }
    }
  }
  const long long nd = many ? 0 : (long long)n * (kNumDirs + 1), total = nd + nmm;
  const long long stride = (long long)nblk * blockDim.x;
  for (long long base = blk * (long long)blockDim.x; base < total; base += stride) {
    const long long e = base + threadIdx.x;
    int cat = 0, v = -1;
    if (e < nd) {
      const int c = dirty[e / (kNumDirs + 1)];
      const int d = (int)(e % (kNumDirs + 1)) - 1;  // -1: the vertex itself
      v = c;
      if (d >= 0) {
        int x, y, z;
        coords(c, g, x, y, z);
        v = -1;
        const int dx = ddx(d), dy = ddy(d), dz = ddz(d);
        if ((unsigned)(x + dx) < (unsigned)g.W && (unsigned)(y + dy) < (unsigned)g.H &&
            (unsigned)(z + dz) < (unsigned)g.D) {
          v = c + dx + dy * g.W + dz * g.W * g.H;
          // From v, c lies in direction d ^ 1: v is c's unless v itself or a
          // neighbour in an earlier direction changed too.
          const int valid = valid_mask(boundary_code(x + dx, y + dy, z + dz, g.W, g.H, g.D));
          bool earlier = bit_of(bits, v);
#pragma unroll
          for (int k = 0; k < kNumDirs; ++k)
            if (k < (d ^ 1) && (valid >> k & 1))
              earlier |= bit_of(bits, v + dir_x(k) + dir_y(k) * g.W + dir_z(k) * g.W * g.H);
          if (earlier) v = -1;
        }
      }
      if (v >= 0) cat = vertex_cats(J, v);
    } else if (e < total) {
      const int ent = J.mm[e - nd];
      v = ent & ((1 << kCatShift) - 1);
      bool near = bit_of(bits, v);
      if (many) {
#pragma unroll
        for (int k = 0; k < kNumDirs; ++k) {
          const int u = v + off[k];
          near |= (unsigned)u < (unsigned)(32 * nw) && bit_of(bits, u);
        }
      } else {
        int x, y, z;
        coords(v, g, x, y, z);
        const int valid = valid_mask(boundary_code(x, y, z, g.W, g.H, g.D));
#pragma unroll
        for (int k = 0; k < kNumDirs; ++k)
          if (valid >> k & 1)
            near |= bit_of(bits, v + dir_x(k) + dir_y(k) * g.W + dir_z(k) * g.W * g.H);
      }
      if (!near) cat = (unsigned)ent >> kCatShift;
    }
    const int slot = warp_append(J.ctr + C_MM_NEXT, cat != 0, 0xffffffffu);
    if (slot >= 0) J.mm_next[slot] = v | (cat << kCatShift);
    count_cats(J.ctr, cat);
  }
  // The bits of the detection before this one, for the next edits.
  const int np = J.ctr[C_DIRTYP];
  const int* prev = odd ? J.dirty : J.dirty1;
  unsigned* pbits = odd ? J.dbits : J.dbits1;
  for (int e = blk * blockDim.x + threadIdx.x; e < np; e += (int)stride) pbits[prev[e] >> 5] = 0u;
  if (blk == 0 && threadIdx.x == 0) J.ctr[C_DETECTED] = 1;
}

// ---------------------------------------------------------------------------
// Steepest directions with tile-local path compression.
//
// Replaces ComputeDirection (:1464-1512) and the first steps of the pointer
// jumping (:1514-1611): each voxel's steepest-ascent (descent) pointer is
// followed inside the tile in shared memory until it leaves the tile or stops
// at a root, so the global jump that follows moves a tile per hop.
// Output: ds/as (original field) or pdd/pda (decompressed field) = first
// vertex outside the tile on the path, or the root.  On the decompressed field
// only tiles marked dirty (a value in the tile or its halo changed) are
// recomputed; the others keep their pointers, which depend on nothing else.
// ---------------------------------------------------------------------------
// Steepest-ascent and steepest-descent directions of one tile voxel: the
// maximum (minimum) of (value, id) over the voxel and its valid neighbours.
// Ids are scanned in ascending order so that ">=" keeps the larger id on a tie;
// the descent scans in descending order with "<=".  (Finite inputs: the scans
// start from -inf / +inf and always meet the centre.)
template <class T>
__device__ __forceinline__ void steepest_dirs(const Tile<T>& s, int tx, int ty, int tz, int valid,
                                              int& hd, int& ld) {
  const T c = s.v[tz + 1][ty + 1][tx + kXOff];
  T hv = -T(INFINITY), lv = T(INFINITY);
  hd = -1;
  ld = -1;
  T nv[kNumDirs];
#pragma unroll
  for (int d = 0; d < kNumDirs; ++d)
    nv[d] = s.v[tz + 1 + dir_z(d)][ty + 1 + dir_y(d)][tx + kXOff + dir_x(d)];
#pragma unroll
  for (int j = 0; j < kNumDirs; ++j) {
    const int d = rank_dir(j);
    if (j == kRankCentre && c >= hv) { hv = c; hd = -1; }
    if ((valid >> d & 1) && nv[d] >= hv) { hv = nv[d]; hd = d; }
  }
#pragma unroll
  for (int j = kNumDirs - 1; j >= 0; --j) {
    const int d = rank_dir(j);
    if ((valid >> d & 1) && nv[d] <= lv) { lv = nv[d]; ld = d; }
    if (j == kRankCentre && c <= lv) { lv = c; ld = -1; }
  }
}

// The same steps voxel by voxel through the exact scans of steepest_dirs, for a
// tile that holds an infinity or a NaN.
template <class T>
__device__ __noinline__ void column_steps_any(const Tile<T>& s, int tx, int ty, int bx, int by, int bz,
                                              const Dims& g, int* up_st, int* dn_st, int* lm) {
  for (int tz = 0; tz < TZ; ++tz) {
    const int x = bx + tx, y = by + ty, z = bz + tz;
    int hd = -1, ld = -1, um;
    lm[tz] = 0;
    if (x < g.W && y < g.H && z < g.D) {
      const int valid = valid_mask(boundary_code(x, y, z, g.W, g.H, g.D));
      steepest_dirs<T>(s, tx, ty, tz, valid, hd, ld);
      tile_masks(s, tx, ty, tz, valid, lm[tz], um);
    }
    up_st[tz] = hd < 0 ? 0 : step_of(ddx(hd), ddy(hd), ddz(hd));
    dn_st[tz] = ld < 0 ? 0 : step_of(ddx(ld), ddy(ld), ddz(ld));
  }
}

// Sets *nan when the tile holds a NaN.
template <class T>
__device__ __noinline__ void note_nans(const Tile<T>& s, int* nan) {
  for (int i = threadIdx.x; i < SX * SY * SZ; i += 256)
    if (isnan((&s.v[0][0][0])[i])) *nan = 1;
}

// Follows the tile's next positions from p, whose own is t, to the path's exit
// from the tile or its root.
__device__ __forceinline__ int follow(const int16_t* nxt, int p, int t, int* err) {
  for (int step = 0; t != p && !(t & kPosOut); ++step) {
    p = t;
    t = nxt[p];
    if (step > TX * TY * TZ) {  // a path never revisits a voxel; guard anyway
      atomicOr(err, kErrTile);
      break;
    }
  }
  return t;
}

// Steepest pointers of one tile, compressed to the tile's exits: every voxel's
// pointer is the first vertex outside the tile on its steepest path, or the
// path's root inside the tile.  kDec = false: f into ds / as (setup), with the
// original classification (otype, olm) from the same tile load; true: g into
// pdd / pda.  Returns false when the tile's load did not complete.
// Bound by the integer pipe (62 % busy: the selects of the two-way choices, then
// the path loops).  A full pass over the 512^3 float64 benchmark field takes
// 1.50 ms, with the classification 2.05 ms; with every voxel scanning its own
// star, and steps checked and indexed by coordinates, 2.08 and 2.69 ms.
template <class T, bool kDec>
__device__ __noinline__ bool direction_tile(const Job<T>& J, Tile<T>& s, uint64_t* bar,
                                            int16_t* hnext, int16_t* lnext, const unsigned* types,
                                            int bx, int by, int bz, unsigned parity) {
  const Dims g = J.dim;
  const int WH = g.W * g.H;
  const T* a = kDec ? J.g : J.f;
  int* ds = kDec ? J.pdd : J.ds;
  int* as = kDec ? J.pda : J.as;
  const bool loaded = load_tile<T>(s, bar, kDec ? J.tma_g : J.tma_f, a, g, bx, by, bz, parity);
  // Whether the tile holds a value that is not finite: v * 0 is then NaN.
  T zero = T(0);
  if (loaded)
    for (int i = threadIdx.x; i < SX * SY * SZ; i += 256) {
      const T v = (&s.v[0][0][0])[i];
      zero = sizeof(T) == 8 ? (T)__fma_rn((double)v, 0.0, (double)zero)
                            : (T)__fmaf_rn((float)v, 0.0f, (float)zero);
    }
  // The block decides together: its threads meet at a barrier further on.
  const bool usual = __syncthreads_and(loaded && zero == T(0));
  if (!usual && !__syncthreads_and(loaded)) {
    if (threadIdx.x == 0) atomicOr(J.ctr + C_ERROR, kErrTile);
    return false;
  }
  if (!kDec && !usual) note_nans(s, J.ctr + C_NAN);
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int x = bx + tx, y = by + ty;
  // A tile off the field's faces has every direction valid at every voxel.
  const bool interior = bx > 0 && by > 0 && bz > 0 && bx + TX < g.W && by + TY < g.H &&
                        bz + TZ < g.D;
  int hs[TZ], ls[TZ], lm[TZ];
  if (!usual) {
    column_steps_any<T>(s, tx, ty, bx, by, bz, g, hs, ls, lm);
  } else if (interior) {
    column_steps<T, false, true, !kDec>(s, tx, ty, ColumnEdges{}, hs, ls, lm);
  } else {
    const ColumnEdges e{x > 0, x + 1 < g.W, y > 0, y + 1 < g.H, bz > 0 ? -1 : 0,
                        min(TZ, g.D - 1 - bz)};
    column_steps<T, true, true, !kDec>(s, tx, ty, e, hs, ls, lm);
  }
  const bool col = x < g.W && y < g.H;
  const int p0 = tx + kPosY * ty;
#pragma unroll
  for (int tz = 0; tz < TZ; ++tz) {
    const int p = p0 + kPosZ * tz;
    hs[tz] += p;
    ls[tz] += p;
    hnext[p] = (int16_t)hs[tz];
    lnext[p] = (int16_t)ls[tz];
    const int z = bz + tz;
    if (!kDec && col && z < g.D) {
      // The original field's classification from the same tile
      // (classifyVertex_CUDA, the type = 0 call :5289): type and lower-star
      // direction mask.
      const int v = x + y * g.W + z * WH;
      const int bc = interior ? 0 : boundary_code(x, y, z, g.W, g.H, g.D);
      const int valid = interior ? (1 << kNumDirs) - 1 : valid_mask(bc);
      const int m = lm[tz] & valid;
      J.otype[v] = (int8_t)(bc == 0 ? interior_type(m, types)
                                    : type_from_masks(m, valid & ~m, valid, bc, J.tb));
      J.olm[v] = (uint16_t)m;
    }
  }
  __syncthreads();
  if (!col) return true;
  // Vertex of an in-tile position, one plane, row and column outside included;
  // flagged when the path ended inside.
  const int base = (bx - 1) + (by - 1) * g.W + (bz - 1) * WH;
  auto vertex = [&](int t) {
    const int q = t + step_of(1, 1, 1);
    const int v = base + (q & (kPosY - 1)) + (q >> 6 & 15) * g.W + (q >> 10) * WH;
    return t & kPosOut ? v : v | kRootFlag;
  };
#pragma unroll
  for (int tz = 0; tz < TZ; ++tz) {
    if (bz + tz >= g.D) break;
    const int p = p0 + kPosZ * tz;
    const int v = x + y * g.W + (bz + tz) * WH;
    ds[v] = vertex(follow(hnext, p, hs[tz], J.ctr + C_ERROR));
    as[v] = vertex(follow(lnext, p, ls[tz], J.ctr + C_ERROR));
  }
  return true;
}

// Setup: every tile of the original field, one block per tile.
template <class T, bool kDec>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 4 : 6) k_direction(const Job<T>* __restrict__ jobs,
                                                   const __grid_constant__ Sel sel) {
  __shared__ Tile<T> s;
  __shared__ uint64_t bar;
  __shared__ int16_t hnext[kPosCount], lnext[kPosCount];
  int bx, by, bz, tile;
  const Job<T>& J = tile_job(jobs, sel, bx, by, bz, &tile);
  if (kDec) {
    if (tile == 0 && threadIdx.x == 0) mf_begin(J.ctr, J.dim.N);
    if (mf_skip(J.ctr)) return;  // same inputs as the last manifold round
    if (!J.tdirty[tile]) return;  // tile and halo unchanged: pointers stand
  }
  if (kDec ? J.tma_g : J.tma_f)
    tile_issue<T>(s, &bar, kDec ? &J.map_g : &J.map_f, bx, by, bz, true);
  // The packed interior types (pack_types, on the host), while the tile is on its way.
  __shared__ uint4 types[kDec ? 1 : kTypeWords / 4];
  if (!kDec) types[threadIdx.x] = reinterpret_cast<const uint4*>(J.tb.packed)[threadIdx.x];
  if (!direction_tile<T, kDec>(J, s, &bar, hnext, lnext, reinterpret_cast<const unsigned*>(types), bx,
                               by, bz, 0))
    return;
  if (kDec && threadIdx.x == 0) J.tdirty[tile] = 0;
}

// A manifold round's steepest pointers of the decompressed field: a fixed
// grid whose blocks take the listed tiles of every selected job in turn, so
// that a round with few changed tiles launches few blocks' worth of work
// instead of one block per tile of the field.  It also marks, per side, the
// current labels of every vertex of a listed tile as touched roots (rtouch2,
// rtouch1): only vertices with a touched label can change label this round
// (k_jump2).
template <class T>
__global__ void __launch_bounds__(256, 4) k_direction_list(const Job<T>* __restrict__ jobs,
                                                        const __grid_constant__ Sel sel) {
  __shared__ Tile<T> s;
  __shared__ uint64_t bar;
  __shared__ int16_t hnext[kPosCount], lnext[kPosCount];
  unsigned loads = 0;  // TMA loads issued by this block: the barrier's phase
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (blk == 0 && threadIdx.x == 0) mf_begin(J.ctr, J.dim.N);
  if (mf_skip(J.ctr)) return;
  const int n = J.ctr[C_TLIST];
  const int ntx = (J.dim.W + TX - 1) / TX, nty = (J.dim.H + TY - 1) / TY;
  for (int k = blk; k < n; k += nblk) {
    const int t = J.cand_next[k];
    const int bx = (t % ntx) * TX, by = ((t / ntx) % nty) * TY, bz = (t / (ntx * nty)) * TZ;
    __syncthreads();  // every thread is done with the shared tile of the last one
    const bool tma = J.tma_g != 0;
    if (tma) tile_issue<T>(s, &bar, &J.map_g, bx, by, bz, loads == 0);
    // While the tile is on its way: the current labels of its vertices.
    const int x = bx + (int)threadIdx.x % TX, y = by + (int)threadIdx.x / TX;
    if (x < J.dim.W && y < J.dim.H) {
      int r2[TZ], r1[TZ];
      unsigned w2[TZ], w1[TZ];
      const int v0 = x + y * J.dim.W + bz * J.dim.W * J.dim.H;
#pragma unroll
      for (int tz = 0; tz < TZ; ++tz) {
        const bool in = bz + tz < J.dim.D;
        r2[tz] = in ? J.dds[v0 + tz * J.dim.W * J.dim.H] : r2[0];
        r1[tz] = in ? J.das[v0 + tz * J.dim.W * J.dim.H] : r1[0];
      }
      // Read first: most roots are marked by many vertices.
#pragma unroll
      for (int tz = 0; tz < TZ; ++tz) {
        w2[tz] = J.rtouch2[r2[tz] >> 5];
        w1[tz] = J.rtouch1[r1[tz] >> 5];
      }
#pragma unroll
      for (int tz = 0; tz < TZ; ++tz) {
        if (!(w2[tz] >> (r2[tz] & 31) & 1u)) atomicOr(J.rtouch2 + (r2[tz] >> 5), 1u << (r2[tz] & 31));
        if (!(w1[tz] >> (r1[tz] & 31) & 1u)) atomicOr(J.rtouch1 + (r1[tz] >> 5), 1u << (r1[tz] & 31));
      }
    }
    if (!direction_tile<T, true>(J, s, &bar, hnext, lnext, nullptr, bx, by, bz, loads & 1u)) return;
    loads += tma;
    if (threadIdx.x == 0) {
      J.tdirty[t] = 0;
      J.tseen[t] = mf_stamp(J.ctr);
      J.tqueue[k] = (unsigned long long)mf_stamp(J.ctr) << 32 | (unsigned)t;
    }
  }
}

// The tiles that hold a vertex whose label may change this round: one with a
// touched root's label (rtouch2 / rtouch1, see k_direction_list).  The vertices
// of one label are connected (each one's path stays in its label), and a touched
// label has a vertex in a recomputed tile, so they are found outwards from the
// recomputed tiles, the queue's first entries: when a tile's halo holds a touched
// label, the halo vertex's tile is next, unless it is stamped already.  A light
// round (a few dozen changed tiles) of a large field then jumps in some hundred
// tiles instead of reading every vertex's two labels (8 B a voxel, 0.29 ms at
// 512^3 for a handful of changes).  With more than a 64th of the tiles
// recomputed, or a quarter found, the jump goes over every vertex.
//
// A block takes the queue's entries by ticket (queue_take).  It waits for its entry
// only while another running block still searches (entries done < entries pushed);
// should that take too long, it asks for the pass over every vertex, which is
// always right, and everyone stops.
__device__ __forceinline__ int load_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int load_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
struct TileQueue {
  int* ctr;
  unsigned long long* at;
  __device__ int ticket() const { return atomicAdd(ctr + C_QHEAD, 1); }
  __device__ int place() const { return atomicAdd(ctr + C_NAFF, 1); }
  // Called by one thread, behind a barrier with those that pushed.
  __device__ void finished() const {
    __threadfence();
    atomicAdd(ctr + C_QDONE, 1);
  }
  __device__ int done() const { return load_acquire(ctr + C_QDONE); }
  __device__ int pushed() const { return load_relaxed(ctr + C_NAFF); }
  __device__ bool dense() const { return load_relaxed(ctr + C_JDENSE) != 0; }
  __device__ void ask_dense() const { atomicExch(ctr + C_JDENSE, 1); }
  __device__ unsigned long long entry(int i) const {
    unsigned long long e;
    asm volatile("ld.relaxed.gpu.b64 %0, [%1];" : "=l"(e) : "l"(at + i) : "memory");
    return e;
  }
  __device__ void store(int i, unsigned long long e) const {
    asm volatile("st.relaxed.gpu.b64 [%0], %1;" ::"l"(at + i), "l"(e) : "memory");
  }
  __device__ void pause() const { __nanosleep(100); }
};
constexpr int kQueueWait = 1 << 16;  // looks at the queue, at least 100 ns apart
template <class T>
__global__ void __launch_bounds__(256) k_touched_tiles(const Job<T>* __restrict__ jobs,
                                                       const __grid_constant__ Sel sel) {
  __shared__ int tile;
  __shared__ unsigned found;
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  int* ctr = J.ctr;
  // A block's threads leave together: on values that nothing writes during this
  // launch, or on the tile that the first thread took.  C_JDENSE, which other blocks
  // set meanwhile, is looked at by that thread alone (a block of which only some
  // threads saw it set would go on without the one that writes `tile`).
  if (mf_skip(ctr)) return;
  const Dims g = J.dim;
  const int WH = g.W * g.H;
  const int ntx = (g.W + TX - 1) / TX, nty = (g.H + TY - 1) / TY, ntz = (g.D + TZ - 1) / TZ;
  const int nt = ntx * nty * ntz;
  const unsigned stamp = (unsigned)mf_stamp(ctr);
  if (ctr[C_TLIST] > nt / 64) {
    if (threadIdx.x == 0) ctr[C_JDENSE] = 1;
    return;
  }
  TileQueue queue{ctr, J.tqueue};  // (its first look finds C_JDENSE set from the start too)
  for (;;) {
    if (threadIdx.x == 0) {
      tile = queue_take(queue, stamp, nt, kQueueWait);
      found = 0u;
    }
    __syncthreads();
    const int t = tile;
    if (t < 0) return;
    const int bx = (t % ntx) * TX, by = ((t / ntx) % nty) * TY, bz = (t / (ntx * nty)) * TZ;
    // The halo around the tile, in which each vertex stands for one of the 26
    // neighbouring tiles.
    unsigned mine = 0u;
    for (int i = threadIdx.x; i < (TX + 2) * (TY + 2) * (TZ + 2); i += 256) {
      const int lx = i % (TX + 2) - 1, r = i / (TX + 2), ly = r % (TY + 2) - 1, lz = r / (TY + 2) - 1;
      const int nx = lx < 0 ? 0 : lx < TX ? 1 : 2, ny = ly < 0 ? 0 : ly < TY ? 1 : 2,
                nz = lz < 0 ? 0 : lz < TZ ? 1 : 2;
      const int which = (nz * 3 + ny) * 3 + nx;
      const int x = bx + lx, y = by + ly, z = bz + lz;
      if (which == 13 || (unsigned)x >= (unsigned)g.W || (unsigned)y >= (unsigned)g.H ||
          (unsigned)z >= (unsigned)g.D)
        continue;
      const int v = x + y * g.W + z * WH;
      if (bit_of(J.rtouch2, J.dds[v]) || bit_of(J.rtouch1, J.das[v])) mine |= 1u << which;
    }
    mine = __reduce_or_sync(0xffffffffu, mine);
    if (lane_id() == 0 && mine) atomicOr(&found, mine);
    __syncthreads();
    if (threadIdx.x < 27 && (found >> threadIdx.x & 1u)) {
      const int q = threadIdx.x;
      const int u = t + (q % 3 - 1) + (q / 3 % 3 - 1) * ntx + (q / 9 - 1) * ntx * nty;
      if (atomicExch(J.tseen + u, (int)stamp) != (int)stamp) queue_push(queue, stamp, u, nt / 4);
    }
    __syncthreads();
    if (threadIdx.x == 0) queue.finished();
  }
}

// Global pointer jumping of both label arrays (ComputeDescendingManifold /
// ComputeAscendingManifold, :1514-1611), the two chains interleaved for
// memory-level parallelism.  A pointer that carries the root flag ends its chain:
// most paths end in their vertex's own tile and load nothing more (without the
// flag, every chain loads its root's entry once to see that it is one: the L1
// was 78 % busy).  Original field, in place: labels always point further along the
// path, so concurrent readers of a label being finalised see either value
// correctly, and a final label is recognised at its own, unflagged, entry.
// Every vertex is resolved (the reference resolves descending labels only next
// to original 2-saddles, the only places they are read).  Iterations are
// capped; hitting the cap sets the error word instead of spinning.  On the
// decompressed field it also writes each vertex's label-mismatch bits
// and changed-input bytes for the saddle pass.  kLater (decompressed field,
// a job's rounds after its first): the label-mismatch bits of a group change
// only with its labels, so the original roots are loaded only for groups
// whose labels changed, after the chase.
template <class T, bool kDec, bool kLater = false>
__global__ void __launch_bounds__(256, 4) k_jump2(const Job<T>* __restrict__ jobs,
                                               const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (kDec) {
    if (mf_skip(J.ctr)) return;
    if (blk == 0 && threadIdx.x == 0) J.ctr[C_TLIST] = 0;  // the listed tiles are done
  }
  // Original field: in place on ds / as.  Decompressed field: from the
  // tile-compressed pointers pdd / pda (kept for the next round) into dds / das.
  const int* a = kDec ? J.pdd : J.ds;
  const int* b = kDec ? J.pda : J.as;
  int* ra = kDec ? J.dds : J.ds;
  int* rb = kDec ? J.das : J.as;
  // Descriptor fields in registers: stores below could alias the descriptor.
  const unsigned* __restrict__ vchg = J.vchg;
  const int* __restrict__ ods = J.ds;
  const int* __restrict__ oas = J.as;
  uint8_t* __restrict__ dirtyv = J.dirtyv;
  uint8_t* __restrict__ mis = J.mis;
  int* err = J.ctr + C_ERROR;
  const int N = J.dim.N;
  const int cap_j = J.iter_cap;
  auto jump_one = [&](int v) {
    int u1 = a[v], u2 = b[v];
    // Decompressed field: this vertex's old labels, original roots and
    // change stamp, loaded while the chains are followed.
    int o1 = 0, o2 = 0, r1 = 0, r2 = 0;
    unsigned c0 = 0;
    if constexpr (kDec) {
      o1 = ra[v];
      o2 = rb[v];
      r1 = ods[v];
      r2 = oas[v];
      c0 = vchg[v >> 5] >> (v & 31);
    }
    int it = 2;  // the limit counts the end of a chain and the look at its root too
    while (it < cap_j && (u1 >= 0 || u2 >= 0)) {
      int w1 = u1, w2 = u2;
      if (u1 >= 0) w1 = a[u1];
      if (u2 >= 0) w2 = b[u2];
      // An entry that names itself is a final label (original field).
      u1 = w1 == u1 ? w1 | kRootFlag : w1;
      u2 = w2 == u2 ? w2 | kRootFlag : w2;
      ++it;
    }
    if (u1 >= 0 || u2 >= 0) {
      u1 = root_at_limit(a, u1);
      u2 = root_at_limit(b, u2);
    }
    if (u1 >= 0 || u2 >= 0 || cap_j < 2) atomicOr(err, kErrJump);
    u1 &= ~kRootFlag;
    u2 &= ~kRootFlag;
    if constexpr (kDec) {
      // For the saddle pass: label-mismatch bits, and whether an input of the
      // rows this vertex feeds changed since the previous computed round (its
      // value, either label, or the value of either label's root).  The
      // change bitset starts full, so the first round marks every vertex.
      const unsigned c1 = vchg[u1 >> 5] >> (u1 & 31), c2 = vchg[u2 >> 5] >> (u2 & 31);
      const bool d = (o1 != u1) | (o2 != u2) | ((c0 | c1 | c2) & 1u);
      dirtyv[v] = d ? (uint8_t)mf_byte(mf_stamp(J.ctr)) : (uint8_t)0;
      if (d) J.bdirty[v >> 10] = mf_stamp(J.ctr);
      mis[v] = (uint8_t)((u1 != r1) | (u2 != r2) << 1);
    }
    ra[v] = u1;
    rb[v] = u2;
  };
  int from = 0;  // the vertices that are left to the loop at the end
  if constexpr (kDec) {
    {
      // Four consecutive vertices per thread: one 16-byte load per array and
      // one 4-byte store per byte array, a quarter of the memory requests of
      // the vertex-per-thread loop, with eight chains interleaved.  A quad
      // with a changed-input byte stamps its 1024-id block (bdirty, read by
      // the saddle pass; its address is read where it is used: kept in a
      // register for the whole loop it costs spills).  Changed-input bytes
      // are the round's (mf_byte): a quad that is not followed leaves its
      // bytes, which then read as unchanged (or, when they are 255 rounds old,
      // as changed, which recomputes rows that have not changed).
      //
      // kLater: a vertex's label on a side can change only when its path
      // crosses a tile whose pointers this round recomputed, and every vertex
      // of a path carries the path's label.  So a quad none of whose old
      // labels is a root marked by k_direction_list (rtouch2 / rtouch1: the
      // old labels of the recomputed tiles' vertices) keeps its labels and
      // mismatch bits and has no changed input (a changed value, own or of a
      // root, lies in a recomputed tile too).
      const int stamp = mf_stamp(J.ctr);
      const unsigned st8 = mf_byte(stamp);
      // Four vertices' chains to their ends.
      auto chase = [&](int* u1, int* u2) {
        // One hop of every unfinished chain per iteration: the loads depend only
        // on their own chain, so they are all in flight at once.
        for (int it = 1; it < cap_j; ++it) {  // (the limit counts the look at the root too)
          bool more = false;
  #pragma unroll
          for (int k = 0; k < 4; ++k) more |= (u1[k] >= 0) | (u2[k] >= 0);
          if (!more) break;
          int w1[4], w2[4];
  #pragma unroll
          for (int k = 0; k < 4; ++k) {
            w1[k] = u1[k];
            w2[k] = u2[k];
            if (u1[k] >= 0) w1[k] = a[u1[k]];
            if (u2[k] >= 0) w2[k] = b[u2[k]];
          }
  #pragma unroll
          for (int k = 0; k < 4; ++k) {
            u1[k] = w1[k];
            u2[k] = w2[k];
          }
        }
        bool open = false;
  #pragma unroll
        for (int k = 0; k < 4; ++k) open |= (u1[k] >= 0) | (u2[k] >= 0);
        if (open) {
          open = false;
          for (int k = 0; k < 8; ++k)
            open |= root_at_limit(k < 4 ? a : b, k < 4 ? u1[k] : u2[k - 4]) >= 0;
        }
  #pragma unroll
        for (int k = 0; k < 4; ++k) {
          u1[k] &= ~kRootFlag;
          u2[k] &= ~kRootFlag;
        }
        if (open) atomicOr(err, kErrJump);
      };
      // Returns the quad's labels through u1 / u2 (the old ones when it is
      // not followed) and the old ones through o1 / o2 (-1 in a first round).
      auto quad = [&](int v0, int* u1, int* u2, int* o1, int* o2) {
        // A job's first round writes every label (its change bitset starts
        // full, and the stored labels may be another job's): no old labels.
        const int4 O1 = kLater ? *reinterpret_cast<const int4*>(ra + v0) : make_int4(-1, -1, -1, -1);
        const int4 O2 = kLater ? *reinterpret_cast<const int4*>(rb + v0) : make_int4(-1, -1, -1, -1);
        o1[0] = O1.x; o1[1] = O1.y; o1[2] = O1.z; o1[3] = O1.w;
        o2[0] = O2.x; o2[1] = O2.y; o2[2] = O2.z; o2[3] = O2.w;
        if constexpr (kLater) {
          unsigned hit = 0u;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            hit |= (J.rtouch2[o1[k] >> 5] >> (o1[k] & 31)) | (J.rtouch1[o2[k] >> 5] >> (o2[k] & 31));
          if (!(hit & 1u)) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              u1[k] = o1[k];
              u2[k] = o2[k];
            }
            return;
          }
        }
        const int4 A = *reinterpret_cast<const int4*>(a + v0);
        const int4 B = *reinterpret_cast<const int4*>(b + v0);
        int4 R1 = make_int4(0, 0, 0, 0), R2 = make_int4(0, 0, 0, 0);
        if constexpr (!kLater) {
          R1 = *reinterpret_cast<const int4*>(ods + v0);
          R2 = *reinterpret_cast<const int4*>(oas + v0);
        }
        const unsigned cw = vchg[v0 >> 5] >> (v0 & 31);
        u1[0] = A.x; u1[1] = A.y; u1[2] = A.z; u1[3] = A.w;
        u2[0] = B.x; u2[1] = B.y; u2[2] = B.z; u2[3] = B.w;
        chase(u1, u2);
        unsigned dv = 0;
        bool n1 = false, n2 = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned c1 = vchg[u1[k] >> 5] >> (u1[k] & 31);
          const unsigned c2 = vchg[u2[k] >> 5] >> (u2[k] & 31);
          n1 |= o1[k] != u1[k];
          n2 |= o2[k] != u2[k];
          const unsigned d = (o1[k] != u1[k]) | (o2[k] != u2[k]) | ((cw >> k | c1 | c2) & 1u);
          dv |= (d ? st8 : 0u) << (8 * k);
        }
        *reinterpret_cast<unsigned*>(dirtyv + v0) = dv;
        // Stores that would rewrite the stored value are skipped.  The
        // mismatch bits follow the labels alone (the original roots are
        // fixed), so a group whose labels did not change keeps last round's
        // bits.
        if (kLater ? (n1 || n2) : true) {
          if constexpr (kLater) {
            R1 = *reinterpret_cast<const int4*>(ods + v0);
            R2 = *reinterpret_cast<const int4*>(oas + v0);
          }
          const int r1[4] = {R1.x, R1.y, R1.z, R1.w}, r2[4] = {R2.x, R2.y, R2.z, R2.w};
          unsigned mv = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mv |= ((unsigned)(u1[k] != r1[k]) | (unsigned)(u2[k] != r2[k]) << 1) << (8 * k);
          *reinterpret_cast<unsigned*>(mis + v0) = mv;
        }
        if (n1) *reinterpret_cast<int4*>(ra + v0) = make_int4(u1[0], u1[1], u1[2], u1[3]);
        if (n2) *reinterpret_cast<int4*>(rb + v0) = make_int4(u2[0], u2[1], u2[2], u2[3]);
        if (dv) J.bdirty[v0 >> 10] = stamp;
      };
      // A light round: only the tiles listed by k_touched_tiles, a thread per
      // tile column (its four vertices' chains together).  Vertices without a
      // touched label keep their labels, as above.
      if (kLater && !J.ctr[C_JDENSE]) {
        const Dims g = J.dim;
        const int WH = g.W * g.H;
        const int ntx = (g.W + TX - 1) / TX, nty = (g.H + TY - 1) / TY;
        const int na = J.ctr[C_NAFF];
        for (int k = blk; k < na; k += nblk) {
          const int t = (int)(unsigned)J.tqueue[k];
          const int x = (t % ntx) * TX + (int)threadIdx.x % TX;
          const int y = ((t / ntx) % nty) * TY + (int)threadIdx.x / TX, z = (t / (ntx * nty)) * TZ;
          if (x >= g.W || y >= g.H) continue;
          const int v0 = x + y * g.W + z * WH;
          int u1[TZ], u2[TZ], o1[TZ], o2[TZ];
          unsigned in = 0u;
#pragma unroll
          for (int q = 0; q < TZ; ++q) {
            if (z + q < g.D) in |= 1u << q;
            o1[q] = in >> q & 1u ? ra[v0 + q * WH] : o1[0];
            o2[q] = in >> q & 1u ? rb[v0 + q * WH] : o2[0];
          }
          bool hit = false;
#pragma unroll
          for (int q = 0; q < TZ; ++q)
            hit |= (in >> q & 1u) && (bit_of(J.rtouch2, o1[q]) || bit_of(J.rtouch1, o2[q]));
          if (!hit) continue;
#pragma unroll
          for (int q = 0; q < TZ; ++q) {
            u1[q] = in >> q & 1u ? a[v0 + q * WH] : kRootFlag;
            u2[q] = in >> q & 1u ? b[v0 + q * WH] : kRootFlag;
          }
          chase(u1, u2);
#pragma unroll
          for (int q = 0; q < TZ; ++q) {
            if (!(in >> q & 1u)) continue;
            const int v = v0 + q * WH;
            const bool d = o1[q] != u1[q] || o2[q] != u2[q] || bit_of(vchg, v) ||
                           bit_of(vchg, u1[q]) || bit_of(vchg, u2[q]);
            dirtyv[v] = d ? (uint8_t)st8 : (uint8_t)0;
            if (d) J.bdirty[v >> 10] = stamp;
            if (o1[q] != u1[q] || o2[q] != u2[q]) {
              mis[v] = (uint8_t)((u1[q] != ods[v]) | (u2[q] != oas[v]) << 1);
              ra[v] = u1[q];
              rb[v] = u2[q];
            }
          }
        }
        return;
      }
      const int nq = N >> 2;
      const int qstride = nblk * blockDim.x;
      for (int q = blk * blockDim.x + threadIdx.x; q < nq; q += qstride) {
        int u1[4], u2[4], o1[4], o2[4];
        quad(q << 2, u1, u2, o1, o2);
      }
      from = nq << 2;
    }
  }
  if constexpr (!kDec) {
    // Four consecutive vertices per thread where the labels' arrays (a caller's
    // own, in extremz_classify) allow 16-byte accesses.
    if (((reinterpret_cast<uintptr_t>(ra) | reinterpret_cast<uintptr_t>(rb)) & 15) == 0) {
      const int nq = N >> 2, qstride = nblk * blockDim.x;
      for (int q = blk * blockDim.x + threadIdx.x; q < nq; q += qstride) {
        const int4 A = reinterpret_cast<const int4*>(ra)[q], B = reinterpret_cast<const int4*>(rb)[q];
        int u[8] = {A.x, A.y, A.z, A.w, B.x, B.y, B.z, B.w};
        // As jump_one, for eight chains; the limit counts the end of a chain and
        // the look at its root too.
        bool open = true;
        for (int it = 2;; ++it) {
          open = false;
#pragma unroll
          for (int k = 0; k < 8; ++k) open |= u[k] >= 0;
          if (!open || it >= cap_j) break;
          int w[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) w[k] = u[k] >= 0 ? (k < 4 ? a : b)[u[k]] : u[k];
#pragma unroll
          for (int k = 0; k < 8; ++k) u[k] = w[k] == u[k] ? w[k] | kRootFlag : w[k];
        }
        if (open) {
          open = false;
#pragma unroll
          for (int k = 0; k < 8; ++k) open |= root_at_limit(k < 4 ? a : b, u[k]) >= 0;
        }
        if (open || cap_j < 2) atomicOr(err, kErrJump);
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] &= ~kRootFlag;
        reinterpret_cast<int4*>(ra)[q] = make_int4(u[0], u[1], u[2], u[3]);
        reinterpret_cast<int4*>(rb)[q] = make_int4(u[4], u[5], u[6], u[7]);
      }
      from = nq << 2;
    }
  }
  const int stride = nblk * blockDim.x;
  for (int v = from + blk * blockDim.x + threadIdx.x; v < N; v += stride) jump_one(v);
}

// ---------------------------------------------------------------------------
// Ordered compaction of the critical-point lists (ExtractCP :1694-1741, here in
// ascending vertex id).  Pass 1 counts per 1024-vertex block, pass 2 scans the
// block counts, pass 3 writes.
// ---------------------------------------------------------------------------
constexpr int kCpBlock = 1024;
static_assert(kCpBlockJ == kCpBlock, "the jump's flags cover the CP-list blocks");

// One warp per 1024-id block, each lane 32 consecutive ids: the types come in
// as two 16-byte loads per lane (one coalesced kilobyte per warp), where one
// 1024-thread block per 1024 ids spent its time scheduling blocks.
constexpr int kCpWarps = 8;  // warps (1024-id blocks) per CTA

// The CP-list membership bits of the lane's 32 ids, one word per list: types 2
// and 3, 1 and 3, 4, 0 (5 and -1 are in none).  Four types at a time: a type's
// three low bits, one per byte, decide each list, and a multiplication gathers
// the four answers.
__device__ __forceinline__ void cp_lane_bits(const int8_t* __restrict__ otype, int N, int v0,
                                             unsigned bits[4]) {
  unsigned w[8];
  if (v0 + 32 <= N) {
    const uint4 q0 = *reinterpret_cast<const uint4*>(otype + v0);
    const uint4 q1 = *reinterpret_cast<const uint4*>(otype + v0 + 16);
    w[0] = q0.x; w[1] = q0.y; w[2] = q0.z; w[3] = q0.w;
    w[4] = q1.x; w[5] = q1.y; w[6] = q1.z; w[7] = q1.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      w[k] = 0u;
      for (int j = 0; j < 4; ++j) {
        const int v = v0 + 4 * k + j;
        w[k] |= (v < N ? (unsigned)(uint8_t)otype[v] : 0xffu) << (8 * j);
      }
    }
  }
#pragma unroll
  for (int l = 0; l < 4; ++l) bits[l] = 0u;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const unsigned b0 = w[k], b1 = w[k] >> 1, b2 = w[k] >> 2, one = 0x01010101u;
    const unsigned in[4] = {b1 & ~b2 & one, b0 & ~b2 & one, b2 & ~b1 & ~b0 & one,
                            ~(b2 | b1 | b0) & one};
#pragma unroll
    for (int l = 0; l < 4; ++l) bits[l] |= (in[l] * 0x01020408u >> 24 & 15u) << (4 * k);
  }
}

// Also counts the entries the original rows will hold (lists 4 and 5): a
// 2-saddle's row has one entry per upper neighbour, a 1-saddle's one per lower
// neighbour (rows keep repeated labels; the persistence filter thr can only
// drop entries, so with thr > 0 this is an upper bound).
__global__ void __launch_bounds__(32 * kCpWarps) k_cp_count(const int8_t* __restrict__ otype,
                                                           const uint16_t* __restrict__ olm,
                                                           Dims g, int nb,
                                                           int* __restrict__ bcount) {
  const int b = blockIdx.x * kCpWarps + (int)(threadIdx.x >> 5);
  if (b >= nb) return;  // whole warps leave together
  const int v0 = b * kCpBlock + (int)lane_id() * 32;
  unsigned bits[4];
  cp_lane_bits(otype, g.N, v0, bits);
  int e2 = 0, e1 = 0;
  if ((bits[0] | bits[1]) != 0u) {
    int x, y, z;
    coords(v0, g, x, y, z);
    if (v0 + 32 <= g.N && x > 0 && x + 31 < g.W - 1 && y > 0 && y < g.H - 1 && z > 0 && z < g.D - 1) {
      // Off the faces every vertex has 14 neighbours; the masks come in together,
      // two to a word.
      int low2 = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint4 q = reinterpret_cast<const uint4*>(olm + v0)[k];
        const unsigned pair[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const unsigned p2 = bits[0] >> (8 * k + 2 * j) & 3u, p1 = bits[1] >> (8 * k + 2 * j) & 3u;
          low2 += __popc(pair[j] & ((p2 & 1u) * 0xffffu | (p2 >> 1) * 0xffff0000u));
          e1 += __popc(pair[j] & ((p1 & 1u) * 0xffffu | (p1 >> 1) * 0xffff0000u));
        }
      }
      e2 = kNumDirs * __popc(bits[0]) - low2;
    } else {
      for (int k = 0; k < 32; ++k) {
        if (((bits[0] | bits[1]) >> k) & 1u) {
          const int nvalid = __popc(valid_mask(boundary_code(x, y, z, g.W, g.H, g.D)));
          const int lower = __popc((unsigned)olm[v0 + k]);
          if ((bits[0] >> k) & 1u) e2 += nvalid - lower;
          if ((bits[1] >> k) & 1u) e1 += lower;
        }
        if (++x == g.W) {
          x = 0;
          if (++y == g.H) {
            y = 0;
            ++z;
          }
        }
      }
    }
  }
  int c[6] = {__popc(bits[0]), __popc(bits[1]), __popc(bits[2]), __popc(bits[3]), e2, e1};
#pragma unroll
  for (int l = 0; l < 6; ++l) {
    for (int o = 16; o > 0; o >>= 1) c[l] += __shfl_xor_sync(0xffffffffu, c[l], o);
    if (lane_id() == 0) bcount[l * nb + b] = c[l];
  }
}

// Exclusive scan of gridDim.x lists of nb counts in place (a block per list),
// list totals to totals[0 .. gridDim.x).  The CP lists use totals = ctr + C_NS2.
// Each thread takes up to 32 consecutive counts per pass, no more than it takes to
// cover the list.  cursor (optional, one list): a second copy of the scanned
// counts.
__global__ void __launch_bounds__(1024) k_scan_lists(int* __restrict__ bcount, int nb, int* totals,
                                                     int* __restrict__ cursor) {
  constexpr int kPer = 32;
  __shared__ int carry;
  __shared__ int warp_sums[32];
  const int l = blockIdx.x;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  int* c = bcount + (long long)l * nb;
  const int per = min(kPer, (nb + 1023) / 1024);
  for (int base = 0; base < nb; base += 1024 * per) {
    const int i0 = base + (int)threadIdx.x * per;
    int x[kPer];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      x[k] = k < per && i0 + k < nb ? c[i0 + k] : 0;
      sum += x[k];
    }
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane_id() >= (unsigned)o) incl += y;
    }
    if (lane_id() == 31) warp_sums[threadIdx.x / 32] = incl;
    __syncthreads();
    if (threadIdx.x < 32) {
      int w = warp_sums[threadIdx.x], wi = w;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane_id() >= (unsigned)o) wi += y;
      }
      warp_sums[threadIdx.x] = wi - w;
    }
    __syncthreads();
    int run = carry + warp_sums[threadIdx.x / 32] + incl - sum;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      if (k < per && i0 + k < nb) {
        c[i0 + k] = run;
        if (cursor) cursor[i0 + k] = run;
      }
      run += x[k];
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry = run;
    __syncthreads();
  }
  if (threadIdx.x == 0) totals[l] = carry;
}

// Exclusive scan in place of lists of n counts (list l at c + l * n, one per
// blockIdx.y) for lists too long for one block: the sum of every 1024-count
// chunk (k_chunk_sums, into sums + l * gridDim.x), a scan of the sums with the
// list totals (k_scan_lists), then each chunk scanned from its offset
// (k_chunk_scan).
__global__ void __launch_bounds__(1024) k_chunk_sums(const int* __restrict__ c, int n,
                                                     int* __restrict__ sums) {
  __shared__ int ws[32];
  c += (long long)blockIdx.y * n;
  sums += (long long)blockIdx.y * gridDim.x;
  const int i = blockIdx.x * 1024 + threadIdx.x;
  int x = i < n ? c[i] : 0;
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if (lane_id() == 0) ws[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    int y = ws[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    if (threadIdx.x == 0) sums[blockIdx.x] = y;
  }
}

__global__ void __launch_bounds__(1024) k_chunk_scan(int* __restrict__ c, int n,
                                                     const int* __restrict__ offs,
                                                     int* __restrict__ cursor) {
  __shared__ int ws[32];
  c += (long long)blockIdx.y * n;
  offs += (long long)blockIdx.y * gridDim.x;
  const int i = blockIdx.x * 1024 + threadIdx.x;
  const int x = i < n ? c[i] : 0;
  int incl = x;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane_id() >= (unsigned)o) incl += y;
  }
  if (lane_id() == 31) ws[threadIdx.x >> 5] = incl;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int w = ws[threadIdx.x];
    int wi = w;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane_id() >= (unsigned)o) wi += y;
    }
    ws[threadIdx.x] = wi - w;
  }
  __syncthreads();
  if (i < n) {
    const int at = offs[blockIdx.x] + ws[threadIdx.x >> 5] + incl - x;
    c[i] = at;
    if (cursor) cursor[i] = at;
  }
}

// The four lists, and ext[v] = the index of a maximum or minimum v in its list
// (computeMaxIndex / computeMinIndex :1928-1939 share one array).
__global__ void __launch_bounds__(32 * kCpWarps) k_cp_write(const int8_t* __restrict__ otype,
                                                           int N, int nb,
                                                           const int* __restrict__ boff,
                                                           int* sad2, int* sad1, int* maxima,
                                                           int* minima, int* __restrict__ ext) {
  const int b = blockIdx.x * kCpWarps + (int)(threadIdx.x >> 5);
  if (b >= nb) return;
  const int v0 = b * kCpBlock + (int)lane_id() * 32;
  unsigned bits[4];
  cp_lane_bits(otype, N, v0, bits);
  // Word by word, a vertex per lane: a list's entries of 32 ids are consecutive,
  // so the stores are coalesced (a lane writing its own 32 ids' entries spread
  // every store over 32 places: 0.40 ms at 512^3, now 0.34).
  int* outs[4] = {sad2, sad1, maxima, minima};
  int pos[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) pos[l] = boff[l * nb + b];
  const unsigned lt = (1u << lane_id()) - 1u;
  for (int j = 0; j < 32; ++j) {
    const int v = b * kCpBlock + 32 * j + (int)lane_id();
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const unsigned word = __shfl_sync(0xffffffffu, bits[l], j);
      if (word >> lane_id() & 1u) {
        const int at = pos[l] + __popc(word & lt);
        outs[l][at] = v;
        if (l >= 2) ext[v] = at;
      }
      pos[l] += __popc(word);
    }
  }
}

// ---------------------------------------------------------------------------
// Saddle rows: findAscPaths (:1832-1926) and findDescPaths (:1956-2049).
// Row i belongs to the i-th ORIGINAL saddle for both fields.  Only [0, count)
// and the count are written, so entries past a shorter row keep their last
// value, as in the reference.
// ---------------------------------------------------------------------------
// The rows of one side of the original field.  A saddle's neighbours on the
// side are the set bits of the direction mask that the classification left
// (upper neighbours of a 2-saddle, lower ones of a 1-saddle): 4.3 of 14 on
// average and 8.2 in the fullest lane of a warp, so the passes below go over
// set bits in groups of four, up to the warp's fullest lane, and no neighbour
// value is read or compared.  Bound by the label and value gathers and by the
// issue of the per-entry work: 1.34 ms for the 22 M 2-saddles of the 512^3
// benchmark field, 2.38 ms when it went over all 14 directions and compared
// their values.
// kNan: the field holds a NaN (a variant of its own: the look for one in every field
// cost 4 %).
template <class T, bool kAsc, bool kNan = false>
__global__ void __launch_bounds__(256, 4) k_rows(Job<T> J) {
  __shared__ int off[kNumDirs];
  fill_offsets(off, J.dim);
  __syncthreads();
  const T* __restrict__ a = J.f;
  const int* __restrict__ lab = kAsc ? J.ds : J.as;
  const int* __restrict__ sad = kAsc ? J.sad2 : J.sad1;
  const int ns = J.ctr[kAsc ? C_NS2 : C_NS1];
  int* __restrict__ rows = kAsc ? J.orow2 : J.orow1;
  const int stride = gridDim.x * blockDim.x;
  const Dims g = J.dim;
  for (int base = blockIdx.x * blockDim.x; base < ns; base += stride) {  // uniform per warp
    const int i = base + threadIdx.x;
    const bool act = i < ns;
    const int s = act ? sad[i] : 0;
    const T sv = a[s];
    unsigned side = act ? J.olm[s] : 0u;
    if (kAsc && act) {
      int x, y, z;
      coords(s, g, x, y, z);
      side = (unsigned)valid_mask(boundary_code(x, y, z, g.W, g.H, g.D)) & ~side;
      // Next to a NaN a path may end at a vertex that is no maximum, whose index
      // in ext is 0 then: in a field without maxima no row names one.
      if (kNan) side = J.ctr[C_NMAX] ? drop_nans(a, off, s, side) : 0u;
      J.smask2[i] = (uint16_t)side;
    }
    const int pmax = (int)__reduce_max_sync(0xffffffffu, __popc(side));
    // The reference sorts each row (insertionSort :1795-1811, descending, for
    // ascending rows; reversed_insertionSort :1813-1829, ascending, for
    // descending rows) by (value, label).  What is read back from an original
    // row is its count, its first and last entry in that order
    // (get_wrong_index_max / _min) and the set of extrema it names
    // (findLargestSaddlePerMax / _Min, get_wrong_index_saddles(_join), where a
    // repeated label adds nothing: only the row decides).  So the row is not
    // sorted: the first and last entry come from one pass, and the entries
    // are kept in direction order as extremum indices, a repeated label's
    // entry as -1.
    int lb[16], mp[16];
    unsigned keep = 0u, dup = 0u;  // by position among the side's neighbours
    int fl = -1, ll = -1;
    T fv = T(0), lv = T(0);
    unsigned rest = side;
#pragma unroll
    for (int h = 0; h < 16; h += 4) {
#pragma unroll
      for (int q = h; q < h + 4; ++q) lb[q] = mp[q] = -1;
      if (h >= pmax) continue;  // uniform per warp
#pragma unroll
      for (int q = h; q < h + 4; ++q) {
        if (rest) lb[q] = lab[s + off[__ffs((int)rest) - 1]];
        rest &= rest - 1u;
      }
      T val[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) val[q] = lb[h + q] >= 0 ? a[lb[h + q]] : T(0);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (lb[h + q] >= 0) mp[h + q] = J.ext[lb[h + q]];
#pragma unroll
      for (int q = h; q < h + 4; ++q) {
        const T v = val[q - h];
        if (lb[q] < 0 || (kAsc && !(tabs(T(v - sv)) >= J.thr))) continue;
        bool again = false;  // an earlier kept entry has the label
#pragma unroll
        for (int e = 0; e < q; ++e) again |= lb[e] == lb[q] && (keep >> e & 1u);
        keep |= 1u << q;
        if (again) {
          dup |= 1u << q;
          continue;
        }
        const bool first = fl < 0 || (kAsc ? above(v, lb[q], fv, fl) : below(v, lb[q], fv, fl));
        const bool last = ll < 0 || (kAsc ? below(v, lb[q], lv, ll) : above(v, lb[q], lv, ll));
        if (first) { fv = v; fl = lb[q]; }
        if (last) { lv = v; ll = lb[q]; }
      }
    }
    const int cnt = __popc(keep);
    int* out = rows + (long long)i * kRowStride;
    if (act) {
      (kAsc ? J.ocnt2 : J.ocnt1)[i] = (uint8_t)cnt;
      (kAsc ? J.oend2 : J.oend1)[i] =
          make_int4(fl, ll, fl >= 0 ? J.ext[fl] : -1, ll >= 0 ? J.ext[ll] : -1);
    }
    // Per kept entry, at its position among the kept ones: the first four in
    // the compact copy, the rest in the row.  And the first pass of
    // findLargestSaddlePerMax / findSmallestSaddlePerMin (:4890-4940) over
    // the row: each named extremum's largest (smallest) saddle key, and the
    // number of rows naming it, for the per-extremum entry lists of the
    // incremental wrong-saddle scan (filled by k_extreme_saddle).  Lanes
    // naming the same extremum share one atomic; a read first skips most key
    // atomics (the key only moves one way).
    using KK = typename KeyOf<T>::K;
    const KK key = KeyOf<T>::enc(sv + T(0));  // -0 and +0 compare equal
    int* mcount = kAsc ? J.moff2 : J.moff1;
    // Entries that count: kept and not a repeat.
#pragma unroll
    for (int q = 0; q < kNumDirs; ++q)
      if (!(keep & ~dup & 1u << q)) mp[q] = -1;
    int m0 = -1, m1 = -1, m2 = -1, m3 = -1;
    int pos = 0;
#pragma unroll
    for (int h = 0; h < 16; h += 4) {
      if (h >= pmax) continue;
#pragma unroll
      for (int q = h; q < h + 4; ++q) {
        if (q >= kNumDirs) continue;
        const unsigned grp = __match_any_sync(0xffffffffu, mp[q]);
        if (mp[q] >= 0 && (grp & ((1u << lane_id()) - 1u)) == 0u) atomicAdd(mcount + mp[q], __popc(grp));
        if (keep >> q & 1u) {
          if (q < 4 || pos < 4) {  // pos <= q
            m0 = pos == 0 ? mp[q] : m0;
            m1 = pos == 1 ? mp[q] : m1;
            m2 = pos == 2 ? mp[q] : m2;
            m3 = pos == 3 ? mp[q] : m3;
          } else {
            out[pos] = mp[q];
          }
          ++pos;
        }
      }
    }
    if (act) (kAsc ? J.orm2 : J.orm1)[i] = make_int4(m0, m1, m2, m3);
    // Then the key reads, four at a time, and the atomics they call for.
#pragma unroll
    for (int h = 0; h < 16; h += 4) {
      if (h >= pmax) continue;
      KK cur[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) cur[q] = mp[h + q] >= 0 ? J.ext_key[mp[h + q]] : KK(0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (mp[h + q] < 0 || !(kAsc ? key > cur[q] : key < cur[q])) continue;
        if (kAsc) atomicMax(J.ext_key + mp[h + q], key);
        else atomicMin(J.ext_key + mp[h + q], key);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Largest saddle per maximum / smallest per minimum on the ORIGINAL field
// (findLargestSaddlePerMax / findSmallestSaddlePerMin :4890-4940): the CSR
// max->saddle table is never materialised; every (row, entry) pair votes.
// k_rows selects the extreme value key per extremum (and counts the entries
// naming it); this pass selects the extreme id at that key and files the
// entries into the per-extremum lists (cursors start at the scanned offsets).
// ---------------------------------------------------------------------------
template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_extreme_saddle(Job<T> J) {
  using K = typename KeyOf<T>::K;
  const int ns = J.ctr[kMax ? C_NS2 : C_NS1];
  const int* sad = kMax ? J.sad2 : J.sad1;
  const int* rows = kMax ? J.orow2 : J.orow1;
  const uint8_t* ocnt = kMax ? J.ocnt2 : J.ocnt1;
  int* cur = J.aff;  // scratch until the first wrong-saddle scan
  int* ent = kMax ? J.ment2 : J.ment1;
  const int stride = gridDim.x * blockDim.x;
  // Uniform per warp: lanes naming the same extremum (neighbouring saddles
  // usually do) share one cursor atomic.
  for (int base = blockIdx.x * blockDim.x; base < ns; base += stride) {
    const int i = base + threadIdx.x;
    const int cnt = i < ns ? ocnt[i] : 0;
    const int s = i < ns ? sad[i] : 0;
    const K key = KeyOf<T>::enc(J.f[s] + T(0));  // -0 and +0 compare equal
    const int* row = rows + (long long)(i < ns ? i : 0) * kRowStride;
    // The first four entries as extremum indices from the compact copy
    // (k_rows), longer rows' tails from the row (stored as extremum indices).
    const int4 m4 = i < ns ? (kMax ? J.orm2 : J.orm1)[i] : make_int4(-1, -1, -1, -1);
    const int pmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    // Seven entries at a time, each step's loads and atomics issued together
    // (a load after an atomic would wait for it).  A row names an extremum in
    // one entry only (a repeat is -1), as counted by k_rows.
#pragma unroll
    for (int h = 0; h < kNumDirs; h += 7) {
      if (h >= pmax) break;
      int m[7];
#pragma unroll
      for (int q = 0; q < 7; ++q) {
        const int p = h + q;
        m[q] = p >= cnt ? -1 : p == 0 ? m4.x : p == 1 ? m4.y : p == 2 ? m4.z : p == 3 ? m4.w : row[p];
      }
      unsigned grp[7];
#pragma unroll
      for (int q = 0; q < 7; ++q) grp[q] = __match_any_sync(0xffffffffu, m[q]);
      int at[7];
#pragma unroll
      for (int q = 0; q < 7; ++q)
        at[q] = (m[q] >= 0 && (grp[q] & ((1u << lane_id()) - 1u)) == 0u)
                    ? atomicAdd(cur + m[q], __popc(grp[q])) : 0;
      K ek[7];
#pragma unroll
      for (int q = 0; q < 7; ++q) ek[q] = m[q] >= 0 ? J.ext_key[m[q]] : K(0);
#pragma unroll
      for (int q = 0; q < 7; ++q) {
        const unsigned below = grp[q] & ((1u << lane_id()) - 1u);
        const int pos = __shfl_sync(0xffffffffu, at[q], __ffs(grp[q]) - 1) + __popc(below);
        if (m[q] < 0) continue;
        if (ek[q] == key) {
          if (kMax) atomicMax(J.largest + m[q], s);
          else atomicMin(J.smallest + m[q], s);
        }
        ent[pos] = i * kRowStride + h + q;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Proposals and their application.
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T midpoint_delta(const Job<T>& J, int i) {
  const T gi = J.g[i];
  return ((J.f[i] - J.bound) + gi) / T(2) - gi;
}
template <class T>
__device__ __forceinline__ T step_delta(const Job<T>& J, int i) {
  return J.edit_type == 1 ? midpoint_delta(J, i) : -J.bound / T(J.q);
}

// Atomic max into the proposal buffer (swap / swap1 / atomicCASDouble
// :2643-2691).  The thread that lifts a vertex off the sentinel records it.
template <class T>
__device__ __forceinline__ void propose(const Job<T>& J, int i, T d) {
  using K = typename KeyOf<T>::K;
  const K k = KeyOf<T>::enc(d);
  const K old = atomicMax(J.delta + i, k);
  if (old == J.sentinel_key && k > old) {
    const int slot = atomicAdd(J.ctr + C_TOUCHED, 1);
    J.touched[slot] = i;
  }
}

// Up to kN proposals of every lane of a warp (bits of `which`): the atomics go out
// together, then the vertices that left the sentinel are listed with one atomic
// per warp.  (With one per thread, half a million of them queued on the same
// counter: 235 us for the first proposals of the 256^3 benchmark field.)
template <class T, int kN>
__device__ __forceinline__ void propose_warp(const Job<T>& J, const int* at, const T* d, unsigned which) {
  using K = typename KeyOf<T>::K;
  K old[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k)
    old[k] = (which >> k & 1u) ? atomicMax(J.delta + at[k], KeyOf<T>::enc(d[k])) : K(0);
  unsigned fresh = 0u;
#pragma unroll
  for (int k = 0; k < kN; ++k)
    if ((which >> k & 1u) && old[k] == J.sentinel_key && KeyOf<T>::enc(d[k]) > old[k]) fresh |= 1u << k;
  const int n = __popc(fresh);
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane_id() >= (unsigned)o) incl += y;
  }
  int slot = 0;
  if (lane_id() == 31 && incl) slot = atomicAdd(J.ctr + C_TOUCHED, incl);
  slot = __shfl_sync(0xffffffffu, slot, 31) + incl - n;
#pragma unroll
  for (int k = 0; k < kN; ++k)
    if (fresh >> k & 1u) J.touched[slot++] = at[k];
}

// c_loop(0..2) (:2887-3055) over the mismatch list.
template <class T>
__global__ void __launch_bounds__(256) k_propose_cp(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const int n = J.ctr[C_MM];
  const int stride = nblk * blockDim.x;
  const Dims g = J.dim;
  const int WH = g.W * g.H;
  for (int base = blk * blockDim.x; base < n; base += stride) {  // uniform per warp
    const int e = base + threadIdx.x;
    const int ent = e < n ? J.mm[e] : 0;
    const int v = ent & ((1 << kCatShift) - 1);
    const int cat = (unsigned)ent >> kCatShift;
    int x, y, z;
    coords(v, g, x, y, z);
    // Neighbours in direction order (the reference's scan order), visited
    // through static indices so that the values stay in registers and their
    // loads go out together.
    const int valid = e < n ? valid_mask(boundary_code(x, y, z, g.W, g.H, g.D)) : 0;
    const int ot = J.otype[v];
    const T gv = J.g[v];
    const bool need_g = (cat & kCatSaddle) || ((cat & kCatMax) && ot == 4);
    T gn[kNumDirs];
#pragma unroll
    for (int d = 0; d < kNumDirs; ++d)
      gn[d] = (need_g && (valid >> d & 1)) ? J.g[v + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH] : T(0);
    // The proposals of c_loop(1), slot 0, and c_loop(0), slot 1.
    int at[4] = {v, v, v, v};
    T dl[4];
    unsigned which = 0u;
    if (cat & kCatMin) {  // c_loop(1) (:2965-3039)
      if (ot != 0) {
        T fn[kNumDirs];
#pragma unroll
        for (int d = 0; d < kNumDirs; ++d)
          fn[d] = (valid >> d & 1) ? J.f[v + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH] : T(0);
        int S = v;
        T sval = J.f[v];
#pragma unroll
        for (int d = 0; d < kNumDirs; ++d) {
          const int r = v + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH;
          if ((valid >> d & 1) && below(fn[d], r, sval, S)) { S = r; sval = fn[d]; }
        }
        const T gs = J.g[S];
        dl[0] = J.edit_type == 1 ? ((sval - J.bound) + gs) / T(2) - gs : -J.bound / T(J.q);
        if (!(gv > gs || (gv == gs && v > S))) {
          at[0] = S;
          which |= 1u;
        }
      } else {
        dl[0] = step_delta(J, v);
        which |= 1u;
      }
    }
    if (cat & kCatMax) {  // c_loop(0) (:2890-2963)
      if (ot != 4) {
        which |= 2u;
      } else {
        T lval = gv;
#pragma unroll
        for (int d = 0; d < kNumDirs; ++d) {
          const int r = v + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH;
          if ((valid >> d & 1) && above(gn[d], r, lval, at[1])) { at[1] = r; lval = gn[d]; }
        }
        if (at[1] != v) which |= 2u;
      }
      if (which & 2u) dl[1] = step_delta(J, at[1]);
    }
    propose_warp<T, 2>(J, at, dl, which);
    // c_loop(2) -> fix_saddle_local (:2804-2884): the original's lower neighbours
    // that are not lower now, four at a time, and the vertex itself when it has
    // lower neighbours it should not have.
    unsigned rest = 0u;
    if (cat & kCatSaddle) {
      int dm = 0;
#pragma unroll
      for (int d = 0; d < kNumDirs; ++d) {
        const int r = v + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH;
        if ((valid >> d & 1) && (gn[d] < gv || (gn[d] == gv && r < v))) dm |= 1 << d;
      }
      const int om = J.olm[v];
      rest = (unsigned)(valid & om & ~dm) | ((dm & ~om) ? 1u << kNumDirs : 0u);
    }
    while (__any_sync(0xffffffffu, rest != 0u)) {
      which = 0u;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        at[q] = v;
        if (rest) {
          const int d = __ffs((int)rest) - 1;
          if (d < kNumDirs) at[q] = v + ddx(d) + ddy(d) * g.W + ddz(d) * WH;
          which |= 1u << q;
        }
        rest &= rest - 1u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) dl[q] = (which >> q & 1u) ? step_delta(J, at[q]) : T(0);
      propose_warp<T, 4>(J, at, dl, which);
    }
  }
}

// applyDeltaBuffer (:3061-3111) over the vertices that received a proposal;
// the proposal buffer is reset to the sentinel on the way (init_delta).
template <class T>
__global__ void __launch_bounds__(256) k_apply(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const bool odd = J.ctr[C_DEPOCH] & 1;
  int* dirty = odd ? J.dirty1 : J.dirty;
  unsigned* bits = odd ? J.dbits1 : J.dbits;
  const int n = J.ctr[C_TOUCHED];
  const int stride = nblk * blockDim.x;
  for (int base = blk * blockDim.x; base < n; base += stride) {  // uniform per warp
    const int e = base + threadIdx.x;
    int v = 0, x = 0, y = 0, z = 0;
    bool fresh = false, changed = false;  // changed, and not in the dirty list yet
    if (e < n) {
      v = J.touched[e];
      const T d = KeyOf<T>::dec(J.delta[v]);
      J.delta[v] = J.sentinel_key;
      const T fv = J.f[v];
      const T g0 = J.g[v];
      T gv = g0;
      if (d == J.sentinel) {
      } else if (J.edit_type == 0) {
        const int c = J.counter[v];
        if (c < J.q - 1 && tabs(T(fv - (gv + d))) <= J.bound) {
          gv += d;
          J.counter[v] = c + 1;
        } else {
          J.counter[v] = J.q;
          gv = fv - J.bound;
        }
      } else {
        if (tabs(T(fv - (gv + d))) <= J.bound) gv += d;
        else gv = fv - J.bound;
      }
      if (KeyOf<T>::enc(gv) != KeyOf<T>::enc(g0)) {
        J.g[v] = gv;
        J.ctr[C_CHANGED] = 1;
        const int w = v >> 5;
        const unsigned bit = 1u << (v & 31);
        fresh = !(atomicOr(bits + w, bit) & bit);
        atomicOr(J.vchg + w, bit);
        atomicOr(J.wchg2 + w, bit);
        if (J.join_rows) atomicOr(J.wchg1 + w, bit);
        if (J.edited) atomicOr(J.edited + w, bit);
        coords(v, J.dim, x, y, z);
        changed = true;
      }
    }
    mark_tiles(J.tdirty, J.cand_next, J.ctr + C_TLIST, J.dim, x, y, z, changed);
    const int slot = warp_append(J.ctr + C_DIRTY, fresh, 0xffffffffu);
    if (slot >= 0) dirty[slot] = v;
  }
}

// ---------------------------------------------------------------------------
// Wrong manifold neighbours (get_wrong_split_neighbors / get_wrong_join_neighbors
// :2400-2513) in the canonical order "saddles in ascending id": saddle s flags
// its first candidate neighbour not flagged by a smaller saddle.
//
// Candidates of s: valid neighbours r (direction order) with r above s in the
// decompressed field and dds[r] != ds[r] (split), or below and das[r] != as[r]
// (join).  Resolution runs in rounds: every unresolved saddle votes (atomic
// max of (round << 32) | ~s) on each of its remaining candidates; a saddle
// commits its first remaining candidate when its own vote won, i.e. no smaller
// unresolved saddle can still take it.  The smallest unresolved saddle always
// commits, and a larger one never takes what a smaller one could still take,
// so the result equals the sequential greedy.
// ---------------------------------------------------------------------------
// Candidate lists this short are resolved by one block (k_wn_resolve) alone.
constexpr int kWnBlockMax = 4096;

template <class T, bool kSplit>
__device__ __forceinline__ int wn_candidates(const Job<T>& J, int s, int* ids) {
  const int n = neighbours(s, J.dim, ids, nullptr);
  const T sv = J.g[s];
  int k = 0;
  for (int j = 0; j < n; ++j) {
    const int r = ids[j];
    const T rv = J.g[r];
    const bool side = kSplit ? above(rv, r, sv, s) : below(rv, r, sv, s);
    const bool wrong = kSplit ? (J.dds[r] != J.ds[r]) : (J.das[r] != J.as[r]);
    if (side && wrong) ids[k++] = r;
  }
  return k;
}

// Row order of the decompressed rows: "comes first in the row" is descending
// for ascending rows, ascending else.
template <class T, bool kSplit>
__device__ __forceinline__ bool row_first(T v, int m, T bv, int bm) {
  return kSplit ? above(v, m, bv, bm) : below(v, m, bv, bm);
}

template <class T, bool kSplit>
__device__ __noinline__ int row_entry_k(const Job<T>& J, int s, int k) {
  const int* lab = kSplit ? J.dds : J.das;
  int ids[kNumDirs];
  const int n = neighbours(s, J.dim, ids, nullptr);
  const T sv = J.g[s];
  int ml[kNumDirs];
  T mv[kNumDirs];
  int cnt = 0;
  for (int j = 0; j < n; ++j) {
    const int r = ids[j];
    const T rv = J.g[r];
    if (kSplit ? above(rv, r, sv, s) : below(rv, r, sv, s)) {
      const int m = lab[r];
      const T v = J.g[m];
      if (!kSplit || tabs(T(v - sv)) >= J.thr) {
        ml[cnt] = m;
        mv[cnt] = v;
        ++cnt;
      }
    }
  }
  for (int a = 0; a < cnt; ++a) {
    int before = 0, same = 0;
    for (int b = 0; b < cnt; ++b) {
      before += row_first<T, kSplit>(mv[b], ml[b], mv[a], ml[a]);
      same += ml[b] == ml[a];
    }
    if (before <= k && k < before + same) return ml[a];
  }
  return -1;
}

// The directions of saddle s's neighbours on the side in the decompressed field.
template <class T, bool kSplit>
__device__ __noinline__ unsigned side_of(const Job<T>& J, int s) {
  const T* __restrict__ gv = J.g;
  const T sv = __ldg(gv + s);
  unsigned side = 0u;
  const Dims g = J.dim;
  const int WH = g.W * g.H;
  int x, y, z;
  coords(s, g, x, y, z);
  const int valid = valid_mask(boundary_code(x, y, z, g.W, g.H, g.D));
  // Values seven at a time (fourteen live values spill at 64 registers).
#pragma unroll
  for (int h = 0; h < kNumDirs; h += 7) {
    T val[7];
#pragma unroll
    for (int q = 0; q < 7; ++q) {
      const int d = h + q;
      val[q] = (valid >> d & 1) ? __ldg(gv + s + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH) : T(0);
    }
#pragma unroll
    for (int q = 0; q < 7; ++q) {
      const int d = h + q;
      const int r = s + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH;
      if ((valid >> d & 1) && (kSplit ? above(val[q], r, sv, s) : below(val[q], r, sv, s)))
        side |= 1u << d;
    }
  }
  return side;
}

// One saddle of one side: its decompressed row summary (count, first and
// last entry in row order) into the row slots, and whether some neighbour on
// the side has a wrong label.
//
// known: no value changed since a detection that found no mismatch, so the
// saddle's neighbours on the side are the original field's (its type and
// lower star matched): the direction mask is read instead of 14 neighbour
// values.  Two thirds of the rounds, the first one (every saddle) among them,
// run right after such a detection (with the 1-saddles' shortcut below, the saddle
// passes of a 512^3 correction went from 7.0 to 5.7 ms; with a kernel of its own for
// the first round and packed queues for the later ones they take 3.1).  The loop goes over the set bits kWide at
// a time, so that a group's gathers (labels and mismatch bits; the labels'
// values) are in flight together.
//
// A 1-saddle's slots are read only with join_rows; else only its seed bit is
// needed: the mismatch bytes of its neighbours.
template <class T, bool kSplit, int kWide = 4>
__device__ __forceinline__ bool saddle_row(const Job<T>& J, const int* __restrict__ off, int i,
                                           int s, bool known) {
  const T* __restrict__ gv = J.g;
  const int* __restrict__ lab = kSplit ? J.dds : J.das;
  const uint8_t* __restrict__ mis = J.mis;
  const T sv = __ldg(gv + s);
  unsigned side = 0u;
  if (known) {
    side = kSplit ? J.smask2[i] : J.olm[s];
  } else {
    side = side_of<T, kSplit>(J, s);
  }
  int mb = 0;
  if (!kSplit && !J.join_rows) {
    while (side) {
#pragma unroll
      for (int q = 0; q < kWide; ++q) {
        if (side) mb |= __ldg(mis + s + off[__ffs((int)side) - 1]);
        side &= side - 1u;
      }
    }
    return (mb >> 1) & 1;
  }
  T fv = T(0), lv = T(0);
  int cnt = 0, fm = -1, lm = -1;
  while (side) {
    int ml[kWide];
    T val[kWide];
#pragma unroll
    for (int q = 0; q < kWide; ++q) {
      ml[q] = -1;
      if (side) {
        const int r = s + off[__ffs((int)side) - 1];
        ml[q] = __ldg(lab + r);
        mb |= __ldg(mis + r);
      }
      side &= side - 1u;
    }
#pragma unroll
    for (int q = 0; q < kWide; ++q) val[q] = ml[q] >= 0 ? __ldg(gv + ml[q]) : T(0);
#pragma unroll
    for (int q = 0; q < kWide; ++q) {
      const int m = ml[q];
      const T v = val[q];
      if (m >= 0 && (!kSplit || tabs(T(v - sv)) >= J.thr)) {
        if (cnt == 0 || row_first<T, kSplit>(v, m, fv, fm)) { fv = v; fm = m; }
        if (cnt == 0 || row_first<T, kSplit>(lv, lm, v, m)) { lv = v; lm = m; }
        ++cnt;
      }
    }
  }
  const int oc = (kSplit ? J.ocnt2 : J.ocnt1)[i];
  if (oc > 0) {
    int* slots = (kSplit ? J.drow2 : J.drow1) + 2ll * i;
    const int k = oc - 1;
    int first = fm, kth = lm;
    if (cnt > k) {
      if (k != cnt - 1) kth = k == 0 ? fm : row_entry_k<T, kSplit>(J, s, k);
      *reinterpret_cast<int2*>(slots) = make_int2(fm, kth);
    } else {  // a shorter row keeps what it does not rewrite
      if (cnt > 0) slots[0] = fm;
      else first = slots[0];
      kth = slots[1];
    }
    const int2 o = *reinterpret_cast<const int2*>((kSplit ? J.oend2 : J.oend1) + i);
    (kSplit ? J.bad2 : J.bad1)[i] = (uint8_t)((o.x != first) | (o.y != kth) << 1);
  }
  return (mb >> (kSplit ? 0 : 1)) & 1;
}

// Whether any input of saddle s's rows changed since the previous computed
// round: the changed-input byte of s or of a neighbour (see k_jump2).  A
// neighbour outside the grid reads as some other vertex, which at worst
// recomputes a row that has not changed, and saves the coordinates.
template <class T>
__device__ __forceinline__ bool saddle_inputs_changed(const Job<T>& J, const int* __restrict__ off,
                                                      int s, unsigned st8) {
  const uint8_t* __restrict__ dirty = J.dirtyv;
  const int last = J.dim.N - 1;
  unsigned d[kNumDirs + 1];
  d[kNumDirs] = __ldg(dirty + s);
#pragma unroll
  for (int k = 0; k < kNumDirs; ++k) d[k] = __ldg(dirty + min(max(s + off[k], 0), last));
  bool hit = false;
#pragma unroll
  for (int k = 0; k <= kNumDirs; ++k) hit |= d[k] == st8;
  return hit;
}

// Fused pass over the original saddles after a manifold round, both sides in
// one grid.  A saddle whose inputs did not change since the previous computed
// round keeps its row slots and reuses its stored seed bit; the others of a later
// round are gathered in shared memory and computed a full block at a time (they
// are a tenth or so of the saddles, and nearly every warp holds one).  A block takes a chunk of the id space (pass_chunk blocks of 1024
// ids) and the entries of both saddle lists in it, so that the two sides read
// the same neighbourhoods together:
//  * decompressed row slots.  The reference rewrites row i (findAscPaths /
//    findDescPaths, :1832-2049) in place each round, and its only reader,
//    get_wrong_index_max / _min (:3113-3171), reads entry 0 and entry k =
//    (original count - 1), possibly stale when the new row is shorter.  So two
//    persistent slots per row reproduce it: slot 0 takes the new entry 0 when
//    the new row is non-empty, slot 1 takes the new entry k when the new row
//    has more than k entries.  Entry 0 is the row's extreme label in the sort
//    order and entry count-1 the opposite extreme, found in one pass; any other
//    entry k is found by ranking the candidates (rare: the rows of both fields
//    usually have the same length).
//  * wrong-neighbour seeds (get_wrong_split_neighbors / _join_ :2400-2513):
//    saddles with a neighbour on the side whose label differs from the
//    original's, 2-saddles to cand, 1-saddles to cand_j.
template <class T>
__global__ void __launch_bounds__(256, 4) k_saddle_pass(const Job<T>* __restrict__ jobs,
                                                        const __grid_constant__ Sel sel) {
  __shared__ int off[kNumDirs];
  __shared__ int queue[512], queued;  // changed rows waiting: index << 1 | side
  __shared__ uint8_t state[256];
  constexpr uint8_t kChunkClean = 0, kChunkSeeds = 1, kChunkChanged = 2;
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (mf_skip(J.ctr)) return;
  if (threadIdx.x == 0) queued = 0;
  fill_offsets(off, J.dim);
  // The bitsets that the round's jump has read, and the flags of the last
  // round's wrong neighbours, start empty again.
  const int nw = (J.dim.N + 31) >> 5;
  for (int w = blk * blockDim.x + threadIdx.x; w < nw; w += nblk * blockDim.x) {
    J.vchg[w] = 0u;
    J.rtouch2[w] = 0u;
    J.rtouch1[w] = 0u;
    J.taken[w] = 0u;
    J.taken1[w] = 0u;
  }
  __syncthreads();
  // No mismatch at the last detection and no value changed since (and no NaN, whose
  // neighbours' sides the masks do not tell).
  const bool known = J.ctr[C_MM] == 0 && J.ctr[C_DIRTY] == 0 && J.ctr[C_NAN] == 0;
  const int ns2 = J.ctr[C_NS2], ns1 = J.ctr[C_NS1];
  const int nb = (J.dim.N + kCpBlock - 1) / kCpBlock;
  const int chunk = J.pass_chunk;
  const int nchunk = (nb + chunk - 1) / chunk;
  // In the first round every changed-input byte is set (the change bitset
  // starts full), so the check is skipped.
  const bool all_new = J.ctr[C_MFDONE] == 0;
  const long long W = J.dim.W, WH = W * J.dim.H, N = J.dim.N;
  // Later rounds first ask the jump's per-block flags whether any changed-input
  // byte is set where a chunk's saddles could see one: the 3 x 3 row windows of
  // the planes and rows next to the chunk, one id wider on each side.  The
  // block's next 256 chunks are asked for together, a thread per chunk and
  // window with its flags' loads in flight at once, so that a light round passes
  // over the clean ones without a barrier each (one thread per chunk took nine
  // windows' loads in turn, 8 us before a small field's pass began).
  const int stamp = mf_stamp(J.ctr);
  auto window_changed = [&](int c, int t) {
    const long long first = (long long)c * chunk * kCpBlock;
    const long long end = min((long long)(c + 1) * chunk, (long long)nb) * kCpBlock;
    const long long shift = (long long)(t / 3 - 1) * WH + (long long)(t % 3 - 1) * W;
    const long long lo = max(0ll, first + shift - 1), hi = min(N - 1, end + shift);
    if (lo > hi) return false;
    const int b0 = (int)(lo >> 10), b1 = (int)(hi >> 10);
    bool seen = false;
    for (int b = b0; b <= b1; b += 6) {
      int f[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) f[k] = J.bdirty[min(b + k, b1)];
#pragma unroll
      for (int k = 0; k < 6; ++k) seen |= f[k] == stamp;
    }
    return seen;
  };
  const unsigned st8 = mf_byte(mf_stamp(J.ctr));  // changed-input bytes of this round
  // Seed s into its side's list.  All lanes of a warp call it.
  auto list = [&](bool split, bool has, int s) {
    const int slot2 = warp_append(J.ctr + C_CAND, has && split, 0xffffffffu);
    if (slot2 >= 0) J.cand[slot2] = s;
    const int slot1 = warp_append(J.ctr + C_CANDJ, has && !split, 0xffffffffu);
    if (slot1 >= 0) J.cand_j[slot1] = s;
  };
  // Row i of a side: slots and seed bit.
  auto row = [&](bool split, int i, int s) {
    const bool has = split ? saddle_row<T, true>(J, off, i, s, known)
                           : saddle_row<T, false>(J, off, i, s, known);
    (split ? J.has2 : J.has1)[i] = (uint8_t)has;
    return has;
  };
  // The last (up to) 256 of the qn queued rows.  The whole block calls it.
  int qn = 0;  // the same in every thread; `queued` hands out the places
  auto drain = [&] {
    const int left = max(qn - (int)blockDim.x, 0), k = left + (int)threadIdx.x;
    bool has = false, split = false;
    int s = 0;
    if (k < qn) {
      const int i = queue[k] >> 1;
      split = queue[k] & 1;
      s = split ? J.sad2[i] : J.sad1[i];
      has = row(split, i, s);
      if (has) atomicAdd(J.hcnt + (s >> 10) / chunk, 1);
    }
    list(split, has, s);
    qn = left;
    __syncthreads();
    if (threadIdx.x == 0) queued = left;
    __syncthreads();
  };
  const int mine = blk < nchunk ? (nchunk - blk + nblk - 1) / nblk : 0;  // chunks of the block
  for (int kc = 0; kc < mine; ++kc) {
    if (!all_new && kc % 256 == 0) {  // what the next 256 chunks ask for
      const int some = min(256, mine - kc);
      __syncthreads();
      if ((int)threadIdx.x < some)
        state[threadIdx.x] = J.hcnt[blk + (kc + (int)threadIdx.x) * nblk] ? kChunkSeeds : kChunkClean;
      __syncthreads();
      for (int p = threadIdx.x; p < 9 * some; p += blockDim.x)
        if (window_changed(blk + (kc + p / 9) * nblk, p % 9)) state[p / 9] = kChunkChanged;
      __syncthreads();
    }
    const uint8_t st = all_new ? kChunkChanged : state[kc % 256];
    if (st == kChunkClean) continue;  // rows and seed bits stand, and no seed bit is set
    const int c = blk + kc * nblk;
    const int b0 = c * chunk, b1 = min(b0 + chunk, nb);
    const int a2 = J.cpoff[b0], e2 = b1 < nb ? J.cpoff[b1] : ns2;
    const int a1 = J.cpoff[nb + b0], e1 = b1 < nb ? J.cpoff[nb + b1] : ns1;
    const int n2 = e2 - a2, n = n2 + (e1 - a1);
    if (st == kChunkSeeds) {  // seed bits as computed in an earlier round
      for (int base = 0; base < n; base += blockDim.x) {
        const int k = base + threadIdx.x;
        const bool split = k < n2;
        bool has = false;
        int s = 0;
        if (k < n) {
          const int i = split ? a2 + k : a1 + k - n2;
          s = split ? J.sad2[i] : J.sad1[i];
          has = (split ? J.has2 : J.has1)[i] != 0;
        }
        list(split, has, s);
      }
      continue;
    }
    if (all_new) {
      int nhas = 0;  // seed bits set in the chunk
      for (int base = 0; base < n; base += blockDim.x) {  // uniform in the block
        const int k = base + threadIdx.x;
        const bool split = k < n2;
        bool has = false;
        int s = 0;
        if (k < n) {
          const int i = split ? a2 + k : a1 + k - n2;
          s = split ? J.sad2[i] : J.sad1[i];
          has = row(split, i, s);
        }
        list(split, has, s);
        nhas += __syncthreads_count(has);
      }
      if (threadIdx.x == 0) J.hcnt[c] = nhas;
      continue;
    }
    if (threadIdx.x == 0) J.hcnt[c] = 0;  // counted as the chunk's saddles are done
    __syncthreads();
    for (int base = 0; base < n; base += blockDim.x) {  // uniform in the block
      const int k = base + threadIdx.x;
      const bool split = k < n2;
      bool has = false, changed = false;
      int s = 0, i = 0;
      if (k < n) {
        i = split ? a2 + k : a1 + k - n2;
        s = split ? J.sad2[i] : J.sad1[i];
        const uint8_t kept = (split ? J.has2 : J.has1)[i];  // loaded with the id
        changed = saddle_inputs_changed(J, off, s, st8);
        has = !changed && kept != 0;
      }
      list(split, has, s);
      const unsigned m = __ballot_sync(0xffffffffu, changed);
      const unsigned h = __ballot_sync(0xffffffffu, has);
      int at = 0;
      if (lane_id() == 0) {
        if (m) at = atomicAdd(&queued, __popc(m));
        if (h) atomicAdd(J.hcnt + c, __popc(h));
      }
      at = __shfl_sync(0xffffffffu, at, 0);
      if (changed) queue[at + __popc(m & ((1u << lane_id()) - 1u))] = i << 1 | (int)split;
      qn += __syncthreads_count(changed);
      if (qn >= (int)blockDim.x) drain();
    }
  }
  if (qn > 0) drain();
}

// The saddle pass of a correction's first round: every saddle, right after a
// detection without mismatch, so the direction masks are the original field's
// (known; a field with a NaN takes k_saddle_pass).  Without the later rounds' checks and queue it holds few registers,
// and its gathers are bound by latency: 2-saddles (rows) and 1-saddles (seed
// bits; rows too with join_rows) in two loops.
template <class T>
__global__ void __launch_bounds__(256, 4) k_saddle_first(const Job<T>* __restrict__ jobs,
                                                         const __grid_constant__ Sel sel) {
  __shared__ int off[kNumDirs];
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (mf_skip(J.ctr)) return;
  fill_offsets(off, J.dim);
  const int stride = nblk * blockDim.x, t0 = blk * blockDim.x + threadIdx.x;
  const int nw = (J.dim.N + 31) >> 5;
  for (int w = t0; w < nw; w += stride) {
    J.vchg[w] = 0u;
    J.rtouch2[w] = 0u;
    J.rtouch1[w] = 0u;
    J.taken[w] = 0u;
    J.taken1[w] = 0u;
  }
  __syncthreads();
  const int chunk = J.pass_chunk;
  auto side = [&](auto split) {
    constexpr bool kSplit = decltype(split)::value;
    const int ns = J.ctr[kSplit ? C_NS2 : C_NS1];
    const int* __restrict__ sad = kSplit ? J.sad2 : J.sad1;
    for (int base = t0 - (int)lane_id(); base < ns; base += stride) {  // uniform per warp
      const int i = base + (int)lane_id();
      bool has = false;
      int s = 0;
      if (i < ns) {
        s = sad[i];
        has = saddle_row<T, kSplit, 8>(J, off, i, s, true);
        (kSplit ? J.has2 : J.has1)[i] = (uint8_t)has;
        if (has) atomicAdd(J.hcnt + (s >> 10) / chunk, 1);
      }
      const int slot = warp_append(J.ctr + (kSplit ? C_CAND : C_CANDJ), has, 0xffffffffu);
      if (slot >= 0) (kSplit ? J.cand : J.cand_j)[slot] = s;
    }
  };
  side(std::true_type{});
  side(std::false_type{});
}

template <class T, bool kSplit>
__global__ void __launch_bounds__(256) k_wn_vote(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel,
                                                 int r) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (mf_skip(J.ctr) || J.wn_lockstep) return;
  if (r == 0) {
    // A short list (every round after the first few of a correction) goes to
    // the block completion whole: the grid rounds would be launches with
    // nothing to do.
    const bool small = J.ctr[C_CAND] <= kWnBlockMax;
    if (blk == 0 && threadIdx.x == 0) J.ctr[C_WNSMALL] = small;
    if (small) return;
  } else if (J.ctr[C_WNSMALL]) {
    return;
  }
  const unsigned long long round = (unsigned)(J.ctr[C_WNROUND] + r + 1);
  const int n = J.ctr[C_CAND + (r & 1)];
  const int* cur = (r & 1) ? J.cand_next : J.cand;
  // The list this round's commit fills (the one read two rounds ago).
  if (blk == 0 && threadIdx.x == 0) J.ctr[C_CAND + ((r + 1) & 1)] = 0;
  const unsigned* taken = kSplit ? J.taken : J.taken1;
  const int stride = nblk * blockDim.x;
  for (int e = blk * blockDim.x + threadIdx.x; e < n; e += stride) {
    const int s = cur[e];
    int ids[kNumDirs];
    const int k = wn_candidates<T, kSplit>(J, s, ids);
    const unsigned long long vote = (round << 32) | (unsigned)(~s);
    for (int j = 0; j < k; ++j)
      if (!bit_of(taken, ids[j])) atomicMax(J.claim + ids[j], vote);
  }
}

template <class T, bool kSplit>
__global__ void __launch_bounds__(256) k_wn_commit(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel,
                                                   int r) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (mf_skip(J.ctr) || J.ctr[C_WNSMALL] || J.wn_lockstep) return;
  const unsigned long long round = (unsigned)(J.ctr[C_WNROUND] + r + 1);
  const int n = J.ctr[C_CAND + (r & 1)];
  const int* cur = (r & 1) ? J.cand_next : J.cand;
  int* nxt = (r & 1) ? J.cand : J.cand_next;
  int* nnext = J.ctr + C_CAND + ((r + 1) & 1);
  unsigned* taken = kSplit ? J.taken : J.taken1;
  int* flagged = kSplit ? J.flagged : J.flagged1;
  int* nflag = J.ctr + (kSplit ? C_NFC : C_NFC1);
  const int stride = nblk * blockDim.x;
  for (int e = blk * blockDim.x + threadIdx.x; e < n; e += stride) {
    const int s = cur[e];
    int ids[kNumDirs];
    const int k = wn_candidates<T, kSplit>(J, s, ids);
    int first = -1;
    for (int j = 0; j < k; ++j)
      if (!bit_of(taken, ids[j])) { first = ids[j]; break; }
    if (first < 0) continue;  // every candidate already flagged: resolved
    const unsigned long long vote = (round << 32) | (unsigned)(~s);
    if (J.claim[first] == vote) {
      atomicOr(taken + (first >> 5), 1u << (first & 31));
      flagged[atomicAdd(nflag, 1)] = first;
    } else {
      nxt[atomicAdd(nnext, 1)] = s;
    }
  }
}

// Grid-wide vote / commit rounds per side before the per-job completion.
// Round r reads the candidate list of parity r & 1 (cand / cand_next, counts
// C_CAND / C_CAND_NEXT) and refills the other; its vote number is the job's
// base round + r + 1.  Lists of at most kWnBlockMax saddles skip them.
constexpr int kWnGridRounds = 3;

// Completion of the arbitration for whatever the grid-wide rounds left
// unresolved: one block per job runs further vote / commit rounds until no
// saddle is left.  Each round commits at least the smallest unresolved saddle
// (its vote wins on every candidate it votes on), so at most n rounds run; the
// device iteration limit bounds them as well.  claim and taken are read
// through L2 (__ldcg): other threads of the block update them with atomics
// and stores between the barriers.
// A flag bit as the last barrier left it: other threads set bits of the same
// word by atomics in L2.
__device__ __forceinline__ bool taken_now(const unsigned* bits, int v) {
  return __ldcg(bits + (v >> 5)) >> (v & 31) & 1u;
}

template <class T, bool kSplit>
__global__ void __launch_bounds__(1024) k_wn_resolve(Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  if (blockIdx.x >= sel.n) return;
  Job<T>& J = jobs[sel.idx[blockIdx.x]];
  if (mf_skip(J.ctr)) return;
  __shared__ int s_next;
  unsigned* taken = kSplit ? J.taken : J.taken1;
  int* flagged = kSplit ? J.flagged : J.flagged1;
  int* nflag = J.ctr + (kSplit ? C_NFC : C_NFC1);
  // The grid-wide rounds left their list in parity kWnGridRounds & 1; a short
  // list skipped them and is still in parity 0.
  const int par = J.ctr[C_WNSMALL] ? 0 : (kWnGridRounds & 1);
  int* cur = par ? J.cand_next : J.cand;
  int* nxt = par ? J.cand : J.cand_next;
  int n = J.ctr[C_CAND + par];
  unsigned long long round = (unsigned)(J.ctr[C_WNROUND] + kWnGridRounds);
  const int cap = J.iter_cap;
  int it = 0;
  while (n > 0) {
    if (it++ >= cap) {
      if (threadIdx.x == 0) atomicOr(J.ctr + C_ERROR, kErrResolve);
      break;
    }
    ++round;
    const unsigned long long hi = round << 32;
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
      const int s = __ldcg(cur + e);
      int ids[kNumDirs];
      const int k = wn_candidates<T, kSplit>(J, s, ids);
      const unsigned long long vote = hi | (unsigned)(~s);
      for (int j = 0; j < k; ++j)
        if (!taken_now(taken, ids[j])) atomicMax(J.claim + ids[j], vote);
    }
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
      const int s = __ldcg(cur + e);
      int ids[kNumDirs];
      const int k = wn_candidates<T, kSplit>(J, s, ids);
      int first = -1;
      for (int j = 0; j < k; ++j)
        if (!taken_now(taken, ids[j])) {
          first = ids[j];
          break;
        }
      if (first < 0) continue;  // every candidate already flagged: resolved
      const unsigned long long vote = hi | (unsigned)(~s);
      if (__ldcg(J.claim + first) == vote) {
        atomicOr(taken + (first >> 5), 1u << (first & 31));
        flagged[atomicAdd(nflag, 1)] = first;
      } else {
        nxt[atomicAdd(&s_next, 1)] = s;
      }
    }
    __syncthreads();
    n = s_next;
    int* t = cur;
    cur = nxt;
    nxt = t;
    __syncthreads();  // every thread has read s_next before it is reset
  }
  if (threadIdx.x == 0) {
    J.ctr[C_WNROUND] = (int)round;
    if (kSplit) {  // the join side's candidates become the list to resolve next
      int* t = J.cand;
      J.cand = J.cand_j;
      J.cand_j = t;
      J.ctr[C_CAND] = J.ctr[C_CANDJ];
    } else {
      J.ctr[C_CAND] = 0;
    }
    J.ctr[C_CAND_NEXT] = 0;
  }
}

// Lockstep resolution of the wrong-neighbour flags (jobs with wn_lockstep).
// Step d flags, for every saddle of a side's candidate list that no earlier
// step resolved, its direction-d neighbour when that neighbour is a candidate
// (on the side, label differs from the original's) and no earlier step flagged
// it.  Two saddles never share their direction-d neighbour, so a step has no
// conflict, and the steps in direction order make each see every earlier one.
// This is how the reference's concurrent launch resolves its check-then-set
// when its threads advance through their neighbour loops in step
// (get_wrong_split_neighbors / _join_, src/ExtreM_cuda.cu:2400-2513): a shared
// candidate goes to the saddle that meets it at the earlier neighbour index.
// The two sides flag into separate arrays, as the reference's two kernels do,
// so one step serves both.  A resolved saddle is complemented in its list (a
// saddle on both lists, type 3, is resolved on each side by itself).
template <class T>
__device__ __forceinline__ void wn_step_entry(const Job<T>& J, int e, int n2, int d) {
  const bool split = e < n2;
  int* const at = split ? J.cand + e : J.cand_j + (e - n2);
  const int s = *at;
  if (s < 0) return;
  const Dims g = J.dim;
  int x, y, z;
  coords(s, g, x, y, z);
  if (!dir_valid(d, boundary_code(x, y, z, g.W, g.H, g.D))) return;
  const int r = s + ddx(d) + ddy(d) * g.W + ddz(d) * g.W * g.H;
  const T sv = J.g[s], rv = J.g[r];
  if (!(split ? above(rv, r, sv, s) : below(rv, r, sv, s))) return;
  unsigned* taken = split ? J.taken : J.taken1;
  if ((split ? J.dds[r] == J.ds[r] : J.das[r] == J.as[r]) || taken_now(taken, r)) return;
  atomicOr(taken + (r >> 5), 1u << (r & 31));
  (split ? J.flagged : J.flagged1)[atomicAdd(J.ctr + (split ? C_NFC : C_NFC1), 1)] = r;
  *at = ~s;
}

// One step over every selected job's two candidate lists (a large list: one
// launch per direction).
template <class T>
__global__ void __launch_bounds__(256) k_wn_step(const Job<T>* __restrict__ jobs,
                                                 const __grid_constant__ Sel sel, int d) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (mf_skip(J.ctr)) return;
  const int n2 = J.ctr[C_CAND], n = n2 + J.ctr[C_CANDJ];
  const int stride = nblk * blockDim.x;
  for (int e = blk * blockDim.x + threadIdx.x; e < n; e += stride) wn_step_entry(J, e, n2, d);
}

// Candidate directions of entry e: the neighbours on its side whose label
// differs from the original's.  All gathers of the fourteen go out together.
template <class T>
__device__ __forceinline__ unsigned wn_mask(const Job<T>& J, bool split, int s) {
  const Dims g = J.dim;
  const int WH = g.W * g.H;
  int x, y, z;
  coords(s, g, x, y, z);
  const int valid = valid_mask(boundary_code(x, y, z, g.W, g.H, g.D));
  const T sv = J.g[s];
  const uint8_t bit = split ? 1 : 2;
  unsigned m = 0u;
#pragma unroll
  for (int d = 0; d < kNumDirs; ++d) {
    if (!(valid >> d & 1)) continue;
    const int r = s + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH;
    const T rv = J.g[r];
    if ((J.mis[r] & bit) && (split ? above(rv, r, sv, s) : below(rv, r, sv, s))) m |= 1u << d;
  }
  return m;
}

// All fourteen steps in one launch for a short list (fourteen grid launches
// would cost more than the work): a cluster of eight blocks per job, with a
// cluster barrier between steps, or its first block alone with a block barrier
// when each of its threads then has at most two entries.  A thread first finds
// its entries' candidate directions (wn_mask; the first kWnHeld entries' in
// registers, the others' in cand_next), so that a step is one look at the flag
// of one neighbour: 4-6 us for a few hundred saddles, where a chain of five
// dependent loads per step took 14-20 us, and a list that outgrew the block
// (several thousand saddles) 500 us.
constexpr int kWnCluster = 8, kWnHeld = 2;
// Lists that go to the cluster: what its threads hold in registers, and, before a
// job's first round, saddles of which a tenth or so will be candidates (fourteen
// launches are 35-70 us on a 64^3 field, the cluster's steps about 25).
constexpr int kWnClusterMax = kWnHeld * kWnCluster * 1024, kWnClusterFirst = 1 << 17;
template <class T>
__global__ void __cluster_dims__(kWnCluster, 1, 1) __launch_bounds__(1024)
    k_wn_steps_block(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  const int job = blockIdx.x / kWnCluster, rank = blockIdx.x % kWnCluster;
  const Job<T>& J = jobs[sel.idx[job]];
  __shared__ int off[kNumDirs];
  fill_offsets(off, J.dim);
  __syncthreads();
  if (mf_skip(J.ctr)) return;  // the whole cluster
  const int n2 = J.ctr[C_CAND], n = n2 + J.ctr[C_CANDJ];
  const bool alone = n <= kWnHeld * 1024;  // the same in every block of the cluster
  if (alone && rank) return;
  const int t0 = alone ? (int)threadIdx.x : rank * 1024 + (int)threadIdx.x;
  const int stride = alone ? 1024 : kWnCluster * 1024;
  auto entry = [&](int e) { return e < n2 ? J.cand[e] : J.cand_j[e - n2]; };
  int hs[kWnHeld];
  unsigned hm[kWnHeld];
#pragma unroll
  for (int k = 0; k < kWnHeld; ++k) {
    const int e = t0 + k * stride;
    hs[k] = e < n ? entry(e) : 0;
    hm[k] = e < n ? wn_mask(J, e < n2, hs[k]) : 0u;
  }
  // cand_next holds N entries; the two lists together may have more only when
  // over half of all vertices are candidates of both sides.
  const int cap = J.dim.N;
  for (int e = t0 + kWnHeld * stride; e < n && e < cap; e += stride)
    J.cand_next[e] = (int)wn_mask(J, e < n2, entry(e));
  // Flags the direction-d candidate of saddle s; true when it was free.
  auto take = [&](bool split, int s, int d) {
    const int r = s + off[d];
    unsigned* taken = split ? J.taken : J.taken1;
    if (taken_now(taken, r)) return false;
    atomicOr(taken + (r >> 5), 1u << (r & 31));
    (split ? J.flagged : J.flagged1)[atomicAdd(J.ctr + (split ? C_NFC : C_NFC1), 1)] = r;
    return true;
  };
  for (int d = 0; d < kNumDirs; ++d) {
#pragma unroll
    for (int k = 0; k < kWnHeld; ++k)
      if ((hm[k] >> d & 1u) && take(t0 + k * stride < n2, hs[k], d)) hm[k] = 0u;
    for (int e = t0 + kWnHeld * stride; e < n; e += stride) {
      if (e < cap) {
        if ((J.cand_next[e] >> d & 1) && take(e < n2, entry(e), d)) J.cand_next[e] = 0;
      } else {
        wn_step_entry(J, e, n2, d);
      }
    }
    if (d + 1 == kNumDirs) break;
    if (alone) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release;\n"
                   "barrier.cluster.wait.acquire;" ::: "memory");
    }
  }
}

// ---------------------------------------------------------------------------
// fixpath (:4046-4206): walk the steepest ascent (descent) of both fields from a
// flagged vertex until they diverge; lower the decompressed choice (split) or
// the original choice (join).  Both sides' lists in one launch: their proposals
// merge by atomic max.
// ---------------------------------------------------------------------------
template <class T, bool kSplit>
__device__ __forceinline__ void fixpath_from(const Job<T>& J, int cur) {
  const Dims g = J.dim;
  const int cap = J.iter_cap;
  int t = -1, fl = -1;
  int steps = 0;
  const int WH = g.W * g.H;
  for (; steps < cap; ++steps) {
    int x, y, z;
    coords(cur, g, x, y, z);
    const int valid = valid_mask(boundary_code(x, y, z, g.W, g.H, g.D));
    int ni = cur, nd = cur;
    T fi = J.f[cur], gd = J.g[cur];
    // Both fields' neighbours through static indices, so that a step's loads are
    // in flight together.
    T fr[kNumDirs], gr[kNumDirs];
#pragma unroll
    for (int d = 0; d < kNumDirs; ++d) {
      const int r = cur + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH;
      fr[d] = (valid >> d & 1) ? J.f[r] : T(0);
      gr[d] = (valid >> d & 1) ? J.g[r] : T(0);
    }
#pragma unroll
    for (int d = 0; d < kNumDirs; ++d) {
      const int r = cur + dir_x(d) + dir_y(d) * g.W + dir_z(d) * WH;
      if (!(valid >> d & 1)) continue;
      if (kSplit ? above(fr[d], r, fi, ni) : below(fr[d], r, fi, ni)) { ni = r; fi = fr[d]; }
      if (kSplit ? above(gr[d], r, gd, nd) : below(gr[d], r, gd, nd)) { nd = r; gd = gr[d]; }
    }
    if (ni != nd) { t = ni; fl = nd; break; }
    if (ni == cur) break;
    cur = ni;
  }
  if (steps == cap) {
    atomicOr(J.ctr + C_ERROR, kErrPath);
    return;
  }
  if (fl == t) return;
  const int target = kSplit ? fl : t;
  propose(J, target, step_delta(J, target));
}

template <class T>
__global__ void __launch_bounds__(256) k_fixpath(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const int n2 = J.ctr[C_NFC], n = n2 + J.ctr[C_NFC1];
  const int stride = nblk * blockDim.x;
  for (int e = blk * blockDim.x + threadIdx.x; e < n; e += stride) {
    if (e < n2) fixpath_from<T, true>(J, J.flagged[e]);
    else fixpath_from<T, false>(J, J.flagged1[e - n2]);
  }
}

// ---------------------------------------------------------------------------
// s_loops (:3465-3487) / s_loops_join (:3489-3512): get_wrong_index_max
// (:3113-3141) and get_wrong_index_min (:3143-3171) with the lowest saddle row
// winning per extremum, followed by the fixes (:3320-3413).
// ---------------------------------------------------------------------------
// The saddle pass has compared each row it computed with the original's (bad2 /
// bad1), so a scan reads a byte per row and goes on only at the wrong ones, and
// lists the extrema they name (in mm_next, free between detections: the index
// times two, plus one for the second kind) for the collecting pass.  Reading
// every row's ends and slots, then every extremum's two arbitration slots, took
// 0.16 ms per scan at 512^3, mostly to find nothing.
template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_wim_scan(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (blk == 0 && threadIdx.x == 0) {  // counted by k_wim_collect
    J.ctr[kMax ? C_WMC : C_WMIN] = 0;
    J.ctr[kMax ? C_WMC2 : C_WMIN2] = 0;
    J.ctr[C_TOUCHED] = 0;  // (the join side's scan follows saddle_loops in one tick)
  }
  const int ns = J.ctr[kMax ? C_NS2 : C_NS1];
  const int4* oend = kMax ? J.oend2 : J.oend1;
  const uint8_t* bad = kMax ? J.bad2 : J.bad1;
  int* first = kMax ? J.first1 : J.first_min1;
  int* flag = kMax ? J.flag2 : J.flag_min2;
  int* count = J.ctr + (kMax ? C_WLIST2 : C_WLIST1);
  const int stride = nblk * blockDim.x;
  for (int q = blk * blockDim.x + threadIdx.x; q < (ns + 15) >> 4; q += stride) {
    // (The arrays are padded; rows past the last are not looked at.)
    const uint4 w = reinterpret_cast<const uint4*>(bad)[q];
    const unsigned word[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      for (unsigned rest = word[j]; rest;) {
        const int byte = (__ffs((int)rest) - 1) >> 3, i = 16 * q + 4 * j + byte;
        const unsigned kinds = rest >> (8 * byte) & 3u;
        rest &= ~(0xffu << (8 * byte));
        if (i >= ns) break;
        const int4 o = oend[i];
        if ((kinds & 1u) && atomicMin(first + o.z, i) == kInf) J.mm_next[atomicAdd(count, 1)] = o.z << 1;
        if ((kinds & 2u) && atomicExch(flag + o.w, 1) == 0)
          J.mm_next[atomicAdd(count, 1)] = o.w << 1 | 1;
      }
    }
  }
}

// Collect per listed extremum, count, propose the fix and reset the arbitration
// slots.  fix = false: detection only (the third block of the outer loop,
// :5932-5951).
template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_wim_collect(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel, int fix) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const int n = J.ctr[kMax ? C_WLIST2 : C_WLIST1];
  const int* ext_list = kMax ? J.maxima : J.minima;
  const int* drow = kMax ? J.drow2 : J.drow1;
  int* first = kMax ? J.first1 : J.first_min1;
  int* flag = kMax ? J.flag2 : J.flag_min2;
  int* c1 = J.ctr + (kMax ? C_WMC : C_WMIN);
  int* c2 = J.ctr + (kMax ? C_WMC2 : C_WMIN2);
  const int stride = nblk * blockDim.x;
  for (int base = blk * blockDim.x; base < n; base += stride) {
    const int e = base + threadIdx.x;
    bool h1 = false, h2 = false;
    if (e < n) {
      const int m = J.mm_next[e] >> 1;
      h2 = J.mm_next[e] & 1;
      h1 = !h2;
      if (h1) {
        const int row = first[m];
        first[m] = kInf;
        if (fix) {
          // split: lower the false maximum, entry 0 of the winning
          // decompressed row (:3326-3344); join: lower the true minimum
          // itself (:3375-3391).
          const int target = kMax ? drow[2ll * row] : ext_list[m];
          propose(J, target, step_delta(J, target));
        }
      } else {
        flag[m] = 0;
        // lower the true maximum (:3346-3364)
        if (fix && kMax) propose(J, ext_list[m], step_delta(J, ext_list[m]));
      }
    }
    const unsigned mask = 0xffffffffu;
    const unsigned b1 = __ballot_sync(mask, h1), b2 = __ballot_sync(mask, h2);
    if (lane_id() == 0) {
      if (b1) atomicAdd(c1, __popc(b1));
      if (b2) atomicAdd(c2, __popc(b2));
    }
  }
}

// get_wrong_index_min direction 1 (:3157-3168, fix :3393-3410) keeps the pair of
// the lowest row per minimum and lowers the row's FALSE last entry, so it needs
// the winning row: one more scan, arbitrating through ext_id (left at kInf;
// first_sj keeps the wrong-saddle results between scans), then the minima of
// the second kind in k_wim_scan's list.
template <class T>
__global__ void __launch_bounds__(256) k_wim_min2_scan(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const int ns = J.ctr[C_NS1];
  const int stride = nblk * blockDim.x;
  for (int q = blk * blockDim.x + threadIdx.x; q < (ns + 15) >> 4; q += stride) {
    const uint4 w = reinterpret_cast<const uint4*>(J.bad1)[q];
    const unsigned word[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      for (unsigned rest = word[j] & 0x02020202u; rest; rest &= rest - 1u) {
        const int i = 16 * q + 4 * j + ((__ffs((int)rest) - 1) >> 3);
        if (i < ns) atomicMin(J.ext_id + J.oend1[i].w, i);
      }
    }
  }
}
template <class T>
__global__ void __launch_bounds__(256) k_wim_min2_collect(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const int n = J.ctr[C_WLIST1];
  const int stride = nblk * blockDim.x;
  for (int e = blk * blockDim.x + threadIdx.x; e < n; e += stride) {
    if (!(J.mm_next[e] & 1)) continue;
    const int m = J.mm_next[e] >> 1;
    const int row = J.ext_id[m];
    J.ext_id[m] = kInf;
    const int target = J.drow1[2ll * row + 1];
    propose(J, target, step_delta(J, target));
  }
}

// ---------------------------------------------------------------------------
// saddle_loops (:4229-4243) / saddle_loops_join (:4245-4261):
// get_wrong_index_saddles(_join) (:3173-3270) -- the first saddle in an
// extremum's CSR list (row order, then entry order) that outranks the true
// largest (smallest) saddle in the decompressed field -- and
// fix_wrong_index_saddle (:3415-3463).
// ---------------------------------------------------------------------------
// The scan is incremental.  An extremum's result -- its first row entry
// (i * kRowStride + p, row order then entry order) whose saddle outranks the
// extremum's true largest (smallest) saddle in the decompressed field, or kInf
// -- depends only on the values of the saddles whose rows name it, and the true
// largest saddle is one of them.  So after the first scan of a correction
// (epoch 1: every extremum) only the extrema named in the rows of saddles whose
// value changed since the previous scan are recomputed, each from its list of
// row entries (moff / ment, built at setup); the others keep their result.
// k_apply marks changed values in wchg2 / wchg1, one bitset per side.

// Row index of vertex v on the side (its index in sad2 / sad1), or -1: a
// binary search among the list entries of v's 1024-id block (cpoff).
template <class T, bool kMax>
__device__ __forceinline__ int side_row(const Job<T>& J, int v) {
  const int t = J.otype[v];
  if (!(kMax ? (t == 2 || t == 3) : (t == 1 || t == 3))) return -1;
  const int nb = (J.dim.N + kCpBlock - 1) / kCpBlock, b = v / kCpBlock;
  const int* off = J.cpoff + (kMax ? 0 : nb);
  const int* sad = kMax ? J.sad2 : J.sad1;
  int lo = off[b], hi = (b + 1 < nb ? off[b + 1] : J.ctr[kMax ? C_NS2 : C_NS1]) - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (sad[mid] < v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Queues the extrema named in the rows of the saddles whose value changed
// (and clears the bitset).  In epoch 1 every extremum is recomputed, so the
// bitset is only cleared.
template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_wis_mark(const Job<T>* __restrict__ jobs,
                                                  const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (blk == 0 && threadIdx.x == 0) J.ctr[kMax ? C_WSC : C_WSCJ] = 0;  // counted by k_wis_collect
  const int epoch = J.ctr[kMax ? C_WEP2 : C_WEP1] + 1;
  unsigned* chg = kMax ? J.wchg2 : J.wchg1;
  const uint8_t* ocnt = kMax ? J.ocnt2 : J.ocnt1;
  const int4* orm = kMax ? J.orm2 : J.orm1;
  const int* rows = kMax ? J.orow2 : J.orow1;
  int* stamp = kMax ? J.wstamp2 : J.wstamp1;
  const int nw = (J.dim.N + 31) >> 5;
  const int stride = nblk * blockDim.x;
  for (int w = blk * blockDim.x + threadIdx.x; w < nw; w += stride) {
    unsigned bits = chg[w];
    if (!bits) continue;
    chg[w] = 0u;
    if (epoch == 1) continue;
    for (; bits; bits &= bits - 1) {
      const int i = side_row<T, kMax>(J, (w << 5) + __ffs(bits) - 1);
      if (i < 0) continue;
      const int cnt = ocnt[i];
      const int4 m4 = orm[i];
      for (int p = 0; p < cnt; ++p) {
        const int m = p == 0 ? m4.x : p == 1 ? m4.y : p == 2 ? m4.z : p == 3 ? m4.w
                                                             : rows[(long long)i * kRowStride + p];
        if (m < 0) continue;  // a repeated label
        if (atomicExch(stamp + m, epoch) != epoch) J.aff[atomicAdd(J.ctr + C_AFF, 1)] = m;
      }
    }
  }
}

// The first entry among ent[k0 + i * step], i >= 0, below k1 whose saddle
// outranks extremum saddle tb (value gt), or kInf.  Four entries at a time:
// their three dependent loads (entry, saddle, value) go out together.
template <class T, bool kMax>
__device__ __forceinline__ int wis_first(const Job<T>& J, const int* sad, const int* ent, int k0,
                                         int k1, int step, int tb, T gt) {
  int hit = kInf;
  for (int k = k0; k < k1; k += 4 * step) {
    int key[4], s[4];
    T gs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) key[j] = k + j * step < k1 ? ent[k + j * step] : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = key[j] >= 0 ? sad[key[j] / kRowStride] : 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) gs[j] = key[j] >= 0 ? J.g[s[j]] : T(0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool wrong = kMax ? (gs[j] > gt || (gs[j] == gt && s[j] > tb))
                              : (gs[j] < gt || (gs[j] == gt && s[j] < tb));
      if (key[j] >= 0 && wrong && key[j] < hit) hit = key[j];
    }
  }
  return hit;
}

// Recomputes the queued extrema (every extremum in epoch 1) from their row
// entries, a thread per extremum; an extremum with more than kWisShort
// entries goes to the long queue (wlong) for a block of its own
// (k_wis_long), so that one long list does not hold up the launch.
constexpr int kWisShort = 48;
template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_wis_update(const Job<T>* __restrict__ jobs,
                                                    const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const bool all = J.ctr[kMax ? C_WEP2 : C_WEP1] == 0;
  const int n = all ? J.ctr[kMax ? C_NMAX : C_NMIN] : J.ctr[C_AFF];
  const int* sad = kMax ? J.sad2 : J.sad1;
  const int* best = kMax ? J.largest : J.smallest;
  const int* off = kMax ? J.moff2 : J.moff1;
  const int* ent = kMax ? J.ment2 : J.ment1;
  int* first = kMax ? J.first_s : J.first_sj;
  const int N = J.dim.N;
  const int stride = nblk * blockDim.x;
  for (int base = blk * blockDim.x; base < n; base += stride) {  // uniform per warp
    const int e = base + threadIdx.x;
    bool lng = false;
    int m = 0;
    if (e < n) {
      m = all ? e : J.aff[e];
      const int tb = best[m];
      const int k0 = off[m], k1 = off[m + 1];
      lng = k1 - k0 > kWisShort;
      // An extremum named by no row has no saddle.
      if (!lng)
        first[m] = (tb >= 0 && tb < N) ? wis_first<T, kMax>(J, sad, ent, k0, k1, 1, tb, J.g[tb])
                                       : kInf;
    }
    const int slot = warp_append(J.ctr + C_WLONG, lng, 0xffffffffu);
    if (slot >= 0) J.wlong[slot] = m;
  }
}

// The long lists of k_wis_update, a block per extremum.
template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_wis_long(const Job<T>* __restrict__ jobs,
                                                  const __grid_constant__ Sel sel) {
  __shared__ int part[8];
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const int n = J.ctr[C_WLONG];
  const int* sad = kMax ? J.sad2 : J.sad1;
  const int* ent = kMax ? J.ment2 : J.ment1;
  const int* off = kMax ? J.moff2 : J.moff1;
  for (int e = blk; e < n; e += nblk) {  // uniform per block
    const int m = J.wlong[e];
    const int tb = (kMax ? J.largest : J.smallest)[m];  // valid: the lists are non-empty
    int hit = wis_first<T, kMax>(J, sad, ent, off[m] + (int)threadIdx.x, off[m + 1], 256, tb,
                                 J.g[tb]);
    for (int o = 16; o > 0; o >>= 1) hit = min(hit, __shfl_xor_sync(0xffffffffu, hit, o));
    if (lane_id() == 0) part[threadIdx.x >> 5] = hit;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) hit = min(hit, part[w]);
      (kMax ? J.first_s : J.first_sj)[m] = hit;
    }
    __syncthreads();
  }
}

template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_wis_collect(const Job<T>* __restrict__ jobs, const __grid_constant__ Sel sel, int fix) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (blk == 0 && threadIdx.x == 0) {  // the scan is over: next epoch, empty queues
    J.ctr[kMax ? C_WEP2 : C_WEP1] += 1;
    J.ctr[C_AFF] = J.ctr[C_WLONG] = 0;
  }
  const int next = J.ctr[kMax ? C_NMAX : C_NMIN];
  const int* sad = kMax ? J.sad2 : J.sad1;
  const int* best = kMax ? J.largest : J.smallest;
  int* first = kMax ? J.first_s : J.first_sj;
  int* cnt = J.ctr + (kMax ? C_WSC : C_WSCJ);
  const int stride = nblk * blockDim.x;
  for (int base = blk * blockDim.x; base < next; base += stride) {
    const int m = base + threadIdx.x;
    bool hit = false;
    if (m < next && first[m] != kInf) {  // kept: the scan is incremental
      hit = true;
      const int s = sad[first[m] / kRowStride];
      const int t = best[m];
      if (fix) {
        const T gt = J.g[t], gs = J.g[s];
        if (kMax) {
          if (!(gt > gs || (gt == gs && t > s))) propose(J, s, step_delta(J, s));
        } else if (!(gt < gs || (gt == gs && t < s))) {
          // store -bound/q, then (edit_type 1) atomic max with the midpoint:
          // max(-bound/q, midpoint) whatever the interleaving (:3447-3458).
          propose(J, t, -J.bound / T(J.q));
          if (J.edit_type == 1) propose(J, t, midpoint_delta(J, t));
        }
      }
    }
    const unsigned b = __ballot_sync(0xffffffffu, hit);
    if (lane_id() == 0 && b) atomicAdd(cnt, __popc(b));
  }
}

// ---------------------------------------------------------------------------
// The final saddle_loops_join (:5997) of a job whose 1-saddle rows nothing
// else reads (join_rows == 0): get_wrong_index_saddles_join looks at them
// once, so no entry lists are built and nothing is kept between scans.  Three
// passes over the 1-saddles of the original field: the extreme value key per
// minimum (k_join_keys, which also leaves each row's distinct minima in orm1 /
// orow1 / ocnt1), the smallest id at that key (k_join_ids: together
// findSmallestSaddlePerMin :4915-4940), and the first row per minimum whose
// saddle comes before that smallest saddle in the decompressed field
// (k_join_scan, into first_sj for k_wis_collect).  ext_key, smallest and first_sj
// were filled at setup.  1.9 ms for the 22 M
// 1-saddles of the 512^3 benchmark field, where their rows, entry lists and
// first full scan took 4.2 ms; a job that ends early does not run them.
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256, 4) k_join_keys(const Job<T>* __restrict__ jobs,
                                                      const __grid_constant__ Sel sel) {
  __shared__ int off[kNumDirs];
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  if (blk == 0 && threadIdx.x == 0) J.ctr[C_WSCJ] = 0;  // counted by k_wis_collect
  fill_offsets(off, J.dim);
  __syncthreads();
  using KK = typename KeyOf<T>::K;
  const int ns = J.ctr[C_NS1];
  const int* __restrict__ lab = J.as;
  const int* __restrict__ ext = J.ext;
  const int stride = nblk * blockDim.x;
  for (int base = blk * blockDim.x; base < ns; base += stride) {  // uniform per warp
    const int i = base + threadIdx.x;
    const bool act = i < ns;
    const int s = act ? J.sad1[i] : 0;
    unsigned rest = act ? J.olm[s] : 0u;
    const int pmax = (int)__reduce_max_sync(0xffffffffu, __popc(rest));
    const KK key = KeyOf<T>::enc(J.f[s] + T(0));  // -0 and +0 compare equal
    // Distinct labels in direction order, kept as extremum indices.
    int lb[16], mp[16];
    int cnt = 0, m0 = -1, m1 = -1, m2 = -1, m3 = -1;
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
#pragma unroll
      for (int q = h; q < h + 8; ++q) lb[q] = mp[q] = -1;
      if (h >= pmax) continue;  // uniform per warp
#pragma unroll
      for (int q = h; q < h + 8; ++q) {
        if (rest) lb[q] = lab[s + off[__ffs((int)rest) - 1]];
        rest &= rest - 1u;
      }
#pragma unroll
      for (int q = h; q < h + 8; ++q) {
        bool fresh = lb[q] >= 0;
#pragma unroll
        for (int e = 0; e < q; ++e) fresh &= lb[e] != lb[q];
        if (fresh) mp[q] = ext[lb[q]];
      }
#pragma unroll
      for (int q = h; q < h + 8; ++q) {
        if (mp[q] < 0) continue;
        m0 = cnt == 0 ? mp[q] : m0;
        m1 = cnt == 1 ? mp[q] : m1;
        m2 = cnt == 2 ? mp[q] : m2;
        m3 = cnt == 3 ? mp[q] : m3;
        if (cnt >= 4) J.orow1[(long long)i * kRowStride + cnt] = mp[q];
        ++cnt;
      }
      KK cur[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) cur[q] = mp[h + q] >= 0 ? J.ext_key[mp[h + q]] : KK(0);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (mp[h + q] >= 0 && key < cur[q]) atomicMin(J.ext_key + mp[h + q], key);
    }
    if (act) {
      J.ocnt1[i] = (uint8_t)cnt;
      J.orm1[i] = make_int4(m0, m1, m2, m3);
    }
  }
}

template <class T>
__global__ void __launch_bounds__(256) k_join_ids(const Job<T>* __restrict__ jobs,
                                                  const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  using KK = typename KeyOf<T>::K;
  const int ns = J.ctr[C_NS1];
  const int stride = nblk * blockDim.x;
  for (int i = blk * blockDim.x + threadIdx.x; i < ns; i += stride) {
    const int s = J.sad1[i], cnt = J.ocnt1[i];
    const int4 m4 = J.orm1[i];
    const KK key = KeyOf<T>::enc(J.f[s] + T(0));
    const int m[4] = {m4.x, m4.y, m4.z, m4.w};
    KK cur[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) cur[q] = m[q] >= 0 ? J.ext_key[m[q]] : KK(0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (m[q] >= 0 && cur[q] == key) atomicMin(J.smallest + m[q], s);
    for (int p = 4; p < cnt; ++p) {
      const int mm = J.orow1[(long long)i * kRowStride + p];
      if (J.ext_key[mm] == key) atomicMin(J.smallest + mm, s);
    }
  }
}

template <class T>
__global__ void __launch_bounds__(256) k_join_scan(const Job<T>* __restrict__ jobs,
                                                   const __grid_constant__ Sel sel) {
  int blk, nblk;
  const Job<T>& J = span_job(jobs, sel, blk, nblk);
  const T* __restrict__ g = J.g;
  const int ns = J.ctr[C_NS1];
  const int stride = nblk * blockDim.x;
  for (int i = blk * blockDim.x + threadIdx.x; i < ns; i += stride) {
    const int s = J.sad1[i], cnt = J.ocnt1[i];
    const int4 m4 = J.orm1[i];
    const T gs = g[s];
    const int m[4] = {m4.x, m4.y, m4.z, m4.w};
    int t[4];
    T gt[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) t[q] = m[q] >= 0 ? J.smallest[m[q]] : s;
#pragma unroll
    for (int q = 0; q < 4; ++q) gt[q] = t[q] != s ? g[t[q]] : T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (t[q] != s && below(gs, s, gt[q], t[q])) atomicMin(J.first_sj + m[q], i * kRowStride);
    for (int p = 4; p < cnt; ++p) {
      const int mm = J.orow1[(long long)i * kRowStride + p], tt = J.smallest[mm];
      if (tt != s && below(gs, s, g[tt], tt)) atomicMin(J.first_sj + mm, i * kRowStride);
    }
  }
}

// ---------------------------------------------------------------------------
// Small helpers.
// ---------------------------------------------------------------------------
// Initial contents of a job's arrays in one launch: segment k is `chunks`
// 16-byte pieces (arrays are padded to 256 bytes) of the 8-byte pattern `value`.
// One launch in place of some twenty fills and clears, whose issue took the host
// longer than a small field's setup takes the device.
constexpr int kMaxFills = 32;
struct FillList {
  int n;
  ulonglong2* at[kMaxFills];
  long long end[kMaxFills];  // inclusive prefix of the segments' pieces
  unsigned long long value[kMaxFills];
};
__global__ void __launch_bounds__(256) k_fill_many(const __grid_constant__ FillList f) {
  const long long total = f.end[f.n - 1], stride = (long long)gridDim.x * blockDim.x;
  int k = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += stride) {
    while (i >= f.end[k]) ++k;
    const unsigned long long v = f.value[k];
    f.at[k][i - (k ? f.end[k - 1] : 0)] = make_ulonglong2(v, v);
  }
}

// End of a tick, one block: the bookkeeping of the first `slots` jobs' phases
// (a thread per job), then, with host set, every counter to the host's mapped
// copy beside the tick's number in the same 8 bytes, so that the host can see
// for each whether it has come and no fence is needed.  (A copy and a stream
// synchronisation behind the kernels took about 8 us longer; a flag written
// behind two system-wide fences about 5 us.)
template <class T>
__global__ void __launch_bounds__(256) k_tick_end(Job<T>* jobs, int* ctr, int slots, unsigned* seq,
                                                  volatile unsigned long long* host) {
  if (threadIdx.x < slots) {
    int* c = ctr + threadIdx.x * C_COUNT;
    c[C_TOUCHED] = 0;
    c[C_WLIST2] = c[C_WLIST1] = 0;
    if (c[C_DETECTED]) {
      c[C_DETECTED] = 0;
      detect_end(jobs[threadIdx.x]);
    }
    if (c[C_MFRUN]) {
      c[C_MFRUN] = 0;
      mf_end(c);
    }
  }
  if (!host) return;
  const unsigned long long s = (unsigned long long)(*seq + 1u) << 32;
  __syncthreads();
  for (int i = threadIdx.x; i < slots * C_COUNT; i += blockDim.x) host[i] = s | (unsigned)ctr[i];
  if (threadIdx.x == 0) *seq = (unsigned)(s >> 32);
}

template <class K>
__global__ void k_fill(K* p, K v, long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) p[i] = v;
}

}  // namespace extremz

// Merge-tree persistence pairs of a field on the device: the extremum-graph
// pairing of the reference's constructPersistencePairs (src/ExtreM.cpp
// :1863-1918, called by compute_MergeT :2930-2952), for the split tree
// (maxima with merge saddles of superlevel sets) and the join tree (minima
// with merge saddles of sublevel sets), from the field's own extrema,
// manifold labels and merge vertices (vertices whose upper, respectively
// lower, link has two or more components).
//
// Order.  The split tree ranks vertices by (value, id); the join tree by the
// reverse order.  Extrema are ranked ascending in the tree's order (the
// global extremum last), saddles descending (the "largest" saddle first).
// Row i of saddle i holds the distinct ranks of the extrema reached by the
// steepest paths of its neighbours on the tree's side (its descending- or
// ascending-manifold labels), ascending; a row with one entry is emptied.
//
// Rounds (:1878-1906): every extremum takes the first (largest) saddle whose
// row holds it; an extremum that is its saddle's smallest entry pairs with it
// and points to the saddle's largest entry; pointers are compressed
// (:1908-1921) and every row is rewritten through them, deduplicated, and
// emptied when one entry is left (:1923-1932).  Rounds repeat until none
// pairs.  The global extremum pairs with the opposite global extremum (:1937).
#pragma once

#include <cub/cub.cuh>

#include "extremz_kernels.cuh"

namespace extremz {

constexpr int kPpRow = 16;  // entries per row (<= 14 neighbours)

// Which of the 2^14 sets of link vertices fall into two or more components, one
// bit per set (kMergeWords words, 2 KB).  An interior vertex whose upper
// neighbours are the set is a 2-saddle (or both kinds of saddle) exactly then,
// so the bits come from the type table's interior entries; the empty and the
// full set have none and one component.  Flooding the link at every voxel took
// 17 ms per pass of a 160x144x128 field; a voxel's test is a bit in shared memory.
constexpr int kMergeWords = (1 << kNumDirs) / 32;
__global__ void __launch_bounds__(256) k_pp_merge_table(DeviceTables tb, unsigned* __restrict__ table) {
  const int set = blockIdx.x * 256 + threadIdx.x;
  const int t = tb.lut[tb.key_offset[0] + set];
  const bool merges = set != 0 && set != (1 << kNumDirs) - 1 && (t == 2 || t == 3);
  const unsigned m = __ballot_sync(0xffffffffu, merges);
  if (lane_id() == 0) table[set >> 5] = m;
}

// Merge vertices of the two trees, from the link itself rather than the
// lookup table (which has no entries for grids thinner than 3 voxels): bit 0
// when the upper link (split tree) has two or more components, bit 1 when the
// lower link (join tree) has.
template <class T>
__device__ __forceinline__ int merge_bits(const T* __restrict__ a, const Dims& g, int v,
                                          const unsigned* table) {
  int x, y, z;
  coords(v, g, x, y, z);
  const int valid = valid_mask(boundary_code(x, y, z, g.W, g.H, g.D));
  const T c = a[v];
  int up = 0;
#pragma unroll
  for (int d = 0; d < kNumDirs; ++d) {
    if (!(valid >> d & 1)) continue;
    const int u = v + dir_x(d) + dir_y(d) * g.W + dir_z(d) * g.W * g.H;
    if (above(a[u], u, c, v)) up |= 1 << d;
  }
  const int lo = valid & ~up;
  return (int)(table[up >> 5] >> (up & 31) & 1u) | (int)(table[lo >> 5] >> (lo & 31) & 1u) << 1;
}

// Ordered compaction of the merge vertices (split list 0, join list 1): block
// counts with each warp's membership words (list l's word of ids 32w .. 32w+31
// at member[l * kCpBlock / 32 * blocks + w]), then (after k_scan_lists) the
// writes in ascending id from those words: the field is read once.
template <class T>
__global__ void __launch_bounds__(kCpBlock) k_pp_cand_count(const T* __restrict__ a, Dims g,
                                                            const unsigned* __restrict__ table,
                                                            unsigned* __restrict__ member,
                                                            int* __restrict__ bcount) {
  __shared__ unsigned tab[kMergeWords];
  __shared__ int cnt[2];
  if (threadIdx.x < kMergeWords) tab[threadIdx.x] = table[threadIdx.x];
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int v = blockIdx.x * kCpBlock + threadIdx.x;
  const int b = v < g.N ? merge_bits(a, g, v, tab) : 0;
  for (int l = 0; l < 2; ++l) {
    const unsigned m = __ballot_sync(0xffffffffu, (b >> l) & 1);
    if (lane_id() == 0) {
      member[(l * gridDim.x + blockIdx.x) * (kCpBlock / 32) + threadIdx.x / 32] = m;
      if (m) atomicAdd(&cnt[l], __popc(m));
    }
  }
  __syncthreads();
  if (threadIdx.x < 2) bcount[threadIdx.x * gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// One warp per 1024-id block and list (blockIdx.y): a lane per membership word.
__global__ void __launch_bounds__(256) k_pp_cand_write(const unsigned* __restrict__ member, int nb,
                                                       const int* __restrict__ boff,
                                                       int* __restrict__ split,
                                                       int* __restrict__ join) {
  const int b = blockIdx.x * 8 + (int)(threadIdx.x >> 5), l = blockIdx.y;
  if (b >= nb) return;  // whole warps leave together
  unsigned m = member[(l * nb + b) * (kCpBlock / 32) + (int)lane_id()];
  const int c = __popc(m);
  int incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane_id() >= (unsigned)o) incl += y;
  }
  int pos = boff[l * nb + b] + incl - c;
  int* out = l ? join : split;
  for (; m; m &= m - 1) out[pos++] = b * kCpBlock + (int)lane_id() * 32 + __ffs(m) - 1;
}

// Sort keys: 64-bit order-preserving value key, complemented for a
// descending sort.  -0 is keyed as +0: the total order compares values, and
// the two zeros are equal values (ties go by id).
template <class T>
__global__ void k_pp_keys(const T* __restrict__ a, const int* __restrict__ list, int n, bool reverse,
                          bool complement, unsigned long long* __restrict__ keys,
                          int* __restrict__ vals) {
  const int stride = gridDim.x * blockDim.x;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
    const int li = reverse ? n - 1 - k : k;  // ties keep the input's id order
    T v = a[list[li]];
    if (v == T(0)) v = T(0);
    const unsigned long long key = (unsigned long long)KeyOf<T>::enc(v);
    keys[k] = complement ? ~key : key;
    vals[k] = li;
  }
}

// rank[list index] = position in the sorted order.
__global__ void k_pp_rank(const int* __restrict__ sorted_li, int n, int* __restrict__ rank) {
  const int stride = gridDim.x * blockDim.x;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) rank[sorted_li[p]] = p;
}

// Stores the distinct entries of r (kInf = none) ascending, unless there is only
// one; returns how many.
__device__ __forceinline__ int pp_store_row(const int* r, int* row) {
  unsigned keep = 0u;
#pragma unroll
  for (int q = 0; q < kPpRow; ++q) {
    bool again = r[q] == kInf;
#pragma unroll
    for (int k = 0; k < q; ++k) again |= r[k] == r[q];
    if (!again) keep |= 1u << q;
  }
  const int n = __popc(keep);
  if (n < 2) return 0;
#pragma unroll
  for (int q = 0; q < kPpRow; ++q) {
    if (!(keep >> q & 1u)) continue;
    int at = 0;
#pragma unroll
    for (int k = 0; k < kPpRow; ++k) at += (keep >> k & 1u) && r[k] < r[q];
    row[at] = r[q];
  }
  return n;
}

// Row of each saddle (by sorted position): distinct extremum ranks of the
// labels of its neighbours on the tree's side, ascending.  The neighbours are
// the classification's direction mask; an entry's place is the number of smaller
// distinct ones, so nothing is sorted in local memory.
template <class T, bool kMax>
__global__ void __launch_bounds__(256) k_pp_rows(const T* __restrict__ a,
                                                 const uint16_t* __restrict__ olm,
                                                 const int* __restrict__ ctr, Dims g,
                                                 const int* __restrict__ sad,
                                                 const int* __restrict__ sorted_li, int ns,
                                                 const int* __restrict__ lab,
                                                 const int* __restrict__ ext,
                                                 const int* __restrict__ erank, int* __restrict__ rows,
                                                 int* __restrict__ cnt) {
  __shared__ int off[kNumDirs];
  fill_offsets(off, g);
  __syncthreads();
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
    const int s = sad[sorted_li[i]];
    unsigned side = olm[s];
    if (kMax) {
      int x, y, z;
      coords(s, g, x, y, z);
      side = (unsigned)valid_mask(boundary_code(x, y, z, g.W, g.H, g.D)) & ~side;
      if (ctr[C_NAN]) side = drop_nans(a, off, s, side);
    }
    int r[kPpRow];
#pragma unroll
    for (int h = 0; h < kPpRow; h += 4) {
#pragma unroll
      for (int q = h; q < h + 4; ++q) {
        r[q] = kInf;
        if (side) r[q] = lab[s + off[__ffs((int)side) - 1]];
        side &= side - 1u;
      }
#pragma unroll
      for (int q = h; q < h + 4; ++q)
        if (r[q] != kInf) r[q] = ext[r[q]];
#pragma unroll
      for (int q = h; q < h + 4; ++q)
        if (r[q] != kInf) r[q] = erank[r[q]];
    }
    cnt[i] = pp_store_row(r, rows + (long long)i * kPpRow);
  }
}

// Largest saddle of every extremum but the global one.
__global__ void __launch_bounds__(256) k_pp_largest(const int* __restrict__ rows,
                                                    const int* __restrict__ cnt, int ns, int glob,
                                                    int* __restrict__ largest) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
    const int c = cnt[i];
    const int* row = rows + (long long)i * kPpRow;
    for (int h = 0; h < c; h += 4) {
      const int4 e = *reinterpret_cast<const int4*>(row + h);
      if (e.x != glob) atomicMin(largest + e.x, i);
      if (h + 1 < c && e.y != glob) atomicMin(largest + e.y, i);
      if (h + 2 < c && e.z != glob) atomicMin(largest + e.z, i);
      if (h + 3 < c && e.w != glob) atomicMin(largest + e.w, i);
    }
  }
}

// Pairing of the round; resets largest for the next round.  lmax keeps the
// extremum each paired one merges into (its saddle row's largest entry, the
// second element of the reference's maximaTriplets, :2187), which ptr then
// loses to compression.
__global__ void k_pp_pair(const int* __restrict__ rows, const int* __restrict__ cnt, int ne, int ns,
                          int* __restrict__ largest, int* __restrict__ ptr, int* __restrict__ pair,
                          int* __restrict__ lmax, int* changed) {
  const int stride = gridDim.x * blockDim.x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += stride) {
    const int i = largest[e];
    largest[e] = kInf;
    if (i >= ns || pair[e] >= 0) continue;
    if (rows[(long long)i * kPpRow] == e) {
      pair[e] = i;
      const int l = rows[(long long)i * kPpRow + cnt[i] - 1];
      ptr[e] = l;
      lmax[e] = l;
      *changed = 1;
    }
  }
}

// Pointer compression to the surviving extremum.
__global__ void k_pp_jump(int* __restrict__ ptr, int ne, int cap, int* err) {
  const int stride = gridDim.x * blockDim.x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += stride) {
    int u = ptr[e], it = 0;
    while (ptr[u] != u && it < cap) {
      u = ptr[u];
      ++it;
    }
    if (it == cap) atomicOr(err, kErrJump);
    ptr[e] = u;
  }
}

// Rows rewritten through the pointers, deduplicated, emptied at one entry.  (Rows
// of up to four entries, nearly all, stay in four registers.)
__global__ void __launch_bounds__(256) k_pp_remap(int* __restrict__ rows, int* __restrict__ cnt, int ns,
                                                  const int* __restrict__ ptr) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += stride) {
    const int c = cnt[i];
    if (c == 0) continue;
    int* row = rows + (long long)i * kPpRow;
    int r[kPpRow];
#pragma unroll
    for (int h = 0; h < kPpRow; h += 4) {
      int4 e = make_int4(kInf, kInf, kInf, kInf);
      if (h < c) e = *reinterpret_cast<const int4*>(row + h);
      r[h] = h < c ? ptr[e.x] : kInf;
      r[h + 1] = h + 1 < c ? ptr[e.y] : kInf;
      r[h + 2] = h + 2 < c ? ptr[e.z] : kInf;
      r[h + 3] = h + 3 < c ? ptr[e.w] : kInf;
    }
    if (c <= 4) {
      int n = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        bool again = r[q] == kInf;
        int at = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k < q) again |= r[k] == r[q];
          // Distinct smaller entries: the first of each value counts.
          bool first = r[k] < r[q];
#pragma unroll
          for (int j = 0; j < k; ++j) first &= r[j] != r[k];
          at += first;
        }
        if (again) continue;
        row[at] = r[q];
        ++n;
      }
      cnt[i] = n < 2 ? 0 : n;
    } else {
      cnt[i] = pp_store_row(r, row);
    }
  }
}

__global__ void k_iota(int* __restrict__ p, int n) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) p[i] = i;
}

// Output pairs (partner vertex, extremum vertex) by extremum rank; the global
// extremum's partner is the opposite global extremum, an unpaired one -1.
// parent (optional): the vertex of the extremum each one merges into (lmax),
// the global extremum its own, an unpaired one -1.
__global__ void k_pp_out(const int* __restrict__ pair, int ne, const int* __restrict__ ext_li,
                         const int* __restrict__ elist, const int* __restrict__ sad_li,
                         const int* __restrict__ slist, int opposite, int* __restrict__ out,
                         const int* __restrict__ lmax, int* __restrict__ parent) {
  const int stride = gridDim.x * blockDim.x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += stride) {
    const int i = pair[e];
    out[2 * e] = e == ne - 1 ? opposite : (i >= 0 ? slist[sad_li[i]] : -1);
    out[2 * e + 1] = elist[ext_li[e]];
    if (parent)
      parent[e] = e == ne - 1 ? elist[ext_li[e]] : (i >= 0 ? elist[ext_li[lmax[e]]] : -1);
  }
}

}  // namespace extremz

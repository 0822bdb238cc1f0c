// k_touched_tiles by itself: `jobs` fields of one size in one launch, each from the
// state that k_direction_list leaves behind for its listed tiles.
#include <cstring>
#include <vector>

#include "extremz_kernels.cuh"

using namespace extremz;

namespace {
template <class V>
V* device(const V* host, size_t n, bool& ok) {
  void* p = nullptr;
  ok = ok && cudaMalloc(&p, (n ? n : 1) * sizeof(V)) == cudaSuccess &&
       cudaMemcpy(p, host, n * sizeof(V), cudaMemcpyHostToDevice) == cudaSuccess;
  return static_cast<V*>(p);
}
}  // namespace

// dds, das: jobs x W*H*D labels; touch2, touch1: jobs x bitsets of the touched ones;
// listed: jobs x nlist tiles.  Per job: dense (C_JDENSE), count (C_NAFF) and the queue
// (nt entries: tiles, or -1 where this round wrote none).
extern "C" int touched_tiles(int jobs, int W, int H, int D, const int* dds, const int* das,
                             const unsigned* touch2, const unsigned* touch1, const int* listed,
                             int nlist, int stamp, int blocks, int* dense, int* count, int* queue) {
  const int N = W * H * D, words = (N + 31) / 32;
  const int nt = ((W + TX - 1) / TX) * ((H + TY - 1) / TY) * ((D + TZ - 1) / TZ);
  if (jobs > kMaxSel || nlist > nt) return 1;
  bool ok = true;
  std::vector<Job<float>> J(jobs);
  Sel sel;
  std::memset(&sel, 0, sizeof(sel));
  sel.n = jobs;
  for (int j = 0; j < jobs; ++j) {
    std::memset(static_cast<void*>(&J[j]), 0, sizeof(J[j]));
    std::vector<int> ctr(C_COUNT, 0), seen(nt, 0);
    std::vector<unsigned long long> q(nt, 0);
    ctr[C_MFDONE] = ctr[C_CHANGED] = 1;
    ctr[C_WNSTAMP] = stamp - 1;
    ctr[C_TLIST] = ctr[C_NAFF] = nlist;
    for (int k = 0; k < nlist; ++k) {
      const int t = listed[j * nlist + k];
      if (t < 0 || t >= nt) return 1;
      seen[t] = stamp;
      q[k] = (unsigned long long)stamp << 32 | (unsigned)t;
    }
    J[j].dim = Dims{W, H, D, N};
    J[j].ctr = device(ctr.data(), ctr.size(), ok);
    J[j].tseen = device(seen.data(), seen.size(), ok);
    J[j].tqueue = device(q.data(), q.size(), ok);
    J[j].dds = device(dds + (size_t)j * N, N, ok);
    J[j].das = device(das + (size_t)j * N, N, ok);
    J[j].rtouch2 = device(touch2 + (size_t)j * words, words, ok);
    J[j].rtouch1 = device(touch1 + (size_t)j * words, words, ok);
    sel.idx[j] = j;
    sel.off[j] = j * blocks;
  }
  sel.off[jobs] = jobs * blocks;
  Job<float>* dj = device(J.data(), J.size(), ok);
  if (ok) {
    k_touched_tiles<float><<<jobs * blocks, 256>>>(dj, sel);
    ok = cudaDeviceSynchronize() == cudaSuccess;
  }
  for (int j = 0; j < jobs && ok; ++j) {
    std::vector<int> ctr(C_COUNT);
    std::vector<unsigned long long> q(nt);
    ok = cudaMemcpy(ctr.data(), J[j].ctr, C_COUNT * sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(q.data(), J[j].tqueue, nt * 8, cudaMemcpyDeviceToHost) == cudaSuccess;
    dense[j] = ctr[C_JDENSE];
    count[j] = ctr[C_NAFF];
    for (int k = 0; k < nt; ++k)
      queue[j * nt + k] = (int)(q[k] >> 32) == stamp ? (int)(unsigned)q[k] : -1;
  }
  for (Job<float>& x : J)
    for (void* p : {(void*)x.ctr, (void*)x.tseen, (void*)x.tqueue, (void*)x.dds, (void*)x.das,
                    (void*)x.rtouch2, (void*)x.rtouch1})
      cudaFree(p);
  cudaFree(dj);
  return ok ? 0 : 2;
}

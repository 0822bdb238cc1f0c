// Runs queue_take / queue_push (csrc/extremz_queue.h) by simulated blocks on a
// model of relaxed memory.  Every write of a location stays readable until the
// reader has seen a newer one of that location, or has acquired a view that holds
// a newer one: a relaxed load returns any of the readable values.  Read-modify-
// writes act on the newest.  finished() releases the block's view; done() acquires
// it, or not (argument "relaxed").
//
// queue_model acquire|relaxed SEEDS: random searches; prints how many ended with an
// entry that nobody took, and in how many a block waited in vain.
#include <ucontext.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <random>
#include <vector>

#include "extremz_queue.h"

namespace {

using u64 = unsigned long long;
using View = std::vector<int>;  // per location: the oldest version still readable

struct Version {
  u64 value;
  View view;  // released with it
};

struct Machine;
struct Fiber {
  ucontext_t ctx;
  std::unique_ptr<char[]> stack{new char[1 << 16]};
  View view;
  bool live = true;
};

constexpr int kHead = 0, kDone = 1, kPushed = 2, kDense = 3, kEntry = 4;

struct Machine {
  bool acquire;
  std::mt19937 rng;
  int tiles, stale = 2;  // a load takes the newest value at least every `stale` times
  std::vector<std::vector<Version>> mem;
  std::vector<std::vector<int>> graph;
  std::vector<int> seen, searched;
  std::vector<Fiber> fibers;
  ucontext_t main_ctx;
  int cur = -1, gave_up = 0;

  void yield() { swapcontext(&fibers[cur].ctx, &main_ctx); }
  u64 load(int loc, bool acq) {
    yield();
    Fiber& f = fibers[cur];
    const int newest = (int)mem[loc].size() - 1, oldest = f.view[loc];
    const int at = rng() % stale == 0 ? newest : oldest + (int)(rng() % (unsigned)(newest - oldest + 1));
    f.view[loc] = at;
    if (acq)
      for (size_t l = 0; l < f.view.size(); ++l)
        if (l < mem[loc][at].view.size()) f.view[l] = std::max(f.view[l], mem[loc][at].view[l]);
    return mem[loc][at].value;
  }
  void write(int loc, u64 value, bool release) {
    Fiber& f = fibers[cur];
    View v = mem[loc].back().view;  // a read-modify-write continues the release sequence
    f.view[loc] = (int)mem[loc].size();
    if (release) {
      v.resize(f.view.size(), 0);
      for (size_t l = 0; l < v.size(); ++l) v[l] = std::max(v[l], f.view[l]);
    }
    mem[loc].push_back({value, v});
  }
  int add(int loc, bool release) {
    yield();
    const u64 old = mem[loc].back().value;
    write(loc, old + 1, release);
    return (int)old;
  }
};

struct Queue {
  Machine& m;
  int ticket() { return m.add(kHead, false); }
  int place() { return m.add(kPushed, false); }
  void finished() { m.add(kDone, true); }
  int done() { return (int)m.load(kDone, m.acquire); }
  int pushed() { return (int)m.load(kPushed, false); }
  bool dense() { return m.load(kDense, false) != 0; }
  u64 entry(int i) { return m.load(kEntry + i, false); }
  void store(int i, u64 e) {
    m.yield();
    m.write(kEntry + i, e, false);
  }
  void ask_dense() {
    ++m.gave_up;
    m.write(kDense, 1, false);
  }
  void pause() { m.yield(); }
};

constexpr unsigned kStamp = 7;

void block(Machine* m) {
  Queue q{*m};
  for (;;) {
    const int t = extremz::queue_take(q, kStamp, m->tiles, 1000);
    if (t < 0) break;
    ++m->searched[t];
    for (int u : m->graph[t])
      if (!m->seen[u]) {
        m->seen[u] = 1;
        extremz::queue_push(q, kStamp, u, m->tiles);
      }
    q.finished();
  }
  m->fibers[m->cur].live = false;
  m->yield();
}

Machine* g_machine;
void entry_point() { block(g_machine); }

// 1: an entry was left, 2: a block waited in vain.
int run(bool acquire, unsigned seed) {
  Machine m;
  m.acquire = acquire;
  m.rng.seed(seed);
  m.tiles = 4 + (int)(m.rng() % 12);
  m.graph.resize(m.tiles);
  for (int t = 1; t < m.tiles; ++t) m.graph[m.rng() % (unsigned)t].push_back(t);  // a tree from 0
  m.seen.assign(m.tiles, 0);
  m.searched.assign(m.tiles, 0);
  m.mem.assign(kEntry + m.tiles, {Version{0, {}}});
  m.mem[kEntry][0].value = (u64)kStamp << 32;  // the first entry: tile 0
  m.mem[kPushed][0].value = 1;
  m.seen[0] = 1;
  m.fibers.resize(2 + m.rng() % 4);
  g_machine = &m;
  for (Fiber& f : m.fibers) {
    f.view.assign(m.mem.size(), 0);
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.get();
    f.ctx.uc_stack.ss_size = 1 << 16;
    f.ctx.uc_link = nullptr;
    makecontext(&f.ctx, entry_point, 0);
  }
  for (int live = (int)m.fibers.size(); live > 0;) {
    m.cur = (int)(m.rng() % m.fibers.size());
    if (!m.fibers[m.cur].live) continue;
    swapcontext(&m.main_ctx, &m.fibers[m.cur].ctx);
    if (!m.fibers[m.cur].live) --live;
  }
  if (m.gave_up) return 2;
  for (int n : m.searched)
    if (n != 1) return 1;
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  const bool acquire = argc > 1 && !std::strcmp(argv[1], "acquire");
  const int seeds = argc > 2 ? std::atoi(argv[2]) : 1000;
  int count[3] = {0, 0, 0};
  for (int s = 0; s < seeds; ++s) ++count[run(acquire, (unsigned)s)];
  std::printf("left %d waited %d\n", count[1], count[2]);
  return 0;
}

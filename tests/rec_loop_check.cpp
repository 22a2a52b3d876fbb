// Host check of rec_loop (csrc/rec_loop.cuh), the loop in which a CTA's warp
// sets hand chunks and phase nodes to one another through shared memory: its
// source is compiled for host threads, one per thread of the CTA, with the last
// thread of every set held up behind each of the set's barriers, so that what it
// reads late must still be what it was.  Every (chunk, node range) has to be
// handed out once, to all threads of one set, with the chunk's own image.
// A barrier that is not reached for 20 seconds counts as a hang.
// Built and run by tests/test_rec_loop.py; prints "<cases> <mismatches>".
#include <algorithm>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

// ---- the CUDA built-ins that the loop uses ---------------------------------
#undef __shared__
#define __shared__ static
using std::acos;
using std::cos;
using std::fabs;
using std::floor;
using std::log10;
using std::pow;
using std::sin;
using std::sqrt;
inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
template <class T>
T atomicAdd(T* p, T v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
inline double atomicAdd(double* p, double v) { const double o = *p; *p = o + v; return o; }  // (not called)
inline unsigned atomicSub(unsigned* p, unsigned v) { return __atomic_fetch_sub(p, v, __ATOMIC_SEQ_CST); }
inline unsigned atomicOr(unsigned* p, unsigned v) { return __atomic_fetch_or(p, v, __ATOMIC_SEQ_CST); }
inline unsigned atomicXor(unsigned* p, unsigned v) { return __atomic_fetch_xor(p, v, __ATOMIC_SEQ_CST); }
inline unsigned atomicAnd(unsigned* p, unsigned v) { return __atomic_fetch_and(p, v, __ATOMIC_SEQ_CST); }
inline unsigned atomicCAS(unsigned* p, unsigned want, unsigned v) {
  __atomic_compare_exchange_n(p, &want, v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST);
  return want;
}
inline void atomicMax(unsigned long long* p, unsigned long long v) {
  unsigned long long o = __atomic_load_n(p, __ATOMIC_SEQ_CST);
  while (o < v && !__atomic_compare_exchange_n(p, &o, v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {
  }
}
inline int __ldcg(const int* p) { return __atomic_load_n(p, __ATOMIC_SEQ_CST); }
inline int4 __ldcg(const int4* p) { return make_int4(__ldcg(&p->x), __ldcg(&p->y), __ldcg(&p->z), __ldcg(&p->w)); }
inline unsigned __float_as_uint(float f) {
  unsigned u;
  std::memcpy(&u, &f, 4);
  return u;
}
inline void __threadfence_block() { __atomic_thread_fence(__ATOMIC_SEQ_CST); }
inline void __nanosleep(unsigned) { std::this_thread::sleep_for(std::chrono::microseconds(20)); }

struct Barrier {
  std::mutex m;
  std::condition_variable cv;
  int n = 0, in = 0;
  long long round = 0;
  void wait() {
    std::unique_lock<std::mutex> lk(m);
    const long long mine = round;
    if (++in == n) {
      in = 0;
      ++round;
      cv.notify_all();
    } else if (!cv.wait_for(lk, std::chrono::seconds(20), [&] { return round != mine; })) {
      std::printf("hang\n");
      std::fflush(stdout);
      std::_Exit(2);
    }
  }
};
Barrier g_set[32], g_block;
thread_local dim3 t_thread;
dim3 g_block_dim, g_block_id, g_grid_dim;
#define threadIdx t_thread
#define blockDim g_block_dim
#define blockIdx g_block_id
#define gridDim g_grid_dim
inline void __syncthreads() { g_block.wait(); }

namespace ppm {
void set_sync(int set, int n) {
  g_set[set].wait();
  if ((int)t_thread.x == set * n + n - 1) std::this_thread::sleep_for(std::chrono::microseconds(300));
}
void cp_async16(void* dst, const void* src) { std::memcpy(dst, src, 16); }
void cp_async_wait_all() {}
}  // namespace ppm

#include "rec_loop.cuh"

namespace ppm {
namespace {

constexpr int kImage = 256, kElems = 16;

struct Check {
  std::vector<std::vector<int>> taken;  // per record and node: threads that worked on it
  std::mutex m;
  int bad = 0;
};

// The work of a set: counts its threads on each node, compares the chunk's image.
struct CountWork {
  int set, st, ST;
  Check* check;
  int take;
  void fill(ChunkCtx& c, const DevProfile&, const DevSpot&, const RingRec& q) {
    c.n_nodes = q.n_nodes;
    c.n_act = q.n_act;
    c.take = take;
    c.u_mod = q.n_nodes;
  }
  void enter(const ChunkCtx&) {}
  void count(int) {}
  void nodes(const ChunkCtx& c, const ChunkBufs& b, int u) {
    std::lock_guard<std::mutex> lk(check->m);
    if (c.rec < 0 || c.rec >= (int)check->taken.size()) {
      ++check->bad;
      return;
    }
    const unsigned char* image = (const unsigned char*)b.P;
    for (int k = 0; k < kImage; ++k) check->bad += image[k] != (unsigned char)(c.rec + 1);
    for (int k = 0; k < c.n_act; ++k) check->bad += b.j[k] != c.rec * 100 + k;
    for (int k = u; k < std::min(u + take, c.n_nodes); ++k) ++check->taken[c.rec][k];
  }
};

// One launch: grid CTAs one after the other; returns the number of mismatches.
int launch(int ST, int sets, int slots, int n_recs, int grid, int nodes, int take) {
  constexpr int kThreads = 512;
  Check check;
  std::vector<RingRec> recs(n_recs);
  std::vector<int4> ctr(n_recs + 1, make_int4(0, 0, 0, 0));
  std::vector<unsigned short> lists((size_t)n_recs * kElems + 8);
  std::vector<unsigned char> data((size_t)n_recs * kImage);
  for (int r = 0; r < n_recs; ++r) {
    const int n = nodes + r % 3, act = 1 + r % kElems;
    recs[r] = RingRec{0, 0, 0, r, act, r * kElems, n, 1};
    ctr[r] = make_int4(0, 0, n, act);
    std::memset(&data[(size_t)r * kImage], r + 1, kImage);
    for (int k = 0; k < kElems; ++k) lists[(size_t)r * kElems + k] = (unsigned short)(r * 100 + k);
    check.taken.emplace_back(n, 0);
  }
  std::vector<DevProfile> profile(1);
  KernelArgs a{};
  a.profiles = profile.data();
  a.shape.rec_slots = slots;
  a.shape.rec_slot_bytes = kImage + 2 * kElems;
  a.shape.off_F = 64;
  RingWork& W = a.rings;
  W.data = data.data();
  W.stride = kImage;
  W.off_hidx = 128;
  W.off_slice = kImage;
  W.recs = recs.data();
  W.ctr = ctr.data();
  W.lists = (unsigned char*)lists.data();
  W.elem_bytes = 2;
  W.n_recs = &n_recs;
  W.rec_cap = n_recs;
  std::vector<unsigned char> sm((size_t)slots * a.shape.rec_slot_bytes);
  g_block_dim = dim3(ST * sets);
  g_grid_dim = dim3(grid);
  g_block.n = ST * sets;
  for (int s = 0; s < sets; ++s) g_set[s].n = ST;
  for (int cta = 0; cta < grid; ++cta) {
    g_block_id = dim3(cta);
    std::vector<std::thread> threads;
    for (int t = 0; t < ST * sets; ++t)
      threads.emplace_back([&, t] {
        t_thread = dim3(t);
        CountWork w{t / ST, t % ST, ST, &check, take};
        rec_loop<kThreads>(a, sm.data(), w);
      });
    for (auto& th : threads) th.join();
  }
  for (const auto& r : check.taken)
    for (int n : r) check.bad += n != ST;
  return check.bad;
}

}  // namespace
}  // namespace ppm

int main() {
  int cases = 0, bad = 0;
  // threads per set, sets, slots, records, CTAs, nodes, nodes a take: sets of one and several warps; records for some
  // of the slots, for all, and more than all CTAs' slots
  const int c[][7] = {{64, 2, 2, 1, 1, 5, 1}, {64, 2, 2, 2, 1, 4, 1},  {64, 2, 2, 9, 1, 3, 1}, {96, 1, 1, 5, 1, 2, 1},
                      {64, 1, 4, 3, 2, 3, 1}, {64, 3, 2, 11, 3, 2, 1}, {32, 4, 2, 7, 1, 6, 2}, {32, 3, 4, 2, 2, 9, 4}};
  for (const auto& k : c) {
    ++cases;
    const int n = ppm::launch(k[0], k[1], k[2], k[3], k[4], k[5], k[6]);
    if (n) std::fprintf(stderr, "case %d: %d\n", cases, n);
    bad += n != 0;
  }
  std::printf("%d %d\n", cases, bad);
  return bad != 0;
}

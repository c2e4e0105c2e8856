// cuda_on_host.h -- test infrastructure: runs the library's own kernels on the host
// CPU, one block at a time, for tests that must not depend on how a GPU happens to
// schedule its warps.
//
// The threads of a block are fibers (ucontext).  A fiber runs until it waits, at a
// block barrier or a warp operation; the lowest-numbered thread that can go on runs
// next.  So thread 0 is as far ahead of the others as the barriers allow: shared
// memory that it overwrites while another thread has still to read it is
// overwritten every time, where a GPU would nearly always be lucky.
// __shared__ variables are function-local statics, device memory is host memory.
#pragma once

#include <cuda_runtime.h>  // vector types; no CUDA library is linked

#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <type_traits>
#include <utility>
#include <vector>

#undef __global__
#undef __device__
#undef __host__
#undef __shared__
#undef __forceinline__
#undef __noinline__
#undef __launch_bounds__
#undef __grid_constant__
#define __global__
#define __device__
#define __host__
#define __shared__ static
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __grid_constant__

inline uint3 threadIdx;
inline uint3 blockIdx;
inline dim3 blockDim;
inline dim3 gridDim;

namespace emu {

struct WarpOp {  // the operation that the lanes of one mask are meeting at
  uint32_t arrived = 0;
  uint64_t gen = 0;
  uint64_t val[2][32];
};
struct Engine {
  static constexpr size_t kStack = 64 * 1024;
  std::vector<ucontext_t> fiber;
  std::vector<unsigned char> done;
  std::vector<char> stacks;
  std::vector<const uint64_t *> wait_at;  // the counter a fiber waits for, and its old value
  std::vector<uint64_t> wait_old;
  std::vector<unsigned char> smem;
  std::map<std::pair<uint32_t, uint32_t>, WarpOp> ops;
  ucontext_t sched;
  unsigned cur = 0, live = 0, at_bar = 0;
  uint64_t bar_gen = 0;
  int bar_or[2], bar_and[2];
  const std::function<void()> *body = nullptr;
};
inline Engine &engine() {
  static Engine e;
  return e;
}
inline void set_thread(unsigned t) {
  engine().cur = t;
  threadIdx = make_uint3(t, 0, 0);
}
inline void wait_change(const uint64_t *at, uint64_t old) {
  Engine &e = engine();
  const unsigned me = e.cur;
  if (*at != old) return;
  e.wait_at[me] = at;
  e.wait_old[me] = old;
  swapcontext(&e.fiber[me], &e.sched);
  e.wait_at[me] = nullptr;
}
inline void release_barrier() {
  Engine &e = engine();
  e.at_bar = 0;
  ++e.bar_gen;
  e.bar_or[e.bar_gen & 1] = 0;
  e.bar_and[e.bar_gen & 1] = 1;
}
// the block's barrier (exited threads do not count, as on a GPU)
inline uint64_t barrier(int pred) {
  Engine &e = engine();
  const uint64_t g = e.bar_gen;
  e.bar_or[g & 1] |= pred != 0;
  e.bar_and[g & 1] &= pred != 0;
  if (++e.at_bar == e.live)
    release_barrier();
  else
    wait_change(&e.bar_gen, g);
  return g;
}
// every lane of mask brings a value; returns the lanes' values
template <class V>
inline const uint64_t *exchange(uint32_t mask, V v) {
  Engine &e = engine();
  const uint32_t lane = e.cur & 31;
  if (!((mask >> lane) & 1u)) {
    std::fprintf(stderr, "emu: lane %u outside its mask %08x\n", lane, mask);
    std::abort();
  }
  WarpOp &op = e.ops[{e.cur >> 5, mask}];
  const uint64_t g = op.gen;
  uint64_t raw = 0;
  std::memcpy(&raw, &v, sizeof(V));
  op.val[g & 1][lane] = raw;
  op.arrived |= 1u << lane;
  if (op.arrived == mask) {
    op.arrived = 0;
    ++op.gen;
  } else {
    wait_change(&op.gen, g);
  }
  return op.val[g & 1];
}
template <class V>
inline V pick(uint64_t raw) {
  V v;
  std::memcpy(&v, &raw, sizeof(V));
  return v;
}

inline void fiber_main() {
  Engine &e = engine();
  (*e.body)();
  e.done[e.cur] = 1;
  if (--e.live && e.at_bar == e.live) release_barrier();
}
inline uint4 *dynamic_smem() { return reinterpret_cast<uint4 *>(engine().smem.data()); }

// Runs body once per thread of every block of the grid; false when threads wait
// for others that never come, or without end.
inline bool launch(unsigned grid, unsigned block, size_t smem, const std::function<void()> &body) {
  Engine &e = engine();
  gridDim = dim3(grid);
  blockDim = dim3(block);
  e.body = &body;
  e.fiber.resize(block);
  e.stacks.resize((size_t)block * Engine::kStack);
  e.wait_at.assign(block, nullptr);
  e.wait_old.assign(block, 0);
  for (unsigned b = 0; b < grid; ++b) {
    e.smem.assign(smem + 16, 0xA5);
    blockIdx = make_uint3(b, 0, 0);
    e.done.assign(block, 0);
    e.ops.clear();
    e.live = block;
    e.at_bar = 0;
    e.bar_or[e.bar_gen & 1] = 0;
    e.bar_and[e.bar_gen & 1] = 1;
    for (unsigned t = 0; t < block; ++t) {
      getcontext(&e.fiber[t]);
      e.fiber[t].uc_stack.ss_sp = e.stacks.data() + (size_t)t * Engine::kStack;
      e.fiber[t].uc_stack.ss_size = Engine::kStack;
      e.fiber[t].uc_link = &e.sched;
      makecontext(&e.fiber[t], fiber_main, 0);
    }
    bool ran = true;
    uint64_t left = 1ull << 26;  // resumptions: a loop that never ends fails the launch
    while (e.live && ran) {
      ran = false;
      for (unsigned t = 0; t < block; ++t) {
        if (e.done[t] || (e.wait_at[t] && *e.wait_at[t] == e.wait_old[t])) continue;
        set_thread(t);
        swapcontext(&e.sched, &e.fiber[t]);
        ran = --left != 0;
        if (!ran) return false;
      }
    }
    if (e.live) return false;
  }
  return true;
}

}  // namespace emu

inline void __syncthreads() { emu::barrier(0); }
inline int __syncthreads_or(int p) {
  const uint64_t g = emu::barrier(p);
  return emu::engine().bar_or[g & 1];
}
inline int __syncthreads_and(int p) {
  const uint64_t g = emu::barrier(p);
  return emu::engine().bar_and[g & 1];
}
inline void __syncwarp(uint32_t m = 0xffffffffu) { emu::exchange(m, 0u); }
inline uint32_t __activemask() { return 0xffffffffu; }
inline void __threadfence() {}
template <class V>
inline V __shfl_sync(uint32_t m, V v, uint32_t src) {
  return emu::pick<V>(emu::exchange(m, v)[src & 31]);
}
template <class V>
inline V __shfl_xor_sync(uint32_t m, V v, uint32_t x) {
  const uint32_t lane = threadIdx.x & 31;
  return emu::pick<V>(emu::exchange(m, v)[lane ^ x]);
}
template <class V>
inline V __shfl_up_sync(uint32_t m, V v, uint32_t d) {
  const uint32_t lane = threadIdx.x & 31;
  return emu::pick<V>(emu::exchange(m, v)[lane >= d ? lane - d : lane]);
}
template <class F>
inline uint32_t emu_fold(uint32_t m, uint32_t v, F f) {
  const uint64_t *p = emu::exchange(m, v);
  bool first = true;
  uint32_t r = 0;
  for (uint32_t l = 0; l < 32; ++l)
    if ((m >> l) & 1u) {
      r = first ? (uint32_t)p[l] : f(r, (uint32_t)p[l]);
      first = false;
    }
  return r;
}
inline uint32_t __ballot_sync(uint32_t m, int p) {
  const uint32_t bit = p ? 1u << (threadIdx.x & 31) : 0u;
  return emu_fold(m, bit, [](uint32_t a, uint32_t b) { return a | b; });
}
inline int __any_sync(uint32_t m, int p) { return __ballot_sync(m, p) != 0; }
inline uint32_t __reduce_add_sync(uint32_t m, uint32_t v) {
  return emu_fold(m, v, [](uint32_t a, uint32_t b) { return a + b; });
}
inline uint32_t __reduce_max_sync(uint32_t m, uint32_t v) {
  return emu_fold(m, v, [](uint32_t a, uint32_t b) { return a > b ? a : b; });
}
inline uint32_t __match_any_sync(uint32_t m, uint32_t v) {
  const uint64_t *p = emu::exchange(m, v);
  uint32_t r = 0;
  for (uint32_t l = 0; l < 32; ++l)
    if (((m >> l) & 1u) && (uint32_t)p[l] == v) r |= 1u << l;
  return r;
}
inline int __popc(uint32_t v) { return __builtin_popcount(v); }
inline int __ffs(uint32_t v) { return __builtin_ffs((int)v); }
inline int __clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }
inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
inline uint32_t __float_as_uint(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  return u;
}
inline float __uint_as_float(uint32_t u) { return emu::pick<float>(u); }
inline long long __double_as_longlong(double d) {
  long long u;
  std::memcpy(&u, &d, 8);
  return u;
}
inline double __longlong_as_double(long long u) { return emu::pick<double>((uint64_t)u); }
inline size_t __cvta_generic_to_shared(const void *) { return 0; }
template <class V>
inline V __ldcg(const V *p) {
  return *p;
}
template <class V, class F>
inline V emu_rmw(V *p, F f) {
  const V old = *p;
  *p = f(old);
  return old;
}
template <class V, class W>
inline V atomicAdd(V *p, W v) { return emu_rmw(p, [v](V o) { return o + (V)v; }); }
template <class V, class W>
inline V atomicSub(V *p, W v) { return emu_rmw(p, [v](V o) { return o - (V)v; }); }
template <class V, class W>
inline V atomicOr(V *p, W v) { return emu_rmw(p, [v](V o) { return o | (V)v; }); }
template <class V, class W>
inline V atomicMin(V *p, W v) { return emu_rmw(p, [v](V o) { return o < (V)v ? o : (V)v; }); }
template <class V, class W>
inline V atomicMax(V *p, W v) { return emu_rmw(p, [v](V o) { return o > (V)v ? o : (V)v; }); }
template <class V, class W>
inline V atomicExch(V *p, W v) { return emu_rmw(p, [v](V) { return (V)v; }); }
template <class V>
inline V atomicCAS(V *p, V c, V v) { return emu_rmw(p, [c, v](V o) { return o == c ? v : o; }); }
template <class V>
inline V min(V a, V b) { return a < b ? a : b; }
template <class V>
inline V max(V a, V b) { return a > b ? a : b; }

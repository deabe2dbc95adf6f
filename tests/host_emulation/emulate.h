// emulate.h -- one thread block on the host, its threads as coroutines.  A
// thread runs without interruption to its next barrier, and the order in
// which the threads of a block take their turns is chosen by the caller: with
// ascending and with descending turns, any two accesses of two threads that no
// barrier orders take place in both orders, so that code which needs one of
// them gives another result in one of the two.  Asynchronous copies land when
// their thread waits for them.
#pragma once
#include <cuda_runtime.h>
#include <ucontext.h>

#include <utility>
#include <vector>

emu_dim3 threadIdx, blockIdx, blockDim, gridDim;

namespace emu {

enum State { READY, AT_WARP, AT_BLOCK, DONE };
struct Thread {
  ucontext_t ctx;
  std::vector<char> stack;
  State state = READY;
  std::vector<std::pair<void *, const void *>> copies;
};
struct Block {
  std::vector<Thread> th;
  ucontext_t sched;
  int cur = -1;
  void (*body)(void *) = nullptr;
  void *arg = nullptr;
};
inline Block *&current() {
  static Block *b = nullptr;
  return b;
}
inline void entry() {
  Block *b = current();
  b->body(b->arg);
  b->th[b->cur].state = DONE;
  swapcontext(&b->th[b->cur].ctx, &b->sched);
}

// Runs body(arg) as every thread of one block; false if the threads wait for
// each other for good (a barrier that some of a warp's threads never reach).
inline bool run_block(int threads, bool descending, emu_dim3 block, void (*body)(void *), void *arg) {
  Block b;
  b.th.resize(threads);
  b.body = body;
  b.arg = arg;
  current() = &b;
  blockDim = {(unsigned)threads, 1, 1};
  blockIdx = block;
  for (Thread &t : b.th) {
    t.stack.resize(1 << 17);
    getcontext(&t.ctx);
    t.ctx.uc_stack.ss_sp = t.stack.data();
    t.ctx.uc_stack.ss_size = t.stack.size();
    t.ctx.uc_link = nullptr;
    makecontext(&t.ctx, entry, 0);
  }
  for (;;) {
    bool ran = false;
    for (int q = 0; q < threads; q++) {
      const int i = descending ? threads - 1 - q : q;
      if (b.th[i].state != READY) continue;
      ran = true;
      b.cur = i;
      threadIdx = {(unsigned)i, 0, 0};
      swapcontext(&b.sched, &b.th[i].ctx);
    }
    int done = 0, at_block = 0;
    for (const Thread &t : b.th) done += t.state == DONE, at_block += t.state == AT_BLOCK;
    if (done == threads) return true;
    bool released = false;
    if (done + at_block == threads) {
      for (Thread &t : b.th)
        if (t.state == AT_BLOCK) t.state = READY;
      released = true;
    }
    for (int w = 0; w < threads; w += 32) {
      const int end = w + 32 < threads ? w + 32 : threads;
      bool all = true, any = false;
      for (int i = w; i < end; i++) {
        all = all && (b.th[i].state == AT_WARP || b.th[i].state == DONE);
        any = any || b.th[i].state == AT_WARP;
      }
      if (!all || !any) continue;
      for (int i = w; i < end; i++)
        if (b.th[i].state == AT_WARP) b.th[i].state = READY;
      released = true;
    }
    if (!ran && !released) return false;
  }
}

}  // namespace emu

void emu_barrier(bool block) {
  emu::Block *b = emu::current();
  emu::Thread &t = b->th[b->cur];
  t.state = block ? emu::AT_BLOCK : emu::AT_WARP;
  swapcontext(&t.ctx, &b->sched);
}
void emu_copy16(void *dst, const void *src) {
  emu::Block *b = emu::current();
  b->th[b->cur].copies.push_back({dst, src});
}
void emu_copies_wait() {
  emu::Block *b = emu::current();
  for (auto &c : b->th[b->cur].copies) memcpy(c.first, c.second, 16);
  b->th[b->cur].copies.clear();
}

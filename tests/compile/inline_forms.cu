// Inline entry methods and invoke_single on the GPU, in SM-level mode and
// (compiled with -DCHARMING_GPU_LEVEL) in GPU-level mode. Every chare sends
// its neighbour M messages whose refnums fall, so all but the last come
// early; the inline entry method that takes them moves the refnum up, hands
// every second one to a block entry method, which reports to chare 0 with
// invoke_single, and after the last waits (async_wait, an inline entry
// method) on a word that is set. The messages from one chare to another stay
// in order, so with the last chare's report all notes must be in, each once.
#include <charming.h>

constexpr int M = 24;

struct Rung : charm::chare {
  int ref, done, notes, bad;
  __device__ Rung() : ref(0), done(0), notes(0), bad(0) {}
};
#ifdef CHARMING_GPU_LEVEL
__device__ charm::chare_proxy<Rung>* rungs;
#else
__shared__ charm::chare_proxy<Rung>* rungs;
#endif
__device__ unsigned long long word = 1;

enum : int { START, TAKE, BLOCK, WOKEN, DONE, NOTE, END };

__device__ void on_start(Rung& c, void*) {
  for (int k = 0; k < M; k++) {
    int b[2] = {c.i, M - 1 - k};
    rungs->invoke((c.i + 1) % c.n, TAKE, b, sizeof(b), M - 1 - k);
  }
}
__device__ int on_take(Rung& c, void* arg) {
  const int* b = static_cast<const int*>(arg);
  if (b[0] != (c.i + c.n - 1) % c.n || b[1] != c.ref) c.bad++;
  rungs->set_refnum(c.i, ++c.ref);
  if (c.ref == M)
    rungs->async_wait(reinterpret_cast<uint64_t*>(&word), 1, charm::CMP_EQ, 1, c.i, WOKEN);
  return c.ref & 1 ? -1 : BLOCK;
}
__device__ void on_block(Rung& c, void* arg) {
  if (threadIdx.x == 0) {  // of every block in GPU-level mode: one message all the same
    const int bad = static_cast<const int*>(arg)[1] != c.ref - 1;
    rungs->invoke_single(0, NOTE, &bad, sizeof(bad));
  }
}
__device__ int on_woken(Rung& c, void* arg) {
  const int bad = c.bad + (arg != nullptr);
  rungs->invoke_single(0, DONE, &bad, sizeof(bad));
  return -1;
}
__device__ int on_done(Rung& c, void* arg) {
  c.bad += *static_cast<const int*>(arg);
  if (++c.done < c.n) return -1;
  printf("inline forms: chares %d, done %d, notes %d of %d, bad %d\n", c.n, c.done, c.notes, c.n * (M / 2), c.bad);
  return END;
}
__device__ int on_note(Rung& c, void* arg) {
  c.bad += *static_cast<const int*>(arg);
  c.notes++;
  return -1;
}
__device__ void on_end(Rung&, void*) { charm::end(); }

__device__ void charm::main(int argc, char** argv, size_t* argvs, int pe) {
  if (charm::pe_thread() == 0) {
    rungs = new charm::chare_proxy<Rung>();
    rungs->add_entry_method<&on_start>();
    rungs->add_inline_entry_method<&on_take>();
    rungs->add_entry_method<&on_block>();
    rungs->add_inline_entry_method<&on_woken>();
    rungs->add_inline_entry_method<&on_done>();
    rungs->add_inline_entry_method<&on_note>();
    rungs->add_entry_method<&on_end>();
    rungs->create(charm::n_pes() > 1 ? 2 * charm::n_pes() : 5);
    for (int c = rungs->start_idx; c <= rungs->end_idx; c++) rungs->set_refnum(c, 0);
  }
  charm::pe_sync();
  charm::barrier();
  const int lo = rungs->start_idx, hi = rungs->end_idx;
  for (int c = lo; c <= hi; c++) rungs->invoke(c, START);
}

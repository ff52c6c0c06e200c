// CPU check of the halo puts' index arithmetic (TEST INFRASTRUCTURE ONLY).
//
// put_rects of apps/jacobi2d.cu, compiled for the host, moves side halos of
// grids whose rows lie so far apart that the last ones start more than 2^31
// elements into the grid (a tall chare has such offsets too; here few rows of
// a huge pitch, so that only a few pages of the reserved address range are
// touched). Every cell must arrive, and the cells around must stay.
//
// The scheduler's part of the runtime is not linked: put_rects calls none of
// it (the Makefile leaves those symbols unresolved).
#include "cuda_host_shim.h"
#include "../../charming_b200/csrc/apps/jacobi2d.cu"

#include <sys/mman.h>

thread_local emu_dim3 threadIdx{0, 0, 0};
thread_local emu_dim3 blockIdx{0, 0, 0};
emu_dim3 blockDim{1, 1, 1};
emu_dim3 gridDim{1, 1, 1};

namespace {

template <typename T>
T* reserve(size_t n) {
  void* p = mmap(nullptr, n * sizeof(T), PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  return p == MAP_FAILED ? nullptr : static_cast<T*>(p);
}

// A halo of nr rows of nc elements; off: first column of both sides.
template <typename T>
int check(int nr, int nc, int src_pitch, int dst_pitch, int off, int nt) {
  const size_t ns = (size_t)nr * src_pitch, nd = (size_t)nr * dst_pitch;
  T *src = reserve<T>(ns), *dst = reserve<T>(nd);
  if (!src || !dst) {
    printf("no address space\n");
    return 1;
  }
  constexpr int V = jac::traits<T>::VEC;
  for (int r = 0; r < nr; r++)
    for (int x = 0; x < nc; x++) src[(size_t)r * src_pitch + off + x] = (T)(1 + r * nc + x);
  const bool vec = nc % V == 0 && off % V == 0;
  put_batch& b = s_puts;
  b.n = 1;
  b.src[0] = src + off;
  b.dst[0] = dst + off;
  b.dst_pitch[0] = dst_pitch;
  b.unit[0] = vec ? V : 1;
  b.nu[0] = vec ? nc / V : nc;
  b.nr[0] = nr;
  for (int t = 0; t < nt; t++) put_rects<T>(1, src_pitch, t, nt);
  int bad = 0;
  for (int r = 0; r < nr; r++)
    for (int x = -1; x <= nc; x++) {
      const T want = x >= 0 && x < nc ? (T)(1 + r * nc + x) : (T)0;
      bad += dst[(size_t)r * dst_pitch + off + x] != want;
    }
  munmap(src, ns * sizeof(T));
  munmap(dst, nd * sizeof(T));
  if (bad) printf("%d bad cells: nr %d nc %d pitches %d %d off %d threads %d\n", bad, nr, nc, src_pitch, dst_pitch, off, nt);
  return bad ? 1 : 0;
}

template <typename T>
int check_all() {
  int bad = 0;
  for (int nt : {1, 32, 96, 480}) {
    bad += check<T>(11, 8, 1 << 28, 1 << 28, 32, nt);         // whole vectors, both sides wide
    bad += check<T>(11, 8, 64, 1 << 28, 32, nt);              // only the neighbour's rows
    bad += check<T>(11, 8, 1 << 28, 64, 32, nt);              // only this chare's
    bad += check<T>(11, 3, (1 << 28) + 32, 1 << 28, 33, nt);  // element copies
    bad += check<T>(600, 4, 96, 128, 32, nt);                 // several turns per thread
  }
  return bad;
}

}  // namespace

int main() {
  const int bad = check_all<float>() + check_all<double>();
  printf(bad ? "failed\n" : "ok\n");
  return bad ? 1 : 0;
}

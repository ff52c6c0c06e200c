// charming_jacobi2d_sweeps_noalloc: Jacobi sweeps of one grid that allocate
// no device memory.
//
// Who needs it: code that runs where allocating is not allowed or not
// possible, e.g. a host that hands this library device buffers from its own
// pool or arena and forbids allocations outside it, a caller inside a
// region where cudaMalloc would synchronise the device, or a process whose
// memory is already fully reserved. charming_jacobi2d_create/run allocate
// the chare grids, staging buffers and the scheduler's inboxes; this entry
// point needs only the caller's input and output grids plus a fixed scratch
// array that is part of the library image.
//
// Scratch: g_noalloc_scratch below, 16 MiB, one per GPU that loads the
// library, held until the process exits. It holds the second (ping-pong)
// grid. Every call overwrites the part it uses before reading it, so
// nothing in it has to start at zero. All calls share it: calls that
// overlap on the GPU (from several host threads, or on several streams)
// race on it and must be serialised by the caller.
//
// The arithmetic is the chares' (jac::stencil), so the result equals the
// grid that charming_jacobi2d_run produces for the same input, bit for bit.
#include "jacobi_sweep.cuh"
#include "../host.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace {

constexpr size_t NOALLOC_SCRATCH_BYTES = 16u << 20;
constexpr int NOALLOC_MAX_DEVICES = 64;

// Device-side scratch; in host code this name is only a host stand-in for
// the symbol, never a device address (see scratch_on_current_device).
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

std::mutex g_scratch_mu;
void* g_scratch_ptr[NOALLOC_MAX_DEVICES];  // device address of the scratch, per device
int g_sm_count[NOALLOC_MAX_DEVICES];       // multiprocessors of each device

// Resolves the scratch's device address and the device's multiprocessor
// count on the current device, once per device (the first call on a device
// does this).
int scratch_on_current_device(void** out, int* sms) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return charm_host::cuda_fail(e, "jacobi2d noalloc: cudaGetDevice");
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
    charm_host::set_error_text("jacobi2d noalloc: device ordinal out of range");
    return CHARMING_ERR_CONFIG;
  }
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return charm_host::cuda_fail(e, "jacobi2d noalloc: cudaGetSymbolAddress");
    int n = 0;
    e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return charm_host::cuda_fail(e, "jacobi2d noalloc: cudaDeviceGetAttribute");
    g_sm_count[dev] = n > 0 ? n : 1;
    g_scratch_ptr[dev] = p;
  }
  *out = g_scratch_ptr[dev];
  *sms = g_sm_count[dev];
  return CHARMING_OK;
}

// L sweeps src -> dst in one pass over a row-major (ny+2) x (nx+2) grid, the
// boundary ring included (it is copied), with the chares' wavefront
// (jac::deep_step): a warp streams the rows of one item, a strip of 32
// vectors times a run of rows, and keeps the levels between in registers.
// Grids of at most 16 vectors a row need no strips: a warp takes 32 / G items
// of G lanes, each a whole row wide (the boundary columns at both ends are kept
// at every level, so what the shuffles bring from the next item is not used).
// 1 x 690000 FP32, 20 sweeps: 98 us; 1033 in strips with most lanes idle, 144
// with one launch per sweep.
// Rows have any alignment here: ALIGNED (16-byte aligned grids whose rows are
// whole vectors) loads and stores vectors, else element by element. The next
// NA_U rows are in flight in registers. FIX: the item's levels can meet the
// boundary ring. The grids stay in L2; small ones are bound by the launch and
// the chain of a warp's rows, large ones by instruction issue. 254^2 FP64, 20
// sweeps: 34 us (96 with one launch per sweep, two copies and a 64-bit division
// per point); 2046^2 FP32, 100 sweeps: 320 us (1870 so).
constexpr int NA_U = 4;

// v: the lane's vector, own: it stores it; rows r0 .. r1 - 1 (none if r1 <= r0)
// in `run` + 2 L steps, the same number for all lanes of the warp. GRP: items of
// fewer lanes than a warp's, compiled apart (one kernel for both made wide grids
// 1 to 2 % slower).
template <typename T, int L, bool ALIGNED, bool FIX, bool GRP>
__device__ __forceinline__ void noalloc_item(const T* __restrict__ src, T* __restrict__ dst, int nx, int ny,
    int v, bool own, int r0, int r1, int run) {
  constexpr int V = jac::traits<T>::VEC, LH = (L + 1) / 2, U = NA_U;
  const int col0 = v * V, W = nx + 2;
  jac::deep_lane<T> ln;
  ln.v = v;
  ln.col0 = col0;
  ln.own = own;
  ln.anyfix = false;
#pragma unroll
  for (int k = 0; k < V; k++) {
    ln.fixc[k] = col0 + k == 0 || col0 + k == nx + 1;
    ln.inw[k] = false;
  }
  ln.fix_r0 = 0;
  ln.fix_r1 = ny + 1;
  const int qs = r0 - L, qe = r1 - 1 + L, qend = GRP ? r0 + run - 1 + L : qe;
  // columns and rows off the grid: its nearest ones, never used by a result
  int off[V];
#pragma unroll
  for (int k = 0; k < V; k++) off[k] = min(max(col0 + k, 0), nx + 1);
  const int voff = min(max(col0, 0), ALIGNED ? W - V : 0);
  T buf[U][V], x[V];
  int next = qs;
  auto load = [&](int u) {
    const T* row = src + (size_t)min(max(next, 0), ny + 1) * W;
    next++;
    if (ALIGNED) {
      const typename jac::vec_of<T>::type t = *reinterpret_cast<const typename jac::vec_of<T>::type*>(row + voff);
      jac::vec_to<T>(t, buf[u]);
    } else {
#pragma unroll
      for (int k = 0; k < V; k++) buf[u][k] = row[off[k]];
    }
  };
#pragma unroll
  for (int u = 0; u < U; u++) load(u);
  jac::deep_state<T, L> S;
#pragma unroll
  for (int l = 0; l < L; l++)
#pragma unroll
    for (int k = 0; k < V; k++) S.P[l][k] = S.X[l][k] = (T)0;
#pragma unroll
  for (int k = 0; k < V; k++) S.D[k] = 0.0;
  double acc = 0.0;
  T* op = dst + (size_t)r0 * W + col0;
  const int nput = ln.own ? W - col0 : 0;
  int q = qs;
  // the first steps of the fill work on the lower half of the levels only
  constexpr int F = 2 * LH / U * U;
#pragma unroll 1
  for (; q < qs + F; q += U) {
#pragma unroll
    for (int u = 0; u < U; u++) {
#pragma unroll
      for (int k = 0; k < V; k++) x[k] = buf[u][k];
      load(u);
      jac::deep_step<T, false, L, LH, FIX>(S, x, q + u, ln, r0, r1, acc);
    }
  }
#pragma unroll 1
  for (; q <= qend; q += U) {
#pragma unroll
    for (int u = 0; u < U; u++) {
#pragma unroll
      for (int k = 0; k < V; k++) x[k] = buf[u][k];
      load(u);
      jac::deep_step<T, false, L, L, FIX>(S, x, q + u, ln, r0, r1, acc);
      const bool full = q + u >= qs + 2 * L && q + u <= qe;  // a row r0 .. r1 - 1 is complete
      const int n = full ? nput : 0;
      if (ALIGNED) {
        jac::put_vec(op, x, n);
      } else {
#pragma unroll
        for (int k = 0; k < V; k++)
          if (k < n) op[k] = x[k];
      }
      op += full ? W : 0;
    }
  }
}

template <typename T, int L, bool ALIGNED, bool GRP>
__global__ void __launch_bounds__(128) noalloc_pass_kernel(const T* __restrict__ src, T* __restrict__ dst, int nx,
    int ny, int strips, int group, int run_rows, int warps) {
  constexpr int V = jac::traits<T>::VEC, E = (L + V - 1) / V, SS = 32 - 2 * E;
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = (int)(threadIdx.x & 31);
  if (w >= warps) return;
  const int nv = (nx + 2 + V - 1) / V;
  if (GRP) {
    const int v = lane & (group - 1), r0 = (w * (32 / group) + lane / group) * run_rows;
    noalloc_item<T, L, ALIGNED, true, true>(src, dst, nx, ny, v, v < nv, r0, min(ny + 2, r0 + run_rows), run_rows);
  } else {
    const int own0 = w % strips * SS, nown = min(SS, nv - own0), v = own0 - E + lane;
    const bool own = lane >= E && lane < E + nown;
    const int r0 = w / strips * run_rows, r1 = min(ny + 2, r0 + run_rows);
    const bool edge = own0 - E <= 0 || (own0 + nown + E) * V > nx + 1 || r0 - L <= 0 || r1 - 1 + L >= ny + 1;
    if (edge) noalloc_item<T, L, ALIGNED, true, false>(src, dst, nx, ny, v, own, r0, r1, 0);
    else noalloc_item<T, L, ALIGNED, false, false>(src, dst, nx, ny, v, own, r0, r1, 0);
  }
}

constexpr int NA_LMAX = 8;

// One pass of L sweeps: how the rows are split, and its cost in SM cycles. A
// pass costs its launch and first loads (5000), then its rows: a warp's step
// through one level takes 55 cycles alone and 38 of its SM sub-partition's
// when several warps share it. (Measured on a B200 to within a quarter; the
// choice only needs their ratio.) Chosen on every call, 8 lengths times about
// 20 splits, so with few divisions.
struct pass_plan {
  int run_rows, strips, group, warps;
  double cycles;
};
template <typename T>
pass_plan plan_pass(int L, int nx, int ny, int sms) {
  constexpr int V = jac::traits<T>::VEC;
  const int E = (L + V - 1) / V, SS = 32 - 2 * E, rows = ny + 2, nv = (nx + 2 + V - 1) / V;
  int group = 32, sh = 0;  // 1 << sh items a warp
  for (; group > 1 && group / 2 >= nv; group /= 2) sh++;
  const int strips = group < 32 ? 1 : (nv + SS - 1) / SS;
  const double inv_parts = 1.0 / (4.0 * sms);
  pass_plan best{0, strips, group, 0, 1e300};
  for (int R = 4; R <= 128; R += R < 16 ? 2 : R < 64 ? 8 : 32) {
    const long long items = (long long)strips * ((rows + R - 1) / R);
    const long long warps = (items + (1 << sh) - 1) >> sh;
    const double per_part = std::ceil((double)warps * inv_parts);
    const double c = 5000.0 + (double)(std::min(R, rows) + 2 * L) * L * std::max(55.0, 38.0 * per_part);
    if (c < best.cycles) best = pass_plan{R, strips, group, (int)warps, c};
    if (R >= rows) break;
  }
  return best;
}

template <typename T, int L>
void launch_pass(const T* src, T* dst, int nx, int ny, const pass_plan& p, bool aligned, int sms) {
  // few warps: blocks of one warp, so that they spread over the SMs
  const int threads = p.warps <= 4 * sms ? 32 : p.warps <= 8 * sms ? 64 : 128;
  const int blocks = (int)(((long long)p.warps * 32 + threads - 1) / threads);
  auto fn = p.group < 32 ? (aligned ? noalloc_pass_kernel<T, L, true, true> : noalloc_pass_kernel<T, L, false, true>)
                         : (aligned ? noalloc_pass_kernel<T, L, true, false> : noalloc_pass_kernel<T, L, false, false>);
  fn<<<blocks, threads, 0, 0>>>(src, dst, nx, ny, p.strips, p.group, p.run_rows, p.warps);
}
template <typename T>
void launch_pass_of(int L, const T* src, T* dst, int nx, int ny, const pass_plan& p, bool aligned, int sms) {
  switch (L) {
    case 1: return launch_pass<T, 1>(src, dst, nx, ny, p, aligned, sms);
    case 2: return launch_pass<T, 2>(src, dst, nx, ny, p, aligned, sms);
    case 3: return launch_pass<T, 3>(src, dst, nx, ny, p, aligned, sms);
    case 4: return launch_pass<T, 4>(src, dst, nx, ny, p, aligned, sms);
    case 5: return launch_pass<T, 5>(src, dst, nx, ny, p, aligned, sms);
    case 6: return launch_pass<T, 6>(src, dst, nx, ny, p, aligned, sms);
    case 7: return launch_pass<T, 7>(src, dst, nx, ny, p, aligned, sms);
    default: return launch_pass<T, 8>(src, dst, nx, ny, p, aligned, sms);
  }
}

template <typename T>
int run_sweeps(int nx, int ny, int sweeps, const T* in, T* out, T* scratch, int sms) {
  const size_t bytes = ((size_t)nx + 2) * ((size_t)ny + 2) * sizeof(T);
  cudaError_t e = cudaSuccess;
  if (sweeps == 0) {
    e = cudaMemcpyAsync(out, in, bytes, cudaMemcpyDeviceToDevice, 0);
  } else {
    // passes of the length that costs least per sweep, as even as they go:
    // the first `longer` of them are one sweep longer than the rest
    int best = 1;
    double cost = 1e300;
    pass_plan plans[NA_LMAX + 1];
    for (int L = 1; L <= NA_LMAX; L++) {
      plans[L] = plan_pass<T>(L, nx, ny, sms);
      const double c = plans[L].cycles * ((sweeps + L - 1) / L);
      if (c < cost) {
        cost = c;
        best = L;
      }
    }
    const int n = (sweeps + best - 1) / best, base = sweeps / n, longer = sweeps % n;
    const bool aligned = ((size_t)nx + 2) * sizeof(T) % 16 == 0 &&
                         ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    // the last pass writes `out`; every pass writes its whole target, ring
    // included
    const T* src = in;
    for (int k = 0; k < n && e == cudaSuccess; k++) {
      T* dst = (n - 1 - k) % 2 == 0 ? out : scratch;
      const int L = base + (k < longer ? 1 : 0);
      launch_pass_of<T>(L, src, dst, nx, ny, plans[L], aligned, sms);
      e = cudaGetLastError();
      src = dst;
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  if (e != cudaSuccess) return charm_host::cuda_fail(e, "jacobi2d noalloc sweeps");
  return CHARMING_OK;
}

}  // namespace

extern "C" int charming_jacobi2d_sweeps_noalloc(int dtype, int nx, int ny, int sweeps,
    const void* dev_in, void* dev_out) {
  if (dtype != CHARMING_F64 && dtype != CHARMING_F32) {
    charm_host::set_error_text("jacobi2d noalloc: dtype must be CHARMING_F64 or CHARMING_F32");
    return CHARMING_ERR_CONFIG;
  }
  if (nx < 1 || ny < 1 || sweeps < 0 || !dev_in || !dev_out) {
    charm_host::set_error_text("jacobi2d noalloc: bad arguments");
    return CHARMING_ERR_CONFIG;
  }
  const size_t esz = dtype == CHARMING_F64 ? 8 : 4;
  // A misaligned element pointer would fault in the kernel's loads.
  if (reinterpret_cast<uintptr_t>(dev_in) % esz || reinterpret_cast<uintptr_t>(dev_out) % esz) {
    charm_host::set_error_text("jacobi2d noalloc: dev_in and dev_out must be aligned to the element size");
    return CHARMING_ERR_CONFIG;
  }
  const unsigned long long cells = ((unsigned long long)nx + 2) * ((unsigned long long)ny + 2);
  if (cells > NOALLOC_SCRATCH_BYTES / esz) {
    charm_host::set_error_text(
        "jacobi2d noalloc: grid larger than the 16 MiB scratch ((nx+2)*(ny+2)*element size must "
        "be <= 16 MiB)");
    return CHARMING_ERR_CONFIG;
  }
  const char* i0 = static_cast<const char*>(dev_in);
  const char* o0 = static_cast<const char*>(dev_out);
  const size_t bytes = cells * esz;
  if (i0 < o0 + bytes && o0 < i0 + bytes) {
    charm_host::set_error_text("jacobi2d noalloc: input and output grids overlap");
    return CHARMING_ERR_CONFIG;
  }
  void* scratch = nullptr;
  int sms = 1;
  int rc = scratch_on_current_device(&scratch, &sms);
  if (rc) return rc;
  if (dtype == CHARMING_F64)
    return run_sweeps<double>(nx, ny, sweeps, static_cast<const double*>(dev_in),
                              static_cast<double*>(dev_out), static_cast<double*>(scratch), sms);
  return run_sweeps<float>(nx, ny, sweeps, static_cast<const float*>(dev_in),
                           static_cast<float*>(dev_out), static_cast<float*>(scratch), sms);
}

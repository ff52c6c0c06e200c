// 3-D Jacobi sweeps (7-point, FP64): the stencil of the reference's
// standalone kernel, examples/jacobi-kernel/jacobi_kernel.cu:36-48,
//   new[i][j][k] = (t + t[i-1] + t[i+1] + t[j-1] + t[j+1] + t[k-1] + t[k+1])
//                  * 0.142857
// added left to right in FP64, then one multiply by the double literal
// 0.142857 (DIVIDEBY7 there, :16). Grid layout as its IDX_3D: x fastest,
// (nx+2) x (ny+2) x (nz+2) doubles with a fixed boundary shell. Unlike the
// reference's benchmark loop (which launches temp -> new_temp every time),
// sweeps alternate between two buffers, so the result is `sweeps` Jacobi
// iterations.
//
// One kernel, L sweeps per pass over the grid (3 or 2; 1 for an odd last
// sweep): a block owns a strip of 32 vectors of 2 columns times the rows of
// its warps (RY each) and marches up z, one plane per step. A thread keeps,
// per level and row, the newest plane of the level below (X) and the partial
// sums of the first six terms around it (P, taken when that plane arrived);
// the next plane closes them, (P + zp) * 0.142857, the adds in the same
// order. So a plane's way through all levels needs no neighbours, and one
// block barrier per plane (the rows at the warps' edges go through shared
// memory, columns by shuffle) serves every level. The planes stream through a
// private ring of shared-memory slots per thread (cp.async). Tiles overlap by
// L cells on each side; the boundary shell is kept at every level and copied.
// Bound by the load/store pipe (ring copies, edge rows, shuffles) and, on
// small grids, by the chain of a plane's step. GLUP/s against one sweep per
// pass (32 x 16 tiles, planes by cp.async): 256^3 399 (255), 512^3 507 (290),
// 640^3 578 (293), 128^3 219, 299 x 300 x 250 432 with its row copies over 300
// sweeps (232).
#include "suite.cuh"
#ifndef CHARMING_HOST_EMULATION
#include "jacobi_sweep.cuh"
#include "../host.cuh"
#include <algorithm>
#include <climits>
#include <cmath>

namespace {

constexpr int J3_S = 4;       // planes in the ring
constexpr int J3_NWMAX = 16;  // warps per block

template <int L>
struct j3_geom {
  static constexpr int E = (L + 1) / 2;      // vectors lost at each strip edge
  static constexpr int SS = 32 - 2 * E;      // vectors a strip owns
};
// rings of J3_S planes (RY rows per warp), and the edge rows of each warp,
// level and step parity
constexpr size_t j3_smem(int warps, int L, int RY) { return (size_t)warps * 512 * (J3_S * RY + 4 * L); }

// Grids of at most 16 vectors a row need no strips: a warp takes the rows of
// 32 >> gs groups of 1 << gs lanes, each a whole row wide (the shell columns at
// both ends are kept at every level, so what the shuffles bring from the next
// group is not used). gs 5: whole warps. 1 x 1 x 300000, 3 sweeps: 154 us (1790
// in strips of whole warps and at most 64 runs, 1279 with one sweep per pass),
// 1 x 200000 x 4 51 (960, 392), 20 x 3000 x 100, 6 sweeps 135 (260, 355).
struct j3_plan {
  int warps, gs, yown, yblocks, zrun, zruns, strips;
  double cost;
};

// GRP: groups of fewer lanes than a warp's (compiled apart: in one kernel with
// them wide grids took 4 to 10 % longer).
template <int L, int RY, bool FIX, bool GRP>
__device__ __forceinline__ void j3_tile(const double* __restrict__ in, double* __restrict__ out, int nx, int ny,
    int nz, int pitch, int zrun, int yown, int gs, double2* smem) {
  using G = j3_geom<L>;
  constexpr unsigned FULL = 0xffffffffu;
  // lane, group of lanes (a warp) and groups; GW lanes lie between two groups
  const int GS = GRP ? gs : 5, GW = 1 << GS, lane = (int)threadIdx.x & (GW - 1), grp = (int)threadIdx.x >> GS;
  const int ngrp = (int)blockDim.x >> GS, NT = (int)blockDim.x, W = nx + 2;
  const size_t plane = (size_t)pitch * (ny + 2);
  constexpr int E = GRP ? 0 : G::E;
  const int own0 = (int)blockIdx.x * G::SS, col0 = (own0 - E + lane) * 2;
  const int nv = (W + 1) / 2;
  const bool own = lane >= E && lane < E + min(GRP ? GW : G::SS, nv - own0);
  const int y0 = (int)blockIdx.y * yown, yt = y0 - L + grp * RY;  // the group's first row
  const int z0 = (int)blockIdx.z * zrun, z1 = min(nz + 2, z0 + zrun);
  const int qs = z0 - L, qe = z1 - 1 + L;
  const bool fixc0 = col0 == 0 || col0 == nx + 1, fixc1 = col0 + 1 == nx + 1;
  // this thread's ring slots and the exchange rows
  double2* ring = smem + threadIdx.x;
  double2* ex = smem + (size_t)J3_S * RY * NT;  // [parity][level][first, last][thread]
  // columns and rows off the grid: its nearest ones, never used by a result
  long long goff[RY];
  int nput[RY];
  bool rowfix[RY];
  const int c0 = min(max(col0, 0), pitch - 2);
#pragma unroll
  for (int i = 0; i < RY; i++) {
    const int y = yt + i;
    goff[i] = (long long)min(max(y, 0), ny + 1) * pitch + c0;
    rowfix[i] = y == 0 || y == ny + 1;
    nput[i] = own && y >= y0 && y < min(y0 + yown, ny + 2) ? W - col0 : 0;
  }
  int next = qs;
  auto fetch = [&](int slot) {
    const double* src = in + (size_t)min(max(next, 0), nz + 1) * plane;
    next++;
#pragma unroll
    for (int i = 0; i < RY; i++) {
      const unsigned dst = jac::smem_u32(ring + (slot * RY + i) * NT);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + goff[i]) : "memory");
    }
    jac::cp_async_commit();
  };
  for (int k = 0; k < J3_S - 1; k++) fetch(k);
  double2 P[L][RY], X[L][RY];
#pragma unroll
  for (int l = 0; l < L; l++)
#pragma unroll
    for (int i = 0; i < RY; i++) P[l][i] = X[l][i] = make_double2(0.0, 0.0);
  int slot = 0, par = 0;
  double* oplane = out + col0;
#pragma unroll 1
  for (int q = qs; q <= qe; q++) {
    double2 v[L + 1][RY];
    jac::cp_async_wait<J3_S - 2>();
#pragma unroll
    for (int i = 0; i < RY; i++) v[0][i] = ring[(slot * RY + i) * NT];
    fetch(slot == 0 ? J3_S - 1 : slot - 1);  // the slot of the plane read before
    slot = slot + 1 == J3_S ? 0 : slot + 1;
    double2* e = ex + (size_t)par * L * 2 * NT + threadIdx.x;
    par ^= 1;
#pragma unroll
    for (int l = 0; l < L; l++) {
      e[(2 * l) * NT] = v[l][0];
      e[(2 * l + 1) * NT] = v[l][RY - 1];
      const int z = q - l - 1;  // plane of level l + 1 computed now
      const bool zfix = FIX && (z == 0 || z == nz + 1);
#pragma unroll
      for (int i = 0; i < RY; i++) {
        double2 o;
        o.x = __dmul_rn(__dadd_rn(P[l][i].x, v[l][i].x), 0.142857);
        o.y = __dmul_rn(__dadd_rn(P[l][i].y, v[l][i].y), 0.142857);
        if (FIX) {
          o.x = zfix || rowfix[i] || fixc0 ? X[l][i].x : o.x;
          o.y = zfix || rowfix[i] || fixc1 ? X[l][i].y : o.y;
        }
        v[l + 1][i] = o;
      }
    }
    const bool full = q >= qs + 2 * L;  // plane q - L is complete
#pragma unroll
    for (int i = 0; i < RY; i++) {
      const int n = full ? nput[i] : 0;
      double* p = oplane + (long long)(q - L) * (long long)plane + (yt + i) * (long long)pitch;
      const double t[2] = {v[L][i].x, v[L][i].y};
      jac::put_vec(p, t, n);
    }
    __syncthreads();  // the edge rows of every group and level are there
#pragma unroll
    for (int l = 0; l < L; l++) {
      // the rows above and below the group's (at the block's edge: its own,
      // never used by a result)
      const double2 up = e[(2 * l + 1) * NT - (grp > 0 ? GW : 0)];
      const double2 dn = e[(2 * l) * NT + (grp + 1 < ngrp ? GW : 0)];
#pragma unroll
      for (int i = 0; i < RY; i++) {
        const double2 c = v[l][i];
        const double left = __shfl_up_sync(FULL, c.y, 1), right = __shfl_down_sync(FULL, c.x, 1);
        const double2 ym = i == 0 ? up : v[l][i - 1], yp = i == RY - 1 ? dn : v[l][i + 1];
        P[l][i].x = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(c.x, left), c.y), ym.x), yp.x), X[l][i].x);
        P[l][i].y = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(c.y, c.x), right), ym.y), yp.y), X[l][i].y);
      }
#pragma unroll
      for (int i = 0; i < RY; i++) X[l][i] = v[l][i];
    }
  }
  jac::cp_async_wait<0>();
}

template <int L, int RY, bool GRP>
__global__ void __launch_bounds__(32 * J3_NWMAX, 1) jacobi3d_pass_kernel(const double* __restrict__ in,
    double* __restrict__ out, int nx, int ny, int nz, int pitch, int zrun, int yown, int gs) {
  extern __shared__ __align__(16) double2 j3_shared[];
  using G = j3_geom<L>;
  const int own0 = (int)blockIdx.x * G::SS, y0 = (int)blockIdx.y * yown, z0 = (int)blockIdx.z * zrun;
  // the tile's levels can meet the shell
  const bool edge = GRP || own0 - G::E <= 0 || (own0 + G::SS + G::E) * 2 > nx + 1 || y0 - L <= 0 ||
                    y0 - L + (int)(blockDim.x >> 5) * RY > ny + 1 || z0 - L <= 0 || z0 + zrun + L > nz + 1;
  if (edge) j3_tile<L, RY, true, GRP>(in, out, nx, ny, nz, pitch, zrun, yown, gs, j3_shared);
  else j3_tile<L, RY, false, false>(in, out, nx, ny, nz, pitch, zrun, yown, gs, j3_shared);
}

// Warps per block, rows per block and planes per run: the fewest steps of
// all resident warps, over the waves that the launch takes. A block's rows
// are its groups' less the 2L of the overlap, a run streams 2L planes more
// than it writes; with few blocks the warps of an SM are bound by latency
// (taken as 8 warps' worth of time). Groups of few lanes make short runs of
// many blocks cheap, so there the three steps that a run takes to start count
// too (in the choice for wide grids they cost 256^3 17 %).
template <int L, int RY>
j3_plan j3_choose(int nx, int ny, int nz, int n_sms) {
  const int nv = (nx + 2 + 1) / 2;
  int gs = 5;
  while (gs > 1 && (1 << (gs - 1)) >= nv) gs--;
  const int start = gs < 5 ? 3 : 0, strips = gs < 5 ? 1 : (nv + j3_geom<L>::SS - 1) / j3_geom<L>::SS;
  j3_plan best{};
  best.cost = 1e300;
  for (int nw = 1; nw <= J3_NWMAX; nw++) {
    const int ymax = (nw * 32 >> gs) * RY - 2 * L;
    if (ymax < 1) continue;
    const int yb = (ny + 2 + ymax - 1) / ymax;
    if (yb > 65535 && nw < J3_NWMAX) continue;  // grid limit
    const int yown = (ny + 2 + yb - 1) / yb;
    const int per_sm = std::max(1, std::min(J3_NWMAX / nw, (int)((227u << 10) / (j3_smem(nw, L, RY) + 1024))));
    const long long tiles = (long long)strips * yb;
    // (past 64 runs in steps of an eighth: tall grids of few rows)
    for (int runs = 1; runs <= 16384; runs += runs < 64 ? 1 : runs / 8) {
      const int zr = (nz + 2 + runs - 1) / runs;
      if (runs > 1 && zr < 4 * L) break;
      const long long blocks = tiles * ((nz + 2 + zr - 1) / zr);
      const double waves = std::ceil((double)blocks / ((double)n_sms * per_sm));
      const double resident = std::min<double>(per_sm, std::ceil((double)blocks / n_sms));
      const double cost = waves * (zr + 2 * L + start) * std::max(8.0, resident * nw) * RY / L;
      if (cost < best.cost * 0.999) best = j3_plan{nw, gs, yown, yb, zr, (nz + 2 + zr - 1) / zr, strips, cost};
      if (zr == 1) break;
    }
  }
  return best;
}

template <int L, int RY>
cudaError_t j3_pass(const double* in, double* out, int nx, int ny, int nz, int pitch, const j3_plan& p,
    cudaStream_t s) {
  auto fn = p.gs < 5 ? jacobi3d_pass_kernel<L, RY, true> : jacobi3d_pass_kernel<L, RY, false>;
  const size_t smem = j3_smem(p.warps, L, RY);
  cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)j3_smem(J3_NWMAX, L, RY));
  if (e != cudaSuccess) return e;
  fn<<<dim3(p.strips, p.yblocks, p.zruns), 32 * p.warps, smem, s>>>(in, out, nx, ny, nz, pitch, p.zrun, p.yown, p.gs);
  return cudaGetLastError();
}

// Rows of an odd number of columns are kept in rows one double longer, so that
// every row starts on a 16-byte boundary (element copies and stores made the
// sweeps of a 255^3 grid 1.65 times as long); these copy them between, inside
// the time that the call reports.
// A block takes a run of rows, its threads every 256th cell of them, eight in
// flight; a thread's next cell is found by adding. Both ways for 299 x 300 x 250
// 139 us (310 with a row per block), 33 x 300 x 3000 203 (428 with a row per
// warp), 0.77 to 0.81 of the copy bandwidth.
__global__ void __launch_bounds__(256) j3_repitch_kernel(const double* __restrict__ src, double* __restrict__ dst,
    int W, int sp, int dp, long long rows, int run) {
  constexpr int B = 8;
  const long long r0 = (long long)blockIdx.x * run;
  const long long left = rows - r0;
  const int nr = (int)(left < run ? left : run), dr = 256 / W, dc = 256 - dr * W;
  src += r0 * sp;
  dst += r0 * dp;
  int r = (int)threadIdx.x / W, c = (int)threadIdx.x - r * W;
  while (r < nr) {
    double v[B];
    long long off[B];
    bool in[B];
#pragma unroll
    for (int k = 0; k < B; k++) {
      in[k] = r < nr;
      if (in[k]) v[k] = src[(long long)r * sp + c];
      off[k] = (long long)r * dp + c;
      r += dr;
      c += dc;
      if (c >= W) {
        c -= W;
        r++;
      }
    }
#pragma unroll
    for (int k = 0; k < B; k++)
      if (in[k]) dst[off[k]] = v[k];
  }
}
cudaError_t j3_repitch(const double* src, double* dst, int W, int sp, int dp, long long rows,
    cudaStream_t s) {
  // runs of about 2048 cells, at most 2^31 - 1 of them
  const long long run = std::max<long long>(std::max(1, 2048 / W), (rows + INT_MAX - 1) / INT_MAX);
  j3_repitch_kernel<<<(unsigned)((rows + run - 1) / run), 256, 0, s>>>(src, dst, W, sp, dp, rows, (int)run);
  return cudaGetLastError();
}

// `sweeps` sweeps from a, alternating between a and b (a pass writes its whole
// target, shell included); returns the buffer holding the result.
double* jacobi3d_run(double* a, double* b, int nx, int ny, int nz, int pitch, int sweeps, cudaStream_t s,
    cudaError_t* err) {
  const int n_sms = charm_host::info().n_sms;
  *err = cudaSuccess;
  const j3_plan p3 = j3_choose<3, 2>(nx, ny, nz, n_sms), p2 = j3_choose<2, 3>(nx, ny, nz, n_sms),
                p1 = j3_choose<1, 3>(nx, ny, nz, n_sms);
  // Three sweeps per pass take fewer plane steps but overlap by more rows, and
  // one of their row steps costs 1.1 to 1.26 of the other's. 256^3: 42 us per
  // sweep against 47 with two, 128^3 9.5 against 12.3; 512^3 276 against 265.
  const bool three = p3.cost * 1.24 < p2.cost;
  while (sweeps > 0 && *err == cudaSuccess) {
    if (three && sweeps >= 3) {
      *err = j3_pass<3, 2>(a, b, nx, ny, nz, pitch, p3, s);
      sweeps -= 3;
    } else if (sweeps >= 2) {
      *err = j3_pass<2, 3>(a, b, nx, ny, nz, pitch, p2, s);
      sweeps -= 2;
    } else {
      *err = j3_pass<1, 3>(a, b, nx, ny, nz, pitch, p1, s);
      sweeps--;
    }
    std::swap(a, b);
  }
  return a;
}

}  // namespace

extern "C" int charming_jacobi3d(int nx, int ny, int nz, int sweeps, double* grid, double* out_ms) {
  int rc = charm_host::ensure_init();
  if (rc) return rc;
  if (nx < 1 || ny < 1 || nz < 1 || sweeps < 0 || !grid) return CHARMING_ERR_CONFIG;
  const size_t n = ((size_t)nx + 2) * ((size_t)ny + 2) * ((size_t)nz + 2);
  // device rows start on 16-byte boundaries; a grid of odd rows passes through
  // b on its way in and through the other buffer on its way out
  const int W = nx + 2, pitch = W + (W & 1);
  const long long rows = ((long long)ny + 2) * ((long long)nz + 2);
  const size_t np = (size_t)pitch * (size_t)rows;
  double *a = nullptr, *b = nullptr;
  cudaError_t e = cudaMalloc(&a, np * 8);
  if (e == cudaSuccess) e = cudaMalloc(&b, np * 8);
  cudaStream_t s = charm_host::stream();
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (e == cudaSuccess) e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(pitch == W ? a : b, grid, n * 8, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaEventRecord(e0, s);
  if (e == cudaSuccess && pitch != W) e = j3_repitch(b, a, W, W, pitch, rows, s);
  double* res = a;
  if (e == cudaSuccess) res = jacobi3d_run(a, b, nx, ny, nz, pitch, sweeps, s, &e);
  double* flat = pitch == W ? res : res == a ? b : a;
  if (e == cudaSuccess && pitch != W) e = j3_repitch(res, flat, W, pitch, W, rows, s);
  if (e == cudaSuccess) e = cudaEventRecord(e1, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(grid, flat, n * 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  float ms = 0.f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
  if (out_ms) *out_ms = ms;
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(a);
  cudaFree(b);
  return charm_host::cuda_fail(e, "jacobi3d");
}
#endif

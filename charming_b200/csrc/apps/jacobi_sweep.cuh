// Jacobi sweep of one chare block, executed inside an entry method by all
// threads of the PE block.
//
// Arithmetic (reference examples/jacobi2d/jacobi2d.cu:327-334):
//   new = (c + l + r + u + d) * 0.2, added left to right in T, one multiply
//   by the double 0.2 for double grids. Float grids (the reference has none)
//   add in float and multiply by 0.2 as the float pair C_HI + C_LO
//   (C_HI = 0.2f, C_LO = the float nearest 0.2 - C_HI) with one FMA:
//   fma(s, C_HI, s * C_LO), within an ulp of the product with the double
//   0.2 and without its two conversions. Written with _rn intrinsics so no
//   contraction can change it.
//
// Block layout in HBM (per chare, two buffers): rows 0..h+1 (0 and h+1 are
// ghost rows), row pitch `pitch` elements (a multiple of 128 bytes); column
// c in 0..w+1 sits at element OFF-1+c, so the first interior column starts
// on a 128-byte boundary (OFF = 128 / sizeof(T)).
//
// Two implementations with identical results:
//   sweep_direct: warps walk column strips down the rows, keeping three
//                 rows in registers (each input row loaded once per strip).
//   sweep_tma:    rows stream through a ring of shared-memory slots filled
//                 by cp.async.bulk (TMA 1-D bulk copies, no multicast), one
//                 mbarrier per slot; each input row is read from HBM once
//                 per column tile, so the compulsory traffic is one read and
//                 one write per point (16 B/LUP FP64, 8 B/LUP FP32).
#pragma once

#include <climits>
#include "suite.cuh"
#include "jacobi_types.cuh"

namespace jac {

template <typename T> struct traits;
template <> struct traits<double> {
  static constexpr int VEC = 2;   // elements per 16-byte vector
  static constexpr int OFF = 16;  // element offset of interior column 1
  static constexpr int TW_MAX = 1024;
};
template <> struct traits<float> {
  static constexpr int VEC = 4;
  static constexpr int OFF = 32;
  static constexpr int TW_MAX = 2048;
};

__device__ __forceinline__ double stencil(double c, double l, double r, double u, double d) {
  return __dmul_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(c, l), r), u), d), 0.2);
}
constexpr float STENCIL_C_HI = 0.2f;                     // 0x3e4ccccd
constexpr float STENCIL_C_LO = -2.9802322831784522e-09f;  // 0xb14ccccd: 0.2 - C_HI, rounded
__device__ __forceinline__ float stencil(float c, float l, float r, float u, float d) {
  float s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(c, l), r), u), d);
  return __fmaf_rn(s, STENCIL_C_HI, __fmul_rn(s, STENCIL_C_LO));
}
// Residual term (S(u) - u)^2 with S in FP64.
template <typename T>
__device__ __forceinline__ double resid2(T c, T l, T r, T u, T d) {
  double s = __dmul_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn((double)c, (double)l), (double)r),
                                           (double)u), (double)d), 0.2);
  double e = __dsub_rn(s, (double)c);
  return __dmul_rn(e, e);
}

template <typename T>
struct block_view {
  T* base;      // element (row 0, column 0 of the pitched layout)
  int pitch;    // elements
  __device__ __forceinline__ T* row(int r) const { return base + (size_t)r * pitch; }
  // pointer to column c (0..w+1) of row r
  __device__ __forceinline__ T* at(int r, int c) const {
    return base + (size_t)r * pitch + traits<T>::OFF - 1 + c;
  }
};

// Computes VEC outputs of one row from the 5 input vectors and stores the
// valid ones. mid points at interior column j0 of the row (vector aligned),
// left/right are the scalars at j0-1 and j0+VEC. Returns the residual sum.
template <typename T, bool RESID>
__device__ __forceinline__ double compute_vec(const T* up, const T* mid, const T* dn, T left,
    T right, T* out, int nvalid) {
  constexpr int V = traits<T>::VEC;
  T u[V], m[V], d[V], o[V];
  if (V == 2) {
    double2 a = *reinterpret_cast<const double2*>(up);
    double2 b = *reinterpret_cast<const double2*>(mid);
    double2 c = *reinterpret_cast<const double2*>(dn);
    u[0] = (T)a.x; u[1] = (T)a.y; m[0] = (T)b.x; m[1] = (T)b.y; d[0] = (T)c.x; d[1] = (T)c.y;
  } else {
    float4 a = *reinterpret_cast<const float4*>(up);
    float4 b = *reinterpret_cast<const float4*>(mid);
    float4 c = *reinterpret_cast<const float4*>(dn);
    u[0] = (T)a.x; u[1] = (T)a.y; u[2] = (T)a.z; u[3] = (T)a.w;
    m[0] = (T)b.x; m[1] = (T)b.y; m[2] = (T)b.z; m[3] = (T)b.w;
    d[0] = (T)c.x; d[1] = (T)c.y; d[2] = (T)c.z; d[3] = (T)c.w;
  }
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < V; k++) {
    T l = (k == 0) ? left : m[k - 1];
    T r = (k == V - 1) ? right : m[k + 1];
    o[k] = stencil(m[k], l, r, u[k], d[k]);
    if (RESID && k < nvalid) acc += resid2<T>(m[k], l, r, u[k], d[k]);
  }
  if (nvalid == V) {
    if (V == 2) {
      *reinterpret_cast<double2*>(out) = make_double2((double)o[0], (double)o[1]);
    } else {
      *reinterpret_cast<float4*>(out) = make_float4((float)o[0], (float)o[1], (float)o[2], (float)o[3]);
    }
  } else {
    #pragma unroll
    for (int k = 0; k < V; k++)  // static indices keep o[] in registers
      if (k < nvalid) out[k] = o[k];
  }
  return acc;
}

// ---------------------------------------------------------------------------
// PTX helpers: mbarriers, bulk copies, per-thread async copies.
// ---------------------------------------------------------------------------
#ifndef CHARMING_HOST_EMULATION
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned long long* b) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" :: "r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(smem_u32(b)),
               "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* b, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done) : "r"(smem_u32(b)), "r"(parity) : "memory");
  return done != 0;
}
// 1-D bulk copy global -> shared, completion counted on the mbarrier.
// Both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes,
    unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(b)) : "memory");
}
// 16-byte asynchronous global -> shared copy (zero fill when src_bytes is 0),
// committed per row; wait_group<N> waits until at most N groups are pending.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, unsigned src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(smem_u32(dst)), "l"(src),
               "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
// The multi-sweep pass's ring of rows, addressed in the shared window, and
// its stores: the first n of a lane's VEC values (n >= VEC: one 16-byte
// store), predicated so that the row loop has no branch in it.
using ring_addr = unsigned;
__device__ __forceinline__ ring_addr to_ring(void* p) { return smem_u32(p); }
__device__ __forceinline__ void ring_fetch(ring_addr a, const void* src, unsigned src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(a), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void ring_read(ring_addr a, double (&x)[2]) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x[0]), "=d"(x[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ring_read(ring_addr a, float (&x)[4]) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void put_vec(double* p, const double (&x)[2], int n) {
  asm volatile("{\n .reg .pred f, h;\n setp.ge.s32 f, %3, 2;\n setp.eq.s32 h, %3, 1;\n"
               " @f st.global.v2.f64 [%0], {%1, %2};\n @h st.global.f64 [%0], %1;\n}"
               :: "l"(p), "d"(x[0]), "d"(x[1]), "r"(n) : "memory");
}
__device__ __forceinline__ void put_vec(float* p, const float (&x)[4], int n) {
  asm volatile("{\n .reg .pred f, a, b, c;\n setp.ge.s32 f, %5, 4;\n setp.eq.s32 a, %5, 1;\n"
               " setp.eq.s32 c, %5, 3;\n setp.eq.or.s32 b, %5, 2, c;\n"
               " @f st.global.v4.f32 [%0], {%1, %2, %3, %4};\n @b st.global.v2.f32 [%0], {%1, %2};\n"
               " @a st.global.f32 [%0], %1;\n @c st.global.f32 [%0+8], %3;\n}"
               :: "l"(p), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "r"(n) : "memory");
}
// Two floats in one instruction, each with the rounding of the single one.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ bool mbar_test_wait(unsigned long long* b, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done) : "r"(smem_u32(b)), "r"(parity) : "memory");
  return done != 0;
}
#else
// The CPU check of the chare code models these (tests/emu).
void mbar_init(unsigned long long* b, unsigned count);
void mbar_inval(unsigned long long* b);
void mbar_expect_tx(unsigned long long* b, unsigned bytes);
bool mbar_try_wait(unsigned long long* b, unsigned parity);
bool mbar_test_wait(unsigned long long* b, unsigned parity);
void mbar_arrive(unsigned long long* b);
void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar);
inline void fence_proxy_async_global() {}
inline void fence_proxy_async_smem() {}
inline void fence_mbar_init() {}
// per-thread copies: done at once on the host
inline void cp_async16(void* dst, const void* src, unsigned src_bytes) {
  memset(dst, 0, 16);
  if (src_bytes) memcpy(dst, src, src_bytes);
}
inline void cp_async_commit() {}
template <int N> inline void cp_async_wait() {}
using ring_addr = char*;
inline ring_addr to_ring(void* p) { return static_cast<char*>(p); }
inline void ring_fetch(ring_addr a, const void* src, unsigned src_bytes) { cp_async16(a, src, src_bytes); }
template <typename T, int V> inline void ring_read(ring_addr a, T (&x)[V]) { memcpy(x, a, 16); }
template <typename T, int V> inline void put_vec(T* p, const T (&x)[V], int n) {
  for (int k = 0; k < V && k < n; k++) p[k] = x[k];
}
struct f32x2 { float a, b; };
inline f32x2 pack2(float a, float b) { return {a, b}; }
inline void unpack2(f32x2 v, float& a, float& b) { a = v.a; b = v.b; }
inline f32x2 add2(f32x2 x, f32x2 y) { return {x.a + y.a, x.b + y.b}; }
inline f32x2 mul2(f32x2 x, f32x2 y) { return {x.a * y.a, x.b * y.b}; }
inline f32x2 fma2(f32x2 x, f32x2 y, f32x2 z) { return {fmaf(x.a, y.a, z.a), fmaf(x.b, y.b, z.b)}; }
#endif

// ---------------------------------------------------------------------------
// Direct-load sweep, simple form: thread i of the block handles vectors
// i, i+n, ... of the (h rows x ceil(w/VEC) vectors) output. Used for blocks
// of fewer than 32 threads.
// ---------------------------------------------------------------------------
template <typename T, bool RESID>
__device__ double sweep_simple(block_view<T> in, block_view<T> out, int w, int h) {
  constexpr int V = traits<T>::VEC;
  const int nv = (w + V - 1) / V;
  const long long total = (long long)nv * h;
  double acc = 0.0;
  for (long long x = threadIdx.x; x < total; x += blockDim.x) {
    int r = (int)(x / nv) + 1;
    int v = (int)(x % nv);
    int j0 = 1 + v * V;
    const T* mid = in.at(r, j0);
    int nvalid = min(V, w - v * V);
    acc += compute_vec<T, RESID>(in.at(r - 1, j0), mid, in.at(r + 1, j0), mid[-1], mid[V],
                                 out.at(r, j0), nvalid);
  }
  return acc;
}

// ---------------------------------------------------------------------------
// Direct-load sweep, strip walker. The block's work is split into items: a
// column strip of 32*J vectors (lane l of a warp owns vectors l, l+32, ...)
// times a run of rows. A warp walks its rows top to bottom keeping the
// rows above, at and below the output row in registers, so each input row
// is loaded once per strip; it loads G rows ahead at a time, which keeps
// G*J 16-byte loads per thread in flight. Left/right neighbours come from
// the neighbouring lanes by shuffle; only the strip's two edge columns are
// loaded as scalars. No block barrier inside the sweep.
// ---------------------------------------------------------------------------
template <typename T> struct vec_of;
template <> struct vec_of<double> { using type = double2; };
template <> struct vec_of<float> { using type = float4; };

template <typename T, int J>
struct walk_row {
  typename vec_of<T>::type v[J];
  T left, right;  // columns just outside the strip (same for all lanes)
};

template <typename T>
__device__ __forceinline__ T vec_elem(const double2& x, int k) { return (T)(k == 0 ? x.x : x.y); }
template <typename T>
__device__ __forceinline__ T vec_elem(const float4& x, int k) {
  return (T)(k == 0 ? x.x : k == 1 ? x.y : k == 2 ? x.z : x.w);
}

// Loads row r of a strip: vector v_j = vbase + lane + 32 j when v_j <= nv
// (vector nv holds the right ghost column and padding, inside the pitched
// row), plus the two edge scalars.
template <typename T, int J>
__device__ __forceinline__ void walk_load(walk_row<T, J>& R, const block_view<T>& in, int r,
    int vbase, int nv, int lane, bool has_right) {
  constexpr int V = traits<T>::VEC;
  using VT = typename vec_of<T>::type;
  const T* row = in.at(r, 1);
#pragma unroll
  for (int j = 0; j < J; j++) {
    int v = vbase + lane + 32 * j;
    if (v <= nv) R.v[j] = *reinterpret_cast<const VT*>(row + (size_t)v * V);
    else R.v[j] = VT{};
  }
  R.left = row[(size_t)vbase * V - 1];
  R.right = has_right ? row[(size_t)(vbase + 32 * J) * V] : (T)0;
}

template <typename T, bool RESID, int J>
__device__ __forceinline__ double walk_compute(const walk_row<T, J>& U, const walk_row<T, J>& M,
    const walk_row<T, J>& D, T* orow, int vbase, int w, int lane) {
  constexpr int V = traits<T>::VEC;
  constexpr unsigned FULL = 0xffffffffu;
  using VT = typename vec_of<T>::type;
  double acc = 0.0;
  T first[J], last[J];
#pragma unroll
  for (int j = 0; j < J; j++) {
    first[j] = vec_elem<T>(M.v[j], 0);
    last[j] = vec_elem<T>(M.v[j], V - 1);
  }
#pragma unroll
  for (int j = 0; j < J; j++) {
    T up_last = __shfl_up_sync(FULL, last[j], 1);
    T dn_first = __shfl_down_sync(FULL, first[j], 1);
    T wrap_l = __shfl_sync(FULL, last[j > 0 ? j - 1 : 0], 31);
    T wrap_r = __shfl_sync(FULL, first[j < J - 1 ? j + 1 : 0], 0);
    T left = lane > 0 ? up_last : (j > 0 ? wrap_l : M.left);
    T right = lane < 31 ? dn_first : (j < J - 1 ? wrap_r : M.right);
    int v = vbase + lane + 32 * j;
    int nvalid = w - v * V;
    if (nvalid > 0) {
      if (nvalid > V) nvalid = V;
      T m[V], u[V], d[V], o[V];
#pragma unroll
      for (int k = 0; k < V; k++) {
        m[k] = vec_elem<T>(M.v[j], k);
        u[k] = vec_elem<T>(U.v[j], k);
        d[k] = vec_elem<T>(D.v[j], k);
      }
#pragma unroll
      for (int k = 0; k < V; k++) {
        T l = (k == 0) ? left : m[k - 1];
        T r = (k == V - 1) ? right : m[k + 1];
        o[k] = stencil(m[k], l, r, u[k], d[k]);
        if (RESID && k < nvalid) acc += resid2<T>(m[k], l, r, u[k], d[k]);
      }
      T* op = orow + (size_t)v * V;
      if (nvalid == V) {
        VT ov;
        if constexpr (V == 2) ov = make_double2((double)o[0], (double)o[1]);
        else ov = make_float4((float)o[0], (float)o[1], (float)o[2], (float)o[3]);
        *reinterpret_cast<VT*>(op) = ov;
      } else {
        #pragma unroll
        for (int k = 0; k < V; k++)  // static indices keep o[] in registers
          if (k < nvalid) op[k] = o[k];
      }
    }
  }
  return acc;
}

// Rows r0..r1-1 of the strip starting at vector vbase (one warp).
template <typename T, bool RESID, int J, int G>
__device__ double walk_item(const block_view<T>& in, const block_view<T>& out, int w, int nv,
    int vbase, int r0, int r1, int lane) {
  const bool has_right = vbase + 32 * J <= nv;
  walk_row<T, J> U, M, D[G];
  walk_load<T, J>(U, in, r0 - 1, vbase, nv, lane, has_right);
  walk_load<T, J>(M, in, r0, vbase, nv, lane, has_right);
  double acc = 0.0;
  for (int r = r0; r < r1; r += G) {
#pragma unroll
    for (int g = 0; g < G; g++) {
      if (r + 1 + g <= r1) walk_load<T, J>(D[g], in, r + 1 + g, vbase, nv, lane, has_right);
    }
#pragma unroll
    for (int g = 0; g < G; g++) {
      if (r + g < r1) {
        acc += walk_compute<T, RESID, J>(U, M, D[g], out.at(r + g, 1), vbase, w, lane);
        U = M;
        M = D[g];
      }
    }
  }
  return acc;
}

template <typename T> struct walk_shape;
template <> struct walk_shape<double> { static constexpr int J = 2, G = 4; };
template <> struct walk_shape<float> { static constexpr int J = 2, G = 4; };

// Not inlined: the walker gets the whole register budget, whatever the
// caller keeps live.
template <typename T, bool RESID>
__device__ __noinline__ double sweep_direct(block_view<T> in, block_view<T> out, int w, int h) {
  if (blockDim.x < 32) return sweep_simple<T, RESID>(in, out, w, h);
  constexpr int V = traits<T>::VEC, J = walk_shape<T>::J, G = walk_shape<T>::G;
  const int nv = (w + V - 1) / V;
  const int n_strips = (nv + 32 * J - 1) / (32 * J);
  const int nw = (int)(blockDim.x / 32), warp = (int)(threadIdx.x / 32), lane = (int)(threadIdx.x & 31);
  if (warp >= nw) return 0.0;  // threads of a partial warp (host emulation only)
  // Enough row runs that every warp gets an item; runs of at least 8 rows.
  int segs = (nw + n_strips - 1) / n_strips;
  if (segs > (h + 7) / 8) segs = (h + 7) / 8;
  if (segs < 1) segs = 1;
  const int items = n_strips * segs;
  double acc = 0.0;
  for (int it = warp; it < items; it += nw) {
    int s = it % n_strips, g = it / n_strips;
    int r0 = 1 + (int)((long long)h * g / segs), r1 = 1 + (int)((long long)h * (g + 1) / segs);
    acc += walk_item<T, RESID, J, G>(in, out, w, nv, s * 32 * J, r0, r1, lane);
  }
  return acc;
}

// ---------------------------------------------------------------------------
// Multi-sweep pass (temporal blocking): L sweeps (2 <= L <= LMAX) from a
// grid whose ghost zone is at least L deep, without writing the
// intermediate sweeps. A warp owns a strip of 32 vectors (one per lane) and
// streams level-0 rows down it; level l row r is computed when level l-1
// row r+1 arrives, so the pass is a wavefront L rows deep. Every level loses
// one valid column at each strip edge (the neighbour value is in another
// warp), so strips overlap by 2*ceil(L/VEC) vectors and each owns the
// 32 - 2*ceil(L/VEC) in the middle; row runs overlap by 2L rows. Cells on
// the domain boundary (row 0 / h+1, column 0 / w+1 of a chare without a
// neighbour there) keep their value at every level; cells beyond it are
// never used by a stored result. Each stored value is computed from the
// same five operands in the same order as a single sweep, so L passes of
// one sweep give the same bits.
// `fixed`: bit 0 top, 1 bottom, 2 left, 3 right side is the domain boundary.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void vec_to(const typename vec_of<T>::type& x, T (&a)[traits<T>::VEC]) {
#pragma unroll
  for (int k = 0; k < traits<T>::VEC; k++) a[k] = vec_elem<T>(x, k);
}
__device__ __forceinline__ double2 vec_from(const double (&a)[2]) { return make_double2(a[0], a[1]); }
__device__ __forceinline__ float4 vec_from(const float (&a)[4]) {
  return make_float4(a[0], a[1], a[2], a[3]);
}

// Per-lane constants of one strip item.
template <typename T>
struct deep_lane {
  bool own;                        // this lane stores its vector / counts the residual
  int v, col0;                     // vector index, its first column
  bool fixc[traits<T>::VEC];       // column on the domain boundary (kept at every level)
  bool inw[traits<T>::VEC];        // column inside the chare (1..w)
  bool anyfix;                     // some fixc[k]
  int fix_r0, fix_r1;              // rows kept at every level (0 / h+1), or INT_MIN
};

// The lane constants of the strip whose owned vectors are own0..own0+nown-1
// (the lane's vector starts E = ceil(L/VEC) vectors before them).
template <typename T, int L>
__device__ __forceinline__ deep_lane<T> make_lane(int w, int h, int fixed, int own0, int nown, int lane) {
  constexpr int V = traits<T>::VEC, E = (L + V - 1) / V;
  deep_lane<T> ln;
  ln.v = own0 - E + lane;
  ln.col0 = 1 + ln.v * V;
  ln.own = ln.v >= own0 && ln.v < own0 + nown;
  ln.anyfix = false;
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int c = ln.col0 + k;
    ln.fixc[k] = (c == 0 && (fixed & 4)) || (c == w + 1 && (fixed & 8));
    ln.inw[k] = c >= 1 && c <= w;
    ln.anyfix = ln.anyfix || ln.fixc[k];
  }
  ln.fix_r0 = (fixed & 1) ? 0 : INT_MIN;
  ln.fix_r1 = (fixed & 2) ? h + 1 : INT_MIN;
  return ln;
}

// What a lane keeps per level between two rows: the newest row of the level
// below (X) and the partial sums ((c + l) + r) + u around it (P), taken as
// soon as that row arrived. When the next row d arrives, the level's output
// is (P + d) * 0.2: the same adds in the same order as `stencil`, but one
// add and one multiply (not two shuffles and five operations) lie between
// the rows of two levels, so a step's chain through the L levels is 2L
// operations long, and two rows per level (three when the whole window is
// kept) fit in registers.
template <typename T, int L>
struct deep_state {
  T P[L][traits<T>::VEC], X[L][traits<T>::VEC];
  double D[traits<T>::VEC];  // level 1's partial sums in FP64 (residual of float grids)
};

__device__ __forceinline__ double resid_close(double p, double d) { return __dmul_rn(__dadd_rn(p, d), 0.2); }
// (P + x) * 0.2, rounded as `stencil` rounds it.
__device__ __forceinline__ void close_vec(double (&o)[2], const double (&P)[2], const double (&x)[2]) {
#pragma unroll
  for (int k = 0; k < 2; k++) o[k] = resid_close(P[k], x[k]);
}
__device__ __forceinline__ void close_vec(float (&o)[4], const float (&P)[4], const float (&x)[4]) {
  const f32x2 hi = pack2(STENCIL_C_HI, STENCIL_C_HI), lo = pack2(STENCIL_C_LO, STENCIL_C_LO);
#pragma unroll
  for (int k = 0; k < 4; k += 2) {
    const f32x2 s = add2(pack2(P[k], P[k + 1]), pack2(x[k], x[k + 1]));
    unpack2(fma2(s, hi, mul2(s, lo)), o[k], o[k + 1]);
  }
}
// P = ((x + l) + r) + X.
__device__ __forceinline__ void open_vec(double (&P)[2], const double (&x)[2], const double (&X)[2], double left,
    double right) {
  P[0] = __dadd_rn(__dadd_rn(__dadd_rn(x[0], left), x[1]), X[0]);
  P[1] = __dadd_rn(__dadd_rn(__dadd_rn(x[1], x[0]), right), X[1]);
}
__device__ __forceinline__ void open_vec(float (&P)[4], const float (&x)[4], const float (&X)[4], float left,
    float right) {
  float t[4];
#pragma unroll
  for (int k = 0; k < 4; k++)
    t[k] = __fadd_rn(__fadd_rn(x[k], k == 0 ? left : x[k - 1]), k == 3 ? right : x[k + 1]);
#pragma unroll
  for (int k = 0; k < 4; k += 2)
    unpack2(add2(pack2(t[k], t[k + 1]), pack2(X[k], X[k + 1])), P[k], P[k + 1]);
}

// One step of the wavefront through levels 1..LM: level-0 row q arrives in x,
// level l's row q - l is computed; x leaves as the row of level LM. FIX: the
// domain boundary is looked for (its cells keep their value at every level);
// without it the step must not meet one. There is no branch in a step: a
// branch in the row loop cost two register moves per value and level.
template <typename T, bool RESID, int L, int LM, bool FIX>
__device__ __forceinline__ void deep_step(deep_state<T, L>& S, T (&x)[traits<T>::VEC], int q,
    const deep_lane<T>& ln, int r0, int r1, double& acc) {
  constexpr int V = traits<T>::VEC;
  constexpr unsigned FULL = 0xffffffffu;
#pragma unroll
  for (int l = 1; l <= LM; l++) {
    const T left = __shfl_up_sync(FULL, x[V - 1], 1);
    const T right = __shfl_down_sync(FULL, x[0], 1);
    T o[V];
    close_vec(o, S.P[l - 1], x);
    if (RESID && l == 1) {
#pragma unroll
      for (int k = 0; k < V; k++) {
        const double c = (double)S.X[0][k];
        const double s = sizeof(T) == 8 ? (double)o[k] : resid_close(S.D[k], (double)x[k]);
        const double e = __dsub_rn(s, c);
        if (ln.own && ln.inw[k] && q - 1 >= r0 && q - 1 < r1) acc += __dmul_rn(e, e);
        if (sizeof(T) == 4) {
          const double lk = (double)(k == 0 ? left : x[k - 1]), rk = (double)(k == V - 1 ? right : x[k + 1]);
          S.D[k] = __dadd_rn(__dadd_rn(__dadd_rn((double)x[k], lk), rk), c);
        }
      }
    }
    if (FIX) {
      const bool row = q - l == ln.fix_r0 || q - l == ln.fix_r1;
#pragma unroll
      for (int k = 0; k < V; k++) o[k] = (row || ln.fixc[k]) ? S.X[l - 1][k] : o[k];
    }
    open_vec(S.P[l - 1], x, S.X[l - 1], left, right);
#pragma unroll
    for (int k = 0; k < V; k++) {
      S.X[l - 1][k] = x[k];
      x[k] = o[k];
    }
  }
}

// The level-0 rows of one lane, in order, through its private ring of P
// 16-byte slots in shared memory (cp.async, P-1 rows ahead; slots lie 32
// vectors apart), so no barrier is needed around it.
template <typename T, int P>
struct deep_stream {
  ring_addr ring;  // this lane's slot 0
  const T* next;   // this lane's vector of the next row to fetch
  int left;        // rows not yet fetched
  int pitch;
  unsigned at;     // byte offset of the next row's slot
  unsigned nb;     // 16, or 0 (zero fill) for a vector outside the pitched row
  __device__ __forceinline__ void fetch(unsigned slot) {
    ring_fetch(ring + slot, next, nb);
    cp_async_commit();
    left--;
    next += left > 0 ? pitch : 0;  // after the last row: that row again, never used
  }
  __device__ __forceinline__ void pop(T (&x)[traits<T>::VEC]) {
    cp_async_wait<P - 2>();
    ring_read(ring + at, x);
    fetch((at + (P - 1) * 512) & (P * 512 - 1));  // the slot of the row read before
    at = (at + 512) & (P * 512 - 1);
  }
};

// One strip item, in four loops: the first half of the fill (L steps, in
// which only the lower half of the levels has a row to work on), the second
// half, the steady steps, and the steps at the bottom domain boundary.
// Level l computes row q - l, so its first row is complete at step qs + 2l,
// and levels 1..L-1 meet the bottom boundary row R at steps R+1..R+L-1. The
// steady loop has no boundary tests (it takes no strip that holds a
// domain-boundary column); it takes 4 rows per turn, so that the rows a lane
// keeps need few register moves. sweep alone, 148 blocks of 2048 x 221, FP64, 6 levels:
// 272 us per pass (1480 GLUP/s), 327 with the whole window kept and a branch
// per level; FP32 155 us (199); 128 x 128 FP64 25.8 us (31.9). The FP64
// pipe is 53 % busy, the shuffles' wavefronts 62 %, the issue slots 69 %.
template <typename T, bool RESID, int L, int P>
__device__ __forceinline__ double deep_item(const block_view<T>& in, const block_view<T>& out, int w,
    const deep_lane<T>& ln, int r0, int r1, int lane, typename vec_of<T>::type* ring, bool lean) {
  constexpr int V = traits<T>::VEC, LH = (L + 1) / 2, U = 4;
  const long long e0 = (long long)traits<T>::OFF - 1 + ln.col0;  // element index in a row
  const bool can_load = e0 >= 0 && e0 + V <= in.pitch;
  const int qs = r0 - L, qe = r1 - 1 + L;  // level-0 rows streamed
  int q_lean_end = (ln.fix_r1 != INT_MIN && ln.fix_r1 + 1 <= qe) ? ln.fix_r1 + 1 : qe + 1;
  if (!lean || __any_sync(0xffffffffu, ln.anyfix)) q_lean_end = INT_MIN;
  deep_stream<T, P> st{to_ring(ring + lane), in.row(qs) + (can_load ? e0 : 0), qe - qs + 1, in.pitch, 0,
                       can_load ? 16u : 0u};
#pragma unroll
  for (int k = 0; k < P - 1; k++) st.fetch(k * 512);
  deep_state<T, L> S;
#pragma unroll
  for (int l = 0; l < L; l++)
#pragma unroll
    for (int k = 0; k < V; k++) S.P[l][k] = S.X[l][k] = (T)0;
#pragma unroll
  for (int k = 0; k < V; k++) S.D[k] = 0.0;
  double acc = 0.0;
  T x[V];
  T* op = out.row(r0) + e0;
  const int nput = ln.own ? w - ln.v * V : 0;
  int q = qs;
#pragma unroll 1
  for (; q < qs + 2 * LH; q++) {
    st.pop(x);
    deep_step<T, RESID, L, LH, true>(S, x, q, ln, r0, r1, acc);
  }
#pragma unroll 1
  for (; q < qs + 2 * L; q++) {
    st.pop(x);
    deep_step<T, RESID, L, L, true>(S, x, q, ln, r0, r1, acc);
  }
#pragma unroll 1
  for (; q + U - 1 < q_lean_end; q += U) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      st.pop(x);
      deep_step<T, RESID, L, L, false>(S, x, q + u, ln, r0, r1, acc);
      put_vec(op, x, nput);
      op += out.pitch;
    }
  }
#pragma unroll 1
  for (; q <= qe; q++) {
    st.pop(x);
    deep_step<T, RESID, L, L, true>(S, x, q, ln, r0, r1, acc);
    put_vec(op, x, nput);
    op += out.pitch;
  }
  cp_async_wait<0>();
  return acc;
}

// The same pass, computed by thread 0 alone for blocks under one warp, with
// levels 1..L-1 kept as three-row rings in the block's scratch.
template <typename T, bool RESID>
__device__ __noinline__ double sweep_deep_simple(block_view<T> in, block_view<T> out, int w, int h, int L,
    int fixed) {
  if (threadIdx.x != 0) return 0.0;
  size_t cap = 0;
  T* ring = reinterpret_cast<T*>(charm::smem_scratch(&cap));
  const int W = w + 2 * L;  // columns 1-L .. w+L
  if ((size_t)(L - 1) * 3 * W * sizeof(T) > cap) {
    charm::detail::report_error(CHARMING_ERR_CONFIG, w, L);
    return 0.0;
  }
  auto slot = [&](int l, int r) -> T* { return ring + ((size_t)(l - 1) * 3 + ((r % 3) + 3) % 3) * W; };
  auto lv = [&](int l, int r, int c) -> T { return l == 0 ? *in.at(r, c) : slot(l, r)[c + L - 1]; };
  double acc = 0.0;
  for (int q = 1 - L; q <= h + L; q++) {
    for (int l = 1; l <= L; l++) {
      const int r = q - l, ext = L - l;
      if (r < 1 - ext || r > h + ext) continue;
      const bool fixr = (r == 0 && (fixed & 1)) || (r == h + 1 && (fixed & 2));
      for (int c = 1 - ext; c <= w + ext; c++) {
        const bool fixc = (c == 0 && (fixed & 4)) || (c == w + 1 && (fixed & 8));
        T m = lv(l - 1, r, c), v = m;
        if (!fixr && !fixc) {
          T lc = lv(l - 1, r, c - 1), rc = lv(l - 1, r, c + 1);
          T up = lv(l - 1, r - 1, c), dn = lv(l - 1, r + 1, c);
          v = stencil(m, lc, rc, up, dn);
          if (RESID && l == 1 && r >= 1 && r <= h && c >= 1 && c <= w)
            acc += resid2<T>(m, lc, rc, up, dn);
        }
        if (l == L) {
          if (r >= 1 && r <= h && c >= 1 && c <= w) *out.at(r, c) = v;
        } else {
          slot(l, r)[c + L - 1] = v;
        }
      }
    }
  }
  return acc;
}

// The items of one pass of L sweeps (one warp); one register allocation per L.
template <typename T, bool RESID, int L>
__device__ __noinline__ double sweep_deep_items(block_view<T> in, block_view<T> out, int w, int h,
    int fixed, typename vec_of<T>::type* ring, int nw, int warp, int lane, bool lean) {
  constexpr int V = traits<T>::VEC, P = 8;
  constexpr int E = (L + V - 1) / V;    // vectors lost at each strip edge over L levels
  constexpr int SS = 32 - 2 * E;        // vectors a strip owns
  const int nv = (w + V - 1) / V;
  const int n_strips = (nv + SS - 1) / SS;
  // Row runs. More runs fill the warps but each streams 2L rows more than it
  // stores. Cost of a split: its rows times the items that share an SM
  // sub-partition's pipes (warps go to the four in turn) plus the items in
  // sequence on the busiest warp (a step's latency is about one more item's
  // worth of issue). Over the splits measured for 64^2 to 2048 x 221 blocks
  // in both types (1 to 12 runs, 16 warps) its choice is within 1 % of the
  // best one on average and 5 % at most; counting rounds of busy warps alone
  // lost 5 % and up to 31 %. One lane per split: a loop over them in every
  // thread took 2 us of a 256^2 block's 58.
  unsigned long long key = ~0ULL;
  {
    const int sg = lane + 1;
    if (sg <= 16 && (sg == 1 || h / sg >= 2 * L)) {
      const int n = n_strips * sg, full = n / nw, rem = n - full * nw;
      const int shared = full * ((nw + 3) / 4) + (rem + 3) / 4, chain = full + (rem > 0 ? 1 : 0);
      key = ((unsigned long long)(unsigned)(shared + chain) * (unsigned)((h + sg - 1) / sg + 2 * L)) << 8 | (unsigned)sg;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long k = __shfl_xor_sync(0xffffffffu, key, o);
      key = k < key ? k : key;
    }
  }
  const int segs = (int)(key & 255);
  const int items = n_strips * segs;
  double acc = 0.0;
  for (int it = warp; it < items; it += nw) {
    int s = it % n_strips, g = it / n_strips;
    int r0 = 1 + (int)((long long)h * g / segs), r1 = 1 + (int)((long long)h * (g + 1) / segs);
    int own0 = s * SS;
    int nown = min(SS, nv - own0);
    const deep_lane<T> ln = make_lane<T, L>(w, h, fixed, own0, nown, lane);
    acc += deep_item<T, RESID, L, P>(in, out, w, ln, r0, r1, lane, ring, lean);
  }
  return acc;
}

// lean: steps that need no boundary or fill tests leave them out (false:
// every step tests); same results bit for bit.
template <typename T, bool RESID>
__device__ __forceinline__ double sweep_deep(block_view<T> in, block_view<T> out, int w, int h, int L,
    int fixed, bool lean = true) {
  if (blockDim.x < 32) return sweep_deep_simple<T, RESID>(in, out, w, h, L, fixed);
  using VT = typename vec_of<T>::type;
  const int P = 8;
  const int nw = (int)(blockDim.x / 32), warp = (int)(threadIdx.x / 32), lane = (int)(threadIdx.x & 31);
  if (warp >= nw) return 0.0;
  size_t sbytes = 0;
  VT* rings = reinterpret_cast<VT*>(charm::smem_scratch(&sbytes));
  if ((size_t)nw * P * 32 * sizeof(VT) > sbytes) {
    if (threadIdx.x == 0) charm::detail::report_error(CHARMING_ERR_CONFIG, (int)sbytes, nw);
    return 0.0;
  }
  VT* ring = rings + (size_t)warp * P * 32;
#define CHARMING_DEEP_CASE(LL)                                                                 \
  if (L == LL) return sweep_deep_items<T, RESID, LL>(in, out, w, h, fixed, ring, nw, warp, lane, lean);
  CHARMING_DEEP_CASE(2)
  CHARMING_DEEP_CASE(3)
  CHARMING_DEEP_CASE(5)
  CHARMING_DEEP_CASE(6)
  CHARMING_DEEP_CASE(7)
  CHARMING_DEEP_CASE(8)
#undef CHARMING_DEEP_CASE
  return sweep_deep_items<T, RESID, 4>(in, out, w, h, fixed, ring, nw, warp, lane, lean);
}

// ---------------------------------------------------------------------------
// TMA row pipeline.
// ---------------------------------------------------------------------------

constexpr int MAX_SLOTS = 64;        // mbarrier pairs in the first 1 KiB
constexpr int BAR_BYTES = 2 * MAX_SLOTS * 8;

// Column tiling and ring size of one sweep. Each warp owns a strip of
// 32 * VEC columns of the tile and walks all rows of it.
struct tma_plan {
  int ntiles;     // column tiles
  int tws;        // tile stride (columns), multiple of VEC
  int NS;         // ring slots (rows in flight)
  int slot_elems; // elements per slot
};

template <typename T>
__host__ __device__ inline size_t tma_slot_bytes(int tws) {
  size_t e = (size_t)tws + 2 * traits<T>::VEC;
  return (e * sizeof(T) + 127) / 128 * 128;
}

template <typename T>
__device__ bool make_plan(int w, int nthreads, size_t smem_bytes, int tile_w_opt, tma_plan* p) {
  constexpr int V = traits<T>::VEC;
  int twmax = (nthreads / 32) * 32 * V;  // one vector per lane
  if (tile_w_opt > 0 && tile_w_opt < twmax) twmax = tile_w_opt;
  twmax = (twmax + V - 1) / V * V;
  p->ntiles = (w + twmax - 1) / twmax;
  int tw = (w + p->ntiles - 1) / p->ntiles;
  p->tws = (tw + V - 1) / V * V;
  size_t sb = tma_slot_bytes<T>(p->tws);
  p->slot_elems = (int)(sb / sizeof(T));
  size_t avail = smem_bytes > (size_t)BAR_BYTES ? smem_bytes - BAR_BYTES : 0;
  long ns = (long)(avail / sb);
  if (ns > MAX_SLOTS) ns = MAX_SLOTS;
  p->NS = (int)ns;
  return p->NS >= 4;
}

// One sweep in -> out. Row segments (tile columns + 16-byte halo each side)
// stream through NS shared-memory slots. full[s] completes when the bulk
// copy into slot s landed; empty[s] when every warp is done with it. Lane 0
// of warp 0 issues copies whenever a slot is empty (it also polls while
// waiting, so it never blocks the pipeline it feeds). Returns false (error
// recorded) if a wait ran out.
template <typename T, bool RESID>
__device__ bool sweep_tma(block_view<T> in, block_view<T> out, int w, int h, void* smem,
    size_t smem_bytes, const tma_plan& P, double* acc_out) {
  constexpr int V = traits<T>::VEC;
  constexpr int H = V;  // halo elements each side of a slot row (16 bytes)
  constexpr unsigned FULL = 0xffffffffu;
  unsigned long long* full = reinterpret_cast<unsigned long long*>(smem);
  unsigned long long* empty = full + MAX_SLOTS;
  T* slots = reinterpret_cast<T*>(reinterpret_cast<char*>(smem) + BAR_BYTES);
  const int rows = h + 2;
  const long long total = (long long)P.ntiles * rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = blockDim.x >> 5;
  __shared__ int s_fail;
  __shared__ long long s_issued;

  fence_proxy_async_global();  // earlier generic writes to `in` -> bulk copies
  if (threadIdx.x == 0) {
    for (int s = 0; s < P.NS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], (unsigned)nw);
    }
    fence_mbar_init();
    s_fail = 0;
  }
  __syncthreads();

  // producer state (lane 0 of warp 0): rows issued, and the next one's slot,
  // round of the ring, tile and row, found by counting (the divisions by the
  // slot count and the rows were most of a row's instructions)
  long long issued = 0;
  int is = 0, iu = 0, it = 0, ir = 0;
  auto try_issue = [&]() {
    while (issued < total) {
      const long long j = issued;
      const int s = is, r = ir;
      if (iu > 0 && !mbar_test_wait(&empty[s], (unsigned)((iu - 1) & 1))) break;
      int c0 = it * P.tws;
      int tw = min(P.tws, w - c0);
      unsigned bytes = (unsigned)(((size_t)(tw + 2 * H) * sizeof(T) + 15) / 16 * 16);
      // checked build: 16-byte aligned source, copy fits its slot
      if (!CHARM_VERIFY(((reinterpret_cast<uintptr_t>(in.row(r) + traits<T>::OFF + c0 - H) & 15) == 0) &&
                        bytes <= (unsigned)(P.slot_elems * sizeof(T)),
                        CHARMING_ERR_PIPELINE, (int)j, (int)bytes))
        break;
      mbar_expect_tx(&full[s], bytes);
      bulk_g2s(slots + (size_t)s * P.slot_elems, in.row(r) + traits<T>::OFF + c0 - H, bytes,
               &full[s]);
      issued = j + 1;
      if (++is == P.NS) {
        is = 0;
        iu++;
      }
      if (++ir == rows) {
        ir = 0;
        it++;
      }
    }
  };
  const bool producer = (warp == 0 && lane == 0);
  if (producer) {
    fence_proxy_async_smem();
    try_issue();
  }
  __syncwarp();

  double acc = 0.0;
  bool fail = false;
  int sc = 0, s1 = 0, s2 = 0;  // slots of the current row and of the two before it
  unsigned parity = 0;
  for (int t = 0; t < P.ntiles && !fail; t++) {
    const int c0 = t * P.tws;
    const int tw = min(P.tws, w - c0);
    const int v = warp * 32 + lane;      // vector of the tile row this lane owns
    const bool active = v * V < tw;
    const bool next_active = (v + 1) * V < tw;
    const int nvalid = active ? min(V, tw - v * V) : 0;
    const int s_off = H + v * V;         // slot element of interior column c0 + v*V
    for (int r = 0; r < rows; r++) {
      unsigned long long* fb = &full[sc];
      unsigned spins = 0;
      while (true) {
        // The producer's warp must not be suspended inside try_wait while
        // copies wait to be issued: it polls with the non-blocking test.
        bool ok = (warp == 0) ? mbar_test_wait(fb, parity) : mbar_try_wait(fb, parity);
        if (__all_sync(FULL, ok)) break;
        if (producer) try_issue();
        __syncwarp();
        if (++spins > (1u << 22) || *reinterpret_cast<volatile int*>(&s_fail)) {
          fail = true;
          break;
        }
      }
      if (fail) break;
      if (r >= 2) {
        const T* up = slots + s2 * P.slot_elems;
        const T* mid = slots + s1 * P.slot_elems;
        const T* dn = slots + sc * P.slot_elems;
        T m[V];
        if (active) {
          if (V == 2) {
            double2 b = *reinterpret_cast<const double2*>(mid + s_off);
            m[0] = (T)b.x;
            m[1] = (T)b.y;
          } else {
            float4 b = *reinterpret_cast<const float4*>(mid + s_off);
            m[0] = (T)b.x; m[1] = (T)b.y; m[2] = (T)b.z; m[3] = (T)b.w;
          }
        } else {
#pragma unroll
          for (int k = 0; k < V; k++) m[k] = (T)0;
        }
        T left = __shfl_up_sync(FULL, m[V - 1], 1);
        T right = __shfl_down_sync(FULL, m[0], 1);
        if (active) {
          if (lane == 0) left = mid[s_off - 1];
          if (lane == 31 || !next_active) right = mid[s_off + V];
          acc += compute_vec<T, RESID>(up + s_off, mid + s_off, dn + s_off, left, right,
                                       out.at(r - 1, 1 + c0 + v * V), nvalid);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s2]);
        if (producer) try_issue();
      }
      s2 = s1;
      s1 = sc;
      if (++sc == P.NS) {
        sc = 0;
        parity ^= 1;
      }
    }
    if (!fail) {
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&empty[s2]);  // rows h and h + 1
        mbar_arrive(&empty[s1]);
      }
    }
  }
  if (fail) atomicExch(&s_fail, 1);
  if (producer) s_issued = issued;
  __syncthreads();
  fail = s_fail != 0;
  if (threadIdx.x == 0) {
    if (fail) {
      // Let copies still in flight land before the slots are reused.
      for (long long j = (s_issued > P.NS ? s_issued - P.NS : 0); j < s_issued; j++) {
        unsigned spins = 0;
        while (!mbar_try_wait(&full[j % P.NS], (unsigned)((j / P.NS) & 1)) && ++spins < (1u << 20)) {
        }
      }
      charm::detail::report_error(CHARMING_ERR_PIPELINE, (int)s_issued, h);
    }
    for (int s = 0; s < P.NS; s++) {
      mbar_inval(&full[s]);
      mbar_inval(&empty[s]);
    }
  }
  fence_proxy_async_global();  // outputs (generic stores) -> next sweep's copies
  __syncthreads();
  *acc_out = acc;
  return !fail;
}

}  // namespace jac

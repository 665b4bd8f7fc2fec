// euler_kernels.cu -- the Euler sibling on sm_100a: one fused kernel per
// dimensionally split 2D step (both sweeps of the reference's
// MUSCL-Hancock + HLLC / HLL step, src/euler/riemann2d_cpu.cpp:295-309, in
// one pass over HBM), its initial max-speed reduction, and a one-CTA kernel
// that runs a whole 1D Riemann problem (src/euler/riemann1d_cpu.cpp:95-196).
//
// 2D step kernels.  Indices are clamped at the walls (the reference's transmissive
// ghost copies, riemann2d_cpu.cpp:160-182); the sweep order alternates with the
// step count (even: x then y); the next step's max signal speeds come from the
// epilogue, so the time step never needs a separate pass.  Small binary64 grids
// and most of the parity build's (see step2d): a CTA of 512 threads owns a 32 x TY
// tile, loads the 36 x (TY + 4) region around it,
// runs the first sweep on the part of it the second needs, then the second on the
// tile, each as reconstruction + Hancock of every cell's two faces, one flux per
// interface and the update, staged in shared memory.  Otherwise: the streaming
// kernel below.
//
// Compiled twice (see Makefile): PMHD_EKNS=exact with -fmad=false (bit
// parity with the reference CPU build) and PMHD_EKNS=fast (contraction,
// approximate binary32 division / square root).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>

#include "euler/euler_api.h"
#include "pmhd/euler.hpp"

#ifndef PMHD_EKNS
#error "PMHD_EKNS must name the build flavour (exact or fast)"
#endif

namespace pmhd {
namespace euler {
namespace PMHD_EKNS {

namespace {

// Point arithmetic of the build: the reference's expressions (exact build,
// bit parity) or the performance forms (fast build, PMHD_EULER_FAST).
#if PMHD_EULER_FAST
namespace pf = ::pmhd::euler::fastform;
template <class T>
__device__ __forceinline__ void k_c2p(const T U[4], T W[4]) {
  pf::cons_to_prim(U, W);
}
template <class T, int NI, int TI>
__device__ __forceinline__ void k_hancock_pair(const T l[4], const T r[4], T lh[4], T rh[4], T fac) {
  pf::hancock_pair<T, NI, TI>(l, r, lh, rh, fac);
}
template <class T, int NI, int TI, bool HLL>
__device__ __forceinline__ void k_flux(const T a[4], const T b[4], T f[4]) {
  if (HLL)
    pf::hll_flux<T, NI, TI>(a, b, f);
  else
    pf::hllc_flux<T, NI, TI>(a, b, f);
}
template <class T>
__device__ __forceinline__ void k_speeds(const T U[4], T& sx, T& sy) {
  pf::cell_speeds(U, sx, sy);
}
#else
template <class T>
__device__ __forceinline__ void k_c2p(const T U[4], T W[4]) {
  cons_to_prim(U, W);
}
template <class T, int NI, int TI>
__device__ __forceinline__ void k_hancock_pair(const T l[4], const T r[4], T lh[4], T rh[4], T fac) {
  hancock<T, NI, TI>(l, l, r, lh, fac);
  hancock<T, NI, TI>(r, l, r, rh, fac);
}
template <class T, int NI, int TI, bool HLL>
__device__ __forceinline__ void k_flux(const T a[4], const T b[4], T f[4]) {
  if (HLL)
    hll_flux<T, NI, TI>(a, b, f);
  else
    hllc_flux<T, NI, TI>(a, b, f);
}
// riemann2d_cpu.cpp:200-210: |u| + c, |v| + c from the primitives.
template <class T>
__device__ __forceinline__ void k_speeds(const T U[4], T& sx, T& sy) {
  T W[4];
  cons_to_prim(U, W);
  const T cs = sound_speed(W[3], W[0]);
  sx = std::fabs(W[1]) + cs;
  sy = std::fabs(W[2]) + cs;
}
#endif

constexpr int NV = 4;

constexpr int TW = 32;  // tile width (cells)
constexpr int RW = TW + 4;

__device__ __forceinline__ unsigned long long speed_bits(double v) {
  return v > 0.0 ? (unsigned long long)__double_as_longlong(v) : 0ull;
}
__device__ __forceinline__ double bits_speed(unsigned long long b) { return __longlong_as_double((long long)b); }

__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}

template <class T, int TY>
struct Tile {
  static constexpr int RH = TY + 4;
  static constexpr int N = RH * RW;  // cells of the region
  T U[NV][N];
  T W[NV][N];   // primitives
  T HL[NV][N];  // Hancock-evolved left (lower) face of each cell; then the interface fluxes
  T HR[NV][N];  // ... right (upper) face
};

// Where the last sweep's updated cells go: the output state (interior cells
// only) and the running maxima of the next step's signal speeds.
template <class T>
struct TileOut {
  T* __restrict__ u;
  long long plane;
  int pitch, i0, j0, nx, ny;
  unsigned long long bx, by;
};

// One sweep over the region cells [r0, r1) x [c0, c1) that are updated;
// DIR 0 = x (along c), 1 = y (along r).  Needs W valid on the cells within
// 2 of them along DIR.  The update phase also does what follows it: the
// first sweep (LAST = false) forms the primitives of each updated cell for
// the second sweep's reconstruction; the last one stores the tile and
// reduces the signal speeds.  (Region rows or columns beyond a wall hold
// copies of the edge cells, and a sweep along them gives the edge cell's
// result bit for bit, so their primitives are the refreshed ghost copies of
// the reference's applyBC between the sweeps.)
template <class T, int TY, int DIR, bool HLL, bool LAST>
__device__ __forceinline__ void sweep(Tile<T, TY>& s, int r0, int r1, int c0, int c1, T fac, T ratio,
                                      TileOut<T>& out) {
  constexpr int NI = DIR == 0 ? 1 : 2, TI = DIR == 0 ? 2 : 1;
  const int step = DIR == 0 ? 1 : RW;
  // Hancock faces of the cells one beyond the updated ones along DIR.
  const int hr0 = DIR == 1 ? r0 - 1 : r0, hr1 = DIR == 1 ? r1 + 1 : r1;
  const int hc0 = DIR == 0 ? c0 - 1 : c0, hc1 = DIR == 0 ? c1 + 1 : c1;
  const int hw = hc1 - hc0, hn = (hr1 - hr0) * hw;
  for (int q = threadIdx.x; q < hn; q += blockDim.x) {
    const int id = (hr0 + q / hw) * RW + hc0 + q % hw;
    T l[NV], r[NV], lh[NV], rh[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) muscl_recon(s.W[k][id - step], s.W[k][id], s.W[k][id + step], l[k], r[k]);
    k_hancock_pair<T, NI, TI>(l, r, lh, rh, fac);
#pragma unroll
    for (int k = 0; k < NV; k++) {
      s.HL[k][id] = lh[k];
      s.HR[k][id] = rh[k];
    }
  }
  __syncthreads();
  // Interface fluxes: F at cell id = flux between id - step and id, for the
  // updated cells and the one past them; stored over HL[id], which only this
  // thread reads.
  const int fr1 = DIR == 1 ? r1 + 1 : r1, fc1 = DIR == 0 ? c1 + 1 : c1;
  const int fw = fc1 - c0, fn = (fr1 - r0) * fw;
  for (int q = threadIdx.x; q < fn; q += blockDim.x) {
    const int id = (r0 + q / fw) * RW + c0 + q % fw;
    T a[NV], b[NV], f[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
      a[k] = s.HR[k][id - step];
      b[k] = s.HL[k][id];
    }
    k_flux<T, NI, TI, HLL>(a, b, f);
#pragma unroll
    for (int k = 0; k < NV; k++) s.HL[k][id] = f[k];
  }
  __syncthreads();
  const int uw = c1 - c0, un = (r1 - r0) * uw;
  for (int q = threadIdx.x; q < un; q += blockDim.x) {
    const int r = r0 + q / uw, c = c0 + q % uw, id = r * RW + c;
    T U4[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) U4[k] = s.U[k][id] - ratio * (s.HL[k][id + step] - s.HL[k][id]);
    if (!LAST) {
      T W4[NV];
      k_c2p(U4, W4);
#pragma unroll
      for (int k = 0; k < NV; k++) {
        s.U[k][id] = U4[k];
        s.W[k][id] = W4[k];
      }
    } else {
      const int i = out.i0 + c - 2, j = out.j0 + r - 2;
      if (i < out.nx && j < out.ny) {
#pragma unroll
        for (int k = 0; k < NV; k++) out.u[k * out.plane + (long long)j * out.pitch + i] = U4[k];
        T vx, vy;
        k_speeds(U4, vx, vy);
        const unsigned long long sx = speed_bits((double)vx), sy = speed_bits((double)vy);
        out.bx = sx > out.bx ? sx : out.bx;
        out.by = sy > out.by ? sy : out.by;
      }
    }
  }
  if (!LAST) __syncthreads();
}

// The step's control values: every CTA reads the same slots; one thread
// (advance) writes the other parity and the speed slot two steps ahead.
template <class T>
struct StepControl {
  T t, dt;
  long long n;
  bool active;
  __device__ __forceinline__ StepControl(const EulerCtrl* ctrl, int p, T dx, T dy, T cfl) {
    t = (T)ctrl->t[p];
    n = ctrl->step[p];
    // t and t + dt are values of type T, so their tests against t_end are
    // exact in binary64 whichever type t_end has.
    active = !ctrl->stop && (double)t < ctrl->t_end && n < ctrl->step_limit;
    dt = (T)0;
    if (active) {
      const T mx = (T)bits_speed(ctrl->sx[n % 3]), my = (T)bits_speed(ctrl->sy[n % 3]);
      const T m = vmin(dx / mx, dy / my);
      dt = ctrl->wide_time ? (T)(ctrl->cfl * (double)m) : cfl * m;
      if ((double)(T)(t + dt) > ctrl->t_end) dt = ctrl->wide_time ? (T)(ctrl->t_end - (double)t) : (T)ctrl->t_end - t;
      if (!(dt > (T)0.0) || t + dt == t) active = false;  // riemann2d_cpu.cpp:298, euler2d_cpu.cpp:309
    }
  }
  __device__ __forceinline__ void advance(EulerCtrl* ctrl, int p) const {
    if (active) {
      ctrl->t[p ^ 1] = (double)(t + dt);
      ctrl->step[p ^ 1] = n + 1;
      ctrl->sx[(n + 2) % 3] = 0ull;
      ctrl->sy[(n + 2) % 3] = 0ull;
    } else {
      ctrl->t[p ^ 1] = ctrl->t[p];
      ctrl->step[p ^ 1] = n;
      if ((double)t < ctrl->t_end && n < ctrl->step_limit) ctrl->stop = 1;
    }
  }
};

// Registers: 64 per thread for two resident CTAs of 512.
template <class T, int TY, int NT, int MINB, bool HLL>
__global__ void __launch_bounds__(NT, MINB) step_kernel(const T* __restrict__ uin, T* __restrict__ uout, int nx, int ny,
                                                   int pitch, long long plane, T dx, T dy, T cfl, EulerCtrl* ctrl,
                                                   int p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Tile<T, TY>& s = *reinterpret_cast<Tile<T, TY>*>(smem_raw);
  constexpr int RH = TY + 4;
  const int i0 = blockIdx.x * TW, j0 = blockIdx.y * TY;
  const StepControl<T> sc(ctrl, p, dx, dy, cfl);
  const T dt = sc.dt;
  const long long n = sc.n;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) sc.advance(ctrl, p);
  if (!sc.active) {
    // Carry the state to the output buffer.
    for (int q = threadIdx.x; q < TW * TY; q += blockDim.x) {
      const int i = i0 + q % TW, j = j0 + q / TW;
      if (i < nx && j < ny)
#pragma unroll
        for (int k = 0; k < NV; k++) uout[k * plane + (long long)j * pitch + i] = uin[k * plane + (long long)j * pitch + i];
    }
    return;
  }
  // Region load with wall clamping, and the primitives of every region cell
  // (same thread, so no barrier between them).  (Measured: asynchronous
  // global -> shared copies of the region, issued ahead of the step-control
  // reads, were 11 % slower in binary64 and no faster in binary32.)
  for (int q = threadIdx.x; q < RH * RW; q += blockDim.x) {
    const int r = q / RW, c = q % RW;
    int j = j0 - 2 + r, i = i0 - 2 + c;
    j = j < 0 ? 0 : (j >= ny ? ny - 1 : j);
    i = i < 0 ? 0 : (i >= nx ? nx - 1 : i);
    T U4[NV], W4[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
      U4[k] = uin[k * plane + (long long)j * pitch + i];
      s.U[k][q] = U4[k];
    }
    k_c2p(U4, W4);
#pragma unroll
    for (int k = 0; k < NV; k++) s.W[k][q] = W4[k];
  }
  __syncthreads();
  const T facx = (T)0.5 * dt / dx, facy = (T)0.5 * dt / dy, rx = dt / dx, ry = dt / dy;
  TileOut<T> out{uout, plane, pitch, i0, j0, nx, ny, 0ull, 0ull};
  if (n % 2 == 0) {
    // x sweep on every region row (columns 2..TW+1), then y sweep on the tile.
    sweep<T, TY, 0, HLL, false>(s, 0, RH, 2, TW + 2, facx, rx, out);
    sweep<T, TY, 1, HLL, true>(s, 2, TY + 2, 2, TW + 2, facy, ry, out);
  } else {
    sweep<T, TY, 1, HLL, false>(s, 2, TY + 2, 0, RW, facy, ry, out);
    sweep<T, TY, 0, HLL, true>(s, 2, TY + 2, 2, TW + 2, facx, rx, out);
  }
  unsigned long long bx = out.bx, by = out.by;
  bx = warp_max(bx);
  by = warp_max(by);
  if ((threadIdx.x & 31) == 0) {
    if (bx) atomicMax(&ctrl->sx[(n + 1) % 3], bx);
    if (by) atomicMax(&ctrl->sy[(n + 1) % 3], by);
  }
}

// ---- streaming step kernel -----------------------------------------------------------
//
// A warp (a CTA of its own) owns a strip of 28 columns -- its 32 lanes are the
// strip and two halo columns on each side -- and marches down a block of rows.
// The sweep along x takes its neighbours by warp shuffles, the sweep along y
// keeps a window of rows in registers, in either order, so there is no shared
// memory and no barrier; per output cell 32 / 28 (x) and (rows + 4) / rows of the
// work is halo.  The next row's loads are issued a row ahead.  Bound by issue and
// by each warp's dependent chain (a row takes 1.03 us at one warp per scheduler
// in binary64, 0.57 in binary32).  Registers: 128 / 64 a thread, 16 / 32 warps per
// SM; one-warp CTAs keep the tile position in uniform registers (four warps a CTA
// with a position per warp: 124 bytes of spills, 10 % slower).  At 4096^2 fp64
// 28.4 and fp32 56.0 G zone-cycles/s, against 12.5 / 26.0 with 32 x 16 / 32 x 32
// shared-memory tiles; at 1024^2 48 / 25 us a step against 99 / 50.
constexpr int kStripW = 28;

template <class T>
struct Cell {
  T v[NV];
};
template <class T>
__device__ __forceinline__ Cell<T> shfl_up1(const Cell<T>& c) {
  Cell<T> r;
#pragma unroll
  for (int k = 0; k < NV; k++) r.v[k] = __shfl_up_sync(0xffffffffu, c.v[k], 1);
  return r;
}
template <class T>
__device__ __forceinline__ Cell<T> shfl_down1(const Cell<T>& c) {
  Cell<T> r;
#pragma unroll
  for (int k = 0; k < NV; k++) r.v[k] = __shfl_down_sync(0xffffffffu, c.v[k], 1);
  return r;
}

// Hancock-evolved lower and upper faces of a cell from its neighbours' and its
// own primitives along direction NI.
template <class T, int NI, int TI>
__device__ __forceinline__ void evolved_faces(const Cell<T>& wm, const Cell<T>& w0, const Cell<T>& wp, T fac,
                                              Cell<T>& lo, Cell<T>& hi) {
  T l[NV], r[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) muscl_recon(wm.v[k], w0.v[k], wp.v[k], l[k], r[k]);
  k_hancock_pair<T, NI, TI>(l, r, lo.v, hi.v, fac);
}

// The x sweep of one row: u is the lane's cell, neighbouring lanes hold its
// neighbours; valid on lanes 2 .. 29.
template <class T, bool HLL>
__device__ __forceinline__ Cell<T> sweep_row_x(const Cell<T>& u, T fac, T ratio) {
  Cell<T> w, lo, hi, f, r;
  k_c2p(u.v, w.v);
  evolved_faces<T, 1, 2>(shfl_up1(w), w, shfl_down1(w), fac, lo, hi);
  k_flux<T, 1, 2, HLL>(shfl_up1(hi).v, lo.v, f.v);
  const Cell<T> fr = shfl_down1(f);
#pragma unroll
  for (int k = 0; k < NV; k++) r.v[k] = u.v[k] - ratio * (fr.v[k] - f.v[k]);
  return r;
}

// The y sweep as a pipeline over rows: push(row r) returns the updated row
// r - 2 (valid from the fifth push on).
template <class T, bool HLL>
struct ColumnSweep {
  Cell<T> w2, w1, u2, u1, hi2, f2;  // rows r - 2 and r - 1; upper face of row r - 2, flux below it
  T fac, ratio;
  __device__ __forceinline__ ColumnSweep(T fac_, T ratio_) : w2{}, w1{}, u2{}, u1{}, hi2{}, f2{}, fac(fac_), ratio(ratio_) {}
  __device__ __forceinline__ Cell<T> push(const Cell<T>& u) {
    Cell<T> w, lo, hi, f, r;
    k_c2p(u.v, w.v);
    evolved_faces<T, 2, 1>(w2, w1, w, fac, lo, hi);  // faces of row r - 1
    k_flux<T, 2, 1, HLL>(hi2.v, lo.v, f.v);          // between rows r - 2 and r - 1
#pragma unroll
    for (int k = 0; k < NV; k++) r.v[k] = u2.v[k] - ratio * (f.v[k] - f2.v[k]);
    w2 = w1, w1 = w, u2 = u1, u1 = u, hi2 = hi, f2 = f;
    return r;
  }
};

template <class T, bool HLL, int MINB>
__global__ void __launch_bounds__(32, MINB) stream_kernel(const T* __restrict__ uin, T* __restrict__ uout, int nx,
                                                           int ny, int pitch, long long plane, T dx, T dy, T cfl,
                                                           int rows, EulerCtrl* ctrl, int p) {
  const StepControl<T> sc(ctrl, p, dx, dy, cfl);
  const int lane = threadIdx.x, strips = (nx + kStripW - 1) / kStripW;
  if (blockIdx.x == 0 && lane == 0) sc.advance(ctrl, p);
  const int strip = (int)(blockIdx.x % (unsigned)strips);
  const int i = strip * kStripW - 2 + lane, j0 = (int)(blockIdx.x / (unsigned)strips) * rows;
  const int j1 = j0 + rows < ny ? j0 + rows : ny;
  const bool owns = lane >= 2 && lane < 2 + kStripW && i < nx;
  if (!sc.active) {  // carry the state to the output buffer
    if (owns)
      for (int j = j0; j < j1; j++)
#pragma unroll
        for (int k = 0; k < NV; k++) uout[k * plane + (long long)j * pitch + i] = uin[k * plane + (long long)j * pitch + i];
    return;
  }
  // Indices clamped at the walls: the reference's transmissive ghost copies.
  const T* col = uin + (i < 0 ? 0 : (i < nx ? i : nx - 1));
  auto load = [&](int j) {
    Cell<T> c;
    const T* q = col + (long long)(j < 0 ? 0 : (j < ny ? j : ny - 1)) * pitch;
#pragma unroll
    for (int k = 0; k < NV; k++) c.v[k] = q[k * plane];
    return c;
  };
  unsigned long long bx = 0ull, by = 0ull;
  auto store = [&](const Cell<T>& c, int j) {
    if (!owns) return;
#pragma unroll
    for (int k = 0; k < NV; k++) uout[k * plane + (long long)j * pitch + i] = c.v[k];
    T vx, vy;
    k_speeds(c.v, vx, vy);
    const unsigned long long sx = speed_bits((double)vx), sy = speed_bits((double)vy);
    bx = sx > bx ? sx : bx;
    by = sy > by ? sy : by;
  };
  const T dt = sc.dt;
  const T facx = (T)0.5 * dt / dx, facy = (T)0.5 * dt / dy, rx = dt / dx, ry = dt / dy;
  ColumnSweep<T, HLL> col_sweep(facy, ry);
  Cell<T> next = load(j0 - 2);
  if (sc.n % 2 == 0) {  // x sweep on every row, then y
#pragma unroll 2
    for (int j = j0 - 2; j < j1 + 2; j++) {
      const Cell<T> u = next;
      next = load(j + 1);
      const Cell<T> r = col_sweep.push(sweep_row_x<T, HLL>(u, facx, rx));
      if (j >= j0 + 2) store(r, j - 2);
    }
  } else {
#pragma unroll 2
    for (int j = j0 - 2; j < j1 + 2; j++) {
      const Cell<T> u = next;
      next = load(j + 1);
      const Cell<T> r = col_sweep.push(u);
      if (j >= j0 + 2) store(sweep_row_x<T, HLL>(r, facx, rx), j - 2);
    }
  }
  bx = warp_max(bx);
  by = warp_max(by);
  if (lane == 0) {
    if (bx) atomicMax(&ctrl->sx[(sc.n + 1) % 3], bx);
    if (by) atomicMax(&ctrl->sy[(sc.n + 1) % 3], by);
  }
}

template <class T>
__global__ void __launch_bounds__(256) speed_kernel(const T* __restrict__ u, int nx, int ny, int pitch,
                                                    long long plane, EulerCtrl* ctrl, int slot) {
  unsigned long long bx = 0, by = 0;
  for (long long q = blockIdx.x * 256LL + threadIdx.x; q < (long long)nx * ny; q += (long long)gridDim.x * 256) {
    const int i = (int)(q % nx), j = (int)(q / nx);
    T U4[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) U4[k] = u[k * plane + (long long)j * pitch + i];
    T vx, vy;
    k_speeds(U4, vx, vy);
    const unsigned long long sx = speed_bits((double)vx), sy = speed_bits((double)vy);
    bx = sx > bx ? sx : bx;
    by = sy > by ? sy : by;
  }
  bx = warp_max(bx);
  by = warp_max(by);
  if ((threadIdx.x & 31) == 0) {
    if (bx) atomicMax(&ctrl->sx[slot], bx);
    if (by) atomicMax(&ctrl->sy[slot], by);
  }
}

// Primitives [ny][nx][4] of the conservative state, in the reference's
// expressions (the parity build's flavour gives the bits of the host's
// cons_to_prim).  Bound by its two passes over memory.
template <class T>
__global__ void __launch_bounds__(256) prims_kernel(const T* __restrict__ u, int nx, int ny, int pitch,
                                                    long long plane, T* __restrict__ out) {
  for (long long q = blockIdx.x * 256LL + threadIdx.x; q < (long long)nx * ny; q += (long long)gridDim.x * 256) {
    const int i = (int)(q % nx), j = (int)(q / nx);
    T U4[NV], W4[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) U4[k] = u[k * plane + (long long)j * pitch + i];
    cons_to_prim(U4, W4);
    struct alignas(16) Pair {
      T a[16 / sizeof(T)];
    };
    Pair* o = reinterpret_cast<Pair*>(out + NV * q);
#pragma unroll
    for (int k = 0; k < NV; k += (int)(16 / sizeof(T))) {
      Pair v;
#pragma unroll
      for (int m = 0; m < (int)(16 / sizeof(T)); m++) v.a[m] = W4[k + m];
      o[k / (int)(16 / sizeof(T))] = v;
    }
  }
}

// The whole 1D run in one CTA (riemann1d_cpu.cpp:95-196); arrays in global
// memory (tiny, L1/L2-resident).  u = [3][N+4] with ghosts, f = [3][N+4].
template <class T, bool HLL>
__global__ void __launch_bounds__(1024) riemann1d_kernel(T* __restrict__ u, T* __restrict__ f, int N, T t_end,
                                                         long long max_iters, double* __restrict__ out_t,
                                                         long long* __restrict__ out_steps, int* __restrict__ err) {
  const int GH = 2, TOT = N + 4;
  T* U0 = u;
  T* U1 = u + TOT;
  T* U2 = u + 2 * TOT;
  T* F0 = f;
  T* F1 = f + TOT;
  T* F2 = f + 2 * TOT;
  const T DX = ((T)1.0 - (T)0.0) / (T)N, CFL = (T)0.8;
  __shared__ unsigned long long red[32];
  T t = (T)0.0;
  long long step = 0;
  while (t < t_end) {
    if (step >= max_iters) {  // the reference has no such limit; a GPU loop must
      if (threadIdx.x == 0) *err = 1;
      break;
    }
    if (threadIdx.x < GH) {
      const int g = threadIdx.x, ir = TOT - 1 - g, in = TOT - 1 - GH;
      U0[g] = U0[GH];
      U1[g] = U1[GH];
      U2[g] = U2[GH];
      U0[ir] = U0[in];
      U1[ir] = U1[in];
      U2[ir] = U2[in];
    }
    unsigned long long m = 0;
    for (int i = GH + threadIdx.x; i < N + GH; i += blockDim.x) {
      const unsigned long long b = speed_bits((double)speed_1d(U0[i], U1[i], U2[i]));
      m = b > m ? b : m;
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) m = red[w] > m ? red[w] : m;
    const T ms = (T)bits_speed(m);
    T dt = CFL * DX / ms;
    if (t + dt > t_end) dt = t_end - t;
    const T fac = (T)0.5 * dt / DX;
    for (int i = GH - 1 + threadIdx.x; i < N + GH; i += blockDim.x) {
      T Wq[4][3];
#pragma unroll
      for (int q = 0; q < 4; q++) cons_to_prim_1d(U0[i - 1 + q], U1[i - 1 + q], U2[i - 1 + q], Wq[q]);
      T Lf[3], Rf[3], L0[3], R0[3], Lh[3], Oh[3], fl[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        muscl_recon(Wq[0][k], Wq[1][k], Wq[2][k], Lf[k], Rf[k]);
        muscl_recon(Wq[1][k], Wq[2][k], Wq[3][k], L0[k], R0[k]);
      }
      hancock_1d(Rf, Lf, Rf, Lh, fac);
      hancock_1d(L0, L0, R0, Oh, fac);
      if (HLL)
        hll_flux_1d(Lh, Oh, fl);
      else
        hllc_flux_1d(Lh, Oh, fl);
      F0[i] = fl[0];
      F1[i] = fl[1];
      F2[i] = fl[2];
    }
    __syncthreads();
    const T ratio = dt / DX;
    for (int i = GH + threadIdx.x; i < N + GH; i += blockDim.x) {
      U0[i] -= ratio * (F0[i] - F0[i - 1]);
      U1[i] -= ratio * (F1[i] - F1[i - 1]);
      U2[i] -= ratio * (F2[i] - F2[i - 1]);
    }
    __syncthreads();
    t += dt;
    step++;
  }
  if (threadIdx.x == 0) {
    *out_t = (double)t;
    *out_steps = step;
  }
}

template <class T, int TY, int NT, int MINB, bool HLL>
cudaError_t launch_step(const void* uin, void* uout, int nx, int ny, int pitch, long long plane, double dx, double dy,
                        double cfl, EulerCtrl* ctrl, int p, cudaStream_t s) {
  auto k = step_kernel<T, TY, NT, MINB, HLL>;  // shared-memory limit set by prepare()
  const size_t smem = sizeof(Tile<T, TY>);
  const dim3 grid((nx + TW - 1) / TW, (ny + TY - 1) / TY);
  k<<<grid, NT, smem, s>>>(static_cast<const T*>(uin), static_cast<T*>(uout), nx, ny, pitch, plane, (T)dx, (T)dy,
                           (T)cfl, ctrl, p);
  return cudaGetLastError();
}

template <class T, int MINB>
cudaError_t launch_stream(int hll, int rows, const void* uin, void* uout, int nx, int ny, int pitch, long long plane,
                          double dx, double dy, double cfl, EulerCtrl* ctrl, int p, cudaStream_t s) {
  const long long grid = (long long)((nx + kStripW - 1) / kStripW) * ((ny + rows - 1) / rows);
  auto k = hll ? stream_kernel<T, true, MINB> : stream_kernel<T, false, MINB>;
  k<<<(unsigned)grid, 32, 0, s>>>(static_cast<const T*>(uin), static_cast<T*>(uout), nx, ny, pitch, plane, (T)dx,
                                    (T)dy, (T)cfl, rows, ctrl, p);
  return cudaGetLastError();
}

template <class T, int TY, int NT, int MINB>
cudaError_t allow_smem() {
  cudaError_t e = cudaFuncSetAttribute(step_kernel<T, TY, NT, MINB, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Tile<T, TY>));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(step_kernel<T, TY, NT, MINB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(Tile<T, TY>));
  return e;
}

template <class T, int TY, int NT, int MINB>
cudaError_t launch_any(int hll, const void* uin, void* uout, int nx, int ny, int pitch, long long plane, double dx,
                       double dy, double cfl, EulerCtrl* ctrl, int p, cudaStream_t s) {
  return hll ? launch_step<T, TY, NT, MINB, true>(uin, uout, nx, ny, pitch, plane, dx, dy, cfl, ctrl, p, s)
             : launch_step<T, TY, NT, MINB, false>(uin, uout, nx, ny, pitch, plane, dx, dy, cfl, ctrl, p, s);
}

}  // namespace

// Rows per warp of the streaming kernel: the candidate of least modelled time.
// With `cap` resident warps per SM and c of them on a scheduler a row takes
// max(t1, t0 + tc c) (fitted at 200^2 .. 4096^2 over 2 .. 128 rows: within 10 % of
// the times measured); full waves take the time of cap, the last one that of what
// is left over.  Few rows cost halo rows, many leave SMs idle.
struct StreamModel {
  int cap;
  double t1, t0, tc;
};
constexpr StreamModel kStream64 = {16, 1.03, 0.45, 0.43}, kStream32 = {32, 0.57, 0.14, 0.25};

int stream_rows(const StreamModel& m, int nx, int ny) {
  const long long strips = (nx + kStripW - 1) / kStripW;
  auto row_time = [&](double warps) {  // per SM
    const double t = m.t0 + m.tc * ((long long)(warps / 4) + ((long long)warps % 4 != 0 || warps != (long long)warps));
    return warps <= 0 ? 0.0 : (t > m.t1 ? t : m.t1);
  };
  int best = 2;
  double best_t = -1;
  for (int rows : {2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128}) {
    const double per_sm = (double)(strips * ((ny + rows - 1) / rows)) / 148.0;
    const long long full = (long long)(per_sm / m.cap);
    const double t = (rows + 4) * (full * row_time(m.cap) + row_time(per_sm - (double)full * m.cap));
    if (best_t < 0 || t < best_t) best_t = t, best = rows;
  }
  return best;
}

// Which kernel steps a grid.  Performance build: binary64 grids of at most one
// wave of 32 x 12 tiles (two 512-thread CTAs per SM) run the shared-memory tile
// kernel, whose phases spread a step over more threads: 200^2 7.9 us a step against
// 8.9 streaming, 500 x 197 10.9 against 12.5; past one wave (400^2) 22 against 15.
// Binary32 streams at every size (200^2: 6.0 against 8.0 us).
//
// Parity build: its expressions take more registers (gamma is a binary64 constant in
// binary32 too), so the streaming kernel spills and each warp's chain is longer,
// and tiles win further up.  Us a step, tiles against streaming: binary32 32 x 32
// 200^2 15 / 23, 1024^2 77 / 96, 3200^2 684 / 728, 3500^2 824 / 821, 4096^2 1118 /
// 1096; binary64 32 x 16 HLLC 500^2 41 / 53, 850^2 100 / 104, 1500^2 270 / 281, 1900^2
// 428 / 421, 4096^2 1909 / 1577; HLL 500^2 38 / 44, 750^2 73 / 73, 1024^2 125 / 113.
constexpr int kTileH = 12, kThreads = 512;
#if !PMHD_EULER_FAST
constexpr int kWideH = 16, kTileH32 = 32;                 // larger tiles, binary64 / binary32
constexpr int kWaves32 = 40, kWavesHllc = 22, kWavesHll = 4;  // tiles up to this many waves
#endif

long long tiles_of(int nx, int ny, int h) { return (long long)((nx + TW - 1) / TW) * ((ny + h - 1) / h); }

// Test hook: PMHD_EULER_STREAM=1 streams at every size.
bool always_stream() {
  const char* e = std::getenv("PMHD_EULER_STREAM");
  return e && e[0] == '1';
}

cudaError_t prepare() {
  cudaError_t e = allow_smem<double, kTileH, kThreads, 2>();
#if !PMHD_EULER_FAST
  if (e == cudaSuccess) e = allow_smem<double, kWideH, kThreads, 2>();
  if (e == cudaSuccess) e = allow_smem<float, kTileH32, kThreads, 2>();
#endif
  return e;
}

cudaError_t step2d(int fp32, int hll, const void* uin, void* uout, int nx, int ny, int pitch, long long plane,
                   double dx, double dy, double cfl, EulerCtrl* ctrl, int p, cudaStream_t s) {
  const long long wave = 2 * 148;
  const bool tiles = !always_stream();
  if (fp32) {
#if !PMHD_EULER_FAST
    if (tiles && tiles_of(nx, ny, kTileH32) <= kWaves32 * wave)
      return launch_any<float, kTileH32, kThreads, 2>(hll, uin, uout, nx, ny, pitch, plane, dx, dy, cfl, ctrl, p, s);
#endif
    return launch_stream<float, kStream32.cap>(hll, stream_rows(kStream32, nx, ny), uin, uout, nx, ny, pitch, plane,
                                               dx, dy, cfl, ctrl, p, s);
  }
  if (tiles && tiles_of(nx, ny, kTileH) <= wave)
    return launch_any<double, kTileH, kThreads, 2>(hll, uin, uout, nx, ny, pitch, plane, dx, dy, cfl, ctrl, p, s);
#if !PMHD_EULER_FAST
  if (tiles && tiles_of(nx, ny, kWideH) <= (hll ? kWavesHll : kWavesHllc) * wave)
    return launch_any<double, kWideH, kThreads, 2>(hll, uin, uout, nx, ny, pitch, plane, dx, dy, cfl, ctrl, p, s);
#endif
  return launch_stream<double, kStream64.cap>(hll, stream_rows(kStream64, nx, ny), uin, uout, nx, ny, pitch, plane, dx,
                                              dy, cfl, ctrl, p, s);
}

cudaError_t speed2d(int fp32, const void* u, int nx, int ny, int pitch, long long plane, EulerCtrl* ctrl, int slot,
                    cudaStream_t s) {
  const long long n = (long long)nx * ny;
  long long g = (n + 255) / 256;
  if (g > 148 * 8) g = 148 * 8;
  if (fp32)
    speed_kernel<float><<<(unsigned)g, 256, 0, s>>>(static_cast<const float*>(u), nx, ny, pitch, plane, ctrl, slot);
  else
    speed_kernel<double><<<(unsigned)g, 256, 0, s>>>(static_cast<const double*>(u), nx, ny, pitch, plane, ctrl, slot);
  return cudaGetLastError();
}

cudaError_t prims2d(int fp32, const void* u, int nx, int ny, int pitch, long long plane, void* out, cudaStream_t s) {
  const long long n = (long long)nx * ny;
  long long g = (n + 255) / 256;
  if (g > 148 * 8) g = 148 * 8;
  if (fp32)
    prims_kernel<float><<<(unsigned)g, 256, 0, s>>>(static_cast<const float*>(u), nx, ny, pitch, plane,
                                                    static_cast<float*>(out));
  else
    prims_kernel<double><<<(unsigned)g, 256, 0, s>>>(static_cast<const double*>(u), nx, ny, pitch, plane,
                                                     static_cast<double*>(out));
  return cudaGetLastError();
}

cudaError_t run1d(int fp32, int hll, void* u, void* f, int n, double t_end, long long max_iters, double* out_t,
                  long long* out_steps, int* err, cudaStream_t s) {
  if (fp32) {
    if (hll)
      riemann1d_kernel<float, true><<<1, 1024, 0, s>>>(static_cast<float*>(u), static_cast<float*>(f), n, (float)t_end,
                                                       max_iters, out_t, out_steps, err);
    else
      riemann1d_kernel<float, false><<<1, 1024, 0, s>>>(static_cast<float*>(u), static_cast<float*>(f), n,
                                                        (float)t_end, max_iters, out_t, out_steps, err);
  } else {
    if (hll)
      riemann1d_kernel<double, true><<<1, 1024, 0, s>>>(static_cast<double*>(u), static_cast<double*>(f), n, t_end,
                                                        max_iters, out_t, out_steps, err);
    else
      riemann1d_kernel<double, false><<<1, 1024, 0, s>>>(static_cast<double*>(u), static_cast<double*>(f), n, t_end,
                                                         max_iters, out_t, out_steps, err);
  }
  return cudaGetLastError();
}

}  // namespace PMHD_EKNS
}  // namespace euler
}  // namespace pmhd

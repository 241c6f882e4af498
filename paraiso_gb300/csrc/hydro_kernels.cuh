// hydro_kernels.cuh -- Hydro step kernels, templated on the real type.
// Included by hydro_exact.cu (no multiply-add contraction: bit-exact with
// the generated code's arithmetic) and hydro_fast.cu (contraction allowed).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "hydro_scheme.cuh"

namespace om {

// Device scalar block of a Hydro handle.  The first fields are the OM's
// statics (HydroMain.hs:44-53); the rest are runtime state.
struct HydroScalars {
  int32_t generation;
  int32_t pad0;
  double time, cfl, dR0, dR1, extent0, extent1;
  // bit pattern of the CFL minimum of the current state (see hk::ts_bits),
  // double-buffered by step parity
  unsigned long long tsmin[2];
  double dt_last;
  // cfl, dR0, dR1 and extent1 rounded to float by the host whenever it
  // uploads the block (hydro_scalars_refresh), so that FP32 kernels need no
  // per-thread conversion from double; (float)x is the same rounding either
  // side
  float cfl_f, dR0_f, dR1_f, ext1_f;
  // raised by a kernel whose bounded wait for its tensor copies ran out
  uint32_t wait_error;
};

// the float copies of a scalar block (host side, before every upload)
inline void hydro_scalars_refresh(HydroScalars *s) {
  s->cfl_f = (float)s->cfl;
  s->dR0_f = (float)s->dR0;
  s->dR1_f = (float)s->dR1;
  s->ext1_f = (float)s->extent1;
}

struct HydroStepArgs {
  const void *rho, *v0, *v1, *p;   // current state (memory-sized arrays)
  void *nrho, *nv0, *nv1, *np;     // next state
  int n0, n1;                      // grid (cyclic, no margins)
  int nt0;                         // tiles along x
  double gamma;
  float gamma_f;                   // (float)gamma
  HydroScalars *sc;
  // words of the scalar block's allocation that hold the CFL minimum of the
  // current state, that of the new one (all ones before the step), and one
  // that the step sets to all ones for the step after (0: none)
  int ts_read, ts_write, ts_clear;
  // persistent kernels: at most this many CTAs (0 = as many as stay
  // resident); read by the host launcher only
  int grid_limit;
  double *dt_hist;                 // dt of this step is written to dt_hist[0]
  // open boundary only (the OPEN kernels): margin width, memory row pitch
  // (n0 + 2 lm) and the CFL timescale minimum of the margin cells
  int lm, ms0;
  const unsigned long long *margin_min;
};

// word of the scalar block that is tsmin[slot]
constexpr int ts_word(int slot) {
  return (int)(offsetof(HydroScalars, tsmin) / sizeof(unsigned long long)) + slot;
}
__device__ __forceinline__ unsigned long long *ts_at(const HydroStepArgs &a, int word) {
  return reinterpret_cast<unsigned long long *>(a.sc) + word;
}

// What a taped step keeps for the reverse sweep (periodic grids; arrays of
// n0 x n1 values of the OM's Real type): the stage-1 state q; per stage the
// flux differences (left wall - right wall) of each axis that the
// conservative update adds, d[4 * axis + k] for k = density, momentum 0,
// momentum 1, energy; and the stage-2 conserved state before the primitive
// recovery, u2 (density, momentum 0, momentum 1, energy).
struct HydroTapeOut {
  void *q[4];
  void *d1[8];
  void *d2[8];
  void *u2[4];
};

namespace hk {

// A CFL minimum is kept as the bit pattern of a positive value of the OM's
// Real type (float bits zero-extended, or double bits): the bit patterns of
// positive IEEE values order like the values, so atomicMin on them is a min.
template <class R> __device__ __forceinline__ unsigned long long ts_bits(R t);
template <> __device__ __forceinline__ unsigned long long ts_bits<float>(float t) {
  return (unsigned long long)__float_as_uint(t);
}
template <> __device__ __forceinline__ unsigned long long ts_bits<double>(double t) {
  return (unsigned long long)__double_as_longlong(t);
}

template <class R> __device__ __forceinline__ R ts_from_bits(unsigned long long b);
template <> __device__ __forceinline__ float ts_from_bits<float>(unsigned long long b) {
  return __uint_as_float((unsigned int)b);
}
template <> __device__ __forceinline__ double ts_from_bits<double>(unsigned long long b) {
  return __longlong_as_double((long long)b);
}

// block-wide min of CFL bit patterns folded into *dst
__device__ __forceinline__ void block_min_to(unsigned long long v, unsigned long long *dst,
                                             unsigned long long *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w < v ? w : v;
  }
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    v = lane < nw ? red[lane] : ~0ull;
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
      v = w < v ? w : v;
    }
    if (lane == 0) atomicMin(dst, v);
  }
}

template <class R>
__device__ __forceinline__ int wrap(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// periodic index for -n <= i < 2n (one add or subtract, no division)
__device__ __forceinline__ int wrap_near(int i, int n) {
  return i < 0 ? i + n : (i >= n ? i - n : i);
}

// boundaryCondition (HydroMain.hs:105-131): a cell of an open grid whose
// index (ix, iy) lies outside [0, n) holds the jet state, in the OM's Real
// type and operation order
template <class R>
__device__ __forceinline__ hs::Prim<R> jet_state(R g, R dR0, R dR1, R ext1, int ix, int iy) {
  const R cx = dR0 * R(ix), cy = dR1 * R(iy);
  const bool region = (cy > R(0.47) * ext1) && ((cy < R(0.53) * ext1) && (cx < R(0)));
  hs::Prim<R> q;
  q.rho = g * g * (region ? R(1) : R(10));
  q.v0 = region ? R(6) : R(0);
  q.v1 = R(0);
  q.p = R(0.6);
  return q;
}

// the flux differences of one cell's update, as hs::update forms them
template <class R>
__device__ __forceinline__ void tape_diffs(void *const *d, size_t gi, const hs::Flux<R> &l0,
                                           const hs::Flux<R> &r0, const hs::Flux<R> &l1,
                                           const hs::Flux<R> &r1) {
  ((R *)d[0])[gi] = l0.fd - r0.fd;
  ((R *)d[1])[gi] = l0.fm0 - r0.fm0;
  ((R *)d[2])[gi] = l0.fm1 - r0.fm1;
  ((R *)d[3])[gi] = l0.fe - r0.fe;
  ((R *)d[4])[gi] = l1.fd - r1.fd;
  ((R *)d[5])[gi] = l1.fm0 - r1.fm0;
  ((R *)d[6])[gi] = l1.fm1 - r1.fm1;
  ((R *)d[7])[gi] = l1.fe - r1.fe;
}

// Scalars in the OM's Real type: the block's float copies for FP32, the
// doubles themselves for FP64 (the same values (R)x would give).
template <class R> struct Reals;
template <> struct Reals<float> {
  static __device__ __forceinline__ float cfl(const HydroScalars *s) { return s->cfl_f; }
  static __device__ __forceinline__ float dR0(const HydroScalars *s) { return s->dR0_f; }
  static __device__ __forceinline__ float dR1(const HydroScalars *s) { return s->dR1_f; }
  static __device__ __forceinline__ float ext1(const HydroScalars *s) { return s->ext1_f; }
  static __device__ __forceinline__ float gamma(const HydroStepArgs &a) { return a.gamma_f; }
};
template <> struct Reals<double> {
  static __device__ __forceinline__ double cfl(const HydroScalars *s) { return s->cfl; }
  static __device__ __forceinline__ double dR0(const HydroScalars *s) { return s->dR0; }
  static __device__ __forceinline__ double dR1(const HydroScalars *s) { return s->dR1; }
  static __device__ __forceinline__ double ext1(const HydroScalars *s) { return s->extent1; }
  static __device__ __forceinline__ double gamma(const HydroStepArgs &a) { return a.gamma; }
};

// Programmatic dependent launch: the next step's blocks may be scheduled while
// this one drains (launch_dependents), and wait for its completion before they
// read or write anything (wait).  Both do nothing in an ordinary launch.
__device__ __forceinline__ void step_begin() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// dt of this step in the OM's Real type: dtG = cfl * reduce Min dts
template <class R> __device__ __forceinline__ R step_dt(const HydroStepArgs &a) {
  const R tsmin = ts_from_bits<R>(*ts_at(a, a.ts_read));
  return Reals<R>::cfl(a.sc) * tsmin;
}

// The margin cells of an open grid beside the tile at (X0, Y0) are set to 0:
// the generated class copies whole manifests, whose margins are zero, into the
// statics.
template <class R>
__device__ __forceinline__ void clear_margins(const HydroStepArgs &a, int X0, int Y0, int tw,
                                              int th, R *const (&out)[4], int tid, int threads) {
  const int n0 = a.n0, n1 = a.n1, lm = a.lm;
  const int xa = X0 == 0 ? -lm : X0, xb = X0 + tw >= n0 ? n0 + lm : X0 + tw;
  const int ya = Y0 == 0 ? -lm : Y0, yb = Y0 + th >= n1 ? n1 + lm : Y0 + th;
  if (xa >= 0 && ya >= 0 && xb <= n0 && yb <= n1) return;
  const int w = xb - xa, cnt = w * (yb - ya);
  for (int i = tid; i < cnt; i += threads) {
    const int y = ya + i / w, x = xa + i % w;
    if (x >= 0 && y >= 0 && x < n0 && y < n1) continue;
    const size_t gi = (size_t)(y + lm) * a.ms0 + (x + lm);
#pragma unroll
    for (int c = 0; c < 4; ++c) out[c][gi] = R(0);
  }
}

// what a step's tile 0 does for the whole step
template <class R, bool OPEN>
__device__ __forceinline__ void step_end(const HydroStepArgs &a, int tile, R dtG) {
  if (tile != 0 || threadIdx.x != 0) return;
  if (OPEN) atomicMin(ts_at(a, a.ts_write), *a.margin_min);
  if (a.ts_clear) *ts_at(a, a.ts_clear) = ~0ull;
  a.dt_hist[0] = (double)dtG;
  a.sc->dt_last = (double)dtG;
  a.sc->time = a.sc->time + (double)dtG;
}

// 4- or 8-byte asynchronous copy global -> shared, and its group fences
template <class R> __device__ __forceinline__ void cp_async(R *dst, const R *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (sizeof(R) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// the scheme's wall flux and update in the exact (generated order) or the
// production algebra
template <bool FA, int AX, class R>
__device__ __forceinline__ hs::Flux<R> wall_flux(R g, const hf::Consts<R> &k,
                                                 const hs::Prim<R> &L, R cl,
                                                 const hs::Prim<R> &Rt, R cr) {
  if constexpr (FA) return hf::hllc<AX>(k, L, cl, Rt, cr);
  else return hs::hllc<AX>(k, L, cl, Rt, cr);
}

// MUSCL face values in the exact or the production algebra
template <bool FA, class R>
__device__ __forceinline__ void muscl(R x0, R x1, R x2, R x3, R &l, R &r) {
  if constexpr (FA) hf::muscl(x0, x1, x2, x3, l, r);
  else hs::muscl(x0, x1, x2, x3, l, r);
}

// sound speed of a state in the exact or the production algebra
template <bool FA, class R>
__device__ __forceinline__ R face_sound(R g, const hf::Consts<R> &k, R rho, R p) {
  if constexpr (FA) return hf::sound(k, rho, p);
  else return hs::sound(g, rho, p);
}

template <bool FA, class R>
__device__ __forceinline__ hs::Prim<R> cell_update(R g, const hf::Consts<R> &k,
                                                   const hs::Prim<R> &b, R dtdx0, R dtdx1,
                                                   const hs::Flux<R> &l0, const hs::Flux<R> &r0,
                                                   const hs::Flux<R> &l1, const hs::Flux<R> &r1,
                                                   R *cons = nullptr) {
  if constexpr (FA) return hf::update(k, b, dtdx0, dtdx1, l0, r0, l1, r1, cons);
  else return hs::update(k, b, dtdx0, dtdx1, l0, r0, l1, r1, cons);
}

}  // namespace hk

// ---------------------------------------------------------------------------
// CFL timescale minimum of a state (used when no fused step has produced it)
// ---------------------------------------------------------------------------
template <class R>
__global__ void __launch_bounds__(256)
hydro_tsmin_kernel(const R *__restrict__ rho, const R *__restrict__ v0,
                   const R *__restrict__ v1, const R *__restrict__ p, size_t n,
                   double gamma, HydroScalars *sc, int slot) {
  __shared__ unsigned long long red[32];
  const R g = (R)gamma, dR0 = (R)sc->dR0, dR1 = (R)sc->dR1;
  unsigned long long m = ~0ull;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const R t = hs::timescale(g, dR0, dR1, rho[i], v0[i], v1[i], p[i]);
    const unsigned long long b = hk::ts_bits<R>(t);
    m = b < m ? b : m;
  }
  hk::block_min_to(m, &sc->tsmin[slot], red);
}

// ---------------------------------------------------------------------------
// Fused two-stage step on a TX x TY tile with a 3-cell cyclic halo.
// Phases: load (with sound speeds) -> stage-1 walls (order 1, one HLLC per
// face) -> stage-1 cells (dt/2) -> stage-2 walls (MUSCL + HLLC) -> stage-2
// cells (dt), written out with the tile's CFL minimum of the new state.
// ---------------------------------------------------------------------------
template <class R, int TX, int TY> struct FusedSmem {
  static constexpr int PX = TX + 6, PY = TY + 6;   // loaded cells
  static constexpr int QX = TX + 4, QY = TY + 4;   // stage-1 cells
  static constexpr int FXX = TX + 5, FXY = TY + 4; // stage-1 x walls
  static constexpr int FYX = TX + 4, FYY = TY + 5; // stage-1 y walls
  R P[4][PY][PX];
  R C[PY][PX];
  R Q[4][QY][QX];
  hs::Flux<R> fx[FXY * FXX];
  hs::Flux<R> fy[FYY * FYX];
};

// One tile of the fused step (tile index `tile` of the grid described by a),
// run by a whole block; the tile with index 0 advances the instance's time.
// OPEN: the grid has margins of width a.lm; box cells outside the interior
// take the jet state of the boundary condition instead of a periodic image,
// and the margin cells' timescale minimum joins the CFL minimum.
// TAPE (periodic grids): the tile's stage-1 states and both stages' flux
// differences are also written to `tape`.
// FA: the production algebra (hf::) instead of the generated order (hs::).
template <class R, int TX, int TY, int NT, bool OPEN = false, bool TAPE = false, bool FA = false>
__device__ __forceinline__ void fused_tile(const HydroStepArgs &a, int tile,
                                           FusedSmem<R, TX, TY> &s, unsigned long long *red,
                                           const HydroTapeOut *tape = nullptr) {
  using S = FusedSmem<R, TX, TY>;
  const int tid = threadIdx.x;
  const int t0 = tile % a.nt0, t1 = tile / a.nt0;
  const int X0 = t0 * TX, Y0 = t1 * TY;
  const int n0 = a.n0, n1 = a.n1;
  const R g = hk::Reals<R>::gamma(a);
  const hf::Consts<R> K = hf::consts<R>(g);
  const R dR0 = hk::Reals<R>::dR0(a.sc), dR1 = hk::Reals<R>::dR1(a.sc);
  const R dtG = hk::step_dt<R>(a);
  const R dtHalf = dtG / R(2);
  const R *rho = (const R *)a.rho, *vx = (const R *)a.v0, *vy = (const R *)a.v1,
          *pr = (const R *)a.p;

  // phase 0: load primitives and sound speeds.  Box indices run from -3 to
  // n + T + 1 (T the tile extent), inside [-n, 2n) once n >= T + 8.
  const bool near = n0 >= TX + 8 && n1 >= TY + 8;
  for (int i = tid; i < S::PY * S::PX; i += NT) {
    const int py = i / S::PX, px = i - py * S::PX;
    R r, u, v, q;
    if (OPEN) {
      const int ix = X0 + px - 3, iy = Y0 + py - 3;
      if (ix < 0 || iy < 0 || ix >= n0 || iy >= n1) {
        const hs::Prim<R> j = hk::jet_state<R>(g, dR0, dR1, hk::Reals<R>::ext1(a.sc), ix, iy);
        r = j.rho; u = j.v0; v = j.v1; q = j.p;
      } else {
        const size_t gi = (size_t)(iy + a.lm) * a.ms0 + (ix + a.lm);
        r = rho[gi]; u = vx[gi]; v = vy[gi]; q = pr[gi];
      }
    } else {
      const int gy = near ? hk::wrap_near(Y0 + py - 3, n1) : hk::wrap<R>(Y0 + py - 3, n1);
      const int gx = near ? hk::wrap_near(X0 + px - 3, n0) : hk::wrap<R>(X0 + px - 3, n0);
      const size_t gi = (size_t)gy * n0 + gx;
      r = rho[gi]; u = vx[gi]; v = vy[gi]; q = pr[gi];
    }
    s.P[0][py][px] = r;
    s.P[1][py][px] = u;
    s.P[2][py][px] = v;
    s.P[3][py][px] = q;
    s.C[py][px] = hk::face_sound<FA>(g, K, r, q);
  }
  __syncthreads();

  // phase 1: stage-1 walls, order-1 reconstruction (L = cell left, R = cell)
  {
    constexpr int NX = S::FXY * S::FXX, NY = S::FYY * S::FYX;
    for (int i = tid; i < NX + NY; i += NT) {
      if (i < NX) {
        const int fy = i / S::FXX, fx = i - fy * S::FXX;
        const int py = fy + 1;
        const hs::Prim<R> L{s.P[0][py][fx], s.P[1][py][fx], s.P[2][py][fx], s.P[3][py][fx]};
        const hs::Prim<R> Rt{s.P[0][py][fx + 1], s.P[1][py][fx + 1], s.P[2][py][fx + 1],
                             s.P[3][py][fx + 1]};
        s.fx[i] = hk::wall_flux<FA, 0>(g, K, L, s.C[py][fx], Rt, s.C[py][fx + 1]);
      } else {
        const int j = i - NX;
        const int fy = j / S::FYX, fx = j - fy * S::FYX;
        const int px = fx + 1;
        const hs::Prim<R> L{s.P[0][fy][px], s.P[1][fy][px], s.P[2][fy][px], s.P[3][fy][px]};
        const hs::Prim<R> Rt{s.P[0][fy + 1][px], s.P[1][fy + 1][px], s.P[2][fy + 1][px],
                             s.P[3][fy + 1][px]};
        s.fy[j] = hk::wall_flux<FA, 1>(g, K, L, s.C[fy][px], Rt, s.C[fy + 1][px]);
      }
    }
  }
  __syncthreads();

  // phase 2: stage-1 cells
  {
    const R dtdx0 = hs::div(dtHalf, dR0), dtdx1 = hs::div(dtHalf, dR1);
    for (int i = tid; i < S::QY * S::QX; i += NT) {
      const int qy = i / S::QX, qx = i - qy * S::QX;
      const int py = qy + 1, px = qx + 1;
      const hs::Prim<R> b{s.P[0][py][px], s.P[1][py][px], s.P[2][py][px], s.P[3][py][px]};
      const hs::Prim<R> q = hk::cell_update<FA>(g, K, b, dtdx0, dtdx1, s.fx[qy * S::FXX + qx],
                                                s.fx[qy * S::FXX + qx + 1], s.fy[qy * S::FYX + qx],
                                                s.fy[(qy + 1) * S::FYX + qx]);
      s.Q[0][qy][qx] = q.rho;
      s.Q[1][qy][qx] = q.v0;
      s.Q[2][qy][qx] = q.v1;
      s.Q[3][qy][qx] = q.p;
      if (TAPE) {
        const int ty = qy - 2, tx = qx - 2;
        if (ty >= 0 && ty < TY && tx >= 0 && tx < TX && Y0 + ty < n1 && X0 + tx < n0) {
          const size_t gi = (size_t)(Y0 + ty) * n0 + (X0 + tx);
          ((R *)tape->q[0])[gi] = q.rho;
          ((R *)tape->q[1])[gi] = q.v0;
          ((R *)tape->q[2])[gi] = q.v1;
          ((R *)tape->q[3])[gi] = q.p;
          hk::tape_diffs<R>(tape->d1, gi, s.fx[qy * S::FXX + qx], s.fx[qy * S::FXX + qx + 1],
                            s.fy[qy * S::FYX + qx], s.fy[(qy + 1) * S::FYX + qx]);
        }
      }
    }
  }
  __syncthreads();

  // phase 3: stage-2 walls with MUSCL-minmod reconstruction of stage-1 cells
  {
    constexpr int NX = TY * (TX + 1), NY = (TY + 1) * TX;
    for (int i = tid; i < NX + NY; i += NT) {
      hs::Prim<R> L, Rt;
      if (i < NX) {
        const int sy = i / (TX + 1), sx = i - sy * (TX + 1);
        const int qy = sy + 2;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          R l, r;
          hk::muscl<FA>(s.Q[f][qy][sx], s.Q[f][qy][sx + 1], s.Q[f][qy][sx + 2], s.Q[f][qy][sx + 3],
                    l, r);
          (&L.rho)[f] = l;
          (&Rt.rho)[f] = r;
        }
        s.fx[i] = hk::wall_flux<FA, 0>(g, K, L, hk::face_sound<FA>(g, K, L.rho, L.p), Rt,
                                       hk::face_sound<FA>(g, K, Rt.rho, Rt.p));
      } else {
        const int j = i - NX;
        const int sy = j / TX, sx = j - sy * TX;
        const int qx = sx + 2;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          R l, r;
          hk::muscl<FA>(s.Q[f][sy][qx], s.Q[f][sy + 1][qx], s.Q[f][sy + 2][qx], s.Q[f][sy + 3][qx],
                    l, r);
          (&L.rho)[f] = l;
          (&Rt.rho)[f] = r;
        }
        s.fy[j] = hk::wall_flux<FA, 1>(g, K, L, hk::face_sound<FA>(g, K, L.rho, L.p), Rt,
                                       hk::face_sound<FA>(g, K, Rt.rho, Rt.p));
      }
    }
  }
  __syncthreads();

  // phase 4: stage-2 cells, written out, with the CFL minimum of the new state
  unsigned long long m = ~0ull;
  {
    const R dtdx0 = hs::div(dtG, dR0), dtdx1 = hs::div(dtG, dR1);
    R *orho = (R *)a.nrho, *ovx = (R *)a.nv0, *ovy = (R *)a.nv1, *opr = (R *)a.np;
    for (int i = tid; i < TY * TX; i += NT) {
      const int oy = i / TX, ox = i - oy * TX;
      const int gy = Y0 + oy, gx = X0 + ox;
      if (gy >= n1 || gx >= n0) continue;
      const int py = oy + 3, px = ox + 3;
      const hs::Prim<R> b{s.P[0][py][px], s.P[1][py][px], s.P[2][py][px], s.P[3][py][px]};
      R cons[4];
      const hs::Prim<R> q = hk::cell_update<FA>(
          g, K, b, dtdx0, dtdx1, s.fx[oy * (TX + 1) + ox], s.fx[oy * (TX + 1) + ox + 1],
          s.fy[oy * TX + ox], s.fy[(oy + 1) * TX + ox], TAPE ? cons : nullptr);
      const size_t gi = OPEN ? (size_t)(gy + a.lm) * a.ms0 + (gx + a.lm) : (size_t)gy * n0 + gx;
      if (TAPE) {
        hk::tape_diffs<R>(tape->d2, gi, s.fx[oy * (TX + 1) + ox], s.fx[oy * (TX + 1) + ox + 1],
                          s.fy[oy * TX + ox], s.fy[(oy + 1) * TX + ox]);
#pragma unroll
        for (int c = 0; c < 4; ++c) ((R *)tape->u2[c])[gi] = cons[c];
      }
      orho[gi] = q.rho;
      ovx[gi] = q.v0;
      ovy[gi] = q.v1;
      opr[gi] = q.p;
      const R t = hs::timescale(g, dR0, dR1, q.rho, q.v0, q.v1, q.p);
      const unsigned long long bits = hk::ts_bits<R>(t);
      m = bits < m ? bits : m;
    }
  }
  if (OPEN) {
    R *out[4] = {(R *)a.nrho, (R *)a.nv0, (R *)a.nv1, (R *)a.np};
    hk::clear_margins<R>(a, X0, Y0, TX, TY, out, tid, NT);
  }
  hk::block_min_to(m, ts_at(a, a.ts_write), red);
  hk::step_end<R, OPEN>(a, tile, dtG);
}

template <class R, int TX, int TY, int NT, bool OPEN = false, bool FA = false>
__global__ void __launch_bounds__(NT)
hydro_fused_kernel(HydroStepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long red[32];
  hk::step_begin();
  fused_tile<R, TX, TY, NT, OPEN, false, FA>(
      a, blockIdx.x, *reinterpret_cast<FusedSmem<R, TX, TY> *>(smem_raw), red);
}

// ---------------------------------------------------------------------------
// The step as two kernels with the stage-1 state in global memory between them.
// A double-precision step is bound by its arithmetic (two results a cycle per
// SM), and the fused tile's halo repeats a third of it: 2.9 stage-1 walls and
// 1.4 stage-1 cells per cell of a 32 x 16 tile.  Here every cell is advanced
// once and the walls of a tile's edge twice (2.1 per cell and stage), for 64
// bytes more per cell, which cost nothing beside that.  1024^2 open: 1.17 ms a
// step fused, 0.92 so, 0.85 with the momenta, energies and differences that
// several walls use formed per cell; 384 x 256: 175 us, 140, 132, and 116 with
// tiles that suit the grid (hydro_f64_tile).  256 threads: 128 leave a small
// grid too few warps (384 x 256: 206 us against 141).  With a part or all of the
// products formed on the integer pipes too, the step was 4 to 27 % slower: the
// double instructions' issue gaps are not free.
// ---------------------------------------------------------------------------
struct HydroStage1 {
  void *q[4];       // stage-1 state, memory-sized arrays
  int tw, th;       // tile, at most kF64Tile a side
  unsigned inv[5];  // 65535 / (tw + k) + 1
  // i / (tw + k) for i < 2000 (exact: the excess of inv over 2^16 / (tw + k)
  // times i stays below 2^16)
  __device__ __forceinline__ int row(int i, int k) const {
    return (int)((unsigned)i * inv[k] >> 16);
  }
};
constexpr int kF64Tile = 16;

namespace hk {
// What a block's threads share of the quotients that are the same for all of
// them (formed by each thread they were a fifth of a step's double operations).
template <class R> struct alignas(16) StageConsts {
  hs::Gas<R> gas;
  R dtdx0, dtdx1;
  StageConsts() = default;
  __device__ StageConsts(R g, R dt, R dR0, R dR1)
      : gas(hs::gas(g)), dtdx0(hs::div(dt, dR0)), dtdx1(hs::div(dt, dR1)) {}
};
}  // namespace hk

template <class R> struct Stage1Smem {
  static constexpr int TX = kF64Tile, TY = kF64Tile;
  static constexpr int PX = TX + 2, PY = TY + 2;
  hk::StageConsts<R> c;
  R P[4][PY][PX];
  R C[PY][PX];
  R M[3][PY][PX];  // momenta and energy
  hs::Flux<R> fx[TY * (TX + 1)];
  hs::Flux<R> fy[(TY + 1) * TX];
  // the momenta and energies of a wall's cells, m and m + step
  template <int AX> struct Wall {
    const R *m;
    int step;
    __device__ __forceinline__ R momL() const { return m[AX * PY * PX]; }
    __device__ __forceinline__ R momR() const { return m[AX * PY * PX + step]; }
    __device__ __forceinline__ hs::Cons<R> side(bool left, R, R, R, R) const {
      const R *x = left ? m : m + step;
      return hs::Cons<R>{x[0], x[PY * PX], x[2 * PY * PX]};
    }
  };
};
template <class R> struct Stage2Smem {
  static constexpr int TX = kF64Tile, TY = kF64Tile;
  static constexpr int QX = TX + 4, QY = TY + 4;
  hk::StageConsts<R> c;
  R Q[4][QY][QX];
  R dx[4][TY][TX + 3];  // differences of a tile row's cells, and of a column's
  R dy[4][TY + 3][TX];
  hs::Flux<R> fx[TY * (TX + 1)];
  hs::Flux<R> fy[(TY + 1) * TX];
};

// Stage 1 of the cells [-e, n + e) of both axes (e = 2 on an open grid, whose
// margin cells step from the jet state; else 0); a.nt0 tiles along x of that
// range.
template <class R, int NT, bool OPEN>
__global__ void __launch_bounds__(NT)
hydro_stage1_kernel(HydroStepArgs a, const __grid_constant__ HydroStage1 o) {
  using S = Stage1Smem<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S &s = *reinterpret_cast<S *>(smem_raw);
  hk::step_begin();
  const int tid = threadIdx.x, tile = blockIdx.x;
  const int t0 = tile % a.nt0, t1 = tile / a.nt0;
  constexpr int e = OPEN ? 2 : 0;
  const int tw = o.tw, th = o.th;
  const int X0 = t0 * tw - e, Y0 = t1 * th - e;
  const int n0 = a.n0, n1 = a.n1;
  const R g = hk::Reals<R>::gamma(a);
  const R dR0 = hk::Reals<R>::dR0(a.sc), dR1 = hk::Reals<R>::dR1(a.sc);
  if (tid == 0) s.c = hk::StageConsts<R>(g, hk::step_dt<R>(a) / R(2), dR0, dR1);
  const R *f[4] = {(const R *)a.rho, (const R *)a.v0, (const R *)a.v1, (const R *)a.p};
  const bool near = n0 >= tw + 2 && n1 >= th + 2;
  for (int i = tid; i < (th + 2) * (tw + 2); i += NT) {
    const int py = o.row(i, 2), px = i - py * (tw + 2);
    const int ix = X0 + px - 1, iy = Y0 + py - 1;
    hs::Prim<R> w;
    if (OPEN) {
      if (ix < 0 || iy < 0 || ix >= n0 || iy >= n1) {
        w = hk::jet_state<R>(g, dR0, dR1, hk::Reals<R>::ext1(a.sc), ix, iy);
      } else {
        const size_t gi = (size_t)(iy + a.lm) * a.ms0 + (ix + a.lm);
        w = hs::Prim<R>{f[0][gi], f[1][gi], f[2][gi], f[3][gi]};
      }
    } else {
      const int gy = near ? hk::wrap_near(iy, n1) : hk::wrap<R>(iy, n1);
      const int gx = near ? hk::wrap_near(ix, n0) : hk::wrap<R>(ix, n0);
      const size_t gi = (size_t)gy * n0 + gx;
      w = hs::Prim<R>{f[0][gi], f[1][gi], f[2][gi], f[3][gi]};
    }
    s.P[0][py][px] = w.rho;
    s.P[1][py][px] = w.v0;
    s.P[2][py][px] = w.v1;
    s.P[3][py][px] = w.p;
    s.C[py][px] = hs::sound(g, w.rho, w.p);
  }
  __syncthreads();
  const hs::Gas<R> k = s.c.gas;
  auto cell = [&](int py, int px) {
    return hs::Prim<R>{s.P[0][py][px], s.P[1][py][px], s.P[2][py][px], s.P[3][py][px]};
  };
  for (int i = tid; i < (th + 2) * (tw + 2); i += NT) {
    const int py = o.row(i, 2), px = i - py * (tw + 2);
    const hs::Prim<R> w = cell(py, px);
    const hs::Cons<R> c = hs::cons_of(k, w.rho, w.v0, w.v1, w.p);
    s.M[0][py][px] = c.m0;
    s.M[1][py][px] = c.m1;
    s.M[2][py][px] = c.e;
  }
  __syncthreads();
  const int NX = th * (tw + 1), NY = (th + 1) * tw;
  for (int i = tid; i < NX + NY; i += NT) {
    if (i < NX) {
      const int sy = o.row(i, 1), sx = i - sy * (tw + 1);
      s.fx[i] = hs::hllc<0>(k, cell(sy + 1, sx), s.C[sy + 1][sx], cell(sy + 1, sx + 1),
                            s.C[sy + 1][sx + 1],
                            typename S::template Wall<0>{&s.M[0][sy + 1][sx], 1});
    } else {
      const int j = i - NX, sy = o.row(j, 0), sx = j - sy * tw;
      s.fy[j] = hs::hllc<1>(k, cell(sy, sx + 1), s.C[sy][sx + 1], cell(sy + 1, sx + 1),
                            s.C[sy + 1][sx + 1],
                            typename S::template Wall<1>{&s.M[0][sy][sx + 1], S::PX});
    }
  }
  __syncthreads();
  const R dtdx0 = s.c.dtdx0, dtdx1 = s.c.dtdx1;
  for (int i = tid; i < th * tw; i += NT) {
    const int oy = o.row(i, 0), ox = i - oy * tw;
    const int iy = Y0 + oy, ix = X0 + ox;
    if (iy >= n1 + e || ix >= n0 + e) continue;
    const hs::Cons<R> c{s.M[0][oy + 1][ox + 1], s.M[1][oy + 1][ox + 1], s.M[2][oy + 1][ox + 1]};
    const hs::Prim<R> q = hs::update_cons<R>(
        k, s.P[0][oy + 1][ox + 1], c, dtdx0, dtdx1, s.fx[oy * (tw + 1) + ox],
        s.fx[oy * (tw + 1) + ox + 1], s.fy[oy * tw + ox], s.fy[(oy + 1) * tw + ox], nullptr);
    const size_t gi = OPEN ? (size_t)(iy + a.lm) * a.ms0 + (ix + a.lm) : (size_t)iy * n0 + ix;
    ((R *)o.q[0])[gi] = q.rho;
    ((R *)o.q[1])[gi] = q.v0;
    ((R *)o.q[2])[gi] = q.v1;
    ((R *)o.q[3])[gi] = q.p;
  }
}

// Stage 2, the new state and its CFL minimum.
template <class R, int NT, bool OPEN>
__global__ void __launch_bounds__(NT)
hydro_stage2_kernel(HydroStepArgs a, const __grid_constant__ HydroStage1 o) {
  using S = Stage2Smem<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long red[32];
  S &s = *reinterpret_cast<S *>(smem_raw);
  hk::step_begin();
  constexpr int T = kF64Tile;
  const int tid = threadIdx.x, tile = blockIdx.x;
  const int t0 = tile % a.nt0, t1 = tile / a.nt0;
  const int tw = o.tw, th = o.th;
  const int X0 = t0 * tw, Y0 = t1 * th;
  const int n0 = a.n0, n1 = a.n1, lm = a.lm;
  const R dR0 = hk::Reals<R>::dR0(a.sc), dR1 = hk::Reals<R>::dR1(a.sc);
  const R dtG = hk::step_dt<R>(a);
  if (tid == 0) s.c = hk::StageConsts<R>(hk::Reals<R>::gamma(a), dtG, dR0, dR1);
  const bool near = n0 >= tw + 4 && n1 >= th + 4;
  for (int i = tid; i < (th + 4) * (tw + 4); i += NT) {
    const int qy = o.row(i, 4), qx = i - qy * (tw + 4);
    const int ix = X0 + qx - 2, iy = Y0 + qy - 2;
    size_t gi;
    if (OPEN) {  // rows and columns beyond the last margin cell feed no cell
      gi = (size_t)(min(iy, n1 + 1) + lm) * a.ms0 + (min(ix, n0 + 1) + lm);
    } else {
      const int gy = near ? hk::wrap_near(iy, n1) : hk::wrap<R>(iy, n1);
      const int gx = near ? hk::wrap_near(ix, n0) : hk::wrap<R>(ix, n0);
      gi = (size_t)gy * n0 + gx;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) s.Q[c][qy][qx] = ((const R *)o.q[c])[gi];
  }
  __syncthreads();
  for (int i = tid; i < th * (tw + 3) + (th + 3) * tw; i += NT) {
    const bool x = i < th * (tw + 3);
    const int j = x ? i : i - th * (tw + 3), r = o.row(j, x ? 3 : 0),
              q = j - r * (x ? tw + 3 : tw);
    const int y0 = x ? r + 2 : r, x0 = x ? q : q + 2;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const R d = s.Q[c][y0 + !x][x0 + x] - s.Q[c][y0][x0];
      (x ? s.dx[c][r][q] : s.dy[c][r][q]) = d;
    }
  }
  __syncthreads();
  const hs::Gas<R> k = s.c.gas;
  const int NX = th * (tw + 1), NY = (th + 1) * tw;
  for (int i = tid; i < NX + NY; i += NT) {
    const bool x = i < NX;
    const int j = x ? i : i - NX;
    const int sy = o.row(j, x ? 1 : 0), sx = j - sy * (x ? tw + 1 : tw);
    // the wall lies between cells 1 and 2 of four along its axis
    const int qy = x ? sy + 2 : sy + 1, qx = x ? sx + 1 : sx + 2, dy = x ? 0 : 1, dx = x ? 1 : 0;
    const int step = x ? 1 : T, field = x ? T * (T + 3) : (T + 3) * T;
    const R *d = x ? &s.dx[0][sy][sx] : &s.dy[0][sy][sx];
    hs::Prim<R> L, Rt;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      hs::muscl_of(s.Q[c][qy][qx], s.Q[c][qy + dy][qx + dx], d[c * field], d[c * field + step],
                   d[c * field + 2 * step], (&L.rho)[c], (&Rt.rho)[c]);
    const R cl = hs::sound(k.g, L.rho, L.p), cr = hs::sound(k.g, Rt.rho, Rt.p);
    if (x) s.fx[j] = hs::hllc<0>(k, L, cl, Rt, cr);
    else s.fy[j] = hs::hllc<1>(k, L, cl, Rt, cr);
  }
  __syncthreads();
  unsigned long long m = ~0ull;
  const R dtdx0 = s.c.dtdx0, dtdx1 = s.c.dtdx1;
  const R *f[4] = {(const R *)a.rho, (const R *)a.v0, (const R *)a.v1, (const R *)a.p};
  R *out[4] = {(R *)a.nrho, (R *)a.nv0, (R *)a.nv1, (R *)a.np};
  for (int i = tid; i < th * tw; i += NT) {
    const int oy = o.row(i, 0), ox = i - oy * tw;
    const int gy = Y0 + oy, gx = X0 + ox;
    if (gy >= n1 || gx >= n0) continue;
    const size_t gi = OPEN ? (size_t)(gy + lm) * a.ms0 + (gx + lm) : (size_t)gy * n0 + gx;
    const hs::Prim<R> b{f[0][gi], f[1][gi], f[2][gi], f[3][gi]};
    const hs::Prim<R> q = hs::update(k, b, dtdx0, dtdx1, s.fx[oy * (tw + 1) + ox],
                                     s.fx[oy * (tw + 1) + ox + 1], s.fy[oy * tw + ox],
                                     s.fy[(oy + 1) * tw + ox]);
    out[0][gi] = q.rho;
    out[1][gi] = q.v0;
    out[2][gi] = q.v1;
    out[3][gi] = q.p;
    const unsigned long long bits =
        hk::ts_bits<R>(hs::timescale(k.g, dR0, dR1, q.rho, q.v0, q.v1, q.p));
    m = bits < m ? bits : m;
  }
  if (OPEN) hk::clear_margins<R>(a, X0, Y0, tw, th, out, tid, NT);
  hk::block_min_to(m, ts_at(a, a.ts_write), red);
  hk::step_end<R, OPEN>(a, tile, dtG);
}

// the fused step that also writes the tape of the reverse sweep (periodic)
template <class R, int TX, int TY, int NT, bool FA = false>
__global__ void __launch_bounds__(NT)
hydro_fused_tape_kernel(HydroStepArgs a, const __grid_constant__ HydroTapeOut t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long red[32];
  fused_tile<R, TX, TY, NT, false, true, FA>(
      a, blockIdx.x, *reinterpret_cast<FusedSmem<R, TX, TY> *>(smem_raw), red, &t);
}

// CFL timescale minimum of the margin cells of an open grid (the jet state
// of the boundary condition; it depends only on the index, gamma, dR and
// extent1)
template <class R>
__global__ void __launch_bounds__(256)
hydro_margin_min_kernel(int n0, int n1, int lm, double gamma, const HydroScalars *sc,
                        unsigned long long *out) {
  __shared__ unsigned long long red[32];
  const R g = (R)gamma, dR0 = (R)sc->dR0, dR1 = (R)sc->dR1, ext1 = (R)sc->extent1;
  const int ms0 = n0 + 2 * lm, ms1 = n1 + 2 * lm;
  const size_t total = (size_t)ms0 * ms1;
  unsigned long long m = ~0ull;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const int y = (int)(i / ms0), x = (int)(i - (size_t)y * ms0);
    const int ix = x - lm, iy = y - lm;
    if (ix >= 0 && iy >= 0 && ix < n0 && iy < n1) continue;
    const hs::Prim<R> q = hk::jet_state<R>(g, dR0, dR1, ext1, ix, iy);
    const unsigned long long b = hk::ts_bits<R>(hs::timescale(g, dR0, dR1, q.rho, q.v0, q.v1, q.p));
    m = b < m ? b : m;
  }
  hk::block_min_to(m, out, red);
}

// CFL minimum of an open grid's current state: the interior cells, then
// the margin cells' minimum
template <class R>
__global__ void __launch_bounds__(256)
hydro_tsmin_open_kernel(const R *__restrict__ rho, const R *__restrict__ v0,
                        const R *__restrict__ v1, const R *__restrict__ p, int n0, int n1, int lm,
                        double gamma, HydroScalars *sc, int slot,
                        const unsigned long long *margin_min) {
  __shared__ unsigned long long red[32];
  const R g = (R)gamma, dR0 = (R)sc->dR0, dR1 = (R)sc->dR1;
  const int ms0 = n0 + 2 * lm;
  const size_t n = (size_t)n0 * n1;
  unsigned long long m = ~0ull;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int y = (int)(i / n0), x = (int)(i - (size_t)y * n0);
    const size_t gi = (size_t)(y + lm) * ms0 + (x + lm);
    const R t = hs::timescale(g, dR0, dR1, rho[gi], v0[gi], v1[gi], p[gi]);
    const unsigned long long b = hk::ts_bits<R>(t);
    m = b < m ? b : m;
  }
  hk::block_min_to(m, &sc->tsmin[slot], red);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicMin(&sc->tsmin[slot], *margin_min);
}

// Ensemble step: every tile of every instance is one work item; the
// persistent grid strides over the flattened item list (prefix[k] = first
// item of instance k), so instances of any size advance in one launch, each
// with its own dt, CFL minimum and time (its HydroStepArgs).  Up to
// kEnsPrefixShared instances, the prefix is kept in shared memory.
constexpr int kEnsPrefixShared = 1024;

template <class R, int TX, int TY, int NT, bool FA = false>
__global__ void __launch_bounds__(NT)
hydro_ensemble_kernel(const HydroStepArgs *__restrict__ args, const int *__restrict__ prefix,
                      int count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long red[32];
  __shared__ int spref[kEnsPrefixShared + 1];
  auto &s = *reinterpret_cast<FusedSmem<R, TX, TY> *>(smem_raw);
  // a block's items increase, so its instance index only moves forward: it
  // advances through the prefix (in shared memory when it fits) instead of
  // searching global memory per item
  const bool shared = count <= kEnsPrefixShared;
  if (shared)
    for (int i = threadIdx.x; i <= count; i += NT) spref[i] = prefix[i];
  __syncthreads();
  const int *pf = shared ? spref : prefix;
  const int total = pf[count];
  int lo = 0;  // instance k with prefix[k] <= item < prefix[k+1]
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    while (lo < count - 1 && pf[lo + 1] <= item) ++lo;
    fused_tile<R, TX, TY, NT, false, false, FA>(args[lo], item - pf[lo], s, red);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Plain path: the structure of the generated code.  One thread per cell,
// every Delayed value recomputed from the four primitive arrays in global
// memory (as Hydro_sub_8 does), grid-stride loops, separate timescale and
// reduce passes, and copies of the manifests back into the statics.
// ---------------------------------------------------------------------------
template <class R>
__global__ void __launch_bounds__(256)
hydro_plain_timescale_kernel(const R *__restrict__ rho, const R *__restrict__ v0,
                             const R *__restrict__ v1, const R *__restrict__ p,
                             R *__restrict__ ts, size_t n, double gamma,
                             const HydroScalars *sc) {
  const R g = (R)gamma, dR0 = (R)sc->dR0, dR1 = (R)sc->dR1;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    ts[i] = hs::timescale(g, dR0, dR1, rho[i], v0[i], v1[i], p[i]);
}

template <class R>
__global__ void __launch_bounds__(256)
hydro_plain_reduce_min_kernel(const R *__restrict__ ts, size_t n, unsigned long long *out) {
  __shared__ unsigned long long red[32];
  unsigned long long m = ~0ull;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const unsigned long long b = hk::ts_bits<R>(ts[i]);
    m = b < m ? b : m;
  }
  hk::block_min_to(m, out, red);
}

template <class R> struct PlainView {
  const R *rho, *v0, *v1, *p;
  int n0, n1;
  __device__ __forceinline__ hs::Prim<R> at(int x, int y) const {
    x = hk::wrap<R>(x, n0);
    y = hk::wrap<R>(y, n1);
    const size_t i = (size_t)y * n0 + x;
    return hs::Prim<R>{rho[i], v0[i], v1[i], p[i]};
  }
};

// stage-1 state at (x, y): order-1 walls recomputed from the primitives
template <class R>
__device__ __forceinline__ hs::Prim<R> plain_stage1(const PlainView<R> &V, const hs::Gas<R> &k,
                                                    R dtdx0, R dtdx1, int x, int y) {
  const hs::Prim<R> c = V.at(x, y), xm = V.at(x - 1, y), xp = V.at(x + 1, y),
                    ym = V.at(x, y - 1), yp = V.at(x, y + 1);
  const R g = k.g;
  const R cc = hs::sound(g, c.rho, c.p);
  const hs::Flux<R> l0 = hs::hllc<0>(k, xm, hs::sound(g, xm.rho, xm.p), c, cc);
  const hs::Flux<R> r0 = hs::hllc<0>(k, c, cc, xp, hs::sound(g, xp.rho, xp.p));
  const hs::Flux<R> l1 = hs::hllc<1>(k, ym, hs::sound(g, ym.rho, ym.p), c, cc);
  const hs::Flux<R> r1 = hs::hllc<1>(k, c, cc, yp, hs::sound(g, yp.rho, yp.p));
  return hs::update(k, c, dtdx0, dtdx1, l0, r0, l1, r1);
}

template <int AX, class R>
__device__ __forceinline__ hs::Flux<R> plain_wall2(const hs::Prim<R> &a0, const hs::Prim<R> &a1,
                                                   const hs::Prim<R> &a2, const hs::Prim<R> &a3,
                                                   const hs::Gas<R> &k) {
  const R g = k.g;
  hs::Prim<R> L, Rt;
  hs::muscl(a0.rho, a1.rho, a2.rho, a3.rho, L.rho, Rt.rho);
  hs::muscl(a0.v0, a1.v0, a2.v0, a3.v0, L.v0, Rt.v0);
  hs::muscl(a0.v1, a1.v1, a2.v1, a3.v1, L.v1, Rt.v1);
  hs::muscl(a0.p, a1.p, a2.p, a3.p, L.p, Rt.p);
  return hs::hllc<AX>(k, L, hs::sound(g, L.rho, L.p), Rt, hs::sound(g, Rt.rho, Rt.p));
}

// (single precision: four blocks an SM; of 136 registers a thread only three fit,
// 640 us for 1024^2 against 440)
template <class R>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 4 : 1)
hydro_plain_step_kernel(PlainView<R> V, R *__restrict__ orho, R *__restrict__ ov0,
                        R *__restrict__ ov1, R *__restrict__ op, double gamma, R dtG, R dR0,
                        R dR1) {
  const hs::Gas<R> g = hs::gas<R>((R)gamma);
  const R dtHalf = dtG / R(2);
  const R h0 = dtHalf / dR0, h1 = dtHalf / dR1;
  const R f0 = dtG / dR0, f1 = dtG / dR1;
  const size_t n = (size_t)V.n0 * V.n1;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int y = (int)(i / V.n0), x = (int)(i - (size_t)y * V.n0);
    // stage-1 cells along the two axes (Delayed: recomputed here)
    const hs::Prim<R> qm2 = plain_stage1(V, g, h0, h1, x - 2, y);
    const hs::Prim<R> qm1 = plain_stage1(V, g, h0, h1, x - 1, y);
    const hs::Prim<R> q00 = plain_stage1(V, g, h0, h1, x, y);
    const hs::Prim<R> qp1 = plain_stage1(V, g, h0, h1, x + 1, y);
    const hs::Prim<R> qp2 = plain_stage1(V, g, h0, h1, x + 2, y);
    const hs::Flux<R> l0 = plain_wall2<0>(qm2, qm1, q00, qp1, g);
    const hs::Flux<R> r0 = plain_wall2<0>(qm1, q00, qp1, qp2, g);
    const hs::Prim<R> ym2 = plain_stage1(V, g, h0, h1, x, y - 2);
    const hs::Prim<R> ym1 = plain_stage1(V, g, h0, h1, x, y - 1);
    const hs::Prim<R> yp1 = plain_stage1(V, g, h0, h1, x, y + 1);
    const hs::Prim<R> yp2 = plain_stage1(V, g, h0, h1, x, y + 2);
    const hs::Flux<R> l1 = plain_wall2<1>(ym2, ym1, q00, yp1, g);
    const hs::Flux<R> r1 = plain_wall2<1>(ym1, q00, yp1, yp2, g);
    const hs::Prim<R> q = hs::update(g, V.at(x, y), f0, f1, l0, r0, l1, r1);
    orho[i] = q.rho;
    ov0[i] = q.v0;
    ov1[i] = q.v1;
    op[i] = q.p;
  }
}

}  // namespace om

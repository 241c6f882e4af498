// hydro_persist.cuh -- the persistent production FP32 step on 32 x 32
// tiles: the fused two-stage MUSCL-HLLC step of hydro_kernels.cuh
// (HydroMain.hs:169-276), in the production algebra (hf::), organised for
// the issue rate of a GB300 SM.
//
//  * A CTA strides over the tiles (single grid) or over the (instance,
//    tile) work list (ensembles).  While it computes one tile, the next
//    tile's 40 x 38 box of the four primitive fields lands in the other of
//    two box buffers: by TMA (four 2-D boxes completing on an mbarrier) for
//    tiles whose box lies inside the grid, by 16-byte cp.async with
//    periodically wrapped addresses for the edge tiles.
//  * The box is kept as four planes of 40 floats per row, starting 4 cells
//    left of the tile (a 16-byte aligned x coordinate) and 3 rows below it.
//  * Lanes run along rows of 32 walls or cells, so shared-memory accesses of
//    a warp are consecutive; the few walls and cells beyond 32 per row form
//    a short remainder list.
//  * The stage-1 state is kept as one float4 record per cell, in rows of 37
//    records (an odd pitch: a warp reading a column of records touches
//    every bank group once).
//  * Stage-2 walls are evaluated in runs of three consecutive walls along
//    the wall normal: the limited slope of a cell is formed once for the
//    right state of one wall and the left state of the next.  The 33 walls
//    of a row (or column) are 11 runs, so the 704 wall runs of a tile are
//    exactly one per thread of the 704-thread CTA.
//  * The paired form (PAIR, 352 threads) evaluates two walls or two cells
//    per thread with packed f32x2 instructions (hf::f2): the x wall left of a
//    cell with the y wall below it, a cell with the one above it, a row's
//    x-wall run with a column's y-wall run.  Walls of either axis share the
//    arithmetic in the frame of the wall.
//  * On large grids the paired form runs as one CTA per SM of two groups
//    (persist_run's GROUPS), each with its own shared-memory block and
//    named barrier, whose phases are offset by about half a tile.
//  * Stage 2 of a tile shares its pass with the next tile's sound speeds.
//  * The tile's CFL minimum is folded in registers over all the tiles of a
//    CTA or group (of one instance) and published once.
// Every value is formed by the production algebra's explicit operations
// (hf:: in hydro_scheme.cuh), as in the tile kernels of hydro_kernels.cuh,
// so all of them give the same bits.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "hydro_kernels.cuh"
#include "tma.cuh"

namespace om {
namespace hp {

constexpr int TX = 32, TY = 32;
constexpr int NT = 704;                 // 22 warps; two CTAs per SM
constexpr int NT2 = 352;                // the paired form: 11 warps; two CTAs (or groups) per SM
constexpr int BW = 40, BH = 38;         // box columns X0-4 .. X0+35, rows Y0-3 .. Y0+34
constexpr int PLANE = 1536;             // floats per field plane: 38 x 40 = 1520, padded to 6144 B
constexpr int QP = 37;                  // stage-1 records per row (36 used)
constexpr int F1X = 37, F1Y = 36;       // stage-1 walls per row: x walls (36 rows), y walls (37 rows)
constexpr int F2X = 33, F2Y = 32;       // stage-2 walls per row: x walls (32 rows), y walls (33 rows)
constexpr uint32_t kBoxBytes = 4u * BH * BW * 4u;  // bytes the four TMA boxes deliver

// stage-1 walls: rows of 32 walls first (x, then y), then the remainders
constexpr int kS1XMain = 36 * 32, kS1YMain = 37 * 32, kS1XRem = 36 * 5, kS1YRem = 37 * 4;
constexpr int kS1Items = kS1XMain + kS1YMain + kS1XRem + kS1YRem;  // 2664
constexpr int kQMain = 36 * 32, kQItems = 36 * 36;                  // stage-1 cells
constexpr int kS1PairMain = 37 * 32, kS1Pairs = 37 * 37;  // paired form
constexpr int kQPairMain = 18 * 32, kQPairs = 18 * 36;    // paired form

using Flux = hs::Flux<float>;
using Prim = hs::Prim<float>;

// What the items of one instance share, formed by one warp when the CTA (or
// group) comes to it and read from shared memory instead of being held in
// registers across phases.  Read and formed by every thread for every tile (with
// the tile's place), it took 453 us of a 4096^2 step where 438 do, and 3.16 ms
// of 64 instances of 256 to 2048 cells a side where 2.86 do: there each tile
// began with a chain of loads from global memory.
struct Inst {
  HydroStepArgs a;  // ensembles only
  int first, end;   // its items
  float dt, dR0, dR1;
  float h0, h1, f0, f1;  // dt/2 and dt over dR0 and dR1
  hf::Consts<float> K;
};

struct alignas(128) Smem {
  float box[2][4 * PLANE];  // two boxes: planes rho, v0, v1, p (128-byte aligned)
  union {
    float c[BH * BW];     // sound speeds of the box cells (stage 1)
    float4 q[36 * QP];    // stage-1 state of the 36 x 36 cells (stage 2)
  } cq;
  union {
    struct {
      Flux x[36 * F1X];
      Flux y[37 * F1Y];
    } s1;
    struct {
      Flux x[32 * F2X];
      Flux y[33 * F2Y];
    } s2;
  } fl;
  uint64_t bar[2];
  uint64_t go;  // two groups per CTA: group 0 releases group 1 (in group 0's block)
  unsigned red[32];
  // of the items in box[0] and box[1]: the tile's origin and whether its box
  // lies inside the grid
  int4 pos[2];
  // the current item's instance and the next one's
  Inst inst[2];
};

// two CTAs per SM, or one CTA of two groups, within the SM's shared memory
// (227 KB per CTA at most)
static_assert(2 * sizeof(Smem) <= 232448, "two shared-memory blocks per SM");

// a warp copies an argument block into shared memory
__device__ __forceinline__ void copy_args(HydroStepArgs *dst, const HydroStepArgs *src,
                                          int lane) {
  static_assert(sizeof(HydroStepArgs) % 4 == 0, "argument block of whole words");
  const uint32_t *s = reinterpret_cast<const uint32_t *>(src);
  uint32_t *d = reinterpret_cast<uint32_t *>(dst);
  for (int i = lane; i < (int)(sizeof(HydroStepArgs) / 4); i += 32) d[i] = s[i];
}

// a warp fills an instance's block; args: its arguments in global memory (ENS)
// or among the kernel's parameters
template <bool ENS>
__device__ __forceinline__ void fill_inst(Inst &o, const HydroStepArgs &A, int first, int end,
                                          int lane) {
  if (ENS) copy_args(&o.a, &A, lane);
  const float dt = hk::step_dt<float>(A), dR0 = A.sc->dR0_f, dR1 = A.sc->dR1_f;
  const float half = dt / 2.0f;
  if (lane == 0) {
    o.first = first;
    o.end = end;
    o.dt = dt;
    o.dR0 = dR0;
    o.dR1 = dR1;
    o.h0 = half / dR0;
    o.h1 = half / dR1;
    o.f0 = dt / dR0;
    o.f1 = dt / dR1;
    o.K = hf::consts<float>(A.gamma_f);
  }
}

// a box lies inside the grid (no periodic image needed)
__device__ __forceinline__ bool box_inside(int X0, int Y0, int n0, int n1) {
  return X0 >= 4 && Y0 >= 3 && X0 + 36 <= n0 && Y0 + 35 <= n1;
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// Start the copy of a tile's box into `dst`.  Inside the grid: thread 0
// posts the byte count on *bar and issues the four TMA boxes (maps[k]
// describes field k of this grid).  Else every thread copies 16-byte
// chunks with wrapped coordinates (rows are multiples of 4 cells, so a
// wrapped chunk stays 16-byte aligned and whole).
// The four fields of a grid: their tensor maps (m, for boxes inside the
// grid) and base pointers (f).
struct FieldRefs {
  const CUtensorMap *m0, *m1, *m2, *m3;
  const float *f0, *f1, *f2, *f3;
};

template <int NTH = NT>
__device__ __forceinline__ void issue_box(float *dst, bool inside, const FieldRefs &r, int n0,
                                          int n1, int X0, int Y0, uint64_t *bar, int tid) {
  if (inside) {
    if (tid == 0) {
      tma::fence_proxy_async();
      tma::mbar_arrive_expect_tx(bar, kBoxBytes);
      tma::load_2d(dst, r.m0, X0 - 4, Y0 - 3, bar);
      tma::load_2d(dst + PLANE, r.m1, X0 - 4, Y0 - 3, bar);
      tma::load_2d(dst + 2 * PLANE, r.m2, X0 - 4, Y0 - 3, bar);
      tma::load_2d(dst + 3 * PLANE, r.m3, X0 - 4, Y0 - 3, bar);
    }
  } else {
    for (int i = tid; i < BH * 10; i += NTH) {
      const int py = i / 10, j = i - py * 10;
      const int gy = hk::wrap_near(Y0 - 3 + py, n1), gx = hk::wrap_near(X0 - 4 + 4 * j, n0);
      const size_t gi = (size_t)gy * n0 + gx;
      float *d = dst + py * BW + 4 * j;
      cp_async16(d, r.f0 + gi);
      cp_async16(d + PLANE, r.f1 + gi);
      cp_async16(d + 2 * PLANE, r.f2 + gi);
      cp_async16(d + 3 * PLANE, r.f3 + gi);
    }
    hk::cp_async_commit();
  }
}

__device__ __forceinline__ Prim box_cell(const float *B, int c) {
  return Prim{B[c], B[PLANE + c], B[2 * PLANE + c], B[3 * PLANE + c]};
}

__device__ __forceinline__ Prim rec(const float4 v) { return Prim{v.x, v.y, v.z, v.w}; }

// Three stage-2 walls along axis AX: wall j lies between records
// q[base + (j+1) st] and q[base + (j+2) st] and reconstructs from
// q[base + j st .. base + (j+3) st] (hf::muscl); its flux goes to
// out[j * ost].  The slope of the record right of wall j serves the left
// state of wall j+1.
template <int AX>
__device__ __forceinline__ void wall_run(const float4 *q, int base, int st, Flux *out, int ost,
                                         const hf::Consts<float> &K) {
  Prim L;
  {
    const Prim x0 = rec(q[base]), x1 = rec(q[base + st]), x2 = rec(q[base + 2 * st]);
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const float a = (&x0.rho)[f], b = (&x1.rho)[f], c = (&x2.rho)[f];
      (&L.rho)[f] = hf::fma(hf::minmod(hf::sub(b, a), hf::sub(c, b)), 0.5f, b);
    }
  }
  float cl = hf::sound(K, L.rho, L.p);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const Prim x1 = rec(q[base + (j + 1) * st]), x2 = rec(q[base + (j + 2) * st]),
               x3 = rec(q[base + (j + 3) * st]);
    Prim R, Ln;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const float b = (&x1.rho)[f], c = (&x2.rho)[f], d = (&x3.rho)[f];
      const float s = hf::minmod(hf::sub(c, b), hf::sub(d, c));
      (&R.rho)[f] = hf::fma(s, -0.5f, c);
      (&Ln.rho)[f] = hf::fma(s, 0.5f, c);
    }
    const float cr = hf::sound(K, R.rho, R.p);
    out[j * ost] = hf::hllc<AX>(K, L, cl, R, cr);
    if (j < 2) {
      L = Ln;
      cl = hf::sound(K, L.rho, L.p);
    }
  }
}

// ---------------------------------------------------------------------------
// item maps shared by both forms
// ---------------------------------------------------------------------------

// stage-1 wall item i: axis, box index of the cell left of (below) the wall,
// and the wall's index in s1.x (axis 0) or s1.y (axis 1).  The wall joins
// box cells c and c + 1 (x) or c and c + BW (y).
__device__ __forceinline__ void s1_item(int i, int &ax, int &c, int &w) {
  int fy, fx;
  if (i < kS1XMain) {
    ax = 0; fy = i >> 5; fx = i & 31;
  } else if (i < kS1XMain + kS1YMain) {
    const int j = i - kS1XMain;
    ax = 1; fy = j >> 5; fx = j & 31;
  } else if (i < kS1XMain + kS1YMain + kS1XRem) {
    const int j = i - (kS1XMain + kS1YMain);
    ax = 0; fy = j / 5; fx = 32 + (j - fy * 5);
  } else {
    const int j = i - (kS1XMain + kS1YMain + kS1XRem);
    ax = 1; fy = j >> 2; fx = 32 + (j & 3);
  }
  // x wall fx of row fy: box cells (fy+1, fx+1), (fy+1, fx+2); y wall fx
  // of row fy: (fy, fx+2), (fy+1, fx+2)
  c = ax == 0 ? (fy + 1) * BW + fx + 1 : fy * BW + fx + 2;
  w = ax == 0 ? fy * F1X + fx : fy * F1Y + fx;
}

// stage-1 wall pair i of the paired form: the x wall left of a cell and the y
// wall below it, for the 37 x 37 cells that are right of or above a wall (rows
// of 32, then the remainder).  The pair's axes are known where the code is
// compiled and it reads three cells; the x walls of the last row and the y walls
// of the last column are no walls of the tile (their cells lie in the box): not
// stored.  (Wall i with the wall 1344 items on, of whatever axis, chose between
// the velocities of each state and flux: 4096^2 took 485 us a step, 438 so, and
// 434 with the common cell and the wall between two paired cells read once; the
// ensembles below 2.86 ms, 2.75.)
__device__ __forceinline__ void s1_pair(int i, int &fy, int &fx) {
  fy = i >> 5;
  fx = i & 31;
  if (i >= kS1PairMain) {
    const int j = i - kS1PairMain;
    fy = j / 5;
    fx = 32 + (j - fy * 5);
  }
}

// stage-1 cell item i: (qy, qx) of the 36 x 36 cells
__device__ __forceinline__ void q_item(int i, int &qy, int &qx) {
  if (i < kQMain) {
    qy = i >> 5; qx = i & 31;
  } else {
    const int j = i - kQMain;
    qy = j >> 2; qx = 32 + (j & 3);
  }
}

// stage-1 cell pair i: cells (qy, qx) and (qy + 1, qx), qy even
__device__ __forceinline__ void q_pair(int i, int &qy, int &qx) {
  if (i < kQPairMain) {
    qy = i >> 5 << 1; qx = i & 31;
  } else {
    const int j = i - kQPairMain;
    qy = j >> 2 << 1; qx = 32 + (j & 3);
  }
}

// ---------------------------------------------------------------------------
// the paired form's helpers
// ---------------------------------------------------------------------------
using hf::f2;

__device__ __forceinline__ hf::NF<f2> pack_flux(const Flux &a, const Flux &b) {
  return hf::NF<f2>{hf::pack(a.fd, b.fd), hf::pack(a.fm0, b.fm0), hf::pack(a.fm1, b.fm1),
                    hf::pack(a.fe, b.fe)};
}

// the fluxes of an x wall and a y wall, back in axis order
__device__ __forceinline__ void split_pair(const hf::NF<f2> &f, Flux &x, Flux &y) {
  float d0, d1, n0, n1, t0, t1, e0, e1;
  hf::unpack(f.fd, d0, d1);
  hf::unpack(f.fn, n0, n1);
  hf::unpack(f.ft, t0, t1);
  hf::unpack(f.fe, e0, e1);
  x = Flux{d0, n0, t0, e0};
  y = Flux{d1, t1, n1, e1};
}

// box cell cx beside an x wall and box cell cy beside a y wall, in the frames
// of their walls
__device__ __forceinline__ hf::NS<f2> pair_state(const float *B, int cx, int cy) {
  return hf::NS<f2>{hf::pack(B[cx], B[cy]), hf::pack(B[PLANE + cx], B[2 * PLANE + cy]),
                    hf::pack(B[2 * PLANE + cx], B[PLANE + cy]),
                    hf::pack(B[3 * PLANE + cx], B[3 * PLANE + cy])};
}

// record k of the x run (row) and of the y run (column), in their walls'
// frames: (rho, un, ut, p)
__device__ __forceinline__ hf::NS<f2> run_rec(const float4 *q, int xa, int ya) {
  const float4 a = q[xa], b = q[ya];
  return hf::NS<f2>{hf::pack(a.x, b.x), hf::pack(a.y, b.z), hf::pack(a.z, b.y),
                    hf::pack(a.w, b.w)};
}

// The x-wall run of row `lane` (walls 3t..3t+2, records xb + 0..5) and the
// y-wall run of column `lane` (walls 3t..3t+2, records yb + 0..5 QP) side
// by side, as wall_run does for one run.
__device__ __forceinline__ void wall_run2(const float4 *q, int xb, int yb, Flux *xo, Flux *yo,
                                          const hf::K<f2> &k) {
  hf::NS<f2> L;
  {
    const hf::NS<f2> x0 = run_rec(q, xb, yb), x1 = run_rec(q, xb + 1, yb + QP),
                     x2 = run_rec(q, xb + 2, yb + 2 * QP);
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const f2 a = (&x0.rho)[f], b = (&x1.rho)[f], c = (&x2.rho)[f];
      (&L.rho)[f] = hf::fma(hf::minmod(hf::sub(b, a), hf::sub(c, b)), k.half, b);
    }
  }
  f2 cl = hf::sound(k, L.rho, L.p);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const hf::NS<f2> x1 = run_rec(q, xb + j + 1, yb + (j + 1) * QP),
                     x2 = run_rec(q, xb + j + 2, yb + (j + 2) * QP),
                     x3 = run_rec(q, xb + j + 3, yb + (j + 3) * QP);
    hf::NS<f2> R, Ln;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const f2 b = (&x1.rho)[f], c = (&x2.rho)[f], d = (&x3.rho)[f];
      const f2 sl = hf::minmod(hf::sub(c, b), hf::sub(d, c));
      (&R.rho)[f] = hf::fma(sl, k.neghalf, c);
      (&Ln.rho)[f] = hf::fma(sl, k.half, c);
    }
    const f2 cr = hf::sound(k, R.rho, R.p);
    split_pair(hf::hllc_ns<f2>(k, L, cl, R, cr), xo[j], yo[j * F2Y]);
    if (j < 2) {
      L = Ln;
      cl = hf::sound(k, L.rho, L.p);
    }
  }
}

// ---------------------------------------------------------------------------
// the tile loop
// ---------------------------------------------------------------------------

// The tiles of one grid (ENS false: args[0], maps m[0..3]) or of an
// ensemble (ENS true: instance k has args[k], maps table[(k * 4) + field]
// and items pf[k] .. pf[k+1]-1).  TAPE: the taped step (single grid).
// PAIR: the paired form (NT2 threads), else one wall or cell per thread
// (NT threads).
// GROUPS 2: the CTA holds two independent groups of NTH threads, each with
// its own shared-memory block (sm[0], sm[1]) and named barrier, working on
// alternate items; group 1 starts once group 0 has passed the second phase
// of its first tile, so the two groups' phases run about half a tile apart
// and one group's barrier tails overlap the other's arithmetic.
// GEN: sides of any size from 64 cells whose rows are whole 16-byte chunks
// (partial tiles); else sides are multiples of 32.
template <bool TAPE, bool ENS, bool PAIR, int GROUPS = 1, bool GEN = false>
__device__ __forceinline__ void persist_run(const HydroStepArgs *__restrict__ args,
                                            const int *__restrict__ pf, int count,
                                            const CUtensorMap *table, const CUtensorMap *m0,
                                            const CUtensorMap *m1, const CUtensorMap *m2,
                                            const CUtensorMap *m3, Smem *sm,
                                            const HydroTapeOut *tape) {
  constexpr int NTH = PAIR ? NT2 : NT;
  const int grp = GROUPS == 2 ? (int)threadIdx.x / NTH : 0;
  Smem &s = sm[grp];
  const int tid = (int)threadIdx.x - grp * NTH, lane = tid & 31, warp = tid >> 5;
  auto sync = [&]() {
    if (GROUPS == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(NTH) : "memory");
  };
  // block-wide (group-wide) min of CFL bit patterns folded into *dst
  auto min_to = [&](unsigned v, unsigned long long *dst) {
    v = __reduce_min_sync(0xffffffffu, v);
    if (lane == 0) s.red[warp] = v;
    sync();
    if (warp == 0) {
      v = __reduce_min_sync(0xffffffffu, lane < NTH / 32 ? s.red[lane] : ~0u);
      if (lane == 0) atomicMin(dst, (unsigned long long)v);
    }
  };
  const int total =
      ENS ? pf[count] : args[0].nt0 * ((args[0].n1 + TY - 1) / TY);
  int item = (int)blockIdx.x * GROUPS + grp;
  const int stride = (int)gridDim.x * GROUPS;
  if (tid == 0) {
    tma::mbar_init(&s.bar[0], 1);
    tma::mbar_init(&s.bar[1], 1);
    if (GROUPS == 2 && grp == 0) tma::mbar_init(&s.go, 1);
    tma::fence_mbar_init();
  }
  __syncthreads();
  bool released = GROUPS == 1 || grp == 1;
  if (item >= total) {
    if (!released && tid == 0) tma::mbar_arrive(&sm[0].go);
    return;
  }
  if (GROUPS == 2 && grp == 1) tma::mbar_wait(&sm[0].go, 0, &args[0].sc->wait_error);

  // start the copy of item `it` of instance k (items from `first` on,
  // arguments A) into box bb, and leave its place in s.pos[bb]
  auto issue = [&](int it, int k, int first, const HydroStepArgs &A, int bb) {
    const int tile = it - first, n0 = A.n0, n1 = A.n1;
    const int t1 = tile / A.nt0, X0 = (tile - t1 * A.nt0) * TX, Y0 = t1 * TY;
    const bool inside = box_inside(X0, Y0, n0, n1);
    if (tid == 0) s.pos[bb] = make_int4(X0, Y0, inside, 0);
    const CUtensorMap *tk = ENS ? table + (size_t)k * 4 : nullptr;
    const FieldRefs r{ENS ? tk : m0,
                      ENS ? tk + 1 : m1,
                      ENS ? tk + 2 : m2,
                      ENS ? tk + 3 : m3,
                      (const float *)A.rho,
                      (const float *)A.v0,
                      (const float *)A.v1,
                      (const float *)A.p};
    issue_box<NTH>(s.box[bb], inside, r, n0, n1, X0, Y0, &s.bar[bb], tid);
  };

  // sound speeds of the box cells into s.cq.c: items [i0, BH*BW/ (PAIR ? 2 : 1))
  // taken by threads t0.. with stride st
  auto sounds = [&](const float *Bx, const hf::Consts<float> &Kx, int first, int stride) {
    if (PAIR) {
      const hf::K<f2> k2 = hf::kconsts<f2>(Kx);
      for (int i = first; i < BH * BW / 2; i += stride) {
        const int j = i + BH * BW / 2;
        const f2 c = hf::sound(k2, hf::pack(Bx[i], Bx[j]),
                               hf::pack(Bx[3 * PLANE + i], Bx[3 * PLANE + j]));
        hf::unpack(c, s.cq.c[i], s.cq.c[j]);
      }
    } else {
      for (int i = first; i < BH * BW; i += stride)
        s.cq.c[i] = hf::sound(Kx, Bx[i], Bx[3 * PLANE + i]);
    }
  };
  // wait until the box of the item in s.pos[bb] has landed (the caller
  // synchronises the block before, so that s.pos holds, and afterwards)
  uint32_t parity = 0;  // bit k: parity of the next completed phase of bar[k]
  auto await_box = [&](int bb, const HydroStepArgs &A) {
    if (s.pos[bb].z) {
      tma::mbar_wait(&s.bar[bb], (parity >> bb) & 1u, &A.sc->wait_error);
      parity ^= 1u << bb;
    } else {
      hk::cp_async_wait_all();
    }
  };

  int lo = 0;  // instance of `item`
  int ai = 0;  // its slot in s.inst
  {
    if (ENS)
      while (lo < count - 1 && pf[lo + 1] <= item) ++lo;
    const int first = ENS ? pf[lo] : 0, end = ENS ? pf[lo + 1] : total;
    issue(item, lo, first, args[lo], 0);
    if (warp == 0) fill_inst<ENS>(s.inst[0], args[lo], first, end, lane);
    sync();
    await_box(0, args[lo]);
    sync();
    sounds(s.box[0], s.inst[0].K, tid, NTH);
  }
  sync();
  int b = 0;
  unsigned m = ~0u;

  for (;;) {
    Inst &I = s.inst[ai];
    const HydroStepArgs &A = ENS ? I.a : args[0];
    const int n0 = A.n0;
    const int X0 = s.pos[b].x, Y0 = s.pos[b].y;
    const float *B = s.box[b];

    // the next item's box goes into the other buffer while this one computes
    // (that buffer's last reader, the previous tile's stage 2, is behind the
    // last barrier, and so is the last reader of the other instance slot)
    const int next = item + stride;
    int lo_n = lo;
    if (next < total) {
      if (!ENS || next < I.end) {
        issue(next, lo, ENS ? I.first : 0, A, b ^ 1);
      } else {
        do ++lo_n;
        while (lo_n < count - 1 && pf[lo_n + 1] <= next);
        const int first = pf[lo_n];
        issue(next, lo_n, first, args[lo_n], b ^ 1);
        if (warp == NTH / 32 - 1)
          fill_inst<ENS>(s.inst[ai ^ 1], args[lo_n], first, pf[lo_n + 1], lane);
      }
    }
    const int an = lo_n == lo ? ai : ai ^ 1;  // the next item's instance

    // stage-1 walls, order-1 reconstruction
    if (PAIR) {
      const hf::K<f2> k2 = hf::kconsts<f2>(I.K);
      for (int i = tid; i < kS1Pairs; i += NTH) {
        int fy, fx;
        s1_pair(i, fy, fx);
        const int c = (fy + 1) * BW + fx + 2;
        // the cell left of, the one below, and the one right of and above
        const hf::NS<f2> L = pair_state(B, c - 1, c - BW), R = pair_state(B, c, c);
        const f2 cl = hf::pack(s.cq.c[c - 1], s.cq.c[c - BW]);
        const f2 cr = hf::pack(s.cq.c[c], s.cq.c[c]);
        Flux x, y;
        split_pair(hf::hllc_ns<f2>(k2, L, cl, R, cr), x, y);
        if (fy < 36) s.fl.s1.x[fy * F1X + fx] = x;
        if (fx < 36) s.fl.s1.y[fy * F1Y + fx] = y;
      }
    } else {
      const hf::Consts<float> K = I.K;
      for (int i = tid; i < kS1Items; i += NTH) {
        int ax, c, w;
        s1_item(i, ax, c, w);
        if (ax == 0)
          s.fl.s1.x[w] =
              hf::hllc<0>(K, box_cell(B, c), s.cq.c[c], box_cell(B, c + 1), s.cq.c[c + 1]);
        else
          s.fl.s1.y[w] =
              hf::hllc<1>(K, box_cell(B, c), s.cq.c[c], box_cell(B, c + BW), s.cq.c[c + BW]);
      }
    }
    sync();

    // stage-1 cells (qy, qx) = box cell (qy+1, qx+2), advanced by dt/2
    {
      const float dtdx0 = I.h0, dtdx1 = I.h1;
      auto tape_cell = [&](int qy, int qx, const float *q, const Flux &l0, const Flux &r0,
                           const Flux &l1, const Flux &r1) {
        const int ty = qy - 2, tx = qx - 2;
        if (ty >= 0 && ty < TY && tx >= 0 && tx < TX) {
          const size_t gi = (size_t)(Y0 + ty) * n0 + (X0 + tx);
#pragma unroll
          for (int f = 0; f < 4; ++f) ((float *)tape->q[f])[gi] = q[f];
          hk::tape_diffs<float>(tape->d1, gi, l0, r0, l1, r1);
        }
      };
      if (PAIR) {
        const hf::K<f2> k2 = hf::kconsts<f2>(I.K);
        const f2 t0 = hf::splat<f2>(dtdx0), t1 = hf::splat<f2>(dtdx1);
        for (int i = tid; i < kQPairs; i += NTH) {
          int qy, qx;
          q_pair(i, qy, qx);
          const int ca = (qy + 1) * BW + qx + 2, cb = ca + BW;
          const Flux &l0a = s.fl.s1.x[qy * F1X + qx], &r0a = s.fl.s1.x[qy * F1X + qx + 1];
          const Flux &l0b = s.fl.s1.x[(qy + 1) * F1X + qx],
                     &r0b = s.fl.s1.x[(qy + 1) * F1X + qx + 1];
          // the wall between the two cells is read once
          const Flux &l1a = s.fl.s1.y[qy * F1Y + qx], &r1b = s.fl.s1.y[(qy + 2) * F1Y + qx];
          const Flux mid = s.fl.s1.y[(qy + 1) * F1Y + qx];
          f2 q[4];
          hf::update_t<f2>(k2, hf::pack(B[ca], B[cb]), hf::pack(B[PLANE + ca], B[PLANE + cb]),
                           hf::pack(B[2 * PLANE + ca], B[2 * PLANE + cb]),
                           hf::pack(B[3 * PLANE + ca], B[3 * PLANE + cb]), t0, t1,
                           pack_flux(l0a, l0b), pack_flux(r0a, r0b), pack_flux(l1a, mid),
                           pack_flux(mid, r1b), q);
          float qa[4], qb[4];
#pragma unroll
          for (int f = 0; f < 4; ++f) hf::unpack(q[f], qa[f], qb[f]);
          if (TAPE) {
            tape_cell(qy, qx, qa, l0a, r0a, l1a, mid);
            tape_cell(qy + 1, qx, qb, l0b, r0b, mid, r1b);
          }
          s.cq.q[qy * QP + qx] = make_float4(qa[0], qa[1], qa[2], qa[3]);
          s.cq.q[(qy + 1) * QP + qx] = make_float4(qb[0], qb[1], qb[2], qb[3]);
        }
      } else {
        const hf::Consts<float> K = I.K;
        for (int i = tid; i < kQItems; i += NTH) {
          int qy, qx;
          q_item(i, qy, qx);
          const int c = (qy + 1) * BW + qx + 2;
          const Flux &l0 = s.fl.s1.x[qy * F1X + qx], &r0 = s.fl.s1.x[qy * F1X + qx + 1];
          const Flux &l1 = s.fl.s1.y[qy * F1Y + qx], &r1 = s.fl.s1.y[(qy + 1) * F1Y + qx];
          const Prim q = hf::update(K, box_cell(B, c), dtdx0, dtdx1, l0, r0, l1, r1);
          if (TAPE) {
            const float qv[4] = {q.rho, q.v0, q.v1, q.p};
            tape_cell(qy, qx, qv, l0, r0, l1, r1);
          }
          s.cq.q[qy * QP + qx] = make_float4(q.rho, q.v0, q.v1, q.p);
        }
      }
    }
    sync();
    if (!released) {  // group 0, first tile: let group 1 start
      if (tid == 0) tma::mbar_arrive(&sm[0].go);
      released = true;
    }

    // stage-2 walls, MUSCL-minmod of the stage-1 state: the x walls
    // 3t..3t+2 of row `lane` and the y walls 3t..3t+2 of column `lane`
    if (PAIR) {
      wall_run2(s.cq.q, (lane + 2) * QP + 3 * warp, 3 * warp * QP + lane + 2,
                &s.fl.s2.x[lane * F2X + 3 * warp], &s.fl.s2.y[3 * warp * F2Y + lane],
                hf::kconsts<f2>(I.K));
    } else if (warp < 11) {
      wall_run<0>(s.cq.q, (lane + 2) * QP + 3 * warp, 1, &s.fl.s2.x[lane * F2X + 3 * warp], 1, I.K);
    } else {
      const int t = warp - 11;
      wall_run<1>(s.cq.q, 3 * t * QP + lane + 2, QP, &s.fl.s2.y[3 * t * F2Y + lane], F2Y, I.K);
    }
    // the next box must have landed before its sound speeds are formed
    if (next < total) await_box(b ^ 1, ENS ? s.inst[an].a : args[0]);
    sync();

    // stage-2 cells (oy, ox) = box cell (oy+3, ox+4), advanced by dt and
    // written out, with the CFL minimum of the new state; the threads with
    // one stage-2 item form the next box's sound speeds (the stage-1 state
    // they overwrite was last read before the barrier above)
    {
      constexpr int P4 = PAIR ? TX * TY / 2 : TX * TY;  // stage-2 items
      constexpr int ONE = P4 - NTH;  // threads from here on take one item
      const float dtdx0 = I.f0, dtdx1 = I.f1, g = I.K.g, dR0 = I.dR0, dR1 = I.dR1;
      float *out[4] = {(float *)A.nrho, (float *)A.nv0, (float *)A.nv1, (float *)A.np};
      auto put = [&](int oy, int ox, const float *q, const float *cons, const Flux &l0,
                     const Flux &r0, const Flux &l1, const Flux &r1) {
        if (GEN && (X0 + ox >= n0 || Y0 + oy >= A.n1)) return;
        const size_t gi = (size_t)(Y0 + oy) * n0 + (X0 + ox);
        if (TAPE) {
          hk::tape_diffs<float>(tape->d2, gi, l0, r0, l1, r1);
#pragma unroll
          for (int k = 0; k < 4; ++k) ((float *)tape->u2[k])[gi] = cons[k];
        }
#pragma unroll
        for (int f = 0; f < 4; ++f) out[f][gi] = q[f];
        const float t = hs::timescale(g, dR0, dR1, q[0], q[1], q[2], q[3]);
        m = min(m, __float_as_uint(t));
      };
      if (PAIR) {
        const hf::K<f2> k2 = hf::kconsts<f2>(I.K);
        const f2 t0 = hf::splat<f2>(dtdx0), t1 = hf::splat<f2>(dtdx1);
        for (int i = tid; i < P4; i += NTH) {
          const int oy = i >> 5 << 1, ox = i & 31;
          const int ca = (oy + 3) * BW + ox + 4, cb = ca + BW;
          const Flux &l0a = s.fl.s2.x[oy * F2X + ox], &r0a = s.fl.s2.x[oy * F2X + ox + 1];
          const Flux &l0b = s.fl.s2.x[(oy + 1) * F2X + ox],
                     &r0b = s.fl.s2.x[(oy + 1) * F2X + ox + 1];
          const Flux &l1a = s.fl.s2.y[oy * F2Y + ox], &r1b = s.fl.s2.y[(oy + 2) * F2Y + ox];
          const Flux mid = s.fl.s2.y[(oy + 1) * F2Y + ox];
          f2 q[4], cons[4];
          hf::update_t<f2>(k2, hf::pack(B[ca], B[cb]), hf::pack(B[PLANE + ca], B[PLANE + cb]),
                           hf::pack(B[2 * PLANE + ca], B[2 * PLANE + cb]),
                           hf::pack(B[3 * PLANE + ca], B[3 * PLANE + cb]), t0, t1,
                           pack_flux(l0a, l0b), pack_flux(r0a, r0b), pack_flux(l1a, mid),
                           pack_flux(mid, r1b), q, TAPE ? cons : nullptr);
          float qa[4], qb[4], ca4[4], cb4[4];
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            hf::unpack(q[f], qa[f], qb[f]);
            if (TAPE) hf::unpack(cons[f], ca4[f], cb4[f]);
          }
          put(oy, ox, qa, ca4, l0a, r0a, l1a, mid);
          put(oy + 1, ox, qb, cb4, l0b, r0b, mid, r1b);
        }
      } else {
        const hf::Consts<float> K = I.K;
        for (int i = tid; i < P4; i += NTH) {
          const int oy = i >> 5, ox = i & 31;
          const int c = (oy + 3) * BW + ox + 4;
          const Flux &l0 = s.fl.s2.x[oy * F2X + ox], &r0 = s.fl.s2.x[oy * F2X + ox + 1];
          const Flux &l1 = s.fl.s2.y[oy * F2Y + ox], &r1 = s.fl.s2.y[(oy + 1) * F2Y + ox];
          float cons[4];
          const Prim q =
              hf::update(K, box_cell(B, c), dtdx0, dtdx1, l0, r0, l1, r1, TAPE ? cons : nullptr);
          const float qv[4] = {q.rho, q.v0, q.v1, q.p};
          put(oy, ox, qv, cons, l0, r0, l1, r1);
        }
      }
      if (next < total && tid >= ONE)
        sounds(s.box[b ^ 1], s.inst[an].K, tid - ONE, NTH - ONE);
    }
    if (X0 == 0 && Y0 == 0 && tid == 0) {
      const float dtG = I.dt;
      if (A.ts_clear) *ts_at(A, A.ts_clear) = ~0ull;
      A.dt_hist[0] = (double)dtG;
      A.sc->dt_last = (double)dtG;
      A.sc->time = A.sc->time + (double)dtG;
    }
    // publish the CFL minimum when this CTA leaves the instance (the
    // reduction ends with a barrier); else one barrier before the next tile
    if (next >= total || lo_n != lo) {
      min_to(m, ts_at(A, A.ts_write));
      m = ~0u;
    } else {
      sync();
    }
    if (next >= total) break;
    item = next;
    lo = lo_n;
    ai = an;
    b ^= 1;
  }
}

template <bool TAPE>
__global__ void __launch_bounds__(NT, 2)
hydro_persist_kernel(HydroStepArgs a, const __grid_constant__ CUtensorMap m0,
                     const __grid_constant__ CUtensorMap m1,
                     const __grid_constant__ CUtensorMap m2,
                     const __grid_constant__ CUtensorMap m3, HydroTapeOut tape) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  hk::step_begin();
  persist_run<TAPE, false, false>(&a, nullptr, 1, nullptr, &m0, &m1, &m2, &m3,
                                  reinterpret_cast<Smem *>(smem_raw), &tape);
}

template <bool TAPE, bool GEN>
__global__ void __launch_bounds__(NT2, 2)
hydro_pair_kernel(HydroStepArgs a, const __grid_constant__ CUtensorMap m0,
                  const __grid_constant__ CUtensorMap m1, const __grid_constant__ CUtensorMap m2,
                  const __grid_constant__ CUtensorMap m3, HydroTapeOut tape) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  hk::step_begin();
  persist_run<TAPE, false, true, 1, GEN>(&a, nullptr, 1, nullptr, &m0, &m1, &m2, &m3,
                                         reinterpret_cast<Smem *>(smem_raw), &tape);
}

// the paired form as one CTA per SM of two groups half a tile apart (two
// shared-memory blocks); 80 registers keep the 22 warps within the SM
// sub-partitions' register files
template <bool TAPE, bool GEN>
__global__ void __maxnreg__(80)
hydro_pair2_kernel(HydroStepArgs a, const __grid_constant__ CUtensorMap m0,
                   const __grid_constant__ CUtensorMap m1, const __grid_constant__ CUtensorMap m2,
                   const __grid_constant__ CUtensorMap m3, HydroTapeOut tape) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  hk::step_begin();
  persist_run<TAPE, false, true, 2, GEN>(&a, nullptr, 1, nullptr, &m0, &m1, &m2, &m3,
                                         reinterpret_cast<Smem *>(smem_raw), &tape);
}

// the paired ensemble step as one CTA per SM of two groups half an item apart
template <bool GEN>
__global__ void __maxnreg__(80)
hydro_pair2_ensemble_kernel(const HydroStepArgs *__restrict__ args,
                            const int *__restrict__ prefix, int count,
                            const CUtensorMap *__restrict__ table) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  persist_run<false, true, true, 2, GEN>(args, prefix, count, table, nullptr, nullptr, nullptr,
                                         nullptr, reinterpret_cast<Smem *>(smem_raw), nullptr);
}

// table: 4 tensor maps per instance for the buffers `args` reads
template <bool PAIR, bool GEN>
__global__ void __launch_bounds__(PAIR ? NT2 : NT, 2)
hydro_persist_ensemble_kernel(const HydroStepArgs *__restrict__ args,
                              const int *__restrict__ prefix, int count,
                              const CUtensorMap *__restrict__ table) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  persist_run<false, true, PAIR, 1, GEN>(args, prefix, count, table, nullptr, nullptr, nullptr,
                                         nullptr, reinterpret_cast<Smem *>(smem_raw), nullptr);
}

}  // namespace hp
}  // namespace om

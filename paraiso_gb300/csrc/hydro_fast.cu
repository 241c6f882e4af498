// hydro_fast.cu -- the production FP32 build of the fused Hydro step:
// the tile code of the exact build (hydro_kernels.cuh) with the production
// algebra (hf:: in hydro_scheme.cuh), compiled with multiply-add
// contraction and fast single-precision division and square root, in the
// tile shapes the tuner chooses from.
#include <cuda_runtime.h>

#include "hydro_launch.cuh"
#include "hydro_sweep.cuh"
#include "om_internal.cuh"

namespace om {

cudaError_t hydro_fused_f32_exact(const HydroStepArgs &a, cudaStream_t s, int *grid_out);

template <int TX, int TY, int NT, bool OPEN = false>
static cudaError_t launch_fast(const HydroStepArgs &a0, cudaStream_t s, int *grid_out) {
  HydroStepArgs a = a0;
  a.nt0 = (a.n0 + TX - 1) / TX;
  const int nt1 = (a.n1 + TY - 1) / TY;
  const size_t smem = sizeof(FusedSmem<float, TX, TY>);
  cudaError_t e = cudaFuncSetAttribute(hydro_fused_kernel<float, TX, TY, NT, OPEN, true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if (grid_out) *grid_out = a.nt0 * nt1;
  return launch_step(hydro_fused_kernel<float, TX, TY, NT, OPEN, true>, a.nt0 * nt1, NT, smem, s,
                     a);
}

// The production sweep over a periodic grid: strips of TX columns, segments
// sized to fill the resident blocks about once.  With `tape`, the taped step.
template <int TX, int TY, int NT, bool TAPE>
static cudaError_t launch_sweep(const HydroStepArgs &a0, const HydroTapeOut *tape,
                                cudaStream_t s, int *grid_out) {
  using K = void (*)(HydroStepArgs, SweepGeom, const HydroTapeOut);
  K k = hydro_sweep_kernel<float, TX, TY, NT, TAPE, true>;
  const size_t smem = sizeof(SweepSmem<float, TX, TY>);
  static int resident_per_sm = 0;  // the same on every device of one kind
  if (!resident_per_sm) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, NT, smem);
    if (e != cudaSuccess) return e;
    resident_per_sm = n > 0 ? n : 1;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  HydroStepArgs a = a0;
  a.nt0 = 0;
  const SweepGeom geo = sweep_geometry(a.n0, a.n1, TX, TY, resident_per_sm * sm_count(dev));
  HydroTapeOut t{};
  if (tape) t = *tape;
  const int grid = geo.strips * geo.segs;
  k<<<grid, NT, smem, s>>>(a, geo, t);
  if (grid_out) *grid_out = grid;
  return cudaGetLastError();
}

cudaError_t hydro_ensemble_f32_exact(const HydroStepArgs *args, const int *prefix, int count,
                                     int grid, cudaStream_t s);
int hydro_ensemble_occupancy_exact(int fp64);

template <int TX, int TY, int NT>
static cudaError_t launch_ens(const HydroStepArgs *args, const int *prefix, int count, int grid,
                              cudaStream_t s) {
  const size_t smem = sizeof(FusedSmem<float, TX, TY>);
  cudaError_t e = cudaFuncSetAttribute(hydro_ensemble_kernel<float, TX, TY, NT, true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  hydro_ensemble_kernel<float, TX, TY, NT, true><<<grid, NT, smem, s>>>(args, prefix, count);
  return cudaGetLastError();
}

template <int TX, int TY, int NT> static int occ_fast() {
  const size_t smem = sizeof(FusedSmem<float, TX, TY>);
  cudaFuncSetAttribute(hydro_ensemble_kernel<float, TX, TY, NT, true>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, hydro_ensemble_kernel<float, TX, TY, NT, true>,
                                                    NT, smem) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = 1;
  }
  return n;
}

cudaError_t hydro_ensemble_f32(const HydroStepArgs *args, const int *prefix, int count, int tile,
                               bool exact, int grid, cudaStream_t s, const CUtensorMap *table,
                               bool general) {
  if (exact) return hydro_ensemble_f32_exact(args, prefix, count, grid, s);
  if (hydro_tile_is_persistent(tile) && table)
    return hydro_persist_ensemble(args, prefix, count, table, hydro_persist_form(tile), general,
                                  grid, s);
  switch (tile) {
    case kTile32x8: return launch_ens<32, 8, 256>(args, prefix, count, grid, s);
    case kTile64x16: return launch_ens<64, 16, 512>(args, prefix, count, grid, s);
    case kTile32x32: return launch_ens<32, 32, 512>(args, prefix, count, grid, s);
    case kTile64x8: return launch_ens<64, 8, 256>(args, prefix, count, grid, s);
    case kTile32x16: return launch_ens<32, 16, 256>(args, prefix, count, grid, s);
    default: return launch_ens<32, 32, 512>(args, prefix, count, grid, s);
  }
}

int hydro_ensemble_occupancy(int fp64, int tile, bool exact) {
  if (fp64 || exact) return hydro_ensemble_occupancy_exact(fp64);
  switch (tile) {
    case kPersist32x32:
    case kPair32x32:
    case kPairGroups32x32: return hydro_persist_occupancy(hydro_persist_form(tile));
    case kTile32x8: return occ_fast<32, 8, 256>();
    case kTile64x16: return occ_fast<64, 16, 512>();
    case kTile32x32: return occ_fast<32, 32, 512>();
    case kTile64x8: return occ_fast<64, 8, 256>();
    case kTile32x16: return occ_fast<32, 16, 256>();
    default: return occ_fast<32, 32, 512>();
  }
}

cudaError_t hydro_fused_tape_exact(int fp64, const HydroStepArgs &a, const HydroTapeOut &t,
                                   cudaStream_t s);

// the taped production step on TX x TY tiles
template <int TX, int TY, int NT>
static cudaError_t launch_tape_fast(const HydroStepArgs &a0, const HydroTapeOut &t,
                                   cudaStream_t s) {
  HydroStepArgs a = a0;
  a.nt0 = (a.n0 + TX - 1) / TX;
  const int nt1 = (a.n1 + TY - 1) / TY;
  const size_t smem = sizeof(FusedSmem<float, TX, TY>);
  cudaError_t e = cudaFuncSetAttribute(hydro_fused_tape_kernel<float, TX, TY, NT, true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  hydro_fused_tape_kernel<float, TX, TY, NT, true><<<a.nt0 * nt1, NT, smem, s>>>(a, t);
  return cudaGetLastError();
}

cudaError_t hydro_fused_tape(int fp64, bool exact, const HydroStepArgs &a0, const HydroTapeOut &t,
                             cudaStream_t s, int tile) {
  if (fp64 || exact) return hydro_fused_tape_exact(fp64, a0, t, s);
  // The forward pass may run another shape of the same algebra (hydro_step_tile,
  // partial persistent tiles): every production kernel rounds each operation of
  // the scheme explicitly, so the states of all shapes are the same bit for bit,
  // and a recomputed state equals the forward pass's.
  switch (tile) {
    case kPersist32x32:
    case kPair32x32:
    case kPairGroups32x32:
      if (hydro_persist_fits(a0.n0, a0.n1))
        return hydro_persist_tape(a0, hydro_persist_form(tile), t, s);
      return launch_tape_fast<32, 32, 512>(a0, t, s);
    case kTile32x8: return launch_tape_fast<32, 8, 256>(a0, t, s);
    case kTile64x16: return launch_tape_fast<64, 16, 512>(a0, t, s);
    case kTile32x16: return launch_tape_fast<32, 16, 256>(a0, t, s);
    case kTile64x8: return launch_tape_fast<64, 8, 256>(a0, t, s);
    case kSweep32x8: return launch_sweep<32, 8, 256, true>(a0, &t, s, nullptr);
    case kSweep32x16: return launch_sweep<32, 16, 512, true>(a0, &t, s, nullptr);
    case kSweep64x8: return launch_sweep<64, 8, 512, true>(a0, &t, s, nullptr);
    default: return launch_tape_fast<32, 32, 512>(a0, t, s);
  }
}

// A grid with at most a tile or two per SM is bound by the chain of a tile's
// five phases, not by throughput: more threads per cell shorten it.  Measured
// per step in a captured run of 50 (us; 32 x 32 or persistent tiles first):
//   64^2   8.5, 16 x 8 by 256 threads 4.3      100^2 8.3, 4.8
//   128^2  8.3, 16 x 8 5.65, 32 x 16 by 1024 5.56
//   256^2  11.4, 32 x 16 by 1024 5.56, by 512 11.6, 32 x 8 by 512 7.5
//   384 x 256 (192 tiles of 32 x 16 on 152 SMs)  12.0, by 512 8.9, by 544 7.8
//   450 x 300 (285)  by 512 10.0, by 544 7.8;  500 x 300 (304)  12.2, 7.7, 7.8
//   560 x 400 (450)  32 x 32 11.8, persistent 11.2, by 512 10.1, by 544 11.5
// (544 threads take the walls of stage 2 in two rounds, and two blocks fill an
// SM; of 512 three do, which evens out only when there are as many.)  Open
// grids: 384 x 256 by 512 10.3, by 544 8.4; 560 x 400 10.5, 12.4, and 12.9 by
// 288; larger ones by 288 threads, 701 x 500 15.8, 16.5 by 256, 3001 x 2500 243,
// 248.
//   600 x 400 (475: more than three to an SM)  12.0, 11.2, 13.1
//   700 x 500 (704)  17.4, 14.7, by 512 16.1;  900 x 500 (928)  21.2, 19.4
//   1000 x 700 (1408)  26.8, 25.6, 28.4;  1200 x 900  40.3, 36.4
//   1500 x 1100  55.5, 47.7;  3000 x 2500  245, 205
// Rows that are no multiples of 4 cells go cell by cell or in pairs into the
// persistent kernel's boxes, which costs what it gains: 1501 x 1100 55.9 with
// 32 x 32 tiles, 58.4; 2002 x 1500 100.2, 99.0; 3001 x 2500 246, 257.
// Large grids that are left to the tile kernels take 32 x 24 tiles by 416 threads,
// whose four phases are 5, 2.4, 3.8 and 1.8 rounds: 1501 x 1100 (11 tiles of
// 32 x 32 per SM) 55.4 against 55.6, 2001 x 1500 (19) 97.7 against 100.1, 3001 x
// 2500 237.8 against 246.6; open 1024^2 37.7 against 37.5 with 32 x 16, 2001 x 1500
// 98.5 against 99.3, 4000^2 498 against 509.
int hydro_step_tile(int tile, int n0, int n1, bool open, int device, int grid_limit) {
  if (grid_limit > 0 || !(open || tile == kPairGroups32x32)) return tile;
  const long long sms = sm_count(device);
  auto tiles = [&](int tx, int ty) { return (long long)((n0 + tx - 1) / tx) * ((n1 + ty - 1) / ty); };
  if (!open && tiles(16, 8) <= sms) return kThin16x8;
  if (tiles(32, 16) <= sms) return kThin32x16;
  if (tiles(32, 16) <= 2 * sms) return kThin32x16h;
  if (tiles(32, 16) <= 3 * sms) return kThin32x16t;
  if (!open && hydro_persist_any(n0, n1)) return tile;
  if (tiles(32, 32) > 16 * sms) return kLarge32x24;
  if (open) return tile;
  if (tiles(32, 32) <= 2 * sms) return kTile32x32;
  return tiles(32, 16) <= 6 * sms ? kThin32x16t : kTile32x32;
}

cudaError_t hydro_fused_f32(const HydroStepArgs &a, int tile, bool exact, cudaStream_t s,
                            int *grid_out) {
  if (exact) return hydro_fused_f32_exact(a, s, grid_out);
  // an open grid (margins, jet boundary condition) runs 32x16 tiles
  if (a.lm > 0) switch (tile) {
    case kThin32x16: return launch_fast<32, 16, 1024, true>(a, s, grid_out);
    case kThin32x16h: return launch_fast<32, 16, 544, true>(a, s, grid_out);
    case kThin32x16t: return launch_fast<32, 16, 512, true>(a, s, grid_out);
    case kLarge32x24: return launch_fast<32, 24, 416, true>(a, s, grid_out);
    default: return launch_fast<32, 16, 288, true>(a, s, grid_out);
  }
  switch (tile) {
    case kThin16x8: return launch_fast<16, 8, 256>(a, s, grid_out);
    case kThin32x16: return launch_fast<32, 16, 1024>(a, s, grid_out);
    case kThin32x16h: return launch_fast<32, 16, 544>(a, s, grid_out);
    case kThin32x16t: return launch_fast<32, 16, 512>(a, s, grid_out);
    case kLarge32x24: return launch_fast<32, 24, 416>(a, s, grid_out);
    case kPersist32x32:
    case kPair32x32:
    case kPairGroups32x32:
      if (hydro_persist_fits(a.n0, a.n1) ||
          (hydro_tile_takes_any(tile) && hydro_persist_any(a.n0, a.n1)))
        return hydro_persist_step(a, hydro_persist_form(tile), s, grid_out);
      return launch_fast<32, 32, 512>(a, s, grid_out);
    case kTile32x8: return launch_fast<32, 8, 256>(a, s, grid_out);
    case kTile64x16: return launch_fast<64, 16, 512>(a, s, grid_out);
    case kTile32x32: return launch_fast<32, 32, 512>(a, s, grid_out);
    case kTile64x8: return launch_fast<64, 8, 256>(a, s, grid_out);
    case kSweep32x8: return launch_sweep<32, 8, 256, false>(a, nullptr, s, grid_out);
    case kSweep32x16: return launch_sweep<32, 16, 512, false>(a, nullptr, s, grid_out);
    case kSweep64x8: return launch_sweep<64, 8, 512, false>(a, nullptr, s, grid_out);
    case kTile32x16: return launch_fast<32, 16, 256>(a, s, grid_out);
    default: return launch_fast<32, 32, 512>(a, s, grid_out);
  }
}

}  // namespace om

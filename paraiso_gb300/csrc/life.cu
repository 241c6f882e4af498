// life.cu -- Conway's Life Orthotope Machine on GB300.
//
// Reference: examples/Life/Generator.hs:67-115 (init, proceed), the
// generated loop examples-old/Life-exampled/dist/Life.cpp:114-183 and the
// CPU/GPU reduce library (Language/Paraiso/Generator/PlanTrans.hs:712-720).
//
//   proceed:  num   = sum of the 8 shifted copies of cell
//             alive = (cell==0 && num==3) || (cell==1 && num>=2 && num<=3)
//             cell' = alive ? 1 : 0
//             population = reduce Sum cell'      generation = generation + 1
//
// The device paths give bit-identical results:
//  * life_general_kernel: one int32 cell per thread with the reference's
//    integer arithmetic; any size, cyclic or open boundary, any cell values.
//  * life_smallreg_kernel: a small grid bit-packed in the registers of one CTA,
//    all generations of a run in one launch.  Cyclic, any width up to 1024.
//  * life_reg_kernel, life_ws_kernel, life_tb*_kernel: bit-packed tiles with a
//    1-word / k-row halo, k generations per launch (temporal blocking).
//  * long runs and rows that are no whole number of words keep the grid packed
//    between launches (proceed_packed).  Cyclic, any width above 32.
// The packed paths require every cell in {0,1}; then num is in [0,8] and
// the rule equals the bit-sliced adder below, so outputs are identical.
// After any external write the first generation runs on the general path,
// whose outputs are always 0/1.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <string>

#include "om_internal.cuh"
#include "tma.cuh"

namespace om {

struct LifeScalars {  // device/host scalar block
  int32_t population;
  int32_t generation;
  uint32_t wait_error;  // raised by a kernel whose bounded wait ran out
};

// Populations kept in pinned host memory beside the scalars.  A run's results
// are a few words that its last kernel writes there: copies around the run
// (scalars in, scalars out, history out) cost more than small runs compute.
static const int kHistory = 4096;

struct LifeState {
  bool binary = true;           // every cell is known to be 0 or 1
  // populations of a run, per generation.  pop_clear: the first kHistory of them
  // are 0, as runs of at most that many generations leave them, whose results
  // go to the host block; those after may hold an earlier, longer run's
  uint32_t *d_pop = nullptr;
  bool pop_clear = false;
  uint32_t *d_flag = nullptr;   // raised by the cell-value check; [1]: a wait ran out
  int pop_cap = 0;
  int last_n = 0;
  int depth = 0, tile_w = 0, tile_h = 0;  // tuned or configured
  uint32_t *packed[2] = {nullptr, nullptr};  // the packed grid between launches
  bool packed_refused = false;  // no memory for it: runs do without
  // tensor maps of the two cell buffers (cells x words x rows) for the TMA
  // kernels, keyed by buffer address, and their one-word maps (32 cells x 1
  // word x 1 row, no swizzle) for the halo word that wraps around;
  // tmap_ok[i] false when encoding failed
  CUtensorMap tmap[2], tpatch[2];
  const void *tmap_ptr[2] = {nullptr, nullptr};
  bool tmap_ok[2] = {false, false};
};

// Index of the cached maps of cell buffer `cells` (n0 x n1 int32, n0 a
// multiple of 32), -1 when the driver does not encode them: dimensions 32
// cells x n0/32 words x n1 rows, boxes of one row of 32 words with 128-byte
// swizzle (st->tmap[i]) and of one word (st->tpatch[i]).
static int life_tmap(LifeState *st, const void *cells, int n0, int n1) {
  for (int i = 0; i < 2; ++i)
    if (st->tmap_ptr[i] == cells) return st->tmap_ok[i] ? i : -1;
  const int i = st->tmap_ptr[0] == nullptr ? 0 : (st->tmap_ptr[1] == nullptr ? 1 : 0);
  const uint64_t dims[3] = {32, (uint64_t)(n0 / 32), (uint64_t)n1};
  const uint64_t strides[2] = {128, (uint64_t)n0 * 4};
  const uint32_t box[3] = {32, 32, 1}, box1[3] = {32, 1, 1};
  st->tmap_ptr[i] = cells;
  st->tmap_ok[i] = tma::encode_tiled(&st->tmap[i], CU_TENSOR_MAP_DATA_TYPE_INT32, 3,
                                     const_cast<void *>(cells), dims, strides, box,
                                     CU_TENSOR_MAP_SWIZZLE_128B) &&
                   tma::encode_tiled(&st->tpatch[i], CU_TENSOR_MAP_DATA_TYPE_INT32, 3,
                                     const_cast<void *>(cells), dims, strides, box1,
                                     CU_TENSOR_MAP_SWIZZLE_NONE);
  return st->tmap_ok[i] ? i : -1;
}

static LifeState *life_state(Handle *h) { return (LifeState *)h->impl; }
static uint32_t *life_history(Handle *h) {
  return (uint32_t *)((char *)h->h_scalars + h->result_offset());
}

cudaError_t life_check_cells_into(const int32_t *cells, size_t n, uint32_t *flag,
                                  cudaStream_t s);

// ---------------------------------------------------------------------------
// device code
// ---------------------------------------------------------------------------

// Next state of 32 cells (one word, bit i = cell 32w+i) from the words of
// the row above (a), the row itself (b) and the row below (c), each with its
// left (L) and right (R) neighbour word.
__device__ __forceinline__ uint32_t life_word(uint32_t aL, uint32_t a, uint32_t aR,
                                              uint32_t bL, uint32_t b, uint32_t bR,
                                              uint32_t cL, uint32_t c, uint32_t cR) {
  const uint32_t aW = __funnelshift_l(aL, a, 1), aE = __funnelshift_r(a, aR, 1);
  const uint32_t bW = __funnelshift_l(bL, b, 1), bE = __funnelshift_r(b, bR, 1);
  const uint32_t cW = __funnelshift_l(cL, c, 1), cE = __funnelshift_r(c, cR, 1);
  // column sums as 2-bit numbers: row a (3 cells), row b (2 cells), row c
  const uint32_t a1 = aW ^ a ^ aE, a2 = (aW & a) | (aE & (aW ^ a));
  const uint32_t c1 = cW ^ c ^ cE, c2 = (cW & c) | (cE & (cW ^ c));
  const uint32_t b1 = bW ^ bE, b2 = bW & bE;
  // num = s0 + 2*(a2 + b2 + c2 + k0)
  const uint32_t s0 = a1 ^ b1 ^ c1;
  const uint32_t k0 = (a1 & b1) | (c1 & (a1 ^ b1));
  // alive' = (num == 3) | (b & num == 2) = exactly-one(a2,b2,c2,k0) & (s0 | b)
  const uint32_t one = (a2 ^ b2 ^ c2 ^ k0) & ~(a2 & b2) & ~(c2 & k0);
  return one & (s0 | b);
}

// One generation on int32 cells, the reference's arithmetic.  Grid covers
// the memory array; open-boundary margins of `next` are written 0 (the
// generated manifest is never written there).
template <bool CYCLIC>
__global__ void __launch_bounds__(256)
life_general_kernel(const int32_t *__restrict__ cur, int32_t *__restrict__ next,
                    int ms0, int ms1, int lm, int tiles_x,
                    uint32_t *__restrict__ pop) {
  const int bx = (int)(blockIdx.x % (unsigned)tiles_x);
  const int by = (int)(blockIdx.x / (unsigned)tiles_x);
  const int x = bx * 32 + threadIdx.x;
  const int y = by * 8 + threadIdx.y;
  uint32_t v = 0;
  if (x < ms0 && y < ms1) {
    const bool interior =
        CYCLIC || (x >= lm && x < ms0 - lm && y >= lm && y < ms1 - lm);
    if (interior) {
      int xm, xp, ym, yp;
      if (CYCLIC) {
        xm = x == 0 ? ms0 - 1 : x - 1;
        xp = x == ms0 - 1 ? 0 : x + 1;
        ym = y == 0 ? ms1 - 1 : y - 1;
        yp = y == ms1 - 1 ? 0 : y + 1;
      } else {
        xm = x - 1; xp = x + 1; ym = y - 1; yp = y + 1;
      }
      const int32_t *rm = cur + (size_t)ym * ms0;
      const int32_t *r0 = cur + (size_t)y * ms0;
      const int32_t *rp = cur + (size_t)yp * ms0;
      // wraparound integer sum, as the generated int arithmetic
      const uint32_t num = (uint32_t)rp[xp] + (uint32_t)rp[x] + (uint32_t)rp[xm] +
                           (uint32_t)r0[xp] + (uint32_t)r0[xm] + (uint32_t)rm[xp] +
                           (uint32_t)rm[x] + (uint32_t)rm[xm];
      const int32_t n = (int32_t)num;
      const int32_t c = r0[x];
      v = ((c == 0 && n == 3) || (c == 1 && n >= 2 && n <= 3)) ? 1u : 0u;
    }
    next[(size_t)y * ms0 + x] = (int32_t)v;
  }
  __shared__ uint32_t ws[8];
  const uint32_t s = __reduce_add_sync(0xffffffffu, v);
  const int warp = threadIdx.y;
  if (threadIdx.x == 0) ws[warp] = s;
  __syncthreads();
  if (warp == 0) {
    uint32_t t = threadIdx.x < 8 ? ws[threadIdx.x] : 0u;
    t = __reduce_add_sync(0xffffffffu, t);
    if (threadIdx.x == 0 && t) atomicAdd(pop, t);
  }
}

// Load an nr x nc block of packed words into shared memory (row stride nc):
// block row r is global row wrap(row0 + r), block column c is global word
// wrap(col0 + c).  One warp per row at a time; each word is 32 coalesced
// int32 loads folded by a ballot, 8 words in flight per warp.  Row and
// word indices advance incrementally (no division per word).
__device__ __forceinline__ void pack_rows(const int32_t *__restrict__ cur, int n0, int n1,
                                          int wd, int row0, int col0, int nc, int nr,
                                          uint32_t *dst, int warp, int nwarps, int lane) {
  int gx0 = col0 % wd;
  if (gx0 < 0) gx0 += wd;
  const bool narrow = nc > wd;  // tiny grids: a tile row wraps more than once
  for (int r = warp; r < nr; r += nwarps) {
    int gy = (row0 + r) % n1;
    if (gy < 0) gy += n1;
    const int32_t *row = cur + (size_t)gy * n0 + lane;
    uint32_t *out = dst + r * nc;
    for (int c0 = 0; c0 < nc; c0 += 8) {
      int32_t v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = c0 + j;
        v[j] = 0;
        if (c < nc) {
          int gx = gx0 + c;
          if (narrow) gx %= wd;
          else if (gx >= wd) gx -= wd;
          v[j] = __ldg(row + (size_t)gx * 32);
        }
      }
      uint32_t mine = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t w = __ballot_sync(0xffffffffu, v[j] != 0);
        if (lane == j) mine = w;
      }
      if (lane < 8 && c0 + lane < nc) out[c0 + lane] = mine;
    }
  }
}

// Bit t of an 8-bit value moved to bit 4t.
__device__ __forceinline__ uint32_t spread4(uint32_t x) {
  x = (x | (x << 12)) & 0x000F000Fu;
  x = (x | (x << 6)) & 0x03030303u;
  x = (x | (x << 3)) & 0x11111111u;
  return x;
}

// pack_rows with 128-bit cell loads: lane L reads cells 4(L%8)..4(L%8)+3 of
// word L/8 of a 4-word group, so one warp instruction moves 512 bytes.
// Ballot j holds cell 4t+j of word m at bit 8m+t; word m is the four bytes
// m of the ballots interleaved.  G groups (4G words, G x 512 bytes) in
// flight per warp.
template <int G>
__device__ __forceinline__ void pack_rows_vec(const int32_t *__restrict__ cur, int n0, int n1,
                                              int wd, int row0, int col0, int nc, int nr,
                                              uint32_t *dst, int warp, int nwarps, int lane) {
  int gx0 = col0 % wd;
  if (gx0 < 0) gx0 += wd;
  const bool narrow = nc > wd;
  const int sub = lane >> 3, quad = (lane & 7) * 4;
  for (int r = warp; r < nr; r += nwarps) {
    int gy = (row0 + r) % n1;
    if (gy < 0) gy += n1;
    const int32_t *row = cur + (size_t)gy * n0 + quad;
    uint32_t *out = dst + r * nc;
    for (int c0 = 0; c0 < nc; c0 += 4 * G) {
      int4 v[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const int cw = c0 + 4 * g + sub;
        v[g] = make_int4(0, 0, 0, 0);
        if (cw < nc) {
          int gx = gx0 + cw;
          if (narrow) gx %= wd;
          else if (gx >= wd) gx -= wd;
          v[g] = __ldg(reinterpret_cast<const int4 *>(row + (size_t)gx * 32));
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const uint32_t b0 = __ballot_sync(0xffffffffu, v[g].x != 0);
        const uint32_t b1 = __ballot_sync(0xffffffffu, v[g].y != 0);
        const uint32_t b2 = __ballot_sync(0xffffffffu, v[g].z != 0);
        const uint32_t b3 = __ballot_sync(0xffffffffu, v[g].w != 0);
        const int cw = c0 + 4 * g + lane;
        if (lane < 4 && cw < nc) {
          const int sh = 8 * lane;
          out[cw] = spread4((b0 >> sh) & 0xFFu) | (spread4((b1 >> sh) & 0xFFu) << 1) |
                    (spread4((b2 >> sh) & 0xFFu) << 2) | (spread4((b3 >> sh) & 0xFFu) << 3);
        }
      }
    }
  }
}

// pack_rows_vec for rows of exactly 32 words (the register kernel), for
// cells that are all 0 or 1: lane L loads cells 4t .. 4t+3 (t = L % 8) of
// word 4g + L / 8 of group g, forms their nibble shifted to bit 4t with
// multiply-adds, and the eight lanes of a word add their nibbles (disjoint
// bits) in three butterfly steps.  Lane 8s of each word's eight stores it.
__device__ __forceinline__ void pack_rows32(const int32_t *__restrict__ cur, int n0, int n1,
                                            int wd, int row0, int col0, int nr, uint32_t *dst,
                                            int warp, int nwarps, int lane) {
  int gx0 = col0 % wd;
  if (gx0 < 0) gx0 += wd;
  const bool narrow = 32 > wd;
  const int sub = lane >> 3, t = lane & 7, quad = t * 4;
  const uint32_t m1 = 1u << quad, m2 = m1 << 1, m4 = m1 << 2, m8 = m1 << 3;
  for (int r = warp; r < nr; r += nwarps) {
    int gy = (row0 + r) % n1;
    if (gy < 0) gy += n1;
    const int32_t *row = cur + (size_t)gy * n0 + quad;
    int4 v[8];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      int gx = gx0 + 4 * g + sub;
      if (narrow) gx %= wd;
      else if (gx >= wd) gx -= wd;
      v[g] = __ldg(reinterpret_cast<const int4 *>(row + (size_t)gx * 32));
    }
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      uint32_t w = (uint32_t)v[g].x * m1 + (uint32_t)v[g].y * m2 + (uint32_t)v[g].z * m4 +
                   (uint32_t)v[g].w * m8;
      w += __shfl_xor_sync(0xffffffffu, w, 1);
      w += __shfl_xor_sync(0xffffffffu, w, 2);
      w += __shfl_xor_sync(0xffffffffu, w, 4);
      if (t == 0) dst[r * 32 + 4 * g + sub] = w;
    }
  }
}

// pack_rows32 with each lane's cells staged in shared memory by
// asynchronous 16-byte copies, two rows in flight per warp: the loads of the
// next row are under way while this row's nibbles are summed, and no
// registers are held by loads in flight.  A lane reads back only the cells it
// copied itself, so the warp needs no barrier.  `stage` is 2 x 256 int4 of
// this warp.
__device__ __forceinline__ void pack_rows32_async(const int32_t *__restrict__ cur, int n0, int n1,
                                                  int wd, int row0, int col0, int nr,
                                                  uint32_t *dst, int warp, int nwarps, int lane,
                                                  int4 *stage) {
  int gx0 = col0 % wd;
  if (gx0 < 0) gx0 += wd;
  const bool narrow = 32 > wd;
  const int sub = lane >> 3, t = lane & 7, quad = t * 4;
  const uint32_t m1 = 1u << quad, m2 = m1 << 1, m4 = m1 << 2, m8 = m1 << 3;
  auto issue = [&](int r, int4 *into) {
    int gy = (row0 + r) % n1;
    if (gy < 0) gy += n1;
    const int32_t *row = cur + (size_t)gy * n0 + quad;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      int gx = gx0 + 4 * g + sub;
      if (narrow) gx %= wd;
      else if (gx >= wd) gx -= wd;
      const unsigned d = (unsigned)__cvta_generic_to_shared(into + g * 32 + lane);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d),
                   "l"(row + (size_t)gx * 32)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  int i = 0;
  if (warp < nr) issue(warp, stage);
  for (int r = warp; r < nr; r += nwarps, ++i) {
    int4 *cur_stage = stage + (i & 1) * 256;
    if (r + nwarps < nr) {
      issue(r + nwarps, stage + ((i + 1) & 1) * 256);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int4 v = cur_stage[g * 32 + lane];
      uint32_t w = (uint32_t)v.x * m1 + (uint32_t)v.y * m2 + (uint32_t)v.z * m4 +
                   (uint32_t)v.w * m8;
      w += __shfl_xor_sync(0xffffffffu, w, 1);
      w += __shfl_xor_sync(0xffffffffu, w, 2);
      w += __shfl_xor_sync(0xffffffffu, w, 4);
      if (t == 0) dst[r * 32 + 4 * g + sub] = w;
    }
  }
}

struct TbParams {
  int n0, n1, wd;   // grid in cells, width in words
  int tw, th, kk;   // tile width (words), height (rows), generations
  int nt0, nt1;     // tiles per axis
  int nb;           // cells in the last word of a row (32 unless n0 % 32 != 0)
};

// A packed grid: rows of wd = ceil(n0 / 32) words, bit i of word w is cell
// (32 w + i) mod n0.  Where n0 is no multiple of 32 the last word of a row
// thus goes on with the row's first cells, so that a tile reads the periodic
// row as a string of words.
//
// Word j of that string for -1 <= j <= wd, as the bits [sh, sh + 32) of words
// o0 (low) and o1 (high).  Word -1 ends at cell n0 - 1, word wd starts at cell
// 32 wd; words further out are never needed right (clamped to wd).
struct ExtWord {
  int o0, o1, sh;
};
__device__ __forceinline__ ExtWord ext_word(int j, int wd, int nb) {
  if (j < 0) {  // cells n0 - 32 .. n0 - 1
    if (nb == 32) return ExtWord{wd - 1, wd - 1, 0};
    return ExtWord{wd - 2, wd - 1, nb};
  }
  if (j >= wd) {  // cells 32 wd mod n0 ..
    if (nb == 32) return ExtWord{0, 0, 0};
    return ExtWord{0, 1, 32 - nb};
  }
  return ExtWord{j, j, 0};
}

// Temporal blocking: each CTA owns a tw x th tile (words x rows), loads it
// with a halo of 1 word and kk rows, advances kk generations in shared
// memory and writes back its owned cells.  After g generations the halo's
// stale front has moved g cells / rows inward; kk <= 32 keeps it inside the
// halo word, and kk rows of vertical halo keep it off the owned rows.
template <bool VEC>
__global__ void __launch_bounds__(256)
life_tb_kernel(const int32_t *__restrict__ cur, int32_t *__restrict__ next,
               TbParams p, uint32_t *__restrict__ pop) {
  extern __shared__ uint32_t sm[];
  __shared__ uint32_t spop[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nthreads = blockDim.x, nwarps = nthreads >> 5;
  const int t = blockIdx.x;
  const int t0 = t % p.nt0, t1 = t / p.nt0;
  const int col0 = t0 * p.tw, row0 = t1 * p.th;
  const int tw_own = min(p.tw, p.wd - col0), th_own = min(p.th, p.n1 - row0);
  const int kk = p.kk;
  const int NC = tw_own + 2, NR = th_own + 2 * kk;
  const int stride = (p.tw + 2) * (p.th + 2 * kk);
  uint32_t *A = sm, *B = sm + stride;
  if (tid < 32) spop[tid] = 0;
  if (VEC)
    pack_rows_vec<4>(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, NC, NR, A, warp, nwarps, lane);
  else
    pack_rows(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, NC, NR, A, warp, nwarps, lane);
  __syncthreads();
  const int NG = max(1, nthreads / NC);
  for (int g = 1; g <= kk; ++g) {
    const int nrows = NR - 2 * g;
    const int chunk = (nrows + NG - 1) / NG;
    uint32_t cnt = 0;
    for (int ci = tid; ci < NC * NG; ci += nthreads) {
      const int c = ci % NC, grp = ci / NC;
      const int rs = g + grp * chunk, re = min(rs + chunk, NR - g);
      if (rs >= re) continue;
      const bool hasL = c > 0, hasR = c < NC - 1;
      const uint32_t *col = A + c;
      uint32_t aL = hasL ? col[(rs - 1) * NC - 1] : 0u, a = col[(rs - 1) * NC],
               aR = hasR ? col[(rs - 1) * NC + 1] : 0u;
      uint32_t bL = hasL ? col[rs * NC - 1] : 0u, b = col[rs * NC],
               bR = hasR ? col[rs * NC + 1] : 0u;
      const bool own_c = c >= 1 && c <= tw_own;
      for (int r = rs; r < re; ++r) {
        const uint32_t cL = hasL ? col[(r + 1) * NC - 1] : 0u, cc = col[(r + 1) * NC],
                       cR = hasR ? col[(r + 1) * NC + 1] : 0u;
        const uint32_t w = life_word(aL, a, aR, bL, b, bR, cL, cc, cR);
        B[r * NC + c] = w;
        if (own_c && r >= kk && r < kk + th_own) cnt += __popc(w);
        aL = bL; a = b; aR = bR;
        bL = cL; b = cc; bR = cR;
      }
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0 && cnt) atomicAdd(&spop[g - 1], cnt);
    __syncthreads();
    uint32_t *tmp = A; A = B; B = tmp;
  }
  if (tid < kk && spop[tid]) atomicAdd(&pop[tid], spop[tid]);
  // write back the owned words, one warp per row
  if (VEC) {
    // lane L writes cells 4(L%8)..+3 of word L/8 of each 4-word group
    const int sub = lane >> 3, quad = (lane & 7) * 4;
    for (int r = warp; r < th_own; r += nwarps) {
      const uint32_t *src = A + (r + kk) * NC + 1;
      int32_t *dst = next + (size_t)(row0 + r) * p.n0 + (size_t)col0 * 32 + quad;
      for (int c0 = 0; c0 < tw_own; c0 += 16) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int cw = c0 + 4 * g + sub;
          if (cw < tw_own) {
            const uint32_t w = src[cw] >> quad;
            *reinterpret_cast<int4 *>(dst + (size_t)cw * 32) =
                make_int4((int)(w & 1u), (int)((w >> 1) & 1u), (int)((w >> 2) & 1u),
                          (int)((w >> 3) & 1u));
          }
        }
      }
    }
  } else {
    // lane i writes bit i of each word
    for (int r = warp; r < th_own; r += nwarps) {
      const uint32_t *src = A + (r + kk) * NC + 1;
      int32_t *dst = next + (size_t)(row0 + r) * p.n0 + (size_t)col0 * 32 + lane;
      for (int c0 = 0; c0 < tw_own; c0 += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = c0 + j;
          if (c < tw_own) dst[(size_t)c * 32] = (int32_t)((src[c] >> lane) & 1u);
        }
      }
    }
  }
}

// Row sums used by the sliding-window update: the two-bit sum (f1 ones, f2
// twos) of the three cells W, C, E of every bit position of one 32-cell word.
struct RowSums {
  uint32_t raw, f1, f2;
};

// one three-input bit operation; LUT bit 4x + 2y + z gives its value at (x, y, z)
template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t x, uint32_t y, uint32_t z) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(x), "r"(y), "r"(z), "n"(LUT));
  return d;
}
__device__ __forceinline__ uint32_t xor3(uint32_t x, uint32_t y, uint32_t z) {
  return lop3<0x96>(x, y, z);
}
__device__ __forceinline__ uint32_t maj3(uint32_t x, uint32_t y, uint32_t z) {
  return lop3<0xE8>(x, y, z);
}

__device__ __forceinline__ RowSums row_sums(uint32_t left, uint32_t w, uint32_t right) {
  const uint32_t W = __funnelshift_l(left, w, 1), E = __funnelshift_r(w, right, 1);
  return RowSums{w, xor3(W, w, E), maj3(W, w, E)};
}

// next state of the middle row b from the sums of rows a (above), b, c.  The
// sum of all nine cells is u0 + 2 (k0 + u1) + 4 u2; a cell lives when it is 3,
// or 4 with the cell itself alive.  With one = exactly one of (k0, u1, u2):
//   u0 = 1: sum 3 is one & ~u2;  u0 = 0: sum 4 is u2 ? one : ~one (sum 0 also
//   gives ~one, but not with the cell alive),
// and the result is that & (u0 | b).  Nine three-input operations a word with
// the two of row_sums; the ALU takes 64 lanes a cycle per SM and these, the
// two shifts and the count are what bounds every packed kernel (the half-adder
// of the middle row that this form does without made it eleven).
__device__ __forceinline__ uint32_t life_from_sums(const RowSums &a, const RowSums &b,
                                                   const RowSums &c) {
  const uint32_t u0 = xor3(a.f1, b.f1, c.f1), k0 = maj3(a.f1, b.f1, c.f1);
  const uint32_t u1 = xor3(a.f2, b.f2, c.f2), u2 = maj3(a.f2, b.f2, c.f2);
  const uint32_t one = lop3<0x16>(k0, u1, u2);
  const uint32_t hit = lop3<0x29>(u0, u2, one);
  return lop3<0xE0>(hit, u0, b.raw);
}

// Two neighbouring rows b, c advanced together between a (above) and d (below):
// the sum of b and c, s0 + 2 s1 + 4 s2, is formed once and serves both, and
// four operations more decide each row (with l = the parity test against the
// cell, m = the test of the twos, found by search over three-input networks):
// eight a word in all instead of nine.
__device__ __forceinline__ uint32_t life_from_pair(uint32_t s0, uint32_t s1, uint32_t s2,
                                                   const RowSums &a, uint32_t cell) {
  const uint32_t l = lop3<0x19>(cell, a.f1, s0), m = lop3<0x19>(s2, a.f2, s1);
  return lop3<0x18>(lop3<0x35>(l, cell, s2), m, l);
}
__device__ __forceinline__ void life_two_rows(const RowSums &a, const RowSums &b,
                                              const RowSums &c, const RowSums &d,
                                              uint32_t &nb, uint32_t &nc) {
  const uint32_t s0 = b.f1 ^ c.f1, k = b.f1 & c.f1;
  const uint32_t s1 = xor3(b.f2, c.f2, k), s2 = maj3(b.f2, c.f2, k);
  nb = life_from_pair(s0, s1, s2, a, b.raw);
  nc = life_from_pair(s0, s1, s2, d, c.raw);
}

// A small grid in the registers of one CTA: all generations of a run in one
// launch, any row length (wd = ceil(n0 / 32) <= 32 words, the last of nb
// cells).
struct SmallParams {
  int n0, n1, wd, nb;
  int gens;  // 1 .. kSmallMaxGens
  int nw;    // warps that advance rows; the block's others only move cells
  int h;     // halo rows each side, and generations between exchanges
  int before;  // generations of the run before these (populations in pop)
};
static const int kSmallThreads = 512;
static const int kSmallMaxGens = 4096;  // populations kept in shared memory

// A warp has rg = 32 / wd groups of lanes, each lane one word of R rows: R rg
// rows of the whole width, of which the middle ones are the warp's own share of
// the grid and h above and below are copies.  A generation needs no other warp:
// west and east words and the row sums above and below a lane's rows come from
// the lanes beside.  Every h generations, when the copies are stale up to the
// own rows, the warps trade own rows for copies through shared memory.
// RAG: nb < 32.  The last word's bits above nb stay 0; the word west of the
// first is the last one with cell n0 - 1 in its top bit, and the last word's
// east neighbour is cell 0 at bit nb - 1.
template <int R, bool RAG>
__global__ void __launch_bounds__(kSmallThreads)
life_smallreg_kernel(const int32_t *__restrict__ cur, int32_t *__restrict__ next, SmallParams p,
                     uint32_t *__restrict__ pop, LifeScalars *scalars, uint32_t *hist) {
  extern __shared__ uint32_t S[];  // 2 x words, then the populations
  const int wd = p.wd, n1 = p.n1, nwords = wd * n1;
  uint32_t *spop = S + 2 * nwords;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWB = kSmallThreads / 32;
  for (int i = tid; i < p.gens; i += kSmallThreads) spop[i] = 0;
  // pack the cells, eight words of the grid in flight per warp
  for (int i0 = warp * 8; i0 < nwords; i0 += NWB * 8) {
    int32_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = min(i0 + j, nwords - 1), y = i / wd, x = (i - y * wd) * 32 + lane;
      v[j] = x < p.n0 ? __ldg(cur + (size_t)y * p.n0 + x) : 0;
    }
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t w = __ballot_sync(0xffffffffu, v[j] != 0);
      if (lane == j) mine = w;
    }
    if (lane < 8 && i0 + lane < nwords) S[i0 + lane] = mine;
  }
  __syncthreads();
  if (warp < p.nw) {
    const int rg = 32 / wd, x = lane % wd, r = lane / wd, h = p.h;
    // this warp's own rows: local rows h .. h + own, row j of the block of
    // copies is row (start - h + j) mod n1 of the grid
    const int start = (int)((long long)warp * n1 / p.nw);
    const int own = (int)((long long)(warp + 1) * n1 / p.nw) - start;
    const int j0 = r * R;
    const int g0 = ((start - h + j0) % n1 + n1) % n1;
    const bool used = r < rg;
    uint32_t rows[R], ownrow = 0;  // own rows of this lane
    {
      int gy = g0;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        rows[i] = S[gy * wd + x];
        if (used && j0 + i >= h && j0 + i < h + own) ownrow |= 1u << i;
        gy = gy + 1 == n1 ? 0 : gy + 1;
      }
    }
    const int west = used && x == 0 ? lane + wd - 1 : (lane == 0 ? 0 : lane - 1);
    const int east = used && x == wd - 1 ? lane - wd + 1 : (lane == 31 ? 31 : lane + 1);
    const int up = (lane - wd) & 31, down = (lane + wd) & 31;
    const bool lastw = x == wd - 1;
    const int lsh = RAG && x == 0 ? 32 - p.nb : 0;       // of the west word
    const int esh = RAG && lastw ? p.nb - 1 : 31;        // of the east word
    const uint32_t keep = RAG && lastw ? (1u << p.nb) - 1u : ~0u;
    auto sums = [&](uint32_t w, uint32_t &f1, uint32_t &f2) {
      const uint32_t wl = __shfl_sync(0xffffffffu, w, west);
      const uint32_t wr = __shfl_sync(0xffffffffu, w, east);
      const uint32_t W = __funnelshift_l(RAG ? wl << lsh : wl, w, 1);
      const uint32_t E = RAG ? (w >> 1) | (wr << esh) : __funnelshift_r(w, wr, 1);
      f1 = xor3(W, w, E);
      f2 = maj3(W, w, E);
    };
    uint32_t *buf = S + nwords;  // the buffer of the next exchange
    // counts of an even generation and the next, and those of the pair before,
    // summed over the warp while the next generation is under way
    uint32_t pair = 0, done = 0;
    int left = h;                // generations until the copies are stale
    for (int g = 0; g < p.gens; ++g) {
      const uint32_t sum = g & 1 ? 0u : __reduce_add_sync(0xffffffffu, done);
      // sums of rows -1 (the lane above's last) .. R (the lane below's first)
      uint32_t f1[R + 2], f2[R + 2];
#pragma unroll
      for (int i = 0; i < R; ++i) sums(rows[i], f1[i + 1], f2[i + 1]);
      f1[0] = __shfl_sync(0xffffffffu, f1[R], up);
      f2[0] = __shfl_sync(0xffffffffu, f2[R], up);
      f1[R + 1] = __shfl_sync(0xffffffffu, f1[1], down);
      f2[R + 1] = __shfl_sync(0xffffffffu, f2[1], down);
      uint32_t cnt = 0;
      auto put = [&](int i, uint32_t w) {
        if (RAG) w &= keep;
        rows[i] = w;
        cnt += ownrow & (1u << i) ? __popc(w) : 0;
      };
#pragma unroll
      for (int i = 0; i < R; i += 2) {
        const RowSums ra{0u, f1[i], f2[i]}, rb{rows[i], f1[i + 1], f2[i + 1]};
        if (i + 1 < R) {
          uint32_t wb, wc;
          life_two_rows(ra, rb, RowSums{rows[i + 1], f1[i + 2], f2[i + 2]},
                        RowSums{0u, f1[i + 3], f2[i + 3]}, wb, wc);
          put(i, wb);
          put(i + 1, wc);
        } else {
          put(i, life_from_sums(ra, rb, RowSums{0u, f1[i + 2], f2[i + 2]}));
        }
      }
      // a warp's count is at most 32 x 32 R < 2^16: two generations a sum
      if (g & 1) {
        done = pair | cnt << 16;
      } else {
        pair = cnt;
        if (g > 0 && lane < 2) atomicAdd(&spop[g - 2 + lane], (sum >> (16 * lane)) & 0xffffu);
      }
      if (--left == 0 && g != p.gens - 1) {
        left = h;
        int gy = g0;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (ownrow & (1u << i)) buf[gy * wd + x] = rows[i];
          gy = gy + 1 == n1 ? 0 : gy + 1;
        }
        asm volatile("bar.sync 1, %0;" ::"r"(p.nw * 32) : "memory");
        gy = g0;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (!(ownrow & (1u << i))) rows[i] = buf[gy * wd + x];
          gy = gy + 1 == n1 ? 0 : gy + 1;
        }
        // the other buffer may be written at the next exchange: its last
        // readers passed this one's barrier
        buf = buf == S ? S + nwords : S;
      }
    }
    {  // the last one or two generations
      const bool odd = p.gens & 1;
      const uint32_t sum = __reduce_add_sync(0xffffffffu, odd ? pair : done);
      if (lane < (odd ? 1 : 2))
        atomicAdd(&spop[p.gens - (odd ? 1 : 2) + lane], (sum >> (16 * lane)) & 0xffffu);
    }
    // into the buffer that no warp still reads
    int gy = g0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (ownrow & (1u << i)) buf[gy * wd + x] = rows[i];
      gy = gy + 1 == n1 ? 0 : gy + 1;
    }
    if (tid == 0) spop[p.gens] = (uint32_t)(buf - S);
  }
  __syncthreads();
  const uint32_t *out = S + spop[p.gens];
  for (int i = tid; i < p.gens; i += kSmallThreads) {
    if (hist) hist[p.before + i] = spop[i];
    else pop[i] += spop[i];
  }
  if (hist && tid == 0) {
    for (int i = 0; i < p.before; ++i) {
      hist[i] = pop[i];
      pop[i] = 0;
    }
    scalars->population = (int32_t)spop[p.gens - 1];
    scalars->generation =
        (int32_t)((uint32_t)scalars->generation + (uint32_t)(p.before + p.gens));
  }
  for (int i = warp; i < nwords; i += NWB) {
    const int y = i / wd, x = (i - y * wd) * 32 + lane;
    if (x < p.n0) next[(size_t)y * p.n0 + x] = (int32_t)((out[i] >> lane) & 1u);
  }
}

// Temporal blocking with one lane per packed word: a tile is 32 words wide
// (30 owned + a halo word each side) and th rows tall plus kk halo rows above
// and below.  Each warp sweeps a contiguous band of rows per generation,
// taking the left/right neighbour words from the adjacent lanes and keeping
// the row sums of the previous two rows in registers.
template <bool VEC>
__global__ void __launch_bounds__(256, 8)
life_tb32_kernel(const int32_t *__restrict__ cur, int32_t *__restrict__ next, TbParams p,
                 uint32_t *__restrict__ pop) {
  extern __shared__ uint32_t sm[];
  __shared__ uint32_t spop[32];
  constexpr int NC = 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  const int t = blockIdx.x;
  const int t0 = t % p.nt0, t1 = t / p.nt0;
  const int col0 = t0 * p.tw, row0 = t1 * p.th;
  const int tw_own = min(p.tw, p.wd - col0), th_own = min(p.th, p.n1 - row0);
  const int kk = p.kk;
  const int NR = th_own + 2 * kk;
  const int stride = NC * (p.th + 2 * kk);
  uint32_t *A = sm, *B = sm + stride;
  if (tid < 32) spop[tid] = 0;
  if (VEC)
    pack_rows_vec<4>(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, NC, NR, A, warp, nwarps, lane);
  else
    pack_rows(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, NC, NR, A, warp, nwarps, lane);
  __syncthreads();
  const bool own_c = lane >= 1 && lane <= tw_own;
  for (int g = 1; g <= kk; ++g) {
    const int lo = g, hi = NR - g;
    const int chunk = (hi - lo + nwarps - 1) / nwarps;
    const int rs = lo + warp * chunk, re = min(rs + chunk, hi);
    uint32_t cnt = 0;
    if (rs < re) {
      uint32_t w = A[(rs - 1) * NC + lane];
      RowSums a = row_sums(__shfl_up_sync(0xffffffffu, w, 1) & (lane ? ~0u : 0u), w,
                           __shfl_down_sync(0xffffffffu, w, 1) & (lane < 31 ? ~0u : 0u));
      w = A[rs * NC + lane];
      RowSums b = row_sums(__shfl_up_sync(0xffffffffu, w, 1) & (lane ? ~0u : 0u), w,
                           __shfl_down_sync(0xffffffffu, w, 1) & (lane < 31 ? ~0u : 0u));
      for (int r = rs; r < re; ++r) {
        w = A[(r + 1) * NC + lane];
        const RowSums c = row_sums(__shfl_up_sync(0xffffffffu, w, 1) & (lane ? ~0u : 0u), w,
                                   __shfl_down_sync(0xffffffffu, w, 1) & (lane < 31 ? ~0u : 0u));
        const uint32_t out = life_from_sums(a, b, c);
        B[r * NC + lane] = out;
        if (own_c && r >= kk && r < kk + th_own) cnt += __popc(out);
        a = b;
        b = c;
      }
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0 && cnt) atomicAdd(&spop[g - 1], cnt);
    __syncthreads();
    uint32_t *tmp = A; A = B; B = tmp;
  }
  if (tid < kk && spop[tid]) atomicAdd(&pop[tid], spop[tid]);
  // write back the owned words (block columns 1..tw_own), one warp per row
  if (VEC) {
    const int sub = lane >> 3, quad = (lane & 7) * 4;
    for (int r = warp; r < th_own; r += nwarps) {
      const uint32_t *src = A + (r + kk) * NC + 1;
      int32_t *dst = next + (size_t)(row0 + r) * p.n0 + (size_t)col0 * 32 + quad;
      for (int c0 = 0; c0 < tw_own; c0 += 16) {
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          const int cw = c0 + 4 * gq + sub;
          if (cw < tw_own) {
            const uint32_t wv = src[cw] >> quad;
            *reinterpret_cast<int4 *>(dst + (size_t)cw * 32) =
                make_int4((int)(wv & 1u), (int)((wv >> 1) & 1u), (int)((wv >> 2) & 1u),
                          (int)((wv >> 3) & 1u));
          }
        }
      }
    }
  } else {
    for (int r = warp; r < th_own; r += nwarps) {
      const uint32_t *src = A + (r + kk) * NC + 1;
      int32_t *dst = next + (size_t)(row0 + r) * p.n0 + (size_t)col0 * 32 + lane;
      for (int c = 0; c < tw_own; ++c) dst[(size_t)c * 32] = (int32_t)((src[c] >> lane) & 1u);
    }
  }
}

// row sums of a row of one word per lane
__device__ __forceinline__ RowSums lane_sums(uint32_t w) {
  return row_sums(__shfl_up_sync(0xffffffffu, w, 1), w, __shfl_down_sync(0xffffffffu, w, 1));
}

// One generation of a warp's R rows of 32 words in registers; the block's
// warps are stacked, and each trades the row sums of its first and last row
// with its neighbours through ex (NW x 2 x 32 pairs, double-buffered by the
// caller).  The rows between are advanced before the wait: a warp's neighbours
// have then written theirs, and only the two edge rows follow it.  `arrive`
// publishes this warp's sums, `wait` waits for the neighbours'.  Returns the
// lane's count of living cells: of all rows (whole) or of the owned rows and
// bits only.
template <int R, int NW, class Arrive, class Wait>
__device__ __forceinline__ uint32_t life_generation(uint32_t (&rows)[R], uint2 (*ex)[2][32],
                                                    int warp, int lane, bool whole,
                                                    uint32_t ownrows, uint32_t colmask, Arrive arrive,
                                                    Wait wait) {
  const RowSums s0 = lane_sums(rows[0]), sl = lane_sums(rows[R - 1]);
  ex[warp][0][lane] = make_uint2(s0.f1, s0.f2);
  ex[warp][1][lane] = make_uint2(sl.f1, sl.f2);
  arrive();
  uint32_t cnt = 0;
  RowSums ra = s0, rb = lane_sums(rows[1]);
  const RowSums s1 = rb;
  auto count = [&](int i) {
    if (whole) cnt += __popc(rows[i]);
    else if (ownrows & (1u << i)) cnt += __popc(rows[i] & colmask);
  };
#pragma unroll
  for (int i = 1; i < R - 1; i += 2) {
    const RowSums rc = i + 1 < R - 1 ? lane_sums(rows[i + 1]) : sl;
    if (i + 1 < R - 1) {
      const RowSums rd = i + 2 < R - 1 ? lane_sums(rows[i + 2]) : sl;
      life_two_rows(ra, rb, rc, rd, rows[i], rows[i + 1]);
      count(i);
      count(i + 1);
      ra = rc;
      rb = rd;
    } else {  // an odd row is left
      rows[i] = life_from_sums(ra, rb, rc);
      count(i);
      ra = rb;
      rb = rc;
    }
  }
  wait();
  const uint2 up = warp > 0 ? ex[warp - 1][1][lane] : make_uint2(0u, 0u);
  const uint2 down = warp < NW - 1 ? ex[warp + 1][0][lane] : make_uint2(0u, 0u);
  rows[0] = life_from_sums(RowSums{0u, up.x, up.y}, s0, s1);
  rows[R - 1] = life_from_sums(ra, sl, RowSums{0u, down.x, down.y});
  if (whole) {
    cnt += __popc(rows[0]) + __popc(rows[R - 1]);
  } else {
    if (ownrows & 1u) cnt += __popc(rows[0] & colmask);
    if (ownrows & (1u << (R - 1))) cnt += __popc(rows[R - 1] & colmask);
  }
  return cnt;
}

// Register-resident temporal blocking.  A block is NW warps x R rows of 32
// packed words (30 owned + halo word each side); warp w keeps rows
// [wR, wR+R) in registers for all kk generations and trades only its first
// and last row with the neighbouring warps through shared memory, once per
// generation.  Rows are not shrunk per generation: the stale front from the
// block's outer rows and columns moves one cell per generation and never
// reaches the owned rows [kk, kk + th_own) and words 1..tw_own.
//
// IO: what the tile is read from and written to.  A run of many generations
// takes the cells in once and out once: its first launch reads int32 cells and
// writes the packed grid, its last one reads the packed grid and writes cells,
// and those between stay packed (1/32 of the bytes, rows loaded straight into
// registers and stored from them).  Any row length is served where both ends
// are packed.
enum LifeIo { kCellsToCells = 0, kCellsToPacked = 1, kPackedToPacked = 2, kPackedToCells = 3 };

template <int R, int NW, bool VEC, int IO = kCellsToCells>
__global__ void __launch_bounds__(NW * 32, (NW >= 32 ? 1 : NW >= 16 ? 2 : 4))
life_reg_kernel(const void *__restrict__ in, void *__restrict__ out, TbParams p,
                uint32_t *__restrict__ pop) {
  constexpr int NC = 32, NR = R * NW;
  constexpr bool PIN = IO == kPackedToPacked || IO == kPackedToCells;
  constexpr bool POUT = IO == kPackedToPacked || IO == kCellsToPacked;
  extern __shared__ uint32_t A[];  // NR x NC packed words (not with both ends packed)
  __shared__ uint2 ex[2][NW][2][NC];
  __shared__ uint32_t spop[32];
  __shared__ int4 nib[16];  // nibble -> its four cells
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!POUT && tid < 16)
    nib[tid] = make_int4(tid & 1, (tid >> 1) & 1, (tid >> 2) & 1, (tid >> 3) & 1);
  const int t = blockIdx.x;
  const int t0 = t % p.nt0, t1 = t / p.nt0;
  // tiles split the grid evenly (sizes differ by at most one word / row)
  const int col0 = (int)((long long)t0 * p.wd / p.nt0);
  const int row0 = (int)((long long)t1 * p.n1 / p.nt1);
  const int tw_own = (int)((long long)(t0 + 1) * p.wd / p.nt0) - col0;
  const int th_own = (int)((long long)(t1 + 1) * p.n1 / p.nt1) - row0;
  const int kk = p.kk;
  if (tid < 32) spop[tid] = 0;
  uint32_t rows[R];
  if (PIN) {
    const uint32_t *src = (const uint32_t *)in;
    const ExtWord e = ext_word(min(col0 - 1 + lane, p.wd), p.wd, p.nb);
    // the block's rows kk + th_own + kk reach; the rest repeat its last one
    int gy = (row0 - kk + min(warp * R, th_own + 2 * kk - 1)) % p.n1;
    if (gy < 0) gy += p.n1;
    int left = th_own + 2 * kk - 1 - min(warp * R, th_own + 2 * kk - 1);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint32_t *row = src + (size_t)gy * p.wd;
      rows[i] = p.nb == 32 ? row[e.o0] : __funnelshift_r(row[e.o0], row[e.o1], e.sh);
      if (left > 0) {
        --left;
        if (++gy == p.n1) gy = 0;
      }
    }
    __syncthreads();
  } else {
    const int32_t *cur = (const int32_t *)in;
    if (VEC)
      pack_rows32(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, min(NR, th_own + 2 * kk), A, warp,
                  NW, lane);
    else
      pack_rows(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, NC, min(NR, th_own + 2 * kk), A, warp,
                NW, lane);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < R; ++i) rows[i] = A[(warp * R + i) * NC + lane];
  }
  // owned rows of this warp as a bit mask; owned columns as a lane mask
  uint32_t ownrows = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int gr = warp * R + i - kk;
    if (gr >= 0 && gr < th_own) ownrows |= 1u << i;
  }
  uint32_t colmask = (lane >= 1 && lane <= tw_own) ? ~0u : 0u;
  // the last word of a row that is no whole number of words counts nb cells
  const bool ragged = PIN && POUT && p.nb != 32 && col0 + tw_own == p.wd;
  if (ragged && lane == tw_own) colmask = (1u << p.nb) - 1u;
  // most warps own all their rows or none: those count every row and keep
  // the lane's count only if the lane and the rows are owned (no per-row
  // test); the warps on the block's halo edges test each row
  constexpr uint32_t allrows = R == 32 ? ~0u : ((1u << R) - 1u);
  const bool whole = ownrows == 0u || (ownrows == allrows && !ragged);
  auto arrive = [] {};
  auto wait = [] { __syncthreads(); };
  for (int g = 0; g < kk; ++g) {
    uint32_t cnt;
    if (whole)
      cnt = life_generation<R, NW>(rows, ex[g & 1], warp, lane, true, ownrows, colmask, arrive,
                                   wait) &
            (ownrows == allrows ? colmask : 0u);
    else
      cnt = life_generation<R, NW>(rows, ex[g & 1], warp, lane, false, ownrows, colmask, arrive,
                                   wait);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0 && cnt) atomicAdd(&spop[g], cnt);
  }
  if (POUT) {
    uint32_t *dst =
        (uint32_t *)out + (ptrdiff_t)(row0 + warp * R - kk) * p.wd + (col0 + lane - 1);
#pragma unroll
    for (int i = 0; i < R; ++i)
      if ((ownrows & (1u << i)) && lane >= 1 && lane <= tw_own) dst[(size_t)i * p.wd] = rows[i];
    __syncthreads();
    if (tid < kk && spop[tid]) atomicAdd(&pop[tid], spop[tid]);
    return;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < R; ++i) A[(warp * R + i) * NC + lane] = rows[i];
  __syncthreads();
  if (tid < kk && spop[tid]) atomicAdd(&pop[tid], spop[tid]);
  const int sub = lane >> 3, quad = (lane & 7) * 4;
  for (int r = warp; r < th_own; r += NW) {
    const uint32_t *src = A + (r + kk) * NC + 1;
    int32_t *dst = (int32_t *)out + (size_t)(row0 + r) * p.n0 + (size_t)col0 * 32;
    if (VEC) {
      // four cells of a word per lane, as the four cells of a nibble
      for (int c0 = 0; c0 < tw_own; c0 += 16) {
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          const int cw = c0 + 4 * gq + sub;
          if (cw < tw_own)
            *reinterpret_cast<int4 *>(dst + (size_t)cw * 32 + quad) =
                nib[(src[cw] >> quad) & 15u];
        }
      }
    } else {
      for (int c = 0; c < tw_own; ++c)
        dst[(size_t)c * 32 + lane] = (int32_t)((src[c] >> lane) & 1u);
    }
  }
}

// The packed grid of cells that are all 0 or 1 (rows of any length), one warp
// per eight words at a time.
__global__ void __launch_bounds__(256)
life_pack_kernel(const int32_t *__restrict__ cells, uint32_t *__restrict__ packed, int n0, int n1,
                 int wd) {
  const int lane = threadIdx.x & 31;
  const int groups = (wd + 7) / 8;
  const long long total = (long long)groups * n1;
  const long long step = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < total;
       i += step) {
    const int y = (int)(i / groups), w0 = (int)(i - (long long)y * groups) * 8;
    const int32_t *row = cells + (size_t)y * n0;
    int32_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      int x = (w0 + j) * 32 + lane;
      if (x >= n0) x -= n0;  // the row goes on with its first cells (n0 > 32)
      v[j] = w0 + j < wd ? __ldg(row + x) : 0;
    }
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t w = __ballot_sync(0xffffffffu, v[j] != 0);
      if (lane == j) mine = w;
    }
    if (lane < 8 && w0 + lane < wd) packed[(size_t)y * wd + w0 + lane] = mine;
  }
}

// and back: one warp per eight words of a row
__global__ void __launch_bounds__(256)
life_unpack_kernel(const uint32_t *__restrict__ packed, int32_t *__restrict__ cells, int n0, int n1,
                   int wd) {
  const int lane = threadIdx.x & 31;
  const int groups = (wd + 7) / 8;
  const long long total = (long long)groups * n1;
  const long long step = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < total;
       i += step) {
    const int y = (int)(i / groups), w0 = (int)(i - (long long)y * groups) * 8;
    const uint32_t mine = packed[(size_t)y * wd + min(w0 + (lane & 7), wd - 1)];
    int32_t *row = cells + (size_t)y * n0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t w = __shfl_sync(0xffffffffu, mine, j);
      const int x = (w0 + j) * 32 + lane;
      if (x < n0) row[x] = (int32_t)((w >> lane) & 1u);
    }
  }
}

// Warp-specialised persistent variant of the register-resident kernel: one
// CTA per SM walks its share of the tiles through a three-stage pipeline
// over three shared-memory tile buffers.  In stage s, producer warps pack
// tile s, consumer warps advance tile s-1 by kk generations in registers
// (edge rows traded through shared memory behind a named barrier that only
// the consumers use), and store warps write tile s-2 back, so loads,
// compute and stores of consecutive tiles overlap.  One __syncthreads ends
// every stage; there are no spin waits.
// whether a warp-specialised variant has room for its producers' staged rows
// (2 x 4 KB each) beside its three tile buffers
template <int R, int NWC, int NWP>
__host__ __device__ constexpr bool kStagedPack() {
  return 3 * 4 * 32 * R * NWC + 8192 * NWP <= 212992;
}

// TMA (the tile's rows arrive by tensor copies): producer warps pack from
// 4 KB row boxes (32 cells x 32 words x 1 row of the grid viewed as cells x
// words x rows, 128-byte swizzle) that land in NS slots per warp, complete
// on an mbarrier per slot and are issued NS - 1 boxes ahead of the row being
// packed.  Each lane packs one whole word from
// eight 16-byte chunks of its 128-byte line (the swizzle puts chunk j of
// line L at j ^ (L mod 8), so the warp's loads hit every bank once).  The box reads
// zeros outside the grid; in the first and last tile columns the one halo
// word that wraps around (word n0/32 - 1 left of word 0, word 0 right of
// the last word) comes in as a second, one-word box (`tpatch`, no swizzle)
// on the same mbarrier.  Words further out stay zero: with at most 32
// generations per launch their error front never reaches an owned word.
// Waits are bounded (tma::mbar_wait raises *err).
// PS: consumer warps synchronise each generation with their two neighbours
// only (an mbarrier per warp and buffer parity, signalled once the warp's
// boundary rows are written), instead of a barrier over all consumers
// IO: the first launch of a long run writes the packed grid and the last one
// reads it (see LifeIo); their store or producer warps then move 1/32 of the
// bytes with plain word accesses.
template <int R, int NWC, int NWP, int NWS, bool TMA = false, int NS = 2, bool PS = false,
          int IO = kCellsToCells>
__global__ void __launch_bounds__((NWC + NWP + NWS) * 32, 1)
life_ws_kernel(const void *__restrict__ in, void *__restrict__ out, TbParams p,
               uint32_t *__restrict__ pop, const __grid_constant__ CUtensorMap tmap,
               const __grid_constant__ CUtensorMap tpatch, uint32_t *err) {
  const int32_t *cur = (const int32_t *)in;
  int32_t *next = (int32_t *)out;
  constexpr int NC = 32, NR = R * NWC;
  extern __shared__ __align__(1024) uint32_t buf[];  // 3 x NR x NC packed words
  __shared__ uint32_t spop[32];
  __shared__ int4 nib[16];  // nibble -> its four cells
  __shared__ uint64_t bars[NWP][NS];
  __shared__ uint64_t cbar[PS ? NWC : 1][2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 16) nib[tid] = make_int4(tid & 1, (tid >> 1) & 1, (tid >> 2) & 1, (tid >> 3) & 1);
  const int kk = p.kk;
  const int ntiles = p.nt0 * p.nt1;
  const int m = ntiles > (int)blockIdx.x ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  if (tid < 32) spop[tid] = 0;
  if (TMA && tid < NS * NWP) {
    tma::mbar_init(&bars[tid / NS][tid % NS], 1);
    tma::fence_mbar_init();
  }
  if (PS && tid < 2 * NWC) tma::mbar_init(&cbar[tid >> 1][tid & 1], 1);
  // consumer generations so far (all tiles): generation G exchanges through
  // buffer G & 1, and is use G >> 1 of that buffer's mbarriers
  uint32_t G = 0;
  __syncthreads();
  constexpr int NWT = NWC + NWP + NWS;
  // write back the owned words of tile t from shared-memory buffer A, by
  // warps sw .. of nsw
  auto store_tile = [&](int t, const uint32_t *A, int sw, int nsw) {
    const int col0 = (t % p.nt0) * p.tw, row0 = (t / p.nt0) * p.th;
    const int tw_own = min(p.tw, p.wd - col0), th_own = min(p.th, p.n1 - row0);
    const int sub = lane >> 3, quad = (lane & 7) * 4;
    if (IO == kCellsToPacked) {
      for (int r = sw; r < th_own; r += nsw)
        if (lane < tw_own)
          ((uint32_t *)out)[(size_t)(row0 + r) * p.wd + col0 + lane] = A[(r + kk) * NC + 1 + lane];
      return;
    }
    for (int r = sw; r < th_own; r += nsw) {
      const uint32_t *src = A + (r + kk) * NC + 1;
      int32_t *dst = next + (size_t)(row0 + r) * p.n0 + (size_t)col0 * 32 + quad;
      for (int c0 = 0; c0 < tw_own; c0 += 16) {
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          const int cw = c0 + 4 * gq + sub;
          if (cw < tw_own)
            *reinterpret_cast<int4 *>(dst + (size_t)cw * 32) = nib[(src[cw] >> quad) & 15u];
        }
      }
    }
  };
  auto pack_tile = [&](int s, int pw, int npw) {
    const int t = blockIdx.x + s * gridDim.x;
    const int col0 = (t % p.nt0) * p.tw, row0 = (t / p.nt0) * p.th;
    if (IO == kPackedToCells) {
      const uint32_t *src =
          (const uint32_t *)in + ext_word(min(col0 - 1 + lane, p.wd), p.wd, 32).o0;
      uint32_t *dst = buf + (s % 3) * NR * NC + lane;
      for (int r0 = pw; r0 < NR; r0 += 4 * npw) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          int gy = (row0 - kk + min(r0 + k * npw, NR - 1)) % p.n1;
          if (gy < 0) gy += p.n1;
          w[k] = src[(size_t)gy * p.wd];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (r0 + k * npw < NR) dst[(r0 + k * npw) * NC] = w[k];
      }
      return;
    }
    pack_rows32(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, NR, buf + (s % 3) * NR * NC, pw,
                npw, lane);
  };
  // TMA slots: after the three tile buffers, 1024-byte aligned (the
  // swizzle's period), NS 4 KB slots per producer warp, then NS 128-byte
  // slots per producer warp for the wrapped halo word
  unsigned char *slots = nullptr, *patches = nullptr;
  if (TMA) {
    unsigned char *after = reinterpret_cast<unsigned char *>(buf + 3 * NR * NC);
    slots = after + ((1024u - (tma::smem_addr(after) & 1023u)) & 1023u);
    patches = slots + (size_t)NWP * NS * 4096;
  }
  // rows this producer warp has packed so far; its rows run pw, pw + NWP,
  // ... of tile 1, then of tile 2, ..., and box q of that sequence goes
  // into slot q mod NS
  uint32_t seq = 0;
  // lane whose word wraps around in tile column col0 (-1: none): lane 0
  // holds word -1 in the first column, lane wd - col0 + 1 word wd in the last
  auto wrap_lane = [&](int col0) {
    if (col0 == 0) return 0;
    const int sr = p.wd - col0 + 1;
    return sr <= 31 ? sr : -1;
  };
  auto row_issue = [&](int s, int r, uint32_t q) {
    const int t = blockIdx.x + s * gridDim.x;
    const int col0 = (t % p.nt0) * p.tw, row0 = (t / p.nt0) * p.th;
    int gy = (row0 - kk + r) % p.n1;
    if (gy < 0) gy += p.n1;
    if (lane == 0) {
      const int pw = warp - NWC;
      const int slot = pw * NS + (int)(q % NS);
      uint64_t *bar = &bars[pw][q % NS];
      const int wl = wrap_lane(col0);
      tma::mbar_arrive_expect_tx(bar, wl >= 0 ? 4096 + 128 : 4096);
      tma::load_3d(slots + (size_t)slot * 4096, &tmap, 0, col0 - 1, gy, bar);
      if (wl >= 0)
        tma::load_3d(patches + (size_t)slot * 128, &tpatch, 0, wl == 0 ? p.wd - 1 : 0, gy, bar);
    }
  };
  auto row_pack = [&](int s, int r, uint32_t q) {
    const int t = blockIdx.x + s * gridDim.x;
    const int col0 = (t % p.nt0) * p.tw;
    const int pw = warp - NWC;
    const int slot = pw * NS + (int)(q % NS);
    tma::mbar_wait(&bars[pw][q % NS], (q / NS) & 1, err);
    const bool patched = lane == wrap_lane(col0);
    const unsigned char *line =
        patched ? patches + (size_t)slot * 128 : slots + (size_t)slot * 4096 + lane * 128;
    const int x7 = patched ? 0 : (lane & 7);
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int4 c = *reinterpret_cast<const int4 *>(line + ((j ^ x7) << 4));
      w += ((uint32_t)c.x << (4 * j)) + ((uint32_t)c.y << (4 * j + 1)) +
           ((uint32_t)c.z << (4 * j + 2)) + ((uint32_t)c.w << (4 * j + 3));
    }
    buf[(s % 3) * NR * NC + r * NC + lane] = w;
    // the slot's reads are done before the next box into it is issued
    tma::fence_proxy_async();
    __syncwarp();
  };
  // the producers' staging rows follow the three tile buffers
  int4 *stage = reinterpret_cast<int4 *>(buf + 3 * NR * NC);
  auto pack_tile_async = [&](int s, int pw) {
    const int t = blockIdx.x + s * gridDim.x;
    const int col0 = (t % p.nt0) * p.tw, row0 = (t / p.nt0) * p.th;
    pack_rows32_async(cur, p.n0, p.n1, p.wd, row0 - kk, col0 - 1, NR, buf + (s % 3) * NR * NC,
                      pw, NWP, lane, stage + pw * 512);
  };
  // Stage 0 only packs and stage m + 1 only stores: there every warp of the
  // block takes part; in stage m the producers, with no tile left to pack,
  // help the store warps.
  for (int s = 0; s < m + 2; ++s) {
    if (s == 0) {
      if (m > 0) pack_tile(0, warp, NWT);
    } else if (s == m + 1) {
      if (m > 0) store_tile(blockIdx.x + (s - 2) * gridDim.x, buf + ((s - 2) % 3) * NR * NC, warp, NWT);
    } else if (warp < NWC) {
      {
        // consumers: advance tile s-1
        const int t = blockIdx.x + (s - 1) * gridDim.x;
        const int col0 = (t % p.nt0) * p.tw, row0 = (t / p.nt0) * p.th;
        const int tw_own = min(p.tw, p.wd - col0), th_own = min(p.th, p.n1 - row0);
        uint32_t *A = buf + ((s - 1) % 3) * NR * NC;
        uint32_t rows[R];
#pragma unroll
        for (int i = 0; i < R; ++i) rows[i] = A[(warp * R + i) * NC + lane];
        // while the rows are in registers their buffer holds the exchange
        static_assert(R >= 8, "the exchange fits in the tile's buffer");
        uint2(*ex)[NWC][2][NC] = reinterpret_cast<uint2(*)[NWC][2][NC]>(A);
        asm volatile("bar.sync 1, %0;" ::"r"(NWC * 32) : "memory");
        uint32_t ownrows = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int gr = warp * R + i - kk;
          if (gr >= 0 && gr < th_own) ownrows |= 1u << i;
        }
        const uint32_t colmask = (lane >= 1 && lane <= tw_own) ? ~0u : 0u;
        constexpr uint32_t allrows = R == 32 ? ~0u : ((1u << R) - 1u);
        const bool whole = ownrows == allrows || ownrows == 0u;
        for (int g = 0; g < kk; ++g) {
          const int b = PS ? (int)(G & 1u) : (g & 1);
          auto arrive = [&] {
            // A neighbour is at most one use ahead on a buffer: to arrive
            // again it must first see this warp's next generation.  It
            // reads a buffer before it signals the next generation, so
            // this warp's rewrite two generations on cannot overtake it.
            if (PS) {
              __syncwarp();
              if (lane == 0) tma::mbar_arrive(&cbar[warp][b]);
            }
          };
          auto wait = [&] {
            if (PS) {
              const uint32_t par = (G >> 1) & 1u;
              if (warp > 0) tma::mbar_wait(&cbar[warp - 1][b], par, err);
              if (warp < NWC - 1) tma::mbar_wait(&cbar[warp + 1][b], par, err);
              ++G;
            } else {
              asm volatile("bar.sync 1, %0;" ::"r"(NWC * 32) : "memory");
            }
          };
          uint32_t cnt;
          if (whole)
            cnt = life_generation<R, NWC>(rows, ex[b], warp, lane, true, ownrows, colmask, arrive,
                                          wait) &
                  (ownrows == allrows ? colmask : 0u);
          else
            cnt = life_generation<R, NWC>(rows, ex[b], warp, lane, false, ownrows, colmask,
                                          arrive, wait);
          cnt = __reduce_add_sync(0xffffffffu, cnt);
          if (lane == 0 && cnt) atomicAdd(&spop[g], cnt);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(NWC * 32) : "memory");
#pragma unroll
        for (int i = 0; i < R; ++i) A[(warp * R + i) * NC + lane] = rows[i];
      }
    } else if (warp < NWC + NWP) {
      if (s < m)
        if (IO == kPackedToCells) {
          pack_tile(s, warp - NWC, NWP);
        } else if (TMA) {
          // rows pw, pw + NWP, ... of tile s, NS - 1 boxes ahead (the first
          // rows of tile s + 1 follow the last of tile s); a slot is issued
          // into only after the row it held was packed
          const int pw = warp - NWC;
          if (s == 1) {  // the sequence's first NS - 1 boxes
            int nr = pw, ns = 1;
            for (int k = 0; k < NS - 1 && ns < m; ++k) {
              row_issue(ns, nr, (uint32_t)k);
              nr += NWP;
              if (nr >= NR) {
                nr = pw;
                ++ns;
              }
            }
          }
          for (int r = pw; r < NR; r += NWP) {
            // the row NS - 1 places further on in the sequence
            int nr = r, ns = s;
#pragma unroll
            for (int k = 0; k < NS - 1; ++k) {
              nr += NWP;
              if (nr >= NR) {
                nr = pw;
                ++ns;
              }
            }
            if (ns < m) row_issue(ns, nr, seq + NS - 1);
            row_pack(s, r, seq);
            ++seq;
          }
        } else if (kStagedPack<R, NWC, NWP>())
          pack_tile_async(s, warp - NWC);
        else
          pack_tile(s, warp - NWC, NWP);
      else if (s >= 2)  // s == m
        store_tile(blockIdx.x + (s - 2) * gridDim.x, buf + ((s - 2) % 3) * NR * NC, warp - NWC,
                   NWP + NWS);
    } else if (s >= 2) {
      // store warps: write back tile s - 2
      const bool helped = s == m;
      store_tile(blockIdx.x + (s - 2) * gridDim.x, buf + ((s - 2) % 3) * NR * NC,
                 helped ? warp - NWC : warp - NWC - NWP, helped ? NWP + NWS : NWS);
    }
    __syncthreads();
  }
  if (tid < kk && spop[tid]) atomicAdd(&pop[tid], spop[tid]);
}

__global__ void life_fill_kernel(int32_t *cell, int n0, int n1, int ms0, int lm,
                                 uint64_t seed_mix, uint64_t thr) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t total = (size_t)n0 * n1;
  if (i >= total) return;
  const size_t y = i / n0, x = i - y * n0;
  const uint64_t h = mix64(seed_mix + (uint64_t)i * 0x9E3779B97F4A7C15ULL);
  cell[(y + lm) * ms0 + (x + lm)] = ((h >> 11) < thr) ? 1 : 0;
}

__global__ void life_reset_kernel(LifeScalars *s) { *s = LifeScalars{}; }

// The run's results into the host block; hist (n <= kHistory): the populations,
// which are cleared for the next run.
__global__ void __launch_bounds__(256)
life_finalize_kernel(LifeScalars *s, uint32_t *hist, uint32_t *pop, uint32_t *wait, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    if (!hist && i != n - 1) continue;
    const uint32_t c = pop[i];
    if (i == n - 1) {
      s->population = (int32_t)c;
      s->generation = (int32_t)((uint32_t)s->generation + (uint32_t)n);
      if (*wait) {
        s->wait_error = 1;
        *wait = 0;
      }
    }
    if (hist) {
      hist[i] = c;
      pop[i] = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

// The small kernel's variants (rows per lane).
static const int kSmallRows[] = {2, 3, 4, 5, 6, 8};
static const int kNumSmallRows = 6;

typedef void (*SmallKernel)(const int32_t *, int32_t *, SmallParams, uint32_t *, LifeScalars *,
                            uint32_t *);
template <bool RAG> static SmallKernel small_kernel(int v) {
  switch (v) {
    case 0: return life_smallreg_kernel<2, RAG>;
    case 1: return life_smallreg_kernel<3, RAG>;
    case 2: return life_smallreg_kernel<4, RAG>;
    case 3: return life_smallreg_kernel<5, RAG>;
    case 4: return life_smallreg_kernel<6, RAG>;
    default: return life_smallreg_kernel<8, RAG>;
  }
}

// The small kernel's plan for a grid: variant, warps and halo of least modelled
// cycles per generation (nw 0: no plan fits).  The model follows 128^2 on
// GB300, where 2 rows x 12 warps take 362 cycles a generation, 2 x 16 390,
// 3 x 8 402, 5 x 4 405, 4 x 8 490, 8 x 4 580 and 3 x 16 560 (one word a thread
// in 16 warps with an exchange every generation: 440).
struct SmallPlan {
  int v, nw, h;
  double cycles;
};
static SmallPlan small_plan(int n0, int n1) {
  SmallPlan best{0, 0, 0, 0};
  const int wd = (n0 + 31) / 32;
  if (wd > 32 || n1 > 2048) return best;
  for (int v = 0; v < kNumSmallRows; ++v) {
    const int R = kSmallRows[v], rows = (32 / wd) * R;
    for (int nw = 1; nw <= kSmallThreads / 32 && nw <= n1; ++nw) {
      const int own = (n1 + nw - 1) / nw, h = (rows - own) / 2;
      if (h < 1) continue;
      const double c = (40.0 + 38.0 * R * ((nw + 3) / 4) + 30.0 * R + 60.0 / h) *
                       (n0 % 32 ? 1.2 : 1.0);
      if (best.nw == 0 || c < best.cycles) best = SmallPlan{v, nw, h, c};
    }
  }
  return best;
}
// Whether a grid runs in one CTA: the small kernel's cycles per generation
// against the packed tiles' (about 1000 at least, with launches, packing and
// unpacking around them).
static bool life_small(const Handle *h) {
  const SmallPlan pl = small_plan(h->size[0], h->size[1]);
  return pl.nw > 0 && pl.cycles < 1000.0;
}

// whether packed kernels serve the grid: every cell 0 or 1, cyclic, rows of
// whole words or of at least one word and a cell
static bool life_packed_ok(const Handle *h) {
  return h->cyclic && h->cfg.variant == 0 &&
         (h->size[0] % 32 == 0 || h->size[0] > 32 || life_small(h));
}

// Launch knobs (om_config depth, tile_x, tile_y, life_kernel) apply to grids of
// more than this many packed words; smaller ones run on whatever fits them.
static const long long kKnobWords = 4096;
static bool life_knobs(const Handle *h) {
  const om_config &c = h->cfg;
  return (long long)((h->size[0] + 31) / 32) * h->size[1] > kKnobWords &&
         (c.depth != 0 || c.tile_x != 0 || c.tile_y != 0 || c.life_kernel != 0 || c.life_io != 0 ||
          c.grid_limit != 0);
}

// Whether a run of n generations goes through the packed grid: rows that are
// no whole number of words from two generations on (a single one is cheaper
// one cell per thread than packed, advanced and unpacked), others with no
// launch knob set, when one launch of at most 32 generations cannot do.
static bool life_run_packed(const Handle *h, int n) {
  if (!life_packed_ok(h) || life_small(h)) return false;
  if (h->size[0] % 32 != 0) return n >= 2;
  return n > 32 && !life_knobs(h);
}

static om_status life_reserve(Handle *h, int kernel_id, int n) {
  LifeState *st = life_state(h);
  if (h->kernels[kernel_id].name == "proceed" && !st->packed[0] && !st->packed_refused &&
      life_run_packed(h, n)) {
    const size_t words = (size_t)((h->size[0] + 31) / 32) * h->size[1];
    for (int i = 0; i < 2 && !st->packed_refused; ++i)
      st->packed_refused = injected_alloc_failure() ||
                           cudaMalloc(&st->packed[i], words * sizeof(uint32_t)) != cudaSuccess;
    if (st->packed_refused) {  // 1/16 more than the cells take: the run goes without
      cudaGetLastError();
      cudaFree(st->packed[0]);
      st->packed[0] = st->packed[1] = nullptr;
    }
  }
  if (n <= st->pop_cap) return OM_OK;
  int cap = std::max(n, kHistory);
  uint32_t *p = nullptr;
  if (cudaMalloc(&p, (size_t)cap * sizeof(uint32_t)) != cudaSuccess) {
    cudaGetLastError();
    set_error("Life: cannot allocate the population history");
    return OM_ERR_NOMEM;
  }
  OM_CUDA_CHECK(cudaStreamSynchronize(h->stream));
  if (st->d_pop) {
    cudaFree(st->d_pop);
    h->replaced++;
  }
  st->d_pop = p;
  st->pop_cap = cap;
  st->pop_clear = false;
  return OM_OK;
}

static om_status life_init(Handle *h, int n) {
  (void)n;
  Array &a = h->arrays[0];
  OM_CUDA_CHECK(cudaMemsetAsync(a.d(), 0, a.count * sizeof(int32_t), h->stream));
  life_reset_kernel<<<1, 1, 0, h->stream>>>((LifeScalars *)h->d_scalars);
  OM_CUDA_CHECK(cudaGetLastError());
  life_state(h)->binary = true;
  life_state(h)->last_n = 0;
  return OM_OK;
}

// Register-resident kernel variants: R rows per warp x NW warps per block.
struct RegVariant {
  int R, NW;
};
static const RegVariant kRegVariants[] = {{16, 8}, {24, 8}, {16, 16}, {32, 8}, {24, 16}, {32, 16}};
static const int kNumRegVariants = 6;

template <bool VEC>
static cudaError_t launch_reg(int v, const int32_t *cur, int32_t *next, const TbParams &p,
                              uint32_t *pop, cudaStream_t s) {
  const RegVariant rv = kRegVariants[v];
  const size_t smem = sizeof(uint32_t) * 32 * rv.R * rv.NW;
  void (*k)(const void *, void *, TbParams, uint32_t *) = nullptr;
  switch (v) {
    case 0: k = life_reg_kernel<16, 8, VEC>; break;
    case 1: k = life_reg_kernel<24, 8, VEC>; break;
    case 2: k = life_reg_kernel<16, 16, VEC>; break;
    case 3: k = life_reg_kernel<32, 8, VEC>; break;
    case 4: k = life_reg_kernel<24, 16, VEC>; break;
    default: k = life_reg_kernel<32, 16, VEC>; break;
  }
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<p.nt0 * p.nt1, rv.NW * 32, smem, s>>>(cur, next, p, pop);
  return cudaGetLastError();
}

// warp-specialised variants: R rows x NWC consumer warps, NWP producer and
// NWS store warps, one CTA per SM
struct WsVariant {
  int R, NWC, NWP, NWS;
  bool tma;  // producers take their rows by TMA
  int ns;    // TMA slots per producer warp
  bool ps;   // consumers synchronise with their neighbours only
};
static const WsVariant kWsVariants[] = {
    {24, 16, 8, 8, false, 0}, {16, 16, 8, 8, false, 0}, {24, 16, 12, 4, false, 0},
    {20, 16, 8, 8, false, 0}, {20, 16, 8, 8, true, 2},  {24, 16, 8, 8, true, 2},
    {20, 16, 4, 12, true, 4}, {20, 16, 6, 10, true, 3}, {24, 16, 4, 12, true, 4},
    {21, 16, 8, 8, true, 2},  {22, 16, 8, 8, true, 2},  {21, 16, 8, 8, false, 0},
    {22, 16, 8, 8, false, 0}, {23, 16, 8, 8, true, 2},  {22, 16, 8, 8, true, 2, true},
    {20, 16, 8, 8, true, 2, true}};
static const int kNumWsVariants = 16;
// the variant the automatic choice takes when TMA serves the grid (rows of
// at least 32 words; fastest on GB300 at 16384^2: 22 rows per consumer warp
// give 990 tiles, at most 7 per SM, where 20 rows give 1098, at most 8),
// else the staged-copy one
static const int kAutoWsVariantTma = 10;
static const int kAutoWsVariant = 3;

// `tmap`, `tpatch`: the tensor maps of `cur` for the TMA variants (ignored
// by the others); at most `ctas` persistent CTAs
// io: kCellsToCells, or the first or last launch of a packed run (automatic
// variants only)
static cudaError_t launch_ws(int v, int io, const void *cur, void *next, const TbParams &p,
                             uint32_t *pop, int ctas, const CUtensorMap &tmap,
                             const CUtensorMap &tpatch, uint32_t *err, cudaStream_t s) {
  const WsVariant wv = kWsVariants[v];
  size_t smem = sizeof(uint32_t) * 3 * 32 * wv.R * wv.NWC;
  if (wv.tma) {
    // three tile buffers, alignment slack, ns 4 KB TMA slots and ns
    // 128-byte wrapped-word slots per producer warp
    smem += 1024 + (size_t)(4096 + 128) * wv.ns * wv.NWP;
  } else if (3 * 4 * 32 * wv.R * wv.NWC + 8192 * wv.NWP <= 212992) {
    // three tile buffers, then two staged rows (2 x 4 KB) per producer warp
    smem += sizeof(int4) * 512 * wv.NWP;
  }
  void (*k)(const void *, void *, TbParams, uint32_t *, const CUtensorMap, const CUtensorMap,
            uint32_t *) = nullptr;
  if (io == kCellsToPacked)
    k = v == kAutoWsVariantTma ? life_ws_kernel<22, 16, 8, 8, true, 2, false, kCellsToPacked>
                               : life_ws_kernel<20, 16, 8, 8, false, 2, false, kCellsToPacked>;
  else if (io == kPackedToCells)
    k = v == kAutoWsVariantTma ? life_ws_kernel<22, 16, 8, 8, true, 2, false, kPackedToCells>
                               : life_ws_kernel<20, 16, 8, 8, false, 2, false, kPackedToCells>;
  else switch (v) {
    case 0: k = life_ws_kernel<24, 16, 8, 8>; break;
    case 1: k = life_ws_kernel<16, 16, 8, 8>; break;
    case 2: k = life_ws_kernel<24, 16, 12, 4>; break;
    case 3: k = life_ws_kernel<20, 16, 8, 8>; break;
    case 4: k = life_ws_kernel<20, 16, 8, 8, true, 2>; break;
    case 5: k = life_ws_kernel<24, 16, 8, 8, true, 2>; break;
    case 6: k = life_ws_kernel<20, 16, 4, 12, true, 4>; break;
    case 7: k = life_ws_kernel<20, 16, 6, 10, true, 3>; break;
    case 8: k = life_ws_kernel<24, 16, 4, 12, true, 4>; break;
    case 9: k = life_ws_kernel<21, 16, 8, 8, true, 2>; break;
    case 10: k = life_ws_kernel<22, 16, 8, 8, true, 2>; break;
    case 11: k = life_ws_kernel<21, 16, 8, 8>; break;
    case 12: k = life_ws_kernel<22, 16, 8, 8>; break;
    case 13: k = life_ws_kernel<23, 16, 8, 8, true, 2>; break;
    case 14: k = life_ws_kernel<22, 16, 8, 8, true, 2, true>; break;
    default: k = life_ws_kernel<20, 16, 8, 8, true, 2, true>; break;
  }
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int ntiles = p.nt0 * p.nt1;
  const int grid = ntiles < ctas ? ntiles : ctas;
  k<<<grid, (wv.NWC + wv.NWP + wv.NWS) * 32, smem, s>>>(cur, next, p, pop, tmap, tpatch, err);
  return cudaGetLastError();
}

// Resident blocks per SM of a register variant (queried once per device;
// handles on other host threads may ask at the same time).
static int reg_occupancy(int device, int v, bool vec) {
  static std::atomic<int> cache[64][kNumRegVariants][2];
  if (device < 0 || device >= 64) return 1;
  std::atomic<int> &c = cache[device][v][vec ? 1 : 0];
  const int known = c.load(std::memory_order_relaxed);
  if (known) return known;
  const RegVariant rv = kRegVariants[v];
  const size_t smem = sizeof(uint32_t) * 32 * rv.R * rv.NW;
  void (*k)(const void *, void *, TbParams, uint32_t *) = nullptr;
  switch (v) {
    case 0: k = vec ? life_reg_kernel<16, 8, true> : life_reg_kernel<16, 8, false>; break;
    case 1: k = vec ? life_reg_kernel<24, 8, true> : life_reg_kernel<24, 8, false>; break;
    case 2: k = vec ? life_reg_kernel<16, 16, true> : life_reg_kernel<16, 16, false>; break;
    case 3: k = vec ? life_reg_kernel<32, 8, true> : life_reg_kernel<32, 8, false>; break;
    case 4: k = vec ? life_reg_kernel<24, 16, true> : life_reg_kernel<24, 16, false>; break;
    default: k = vec ? life_reg_kernel<32, 16, true> : life_reg_kernel<32, 16, false>; break;
  }
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, rv.NW * 32, smem) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = 1;
  }
  c.store(n, std::memory_order_relaxed);
  return n;
}

// Launch plan for the register kernel: the variant and tile grid (nt0 x nt1,
// tiles split evenly).  The kernel is issue-bound and a warp issues for all
// 32 lanes however many words its tile owns, so a block costs its rows
// (NR) whatever its width.  The plan minimises the rows the busiest SM
// issues (ceil(tiles / SMs) x NR), then the rows issued in all (tiles x
// NR).  The 32-row variants need more than the 64 registers a thread has
// at their occupancy and spill: the plan leaves them out.  Returns the
// variant.
static int reg_plan(int device, bool vec, int wd, int n1, int kk, int *nt0_out, int *nt1_out) {
  const int sms = sm_count(device);
  double best_cost = 1e300, best_work = 1e300;
  int best_v = 1, best0 = (wd + 29) / 30, best1 = 1;
  for (int v = 0; v < kNumRegVariants; ++v) {
    if (kRegVariants[v].R > 24) continue;
    const int NR = kRegVariants[v].R * kRegVariants[v].NW;
    const int thm = NR - 2 * kk;
    if (thm < 8) continue;
    if (reg_occupancy(device, v, vec) < 1) continue;
    const int nt0min = (wd + 29) / 30;
    const int nt1min = (n1 + thm - 1) / thm;
    for (int nt0 = nt0min; nt0 <= nt0min + 2 && nt0 <= wd; ++nt0)
      for (int nt1 = nt1min; nt1 <= nt1min + 24 && nt1 <= n1; ++nt1) {
        const long long tiles = (long long)nt0 * nt1;
        const double cost = (double)((tiles + sms - 1) / sms) * NR;
        const double work = (double)tiles * NR;
        if (cost < best_cost - 1e-9 || (cost < best_cost + 1e-9 && work < best_work - 1e-9)) {
          best_cost = cost;
          best_work = work;
          best_v = v;
          best0 = nt0;
          best1 = nt1;
        }
      }
  }
  *nt0_out = best0;
  *nt1_out = best1;
  return best_v;
}

// Variants of the register kernel with a packed end or two (R rows x NW
// warps): short blocks let a grid of a few million cells spread over every SM
// (2048^2 x 100: 126-128 us with 64- to 128-row blocks, 168 with 192 rows, 230
// with 320), tall ones waste less on halo rows where tiles are many (16384^2:
// 1936 us with 64 rows, 1290 with 192, 1176 with 384).
static const RegVariant kPackedVariants[] = {{4, 16}, {6, 16}, {8, 16}, {12, 16},
                                             {16, 16}, {20, 16}, {24, 16}, {8, 8}};
static const int kNumPackedVariants = 8;

typedef void (*RegKernel)(const void *, void *, TbParams, uint32_t *);
template <int IO> static RegKernel packed_kernel(int v) {
  switch (v) {
    case 0: return life_reg_kernel<4, 16, true, IO>;
    case 1: return life_reg_kernel<6, 16, true, IO>;
    case 2: return life_reg_kernel<8, 16, true, IO>;
    case 3: return life_reg_kernel<12, 16, true, IO>;
    case 4: return life_reg_kernel<16, 16, true, IO>;
    case 5: return life_reg_kernel<20, 16, true, IO>;
    case 6: return life_reg_kernel<24, 16, true, IO>;
    default: return life_reg_kernel<8, 8, true, IO>;
  }
}
static RegKernel packed_kernel(int v, int io) {
  return io == kCellsToPacked   ? packed_kernel<kCellsToPacked>(v)
         : io == kPackedToCells ? packed_kernel<kPackedToCells>(v)
                                : packed_kernel<kPackedToPacked>(v);
}
static size_t packed_smem(int v, int io) {
  return io == kPackedToPacked
             ? 0
             : sizeof(uint32_t) * 32 * kPackedVariants[v].R * kPackedVariants[v].NW;
}

// resident blocks per SM of a packed variant (queried once per device)
static int packed_occupancy(int device, int v, int io) {
  static std::atomic<int> cache[64][kNumPackedVariants][4];
  if (device < 0 || device >= 64) return 1;
  std::atomic<int> &c = cache[device][v][io];
  const int known = c.load(std::memory_order_relaxed);
  if (known) return known;
  const RegKernel k = packed_kernel(v, io);
  const size_t smem = packed_smem(v, io);
  int n = 0;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kPackedVariants[v].NW * 32, smem) !=
          cudaSuccess ||
      n < 1) {
    cudaGetLastError();
    n = 1;
  }
  c.store(n, std::memory_order_relaxed);
  return n;
}

// A launch of the packed register kernel: variant, generations, tile grid.
struct PackedPlan {
  int v, kk, nt0, nt1;
  double cycles;  // of the model below
  double rate() const { return cycles / kk; }
};

// The plan of least modelled time over depths kmin .. kmax: per generation
// (rate 0), or, for a run's first and last launch, beyond what its generations
// would take at `rate` cycles each between them.
// Per generation a block keeps a sub-partition's ALU busy for 22 cycles per
// row of each of its warps (nine bit operations and two shifts at 16 lanes a
// cycle), about two rows' worth for the exchanged rows and 40 for the count; a
// block alone on its SM also waits about 250 for the exchange.  A launch costs
// about 4000 cycles before and after, the packed rows' load and store 1500 a
// round, and cells that are read or written 4 KB a row at about 48 bytes a
// cycle.
static PackedPlan packed_plan(int device, int wd, int n1, int io, int kmin, int kmax,
                              double rate = 0) {
  const int sms = sm_count(device);
  PackedPlan best{-1, 1, 1, 1, 0};
  double best_cost = 1e300;
  for (int v = 0; v < kNumPackedVariants; ++v) {
    const RegVariant rv = kPackedVariants[v];
    const int NR = rv.R * rv.NW;
    const int occ = packed_occupancy(device, v, io);
    const double alu = rv.NW * ((rv.R + 2) * 22.0 + 40.0) / 4.0;
    for (int kk = kmin; kk <= kmax; ++kk) {
      const int thm = NR - 2 * kk;
      if (thm < 4) break;
      const int nt0min = (wd + 29) / 30, nt1min = (n1 + thm - 1) / thm;
      for (int nt0 = nt0min; nt0 <= nt0min + 1 && nt0 <= wd; ++nt0) {
        const long long tiles = (long long)nt0 * nt1min;
        const long long per = (tiles + sms - 1) / sms;
        const long long rounds = (per + occ - 1) / occ;
        const double c = (double)std::min<long long>(per, occ);
        double gen = std::max(c * alu, alu + 250.0) * (double)(per / occ);
        if (per % occ) gen += std::max((double)(per % occ) * alu, alu + 250.0);
        double cyc = 4000.0 + kk * gen + 1500.0 * (double)rounds;
        if (io != kPackedToPacked) {
          const int rows = (n1 + nt1min - 1) / nt1min + (io == kCellsToPacked ? 2 * kk : 0);
          cyc += (double)per * rows * 4096.0 / 48.0;
        }
        const double cost = rate > 0 ? cyc - kk * rate : cyc / kk;
        if (cost < best_cost) {
          best_cost = cost;
          best = PackedPlan{v, kk, nt0, nt1min, cyc};
        }
      }
    }
  }
  return best;
}

static om_status launch_packed(Handle *h, const PackedPlan &pl, int io, const void *in, void *out,
                               TbParams p, uint32_t *pop) {
  p.kk = pl.kk;
  p.nt0 = pl.nt0;
  p.nt1 = pl.nt1;
  const RegKernel k = packed_kernel(pl.v, io);
  const size_t smem = packed_smem(pl.v, io);
  OM_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaEvent_t ev = prof_begin(h);
  k<<<pl.nt0 * pl.nt1, kPackedVariants[pl.v].NW * 32, smem, h->stream>>>(in, out, p, pop);
  OM_CUDA_CHECK(cudaGetLastError());
  prof_end(h, ev, io == kPackedToPacked ? "life_packed_kernel" : "life_reg_kernel",
           (double)p.n0 * p.n1 * pl.kk);
  h->launches++;
  return OM_OK;
}

// register variant for kk generations: the smallest block whose owned rows
// (block rows - 2kk) reach the requested tile height (default 320, the
// 24-row x 16-warp block at depth 32: fastest in the GB300 tile sweep)
static int reg_variant(int kk, int want_th) {
  const int want = want_th > 0 ? want_th : 320;
  int best = -1;
  for (int v = 0; v < kNumRegVariants; ++v) {
    const int th = kRegVariants[v].R * kRegVariants[v].NW - 2 * kk;
    if (th >= want) { best = v; break; }
    if (th >= 1) best = v;
  }
  return best < 0 ? kNumRegVariants - 1 : best;
}

// Tile choice: tile_w 0 (default) selects the register-resident kernel,
// 30 the one-lane-per-word shared-memory kernel, other widths the general
// tile kernel.  Depth defaults to 32 generations per launch.
static bool life_pick_tiles(Handle *h, TbParams &p, bool knobs) {
  LifeState *st = life_state(h);
  const bool lane_per_word = !knobs || st->tile_w == 0 || st->tile_w == 30;
  p.kk = knobs && st->depth > 0 ? std::min(st->depth, 32) : 32;
  p.tw = lane_per_word ? 30 : st->tile_w;
  p.th = st->tile_h > 0 ? st->tile_h : 128;
  p.tw = std::min(p.tw, p.wd);
  p.th = std::min(p.th, p.n1);
  return lane_per_word;
}

static size_t tb_smem_bytes(const TbParams &p, bool lane_per_word) {
  const int nc = lane_per_word ? 32 : p.tw + 2;
  return 2 * sizeof(uint32_t) * (size_t)nc * (p.th + 2 * p.kk);
}

static om_status launch_general(Handle *h, uint32_t *pop) {
  Array &a = h->arrays[0];
  const int ms0 = (int)h->memory_size(0), ms1 = (int)h->memory_size(1);
  const int tiles_x = (ms0 + 31) / 32;
  const size_t blocks = (size_t)tiles_x * ((ms1 + 7) / 8);
  dim3 block(32, 8);
  cudaEvent_t ev = prof_begin(h);
  if (h->cyclic)
    life_general_kernel<true><<<(unsigned)blocks, block, 0, h->stream>>>(
        (const int32_t *)a.d(), (int32_t *)a.d_next(), ms0, ms1, 0, tiles_x, pop);
  else
    life_general_kernel<false><<<(unsigned)blocks, block, 0, h->stream>>>(
        (const int32_t *)a.d(), (int32_t *)a.d_next(), ms0, ms1, h->lower_margin[0],
        tiles_x, pop);
  OM_CUDA_CHECK(cudaGetLastError());
  prof_end(h, ev, "life_general_kernel", (double)h->size[0] * h->size[1]);
  h->launches++;
  a.swap();
  return OM_OK;
}

// the warp-specialised variant the automatic choice takes for tiles of depth
// kk: on grids of at least 1.5 of its tiles per SM; -1 on smaller ones
static int auto_ws_variant(Handle *h, int wd, int n1, int kk, bool tma_ok) {
  const int av = tma_ok ? kAutoWsVariantTma : kAutoWsVariant;
  const WsVariant wv = kWsVariants[av];
  const int th = std::min(wv.R * wv.NWC - 2 * kk, n1);
  const long long tiles = (long long)((wd + 29) / 30) * ((n1 + th - 1) / th);
  return th > 0 && 2 * tiles >= 3LL * sm_count(h->device) ? av : -1;
}

static om_status launch_ws_tiles(Handle *h, int v, int io, const void *in, void *out, TbParams q,
                                 int mi, uint32_t *pop) {
  LifeState *st = life_state(h);
  const WsVariant wv = kWsVariants[v];
  q.tw = std::min(30, q.wd);
  q.th = std::min(wv.R * wv.NWC - 2 * q.kk, q.n1);
  q.nt0 = (q.wd + q.tw - 1) / q.tw;
  q.nt1 = (q.n1 + q.th - 1) / q.th;
  cudaEvent_t ev = prof_begin(h);
  const int ctas = h->cfg.grid_limit > 0 ? std::min(h->cfg.grid_limit, sm_count(h->device))
                                         : sm_count(h->device);
  cudaError_t e = launch_ws(v, io, in, out, q, pop, ctas, st->tmap[mi < 0 ? 0 : mi],
                            st->tpatch[mi < 0 ? 0 : mi],
                            st->d_flag + 1, h->stream);
  if (e != cudaSuccess) {
    set_error(std::string("life_ws_kernel: ") + cudaGetErrorString(e));
    return OM_ERR_CUDA;
  }
  prof_end(h, ev, wv.tma ? "life_ws_tma_kernel" : "life_ws_kernel",
           (double)q.n0 * q.n1 * q.kk);
  h->launches++;
  return OM_OK;
}

// Generations per launch at the two ends of a packed run on the
// warp-specialised kernel: fewer leave it waiting for the cells' 4 bytes each
// (16384^2 x 100 generations: 1280 us at 8, 1230 at 12, 1176 at 22), more only
// add halo rows (1189 at 26, 1207 at 30).  These and the block heights' figures
// were taken with each row's sums formed alone; shared by two rows
// (life_two_rows), 22 takes 1133.
static const int kWsEdgeDepth = 22;

// Generations g .. n - 1 of a run through the packed grid.  With every launch
// reading and writing int32 cells a 16384^2 run of 100 generations moved 9 GB
// in four launches (1955 us); with the cells read once and written once it
// takes 1133 us, bound by the ALU's bit operations (78 % of its cycles) between
// the ends.  2048^2 x 100: 205 -> 102 us.  Rows of 1000 cells (1000 x 700 x
// 100) no longer take a launch of the one-cell kernel per generation: 496 ->
// 79 us.  A kernel of the warp-specialised form between the ends too was no
// faster (1144 to 1208 us over its row counts, warps and depths).
static om_status proceed_packed(Handle *h, int n, int g) {
  LifeState *st = life_state(h);
  Array &a = h->arrays[0];
  TbParams p{};
  p.n0 = h->size[0];
  p.n1 = h->size[1];
  p.wd = (p.n0 + 31) / 32;
  p.nb = p.n0 - 32 * (p.wd - 1);
  const bool ragged = p.nb != 32;
  uint32_t **pk = st->packed;
  int cur = 0;
  const long long rows8 = (long long)((p.wd + 7) / 8) * p.n1;
  const unsigned io_grid =
      (unsigned)std::max<long long>(1, std::min<long long>((rows8 + 7) / 8, 8LL * sm_count(h->device)));
  int ws = -1, mi = -1, edge = 0;
  PackedPlan first{}, last{};
  if (ragged) {
    cudaEvent_t ev = prof_begin(h);
    life_pack_kernel<<<io_grid, 256, 0, h->stream>>>((const int32_t *)a.d(), pk[0], p.n0, p.n1,
                                                     p.wd);
    OM_CUDA_CHECK(cudaGetLastError());
    prof_end(h, ev, "life_pack_kernel", 0.0);
    h->launches++;
  } else {
    mi = p.wd >= 32 ? life_tmap(st, a.d(), p.n0, p.n1) : -1;
    ws = auto_ws_variant(h, p.wd, p.n1, 32, mi >= 0);
    if (ws >= 0) {
      edge = std::min(kWsEdgeDepth, (n - g) / 2);
      p.kk = edge;
      OM_TRY(launch_ws_tiles(h, ws, kCellsToPacked, a.d(), pk[0], p, mi, st->d_pop + g));
    } else {
      const double rate = packed_plan(h->device, p.wd, p.n1, kPackedToPacked, 4, 32).rate();
      const int most = std::min(24, (n - g) / 2);
      first = packed_plan(h->device, p.wd, p.n1, kCellsToPacked, 1, most, rate);
      last = packed_plan(h->device, p.wd, p.n1, kPackedToCells, 1, most, rate);
      OM_TRY(launch_packed(h, first, kCellsToPacked, a.d(), pk[0], p, st->d_pop + g));
      edge = last.kk;
      g += first.kk - edge;
    }
    g += edge;
  }
  const int rem = n - g - edge;
  if (rem > 0) {
    // launches of near-equal depth, at most the best one
    const int kbest =
        packed_plan(h->device, p.wd, p.n1, kPackedToPacked, std::min(4, rem), std::min(32, rem)).kk;
    const int nl = (rem + kbest - 1) / kbest;
    for (int l = 0; l < nl; ++l) {
      const int kk = rem / nl + (l < rem % nl ? 1 : 0);
      const PackedPlan pl = packed_plan(h->device, p.wd, p.n1, kPackedToPacked, kk, kk);
      OM_TRY(launch_packed(h, pl, kPackedToPacked, pk[cur], pk[1 - cur], p, st->d_pop + g));
      cur = 1 - cur;
      g += kk;
    }
  }
  if (ragged) {
    cudaEvent_t ev = prof_begin(h);
    life_unpack_kernel<<<io_grid, 256, 0, h->stream>>>(pk[cur], (int32_t *)a.d_next(), p.n0, p.n1,
                                                       p.wd);
    OM_CUDA_CHECK(cudaGetLastError());
    prof_end(h, ev, "life_unpack_kernel", 0.0);
    h->launches++;
  } else if (ws >= 0) {
    p.kk = edge;
    OM_TRY(launch_ws_tiles(h, ws, kPackedToCells, pk[cur], a.d_next(), p, -1, st->d_pop + g));
  } else {
    OM_TRY(launch_packed(h, last, kPackedToCells, pk[cur], a.d_next(), p, st->d_pop + g));
  }
  a.swap();
  return OM_OK;
}

// whether a run is one launch of the small kernel, which writes its results too
static bool life_one_launch(const Handle *h, int n) {
  return life_packed_ok(h) && life_small(h) && ((const LifeState *)h->impl)->binary &&
         n <= kHistory;
}

// gens generations of a small grid; populations added to pop, or with hist
// written there with the run's other results (and those of the `before`
// generations in pop)
static om_status launch_small(Handle *h, int gens, uint32_t *pop, uint32_t *hist, int before) {
  Array &a = h->arrays[0];
  const int n0 = h->size[0], n1 = h->size[1];
  const SmallPlan pl = small_plan(n0, n1);
  SmallParams sp{n0, n1, (n0 + 31) / 32, 0, gens, pl.nw, pl.h, before};
  sp.nb = n0 - 32 * (sp.wd - 1);
  const SmallKernel k = n0 % 32 ? small_kernel<true>(pl.v) : small_kernel<false>(pl.v);
  const size_t smem = sizeof(uint32_t) * (2 * (size_t)sp.wd * n1 + gens + 1);
  if (smem > 48 * 1024)
    OM_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaEvent_t ev = prof_begin(h);
  k<<<1, kSmallThreads, smem, h->stream>>>((const int32_t *)a.d(), (int32_t *)a.d_next(), sp, pop,
                                           (LifeScalars *)h->d_scalars, hist);
  OM_CUDA_CHECK(cudaGetLastError());
  prof_end(h, ev, "life_smallreg_kernel", (double)n0 * n1 * gens);
  h->launches++;
  a.swap();
  return OM_OK;
}

static om_status life_proceed(Handle *h, int n) {
  LifeState *st = life_state(h);
  if (n > st->pop_cap) {
    set_error("Life: population history not reserved");
    return OM_ERR_STATE;
  }
  Array &a = h->arrays[0];
  uint32_t *hist = n <= kHistory ? life_history(h) : nullptr;
  const int n0 = h->size[0], n1 = h->size[1];
  const bool ragged = n0 % 32 != 0;
  const bool small = life_small(h);
  // on rows that are no whole number of words, a single generation is cheaper
  // one cell per thread than packed, advanced and unpacked; without memory for
  // the packed grid all of them go so, and runs of whole words go in launches of
  // at most 32 generations
  const bool packed_ok =
      life_packed_ok(h) && (!ragged || small || (n >= 2 && st->packed[0]));
  if (life_one_launch(h, n)) {
    OM_TRY(launch_small(h, n, nullptr, hist, 0));
    st->last_n = n;
    return OM_OK;
  }
  if (!hist || !st->pop_clear)
    OM_CUDA_CHECK(cudaMemsetAsync(st->d_pop, 0, sizeof(uint32_t) * (size_t)std::max(n, kHistory),
                                  h->stream));
  st->pop_clear = false;
  int g = 0;
  if (!packed_ok || !st->binary) {
    const int first = packed_ok ? 1 : n;
    for (; g < first; ++g) OM_TRY(launch_general(h, st->d_pop + g));
    st->binary = true;
  }
  if (g < n && packed_ok && small) {
    if (hist) {
      OM_TRY(launch_small(h, n - g, st->d_pop, hist, g));
      st->pop_clear = true;
      st->last_n = n;
      return OM_OK;
    }
    for (int gens; g < n; g += gens) {
      gens = std::min(n - g, kSmallMaxGens);
      OM_TRY(launch_small(h, gens, st->d_pop + g, nullptr, 0));
    }
  } else if (g < n && (ragged || (st->packed[0] && life_run_packed(h, n - g)))) {
    OM_TRY(proceed_packed(h, n, g));
  } else if (g < n) {
    const int wd = n0 / 32;
    {
      TbParams p;
      p.n0 = n0; p.n1 = n1; p.wd = wd; p.nb = 32;
      const bool knobs = life_knobs(h);
      const bool l32 = life_pick_tiles(h, p, knobs);
      const bool reg = !knobs || st->tile_w == 0;
      const int tile_h = knobs ? st->tile_h : 0;
      const int kmax = p.kk;
      p.nt0 = (p.wd + p.tw - 1) / p.tw;
      p.nt1 = (p.n1 + p.th - 1) / p.th;
      // split the remaining generations into launches of near-equal depth
      const int rem = n - g;
      const int nl = (rem + kmax - 1) / kmax;
      const size_t smem_max = tb_smem_bytes(p, l32);
      const bool vec = h->cfg.life_io != 1;
      auto kern = l32 ? (vec ? life_tb32_kernel<true> : life_tb32_kernel<false>)
                      : (vec ? life_tb_kernel<true> : life_tb_kernel<false>);
      const char *kname = l32 ? "life_tb32_kernel" : "life_tb_kernel";
      if (!reg)
        OM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem_max));
      // the packed kernel: life_kernel >= 1 selects the warp-specialised
      // persistent kernel (variant life_kernel - 1); 0 with no tile shape
      // given takes it too on grids of at least 1.5 of its tiles per SM,
      // where it overlaps one tile's loads and stores with another's
      // generations, and the register-resident blocks on smaller grids
      int ws = knobs ? h->cfg.life_kernel : 0;
      // TMA rows need a grid at least one box (32 words) wide whose buffers
      // the driver describes
      const bool tma_ok = wd >= 32 && life_tmap(st, a.d(), n0, n1) >= 0 &&
                          life_tmap(st, a.d_next(), n0, n1) >= 0;
      if (reg && ws == 0 && tile_h == 0) ws = auto_ws_variant(h, wd, n1, kmax, tma_ok) + 1;
      if (ws >= 1 && kWsVariants[std::min(ws - 1, kNumWsVariants - 1)].tma && !tma_ok) {
        set_error("Life: the TMA kernel variants need rows of at least 1024 cells and a "
                  "tensor map of the grid");
        return OM_ERR_UNSUPPORTED;
      }
      for (int l = 0; l < nl; ++l) {
        const int kk = rem / nl + (l < rem % nl ? 1 : 0);
        p.kk = kk;
        if (reg && ws >= 1) {
          // warp-specialised persistent kernel, variant ws - 1
          const int v = std::min(ws - 1, kNumWsVariants - 1);
          OM_TRY(launch_ws_tiles(h, v, kCellsToCells, a.d(), a.d_next(), p,
                                 kWsVariants[v].tma ? life_tmap(st, a.d(), n0, n1) : -1,
                                 st->d_pop + g));
          a.swap();
          g += kk;
          continue;
        }
        if (reg) {
          TbParams q = p;
          const int v = tile_h > 0 ? reg_variant(kk, tile_h)
                                       : reg_plan(h->device, vec, wd, n1, kk, &q.nt0, &q.nt1);
          if (tile_h > 0) {
            const int thm = std::min(kRegVariants[v].R * kRegVariants[v].NW - 2 * kk, n1);
            q.nt0 = (wd + 29) / 30;
            q.nt1 = (n1 + thm - 1) / thm;
          }
          q.tw = (wd + q.nt0 - 1) / q.nt0;
          q.th = (n1 + q.nt1 - 1) / q.nt1;
          cudaEvent_t ev = prof_begin(h);
          cudaError_t e = vec ? launch_reg<true>(v, (const int32_t *)a.d(), (int32_t *)a.d_next(),
                                                 q, st->d_pop + g, h->stream)
                              : launch_reg<false>(v, (const int32_t *)a.d(),
                                                  (int32_t *)a.d_next(), q, st->d_pop + g,
                                                  h->stream);
          if (e != cudaSuccess) {
            set_error(std::string("life_reg_kernel: ") + cudaGetErrorString(e));
            return OM_ERR_CUDA;
          }
          prof_end(h, ev, "life_reg_kernel", (double)n0 * n1 * kk);
          h->launches++;
          a.swap();
          g += kk;
          continue;
        }
        cudaEvent_t ev = prof_begin(h);
        kern<<<p.nt0 * p.nt1, 256, tb_smem_bytes(p, l32), h->stream>>>(
            (const int32_t *)a.d(), (int32_t *)a.d_next(), p, st->d_pop + g);
        OM_CUDA_CHECK(cudaGetLastError());
        prof_end(h, ev, kname, (double)n0 * n1 * kk);
        h->launches++;
        a.swap();
        g += kk;
      }
    }
  }
  life_finalize_kernel<<<1, 256, 0, h->stream>>>((LifeScalars *)h->d_scalars, hist, st->d_pop,
                                                 st->d_flag + 1, n);
  OM_CUDA_CHECK(cudaGetLastError());
  st->pop_clear = hist != nullptr;
  h->launches++;
  st->last_n = n;
  return OM_OK;
}

static uint64_t life_state_key(Handle *h) {
  const LifeState *st = life_state(h);
  return (st->binary ? 1 : 0) | (st->pop_clear ? 2 : 0);
}

static void life_after_replay(Handle *h, int kernel_id, int n) {
  LifeState *st = life_state(h);
  if (h->kernels[kernel_id].name == "proceed") {
    if (!life_one_launch(h, n)) st->pop_clear = n <= kHistory;
    st->binary = true;
    st->last_n = n;
  } else {
    st->binary = true;
    st->last_n = 0;
  }
}

static void life_restore_key(Handle *h, uint64_t key) {
  LifeState *st = life_state(h);
  st->binary = (key & 1) != 0;
  st->pop_clear = (key & 2) != 0;
}

// New cell contents came from the host.  The packed kernels need every cell
// in {0, 1}; one read-only pass (HBM speed, a fraction of one generation)
// settles that here, outside any stream capture, so that only grids that do
// hold other values pay for a generation of the general integer kernel.
static void life_array_written(Handle *h, Array *a) {
  LifeState *st = life_state(h);
  st->binary = false;
  if (!life_packed_ok(h) || !st->d_flag || h->capturing) return;
  uint32_t bad = 1;
  if (cudaMemsetAsync(st->d_flag, 0, sizeof(uint32_t), h->stream) != cudaSuccess ||
      life_check_cells_into((const int32_t *)a->d(), a->count, st->d_flag, h->stream) !=
          cudaSuccess ||
      cudaMemcpyAsync(&bad, st->d_flag, sizeof(bad), cudaMemcpyDeviceToHost, h->stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(h->stream) != cudaSuccess)
    return;  // binary stays false: the general kernel handles any values
  st->binary = bad == 0;
}

static void life_free(Handle *h) {
  LifeState *st = life_state(h);
  if (st) {
    if (st->d_pop) cudaFree(st->d_pop);
    if (st->d_flag) cudaFree(st->d_flag);
    cudaFree(st->packed[0]);
    cudaFree(st->packed[1]);
    delete st;
  }
  h->impl = nullptr;
}

// Raises *flag when any of the n cells is outside {0, 1}.  128-bit loads when
// the array is 16-byte aligned; a value v is outside {0, 1} iff v & ~1 != 0,
// so the OR of four cells is tested at once.
__global__ void __launch_bounds__(256)
life_check_kernel(const int32_t *__restrict__ cells, size_t n, uint32_t *flag) {
  bool bad = false;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t tail = 0;
  if ((reinterpret_cast<uintptr_t>(cells) & 15) == 0) {
    const int4 *v = reinterpret_cast<const int4 *>(cells);
    const size_t nv = n / 4;
    for (size_t i = i0; i < nv; i += stride) {
      const int4 c = __ldcs(v + i);
      bad |= ((c.x | c.y | c.z | c.w) & ~1) != 0;
    }
    tail = nv * 4;
  }
  for (size_t i = tail + i0; i < n; i += stride) bad |= (cells[i] & ~1) != 0;
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1u);
}

// Launches the cell-value check on stream s (allocates nothing; *flag must
// be cleared by the caller).
cudaError_t life_check_cells_into(const int32_t *cells, size_t n, uint32_t *flag,
                                  cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const size_t want = (n / 4 + 255) / 256;
  const unsigned grid = (unsigned)std::max<size_t>(1, std::min<size_t>(want, 8 * (size_t)sms));
  life_check_kernel<<<grid, 256, 0, s>>>(cells, n, flag);
  return cudaGetLastError();
}

// One launch of the temporally blocked tile kernel from `cur` into `next`
// (cyclic, width % 32 == 0, 1 <= gens <= 32, cells 0/1), with the default
// 32-word x 64-row tiles.  Allocates nothing; used by the caller-buffer
// entry point in life_noalloc.cu.
cudaError_t life_tb_launch_into(const int32_t *cur, int32_t *next, int n0, int n1, int gens,
                                uint32_t *pop, cudaStream_t s) {
  TbParams p;
  p.n0 = n0; p.n1 = n1; p.wd = n0 / 32; p.nb = 32;
  p.kk = gens;
  p.tw = std::min(32, p.wd);
  p.th = std::min(64, n1);
  p.nt0 = (p.wd + p.tw - 1) / p.tw;
  p.nt1 = (p.n1 + p.th - 1) / p.th;
  const size_t smem = tb_smem_bytes(p, false);
  cudaError_t e = cudaFuncSetAttribute(life_tb_kernel<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  life_tb_kernel<false><<<p.nt0 * p.nt1, 256, smem, s>>>(cur, next, p, pop);
  return cudaGetLastError();
}

om_status life_setup(Handle *h) {
  const int lm = h->cyclic ? 0 : 1;  // stencil radius 1 (OMTrans.hs:103-116)
  for (int ax = 0; ax < 2; ++ax) {
    h->lower_margin[ax] = lm;
    h->upper_margin[ax] = lm;
  }
  LifeState *st = new LifeState();
  st->depth = h->cfg.depth;
  st->tile_w = h->cfg.tile_x;
  st->tile_h = h->cfg.tile_y;
  h->impl = st;
  h->impl_free = life_free;
  h->ops.state_key = life_state_key;
  h->ops.after_replay = life_after_replay;
  h->ops.restore_key = life_restore_key;
  h->ops.array_written = life_array_written;
  h->ops.reserve = life_reserve;
  h->ops.after_run = [](Handle *hh) -> om_status {
    LifeScalars *sc = (LifeScalars *)hh->h_scalars;
    if (!sc->wait_error) return OM_OK;
    sc->wait_error = 0;
    set_error("Life: a kernel's bounded wait for its tensor copies ran out; the cells of "
              "this run are unspecified");
    return OM_ERR_CUDA;
  };
  OM_TRY(alloc_array(h, "cell", sizeof(int32_t)));
  if (cudaMalloc(&st->d_flag, 2 * sizeof(uint32_t)) != cudaSuccess) {
    set_error("Life: cannot allocate the cell-value flag");
    return OM_ERR_NOMEM;
  }
  OM_CUDA_CHECK(cudaMemsetAsync(st->d_flag, 0, 2 * sizeof(uint32_t), h->stream));
  h->scalars.push_back({"population", kInt, offsetof(LifeScalars, population)});
  h->scalars.push_back({"generation", kInt, offsetof(LifeScalars, generation)});
  h->scalar_bytes = sizeof(LifeScalars);
  h->result_bytes = kHistory * sizeof(uint32_t);
  h->scalars_on_host = true;
  h->kernels.push_back({"init", life_init});
  h->kernels.push_back({"proceed", life_proceed});
  return OM_OK;
}

}  // namespace om

using namespace om;

extern "C" om_status om_life_fill_random(om_handle H, uint64_t seed, double p) {
  if (!H) { set_error("om_life_fill_random: null handle"); return OM_ERR_ARG; }
  Handle *h = handle_of(H);
  if (h->kind != OM_KIND_LIFE) { set_error("not a Life handle"); return OM_ERR_ARG; }
  if (!(p >= 0.0 && p <= 1.0)) { set_error("p must be in [0,1]"); return OM_ERR_ARG; }
  OM_CUDA_CHECK(cudaSetDevice(h->device));
  Array &a = h->arrays[0];
  OM_CUDA_CHECK(cudaMemsetAsync(a.d(), 0, a.count * sizeof(int32_t), h->stream));
  const uint64_t thr = (uint64_t)floor(p * 9007199254740992.0);
  const size_t total = (size_t)h->size[0] * h->size[1];
  const int block = 256;
  life_fill_kernel<<<(unsigned)((total + block - 1) / block), block, 0, h->stream>>>(
      (int32_t *)a.d(), h->size[0], h->size[1], (int)h->memory_size(0),
      h->lower_margin[0], mix64(seed), thr);
  OM_CUDA_CHECK(cudaGetLastError());
  OM_CUDA_CHECK(cudaStreamSynchronize(h->stream));
  a.newer = a.host ? Newer::kDevice : Newer::kBoth;
  life_state(h)->binary = true;
  return OM_OK;
}

extern "C" om_status om_life_population_history(om_handle H, int32_t *out, int n,
                                                int *written) {
  if (!H || (!out && n > 0)) { set_error("om_life_population_history: null argument"); return OM_ERR_ARG; }
  Handle *h = handle_of(H);
  if (h->kind != OM_KIND_LIFE) { set_error("not a Life handle"); return OM_ERR_ARG; }
  LifeState *st = life_state(h);
  const int m = std::min(n, st->last_n);
  if (m > 0 && st->last_n <= kHistory) {
    std::memcpy(out, life_history(h), (size_t)m * sizeof(int32_t));
  } else if (m > 0) {
    OM_CUDA_CHECK(cudaSetDevice(h->device));
    OM_CUDA_CHECK(cudaMemcpyAsync(out, st->d_pop, (size_t)m * sizeof(int32_t),
                                  cudaMemcpyDeviceToHost, h->stream));
    OM_CUDA_CHECK(cudaStreamSynchronize(h->stream));
  }
  if (written) *written = std::max(m, 0);
  return OM_OK;
}

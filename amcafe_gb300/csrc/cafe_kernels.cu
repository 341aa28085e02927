// CUDA kernels of the CA step (VoxelsCA::UpdateVoxels and TempField::
// AnalyticTempCurr, AMCAFE src/src-mpi/VoxelsCA.C:232-655, TempField.C:139-217)
// and of the per-layer operations (CleanLayer, AddLayer1 Voronoi assignment).
//
// Step pipeline (one realisation, launched by cafe_host.cu on one stream):
//   k_melt          pool box only: SetLiquid3 + BuildjID + "any cell at the
//                   liquidus" flag (VoxelsCA.C:1098-1116, TempField.C:191-206)
//   k_solid2mushy   ConvertSolid1(1) (VoxelsCA.C:780-797), in place
//   k_active_count  \ order-preserving compaction of the active set
//   k_scan_blocks    > (VoxelsCA.C:262-275): mushy, undercooled liquid and
//   k_active_scatter/  their neighbours at/above the liquidus, in index order
//   k_gather        per-position copies, neighbour positions (VoxelsCA.C:
//                   283-335), ruq offsets (VoxelsCA.C:380) by RNG jump-ahead
//   k_lists_*       vs2ind (mushy positions in order) and frontier rows
//   k_rows_*        (cafe_events.cuh) bounds on the rows' capture times; for
//                   the rows that may capture soon the numerators per liquid
//                   neighbour, sorted per cell
//   k_children      (cafe_events.cuh) rows of the cells that those rows will
//                   capture within the step, two generations ahead
//   k_event_loop    (cafe_events.cuh) the sequential capture/nucleation loop
//                   (VoxelsCA.C:381-610), one thread block
//   k_rows_finalize growth of the rows the loop left aside (VoxelsCA.C:511-516)
//   k_writeback     VoxelsCA.C:633-643
//   k_mushy2solid   ConvertSolid1(0) (VoxelsCA.C:739-758), in place
// All FP64 arithmetic follows the reference's expression order; the file is
// compiled with --fmad=false so no product is fused into an add.
#include <cuda_runtime.h>
#include <stdint.h>

#include "cafe_device.cuh"

#define CAFE_DENSE_THREADS 256
#define CAFE_CELLS_PER_THREAD 8
#define CAFE_CELLS_PER_BLOCK (CAFE_DENSE_THREADS * CAFE_CELLS_PER_THREAD)
// The active-set compaction takes `chunks` (1..4) 8-cell chunks per thread: one,
// so that the cell-by-cell tests inside the pool box spread over the GPU, unless a
// batch's autotuner finds more to be faster (many realisations fill the GPU).
#define CAFE_ACT_MAX_CHUNKS 4
#define CAFE_LOOP_THREADS 512

// ------------------------------------------------------------------ helpers
// Growth velocity of active position p (VoxelsCA.C:405): per temperature class
// with the analytic field, per cell with the EASM field.
__device__ __forceinline__ double cafe_vh(const CafeDev &D, const CafeConsts &K, int p) {
  return K.easm ? D.a_vh[p] : K.vhat_cls[D.a_cls[p]];
}

// Nucleation probability of a capture event that takes active position icap
// (VoxelsCA.C:483): rX, or with the Gaussian-undercooling extension
// rX exp(-.5 x1^2), x1 = ((tL - T) - mean) / sd / sqrt(2), the form of
// VoxelsCA.C:2545-2548, with T the captured cell's temperature.
__device__ __forceinline__ double cafe_nuc_rate(const CafeDev &D, const CafeConsts &K, int icap) {
  if (!K.nuc_gauss) return K.rX;
  double T = K.easm ? D.temp[D.act[icap]] : K.Tcls[D.a_cls[icap]];
  double x1 = ((K.tL - T) - K.nuc_mean) / K.nuc_sd / 1.4142135623730951;
  return K.rX * crm_exp(-.5 * (x1 * x1));
}

// ... as k_gather stored it for the step
__device__ __forceinline__ double cafe_nuc_rate_at(const CafeDev &D, const CafeConsts &K, int icap) {
  return K.nuc_gauss ? D.a_nuc[icap] : K.rX;
}

__device__ __forceinline__ int cafe_hot(const CafeDev &D, const CafeConsts &K, const CafeStepParams &P,
                                        int i, int j, int k) {
  return K.hot_cls[cafe_cls(D, P, i, j, k)];
}

// Moore neighbours in ascending linear-index order (Grid.C:399-414 + sort at
// Grid.C:375); writes cell indices, returns the count.
__device__ __forceinline__ int cafe_moore(const CafeConsts &K, int i, int j, int k, long long *nb) {
  int n = 0;
  for (int dz = -1; dz <= 1; ++dz) {
    int z = k + dz;
    if (z < 0 || z >= K.nz) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      int y = j + dy;
      if (y < 0 || y >= K.ny) continue;
      for (int dx = -1; dx <= 1; ++dx) {
        int x = i + dx;
        if (x < 0 || x >= K.nx) continue;
        if (dx == 0 && dy == 0 && dz == 0) continue;
        nb[n++] = (long long)K.nxy * z + (long long)K.nx * y + x;
      }
    }
  }
  return n;
}

// ------------------------------------------------------------------ K: melt
// Over the box where T may reach the liquidus: SetLiquid3 and BuildjID, a warp
// per row of the box. A cell's class is a test of two or three quotients against
// one, so single precision decides all cells but those near the pool's
// surface, which take the FP64 evaluation: with it for every cell the pass was
// bound by FP64 issue (three divisions a cell; 88 us a step for the rotated pool
// of the 1024x1024x256 deck).
__device__ __forceinline__ void d_melt(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, const int cafe_bid, const int cafe_nblk) {
  const CafeStepParams P = *Pp;
  const int bx = P.hi[0] - P.lo[0], by = P.hi[1] - P.lo[1], bz = P.hi[2] - P.lo[2];
  const int lane = threadIdx.x & 31, warps = (cafe_nblk * blockDim.x) >> 5;
  const long long iz1 = (long long)P.ilaserLoc * K.nxy;
  int any = 0;
  const CafeClassStep C = cafe_class_step(K.ra1, K.bmDX0, P.dirp, P.cg, P.sg, K.dx[0], P.any_hot_full != 0);
  for (int row = (cafe_bid * blockDim.x + threadIdx.x) >> 5; row < by * bz; row += warps) {
    const int j = P.lo[1] + row % by, k = P.lo[2] + row / by;
    const double zp = ((double)k + .5) * K.dx[2], y0 = ((double)j + .5) * K.dx[1];
    const double X = ((double)P.lo[0] + .5) * K.dx[0] - K.hLX0, Y = y0 - K.hLX1;
    const CafeClassRow W = cafe_class_row(C, P.cg, P.sg, K.hLX0, K.hLX1, P.lx, P.ly, P.lz, X, Y, zp, bx);
    const long long base = (long long)K.nxy * k + (long long)K.nx * j + P.lo[0];
    for (int x = lane; x < bx; x += 32) {
      int c = cafe_class_fast(C, W, x);
      const int i = P.lo[0] + x;
      if (c < 0) c = cafe_temp_class_exact(K, P, i, j, k);
      D.tcls[(long long)row * bx + x] = (uint8_t)c;
      const long long idx = base + x;
      if (K.gt_cls[c]) D.buildj[idx] = 1;
      if (K.hot_cls[c]) {
        any = 1;
        if (idx < K.nxy) {
          D.state[idx] = 2;
        } else if (idx < iz1) {
          D.state[idx] = 1;
          D.gid[idx] = 0;
        }
        D.ext[idx] = 0.0;
      }
    }
  }
  if (__syncthreads_or(any) && threadIdx.x == 0) atomicOr(&D.ctr[CTR_HOT], 1);
}
__global__ void k_melt(CafeDev D, CafeConsts K, const CafeStepParams *__restrict__ Pp) {
  d_melt(D, K, Pp, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------ K: solid -> mushy
// ConvertSolid1(1): solid cells with a liquid neighbour become mushy. In place
// is equivalent to the reference's collect-then-apply: the test reads only
// "neighbour == liquid", which this pass never changes. Liquid cells can only
// be (a) cells listed by the previous step's write-back, (b) cells of the
// previous step's pool box, (c) cells of this step's pool box; k_solid2mushy
// covers these, the dense kernel every cell (after an upload or restore).
__global__ void k_solid2mushy_dense(CafeDev D, CafeConsts K) {
  long long base = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * CAFE_CELLS_PER_THREAD;
  for (int c = 0; c < CAFE_CELLS_PER_THREAD; ++c) {
    long long idx = base + c;
    if (idx >= K.N) return;
    if (D.state[idx] != 3) continue;
    int i, j, k;
    cafe_cell_xyz(K, idx, i, j, k);
    long long nb[26];
    int n = cafe_moore(K, i, j, k, nb);
    bool liq = false;
    for (int a = 0; a < n && !liq; ++a) liq = (D.state[nb[a]] == 1);
    if (liq) D.state[idx] = 2;
  }
}

// Eight bytes a[i .. i+7] as one word for any i (a is 8-byte aligned and padded).
__device__ __forceinline__ unsigned long long cafe_load8(const uint8_t *a, long long i) {
  const unsigned long long *w = (const unsigned long long *)(a + (i & ~7LL));
  const int sh = (int)(i & 7) * 8;
  unsigned long long v = w[0];
  if (sh) v = (v >> sh) | (w[1] << (64 - sh));
  return v;
}
// The lowest bits of the eight bytes of w (each 0 or 1) as a mask, bit c for byte c.
__device__ __forceinline__ uint32_t cafe_gather8(unsigned long long w) {
  return (uint32_t)((w * 0x0102040810204080ULL) >> 56);
}

// ConvertSolid1(1) for the eight cells i0..i0+7 of row (j, k): the states of the
// 3 x 3 rows around them as words (a state is 0..3: solid has both low bits,
// liquid the lowest only), the liquid cells of the nine rows as one mask, and
// its three-wide window. Cells past the row's end are masked out.
__device__ __forceinline__ void cafe_chunk_solid2mushy(const CafeDev &D, const CafeConsts &K, int i0, int j, int k) {
  const int n = min(8, K.nx - i0);
  const uint32_t valid = (1u << n) - 1u;
  const long long base = (long long)K.nxy * k + (long long)K.nx * j + i0;
  const unsigned long long w0 = cafe_load8(D.state, base);
  const uint32_t solid = cafe_gather8(w0 & (w0 >> 1) & 0x0101010101010101ULL) & valid;
  if (!solid) return;
  uint32_t liq = 0;  // bit x: cell i0 - 1 + x of some row
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const int y = j + r % 3 - 1, z = k + r / 3 - 1;
    if (y < 0 || y >= K.ny || z < 0 || z >= K.nz) continue;
    const long long rb = (long long)K.nxy * z + (long long)K.nx * y + i0;
    const unsigned long long w = cafe_load8(D.state, rb);
    liq |= (cafe_gather8(w & ~(w >> 1) & 0x0101010101010101ULL) & valid) << 1;
    if (i0 > 0 && D.state[rb - 1] == 1) liq |= 1u;
    if (i0 + 8 < K.nx && D.state[rb + 8] == 1) liq |= 1u << 9;
  }
  uint32_t hit = solid & ((liq | (liq << 1) | (liq >> 1)) >> 1);
  for (; hit; hit &= hit - 1) D.state[base + __ffs(hit) - 1] = 2;
}

// ConvertSolid1(1) where liquid cells can be: this step's pool box and the
// previous one, each dilated by one cell (as one box when that is no larger),
// in chunks of eight cells, and around the cells that the previous step listed.
// Eight cells per thread: the cell-by-cell form (26 loads for every solid cell,
// two boxes and the list in launches of their own) took 98 us a step on
// 1024x1024x256 cells, bound by its dependent loads.
__device__ __forceinline__ void d_solid2mushy(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, const int cafe_bid, const int cafe_nblk) {
  int lo[2][3], hi[2][3];
  long long cnt[2] = {0, 0}, vol[2] = {0, 0};
  const bool prev = Pp->phi[0] > Pp->plo[0] && Pp->phi[1] > Pp->plo[1] && Pp->phi[2] > Pp->plo[2];
  const int nmax[3] = {K.nx, K.ny, K.nz};
#pragma unroll
  for (int b = 0; b < 2; ++b) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[b][a] = max((b ? Pp->plo[a] : Pp->lo[a]) - 1, 0);
      hi[b][a] = min((b ? Pp->phi[a] : Pp->hi[a]) + 1, nmax[a]);
    }
    vol[b] = (long long)max(hi[b][0] - lo[b][0], 0) * max(hi[b][1] - lo[b][1], 0) * max(hi[b][2] - lo[b][2], 0);
  }
  if (!prev) vol[1] = 0;
  if (vol[0] > 0 && vol[1] > 0) {
    int ul[3], uh[3];
    long long uv = 1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ul[a] = min(lo[0][a], lo[1][a]);
      uh[a] = max(hi[0][a], hi[1][a]);
      uv *= uh[a] - ul[a];
    }
    if (uv <= vol[0] + vol[1]) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        lo[0][a] = ul[a];
        hi[0][a] = uh[a];
      }
      vol[1] = 0;
    }
  }
  int cx[2];
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    lo[b][0] &= ~7;
    cx[b] = (hi[b][0] - lo[b][0] + 7) >> 3;
    if (vol[b] > 0) cnt[b] = (long long)cx[b] * (hi[b][1] - lo[b][1]) * (hi[b][2] - lo[b][2]);
  }
  const long long total = cnt[0] + cnt[1] + D.ctr[CTR_NLIQ];
  for (long long t = cafe_bid * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)cafe_nblk * blockDim.x) {
    if (t < cnt[0] + cnt[1]) {
      const int b = t < cnt[0] ? 0 : 1;
      const unsigned int u = (unsigned int)(b ? t - cnt[0] : t), nxc = b ? cx[1] : cx[0];
      const unsigned int ny = b ? hi[1][1] - lo[1][1] : hi[0][1] - lo[0][1];
      const unsigned int r = u / nxc, z = r / ny;
      cafe_chunk_solid2mushy(D, K, (b ? lo[1][0] : lo[0][0]) + 8 * (int)(u - r * nxc),
                             (b ? lo[1][1] : lo[0][1]) + (int)(r - z * ny), (b ? lo[1][2] : lo[0][2]) + (int)z);
    } else {
      const long long idx = D.liq[t - cnt[0] - cnt[1]];
      if (D.state[idx] != 1) continue;
      int i, j, k;
      cafe_cell_xyz(K, idx, i, j, k);
#pragma unroll
      for (int d = 0; d < 27; ++d) {
        const int x = i + d % 3 - 1, y = j + d / 3 % 3 - 1, z = k + d / 9 - 1;
        if (x < 0 || x >= K.nx || y < 0 || y >= K.ny || z < 0 || z >= K.nz) continue;
        const long long nb = (long long)K.nxy * z + (long long)K.nx * y + x;
        if (D.state[nb] == 3) D.state[nb] = 2;
      }
    }
  }
}
__global__ void k_solid2mushy(CafeDev D, CafeConsts K, const CafeStepParams *__restrict__ Pp) {
  d_solid2mushy(D, K, Pp, blockIdx.x, gridDim.x);
}

// The step parameters into device memory (kernel arguments are copied at
// launch, so the host copy may change right after).
__global__ void k_put_params(CafeStepParams *Pd, CafeStepParams P) { *Pd = P; }


// ------------------------------------------------------------------ active set
// Box that can hold active cells this step: the mushy and liquid cells left by
// the previous step (k_writeback), this and the previous pool box, widened by
// one cell. Every active cell is mushy, liquid, or at/above the liquidus
// (inside the pool box); a cell turns mushy this step only next to a liquid
// cell (ConvertSolid1(1)), and liquid cells are those left by the previous
// step or melted in the pool box; new layers bring solid and powder cells
// only. In chunks of eight cells along x (x0 a multiple of 8), whose order is
// the order of their cells. (Whole z planes instead, 62 M cells a step on
// 1024x1024x256, made the compaction 130 us by instruction issue; the box's cells
// take 22, bound by the latency of their loads.)
struct CafeBox {
  int x0, y0, z0, nxc, ny;
  long long n;  // chunks
};
__device__ __forceinline__ CafeBox cafe_active_box(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ P) {
  const bool cur = P->hi[0] > P->lo[0] && P->hi[1] > P->lo[1] && P->hi[2] > P->lo[2];
  const bool prev = P->phi[0] > P->plo[0] && P->phi[1] > P->plo[1] && P->phi[2] > P->plo[2];
  const int nmax[3] = {K.nx, K.ny, K.nz};
  int lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = D.ctr[CTR_BOX + a];
    hi[a] = D.ctr[CTR_BOX + 3 + a];
    if (cur) {
      lo[a] = min(lo[a], P->lo[a]);
      hi[a] = max(hi[a], P->hi[a] - 1);
    }
    if (prev) {
      lo[a] = min(lo[a], P->plo[a]);
      hi[a] = max(hi[a], P->phi[a] - 1);
    }
    lo[a] = max(lo[a] - 1, 0);
    hi[a] = min(hi[a] + 1, nmax[a] - 1);
  }
  CafeBox b;
  b.x0 = lo[0] & ~7;
  b.y0 = lo[1];
  b.z0 = lo[2];
  b.nxc = (hi[0] - b.x0 + 8) >> 3;
  b.ny = hi[1] - lo[1] + 1;
  b.n = hi[0] < lo[0] || hi[1] < lo[1] || hi[2] < lo[2] ? 0 : (long long)b.nxc * b.ny * (hi[2] - lo[2] + 1);
  return b;
}

// Flags of the eight state bytes of w (bit c for byte c): the byte is 1
// (liquid) or 2 (mushy). Bit arithmetic on the word: a byte is 1 or 2 when
// it is below 4 and its two low bits differ; the eight results, one per
// byte's lowest bit, are gathered into the top byte by one multiplication.
__device__ __forceinline__ uint32_t cafe_liq_or_mushy8(unsigned long long w) {
  const unsigned long long t = w & 0xFCFCFCFCFCFCFCFCULL;
  const unsigned long long u = (t | (t >> 2) | (t >> 4)) & 0x0C0C0C0C0C0C0C0CULL;
  const unsigned long long ge4 = (u | (u >> 1)) & 0x0404040404040404ULL;  // bit 2: the byte is >= 4
  const unsigned long long a = (w ^ (w >> 1)) & ~(ge4 >> 2) & 0x0101010101010101ULL;
  return (uint32_t)((a * 0x0102040810204080ULL) >> 56);
}

// Activity flags of the eight cells i0..i0+7 of row (j, k), i0 a multiple of 8
// (bit c for cell i0 + c; cells past the row's end are not active). A cell that
// cannot be at or above the liquidus (outside the pool box, or not below the
// laser plane) is active exactly when it is liquid or mushy, so a chunk outside
// the hot region is decided from its state bytes, loaded as one word. In the
// hot region the chunk's own classes come next: when no cell of it is at or
// above the liquidus, the same holds. Otherwise the states of the 3 x 3 rows
// around the chunk over i0-1..i0+8 (a word and two bytes per row) and the
// classes of their liquid cells are loaded, all before any test, so that no
// load waits on another's outcome. A neighbour "emits" when it is mushy or
// liquid below the liquidus; a cell at or above the liquidus is active when
// mushy or when an emitter lies among its 26 neighbours, i.e. in the
// three-wide window of the nine rows' emitter masks (the cell itself, at or
// above the liquidus, emits only if mushy, and then it is active anyway).
__device__ __forceinline__ uint32_t cafe_chunk_active(const CafeDev &D, const CafeConsts &K, const CafeStepParams &P,
                                                      int i0, int j, int k) {
  const int n = min(8, K.nx - i0);
  const uint32_t valid = (1u << n) - 1u;
  const unsigned long long wown = cafe_load8(D.state, (long long)K.nxy * k + (long long)K.nx * j + i0);
  const uint32_t own_lm = cafe_liq_or_mushy8(wown) & valid;
  // (with any_hot_full, T0 or tS reaches the liquidus and no class is cold)
  if (!P.any_hot_full && (k >= P.kabove || k < P.lo[2] || k >= P.hi[2] || j < P.lo[1] || j >= P.hi[1] ||
                          i0 + 7 < P.lo[0] || i0 >= P.hi[0]))
    return own_lm;
  const uint32_t hotmask = (K.hot_cls[0] ? 1u : 0u) | (K.hot_cls[1] ? 2u : 0u) | (K.hot_cls[2] ? 4u : 0u);
  uint32_t own_hot = 0;  // bit c: cell i0 + c at or above the liquidus
#pragma unroll
  for (int c = 0; c < 8; ++c)
    if (c < n) own_hot |= ((hotmask >> cafe_cls(D, P, i0 + c, j, k)) & 1u) << c;
  if (own_hot == 0) return own_lm;
  uint32_t own_mushy = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) own_mushy |= (((wown >> (8 * c)) & 0xffu) == 2u ? 1u : 0u) << c;
  uint32_t win = 0;  // bit x: an emitter at x - 1..x + 1 (x = 0..9 for i0 - 1 + x) in some row
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const int y = j + r % 3 - 1, z = k + r / 3 - 1;
    const bool rowin = y >= 0 && y < K.ny && z >= 0 && z < K.nz;
    const long long rb = (long long)K.nxy * (rowin ? z : 0) + (long long)K.nx * (rowin ? y : 0);
    const unsigned long long w = rowin ? cafe_load8(D.state, rb + i0) : 0ULL;
    const unsigned int sl = (rowin && i0 > 0) ? D.state[rb + i0 - 1] : 0u;
    const unsigned int sr = (rowin && i0 + 8 < K.nx) ? D.state[rb + i0 + 8] : 0u;
    uint32_t e = 0;
#pragma unroll
    for (int x = 0; x < 10; ++x) {
      const unsigned int s =
          x == 0 ? sl : (x == 9 ? sr : (x - 1 < n ? (unsigned int)(w >> (8 * (x - 1))) & 0xffu : 0u));
      // the class of a liquid neighbour
      const int c = s == 1u ? cafe_cls(D, P, i0 - 1 + x, y, z) : 1;
      const bool hot = (hotmask >> c) & 1u;
      e |= (s == 2u || (s == 1u && !hot)) ? 1u << x : 0u;
    }
    win |= e | (e << 1) | (e >> 1);
  }
  // cell i0 + c is bit c + 1 of the window
  const uint32_t nb = (win >> 1) & 0xffu;
  return ((~own_hot & own_lm) | (own_hot & (own_mushy | nb))) & valid;
}

// A thread's `chunks` consecutive chunks of the box, from chunk t on: f(c, i0, j,
// k) for each (coordinates formed once, then stepped).
template <class F>
__device__ __forceinline__ void cafe_for_chunks(const CafeBox &b, long long t, int chunks, F f) {
  if (t >= b.n) return;
  const unsigned int u = (unsigned int)t, r = u / (unsigned int)b.nxc, z = r / (unsigned int)b.ny;
  int xc = (int)(u - r * b.nxc), y = (int)(r - z * b.ny), k = b.z0 + (int)z;
#pragma unroll
  for (int c = 0; c < CAFE_ACT_MAX_CHUNKS; ++c) {
    if (c >= chunks || t + c >= b.n) break;
    f(c, b.x0 + 8 * xc, b.y0 + y, k);
    if (++xc == b.nxc) {
      xc = 0;
      if (++y == b.ny) {
        y = 0;
        ++k;
      }
    }
  }
}

// The compaction runs over "virtual blocks" of CAFE_DENSE_THREADS threads x
// `chunks` chunks of the box; a persistent grid strides over them.
__device__ __forceinline__ long long cafe_box_vblocks(const CafeBox &b, int chunks) {
  const long long per = (long long)CAFE_DENSE_THREADS * chunks;
  return (b.n + per - 1) / per;
}
__device__ __forceinline__ void d_active_count(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, int chunks, const int cafe_bid, const int cafe_nblk) {
  const CafeStepParams P = *Pp;
  __shared__ int wsum[CAFE_DENSE_THREADS / 32];
  const CafeBox B = cafe_active_box(D, K, Pp);
  const long long nvb = cafe_box_vblocks(B, chunks);
  for (long long vb = cafe_bid; vb < nvb; vb += cafe_nblk) {
    uint32_t f = 0;
    cafe_for_chunks(B, (vb * CAFE_DENSE_THREADS + threadIdx.x) * chunks, chunks,
                    [&](int c, int i0, int j, int k) { f |= cafe_chunk_active(D, K, P, i0, j, k) << (8 * c); });
    D.act_flags[vb * CAFE_DENSE_THREADS + threadIdx.x] = f;
    const int cnt = __reduce_add_sync(0xffffffffu, __popc(f));
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
      int sum = 0;
      for (int w = 0; w < CAFE_DENSE_THREADS / 32; ++w) sum += wsum[w];
      D.blk[vb] = sum;
    }
    __syncthreads();
  }
}
__global__ void k_active_count(CafeDev D, CafeConsts K, const CafeStepParams *__restrict__ Pp, int chunks) {
  d_active_count(D, K, Pp, chunks, blockIdx.x, gridDim.x);
}

// Exclusive scan over the block of one value per thread (blockDim.x a multiple
// of 32, at most 1024; every thread must call it): returns this thread's
// prefix and leaves the block total in tot. ws: 33 shared words.
__device__ __forceinline__ long long cafe_block_excl_scan(long long v, long long *ws, long long &tot) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  long long incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const long long t = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  if (w == 0) {
    const long long x = lane < nw ? ws[lane] : 0;
    long long xi = x;
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(FULL, xi, o);
      if (lane >= o) xi += t;
    }
    if (lane < nw) ws[lane] = xi - x;
    if (lane == 31) ws[32] = xi;
  }
  __syncthreads();
  tot = ws[32];
  return ws[w] + incl - v;
}

// Exclusive scan of the compaction's block counts in place; the total is the
// active-list length.
__device__ __forceinline__ void d_scan_blocks(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, int chunks) {
  int32_t *blk = D.blk;
  const long long n = cafe_box_vblocks(cafe_active_box(D, K, Pp), chunks);
  __shared__ long long ws[33];
  // each thread's segment is a multiple of four counts, so that its groups of
  // four are aligned 16-byte loads and stores (a warp's lanes read segments
  // apart, and one vector access serves four counts)
  const long long per = ((n + blockDim.x - 1) / blockDim.x + 3) & ~3LL;
  long long b0 = threadIdx.x * per, b1 = b0 + per < n ? b0 + per : n;
  if (b0 > n) b0 = n;
  long long s = 0;
  for (long long b = b0; b < b1; b += 16) {
    int4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long g = b + 4 * i;
      if (g + 4 <= b1)
        v[i] = *(const int4 *)(blk + g);
      else
        v[i] = make_int4(g < b1 ? blk[g] : 0, g + 1 < b1 ? blk[g + 1] : 0, g + 2 < b1 ? blk[g + 2] : 0, 0);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) s += (long long)v[i].x + v[i].y + v[i].z + v[i].w;
  }
  long long tot;
  long long acc = cafe_block_excl_scan(s, ws, tot);
  if (threadIdx.x == 0) D.ctr[CTR_NA] = (int)tot;
  for (long long b = b0; b < b1; b += 16) {
    int4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long g = b + 4 * i;
      if (g + 4 <= b1)
        v[i] = *(const int4 *)(blk + g);
      else
        v[i] = make_int4(g < b1 ? blk[g] : 0, g + 1 < b1 ? blk[g + 1] : 0, g + 2 < b1 ? blk[g + 2] : 0, 0);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long g = b + 4 * i;
      int4 o;
      o.x = (int32_t)acc;
      acc += v[i].x;
      o.y = (int32_t)acc;
      acc += v[i].y;
      o.z = (int32_t)acc;
      acc += v[i].z;
      o.w = (int32_t)acc;
      acc += v[i].w;
      if (g + 4 <= b1) {
        *(int4 *)(blk + g) = o;
      } else {
        if (g < b1) blk[g] = o.x;
        if (g + 1 < b1) blk[g + 1] = o.y;
        if (g + 2 < b1) blk[g + 2] = o.z;
      }
    }
  }
}
__global__ void __launch_bounds__(1024) k_scan_blocks(CafeDev D, CafeConsts K, const CafeStepParams *__restrict__ Pp, int chunks) {
  d_scan_blocks(D, K, Pp, chunks);
}

__device__ __forceinline__ void d_active_scatter(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, int chunks, const int cafe_bid, const int cafe_nblk) {
  __shared__ int wsum[CAFE_DENSE_THREADS / 32];
  const CafeBox B = cafe_active_box(D, K, Pp);
  const long long nvb = cafe_box_vblocks(B, chunks);
  for (long long vb = cafe_bid; vb < nvb; vb += cafe_nblk) {
  const uint32_t flags = D.act_flags[vb * CAFE_DENSE_THREADS + threadIdx.x];  // from k_active_count
  const int cnt = __popc(flags);
  // block-exclusive scan of per-thread counts
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  if (threadIdx.x < 32) {
    int v = threadIdx.x < CAFE_DENSE_THREADS / 32 ? wsum[threadIdx.x] : 0;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (threadIdx.x >= o) inc += u;
    }
    if (threadIdx.x < CAFE_DENSE_THREADS / 32) wsum[threadIdx.x] = inc - v;
  }
  __syncthreads();
  long long pos = (long long)D.blk[vb] + wsum[w] + (incl - cnt);
  if (flags)
    cafe_for_chunks(B, (vb * CAFE_DENSE_THREADS + threadIdx.x) * chunks, chunks, [&](int c, int i0, int j, int k) {
      const long long base = (long long)K.nxy * k + (long long)K.nx * j + i0;
      for (uint32_t m = (flags >> (8 * c)) & 0xffu; m; m &= m - 1) {
        const long long idx = base + __ffs(m) - 1;
        if (pos < D.act_cap) {
          D.act[pos] = (int32_t)idx;
          D.pos_of[idx] = (int32_t)pos;
        } else {
          atomicOr(D.err, CAFE_ERR_ACTIVE_CAP);
        }
        ++pos;
      }
    });
  __syncthreads();  // wsum is reused by the next virtual block
  }
}
__global__ void k_active_scatter(CafeDev D, CafeConsts K, const CafeStepParams *__restrict__ Pp, int chunks) {
  d_active_scatter(D, K, Pp, chunks, blockIdx.x, gridDim.x);
}

// Counters of the step from the gather on (one thread, before the row set-up and
// after k_solid2mushy and the compaction read last step's): the active box, rebuilt
// by k_writeback, and the row set-up's.
__device__ __forceinline__ void d_reset_rows(const CafeDev &D, const CafeConsts &K) {
  for (int a = 0; a < 3; ++a) {
    D.ctr[CTR_BOX + a] = 0x7fffffff;
    D.ctr[CTR_BOX + 3 + a] = -1;
  }
  D.row_mag[0] = D.row_mag[1] = 0ULL;  // formed by k_rows_order and k_children
  D.row_mag[2] = ~0ULL;
  D.row_mag[3] = 0ULL;
  // the row set-up's counters; a per-cell field grows rows with their own velocities
  D.ctr[CTR_SLOW] = K.easm ? 1 : 0;
  D.ctr[CTR_NPAIRS] = D.ctr[CTR_NDUE] = D.ctr[CTR_NKEY] = 0;
  for (int d = 0; d < CAFE_CHILD_DEPTH; ++d) D.ctr[CTR_NCHILD + d] = 0;
  D.ctr[CTR_NLIQ] = 0;  // listed again by k_writeback (k_solid2mushy has read it)
}

// ------------------------------------------------------------------ gather
// Per active position: copies of the cell data, temperature class, neighbour
// positions by direction (CAFE_NSLOT, in ascending index order; -1 = not active
// or outside the grid), kind (a_kind),
// all-neighbours-below-liquidus flag and the ruq offset (VoxelsCA.C:380:
// ruq[p] = (U_p - .5) dX / 100, U_p the p-th uniform of minstd(30 tInd + seed1)).
// A warp takes 32 positions: one value per position a lane each, then a position's
// 26 neighbours a lane each, bound by the latency of the scattered loads. With a
// thread per position it and the lists took 36 us more on 1024x1024x256.
__device__ __forceinline__ void d_gather(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, const int cafe_bid, const int cafe_nblk) {
  const CafeStepParams P = *Pp;
  int na = D.ctr[CTR_NA];
  if (na > D.act_cap) na = (int)D.act_cap;
  uint32_t seed = cafe_minstd_seed((uint64_t)(uint32_t)(30 * P.tInd + (int)K.seed1));
  // A warp takes 32 positions: their copies with a position per lane, then their
  // neighbours with a direction per lane, one position after another (a
  // position's 26 neighbours loaded by one thread took 28 us for 36 thousand,
  // waiting on each load in turn).
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int warps = (cafe_nblk * blockDim.x) >> 5;
  const uint32_t pw = cafe_minstd_pow(2 * lane);  // the stream's step to lane's position from the warp's first
  const int d27 = lane < 13 ? lane : lane + 1;    // direction of this lane (CAFE_NSLOT of them)
  const int dx = d27 % 3 - 1, dy = d27 / 3 % 3 - 1, dz = d27 / 9 - 1;
  for (int w = (cafe_bid * blockDim.x + threadIdx.x) >> 5; w * 32 < na; w += warps) {
    const int p0 = w * 32, p = p0 + lane, n = min(32, na - p0);
    int i = 0, j = 0, k = 0;
    uint8_t st = 0;
    if (lane < n) {
      const long long idx = D.act[p];
      cafe_cell_xyz(K, idx, i, j, k);
      st = D.state[idx];
      D.a_state[p] = st;
      D.a_gid[p] = D.gid[idx];
      D.a_ext[p] = D.ext[idx];
      D.a_cx[p] = D.cx[idx];
      D.a_cy[p] = D.cy[idx];
      D.a_cz[p] = D.cz[idx];
      D.a_cls[p] = (uint8_t)cafe_cls(D, P, i, j, k);
      if (K.easm) {
        // VoxelsCA.C:405: T >= tL ? 0 : Avel pow(tL - T, nvel)
        double T = D.temp[idx];
        D.a_vh[p] = T >= K.tL ? 0.0 : K.Avel * crm_pow_int(K.tL - T, K.nvel_i);
      }
      D.a_frow[p] = -1;
      D.a_ev[p] = 0;
      if (K.nuc_gauss) D.a_nuc[p] = cafe_nuc_rate(D, K, p);
      // the p-th uniform of the stream: outputs 2 p + 1 and 2 p + 2
      const uint32_t x1 = (uint32_t)(((uint64_t)cafe_minstd_skip(seed, 2ULL * p0 + 1) * pw) % CAFE_MINSTD_M);
      const double U = cafe_canonical(x1, cafe_minstd_next(x1));
      D.a_ruq[p] = (U - .5) * K.ruq_dx / 100.;
    }
    bool liq = false, cold = false;
#pragma unroll 4
    for (int t = 0; t < n; ++t) {
      const int x = __shfl_sync(FULL, i, t) + dx, y = __shfl_sync(FULL, j, t) + dy, z = __shfl_sync(FULL, k, t) + dz;
      int q = -1;
      bool l = false, h = false;
      if (lane < CAFE_NSLOT) {
        if (x >= 0 && x < K.nx && y >= 0 && y < K.ny && z >= 0 && z < K.nz) {
          const long long nb = (long long)K.nxy * z + (long long)K.nx * y + x;
          q = D.pos_of[nb];
          l = q >= 0 && D.state[nb] == 1;
          h = q >= 0 && cafe_hot(D, K, P, x, y, z);
        }
        D.a_nbr[(long long)(p0 + t) * CAFE_NSLOT + lane] = q;
      }
      const uint32_t bl = __ballot_sync(FULL, l), bh = __ballot_sync(FULL, h);
      if (lane == t) {
        liq = bl != 0u;
        cold = bh == 0u;
      }
    }
    if (lane < n) {
      D.a_cold[p] = cold;
      // mushy; able to capture (VoxelsCA.C:396-397)
      D.a_kind[p] = st == 2 ? (liq && cold ? 3 : 1) : 0;
    }
  }
}
__global__ void k_gather(CafeDev D, CafeConsts K, const CafeStepParams *__restrict__ Pp) {
  if (blockIdx.x == 0 && threadIdx.x == 0) d_reset_rows(D, K);
  d_gather(D, K, Pp, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------ vs2ind + frontier rows
// Two order-preserving compactions over positions: mushy positions (vs2ind,
// VoxelsCA.C:346-353) and, among them, those with a liquid neighbour and no
// neighbour at the liquidus (the cells that can capture, VoxelsCA.C:396-397).
// Eight positions per thread, their kinds as one word (positions past the
// list's end count as nothing).
__device__ __forceinline__ unsigned long long cafe_kinds8(const CafeDev &D, long long base, int na) {
  if (base >= na) return 0ULL;
  unsigned long long w = *(const unsigned long long *)(D.a_kind + base);
  if (base + 8 > na) w &= (1ULL << (8 * (na - base))) - 1ULL;
  return w;
}
__device__ __forceinline__ void d_lists_count(const CafeDev &D, const int cafe_bid, const int cafe_nblk) {
  __shared__ int ws[2][CAFE_DENSE_THREADS / 32];
  int na = D.ctr[CTR_NA];
  if (na > D.act_cap) na = (int)D.act_cap;
  const int nvb = (na + CAFE_CELLS_PER_BLOCK - 1) / CAFE_CELLS_PER_BLOCK;
  for (int vb = cafe_bid; vb < nvb; vb += cafe_nblk) {
    const unsigned long long w =
        cafe_kinds8(D, ((long long)vb * CAFE_DENSE_THREADS + threadIdx.x) * CAFE_CELLS_PER_THREAD, na);
    const int c2 = __reduce_add_sync(0xffffffffu, __popcll(w & 0x0101010101010101ULL));
    const int cf = __reduce_add_sync(0xffffffffu, __popcll(w & 0x0202020202020202ULL));
    if ((threadIdx.x & 31) == 0) {
      ws[0][threadIdx.x >> 5] = c2;
      ws[1][threadIdx.x >> 5] = cf;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int s2 = 0, sf = 0;
      for (int q = 0; q < CAFE_DENSE_THREADS / 32; ++q) {
        s2 += ws[0][q];
        sf += ws[1][q];
      }
      D.blk[2 * vb] = s2;
      D.blk[2 * vb + 1] = sf;
    }
    __syncthreads();
  }
}
__global__ void k_lists_count(CafeDev D) {
  d_lists_count(D, blockIdx.x, gridDim.x);
}

// Exclusive scan of interleaved pairs (blk[2b], blk[2b+1]), b < n, one block.
// Exclusive scan of the (mushy, frontier) count pairs of the position blocks
// that hold active positions (na from *na_ptr); totals to *tot0, *tot1.
__device__ __forceinline__ void d_scan_pairs(int32_t *blk, long long n, const int *na_ptr, int *tot0, int *tot1, const int cafe_bid, const int cafe_nblk) {
  __shared__ long long ws[2][33];
  {
    long long used = ((long long)*na_ptr + CAFE_CELLS_PER_BLOCK - 1) / CAFE_CELLS_PER_BLOCK;
    if (used < n) n = used;
  }
  long long per = (n + blockDim.x - 1) / blockDim.x;
  long long b0 = threadIdx.x * per, b1 = b0 + per < n ? b0 + per : n;
  const int2 *p2 = (const int2 *)blk;  // (count 0, count 1) of block b
  long long s0 = 0, s1 = 0;
  for (long long b = b0; b < b1; b += 8) {
    int2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = b + i < b1 ? p2[b + i] : make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      s0 += v[i].x;
      s1 += v[i].y;
    }
  }
  long long t0, t1;
  long long a0 = cafe_block_excl_scan(s0, ws[0], t0);
  long long a1 = cafe_block_excl_scan(s1, ws[1], t1);
  if (threadIdx.x == 0) {
    *tot0 = (int)t0;
    *tot1 = (int)t1;
  }
  int2 *q2 = (int2 *)blk;
  for (long long b = b0; b < b1; b += 8) {
    int2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = b + i < b1 ? q2[b + i] : make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (b + i < b1) {
        q2[b + i] = make_int2((int32_t)a0, (int32_t)a1);
        a0 += v[i].x;
        a1 += v[i].y;
      }
  }
}
__global__ void __launch_bounds__(1024) k_scan_pairs(int32_t *blk, long long n, const int *na_ptr, int *tot0, int *tot1) {
  d_scan_pairs(blk, n, na_ptr, tot0, tot1, blockIdx.x, gridDim.x);
}

__device__ __forceinline__ void d_lists_scatter(const CafeDev &D, const int cafe_bid, const int cafe_nblk) {
  __shared__ int ws[2][CAFE_DENSE_THREADS / 32];
  int na = D.ctr[CTR_NA];
  if (na > D.act_cap) na = (int)D.act_cap;
  const int nvb = (na + CAFE_CELLS_PER_BLOCK - 1) / CAFE_CELLS_PER_BLOCK;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int vb = cafe_bid; vb < nvb; vb += cafe_nblk) {
    const long long base = ((long long)vb * CAFE_DENSE_THREADS + threadIdx.x) * CAFE_CELLS_PER_THREAD;
    const unsigned long long kinds = cafe_kinds8(D, base, na);
    const int c2 = __popcll(kinds & 0x0101010101010101ULL), cf = __popcll(kinds & 0x0202020202020202ULL);
    int i2 = c2, i_f = cf;
    for (int o = 1; o < 32; o <<= 1) {
      int v2 = __shfl_up_sync(0xffffffffu, i2, o), vf = __shfl_up_sync(0xffffffffu, i_f, o);
      if (lane >= o) {
        i2 += v2;
        i_f += vf;
      }
    }
    if (lane == 31) {
      ws[0][w] = i2;
      ws[1][w] = i_f;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int a2 = 0, af = 0;
      for (int q = 0; q < CAFE_DENSE_THREADS / 32; ++q) {
        int v2 = ws[0][q], vf = ws[1][q];
        ws[0][q] = a2;
        ws[1][q] = af;
        a2 += v2;
        af += vf;
      }
    }
    __syncthreads();
    long long j2 = (long long)D.blk[2 * vb] + ws[0][w] + (i2 - c2);
    long long jf = (long long)D.blk[2 * vb + 1] + ws[1][w] + (i_f - cf);
    for (int c = 0; c < CAFE_CELLS_PER_THREAD; ++c) {
      const int kind = (int)(kinds >> (8 * c)) & 0xff;
      if (!kind) continue;
      const long long p = base + c;
      if (j2 < D.vs2_cap)
        D.vs2[j2] = (int32_t)p;
      else
        atomicOr(D.err, CAFE_ERR_MUSHY_CAP);
      if (kind & 2) {
        if (jf < D.row_cap) {
          D.row_pos[jf] = (int32_t)p;
          D.row_j[jf] = (int32_t)j2;
          D.a_frow[p] = (int32_t)jf;
        } else {
          atomicOr(D.err, CAFE_ERR_ROW_CAP);
        }
        ++jf;
      }
      ++j2;
    }
    __syncthreads();  // ws is reused by the next virtual block
  }
}
__global__ void k_lists_scatter(CafeDev D) {
  d_lists_scatter(D, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------ frontier rows
// Order keys: an unsigned integer order equal to the numeric order of the
// doubles (negative values included); cafe_key_canon maps -0 to +0 first so
// that equal values get equal keys.
#define CAFE_KEY_NONE 0xffffffffffffffffULL
__device__ __forceinline__ unsigned long long cafe_key(double x) {
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}
__device__ __forceinline__ double cafe_unkey(unsigned long long k) {
  unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffULL) : ~k;
  return __longlong_as_double((long long)b);
}
__device__ __forceinline__ unsigned long long cafe_key_canon(double x) {
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  if (b == 0x8000000000000000ULL) b = 0;
  return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}
__device__ __forceinline__ unsigned long long cafe_shfl_u64(unsigned long long v, int src) {
  return (unsigned long long)__shfl_sync(0xffffffffu, (long long)v, src);
}
__device__ __forceinline__ unsigned long long cafe_shfl_u64_xor(unsigned long long v, int o) {
  return (unsigned long long)__shfl_xor_sync(0xffffffffu, (long long)v, o);
}
__device__ __forceinline__ bool cafe_is_nan(double x) { return (crm_bits(x) & CRM_ABS_MASK) > CRM_BITS_INF; }
// x < 0.0 (negative, nonzero, not NaN)
__device__ __forceinline__ bool cafe_is_neg(double x) {
  long long b = crm_bits(x);
  return b < 0 && (b & CRM_ABS_MASK) != 0 && (b & CRM_ABS_MASK) <= CRM_BITS_INF;
}
#include "cafe_events.cuh"

// Brings every row's extent up to the end of the step (the lazily applied
// growth of VoxelsCA.C:511-516), spread over the whole GPU, and copies it back
// to the row cell's active-list position.
// The growths come through shared memory, a batch at a time, so that a row's
// chain is its additions (64 cycles each, up to a hundred a step: 20 us) and no
// load waits on it.
#define CAFE_FINAL_BATCH 512
__device__ __forceinline__ void d_rows_finalize(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  __shared__ double vd[CAFE_FINAL_BATCH];
  int nrows = D.ctr[CTR_NROWS_END];
  if (nrows > D.row_cap) nrows = (int)D.row_cap;
  const int nev = D.ctr[CTR_NEV];
  const bool pr = D.ctr[CTR_EVLOG] != 0;
  const int nrows0 = D.ctr[CTR_NROWS];
  for (int k0 = cafe_bid * blockDim.x; k0 < nrows; k0 += cafe_nblk * blockDim.x) {
    const int k = k0 + threadIdx.x;
    int r = -1, p = 0, m = 0, stop = 0;
    double E = 0.0, v = 0.0;
    if (k < nrows) {
      r = cafe_row_at(D, nrows0, k);
      p = D.row_pos[r];
      m = D.row_m[r];
      E = D.row_E[r];
      if (pr) v = cafe_vh(D, K, p);
      if (m >= nev)
        m = 0;  // (its extent is final: nothing to apply)
      else
        stop = min(nev, cafe_row_death(D, r));
    }
    for (int e0 = 1; e0 <= nev; e0 += CAFE_FINAL_BATCH) {
      const int n = min(CAFE_FINAL_BATCH, nev - e0 + 1);
      __syncthreads();
      for (int e = threadIdx.x; e < n; e += blockDim.x) vd[e] = D.ev_vd[e0 + e];
      __syncthreads();
      const int a = max(m + 1 - e0, 0), b = min(stop - e0 + 1, n);
      if (pr) {
#pragma unroll 4
        for (int e = a; e < b; ++e) E = cafe_grow(E, v * vd[e]);
      } else {
#pragma unroll 4
        for (int e = a; e < b; ++e) E = cafe_grow(E, vd[e]);
      }
    }
    if (r >= 0) D.a_ext[p] = E;
  }
}
__global__ void k_rows_finalize(CafeDev D, CafeConsts K) {
  d_rows_finalize(D, K, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------ write back
__device__ __forceinline__ void d_writeback(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  int na = D.ctr[CTR_NA];
  if (na > D.act_cap) na = (int)D.act_cap;
  int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-1, -1, -1};
  for (int p = cafe_bid * blockDim.x + threadIdx.x; p < na; p += cafe_nblk * blockDim.x) {
    long long idx = D.act[p];
    if (D.a_state[p] == 1 || D.a_state[p] == 2) {
      int c[3];
      cafe_cell_xyz(K, idx, c[0], c[1], c[2]);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        lo[a] = min(lo[a], c[a]);
        hi[a] = max(hi[a], c[a]);
      }
    }
    D.state[idx] = D.a_state[p];
    D.gid[idx] = D.a_gid[p];
    D.ext[idx] = D.a_ext[p];
    D.cx[idx] = D.a_cx[p];
    D.cy[idx] = D.a_cy[p];
    D.cz[idx] = D.a_cz[p];
    D.pos_of[idx] = -1;
    if (D.a_state[p] == 1) {
      int t = atomicAdd(&D.ctr[CTR_NLIQ], 1);
      D.liq[t] = (int32_t)idx;  // t < na <= act_cap = liq capacity
    }
  }
  __shared__ int box[6];
  if (threadIdx.x < 6) box[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : -1;
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int l = __reduce_min_sync(0xffffffffu, lo[a]), h = __reduce_max_sync(0xffffffffu, hi[a]);
    if ((threadIdx.x & 31) == 0 && h >= 0) {
      atomicMin(&box[a], l);
      atomicMax(&box[3 + a], h);
    }
  }
  __syncthreads();
  if (threadIdx.x < 3 && box[3] >= 0) {
    atomicMin(&D.ctr[CTR_BOX + threadIdx.x], box[threadIdx.x]);
    atomicMax(&D.ctr[CTR_BOX + 3 + threadIdx.x], box[3 + threadIdx.x]);
  }
}
__global__ void k_writeback(CafeDev D, CafeConsts K) {
  d_writeback(D, K, blockIdx.x, gridDim.x);
}

// ConvertSolid1(0): mushy cells whose neighbours are all mushy or solid become
// solid with zero extent. Every mushy cell is in this step's active list. In
// place is equivalent to collect-then-apply: 2 -> 3 keeps "neighbour >= 2". A row of
// three neighbours is read as a word; bound by load latency (7 us; byte by byte
// through a local array 11).
__device__ __forceinline__ void d_mushy2solid(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  int na = D.ctr[CTR_NA];
  if (na > D.act_cap) na = (int)D.act_cap;
  for (int p = cafe_bid * blockDim.x + threadIdx.x; p < na; p += cafe_nblk * blockDim.x) {
    if (D.a_state[p] != 2) continue;
    long long idx = D.act[p];
    int i, j, k;
    cafe_cell_xyz(K, idx, i, j, k);
    // the two or three states around i of each neighbouring row as bytes of one
    // word: mushy and solid (2, 3) have the second bit
    const int x0 = i > 0 ? i - 1 : 0, n = min(i + 1, K.nx - 1) - x0 + 1;
    const unsigned long long need = 0x020202ULL & ((1ULL << (8 * n)) - 1ULL);
    bool all = true;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      const int y = j + r % 3 - 1, z = k + r / 3 - 1;
      if (y < 0 || y >= K.ny || z < 0 || z >= K.nz) continue;
      all = all && (cafe_load8(D.state, (long long)K.nxy * z + (long long)K.nx * y + x0) & need) == need;
    }
    if (all) {
      D.state[idx] = 3;
      D.ext[idx] = 0.0;
    }
  }
}
__global__ void k_mushy2solid(CafeDev D, CafeConsts K) {
  d_mushy2solid(D, K, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------ grains
__global__ void k_rot_range(CafeDev D, int g0, int g1) {
  for (int g = g0 + blockIdx.x * blockDim.x + threadIdx.x; g < g1; g += gridDim.x * blockDim.x)
    cafe_rot_from_cth(D.cth + 4LL * g, D.rot + 9LL * g);
}

// CleanLayer (VoxelsCA.C:800-839): grain volumes, renumbering, compaction.
__global__ void k_grain_count(CafeDev D, CafeConsts K, int32_t *cnt) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K.N;
       idx += (long long)gridDim.x * blockDim.x) {
    int g = D.gid[idx];
    if (g > 0) atomicAdd(&cnt[g - 1], 1);
  }
}
// Single block: newid[g] (1-based, 0 = dropped) and compacted grain tables.
__global__ void k_grain_renumber(CafeDev D, const int32_t *cnt, int32_t *newid, double *cth2,
                                 double *rot2) {
  __shared__ int part[1024];
  int ng = D.ctr[CTR_NGRAIN];
  int per = (ng + blockDim.x - 1) / blockDim.x;
  int b0 = threadIdx.x * per, b1 = min(b0 + per, ng);
  int s = 0;
  for (int g = b0; g < b1; ++g) s += cnt[g] > 0;
  part[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int t = 0; t < (int)blockDim.x; ++t) {
      int v = part[t];
      part[t] = acc;
      acc += v;
    }
    D.ctr[CTR_NVS2_END] = acc;  // scratch: new grain count
  }
  __syncthreads();
  int k = part[threadIdx.x];
  for (int g = b0; g < b1; ++g) {
    if (cnt[g] > 0) {
      newid[g] = k + 1;
      for (int a = 0; a < 4; ++a) cth2[4LL * k + a] = D.cth[4LL * g + a];
      for (int a = 0; a < 9; ++a) rot2[9LL * k + a] = D.rot[9LL * g + a];
      ++k;
    } else {
      newid[g] = 0;
    }
  }
}
__global__ void k_gid_remap(CafeDev D, CafeConsts K, const int32_t *newid) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K.N;
       idx += (long long)gridDim.x * blockDim.x) {
    int g = D.gid[idx];
    if (g != 0) D.gid[idx] = newid[g - 1];
  }
}

// ------------------------------------------------------------------ Voronoi
// Nearest site with the reference's distance (dx^2 + dy^2) + dz^2 and its
// first-minimum rule (BasePlate.C:269-272, VoxelsCA.C:925-930). Sites are
// bucketed on a uniform grid; rings of buckets are searched until no unvisited
// bucket can hold a site whose rounded distance could reach the best found.
struct CafeSiteGrid {
  const double *xyz;      // 3 per site
  const float4 *near;     // per entry of idx: the site in single precision and its index
  const int32_t *start;   // bucket CSR
  const int32_t *idx;     // site indices, ascending inside a bucket
  double lo[3], h;
  float top;              // largest magnitude of a site's coordinates and the grid's corners
  int nb[3];
};

// The nearest site when single precision tells it from all others, else -1. A
// cell meets about ninety sites; their distances in double precision (8 operations of
// 64 cycles each) made the baseplate of 512 x 256 x 80 cells 28 ms. A coordinate
// difference is in error by at most 2^-23 (|q| + |site|) < e, a distance by
// sqrt(3) e and a relative 2^-22; the sites left out lie beyond `gap`.
__device__ __forceinline__ int cafe_nearest_site_f32(const CafeSiteGrid &G, double q0, double q1, double q2) {
  const float q[3] = {(float)q0, (float)q1, (float)q2}, h = (float)G.h;
  const float e = 1.3e-7f * (fmaxf(fmaxf(fabsf(q[0]), fabsf(q[1])), fabsf(q[2])) + G.top);
  float lo[3];
  int qb[3];
  for (int a = 0; a < 3; ++a) {
    lo[a] = (float)G.lo[a];
    qb[a] = min(max((int)((q[a] - lo[a]) / h), 0), G.nb[a] - 1);
  }
  float best = INFINITY, second = INFINITY;
  int besti = -1;
  const int rmax = max(G.nb[0], max(G.nb[1], G.nb[2]));
  for (int r = 0; r <= rmax; ++r) {
    for (int bz = max(qb[2] - r, 0); bz <= min(qb[2] + r, G.nb[2] - 1); ++bz) {
      for (int by = max(qb[1] - r, 0); by <= min(qb[1] + r, G.nb[1] - 1); ++by) {
        // the ring's buckets of this row: all of them, or the two ends
        const int row = (bz * G.nb[1] + by) * G.nb[0];
        const bool edge = bz == qb[2] - r || bz == qb[2] + r || by == qb[1] - r || by == qb[1] + r;
        for (int end = 0; end < (edge ? 1 : 2); ++end) {
          const int x0 = edge ? max(qb[0] - r, 0) : (end ? qb[0] + r : qb[0] - r);
          const int x1 = edge ? min(qb[0] + r, G.nb[0] - 1) : x0;
          if (x0 < 0 || x1 >= G.nb[0]) continue;
          const int t1 = G.start[row + x1 + 1];
          for (int t = G.start[row + x0]; t < t1; ++t) {
            const float4 p = G.near[t];
            const float a = q[0] - p.x, b = q[1] - p.y, c = q[2] - p.z;
            const float d = a * a + b * b + c * c;
            if (d < best) {
              second = best;
              best = d;
              besti = __float_as_int(p.w);
            } else if (d < second) {
              second = d;
            }
          }
        }
      }
    }
    // lower bound on the distance to any bucket outside rings 0..r
    float gap = INFINITY;
    for (int a = 0; a < 3; ++a) {
      if (qb[a] - r - 1 >= 0) gap = fminf(gap, q[a] - (lo[a] + (float)(qb[a] - r) * h));
      if (qb[a] + r + 1 < G.nb[a]) gap = fminf(gap, (lo[a] + (float)(qb[a] + r + 1) * h) - q[a]);
    }
    if (gap == INFINITY) break;  // (no bucket is left)
    if (gap - 4.f * e > sqrtf(best) * (1.f + 1e-6f) + 4.f * e) break;
  }
  const float s1 = sqrtf(best), s2 = sqrtf(second);
  return second == INFINITY || s2 - s1 > 4.f * e + 1e-6f * s2 ? besti : -1;
}
__device__ int cafe_nearest_site(const CafeSiteGrid &G, double q0, double q1, double q2) {
  const int near = cafe_nearest_site_f32(G, q0, q1, q2);
  if (near >= 0) return near;
  double q[3] = {q0, q1, q2};
  int qb[3];
  for (int a = 0; a < 3; ++a) {
    double f = floor((q[a] - G.lo[a]) / G.h);
    int b = f < 0 ? 0 : (f > G.nb[a] - 1 ? G.nb[a] - 1 : (int)f);
    qb[a] = b;
  }
  double best = INFINITY;
  int besti = -1;
  int rmax = max(G.nb[0], max(G.nb[1], G.nb[2]));
  for (int r = 0; r <= rmax; ++r) {
    for (int dz = -r; dz <= r; ++dz) {
      int bz = qb[2] + dz;
      if (bz < 0 || bz >= G.nb[2]) continue;
      for (int dy = -r; dy <= r; ++dy) {
        int by = qb[1] + dy;
        if (by < 0 || by >= G.nb[1]) continue;
        bool edge = (abs(dz) == r || abs(dy) == r);
        for (int dxx = -r; dxx <= r; dxx += (edge ? 1 : (2 * r > 0 ? 2 * r : 1))) {
          int bx = qb[0] + dxx;
          if (bx < 0 || bx >= G.nb[0]) continue;
          int b = (bz * G.nb[1] + by) * G.nb[0] + bx;
          for (int t = G.start[b]; t < G.start[b + 1]; ++t) {
            int i = G.idx[t];
            double a = q0 - G.xyz[3LL * i], bb = q1 - G.xyz[3LL * i + 1], c = q2 - G.xyz[3LL * i + 2];
            double d = a * a + bb * bb + c * c;
            if (d < best || (d == best && i < besti)) {
              best = d;
              besti = i;
            }
          }
          if (r == 0) break;
        }
      }
    }
    // lower bound on the distance to any bucket outside rings 0..r
    double gap = INFINITY;
    bool more = false;
    for (int a = 0; a < 3; ++a) {
      if (qb[a] - r - 1 >= 0) {
        more = true;
        double g = q[a] - (G.lo[a] + (qb[a] - r) * G.h);
        gap = g < gap ? g : gap;
      }
      if (qb[a] + r + 1 < G.nb[a]) {
        more = true;
        double g = (G.lo[a] + (qb[a] + r + 1) * G.h) - q[a];
        gap = g < gap ? g : gap;
      }
    }
    if (!more) break;
    gap -= 1e-9 * G.h;
    if (besti >= 0 && gap > 0 && gap * gap > best * (1.0 + 1e-9)) break;
  }
  return besti;
}

// Baseplate (BasePlate.C:262-273 + VoxelsCA.C:133-141, 148-156): cell centres,
// cells below z = Nzh-1 solid, the top baseplate plane mushy.
__global__ void k_baseplate(CafeDev D, CafeConsts K, CafeSiteGrid G, int Nzh) {
  long long nbp = (long long)Nzh * K.nxy;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < nbp;
       idx += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    cafe_cell_xyz(K, idx, i, j, k);
    double x = (i + .5) * K.dx[0], y = (j + .5) * K.dx[1], z = (k + .5) * K.dx[2];
    int s = cafe_nearest_site(G, x, y, z);
    D.gid[idx] = s + 1;
    D.state[idx] = idx < (long long)(Nzh - 1) * K.nxy ? 3 : 2;
    D.cx[idx] = ((double)i + .5) * K.dx[0];
    D.cy[idx] = ((double)j + .5) * K.dx[1];
    D.cz[idx] = ((double)k + .5) * K.dx[2];
  }
}

// AddLayer1 part 1 (VoxelsCA.C:922-936): nearest site (corner coordinates) for
// every cell of the layer slab [iz1, ilaserLoc) (also beyond the box top, as
// the reference does), and the used-site flags.
__global__ void k_layer_voronoi(CafeConsts K, CafeSiteGrid G, int iz1, int ilaser, int32_t *gtmp,
                                int32_t *used) {
  long long nslab = (long long)K.nxy * (ilaser - iz1);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nslab;
       t += (long long)gridDim.x * blockDim.x) {
    int k = iz1 + (int)(t / K.nxy);
    long long r = t % K.nxy;
    int j = (int)(r / K.nx), i = (int)(r % K.nx);
    double x = i * K.dx[0], y = j * K.dx[1], z = k * K.dx[2];
    int s = cafe_nearest_site(G, x, y, z);
    gtmp[t] = s;
    used[s] = 1;
  }
}
// AddLayer1 part 2 (VoxelsCA.C:952-981): new grain IDs, solid state, cell
// centres inside the slab; empty state above the laser plane.
__global__ void k_layer_apply(CafeDev D, CafeConsts K, int iz1, int ilaser, const int32_t *gtmp,
                              const int32_t *map, int ngrain0) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K.N;
       idx += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    cafe_cell_xyz(K, idx, i, j, k);
    if (k >= iz1 && k < ilaser) {
      long long t = (long long)(k - iz1) * K.nxy + (long long)j * K.nx + i;
      D.gid[idx] = ngrain0 + map[gtmp[t]] + 1;
      D.state[idx] = 3;
      D.cx[idx] = ((double)i + .5) * K.dx[0];
      D.cy[idx] = ((double)j + .5) * K.dx[1];
      D.cz[idx] = ((double)k + .5) * K.dx[2];
    }
    if (idx >= (long long)K.nxy * ilaser) {
      D.state[idx] = 0;
      D.gid[idx] = 0;
    }
  }
}

// TempField::TempCurr for output (the step computes it on the fly).
__global__ void k_temperature(CafeConsts K, CafeStepParams P, double *T) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K.N;
       idx += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    cafe_cell_xyz(K, idx, i, j, k);
    T[idx] = K.Tcls[cafe_temp_class_exact(K, P, i, j, k)];
  }
}

// ------------------------------------------------------------------ host transfers
// Layout conversions between the device state and the C ABI's host layout
// (int32 vState/BuildjID, interleaved centres), one staging chunk at a time.
__global__ void k_u8_to_i32(const uint8_t *src, int32_t *dst, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}
// Converts and checks 0 <= v <= vmax; a bad value sets bit `bad_bit` of *bad.
__global__ void k_i32_to_u8_check(const int32_t *src, uint8_t *dst, long long n, int vmax, int *bad, int bad_bit) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    int v = src[i];
    if (v < 0 || v > vmax) atomicOr(bad, bad_bit);
    dst[i] = (uint8_t)v;
  }
}
__global__ void k_check_range_i32(const int32_t *a, long long n, int vmax, int *bad, int bad_bit) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    int v = a[i];
    if (v < 0 || v > vmax) atomicOr(bad, bad_bit);
  }
}
__global__ void k_interleave3(const double *x, const double *y, const double *z, double *dst, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    dst[3 * i] = x[i];
    dst[3 * i + 1] = y[i];
    dst[3 * i + 2] = z[i];
  }
}
__global__ void k_deinterleave3(const double *src, double *x, double *y, double *z, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    x[i] = src[3 * i];
    y[i] = src[3 * i + 1];
    z[i] = src[3 * i + 2];
  }
}

// ------------------------------------------------------------------ output
// VoxelsCA::Build. InitializeVoxels marks the baseplate cells that carry a
// grain (VoxelsCA.C:156-159); SetBuild (VoxelsCA.C:76-115) marks every cell of
// every grain that has a melted cell (BuildjID = 1) or a Build cell. The
// reference does this in two passes; the grains of its second pass are those
// of the first plus those of the Build cells, so one flag pass over both
// conditions and one marking pass give the same field.
__global__ void k_build_init(CafeDev D, CafeConsts K) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K.N;
       idx += (long long)gridDim.x * blockDim.x)
    D.build[idx] = D.gid[idx] != 0;
}
__global__ void k_build_flag(CafeDev D, CafeConsts K, uint8_t *gflag) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K.N;
       idx += (long long)gridDim.x * blockDim.x) {
    int g = D.gid[idx];
    if (g > 0 && (D.buildj[idx] == 1 || D.build[idx] == 1)) gflag[g] = 1;
  }
}
__global__ void k_build_mark(CafeDev D, CafeConsts K, const uint8_t *gflag) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K.N;
       idx += (long long)gridDim.x * blockDim.x) {
    int g = D.gid[idx];
    if (g > 0 && gflag[g]) D.build[idx] = 1;
  }
}

// One direction of the IPF colouring (VoxelsCA.C:1645-1702 for z, 1703-1760
// for x, 1761-1810 for y) for rotation R. With own_hue false the hue starts
// from H as given (the reference's y direction adds to the x direction's hue),
// and the hue fraction is H/6 as the reference writes it.
__device__ void cafe_ipf_dir(const CafeIpfConsts &C, const double R[3][3], int dir, bool own_hue, double &H,
                             float *rgb) {
  const double v[3] = {dir == 1 ? 1.0 : 0.0, dir == 2 ? 1.0 : 0.0, dir == 0 ? 1.0 : 0.0};
  double a = fabs(R[0][0] * v[0] + R[1][0] * v[1] + R[2][0] * v[2]);
  double b = fabs(R[0][1] * v[0] + R[1][1] * v[1] + R[2][1] * v[2]);
  double c = fabs(R[0][2] * v[0] + R[1][2] * v[1] + R[2][2] * v[2]);
  // std::sort of three (libstdc++'s insertion sort, order of comparisons
  // kept), then the swap of the first two
  if (b < a) { double t = a; a = b; b = t; }
  if (c < a) { double t = c; c = b; b = a; a = t; }
  else if (c < b) { double t = c; c = b; b = t; }
  double v0 = b, v1 = a, v2 = (1.0 < c) ? 1.0 : c;
  double xp = 2. * v0 / (1. + v2);
  double yp = 2. * v1 / (1. + v2);
  if (own_hue) {
    H = crm_atan2((yp - C.y0) / (xp - C.x0), 1.0) * 180. / 3.14159265358979323846;
    if (xp < C.x0) H += 180;
  }
  H = H + 240 - C.hoff;
  const double V = 1.;
  double S = crm_pow_half((xp - C.x0) * (xp - C.x0) + (yp - C.y0) * (yp - C.y0));
  S = S / C.sMax * 0.8 + 0.2;
  if (H >= 360.0) H = 0.0;
  int icase = (int)floor(H / 60.0);
  double ff = H / 6.0 - icase;
  double p = V * (1. - S), q = V * (1. - S * ff), tt = V * (1. - (S * (1. - ff)));
  float r0 = 0.0f, r1 = 0.0f, r2 = 0.0f;
  if (!(S <= 0.0)) {
    switch (icase) {
      case 0: r0 = (float)V; r1 = (float)tt; r2 = (float)p; break;
      case 1: r0 = (float)q; r1 = (float)V; r2 = (float)p; break;
      case 2: r0 = (float)p; r1 = (float)V; r2 = (float)tt; break;
      case 3: r0 = (float)p; r1 = (float)q; r2 = (float)V; break;
      case 4: r0 = (float)tt; r1 = (float)p; r2 = (float)V; break;
      case 5: r0 = (float)V; r1 = (float)p; r2 = (float)q; break;
      default: break;
    }
  }
  rgb[0] = r0;
  rgb[1] = r1;
  rgb[2] = r2;
}
// IPF colours of grains [0, ngrain): 9 floats per grain (z, x, y directions).
__global__ void k_ipf_grains(const double *cth, int ngrain, CafeIpfConsts C, float *out) {
  for (int gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngrain; gi += gridDim.x * blockDim.x) {
    const double *cc = cth + 4LL * gi;
    double omega = cc[0], ax[3] = {cc[1], cc[2], cc[3]};
    double co = crm_cos(omega), so = crm_sin(omega);
    double R[3][3];
    // VoxelsCA.C:1635-1644, with pow(a, 2.0) = a*a
    R[0][0] = co + (ax[0] * ax[0]) * (1 - co);
    R[0][1] = ax[0] * ax[1] * (1 - co) - ax[2] * so;
    R[0][2] = ax[0] * ax[2] * (1 - co) + ax[1] * so;
    R[1][0] = ax[0] * ax[1] * (1 - co) + ax[2] * so;
    R[1][1] = co + (ax[1] * ax[1]) * (1 - co);
    R[1][2] = ax[1] * ax[2] * (1 - co) - ax[0] * so;
    R[2][0] = ax[2] * ax[0] * (1 - co) - ax[1] * so;
    R[2][1] = ax[2] * ax[1] * (1 - co) + ax[0] * so;
    R[2][2] = co + (ax[2] * ax[2]) * (1 - co);
    double H = 0.0;
    float *o = out + 9LL * gi;
    cafe_ipf_dir(C, R, 0, true, H, o);
    cafe_ipf_dir(C, R, 1, true, H, o + 3);
    cafe_ipf_dir(C, R, 2, false, H, o + 6);
  }
}
// Per-cell colours of direction `d` (0 z, 1 x, 2 y) for cells [off, off+n).
__global__ void k_ipf_cells(CafeDev D, const float *gcol, int d, long long off, long long n, float *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    int g = D.gid[off + i];
    float r = 0.0f, gg = 0.0f, b = 0.0f;
    if (g >= 1) {
      const float *c = gcol + 9LL * (g - 1) + 3 * d;
      r = c[0];
      gg = c[1];
      b = c[2];
    }
    out[3 * i] = r;
    out[3 * i + 1] = gg;
    out[3 * i + 2] = b;
  }
}
// TempField::TempCurr as float for cells [off, off+n) (WriteToHDF1's TempOut).
__global__ void k_temperature_f(CafeConsts K, CafeStepParams P, long long off, long long n, float *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    int a, b, c;
    cafe_cell_xyz(K, off + i, a, b, c);
    out[i] = (float)K.Tcls[cafe_temp_class_exact(K, P, a, b, c)];
  }
}
// Build as int32 for cells [off, off+n).
__global__ void k_build_i32(CafeDev D, long long off, long long n, int32_t *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = D.build[off + i];
}

// ------------------------------------------------------------------ EASM
// TempField::EASM (TempField.C:79-137): per cell below the laser plane the
// damped fixed point of Utilities::EASM_Temp_LG (Utilities.C:128-140) on
// Utilities::Integral (Utilities.C:105-124) = 300 + sum_i w_i f(x_i), f the
// moving-Gaussian-source kernel Temp_Fun_G (Utilities.C:228-249) with the 316L
// properties at the iterate (Utilities.C:39-76). Expressions keep the
// reference's order; pow(x, 2) is x*x, pow(t - x, -0.5) and exp are the
// correctly rounded functions of cafe_crmath.h.
__device__ __forceinline__ void cafe_easm_materials(double T, double M[4]) {
  double rho, cP, k;
  if (T < 1660)
    rho = 8084.2 - 0.42086 * T - 3.8942 * 1e-5 * T * T;
  else if (T >= 1660 && T < 3090)
    rho = 7432.7 + 3.9338 * 1e-2 * T - 1.8007 * 1e-4 * T * T;
  else
    rho = 6124.72;
  if (T < 1660)
    cP = 458.984 + 0.1328 * T;
  else
    cP = 769.855;
  if (T < 1660)
    k = 9.248 + 1.571 * 1e-2 * T;
  else if (T >= 1660 && T < 3090)
    k = 12.41 + 3.279 * 1e-3 * T;
  else
    k = 21.6465;
  M[0] = cP;
  M[1] = k;
  M[2] = rho;
  M[3] = crm_div_int(k, rho * cP);
}
// What an integral's nodes share: C of Temp_Fun_G, the material's M[3], the
// squared distances across and below.
struct CafeEasmPoint {
  double C, M3, dy2, dz2;
};
__device__ __forceinline__ CafeEasmPoint cafe_easm_point(const CafeEasm &E, double R1, double R2, double Ly, double Lz,
                                                         double T) {
  const double eta = 0.56, pi = 3.14159265358979323846;
  double M[4];
  cafe_easm_materials(T, M);
  const double dy = R1 - Ly, dz = fabs(R2 - Lz);
  CafeEasmPoint p;
  p.C = crm_div_int(eta * E.Q, pi * M[2] * M[0] * crm_sqrt_int(4 * pi * M[3]));
  p.M3 = M[3];
  p.dy2 = dy * dy;
  p.dz2 = dz * dz;
  return p;
}
// Term i of the rule. The field is bound by FP64 issue: with floating-point
// divisions and exp a node took ~110 FP64 instructions, with the integer ones
// (cafe_intmath.h, the same bits) ten.
__device__ __forceinline__ double cafe_easm_node(const CafeEasm &E, const CafeEasmPoint &p, int i, double Lx, double R0) {
  const double sigma = 50.0e-6;
  const double m = 2 * p.M3 * E.tx[i], d = m + sigma * sigma, dx = R0 - Lx;
  // (4 M3 tx + 2 sigma^2 and 4 M3 tx are exactly 2 d and 2 m)
  const crm_recip rd = crm_reciprocal(d);
  const double a = crm_quotient(p.C * E.r[i], rd, d, 0);
  const double arg = -crm_quotient(dx * dx + p.dy2, rd, d, 1) - crm_quotient(p.dz2, crm_reciprocal(m), m, 1);
  return E.qw[i] * (a * crm_exp_int(arg));
}
__device__ __forceinline__ double cafe_easm_integral(const CafeEasm &E, const double *Lx, double R0, double R1,
                                                     double R2, double Ly, double Lz, double T) {
  const CafeEasmPoint p = cafe_easm_point(E, R1, R2, Ly, Lz, T);
  double s = 0.0;
  for (int i = 0; i < CAFE_EASM_NODES; ++i) s += cafe_easm_node(E, p, i, Lx[i], R0);
  return 300 + s;
}
__global__ void k_set_int(int *p, int v) { *p = v; }
__global__ void k_easm_reset(CafeDev D) {
  int t = threadIdx.x;
  if (t < 3) D.ctr[CTR_EASM_BOX + t] = 0x7fffffff;
  else if (t < 6) D.ctr[CTR_EASM_BOX + t] = -1;
  else if (t == 6) D.ctr[CTR_EASM_COLD] = 0;
  else if (t == 7) *(unsigned long long *)&D.ctr[CTR_EASM_CURSOR] = 0ULL;
  else if (t == 8) D.ctr[CTR_EASM_QN] = 0;
  else if (t == 9) D.ctr[CTR_EASM_QHEAD] = 0;
}
// Cells [0, ncell) (cells above the laser plane keep T = 0). Writes temp,
// BuildjID, the box of the cells at or above the liquidus and the "some cell
// below the liquidus" flag. Cells need 2 to 100 integrals each, so each
// thread takes the next cell from a shared cursor whenever its own has
// converged: the lanes of a warp then run the same 25-node loop together
// instead of idling behind the slowest cell of a fixed assignment.
__global__ void k_easm(CafeDev D, CafeConsts K, CafeStepParams P, CafeEasm E, long long ncell) {
  __shared__ double s_Lx[CAFE_EASM_NODES];
  __shared__ int s_box[6], s_cold;
  __shared__ unsigned long long s_integrals;
  const double t = 80.0e-5;
  if (threadIdx.x < CAFE_EASM_NODES) {
    double x0 = P.lx - E.bmV * t;  // Utilities.C:243-244
    s_Lx[threadIdx.x] = x0 + E.bmV * E.qx[threadIdx.x];
  }
  if (threadIdx.x < 3) {
    s_box[threadIdx.x] = 0x7fffffff;
    s_box[3 + threadIdx.x] = -1;
  }
  if (threadIdx.x == 0) {
    s_cold = 0;
    s_integrals = 0;
  }
  __syncthreads();
  unsigned long long nint = 0;
  int bx0 = 0x7fffffff, by0 = 0x7fffffff, bz0 = 0x7fffffff, bx1 = -1, by1 = -1, bz1 = -1, cold = 0;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  long long idx = -1;  // this lane's cell, -1 when it needs one
  bool exhausted = false;
  int ci = 0, cj = 0, ck = 0, n = 0, done_here = 0;
  bool first = true;
  double xp = 0, yp = 0, zp = 0, Told = 0, Tnew = 0, Tin = 0;
  // warp-synchronous rounds: lanes without a cell take new ones together (one
  // atomic per warp), then every lane evaluates one integral (lanes without a
  // cell on dummy inputs, discarded), so the warp stays converged
  while (true) {
    bool need = idx < 0 && !exhausted;
    unsigned needm = __ballot_sync(FULL, need);
    if (needm) {
      unsigned long long base = 0;
      int leader = __ffs(needm) - 1;
      if (lane == leader) base = atomicAdd((unsigned long long *)&D.ctr[CTR_EASM_CURSOR], (unsigned long long)__popc(needm));
      base = __shfl_sync(FULL, base, leader);
      if (need) {
        long long r = (long long)(base + __popc(needm & ((1u << lane) - 1u)));
        // from the top down: the cells just below the laser plane take the most
        // integrals, and handing them out first keeps the end of the pass from
        // waiting on a few long cells
        long long c = ncell - 1 - r;
        if (r >= ncell) {
          exhausted = true;
        } else {
          cafe_cell_xyz(K, c, ci, cj, ck);
          double x0 = ((double)ci + .5) * K.dx[0];
          double y0 = ((double)cj + .5) * K.dx[1];
          zp = ((double)ck + .5) * K.dx[2];
          if (zp > P.lz) {
            // above the laser plane: T stays 0 (TempField.C:99)
          } else if ((x0 > P.lx) && (zp > (P.lz - E.layerT))) {
            double T = .99 * K.T0;
            D.temp[c] = T;
            if (T > K.tL)
              D.buildj[c] = 1;
            else if (T < K.T0)
              D.buildj[c] = 0;
            if (T >= K.tL) {
              bx0 = min(bx0, ci); by0 = min(by0, cj); bz0 = min(bz0, ck);
              bx1 = max(bx1, ci); by1 = max(by1, cj); bz1 = max(bz1, ck);
            } else {
              cold = 1;
            }
          } else {
            xp = P.cg * (x0 - K.hLX0) + P.sg * (y0 - K.hLX1) + K.hLX0;
            yp = -P.sg * (x0 - K.hLX0) + P.cg * (y0 - K.hLX1) + K.hLX1;
            idx = c;
            first = true;
            Told = 0.0;
            Tin = 0.0;
            n = 0;
            done_here = 0;
          }
        }
      }
    }
    const bool work = idx >= 0;
    if (__all_sync(FULL, !work && exhausted)) break;
    if (!__any_sync(FULL, work)) continue;  // only cells without integrals were taken
    // one integral per lane; then the step of Utilities::EASM_Temp_LG's loop
    double Tres = cafe_easm_integral(E, s_Lx, xp, yp, zp, P.ly, P.lz, Tin);
    if (!work) continue;
    ++nint;
    if (first) {
      Tnew = Tres;
      first = false;
    } else {
      Tnew = 0.5 * (Told + Tres);
      n++;
    }
    if (fabs(Told - Tnew) > 10.0 && n < 100) {
      // a long fixed point goes on in the warp-per-cell pass (when the queue
      // has room), from this point of the loop: test passed, next integral due
      if (++done_here >= CAFE_EASM_LANE_INTEGRALS) {
        int slot = atomicAdd(&D.ctr[CTR_EASM_QN], 1);
        if (slot < D.easm_qcap) {
          CafeEasmItem it;
          it.idx = idx;
          it.Told = Told;
          it.Tnew = Tnew;
          it.n = n;
          it.pad = 0;
          D.easm_q[slot] = it;
          idx = -1;
          continue;
        }
      }
      Told = Tnew;
      Tin = Told;
      continue;
    }
    double T = Tnew;
    D.temp[idx] = T;
    if (T > K.tL)
      D.buildj[idx] = 1;
    else if (T < K.T0)
      D.buildj[idx] = 0;
    if (T >= K.tL) {
      bx0 = min(bx0, ci); by0 = min(by0, cj); bz0 = min(bz0, ck);
      bx1 = max(bx1, ci); by1 = max(by1, cj); bz1 = max(bz1, ck);
    } else {
      cold = 1;
    }
    idx = -1;
  }
  if (bx1 >= 0) {
    atomicMin(&s_box[0], bx0); atomicMin(&s_box[1], by0); atomicMin(&s_box[2], bz0);
    atomicMax(&s_box[3], bx1); atomicMax(&s_box[4], by1); atomicMax(&s_box[5], bz1);
  }
  if (cold) s_cold = 1;
  if (nint) atomicAdd(&s_integrals, nint);
  __syncthreads();
  if (threadIdx.x == 0 && s_integrals) atomicAdd(&D.stat[STAT_EASM_INTEGRALS], s_integrals);
  if (threadIdx.x < 3 && s_box[3 + threadIdx.x] >= 0) {
    atomicMin(&D.ctr[CTR_EASM_BOX + threadIdx.x], s_box[threadIdx.x]);
    atomicMax(&D.ctr[CTR_EASM_BOX + 3 + threadIdx.x], s_box[3 + threadIdx.x]);
  }
  if (threadIdx.x == 0 && s_cold) D.ctr[CTR_EASM_COLD] = 1;
}
// Utilities::Integral for one cell with the 25 nodes spread over the lanes of
// a warp; the weighted terms are added in node order on every lane, as the
// quadrature sum does, so the result is that of cafe_easm_integral.
__device__ __forceinline__ double cafe_easm_integral_warp(const CafeEasm &E, const double *Lx, double R0, double R1,
                                                          double R2, double Ly, double Lz, double T, int lane) {
  const unsigned FULL = 0xffffffffu;
  const CafeEasmPoint pt = cafe_easm_point(E, R1, R2, Ly, Lz, T);
  const double p = lane < CAFE_EASM_NODES ? cafe_easm_node(E, pt, lane, Lx[lane], R0) : 0.0;
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < CAFE_EASM_NODES; ++i) s += __shfl_sync(FULL, p, i);
  return 300 + s;
}

// The cells queued by k_easm: one warp per cell until its fixed point ends.
__global__ void k_easm_long(CafeDev D, CafeConsts K, CafeStepParams P, CafeEasm E) {
  __shared__ double s_Lx[CAFE_EASM_NODES];
  __shared__ int s_box[6], s_cold;
  __shared__ unsigned long long s_integrals;
  const double t = 80.0e-5;
  if (threadIdx.x < CAFE_EASM_NODES) {
    double x0 = P.lx - E.bmV * t;
    s_Lx[threadIdx.x] = x0 + E.bmV * E.qx[threadIdx.x];
  }
  if (threadIdx.x < 3) {
    s_box[threadIdx.x] = 0x7fffffff;
    s_box[3 + threadIdx.x] = -1;
  }
  if (threadIdx.x == 0) {
    s_cold = 0;
    s_integrals = 0;
  }
  __syncthreads();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int nq = D.ctr[CTR_EASM_QN];
  if (nq > D.easm_qcap) nq = (int)D.easm_qcap;
  unsigned long long nint = 0;
  int bx0 = 0x7fffffff, by0 = 0x7fffffff, bz0 = 0x7fffffff, bx1 = -1, by1 = -1, bz1 = -1, cold = 0;
  while (true) {
    int q = 0;
    if (lane == 0) q = atomicAdd(&D.ctr[CTR_EASM_QHEAD], 1);
    q = __shfl_sync(FULL, q, 0);
    if (q >= nq) break;
    CafeEasmItem it = D.easm_q[q];
    int ci, cj, ck;
    cafe_cell_xyz(K, it.idx, ci, cj, ck);
    double x0 = ((double)ci + .5) * K.dx[0];
    double y0 = ((double)cj + .5) * K.dx[1];
    double zp = ((double)ck + .5) * K.dx[2];
    double xp = P.cg * (x0 - K.hLX0) + P.sg * (y0 - K.hLX1) + K.hLX0;
    double yp = -P.sg * (x0 - K.hLX0) + P.cg * (y0 - K.hLX1) + K.hLX1;
    double Told = it.Told, Tnew = it.Tnew;
    int n = it.n;
    // continue Utilities::EASM_Temp_LG's loop where the lane pass left it
    while (fabs(Told - Tnew) > 10.0 && n < 100) {
      Told = Tnew;
      double Tt = cafe_easm_integral_warp(E, s_Lx, xp, yp, zp, P.ly, P.lz, Told, lane);
      Tnew = 0.5 * (Told + Tt);
      n++;
      ++nint;
    }
    if (lane == 0) {
      double T = Tnew;
      D.temp[it.idx] = T;
      if (T > K.tL)
        D.buildj[it.idx] = 1;
      else if (T < K.T0)
        D.buildj[it.idx] = 0;
      if (T >= K.tL) {
        bx0 = min(bx0, ci); by0 = min(by0, cj); bz0 = min(bz0, ck);
        bx1 = max(bx1, ci); by1 = max(by1, cj); bz1 = max(bz1, ck);
      } else {
        cold = 1;
      }
    }
  }
  if (bx1 >= 0) {
    atomicMin(&s_box[0], bx0); atomicMin(&s_box[1], by0); atomicMin(&s_box[2], bz0);
    atomicMax(&s_box[3], bx1); atomicMax(&s_box[4], by1); atomicMax(&s_box[5], bz1);
  }
  if (cold) s_cold = 1;
  if (lane == 0 && nint) atomicAdd(&s_integrals, nint);
  __syncthreads();
  if (threadIdx.x == 0 && s_integrals) atomicAdd(&D.stat[STAT_EASM_INTEGRALS], s_integrals);
  if (threadIdx.x < 3 && s_box[3 + threadIdx.x] >= 0) {
    atomicMin(&D.ctr[CTR_EASM_BOX + threadIdx.x], s_box[threadIdx.x]);
    atomicMax(&D.ctr[CTR_EASM_BOX + 3 + threadIdx.x], s_box[3 + threadIdx.x]);
  }
  if (threadIdx.x == 0 && s_cold) D.ctr[CTR_EASM_COLD] = 1;
}

// SetLiquid3 (VoxelsCA.C:1098-1116) and the class map over the box of the
// cells at or above the liquidus, from the EASM temperatures.
// The Rosenthal field (extension) over cells [0, ncell): temp, BuildjID as
// AnalyticTempCurr sets it (TempField.C:180-185), the box of the cells at or
// above the liquidus and the "some cell below the liquidus" flag, in the slots
// the EASM field uses. Bound by FP64 issue: the distance's root, the division and
// exp in integers (cafe_intmath.h) took the field from 0.19 to 0.09 ms a step on
// 256x128x64 cells.
__global__ void k_rosenthal(CafeDev D, CafeConsts K, CafeStepParams P, long long ncell) {
  __shared__ int s_box[6], s_cold;
  if (threadIdx.x < 3) {
    s_box[threadIdx.x] = 0x7fffffff;
    s_box[3 + threadIdx.x] = -1;
  }
  if (threadIdx.x == 0) s_cold = 0;
  __syncthreads();
  int bx0 = 0x7fffffff, by0 = 0x7fffffff, bz0 = 0x7fffffff, bx1 = -1, by1 = -1, bz1 = -1, cold = 0;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell;
       c += (long long)gridDim.x * blockDim.x) {
    int ci, cj, ck;
    cafe_cell_xyz(K, c, ci, cj, ck);
    double T = cafe_rosenthal_T(K, P, ci, cj, ck);
    D.temp[c] = T;
    if (T > K.tL)
      D.buildj[c] = 1;
    else if (T < K.T0)
      D.buildj[c] = 0;
    if (T >= K.tL) {
      bx0 = min(bx0, ci); by0 = min(by0, cj); bz0 = min(bz0, ck);
      bx1 = max(bx1, ci); by1 = max(by1, cj); bz1 = max(bz1, ck);
    } else {
      cold = 1;
    }
  }
  if (bx1 >= 0) {
    atomicMin(&s_box[0], bx0); atomicMin(&s_box[1], by0); atomicMin(&s_box[2], bz0);
    atomicMax(&s_box[3], bx1); atomicMax(&s_box[4], by1); atomicMax(&s_box[5], bz1);
  }
  if (cold) s_cold = 1;
  __syncthreads();
  if (threadIdx.x < 3 && s_box[3 + threadIdx.x] >= 0) {
    atomicMin(&D.ctr[CTR_EASM_BOX + threadIdx.x], s_box[threadIdx.x]);
    atomicMax(&D.ctr[CTR_EASM_BOX + 3 + threadIdx.x], s_box[3 + threadIdx.x]);
  }
  if (threadIdx.x == 0 && s_cold) D.ctr[CTR_EASM_COLD] = 1;
}
__global__ void k_fill_f64(double *p, long long n, double v) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = v;
}
__global__ void k_melt_easm(CafeDev D, CafeConsts K, CafeStepParams P) {
  int bx = P.hi[0] - P.lo[0], by = P.hi[1] - P.lo[1], bz = P.hi[2] - P.lo[2];
  long long nbox = (long long)bx * by * bz;
  long long iz1 = (long long)P.ilaserLoc * K.nxy;
  int any = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nbox;
       t += (long long)gridDim.x * blockDim.x) {
    int i = P.lo[0] + (int)(t % bx);
    long long r = t / bx;
    int j = P.lo[1] + (int)(r % by);
    int k = P.lo[2] + (int)(r / by);
    long long idx = (long long)K.nxy * k + (long long)K.nx * j + i;
    double zp = ((double)k + .5) * K.dx[2];
    double T = D.temp[idx];
    int c = zp > P.lz ? 0 : (T >= K.tL ? 2 : 1);
    D.tcls[t] = (uint8_t)c;
    if (c == 2) {
      any = 1;
      if (idx < K.nxy) {
        D.state[idx] = 2;
      } else if (idx < iz1) {
        D.state[idx] = 1;
        D.gid[idx] = 0;
      }
      D.ext[idx] = 0.0;
    }
  }
  if (__syncthreads_or(any) && threadIdx.x == 0) atomicOr(&D.ctr[CTR_HOT], 1);
}
// Temperatures of cells [off, off+n) as float (output) from the EASM field.
__global__ void k_temp_copy_f(const double *T, long long off, long long n, float *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = (float)T[off + i];
}

// Sets bit `bit` of *bad if some v[i] > maxv.
__global__ void k_check_range_u8(const uint8_t *v, long long n, int maxv, int *bad, int bit) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (v[i] > maxv) atomicOr(bad, bit);
}

// ------------------------------------------------------------------ growth log
// Before k_rows_finalize: every frontier row of the step (those present at
// the start and those created by captures) gets a log entry holding its cell
// and its extent before the step's growth (a_ext still holds it: the start
// value, or the value set at capture). tau temporarily holds that extent.
__global__ void k_glog_begin(CafeDev D, const CafeStepParams *__restrict__ Pp) {
  int nrows = D.ctr[CTR_NROWS_END];
  if (nrows > D.row_cap) nrows = (int)D.row_cap;
  long long base = D.ctr[CTR_GLOG_N];
  if (base + nrows > D.glog_cap) {
    if (blockIdx.x == 0 && threadIdx.x == 0) D.ctr[CTR_GLOG_OVER] = 1;
    return;
  }
  const int tind = Pp->tInd, nrows0 = D.ctr[CTR_NROWS];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nrows; k += gridDim.x * blockDim.x) {
    int p = D.row_pos[cafe_row_at(D, nrows0, k)];
    D.glog_cell[base + k] = (int32_t)D.act[p];
    D.glog_step[base + k] = tind;
    D.glog_tau[base + k] = D.a_ext[p];
  }
}
// After k_rows_finalize: growth time = (final extent - extent before) / v
// (0 for a row that does not grow).
__global__ void k_glog_end(CafeDev D, CafeConsts K) {
  int nrows = D.ctr[CTR_NROWS_END];
  if (nrows > D.row_cap) nrows = (int)D.row_cap;
  long long base = D.ctr[CTR_GLOG_N];
  if (base + nrows > D.glog_cap) return;
  const int nrows0 = D.ctr[CTR_NROWS];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nrows; k += gridDim.x * blockDim.x) {
    int p = D.row_pos[cafe_row_at(D, nrows0, k)];
    double v = cafe_vh(D, K, p);
    double e0 = D.glog_tau[base + k];
    D.glog_tau[base + k] = v > 0.0 ? (D.a_ext[p] - e0) / v : 0.0;
  }
}
__global__ void k_glog_advance(CafeDev D) {
  int nrows = D.ctr[CTR_NROWS_END];
  if (nrows > D.row_cap) nrows = (int)D.row_cap;
  long long base = D.ctr[CTR_GLOG_N];
  if (base + nrows <= D.glog_cap) D.ctr[CTR_GLOG_N] = (int)(base + nrows);
}

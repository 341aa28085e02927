// Frontier rows and the event loop of one step (VoxelsCA.C:381-610), part of
// cafe_kernels.cu.
//
// A frontier row is a mushy cell with a liquid neighbour. Its slots are the 26
// neighbour directions; those that hold a liquid neighbour are candidates with
// capture time t = fl(fl(g - E)/v), g the slot's numerator, E the row cell's
// extent and v its growth velocity. A row's record lists its slots by g
// (CafeSlot row_slot[26]), so that its earliest candidate is the first one
// still live; row_live is the mask of live slots in that order.

// ------------------------------------------------------------------ row set-up
// Captures that can happen within the step are foreseen: when a record is
// sorted, each of its candidates that comes due before the limit tmax is
// entered in a list with the time it would be captured at, and k_children makes
// the captured cell's own row ahead of the event loop (its geometry depends
// only on the capturing row's slot), again listing its candidates. A listed
// slot carries its row's number in the upper bits of CafeSlot::m.
struct CafeChildList {
  int *n;    // entries listed so far
  int off, cap;  // first entry, one past the last one (entries are children, row D.row_cap + entry)
  double tmax;
};
__device__ __forceinline__ int cafe_slot_child(uint32_t m) { return (int)(m >> 5) - 1; }

// Sorts the slots of row r (one per lane: liv, numerator gv, neighbour position
// q) by g (NaN last among the live ones, ties by slot, the other slots after
// them) into the row's record, and forms the row's key: the order key of T + t
// for its first candidate, a lower bound of the row's absolute capture time
// (CAFE_KEY_NONE without a candidate). E and v are the row's. Returns, in every
// lane, the order key of the largest |g| of the live slots (0 when none).
__device__ __forceinline__ unsigned long long cafe_row_sort_warp(const CafeDev &D, long long r, bool liv, double gv,
                                                                 int q, double E, double v, double T, int gid,
                                                                 const CafeChildList &C) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t live = __ballot_sync(FULL, liv);
  const bool gfin = !cafe_is_nan(gv);
  const unsigned long long key = (liv && gfin) ? cafe_key_canon(gv) : CAFE_KEY_NONE;
  int rank = liv ? 0 : __popc(live);
#pragma unroll
  for (int t = 0; t < CAFE_NSLOT; ++t) {
    unsigned long long kt = cafe_shfl_u64(key, t);
    bool lt = (live >> t) & 1u;
    if (liv)
      rank += lt && (kt < key || (kt == key && t < lane));
    else
      rank += !lt && t < lane;
  }
  // the slot's capture time and, when it comes due within the step, its child
  double t = NAN;
  uint32_t child = 0;
  if (liv) {
    t = (gv - E) / v;
    if (C.off < C.cap && T + t < C.tmax) {
      const int i = C.off + atomicAdd(C.n, 1);
      if (i < C.cap) {
        child = (uint32_t)(D.row_cap + i + 1) << 5;
        D.row_pos[D.row_cap + i] = q;
        D.ch_src[i] = (int32_t)(r * CAFE_NSLOT + lane);
        D.ch_gid[i] = gid;
        D.ch_T[i] = T + t;
      }
    }
  }
  if (lane < CAFE_NSLOT) {
    CafeSlot s;
    s.g = liv ? gv : NAN;
    s.q = q;
    s.m = (uint32_t)lane | child;
    D.row_slot[r * CAFE_NSLOT + rank] = s;
    D.row_rank[r * 32 + lane] = (uint8_t)rank;
    if (lane == 0) D.row_live[r] = (1u << __popc(live)) - 1u;
  }
  if (liv && rank == 0) {
    D.row_key[r] = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(T + t);
  }
  if (lane == 0 && live == 0) D.row_key[r] = CAFE_KEY_NONE;
  unsigned long long ak = (liv && gfin) ? cafe_key(fabs(gv)) : 0ULL;
  for (int o = 16; o > 0; o >>= 1) ak = max(ak, cafe_shfl_u64_xor(ak, o));
  return ak;
}

// The captured cell's grain, centre and extent as the capture just stored
// them, handed to the fill through shared memory.
struct CafeNewCell {
  double c[3], ext;
  int gid;
};
// Per-slot partial results passed between the four warps of cafe_row_fill_quad.
struct CafeQuadScratch {
  double cth[32], sph[32], l[32], d1I[32], dI2[32], d1J[32], dJ3[32], dr[32];
};
#define CAFE_QUAD_THREADS 128
__device__ __forceinline__ void cafe_bar_quad() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Fills row r for position p, the cell just captured (nc), at time T with warps
// 0-3 of the block together (all 128 threads must call it): every liquid
// neighbour slot gets its numerator g and capture result (extent, centre), and
// the record is sorted. A warp issues one FP64 instruction per ~64 cycles
// whatever its active lanes, so the independent chains of each slot's geometry
// run in different warps, lane s of each warp on slot s. First stage:
//   warp 0: cos th and the cell distance l; warp 1: sin ph;
//   warp 2: |R^T dn|_1 and the projection on edge p0-p1;
//   warp 3: the projection on edge p0-p2.
// Second stage, after one barrier: warp 0 forms g and sorts; warp 2 the extent
// and warp 3 the centre a capture from this row gives. The return value (the
// order key of the row's largest |g|) is valid in warp 0.
__device__ __noinline__ unsigned long long cafe_row_fill_quad(const CafeDev &D, const CafeConsts &K, long long r, int p,
                                                              double T, CafeQuadScratch &S, const CafeNewCell &nc,
                                                              const CafeChildList &C) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gp = nc.gid;
  const bool grain_ok = gp >= 1 && gp <= D.grain_cap;
  bool liv = false;
  int q = -1;
  double dn[3] = {0.0, 0.0, 0.0}, cs[3] = {0.0, 0.0, 0.0};
  int ci = 0, cj = 0, ck = 0, si = 0, sj = 0, sk = 0;
  if (lane < CAFE_NSLOT) {
    q = D.a_nbr[(long long)p * CAFE_NSLOT + lane];
    liv = q >= 0 && D.a_state[q] == 1;
  }
  const bool work = liv && grain_ok;
  double R[9], loc[3], dr = 0.0, pk[3][3];
  int s0i = 0;
  if (work) {
    cafe_cell_xyz(K, D.act[q], ci, cj, ck);
    cafe_cell_xyz(K, D.act[p], si, sj, sk);
    cs[0] = nc.c[0];
    cs[1] = nc.c[1];
    cs[2] = nc.c[2];
    cafe_geo_dn(K, ci, cj, ck, cs, dn);
    if (w == 0) {
      S.cth[lane] = cafe_geo_costh(dn);
      S.l[lane] = cafe_geo_l(K, ci, cj, ck, si, sj, sk);
    } else if (w == 1) {
      S.sph[lane] = cafe_geo_sinph(dn);
    } else {
      const double *Rg = D.rot + 9LL * (gp - 1);
      for (int a = 0; a < 9; ++a) R[a] = Rg[a];
      dr = cafe_geo_loc(R, dn, loc);
      s0i = cafe_geo_corners(loc, dr, pk);
      if (w == 2) {
        S.dr[lane] = dr;
        cafe_geo_edge(loc, pk[0], pk[1], &S.d1I[lane], &S.dI2[lane]);
      } else {
        cafe_geo_edge(loc, pk[0], pk[2], &S.d1J[lane], &S.dJ3[lane]);
      }
    }
  }
  cafe_bar_quad();
  unsigned long long ak = 0ULL;
  if (w == 0) {
    double gv = liv ? NAN : 0.0;  // a capturing cell without a grain never captures
    if (work) gv = crm_pow_half(S.cth[lane] * S.sph[lane]) * S.dr[lane];
    ak = cafe_row_sort_warp(D, r, liv, gv, q, nc.ext, cafe_vh(D, K, p), T, gp, C);
  } else if (w >= 2 && work) {
    double Lmud = cafe_geo_lmud(K, S.l[lane], S.d1I[lane], S.dI2[lane], S.d1J[lane], S.dJ3[lane]);
    double *o = D.row_geo + (r * CAFE_NSLOT + lane) * 4;
    if (w == 2) {
      double f = crm_pow_half(S.cth[lane] * S.sph[lane]);
      o[0] = f * Lmud * 1.0;
    } else {
      double cn[3];
      cafe_geo_centre(R, cs, pk[0], s0i, Lmud, cn);
      o[1] = cn[0];
      o[2] = cn[1];
      o[3] = cn[2];
    }
  }
  return ak;
}

// ------------------------------------------------------------------ candidates
// A capture candidate: time t and tie-break ruqs, compared through their
// order keys (equal doubles give equal keys; NaN times are never candidates).
struct CafeCand {
  unsigned long long tk, rk;
  double t;
  int j, s;     // vs2 index and neighbour slot of the capturing cell; j < 0 = none
  int r, q, child;  // (not compared) its row, the captured position and that cell's foreseen row
};
__device__ __forceinline__ CafeCand cafe_cand_none() {
  CafeCand c;
  c.tk = c.rk = CAFE_KEY_NONE;
  c.t = 0.0;
  c.j = -1;
  c.s = 0;
  c.r = c.q = 0;
  c.child = -1;
  return c;
}
__device__ __forceinline__ bool cafe_cand_better(const CafeCand &a, const CafeCand &b) {
  // lexicographic (t, ruqs, scan position): VoxelsCA.C:427-440 keeps the first
  // scanned candidate among full ties
  if (a.j < 0) return false;
  if (b.j < 0) return true;
  if (a.tk != b.tk) return a.tk < b.tk;
  if (a.rk != b.rk) return a.rk < b.rk;
  if (a.j != b.j) return a.j < b.j;
  return a.s < b.s;
}
// Best candidate of the warp, in every lane.
__device__ __forceinline__ CafeCand cafe_warp_best(CafeCand best) {
  for (int o = 16; o > 0; o >>= 1) {
    CafeCand c;
    c.tk = cafe_shfl_u64_xor(best.tk, o);
    c.rk = cafe_shfl_u64_xor(best.rk, o);
    c.t = __shfl_xor_sync(0xffffffffu, best.t, o);
    c.j = __shfl_xor_sync(0xffffffffu, best.j, o);
    c.s = __shfl_xor_sync(0xffffffffu, best.s, o);
    c.r = __shfl_xor_sync(0xffffffffu, best.r, o);
    c.q = __shfl_xor_sync(0xffffffffu, best.q, o);
    c.child = __shfl_xor_sync(0xffffffffu, best.child, o);
    if (cafe_cand_better(c, best)) best = c;
  }
  return best;
}
#define CAFE_KEY_1E6 0xc12e848000000000ULL  // cafe_key(1e6)

// Best candidate of frontier row r (VoxelsCA.C:386-445 restricted to one cell)
// with extent E, velocity v and live slots `live`. For a
// positive finite velocity the capture time is non-decreasing in g, so the
// visit in g order stops at the first time above the row's minimum; otherwise
// every live slot is evaluated. The reference's acceptance limit t <= 1e6
// (VoxelsCA.C:383, 427) applies.
__device__ __noinline__ void cafe_row_best(const CafeDev &D, int r, double E, double v, uint32_t live,
                                           CafeCand &best) {
  const int p = D.row_pos[r];
  const long long vb = crm_bits(v);
  const bool mono = vb > 0 && vb < CRM_BITS_INF;  // 0 < v < inf
  bool have = false;
  unsigned long long tfirst = 0;
  for (; live; live &= live - 1) {
    const CafeSlot s = D.row_slot[(long long)r * CAFE_NSLOT + __ffs(live) - 1];
    double dr = s.g - E;
    double t = dr / v;
    if (cafe_is_nan(t)) continue;
    unsigned long long tk = cafe_key_canon(t);
    if (!(tk <= CAFE_KEY_1E6)) {
      if (mono) break;
      continue;
    }
    if (mono && have && tk > tfirst) break;
    CafeCand c;
    c.t = t;
    c.tk = tk;
    c.rk = cafe_key_canon(.5 * (D.a_ruq[p] + D.a_ruq[s.q]));
    c.j = D.row_j[r];
    c.s = (int)(s.m & 31u);
    c.r = r;
    c.q = s.q;
    c.child = cafe_slot_child(s.m);
    if (cafe_cand_better(c, best)) best = c;
    if (!have) {
      have = true;
      tfirst = tk;
    }
  }
}

// ------------------------------------------------------------------ growth log
// Every event's growth is logged and applied to a row outside the resident set
// only when the row is needed or at the end of the step (k_rows_finalize). The
// log holds fl(v * DtMin) when the step's rows share one velocity (v NaN here),
// else DtMin, which each row multiplies by its own velocity.
#define CAFE_ALIVE 0x7fffffff   // row_death of a row that is still alive
#define CAFE_M_DONE 0x7fffffff  // row_m of a row whose extent is kept current

// One event's growth of an extent (VoxelsCA.C:511-516).
__device__ __forceinline__ double cafe_grow(double E, double vd) {
  E = E + vd;
  return cafe_is_neg(E) ? 0.0 : E;  // (E < 0.0) ? 0.0 : E
}
// Extent of row r after the logged growth of events row_m+1 .. min(upto,
// row_death). A nucleation logs +0, which leaves an extent unchanged (extents
// are never -0).
template <bool PR>
__device__ __forceinline__ double cafe_row_replayed(const CafeDev &D, int r, int upto, double v, int &stop) {
  const int m = D.row_m[r];
  stop = min(upto, D.row_death[r]);
  double E = D.row_E[r];
  if (stop <= m) {
    stop = m;
    return E;
  }
  for (int k = m + 1; k <= stop; ++k) E = cafe_grow(E, PR ? v * D.ev_vd[k] : D.ev_vd[k]);
  return E;
}
__device__ __forceinline__ void cafe_row_replay(const CafeDev &D, const CafeConsts &K, int r, int upto, bool pr) {
  int stop;
  const double E = pr ? cafe_row_replayed<true>(D, r, upto, cafe_vh(D, K, D.row_pos[r]), stop)
                      : cafe_row_replayed<false>(D, r, upto, 0.0, stop);
  D.row_E[r] = E;
  D.row_m[r] = stop;
}

// A velocity whose reciprocal and products stay in the normal range.
__device__ __forceinline__ bool cafe_v_ordinary(double v) { return v > 0x1p-100 && v < 0x1p100; }

// ------------------------------------------------------------------ row kernels
// Frontier rows of the step, in three passes so that the capture geometry,
// the expensive part, runs with one (row, slot) pair per lane:
// k_rows_prep (one warp per row) finds each row's liquid neighbours, sets the
// row's extent and growth watermark, and lists the pairs that need geometry;
// k_rows_geo evaluates the listed pairs; k_rows_order (one warp per row) sorts
// each row's record. CTR_SLOW: bit 0 some row grows with another velocity, bit 1
// some row has a velocity or extent that only the full scan handles.
__device__ __forceinline__ void d_rows_prep(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  int nrows = D.ctr[CTR_NROWS];
  if (nrows > D.row_cap) nrows = (int)D.row_cap;
  const int warps = (cafe_nblk * blockDim.x) >> 5;
  const int w = (cafe_bid * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  for (int r = w; r < nrows; r += warps) {
    int p = D.row_pos[r];
    int gp = D.a_gid[p];
    bool grain_ok = gp >= 1 && gp <= D.grain_cap;
    bool liv = false;
    if (lane < CAFE_NSLOT) {
      const int q = D.a_nbr[(long long)p * CAFE_NSLOT + lane];
      liv = q >= 0 && D.a_state[q] == 1;
    }
    if (liv && !grain_ok) D.row_slot[(long long)r * CAFE_NSLOT + lane].g = NAN;  // never captures
    uint32_t work = __ballot_sync(FULL, liv && grain_ok);
    int base = 0;
    if (lane == 0 && work) base = atomicAdd(&D.ctr[CTR_NPAIRS], __popc(work));
    base = __shfl_sync(FULL, base, 0);
    if (work >> lane & 1u) D.row_pairs[base + __popc(work & ((1u << lane) - 1u))] = r * 32 + lane;
    if (lane == 0) {
      const double E = D.a_ext[p];
      D.row_E[r] = E;
      D.row_m[r] = 0;
      D.row_death[r] = CAFE_ALIVE;
      const double v = cafe_vh(D, K, p);
      const int bad = (cafe_v_ordinary(v) && fabs(E) != INFINITY) ? 0 : 2;
      const int slow = bad | (D.a_cls[p] != 1 ? 1 : 0);
      if (slow) atomicOr(&D.ctr[CTR_SLOW], slow);
    }
  }
}
__global__ void k_rows_prep(CafeDev D, CafeConsts K) {
  d_rows_prep(D, K, blockIdx.x, gridDim.x);
}

__device__ __forceinline__ void d_rows_geo(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  int n = D.ctr[CTR_NPAIRS];
  const long long cap = D.row_cap * CAFE_NSLOT;
  if (n > cap) n = (int)cap;
  for (int i = cafe_bid * blockDim.x + threadIdx.x; i < n; i += cafe_nblk * blockDim.x) {
    int v = D.row_pairs[i];
    int r = v >> 5, sl = v & 31;
    int p = D.row_pos[r];
    int q = D.a_nbr[(long long)p * CAFE_NSLOT + sl];
    const double *Rg = D.rot + 9LL * (D.a_gid[p] - 1);
    double Rm[9];
    for (int a = 0; a < 9; ++a) Rm[a] = Rg[a];
    int i0, j0, k0, si, sj, sk;
    cafe_cell_xyz(K, D.act[q], i0, j0, k0);
    cafe_cell_xyz(K, D.act[p], si, sj, sk);
    double cs[3] = {D.a_cx[p], D.a_cy[p], D.a_cz[p]};
    double g, e, cn[3];
    cafe_capture_geometry(K, i0, j0, k0, si, sj, sk, cs, Rm, &g, &e, cn);
    long long o = (long long)r * CAFE_NSLOT + sl;
    D.row_slot[o].g = g;  // by slot; k_rows_order sorts the record in place
    double *og = D.row_geo + o * 4;
    og[0] = e;
    og[1] = cn[0];
    og[2] = cn[1];
    og[3] = cn[2];
  }
}
__global__ void k_rows_geo(CafeDev D, CafeConsts K) {
  d_rows_geo(D, K, blockIdx.x, gridDim.x);
}

// Also the magnitudes that bound the keys' rounding: the largest |g| and
// extent, the smallest and the largest velocity over the rows (order keys, in row_mag).
__device__ __forceinline__ void d_rows_order(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  int nrows = D.ctr[CTR_NROWS];
  if (nrows > D.row_cap) nrows = (int)D.row_cap;
  const int warps = (cafe_nblk * blockDim.x) >> 5;
  const int w = (cafe_bid * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  unsigned long long gk = 0ULL, ek = 0ULL, vk = CAFE_KEY_NONE, xk = 0ULL;
  const CafeChildList C = {&D.ctr[CTR_NCHILD], 0, D.ch_cap, K.DelT * CAFE_CHILD_REACH};
  for (int r = w; r < nrows; r += warps) {
    int p = D.row_pos[r];
    int q = -1;
    bool liv = false;
    double gv = 0.0;
    if (lane < CAFE_NSLOT) {
      q = D.a_nbr[(long long)p * CAFE_NSLOT + lane];
      liv = q >= 0 && D.a_state[q] == 1;
      if (liv) gv = D.row_slot[(long long)r * CAFE_NSLOT + lane].g;
    }
    __syncwarp();  // the record is read before it is written in order
    const double E = D.row_E[r], v = cafe_vh(D, K, p);
    gk = max(gk, cafe_row_sort_warp(D, r, liv, gv, q, E, v, 0.0, D.a_gid[p], C));
    if (!cafe_is_nan(E)) ek = max(ek, cafe_key(fabs(E)));  // NaN extents occur (the reference's 0/0)
    vk = min(vk, cafe_key(v));
    xk = max(xk, cafe_key(v));
  }
  if (lane == 0 && w < nrows) {
    atomicMax(&D.row_mag[0], gk);
    atomicMax(&D.row_mag[1], ek);
    atomicMin(&D.row_mag[2], vk);
    atomicMax(&D.row_mag[3], xk);
  }
}
__global__ void k_rows_order(CafeDev D, CafeConsts K) {
  d_rows_order(D, K, blockIdx.x, gridDim.x);
}

// The rows of foreseen captures, one per block of four warps: generation `depth`
// lists the next one (in CTR_NCHILD + depth + 1) up to CAFE_CHILD_DEPTH. An
// event's chain of dependent captures within one step is rarely longer; a row
// that is not foreseen is filled by the event loop itself.
#define CAFE_CHILD_BLOCKS_PER_SM 4
__device__ __forceinline__ void d_children(const CafeDev &D, const CafeConsts &K, int depth, const int cafe_bid, const int cafe_nblk) {
  __shared__ CafeQuadScratch Q;
  __shared__ CafeNewCell nc;
  int off = 0, n = 0;
  for (int d = 0; d <= depth; ++d) {
    off += n;
    n = min(D.ctr[CTR_NCHILD + d], D.ch_cap - off);
  }
  const int last = off + n;
  const CafeChildList C = {&D.ctr[CTR_NCHILD + min(depth + 1, CAFE_CHILD_DEPTH - 1)], last,
                           depth + 1 < CAFE_CHILD_DEPTH ? D.ch_cap : last, K.DelT * CAFE_CHILD_REACH};
  for (int i = off + cafe_bid; i < last; i += cafe_nblk) {
    const long long id = D.row_cap + i;
    const int p = D.row_pos[id];
    if (threadIdx.x < 4) {
      const double x = D.row_geo[(long long)D.ch_src[i] * 4 + threadIdx.x];
      if (threadIdx.x == 0) nc.ext = x; else nc.c[threadIdx.x - 1] = x;
    } else if (threadIdx.x == 4) {
      nc.gid = D.ch_gid[i];
    }
    __syncthreads();
    const unsigned long long gk = cafe_row_fill_quad(D, K, id, p, D.ch_T[i], Q, nc, C);
    if (threadIdx.x == 0) {
      D.row_key[id] = CAFE_KEY_NONE;  // until the row exists
      atomicMax(&D.row_mag[0], gk);
      if (!cafe_is_nan(nc.ext)) atomicMax(&D.row_mag[1], cafe_key(fabs(nc.ext)));
      const double v = cafe_vh(D, K, p);
      if (cafe_v_ordinary(v)) {
        atomicMin(&D.row_mag[2], cafe_key(v));
        atomicMax(&D.row_mag[3], cafe_key(v));
      }
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(CAFE_QUAD_THREADS) k_children(const __grid_constant__ CafeDev D, const __grid_constant__ CafeConsts K, int depth) {
  d_children(D, K, depth, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------ event loop
// The capture/nucleation loop of one step (VoxelsCA.C:381-610), one block.
//
// Every event is a global argmin over the frontier, the growth of every
// frontier cell and the capture, one after another. Only a few hundred of the
// ~10 thousand rows can capture within a step, so the loop works on a resident
// set: the rows whose key (lower bound of the absolute capture time T + t when
// last evaluated) lies at or below a window bound W, and the rows created by
// captures (made ahead by k_children when the capture was foreseen, filled in
// the loop otherwise). A resident row has its extent in a register of the thread that owns
// its index and its first live slot in shared memory. Per event:
//   select   every resident's g - E, the minimum over the block by integer order
//            keys (two redux per warp and level), and a test that no other
//            candidate lies within the rounding of the division by v. A tie (or
//            a near one) is resolved by evaluating the close rows exactly in the
//            reference's order (time, ruqs, vs2 index, slot);
//   apply    one warp updates the captured cell and its neighbours' rows while
//            one thread divides out the capture time and advances the clock and
//            another draws the next event's uniform;
//   grow     every resident's extent by the logged growth, in the reference's
//            order of additions (the rows outside the set replay the log when
//            they enter it or at the step's end).
// Exactness: a row outside the set has key K > W, and its exact time is at least
// K - T - delta, delta = (ev+16) 2^-47 (|W| + |T| + 2 sum|dt| + (gmax+emax)/v)
// for the roundings of ev growth additions. A winner at T + t below W - delta is
// the global one; otherwise the set is written back and opened again with a later
// window. Rows with another velocity than the step's class-1 velocity switch the
// step to per-row velocities (PR); a velocity that is not positive and finite,
// or a window that does not fit, to the full scan of every row per event.
#define CAFE_RES_PER 2  // resident rows per thread
#define CAFE_RES_MAX (CAFE_RES_PER * CAFE_LOOP_THREADS)
#define CAFE_RES_TARGET 320  // rows an opened window aims at: one per thread with room for the step's new rows
#define CAFE_OPEN_TRIES 48   // windows in a row without an event before the step takes the full scan
#define CAFE_CAP_WARP (CAFE_LOOP_THREADS / 32 - 1)     // captures
#define CAFE_CLOCK_WARP (CAFE_LOOP_THREADS / 32 - 2)   // capture time and clock
#define CAFE_DRAW_WARP (CAFE_LOOP_THREADS / 32 - 3)    // nucleation draws
static_assert(CAFE_CAP_WARP >= 6, "warps 0-3 fill rows");
// Row of the k-th frontier row of the step: the rows present at its start, then
// the rows that captures created, in their order (row_new).
__device__ __forceinline__ int cafe_row_at(const CafeDev &D, int nrows0, int k) {
  return k < nrows0 ? k : D.row_new[k - nrows0];
}

struct CafeLoop {
  // the loop's scalars (VoxelsCA.C:381-610)
  double tinc, dt, vd, vs, vneg, vmin, vmax, dsum, gmax, emax;
  double unext[2];  // unext[e & 1]: event e's draw
  int fill, nvs2, countS, nrows0, nrows, ngrain, done, nuc, ev, sw, na, newrow, slow;
  uint32_t rng;
  unsigned int sdloc;
  long long nnuc, negdt, opens, cyc[4];
  CafeNewCell nc;
};
struct CafeResident {
  double g[CAFE_RES_MAX];      // numerator of the first live slot, NaN when none
  double v[CAFE_RES_MAX];      // growth velocity (PR)
  int r[CAFE_RES_MAX];         // row, -1 when free
  int q[CAFE_RES_MAX];         // the first live slot's neighbour position
  uint32_t m[CAFE_RES_MAX];    // ... and its slot
  uint32_t live[CAFE_RES_MAX];  // live slots in g order
  unsigned char flag[CAFE_RES_MAX];  // CAFE_RF_*
  unsigned short free[CAFE_RES_MAX];
  unsigned long long wk[CAFE_LOOP_THREADS / 32], thr[32];
  double wd[CAFE_LOOP_THREADS / 32];
  int wi[CAFE_LOOP_THREADS / 32], hist[32];
  int top, nfree, newslot, overflow;
  double newE;              // extent of the row that enters at newslot
  unsigned long long klim;  // a smallest key below it needs no further test
  unsigned long long kw;    // rows with keys at or below it are resident
  double wlim, dsum_cap;    // latest safe T + t; the window holds while dsum <= dsum_cap and ev <= ev_cap
  int ev_cap, all;          // all: every row with a candidate is resident
  CafeCand red[CAFE_LOOP_THREADS / 32];
};
#define CAFE_RF_NEAR 1   // the next live slot's g is within a relative 2^-19
#define CAFE_RF_DYING 2  // no live slot is left: the row grew at this event for the last time

// (smallest key, its lane's index) of a warp, in every lane: two redux steps
// on the 32-bit halves.
__device__ __forceinline__ unsigned long long cafe_warp_min_key(unsigned long long k, int &src) {
  const uint32_t hi = (uint32_t)(k >> 32), lo = (uint32_t)k;
  const uint32_t mh = __reduce_min_sync(0xffffffffu, hi);
  const uint32_t ml = __reduce_min_sync(0xffffffffu, hi == mh ? lo : 0xffffffffu);
  src = __ffs(__ballot_sync(0xffffffffu, hi == mh && lo == ml)) - 1;
  return ((unsigned long long)mh << 32) | ml;
}

// The first live slot of a row's record and whether the next one is close.
__device__ __forceinline__ void cafe_res_first(const CafeDev &D, CafeResident &S, int i, int r, uint32_t live) {
  const CafeSlot *rec = D.row_slot + (long long)r * CAFE_NSLOT;
  if (!live) {
    S.g[i] = NAN;
    S.flag[i] = 0;
    return;
  }
  const uint32_t rest = live & (live - 1);
  const CafeSlot a = rec[__ffs(live) - 1];
  const double g2 = rest ? rec[__ffs(rest) - 1].g : NAN;
  S.g[i] = a.g;
  S.q[i] = a.q;
  S.m[i] = a.m;
  const unsigned long long k1 = cafe_key_canon(a.g), k2 = cafe_key_canon(g2);
  S.flag[i] = (rest && !cafe_is_nan(g2) && k2 - k1 < (1ULL << 33)) ? CAFE_RF_NEAR : 0;
}

// Keyed loop over the resident set; every thread of the block calls it. Leaves
// with L.done set, or with L.sw set when the step must continue with the full
// scan (every row's extent and live mask are then in the row arrays).
template <bool PR>
__device__ __forceinline__ void cafe_events_resident(const CafeDev &D, const CafeConsts &K, long long max_events,
                                                     CafeLoop &L, CafeResident &S, CafeQuadScratch &Q) {
  const unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = CAFE_LOOP_THREADS, NW = CAFE_LOOP_THREADS / 32;
  const double V = K.vhat_cls[1];
  // key distance within which two approximate values may belong to equal times:
  // a few ulps of g - E; with PR the value is (g - E) times a reciprocal good
  // to about 2^-44
  const unsigned long long TOL = PR ? (1ULL << 14) : 8ULL;
  const unsigned long long KTINY = cafe_key(0x1p-900);
  double E[CAFE_RES_PER], rv[CAFE_RES_PER];
#pragma unroll
  for (int c = 0; c < CAFE_RES_PER; ++c) E[c] = rv[c] = 0.0;
  int ev = 0;
  int tries = 0;  // windows opened since the last event
  bool need_open = true;
  if (tid == 0) S.top = 0;
  __syncthreads();
  long long t0 = clock64();
  // every resident's extent, live mask and key back to the row arrays
  auto flush = [&](bool keys) {
#pragma unroll
    for (int c = 0; c < CAFE_RES_PER; ++c) {
      const int i = tid + c * NT;
      if (i >= S.top || S.r[i] < 0) continue;
      const int r = S.r[i];
      D.row_E[r] = E[c];
      D.row_m[r] = ev;
      D.row_live[r] = S.live[i];
      D.row_res[r] = -1;
      if (keys) {
        const double t = (S.g[i] - E[c]) / (PR ? S.v[i] : V);
        D.row_key[r] = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(L.tinc + t);
      }
    }
  };
  auto load_resident = [&](int c, int i) {
    const int r = S.r[i];
    const uint32_t live = D.row_live[r];
    double v = 0.0;
    if (PR) {
      v = cafe_vh(D, K, D.row_pos[r]);
      S.v[i] = v;
      rv[c] = 1.0 / v;
    }
    int stop;
    E[c] = cafe_row_replayed<PR>(D, r, ev, v, stop);
    S.live[i] = live;
    cafe_res_first(D, S, i, r, live);
    D.row_res[r] = i;
  };
  while (true) {
    if (need_open) {
      // ---- open the window: the earliest rows by key
      need_open = false;
      ++tries;
      flush(true);
      __syncthreads();
      const int nrows = L.nrows, nrows0 = L.nrows0;
      unsigned long long mn = CAFE_KEY_NONE;
      int cnt = 0;
      for (int r0 = tid; r0 < nrows; r0 += 8 * NT) {
        unsigned long long kk[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) kk[u] = r0 + u * NT < nrows ? D.row_key[cafe_row_at(D, nrows0, r0 + u * NT)] : CAFE_KEY_NONE;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          mn = min(mn, kk[u]);
          cnt += kk[u] != CAFE_KEY_NONE;
        }
      }
      int src;
      mn = cafe_warp_min_key(mn, src);
      cnt = __reduce_add_sync(FULL, cnt);
      if (lane == 0) {
        S.wk[warp] = mn;
        S.wi[warp] = cnt;
      }
      if (tid < 32) S.hist[tid] = 0;
      __syncthreads();
      mn = cafe_warp_min_key(lane < NW ? S.wk[lane] : CAFE_KEY_NONE, src);
      cnt = __reduce_add_sync(FULL, lane < NW ? S.wi[lane] : 0);
      const bool all = cnt <= CAFE_RES_TARGET;
      // rounding bound of the keys for the next 4096 events and 64 DelT of growth
      const double dcap = L.dsum + 64.0 * K.DelT;
      const double base = (mn == CAFE_KEY_NONE ? 0.0 : cafe_unkey(mn));
      const double slack = (double)(ev + 4096 + 16) * 0x1p-47 *
                           (fabs(base) + 64.0 * K.DelT + fabs(L.tinc) + 2.0 * dcap +
                            (L.gmax + L.emax) / (PR ? L.vmin : V) + 1e-300);
      int pick = 31;
      if (!all) {
        if (tid < 32) {
          // thresholds in steps of a factor sqrt(2), DelT/1024 .. 45 DelT beyond the smallest key
          const double f = (tid & 1) ? 1.4142135623730951 : 1.0;
          const double wj = base + 4.0 * slack + K.DelT * (f * crm_from_bits((long long)(1023 - 10 + (tid >> 1)) << 52));
          S.thr[tid] = cafe_is_nan(wj) ? CAFE_KEY_NONE - 1 : cafe_key(wj);
        }
        __syncthreads();
        const unsigned long long last = S.thr[31];
        for (int r = tid; r < nrows; r += NT) {
          const unsigned long long k = D.row_key[cafe_row_at(D, nrows0, r)];
          if (k > last) continue;
          int lo = 0, hi = 31;  // first threshold at or above the key
          while (lo < hi) {
            const int md = (lo + hi) >> 1;
            if (k <= S.thr[md]) hi = md; else lo = md + 1;
          }
          atomicAdd(&S.hist[lo], 1);
        }
        __syncthreads();
        int h = S.hist[lane];
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(FULL, h, o);
          if (lane >= o) h += u;
        }
        const uint32_t fits = __ballot_sync(FULL, h <= CAFE_RES_TARGET);
        // the counts ascend: the last threshold that fits the target, else the first if it fits at all
        pick = fits ? 31 - __clz(fits) : 0;
        const int n0 = __shfl_sync(FULL, h, 0);
        if (tid == 0) S.overflow = !fits && n0 > CAFE_RES_MAX - 64;
      }
      const unsigned long long kw = all ? CAFE_KEY_NONE - 1 : S.thr[pick];
      if (tid == 0) {
        if (all) S.overflow = 0;
        if (!(slack < 1e300) || tries >= CAFE_OPEN_TRIES) S.overflow = 1;
        S.kw = kw;
        S.all = all;
        S.top = 0;
        S.nfree = 0;
        S.ev_cap = ev + 4096;
        S.dsum_cap = dcap;
        S.wlim = all ? INFINITY : cafe_unkey(kw) - slack;
        L.opens++;
        // the bound of the next winner's key
        const double v = PR ? 1.0 : V;
        const double lim = fmin(S.wlim - L.tinc, 0x1.e847fp19) * v;  // 0x1.e847fp19 < 1e6
        S.klim = cafe_key(lim - fabs(lim) * 0x1p-30);
      }
      __syncthreads();
      if (S.overflow) {
        if (tid == 0) L.sw = 1;
        __syncthreads();
        break;
      }
      for (int k = tid; k < nrows; k += NT) {
        const int r = cafe_row_at(D, nrows0, k);
        if (D.row_key[r] <= kw) {
          const int i = atomicAdd(&S.top, 1);
          if (i < CAFE_RES_MAX) S.r[i] = r;
        }
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < CAFE_RES_PER; ++c) {
        const int i = tid + c * NT;
        if (i < S.top) load_resident(c, i);
      }
      __syncthreads();
      if (tid == 0) {
        const long long t1 = clock64();
        L.cyc[3] += t1 - t0;
        t0 = t1;
      }
    }
    // ---- select: the smallest (g - E) / v over the resident rows
    unsigned long long kk[CAFE_RES_PER], bk = CAFE_KEY_NONE;
    double bd = 0.0;
    int bi = -1;
    const int top = S.top;
#pragma unroll
    for (int c = 0; c < CAFE_RES_PER; ++c) {
      const int i = tid + c * NT;
      kk[c] = CAFE_KEY_NONE;
      if (i < top && S.r[i] >= 0) {
        const double d = S.g[i] - E[c];
        const double x = PR ? d * rv[c] : d;
        if (!cafe_is_nan(x)) kk[c] = cafe_key_canon(x);
        if (kk[c] < bk) {
          bk = kk[c];
          bd = d;
          bi = i;
        }
      }
    }
    int src;
    {
      const unsigned long long wm = cafe_warp_min_key(bk, src);
      if (lane == src) {
        S.wk[warp] = wm;
        S.wi[warp] = bi;
        S.wd[warp] = bd;
      }
    }
    __syncthreads();
    const unsigned long long kmin = cafe_warp_min_key(lane < NW ? S.wk[lane] : CAFE_KEY_NONE, src);
    const int win = S.wi[src];
    const double wd = S.wd[src];
    // (read before the next barrier: the captures change them after it)
    int wr = -1, wq = 0, ws = 0, child = -1;
    if (kmin != CAFE_KEY_NONE) {
      wr = S.r[win];
      wq = S.q[win];
      ws = (int)(S.m[win] & 31u);
      child = cafe_slot_child(S.m[win]);
    }
    // another candidate within the rounding of the division?
    bool tie = false;
    if (kmin != CAFE_KEY_NONE) {
      unsigned long long thr = kmin + TOL;
      const int ex = (int)((crm_bits(cafe_unkey(kmin)) >> 52) & 0x7ff);
      if (ex < 1023 - 900) thr = KTINY;  // zero or tiny: times may round together
      bool close = false;
#pragma unroll
      for (int c = 0; c < CAFE_RES_PER; ++c) {
        const int i = tid + c * NT;
        if (kk[c] <= thr) {
          if (i != win) {
            close = true;
          } else {
            // its own next slot: g apart by 2^-19 relative cannot round together
            // unless the extent dwarfs g
            const int ed = (int)((crm_bits(wd) >> 52) & 0x7ff), eg = (int)((crm_bits(S.g[i]) >> 52) & 0x7ff);
            close = close || (S.flag[i] & CAFE_RF_NEAR) || ed > eg + 20 || thr == KTINY;
          }
        }
      }
      tie = __syncthreads_or(close);
    }
    const bool plain = kmin != CAFE_KEY_NONE && !tie && kmin < S.klim;
    CafeCand wc = cafe_cand_none();
    if (!plain) {
      if (!S.all && !(kmin < S.klim)) {  // beyond the window (or nothing in it)
        __syncthreads();
        need_open = true;
        continue;
      }
      // exact candidates of the close rows, the reference's order among them
      if (kmin != CAFE_KEY_NONE) {
        const int ex = (int)((crm_bits(cafe_unkey(kmin)) >> 52) & 0x7ff);
        const unsigned long long thr = ex < 1023 - 900 ? KTINY : kmin + TOL;
#pragma unroll
        for (int c = 0; c < CAFE_RES_PER; ++c) {
          const int i = tid + c * NT;
          if (kk[c] <= thr) cafe_row_best(D, S.r[i], E[c], PR ? S.v[i] : V, S.live[i], wc);
        }
        wc = cafe_warp_best(wc);
        if (lane == 0) S.red[warp] = wc;
        __syncthreads();
        wc = cafe_warp_best(lane < NW ? S.red[lane] : cafe_cand_none());
        __syncthreads();
      }
      if (wc.j < 0 || !(wc.tk < CAFE_KEY_1E6)) {  // no candidate is left
        if (tid == 0) L.done = 1;
        __syncthreads();
        break;
      }
      wr = wc.r;
      wq = wc.q;
      ws = wc.s;
      child = wc.child;
    }
    if (ev >= max_events) {
      if (tid == 0) {
        atomicOr(D.err, CAFE_ERR_ITER_CAP);
        L.done = 1;
      }
      __syncthreads();
      break;
    }
    ++ev;
    tries = 0;
    if (tid == 0) {
      const long long t1 = clock64();
      L.cyc[0] += t1 - t0;
      t0 = t1;
    }
    // ---- apply the event
    const int icap = wq;
    if (warp == CAFE_CAP_WARP) {
      const int p = D.row_pos[wr];
      const bool cold = D.a_cold[icap] != 0;
      const int cls = D.a_cls[icap];
      const bool nuc = L.unext[ev & 1] < cafe_nuc_rate_at(D, K, icap);
      // level 1: the neighbours; the capture result of this slot (lanes 26-29:
      // extent and centre, computed when the row was filled) and the grain
      int q = -1, gcap = 0;
      double gx = 0.0;
      if (lane < CAFE_NSLOT) q = D.a_nbr[(long long)icap * CAFE_NSLOT + lane];
      else if (lane < 30) gx = D.row_geo[((long long)wr * CAFE_NSLOT + ws) * 4 + lane - 26];
      else if (lane == 30) gcap = D.a_gid[p];
      // ... and the foreseen row's record
      CafeSlot cr;
      cr.g = NAN;
      cr.q = -1;
      cr.m = 0;
      int crk = 0;
      const bool foreseen = child >= 0 && !nuc;
      if (foreseen && lane < CAFE_NSLOT) {
        cr = D.row_slot[(long long)child * CAFE_NSLOT + lane];
        crk = D.row_rank[(long long)child * 32 + lane];
      }
      // level 2
      int st = 0, fr = -1;
      if (q >= 0) {
        st = D.a_state[q];
        fr = D.a_frow[q];
      }
      const uint32_t clive = __reduce_or_sync(FULL, st == 1 ? 1u << crk : 0u);
      const bool grows = clive != 0u && cold;
      // a foreseen row enters the resident set at once (its neighbours that were
      // captured meanwhile are no longer live)
      int ci = -1;
      if (foreseen && grows) {
        if (lane == 0) {
          if (S.nfree > 0) ci = S.free[--S.nfree];
          else if (S.top < CAFE_RES_MAX) ci = S.top++;
        }
        ci = __shfl_sync(FULL, ci, 0);
        const uint32_t rest = clive & (clive - 1u);
        const int k1 = __ffs(clive) - 1, k2 = rest ? __ffs(rest) - 1 : 31;
        const double g2 = __shfl_sync(FULL, cr.g, k2);  // (lane 31: NaN)
        if (ci >= 0) {
          if (lane == k1) {
            S.g[ci] = cr.g;
            S.q[ci] = cr.q;
            S.m[ci] = cr.m;
            S.live[ci] = clive;
            S.flag[ci] = (!cafe_is_nan(g2) && cafe_key_canon(g2) - cafe_key_canon(cr.g) < (1ULL << 33)) ? CAFE_RF_NEAR : 0;
            S.r[ci] = child;
            if (PR) S.v[ci] = cafe_vh(D, K, icap);
          }
          if (lane == 26) S.newE = gx;
        } else if (lane == 0) {
          D.row_live[child] = clive;
        }
      }
      if (lane == 0) S.newslot = ci;
      // level 3: the neighbours' rows
      if (fr >= 0) {
        const int rs = D.row_res[fr];
        const uint32_t lg = D.row_live[fr];
        const int rk = D.row_rank[(long long)fr * 32 + (CAFE_NSLOT - 1 - lane)];
        const uint32_t live = rs >= 0 ? S.live[rs] : lg;
        const uint32_t bit = 1u << rk;
        if (live & bit) {
          const uint32_t nl = live & ~bit;
          if (rs >= 0) {
            S.live[rs] = nl;
            if (!nl) {
              S.g[rs] = NAN;
              S.flag[rs] = CAFE_RF_DYING;
              D.row_death[fr] = ev;  // it grew at this event too
            } else if ((live & (bit - 1u)) == 0u) {
              cafe_res_first(D, S, rs, fr, nl);
            }
          } else {
            D.row_live[fr] = nl;
            if (!nl) {
              D.row_death[fr] = ev;
              D.row_key[fr] = CAFE_KEY_NONE;
            }
          }
        }
      }
      // the captured cell (VoxelsCA.C:483-505 and 518-605)
      if (nuc) {
        if (lane == 0) {
          int ci, cj, ck;
          cafe_cell_xyz(K, D.act[icap], ci, cj, ck);
          if (L.ngrain < D.grain_cap) {
            double q4[4];
            cafe_sample_orientation(K, L.sdloc, q4);
            double *cc = D.cth + 4LL * L.ngrain;
            for (int a = 0; a < 4; ++a) cc[a] = q4[a];
            cafe_rot_from_cth(cc, D.rot + 9LL * L.ngrain);
          } else {
            atomicOr(D.err, CAFE_ERR_GRAIN_CAP);
            L.done = 1;
          }
          L.ngrain += 1;
          D.a_gid[icap] = L.nc.gid = L.ngrain;
          D.a_cx[icap] = L.nc.c[0] = ((double)ci + .5) * K.dx[0];
          D.a_cy[icap] = L.nc.c[1] = ((double)cj + .5) * K.dx[1];
          D.a_cz[icap] = L.nc.c[2] = ((double)ck + .5) * K.dx[2];
          L.sdloc += 10u;
          D.a_ext[icap] = L.nc.ext = 0.0;
          L.nnuc++;
        }
      } else if (lane == 26) {
        D.a_ext[icap] = L.nc.ext = gx;
        if (fabs(gx) == INFINITY) L.sw = 1;  // its times need the full scan
      } else if (lane == 27) {
        D.a_cx[icap] = L.nc.c[0] = gx;
      } else if (lane == 28) {
        D.a_cy[icap] = L.nc.c[1] = gx;
      } else if (lane == 29) {
        D.a_cz[icap] = L.nc.c[2] = gx;
      } else if (lane == 30) {
        D.a_gid[icap] = L.nc.gid = gcap;
      }
      if (lane == 31) {
        D.a_state[icap] = 2;
        if (L.nvs2 < D.vs2_cap) {
          D.vs2[L.nvs2] = icap;
        } else {
          atomicOr(D.err, CAFE_ERR_MUSHY_CAP);
          L.done = 1;
        }
        L.countS = L.nvs2;
        L.nvs2 += 1;
        L.newrow = -1;
        if (grows) {
          const int k = L.nrows;
          if (k < D.row_cap) {
            const int r = foreseen ? child : k;
            D.row_pos[r] = icap;
            D.row_j[r] = L.nvs2 - 1;
            D.row_res[r] = ci;
            D.a_frow[icap] = r;
            D.row_death[r] = CAFE_ALIVE;
            D.row_m[r] = ev;
            D.row_new[k - L.nrows0] = r;
            L.nrows = k + 1;
            L.newrow = r;
            L.fill = !foreseen;
            // a cell of another growth velocity
            if (PR) {
              const double v = cafe_vh(D, K, icap);
              if (!cafe_v_ordinary(v)) L.sw = 1;
              L.vmin = fmin(L.vmin, v);
              L.vmax = fmax(L.vmax, v);
            } else if (cls != 1) {
              L.sw = 1;
            }
          } else {
            atomicOr(D.err, CAFE_ERR_ROW_CAP);
            L.done = 1;
          }
        }
      }
    } else if (tid == CAFE_CLOCK_WARP * 32) {
      // the capture time, the clock (VoxelsCA.C:381, 483-516) and the growth log
      const bool nuc = L.unext[ev & 1] < cafe_nuc_rate_at(D, K, icap);
      const double t = plain ? wd / (PR ? S.v[win] : V) : wc.t;
      const double dt = nuc ? 0.0 : t;
      L.dt = dt;
      const double vd = PR ? dt : (nuc ? 0.0 : V * dt);
      L.vd = vd;
      D.ev_vd[ev] = vd;
      L.tinc += dt;
      L.dsum += fabs(dt);
      L.vs += vd;
      D.ev_vs[ev] = L.vs;
      if (cafe_is_neg(dt)) {
        L.negdt++;
        L.vneg += fabs(vd);
      }
      L.nuc = nuc;
    } else if (tid == CAFE_DRAW_WARP * 32) {
      // the next event's draw (VoxelsCA.C:483; two engine outputs per event)
      cafe_uniform_stream st;
      st.x = L.rng;
      L.unext[(ev + 1) & 1] = cafe_uniform_next(&st);
      L.rng = st.x;
    }
    __syncthreads();
    // ---- grow (VoxelsCA.C:511-516); a row that lost its last slot leaves
    {
      const double vd = L.vd;
      const int top2 = S.top, born = S.newslot;
#pragma unroll
      for (int c = 0; c < CAFE_RES_PER; ++c) {
        const int i = tid + c * NT;
        if (i == born) {  // created by this event: grows from the next one on
          E[c] = S.newE;
          if (PR) {
            const double v = S.v[i], y = (double)(1.0f / (float)v);
            rv[c] = y * (2.0 - v * y);
          }
        } else if (i < top2 && S.r[i] >= 0) {
          E[c] = cafe_grow(E[c], PR ? S.v[i] * vd : vd);
          if (S.flag[i] & CAFE_RF_DYING) {
            const int r = S.r[i];
            D.row_E[r] = E[c];
            D.row_m[r] = ev;
            D.row_live[r] = 0u;
            D.row_key[r] = CAFE_KEY_NONE;
            D.row_res[r] = -1;
            S.flag[i] = 0;
            S.r[i] = -1;
            S.free[atomicAdd(&S.nfree, 1)] = (unsigned short)i;
          }
        }
      }
    }
    if (tid == CAFE_CLOCK_WARP * 32) {
      // while (vSind2 != countS && tinc < DelT)
      const bool tin = !cafe_is_nan(L.tinc) && cafe_key(L.tinc) < cafe_key(K.DelT);
      if (!(L.nvs2 != L.countS && tin)) L.done = 1;
      const double lim = fmin(S.wlim - L.tinc, 0x1.e847fp19) * (PR ? 1.0 : V);
      S.klim = (ev < S.ev_cap && L.dsum <= S.dsum_cap) || S.all ? cafe_key(lim - fabs(lim) * 0x1p-30) : 0ULL;
    }
    __syncthreads();
    if (tid == 0) {
      const long long t1 = clock64();
      L.cyc[1] += t1 - t0;
      t0 = t1;
    }
    // ---- a negative event may clamp a small extent at zero (VoxelsCA.C:515),
    // which breaks the key bound of a row outside the set: the rows whose
    // extrapolated extent comes near zero are brought up to date with a new key
    if (cafe_is_neg(L.vd)) {
      const double vd = L.vd, vsp = D.ev_vs[ev - 1], vx = PR ? L.vmax : V;
      const double margin = (double)(ev + 16) * 0x1p-48 * (L.emax + L.gmax + vx * L.dsum + 1e-300);
      // an extent above all the negative growth so far cannot have come near zero
      const long long safe = crm_bits((PR ? L.vneg * vx : L.vneg) * (1.0 + 0x1p-20) + 2.0 * margin);
      bool again = false;
      const int nrows = L.nrows, nrows0 = L.nrows0;
      for (int k = tid; k < nrows; k += NT) {
        const int r = cafe_row_at(D, nrows0, k);
        if (crm_bits(D.row_E[r]) >= safe) continue;  // (NaN too: it never captures)
        if (D.row_res[r] >= 0 || D.row_death[r] < ev) continue;
        const int m = D.row_m[r];
        if (m >= ev) continue;
        const double v = PR ? cafe_vh(D, K, D.row_pos[r]) : V;
        const double gr = (vsp - D.ev_vs[m]) + vd;
        if (D.row_E[r] + (PR ? v * gr : gr) >= margin) continue;
        int stop;
        const double En = cafe_row_replayed<PR>(D, r, ev, v, stop);
        D.row_E[r] = En;
        D.row_m[r] = stop;
        const uint32_t live = D.row_live[r];
        if (live) {
          const double t = (D.row_slot[(long long)r * CAFE_NSLOT + __ffs(live) - 1].g - En) / v;
          const unsigned long long key = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(L.tinc + t);
          D.row_key[r] = key;
          again = again || key <= S.kw;
        }
      }
      if (__syncthreads_or(again)) need_open = true;
    }
    // ---- the captured cell's own row
    const int nr = L.newrow;
    if (nr >= 0 && !L.fill) {
      if (S.newslot < 0) {  // no room: write the set back and open a new window
        if (tid == 0) {
          D.row_E[nr] = L.nc.ext;
          const double t = (D.row_slot[(long long)nr * CAFE_NSLOT + __ffs(D.row_live[nr]) - 1].g - L.nc.ext) /
                           (PR ? cafe_vh(D, K, icap) : V);
          D.row_key[nr] = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(L.tinc + t);
        }
        need_open = true;
        __syncthreads();
      }
    } else if (nr >= 0) {
      if (warp < CAFE_QUAD_THREADS / 32) {
        const CafeChildList none = {nullptr, 0, 0, 0.0};
        const unsigned long long gk = cafe_row_fill_quad(D, K, nr, icap, L.tinc, Q, L.nc, none);
        if (tid == 0) {
          D.row_E[nr] = L.nc.ext;
          if (gk != 0ULL) L.gmax = fmax(L.gmax, cafe_unkey(gk));
          if (!cafe_is_nan(L.nc.ext)) L.emax = fmax(L.emax, fabs(L.nc.ext));
          int i = -1;
          if (S.nfree > 0) i = S.free[--S.nfree];
          else if (S.top < CAFE_RES_MAX) i = S.top++;
          S.newslot = i;
          if (i >= 0) S.r[i] = nr;
        }
      }
      __syncthreads();
      const int i = S.newslot;
      if (i < 0) {
        need_open = true;  // no room: write the set back and open a new window
      } else if (i % NT == tid) {
#pragma unroll
        for (int c = 0; c < CAFE_RES_PER; ++c)
          if (i == tid + c * NT) load_resident(c, i);
      }
      __syncthreads();
      if (tid == 0) {
        const long long t1 = clock64();
        L.cyc[2] += t1 - t0;
        t0 = t1;
      }
    }
    if (L.done || L.sw) break;
  }
  flush(false);
  if (tid == 0) {
    L.ev = ev;
    D.ctr[CTR_EVLOG] = PR ? 1 : 0;
  }
  __syncthreads();
}

__device__ __forceinline__ void d_event_loop(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, long long max_events, int allow_fast, const int cafe_bid, const int cafe_nblk) {
  __shared__ CafeLoop L;
  __shared__ CafeResident S;
  __shared__ CafeQuadScratch Q;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = CAFE_LOOP_THREADS, NW = CAFE_LOOP_THREADS / 32;
  if (cafe_bid != 0) return;  // event_fill_helper's second block: the loop leaves it nothing to do
  if (tid == 0) {
    L.na = D.ctr[CTR_NA];
    L.nvs2 = D.ctr[CTR_NVS2];
    L.nrows = L.nrows0 = D.ctr[CTR_NROWS];
    L.ngrain = D.ctr[CTR_NGRAIN];
    const int tInd = Pp->tInd;
    uint32_t seed = cafe_minstd_seed((uint64_t)(uint32_t)(30 * tInd + (int)K.seed1));
    cafe_uniform_stream st;
    st.x = cafe_minstd_skip(seed, 2ULL * (uint64_t)L.na);
    L.unext[1] = cafe_uniform_next(&st);  // the first event's draw; later draws are made one event ahead
    L.rng = st.x;
    L.sdloc = K.seed0 + 32u * (unsigned int)tInd + 64u * (unsigned int)L.ngrain;
    L.tinc = L.dsum = L.vd = L.dt = L.vs = L.vneg = 0.0;
    L.gmax = D.row_mag[0] ? cafe_unkey(D.row_mag[0]) : 0.0;
    L.emax = D.row_mag[1] ? cafe_unkey(D.row_mag[1]) : 0.0;
    L.vmin = D.row_mag[2] != CAFE_KEY_NONE ? cafe_unkey(D.row_mag[2]) : 1.0;
    L.vmax = D.row_mag[3] ? cafe_unkey(D.row_mag[3]) : 1.0;
    L.countS = L.na;
    L.nnuc = L.negdt = L.opens = 0;
    L.ev = L.sw = 0;
    L.newrow = -1;
    L.cyc[0] = L.cyc[1] = L.cyc[2] = L.cyc[3] = 0;
    D.ev_vd[0] = D.ev_vs[0] = 0.0;
    D.ctr[CTR_EVLOG] = 0;
    const int slow = D.ctr[CTR_SLOW];
    // 0: rows share one velocity; 1: per-row velocities; 2: full scan
    L.slow = (!allow_fast || (slow & 2)) ? 2 : (slow & 1);
    L.done = (*D.err != 0) || (L.na > D.act_cap) || (L.nvs2 > D.vs2_cap) || (L.nrows > D.row_cap);
    if (L.na + 2 > D.ev_cap) {
      atomicOr(D.err, CAFE_ERR_ITER_CAP);
      L.done = 1;
    }
    // while (vSind2 != countS && tinc < DelT)
    if (!(L.nvs2 != L.countS && L.tinc < K.DelT)) L.done = 1;
  }
  __syncthreads();
  const int mode = L.slow;
  if (!L.done) {
    if (mode == 0)
      cafe_events_resident<false>(D, K, max_events, L, S, Q);
    else if (mode == 1)
      cafe_events_resident<true>(D, K, max_events, L, S, Q);
  }
  const bool scan = mode == 2 || L.sw;
  if (scan && !L.done) {
    // extents are kept current from here on
    const int e0 = L.ev;
    for (int k = tid; k < L.nrows; k += NT) {
      const int r = cafe_row_at(D, L.nrows0, k);
      if (e0) cafe_row_replay(D, K, r, e0, mode == 1);
      D.row_m[r] = CAFE_M_DONE;
    }
    __syncthreads();
  }
  // ======================================================== full scan
  bool first = true;
  while (scan && !L.done) {
    if (tid == 0 && !first) {
      // while (vSind2 != countS && tinc < DelT)
      if (!(L.nvs2 != L.countS && L.tinc < K.DelT)) L.done = 1;
    }
    first = false;
    __syncthreads();
    if (L.done) break;
    // ---- every row's best candidate (VoxelsCA.C:386-445)
    CafeCand best = cafe_cand_none();
    for (int k = tid; k < L.nrows; k += NT) {
      const int r = cafe_row_at(D, L.nrows0, k);
      const uint32_t live = D.row_live[r];
      if (live) cafe_row_best(D, r, D.row_E[r], cafe_vh(D, K, D.row_pos[r]), live, best);
    }
    best = cafe_warp_best(best);
    if (lane == 0) S.red[warp] = best;
    __syncthreads();
    best = cafe_warp_best(lane < NW ? S.red[lane] : cafe_cand_none());
    __syncthreads();
    if (best.j < 0 || !(best.tk < CAFE_KEY_1E6) || L.ev >= max_events) {
      if (tid == 0) {
        if (best.j >= 0 && best.tk < CAFE_KEY_1E6) atomicOr(D.err, CAFE_ERR_ITER_CAP);
        L.done = 1;
      }
      __syncthreads();
      break;
    }
    const int icap = best.q, wr = best.r;
    if (tid == 0) {
      const double U = L.unext[(L.ev + 1) & 1];
      cafe_uniform_stream st;
      st.x = L.rng;
      L.unext[L.ev & 1] = cafe_uniform_next(&st);
      L.rng = st.x;
      L.nuc = U < cafe_nuc_rate_at(D, K, icap);
      L.dt = L.nuc ? 0.0 : best.t;
      if (L.dt < 0.0) L.negdt++;
      L.ev += 1;
      L.countS = L.nvs2;
    }
    __syncthreads();
    const int ev = L.ev;
    // ---- growth of every mushy cell of the list (VoxelsCA.C:511-516)
    if (!L.nuc) {
      double d = L.dt;
      if (isfinite(d)) {
        for (int k = tid; k < L.nrows; k += NT) {
          const int r = cafe_row_at(D, L.nrows0, k);
          if (!D.row_live[r]) continue;
          double e = D.row_E[r] + cafe_vh(D, K, D.row_pos[r]) * d;
          D.row_E[r] = (e < 0.0) ? 0.0 : e;
        }
      } else {
        // a non-finite DtMin also reaches the cells that have no liquid
        // neighbour (0 * inf)
        for (int j = tid; j < L.countS; j += NT) {
          int p = D.vs2[j];
          int r = D.a_frow[p];
          double v = (r >= 0 && D.row_live[r]) ? cafe_vh(D, K, p) : 0.0;
          double *ep = r >= 0 ? &D.row_E[r] : &D.a_ext[p];
          double e = *ep + v * d;
          *ep = (e < 0.0) ? 0.0 : e;
        }
      }
    }
    __syncthreads();
    // ---- the captured cell (VoxelsCA.C:483-505 and 518-605)
    if (tid == 0) {
      D.a_state[icap] = 2;
      if (L.nvs2 < D.vs2_cap) {
        D.vs2[L.nvs2] = icap;
      } else {
        atomicOr(D.err, CAFE_ERR_MUSHY_CAP);
        L.done = 1;
      }
      L.nvs2 += 1;
      if (L.nuc) {
        int ci, cj, ck;
        cafe_cell_xyz(K, D.act[icap], ci, cj, ck);
        if (L.ngrain < D.grain_cap) {
          double q4[4];
          cafe_sample_orientation(K, L.sdloc, q4);
          double *c = D.cth + 4LL * L.ngrain;
          for (int a = 0; a < 4; ++a) c[a] = q4[a];
          cafe_rot_from_cth(c, D.rot + 9LL * L.ngrain);
        } else {
          atomicOr(D.err, CAFE_ERR_GRAIN_CAP);
          L.done = 1;
        }
        L.ngrain += 1;
        L.nc.gid = L.ngrain;
        L.nc.c[0] = ((double)ci + .5) * K.dx[0];
        L.nc.c[1] = ((double)cj + .5) * K.dx[1];
        L.nc.c[2] = ((double)ck + .5) * K.dx[2];
        L.nc.ext = 0.0;
        L.sdloc += 10u;
        L.nnuc++;
      } else {
        const double *gq = D.row_geo + ((long long)wr * CAFE_NSLOT + best.s) * 4;
        L.nc.gid = D.a_gid[D.row_pos[wr]];
        L.nc.ext = gq[0];
        L.nc.c[0] = gq[1];
        L.nc.c[1] = gq[2];
        L.nc.c[2] = gq[3];
      }
      D.a_gid[icap] = L.nc.gid;
      D.a_ext[icap] = L.nc.ext;
      D.a_cx[icap] = L.nc.c[0];
      D.a_cy[icap] = L.nc.c[1];
      D.a_cz[icap] = L.nc.c[2];
      L.tinc += L.dt;
    } else if (warp == 1) {
      // ---- neighbours of the captured cell lose one liquid neighbour
      const int q = lane < CAFE_NSLOT ? D.a_nbr[(long long)icap * CAFE_NSLOT + lane] : -1;
      const bool liq = q >= 0 && D.a_state[q] == 1;
      const bool any = __ballot_sync(0xffffffffu, liq) != 0u;
      if (lane == 0) L.newrow = any && D.a_cold[icap] ? 1 : 0;
      const int r = q >= 0 ? D.a_frow[q] : -1;
      if (r >= 0) {
        const uint32_t live = D.row_live[r], bit = 1u << D.row_rank[(long long)r * 32 + (CAFE_NSLOT - 1 - lane)];
        if (live & bit) {
          D.row_live[r] = live & ~bit;
          if (live == bit) {
            D.row_death[r] = ev;
            D.row_key[r] = CAFE_KEY_NONE;
          }
        }
      }
    }
    __syncthreads();
    // ---- the captured cell becomes a capturing cell if it qualifies
    if (warp < CAFE_QUAD_THREADS / 32 && L.newrow && !L.done) {
      const int r = L.nrows;
      if (r < D.row_cap) {
        if (tid == 0) {
          D.row_pos[r] = icap;
          D.row_j[r] = L.nvs2 - 1;
          D.row_res[r] = -1;
          D.a_frow[icap] = r;
          D.row_death[r] = CAFE_ALIVE;
          D.row_E[r] = L.nc.ext;
          D.row_m[r] = CAFE_M_DONE;
          D.row_new[r - L.nrows0] = r;
        }
        const CafeChildList none = {nullptr, 0, 0, 0.0};
        cafe_row_fill_quad(D, K, r, icap, L.tinc, Q, L.nc, none);
        if (tid == 0) L.nrows = r + 1;
      } else if (tid == 0) {
        atomicOr(D.err, CAFE_ERR_ROW_CAP);
        L.done = 1;
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    D.ctr[CTR_NGRAIN] = L.ngrain;
    D.ctr[CTR_NVS2_END] = L.nvs2;
    D.ctr[CTR_NROWS_END] = L.nrows;
    D.ctr[CTR_NEV] = L.ev;
    D.ctr[CTR_NNUC] = (int)L.nnuc;
    atomicAdd(&D.stat[STAT_EVENTS], (unsigned long long)L.ev);
    atomicAdd(&D.stat[STAT_NUC], (unsigned long long)L.nnuc);
    atomicAdd(&D.stat[STAT_NEGDT], (unsigned long long)L.negdt);
    atomicMax(&D.stat[STAT_MAXNA], (unsigned long long)L.na);
    atomicMax(&D.stat[STAT_MAXROWS], (unsigned long long)L.nrows);
    atomicAdd(&D.stat[STAT_STEPS], 1ULL);
    atomicAdd(&D.stat[STAT_SUMNA], (unsigned long long)L.na);
    atomicAdd(&D.stat[STAT_SUMROWS], (unsigned long long)L.nrows);
    atomicAdd(&D.stat[STAT_EVALS], (unsigned long long)L.opens);
    if (mode || L.sw) atomicAdd(&D.stat[STAT_SLOWSTEPS], 1ULL);
    for (int c = 0; c < 4; ++c) atomicAdd(&D.stat[STAT_CYC_SELECT + c], (unsigned long long)L.cyc[c]);
  }
}
__global__ void __launch_bounds__(CAFE_LOOP_THREADS, 1)
    k_event_loop(const __grid_constant__ CafeDev D, const __grid_constant__ CafeConsts K, const CafeStepParams *__restrict__ Pp, long long max_events, int allow_fast) {
  d_event_loop(D, K, Pp, max_events, allow_fast, blockIdx.x, gridDim.x);
}

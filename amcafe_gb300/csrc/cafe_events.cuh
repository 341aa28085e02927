// Frontier rows and the event loop of one step (VoxelsCA.C:381-610), part of
// cafe_kernels.cu.
//
// A frontier row is a mushy cell with a liquid neighbour. Its slots are the 26
// neighbour directions; those that hold a liquid neighbour are candidates with
// capture time t = fl(fl(g - E)/v), g the slot's numerator, E the row cell's
// extent and v its growth velocity. A row's record lists the slots that held a
// liquid neighbour when it was made by g (CafeSlot row_slot[26], row_n of
// them), so that its earliest candidate is the first one whose neighbour has not
// been captured since (a_ev, the event that captured a position, 0 for none);
// row_k is the place to look from.

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

#define CAFE_DUE_REACH 1.5      // time steps
#define CAFE_OUTSIDE_REACH 1.5  // ... for a row that a capture creates
#define CAFE_SHORT_REACH 1.1    // ... to which a window may shrink
#define CAFE_FEW_ROWS 512       // up to here every row gets its record (one wave of k_rows_geo)

// The extent that a row's growth starts from, for the bounds of its capture time: the
// first capture lifts a negative one (a host program's state may hold such) to zero
// (VoxelsCA.C:515), so it grows by no more than from there.
__device__ __forceinline__ double cafe_lifted(double E) { return cafe_is_neg(E) ? 0.0 : E; }

// Sorts the slots of row r (one per lane: liv, numerator gv, neighbour position
// q) by g (NaN last, ties by slot) into the row's record, and forms the row's key: the order key of T + t
// for its first candidate, a lower bound of the row's absolute capture time
// (CAFE_KEY_NONE without a candidate). E, v and ruq are the row's. Returns, in every
// lane, the order key of the largest |g| of the live slots (0 when none).
__device__ __forceinline__ unsigned long long cafe_row_sort_warp(const CafeDev &D, long long r, bool liv, double gv,
                                                                 int q, double E, double v, double T, int gid, double ruq,
                                                                 const CafeChildList &C, bool fill) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t live = __ballot_sync(FULL, liv);
  const bool gfin = !cafe_is_nan(gv);
  const unsigned long long key = (liv && gfin) ? cafe_key_canon(gv) : CAFE_KEY_NONE;
  int rank = 0;
#pragma unroll
  for (int t = 0; t < CAFE_NSLOT; ++t) {
    unsigned long long kt = cafe_shfl_u64(key, t);
    rank += ((live >> t) & 1u) && (kt < key || (kt == key && t < lane));
  }
  // the slot's capture time and, when it comes due within the step, its child
  double t = NAN;
  uint32_t child = 0;
  if (liv) {
    t = (gv - cafe_lifted(E)) / v;
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
  if (liv) {
    CafeSlot s;
    s.g = gv;
    s.q = q;
    s.m = (uint32_t)lane | child;
    s.rk = cafe_key_canon(.5 * (ruq + D.a_ruq[q]));
    D.row_slot[r * CAFE_NSLOT + rank] = s;
  } else if (fill && lane < CAFE_NSLOT) {
    // (the rest of the record is read along with it: keep it in cache)
    CafeSlot s;
    s.g = NAN;
    s.rk = CAFE_KEY_NONE;
    s.q = 0;
    s.m = 0;
    D.row_slot[r * CAFE_NSLOT + __popc(live) + __popc(~live & ((1u << lane) - 1u))] = s;
  }
  if (lane == 0) {
    D.row_n[r] = (uint8_t)__popc(live);
    D.row_k[r] = 0;
  }
  if (liv && rank == 0) {
    D.row_key[r] = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(T + t);
  }
  if (lane == 0 && live == 0) D.row_key[r] = CAFE_KEY_NONE;
  unsigned long long ak = (liv && gfin) ? cafe_key(fabs(gv)) : 0ULL;
  for (int o = 16; o > 0; o >>= 1) ak = max(ak, cafe_shfl_u64_xor(ak, o));
  return ak;
}

// ------------------------------------------------------------------ lower bounds
// Most rows cannot capture within the step, and their exact geometry (~600 FP64
// instructions a slot, 64 cycles each on this GPU) would only tell that they
// cannot. So every slot's numerator is first bounded in single precision
// (cafe_glb_slot).
// A row whose bound says that it is not due within CAFE_DUE_REACH time steps gets
// no record (row_n = CAFE_NO_RECORD, row_glb its bound), only a key; the event
// loop makes the record if the row is needed after all.
#define CAFE_NO_RECORD 255
// The offsets c0 of a cell (si, sj, sk) from octahedron centre cs.
__device__ __forceinline__ void cafe_glb_centre(const CafeConsts &K, int si, int sj, int sk, const double *cs, float *c0) {
  double dn[3];
  cafe_geo_dn(K, si, sj, sk, cs, dn);
  for (int a = 0; a < 3; ++a) c0[a] = cafe_trunc_f32(dn[a]);
}
// The rotation Rg in single precision, the same in every lane, and its largest entry: an
// entry a lane and shuffles, in place of nine conversions (eight operations each) in every lane.
__device__ __forceinline__ void cafe_glb_rot(const double *Rg, float *R, float &rm) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const float x = lane < 9 ? cafe_trunc_f32(Rg[lane]) : 1.f;
  rm = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(fabsf(x))));
  for (int a = 0; a < 9; ++a) R[a] = __shfl_sync(FULL, x, a);
}
// Smallest lower and largest upper bound over the slots `liv` of a warp; any NaN gives NaN.
__device__ __forceinline__ void cafe_glb_range(bool liv, float &lo, float &hi) {
  const unsigned FULL = 0xffffffffu;
  const bool nan = __any_sync(FULL, liv && !(lo >= 0.f));
  lo = __uint_as_float(__reduce_min_sync(FULL, liv ? __float_as_uint(lo) : 0x7f800000u));
  hi = __uint_as_float(__reduce_max_sync(FULL, liv ? __float_as_uint(hi) : 0u));
  if (nan) lo = hi = NAN;
}
// Lower bound of a row's capture time from the bound of its g.
__device__ __forceinline__ double cafe_lb_time(float glb, double E, double v) {
  const double t = ((double)glb - E) / v;
  return t - fabs(t) * 0x1p-40;
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
  CafeNewCell nc;
};
#define CAFE_QUAD_THREADS 128
__device__ __forceinline__ void cafe_bar_quad(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }

// Geometry of up to 32 slots with four warps of the block together (all 128
// threads call it, with a barrier `bar` of their own): lane t of every warp holds
// slot t (work: the neighbour (ci, cj, ck) of cell (si, sj, sk) with centre cs and
// rotation Rg). A warp issues one FP64 instruction per ~64 cycles whatever its
// active lanes, so the independent chains of a slot run in different warps. First
// stage:
//   warp 0: cos th and the cell distance l; warp 1: sin ph;
//   warp 2: |R^T dn|_1 and the projection on edge p0-p1;
//   warp 3: the projection on edge p0-p2.
// Second stage, after one barrier: warp 0 forms g (returned in warp 0), warp 2 the
// extent and warp 3 the centre a capture through the slot gives (into o).
__device__ __forceinline__ double cafe_geo_quad(const CafeConsts &K, bool work, int ci, int cj, int ck, int si, int sj,
                                                int sk, const double *cs, const double *Rg, CafeQuadScratch &S, int bar,
                                                double *o) {
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3;
  double R[9], loc[3], dr = 0.0, pk[3][3];
  int s0i = 0;
  if (work) {
    double dn[3];
    cafe_geo_dn(K, ci, cj, ck, cs, dn);
    if (w == 0) {
      S.cth[lane] = cafe_geo_costh(dn);
      S.l[lane] = cafe_geo_l(K, ci, cj, ck, si, sj, sk);
    } else if (w == 1) {
      S.sph[lane] = cafe_geo_sinph(dn);
    } else {
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
  cafe_bar_quad(bar);
  if (!work) return 0.0;
  if (w == 0) return crm_pow_half_int(S.cth[lane] * S.sph[lane]) * S.dr[lane];
  if (w >= 2) {
    double Lmud = cafe_geo_lmud(K, S.l[lane], S.d1I[lane], S.dI2[lane], S.d1J[lane], S.dJ3[lane]);
    if (w == 2) {
      double f = crm_pow_half_int(S.cth[lane] * S.sph[lane]);
      o[0] = f * Lmud * 1.0;
    } else {
      double cn[3];
      cafe_geo_centre(R, cs, pk[0], s0i, Lmud, cn);
      o[1] = cn[0];
      o[2] = cn[1];
      o[3] = cn[2];
    }
  }
  return 0.0;
}

// Makes the record of row r, position p, cell nc, at time T with four warps
// (cafe_geo_quad): every slot whose neighbour was liquid at the step's start gets
// its numerator and capture result, and warp 0 sorts. The return value (the order
// key of the row's largest |g|) is valid in warp 0.
__device__ __noinline__ unsigned long long cafe_row_fill_quad(const CafeDev &D, const CafeConsts &K, long long r, int p,
                                                              double T, CafeQuadScratch &S, const CafeNewCell &nc,
                                                              const CafeChildList &C, int bar = 1) {
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3;
  const int gp = nc.gid;
  const bool grain_ok = gp >= 1 && gp <= D.grain_cap;
  bool liv = false;
  int q = -1;
  if (lane < CAFE_NSLOT) {
    q = D.a_nbr[(long long)p * CAFE_NSLOT + lane];
    liv = q >= 0 && (D.a_state[q] == 1 || D.a_ev[q] != 0);
  }
  const bool work = liv && grain_ok;
  int ci = 0, cj = 0, ck = 0, si = 0, sj = 0, sk = 0;
  if (work) {
    cafe_cell_xyz(K, D.act[q], ci, cj, ck);
    cafe_cell_xyz(K, D.act[p], si, sj, sk);
  }
  const double gq = cafe_geo_quad(K, work, ci, cj, ck, si, sj, sk, nc.c, D.rot + 9LL * (grain_ok ? gp - 1 : 0), S, bar,
                                  D.row_geo + (r * CAFE_NSLOT + lane) * 4);
  if (w != 0) return 0ULL;
  // (a capturing cell without a grain never captures)
  return cafe_row_sort_warp(D, r, liv, work ? gq : (liv ? NAN : 0.0), q, nc.ext, cafe_vh(D, K, p), T, gp, D.a_ruq[p], C,
                            true);
}

// ------------------------------------------------------------------ candidates
// A capture candidate: time t and tie-break ruqs, compared through their
// order keys (equal doubles give equal keys; NaN times are never candidates).
struct CafeCand {
  unsigned long long tk, rk;
  double t;
  int j, s;     // vs2 index and neighbour slot of the capturing cell; j < 0 = none
  int r, q;     // (not compared) its row and the captured position
  uint32_t m;   // ... and the slot's CafeSlot::m
};
__device__ __forceinline__ CafeCand cafe_cand_none() {
  CafeCand c;
  c.tk = c.rk = CAFE_KEY_NONE;
  c.t = 0.0;
  c.j = -1;
  c.s = 0;
  c.r = c.q = 0;
  c.m = 0;
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
    c.m = __shfl_xor_sync(0xffffffffu, best.m, o);
    if (cafe_cand_better(c, best)) best = c;
  }
  return best;
}
#define CAFE_KEY_1E6 0xc12e848000000000ULL  // cafe_key(1e6)

// First place from k on in row r's record whose neighbour is not captured;
// row_n[r] when none is left.
__device__ __forceinline__ int cafe_row_next(const CafeDev &D, int r, int k) {
  const int n = D.row_n[r];
  const CafeSlot *rec = D.row_slot + (long long)r * CAFE_NSLOT;
  while (k < n && D.a_ev[rec[k].q] != 0) ++k;
  return k;
}
// Event at which row r lost its last liquid neighbour (it grew at that event
// too), CAFE_ALIVE when one is left. The slots of largest g are captured last,
// so the first look nearly always ends it.
#define CAFE_ALIVE 0x7fffffff
__device__ __forceinline__ int cafe_row_death(const CafeDev &D, int r) {
  if (D.row_n[r] == CAFE_NO_RECORD) {
    const int32_t *nb = D.a_nbr + (long long)D.row_pos[r] * CAFE_NSLOT;
    bool liq = false;
#pragma unroll
    for (int s = 0; s < CAFE_NSLOT; ++s) {
      const int q = nb[s];
      liq |= q >= 0 && D.a_state[q] == 1;
    }
    if (liq) return CAFE_ALIVE;
    int d = 0;
    for (int s = 0; s < CAFE_NSLOT; ++s)
      if (nb[s] >= 0) d = max(d, D.a_ev[nb[s]]);
    return d;
  }
  const CafeSlot *rec = D.row_slot + (long long)r * CAFE_NSLOT;
  int d = 0;
  for (int k = (int)D.row_n[r] - 1; k >= 0; --k) {
    const int e = D.a_ev[rec[k].q];
    if (e == 0) return CAFE_ALIVE;
    d = max(d, e);
  }
  return d;
}

// Best candidate of frontier row r (VoxelsCA.C:386-445 restricted to one cell)
// with extent E and velocity v, looking from place k of its record on. For a
// positive finite velocity the capture time is non-decreasing in g, so the
// visit in g order stops at the first time above the row's minimum; otherwise
// every live slot is evaluated. The reference's acceptance limit t <= 1e6
// (VoxelsCA.C:383, 427) applies.
__device__ __noinline__ void cafe_row_best(const CafeDev &D, int r, double E, double v, int k, CafeCand &best) {
  const long long vb = crm_bits(v);
  const bool mono = vb > 0 && vb < CRM_BITS_INF;  // 0 < v < inf
  bool have = false;
  unsigned long long tfirst = 0;
  for (const int n = D.row_n[r]; k < n; ++k) {
    const CafeSlot s = D.row_slot[(long long)r * CAFE_NSLOT + k];
    if (D.a_ev[s.q] != 0) continue;
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
    c.rk = s.rk;
    c.j = D.row_j[r];
    c.s = (int)(s.m & 31u);
    c.r = r;
    c.q = s.q;
    c.m = s.m;
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
#define CAFE_M_DONE 0x7fffffff  // row_m of a row whose extent is kept current elsewhere

// One event's growth of an extent (VoxelsCA.C:511-516): (E < 0.0) ? 0.0 : E after the
// addition. A nucleation grows no extent (VoxelsCA.C:483-505) and logs -0, which leaves
// every one as it is; one below zero (a host program's state may hold such) is
// lifted by the first event that grows it. On an event's chain, hence one test of the
// sum's high word: a NaN that an addition returns is quiet (above infinity's high
// word), and only -0 with -0 adds up to -0.
__device__ __forceinline__ double cafe_grow(double E, double vd) {
  const bool grows = crm_bits(vd) != ~CRM_ABS_MASK;
  E = E + vd;
  return grows && ((unsigned)__double2hiint(E) ^ 0x80000000u) <= 0x7ff00000u ? 0.0 : E;
}
// Extent of row r after the logged growth of events row_m+1 .. min(upto, its
// last).
template <bool PR>
__device__ __forceinline__ double cafe_row_replayed(const CafeDev &D, int r, int upto, double v, int &stop) {
  const int m = D.row_m[r];
  stop = m < upto ? min(upto, cafe_row_death(D, r)) : m;
  double E = D.row_E[r];
  if (stop <= m) {
    stop = m;
    return E;
  }
  // (the sums are a serial chain: its terms are loaded eight at a time)
  for (int k = m + 1; k <= stop; k += 8) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = D.ev_vd[min(k + u, stop)];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k + u <= stop) E = cafe_grow(E, PR ? v * x[u] : x[u]);
  }
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
// k_rows_prep (eight rows per warp) sets the row's extent and growth watermark, bounds
// its numerators and, when it may be due, lists it and its (row, slot) pairs;
// k_rows_geo evaluates the listed pairs, 32 at a time by four warps; k_rows_order (one warp per listed row)
// sorts the records. CTR_SLOW: bit 0 some row grows with another velocity, bit 1
// some row has a velocity or extent that only the full scan handles. row_mag: the
// magnitudes that bound the keys' rounding, the largest |g| and extent, the
// smallest and the largest velocity over the rows (order keys). Geometry of every
// slot of every row instead took 145 us a step, its sort 26 (512x256x128); now
// k_rows_prep takes 19, k_rows_geo 15 and k_rows_order 8, the longest chain of one
// row each.
#define CAFE_PREP_ROWS 8
__device__ __forceinline__ void d_rows_prep(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  int nrows = D.ctr[CTR_NROWS];
  if (nrows > D.row_cap) nrows = (int)D.row_cap;
  // A warp takes CAFE_PREP_ROWS rows: what is one value per row with a row per
  // lane, then the slots with a direction per lane, one row after another.
  const int warps = (cafe_nblk * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  __shared__ unsigned int mag[4];  // high words of the magnitudes' order keys
  if (threadIdx.x < 4) mag[threadIdx.x] = threadIdx.x == 2 ? 0xffffffffu : 0u;
  __syncthreads();
  int nkey = 0;  // rows without a record that may be candidates
  const double lim = K.DelT * CAFE_DUE_REACH, V1 = K.vhat_cls[1], rV1 = 1.0 / V1;
  const float dx = (float)K.dx[0];
  const bool all = K.all_rows || nrows <= CAFE_FEW_ROWS;
  for (int w = (cafe_bid * blockDim.x + threadIdx.x) >> 5; w * CAFE_PREP_ROWS < nrows; w += warps) {
    const int r0 = w * CAFE_PREP_ROWS, n = min(CAFE_PREP_ROWS, nrows - r0);
    int p = 0, gp = 0;
    float c0[3] = {0.f, 0.f, 0.f}, gmax = 0.f;
    double E = 0.0, v = 1.0;
    if (lane < n) {
      const int r = r0 + lane;
      p = D.row_pos[r];
      gp = D.a_gid[p];
      if (gp < 1 || gp > D.grain_cap) gp = 0;
      E = D.a_ext[p];
      v = cafe_vh(D, K, p);
      int si, sj, sk;
      cafe_cell_xyz(K, D.act[p], si, sj, sk);
      const double cs[3] = {D.a_cx[p], D.a_cy[p], D.a_cz[p]};
      cafe_glb_centre(K, si, sj, sk, cs, c0);
      D.row_E[r] = E;
      D.row_m[r] = 0;
      const int bad = (cafe_v_ordinary(v) && fabs(E) != INFINITY) ? 0 : 2;
      const int slow = bad | (D.a_cls[p] != 1 ? 1 : 0);
      if (slow) atomicOr(&D.ctr[CTR_SLOW], slow);
    }
    float lo = NAN;  // this lane's row
    uint32_t liq = 0u;
    for (int t = 0; t < n; ++t) {
      const int pt = __shfl_sync(FULL, p, t), gt = __shfl_sync(FULL, gp, t);
      float ct[3];
      for (int a = 0; a < 3; ++a) ct[a] = __shfl_sync(FULL, c0[a], t);
      bool liv = false;
      if (lane < CAFE_NSLOT) {
        const int q = D.a_nbr[(long long)pt * CAFE_NSLOT + lane];
        liv = q >= 0 && D.a_state[q] == 1;
      }
      float l = 0.f, h = 0.f;
      if (gt) {
        float R[9], rm;
        cafe_glb_rot(D.rot + 9LL * (gt - 1), R, rm);
        if (liv) cafe_glb_slot(lane, ct, dx, R, rm, l, h);
        cafe_glb_range(liv, l, h);
        gmax = fmaxf(gmax, h);  // (fmaxf drops NaN: such a row's times are NaN)
      }
      const uint32_t bl = __ballot_sync(FULL, liv);
      if (lane == t) {
        lo = gt ? l : NAN;
        liq = bl;
      }
    }
    // the rows that may be due are listed with their pairs
    double tl = ((double)lo - cafe_lifted(E)) * (v == V1 ? rV1 : 1.0 / v);
    tl -= fabs(tl) * 0x1p-40;
    const bool due = lane < n && (all || !gp || !(tl > lim));
    const uint32_t work = due && gp ? liq : 0u;
    const uint32_t bd = __ballot_sync(FULL, due);
    int cnt = __popc(work), incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += u;
    }
    int base = 0, ib = 0;
    if (lane == 31 && incl) base = atomicAdd(&D.ctr[CTR_NPAIRS], incl);
    if (lane == 0 && bd) ib = atomicAdd(&D.ctr[CTR_NDUE], __popc(bd));
    base = __shfl_sync(FULL, base, 31) + incl - cnt;
    ib = __shfl_sync(FULL, ib, 0);
    if (lane < n) {
      const int r = r0 + lane;
      if (due) {
        D.row_due[ib + __popc(bd & ((1u << lane) - 1u))] = r;
        for (uint32_t m = work; m; m &= m - 1) D.row_pairs[base++] = r * 32 + __ffs(m) - 1;
        if (!gp)  // never captures
          for (uint32_t m = liq; m; m &= m - 1) D.row_slot[(long long)r * CAFE_NSLOT + __ffs(m) - 1].g = NAN;
      } else {
        D.row_n[r] = CAFE_NO_RECORD;
        D.row_glb[r] = lo;
        D.row_key[r] = cafe_key(tl);
      }
    }
    nkey += n - __popc(bd);
    // magnitudes, rounded outwards to the keys' high words
    const bool in = lane < n;
    const uint32_t ekey = in && !cafe_is_nan(E) ? (uint32_t)(cafe_key(fabs(E)) >> 32) + 1u : 0u;  // NaN extents occur (the reference's 0/0)
    const uint32_t vkey = (uint32_t)(cafe_key(v) >> 32);
    // (a sign, that of -0.0 too, counts as the smallest; NaN never captures)
    const uint32_t elow =
        __reduce_min_sync(FULL, in && !cafe_is_nan(E) ? (uint32_t)max(__double2hiint(E), 0) : 0xffffffffu);
    if (lane == 0) D.row_low[w] = elow;
    const uint32_t e1 = __reduce_max_sync(FULL, ekey), v0 = __reduce_min_sync(FULL, in ? vkey : 0xffffffffu),
                   v1 = __reduce_max_sync(FULL, in ? vkey + 1u : 0u);
    if (lane == 0) {
      if (gmax > 0.f) atomicMax(&mag[0], (uint32_t)(cafe_key((double)gmax) >> 32) + 1u);
      atomicMax(&mag[1], e1);
      atomicMin(&mag[2], v0);
      atomicMax(&mag[3], v1);
    }
  }
  __syncthreads();
  if (threadIdx.x < 4 && mag[2] != 0xffffffffu) {
    const unsigned long long k = (unsigned long long)mag[threadIdx.x] << 32;
    if (threadIdx.x == 2)
      atomicMin(&D.row_mag[2], k);
    else
      atomicMax(&D.row_mag[threadIdx.x], k);
  }
  if (lane == 0 && nkey) atomicAdd(&D.ctr[CTR_NKEY], nkey);
}
__global__ void k_rows_prep(CafeDev D, CafeConsts K) {
  d_rows_prep(D, K, blockIdx.x, gridDim.x);
}

__device__ __forceinline__ void d_rows_geo(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  __shared__ CafeQuadScratch Q;
  const int lane = threadIdx.x & 31;
  int n = D.ctr[CTR_NPAIRS];
  const long long cap = D.row_cap * CAFE_NSLOT;
  if (n > cap) n = (int)cap;
  for (int i0 = cafe_bid * 32; i0 < n; i0 += cafe_nblk * 32) {
    const bool work = i0 + lane < n;
    int ci = 0, cj = 0, ck = 0, si = 0, sj = 0, sk = 0;
    double cs[3] = {0.0, 0.0, 0.0};
    const double *Rg = D.rot;
    long long o = 0;
    if (work) {
      const int v = D.row_pairs[i0 + lane], r = v >> 5, sl = v & 31, p = D.row_pos[r];
      cafe_cell_xyz(K, D.act[p], si, sj, sk);
      const int d27 = sl < 13 ? sl : sl + 1;
      ci = si + d27 % 3 - 1;
      cj = sj + d27 / 3 % 3 - 1;
      ck = sk + d27 / 9 - 1;
      Rg = D.rot + 9LL * (D.a_gid[p] - 1);
      cs[0] = D.a_cx[p];
      cs[1] = D.a_cy[p];
      cs[2] = D.a_cz[p];
      o = (long long)r * CAFE_NSLOT + sl;
    }
    const double g = cafe_geo_quad(K, work, ci, cj, ck, si, sj, sk, cs, Rg, Q, 1, D.row_geo + o * 4);
    if (work && threadIdx.x < 32) D.row_slot[o].g = g;  // by slot; k_rows_order sorts the record in place
    __syncthreads();  // the scratch is used again
  }
}
__global__ void __launch_bounds__(CAFE_QUAD_THREADS) k_rows_geo(CafeDev D, CafeConsts K) {
  d_rows_geo(D, K, blockIdx.x, gridDim.x);
}

__device__ __forceinline__ void d_rows_order(const CafeDev &D, const CafeConsts &K, const int cafe_bid, const int cafe_nblk) {
  const int n = D.ctr[CTR_NDUE];
  const int warps = (cafe_nblk * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  unsigned long long gk = 0ULL;
  const CafeChildList C = {&D.ctr[CTR_NCHILD], 0, D.ch_cap, K.DelT * CAFE_CHILD_REACH};
  for (int i = (cafe_bid * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const int r = D.row_due[i], p = D.row_pos[r];
    int q = -1;
    bool liv = false;
    double gv = 0.0;
    if (lane < CAFE_NSLOT) {
      q = D.a_nbr[(long long)p * CAFE_NSLOT + lane];
      liv = q >= 0 && D.a_state[q] == 1;
      if (liv) gv = D.row_slot[(long long)r * CAFE_NSLOT + lane].g;
    }
    __syncwarp();  // the record is read before it is written in order
    gk = max(gk, cafe_row_sort_warp(D, r, liv, gv, q, D.row_E[r], cafe_vh(D, K, p), 0.0, D.a_gid[p], D.a_ruq[p], C, false));
  }
  if (lane == 0 && gk) atomicMax(&D.row_mag[0], gk);
}
__global__ void k_rows_order(CafeDev D, CafeConsts K) {
  d_rows_order(D, K, blockIdx.x, gridDim.x);
}

// The rows of foreseen captures, one per block of four warps: generation `depth`
// lists the next one (in CTR_NCHILD + depth + 1) up to ndepth <= CAFE_CHILD_DEPTH. An
// event's chain of dependent captures within one step is rarely longer; a row
// that is not foreseen is filled by the event loop itself (10 us against 30
// for a launch that makes a hundred). Bound by the chain of one row's geometry.
#define CAFE_CHILD_BLOCKS_PER_SM 4
__device__ __forceinline__ void d_children(const CafeDev &D, const CafeConsts &K, int depth, int ndepth, const int cafe_bid, const int cafe_nblk) {
  __shared__ CafeQuadScratch Q;
  __shared__ CafeNewCell nc;
  int off = 0, n = 0;
  for (int d = 0; d <= depth; ++d) {
    off += n;
    n = min(D.ctr[CTR_NCHILD + d], D.ch_cap - off);
  }
  const int last = off + n;
  const CafeChildList C = {&D.ctr[CTR_NCHILD + min(depth + 1, CAFE_CHILD_DEPTH - 1)], last,
                           depth + 1 < ndepth ? D.ch_cap : last, K.DelT * CAFE_CHILD_REACH};
  const int lane = threadIdx.x & 31;
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
    // (every warp evaluates the bound)
    const double T = D.ch_T[i], v = cafe_vh(D, K, p);
    bool liv = false;
    if (lane < CAFE_NSLOT) {
      const int q = D.a_nbr[(long long)p * CAFE_NSLOT + lane];
      liv = q >= 0 && D.a_state[q] == 1;
    }
    bool due = true;
    double tl = 0.0;
    float lo = 0.f, hi = 0.f;
    if (nc.gid >= 1 && nc.gid <= D.grain_cap) {
      int si, sj, sk;
      cafe_cell_xyz(K, D.act[p], si, sj, sk);
      float R[9], c0[3], rm;
      cafe_glb_rot(D.rot + 9LL * (nc.gid - 1), R, rm);
      const float dx = (float)K.dx[0];
      cafe_glb_centre(K, si, sj, sk, nc.c, c0);
      if (liv) cafe_glb_slot(lane, c0, dx, R, rm, lo, hi);
      cafe_glb_range(liv, lo, hi);
      tl = cafe_lb_time(lo, nc.ext, v);
      due = K.all_rows || !(T + tl > K.DelT * CAFE_DUE_REACH) || !cafe_v_ordinary(v);
    }
    unsigned long long gk = 0ULL;
    if (due) {
      gk = cafe_row_fill_quad(D, K, id, p, T, Q, nc, C);
    } else if (threadIdx.x == 0) {
      D.row_n[id] = CAFE_NO_RECORD;
      D.row_glb[id] = lo;
      if (hi > 0.f) gk = cafe_key((double)hi);
    }
    __syncthreads();  // (every warp has read ch_T)
    if (threadIdx.x == 0) {
      D.row_key[id] = CAFE_KEY_NONE;  // until the row exists
      D.row_m[id] = CAFE_M_DONE;  // (set when it leaves the resident set)
      D.ch_T[i] = tl;  // from here on: the bound of the time from its capture to its first
      atomicMax(&D.row_mag[0], gk);
      if (!cafe_is_nan(nc.ext)) atomicMax(&D.row_mag[1], cafe_key(fabs(nc.ext)));
      if (cafe_v_ordinary(v)) {
        atomicMin(&D.row_mag[2], cafe_key(v));
        atomicMax(&D.row_mag[3], cafe_key(v));
      }
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(CAFE_QUAD_THREADS) k_children(const __grid_constant__ CafeDev D, const __grid_constant__ CafeConsts K, int depth, int ndepth) {
  d_children(D, K, depth, ndepth, blockIdx.x, gridDim.x);
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
// the loop otherwise). A resident row's extent and first live slot are in shared
// memory; one thread owns it. What an event costs is instructions on its chain
// (~11 SM cycles each, against ~700 for a load that misses L1), so rows keep no
// live masks: a row looks for its next slot when its first one is captured. Per event:
//   select   every resident's g - E, its minimum over the block by 32-bit order
//            keys (the high word; with PR a single-precision time). When no other
//            candidate's key is within the keys' resolution the minimum stands;
//            else the close ones are compared in full: equal g - E by ruqs, and
//            what only exact times decide in the reference's order (time, ruqs,
//            vs2 index, slot);
//   apply    the owner of a row whose first slot was captured moves it on; one
//            warp updates the captured cell and brings in its row, one thread
//            divides out the capture time and advances the clock, another draws
//            the next event's uniform;
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
#define CAFE_RES_MAX 640  // resident rows
#define CAFE_QUADS 4  // groups of four warps that fill rows side by side
#define CAFE_RES_TARGET 320  // rows an opened window aims at: one per thread with room for the step's new rows
#define CAFE_OPEN_TRIES 48   // windows in a row without an event before the step takes the full scan
#define CAFE_WARPS (CAFE_LOOP_THREADS / 32)
#define CAFE_CAP_WARP (CAFE_LOOP_THREADS / 32 - 1)     // captures
#define CAFE_CLOCK_WARP (CAFE_LOOP_THREADS / 32 - 2)   // capture time and clock
#define CAFE_DRAW_WARP (CAFE_LOOP_THREADS / 32 - 3)    // nucleation draws
#define CAFE_AHEAD_WARP (CAFE_LOOP_THREADS / 32 - 4)   // loads the likely next events' data ahead
#define CAFE_CELL_WARP (CAFE_LOOP_THREADS / 32 - 5)    // the captured cell's state
static_assert(CAFE_CELL_WARP >= 8, "warps 0-3 fill rows");
// Row of the k-th frontier row of the step: the rows present at its start, then
// the rows that captures created, in their order (row_new).
__device__ __forceinline__ int cafe_row_at(const CafeDev &D, int nrows0, int k) {
  return k < nrows0 ? k : D.row_new[k - nrows0];
}

struct CafeLoop {
  // the loop's scalars (VoxelsCA.C:381-610)
  double tinc, dt, vd, vs, rV, vmin, vmax, dsum, gmax, emax;
  double unext[2];  // unext[e & 1]: event e's draw
  int fill, nvs2, countS, nrows0, nrows, ngrain, done, nuc, ev, sw, na, newrow, slow;
  uint32_t rng;
  unsigned int sdloc;
  long long nnuc, negdt, opens, cyc[4];
  int late, outside, filled;  // cafe_event_paths
  CafeNewCell nc;
};
struct CafeResident {
  double g[CAFE_RES_MAX];      // numerator of the first live slot, NaN when none
  double E[CAFE_RES_MAX];      // extent
  double v[CAFE_RES_MAX];      // growth velocity (PR)
  float rv[CAFE_RES_MAX];      // ... and its reciprocal
  unsigned long long rk[CAFE_RES_MAX];  // the first live slot's tie-break ruqs (order key)
  int r[CAFE_RES_MAX];         // row, -1 when free
  int q[CAFE_RES_MAX];         // the first live slot's neighbour position, -1 when none
  uint32_t m[CAFE_RES_MAX];    // ... and its CafeSlot::m
  unsigned char k[CAFE_RES_MAX];     // ... and its place in the record
  unsigned char flag[CAFE_RES_MAX];  // CAFE_RF_*
  unsigned short free[CAFE_RES_MAX];
  // each warp's smallest candidate: key, index, row, position, slot, g - E, tie-break
  uint32_t wh[CAFE_WARPS], wm[CAFE_WARPS];
  int wi[CAFE_WARPS], wr[CAFE_WARPS], wq[CAFE_WARPS], wf[CAFE_WARPS];
  double wd[CAFE_WARPS];
  unsigned long long wrk[CAFE_WARPS];
  unsigned long long wk[CAFE_WARPS], thr[32];  // (opening a window)
  int hist[32];
  int top, nfree, newslot, overflow, nfill, sink[32];
  uint32_t klim[2];  // [e & 1]: a smallest key below it needs no further test at event e
  unsigned long long kw;    // rows with keys at or below it are resident
  double slack;             // rounding bound of the keys
  int outside;              // the row created by this event stays outside the set
  double wlim, dsum_cap;    // latest safe T + t; the window holds while dsum <= dsum_cap and ev <= ev_cap
  int ev_cap, all;          // all: every row with a candidate is resident
  CafeCand red[CAFE_WARPS];
};
#define CAFE_RF_NEAR 1   // the next slot's g is within a relative 2^-19
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

// Place k of the record of row r, resident index i, becomes its first slot;
// place n: none is left.
__device__ __forceinline__ void cafe_res_first(const CafeDev &D, CafeResident &S, int i, int r, int k) {
  const int n = D.row_n[r];
  const CafeSlot *rec = D.row_slot + (long long)r * CAFE_NSLOT;
  // the slots from k on with their capture state, two at a time
  CafeSlot a;
  a.q = -1;
  while (k < n) {
    const CafeSlot x = rec[k], y = rec[min(k + 1, n - 1)];
    const int ex = D.a_ev[x.q], ey = D.a_ev[y.q];
    a = x;
    if (ex == 0) break;
    a = y;
    ++k;
    if (k < n && ey == 0) break;
    ++k;
  }
  if (k >= n) {
    S.g[i] = NAN;
    S.q[i] = -1;
    S.flag[i] = CAFE_RF_DYING;
    return;
  }
  // (a captured next slot may leave the flag set: that only costs a comparison)
  const unsigned long long k1 = cafe_key_canon(a.g);
  const unsigned long long k2 = k + 1 < n ? cafe_key_canon(rec[k + 1].g) : CAFE_KEY_NONE;
  S.g[i] = a.g;
  S.q[i] = a.q;
  S.m[i] = a.m;
  S.rk[i] = a.rk;
  S.k[i] = (unsigned char)k;
  S.flag[i] = k2 - k1 < (1ULL << 33) ? CAFE_RF_NEAR : 0;
}

// A nucleation takes position icap (VoxelsCA.C:483-505).
__device__ __noinline__ void cafe_nucleate(const CafeDev &D, const CafeConsts &K, CafeLoop &L, int icap) {
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
  D.a_gid[icap] = L.nc.gid = L.ngrain;
  D.a_cx[icap] = L.nc.c[0] = ((double)ci + .5) * K.dx[0];
  D.a_cy[icap] = L.nc.c[1] = ((double)cj + .5) * K.dx[1];
  D.a_cz[icap] = L.nc.c[2] = ((double)ck + .5) * K.dx[2];
  L.sdloc += 10u;
  D.a_ext[icap] = L.nc.ext = 0.0;
  L.nnuc++;
}

// Keys within KC of each other may belong to equal times, or be out of order:
// the high word resolves 2^-20; a single-precision time is good to 2^-22. Keys of
// magnitudes at or below KTINY (2^-900, 2^-100) are all close to each other.
template <bool PR>
constexpr __host__ __device__ uint32_t cafe_kc() { return PR ? 16u : 2u; }
template <bool PR>
constexpr __host__ __device__ uint32_t cafe_ktiny() { return 0x80000000u | (PR ? 0x0d800000u : (1023u - 900u) << 20); }
template <bool PR>
constexpr __host__ __device__ int cafe_xm() { return PR ? 0x7f800000 : 0x7ff00000; }
// The largest key that is close to the smallest one, k.
template <bool PR>
__device__ __forceinline__ uint32_t cafe_close_key(uint32_t k) {
  const uint32_t t = k + cafe_kc<PR>(), mag = k & 0x80000000u ? k : ~k;
  return mag <= cafe_ktiny<PR>() ? max(t, cafe_ktiny<PR>()) : t;
}

// The largest key that a winner at clock T may have and be the global one; Vf:
// the common velocity, rounded down.
template <bool PR>
__device__ __forceinline__ uint32_t cafe_window_limit(const CafeResident &S, float Vf, int ev, double T, double dsum) {
  if (!S.all && !(ev < S.ev_cap && (unsigned long long)crm_bits(dsum) <= (unsigned long long)crm_bits(S.dsum_cap))) return 0u;
  double lim = S.wlim - T;
  if (cafe_key(lim) > cafe_key(0x1.e847fp19)) lim = 0x1.e847fp19;  // 0x1.e847fp19 < 1e6
  return cafe_limit_key(lim, Vf, PR);
}

// The loop's rare parts, out of line: an event's chain pays for every
// instruction line that the loop spreads over. They read the device state
// from a copy in shared memory, so that the loop's own stays in constant memory.

// Every resident's extent, place and (keys) key back to the row arrays.
template <bool PR>
__device__ __noinline__ void cafe_res_flush(const CafeDev &D, const CafeConsts &K, CafeLoop &L, CafeResident &S, int ev, bool keys) {
  const double V = K.vhat_cls[1];
  for (int i = threadIdx.x; i < S.top; i += CAFE_LOOP_THREADS) {
    const int r = S.r[i];
    if (r < 0) continue;
    D.row_E[r] = S.E[i];
    D.row_m[r] = ev;
    if (r < L.nrows0) D.row_low[r / CAFE_PREP_ROWS] = 0u;
    D.row_k[r] = S.k[i];
    if (keys) {
      const double t = (S.g[i] - cafe_lifted(S.E[i])) / (PR ? S.v[i] : V);
      D.row_key[r] = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(L.tinc + t);
    }
  }
}

// Row S.r[i] enters: its growth so far, its first live slot.
template <bool PR>
__device__ __noinline__ void cafe_load_resident(const CafeDev &D, const CafeConsts &K, CafeResident &S, int i, int ev) {
  const int r = S.r[i];
  double v = 0.0;
  if (PR) {
    v = cafe_vh(D, K, D.row_pos[r]);
    S.v[i] = v;
    S.rv[i] = 1.0f / (float)v;
  }
  int stop;
  const double E = cafe_row_replayed<PR>(D, r, ev, v, stop);
  S.E[i] = E;
  cafe_res_first(D, S, i, r, D.row_k[r]);
  if (S.flag[i] & CAFE_RF_DYING) {  // every neighbour is captured: not a candidate any more
    D.row_E[r] = E;
    D.row_m[r] = stop;
    D.row_key[r] = CAFE_KEY_NONE;
    S.flag[i] = 0;
    S.r[i] = -1;
    S.free[atomicAdd(&S.nfree, 1)] = (unsigned short)i;
  } else {
    D.row_m[r] = CAFE_M_DONE;  // until it is written back
  }
}

// The record of row r, made by the four warps that call it together (its cell's
// grain, centre and extent are in the active list).
__device__ __forceinline__ void cafe_make_record(const CafeDev &D, const CafeConsts &K, CafeLoop &L, CafeQuadScratch *Q, int r) {
  const int quad = threadIdx.x >> 7, p = D.row_pos[r];
  CafeNewCell &nc = Q[quad].nc;
  if ((threadIdx.x & 127) == 0) {
    nc.gid = D.a_gid[p];
    nc.ext = D.row_E[r];
    nc.c[0] = D.a_cx[p];
    nc.c[1] = D.a_cy[p];
    nc.c[2] = D.a_cz[p];
  }
  cafe_bar_quad(1 + quad);
  const CafeChildList none = {nullptr, 0, 0, 0.0};
  cafe_row_fill_quad(D, K, r, p, L.tinc, Q[quad], nc, none, 1 + quad);
  cafe_bar_quad(1 + quad);  // (the scratch is used again)
}

// Opens the window: the earliest rows by key become resident.
template <bool PR>
__device__ __noinline__ void cafe_window_open(const CafeDev &D, const CafeConsts &K, CafeLoop &L, CafeResident &S, CafeQuadScratch *Q, int ev, int tries) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = CAFE_LOOP_THREADS, NW = CAFE_WARPS;
  const unsigned FULL = 0xffffffffu;
  const double V = K.vhat_cls[1];
  cafe_res_flush<PR>(D, K, L, S, ev, true);
  __syncthreads();
  // the first window takes its rows from the list of those that may be due
  // soon (k_rows_order), later ones from all rows of the step
  const bool first = ev == 0 && tries == 1;
  const int nrows0 = L.nrows0, nrows = first ? D.ctr[CTR_NDUE] : L.nrows;
  auto row_at = [&](int k) -> int { return first ? D.row_due[k] : cafe_row_at(D, nrows0, k); };
  // (a row without a record has to be filled: it counts for twenty)
  auto weight = [&](int r) -> int { return D.row_n[r] == CAFE_NO_RECORD ? 20 : 1; };
  unsigned long long mn = CAFE_KEY_NONE;
  int cnt = 0;
  for (int r0 = tid; r0 < nrows; r0 += 8 * NT) {
    unsigned long long kk[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) kk[u] = r0 + u * NT < nrows ? D.row_key[row_at(r0 + u * NT)] : CAFE_KEY_NONE;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      mn = min(mn, kk[u]);
      if (kk[u] != CAFE_KEY_NONE) cnt += weight(row_at(r0 + u * NT));
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
  if (tid == 0) S.nfill = 0;  // (rows in the first bin)
  for (int i = tid; i < CAFE_RES_MAX; i += NT) {
    S.g[i] = NAN;
    S.q[i] = S.r[i] = -1;
    S.flag[i] = 0;
  }
  __syncthreads();
  mn = cafe_warp_min_key(lane < NW ? S.wk[lane] : CAFE_KEY_NONE, src);
  cnt = __reduce_add_sync(FULL, lane < NW ? S.wi[lane] : 0);
  const bool all = cnt <= CAFE_RES_TARGET;
  // rounding bound of the keys for the next 4096 events and 64 DelT of growth
  // (by one warp: a double-precision operation of all sixteen takes 256 cycles)
  double dcap = 0.0, base = 0.0, slack = 0.0;
  if (warp == 0) {
    dcap = L.dsum + 64.0 * K.DelT;
    base = (mn == CAFE_KEY_NONE ? 0.0 : cafe_unkey(mn));
    slack = (double)(ev + 4096 + 16) * 0x1p-47 *
            (fabs(base) + 64.0 * K.DelT + fabs(L.tinc) + 2.0 * dcap +
             (L.gmax + L.emax) * (PR ? 1.0 / L.vmin : L.rV) * (1.0 + 0x1p-40) + 1e-300);
  }
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
      const int rr = row_at(r);
      const unsigned long long k = D.row_key[rr];
      if (k > last) continue;
      int lo = 0, hi = 31;  // first threshold at or above the key
      while (lo < hi) {
        const int md = (lo + hi) >> 1;
        if (k <= S.thr[md]) hi = md; else lo = md + 1;
      }
      atomicAdd(&S.hist[lo], weight(rr));
      if (lo == 0) atomicAdd(&S.nfill, 1);
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
    if (tid == 0) S.overflow = !fits && S.nfill > CAFE_RES_MAX - 64;
  }
  if (tid == 0) {
    // the rows that are not listed have keys above the listed ones' reach
    const unsigned long long kdue = first && D.ctr[CTR_NKEY] > 0 ? cafe_key(K.DelT * CAFE_DUE_REACH) : CAFE_KEY_NONE - 1;
    const unsigned long long kw = min(kdue, all ? CAFE_KEY_NONE - 1 : S.thr[pick]);
    const bool every = kw == CAFE_KEY_NONE - 1;
    if (all) S.overflow = 0;
    if (!every && !(cafe_unkey(kw) < 1e300)) S.overflow = 1;
    if (!(slack < 1e300) || tries >= CAFE_OPEN_TRIES) S.overflow = 1;
    S.kw = kw;
    S.all = every;
    S.top = 0;
    S.nfree = 0;
    S.ev_cap = ev + 4096;
    S.dsum_cap = dcap;
    S.wlim = every ? INFINITY : cafe_unkey(kw) - slack;
    S.slack = slack;
    S.nfill = 0;
    L.opens++;
    S.klim[(ev + 1) & 1] = cafe_window_limit<PR>(S, __double2float_rd(V), ev, L.tinc, L.dsum);
  }
  __syncthreads();
  if (S.overflow) return;
  const unsigned long long kw = S.kw;
  for (int k = tid; k < nrows; k += NT) {
    const int r = row_at(k);
    if (D.row_key[r] <= kw) {
      const int i = atomicAdd(&S.top, 1);
      if (i < CAFE_RES_MAX) {
        S.r[i] = r;
        if (D.row_n[r] == CAFE_NO_RECORD) S.free[atomicAdd(&S.nfill, 1)] = (unsigned short)i;
      }
    }
  }
  __syncthreads();
  // the records that were not made, four rows at a time
  if (tid == 0) L.late += S.nfill;
  for (int j = warp >> 2; j < S.nfill; j += CAFE_QUADS) cafe_make_record(D, K, L, Q, S.r[S.free[j]]);
  __syncthreads();
  {
    const int top = S.top;
    for (int i = tid; i < top; i += NT) cafe_load_resident<PR>(D, K, S, i, ev);
  }
  __syncthreads();
}

// Exact candidates of the rows with keys at or below kthr, the reference's order
// among them; the best one is left in S.red[0].
template <bool PR>
__device__ __noinline__ void cafe_select_exact(const CafeDev &D, const CafeConsts &K, CafeResident &S, uint32_t kthr) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = CAFE_LOOP_THREADS, NW = CAFE_WARPS;
  const double V = K.vhat_cls[1];
  CafeCand wc = cafe_cand_none();
  const int top = S.top;
  for (int i = tid; i < top; i += NT) {
    const double d = S.g[i] - S.E[i];
    const uint32_t k = cafe_key32(PR ? __float_as_int((float)d * S.rv[i]) : __double2hiint(d), cafe_xm<PR>());
    if (k <= kthr && k != 0xffffffffu) cafe_row_best(D, S.r[i], S.E[i], PR ? S.v[i] : V, S.k[i], wc);
  }
  wc = cafe_warp_best(wc);
  if (lane == 0) S.red[warp] = wc;
  __syncthreads();
  if (warp == 0) {
    wc = cafe_warp_best(lane < NW ? S.red[lane] : cafe_cand_none());
    __syncwarp();
    if (lane == 0) S.red[0] = wc;
  }
  __syncthreads();
}

// A negative event may clamp a small extent at zero (VoxelsCA.C:515),
// which breaks the key bound of a row outside the set: the rows whose
// extrapolated extent comes near zero are brought up to date with a new key
// (true: one of them may be due within the step). A few rows of thousands: those
// of the groups whose smallest extent (row_low) is below the threshold or that
// hold a row brought up to date before, and the step's new rows, are listed in
// shared memory and take a thread each.
template <bool PR>
__device__ __noinline__ bool cafe_negative_event(const CafeDev &D, const CafeConsts &K, CafeLoop &L, CafeResident &S, CafeQuadScratch *Q, int ev) {
  const int tid = threadIdx.x;
  constexpr int NT = CAFE_LOOP_THREADS;
  constexpr int CAP = (int)(sizeof(CafeQuadScratch) * CAFE_QUADS / sizeof(int));
  int *list = (int *)Q;  // (no record is being made)
  const double V = K.vhat_cls[1], rV = L.rV;
  const int nrows = L.nrows, nrows0 = L.nrows0, groups = (nrows0 + CAFE_PREP_ROWS - 1) / CAFE_PREP_ROWS;
  uint32_t lo[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) lo[u] = tid + u * NT < groups ? D.row_low[tid + u * NT] : 0xffffffffu;
  const double vd = L.vd;
  if (tid == 0) {  // (one warp's double-precision work, not sixteen's)
    const double vsp = D.ev_vs[ev - 1], vx = PR ? L.vmax : V;
    const double margin = (double)(ev + 16) * 0x1p-48 * (L.emax + L.gmax + vx * L.dsum + 1e-300);
    // rows that still hold the step's first extents (row_m 0, nearly all) have
    // grown by the whole running sum: they are decided by one threshold
    const double g0 = vsp + vd;
    const double need = PR ? (g0 >= 0.0 ? margin - g0 * L.vmin : margin - g0 * L.vmax) : margin - g0;
    S.thr[0] = need > 0.0 ? (unsigned long long)crm_bits(need * (1.0 + 0x1p-40)) : 0ULL;
    S.thr[1] = (unsigned long long)crm_bits(margin);
    S.thr[2] = (unsigned long long)crm_bits(vsp);
    S.thr[3] = cafe_key(K.DelT * CAFE_SHORT_REACH);
    S.nfill = 0;
  }
  __syncthreads();
  const long long thr0 = (long long)S.thr[0];
  const uint32_t thi = (uint32_t)(S.thr[0] >> 32);
  auto expand = [&](int g) {
    const int n = min(CAFE_PREP_ROWS, nrows0 - g * CAFE_PREP_ROWS), b = atomicAdd(&S.nfill, n);
    for (int u = 0; u < n && b + u < CAP; ++u) list[b + u] = g * CAFE_PREP_ROWS + u;
  };
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (lo[u] <= thi) expand(tid + u * NT);
  for (int g = tid + 4 * NT; g < groups; g += NT)
    if (D.row_low[g] <= thi) expand(g);
  __syncthreads();
  const int nl = S.nfill, nnew = nrows - nrows0;
  const bool listed = nl <= CAP;  // else: every row
  const int n = listed ? nl + nnew : nrows;
  const double margin = crm_from_bits((long long)S.thr[1]), vsp = crm_from_bits((long long)S.thr[2]);
  unsigned long long near = CAFE_KEY_NONE;  // smallest new key
  for (int k = tid; k < n; k += NT) {
    const int r = !listed ? cafe_row_at(D, nrows0, k) : k < nl ? list[k] : D.row_new[k - nl];
    const int m = D.row_m[r];
    const double E = D.row_E[r];
    if (m >= ev || (m == 0 && crm_bits(E) >= thr0)) continue;  // (NaN too: it never captures)
    const double v = PR ? cafe_vh(D, K, D.row_pos[r]) : V;
    const double gr = (vsp - D.ev_vs[m]) + vd;
    if (E + (PR ? v * gr : gr) >= margin) continue;
    int stop;
    const double En = cafe_row_replayed<PR>(D, r, ev, v, stop);
    D.row_E[r] = En;
    D.row_m[r] = stop < ev ? CAFE_M_DONE : ev;  // (a row that stopped growing keeps its extent)
    if (r < nrows0) D.row_low[r / CAFE_PREP_ROWS] = 0u;
    double t = NAN;
    if (D.row_n[r] == CAFE_NO_RECORD) {
      t = ((double)D.row_glb[r] - En) * (PR ? 1.0 / v : rV);
      t -= fabs(t) * 0x1p-40;
    } else {
      const int kn = cafe_row_next(D, r, D.row_k[r]);
      D.row_k[r] = (uint8_t)kn;
      if (kn < D.row_n[r]) {
        const double d = D.row_slot[(long long)r * CAFE_NSLOT + kn].g - En;
        t = PR ? d / v : cafe_div_by(d, V, rV);
      }
    }
    const unsigned long long key = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(L.tinc + t);
    D.row_key[r] = key;
    if (key < near) near = key;
  }
  // one of them due within the step: a new window; else the window ends before it
  if (__syncthreads_or(near <= S.thr[3])) return true;
  if (near < S.kw) atomicMin(&S.kw, near);
  __syncthreads();
  if (tid == 0 && S.kw < CAFE_KEY_NONE - 1) {
    S.all = 0;
    S.wlim = fmin(S.wlim, cafe_unkey(S.kw) - S.slack);
    S.klim[(ev + 1) & 1] = cafe_window_limit<PR>(S, __double2float_rd(V), ev, L.tinc, L.dsum);
  }
  __syncthreads();
  return false;
}

// The captured cell's own row when it was not foreseen, or found no room in the
// resident set (true: open a new window).
template <bool PR>
__device__ __noinline__ bool cafe_new_row(const CafeDev &D, const CafeConsts &K, CafeLoop &L, CafeResident &S, CafeQuadScratch *Q, int ev, int icap) {
  const int tid = threadIdx.x, warp = tid >> 5;
  constexpr int NT = CAFE_LOOP_THREADS;
  const double V = K.vhat_cls[1];
  const int nr = L.newrow;
  if (!L.fill) {
    if (tid == 0) {
      D.row_E[nr] = L.nc.ext;
      const int k = cafe_row_next(D, nr, 0);
      const double t = (D.row_slot[(long long)nr * CAFE_NSLOT + k].g - L.nc.ext) / (PR ? cafe_vh(D, K, icap) : V);
      D.row_key[nr] = cafe_is_nan(t) ? CAFE_KEY_NONE : cafe_key(L.tinc + t);
    }
    __syncthreads();
    return true;
  }
  __syncthreads();
  if (warp < CAFE_QUAD_THREADS / 32) {
    const CafeChildList none = {nullptr, 0, 0, 0.0};
    const unsigned long long gk = cafe_row_fill_quad(D, K, nr, icap, L.tinc, Q[0], L.nc, none);
    if (tid == 0) {
      L.filled++;
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
  if (i >= 0 && i % NT == tid) cafe_load_resident<PR>(D, K, S, i, ev);
  __syncthreads();
  return i < 0;
}

// Keyed loop over the resident set; every thread of the block calls it. Bound by the
// chain of an event, ~6.2k cycles on 512x256x128 (36k when the winner was searched
// among all rows and the captured cell's row made behind it), ~11 cycles an
// instruction: hence one warp per independent part, two barriers, and the rare
// parts out of line. Leaves
// with L.done set, or with L.sw set when the step must continue with the full
// scan (every row's extent and place are then in the row arrays).
template <bool PR>
__device__ __forceinline__ void cafe_events_resident(const CafeDev &D, const CafeConsts &K, long long max_events,
                                                     CafeLoop &L, CafeResident &S, CafeQuadScratch *Q,
                                                     const CafeDev &sD, const CafeConsts &sK) {
  const unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = CAFE_LOOP_THREADS, NW = CAFE_LOOP_THREADS / 32;
  const double V = K.vhat_cls[1];
  constexpr uint32_t KTINY = cafe_ktiny<PR>();
  constexpr int XM = cafe_xm<PR>();
  int ev = 0;
  int tries = 0;  // windows opened since the last event
  bool need_open = true;
  if (tid == 0) S.top = 0;
  __syncthreads();
  long long t0 = clock64();
  const float Vf = __double2float_rd(V);
  const double rV = L.rV, kout = K.DelT * CAFE_OUTSIDE_REACH;
  int cnv = L.nvs2, cnr = L.nrows;  // (capturing warps) list and row counts
  // this thread's smallest and second smallest keys; whether they are known
  uint32_t bk = 0xffffffffu, b2 = 0xffffffffu;
  double bd = 0.0;
  int bi = -1;
  bool have = false;
  auto consider = [&](int i, double d) {  // (g is NaN where no row is)
    const uint32_t k = cafe_key32(PR ? __float_as_int((float)d * S.rv[i]) : __double2hiint(d), XM);
    b2 = min(b2, max(k, bk));
    if (k < bk) {
      bk = k;
      bd = d;
      bi = i;
    }
  };
  while (true) {
    if (need_open) {
      // ---- open the window: the earliest rows by key
      need_open = have = false;
      ++tries;
      cafe_window_open<PR>(sD, sK, L, S, Q, ev, tries);
      if (tid == 0) {
        const long long t1 = clock64();
        L.cyc[3] += t1 - t0;
        t0 = t1;
      }
      if (S.overflow) {
        if (tid == 0) L.sw = 1;
        __syncthreads();
        break;
      }
    }
    // ---- select: the smallest (g - E) / v over the resident rows
    if (!have) {
      bk = b2 = 0xffffffffu;
      const int top = S.top;
      for (int i = tid; i < top; i += NT) consider(i, S.g[i] - S.E[i]);
    }
    {
      const uint32_t wmin = __reduce_min_sync(FULL, bk);
      const uint32_t thr = cafe_close_key<PR>(wmin);
      const uint32_t cl = wmin == 0xffffffffu ? 0u : __ballot_sync(FULL, bk <= thr);
      if (cl == 0u) {
        if (lane == 0) S.wh[warp] = wmin;
      } else {
        int lead = __ffs(cl) - 1;
        // a candidate's own next slot: g apart by 2^-19 relative cannot round
        // together unless the extent dwarfs g
        bool hard = false;
        unsigned long long kf = CAFE_KEY_NONE;
        if (bk <= thr) {
          const int ed = (__double2hiint(bd) >> 20) & 0x7ff, eg = (__double2hiint(S.g[bi]) >> 20) & 0x7ff;
          hard = S.flag[bi] || ed > eg + 20 || b2 <= thr;
          // a tiny g - E is decided here only when it is zero, so that the time is,
          // and g is ordinary, so that the row's next slot is not tiny as well
          if (bk <= KTINY && ~bk <= KTINY) hard = hard || PR || bd != 0.0 || eg < 400;
          kf = cafe_key_canon(bd);
        }
        if (cl & (cl - 1u)) {
          // several close ones: by g - E, then by ruqs (equal g - E gives equal
          // times); apart by less than the division's rounding, or equal in
          // both: undecided here
          const unsigned long long k1 = cafe_warp_min_key(kf, lead);
          const unsigned long long rf = kf == k1 ? S.rk[bi] : CAFE_KEY_NONE;
          const unsigned long long r1 = cafe_warp_min_key(rf, lead);
          const uint32_t eq = __ballot_sync(FULL, kf == k1 && rf == r1);
          hard = __any_sync(FULL, hard || (kf != k1 && kf - k1 < 8)) || (eq & (eq - 1u)) || PR;
        }
        if (lane == lead) {
          S.wh[warp] = wmin;
          S.wf[warp] = hard;
          S.wd[warp] = bd;
          S.wrk[warp] = S.rk[bi];
          S.wi[warp] = bi;
          S.wr[warp] = S.r[bi];
          S.wq[warp] = S.q[bi];
          S.wm[warp] = S.m[bi];
        }
      }
    }
    __syncthreads();
    const uint32_t wkey = lane < NW ? S.wh[lane] : 0xffffffffu;
    const uint32_t kmin = __reduce_min_sync(FULL, wkey);
    const bool inside = kmin < S.klim[(ev + 1) & 1];
    const uint32_t kthr = cafe_close_key<PR>(kmin);
    const uint32_t wcl = __ballot_sync(FULL, wkey <= kthr && wkey != 0xffffffffu);
    int src = __ffs(wcl | 0x80000000u) - 1;
    bool exact = !inside;
    if (!exact) {
      if (wcl & (wcl - 1u)) {  // several warps' candidates are close: likewise among them
        const bool c = wcl >> lane & 1u;
        const unsigned long long kf = c ? cafe_key_canon(S.wd[lane]) : CAFE_KEY_NONE;
        const unsigned long long k1 = cafe_warp_min_key(kf, src);
        const unsigned long long rf = kf == k1 ? S.wrk[lane] : CAFE_KEY_NONE;
        const unsigned long long r1 = cafe_warp_min_key(rf, src);
        const uint32_t eq = __ballot_sync(FULL, kf == k1 && rf == r1);
        exact = __any_sync(FULL, c && (S.wf[lane] || (kf != k1 && kf - k1 < 8))) || (eq & (eq - 1u)) || PR;
      } else {
        exact = S.wf[src];
      }
    }
    src &= NW - 1;
    const double wd = S.wd[src];
    const int win = S.wi[src];
    int wr = S.wr[src], wq = S.wq[src];
    uint32_t wm = S.wm[src];
    if (exact) {
      if (!S.all && !inside) {  // beyond the window (or nothing in it)
        __syncthreads();
        need_open = true;
        continue;
      }
      // exact candidates of the close rows, the reference's order among them
      if (kmin != 0xffffffffu) cafe_select_exact<PR>(sD, sK, S, kthr);
      const bool none = kmin == 0xffffffffu || S.red[0].j < 0 || !(S.red[0].tk < CAFE_KEY_1E6);
      wr = S.red[0].r;
      wq = S.red[0].q;
      wm = S.red[0].m;
      __syncthreads();
      if (none) {  // no candidate is left
        if (tid == 0) L.done = 1;
        __syncthreads();
        break;
      }
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
    const int icap = wq, child = cafe_slot_child(wm);
    double kc = 0.0, dta = 0.0;  // (clock thread) the outside row's key, |dt|
    if (warp == CAFE_CAP_WARP) {
      // the captured cell's row. Level 1: the foreseen row's record (lane = place)
      // and its cell's extent, computed when the capturing row was filled
      int cn = 0;
      double gx = 0.0;
      CafeSlot cr;
      cr.g = NAN;
      cr.rk = CAFE_KEY_NONE;
      cr.q = -1;
      cr.m = 0;
      const bool nuc = L.unext[ev & 1] < cafe_nuc_rate_at(D, K, icap);
      const bool foreseen = child >= 0 && !nuc;
      if (foreseen) {
        cn = D.row_n[child];  // (the record's entries are not valid when there is none)
        if (lane < CAFE_NSLOT) cr = D.row_slot[(long long)child * CAFE_NSLOT + lane];
        if (lane == CAFE_NSLOT) gx = D.row_geo[((long long)wr * CAFE_NSLOT + (wm & 31u)) * 4];
      }
      const bool cold = D.a_cold[icap] != 0;
      const int cls = D.a_cls[icap];
      const double vq = PR ? cafe_vh(D, K, icap) : V;
      const int nf = S.nfree, tp = S.top;
      // level 2: which of its neighbours (all but the captured ones) are left
      const bool rec = foreseen && cn != CAFE_NO_RECORD;
      bool left = false;
      if (rec) {
        left = lane < cn && D.a_ev[cr.q] == 0;
      } else if (lane < CAFE_NSLOT) {
        const int q = D.a_nbr[(long long)icap * CAFE_NSLOT + lane];
        left = q >= 0 && D.a_state[q] == 1;
      }
      const uint32_t clive = __ballot_sync(FULL, left);
      const bool grows = clive != 0u && cold, room = cnr < D.row_cap;
      const int row = foreseen ? child : cnr;
      // a foreseen row enters the resident set at once
      const bool enter = grows && rec && room && (nf > 0 || tp < CAFE_RES_MAX);
      const int ci = !enter ? -1 : nf > 0 ? (int)S.free[nf - 1] : tp;
      const int k1 = __ffs(clive | 0x80000000u) - 1;
      const double g2 = __shfl_sync(FULL, cr.g, (k1 + 1) & 31);
      if (enter) {
        if (lane == k1) {
          const unsigned long long d2 = k1 + 1 < cn ? cafe_key_canon(g2) - cafe_key_canon(cr.g) : CAFE_KEY_NONE;
          S.g[ci] = cr.g;
          S.q[ci] = cr.q;
          S.m[ci] = cr.m;
          S.rk[ci] = cr.rk;
          S.k[ci] = (unsigned char)k1;
          S.flag[ci] = d2 < (1ULL << 33) ? CAFE_RF_NEAR : 0;
          S.r[ci] = child;
          if (PR) {
            S.v[ci] = vq;
            S.rv[ci] = 1.0f / (float)vq;
          }
        }
        if (lane == CAFE_NSLOT) S.E[ci] = gx;
        if (lane == 30) {
          if (nf > 0) S.nfree = nf - 1;
          else S.top = tp + 1;
        }
      }
      if (lane == CAFE_NSLOT && foreseen && !rec) D.row_E[child] = gx;
      if (lane == 31) {
        L.newrow = grows && room ? row : -1;
        L.fill = !rec;
        S.newslot = ci;
        if (grows) {
          if (room) {
            D.row_j[row] = cnv;
            D.a_frow[icap] = row;
            D.row_new[cnr - L.nrows0] = row;
            L.nrows = cnr + 1;
            if (ci < 0) {
              D.row_pos[row] = icap;
              D.row_m[row] = ev;
            }
            // a cell of another growth velocity
            if (PR) {
              if (!cafe_v_ordinary(vq)) L.sw = 1;
              L.vmin = fmin(L.vmin, vq);
              L.vmax = fmax(L.vmax, vq);
            } else if (cls != 1) {
              L.sw = 1;
            }
          } else {
            atomicOr(D.err, CAFE_ERR_ROW_CAP);
            L.done = 1;
          }
        }
      }
      cnv += 1;
      cnr += grows && room;
    } else if (warp == CAFE_CELL_WARP) {
      // the captured cell (VoxelsCA.C:483-505 and 518-605): the capture result of
      // this slot (lanes 26-29: extent and centre), the grain
      if (lane == 31) {
        D.a_state[icap] = 2;
        D.a_ev[icap] = ev;
        if (cnv < D.vs2_cap) {
          D.vs2[cnv] = icap;
        } else {
          atomicOr(D.err, CAFE_ERR_MUSHY_CAP);
          L.done = 1;
        }
      }
      cnv += 1;
      if (L.unext[ev & 1] < cafe_nuc_rate_at(D, K, icap)) {
        if (lane == 0) cafe_nucleate(sD, sK, L, icap);
      } else if (lane >= CAFE_NSLOT && lane < 30) {
        const double gx = D.row_geo[((long long)wr * CAFE_NSLOT + (wm & 31u)) * 4 + lane - 26];
        // (one store each: the destination by lane)
        double *gd = lane == 26 ? D.a_ext : lane == 27 ? D.a_cx : lane == 28 ? D.a_cy : D.a_cz;
        double *sd = lane == 26 ? &L.nc.ext : &L.nc.c[(lane - 27) & 3];
        gd[icap] = gx;
        *sd = gx;
        if (lane == 26 && fabs(gx) == INFINITY) L.sw = 1;  // its times need the full scan
      } else if (lane == 30) {
        D.a_gid[icap] = L.nc.gid = D.a_gid[D.row_pos[wr]];
      }
    } else if (tid == CAFE_CLOCK_WARP * 32) {
      // the capture time, the clock (VoxelsCA.C:381, 483-516) and the growth log
      const bool nuc = L.unext[ev & 1] < cafe_nuc_rate_at(D, K, icap);
      int cn = 0;
      if (child >= 0) {
        cn = D.row_n[child];
        kc = D.ch_T[child - (int)D.row_cap];
      }
      const double t = exact ? S.red[0].t : (PR ? wd / S.v[win] : cafe_div_by(wd, V, rV));
      const double dt = nuc ? 0.0 : t;
      const double vd = nuc ? -0.0 : PR ? dt : V * dt;  // (cafe_grow)
      const double tinc = L.tinc + dt;
      L.vd = vd;
      D.ev_vd[ev] = vd;
      L.tinc = tinc;
      // while (vSind2 != countS && tinc < DelT): an event always lengthens the list
      if (cafe_is_nan(tinc) || !(cafe_key(tinc) < cafe_key(K.DelT))) L.done = 1;
      const double vs = L.vs + vd;
      L.vs = vs;
      D.ev_vs[ev] = vs;
      if (cafe_is_neg(dt)) L.negdt++;
      dta = fabs(dt);
      // a foreseen row that is not due within the step stays outside the set, and
      // the window ends before its key
      kc = tinc + kc;
      S.outside = child >= 0 && !nuc && cn == CAFE_NO_RECORD && kc > kout;
    } else if (tid == CAFE_DRAW_WARP * 32) {
      // the next event's draw (VoxelsCA.C:483; two engine outputs per event)
      cafe_uniform_stream st;
      st.x = L.rng;
      L.unext[(ev + 1) & 1] = cafe_uniform_next(&st);
      L.rng = st.x;
    } else if (warp == CAFE_AHEAD_WARP) {
      // the event most likely to follow (the smallest candidate of the other
      // warps that does not aim at the captured cell; right in two of three
      // events): what its capture loads, into this SM's L1
      const uint32_t a = lane < NW && lane != src && wkey != 0xffffffffu && S.wq[lane] != icap ? wkey : 0xffffffffu;
      const uint32_t k2 = __reduce_min_sync(FULL, a);
      if (k2 != 0xffffffffu) {
        const int s2 = __ffs(__ballot_sync(FULL, a == k2)) - 1;
        const int q2 = S.wq[s2], r2 = S.wr[s2], c2 = cafe_slot_child(S.wm[s2]);
        int x = 0;  // (kept, so that the loads are)
        if (lane < CAFE_NSLOT) {
          if (c2 >= 0) {
            if (D.row_n[c2] != CAFE_NO_RECORD) {
              const CafeSlot cs = D.row_slot[(long long)c2 * CAFE_NSLOT + lane];
              x = D.a_ev[cs.q] + (int)cs.m + __double2hiint(cs.g) + (int)cs.rk;
            } else {
              x = D.a_nbr[(long long)q2 * CAFE_NSLOT + lane];
              if (x >= 0) x = D.a_state[x];
            }
          }
        } else if (lane < 30) {
          x = __double2hiint(D.row_geo[((long long)r2 * CAFE_NSLOT + (S.wm[s2] & 31u)) * 4 + lane - 26]);
        } else if (lane == 30) {
          x = D.a_gid[D.row_pos[r2]];
        } else {
          x = D.a_cold[q2] + D.a_cls[q2];
        }
        S.sink[lane] = x;
      }
    }
    // a row whose first slot is the captured cell moves on to its next one (the
    // captured cell itself counts as captured by then)
    {
      const int top = S.top;
      for (int i = tid; i < top; i += NT)
        if (S.q[i] == icap) cafe_res_first(D, S, i, S.r[i], S.k[i] + 1);
    }
    __syncthreads();
    // ---- grow (VoxelsCA.C:511-516), and the next event's smallest candidates; a
    // row that lost its last slot leaves
    const int born = S.newslot;
    {
      const double vd = L.vd;
      const int top = S.top;
      bk = b2 = 0xffffffffu;
      for (int i = tid; i < top; i += NT) {
        double E = S.E[i];
        // (a row created by this event grows from the next one on)
        if (i != born && S.r[i] >= 0) {
          E = cafe_grow(E, PR ? S.v[i] * vd : vd);
          S.E[i] = E;
          if (S.flag[i] & CAFE_RF_DYING) {
            const int r = S.r[i];
            D.row_E[r] = E;
            D.row_m[r] = ev;
            D.row_key[r] = CAFE_KEY_NONE;
            S.flag[i] = 0;
            S.r[i] = -1;
            S.free[atomicAdd(&S.nfree, 1)] = (unsigned short)i;
          }
        }
        consider(i, S.g[i] - E);
      }
      have = true;
    }
    if (tid == CAFE_CLOCK_WARP * 32) {
      // the window's limit for the next event
      const double dsum = L.dsum + dta;
      L.dsum = dsum;
      if (S.outside) {
        const unsigned long long key = cafe_key(kc);
        D.row_key[child] = key;
        if (key < S.kw) {
          S.kw = key;
          S.wlim = kc - S.slack;
        }
        S.all = 0;
      }
      S.klim[(ev + 1) & 1] = cafe_window_limit<PR>(S, Vf, ev, L.tinc, dsum);
      L.outside += S.outside;
    }
    if (tid == 0) {
      const long long t1 = clock64();
      L.cyc[1] += t1 - t0;
      t0 = t1;
    }
    // ---- events with more to do than the row that was foreseen
    const bool neg = cafe_is_neg(L.vd), fresh = L.newrow >= 0 && born < 0 && !S.outside;
    if (neg || fresh) {
      __syncthreads();
      have = false;
      if (neg && cafe_negative_event<PR>(sD, sK, L, S, Q, ev)) need_open = true;
      if (fresh) {
        if (cafe_new_row<PR>(sD, sK, L, S, Q, ev, icap)) need_open = true;
        if (tid == 0) {
          const long long t1 = clock64();
          L.cyc[2] += t1 - t0;
          t0 = t1;
        }
      }
    }
    if (L.done || L.sw) break;
  }
  cafe_res_flush<PR>(sD, sK, L, S, ev, false);
  if (tid == CAFE_CAP_WARP * 32) {
    L.nvs2 = cnv;
    L.countS = cnv - 1;
  }
  if (tid == 0) {
    L.ev = ev;
    D.ctr[CTR_EVLOG] = PR ? 1 : 0;
  }
  __syncthreads();
}

// The reference's scan of every row per event: from the start (mode 2), or where
// the resident loop stopped with L.sw.
__device__ __noinline__ void cafe_events_scan(const CafeDev &D, const CafeConsts &K, long long max_events, CafeLoop &L,
                                              CafeResident &S, CafeQuadScratch *Q, int mode) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = CAFE_LOOP_THREADS, NW = CAFE_WARPS;
  if (L.done || !(mode == 2 || L.sw)) return;
  if (tid == 0) atomicAdd(&D.stat[STAT_FULLSCAN], 1ULL);
  {
    // every row needs its record, and extents are kept current from here on
    for (int k = warp >> 2; k < L.nrows; k += CAFE_QUADS) {
      const int r = cafe_row_at(D, L.nrows0, k);
      if (D.row_n[r] == CAFE_NO_RECORD) cafe_make_record(D, K, L, Q, r);
    }
    __syncthreads();
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
  while (!L.done) {
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
      const int k0 = D.row_k[r], k1 = cafe_row_next(D, r, k0);
      if (k1 != k0) D.row_k[r] = (uint8_t)k1;
      if (k1 < D.row_n[r]) cafe_row_best(D, r, D.row_E[r], cafe_vh(D, K, D.row_pos[r]), k1, best);
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
          if (D.row_k[r] >= D.row_n[r]) continue;  // (no liquid neighbour)
          double e = D.row_E[r] + cafe_vh(D, K, D.row_pos[r]) * d;
          D.row_E[r] = (e < 0.0) ? 0.0 : e;
        }
      } else {
        // a non-finite DtMin also reaches the cells that have no liquid
        // neighbour (0 * inf)
        for (int j = tid; j < L.countS; j += NT) {
          int p = D.vs2[j];
          int r = D.a_frow[p];
          double v = (r >= 0 && D.row_k[r] < D.row_n[r]) ? cafe_vh(D, K, p) : 0.0;
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
      D.a_ev[icap] = ev;
      if (L.nvs2 < D.vs2_cap) {
        D.vs2[L.nvs2] = icap;
      } else {
        atomicOr(D.err, CAFE_ERR_MUSHY_CAP);
        L.done = 1;
      }
      L.nvs2 += 1;
      if (L.nuc) {
        cafe_nucleate(D, K, L, icap);
      } else {
        const double *gq = D.row_geo + ((long long)wr * CAFE_NSLOT + best.s) * 4;
        D.a_gid[icap] = L.nc.gid = D.a_gid[D.row_pos[wr]];
        D.a_ext[icap] = L.nc.ext = gq[0];
        D.a_cx[icap] = L.nc.c[0] = gq[1];
        D.a_cy[icap] = L.nc.c[1] = gq[2];
        D.a_cz[icap] = L.nc.c[2] = gq[3];
      }
      L.tinc += L.dt;
    } else if (warp == 1) {
      const int q = lane < CAFE_NSLOT ? D.a_nbr[(long long)icap * CAFE_NSLOT + lane] : -1;
      const bool any = __any_sync(0xffffffffu, q >= 0 && D.a_state[q] == 1);
      if (lane == 0) L.newrow = any && D.a_cold[icap] ? 1 : 0;
    }
    __syncthreads();
    // ---- the captured cell becomes a capturing cell if it qualifies
    if (warp < CAFE_QUAD_THREADS / 32 && L.newrow && !L.done) {
      const int r = L.nrows;
      if (r < D.row_cap) {
        if (tid == 0) {
          D.row_pos[r] = icap;
          D.row_j[r] = L.nvs2 - 1;
          D.a_frow[icap] = r;
          D.row_E[r] = L.nc.ext;
          D.row_m[r] = CAFE_M_DONE;
          D.row_new[r - L.nrows0] = r;
        }
        const CafeChildList none = {nullptr, 0, 0, 0.0};
        cafe_row_fill_quad(D, K, r, icap, L.tinc, Q[0], L.nc, none);
        if (tid == 0) L.nrows = r + 1;
      } else if (tid == 0) {
        atomicOr(D.err, CAFE_ERR_ROW_CAP);
        L.done = 1;
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void d_event_loop(const CafeDev &D, const CafeConsts &K, const CafeStepParams *__restrict__ Pp, long long max_events, int allow_fast, const int cafe_bid, const int cafe_nblk) {
  __shared__ CafeLoop L;
  __shared__ CafeResident S;
  __shared__ CafeQuadScratch Q[CAFE_QUADS];
  __shared__ CafeDev sD;
  __shared__ CafeConsts sK;
  const int tid = threadIdx.x;
  constexpr int NT = CAFE_LOOP_THREADS;
  if (cafe_bid != 0) return;  // event_fill_helper's second block: the loop leaves it nothing to do
  for (int i = tid; i < (int)(sizeof(CafeDev) / 4); i += NT) ((uint32_t *)&sD)[i] = ((const uint32_t *)&D)[i];
  for (int i = tid; i < (int)(sizeof(CafeConsts) / 4); i += NT) ((uint32_t *)&sK)[i] = ((const uint32_t *)&K)[i];
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
    L.rV = 1.0 / K.vhat_cls[1];
    L.tinc = L.dsum = L.vd = L.dt = L.vs = 0.0;
    L.gmax = D.row_mag[0] ? cafe_unkey(D.row_mag[0]) : 0.0;
    L.emax = D.row_mag[1] ? cafe_unkey(D.row_mag[1]) : 0.0;
    L.vmin = D.row_mag[2] != CAFE_KEY_NONE ? cafe_unkey(D.row_mag[2]) : 1.0;
    L.vmax = D.row_mag[3] ? cafe_unkey(D.row_mag[3]) : 1.0;
    L.countS = L.na;
    L.nnuc = L.negdt = L.opens = 0;
    L.late = L.outside = L.filled = 0;
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
      cafe_events_resident<false>(D, K, max_events, L, S, Q, sD, sK);
    else if (mode == 1)
      cafe_events_resident<true>(D, K, max_events, L, S, Q, sD, sK);
  }
  cafe_events_scan(sD, sK, max_events, L, S, Q, mode);
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
    if (L.late) atomicAdd(&D.stat[STAT_LATE], (unsigned long long)L.late);
    if (L.outside) atomicAdd(&D.stat[STAT_OUTSIDE], (unsigned long long)L.outside);
    if (L.filled) atomicAdd(&D.stat[STAT_FILLED], (unsigned long long)L.filled);
    for (int c = 0; c < 4; ++c) atomicAdd(&D.stat[STAT_CYC_SELECT + c], (unsigned long long)L.cyc[c]);
  }
}
__global__ void __launch_bounds__(CAFE_LOOP_THREADS, 1)
    k_event_loop(const __grid_constant__ CafeDev D, const __grid_constant__ CafeConsts K, const CafeStepParams *__restrict__ Pp, long long max_events, int allow_fast) {
  d_event_loop(D, K, Pp, max_events, allow_fast, blockIdx.x, gridDim.x);
}

// DOM sweep, register-patch kernel (path 8, kernel 3).
//
// As in the pencil kernel, one thread-block cluster sweeps an octant, its CTAs
// split the k' rows and hand their last row to the next CTA through a ring in
// its shared memory.  What differs is where the values live and how they move:
//
//  * A thread owns RK rows of one column of pencils and keeps their intensities
//    of all MO ordinates in registers, so the x-inflow is a register, and so is
//    the z-inflow inside the patch; the rest passes through shared memory (one
//    plane double-buffered, 16-byte accesses, conflict-free because a pencil's
//    MO values are contiguous).  The quadrature's few distinct constants stay
//    in registers too.
//  * (kappa, kappa B) and the y-inflow rows are held by hyperplane (four
//    orientations of the former serve the eight octants), so what all of a
//    CTA's rows read on one hyperplane is one run: two bulk copies
//    (cp.async.bulk) a step, RP_KS steps ahead, and no thread loads from global
//    memory.  The octant partials of G and the ground flux are in skewed arrays
//    [k'][i' + j'][j'], so a warp's stores are runs too.  In the natural layout
//    every lane touches a line of its own.
//  * The last row's pencils store into the next CTA's ring themselves (16-byte
//    st.async, counted on its mbarrier), and each warp of the first row block
//    releases the slot it has read; only the warps concerned wait for the ring.
//    There is no helper warp: with one, the
//    register file would leave the twelve compute warps 128 registers a thread
//    (FP64, ten ordinates: spills) instead of 160.
//  * The quotient's reciprocal is shared by the ordinates of a pair (m, m')
//    that differ by swapping the x and y components: on a grid with dx == dy
//    their denominators are the same numbers (PAIR; checked on the host).
//
// Time is counted per CTA: at step t its row r holds the cells with
// i' + j' = t - r, so a CTA with rows rows runs S + rows - 1 steps (S = nx + ny
// - 1) and needs item t of the CTA before it at step t.  The arithmetic of a
// cell, the order in which an octant's ordinates are summed and the order of
// the octants are the pencil kernel's, so the results are the same bit for bit.
//
// Measured, a sweep of 400 x 120 x 60 with S8 (10 CTAs of 6 rows an octant):
// FP64 890 us, FP32 620 us (pencil kernel 1810 and 1357); 97 x 41 x 23 with S4:
// 110 us (167).  What bounds it is latency: a step takes about 3300 cycles, of
// which the busiest scheduler's FP64 pipe works 1300 and issues 1500; a warp by
// itself needs 1700 (about four cycles an instruction), and the barrier waits
// for the slowest of twelve.
#pragma once

#define RP_KS 4      // steps of prefetched inputs
#define RP_ZS_MAX 8  // slots of the row hand-off ring (4 where shared memory is short)
template <int MO> struct RpShape;
// Rows per thread and warps at most: 6 rows of 97 to 128 pencils, what a CTA has to
// hold for 60 levels to run in one wave of clusters.  Ten ordinates: two rows a
// thread at 168 registers.  Six and three: one row at 80, which the FP64 form of six
// exceeds by 36 bytes of spill loads; with them its sweep takes 790 us at
// 400 x 120 x 60 (FP32 528), the pencil kernel's 1359 (1051), and at 133 x 45 x 37
// 168 (147) against 301 (242).  Three: 542 (451) against 857 (736).
template <> struct RpShape<10> { static constexpr int RK = 2, MAXW = 12; };
template <> struct RpShape<6> { static constexpr int RK = 1, MAXW = 24; };
template <> struct RpShape<3> { static constexpr int RK = 1, MAXW = 24; };

// The level-symmetric point order of an octant (points (i, j, k) of levels with
// i + j + k = NL - 1, k fastest), one hexadecimal digit per ordinate from the
// right: the level of each component, the weight class, and the first ordinate
// of the class of equal denominators (x and y components swapped).
template <int MO> struct RpPoints;
template <> struct RpPoints<10> {
  static constexpr int NL = 4, NW = 3;
  static constexpr unsigned long long X = 0x3221110000, Y = 0x0102103210, Z = 0x0010120123,
                                      W = 0x0111210110, PAIR = 0x3626513210;
};
template <> struct RpPoints<6> {
  static constexpr int NL = 3, NW = 2;
  static constexpr unsigned long long X = 0x211000, Y = 0x010210, Z = 0x001012, W = 0x011010,
                                      PAIR = 0x241210;
};
template <> struct RpPoints<3> {
  static constexpr int NL = 2, NW = 1;
  static constexpr unsigned long long X = 0x100, Y = 0x010, Z = 0x001, W = 0x000, PAIR = 0x110;
};
__host__ __device__ constexpr int rp_digit(unsigned long long d, int m) {
  return (int)((d >> (4 * m)) & 15);
}

template <typename T, int MO>
struct RpArgs {
  // (kappa, kappa B) by hyperplane, [plane][k][j], for the four orientations
  // of an octant up to reversal (rp_class)
  const typename Vec2Of<T>::type* kb[4];
  const T *igA, *igB;  // ground intensity, [i + j][j] and [i - j + ny - 1][j]
  T *Goct, *Qoct, *wrap;
  const double *ox, *oy, *oz;  // ordinate components (the first MO: the first octant's)
  double I_amb, dz0;
  // |component| / spacing by level, the denominators' constant part by ordinate,
  // the weights by class; az and as hold for levels of height dz0 (other
  // levels: a table in shared memory)
  T ax[RpPoints<MO>::NL], ay[RpPoints<MO>::NL], az[RpPoints<MO>::NL], as[MO], w[RpPoints<MO>::NW],
      wq[MO];
  int C, rows, pitch, zs;
  unsigned char fx[8], fy[8], fz[8];
  signed char slot[8];  // ground-flux slot of a downward octant, -1 upward
  const int* done;
  int* err;
  int withhold;
};

// a pencil's MO values, padded to whole 16-byte runs where a bulk copy moves them
__host__ __device__ constexpr int rp_pad(int tsize, int MO) {
  return tsize == 8 ? (MO + 1) / 2 * 2 : (MO + 3) / 4 * 4;
}
__host__ __device__ inline int rp_pitch(int ny) { return (ny + 3) / 4 * 4; }
// an octant's orientation class and whether its planes run backwards in it
__host__ __device__ inline int rp_class(bool fx, bool fy, bool fz) {
  return (fx == fy ? 0 : 1) + (fx == fz ? 0 : 2);
}

struct RpLayout {
  size_t bars, kab, yin, ig, xb, spare, zin, tz, total, rowb;
};
__host__ __device__ inline RpLayout rp_layout(int tsize, int Mo, int rows, int ny, int zs) {
  RpLayout L;
  const size_t pitch = (size_t)rp_pitch(ny);
  size_t o = 0;
  L.rowb = up16((size_t)ny * Mo * tsize);
  // (and two words: the step and the row of the ring whose wait gave up)
  L.bars = o; o = up16(o + (RP_KS + 2 * RP_ZS_MAX + 1) * sizeof(unsigned long long));
  L.kab = o; o = up16(o + RP_KS * rows * pitch * 2 * tsize);
  L.yin = o; o = up16(o + RP_KS * (size_t)rows * rp_pad(tsize, Mo) * tsize);
  L.ig = o; o = up16(o + RP_KS * pitch * tsize);
  L.spare = o; o = up16(o + 2 * (size_t)Mo * tsize);  // of patch rows that do not exist
  L.xb = o; o = up16(o + 2 * (size_t)rows * L.rowb);
  L.zin = o; o = up16(o + zs * L.rowb);
  L.tz = o; o = up16(o + (size_t)rows * Mo * 2 * tsize);
  L.total = o;
  return L;
}

// contiguous global bytes into this CTA's shared memory, counted on its mbarrier
__device__ __forceinline__ void rp_bulk_in(uint32_t dst, const void* src, uint32_t bytes,
                                           uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
// two adjacent values into another CTA's shared memory, counted on its mbarrier
__device__ __forceinline__ void rp_st_async2(uint32_t a, double x, double y, uint32_t bar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(a),
      "d"(x), "d"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void rp_st_async2(uint32_t a, float x, float y, uint32_t bar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(a),
      "f"(x), "f"(y), "r"(bar)
      : "memory");
}
template <typename T, int MO>
__device__ __forceinline__ void rp_send(uint32_t p, uint32_t bar, const T (&v)[MO]) {
  if constexpr (MO % 2 == 0) {
#pragma unroll
    for (int m = 0; m < MO; m += 2)
      rp_st_async2(p + (uint32_t)(m * sizeof(T)), v[m], v[m + 1], bar);
  } else {
#pragma unroll
    for (int m = 0; m < MO; ++m) cl_st_async(p + (uint32_t)(m * sizeof(T)), v[m], bar);
  }
}

// cl_wait and cl_arrive_remote at CTA scope: with the cluster scope's release
// and acquire every wait and signal would also order this thread's global
// stores (the partials of G), about a thousand cycles a step.  What passes
// through the ring is ordered without them: the values arrive by st.async,
// whose bytes complete the barrier phase, and a slot is released after its
// values were used.
__device__ __forceinline__ bool rp_poll(uint32_t addr, uint32_t parity, int limit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// Bounded wait.  A thread whose wait gave up does not wait, signal or send
// again on what it waited for: the row ring (RP_RING) or the inputs (RP_IN).
// The two are separate, as the thread that waits for the inputs may be one that
// sends or takes rows: with the ring given up it must go on waiting for its
// copies, or it would announce new ones on phases that are still open.
#define RP_RING 1u
#define RP_IN 2u
__device__ __forceinline__ bool rp_wait(uint32_t addr, uint32_t parity, unsigned& failed,
                                        unsigned what, int* err) {
  if (failed & what) return true;
  if (rp_poll(addr, parity, CL_WAIT_LIMIT)) return true;
  failed |= what;
  if (err) atomicExch(err, 1);
  return false;  // once
}
// try_wait rounds for copies and rows still under way when a CTA leaves, over
// all the phases it asks about
#define RP_DRAIN_LIMIT (1 << 16)
__device__ __forceinline__ void rp_release(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// N consecutive values from m0 on by 32-bit shared address, two at a time where
// MO is even; volatile, so a batch's loads and stores stay where they are put
// (the register budget depends on it)
template <typename T, int MO, int N>
__device__ __forceinline__ void rp_ld(uint32_t p, int m0, T (&v)[N]) {
  if constexpr (MO % 2 == 0) {
#pragma unroll
    for (int m = 0; m < N; m += 2) {
      const auto x = sh_ld2<typename Vec2Of<T>::type>(p + (uint32_t)((m0 + m) * sizeof(T)));
      v[m] = x.x;
      v[m + 1] = x.y;
    }
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m) v[m] = sh_ld<T>(p + (uint32_t)((m0 + m) * sizeof(T)));
  }
}
__device__ __forceinline__ void rp_st2(uint32_t a, double x, double y) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ void rp_st2(uint32_t a, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}
template <typename T, int MO>
__device__ __forceinline__ void rp_st(uint32_t p, int m0, int n, const T (&v)[MO]) {
  if constexpr (MO % 2 == 0) {
#pragma unroll
    for (int m = 0; m < n; m += 2)
      rp_st2(p + (uint32_t)((m0 + m) * sizeof(T)), v[m0 + m], v[m0 + m + 1]);
  } else {
#pragma unroll
    for (int m = 0; m < n; ++m) sh_st(p + (uint32_t)((m0 + m) * sizeof(T)), v[m0 + m]);
  }
}
// sweep_quot's two halves: the refined reciprocal, and the quotient from it
__device__ __forceinline__ double rp_recip(double den) {
  const double r0 = rcp_approx(den);
  return __fma_rn(r0, __fma_rn(-den, r0, 1.0), r0);
}
__device__ __forceinline__ double rp_quot(double num, double den, double r1) {
  const double q0 = num * r1;
  return __fma_rn(r1, __fma_rn(-den, q0, num), q0);
}
__device__ __forceinline__ float rp_recip(float) { return 0.0f; }
__device__ __forceinline__ float rp_quot(float num, float den, float) { return __fdividef(num, den); }

template <typename T, int MO, bool PAIR>
__global__ void __launch_bounds__(32 * RpShape<MO>::MAXW, 1)
    k_dom_octant_rp(GridDev g, const __grid_constant__ RpArgs<T, MO> a) {
  using T2 = typename Vec2Of<T>::type;
  using PT = RpPoints<MO>;
  constexpr int RK = RpShape<MO>::RK;
  constexpr int MOW = rp_pad((int)sizeof(T), MO);
  constexpr uint32_t TS = (uint32_t)sizeof(T), PS = MO * TS;
  extern __shared__ __align__(16) unsigned char shraw[];
  if (a.done && *(volatile const int*)a.done) return;
  cg::cluster_group cl = cg::this_cluster();
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int C = a.C, rows = a.rows, pitch = a.pitch;
  const int rank = (int)cl.block_rank();
  const int oct = blockIdx.x / C;
  const bool fx = a.fx[oct] != 0, fy = a.fy[oct] != 0, fz = a.fz[oct] != 0;
  const int zm = a.zs - 1, zlog = 31 - __clz(a.zs);
  const RpLayout L = rp_layout((int)sizeof(T), MO, rows, ny, a.zs);
  unsigned long long* bars = (unsigned long long*)(shraw + L.bars);
  const uint32_t full_k = smem_u32(bars), full_z = full_k + 8u * RP_KS,
                 empty_z = full_z + 8u * RP_ZS_MAX;
  volatile int* const gave_up = (volatile int*)(bars + RP_KS + 2 * RP_ZS_MAX);
  T* igr = (T*)(shraw + L.ig);
  T2* tz = (T2*)(shraw + L.tz);
  const int S = nx + ny - 1;
  const int r0 = rank * rows;
  const int nrows = min(rows, nz - r0);
  const int steps = S + nrows - 1;
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  const int nwj = (ny + 31) / 32, nw = (int)blockDim.x / 32;
  const int rb = warp / nwj, jb = warp - rb * nwj;
  const uint32_t row_bytes = (uint32_t)L.rowb, fill_bytes = (uint32_t)ny * PS;
  const bool ground_in = rank == 0 && fz;  // the ground's intensity flows in
  for (int q = threadIdx.x; q < nrows * MO; q += blockDim.x) {
    const int r = q / MO, m = q - r * MO;
    const int kp = r0 + r, k = fz ? kp : nz - 1 - kp;
    const double axd = fabs(a.ox[m]) / g.dx, ayd = fabs(a.oy[m]) / g.dy;
    const double azd = fabs(a.oz[m]) / g.dz[k];
    T2 v;
    v.x = (T)azd;
    v.y = (T)(axd + ayd + azd);
    tz[q] = v;
  }
  // full_k: the inputs of a step (one arrival for each of their arrays); full_z:
  // the row handed on to this CTA; empty_z: the next CTA's first row block has
  // read what this CTA sent into its ring
  if (threadIdx.x == 0) {
    gave_up[0] = steps;
    gave_up[1] = S;
    for (int q = 0; q < RP_KS; ++q) cl_mbar_init(bars + q, 3u);
    for (int q = 0; q < RP_ZS_MAX; ++q) {
      cl_mbar_init(bars + RP_KS + q, 1u);
      cl_mbar_init(bars + RP_KS + RP_ZS_MAX + q, (unsigned)nwj);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (rank > 0)
      for (int q = 0; q < min(a.zs, S); ++q) cl_arrive_expect(full_z + 8u * q, fill_bytes);
  }
  __syncthreads();
  cluster_arrive_release();
  cluster_wait_acquire();

  const uint32_t a_xb = smem_u32(shraw + L.xb), a_spare = smem_u32(shraw + L.spare);
  const uint32_t a_zin = smem_u32(shraw + L.zin), a_yin = smem_u32(shraw + L.yin);
  const uint32_t a_kab = smem_u32(shraw + L.kab), kstep = (uint32_t)(rows * pitch) * 2 * TS;
  // The inputs of a step into slot t % RP_KS, an array each by the first lanes of
  // a warp in the middle of the CTA: all rows of a plane are one run (k ascends
  // in memory), planes are step bytes apart, a step past last brings nothing.
  // Every one of these lanes waits for the inputs itself, so what it may announce
  // next is its own knowledge; in lanes of one warp that costs a single wait (in
  // one lane of three warps each, with a word in shared memory to tell the others
  // of a wait that gave up: 119 us a sweep at 97 x 41 x 23, S4, against 110).
  const int P = nx + ny + nz - 2, Pw = nx + nz - 1;
  const bool loads = warp == (nw / (2 * nwj)) * nwj + (nwj > 2 ? 1 : 0) && lane < 3;
  struct Load {
    const char* src;
    int64_t step;
    uint32_t dst, size, slot;
    int last;
  } ld = {};
  if (loads && lane == 0) {
    const int64_t plane = (int64_t)nz * pitch * 2 * TS;
    ld = Load{(const char*)a.kb[rp_class(fx, fy, fz)] + (fx ? r0 : P - 1 - r0) * plane +
                  (int64_t)(fz ? r0 : nz - r0 - nrows) * pitch * 2 * TS,
              fx ? plane : -plane, a_kab, (uint32_t)(nrows * pitch) * 2 * TS, kstep, steps};
  } else if (loads && lane == 1) {
    const int64_t plane = (int64_t)nz * MOW * TS;
    ld = Load{(const char*)a.wrap + ((int64_t)oct * Pw + r0) * plane + (int64_t)r0 * MOW * TS,
              plane, a_yin, (uint32_t)(nrows * MOW) * TS, (uint32_t)(rows * MOW) * TS,
              min(steps, Pw - r0)};
  } else if (loads) {
    const int64_t plane = (int64_t)pitch * TS;
    ld = Load{(const char*)(fx == fy ? a.igA : a.igB) + (fx ? 0 : S - 1) * plane,
              fx ? plane : -plane, smem_u32(igr), (uint32_t)plane, (uint32_t)plane,
              ground_in ? min(steps, S) : 0};
  }
  auto load = [&](int t) {
    const int sl = t & (RP_KS - 1);
    const uint32_t bar = full_k + 8u * sl;
    const bool on = t < ld.last;
    cl_arrive_expect(bar, on ? ld.size : 0u);
    if (on) rp_bulk_in(ld.dst + (uint32_t)sl * ld.slot, ld.src + t * ld.step, ld.size, bar);
  };
  if (loads)
    for (int t = 0; t < min(RP_KS, steps); ++t) load(t);
  // the row hand-off: the last row block's warps send, the first one's release
  const int row0 = rb * RK;
  const bool sends = rank < C - 1 && row0 + RK >= rows && row0 < rows;
  const bool takes = rank > 0 && rb == 0;
  // lanes past the last column double it, value for value
  const int j = min(jb * 32 + lane, ny - 1), jk = fy ? j : ny - 1 - j;
  const uint32_t dn_zin =
      sends ? cl_mapa(a_zin, (unsigned)(rank + 1)) + (uint32_t)j * PS : 0u;
  const uint32_t dn_full = sends ? cl_mapa(full_z, (unsigned)(rank + 1)) : 0u;
  const uint32_t up_empty = takes ? cl_mapa(empty_z, (unsigned)(rank - 1)) : 0u;
  const bool own = jb * 32 + lane < ny;  // a doubling lane sends nothing
  unsigned failed = 0;  // RP_RING, RP_IN: this thread's wait gave up
  const T I_amb = (T)a.I_amb;
  T I[RK][MO];
#pragma unroll
  for (int r = 0; r < RK; ++r)
#pragma unroll
    for (int m = 0; m < MO; ++m) I[r][m] = I_amb;
  // steps in which some pencil of the warp has a cell, and the step from which
  // all have begun
  const int t_lo = row0 + jb * 32;
  const int t_hi = row0 < nrows
                       ? min(row0 + RK, nrows) - 1 + min(ny - 1, jb * 32 + 31) + nx - 1 : -1;
  const int t_all = row0 + RK - 1 + jb * 32 + 31;
  // this thread's place in each row's buffers of this step and the last one
  // (they swap); a patch row that does not exist has a spare place
  uint32_t cur[RK], prv[RK], swp[RK], koff[RK];
  int lim[RK];  // nx, or 0 for a pencil that does not exist
  T* Gp[RK];
  const uint32_t half = (uint32_t)rows * row_bytes;
#pragma unroll
  for (int r = 0; r < RK; ++r) {
    const bool has = row0 + r < nrows;
    const int row = min(row0 + r, nrows - 1);
    cur[r] = has ? a_xb + (uint32_t)row * row_bytes + (uint32_t)j * PS : a_spare + PS;
    prv[r] = has ? cur[r] + half : cur[r];
    swp[r] = cur[r] ^ prv[r];
    koff[r] = a_kab + (uint32_t)((fz ? row : nrows - 1 - row) * pitch + jk) * 2 * TS;
    lim[r] = has ? nx : 0;
    // its partial of G at step 0 (a pointer that steps with t; used only where
    // the pencil has a cell)
    Gp[r] = a.Goct + (((int64_t)oct * nz + r0 + row) * S - row) * pitch + j;
  }
  // z-inflow of the first row: the row below, or the ring
  uint32_t zprv = a_xb + (uint32_t)max(row0 - 1, 0) * row_bytes + (uint32_t)j * PS + half;
  const uint32_t zswp = zprv ^ (zprv - half), zring = a_zin + (uint32_t)j * PS;
  const uint32_t yoff = a_yin + (uint32_t)(min(row0, nrows - 1) * MOW) * TS;
  const int slot = a.slot[oct];
  const bool ground_row = slot >= 0 && r0 + nrows == nz && row0 + RK >= nrows && row0 < nrows;
  const bool last_col = jb == nwj - 1;
  // every level of the CTA is dz0 high: az and as are launch constants
  bool uni = true;
  for (int r = 0; r < nrows; ++r) uni = uni && g.dz[fz ? r0 + r : nz - 1 - (r0 + r)] == a.dz0;
  auto march = [&](auto tab) {
    constexpr bool TAB = decltype(tab)::value;
    T cx[PT::NL], cy[PT::NL], cz[PT::NL], cw[PT::NW], cs[MO];
#pragma unroll
    for (int q = 0; q < PT::NL; ++q) {
      cx[q] = a.ax[q];
      cy[q] = PAIR ? cx[q] : a.ay[q];
      if (!TAB) cz[q] = a.az[q];
    }
#pragma unroll
    for (int q = 0; q < PT::NW; ++q) cw[q] = a.w[q];
#pragma unroll
    for (int m = 0; m < MO; ++m)
      if (!TAB)
        cs[m] = PAIR && rp_digit(PT::PAIR, m) != m ? cs[rp_digit(PT::PAIR, m)] : a.as[m];
    int ip = -row0 - j;  // the first row's cell at step t
    uint32_t zslot = 0, kslot = 0, yslot = 0;  // slot offsets of the rings
    for (int t = 0; t < steps; ++t, ++ip) {
      // the inputs of step t are there (one warp waits; the barrier passes it on)
      if (loads && !rp_wait(full_k + 8u * (t & (RP_KS - 1)), (uint32_t)((t / RP_KS) & 1), failed,
                            RP_IN, a.err))
        gave_up[0] = t;
      __syncthreads();  // step t - 1 complete in this CTA
      if (loads && t > 0 && t - 1 + RP_KS < steps && !(failed & RP_IN)) load(t - 1 + RP_KS);
      const int q = t - (rows - 1);  // the item that this step hands on
      if (sends && q > zm && q < S)  // its slot in the next CTA is free again
        rp_wait(empty_z + 8u * (q & zm), (uint32_t)(((q >> zlog) - 1) & 1), failed, RP_RING, a.err);
      if (takes && t < S) {
        if (!rp_wait(full_z + 8u * (t & zm), (uint32_t)((t >> zlog) & 1), failed, RP_RING, a.err) &&
            threadIdx.x == 0)
          gave_up[1] = t;
        if (jb == 0 && lane == 0 && !(failed & RP_RING) && t + zm + 1 < S)
          cl_arrive_expect(full_z + 8u * (t & zm), fill_bytes);
      }
      if (t >= t_lo && t <= t_hi) {
        const uint32_t az = row0 > 0 ? zprv : zring + zslot;
        uint32_t ay[RK];
        T2 k2[RK];
        T gs[RK], rc[RK][MO];
#pragma unroll
        for (int r = 0; r < RK; ++r) {
          // y-inflow: the pencil to the left, in the first column the values
          // that the sweep before left at the row's other end
          ay[r] = prv[r] - PS;
          k2[r] = sh_ld2<T2>(koff[r] + kslot);
          gs[r] = (T)0;
        }
        if (j == 0) {
#pragma unroll
          for (int r = 0; r < RK; ++r)
            ay[r] = yoff + yslot + (uint32_t)(min(r, nrows - 1 - row0) * MOW) * TS;
        }
        if (row0 == 0 && rank == 0) {
          // no row below: the ground's (the ambient) intensity for every
          // ordinate, into this column's place in the ring
          const T zg = fz ? igr[(t & (RP_KS - 1)) * pitch + jk] : I_amb;
          T z[MO];
#pragma unroll
          for (int m = 0; m < MO; ++m) z[m] = zg;
          rp_st<T, MO>(az, 0, MO, z);
        }
        // the batches: all loads of one before its updates, its stores after
        // the loads of the next
        constexpr int N0 = MO > 6 ? 6 : MO, N1 = MO - N0;
        T Iy0[RK][N0], Iz0[N0];
#pragma unroll
        for (int r = 0; r < RK; ++r) rp_ld<T, MO>(ay[r], 0, Iy0[r]);
        rp_ld<T, MO>(az, 0, Iz0);
        auto update = [&](int r, int m, T Iy, T Iz) {
          T zc, as;
          if constexpr (TAB) {
            const T2 z = tz[min(row0 + r, nrows - 1) * MO + m];
            zc = z.x;
            as = z.y;
          } else {
            zc = cz[rp_digit(PT::Z, m)];
            as = cs[m];
          }
          const T den = k2[r].x + as;
          const bool share = PAIR && rp_digit(PT::PAIR, m) != m;
          rc[r][m] = share ? rc[r][rp_digit(PT::PAIR, m)] : rp_recip(den);
          const T num = fmat(zc, Iz, fmat(cy[rp_digit(PT::Y, m)], Iy,
                                          fmat(cx[rp_digit(PT::X, m)], I[r][m], k2[r].y)));
          I[r][m] = rp_quot(num, den, rc[r][m]);
          gs[r] = fmat(cw[rp_digit(PT::W, m)], I[r][m], gs[r]);
        };
        // from the far row, so that the row below still holds its value of the
        // step before
#pragma unroll
        for (int m = 0; m < N0; ++m)
#pragma unroll
          for (int r = RK - 1; r >= 0; --r)
            update(r, m, Iy0[r][m], r > 0 ? I[r > 0 ? r - 1 : 0][m] : Iz0[m]);
        if constexpr (N1 > 0) {
          T Iy1[RK][N1], Iz1[N1];
#pragma unroll
          for (int r = 0; r < RK; ++r) rp_ld<T, MO>(ay[r], N0, Iy1[r]);
          rp_ld<T, MO>(az, N0, Iz1);
#pragma unroll
          for (int r = 0; r < RK; ++r) rp_st<T, MO>(cur[r], 0, N0, I[r]);
#pragma unroll
          for (int m = 0; m < N1; ++m)
#pragma unroll
            for (int r = RK - 1; r >= 0; --r)
              update(r, N0 + m, Iy1[r][m], r > 0 ? I[r > 0 ? r - 1 : 0][N0 + m] : Iz1[m]);
#pragma unroll
          for (int r = 0; r < RK; ++r) rp_st<T, MO>(cur[r], N0, N1, I[r]);
        } else {
#pragma unroll
          for (int r = 0; r < RK; ++r) rp_st<T, MO>(cur[r], 0, N0, I[r]);
        }
        bool act[RK];
#pragma unroll
        for (int r = 0; r < RK; ++r) {
          act[r] = (unsigned)(ip - r) < (unsigned)lim[r];
          if (act[r]) *Gp[r] = gs[r];
        }
        if (ground_row) {
#pragma unroll
          for (int r = 0; r < RK; ++r) {
            const int row = row0 + r;
            if (act[r] && row == nrows - 1) {
              T qs = (T)0;
#pragma unroll
              for (int m = 0; m < MO; ++m) qs = fmat(a.wq[m], I[r][m], qs);
              a.Qoct[((int64_t)slot * S + t - row) * pitch + j] = qs;
            }
          }
        }
        if (last_col) {
          // the y-outflow, read by the next sweep at the row's other end
#pragma unroll
          for (int r = 0; r < RK; ++r)
            if (j == ny - 1 && own && act[r]) {
              const int row = row0 + r;
              T* wo = a.wrap + (((int64_t)oct * Pw + ip - r + r0 + row) * nz + r0 + row) * MOW;
              if constexpr (MO % 2 == 0) {
#pragma unroll
                for (int m = 0; m < MO; m += 2) {
                  T2 v;
                  v.x = I[r][m];
                  v.y = I[r][m + 1];
                  *reinterpret_cast<T2*>(wo + m) = v;
                }
              } else {
#pragma unroll
                for (int m = 0; m < MO; ++m) wo[m] = I[r][m];
              }
            }
        }
        if (t < t_all) {
          // a pencil that has not begun: its first x-inflow is the ambient one
#pragma unroll
          for (int r = 0; r < RK; ++r)
            if (ip - r < 0) {
#pragma unroll
              for (int m = 0; m < MO; ++m) I[r][m] = I_amb;
            }
        }
      }
#pragma unroll
      for (int r = 0; r < RK; ++r) {
        Gp[r] += pitch;
        cur[r] ^= swp[r];
        prv[r] ^= swp[r];
      }
      zprv ^= zswp;
      const bool kwrap = ((t + 1) & (RP_KS - 1)) == 0;
      kslot = kwrap ? 0u : kslot + kstep;
      yslot = kwrap ? 0u : yslot + (uint32_t)(rows * MOW) * TS;
      zslot = ((t + 1) & zm) == 0 ? 0u : zslot + row_bytes;
      if (sends && q >= 0 && q < S && own && !(failed & RP_RING) &&
          !(rank == 0 && q == a.withhold)) {
        const uint32_t dst = dn_zin + (uint32_t)(q & zm) * row_bytes;
        const uint32_t bar = dn_full + 8u * (q & zm);
#pragma unroll
        for (int r = 0; r < RK; ++r)
          if (row0 + r == rows - 1) rp_send<T, MO>(dst, bar, I[r]);
      }
      if (takes && t < S) {
        __syncwarp();
        if (lane == 0 && !(failed & RP_RING)) rp_release(up_empty + 8u * (t & zm));
      }
    }
  };
  if (uni) march(std::false_type{});
  else march(std::true_type{});
  // no CTA leaves while another may still signal its barriers or write its ring
  cluster_arrive_release();
  cluster_wait_acquire();
  // Nobody sends or loads any more.  Where a wait gave up, copies and rows that
  // were announced may still be on their way into this CTA: they land before it
  // leaves (those that were never sent run into the limit).
  int rounds = RP_DRAIN_LIMIT;
  auto drain = [&](uint32_t bar, uint32_t parity) {
    while (rounds > 0 && !rp_poll(bar, parity, 1)) --rounds;
  };
  if (loads) {
    const int t0 = gave_up[0];
    for (int t = t0; t < min(steps, max(t0 - 1, 0) + RP_KS); ++t)
      drain(full_k + 8u * (t & (RP_KS - 1)), (uint32_t)((t / RP_KS) & 1));
  }
  if (threadIdx.x == 0 && rank > 0) {
    for (int t = gave_up[1]; t < min(S, gave_up[1] + a.zs); ++t)
      drain(full_z + 8u * (t & zm), (uint32_t)((t >> zlog) & 1));
  }
}

// ---- the arrays in skewed layout ------------------------------------------------
#define RP_T 32
#define RP_TP 34  // tile stride: rows, and both diagonals (33, 35), free of bank conflicts
// Tile of RP_T x RP_T cells of one level in the skewed layouts.  A pass u takes
// one cell of every tile row jj (the lane): column u - jj (type A, i + j) or
// u + jj (type B, i - j), modulo the tile, so the lanes lie on two skewed rows,
// a run of each.
__device__ __forceinline__ int rp_col(bool A, int u, int jj) {
  return (A ? u - jj : u + jj) & (RP_T - 1);
}

// Absorption and emission as k_dom_setup's, with (kappa, kappa B) in the four
// orientations' hyperplane order; a block owns a 32 x 32 tile of one level and
// turns it in shared memory, so both sides are runs.
template <typename T2>
struct RpKb {
  T2* kb[4];
};
template <typename T>
__global__ void __launch_bounds__(256)
    k_dom_setup_skew(GridDev g, DomSetupArgs s, double* ks, double* kg, double* ksafe, double* B,
                     RpKb<typename Vec2Of<T>::type> o, int pitch) {
  using T2 = typename Vec2Of<T>::type;
  __shared__ T2 tile[RP_T][RP_TP];
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int i0 = blockIdx.x * RP_T, j0 = blockIdx.y * RP_T, k = blockIdx.z;
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  for (int jj = wy; jj < RP_T; jj += 8) {
    const int i = i0 + lane, j = j0 + jj;
    if (i < nx && j < ny) {
      const int64_t c = cidx(g, k, j, i);
      double ksf, Bc;
      dom_setup_cell(s, c, ks, kg, ksafe, B, ksf, Bc);
      T2 v;
      v.x = (T)ksf;
      v.y = (T)(ksf * Bc);
      tile[jj][lane] = v;
    }
  }
  __syncthreads();
  const int j = j0 + lane;
  for (int u = wy; u < RP_T; u += 8) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool A = (q & 1) == 0;
      const int x = rp_col(A, u, lane), i = i0 + x;
      if (i < nx && j < ny) {
        const int p = i + (A ? j : ny - 1 - j) + ((q & 2) == 0 ? k : nz - 1 - k);
        o.kb[q][((int64_t)p * nz + k) * pitch + j] = tile[lane][x];
      }
    }
  }
}

// The octant signs for the reduction over skewed partials.
struct RpOct {
  unsigned char fx[8], fy[8], fz[8];
  signed char slot[8];
};

// G = sum over the octants in octant order, max G and max |G - G_prev|.  A
// thread has all its loads (RP_TQ cells of eight octants) in flight before it
// adds any; runs of octants of one skew type then pass through the tile in
// turn.  400 x 120 x 60, FP64: 55 us (230 MB read, 23 written: 4.6 TB/s); with
// two octants at a time and one skewed row a pass, half of its lanes idle, 100.
#define RP_GW 16  // warps of a block
#define RP_TQ (RP_T / RP_GW)
template <typename T>
__global__ void __launch_bounds__(32 * RP_GW, 2)
    k_dom_G_skew(GridDev g, const __grid_constant__ RpOct o8, const T* __restrict__ Goct, int pitch,
                 double* G, const double* __restrict__ Gp, unsigned long long* keys,
                 const int* done) {
  if (done && *done) return;
  __shared__ double tile[RP_T][RP_TP];
  const int nx = g.nx, ny = g.ny, nz = g.nz, S = nx + ny - 1;
  const int i0 = blockIdx.x * RP_T, j0 = blockIdx.y * RP_T, k = blockIdx.z;
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int j = j0 + lane;
  T v[8][RP_TQ];
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const bool fx = o8.fx[o] != 0, fy = o8.fy[o] != 0;
    const int jp = fy ? j : ny - 1 - j, kp = o8.fz[o] ? k : nz - 1 - k;
    const T* src = Goct + ((int64_t)o * nz + kp) * S * pitch + jp;
#pragma unroll
    for (int q = 0; q < RP_TQ; ++q) {
      const int i = i0 + rp_col(fx == fy, wy + RP_GW * q, lane);
      v[o][q] = i < nx && j < ny ? src[((fx ? i : nx - 1 - i) + jp) * pitch] : (T)0;
    }
  }
  double s[RP_TQ], gp[RP_TQ];
#pragma unroll
  for (int q = 0; q < RP_TQ; ++q) {
    const int i = i0 + lane, jc = j0 + wy + RP_GW * q;
    s[q] = 0.0;
    gp[q] = i < nx && jc < ny ? Gp[cidx(g, k, jc, i)] : 0.0;
  }
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const bool A = o8.fx[o] == o8.fy[o];
    if (o > 0 && A != (o8.fx[o - 1] == o8.fy[o - 1])) {
      // the other skew type's threads go on with the sums so far
#pragma unroll
      for (int q = 0; q < RP_TQ; ++q) tile[lane][rp_col(!A, wy + RP_GW * q, lane)] = s[q];
      __syncthreads();
#pragma unroll
      for (int q = 0; q < RP_TQ; ++q) s[q] = tile[lane][rp_col(A, wy + RP_GW * q, lane)];
      __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < RP_TQ; ++q) s[q] += (double)v[o][q];
  }
  {
    const bool A = o8.fx[7] == o8.fy[7];
#pragma unroll
    for (int q = 0; q < RP_TQ; ++q) tile[lane][rp_col(A, wy + RP_GW * q, lane)] = s[q];
    __syncthreads();
  }
  unsigned long long bg = 0, bd = 0;
#pragma unroll
  for (int q = 0; q < RP_TQ; ++q) {
    const int i = i0 + lane, jj = wy + RP_GW * q;
    if (i < nx && j0 + jj < ny) {
      const double t = tile[jj][lane];
      G[cidx(g, k, j0 + jj, i)] = t;
      dom_G_keys(t, gp[q], bg, bd);
    }
  }
  // one pair of atomics a block: with one a warp, the 25,000 warps of the
  // workload's grid queued at the two addresses for longer than the sums take
  __shared__ unsigned long long best[2];
  if (threadIdx.x < 2) best[threadIdx.x] = 0;
  __syncthreads();
  dom_G_max(bg, bd, best);
  __syncthreads();
  if (threadIdx.x < 2) atomicMax(keys + threadIdx.x, best[threadIdx.x]);
}

// the y-inflow rows in the kernel's order, [octant][i' + k'][k'][MOW], from and
// to the M x Nz x Nx form
template <typename A, typename B>
__global__ void k_dom_wrap_copy(GridDev g, RpOct o8, int M, int Mo, int MOW,
                                const A* __restrict__ src, B* dst, int to_rows) {
  const int64_t tot = (int64_t)M * g.nz * g.nx;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= tot) return;
  const int n = (int)(t / ((int64_t)g.nz * g.nx));
  const int r = (int)(t - (int64_t)n * g.nz * g.nx);
  const int k = r / g.nx, i = r - k * g.nx;
  const int o = n / Mo, m = n - o * Mo;
  const int ip = o8.fx[o] ? i : g.nx - 1 - i, kp = o8.fz[o] ? k : g.nz - 1 - k;
  const int64_t q = (((int64_t)o * (g.nx + g.nz - 1) + ip + kp) * g.nz + kp) * MOW + m;
  if (to_rows) dst[q] = (B)src[t];
  else dst[t] = (B)src[q];
}

// ground exchange from the skewed partial fluxes; the new ground intensity in
// the natural order and in both skewed layouts (nslots = 0: the solve's start)
template <typename T>
__global__ void k_dom_ground_skew(GridDev g, RpOct o8, int start, const T* __restrict__ Qoct,
                                  int pitch, const double* __restrict__ Isoil, double refl,
                                  double relax, double* Ig, double* qin, T* igA, T* igB,
                                  const int* done) {
  if (done && *done) return;
  const int nx = g.nx, ny = g.ny, S = nx + ny - 1;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nx * ny) return;
  const int j = q / nx, i = q - j * nx;
  double v;
  if (start) {
    v = Ig[q];
  } else {
    double s = 0.0;
    for (int o = 0; o < 8; ++o) {
      if (o8.slot[o] < 0) continue;
      const int ip = o8.fx[o] ? i : nx - 1 - i, jp = o8.fy[o] ? j : ny - 1 - j;
      s += (double)Qoct[((int64_t)o8.slot[o] * S + ip + jp) * pitch + jp];
    }
    qin[q] = s;
    const double Inew = Isoil[q] + refl * s;
    v = relax * Inew + (1.0 - relax) * Ig[q];
    Ig[q] = v;
  }
  igA[(int64_t)(i + j) * pitch + j] = (T)v;
  igB[(int64_t)(i - j + ny - 1) * pitch + j] = (T)v;
}

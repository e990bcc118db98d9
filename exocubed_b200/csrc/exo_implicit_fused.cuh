// exo_implicit_fused.cuh -- the mixed build's 5x5 solve in FP64 blocks with its
// back substitution in the same kernel (textually part of exo_kernels.cuh).
//
// The same algorithm as implicit_column and kb_implicit_bwd in one kernel.  The
// split form is faster (6x24^2x32 109 us a solve against 123, 6x96^2x64 761
// against 785, 6x192^2x96 4017 against 4166, with 128 columns a block 4025
// against 3861; with the blocks kept by their structure 617 at 6x96^2x64);
// but compiled with fused multiply-adds it does not round as this one does:
// the last bits of u it changes reach the FP32 copy of the primitives, and a
// run differs by 1e-7 within some tens of steps.  (The boundary terms as
// branches change the roundings too.)  FP32 blocks, the 3x3 blocks and the FP64 build, whose
// results the split form leaves to the bit, take the split form.
//
// What bounds it: dependent FP64 operations at eight to nine warps per SM, on
// large grids the scratch's traffic (480 of 640 bytes a level and column,
// 2.1 ms at the copy rate at 6x192^2x96), and the L1 beside the blocks' shared
// memory, whose lines hold the columns' strided loads in flight (fused_tiles).
// More warps do not help (200 registers, ten warps: the same; 168: twice the
// time, the lines of L1 in flight being what limits them).

// Solve with the LU factors of implicit_column's mixed build (rows taken in
// the order 1, 4, 2, 3, 0, threshold row swaps packed 3 bits per step): y
// holds the right-hand side with its rows in natural order on entry and the
// solution, unknowns in order, on exit.
template <class R>
__device__ __forceinline__ void lu_solve_swapped(const R (&t)[5][5], const R (&idg)[5],
                                              unsigned perm, bool swapped, R* y) {
  constexpr int O[5] = {1, 4, 2, 3, 0};
  if (swapped) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned pk = (perm >> (3 * k)) & 7u;
#pragma unroll
      for (int r = k + 1; r < 5; ++r) {
        const bool sw = (pk == (unsigned)r);
        const R a = y[O[k]], b = y[O[r]];
        y[O[k]] = sw ? b : a;
        y[O[r]] = sw ? a : b;
      }
    }
  }
#pragma unroll
  for (int r = 1; r < 5; ++r)
#pragma unroll
    for (int k = 0; k < r; ++k) y[O[r]] -= t[O[r]][k] * y[O[k]];
  R z[5];
#pragma unroll
  for (int r = 4; r >= 0; --r) {
    R acc = y[O[r]];
#pragma unroll
    for (int q = r + 1; q < 5; ++q) acc -= t[O[r]][q] * z[q];
    z[r] = acc * idg[r];
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) y[r] = z[r];
}

// The back substitution of the stepping kernel's FP64 blocks (mixed build)
// with the state u moved through shared memory by the warp: the warp's 32
// columns go down BWD_TL levels at a time; each lane copies four levels of
// a column for one variable in one 32-byte run (the per-lane accesses of
// one level are 816 bytes apart, a sector each), the next chunk's copies in
// flight while a chunk is corrected.  The factors are read per lane, one
// level ahead (they are contiguous across the warp).  io.live: the lanes of
// the warp with a column.  wtile: 2 x 5 x 32 x (BWD_TL + 1) doubles of shared
// memory for the warp alone.
constexpr int BWD_TL = 4;
// the two u tiles of a warp's back substitution (5 variables x 32 columns x
// BWD_TL levels, padded)
constexpr int WARP_TILE_DOUBLES = 2 * 5 * 32 * (BWD_TL + 1);
// a warp's shared memory: the inputs (a level tile, or w and du of the next
// level), then two face matrices (entry e of lane l at [e * 32 + l])
template <bool kTile>
__host__ __device__ constexpr int fused_input_doubles() {
  return kTile ? LEVEL_TILE_DOUBLES : 10 * 32;
}
template <bool kTile>
__host__ __device__ constexpr int fused_warp_doubles() {
  return fused_input_doubles<kTile>() + 50 * 32;
}
static_assert(fused_warp_doubles<false>() >= WARP_TILE_DOUBLES,
              "the tiled back substitution's buffers fit in the warp's memory");
template <class IO>
__device__ __forceinline__ void implicit_backward_tiled(IO& io, int is, int ie,
                                                        typename IO::Real* dp, double* wtile) {
  static_assert(BWD_TL == 4, "the lane -> (column, level) split below assumes 4 levels");
  constexpr int NB = 5;
  constexpr int NF = NB * NB + NB;  // factors per level: (A c)_i and delta_i
  constexpr int TS = BWD_TL + 1;
  constexpr int TW = 5 * 32 * TS;
  const unsigned live = io.live;
  const int lane = (int)(threadIdx.x & 31);
  __syncwarp(live);
  // lane copies level (lane & 3) of columns (lane >> 2) + 8 m, m = 0..3
  // (in a warp with a column in every lane)
  double* ub[4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
    ub[m] = reinterpret_cast<double*>(__shfl_sync(
        live, reinterpret_cast<unsigned long long>(io.xc), ((lane >> 2) + 8 * m) & 31));
  const int l = lane & 3;
  const int nch = (ie - is + BWD_TL) / BWD_TL;
  auto range = [&](int c, int& lo, int& hi) {
    hi = ie - c * BWD_TL;
    lo = max(is, hi - BWD_TL + 1);
  };
  // a warp with a column in every lane copies in 32-byte runs; the last warp
  // of a member may have fewer, and there each lane copies its own column
  const bool full = live == 0xffffffffu;
  auto load = [&](int c) {
    double* t = wtile + (c & 1) * TW;
    int lo, hi;
    range(c, lo, hi);
    if (full) {
      if (lo + l <= hi) {
#pragma unroll
        for (int e = 0; e < 20; ++e) {
          const int m = e & 3, n = e >> 2;
          cp_async8(&t[(n * 32 + (lane >> 2) + 8 * m) * TS + l], ub[m] + n * io.vs + lo + l);
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < 20; ++e) {
        const int ll = e & 3, n = e >> 2;
        if (lo + ll <= hi) cp_async8(&t[(n * 32 + lane) * TS + ll], io.xc + n * io.vs + lo + ll);
      }
    }
    cp_async_commit();
  };
  load(0);
  if (nch > 1) load(1);
  using R = typename IO::Real;
  // the factors of the next level, in flight while a level is corrected
  R cur_s[NF];
  if (ie > is) {
#pragma unroll
    for (int e = 0; e < NF; ++e) cur_s[e] = io.scr(ie - 1 - is, e);
  }
  for (int c = 0; c < nch; ++c) {
    if (c + 1 < nch) cp_async_wait_one();
    else cp_async_wait_all();
    __syncwarp(live);
    double* t = wtile + (c & 1) * TW;
    int lo, hi;
    range(c, lo, hi);
    for (int i = hi; i >= lo; --i) {
      if (i < ie) {
        R nxt_s[NF];
        const int ahead = i - 1;  // the level whose factors load now
        if (ahead >= is) {
#pragma unroll
          for (int e = 0; e < NF; ++e) nxt_s[e] = io.scr(ahead - is, e);
        }
        R dl[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) {
          R ad = cur_s[r * NB] * dp[0];
#pragma unroll
          for (int k = 1; k < NB; ++k) ad += cur_s[r * NB + k] * dp[k];
          dl[r] = cur_s[NB * NB + r] - ad;
        }
#pragma unroll
        for (int r = 0; r < NB; ++r) dp[r] = dl[r];
#pragma unroll
        for (int e = 0; e < NF; ++e) cur_s[e] = nxt_s[e];
      }
      // the corrected update of every variable
      double uu[5];
#pragma unroll
      for (int n = 0; n < 5; ++n) uu[n] = io.stage < 0 ? dp[n] : t[(n * 32 + lane) * TS + (i - lo)] + 1. * dp[n];
      if (io.stage == 2) airparcel_round_trip(uu, io.Rd, io.gamma);
#pragma unroll
      for (int n = 0; n < 5; ++n) t[(n * 32 + lane) * TS + (i - lo)] = uu[n];
    }
    __syncwarp(live);
    if (full) {
      if (lo + l <= hi) {
#pragma unroll
        for (int e = 0; e < 20; ++e) {
          const int m = e & 3, n = e >> 2;
          ub[m][n * io.vs + lo + l] = t[(n * 32 + (lane >> 2) + 8 * m) * TS + l];
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < 20; ++e) {
        const int ll = e & 3, n = e >> 2;
        if (lo + ll <= hi) io.xc[n * io.vs + lo + ll] = t[(n * 32 + lane) * TS + ll];
      }
    }
    __syncwarp(live);
    if (c + 2 < nch) load(c + 2);
  }
}

template <bool kTile, class IO>
__device__ __forceinline__ void implicit_column_fused(IO& io, typename IO::Real* sa, int ss, double* in,
                                                double cos_theta, double sin_theta, double d2,
                                                double d3, const double* x1f, const double* x1v,
                                                const double* dx1f, int is, int ie, double dt,
                                                double gamma, double grav, double* wt) {
  using R = typename IO::Real;
  using ColCell = exo::EXO_KNS::ColCell<R>;
  const double s = sin_theta;
  // gmm1 of every cell; the face average equals it
  const R gm1 = R((gamma - 1.) * 1. / 1.);
  const R gp = (gm1 + R(1)) / gm1;
  const R gam = R(gamma);
  const R grv = R(grav);
  // the reference's Dt = 1/dt, the same value every time
  const R rdt = R(1. / dt);
  auto cell = [&](const double* w) {
    ColCell c;
    c.rho = R(w[IDN]);
    c.v1 = R(w[IVX]);
    c.v2 = R(w[IVY] + w[IVZ] * cos_theta);
    c.v3 = R(w[IVZ] * sin_theta);
    c.p = R(w[IPR]);
    c.s2 = c.v1 * c.v1 + c.v2 * c.v2 + c.v3 * c.v3;
    if constexpr (sizeof(R) == 4) {
      c.isq = rsqrt_r(c.rho);
      c.sq = c.rho * c.isq;
      c.hr = gp * c.p * (c.isq * c.isq);
    } else {
      c.hr = gp * c.p * inv_r(c.rho);
    }
    return c;
  };
  auto AMs = [&](int slot, int r, int q) -> R& { return sa[(slot * 25 + r * 5 + q) * ss]; };

  // w(i+1) and du(i): with kTile four levels at a time by the whole warp (the
  // last warp of a member, where some lanes have no column, copies per lane),
  // else each lane its own, a level ahead
  LevelTile<IO, 5> lt(io, in, is, ie - is + 1);
  auto ready = [&](int k0) {
    if (io.live == 0xffffffffu) {
      lt.ready(io, k0);
    } else if ((k0 & 3) == 0) {
      __syncwarp(io.live);
      for (int k = k0; k < min(k0 + 4, ie - is + 1); ++k) {
#pragma unroll
        for (int n = 0; n < 5; ++n) {
          cp_async8(lt.place(n, k), io.wptr(is + 1 + k, n));
          cp_async8(lt.place(5 + n, k), io.duptr(is + k, n));
        }
      }
      cp_async_commit();
      cp_async_wait_all();
      __syncwarp(io.live);
    }
  };
  double* const next = in + (threadIdx.x & 31);
  auto prefetch = [&](int iw, int idu) {
#pragma unroll
    for (int n = 0; n < 5; ++n) cp_async8(next + n * 32, io.wptr(iw, n));
    if (idu >= 0) {
#pragma unroll
      for (int n = 0; n < 5; ++n) cp_async8(next + (5 + n) * 32, io.duptr(idu, n));
    }
    cp_async_commit();
  };
  double raw[5];
  io.w(is - 1, raw);
  ColCell cm = cell(raw);
  io.w(is, raw);
  ColCell c0 = cell(raw);
  if constexpr (!kTile) prefetch(is + 1, is);
  {
    R A[5][5];
    abs_jacobian(cm, c0, gm1, gam, A);
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int q = 0; q < 5; ++q) AMs(0, r, q) = A[r][q];
  }
  R Ap[5][5];
  R dp[5];  // delta_{i-1}
  int cur = 0;
  for (int i = is; i <= ie; ++i) {
    if constexpr (kTile) ready(i - is);
    else cp_async_wait_all();
    double rhs[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      raw[n] = kTile ? lt.get(n, i - is) : next[n * 32];
      rhs[n] = kTile ? lt.get(5 + n, i - is) : next[(5 + n) * 32];
    }
    ColCell cp = cell(raw);
    if constexpr (!kTile) prefetch(i + 2, i < ie ? i + 1 : -1);
    const int nxt = cur ^ 1;
    {
      R A[5][5];
      abs_jacobian(c0, cp, gm1, gam, A);
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int q = 0; q < 5; ++q) AMs(nxt, r, q) = A[r][q];
    }
    const double aleft = d2 * d3 * x1f[i] * x1f[i] * s;
    const double aright = d2 * d3 * x1f[i + 1] * x1f[i + 1] * s;
    const double vol = dx1f[i] * d2 * d3 * x1v[i] * x1v[i] * s;
    const double i2v = 0.5 / vol;
    const R bl = R(aleft * i2v), cr = R(aright * i2v), dd = R((aright - aleft) * i2v);
    const bool first = (i == is), last = (i == ie);
    R x[5];
    // rows of a, b (and c at the top boundary), then of t = a - b (A c)_{i-1},
    // written over row r of |A|(i-1/2) once that row has been read; and x
    unroll<5>([&](auto Row) {
      constexpr int r = decltype(Row)::value;
      R brow[5], trow[5];
      unroll<5>([&](auto Q) {
        constexpr int q = decltype(Q)::value;
        const R am = AMs(cur, r, q), ap = AMs(nxt, r, q);
        R a = am * bl + ap * cr;
        if constexpr (fj_nz(r, q)) a += dd * fj_entry<r, q>(c0, gm1);
        if constexpr (r == q) a += rdt;
        if constexpr ((r == IVX && q == IDN) || (r == IEN && q == IVX)) a -= grv;
        R bm = am;
        if constexpr (fj_nz(r, q)) bm += fj_entry<r, q>(cm, gm1);
        R b = -bm * bl;
        if (first) a += (q == IVX) ? -b : b;
        if (last) {
          R cmv = ap;
          if constexpr (fj_nz(r, q)) cmv -= fj_entry<r, q>(cp, gm1);
          R c = -cmv * cr;
          a += (q == IVX) ? -c : c;
        }
        brow[q] = b;
        trow[q] = a;
      });
      x[r] = R(rhs[r]) * rdt;
      if (!first) {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          R ba = brow[0] * Ap[0][q];
#pragma unroll
          for (int k = 1; k < 5; ++k) ba += brow[k] * Ap[k][q];
          trow[q] = trow[q] - ba;
        }
        R bd = brow[0] * dp[0];
#pragma unroll
        for (int k = 1; k < 5; ++k) bd += brow[k] * dp[k];
        x[r] = x[r] - bd;
      }
#pragma unroll
      for (int q = 0; q < 5; ++q) AMs(cur, r, q) = trow[q];
    });
    R t[5][5];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int q = 0; q < 5; ++q) t[r][q] = AMs(cur, r, q);
    // c_i column by column, from |A|(i+1/2) in shared memory and the upper cell
    auto ccol = [&](auto Q, R* c) {
      constexpr int q = decltype(Q)::value;
      unroll<5>([&](auto Row) {
        constexpr int r = decltype(Row)::value;
        R cmv = AMs(nxt, r, q);
        if constexpr (fj_nz(r, q)) cmv -= fj_entry<r, q>(cp, gm1);
        c[r] = -cmv * cr;
      });
    };
    // LU with the rows taken in the order 1, 4, 2, 3, 0 -- the order partial
    // pivoting ends with for nearly every block of this solve (density last,
    // energy and x1 momentum first) -- and threshold partial pivoting on top:
    // a row swap only where the diagonal falls below a tenth of the largest
    // entry of its column, so the swap code is skipped almost always.
    constexpr int O[5] = {1, 4, 2, 3, 0};
    unsigned perm = 0;  // 3 bits per step: the position swapped in
    bool swapped = false;
    R idg[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      if (k < 4) {
        const R dk = abs_r(t[O[k]][k]);
        R best = dk;
        int piv = k;
#pragma unroll
        for (int r = k + 1; r < 5; ++r) {
          const R m = abs_r(t[O[r]][k]);
          if (m > best) { best = m; piv = r; }
        }
        const bool take = dk < R(0.1) * best;
        if (!take) piv = k;
        perm |= (unsigned)piv << (3 * k);
        // the warp decides: as a lane's own branch the swaps become selects
        // that every level pays for
        if (__any_sync(io.live, take)) {
          swapped = true;
#pragma unroll
          for (int r = k + 1; r < 5; ++r) {
            const bool sw = (piv == r);
#pragma unroll
            for (int q = 0; q < 5; ++q) {
              const R a = t[O[k]][q], b = t[O[r]][q];
              t[O[k]][q] = sw ? b : a;
              t[O[r]][q] = sw ? a : b;
            }
          }
        }
      }
      idg[k] = inv_r(t[O[k]][k]);
#pragma unroll
      for (int r = k + 1; r < 5; ++r) {
        const R l = t[O[r]][k] * idg[k];
        t[O[r]][k] = l;
#pragma unroll
        for (int q = k + 1; q < 5; ++q) t[O[r]][q] -= l * t[O[k]][q];
      }
    }
    auto solve = [&](R* y) { lu_solve_swapped(t, idg, perm, swapped, y); };
    solve(x);
    unroll<5>([&](auto Q) {
      constexpr int q = decltype(Q)::value;
      R c[5];
      ccol(Q, c);
      solve(c);
#pragma unroll
      for (int r = 0; r < 5; ++r) Ap[r][q] = c[r];
    });
#pragma unroll
    for (int r = 0; r < 5; ++r) dp[r] = x[r];
    R* const sl = &io.scr(i - is, 0);
    if (!last) {
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int q = 0; q < 5; ++q) sl[(r * 5 + q) * 32] = Ap[r][q];
#pragma unroll
      for (int r = 0; r < 5; ++r) sl[(25 + r) * 32] = dp[r];
    }
    cm = c0;
    c0 = cp;
    cur = nxt;
  }
  // the warp's shared memory, free once every lane has finished its forward
  // sweep and its last copies (unused) have landed, holds the back
  // substitution's tiles
  if constexpr (!kTile) cp_async_wait_all();
  implicit_backward_tiled(io, is, ie, dp, wt);
}

// shared memory: fused_warp_doubles for each warp, then the radial tables
template <bool kTile>
constexpr size_t fused_smem(int threads, int nc1) {
  return ((size_t)fused_warp_doubles<kTile>() * (threads / 32) + 3 * (size_t)(nc1 + 1)) * sizeof(double);
}
// How the inputs come in.  A level tile reads each sector once but takes 23 KB
// a warp; per lane (15 KB) a sector is read four times, mostly from L2 (L1 hits
// 3 %).  An SM's shared memory goes up in steps, and what is left of 256 KB is
// L1, a line of which every load in flight holds: at the default 64 columns a block, four blocks with tiles leave 60 KB as
// long as they stay within the step of 196 KB (99 levels), past it 28 KB, too
// few lines for the copies in flight.  At 32 columns eight blocks with tiles
// leave 28 KB, nine without 60; at 128 two without leave 124 KB.  us a solve,
// tiles / per lane:
//   64 columns:   6x96^2x64 785 / 800, 96 levels 1168 / 1180, 99 1199 / 1230,
//                 100 1587 / 1235, 110 1720 / 1306, 6x192^2x96 4128 / 4055
//   32 columns:   6x96^2x64 998 / 805, 6x192^2x96 5600 / 4055
//   128 columns:  6x96^2x64 778 / 799, 6x192^2x96 4128 / 3838
// With three contexts' steps in turn on the GPU the tiles, which ask less of L1
// and L2, gain 5 % of a step at 6x96^2x64 (4450 against 4690 us) and 6x192^2x96
// (25650 against 26880), at 64 and at 128 columns; 128 is no default but an
// autotuner's choice for steps by themselves.  Grids of few blocks gain nothing
// from tiles even so (us a step, alone and in turn, tiles / per lane: 24 blocks,
// 6x16^2x90, 1173 / 1122 and 494 / 473; 54, 6x24^2x32, 496 / 468 and 266 / 264;
// but 85, 6x30^2x60, 1063 / 1034 and 596 / 628; 384, 6x64^2x33, 1320 / 1301 and
// 1169 / 1231): the line is a block for every second SM.  Tiles of
// two levels (18 KB a warp): 4416, 4004 and 3995 us a solve at 6x192^2x96 and
// 32, 64 and 128 columns.
constexpr bool fused_tiles(unsigned blocks, int threads, int nc1) {
  const size_t block = (fused_smem<true>(threads, nc1) + sizeof(DevView) + 127) / 128 * 128 + 1024;
  return threads == 64 && blocks > 148 / 2 && 4 * block <= 196 * 1024;
}

// A column of the stepping context: primitives and update from the state
// arrays, the corrected update added to u (with the AirParcel round trip on
// the last stage).
template <class R>
struct FusedColumnIO {
  using Real = R;
  const double* wc;
  const double* duc;
  double* xc;      // what is corrected: u, or for stage < 0 du
  size_t vs;       // stride between variables
  R* scr0;         // scratch of this column: [level][entry][32 lanes] per warp of columns
  int stage;       // < 0: write the corrected update into du, leave u alone
  double Rd, gamma;
  __device__ __forceinline__ void w(int i, double* out) const {
#pragma unroll
    for (int n = 0; n < 5; ++n) out[n] = wc[n * vs + i];
  }
  __device__ __forceinline__ size_t wstride() const { return vs; }
  __device__ __forceinline__ size_t dstride() const { return vs; }
  __device__ __forceinline__ const double* wptr(int i, int n) const { return wc + n * vs + i; }
  __device__ __forceinline__ const double* duptr(int i, int n) const { return duc + n * vs + i; }
  __device__ __forceinline__ R& scr(int lev, int e) const {
    return scr0[(lev * 30 + e) * 32];
  }
  unsigned live;   // the lanes of the warp with a column
};


template <class R, bool kTile>
__device__ __forceinline__ void implicit_fused_block(const DevView& v, unsigned blk, int stage,
                                               double dt_given = 0.) {
  extern __shared__ double ism[];
  const int ncol = 6 * v.N * v.N;
  const int col = (int)(blk * blockDim.x + threadIdx.x);
  // the radial geometry, read every level by every column, staged once per
  // block: kept out of L1, which the columns' strided loads churn each level
  const double* x1f;
  const double* x1v;
  const double* dx1f;
  stage_radial(ism + (blockDim.x >> 5) * fused_warp_doubles<kTile>(), v.nc1, v.x1f, v.x1v, v.dx1f, x1f, x1v, dx1f);
  const unsigned live = __ballot_sync(0xffffffffu, col < ncol);
  if (col >= ncol) return;
  const int j = v.js + col % v.N;
  const int k = v.ks + (col / v.N) % v.N;
  const int p = col / (v.N * v.N);
  const double dt = stage < 0 ? dt_given : rk_beta(stage) * v.sc->dt;
  const size_t base = idx(v, p, 0, k, j, 0);
  // scratch in blocks of 32 columns: a warp's 32 entries are 128 (FP32) or
  // 256 (FP64) contiguous bytes
  R* scr0 = reinterpret_cast<R*>(v.scratch) + (size_t)(col >> 5) * v.L * 30 * 32 + (col & 31);
  FusedColumnIO<R> io{v.w + base, v.du + base, (stage < 0 ? v.du : v.u) + base, v.cells, scr0,
                      stage,       v.Rd,        v.gamma,                          live};
  double* const wt = ism + (threadIdx.x >> 5) * fused_warp_doubles<kTile>();
  implicit_column_fused<kTile>(io, wt + fused_input_doubles<kTile>() + (threadIdx.x & 31), 32, wt,
                        geo(v, GCOSC, p, k, j), geo(v, GSINC, p, k, j), geo(v, GDX2A, p, k, j),
                        geo(v, GDX3A, p, k, j), x1f, x1v, dx1f, v.is, v.ie, dt, v.gamma, v.grav,
                        wt);
}

// panel.cuh -- LU panel with partial pivoting and implicit interchanges
// (included by lu.cu after its complex and cluster helpers).
//
// A panel of w <= 64 columns is factored by a cluster of cs CTAs, CTA `rank`
// owning rows [k + rank * rp, ...).  Columns advance in slices of `sl` (the
// widest multiple of 8 up to 64 whose rows fit shared memory) and, inside a
// slice, in sub-panels of 8 columns whose values stay in registers (RPT rows
// per thread of the first RW warps; the last four warps do the bookkeeping).
//
// What bounds it: a chain of w pivot steps, each a reduction over all rows,
// one exchange between the CTAs and one rank-1 update.  Measured on B200 with
// the arithmetic taken out, a step costs about 300 cycles inside one CTA (one
// barrier) and 820 to 900 with st.async mailboxes in clusters of 2 to 8 CTAs,
// 960 to 1150 in clusters of 16; the reduction and the update are bound by
// instruction issue, so:
//
//  - rows never move while the panel runs.  A thread keeps its rows and each
//    row's current position; choosing a pivot only changes positions.  The
//    step needs no second row, a sub-panel's end moves nothing, and the
//    interchanges become real once, when the finished panel is written.
//  - few warps own rows, several rows per thread: the per-warp work of a step
//    (keys, reduction, pivot row, reciprocal) is paid once for all of them.
//    Candidates are pushed and lists kept by warps that own none.
//  - fewer, taller CTAs: shared memory holds one slice, not the panel.  The
//    finished slices lie in A (each row still at its old place) and update a
//    new slice in one pass from L2.
//  - the winner's values right of the sub-panel leave for every CTA as soon
//    as it is known, under the following steps; the sub-panel's end waits on
//    that mailbox instead of a cluster barrier.
//
// Pivot choice is LAPACK's (largest |re| + |im|, first position on ties).
#pragma once

// Orders candidates by (key, position): the lane with the largest key and,
// among equal keys, the lowest position.  FP32 keys are one word (lo unused).
template <typename R>
__device__ __forceinline__ int warp_best(unsigned hi, unsigned lo, int pos) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned mh = __reduce_max_sync(FULL, hi);
  bool e = hi == mh;
  unsigned m = __ballot_sync(FULL, e);
  if ((m & (m - 1)) && mh != 0u) {
    if constexpr (sizeof(R) == 8) {
      const unsigned ml = __reduce_max_sync(FULL, e ? lo : 0u);
      e = e && lo == ml;
    }
    const int pm = __reduce_min_sync(FULL, e ? pos : INT_MAX);
    m = __ballot_sync(FULL, e && pos == pm);
  }
  return __ffs(m) - 1;
}

// A row's pivot key: 0 when it cannot be chosen, else the bits of |re| + |im|
// (>= 0, so they order as the value does; a NaN counts as 0) with the high
// word raised by one.
__device__ __forceinline__ void pivot_key(zf z, bool elig, unsigned& hi, unsigned& lo) {
  float b = cabs1(z);
  if (!(b >= 0.f)) b = 0.f;
  hi = elig ? __float_as_uint(b) + 1u : 0u;
  lo = 0u;
}
__device__ __forceinline__ void pivot_key(zd z, bool elig, unsigned& hi, unsigned& lo) {
  double b = cabs1(z);
  if (!(b >= 0.0)) b = 0.0;
  const unsigned long long q = elig ? (unsigned long long)__double_as_longlong(b) + (1ull << 32) : 0ull;
  hi = (unsigned)(q >> 32);
  lo = (unsigned)q;
}

template <typename R>
struct PanelIp {
  // the slice (16 elements of slack for the last row tile) and, with more than
  // one slice, the U12 block: U rows of the slices before, pitch sl + kPad
  static constexpr int kPad = sizeof(R) == 4 ? 4 : 2;  // pitch padding of the U blocks: conflict-free fragments
  // elements of the slice, which also holds L11 of the slices before while U12 is formed
  __host__ __device__ static int slice(int sl, int rps, int w) {
    const int e = (w - 1) / sl * sl, a = sl * rps + 16, b = e * e + 64;
    return e > 0 && b > a ? b : a;
  }
  static size_t smem(int sl, int rps, int w) {
    return ((size_t)slice(sl, rps, w) + (size_t)((w - 1) / sl * sl) * (sl + kPad)) * sizeof(cpx<R>);
  }
};

// `cols` entries of one row from shared memory to A, eight loads in flight.
template <typename R>
__device__ __forceinline__ void panel_store_row(typename Elt<R>::T* dst, size_t lda, const cpx<R>* src, int rps,
                                                int cols) {
  for (int c = 0; c < cols; c += 8) {
    cpx<R> t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = src[(size_t)min(c + u, cols - 1) * rps];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (c + u < cols) stc<R>(&dst[(size_t)(c + u) * lda], t[u]);
  }
}

// Rows [row0, row0 + rcount) of `cols` columns from col0 into s (pitch rps),
// issued by one thread as one bulk copy per column (size rounded up to 16
// bytes: lda and the rows are even) completing on bar; false when the
// addresses do not allow it.
template <typename R>
__device__ __forceinline__ bool panel_bulk_ok(const typename Elt<R>::T* A, size_t lda, int row0) {
  return sizeof(R) == 8 || ((((size_t)A | (lda * sizeof(float2)) | ((size_t)row0 * sizeof(float2))) & 15) == 0);
}
template <typename R>
__device__ __forceinline__ void panel_bulk_load(const typename Elt<R>::T* A, size_t lda, int row0, int col0, int rcount,
                                                int cols, cpx<R>* s, int rps, uint64_t* bar) {
  const unsigned bytes = (unsigned)((rcount * sizeof(cpx<R>) + 15) & ~(size_t)15);
  mbar_expect_tx(bar, bytes * (unsigned)cols);
  for (int c = 0; c < cols; ++c) bulk_g2s(s + (size_t)c * rps, A + (size_t)(col0 + c) * lda + row0, bytes, bar);
}

// C(16 rows x 32 columns from column n0) -= L U for one warp, TF32 operands
// (FP32 accumulation): kk rows of U, U(t, c) = ub[t * uld + c], L's fragments
// from lf(kstep, part) and C, once ready() returns, through cld / cst (row
// half h, column c).
template <typename LF, typename WT, typename CL, typename CS>
__device__ __forceinline__ void panel_tile(int kk, int ncol, const zf* ub, int uld, LF lf, WT ready, CL cld, CS cst) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  float pr[4][4], pi[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) pr[nt][e] = pi[nt][e] = 0.f;
#pragma unroll 4
  for (int ks = 0; ks < kk; ks += 8) {
    const zf x0 = lf(ks + t4, 0), x1 = lf(ks + t4, 8), x2 = lf(ks + t4 + 4, 0), x3 = lf(ks + t4 + 4, 8);
    const unsigned ar[4] = {to_tf32(x0.re), to_tf32(x1.re), to_tf32(x2.re), to_tf32(x3.re)};
    const unsigned ai[4] = {to_tf32(x0.im), to_tf32(x1.im), to_tf32(x2.im), to_tf32(x3.im)};
    const unsigned an[4] = {ai[0] ^ 0x80000000u, ai[1] ^ 0x80000000u, ai[2] ^ 0x80000000u, ai[3] ^ 0x80000000u};
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
      if (nt * 8 < ncol) {
        const zf y0 = ub[(ks + t4) * uld + nt * 8 + g], y1 = ub[(ks + t4 + 4) * uld + nt * 8 + g];
        const unsigned br[2] = {to_tf32(y0.re), to_tf32(y1.re)}, bi[2] = {to_tf32(y0.im), to_tf32(y1.im)};
        mma_tf32(pr[nt], ar, br);
        mma_tf32(pr[nt], an, bi);
        mma_tf32(pi[nt], ar, bi);
        mma_tf32(pi[nt], ai, br);
      }
  }
  ready();
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
    if (nt * 8 < ncol) {
      zf z[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) z[e] = cld((e >> 1) << 3, nt * 8 + 2 * t4 + (e & 1));
#pragma unroll
      for (int e = 0; e < 4; ++e)
        cst((e >> 1) << 3, nt * 8 + 2 * t4 + (e & 1), zf{z[e].re - pr[nt][e], z[e].im - pi[nt][e]});
    }
}

// The same for FP64 on the DMMA units, 16 rows x 16 columns (C loaded first
// and accumulated onto): SIMT rank-8 updates at two or three warps per
// scheduler reached 0.4 of the FP64 rate, DMMA needs far fewer instructions
// and shared-memory reads in flight.
template <typename LF, typename WT, typename CL, typename CS>
__device__ __forceinline__ void panel_tile(int kk, int ncol, const zd* ub, int uld, LF lf, WT ready, CL cld, CS cst) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  double re[2][2][2], im[2][2][2];  // [row half][column half][pair]
  ready();
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const zd z = nt * 8 < ncol ? cld(8 * h, nt * 8 + 2 * t4 + e) : zd{0.0, 0.0};
        re[h][nt][e] = z.re;
        im[h][nt][e] = z.im;
      }
#pragma unroll 2
  for (int ks = 0; ks < kk; ks += 4) {
    const zd x[2] = {lf(ks + t4, 0), lf(ks + t4, 8)};
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
      if (nt * 8 < ncol) {
        const zd y = ub[(ks + t4) * uld + nt * 8 + g];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          dmma(re[h][nt][0], re[h][nt][1], -x[h].re, y.re);
          dmma(im[h][nt][0], im[h][nt][1], -x[h].re, y.im);
          dmma(re[h][nt][0], re[h][nt][1], x[h].im, y.im);
          dmma(im[h][nt][0], im[h][nt][1], -x[h].im, y.re);
        }
      }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
      if (nt * 8 < ncol)
#pragma unroll
        for (int e = 0; e < 2; ++e) cst(8 * h, nt * 8 + 2 * t4 + e, zd{re[h][nt][e], im[h][nt][e]});
}

template <typename R, int RW, int RPT>
__global__ void __launch_bounds__(RW * 32 + 128, 1) k_panel_ip(PanelArgs a) {
  using E = typename Elt<R>::T;
  using C = cpx<R>;
  constexpr int SW = 8, NB = 64, NT = RW * 32 + 128, NW = NT / 32, RT = RW * 32;
  constexpr int UP = NB + PanelIp<R>::kPad;  // pitch of s_u (conflict-free fragments)
  constexpr int TN = sizeof(R) == 4 ? 32 : 16;  // columns of a panel_tile
  constexpr int KW = RowWords<R>::kN, CW = SW / KW;  // 16-byte words per row, columns per word
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const s_a = reinterpret_cast<C*>(smem_raw);          // [sl][rps] the slice, rows at their old places
  const int SL = a.sl, rps = a.rps, ULD = SL + PanelIp<R>::kPad;
  C* const s_u12 = s_a + PanelIp<R>::slice(SL, rps, a.w);           // [sb][ULD] U rows of the finished slices, this slice's columns
  __shared__ uint4 s_box[2][16][1 + KW];                  // [column parity][CTA]: candidate (key, position, row), 8 values
  __shared__ uint4 s_wt[2][RW][1 + KW];                   // the same, staged by every warp's best row
  __shared__ uint4 s_k[2][RW];                            // its key and position (for the CTA's reduction)
  __shared__ __align__(16) C s_u[SW][UP];                 // U of the sub-panel's pivot rows, from its first column on
  __shared__ __align__(16) C s_l8[SW][SW];                // their L in the sub-panel
  __shared__ int s_orig[NB], s_prow[NB];                  // pivot t: its row at the panel's start, its position when chosen
  __shared__ int s_dsrc[NB], s_ddst[NB], s_nd;            // displaced rows: start row, final position
  __shared__ uint64_t s_mb[2], s_mbu, s_mbl;              // mailboxes: a column's candidates, a sub-panel's U rows; slice loads

  const unsigned long long wlim = wait_limit(a.status);
  const int cs = a.cs;
  const int rank = cs > 1 ? (int)cluster_rank() : 0;
  const int prob = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool rows = warp < RW;   // this warp owns rows
  const int ht = tid - RT;       // thread among the helpers
  E* const A = static_cast<E*>(a.A) + (size_t)prob * a.bstride;
  const size_t lda = a.lda;
  const int rp = a.rp, w = a.w, k = a.k;
  const int rbase = k + rank * rp;
  const int rcount = max(0, min(rp, a.nn - rbase));
  E* const ubuf = static_cast<E*>(a.ubuf) + (size_t)prob * NB * NB;  // [c][t] U of all but the last slice

  const bool bulk = panel_bulk_ok<R>(A, lda, rbase);
  if (tid == 0) {
    mbar_init(&s_mb[0], 1);
    mbar_init(&s_mb[1], 1);
    mbar_init(&s_mbu, 1);
    mbar_init(&s_mbl, 1);
    if (bulk && rcount > 0) panel_bulk_load<R>(A, lda, rbase, k, rcount, min(SL, w), s_a, rps, &s_mbl);
  }
  if (!bulk) load_slice_async<R>(A, lda, rbase, k, rcount, min(SL, w), s_a, rps);
  if (rank == 0 && prob == 0 && tid == 0 && a.pstart) {
    a.pstart[a.pidx] = k;
    a.pstart[a.pidx + 1] = k + w;
  }
  __syncthreads();
  if (cs > 1) cluster_sync();  // every CTA's mbarriers exist before the first push
  unsigned mph = 0, uph = 0, lph = 0;  // phase bits of s_mb[0], s_mb[1], of s_mbu and of s_mbl
  bool gave_up = false;        // a wait of this thread ran out: later waits are skipped
  auto wait_mail = [&](uint64_t* bar, unsigned parity) {
    if (!gave_up && !mbar_wait(bar, parity, wlim)) {
      gave_up = true;
      atomicExch(&a.status[ST_TIMEOUT], 1);
    }
  };
  // a slice load must land before its buffer is used or the CTA leaves: waited
  // for even after another wait ran out
  auto wait_slice = [&]() {
    if (bulk && rcount > 0) {
      if (!mbar_wait(&s_mbl, lph, wlim)) {
        gave_up = true;
        atomicExch(&a.status[ST_TIMEOUT], 1);
      }
      lph ^= 1u;
    }
  };
  wait_slice();

  // Current position of my rows: >= the column's row while it can be chosen,
  // its final position once it is a pivot (-1: no row).
  int pos[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) pos[i] = rows && tid + i * RT < rcount ? rbase + tid + i * RT : -1;
  // every CTA's last warp follows the panel's first w rows, the only ones an
  // interchange can displace (lane l: rows k + l and k + 32 + l)
  int t0 = k + lane, t1 = k + 32 + lane;
  C v[RPT][SW];
  const C czero{R(0), R(0)};

  for (int sb = 0; sb < w; sb += SL) {
    const int se = min(w, sb + SL), wsl = se - sb;
    const bool last = se >= w;
    if (sb > 0) {
      // The finished slices update this one: U12 = L11^-1 (pivot rows of A),
      // then C - L U12, C and L straight from A (rows at their old places).
      C* const s_l = s_a;  // L11 by columns [t][sb]; the slice is written only after the solve
{
        const int total = sb * (sb + wsl);  // L11, then the pivot rows of A; four loads in flight
        for (int i0 = tid; i0 < total; i0 += 4 * NT) {
          C t[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * NT, c = i / sb, r = i - c * sb;
            t[u] = i < total && (c >= sb || r > c) ? ldc_cg<R>(&A[(size_t)(k + c) * lda + s_orig[r]]) : czero;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * NT, c = i / sb, r = i - c * sb;
            if (i >= total) continue;
            if (c < sb)
              s_l[i] = t[u];
            else
              s_u12[r * ULD + c - sb] = t[u];
          }
        }
      }
      __syncthreads();
      {
        // lanes = rows (and rows + 32), up to four columns per warp; L11 is
        // stored with zeros on and above the diagonal, and lanes past sb
        // compute values nobody reads
        constexpr int QC = 4;
        const bool tall = sb > 32;
        for (int c0 = warp; c0 < wsl; c0 += NW * QC) {
          C x[QC][2];
#pragma unroll
          for (int q = 0; q < QC; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              x[q][h] = c0 + q * NW < wsl && lane + 32 * h < sb ? s_u12[(lane + 32 * h) * ULD + c0 + q * NW] : czero;
#pragma unroll 4
          for (int t = 0; t < sb; ++t) {
            const C l0 = s_l[t * sb + lane], l1 = tall ? s_l[t * sb + lane + 32] : czero;
#pragma unroll
            for (int q = 0; q < QC; ++q) {
              const C src = t < 32 ? x[q][0] : x[q][1];
              const C u{__shfl_sync(FULL, src.re, t & 31), __shfl_sync(FULL, src.im, t & 31)};
              if (t < 31) cfms(x[q][0], l0, u);
              if (tall) cfms(x[q][1], l1, u);
            }
          }
#pragma unroll
          for (int q = 0; q < QC; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (c0 + q * NW < wsl && lane + 32 * h < sb) s_u12[(lane + 32 * h) * ULD + c0 + q * NW] = x[q][h];
        }
      }
      __syncthreads();
      if (rank == 0 && !last)  // U of this slice's columns (the last slice's follows at the end)
        for (int i = tid; i < sb * wsl; i += NT)
          stc<R>(&ubuf[(size_t)(sb + i / sb) * NB + i % sb], s_u12[(i % sb) * ULD + i / sb]);
      // C lands in s_a (over L11, whose readers are past the barrier) while L
      // comes from L2
      if (tid == 0 && bulk && rcount > 0) {
        asm volatile("fence.proxy.async;" ::: "memory");
        panel_bulk_load<R>(A, lda, rbase, k + sb, rcount, wsl, s_a, rps, &s_mbl);
      }
      if (!bulk) {
        load_slice_async<R>(A, lda, rbase, k + sb, rcount, wsl, s_a, rps);
        __syncthreads();
      }
{
        const int g = lane >> 2;
        const E* const Lp = A + (size_t)k * lda + rbase;
        bool landed = false;
        for (int rb = warp * 16; rb < rcount; rb += NW * 16) {
          C* const sr = s_a + rb + g;
          const int ra = min(rb + g, rcount - 1), rb2 = min(rb + g + 8, rcount - 1);
          for (int n0 = 0; n0 < wsl; n0 += TN)
            panel_tile(
                sb, wsl - n0, s_u12 + n0, ULD,
                [&](int t, int h) { return ldc_cg<R>(&Lp[(size_t)t * lda + (h ? rb2 : ra)]); },
                [&]() {
                  if (!landed) wait_slice();
                  landed = true;
                },
                [&](int h, int c) { return sr[min(n0 + c, wsl - 1) * rps + h]; },
                [&](int h, int c, C z) {
                  if (rb + g + h < rcount && n0 + c < wsl) sr[(n0 + c) * rps + h] = z;
                });
        }
        if (!landed) wait_slice();
      }
      __syncthreads();
    }

    for (int s0 = 0; s0 < wsl; s0 += SW) {  // columns relative to the slice
      const int sw = min(SW, wsl - s0);
      const int nright = wsl - s0 - SW;  // columns right of the sub-panel (<= 0: the slice's last)
      const int nrw = sizeof(R) == 4 ? (nright + 1) / 2 : nright;  // ... as 16-byte words
      if (cs > 1 && nright > 0 && tid == 0) mbar_expect_tx(&s_mbu, (unsigned)(SW * (KW + nrw)) * 16u);
#pragma unroll
      for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int c = 0; c < SW; ++c)
          v[i][c] = (rows && tid + i * RT < rcount && c < sw) ? s_a[(s0 + c) * rps + tid + i * RT] : czero;

      // One code path for all columns: v[.][0] is the current column, and the
      // update moves every value one column down.
      unsigned hi = 0, lo = 0;  // my best row for the current column: key, index, position
      int bi = 0, bp = 0;
      auto my_best = [&](int g) {
        bi = 0;
        bp = pos[0];
        pivot_key(v[0][0], pos[0] >= g, hi, lo);
#pragma unroll
        for (int i = 1; i < RPT; ++i) {
          unsigned h2, l2;
          pivot_key(v[i][0], pos[i] >= g, h2, l2);
          const bool gt = h2 > hi || (h2 == hi && (l2 > lo || (l2 == lo && pos[i] < bp)));
          hi = gt ? h2 : hi;
          lo = gt ? l2 : lo;
          bi = gt ? i : bi;
          bp = gt ? pos[i] : bp;
        }
      };
      if (rows) my_best(k + sb + s0);
      // the steps jj < 4 update 7 columns, the others the 3 that are left
      auto step = [&](auto nupd, int jj) {
        constexpr int NU = decltype(nupd)::value;
        const int j = sb + s0 + jj, gj = k + j, par = j & 1;
        if (rows) {
          // 1. The warp's best row, its values staged for the CTA.
          const int wl = warp_best<R>(hi, lo, bp);
          if (lane == wl) {
            s_k[par][warp] = make_uint4(hi, lo, (unsigned)bp, 0u);
            s_wt[par][warp][0] = make_uint4(hi, lo, (unsigned)bp, (unsigned)(rbase + tid + bi * RT));
#pragma unroll
            for (int i = 0; i < RPT; ++i)
              if (i == bi)
#pragma unroll
                for (int q = 0; q < KW; ++q) s_wt[par][warp][1 + q] = row_word<R>(v[i], q);
          }
        } else if (cs > 1 && ht == 0) {
          mbar_expect_tx(&s_mb[par], (unsigned)(cs * (1 + KW)) * 16u);
        }
        __syncthreads();
        // 2. The CTA's candidate; in a cluster the helper warps send it to
        //    every CTA's mailbox, and the winner is found there.
        const uint4* win;
        int wsrc = 0;
        if (cs == 1 || !rows) {
          const uint4 q = lane < RW ? s_k[par][lane] : make_uint4(0u, 0u, INT_MAX, 0u);
          const int ww = warp_best<R>(q.x, q.y, (int)q.z);
          win = &s_wt[par][ww][0];
          if (cs > 1 && lane < cs)
            for (int wi = warp - RW; wi < 1 + KW; wi += NW - RW)
              dsm_st4_async(&s_box[par][rank][wi], lane, win[wi], &s_mb[par]);
        }
        if (cs > 1) {
          wait_mail(&s_mb[par], (mph >> par) & 1u);
          mph ^= 1u << par;
          const uint4 q = lane < cs ? s_box[par][lane][0] : make_uint4(0u, 0u, INT_MAX, 0u);
          wsrc = warp_best<R>(q.x, q.y, (int)q.z);
          win = &s_box[par][wsrc][0];
        }
        C piv[SW];
        row_unword<R>(win + 1, piv);
        const uint4 head = win[0];
        int prow = (int)head.z, orig = (int)head.w;
        if (prow < gj || prow >= a.nn || orig < k || orig >= a.nn) prow = orig = gj;  // only after a timeout
        const bool zero = piv[0].re == R(0) && piv[0].im == R(0);
        if (rows) {
          // 3. Multipliers and the rank-1 update, in registers.
          const C rpv = zero ? czero : crcp(piv[0]);
          C l[RPT];
#pragma unroll
          for (int i = 0; i < RPT; ++i) {
            // no branch: rows that are done get values nobody reads
            pos[i] = pos[i] == prow ? gj : (pos[i] == gj ? prow : pos[i]);
            l[i] = v[i][0] * rpv;
            v[i][0] = v[i][1];
            cfms(v[i][0], l[i], piv[1]);  // the next column first: its search is the critical path
          }
          my_best(gj + 1);
#pragma unroll
          for (int i = 0; i < RPT; ++i) {
            if (pos[i] > gj) s_a[(s0 + jj) * rps + tid + i * RT] = l[i];
#pragma unroll
            for (int c = 1; c < NU; ++c) {
              C x = v[i][c + 1];
              cfms(x, l[i], piv[c + 1]);
              v[i][c] = x;
            }
            v[i][NU] = czero;
          }
        } else {
          // 4. Bookkeeping: positions, the pivot's row, its U in the sub-panel,
          //    and (from its owner) its L in the sub-panel and its values right of it.
          if (ht < SW - jj) s_u[jj][jj + ht] = reinterpret_cast<const C*>(win + 1)[ht];
          if (ht == 0) {
            s_orig[j] = orig;
            s_prow[j] = prow;
            if (zero && rank == 0 && !a.no_singular) atomicCAS(&a.status[ST_SINGULAR], 0, gj + 1);
          }
          if (warp == NW - 1) {
            t0 = t0 == prow ? gj : (t0 == gj ? prow : t0);
            t1 = t1 == prow ? gj : (t1 == gj ? prow : t1);
          }
          if (nright > 0 && wsrc == rank) {
            const int lr = min(max(orig - rbase, 0), rp - 1);
            if (cs == 1) {
              if (ht < jj) s_l8[jj][ht] = s_a[(s0 + ht) * rps + lr];
              if (ht >= SW && ht < SW + nright) s_u[jj][ht] = s_a[(s0 + ht) * rps + lr];
            } else {
              for (int i = ht; i < (KW + nrw) * cs; i += NT - RT) {
                const int q = i / cs, dst = i % cs;
                const C* src = &s_a[(s0 + q * CW) * rps + lr];
                uint4 word;
                if constexpr (sizeof(R) == 4) {
                  const C x = src[0], y = src[rps];
                  word = make_uint4(__float_as_uint(x.re), __float_as_uint(x.im), __float_as_uint(y.re),
                                    __float_as_uint(y.im));
                } else {
                  word = *reinterpret_cast<const uint4*>(src);
                }
                dsm_st4_async(q < KW ? reinterpret_cast<uint4*>(&s_l8[jj][0]) + q
                                     : reinterpret_cast<uint4*>(&s_u[jj][0]) + q,
                              (unsigned)dst, word, &s_mbu);
              }
            }
          }
        }
      };
#pragma unroll 1
      for (int jj = 0; jj < min(sw, SW / 2); ++jj) step(std::integral_constant<int, SW - 1>{}, jj);
#pragma unroll 1
      for (int jj = SW / 2; jj < sw; ++jj) step(std::integral_constant<int, SW / 2 - 1>{}, jj);

      // End of the sub-panel.
      if (cs > 1 && nright > 0) {
        wait_mail(&s_mbu, uph);
        uph ^= 1u;
      }
      __syncthreads();
      if (nright > 0) {
        // U right of the sub-panel: U(i,c) = A(i,c) - sum_{t<i} L(i,t) U(t,c).
        if (tid < nright) {
          C x[SW];
#pragma unroll
          for (int i = 0; i < SW; ++i) x[i] = s_u[i][SW + tid];
#pragma unroll
          for (int i = 1; i < SW; ++i) {
#pragma unroll
            for (int t = 0; t < i; ++t) cfms(x[i], s_l8[i][t], x[t]);
            s_u[i][SW + tid] = x[i];
          }
        }
        __syncthreads();
      }
      if (rank == 0) {  // the sub-panel's U rows, from each pivot's column on
        E* const ud = last ? A + (size_t)(k + sb + s0) * lda + k + sb + s0 : ubuf + (size_t)(sb + s0) * NB + sb + s0;
        const size_t ul = last ? lda : NB;
        const int wr = wsl - s0;
        for (int i = tid; i < SW * wr; i += NT) {
          const int t = i % SW, c = i / SW;
          if (c >= t && t < sw) stc<R>(&ud[(size_t)c * ul + t], s_u[t][c]);
        }
      }
      if (nright > 0) {
        // Rank-8 update of the slice's columns right of the sub-panel (rows
        // that are pivots already get values nobody reads).
        const int g = lane >> 2;
        for (int rb = warp * 16; rb < rcount; rb += NW * 16) {
          C* const sr = s_a + (size_t)s0 * rps + rb + g;
          for (int n0 = 0; n0 < nright; n0 += TN)
            panel_tile(
                SW, nright - n0, &s_u[0][SW + n0], UP, [&](int t, int h) { return sr[t * rps + h]; }, []() {},
                [&](int h, int c) { return sr[min(SW + n0 + c, wsl - s0 - 1) * rps + h]; },
                [&](int h, int c, C z) {
                  if (rb + g + h < rcount && n0 + c < nright) sr[(SW + n0 + c) * rps + h] = z;
                });
        }
        __syncthreads();
      }
    }
    if (!last) {
      // The finished slice to A, every row still at its old place.
      for (int r = tid; r < rcount; r += NT)
        panel_store_row<R>(A + (size_t)(k + sb) * lda + rbase + r, lda, s_a + r, rps, wsl);
    } else {
      // No pushes any more.  A CTA whose waits ran out gets here early; it
      // must not leave while others may still write to its mailboxes.
      if (cs > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
      // U12 and the rows to their final positions (pivot t: its L; its U in the
      // slice is there): every CTA has long read what it needs of these columns.
      if (rank == 0)
        for (int i = tid; i < sb * wsl; i += NT)
          stc<R>(&A[(size_t)(k + sb + i / sb) * lda + k + i % sb], s_u12[(i % sb) * ULD + i / sb]);
      if (rows)
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          if (pos[i] < 0) continue;
          const int lim = min(wsl, pos[i] < k + w ? pos[i] - k - sb : wsl);
          panel_store_row<R>(A + (size_t)(k + sb) * lda + pos[i], lda, s_a + tid + i * RT, rps, lim);
        }
      if (warp == NW - 1) {  // displaced rows: the first w rows that did not become pivots
        const bool d0 = lane < w && t0 >= k + w, d1 = lane + 32 < w && t1 >= k + w;
        const unsigned m0 = __ballot_sync(FULL, d0), m1 = __ballot_sync(FULL, d1);
        const unsigned below = (1u << lane) - 1;
        if (d0) {
          s_dsrc[__popc(m0 & below)] = k + lane;
          s_ddst[__popc(m0 & below)] = t0;
        }
        if (d1) {
          s_dsrc[__popc(m0) + __popc(m1 & below)] = k + 32 + lane;
          s_ddst[__popc(m0) + __popc(m1 & below)] = t1;
        }
        if (lane == 0) s_nd = __popc(m0) + __popc(m1);
      }
    }
    if (cs > 1 && !last)
      cluster_sync();
    else
      __syncthreads();
  }
  // The interchanges on the earlier slices, whole columns per CTA: pivot t's
  // row to position k + t (its L from A, its U from ubuf), the displaced rows
  // to the places they took.
  const int nd = s_nd, early = (w - 1) / SL * SL;  // columns before the last slice
  constexpr int PU = 8, CB = PU * NT / NB;         // columns handled at a time
  for (int cb = rank; cb < early; cb += CB * cs) {
    C f[PU], d[PU];
#pragma unroll
    for (int u = 0; u < PU; ++u) {
      const int i = tid + u * NT, c = cb + (i / NB) * cs, t = i % NB;
      if (c < early && t < w)
        f[u] = c < t ? ldc_cg<R>(&A[(size_t)(k + c) * lda + s_orig[t]]) : ldc_cg<R>(&ubuf[(size_t)c * NB + t]);
      if (c < early && t < nd) d[u] = ldc_cg<R>(&A[(size_t)(k + c) * lda + s_dsrc[t]]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PU; ++u) {
      const int i = tid + u * NT, c = cb + (i / NB) * cs, t = i % NB;
      if (c < early && t < w) stc<R>(&A[(size_t)(k + c) * lda + k + t], f[u]);
      if (c < early && t < nd) stc<R>(&A[(size_t)(k + c) * lda + s_ddst[t]], d[u]);
    }
  }
  if (rank == 0) {
    int* ipiv = a.ipiv + (size_t)prob * a.ipiv_stride;
    int* perm = a.perm + (size_t)prob * a.perm_stride;
    if (tid == 0) perm[0] = w + nd;
    if (tid < w) {
      ipiv[k + tid] = s_prow[tid] + 1;
      perm[1 + 2 * tid] = k + tid;
      perm[2 + 2 * tid] = s_orig[tid];
    }
    if (tid < nd) {
      perm[1 + 2 * (w + tid)] = s_ddst[tid];
      perm[2 + 2 * (w + tid)] = s_dsrc[tid];
    }
  }
  if (cs > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

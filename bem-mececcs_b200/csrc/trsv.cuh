// trsv.cuh -- FP32 triangular solves with the LU factors in one thread-block
// cluster per problem (included by lu.cu after its helpers).
//
// The refinement solves L U d = r two or three times per factorisation.  What
// bounds a solve is the chain of 64-row steps, then the factors' bytes: the
// cooperative kernel (k_trsv_f32) gathers the step's rows, applies the block
// inverse, updates every row and meets at a grid barrier in global memory, 5
// to 7 us a step (1.46 ms for a solve of 7 x 6480 unknowns whose factors take
// 0.36 ms to read).  Here
//
//  - L is put into its final row order once per factorisation (k_row_maps,
//    k_lperm: later panels' interchanges applied to earlier columns, only to
//    rows that move), so the right-hand side is permuted once and a step
//    gathers nothing;
//  - the CTAs of a cluster own 64-row blocks cyclically.  A step's 64 values
//    go to every CTA by st.async; the owner of the next block updates that
//    block first, applies its inverse and sends its values on, while the other
//    rows' updates follow behind.  A step costs one block product, one inverse
//    product and one exchange;
//  - a producer warp streams the CTA's tiles (64 x 64) in the order they are
//    used, as far ahead as its ring of stages allows, whatever the chain does.
#pragma once

constexpr int kTclSlots = 16;               // steps whose values a CTA can hold
constexpr int kTclStage = 64 * 64;          // complex elements of a tile
constexpr int kTclThreads = 8 * 32 + 32;    // eight consumer warps, one producer

struct TrsvClArgs {
  float2* v;              // problem b at v + b * vstride: right-hand side in, solution out
  size_t vstride;
  int nn, nb, npan;       // unknowns, 64-row blocks, forward inverses per problem
  int forward;            // forward and back substitution, or back substitution only
  int stages, own;        // ring stages, blocks a CTA may own
  const float2* tinv;     // [problem][npan + nb][64][64] by columns: inverses of L11, then of the U blocks
  const int* rows;        // [problem][npan + 1][nn]: the last one gives the row at each final position
  int* status;
};

// Row maps of a factorisation whose panels are 64 wide, one CTA per problem:
// map p (p < npan) gives for a final position q >= 64 (p + 1) the position
// where panel p left its row, moved[p] whether any differs; map npan the row
// that starts at the top and ends at q.  From the last panel back, a row's
// position before panel p's interchanges is read from the panel's list.
__global__ void __launch_bounds__(1024) k_row_maps(int nn, int npan, int batch, const int* __restrict__ perm,
                                                   int* rows, int* moved) {
  extern __shared__ int s_mem[];
  int* const m = s_mem;        // [nn] position of the row that ends at q
  int* const tbl = s_mem + nn;  // [nn] the panel's list as a table
  const int prob = blockIdx.x, tid = threadIdx.x;
  rows += (size_t)prob * (npan + 1) * nn;
  moved += (size_t)prob * npan;
  for (int q = tid; q < nn; q += 1024) m[q] = tbl[q] = q;
  auto entry = [&](int p, int& dst, int& src) {
    const int* pl = perm + ((size_t)p * batch + prob) * kPermStride;
    dst = -1;
    if (p >= 0 && tid < 128 && tid < pl[0]) {
      dst = pl[1 + 2 * tid];
      src = pl[2 + 2 * tid];
    }
  };
  int dst, src = 0;
  entry(npan - 1, dst, src);
  __syncthreads();
  for (int p = npan - 1; p >= 0; --p) {
    int any = 0;
    for (int q = 64 * (p + 1) + tid; q < nn; q += 1024) {
      const int x = m[q];
      rows[(size_t)p * nn + q] = x;
      any |= x != q;
    }
    if (dst >= 0) tbl[dst] = src;
    any = __syncthreads_or(any);
    if (tid == 0) moved[p] = any;
    for (int q = 64 * p + tid; q < nn; q += 1024) m[q] = tbl[m[q]];
    __syncthreads();
    if (dst >= 0) tbl[dst] = dst;
    if (p > 0) entry(p - 1, dst, src);
    __syncthreads();
  }
  for (int q = tid; q < nn; q += 1024) rows[(size_t)npan * nn + q] = m[q];
}

// L of panel blockIdx.x into its final row order (4 of its 64 columns per
// CTA), in place: the rows that move are read, then written.
__global__ void __launch_bounds__(256) k_lperm(float2* Abase, size_t lda, size_t bstride, int nn, int npan,
                                               const int* __restrict__ rows, const int* __restrict__ moved) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* const s = reinterpret_cast<float2*>(smem_raw);
  const int p = blockIdx.x, prob = blockIdx.z, r0 = 64 * (p + 1);
  if (!moved[(size_t)prob * npan + p]) return;
  const int* const map = rows + ((size_t)prob * (npan + 1) + p) * nn;
  float2* const A = Abase + (size_t)prob * bstride;
  for (int c = 64 * p + 4 * blockIdx.y; c < 64 * p + 4 * (int)blockIdx.y + 4; ++c) {
    float2* const col = A + (size_t)c * lda;
    for (int q = r0 + threadIdx.x; q < nn; q += 256) {
      const int x = map[q];
      if (x != q) s[q - r0] = col[x];
    }
    __syncthreads();
    for (int q = r0 + threadIdx.x; q < nn; q += 256)
      if (map[q] != q) col[q] = s[q - r0];
    __syncthreads();
  }
}

// Inverses of the diagonal blocks the solves step through, by columns
// [64][64], zero outside the block: blocks [0, npan) the unit-lower L11 of
// panel b, blocks [npan, npan + nb) the upper triangles.  An upper block is
// inverted as the lower one it is with rows and columns reversed.  16 x 16
// diagonal blocks first (a warp each, lane = column), then X21 = -X22 L21 X11
// at 16 and 32, as k_l11_inv; a thread per column of the whole block took a
// chain of 64 dependent sums (119 us for 32 x 720 unknowns).
__global__ void __launch_bounds__(256) k_tri_inv_cl(const float2* __restrict__ Abase, size_t lda, size_t bstride, int nn,
                                                    int npan, int b0, int nblocks, float2* inv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* const s_x = reinterpret_cast<float2*>(smem_raw);  // [64][kLtLd] the inverse, row-major
  float2* const s_l = s_x + 64 * kLtLd;                      // [64][kLtLd] the block, row-major
  const int b = b0 + blockIdx.x, prob = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float2* A = Abase + (size_t)prob * bstride;
  float2* const out = inv + ((size_t)prob * nblocks + b) * kTclStage;
  const bool lower = b < npan;
  const int k0 = 64 * (lower ? b : b - npan), w = min(64, nn - k0);
  auto at = [](float2* M, int i, int j) -> float2& { return M[i * kLtLd + j]; };
  for (int q = tid; q < 64 * 64; q += 256) {
    const int i = q & 63, c = q >> 6;  // row, column of the block
    float2 z = make_float2(0.f, 0.f);
    if (i < w && c < w && (lower ? i > c : i <= c)) z = A[(size_t)(k0 + c) * lda + k0 + i];
    if (lower ? i == c : i == c && i >= w) z = make_float2(1.f, 0.f);
    const int ii = lower ? i : 63 - i, cc = lower ? c : 63 - c;
    at(s_l, ii, cc) = z;
    at(s_x, ii, cc) = make_float2(0.f, 0.f);
  }
  __syncthreads();
  if (warp < 4 && lane < 16) {
    const int o = 16 * warp, c = lane;
    zf x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      zf acc{i == c ? 1.f : 0.f, 0.f}, acc2{0.f, 0.f};
#pragma unroll
      for (int t = 0; t < i; ++t) {
        const float2 l = at(s_l, o + i, o + t);
        cfms((t & 1) ? acc2 : acc, zf{l.x, l.y}, x[t]);
      }
      acc = acc + acc2;
      const float2 d = at(s_l, o + i, o + i);
      x[i] = i < c ? zf{0.f, 0.f} : lower ? acc : (d.x == 0.f && d.y == 0.f) ? zf{0.f, 0.f} : acc * crcp(zf{d.x, d.y});
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) at(s_x, o + i, o + c) = make_float2(x[i].re, x[i].im);
  }
  __syncthreads();
  // the strict upper half of s_x (rows 0-31, columns 32-63) holds L21 X11 meanwhile
  for (int h = 16; h <= 32; h *= 2) {
    const int outs = 32 * h;  // (64 / 2h) blocks of h x h
    for (int q = tid; q < outs; q += 256) {
      const int pp = q / (h * h), i = (q / h) % h, j = q % h, o = pp * 2 * h;
      zf acc{0.f, 0.f}, acc2{0.f, 0.f};
      for (int t = 0; t < h; t += 2) {
        const float2 l = at(s_l, o + h + i, o + t), x = at(s_x, o + t, o + j);
        const float2 l2 = at(s_l, o + h + i, o + t + 1), x2 = at(s_x, o + t + 1, o + j);
        cfms(acc, zf{l.x, l.y}, zf{x.x, x.y});
        cfms(acc2, zf{l2.x, l2.y}, zf{x2.x, x2.y});
      }
      at(s_x, pp * h + i, 32 + j) = make_float2(acc.re + acc2.re, acc.im + acc2.im);  // -L21 X11
    }
    __syncthreads();
    for (int q = tid; q < outs; q += 256) {
      const int pp = q / (h * h), i = (q / h) % h, j = q % h, o = pp * 2 * h;
      zf acc{0.f, 0.f}, acc2{0.f, 0.f};
      for (int t = 0; t < h; t += 2) {
        const float2 x = at(s_x, o + h + i, o + h + t), u = at(s_x, pp * h + t, 32 + j);
        const float2 x2 = at(s_x, o + h + i, o + h + t + 1), u2 = at(s_x, pp * h + t + 1, 32 + j);
        cfms(acc, zf{-x.x, -x.y}, zf{u.x, u.y});
        cfms(acc2, zf{-x2.x, -x2.y}, zf{u2.x, u2.y});
      }
      at(s_x, o + h + i, o + j) = make_float2(acc.re + acc2.re, acc.im + acc2.im);
    }
    __syncthreads();
  }
  for (int q = tid; q < 64 * 64; q += 256) {
    const int i = q & 63, c = q >> 6;
    const bool in = i < w && c < w && (lower ? i >= c : i <= c);
    out[q] = in ? (lower ? at(s_x, i, c) : at(s_x, 63 - i, 63 - c)) : make_float2(0.f, 0.f);
  }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(const uint64_t* bar, unsigned rank) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_rank(bar, rank)) : "memory");
}
// mbar_wait that also orders the remote arrivals' reads before what follows.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, unsigned parity, unsigned long long limit_ns) {
  const bool ok = mbar_wait(bar, parity, limit_ns);
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
  return ok;
}

__global__ void __launch_bounds__(kTclThreads, 1) k_trsv_cl(const __grid_constant__ CUtensorMap tm, TrsvClArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  zf* const ring = reinterpret_cast<zf*>(smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u));
  zf* const s_acc = ring + (size_t)a.stages * kTclStage;  // [4 column groups][own][64] sums of T x
  zf* const s_y = s_acc + (size_t)4 * a.own * 64;         // [own][64] right-hand side, then solution
  __shared__ __align__(16) zf s_x[kTclSlots][64];         // the steps' values
  __shared__ __align__(16) zf s_xo[64];
  __shared__ zf s_g[64], s_part[4][64];
  __shared__ uint64_t s_full[8], s_empty[8], s_xfull[kTclSlots], s_xfree[kTclSlots];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, prob = blockIdx.y;
  const int G = gridDim.x, rank = G > 1 ? (int)cluster_rank() : 0;
  const int nn = a.nn, nb = a.nb, NS = a.stages;
  const unsigned long long wlim = wait_limit(a.status);
  float2* const v = a.v + (size_t)prob * a.vstride;
  const float2* const inv = a.tinv + (size_t)prob * (a.npan + nb) * kTclStage;
  const int nf = a.forward ? nb - 1 : 0, nsteps = nf + nb - 1;  // steps whose values are sent
  auto source = [&](int s) { return (s < nf ? s : nb - 1 - (s - nf)) % G; };  // the CTA that sends step s

  if (tid == 0) {
    for (int i = 0; i < 8; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], 8);
    }
    for (int i = 0; i < kTclSlots; ++i) {
      mbar_init(&s_xfull[i], 1);
      mbar_init(&s_xfree[i], 8 * G);
    }
    for (int s = 0; s < min(kTclSlots, nsteps); ++s) mbar_expect_tx(&s_xfull[s], 64 * sizeof(zf));
  }
  const int* const start = a.rows ? a.rows + ((size_t)prob * (a.npan + 1) + a.npan) * nn : nullptr;
  for (int i = tid; i < a.own * 64; i += kTclThreads) {
    const int q = ((i >> 6) * G + rank) * 64 + (i & 63);
    s_y[i] = q < nn ? ldc_cg<float>(&v[a.forward ? start[q] : q]) : zf{0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 4; ++c) s_acc[c * a.own * 64 + i] = zf{0.f, 0.f};
  }
  __syncthreads();
  if (G > 1) cluster_sync();  // every CTA's barriers exist and v has been read

  // The CTA's work in order: inv(b, ib, s) solves its block b with inverse ib
  // (its values are sent as step s, or not when s < 0), tile(b, p) updates its
  // block b with step values of block p, between begin(s) and end(s).
  auto run = [&](auto inv_b, auto tile, auto begin, auto end) {
    int s = 0;
    if (a.forward) {
      if (rank == 0) inv_b(0, 0, nf > 0 ? 0 : -1);
      for (int p = 0; p < nb - 1; ++p, ++s) {
        begin(s);
        int b = p + 1 + ((rank - (p + 1)) % G + G) % G;
        if (b == p + 1) {
          tile(b, p);
          inv_b(b, b, b < nb - 1 ? s + 1 : -1);
          b += G;
        }
        for (; b < nb; b += G) tile(b, p);
        end(s);
      }
    }
    if ((nb - 1) % G == rank) inv_b(nb - 1, a.npan + nb - 1, nb > 1 ? s : -1);
    for (int p = nb - 1; p > 0; --p, ++s) {
      begin(s);
      int b = p - 1 - (((p - 1) - rank) % G + G) % G;
      if (b == p - 1) {
        tile(b, p);
        inv_b(b, a.npan + b, b > 0 ? s + 1 : -1);
        b -= G;
      }
      for (; b >= 0; b -= G) tile(b, p);
      end(s);
    }
  };

  bool gave_up = false;
  int t = 0;  // tiles so far
  if (warp == 8) {
    if (lane == 0) {
      auto stage = [&]() -> int {
        const int st = t % NS;
        if (t >= NS && !gave_up && !mbar_wait(&s_empty[st], (t / NS - 1) & 1, wlim)) {
          gave_up = true;
          atomicExch(&a.status[ST_TIMEOUT], 1);
        }
        return st;
      };
      auto load_inv = [&](int, int ib, int) {
        const int st = stage();
        if (gave_up) return;
        mbar_expect_tx(&s_full[st], kTclStage * sizeof(zf));
        bulk_g2s(ring + (size_t)st * kTclStage, inv + (size_t)ib * kTclStage, kTclStage * sizeof(zf), &s_full[st]);
        ++t;
      };
      auto load_tile = [&](int b, int p) {
        const int st = stage();
        if (gave_up) return;
        mbar_expect_tx(&s_full[st], kTclStage * sizeof(zf));
        tma_rows_load(ring + (size_t)st * kTclStage, &tm, 64 * b, 64 * p, prob, &s_full[st]);
        ++t;
      };
      run(load_inv, load_tile, [](int) {}, [](int) {});
      for (int i = max(0, t - NS); i < t; ++i) mbar_wait(&s_full[i % NS], (i / NS) & 1, wlim);  // all loads have landed
    }
    __syncwarp();
  } else {
    const int row = 32 * (warp & 1) + lane, cg = warp >> 1;  // one row, 16 columns of every tile
    unsigned freeph = 0;  // phase bits of s_xfree
    auto give_up = [&]() {
      gave_up = true;
      atomicExch(&a.status[ST_TIMEOUT], 1);
    };
    auto bar = []() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    // sum over this thread's 16 columns of the next tile times x; the stage is
    // handed back once the warp has read it
    auto product = [&](const zf* x) -> zf {
      const int st = t % NS;
      if (!gave_up && !mbar_wait(&s_full[st], (t / NS) & 1, wlim)) give_up();
      const zf* T = ring + (size_t)st * kTclStage + (size_t)(16 * cg) * 64 + row;
      zf s0{0.f, 0.f}, s1{0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 16; c += 2) {
        cfma(s0, T[c * 64], x[16 * cg + c]);
        cfma(s1, T[(c + 1) * 64], x[16 * cg + c + 1]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[st]);
      ++t;
      return s0 + s1;
    };
    const zf* x = nullptr;
    auto solve = [&](int b, int, int s) {
      const int o = (b - rank) / G * 64;
      bar();  // every warp's sums for this block are there
      if (tid < 64) {
        zf g = s_y[o + tid];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          zf& z = s_acc[c * a.own * 64 + o + tid];
          g = g - z;
          z = zf{0.f, 0.f};
        }
        s_g[tid] = g;
      }
      bar();
      s_part[cg][row] = product(s_g);
      if (s >= kTclSlots) {  // every CTA is done with the values 16 steps back
        const int slot = s % kTclSlots;
        if (!gave_up && !mbar_wait_cluster(&s_xfree[slot], (freeph >> slot) & 1u, wlim)) give_up();
        freeph ^= 1u << slot;
      }
      bar();
      if (tid < 64) {
        const zf z = (s_part[0][tid] + s_part[1][tid]) + (s_part[2][tid] + s_part[3][tid]);
        s_y[o + tid] = z;
        s_xo[tid] = z;
      }
      bar();
      if (s >= 0)
        for (int dst = warp; dst < G; dst += 8)
          dsm_st4_async(reinterpret_cast<uint4*>(&s_x[s % kTclSlots][0]) + lane, (unsigned)dst,
                        reinterpret_cast<const uint4*>(s_xo)[lane], &s_xfull[s % kTclSlots]);
    };
    auto update = [&](int b, int) {
      const zf d = product(x);
      zf& z = s_acc[cg * a.own * 64 + (b - rank) / G * 64 + row];
      z = z + d;
    };
    auto begin = [&](int s) {
      const int slot = s % kTclSlots;
      if (!gave_up && !mbar_wait(&s_xfull[slot], (s / kTclSlots) & 1, wlim)) give_up();
      if (tid == 0 && s + kTclSlots < nsteps) mbar_expect_tx(&s_xfull[slot], 64 * sizeof(zf));
      x = s_x[slot];
    };
    auto end = [&](int s) {
      __syncwarp();
      if (lane == 0 && s + kTclSlots < nsteps) mbar_arrive_remote(&s_xfree[s % kTclSlots], source(s + kTclSlots));
    };
    run(solve, update, begin, end);
    bar();
    for (int i = tid; i < a.own * 64; i += 256) {
      const int q = ((i >> 6) * G + rank) * 64 + (i & 63);
      if (q < nn) stc<float>(&v[q], s_y[i]);
    }
  }
  if (G > 1) cluster_sync();  // no CTA leaves while others may still write to it
}

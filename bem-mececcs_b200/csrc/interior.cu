// interior.cu -- displacements and stresses at interior points on the device.
//
// INTEREC's interior part: the displacement at interior point K is
//   ZDSOL(3K+i) = sum_J  ZG_KJ(i,:) . ZDFI_J  -  ZH_KJ(i,:) . ZFI_J
// with NONSINGD's Stokes U and T over boundary element J seen from K
// (src/Interec.for:86-135, the computation cuda_interec1_ does on the
// reference's GPU, src/kernels/Interec1_cu.cu:44-237), and the stress is
//   ZSSOL(9K+i+3j) = sum_J sum_k ZDFI_J(k) ZD(k,i,j) - ZFI_J(k) ZS(k,i,j)
// with SIGMAEC's derivative kernels (src/Interec.for:186-285,
// src/Sigmaec.for:9-212).  ZFI / ZDFI are the boundary displacements and
// tractions after the un-swap.
//
// One thread per (interior point, boundary element): the NPG^2 Gauss points
// of the element (the per-mesh table of k_geometry) are visited once.  The
// boundary values t, u and the normal n are constant on the element, so the
// sums over the Gauss points keep only what varies: the coefficients of t_i,
// u_i, n_i and rd_i in the displacement (6 complex sums) and of rd_i rd_j,
// rd_i t_j, rd_i u_j, rd_i n_j, u_i n_j and the identity in the symmetric
// stress (17); the vectors are multiplied in once per element.  That and the
// radial functions of bem_device.cuh take about 350 FP64 operations per point
// where contracting every tensor at every point took some 900; the FP64 pipe
// bounds the kernel (960 elements x 1000 points, NPG = 4, with stresses:
// 1078 us before).  A
// CTA reduces its 64 elements in a fixed order and writes one partial per
// (point, element chunk); k_interior_reduce sums the chunks in order, so the
// result does not depend on scheduling.
#include <cuda_runtime.h>

#include <algorithm>
#include <complex>
#include <vector>

#include "bem_internal.h"

namespace bem {

namespace {

constexpr int kIntThreads = 64;   // boundary elements per CTA, one per thread (128 left more of the last CTA idle)
constexpr int kIntOut = 12;       // 3 displacement + 9 stress components
constexpr int kIntAcc = 9;        // 3 displacement + 6 symmetric stress components

struct InteriorParams {
  int nbe, ng, l, chunks, want_stress;
  const double4* gq;   // [N][ng] Gauss point (x, y, z, w1*w2*|J|)
  const double4* eta;  // [N] unit normals
  const double4* pts;  // [l] interior points
  const double2* u;    // [3nbe] boundary displacements
  const double2* t;    // [3nbe] boundary tractions
  StokesConsts kc;
  zd zmu, lm;          // shear modulus ZGE, and lambda / mu
  double2* part;       // [l][chunks][12]
};

__device__ __forceinline__ zd ldz(const double2* p) {
  const double2 v = *p;
  return zd{v.x, v.y};
}

// Symmetric index (i <= j) -> 0..5: 00 01 02 11 12 22.
__host__ __device__ constexpr int sidx(int i, int j) {
  return i <= j ? (i == 0 ? j : (i == 1 ? 2 + j : 5)) : (j == 0 ? i : (j == 1 ? 2 + i : 5));
}

__global__ void __launch_bounds__(kIntThreads) k_interior(InteriorParams p) {
  __shared__ zd s_red[kIntThreads / 32][kIntAcc];
  __shared__ CexpTable tab;
  cexp_table_fill(tab);
  __syncthreads();
  const int K = blockIdx.y;
  const int J = blockIdx.x * kIntThreads + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  zd acc[kIntAcc];
#pragma unroll
  for (int i = 0; i < kIntAcc; ++i) acc[i] = zd{0.0, 0.0};

  if (J < p.nbe) {
    const StokesConsts& kc = p.kc;
    const double4 P = p.pts[K];
    const double4 nv = p.eta[J];
    const double n[3] = {nv.x, nv.y, nv.z};
    zd u[3], t[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      u[i] = ldz(&p.u[3 * J + i]);
      t[i] = ldz(&p.t[3 * J + i]);
    }
    zd un{0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 3; ++i) cfma(un, u[i], n[i]);
    const double4* q = p.gq + (size_t)J * p.ng;
    // displacement: sums of FHI, AA dr/dn, AA (rd.u), and the two rd_i
    // coefficients CAPPA (rd.t) and BB dr/dn (rd.u) + CC (n.u)
    zd sf{0.0, 0.0}, sa{0.0, 0.0}, sb{0.0, 0.0}, sk[3], sc[3];
    // stress: c4 (rd.t), c5 dr/dn (rd.u) + c9 (n.u) with rd_i rd_j; c3, c6
    // dr/dn, c6 (rd.u) with rd_i; c12; the identity's coefficient
    zd sp[6], s3[3], s6[3], s7[3], s12{0.0, 0.0}, sd{0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 3; ++i) sk[i] = sc[i] = s3[i] = s6[i] = s7[i] = zd{0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 6; ++i) sp[i] = zd{0.0, 0.0};
    const zd mu4 = p.zmu * kc.inv4pi;
    for (int g = 0; g < p.ng; ++g) {
      const double4 qq = q[g];
      const double r1 = qq.x - P.x, r2 = qq.y - P.y, r3 = qq.z - P.z;
      const double rr = fma(r1, r1, fma(r2, r2, r3 * r3));
      const double ir = rsqrt_fast(rr);  // r and 1/r from one reciprocal square root
      const double r = rr * ir;
      const double rd[3] = {r1 * ir, r2 * ir, r3 * ir};
      const double drn = rd[0] * n[0] + rd[1] * n[1] + rd[2] * n[2];
      const double wt = qq.w;
      const StokesRadial s = stokes_radial(kc, tab, r, ir);
      zd rt = t[0] * rd[0], ru = u[0] * rd[0];
      cfma(rt, t[1], rd[1]);
      cfma(rt, t[2], rd[2]);
      cfma(ru, u[1], rd[1]);
      cfma(ru, u[2], rd[2]);
      const zd rud = ru * drn;
      const double w3[3] = {wt * rd[0], wt * rd[1], wt * rd[2]};
      cfma(sf, s.fhi, wt);
      cfma(sa, s.aa, wt * drn);
      cfma(sb, s.aa * ru, wt);
      const zd kt = s.cappa * rt;
      zd bc = s.cc * un;
      cfma(bc, s.bbh * 2.0, rud);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        cfma(sk[i], kt, w3[i]);
        cfma(sc[i], bc, w3[i]);
      }
      if (p.want_stress) {
        // SIGMAEC's coefficients (src/Sigmaec.for:96-160).  With D = V - Ep/r
        // (the derivative of Ep) the second derivatives of the radial
        // functions enter only through
        //   FHI'' = zks W - 3 W/r + V/r + (7 Es - 5 Ep + 12 Q)/r^2
        //   CAPPA'' = zks W - zkp V - 5 (W - V)/r + (17 S + 36 Q)/r^2
        // and the dilatational terms reduce to lm D and lm zkp V:
        //   c2 = lm D, c8 = 3 lm D/r - lm zkp V, c10 = 4 CAPPA/r^2 - 4 lm D/r,
        //   c11 = -lm^2 zkp V.
        const double ir2 = ir * ir;
        const zd cr = s.cr, cr2 = cr * ir;
        const zd wv = s.w - s.v, ksw = kc.zks * s.w, kpv = kc.zkp * s.v;
        zd cdr = wv;  // CAPPA' = W - V - (3 CAPPA + S)/r
        cfma(cdr, cr, -3.0);
        cfma(cdr, s.s, -ir);
        zd fdr = s.w;  // FHI' = W - (CAPPA + Es)/r
        cfma(fdr, cr, -1.0);
        cfma(fdr, s.es, -ir);
        const zd fr1 = fdr * ir, cr1 = cdr * ir;
        zd f2 = ksw;
        cfma(f2, s.w, -3.0 * ir);
        cfma(f2, s.v, ir);
        zd t2 = s.es * 7.0;
        cfma(t2, s.ep, -5.0);
        cfma(t2, s.q, 12.0);
        cfma(f2, t2, ir2);
        zd k2 = ksw - kpv;
        cfma(k2, wv, -5.0 * ir);
        zd t3 = s.s * 17.0;
        cfma(t3, s.q, 36.0);
        cfma(k2, t3, ir2);
        const zd ld = p.lm * s.d, lv = p.lm * kpv;
        const zd c3 = s.aa;                 // FHI' - CAPPA/r
        zd c4 = cdr * 2.0;
        cfma(c4, cr, -4.0);
        zd c5 = k2 * 4.0;
        cfma(c5, cr1, -20.0);
        cfma(c5, cr2, 32.0);
        zd c6 = f2 - fr1;
        cfma(c6, cr1, -3.0);
        cfma(c6, cr2, 6.0);
        zd c9 = cr1 * 4.0;                  // 2 (c7 + c8), c7 = 2 CAPPA'/r - 4 CAPPA/r^2
        cfma(c9, cr2, -8.0);
        cfma(c9, ld, 6.0 * ir);
        cfma(c9, lv, -2.0);
        zd c1011 = cr2 * 4.0;
        cfma(c1011, ld, -4.0 * ir);
        cfma(c1011, -p.lm, lv);
        zd c12 = fr1 * 2.0;
        cfma(c12, cr2, -2.0);
        zd c12a = cr * 2.0;                 // c1 - c2
        c12a = c12a - ld;
        // rd_i rd_j: c4 (rd.t) / 4 pi - mu/(4 pi) (c5 dr/dn (rd.u) + c9 (n.u))
        zd h = c5 * rud;
        cfma(h, c9, un);
        zd pij = (c4 * rt) * kc.inv4pi;
        cfma(pij, -mu4, h);
        cfma(sp[0], pij, w3[0] * rd[0]);
        cfma(sp[1], pij, w3[0] * rd[1]);
        cfma(sp[2], pij, w3[0] * rd[2]);
        cfma(sp[3], pij, w3[1] * rd[1]);
        cfma(sp[4], pij, w3[1] * rd[2]);
        cfma(sp[5], pij, w3[2] * rd[2]);
        const zd c6d = c6 * drn, c6u = c6 * ru;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          cfma(s3[i], c3, w3[i]);
          cfma(s6[i], c6d, w3[i]);
          cfma(s7[i], c6u, w3[i]);
        }
        cfma(s12, c12, wt);
        zd id = c9 * rud;
        cfma(id, c1011, un);
        zd di = (c12a * rt) * kc.inv4pi;
        cfma(di, -mu4, id);
        cfma(sd, di, wt);
      }
    }
    // Displacements: U(i,:) . t - T(i,:) . u   (Solfund.for:50-60 layouts)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      zd ug = sf * t[i] - sk[i];
      zd th = sc[i];
      cfma(th, sa, u[i]);
      cfma(th, sb, n[i]);
      acc[i] = kc.zc0 * ug - kc.inv4pi * th;
    }
    if (p.want_stress) {
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j) {
          zd d = s3[i] * t[j];  // c3 (t_j rd_i + t_i rd_j)
          cfma(d, s3[j], t[i]);
          zd m = s6[i] * u[j];  // c6 dr/dn (u_j rd_i + u_i rd_j) + c6 (rd.u) (rd_i n_j + rd_j n_i)
          cfma(m, s6[j], u[i]);
          cfma(m, s7[i], n[j]);
          cfma(m, s7[j], n[i]);
          zd un2 = u[i] * n[j];  // c12 (u_i n_j + u_j n_i)
          cfma(un2, u[j], n[i]);
          cfma(m, s12, un2);
          zd a = sp[sidx(i, j)] - kc.inv4pi * d;
          cfma(a, mu4, m);
          if (i == j) a = a + sd;
          acc[3 + sidx(i, j)] = a;
        }
    }
  }
  // CTA reduction in a fixed order: warp tree, then the warps in order.
#pragma unroll
  for (int i = 0; i < kIntAcc; ++i) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      acc[i].re += __shfl_down_sync(0xffffffffu, acc[i].re, off);
      acc[i].im += __shfl_down_sync(0xffffffffu, acc[i].im, off);
    }
    if (lane == 0) s_red[warp][i] = acc[i];
  }
  __syncthreads();
  if (threadIdx.x < kIntOut) {
    const int o = threadIdx.x;
    // output o: 0..2 displacement, 3 + (i + 3j) stress component (i, j)
    const int a = o < 3 ? o : 3 + sidx((o - 3) % 3, (o - 3) / 3);
    zd sum = s_red[0][a];
#pragma unroll
    for (int w = 1; w < kIntThreads / 32; ++w) sum = sum + s_red[w][a];
    p.part[((size_t)K * p.chunks + blockIdx.x) * kIntOut + o] = make_double2(sum.re, sum.im);
  }
}

__global__ void k_interior_reduce(const double2* __restrict__ part, int l, int chunks, double2* out) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= l * kIntOut) return;
  const int K = idx / kIntOut, o = idx % kIntOut;
  double2 s = make_double2(0.0, 0.0);
  for (int c = 0; c < chunks; ++c) {
    const double2 v = part[((size_t)K * chunks + c) * kIntOut + o];
    s.x += v.x;
    s.y += v.y;
  }
  out[idx] = s;
}

}  // namespace

void release_interior(bem_ctx* ctx) {
  dev_free(ctx, ctx->int_pts);
  dev_free(ctx, ctx->int_ut);
  dev_free(ctx, ctx->int_part);
  dev_free(ctx, ctx->int_out);
  ctx->int_pts = nullptr;
  ctx->int_ut = nullptr;
  ctx->int_part = nullptr;
  ctx->int_out = nullptr;
  ctx->int_cap_l = ctx->int_cap_nn = 0;
}

int interior_points(bem_ctx* ctx, const double zge[2], const double zcs[2], const double zcp[2], double rho,
                    double fr, int l, const double* cxi, const double* cyi, const double* czi, const double* disp,
                    const double* trac, double* zdsol, double* zssol) {
  const Mesh& m = ctx->mesh;
  const int nbe = m.nbe, nn = 3 * nbe;
  if (l <= 0) return BEM_OK;
  const int chunks = (nbe + kIntThreads - 1) / kIntThreads;
  if ((size_t)l > ctx->int_cap_l || (size_t)nn > ctx->int_cap_nn) {
    release_interior(ctx);
    BEM_CUDA(ctx, dev_alloc(ctx, &ctx->int_pts, (size_t)l * sizeof(double4)));
    BEM_CUDA(ctx, dev_alloc(ctx, &ctx->int_ut, (size_t)2 * nn * sizeof(double2)));
    BEM_CUDA(ctx, dev_alloc(ctx, &ctx->int_part, (size_t)l * chunks * kIntOut * sizeof(double2)));
    BEM_CUDA(ctx, dev_alloc(ctx, &ctx->int_out, (size_t)l * kIntOut * sizeof(double2)));
    ctx->int_cap_l = (size_t)l;
    ctx->int_cap_nn = (size_t)nn;
  }
  std::vector<double4> pts((size_t)l);
  for (int k = 0; k < l; ++k) pts[k] = make_double4(cxi[k], cyi[k], czi[k], 0.0);
  BEM_CUDA(ctx, cudaMemcpyAsync(ctx->int_pts, pts.data(), (size_t)l * sizeof(double4), cudaMemcpyHostToDevice,
                                ctx->stream));
  BEM_CUDA(ctx, cudaMemcpyAsync(ctx->int_ut, disp, (size_t)nn * sizeof(double2), cudaMemcpyHostToDevice,
                                ctx->stream));
  BEM_CUDA(ctx, cudaMemcpyAsync(ctx->int_ut + nn, trac, (size_t)nn * sizeof(double2), cudaMemcpyHostToDevice,
                                ctx->stream));
  using cd = std::complex<double>;
  const cd zmu(zge[0], zge[1]), cp(zcp[0], zcp[1]);
  const cd lm = (cp * cp * rho - 2.0 * zmu) / zmu;  // Sigmaec.for: ZLAMB / ZMU
  InteriorParams p{};
  p.nbe = nbe;
  p.ng = m.ng;
  p.l = l;
  p.chunks = chunks;
  p.want_stress = zssol ? 1 : 0;
  p.gq = m.gq;
  p.eta = m.eta;
  p.pts = ctx->int_pts;
  p.u = ctx->int_ut;
  p.t = ctx->int_ut + nn;
  p.kc = make_consts(zge, zcs, zcp, fr);
  p.zmu = zd{zmu.real(), zmu.imag()};
  p.lm = zd{lm.real(), lm.imag()};
  p.part = ctx->int_part;
  k_interior<<<dim3(chunks, l), kIntThreads, 0, ctx->stream>>>(p);
  ctx->launches++;
  BEM_CUDA(ctx, cudaGetLastError());
  k_interior_reduce<<<(l * kIntOut + 255) / 256, 256, 0, ctx->stream>>>(ctx->int_part, l, chunks, ctx->int_out);
  ctx->launches++;
  BEM_CUDA(ctx, cudaGetLastError());
  std::vector<double2> out((size_t)l * kIntOut);
  BEM_CUDA(ctx, cudaMemcpyAsync(out.data(), ctx->int_out, out.size() * sizeof(double2), cudaMemcpyDeviceToHost,
                                ctx->stream));
  BEM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (int k = 0; k < l; ++k) {
    for (int i = 0; i < 3; ++i) {
      zdsol[2 * (3 * k + i)] = out[(size_t)k * kIntOut + i].x;
      zdsol[2 * (3 * k + i) + 1] = out[(size_t)k * kIntOut + i].y;
    }
    if (zssol)
      for (int mm = 0; mm < 9; ++mm) {
        zssol[2 * (9 * k + mm)] = out[(size_t)k * kIntOut + 3 + mm].x;
        zssol[2 * (9 * k + mm) + 1] = out[(size_t)k * kIntOut + 3 + mm].y;
      }
  }
  return BEM_OK;
}

}  // namespace bem

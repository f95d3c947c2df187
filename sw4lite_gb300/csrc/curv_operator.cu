// The curvilinear operator rhs4sgcurv (src/rhs4sgcurv.C:34, src/rhs4sgcurv_rev.C:34) on the
// rows away from the SBP top, either component layout, sm_103a, FP64: lu = L(u) for the
// kernel-level entry point.
//
// FP64 operations bound it (1.7 per clock and SM).  One thread per point that forms every
// coefficient and inner difference of its stencil anew takes about 1500; here each is
// formed once per point and shared, about 450 (and what the tiles' halos repeat):
//  * CTA = 32 x 6 columns marching up r through a 5-plane ring of the field in shared
//    memory; a cross term D_a(C D_b u) is an outer difference of per-point products
//    G = C D_b u, staged over a p or q halo or, along r, in a register queue (as in
//    curv_stage.cu, whose coefficients are prepared with the material; a kernel-level call
//    prepares and allocates nothing);
//  * the coefficients of a point's second differences along p and q are staged with the
//    products, the six along r ride a shared-memory queue of the own column;
//  * weights are formed from five coefficients, 10 operations for each kind.
// 130 x 121 x 64 points (tiles three quarters full): 1.35 ms against 2.86 ms; tiles of 8,
// 10 or 12 rows and one CTA per SM measured 1.37 to 1.39 ms.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "stencil.cuh"

namespace sw4g {
namespace {

constexpr int TX = 32, TY = 6, HALO = 2, CTAS = 2;
constexpr int PX = TX + 2 * HALO, PY = TY + 2 * HALO, PLANE = PX * PY;
constexpr int NTHREADS = TX * TY;
constexpr int NX = TY * PX, NY = PY * TX;

struct CurvOp {
   Box b;
   int k1, k2, kchunk;
   long long mcs, mps;  // metric component / point stride
   const double* __restrict__ u;
   const double* __restrict__ mu;
   const double* __restrict__ la;
   const double* __restrict__ met;
   const double* __restrict__ jac;
   const double* __restrict__ sx;
   const double* __restrict__ sy;
   double* __restrict__ lu;
};

struct Smem {
   double v[5][3][PLANE];       // field, ring of planes
   double gx[3][NX], gy[3][NY]; // products for the p and q outer differences
   double ax[2][NX];            // (2 mu + la) m1^2 sx, mu m1^2 sx along p,
   double ay[2][NY];            // ... sy along q
   double ar[5][6][NTHREADS];   // A00, A11, A22, A01, A02, A12 of the own column, ring
   double isx[PX], isy[PY];     // reciprocal stretching of the tile
};

// the products of a point: mu and la times m1^2, m2 m1, m3 m1, m4 m1
struct Coefs {
   double m11, l11, m21, l21, m31, l31, m41, l41;
};

__device__ __forceinline__ Coefs coefs(double m, double l, double m1, double m2, double m3, double m4)
{
   const double a = m * m1, b = l * m1;
   return Coefs{a * m1, b * m1, a * m2, b * m2, a * m3, b * m3, a * m4, b * m4};
}

// weights of the variable-coefficient second difference at the middle of five
// coefficients, times 6 (src/rhs4sgcurv_rev.C)
__device__ __forceinline__ void weights(const double a[5], double w[4])
{
   w[0] = fma(-0.75, a[2] + a[0], a[1]);
   w[1] = fma(3.0, a[2] + a[1], a[0] + a[3]);
   w[2] = fma(3.0, a[3] + a[2], a[1] + a[4]);
   w[3] = fma(-0.75, a[2] + a[4], a[3]);
}

__global__ void __launch_bounds__(NTHREADS, CTAS) curv_operator_kernel(CurvOp a)
{
   extern __shared__ __align__(16) unsigned char shared[];
   Smem& sm = *reinterpret_cast<Smem*>(shared);
   const Box& b = a.b;
   const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty;
   const int i0 = b.ib + 2 + blockIdx.x * TX, j0 = b.jb + 2 + blockIdx.y * TY;
   const int kbeg = a.k1 + blockIdx.z * a.kchunk;
   if (kbeg > a.k2) return;
   const int kend = min(kbeg + a.kchunk - 1, a.k2);
   const int i = i0 + tx, j = j0 + ty, ni = (int)b.ni;
   const bool active = i <= b.ie - 2 && j <= b.je - 2;
   const int own = (ty + HALO) * PX + tx + HALO;
   const int col = (i - b.ib) + ni * (j - b.jb);

   if (tid < PX) sm.isx[tid] = i0 - HALO + tid <= b.ie ? 1 / __ldg(a.sx + (i0 - HALO + tid - b.ib)) : 0.0;
   if (tid < PY) sm.isy[tid] = j0 - HALO + tid <= b.je ? 1 / __ldg(a.sy + (j0 - HALO + tid - b.jb)) : 0.0;
   const double sxi = active ? __ldg(a.sx + (i - b.ib)) : 1.0, syj = active ? __ldg(a.sy + (j - b.jb)) : 1.0;

   constexpr int kPre = (PLANE + NTHREADS - 1) / NTHREADS;
   double pv[kPre][3];
   int pcol[kPre];  // -1: beyond the tile or the array
#pragma unroll
   for (int r = 0; r < kPre; r++) {
      const int idx = tid + r * NTHREADS, gi = i0 - HALO + idx % PX, gj = j0 - HALO + idx / PX;
      pcol[r] = idx < PLANE && gi <= b.ie && gj <= b.je ? (gi - b.ib) + ni * (gj - b.jb) : -1;
   }
   auto fetch = [&](int kk) {
      const long long plane = b.nij * (long long)(kk - b.kb);
#pragma unroll
      for (int r = 0; r < kPre; r++)
#pragma unroll
         for (int c = 0; c < 3; c++) pv[r][c] = pcol[r] >= 0 ? __ldg(a.u + c * b.cs + b.ps * (plane + pcol[r])) : 0.0;
   };
   auto store = [&](int q) {
#pragma unroll
      for (int r = 0; r < kPre; r++)
         if (tid + r * NTHREADS < PLANE)
#pragma unroll
            for (int c = 0; c < 3; c++) sm.v[q][c][tid + r * NTHREADS] = pv[r][c];
   };
   auto metric = [&](int c, long long p) { return __ldg(a.met + c * a.mcs + a.mps * p); };

   // Own column at a plane whose field is in slot q: the r-r coefficients into their queue
   // and the products for the r outer difference.
   auto column = [&](int kk, int q, double g[3]) {
      if (!active) return;
      const long long p = b.nij * (long long)(kk - b.kb) + col;
      const double m = __ldg(a.mu + p), l = __ldg(a.la + p), m1 = metric(0, p), m2 = metric(1, p), m3 = metric(2, p),
                   m4 = metric(3, p);
      const double s2 = m2 * sxi, s3 = m3 * syj, q2 = s2 * s2, q3 = s3 * s3, q4 = m4 * m4, l2m = fma(2.0, m, l), lm = l + m;
      sm.ar[q][0][tid] = fma(l2m, q2, m * (q3 + q4));
      sm.ar[q][1][tid] = fma(l2m, q3, m * (q2 + q4));
      sm.ar[q][2][tid] = fma(l2m, q4, m * (q2 + q3));
      const double b2 = lm * m2;
      sm.ar[q][3][tid] = b2 * m3;
      sm.ar[q][4][tid] = b2 * m4;
      sm.ar[q][5][tid] = lm * m3 * m4;
      const Coefs c = coefs(m, l, m1, m2, m3, m4);
      const double isx = sm.isx[tx + HALO], isy = sm.isy[ty + HALO];
      double dp[3], dq[3];
#pragma unroll
      for (int n = 0; n < 3; n++) {
         const double* f = sm.v[q][n] + own;
         dp[n] = d1c(f[-2], f[-1], f[1], f[2]);
         dq[n] = d1c(f[-2 * PX], f[-PX], f[PX], f[2 * PX]);
      }
      const double x21 = c.m21 * sxi, y31 = c.m31 * syj;
      g[0] = isy * (fma(2.0, c.m21, c.l21) * sxi * dp[0] + c.m41 * dp[2]) + c.m31 * dp[1] + y31 * isx * dq[0] + c.l21 * dq[1];
      g[1] = isx * (fma(2.0, c.m31, c.l31) * syj * dq[1] + c.m41 * dq[2]) + c.l31 * dp[0] + x21 * isy * dp[1] + c.m21 * dq[0];
      g[2] = isy * (c.l41 * dp[0] + x21 * dp[2]) + isx * (y31 * dq[2] + c.l41 * dq[1]);
   };

   double gr[5][3];  // products for the r outer difference at planes k-2..k+2
#pragma unroll
   for (int q = 0; q < 5; q++) gr[q][0] = gr[q][1] = gr[q][2] = 0;
   // ring slots of planes k-2..k+2
   int qm2 = 0, qm1 = 1, q0 = 2, qp1 = 3, qp2 = 4;
   for (int q = 0; q < 4; q++) {
      fetch(kbeg - 2 + q);
      store(q);
   }
   fetch(kbeg + 2);
   __syncthreads();
#pragma unroll
   for (int q = 0; q < 4; q++) column(kbeg - 2 + q, q, gr[q + 1]);

   for (int k = kbeg; k <= kend; k++) {
      store(qp2);
      __syncthreads();
      if (k < kend) fetch(k + 3);
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
         for (int c = 0; c < 3; c++) gr[q][c] = gr[q + 1][c];
      column(k + 2, qp2, gr[4]);
      const long long plane = b.nij * (long long)(k - b.kb);
      const double(*vm2)[PLANE] = sm.v[qm2], (*vm1)[PLANE] = sm.v[qm1], (*v0)[PLANE] = sm.v[q0], (*vp1)[PLANE] = sm.v[qp1],
            (*vp2)[PLANE] = sm.v[qp2];
      auto dr = [&](int c, int s) { return d1c(vm2[c][s], vm1[c][s], vp1[c][s], vp2[c][s]); };
      // p products and coefficients over the x-extended rows, then q over the y-extended columns
#pragma unroll 1
      for (int idx = tid; idx < NX + NY; idx += NTHREADS) {
         const bool xp = idx < NX;
         const int q = xp ? idx : idx - NX;
         const int li = xp ? q % PX : q % TX + HALO, lj = xp ? q / PX + HALO : q / TX;
         const int gi = i0 - HALO + li, gj = j0 - HALO + lj, s = lj * PX + li;
         if (gi > b.ie || gj > b.je) continue;
         const long long p = plane + (gi - b.ib) + b.ni * (gj - b.jb);
         const Coefs c = coefs(__ldg(a.mu + p), __ldg(a.la + p), metric(0, p), metric(1, p), metric(2, p), metric(3, p));
         const double sxx = __ldg(a.sx + (gi - b.ib)), syy = __ldg(a.sy + (gj - b.jb));
         const double x21 = c.m21 * sxx, y31 = c.m31 * syy;
         const double r0 = dr(0, s), r1 = dr(1, s), r2 = dr(2, s);
         if (xp) {
            const double isy = sm.isy[lj];
            const double d0 = d1c(v0[0][s - 2 * PX], v0[0][s - PX], v0[0][s + PX], v0[0][s + 2 * PX]);
            const double d1 = d1c(v0[1][s - 2 * PX], v0[1][s - PX], v0[1][s + PX], v0[1][s + 2 * PX]);
            sm.gx[0][q] = c.l11 * d1 + isy * (fma(2.0, c.m21, c.l21) * sxx * r0 + c.l31 * syy * r1 + c.l41 * r2);
            sm.gx[1][q] = c.m11 * d0 + c.m31 * r0 + x21 * isy * r1;
            sm.gx[2][q] = isy * (c.m41 * r0 + x21 * r2);
            sm.ax[0][q] = fma(2.0, c.m11, c.l11) * sxx;
            sm.ax[1][q] = c.m11 * sxx;
         } else {
            const double isx = sm.isx[li];
            const double d0 = d1c(v0[0][s - 2], v0[0][s - 1], v0[0][s + 1], v0[0][s + 2]);
            const double d1 = d1c(v0[1][s - 2], v0[1][s - 1], v0[1][s + 1], v0[1][s + 2]);
            sm.gy[0][q] = c.m11 * d1 + y31 * isx * r0 + c.m21 * r1;
            sm.gy[1][q] = c.l11 * d0 + c.l21 * r0 + isx * (fma(2.0, c.m31, c.l31) * syy * r1 + c.l41 * r2);
            sm.gy[2][q] = isx * (y31 * r2 + c.m41 * r1);
            sm.ay[0][q] = fma(2.0, c.m11, c.l11) * syy;
            sm.ay[1][q] = c.m11 * syy;
         }
      }
      __syncthreads();

      if (active) {
         double r[3];
         const double isx = sm.isx[tx + HALO], isy = sm.isy[ty + HALO];
         // second differences along p and q: the first kind for the component along the axis
         double sp[3], sq[3];
#pragma unroll
         for (int ax = 0; ax < 2; ax++) {
            double w[2][4];
#pragma unroll
            for (int t = 0; t < 2; t++) {
               double c[5];
#pragma unroll
               for (int m = 0; m < 5; m++) c[m] = ax == 0 ? sm.ax[t][ty * PX + tx + m] : sm.ay[t][(ty + m) * TX + tx];
               weights(c, w[t]);
            }
            const int st = ax == 0 ? 1 : PX;
#pragma unroll
            for (int c = 0; c < 3; c++) {
               const double* f = v0[c] + own;
               const double* wc = w[c == ax ? 0 : 1];
               const double s = wc[0] * (f[-2 * st] - f[0]) + wc[1] * (f[-st] - f[0]) + wc[2] * (f[st] - f[0]) + wc[3] * (f[2 * st] - f[0]);
               if (ax == 0) sp[c] = s;
               else sq[c] = s;
            }
         }
         // along r: the symmetric matrix A
         double f[3][4], sd[3], so[3] = {0, 0, 0};
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const double f0 = v0[c][own];
            f[c][0] = vm2[c][own] - f0;
            f[c][1] = vm1[c][own] - f0;
            f[c][2] = vp1[c][own] - f0;
            f[c][3] = vp2[c][own] - f0;
         }
         const double rs[3] = {1.0, isy, isx};  // of A01, A02, A12
#pragma unroll
         for (int t = 0; t < 6; t++) {
            const double c[5] = {sm.ar[qm2][t][tid], sm.ar[qm1][t][tid], sm.ar[q0][t][tid], sm.ar[qp1][t][tid], sm.ar[qp2][t][tid]};
            double w[4];
            weights(c, w);
            auto sum = [&](int n) { return w[0] * f[n][0] + w[1] * f[n][1] + w[2] * f[n][2] + w[3] * f[n][3]; };
            if (t < 3) {
               sd[t] = sum(t);
            } else {
               const int x = t == 5 ? 1 : 0, y = t == 3 ? 1 : 2;
               so[x] = fma(rs[t - 3], sum(y), so[x]);
               so[y] = fma(rs[t - 3], sum(x), so[y]);
            }
         }
         const long long p = plane + col;
         const double ijac = sxi * syj / __ldg(a.jac + p), isxy = isx * isy;
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const double* gx = sm.gx[c] + ty * PX + tx;
            const double* gy = sm.gy[c] + ty * TX + tx;
            const double cross = d1c(gx[0], gx[1], gx[3], gx[4]) + d1c(gy[0], gy[TX], gy[3 * TX], gy[4 * TX]) +
                                 d1c(gr[0][c], gr[1][c], gr[3][c], gr[4][c]);
            r[c] = (isy * sp[c] + isx * sq[c] + isxy * sd[c] + so[c]) * (1.0 / 6) + cross * (1.0 / 144);
            a.lu[c * b.cs + b.ps * p] = r[c] * ijac;
         }
      }
      __syncthreads();
      const int next = qm2;
      qm2 = qm1;
      qm1 = q0;
      q0 = qp1;
      qp1 = qp2;
      qp2 = next;
   }
}

}  // namespace

int launch_curv_operator(const CurvSpec& s, int k1, int k2, double* lu, cudaStream_t st)
{
   if (k2 < k1) return kOk;
   CurvOp a;
   a.b = make_box(s.soa, s.ib, s.ie, s.jb, s.je, s.kb, s.ke);
   a.k1 = k1;
   a.k2 = k2;
   a.mcs = s.soa ? a.b.npts : 1;
   a.mps = s.soa ? 1 : 4;
   a.u = s.u;
   a.mu = s.mu;
   a.la = s.la;
   a.met = s.met;
   a.jac = s.jac;
   a.sx = s.strx;
   a.sy = s.stry;
   a.lu = lu;
   static_assert(sizeof(Smem) <= 113 * 1024, "two CTAs per SM");
   static std::atomic<int> resident[64];
   const int slots = resident_slots(resident, (const void*)curv_operator_kernel, NTHREADS, sizeof(Smem));
   if (slots < 1) return kCudaError;
   const int gx = blocks_for(s.ie - s.ib - 3, TX), gy = blocks_for(s.je - s.jb - 3, TY), nk = k2 - k1 + 1;
   a.kchunk = planes_per_cta((long long)gx * gy, nk, slots);
   const dim3 grid(gx, gy, (nk + a.kchunk - 1) / a.kchunk), block(TX, TY);
   curv_operator_kernel<<<grid, block, sizeof(Smem), st>>>(a);
   return launch_status();
}

}  // namespace sw4g

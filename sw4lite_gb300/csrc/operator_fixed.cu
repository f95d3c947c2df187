// The Cartesian operator rhs4sg (src/rhs4sg.C:38, src/rhs4sg_rev.C:44) on the centred rows,
// either component layout, sm_103a: lu = L(u) for the kernel-level entry point, with the
// sums in block fixed-point arithmetic on the integer pipes (fixed.cuh).
//
// The march, tiles and products are those of stage_fixed.cu.  A kernel-level call prepares
// nothing and allocates nothing, so the material comes with each plane: the products
// a = c s of a coefficient (mu, 2 mu + lambda) and the stretching along each axis are
// formed in FP64, aligned as integers like the field, and the weights of the second
// differences are integer sums of five of them.  Stretching factors of the point itself
// multiply finished sums and keep their own exponents: any finite profile is accepted.
//
// What bounds it: the integer pipes, about 3500 instructions a warp of 32 points, and 20
// FP64 operations a point, against 410 for one thread per point that forms every weight and
// inner difference anew: 256 x 200 x 150 points 1.74 ms against 5.97 ms.  The error against
// quad precision is 0.5 to 0.9 times that of the FP64 sums (smooth and random fields, profiles
// random and falling to 1e-4).
#include <algorithm>

#include "common.cuh"
#include "fixed.cuh"
#include "kernels.h"

namespace sw4g {
namespace {

constexpr int TX = 32, TY = 6, HALO = 2;
constexpr int PX = TX + 2 * HALO, PY = TY + 2 * HALO, PLANE = PX * PY;
constexpr int NTHREADS = TX * TY;
constexpr int NX = TY * PX, NY = PY * TX;
constexpr int kNone = -20000;  // below any exponent, in 16 bits

struct OpFixed {
   Box b;
   int k1, k2, kchunk;
   const double* __restrict__ u;
   const double* __restrict__ mu;
   const double* __restrict__ la;
   const double* __restrict__ sx;
   const double* __restrict__ sy;
   const double* __restrict__ sz;
   double* __restrict__ lu;
   double cof;  // 1 / (144 h^2)
};

struct Smem {
   i64 v[5][3][PLANE];   // field, ring of planes
   i64 gx[3][NX];        // products for the x outer difference: la (v_y + w_z), mu u_y, mu u_z
   i64 gy[3][NY];        // for the y outer difference: mu v_x, la (u_x + w_z), mu v_z
   i64 gz[4][3][NTHREADS];  // for the z one: mu w_x, mu w_y, la (u_x + v_y), four planes back
   i64 ax[2][NX];        // mu s_x, (2 mu + la) s_x of the plane along x,
   i64 ay[2][NY];        // ... s_y along y,
   i64 az[5][2][NTHREADS];  // ... s_z of the own column, ring of planes
   int gxe[NX], gye[NY], gze[4][NTHREADS];  // exponents: la's product << 16 | mu's
   short ve[5][PLANE], axe[NX], aye[NY], aze[5][NTHREADS];
   int bad;
};

// Products of one point for one outer direction: la f0 s0 + la f1 s1, mu m0 and mu m1 (as in
// stage_fixed.cu, the first with its own exponent).  c: mu and la as integers, ec their
// exponent - 1022.
struct Triple {
   i64 la, m0, m1;
   int el, em;
};

__device__ __forceinline__ int2 limbs(i64 c) { return make_int2((int)(c >> kSplit), (int)(c & kMask) << 5); }

__device__ __forceinline__ Triple products(i64 s0, i64 s1, i64 m0, i64 m1, int es0, int es1, i64 mu, i64 la, int ec,
                                           double f0, double f1)
{
   const int es = max(es0, es1), d0 = es - es0 + 1, d1 = es - es1 + 1;
   const int2 cm = limbs(mu);
   Triple t;
   t.m0 = mulc(sar(m0, d0), cm);
   t.m1 = mulc(sar(m1, d1), cm);
   t.em = es + ec;
   const Scale a(f0), b(f1);
   const int ea = es0 + a.e, eb = es1 + b.e, el = max(ea, eb);
   t.la = mulc(sar(a(s0 >> 1), el - ea) + sar(b(s1 >> 1), el - eb), limbs(la));
   t.el = el + ec;
   return t;
}

__device__ __forceinline__ int pack(int el, int em) { return (int)((unsigned)max(el, kNone) << 16 | (unsigned)(max(em, kNone) & 0xffff)); }
__device__ __forceinline__ int upper(int e) { return e >> 16; }
__device__ __forceinline__ int lower(int e) { return (short)(e & 0xffff); }

// The points of a column whose sums read a field or material value or a stretching factor
// that is not finite, set to NaN after the march (see stage_fixed.cu: of the material a
// component reads mu at every point of the three axes, lambda at its own point and along
// its own axis).
__device__ void mark_not_finite(const OpFixed& a, int i, int j, int kbeg, int kend)
{
   const Box& b = a.b;
   const long long st[3] = {1, b.ni, b.nij};
   const double* str[3] = {a.sx + (i - b.ib), a.sy + (j - b.jb), a.sz - b.kb};
   for (int k = kbeg; k <= kend; k++) {
      const long long p = pidx(b, i, j, k);
      auto bad = [&](int c, long long q) { return !isfinite(a.u[c * b.cs + b.ps * q]); };
      bool nan[3] = {bad(0, p), bad(1, p), bad(2, p)}, all = !isfinite(a.mu[p]) || !isfinite(a.la[p]);
      for (int ax = 0; ax < 3; ax++)
         for (int m = -2; m <= 2; m++) {
            all = all || !isfinite(str[ax][(ax == 2 ? k : 0) + m]);
            if (m == 0) continue;
            const long long q = p + m * st[ax];
            all = all || !isfinite(a.mu[q]);
            nan[ax] = nan[ax] || !isfinite(a.la[q]);
            for (int c = 0; c < 3; c++) {
               nan[c] = nan[c] || bad(c, q);
               if (c == ax) continue;
               for (int n = -2; n <= 2; n++) {
                  if (n == 0) continue;
                  nan[ax] = nan[ax] || bad(c, q + n * st[c]);
                  nan[c] = nan[c] || bad(ax, q + n * st[c]);
               }
            }
         }
      for (int c = 0; c < 3; c++)
         if (all || nan[c]) a.lu[c * b.cs + b.ps * p] = __longlong_as_double(0x7ff8000000000000LL);
   }
}

__global__ void __launch_bounds__(NTHREADS, 2) operator_fixed_kernel(OpFixed a)
{
   extern __shared__ __align__(16) unsigned char shared[];
   Smem& sm = *reinterpret_cast<Smem*>(shared);
   const Box& b = a.b;
   const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty;
   const int i0 = b.ib + 2 + blockIdx.x * TX, j0 = b.jb + 2 + blockIdx.y * TY;
   const int kbeg = a.k1 + blockIdx.z * a.kchunk;
   if (kbeg > a.k2) return;
   const int kend = min(kbeg + a.kchunk - 1, a.k2);
   const int i = i0 + tx, j = j0 + ty;
   const bool active = i <= b.ie - 2 && j <= b.je - 2, inside = i <= b.ie && j <= b.je;
   const int own = (ty + HALO) * PX + tx + HALO;
   const int ni = (int)b.ni, col = (i - b.ib) + ni * (j - b.jb);

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
      for (int r = 0; r < kPre; r++) {
         const int idx = tid + r * NTHREADS;
         if (idx < PLANE) {
            i64 m[3];
            int e;
            if (to_block(pv[r][0], pv[r][1], pv[r][2], m, e)) sm.bad = 1;
#pragma unroll
            for (int c = 0; c < 3; c++) sm.v[q][c][idx] = m[c];
            sm.ve[q][idx] = (short)e;
         }
      }
   };
   // c s of a point's two coefficients as integers
   auto put = [&](double m, double l, double s, i64* a0, i64* a1, short* e) {
      i64 t[3];
      int x;
      if (to_block(m * s, fma(2.0, m, l) * s, 0.0, t, x)) sm.bad = 1;
      *a0 = t[0];
      *a1 = t[1];
      *e = (short)x;
   };
   // the own column's material two planes ahead (z weights)
   auto put_z = [&](int kk, int q) {
      double m = 0, l = 0;
      if (inside) {
         const long long p = b.nij * (long long)(kk - b.kb) + col;
         m = __ldg(a.mu + p);
         l = __ldg(a.la + p);
      }
      put(m, l, __ldg(a.sz + kk - b.kb), &sm.az[q][0][tid], &sm.az[q][1][tid], &sm.aze[q][tid]);
   };

   const double sxi = inside ? __ldg(a.sx + (i - b.ib)) : 0.0, syj = inside ? __ldg(a.sy + (j - b.jb)) : 0.0;

   // the halo's products and x, y weights: rows -2, -1, TY, TY + 1 by the first four warps,
   // columns -2, -1, 32, 33 by the next 4 TY threads
   const bool halo = tid < 4 * TX + 4 * TY, yh = ty < 4;
   const int hrow = yh ? (ty < 2 ? ty : ty + TY) : ((tid - 4 * TX) >> 2) + HALO;
   const int hcl = yh ? tx + HALO : ((tx & 3) < 2 ? (tx & 3) : (tx & 3) + TX);
   int hcol = -1;
   double hin = 0, hst = 0;  // stretching of the point across and along its outer direction
   if (halo) {
      const int gi = i0 - HALO + hcl, gj = j0 - HALO + hrow;
      if (gi <= b.ie && gj <= b.je) {
         hcol = (gi - b.ib) + ni * (gj - b.jb);
         hin = yh ? __ldg(a.sx + (gi - b.ib)) : __ldg(a.sy + (gj - b.jb));
         hst = yh ? __ldg(a.sy + (gj - b.jb)) : __ldg(a.sx + (gi - b.ib));
      }
   }

   i64 pq[2][3];  // sums of planes k-2, k-1 and their exponents
   int pe[2][3];
#pragma unroll
   for (int q = 0; q < 4; q++) sm.gze[q][tid] = pack(kNone, kNone), sm.gz[q][0][tid] = sm.gz[q][1][tid] = sm.gz[q][2][tid] = 0;
#pragma unroll
   for (int q = 0; q < 2; q++)
#pragma unroll
      for (int c = 0; c < 3; c++) pe[q][c] = kNone, pq[q][c] = 0;

   if (tid == 0) sm.bad = 0;
   __syncthreads();
   // ring slots of planes k-2..k+2
   int qm2 = 3, qm1 = 4, q0 = 0, qp1 = 1, qp2 = 2;
   fetch(kbeg - 2);
   store(q0);
   put_z(kbeg - 2, q0);
   fetch(kbeg - 1);
   store(qp1);
   put_z(kbeg - 1, qp1);
   fetch(kbeg);
   for (int k = kbeg - 2; k <= kend + 2; k++) {
      const bool full = k >= kbeg && k <= kend;
      const long long plane = b.nij * (long long)(k - b.kb);
      // material of the plane, own point and halo
      i64 cm[3];
      int ec;
      {
         double m = 0, l = 0;
         if (inside) {
            m = __ldg(a.mu + plane + col);
            l = __ldg(a.la + plane + col);
         }
         if (to_block(m, l, 0.0, cm, ec)) sm.bad = 1;
         ec -= 1022;
         if (full) {
            const int qx = ty * PX + tx + HALO, qy = (ty + HALO) * TX + tx;
            put(m, l, sxi, &sm.ax[0][qx], &sm.ax[1][qx], &sm.axe[qx]);
            put(m, l, syj, &sm.ay[0][qy], &sm.ay[1][qy], &sm.aye[qy]);
         }
      }
      i64 hm[3] = {0, 0, 0};
      int he = 0;
      if (full && halo) {
         double m = 0, l = 0;
         if (hcol >= 0) {
            m = __ldg(a.mu + plane + hcol);
            l = __ldg(a.la + plane + hcol);
         }
         if (to_block(m, l, 0.0, hm, he)) sm.bad = 1;
         he -= 1022;
         if (yh) {
            const int q = hrow * TX + tx;
            put(m, l, hst, &sm.ay[0][q], &sm.ay[1][q], &sm.aye[q]);
         } else {
            const int q = (hrow - HALO) * PX + hcl;
            put(m, l, hst, &sm.ax[0][q], &sm.ax[1][q], &sm.axe[q]);
         }
      }
      if (k <= kend) {
         store(qp2);
         put_z(k + 2, qp2);
      }
      __syncthreads();
      if (k < kend) fetch(k + 3);
      const double szk = __ldg(a.sz + (k - b.kb));
      const i64* v0 = &sm.v[q0][0][0];
      const short* e0 = sm.ve[q0];
      int ex[4], ey[4], ez[4] = {0, 0, 0, 0};
#pragma unroll
      for (int m = 0; m < 4; m++) {
         const int s = m < 2 ? m - 2 : m - 1;
         ex[m] = e0[own + s];
         ey[m] = e0[own + s * PX];
      }
      const int Ex = max4(ex[0], ex[1], ex[2], ex[3]), Ey = max4(ey[0], ey[1], ey[2], ey[3]);
      int Ez = 0;
      i64 dx[3], dy[3], dz[3], S[3] = {0, 0, 0};
      int eS = kNone;
      const int qz[4] = {qm2, qm1, qp1, qp2};
      if (!full) {
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const i64* v = v0 + c * PLANE + own;
            if (c != 1) dx[c] = d1i(sar(v[-2], Ex - ex[0]), sar(v[-1], Ex - ex[1]), sar(v[1], Ex - ex[2]), sar(v[2], Ex - ex[3]));
            if (c != 0) dy[c] = d1i(sar(v[-2 * PX], Ey - ey[0]), sar(v[-PX], Ey - ey[1]), sar(v[PX], Ey - ey[2]), sar(v[2 * PX], Ey - ey[3]));
         }
      } else {
#pragma unroll
         for (int m = 0; m < 4; m++) ez[m] = sm.ve[qz[m]][own];
         Ez = max4(ez[0], ez[1], ez[2], ez[3]);
         const int eo = e0[own], E = max(max(Ex, Ey), max(Ez, eo));
         i64 x0[3];
#pragma unroll
         for (int c = 0; c < 3; c++) x0[c] = sar(v0[c * PLANE + own], E - eo);
#pragma unroll
         for (int ax = 0; ax < 3; ax++) {
            // weights: 4 a(q-1) - 3 (a(q) + a(q-2)) and 4 (a(q-2) + a(q+1)) + 12 (a(q) + a(q-1)) and
            // their mirrors, below 2^62, kept to 2^-5 and split at bit 30, so that an axis'
            // sums of products fit.  The centre's is minus the sum of the limbs.
            int ae[5];
            i64 av[2][5];
            const int qx = ty * PX + tx, qy = ty * TX + tx;
#pragma unroll
            for (int m = 0; m < 5; m++) {
               const int zq = m == 0 ? qm2 : m == 1 ? qm1 : m == 2 ? q0 : m == 3 ? qp1 : qp2;
               ae[m] = ax == 0 ? sm.axe[qx + m] : ax == 1 ? sm.aye[qy + m * TX] : sm.aze[zq][tid];
#pragma unroll
               for (int t = 0; t < 2; t++) av[t][m] = ax == 0 ? sm.ax[t][qx + m] : ax == 1 ? sm.ay[t][qy + m * TX] : sm.az[zq][t][tid];
            }
            const int ea = max(max4(ae[0], ae[1], ae[2], ae[3]), ae[4]);
            int2 w[2][4];
            int ch[2], cl[2];
#pragma unroll
            for (int t = 0; t < 2; t++) {
               i64 A[5];
#pragma unroll
               for (int m = 0; m < 5; m++) A[m] = sar(av[t][m], ea - ae[m]);
               const i64 o0 = A[2] + A[0], o1 = A[2] + A[4], i0s = A[2] + A[1], i1s = A[3] + A[2];
               const i64 W[4] = {(A[1] << 2) - (o0 + (o0 << 1)), (A[0] + A[3] + i0s + (i0s << 1)) << 2,
                                 (A[1] + A[4] + i1s + (i1s << 1)) << 2, (A[3] << 2) - (o1 + (o1 << 1))};
               i64 lows = 0;
               ch[t] = 0;
#pragma unroll
               for (int m = 0; m < 4; m++) {
                  const i64 r = (W[m] + 16) >> 5, h = (r + (1 << 29)) >> 30;
                  w[t][m] = make_int2((int)h, (int)(r - (h << 30)));
                  ch[t] -= w[t][m].x;
                  lows -= w[t][m].y;
               }
               const i64 h = (lows + (1 << 29)) >> 30;
               ch[t] += (int)h;
               cl[t] = (int)(lows - (h << 30));
            }
            const int Ea = ax == 0 ? Ex : ax == 1 ? Ey : Ez;
            i64 hh[3], xw[3], wx[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
               i64 x[4];
#pragma unroll
               for (int m = 0; m < 4; m++) {
                  const int o = m < 2 ? m - 2 : m - 1;
                  x[m] = ax == 0 ? v0[c * PLANE + own + o] : ax == 1 ? v0[c * PLANE + own + o * PX] : sm.v[qz[m]][c][own];
               }
               const int* e = ax == 0 ? ex : ax == 1 ? ey : ez;
               const i64 d = d1i(sar(x[0], Ea - e[0]), sar(x[1], Ea - e[1]), sar(x[2], Ea - e[2]), sar(x[3], Ea - e[3]));
               if (ax == 0) dx[c] = d;
               if (ax == 1) dy[c] = d;
               if (ax == 2) dz[c] = d;
               const int t = ax == c ? 1 : 0;
               hh[c] = xw[c] = wx[c] = 0;
#pragma unroll
               for (int m = 0; m < 5; m++) {
                  const i64 y = m < 4 ? sar(x[m], E - e[m]) : x0[c];
                  const int wh = m < 4 ? w[t][m].x : ch[t], wl = m < 4 ? w[t][m].y : cl[t];
                  const int xh = (int)(y >> kSplit), xl = (int)y & kMask;
                  hh[c] = madw(xh, wh, hh[c]);
                  xw[c] = madw(xh, wl, xw[c]);
                  wx[c] = madw(xl, wh, wx[c]);
               }
            }
            // the sum of a smooth field is a small part of its terms: shifted up to keep
            // its low bits
            auto top = [](i64 x) { return (unsigned)((int)(x >> 32) ^ (int)(x >> 63)); };
            const int up = min(max(__clz((int)(top(hh[0]) | top(hh[1]) | top(hh[2]))) - 3, 0), 24);
            i64 s[3];
#pragma unroll
            for (int c = 0; c < 3; c++) s[c] = (hh[c] << up) + sar(xw[c], 30 - up) + sar(wx[c], kSplit - up);
            // times the point's own factor; running sums to the larger exponent
            const Scale f(ax == 0 ? sxi : ax == 1 ? syj : szk);
            const int es = E + ea + f.e - up;
            if (ax == 0) {
               eS = es;
#pragma unroll
               for (int c = 0; c < 3; c++) S[c] = f(s[c]);
            } else {
               const int en = max(eS, es);
               const Round down(en - eS), add(en - es);
#pragma unroll
               for (int c = 0; c < 3; c++) S[c] = down(S[c]) + add(f(s[c]));
               eS = en;
            }
         }
         eS -= 1021;
      }

      // products of the own point
      const Triple z = products(dx[0], dy[1], dx[2], dy[2], Ex, Ey, cm[0], cm[1], ec, sxi, syj);
      if (full) {
         Triple t = products(dy[1], dz[2], dy[0], dz[0], Ey, Ez, cm[0], cm[1], ec, syj, szk);
         const int qx = ty * PX + tx + HALO;
         sm.gx[0][qx] = t.la;
         sm.gx[1][qx] = t.m0;
         sm.gx[2][qx] = t.m1;
         sm.gxe[qx] = pack(t.el, t.em);
         t = products(dx[0], dz[2], dx[1], dz[1], Ex, Ez, cm[0], cm[1], ec, sxi, szk);
         const int qy = (ty + HALO) * TX + tx;
         sm.gy[0][qy] = t.m0;
         sm.gy[1][qy] = t.la;
         sm.gy[2][qy] = t.m1;
         sm.gye[qy] = pack(t.el, t.em);
         if (halo) {
            const int s = hrow * PX + hcl, o = yh ? 1 : PX;
            int eh[4], ezh[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
               eh[m] = e0[s + (m < 2 ? m - 2 : m - 1) * o];
               ezh[m] = sm.ve[qz[m]][s];
            }
            const int Eh = max4(eh[0], eh[1], eh[2], eh[3]), Ezh = max4(ezh[0], ezh[1], ezh[2], ezh[3]);
#pragma unroll
            for (int m = 0; m < 4; m++) {
               eh[m] = Eh - eh[m];
               ezh[m] = Ezh - ezh[m];
            }
            const int cs = (yh ? 0 : PLANE) + s, cc = (yh ? PLANE : 0) + s;
            auto along = [&](int q) { return d1i(sar(v0[q - 2 * o], eh[0]), sar(v0[q - o], eh[1]), sar(v0[q + o], eh[2]), sar(v0[q + 2 * o], eh[3])); };
            auto down = [&](int q) {
               return d1i(sar(sm.v[qm2][0][q], ezh[0]), sar(sm.v[qm1][0][q], ezh[1]), sar(sm.v[qp1][0][q], ezh[2]), sar(sm.v[qp2][0][q], ezh[3]));
            };
            t = products(along(cs), down(2 * PLANE + s), along(cc), down(cc), Eh, Ezh, hm[0], hm[1], he, hin, szk);
            if (yh) {
               const int q = hrow * TX + tx;
               sm.gy[0][q] = t.m0;
               sm.gy[1][q] = t.la;
               sm.gy[2][q] = t.m1;
               sm.gye[q] = pack(t.el, t.em);
            } else {
               const int q = (hrow - HALO) * PX + hcl;
               sm.gx[0][q] = t.la;
               sm.gx[1][q] = t.m0;
               sm.gx[2][q] = t.m1;
               sm.gxe[q] = pack(t.el, t.em);
            }
         }
      }
      __syncthreads();

      // plane k: second differences and the x and y outer differences
      i64 P[3] = {0, 0, 0};
      int eP[3] = {kNone, kNone, kNone};
      if (full) {
         const i64* gx = &sm.gx[0][ty * PX + tx];
         const i64* gy = &sm.gy[0][ty * TX + tx];
         int hx[2][4], hy[2][4], Gx[2], Gy[2];  // mu's products, la's
#pragma unroll
         for (int m = 0; m < 4; m++) {
            const int n = m < 2 ? m : m + 1, x = sm.gxe[ty * PX + tx + n], y = sm.gye[(ty + n) * TX + tx];
            hx[0][m] = lower(x);
            hx[1][m] = upper(x);
            hy[0][m] = lower(y);
            hy[1][m] = upper(y);
         }
#pragma unroll
         for (int q = 0; q < 2; q++) {
            Gx[q] = max4(hx[q][0], hx[q][1], hx[q][2], hx[q][3]);
            Gy[q] = max4(hy[q][0], hy[q][1], hy[q][2], hy[q][3]);
#pragma unroll
            for (int m = 0; m < 4; m++) {
               hx[q][m] = Gx[q] - hx[q][m] + 3;
               hy[q][m] = Gy[q] - hy[q][m] + 3;
            }
         }
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const i64* x = gx + c * NX;
            const i64* y = gy + c * NY;
            const int lx = c == 0, ly = c == 1;
            const Scale fx(c == 0 ? sxi : c == 1 ? sxi * syj : sxi * szk), fy(c == 0 ? syj * sxi : c == 1 ? syj : syj * szk);
            const i64 cx = fx(d1i(sar(x[0], hx[lx][0]), sar(x[1], hx[lx][1]), sar(x[3], hx[lx][2]), sar(x[4], hx[lx][3])) >> 1);
            const i64 cy = fy(d1i(sar(y[0], hy[ly][0]), sar(y[TX], hy[ly][1]), sar(y[3 * TX], hy[ly][2]), sar(y[4 * TX], hy[ly][3])) >> 1);
            const int tx_ = Gx[lx] + fx.e, ty_ = Gy[ly] + fy.e;
            eP[c] = max(eS, max(tx_, ty_));
            const i64 s8 = Round(eP[c] - eS + 3)(S[c]);  // second differences carry 1/6, mixed terms 1/144
            P[c] = s8 + (s8 << 1) + Round(eP[c] - tx_ + 2)(cx) + Round(eP[c] - ty_ + 2)(cy);
         }
      }

      // plane k - 2: the z outer difference
      const int kp = k - 2;
      if (kp >= kbeg && active) {
         const int z0 = k & 3, z1 = (k + 1) & 3, z3 = (k + 3) & 3;  // planes k-4, k-3, k-1
         const int g0 = sm.gze[z0][tid], g1 = sm.gze[z1][tid], g3 = sm.gze[z3][tid];
         const double szp = __ldg(a.sz + (kp - b.kb));
         const i64 zn[3] = {z.m0, z.m1, z.la};
         const long long pp = col + b.nij * (long long)(kp - b.kb);
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const bool l = c == 2;
            const int h0 = l ? upper(g0) : lower(g0), h1 = l ? upper(g1) : lower(g1), h3 = l ? upper(g3) : lower(g3),
                      h4 = l ? z.el : z.em;
            const int Eg = max4(h0, h1, h3, h4);
            const Scale f(c == 0 ? szp * sxi : c == 1 ? szp * syj : szp);
            const i64 cz = f(d1i(sar(sm.gz[z0][c][tid], Eg - h0 + 3), sar(sm.gz[z1][c][tid], Eg - h1 + 3),
                                 sar(sm.gz[z3][c][tid], Eg - h3 + 3), sar(zn[c], Eg - h4 + 3)) >> 1);
            const int tz = Eg + f.e, eF = max(pe[0][c], tz);
            a.lu[c * b.cs + b.ps * pp] = a.cof * from_block(Round(eF - pe[0][c])(pq[0][c]) + Round(eF - tz + 2)(cz), eF - 1072);
         }
      }
      sm.gz[k & 3][0][tid] = z.m0;
      sm.gz[k & 3][1][tid] = z.m1;
      sm.gz[k & 3][2][tid] = z.la;
      sm.gze[k & 3][tid] = pack(z.el, z.em);
#pragma unroll
      for (int c = 0; c < 3; c++) {
         pq[0][c] = pq[1][c];
         pq[1][c] = P[c];
         pe[0][c] = pe[1][c];
         pe[1][c] = eP[c];
      }
      const int next = qm2;
      qm2 = qm1;
      qm1 = q0;
      q0 = qp1;
      qp1 = qp2;
      qp2 = next;
   }
   if (sm.bad && active) mark_not_finite(a, i, j, kbeg, kend);
}

}  // namespace

int launch_operator_fixed(const Box& b, int k1, int k2, double* lu, const double* u, const double* mu, const double* la,
                          double h, const double* sx, const double* sy, const double* sz, cudaStream_t s)
{
   if (k2 < k1) return kOk;
   OpFixed a;
   a.b = b;
   a.k1 = k1;
   a.k2 = k2;
   a.u = u;
   a.mu = mu;
   a.la = la;
   a.sx = sx;
   a.sy = sy;
   a.sz = sz;
   a.lu = lu;
   a.cof = 1.0 / (144 * h * h);
   static_assert(sizeof(Smem) <= 113 * 1024, "two CTAs per SM");
   // the opt-in shared-memory size is a per-device function attribute
   int dev = 0;
   if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return kCudaError;
   static int slots[64] = {};  // CTAs resident at once
   if (!slots[dev]) {
      int sms = 0;
      if (cudaFuncSetAttribute(operator_fixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)) != cudaSuccess ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
         return kCudaError;
      slots[dev] = std::max(1, sms) * resident_ctas((const void*)operator_fixed_kernel, NTHREADS, sizeof(Smem));
   }
   const int gx = blocks_for(b.ie - b.ib - 3, TX), gy = blocks_for(b.je - b.jb - 3, TY), nk = k2 - k1 + 1;
   a.kchunk = planes_per_cta((long long)gx * gy, nk, slots[dev]);
   const dim3 grid(gx, gy, (nk + a.kchunk - 1) / a.kchunk), block(TX, TY);
   operator_fixed_kernel<<<grid, block, sizeof(Smem), s>>>(a);
   return launch_status();
}

}  // namespace sw4g

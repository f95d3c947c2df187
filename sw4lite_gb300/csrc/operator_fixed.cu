// The Cartesian operator rhs4sg (src/rhs4sg.C:38, src/rhs4sg_rev.C:44) on the centred rows,
// either component layout, sm_103a: lu = L(u) for the kernel-level entry point, with the
// sums in block fixed-point arithmetic on the integer pipes (fixed.cuh).
//
// The march, tiles and products are those of stage_fixed.cu.  A kernel-level call prepares
// nothing and allocates nothing, so the material comes with each plane: the products
// a = c s of a coefficient (mu, 2 mu + lambda) and the stretching along each axis are
// formed in FP64, aligned as integers like the field, and the weights of the second
// differences are integer sums of five of them.  Stretching factors of the point itself
// multiply finished sums and keep their own exponents, as everything does that is not yet
// added: any finite profile is accepted, and each component, coefficient and axis keeps its
// digits beside others any power of two larger.
//
// What bounds it: the latency of twelve warps an SM and the integer pipes, about 5000
// instructions a warp of 32 points, and 20 FP64 operations a point, against 410 for one thread
// per point that forms every weight and inner difference anew: 256 x 200 x 150 points 2.15 ms
// against 5.97 ms.  (One exponent for a point's components and coefficients: 1.74 ms, and the
// smaller ones lost digits.)
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
   unsigned ve[5][PLANE];   // exponents of the three components (pack)
   short gxe[3][NX], gye[3][NY], gze[4][3][NTHREADS], axe[2][NX], aye[2][NY];
   int bad;
};

// Exponents of a point's three components in one word: 11 bits each for the first two, and the
// third, whose integer is brought to an even one, halved.
__device__ __forceinline__ unsigned pack(int e0, int e1, int e2) { return (unsigned)e2 << 21 | (unsigned)e1 << 11 | (unsigned)e0; }
__device__ __forceinline__ int unpack(int c, unsigned e)
{
   return c == 0 ? (int)(e & 0x7ff) : c == 1 ? (int)(e >> 11 & 0x7ff) : (int)(e >> 22) << 1;
}

__device__ __forceinline__ int2 limbs(i64 c) { return make_int2((int)(c >> kSplit), (int)(c & kMask) << 5); }

// The sum of two numbers, halved once so that sums of sums fit
__device__ __forceinline__ Num add(const Num& a, const Num& b)
{
   const int e = max(a.e, b.e);
   return Num{to_odd(a.m, e - a.e + 1) + to_odd(b.m, e - b.e + 1), e + 1};
}

// The points of a column whose sums read a field value, a product c s or a product of two
// stretching factors that is not finite, set to NaN after the march (see stage_fixed.cu: of the
// coefficients along an axis the component of the axis reads (2 mu + lambda) s and lambda, the
// others mu s and mu, and c s is not finite where c is not).
__device__ void mark_not_finite(const OpFixed& a, int i, int j, int kbeg, int kend)
{
   const Box& b = a.b;
   const long long st[3] = {1, b.ni, b.nij};
   const double* str[3] = {a.sx + (i - b.ib), a.sy + (j - b.jb), a.sz - b.kb};
   for (int k = kbeg; k <= kend; k++) {
      const long long p = pidx(b, i, j, k);
      auto bad = [&](int c, long long q) { return !isfinite(a.u[c * b.cs + b.ps * q]); };
      const double sx = str[0][0], sy = str[1][0], sz = str[2][k];
      const bool xy = !isfinite(sx * sy), xz = !isfinite(sx * sz), yz = !isfinite(sy * sz);
      bool nan[3] = {bad(0, p) || xy || xz, bad(1, p) || xy || yz, bad(2, p) || xz || yz};
      for (int ax = 0; ax < 3; ax++)
         for (int m = -2; m <= 2; m++) {
            const long long q = p + m * st[ax];
            const double s = str[ax][(ax == 2 ? k : 0) + m], mu = a.mu[q];
            const bool shear = !isfinite(mu * s), normal = !isfinite(fma(2.0, mu, a.la[q]) * s);
            for (int c = 0; c < 3; c++) {
               nan[c] = nan[c] || (c == ax ? normal : shear);
               if (m == 0) continue;
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
         if (nan[c]) a.lu[c * b.cs + b.ps * p] = __longlong_as_double(0x7ff8000000000000LL);
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
            int e[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
               i64 m;
               if (to_fixed(pv[r][c], m, e[c])) sm.bad = 1;
               if (c == 2) {
                  m >>= e[2] & 1;
                  e[2] += e[2] & 1;
               }
               sm.v[q][c][idx] = m;
            }
            sm.ve[q][idx] = pack(e[0], e[1], e[2]);
         }
      }
   };
   // c s of a point's two coefficients as integers
   auto put = [&](double m, double l, double s, i64* a0, i64* a1, int& e0, int& e1) {
      const bool b0 = to_fixed(m * s, *a0, e0), b1 = to_fixed(fma(2.0, m, l) * s, *a1, e1);
      if (b0 || b1) sm.bad = 1;
   };
   auto put_xy = [&](double m, double l, double s, i64* a0, i64* a1, short* e0, short* e1) {
      int x0, x1;
      put(m, l, s, a0, a1, x0, x1);
      *e0 = (short)x0;
      *e1 = (short)x1;
   };
   // the own column's material two planes ahead (z weights), exponents (2 mu + la) << 16 | mu
   int aze[5] = {0, 0, 0, 0, 0};  // of the planes k-2..k+2
   auto put_z = [&](int kk, int q) {
      double m = 0, l = 0;
      if (inside) {
         const long long p = b.nij * (long long)(kk - b.kb) + col;
         m = __ldg(a.mu + p);
         l = __ldg(a.la + p);
      }
      int e0, e1;
      put(m, l, __ldg(a.sz + kk - b.kb), &sm.az[q][0][tid], &sm.az[q][1][tid], e0, e1);
      return e1 << 16 | e0;
   };

   const double sxi = inside ? __ldg(a.sx + (i - b.ib)) : 0.0, syj = inside ? __ldg(a.sy + (j - b.jb)) : 0.0;

   const bool stx = !is_one(sxi), sty = !is_one(syj);

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

   Num pq[2][3];  // sums of planes k-2, k-1, value m * 2^(e - 1072)
#pragma unroll
   for (int c = 0; c < 3; c++) {
#pragma unroll
      for (int q = 0; q < 4; q++) sm.gze[q][c][tid] = (short)kNone, sm.gz[q][c][tid] = 0;
      pq[0][c] = pq[1][c] = Num{0, kNone};
   }

   if (tid == 0) sm.bad = 0;
   __syncthreads();
   // a product of two factors may overflow where their biased exponents add to this
   constexpr int kOver = 2 * 1023 + 1023;
   auto exponent = [](double s) { return (__double2hiint(s) >> 20) & 0x7ff; };
   const int exy = max(exponent(sxi), exponent(syj));
   if (exponent(sxi) + exponent(syj) >= kOver) sm.bad = 1;
   // ring slots of planes k-2..k+2
   int qm2 = 3, qm1 = 4, q0 = 0, qp1 = 1, qp2 = 2;
   fetch(kbeg - 2);
   store(q0);
   aze[2] = put_z(kbeg - 2, q0);
   fetch(kbeg - 1);
   store(qp1);
   aze[3] = put_z(kbeg - 1, qp1);
   fetch(kbeg);
   for (int k = kbeg - 2; k <= kend + 2; k++) {
      const bool full = k >= kbeg && k <= kend;
      const long long plane = b.nij * (long long)(k - b.kb);
      // material of the plane, own point and halo
      i64 cm[2];
      int ec[2];
      {
         double m = 0, l = 0;
         if (inside) {
            m = __ldg(a.mu + plane + col);
            l = __ldg(a.la + plane + col);
         }
         const bool b0 = to_fixed(m, cm[0], ec[0]), b1 = to_fixed(l, cm[1], ec[1]);
         if (b0 || b1) sm.bad = 1;
         if (full) {
            const int qx = ty * PX + tx + HALO, qy = (ty + HALO) * TX + tx;
            put_xy(m, l, sxi, &sm.ax[0][qx], &sm.ax[1][qx], &sm.axe[0][qx], &sm.axe[1][qx]);
            put_xy(m, l, syj, &sm.ay[0][qy], &sm.ay[1][qy], &sm.aye[0][qy], &sm.aye[1][qy]);
         }
      }
      i64 hm[2] = {0, 0};
      int he[2] = {0, 0};
      if (full && halo) {
         double m = 0, l = 0;
         if (hcol >= 0) {
            m = __ldg(a.mu + plane + hcol);
            l = __ldg(a.la + plane + hcol);
         }
         const bool b0 = to_fixed(m, hm[0], he[0]), b1 = to_fixed(l, hm[1], he[1]);
         if (b0 || b1) sm.bad = 1;
         if (yh) {
            const int q = hrow * TX + tx;
            put_xy(m, l, hst, &sm.ay[0][q], &sm.ay[1][q], &sm.aye[0][q], &sm.aye[1][q]);
         } else {
            const int q = (hrow - HALO) * PX + hcl;
            put_xy(m, l, hst, &sm.ax[0][q], &sm.ax[1][q], &sm.axe[0][q], &sm.axe[1][q]);
         }
      }
      if (k <= kend) {
         store(qp2);
         aze[4] = put_z(k + 2, qp2);
      }
      __syncthreads();
      if (k < kend) fetch(k + 3);
      const double szk = __ldg(a.sz + (k - b.kb));
      if (exy + exponent(szk) >= kOver) sm.bad = 1;
      const i64* v0 = &sm.v[q0][0][0];
      const unsigned* e0 = sm.ve[q0];
      const int qz[4] = {qm2, qm1, qp1, qp2};
      // differences of component c at the point s along an axis of the plane (stride o) or
      // across the planes
      auto along = [&](int c, int s, int o, bool& tiny) {
         const i64* v = v0 + c * PLANE + s;
         const int x0 = unpack(c, e0[s - 2 * o]), x1 = unpack(c, e0[s - o]), x2 = unpack(c, e0[s + o]), x3 = unpack(c, e0[s + 2 * o]);
         return difference(v[-2 * o], v[-o], v[o], v[2 * o], x0, x1, x2, x3, max4(x0, x1, x2, x3), tiny);
      };
      auto down = [&](int c, int s, bool& tiny) {
         const int x0 = unpack(c, sm.ve[qm2][s]), x1 = unpack(c, sm.ve[qm1][s]), x2 = unpack(c, sm.ve[qp1][s]), x3 = unpack(c, sm.ve[qp2][s]);
         return difference(sm.v[qm2][c][s], sm.v[qm1][c][s], sm.v[qp1][c][s], sm.v[qp2][c][s], x0, x1, x2, x3, max4(x0, x1, x2, x3), tiny);
      };

      Num D[3][3];  // differences along x, y, z of the components
      bool few = false;  // one of them has lost nearly all its bits
      Num S[3] = {{0, kNone}, {0, kNone}, {0, kNone}};
      if (!full) {
         D[0][0] = along(0, own, 1, few);
         D[0][2] = along(2, own, 1, few);
         D[1][1] = along(1, own, PX, few);
         D[1][2] = along(2, own, PX, few);
         if (few) rest(D[0][0]), rest(D[0][2]), rest(D[1][1]), rest(D[1][2]);
      } else {
         const int qx = ty * PX + tx, qy = ty * TX + tx;
#pragma unroll
         for (int ax = 0; ax < 3; ax++) {
            unsigned en[4];  // exponents of the four neighbours
#pragma unroll
            for (int m = 0; m < 4; m++) {
               const int s = m < 2 ? m - 2 : m - 1;
               en[m] = ax == 0 ? e0[own + s] : ax == 1 ? e0[own + s * PX] : sm.ve[qz[m]][own];
            }
            const double f = ax == 0 ? sxi : ax == 1 ? syj : szk;
#pragma unroll
            for (int t = 0; t < 2; t++) {
               // weights: 4 a(q-1) - 3 (a(q) + a(q-2)) and 4 (a(q-2) + a(q+1)) + 12 (a(q) + a(q-1)) and
               // their mirrors, four times the operator's, below 2^62, kept to 2^-5 and split at bit
               // 30; each with the exponent of the largest a that it reads
               i64 A[5];
               int ae[5];
#pragma unroll
               for (int m = 0; m < 5; m++) {
                  const int zq = m == 0 ? qm2 : m == 1 ? qm1 : m == 2 ? q0 : m == 3 ? qp1 : qp2;
                  ae[m] = ax == 0 ? sm.axe[t][qx + m] : ax == 1 ? sm.aye[t][qy + m * TX] : t == 1 ? aze[m] >> 16 : aze[m] & 0xffff;
                  A[m] = ax == 0 ? sm.ax[t][qx + m] : ax == 1 ? sm.ay[t][qy + m * TX] : sm.az[zq][t][tid];
               }
               int2 w[4];
               int we[4];
#pragma unroll
               for (int m = 0; m < 4; m++) {
                  const int far = m == 0 ? 0 : 4;
                  i64 W;
                  if (m == 0 || m == 3) {
                     const int e = max(max(ae[2], ae[far]), ae[m == 0 ? 1 : 3]);
                     const i64 o = sar(A[2], e - ae[2]) + sar(A[far], e - ae[far]);
                     W = (sar(A[m == 0 ? 1 : 3], e - ae[m == 0 ? 1 : 3]) << 2) - (o + (o << 1));
                     we[m] = e;
                  } else {
                     const int q = m - 1;  // a(q), a(q + 3) with weight 1, the two between with 3
                     const int e = max4(ae[q], ae[q + 1], ae[q + 2], ae[q + 3]);
                     const i64 i = sar(A[q + 1], e - ae[q + 1]) + sar(A[q + 2], e - ae[q + 2]);
                     W = (sar(A[q], e - ae[q]) + sar(A[q + 3], e - ae[q + 3]) + i + (i << 1)) << 2;
                     we[m] = e;
                  }
                  const i64 r = (W + 16) >> 5, h = (r + (1 << 29)) >> 30;
                  w[m] = make_int2((int)h, (int)(r - (h << 30)));
               }
#pragma unroll
               for (int c = 0; c < 3; c++) {
                  if ((ax == c) != (t == 1)) continue;
                  int e[4];
#pragma unroll
                  for (int m = 0; m < 4; m++) e[m] = unpack(c, en[m]);
                  const int E = max4(e[0], e[1], e[2], e[3]), eo = unpack(c, e0[own]), Ec = max(E, eo);
                  i64 x[4];
#pragma unroll
                  for (int m = 0; m < 4; m++) {
                     const int s = m < 2 ? m - 2 : m - 1;
                     x[m] = sar(ax == 0 ? v0[c * PLANE + own + s] : ax == 1 ? v0[c * PLANE + own + s * PX] : sm.v[qz[m]][c][own], E - e[m]);
                  }
                  D[ax][c] = normal(d1i(x[0], x[1], x[2], x[3]), E, few);
                  // differences to the own value, aligned by the size of their products with the weights,
                  // the largest brought to bit 57
                  const i64 x0 = sar(v0[c * PLANE + own], Ec - eo);
                  int pe[4];
                  bool tiny = false;
#pragma unroll
                  for (int m = 0; m < 4; m++) {
                     const i64 d = sar(x[m], Ec - E) - x0;
                     const int n = headroom<57>(d);
                     x[m] = d << n;
                     pe[m] = we[m] - n;
                     tiny = tiny || (unsigned)((int)(d >> 32) + 1) < 2u;  // its upper word is sign
                  }
                  if (tiny)
#pragma unroll
                     for (int m = 0; m < 4; m++) {
                        const int n = max(__clzll(x[m] ^ (x[m] >> 63)) - 6, 0), e = pe[m];
                        pe[m] = x[m] == 0 ? kNone : e - n;
                        x[m] <<= n;
                     }
                  const int ep = max4(pe[0], pe[1], pe[2], pe[3]);
                  i64 hh = 0, xw = 0, wx = 0;
#pragma unroll
                  for (int m = 0; m < 4; m++) {
                     const i64 y = sar(x[m], ep - pe[m]);
                     const int xh = (int)(y >> 27), xl = (int)y & ((1 << 27) - 1);
                     hh = madw(xh, w[m].x, hh);
                     xw = madw(xh, w[m].y, xw);
                     wx = madw(xl, w[m].x, wx);
                  }
                  // the sum of a smooth field is a small part of its terms: with as many of the
                  // lower bits as there is room for
                  const int up = min(headroom<60>(hh), 27);  // |s| < 2^62, as Scale takes it
                  const i64 s = (hh << up) + to_odd((xw >> 3) + wx, 27 - up);
                  // times the point's own factor
                  Num T = {s, s == 0 ? kNone : Ec + ep - up};
                  if (!is_one(f)) T = stretched<true>(T, f);
                  S[c] = ax == 0 ? T : add(S[c], T);
               }
            }
         }
#pragma unroll
         for (int c = 0; c < 3; c++) S[c].e = max(S[c].e - 1020, kNone);
      }

      if (full && few)
#pragma unroll
         for (int ax = 0; ax < 3; ax++)
#pragma unroll
            for (int c = 0; c < 3; c++) rest(D[ax][c]);
      // products of the own point
      const int2 lm = limbs(cm[0]), ll = limbs(cm[1]);
      const int emu = ec[0] - 1022, ela = ec[1] - 1022;
      const Triple z = products<true>(D[0][0], D[1][1], D[0][2], D[1][2], lm, emu, ll, ela, sxi, syj);
      if (full) {
         auto to_x = [&](const Triple& t, int q) {
            sm.gx[0][q] = t.la.m;
            sm.gx[1][q] = t.m0.m;
            sm.gx[2][q] = t.m1.m;
            sm.gxe[0][q] = (short)max(t.la.e, kNone);
            sm.gxe[1][q] = (short)max(t.m0.e, kNone);
            sm.gxe[2][q] = (short)max(t.m1.e, kNone);
         };
         auto to_y = [&](const Triple& t, int q) {
            sm.gy[0][q] = t.m0.m;
            sm.gy[1][q] = t.la.m;
            sm.gy[2][q] = t.m1.m;
            sm.gye[0][q] = (short)max(t.m0.e, kNone);
            sm.gye[1][q] = (short)max(t.la.e, kNone);
            sm.gye[2][q] = (short)max(t.m1.e, kNone);
         };
         to_x(products<true>(D[1][1], D[2][2], D[1][0], D[2][0], lm, emu, ll, ela, syj, szk), ty * PX + tx + HALO);
         to_y(products<true>(D[0][0], D[2][2], D[0][1], D[2][1], lm, emu, ll, ela, sxi, szk), (ty + HALO) * TX + tx);
         if (halo) {
            const int s = hrow * PX + hcl, o = yh ? 1 : PX, cs = yh ? 0 : 1, cc = 1 - cs;
            bool some = false;
            Num d0 = along(cs, s, o, some), d1 = down(2, s, some), d2 = along(cc, s, o, some), d3 = down(cc, s, some);
            if (some) rest(d0), rest(d1), rest(d2), rest(d3);
            const Triple t = products<true>(d0, d1, d2, d3, limbs(hm[0]), he[0] - 1022, limbs(hm[1]), he[1] - 1022, hin, szk);
            if (yh) to_y(t, hrow * TX + tx);
            else to_x(t, (hrow - HALO) * PX + hcl);
         }
      }
      __syncthreads();

      // plane k: second differences and the x and y outer differences
      Num P[3] = {{0, kNone}, {0, kNone}, {0, kNone}};
      if (full) {
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const i64* x = &sm.gx[c][ty * PX + tx];
            const i64* y = &sm.gy[c][ty * TX + tx];
            const short* xe = &sm.gxe[c][ty * PX + tx];
            const short* ye = &sm.gye[c][ty * TX + tx];
            const int hx[4] = {xe[0], xe[1], xe[3], xe[4]}, hy[4] = {ye[0], ye[TX], ye[3 * TX], ye[4 * TX]};
            Num cx = outer(x[0], x[1], x[3], x[4], hx[0], hx[1], hx[2], hx[3], max4(hx[0], hx[1], hx[2], hx[3]));
            Num cy = outer(y[0], y[TX], y[3 * TX], y[4 * TX], hy[0], hy[1], hy[2], hy[3], max4(hy[0], hy[1], hy[2], hy[3]));
            if (stx || sty || !is_one(szk)) {
               cx = stretched<true>(cx, c == 0 ? sxi : c == 1 ? sxi * syj : sxi * szk);
               cy = stretched<true>(cy, c == 0 ? syj * sxi : c == 1 ? syj : syj * szk);
            }
            P[c].e = max(S[c].e, max(cx.e, cy.e));
            const i64 s8 = to_odd(S[c].m, P[c].e - S[c].e + 3);  // second differences carry 1/6, mixed terms 1/144
            P[c].m = s8 + (s8 << 1) + to_odd(cx.m, P[c].e - cx.e + 2) + to_odd(cy.m, P[c].e - cy.e + 2);
         }
      }

      // plane k - 2: the z outer difference
      const int kp = k - 2;
      if (kp >= kbeg && active) {
         const int z0 = k & 3, z1 = (k + 1) & 3, z3 = (k + 3) & 3;  // planes k-4, k-3, k-1
         const double szp = __ldg(a.sz + (kp - b.kb));
         const Num zn[3] = {z.m0, z.m1, z.la};
         const long long pp = col + b.nij * (long long)(kp - b.kb);
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const int h0 = sm.gze[z0][c][tid], h1 = sm.gze[z1][c][tid], h3 = sm.gze[z3][c][tid], h4 = zn[c].e;
            Num g = outer(sm.gz[z0][c][tid], sm.gz[z1][c][tid], sm.gz[z3][c][tid], zn[c].m, h0, h1, h3, h4, max4(h0, h1, h3, h4));
            if (stx || sty || !is_one(szp)) g = stretched<true>(g, c == 0 ? szp * sxi : c == 1 ? szp * syj : szp);
            const int eF = max(pq[0][c].e, g.e);
            bool low;
            const double lu = from_block(to_odd(pq[0][c].m, eF - pq[0][c].e) + to_odd(g.m, eF - g.e + 2), eF - 1072, low);
            a.lu[c * b.cs + b.ps * pp] = (low ? lowered(a.cof) : a.cof) * lu;
         }
      }
      const Num zn[3] = {z.m0, z.m1, z.la};
#pragma unroll
      for (int c = 0; c < 3; c++) {
         sm.gz[k & 3][c][tid] = zn[c].m;
         sm.gze[k & 3][c][tid] = (short)max(zn[c].e, kNone);
         pq[0][c] = pq[1][c];
         pq[1][c] = P[c];
      }
#pragma unroll
      for (int q = 0; q < 4; q++) aze[q] = aze[q + 1];
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
   static std::atomic<int> resident[64];
   const int slots = resident_slots(resident, (const void*)operator_fixed_kernel, NTHREADS, sizeof(Smem));
   if (slots < 1) return kCudaError;
   const int gx = blocks_for(b.ie - b.ib - 3, TX), gy = blocks_for(b.je - b.jb - 3, TY), nk = k2 - k1 + 1;
   a.kchunk = planes_per_cta((long long)gx * gy, nk, slots);
   const dim3 grid(gx, gy, (nk + a.kchunk - 1) / a.kchunk), block(TX, TY);
   operator_fixed_kernel<<<grid, block, sizeof(Smem), s>>>(a);
   return launch_status();
}

}  // namespace sw4g

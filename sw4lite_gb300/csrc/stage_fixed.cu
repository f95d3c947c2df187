// FP64 stage kernels of the elastic time step on Cartesian grids, sm_103a, with the
// stencil sums in block fixed-point arithmetic on the integer pipes (fixed.cuh).
//
// One launch computes, for every centred row k1..k2 of the interior,
//   form 0  out = 2u - um + coef/rho * L(u)                            (predictor)
//   form 1  out = up + coef/rho * L(up - 2u + um)                      (corrector)
//   form 2  out = 2u - um + coef/rho * L(up)                           (adjoint)
// with L the divergence of stress of the reference's rhs4sg (src/rhs4sg_rev.C:111-348),
// in place of the reference's RHSPredCU_center / evalDpDmInTimeCU / RHSCorrCU_center
// (src/EW_cuda.C:1228-1509); the supergrid damping of forms 1 and 2 follows on the layers
// alone (damping_layers.cu).
//
//  * CTA = 32 x 6 columns marching up z through a 5-plane ring of the stage field in
//    shared memory, 2-point halo: per point three 57-bit integers with one exponent.
//    Two CTAs per SM at 168 registers: the 128 registers of 2 x 256 threads spill into an
//    L1 that the shared memory leaves at a few KB (predictor at 512^3 19.6 ms, 32 x 6
//    15.2 ms, one CTA of 32 x 12 18.3 ms).
//  * Every sum has the exponent of the largest value it reads: per axis for the centred
//    differences and the second differences along it, their largest for the point's sum.
//  * The second differences' 24 weights per point (stretching folded in) are integers
//    with one exponent per point, prepared once per material and stored by blocks of 32
//    points, so that a warp reads 24 contiguous lines; each warp copies its own
//    asynchronously, two axes ahead of their use.
//  * A mixed derivative is the outer difference of a product G = c * D f formed once per
//    point.  The nine first differences of a point serve its second differences' values
//    and all three of its products: those for the x and y outer differences go to shared
//    memory, those for the z outer difference into a register queue, so a plane is
//    finished two planes later, when the last product along z is known.
//  * FP64 remains in forming up - 2u + um and in the update.
// What bounds them: the integer pipes (about 2300 instructions a warp of 32 points, half of
// them at half rate), the corrector also the FP64 operations of its stage field.  At 512^3
// the predictor takes 15.2 ms and the corrector 22.5 ms with the damping (28.2 ms with the
// damping inside the kernel), against 40.6 and 53.8 ms with the sums in FP64 (stage_fused.cu), whose 160 and 198 FP64 operations a point saturate the
// 1.7 that an SM completes per clock.  Against quad precision the levels after 50 steps are off
// by 0.5 to 0.65 times what they were.
#include <algorithm>

#include "common.cuh"
#include "fixed.cuh"
#include "kernels.h"
#include "stencil.cuh"

namespace sw4g {
namespace {

constexpr int TX = kFixedBlock, TY = 6, HALO = 2;
constexpr int PX = TX + 2 * HALO;  // 36
constexpr int PY = TY + 2 * HALO;
constexpr int PLANE = PX * PY;
constexpr int NTHREADS = TX * TY;
constexpr int NX = TY * PX, NY = PY * TX;  // products for the x and y outer differences

struct FixedArgs {
   int ib, ie, jb, je, kb, ke;
   long long ni, nij, npts;
   int k1, k2, kchunk;
   const double* __restrict__ u;
   const double* __restrict__ um;
   const double* __restrict__ up;
   double* __restrict__ out;
   const double* __restrict__ irho;
   const int2* __restrict__ w;    // second-difference weights, by blocks of 32 points
   const int4* __restrict__ c;    // lambda and mu coefficients of the mixed terms
   const int* __restrict__ e;     // exponents of both: weights << 16 | coefficients
   const int* __restrict__ bad;   // nonzero: the material is not finite everywhere
   const double* __restrict__ mu;  // read where the material is not finite
   const double* __restrict__ la;
   int wbx, wny;                  // blocks per row and rows per plane of w
   const double* __restrict__ sx;
   const double* __restrict__ sy;
   const double* __restrict__ sz;
   double coef;
   int* emax;
};

// Exponent of coefficients beyond the range
constexpr int kCoefBad = 0x7fff;

struct Smem {
   i64 v[5][3][PLANE];         // stage field, ring of planes
   i64 gx[3][NX];              // products for the x outer difference: la (v_y + w_z), mu u_y, mu u_z
   i64 gy[3][NY];              // for the y outer difference: mu v_x, la (u_x + w_z), mu v_z
   int2 w[TY][2][8][TX];       // weights of one axis for a row of points, two stages per warp
   i64 gz[4][3][NTHREADS];     // products for the z outer difference: mu w_x, mu w_y, la (u_x + v_y)
   int gze[4][NTHREADS];       // of the four planes before, each thread its own column
   int ve[5][PLANE];
   int gxe[NX], gye[NY];
   int bad;                    // a value of the stage field or of the material is not finite
};

__device__ __forceinline__ bool is_one(double x) { return __double_as_longlong(x) == 0x3ff0000000000000LL; }

// Products of one point for one outer direction; la multiplies the sum of the two
// differences s0, s1 (exponents es0, es1; stretching factors f0, f1), mu the differences
// m0 (exponent es0) and m1 (exponent es1); value g * 2^(e - 1078).
struct Triple {
   i64 la, m0, m1;
   int e;
};

__device__ __forceinline__ Triple products(i64 s0, i64 s1, i64 m0, i64 m1, int es0, int es1, int4 c, int ec,
                                           double f0, double f1)
{
   const int es = max(es0, es1);
   const int d0 = es - es0 + 1, d1 = es - es1 + 1;
   i64 a = sar(s0, d0), b = sar(s1, d1);
   if (!is_one(f0)) a = Factor(f0)(a);
   if (!is_one(f1)) b = Factor(f1)(b);
   Triple t;
   t.la = mulc(a + b, make_int2(c.z, c.w));
   t.m0 = mulc(sar(m0, d0), make_int2(c.x, c.y));
   t.m1 = mulc(sar(m1, d1), make_int2(c.x, c.y));
   t.e = es + ec;
   return t;
}

__device__ __forceinline__ void copy16(void* dst, const void* src)
{
   asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                : "memory");
}

// The stage field: u, up - 2u + um or up
template <int FORM>
__device__ __forceinline__ double stage_value(const FixedArgs& a, long long q)
{
   // fma: 2 * x compiles to x + x, an FP64 operation more
   if (FORM == 1) return fma(-2.0, __ldg(a.u + q), __ldg(a.up + q)) + __ldg(a.um + q);
   return __ldg((FORM == 0 ? a.u : a.up) + q);
}

// The points of a column whose sums read a value that is not finite, set to NaN after the
// march: the sums themselves took it as zero.  A component's second differences read the
// component along the three axes; its mixed terms read another component at the points
// off both axes in the plane of the two.  Of the material a component reads mu at every
// point of the three axes, lambda at its own point and along its own axis.
// Returns the exponent field of NaN if there was such a point.
template <int FORM>
__device__ int mark_not_finite(const FixedArgs& a, int i, int j, int kbeg, int kend)
{
   int em = 0;
   for (int k = kbeg; k <= kend; k++) {
      const long long p = (i - a.ib) + a.ni * (j - a.jb) + a.nij * (long long)(k - a.kb);
      const long long st[3] = {1, a.ni, a.nij};
      auto bad = [&](int c, long long q) {
         return !isfinite(stage_value<FORM>(a, q + c * a.npts));
      };
      bool coef = !isfinite(a.mu[p]) || !isfinite(a.la[p]), all = coef;
      bool nan[3] = {bad(0, p), bad(1, p), bad(2, p)};
      for (int ax = 0; ax < 3; ax++)
         for (int m = -2; m <= 2; m++) {
            if (m == 0) continue;
            const long long q = p + m * st[ax];
            const bool mu = !isfinite(a.mu[q]), la = !isfinite(a.la[q]);
            all = all || mu;
            nan[ax] = nan[ax] || la;
            coef = coef || mu || la;
            for (int c = 0; c < 3; c++) {
               nan[c] = nan[c] || bad(c, q);
               if (c == ax) continue;
               for (int n = -2; n <= 2; n++)
                  if (n != 0 && bad(c, q + n * st[c])) nan[ax] = true;  // c_c of another component ...
               for (int n = -2; n <= 2; n++)
                  if (n != 0 && bad(ax, q + n * st[c])) nan[c] = true;  // ... in both of the plane's
            }
         }
      if (!coef && (a.e[p] >> 16) == kCoefBad) all = true;  // weights beyond the range
      for (int c = 0; c < 3; c++)
         if (all || nan[c]) {
            a.out[p + c * a.npts] = __longlong_as_double(0x7ff8000000000000LL);
            em = 0x7ff;
         }
   }
   return em;
}

template <int FORM>
__global__ void __launch_bounds__(NTHREADS, 2) fixed_stage_kernel(FixedArgs a)
{
   extern __shared__ __align__(16) unsigned char shared[];
   Smem& sm = *reinterpret_cast<Smem*>(shared);

   const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty;
   const int i0 = a.ib + 2 + blockIdx.x * TX;
   const int j0 = a.jb + 2 + blockIdx.y * TY;
   const int kbeg = a.k1 + blockIdx.z * a.kchunk;
   if (kbeg > a.k2) return;
   const int kend = min(kbeg + a.kchunk - 1, a.k2);
   const int i = i0 + tx, j = j0 + ty;
   const bool active = (i <= a.ie - 2) && (j <= a.je - 2);
   const bool inside = (i <= a.ie) && (j <= a.je);
   const bool row = j <= a.je - 2;  // the warp's row has interior points
   const int own = (ty + HALO) * PX + (tx + HALO);
   const long long npts = a.npts;
   const int col = (i - a.ib) + (int)a.ni * (j - a.jb);

   // the stage field's next plane, loaded one plane ahead of its use
   constexpr int kPre = (PLANE + NTHREADS - 1) / NTHREADS;
   double pv[kPre][3];
   int pcol[kPre];  // -1: beyond the tile or the array
#pragma unroll
   for (int r = 0; r < kPre; r++) {
      const int idx = tid + r * NTHREADS;
      const int gi = i0 - HALO + idx % PX, gj = j0 - HALO + idx / PX;
      pcol[r] = idx < PLANE && gi <= a.ie && gj <= a.je ? (gi - a.ib) + (int)a.ni * (gj - a.jb) : -1;
   }
   auto fetch = [&](int kk) {
      const long long plane = a.nij * (long long)(kk - a.kb);
#pragma unroll
      for (int r = 0; r < kPre; r++) {
         const long long p = plane + pcol[r];
#pragma unroll
         for (int c = 0; c < 3; c++) {
            pv[r][c] = pcol[r] >= 0 ? stage_value<FORM>(a, p + c * npts) : 0.0;
         }
      }
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
            sm.ve[q][idx] = e;
         }
      }
   };
   // The weights of the warp's row, axis by axis, through two stages of shared memory
   // two axes ahead of their use; wsrc: the next ones to copy, two planes end to end
   // wstride apart
   const int2* wsrc = a.w + (((long long)(kbeg - a.kb - 2) * a.wny + (j - a.jb - 2)) * a.wbx + blockIdx.x) * (24 * TX);
   const long long wstride = (long long)a.wny * a.wbx * (24 * TX) - 16 * TX;
   int wax = 0, wk = kbeg;
   auto copy_weights = [&](int stage) {
      if (row && wk <= kend) {
#pragma unroll
         for (int r = 0; r < 4; r++)
            copy16(&sm.w[ty][stage][0][0] + (r * 32 + tx) * 2, wsrc + (r * 32 + tx) * 2);
         wax = wax == 2 ? 0 : wax + 1;
         wk += wax == 0 ? 1 : 0;
         wsrc += wax == 0 ? wstride : 8 * TX;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
   };

   // Stretching of the own column, applied where it is not 1
   const double sxi = inside ? __ldg(a.sx + (i - a.ib)) : 1.0, syj = inside ? __ldg(a.sy + (j - a.jb)) : 1.0;
   const bool stx = !is_one(sxi), sty = !is_one(syj);

   // The halo's products: rows -2, -1, TY, TY + 1 (y outer) by the first four warps, columns
   // -2, -1, 32, 33 (x outer) by the next 4 TY threads
   const bool halo = tid < 4 * TX + 4 * TY, yh = ty < 4;
   const int hrow = yh ? (ty < 2 ? ty : ty + TY) : ((tid - 4 * TX) >> 2) + HALO;  // in the plane
   const int hcl = yh ? tx + HALO : ((tx & 3) < 2 ? (tx & 3) : (tx & 3) + TX);
   int hcol = -1;
   double hst = 1;
   if (halo) {
      const int gi = i0 - HALO + hcl, gj = j0 - HALO + hrow;
      if (gi <= a.ie && gj <= a.je) {
         hcol = (gi - a.ib) + (int)a.ni * (gj - a.jb);
         hst = yh ? __ldg(a.sx + (gi - a.ib)) : __ldg(a.sy + (gj - a.jb));
      }
   }

   i64 pq[2][3];  // sums of planes k-2, k-1
   int pe[2];
#pragma unroll
   for (int q = 0; q < 4; q++) sm.gze[q][tid] = kExpNone, sm.gz[q][0][tid] = sm.gz[q][1][tid] = sm.gz[q][2][tid] = 0;
#pragma unroll
   for (int q = 0; q < 2; q++) pe[q] = kExpNone, pq[q][0] = pq[q][1] = pq[q][2] = 0;
   int em = 0;

   if (tid == 0) sm.bad = *a.bad;
   __syncthreads();
   // ring slots of planes k-2..k+2
   int qm2 = 3, qm1 = 4, q0 = 0, qp1 = 1, qp2 = 2;
   fetch(kbeg - 2);
   store(q0);
   fetch(kbeg - 1);
   store(qp1);
   fetch(kbeg);
   copy_weights(0);
   copy_weights(1);
   int stage = 0;
   for (int k = kbeg - 2; k <= kend + 2; k++) {
      const bool full = k >= kbeg && k <= kend;
      const long long plane = a.nij * (long long)(k - a.kb);
      // planes up to kend + 2 are read (kend + 2 <= the last array plane)
      if (k <= kend) store(qp2);
      __syncthreads();
      // coefficients, used after the second differences
      int4 cc = make_int4(0, 0, 0, 0), hc = make_int4(0, 0, 0, 0);
      int ee = 0, he = 0;
      if (inside) {
         cc = __ldg(a.c + plane + col);
         ee = __ldg(a.e + plane + col);
      }
      if (hcol >= 0) {
         hc = __ldg(a.c + plane + hcol);
         he = __ldg(a.e + plane + hcol);
      }
      const double szk = __ldg(a.sz + (k - a.kb));
      const i64* v0 = &sm.v[q0][0][0];
      const int* e0 = sm.ve[q0];
      const int ec = (int)(short)(ee & 0xffff), ew = ee >> 16;

      int ex[4], ey[4];
#pragma unroll
      for (int m = 0; m < 4; m++) {
         const int s = m < 2 ? m - 2 : m - 1;
         ex[m] = e0[own + s];
         ey[m] = e0[own + s * PX];
      }
      const int Ex = max4(ex[0], ex[1], ex[2], ex[3]), Ey = max4(ey[0], ey[1], ey[2], ey[3]);
      int Ez = 0;
      i64 dx[3], dy[3], dz[3];
      i64 S[3] = {0, 0, 0};
      int eS = kExpNone;

      if (!full) {
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const i64* v = v0 + c * PLANE + own;
            if (c != 1) dx[c] = d1i(sar(v[-2], Ex - ex[0]), sar(v[-1], Ex - ex[1]), sar(v[1], Ex - ex[2]), sar(v[2], Ex - ex[3]));
            if (c != 0) dy[c] = d1i(sar(v[-2 * PX], Ey - ey[0]), sar(v[-PX], Ey - ey[1]), sar(v[PX], Ey - ey[2]), sar(v[2 * PX], Ey - ey[3]));
         }
      } else {
         const int qz[4] = {qm2, qm1, qp1, qp2};
         int ez[4];
#pragma unroll
         for (int m = 0; m < 4; m++) ez[m] = sm.ve[qz[m]][own];
         Ez = max4(ez[0], ez[1], ez[2], ez[3]);
         const int eo = e0[own];
         const int E = max(max(Ex, Ey), max(Ez, eo));
         i64 cr[3] = {1 << (kSplit - 1), 1 << (kSplit - 1), 1 << (kSplit - 1)};
         int ch[3] = {0, 0, 0}, cl[3] = {0, 0, 0};  // limb sums of the weights: the centre's
#pragma unroll
         for (int ax = 0; ax < 3; ax++) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            int2 w[2][4];
#pragma unroll
            for (int t = 0; t < 2; t++)
#pragma unroll
               for (int m = 0; m < 4; m++) w[t][m] = sm.w[ty][stage][t * 4 + m][tx];
            __syncwarp();
            copy_weights(stage);
            stage ^= 1;
            const int Ea = ax == 0 ? Ex : ax == 1 ? Ey : Ez;
#pragma unroll
            for (int c = 0; c < 3; c++) {
               i64 x[4];
#pragma unroll
               for (int m = 0; m < 4; m++) {
                  const int s = m < 2 ? m - 2 : m - 1;
                  x[m] = ax == 0 ? v0[c * PLANE + own + s] : ax == 1 ? v0[c * PLANE + own + s * PX] : sm.v[qz[m]][c][own];
               }
               const int* e = ax == 0 ? ex : ax == 1 ? ey : ez;
               const i64 d = d1i(sar(x[0], Ea - e[0]), sar(x[1], Ea - e[1]), sar(x[2], Ea - e[2]), sar(x[3], Ea - e[3]));
               if (ax == 0) dx[c] = d;
               if (ax == 1) dy[c] = d;
               if (ax == 2) dz[c] = d;
               const int2* wc = w[ax == c ? 1 : 0];
#pragma unroll
               for (int m = 0; m < 4; m++) {
                  const i64 y = sar(x[m], E - e[m]);
                  const int xh = (int)(y >> kSplit), xl = (int)y & kMask;
                  S[c] = madw(xh, wc[m].x, S[c]);
                  cr[c] = madw(xh, wc[m].y, cr[c]);
                  cr[c] = madw(xl, wc[m].x, cr[c]);
               }
            }
#pragma unroll
            for (int t = 0; t < 2; t++) {
               const int sh = (w[t][0].x + w[t][1].x) + (w[t][2].x + w[t][3].x);
               const int sl = (w[t][0].y + w[t][1].y) + (w[t][2].y + w[t][3].y);
#pragma unroll
               for (int c = 0; c < 3; c++)
                  if ((ax == c) == (t == 1)) {
                     ch[c] -= sh;
                     cl[c] -= sl;
                  }
            }
         }
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const i64 x = sar(v0[c * PLANE + own], E - eo);
            const int xh = (int)(x >> kSplit), xl = (int)x & kMask;
            cr[c] = madw(xl, ch[c], madw(xh, cl[c], cr[c]));
            S[c] = madw(xh, ch[c], S[c]) + (cr[c] >> kSplit);
         }
         eS = E + ew - 11;
      }

      // Products of the own point
      const bool stz = !is_one(szk);
      const Triple z = products(dx[0], dy[1], dx[2], dy[2], Ex, Ey, cc, ec, sxi, syj);
      if (full) {
         Triple t = products(dy[1], dz[2], dy[0], dz[0], Ey, Ez, cc, ec, syj, szk);
         const int qx = ty * PX + tx + HALO;
         sm.gx[0][qx] = t.la;
         sm.gx[1][qx] = t.m0;
         sm.gx[2][qx] = t.m1;
         sm.gxe[qx] = t.e;
         t = products(dx[0], dz[2], dx[1], dz[1], Ex, Ez, cc, ec, sxi, szk);
         const int qy = (ty + HALO) * TX + tx;
         sm.gy[0][qy] = t.m0;
         sm.gy[1][qy] = t.la;
         sm.gy[2][qy] = t.m1;
         sm.gye[qy] = t.e;
         if (halo) {
            const int s = hrow * PX + hcl, o = yh ? 1 : PX;
            const int qz[4] = {qm2, qm1, qp1, qp2};
            int eh[4], ez[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
               eh[m] = e0[s + (m < 2 ? m - 2 : m - 1) * o];
               ez[m] = sm.ve[qz[m]][s];
            }
            const int Eh = max4(eh[0], eh[1], eh[2], eh[3]), Ezh = max4(ez[0], ez[1], ez[2], ez[3]);
#pragma unroll
            for (int m = 0; m < 4; m++) {
               eh[m] = Eh - eh[m];
               ez[m] = Ezh - ez[m];
            }
            // y outer: mu v_x, la (u_x + w_z), mu v_z;  x outer: la (v_y + w_z), mu u_y, mu u_z
            const int cs = (yh ? 0 : PLANE) + s, cm = (yh ? PLANE : 0) + s;
            auto along = [&](int q) { return d1i(sar(v0[q - 2 * o], eh[0]), sar(v0[q - o], eh[1]), sar(v0[q + o], eh[2]), sar(v0[q + 2 * o], eh[3])); };
            auto down = [&](int q) {
               return d1i(sar(sm.v[qm2][0][q], ez[0]), sar(sm.v[qm1][0][q], ez[1]), sar(sm.v[qp1][0][q], ez[2]), sar(sm.v[qp2][0][q], ez[3]));
            };
            t = products(along(cs), down(2 * PLANE + s), along(cm), down(cm), Eh, Ezh, hc, (int)(short)(he & 0xffff), hst, szk);
            if (yh) {
               const int q = hrow * TX + tx;
               sm.gy[0][q] = t.m0;
               sm.gy[1][q] = t.la;
               sm.gy[2][q] = t.m1;
               sm.gye[q] = t.e;
            } else {
               const int q = (hrow - HALO) * PX + hcl;
               sm.gx[0][q] = t.la;
               sm.gx[1][q] = t.m0;
               sm.gx[2][q] = t.m1;
               sm.gxe[q] = t.e;
            }
         }
      }
      __syncthreads();

      // the values plane k - 2 is finished with, and the next plane of the stage field
      const int kp = k - 2;
      const bool finish = kp >= kbeg && active;
      const long long pp = col + a.nij * (long long)(kp - a.kb);
      double ir = 0, base[3] = {0, 0, 0};
      if (finish) {
         ir = __ldg(a.irho + pp);
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const long long q = pp + c * npts;
            base[c] = FORM == 1 ? __ldg(a.up + q) : fma(2.0, __ldg(a.u + q), -__ldg(a.um + q));
         }
      }
      if (k < kend) fetch(k + 3);

      // plane k: second differences and the x and y outer differences
      i64 P[3] = {0, 0, 0};
      int eP = kExpNone;
      if (full) {
         const i64* gx = &sm.gx[0][ty * PX + tx];
         const i64* gy = &sm.gy[0][ty * TX + tx];
         int hx[4], hy[4];
#pragma unroll
         for (int m = 0; m < 4; m++) {
            const int n = m < 2 ? m : m + 1;
            hx[m] = sm.gxe[ty * PX + tx + n];
            hy[m] = sm.gye[(ty + n) * TX + tx];
         }
         const int Eg = max(max4(hx[0], hx[1], hx[2], hx[3]), max4(hy[0], hy[1], hy[2], hy[3]));
         eP = max(eS, Eg);
         const Round of_s(eP - eS + 1), of_g(eP - Eg + 2);
#pragma unroll
         for (int m = 0; m < 4; m++) {
            hx[m] = Eg - hx[m] + 4;
            hy[m] = Eg - hy[m] + 4;
         }
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const i64* x = gx + c * NX;
            const i64* y = gy + c * NY;
            i64 cx = d1i(sar(x[0], hx[0]), sar(x[1], hx[1]), sar(x[3], hx[2]), sar(x[4], hx[3]));
            i64 cy = d1i(sar(y[0], hy[0]), sar(y[TX], hy[1]), sar(y[3 * TX], hy[2]), sar(y[4 * TX], hy[3]));
            if (stx || sty || stz) {
               cx = Factor(c == 0 ? sxi : c == 1 ? sxi * syj : sxi * szk)(cx);
               cy = Factor(c == 0 ? syj * sxi : c == 1 ? syj : syj * szk)(cy);
            }
            P[c] = of_s(S[c]) + of_g(cx + cy);
         }
      }

      // plane k - 2: the z outer difference, then the update
      if (finish) {
         const int z0 = k & 3, z1 = (k + 1) & 3, z3 = (k + 3) & 3;  // planes k-4, k-3, k-1
         int h0 = sm.gze[z0][tid], h1 = sm.gze[z1][tid], h3 = sm.gze[z3][tid];
         const int Eg = max4(h0, h1, h3, z.e);
         const int eF = max(pe[0], Eg);
         const Round of_p(eF - pe[0]), of_z(eF - Eg + 2);
         h0 = Eg - h0 + 4, h1 = Eg - h1 + 4, h3 = Eg - h3 + 4;
         const int h4 = Eg - z.e + 4;
         const double szp = __ldg(a.sz + (kp - a.kb));
         const bool st = stx || sty || !is_one(szp);
         const i64 zn[3] = {z.m0, z.m1, z.la};
         const double cr = a.coef * ir;
#pragma unroll
         for (int c = 0; c < 3; c++) {
            i64 cz = d1i(sar(sm.gz[z0][c][tid], h0), sar(sm.gz[z1][c][tid], h1), sar(sm.gz[z3][c][tid], h3), sar(zn[c], h4));
            if (st) cz = Factor(c == 0 ? szp * sxi : c == 1 ? szp * syj : szp)(cz);
            const double lu = from_block(of_p(pq[0][c]) + of_z(cz), eF - 1072);
            const double v = base[c] + cr * lu;
            if (FORM != 0) em = max(em, (__double2hiint(v) >> 20) & 0x7ff);
            a.out[pp + c * npts] = v;
         }
      }

      // queues
      sm.gz[k & 3][0][tid] = z.m0;
      sm.gz[k & 3][1][tid] = z.m1;
      sm.gz[k & 3][2][tid] = z.la;
      sm.gze[k & 3][tid] = z.e;
#pragma unroll
      for (int c = 0; c < 3; c++) {
         pq[0][c] = pq[1][c];
         pq[1][c] = P[c];
      }
      pe[0] = pe[1];
      pe[1] = eP;
      const int next = qm2;
      qm2 = qm1;
      qm1 = q0;
      q0 = qp1;
      qp1 = qp2;
      qp2 = next;
   }
   if (sm.bad && active) em = max(em, mark_not_finite<FORM>(a, i, j, kbeg, kend));
   if (a.emax) {
      em = __reduce_max_sync(0xffffffffu, em);
      if (tx == 0 && em > 0) atomicMax(a.emax, em);
   }
}

// The smallest e with x < 2^e, from the bit pattern of a positive x (-1022 for zero).
__device__ __forceinline__ int exponent_above(double x) { return ((__double2hiint(x) >> 20) & 0x7ff) - 1022; }

// Coefficients of the fixed-point stages.  For every array point: mu and lambda over
// 144 h^2 with the exponent of the larger; for every interior point the weights of its
// second differences (src/rhs4sg_rev.C:114-136)
//   a(q-1) - 3/4 (a(q) + a(q-2)),  a(q-2) + a(q+1) + 3 (a(q) + a(q-1))  and their mirrors
// of a = mu s and a = (2 mu + lambda) s along each axis, times s / (6 h^2), with the
// exponent of twice the largest sum of absolute values of one component's twelve.
__global__ void fixed_coef_kernel(Box b, const double* __restrict__ mu, const double* __restrict__ la,
                                  const double* __restrict__ sx, const double* __restrict__ sy,
                                  const double* __restrict__ sz, double scale, double cof144, int wbx, int wny,
                                  int2* __restrict__ w, int4* __restrict__ c, int* __restrict__ e,
                                  int* __restrict__ bad)
{
   for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < b.npts;
        p += (long long)gridDim.x * blockDim.x) {
      const int i = b.ib + (int)(p % b.ni);
      const int j = b.jb + (int)((p / b.ni) % (b.je - b.jb + 1));
      const int k = b.kb + (int)(p / b.nij);
      // a coefficient that is not finite counts as zero; the points that read it are marked
      // after the march
      bool finite = true;
      auto clean = [&](double v) {
         if (isfinite(v)) return v;
         finite = false;
         return 0.0;
      };
      const double m = clean(mu[p] * cof144), l = clean(la[p] * cof144);
      int ec = max(exponent_above(fmax(fabs(m), fabs(l))), -900);
      const int2 cm = to_coef(m, ec), cl = to_coef(l, ec);
      c[p] = make_int4(cm.x, cm.y, cl.x, cl.y);
      if (!(fabs(m) <= 1e300 && fabs(l) <= 1e300)) ec = kCoefBad;
      int ew = -1022;
      if (i >= b.ib + 2 && i <= b.ie - 2 && j >= b.jb + 2 && j <= b.je - 2 && k >= b.kb + 2 && k <= b.ke - 2) {
         const long long st[3] = {1, b.ni, b.nij};
         const double* sv[3] = {sx + (i - b.ib), sy + (j - b.jb), sz + (k - b.kb)};
         double wt[3][2][4], sum[3][2];
#pragma unroll
         for (int ax = 0; ax < 3; ax++) {
            double av[2][5];
#pragma unroll
            for (int q = -2; q <= 2; q++) {
               const long long pq = p + q * st[ax];
               const double s = sv[ax][q];
               av[0][q + 2] = mu[pq] * s;
               av[1][q + 2] = (2 * mu[pq] + la[pq]) * s;
            }
            const double f = scale * sv[ax][0];
#pragma unroll
            for (int t = 0; t < 2; t++) {
               const double* v = av[t];
               wt[ax][t][0] = f * (v[1] - 0.75 * (v[2] + v[0]));
               wt[ax][t][1] = f * (v[0] + v[3] + 3 * (v[2] + v[1]));
               wt[ax][t][2] = f * (v[1] + v[4] + 3 * (v[3] + v[2]));
               wt[ax][t][3] = f * (v[3] - 0.75 * (v[2] + v[4]));
#pragma unroll
               for (int q = 0; q < 4; q++) wt[ax][t][q] = clean(wt[ax][t][q]);
               sum[ax][t] = fabs(wt[ax][t][0]) + fabs(wt[ax][t][1]) + fabs(wt[ax][t][2]) + fabs(wt[ax][t][3]);
            }
         }
         double most = 0;
#pragma unroll
         for (int q = 0; q < 3; q++) {
            double s = 0;
#pragma unroll
            for (int ax = 0; ax < 3; ax++) s += sum[ax][ax == q ? 1 : 0];
            most = fmax(most, s);
         }
         ew = max(exponent_above(2 * most), -900);
         if (!(most <= 1e300)) ew = kCoefBad;
         const int ii = i - b.ib - 2;
         int2* o = w + ((((long long)(k - b.kb - 2) * wny + (j - b.jb - 2)) * wbx + ii / kFixedBlock) * 24) * kFixedBlock +
                   ii % kFixedBlock;
         const double up = ew == kCoefBad ? 0.0 : scalbn(1.0, 57 - ew);
#pragma unroll
         for (int ax = 0; ax < 3; ax++)
#pragma unroll
            for (int t = 0; t < 2; t++)
#pragma unroll
               for (int q = 0; q < 4; q++) {
                  const i64 v = __double2ll_rn(wt[ax][t][q] * up);
                  const i64 hi = (v + (1 << (kSplit - 1))) >> kSplit;
                  o[((ax * 2 + t) * 4 + q) * kFixedBlock] = make_int2((int)hi, (int)(v - (hi << kSplit)));
               }
      }
      if (!finite || ew == kCoefBad || ec == kCoefBad) *bad = 1;
      e[p] = (int)((unsigned)ew << 16 | ((unsigned)ec & 0xffffu));
   }
}

}  // namespace

long long fixed_weight_len(const Box& b)
{
   const long long nx = b.ie - b.ib - 3, ny = b.je - b.jb - 3, nz = b.ke - b.kb - 3;
   return (nx + kFixedBlock - 1) / kFixedBlock * ny * nz * 24 * kFixedBlock;
}

int launch_fixed_coef(const Box& b, const double* mu, const double* la, const double* sx, const double* sy,
                      const double* sz, double h, const FixedCoef& c, cudaStream_t s)
{
   SW4G_TRY(cuda_ok(cudaMemsetAsync(c.bad, 0, sizeof(int), s)));
   const int nx = (int)(b.ie - b.ib - 3), ny = (int)(b.je - b.jb - 3);
   const long long blocks = std::min<long long>((b.npts + 127) / 128, 152LL * 32);
   fixed_coef_kernel<<<(int)blocks, 128, 0, s>>>(b, mu, la, sx, sy, sz, 1.0 / (6 * h * h), 1.0 / (144 * h * h),
                                                 blocks_for(nx, kFixedBlock), ny, c.w, c.c, c.e, c.bad);
   return launch_status();
}

// Planes per CTA.  A CTA's march costs its planes and about four more (two planes of ring
// and two of z products at each end).  Launches that fill the resident slots more than
// once cost their waves and a tail of CTAs finishing apart; ones that fit at once cost
// their longest CTA, 1.3 times as much a plane as the share of a full GPU.  Against
// stage_kchunk's rule (3.5 waves, at least 12 planes): 64^3 121 -> 70 us a stage, a step
// at 48 x 40 x 36 363 -> 258 us, 101^3 752 -> 710 us, 512^3 unchanged.
int planes_per_cta(long long cols, int nk, int slots)
{
   if (stage_chunks_override() > 0) return stage_kchunk(cols, nk, 1, 1);
   int best = nk;
   double least = 1e30;
   for (int c = 1; c <= nk; c++) {
      const int per = (nk + c - 1) / c;
      if (per < 2 && c > 1) break;
      const double waves = (double)(cols * ((nk + per - 1) / per)) / slots;
      const double cost = (per + 4) * (waves <= 1 ? 1.3 : waves + 0.7);
      if (cost < least * 0.999) {
         least = cost;
         best = per;
      }
   }
   return best;
}

int launch_fixed_stage(const FusedStage& st, cudaStream_t stream)
{
   if (st.k2 < st.k1) return kOk;
   const Box& b = st.b;
   if (b.cs != b.npts) return kNotSupported;  // SoA only
   FixedArgs a;
   a.ib = b.ib; a.ie = b.ie; a.jb = b.jb; a.je = b.je; a.kb = b.kb; a.ke = b.ke;
   a.ni = b.ni; a.nij = b.nij; a.npts = b.npts;
   a.k1 = st.k1;
   a.k2 = st.k2;
   a.u = st.u;
   a.um = st.um;
   a.up = st.up;
   a.out = st.out;
   a.irho = st.irho;
   a.w = st.fc.w;
   a.c = st.fc.c;
   a.e = st.fc.e;
   a.bad = st.fc.bad;
   a.mu = st.mu;
   a.la = st.la;
   a.sx = st.st[0];
   a.sy = st.st[1];
   a.sz = st.st[2];
   a.coef = st.coef > 0 ? st.coef : (st.corrector ? st.dt * st.dt / 12 : st.dt * st.dt);
   a.emax = st.emax;
   const int ni = b.ie - b.ib - 3, nj = b.je - b.jb - 3, nk = st.k2 - st.k1 + 1;
   const int gx = blocks_for(ni, TX), gy = blocks_for(nj, TY);
   a.wbx = gx;
   a.wny = nj;
   const int form = st.corrector;  // 0, 1 or 2
   if (form < 0 || form > 2) return kBadArgument;
   const size_t smem = sizeof(Smem);
   static_assert(sizeof(Smem) <= 113 * 1024, "CTAs per SM");
   const void* kern = form == 0 ? (const void*)fixed_stage_kernel<0>
                      : form == 1 ? (const void*)fixed_stage_kernel<1>
                                  : (const void*)fixed_stage_kernel<2>;
   // the opt-in shared-memory size is a per-device function attribute
   int dev = 0;
   if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return kCudaError;
   static bool attr_set[3][64] = {};
   static int slots[3][64] = {};  // CTAs resident at once
   if (!attr_set[form][dev]) {
      int sms = 0;
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
         return kCudaError;
      slots[form][dev] = std::max(1, sms) * resident_ctas(kern, NTHREADS, smem);
      attr_set[form][dev] = true;
   }
   a.kchunk = st.kchunk > 0 ? st.kchunk : planes_per_cta((long long)gx * gy, nk, slots[form][dev]);
   const dim3 grid(gx, gy, (nk + a.kchunk - 1) / a.kchunk), block(TX, TY, 1);
   if (form == 0)
      fixed_stage_kernel<0><<<grid, block, smem, stream>>>(a);
   else if (form == 1)
      fixed_stage_kernel<1><<<grid, block, smem, stream>>>(a);
   else
      fixed_stage_kernel<2><<<grid, block, smem, stream>>>(a);
   SW4G_TRY(launch_status());
   if (form == 0 || st.beta == 0) return kOk;
   return launch_damping_layers(4, b, st.k1, st.k2, st.u, st.um, st.out, st.rho, st.irho, st.dc, st.st, st.co,
                               st.beta, st.emax, stream);
}

}  // namespace sw4g

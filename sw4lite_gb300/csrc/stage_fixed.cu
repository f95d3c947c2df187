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
//    shared memory, 2-point halo: three 57-bit integers and their exponents a point.
//    Two CTAs per SM at 168 registers: the 128 registers of 2 x 256 threads spill into an
//    L1 that the shared memory leaves at a few KB (measured with one exponent a point:
//    predictor at 512^3 19.6 ms, 32 x 6 15.2 ms, one CTA of 32 x 12 18.3 ms).
//  * A value, a difference, a product and a weight each have their own exponent, so a
//    component keeps its digits beside one that is any power of two larger.  A component's
//    second differences are sums over w (x - x_0) on all three axes, aligned to the largest
//    w x among them; the products of the mixed terms are aligned by the outer difference
//    that reads them.
//  * The second differences' 24 weights per point (stretching folded in) are integers with
//    an exponent for each axis and coefficient, prepared once per material and stored by
//    blocks of 32 points, so that a warp reads 24 contiguous lines; each warp copies its own
//    asynchronously, three axes' and coefficients' lines ahead of their use.
//  * A mixed derivative is the outer difference of a product G = c * D f formed once per
//    point.  The nine first differences of a point serve its second differences' values
//    and all three of its products: those for the x and y outer differences go to shared
//    memory, those for the z outer difference into a register queue, so a plane is
//    finished two planes later, when the last product along z is known.
//  * FP64 remains in forming up - 2u + um and in the update.
// What bounds them: the latency of twelve warps an SM and the integer pipes (about 2900
// instructions a warp of 32 points, half of them at half rate), the corrector also the FP64
// operations of its stage field.  At 512^3 the predictor takes 17.9 ms and the corrector 25.8 ms
// with the damping, against 40.6 and 53.8 ms with the sums in FP64 (stage_fused.cu), whose 160
// and 198 FP64 operations a point saturate the 1.7 that an SM completes per clock.  (One
// exponent for a point's three components, and one for all its weights, took 15.2 and 22.5 ms,
// and cost a component below the others its digits.)  Against quad precision the levels after 50
// steps are off by 0.47 to 0.69 times what they are with the sums in FP64.
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
   const int* __restrict__ e;     // exponents of both: lambda << 16 | mu
   const int* __restrict__ ew;    // of the weights, npts for each axis: (2 mu + lambda) << 16 | mu
   const int* __restrict__ bad;   // nonzero: the material is not finite everywhere
   int wbx, wny;                  // blocks per row and rows per plane of w
   const double* __restrict__ sx;
   const double* __restrict__ sy;
   const double* __restrict__ sz;
   double coef;
   int* emax;
};

// Exponent of weights and coefficients that are not finite
constexpr int kCoefBad = 0x7fff;

constexpr int kStages = 3;     // of weights, four lines each
constexpr int kLimb = 27;      // low limb of the second differences' factors

struct Smem {
   i64 v[5][3][PLANE];         // stage field, ring of planes
   i64 gx[3][NX];              // products for the x outer difference: la (v_y + w_z), mu u_y, mu u_z
   i64 gy[3][NY];              // for the y outer difference: mu v_x, la (u_x + w_z), mu v_z
   int2 w[TY][kStages][4][TX]; // weights of one axis and coefficient for a row of points
   i64 gz[4][3][NTHREADS];     // products for the z outer difference: mu w_x, mu w_y, la (u_x + v_y)
                               // of the four planes before, each thread its own column
   short ve[5][3][PLANE];      // exponents of all these
   short gxe[3][NX], gye[3][NY], gze[4][3][NTHREADS];
   int bad;                    // a value of the stage field or of the material is not finite
};

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
// component and its weights along the three axes; its mixed terms read another component at
// the points off both axes in the plane of the two, lambda along its own axis and mu along
// the others.
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
      bool nan[3] = {bad(0, p), bad(1, p), bad(2, p)};
      for (int ax = 0; ax < 3; ax++) {
         const int ew = a.ew[p + ax * a.npts];
         for (int c = 0; c < 3; c++)
            if ((c == ax ? ew >> 16 : (int)(short)(ew & 0xffff)) == kCoefBad) nan[c] = true;
         for (int m = -2; m <= 2; m++) {
            if (m == 0) continue;
            const long long q = p + m * st[ax];
            const bool mu = (short)(a.e[q] & 0xffff) == kCoefBad, la = (a.e[q] >> 16) == kCoefBad;
            for (int c = 0; c < 3; c++) {
               nan[c] = nan[c] || bad(c, q) || (c == ax ? la : mu);
               if (c == ax) continue;
               for (int n = -2; n <= 2; n++)
                  if (n != 0 && bad(c, q + n * st[c])) nan[ax] = true;  // c_c of another component ...
               for (int n = -2; n <= 2; n++)
                  if (n != 0 && bad(ax, q + n * st[c])) nan[c] = true;  // ... in both of the plane's
            }
         }
      }
      for (int c = 0; c < 3; c++)
         if (nan[c]) {
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
#pragma unroll
            for (int c = 0; c < 3; c++) {
               i64 m;
               int e;
               if (to_fixed(pv[r][c], m, e)) sm.bad = 1;
               sm.v[q][c][idx] = m;
               sm.ve[q][c][idx] = (short)e;
            }
         }
      }
   };
   // The weights of the warp's row, four lines (one axis and coefficient) at a time, through
   // three stages of shared memory; wsrc: the next ones to copy, two planes end to end
   // wstride apart
   const int2* wsrc = a.w + (((long long)(kbeg - a.kb - 2) * a.wny + (j - a.jb - 2)) * a.wbx + blockIdx.x) * (24 * TX);
   const long long wstride = (long long)a.wny * a.wbx * (24 * TX) - 20 * TX;
   int wunit = 0, wk = kbeg;
   auto copy_weights = [&](int stage) {
      if (row && wk <= kend) {
#pragma unroll
         for (int r = 0; r < 2; r++)
            copy16(&sm.w[ty][stage][0][0] + (r * 32 + tx) * 2, wsrc + (r * 32 + tx) * 2);
         wunit = wunit == 5 ? 0 : wunit + 1;
         wk += wunit == 0 ? 1 : 0;
         wsrc += wunit == 0 ? wstride : 4 * TX;
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

   Num pq[2][3];  // sums of planes k-2, k-1, value m * 2^(e - 1072)
#pragma unroll
   for (int c = 0; c < 3; c++) {
#pragma unroll
      for (int q = 0; q < 4; q++) sm.gze[q][c][tid] = (short)kNone, sm.gz[q][c][tid] = 0;
      pq[0][c] = pq[1][c] = Num{0, kNone};
   }
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
   copy_weights(2);
   for (int k = kbeg - 2; k <= kend + 2; k++) {
      const bool full = k >= kbeg && k <= kend;
      const long long plane = a.nij * (long long)(k - a.kb);
      // planes up to kend + 2 are read (kend + 2 <= the last array plane)
      if (k <= kend) store(qp2);
      __syncthreads();
      // coefficients, used after the second differences
      int4 cc = make_int4(0, 0, 0, 0), hc = make_int4(0, 0, 0, 0);
      int ee = 0, he = 0, ew[3] = {0, 0, 0};
      if (inside) {
         cc = __ldg(a.c + plane + col);
         ee = __ldg(a.e + plane + col);
         if (full)
#pragma unroll
            for (int ax = 0; ax < 3; ax++) ew[ax] = __ldg(a.ew + plane + col + ax * npts);
      }
      if (hcol >= 0) {
         hc = __ldg(a.c + plane + hcol);
         he = __ldg(a.e + plane + hcol);
      }
      const double szk = __ldg(a.sz + (k - a.kb));
      const i64* v0 = &sm.v[q0][0][0];
      const short* e0 = &sm.ve[q0][0][0];
      const int qz[4] = {qm2, qm1, qp1, qp2};
      // value and exponent of component c at the point s, m points along an axis of the plane
      // (stride o) or, as down, planes
      auto along = [&](int c, int s, int o, bool& tiny) {
         const i64* v = v0 + c * PLANE + s;
         const short* e = e0 + c * PLANE + s;
         const int x0 = e[-2 * o], x1 = e[-o], x2 = e[o], x3 = e[2 * o];
         return difference(v[-2 * o], v[-o], v[o], v[2 * o], x0, x1, x2, x3, max4(x0, x1, x2, x3), tiny);
      };
      auto down = [&](int c, int s, bool& tiny) {
         const int x0 = sm.ve[qm2][c][s], x1 = sm.ve[qm1][c][s], x2 = sm.ve[qp1][c][s], x3 = sm.ve[qp2][c][s];
         return difference(sm.v[qm2][c][s], sm.v[qm1][c][s], sm.v[qp1][c][s], sm.v[qp2][c][s], x0, x1, x2, x3, max4(x0, x1, x2, x3), tiny);
      };

      Num D[3][3];  // differences along x, y, z of the components
      bool tiny = false;
      i64 S[3] = {0, 0, 0};
      int eS[3] = {kNone, kNone, kNone};

      if (!full) {
         D[0][0] = along(0, own, 1, tiny);
         D[0][2] = along(2, own, 1, tiny);
         D[1][1] = along(1, own, PX, tiny);
         D[1][2] = along(2, own, PX, tiny);
      } else {
         // the largest exponent along each axis, and of a component's w x
         int E[3][3], eo[3];
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const short* e = e0 + c * PLANE + own;
            eo[c] = e[0];
            E[0][c] = max4(e[-2], e[-1], e[1], e[2]);
            E[1][c] = max4(e[-2 * PX], e[-PX], e[PX], e[2 * PX]);
            E[2][c] = max4(sm.ve[qm2][c][own], sm.ve[qm1][c][own], sm.ve[qp1][c][own], sm.ve[qp2][c][own]);
#pragma unroll
            for (int ax = 0; ax < 3; ax++)
               eS[c] = max(eS[c], max(E[ax][c], eo[c]) + (ax == c ? ew[ax] >> 16 : (int)(short)(ew[ax] & 0xffff)));
         }
         i64 cr[3] = {0, 0, 0};  // products of high and low limbs
#pragma unroll
         for (int unit = 0; unit < 6; unit++) {
            const int ax = unit / 2, t = unit % 2;
            asm volatile("cp.async.wait_group 2;" ::: "memory");
            __syncwarp();
            int2 w[4];
#pragma unroll
            for (int m = 0; m < 4; m++) w[m] = sm.w[ty][unit % kStages][m][tx];
            __syncwarp();
            copy_weights(unit % kStages);
            const int et = t == 1 ? ew[ax] >> 16 : (int)(short)(ew[ax] & 0xffff);
#pragma unroll
            for (int c = 0; c < 3; c++) {
               if ((ax == c) != (t == 1)) continue;
               const int E_ = E[ax][c], A = eS[c] - et;
               i64 x[4];
#pragma unroll
               for (int m = 0; m < 4; m++) {
                  const int s = m < 2 ? m - 2 : m - 1;
                  const int e = ax == 0 ? e0[c * PLANE + own + s] : ax == 1 ? e0[c * PLANE + own + s * PX] : sm.ve[qz[m]][c][own];
                  x[m] = sar(ax == 0 ? v0[c * PLANE + own + s] : ax == 1 ? v0[c * PLANE + own + s * PX] : sm.v[qz[m]][c][own], E_ - e);
               }
               D[ax][c] = normal(d1i(x[0], x[1], x[2], x[3]), E_, tiny);
               const i64 x0 = sar(v0[c * PLANE + own], A - eo[c]);
#pragma unroll
               for (int m = 0; m < 4; m++) {
                  const i64 y = sar(x[m], A - E_) - x0;
                  const int xh = (int)(y >> kLimb), xl = (int)y & ((1 << kLimb) - 1);
                  S[c] = madw(xh, w[m].x, S[c]);
                  cr[c] = madw(xh, w[m].y, cr[c]);
                  cr[c] = madw(xl, w[m].x, cr[c]);
               }
            }
         }
#pragma unroll
         for (int c = 0; c < 3; c++) {  // with as many of the lower bits as there is room for
            const int n = min(headroom<61>(S[c]), kLimb);
            S[c] = (S[c] << n) + to_odd(cr[c], kLimb - n);
            eS[c] -= 9 + n;
         }
      }

      // differences that cancelled almost
      if (tiny) {
         if (!full) {
            rest(D[0][0]), rest(D[0][2]), rest(D[1][1]), rest(D[1][2]);
         } else {
#pragma unroll
            for (int ax = 0; ax < 3; ax++)
#pragma unroll
               for (int c = 0; c < 3; c++) rest(D[ax][c]);
         }
      }

      // Products of the own point
      const bool stz = !is_one(szk);
      const int2 cm = make_int2(cc.x, cc.y), cl = make_int2(cc.z, cc.w);
      const int emu = (int)(short)(ee & 0xffff), el = ee >> 16;
      const Triple z = products<false>(D[0][0], D[1][1], D[0][2], D[1][2], cm, emu, cl, el, sxi, syj);
      if (full) {
         auto to_x = [&](const Triple& t, int q) {
            sm.gx[0][q] = t.la.m;
            sm.gx[1][q] = t.m0.m;
            sm.gx[2][q] = t.m1.m;
            sm.gxe[0][q] = (short)t.la.e;
            sm.gxe[1][q] = (short)t.m0.e;
            sm.gxe[2][q] = (short)t.m1.e;
         };
         auto to_y = [&](const Triple& t, int q) {
            sm.gy[0][q] = t.m0.m;
            sm.gy[1][q] = t.la.m;
            sm.gy[2][q] = t.m1.m;
            sm.gye[0][q] = (short)t.m0.e;
            sm.gye[1][q] = (short)t.la.e;
            sm.gye[2][q] = (short)t.m1.e;
         };
         to_x(products<false>(D[1][1], D[2][2], D[1][0], D[2][0], cm, emu, cl, el, syj, szk), ty * PX + tx + HALO);
         to_y(products<false>(D[0][0], D[2][2], D[0][1], D[2][1], cm, emu, cl, el, sxi, szk), (ty + HALO) * TX + tx);
         if (halo) {
            // y outer: mu v_x, la (u_x + w_z), mu v_z;  x outer: la (v_y + w_z), mu u_y, mu u_z
            const int s = hrow * PX + hcl, o = yh ? 1 : PX, cs = yh ? 0 : 1, cm = 1 - cs;
            bool some = false;
            Num d0 = along(cs, s, o, some), d1 = down(2, s, some), d2 = along(cm, s, o, some), d3 = down(cm, s, some);
            if (some) rest(d0), rest(d1), rest(d2), rest(d3);
            const Triple t = products<false>(d0, d1, d2, d3, make_int2(hc.x, hc.y), (int)(short)(he & 0xffff), make_int2(hc.z, hc.w), he >> 16, hst, szk);
            if (yh) to_y(t, hrow * TX + tx);
            else to_x(t, (hrow - HALO) * PX + hcl);
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
            if (stx || sty || stz) {
               cx = stretched<false>(cx, c == 0 ? sxi : c == 1 ? sxi * syj : sxi * szk);
               cy = stretched<false>(cy, c == 0 ? syj * sxi : c == 1 ? syj : syj * szk);
            }
            P[c].e = max(eS[c], max(cx.e, cy.e));
            P[c].m = to_odd(S[c], P[c].e - eS[c] + 1) + to_odd(cx.m, P[c].e - cx.e + 2) + to_odd(cy.m, P[c].e - cy.e + 2);
         }
      }

      // plane k - 2: the z outer difference, then the update
      if (finish) {
         const int z0 = k & 3, z1 = (k + 1) & 3, z3 = (k + 3) & 3;  // planes k-4, k-3, k-1
         const double szp = __ldg(a.sz + (kp - a.kb));
         const bool st = stx || sty || !is_one(szp);
         const Num zn[3] = {z.m0, z.m1, z.la};
         const double cr = a.coef * ir;
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const int h0 = sm.gze[z0][c][tid], h1 = sm.gze[z1][c][tid], h3 = sm.gze[z3][c][tid], h4 = zn[c].e;
            Num g = outer(sm.gz[z0][c][tid], sm.gz[z1][c][tid], sm.gz[z3][c][tid], zn[c].m, h0, h1, h3, h4, max4(h0, h1, h3, h4));
            if (st) g = stretched<false>(g, c == 0 ? szp * sxi : c == 1 ? szp * syj : szp);
            const int eF = max(pq[0][c].e, g.e);
            const i64 F = to_odd(pq[0][c].m, eF - pq[0][c].e) + to_odd(g.m, eF - g.e + 2);
            bool low;
            const double lu = from_block(F, eF - 1072, low);
            const double v = base[c] + (low ? lowered(cr) : cr) * lu;
            if (FORM != 0) em = max(em, (__double2hiint(v) >> 20) & 0x7ff);
            a.out[pp + c * npts] = v;
         }
      }

      // queues
      const Num zn[3] = {z.m0, z.m1, z.la};
#pragma unroll
      for (int c = 0; c < 3; c++) {
         sm.gz[k & 3][c][tid] = zn[c].m;
         sm.gze[k & 3][c][tid] = (short)zn[c].e;
         pq[0][c] = pq[1][c];
         pq[1][c] = P[c];
      }
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

// Coefficients of the fixed-point stages.  For every array point: mu and lambda over
// 144 h^2; for every interior point the weights of its second differences
// (src/rhs4sg_rev.C:114-136)
//   a(q-1) - 3/4 (a(q) + a(q-2)),  a(q-2) + a(q+1) + 3 (a(q) + a(q-1))  and their mirrors
// of a = mu s and a = (2 mu + lambda) s along each axis, times s / (6 h^2), each four with
// the exponent that leaves the sum of their magnitudes below 2^56.  What is not finite counts
// as zero and has the exponent kCoefBad; the points that read it are marked after a march.
__global__ void fixed_coef_kernel(Box b, const double* __restrict__ mu, const double* __restrict__ la,
                                  const double* __restrict__ sx, const double* __restrict__ sy,
                                  const double* __restrict__ sz, double scale, double cof144, int wbx, int wny,
                                  int2* __restrict__ w, int4* __restrict__ c, int* __restrict__ e,
                                  int* __restrict__ ew, int* __restrict__ bad)
{
   for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < b.npts;
        p += (long long)gridDim.x * blockDim.x) {
      const int i = b.ib + (int)(p % b.ni);
      const int j = b.jb + (int)((p / b.ni) % (b.je - b.jb + 1));
      const int k = b.kb + (int)(p / b.nij);
      bool any = false;
      auto coef = [&](double v, int2& limbs) {
         i64 m;
         int x;
         const bool nf = to_fixed(v, m, x);
         any = any || nf;
         if (nf) m = 0;
         limbs = make_int2((int)(m >> kSplit), (int)(m & kMask) << 5);
         return nf ? kCoefBad : x - 1022;
      };
      int2 cm, cl;
      const int em = coef(mu[p] * cof144, cm), el = coef(la[p] * cof144, cl);
      c[p] = make_int4(cm.x, cm.y, cl.x, cl.y);
      e[p] = (int)((unsigned)el << 16 | ((unsigned)em & 0xffffu));
      if (i >= b.ib + 2 && i <= b.ie - 2 && j >= b.jb + 2 && j <= b.je - 2 && k >= b.kb + 2 && k <= b.ke - 2) {
         const long long st[3] = {1, b.ni, b.nij};
         const double* sv[3] = {sx + (i - b.ib), sy + (j - b.jb), sz + (k - b.kb)};
         const int ii = i - b.ib - 2;
         int2* o = w + ((((long long)(k - b.kb - 2) * wny + (j - b.jb - 2)) * wbx + ii / kFixedBlock) * 24) * kFixedBlock +
                   ii % kFixedBlock;
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
            int et[2];
#pragma unroll
            for (int t = 0; t < 2; t++) {
               const double* v = av[t];
               const double wt[4] = {f * (v[1] - 0.75 * (v[2] + v[0])), f * (v[0] + v[3] + 3 * (v[2] + v[1])),
                                     f * (v[1] + v[4] + 3 * (v[3] + v[2])), f * (v[3] - 0.75 * (v[2] + v[4]))};
               i64 m[4], sum = 0;
               int x[4];
               bool nf = false;
#pragma unroll
               for (int q = 0; q < 4; q++)
                  if (to_fixed(wt[q], m[q], x[q])) nf = true;
               const int most = max4(x[0], x[1], x[2], x[3]);
#pragma unroll
               for (int q = 0; q < 4; q++) {
                  const i64 r = sar(m[q], most - x[q]);
                  sum += r < 0 ? -r : r;
               }
               const int down = nf ? 62 : max(8 - __clzll(sum), 0);  // sum < 2^(64 - clz)
#pragma unroll
               for (int q = 0; q < 4; q++) {
                  const i64 r = nf ? 0 : Round(most - x[q] + down)(m[q]), hi = (r + (1 << (kLimb - 1))) >> kLimb;
                  o[((ax * 2 + t) * 4 + q) * kFixedBlock] = make_int2((int)hi, (int)(r - (hi << kLimb)));
               }
               et[t] = nf ? kCoefBad : most + down - 1022;
               any = any || nf;
            }
            ew[p + ax * b.npts] = (int)((unsigned)et[1] << 16 | ((unsigned)et[0] & 0xffffu));
         }
      }
      // ghost points off two axes' interiors are in no stencil
      const int off = (i < b.ib + 2 || i > b.ie - 2) + (j < b.jb + 2 || j > b.je - 2) + (k < b.kb + 2 || k > b.ke - 2);
      if (any && off < 2) *bad = 1;
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
                                                 blocks_for(nx, kFixedBlock), ny, c.w, c.c, c.e, c.ew, c.bad);
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
   a.ew = st.fc.ew;
   a.bad = st.fc.bad;
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
   static std::atomic<int> resident[3][64];
   const int slots = resident_slots(resident[form], kern, NTHREADS, smem);
   if (slots < 1) return kCudaError;
   a.kchunk = st.kchunk > 0 ? st.kchunk : planes_per_cta((long long)gx * gy, nk, slots);
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

// Supergrid damping of an FP64 level in the layers alone, sm_103a.
//
//   order 4:  out -= beta/rho   sum_a w_a D2_a(e_a D2_a(u - um))
//   order 6:  out += beta/2/rho sum_a w_a D3_a((e_a(m) + e_a(m+1)) D3_a(u - um))
//
// with e_a = rho dc_a, w_a the axis' stretching times the corner tapers of the other two
// (addsgd4fort, addsgd6fort: src/ew-cfromfort.C:748-1158).  An axis' term is exactly zero
// where its profile dc vanishes within the stencil, so only the layers' points are touched.
//
// FP64 operations bound it (1.7 per clock and SM), so each is done once: a thread marches
// along the damped axis with the inner differences and their products in registers, 8
// operations per point and component (order 4) instead of 17 where each point evaluates
// its own five.  Threads of a warp lie along x for the y and z layers and along y for the
// x layers.  A point in two or three layers is done whole by the first of them in the
// order x, y, z, the other axes' terms evaluated at the point, so a level is rounded once.
//
// Measured with 30-point layers: order 4 at 512^3, 3.2 ms against 8.6 ms inside the
// corrector stage; order 6 at 160 x 144 x 128, 0.3 ms against 1.3 ms for the kernel that
// visits every point (pointwise.cu, the kernel-level entry points).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "stencil.cuh"

namespace sw4g {
namespace {

// 64-thread CTAs at 168 registers: the loads of four points in flight in each thread
// measured better than more threads (at 512^3: 128 registers +0.2 ms, 64 registers +3 ms,
// by spills).
constexpr int kThreads = 64, kUnroll = 4;

struct LineArgs {
   Box b;
   int lo[3], hi[3];  // the points that may be damped, as array indices from 0
   DampSegs seg;
   int len;               // points per thread
   int chunks[3];         // per line of each axis
   int block0[3];         // first block of each axis
   const double* __restrict__ u;
   const double* __restrict__ um;
   double* __restrict__ out;
   const double* __restrict__ rho;
   const double* __restrict__ irho;
   const double* dc[3];
   const double* st[3];
   const double* co[3];
   double beta;
   int* emax;
};

template <int ORDER>
__device__ __forceinline__ bool damped(const double* __restrict__ dc, int n)
{
   constexpr int R = ORDER == 4 ? 1 : 2;
   bool any = false;
#pragma unroll
   for (int m = -R; m <= R; m++) any = any || nonzero_bits(__ldg(dc + n + m));
   return any;
}

// w * (the outer difference) of one axis at one point, all components
template <int ORDER, int ax>
__device__ __forceinline__ void term_at(const LineArgs& a, const int n[3], long long p, long long o, double sg[3])
{
   constexpr int R = ORDER == 4 ? 1 : 2;
   double e[2 * R + 1];
#pragma unroll
   for (int m = -R; m <= R; m++) e[m + R] = __ldg(a.rho + p + m * o) * __ldg(a.dc[ax] + n[ax] + m);
   constexpr int b0 = ax == 0 ? 1 : 0, b1 = ax == 2 ? 1 : 2;
   const double w = __ldg(a.st[ax] + n[ax]) * __ldg(a.co[b0] + n[b0]) * __ldg(a.co[b1] + n[b1]);
#pragma unroll
   for (int c = 0; c < 3; c++) {
      double d[2 * R + 3];
#pragma unroll
      for (int m = -R - 1; m <= R + 1; m++) {
         const long long q = p + c * a.b.npts + m * o;
         d[m + R + 1] = __ldg(a.u + q) - __ldg(a.um + q);
      }
      double s = 0;
      if (ORDER == 4) {
         s = e[2] * (d[4] - 2 * d[3] + d[2]) - 2 * e[1] * (d[3] - 2 * d[2] + d[1]) + e[0] * (d[2] - 2 * d[1] + d[0]);
      } else {
         const double sign[4] = {-1, 3, -3, 1};
#pragma unroll
         for (int m = 0; m < 4; m++)
            s += sign[m] * (e[m + 1] + e[m]) * (d[m + 3] - 3 * d[m + 2] + 3 * d[m + 1] - d[m]);
      }
      sg[c] += w * s;
   }
}

// The t-th thread of axis ax's layers; returns the largest exponent field written
template <int ORDER, int ax>
__device__ __forceinline__ int march(const LineArgs& a, long long t)
{
   const long long st[3] = {1, a.b.ni, a.b.nij};
   constexpr int lane_ax = ax == 0 ? 1 : 0, row_ax = ax == 2 ? 1 : 2;
   const int nl = a.hi[lane_ax] - a.lo[lane_ax] + 1, nr = a.hi[row_ax] - a.lo[row_ax] + 1;
   const int lanes = (nl + 31) / 32 * 32;
   const int il = (int)(t % lanes);
   t /= lanes;
   const int ir = (int)(t % nr), chunk = (int)(t / nr);
   int em = 0;
   if (il < nl && chunk < a.chunks[ax]) {
      int n[3];
      n[lane_ax] = a.lo[lane_ax] + il;
      n[row_ax] = a.lo[row_ax] + ir;
      // the chunk's points along the axis
      const int first = (a.seg.hi[ax][0] - a.seg.lo[ax][0] + a.len) / a.len;
      const int s = chunk < first ? 0 : 1;
      const int from = a.seg.lo[ax][s] + (chunk - (s ? first : 0)) * a.len, to = min(from + a.len - 1, a.seg.hi[ax][s]);
      // points of an earlier axis' layers are done there
      const bool other0 = damped<ORDER>(a.dc[lane_ax], n[lane_ax]), other1 = damped<ORDER>(a.dc[row_ax], n[row_ax]);
      const bool skip = (ax > 0 && other0) || (ax == 2 && other1);
      const bool also_y = ax == 0 && other0, also_z = (ax == 0 || ax == 1) && other1;
      if (!skip) {
         constexpr int R = ORDER == 4 ? 1 : 2;
         const long long o = st[ax];
         n[ax] = from;
         long long p = n[0] + a.b.ni * n[1] + a.b.nij * (long long)n[2];
         constexpr int b0 = ax == 0 ? 1 : 0, b1 = ax == 2 ? 1 : 2;
         const double c0 = __ldg(a.co[b0] + n[b0]), c1 = __ldg(a.co[b1] + n[b1]);
         auto diff = [&](int c, int m) {
            const long long q = p + c * a.b.npts + m * o;
            return __ldg(a.u + q) - __ldg(a.um + q);
         };
         auto coef = [&](int m) { return __ldg(a.rho + p + m * o) * __ldg(a.dc[ax] + n[ax] + m); };
         // windows at the point n: differences d up to n + R, inner products g before the
         // one that the next difference completes
         double d[3][ORDER / 2], g[3][ORDER / 2], e = 0;
         if (ORDER == 4) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
               const double dm2 = diff(c, -2), dm1 = diff(c, -1), d0 = diff(c, 0), d1 = diff(c, 1);
               g[c][0] = coef(-1) * (d0 - 2 * dm1 + dm2);
               g[c][1] = coef(0) * (d1 - 2 * d0 + dm1);
               d[c][0] = d0;
               d[c][1] = d1;
            }
         } else {
            const double em2 = coef(-2), em1 = coef(-1), e0 = coef(0);
            e = coef(1);
#pragma unroll
            for (int c = 0; c < 3; c++) {
               const double dm3 = diff(c, -3), dm2 = diff(c, -2), dm1 = diff(c, -1), d0 = diff(c, 0), d1 = diff(c, 1), d2 = diff(c, 2);
               g[c][0] = (em1 + em2) * (d0 - 3 * dm1 + 3 * dm2 - dm3);
               g[c][1] = (e0 + em1) * (d1 - 3 * d0 + 3 * dm1 - dm2);
               g[c][ORDER / 2 - 1] = (e + e0) * (d2 - 3 * d1 + 3 * d0 - dm1);
               d[c][0] = d0;
               d[c][1] = d1;
               d[c][ORDER / 2 - 1] = d2;
            }
         }
#pragma unroll kUnroll
         for (; n[ax] <= to; n[ax]++, p += o) {
            const double w = __ldg(a.st[ax] + n[ax]) * c0 * c1;
            const double en = coef(R);
            double sg[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
               const double dn = diff(c, R + 1);
               double s;
               if (ORDER == 4) {
                  const double gn = en * (dn - 2 * d[c][1] + d[c][0]);
                  s = gn - 2 * g[c][1] + g[c][0];
                  g[c][0] = g[c][1];
                  g[c][1] = gn;
                  d[c][0] = d[c][1];
                  d[c][1] = dn;
               } else {
                  constexpr int L = ORDER / 2 - 1;
                  const double gn = (en + e) * (dn - 3 * d[c][L] + 3 * d[c][1] - d[c][0]);
                  s = gn - 3 * g[c][L] + 3 * g[c][1] - g[c][0];
                  g[c][0] = g[c][1];
                  g[c][1] = g[c][L];
                  g[c][L] = gn;
                  d[c][0] = d[c][1];
                  d[c][1] = d[c][L];
                  d[c][L] = dn;
               }
               sg[c] = w * s;
            }
            e = en;
            if (also_y) term_at<ORDER, 1>(a, n, p, st[1], sg);
            if (also_z) term_at<ORDER, 2>(a, n, p, st[2], sg);
            const double f = a.beta * __ldg(a.irho + p);
#pragma unroll
            for (int c = 0; c < 3; c++) {
               const long long q = p + c * a.b.npts;
               const double v = a.out[q] - f * sg[c];
               a.out[q] = v;
               em = max(em, (__double2hiint(v) >> 20) & 0x7ff);
            }
         }
      }
   }
   return em;
}

template <int ORDER>
__global__ void __launch_bounds__(kThreads, 6) damping_lines_kernel(LineArgs a)
{
   const int ax = blockIdx.x >= a.block0[2] ? 2 : blockIdx.x >= a.block0[1] ? 1 : 0;
   const long long t = (long long)(blockIdx.x - a.block0[ax]) * kThreads + threadIdx.x;
   int em = ax == 0 ? march<ORDER, 0>(a, t) : ax == 1 ? march<ORDER, 1>(a, t) : march<ORDER, 2>(a, t);
   if (a.emax) {
      em = __reduce_max_sync(0xffffffffu, em);
      if ((threadIdx.x & 31) == 0 && em > 0) atomicMax(a.emax, em);
   }
}

}  // namespace

DampSegs damp_segments(int order, const double* const dc[3], const int n[3], const int lo[3], const int hi[3])
{
   const int reach = order == 4 ? 1 : 2;
   DampSegs s;
   for (int ax = 0; ax < 3; ax++) {
      s.lo[ax][0] = s.lo[ax][1] = lo[ax];
      s.hi[ax][0] = s.hi[ax][1] = lo[ax] - 1;
      auto on = [&](int q) {
         for (int m = std::max(0, q - reach); m <= std::min(n[ax] - 1, q + reach); m++)
            if (dc[ax][m] != 0) return true;
         return false;
      };
      int a = lo[ax], b = hi[ax];
      while (a <= hi[ax] && on(a)) a++;
      while (b >= a && on(b)) b--;
      bool between = false;
      for (int q = a; q <= b; q++) between = between || on(q);
      if (a > b || between) {
         s.hi[ax][0] = hi[ax];  // one segment, the whole line
      } else {
         s.hi[ax][0] = a - 1;
         s.lo[ax][1] = b + 1;
         s.hi[ax][1] = hi[ax];
      }
   }
   return s;
}

int launch_damping_lines(int order, const Box& b, int k1, int k2, const DampSegs& seg, const double* u,
                         const double* um, double* out, const double* rho, const double* irho,
                         const double* const dc[3], const double* const st[3], const double* const co[3],
                         double beta, int* emax, cudaStream_t s)
{
   if (beta == 0) return kOk;
   if ((order != 4 && order != 6) || b.cs != b.npts) return kBadArgument;
   const int g = order == 4 ? 2 : 3;
   LineArgs a;
   a.b = b;
   a.lo[0] = a.lo[1] = g;
   a.hi[0] = b.ie - b.ib - g;
   a.hi[1] = b.je - b.jb - g;
   a.lo[2] = std::max(g, k1 - b.kb);
   a.hi[2] = std::min(b.ke - b.kb - g, k2 - b.kb);
   if (a.hi[0] < a.lo[0] || a.hi[1] < a.lo[1] || a.hi[2] < a.lo[2]) return kOk;
   a.seg = seg;
   for (int q = 0; q < 2; q++) {
      a.seg.lo[2][q] = std::max(seg.lo[2][q], a.lo[2]);
      a.seg.hi[2][q] = std::min(seg.hi[2][q], a.hi[2]);
      if (a.seg.hi[2][q] < a.seg.lo[2][q]) a.seg.hi[2][q] = a.seg.lo[2][q] - 1;
   }
   a.u = u;
   a.um = um;
   a.out = out;
   a.rho = rho;
   a.irho = irho;
   for (int q = 0; q < 3; q++) {
      a.dc[q] = dc[q];
      a.st[q] = st[q];
      a.co[q] = co[q];
   }
   a.beta = order == 4 ? beta : -0.5 * beta;
   a.emax = emax;
   // Points per thread: a longer march wastes less on its start (order + 1 differences),
   // a shorter one gives a small grid more threads.
   const long long ni = a.hi[0] - a.lo[0] + 1, nj = a.hi[1] - a.lo[1] + 1, nk = a.hi[2] - a.lo[2] + 1;
   a.len = ni * nj + nj * nk + ni * nk < 100000 ? 8 : 32;
   long long blocks = 0;
   const long long rows[3] = {nk, nk, nj}, lanes[3] = {(nj + 31) / 32 * 32, (ni + 31) / 32 * 32, (ni + 31) / 32 * 32};
   for (int ax = 0; ax < 3; ax++) {
      a.chunks[ax] = 0;
      for (int q = 0; q < 2; q++) a.chunks[ax] += (a.seg.hi[ax][q] - a.seg.lo[ax][q] + a.len) / a.len;
      a.block0[ax] = (int)blocks;
      blocks += (lanes[ax] * rows[ax] * a.chunks[ax] + kThreads - 1) / kThreads;
   }
   if (blocks == 0) return kOk;
   if (order == 4)
      damping_lines_kernel<4><<<(int)blocks, kThreads, 0, s>>>(a);
   else
      damping_lines_kernel<6><<<(int)blocks, kThreads, 0, s>>>(a);
   return launch_status();
}

}  // namespace sw4g

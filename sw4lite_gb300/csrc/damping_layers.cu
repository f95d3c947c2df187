// Supergrid damping of an FP64 level in the layers alone, sm_103a.
//
//   order 4:  out -= beta/rho   sum_a w_a D2_a(e_a D2_a(u - um))
//   order 6:  out += beta/2/rho sum_a w_a D3_a((e_a(m) + e_a(m+1)) D3_a(u - um))
//
// with e_a = rho dc_a, w_a the axis' stretching times the corner tapers of the other two
// (addsgd4fort, addsgd6fort: src/ew-cfromfort.C:748-1158).  An axis' term is exactly zero
// where its profile dc vanishes within the stencil, so only the layers' points are touched.
//
// FP64 operations bound it (1.7 per clock and SM), so each is done once: a CTA of 32 x 8
// columns marches along z, the inner differences times e are formed once per point and
// axis, those along x and y from a plane of u - um with its halo and shared through shared
// memory, those along z kept in registers: per point and component 8 operations in one
// layer and about 22 in three, where a point that evaluates its own five differences takes
// 17 for each axis.
//
// Measured with 30-point layers: order 4 at 512^3 3.1 ms (8.6 ms inside the corrector stage,
// 3.2 ms by threads that march along the damped axis), at 64^3 with 15-point layers 45 us
// (114 us by marching threads, most of whose points lie in two or three layers); order 6
// at 160 x 144 x 128 0.25 ms against 1.3 ms for the kernel that visits every point
// (pointwise.cu, the kernel-level entry points).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "stencil.cuh"

namespace sw4g {
namespace {

constexpr int TX = 32, TY = 8, kThreads = TX * TY;

struct DampArgs {
   Box b;
   int i0, i1, j0, j1, k0, k1;  // the points that may be damped
   int kchunk;
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

// ORDER 4: the inner difference at m reads d(m-1..m+1), the outer one m-1..m+1;
// ORDER 6: the inner one of the half point m + 1/2 reads d(m-1..m+2), the outer m-2..m+1.
template <int ORDER>
struct Shape {
   static constexpr int H = ORDER / 2;                       // halo of u - um
   static constexpr int PX = TX + 2 * H, PY = TY + 2 * H, PLANE = PX * PY;
   static constexpr int LO = ORDER == 4 ? 1 : 2;             // inner differences at -LO..+1
   static constexpr int GX = TX + LO + 1, GY = TY + LO + 1;
   double d[3][PLANE];  // u - um of the plane
   double gx[3][TY * GX];
   double gy[3][GY * TX];
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

// coefficient times the inner difference at a point, from v = &d and its stride
template <int ORDER>
__device__ __forceinline__ double inner(double e, const double* v, int o)
{
   // fma: 2 * x compiles to x + x, an operation more
   if (ORDER == 4) return e * (fma(-2.0, v[0], v[o]) + v[-o]);
   return e * (fma(3.0, v[0], fma(-3.0, v[o], v[2 * o])) - v[-o]);
}

// the outer difference of products at g[-LO], ..., g[1]
template <int ORDER>
__device__ __forceinline__ double outer(const double* g, int o)
{
   if (ORDER == 4) return fma(-2.0, g[0], g[o]) + g[-o];
   return fma(3.0, g[-o], fma(-3.0, g[0], g[o])) - g[-2 * o];
}

// e of the inner difference at an axis' array index n: e(n), or e(n) + e(n+1)
template <int ORDER>
__device__ __forceinline__ double coef_of(const double* __restrict__ rho, const double* __restrict__ dc, long long p, int n,
                                          long long o)
{
   const double e = __ldg(rho + p) * __ldg(dc + n);
   return ORDER == 4 ? e : __ldg(rho + p + o) * __ldg(dc + n + 1) + e;
}

template <int ORDER>
__global__ void __launch_bounds__(kThreads, 2) damping_layers_kernel(DampArgs a)
{
   using S = Shape<ORDER>;
   constexpr int H = S::H, LO = S::LO;
   extern __shared__ __align__(16) unsigned char shared[];
   S& sm = *reinterpret_cast<S*>(shared);
   const Box& b = a.b;
   const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TX * ty;
   // tiles count from both sides of the grid inwards, so that a layer fills its tiles from
   // its own side; the middle tile of an axis leaves out what the lower half has
   const int lx = gridDim.x / 2, ly = gridDim.y / 2, bx = blockIdx.x, by = blockIdx.y;
   const int i0 = bx < lx ? a.i0 + bx * TX : a.i1 + 1 - (int)(gridDim.x - bx) * TX;
   const int j0 = by < ly ? a.j0 + by * TY : a.j1 + 1 - (int)(gridDim.y - by) * TY;
   int kbeg = a.k0 + blockIdx.z * a.kchunk, kend = min(kbeg + a.kchunk - 1, a.k1);
   const int i = i0 + tx, j = j0 + ty;
   const bool active = i >= a.i0 + (bx < lx ? 0 : lx * TX) && j >= a.j0 + (by < ly ? 0 : ly * TY);
   const bool dampx = active && damped<ORDER>(a.dc[0], i - b.ib), dampy = active && damped<ORDER>(a.dc[1], j - b.jb);
   const bool anyx = __syncthreads_or(dampx) != 0, anyy = __syncthreads_or(dampy) != 0, halo = anyx || anyy;
   bool z = false;
   for (int k = kbeg + tid; k <= kend; k += kThreads) z = z || damped<ORDER>(a.dc[2], k - b.kb);
   const bool anyz = __syncthreads_or(z) != 0;
   if (!halo) {  // only the planes of the z layers
      while (kbeg <= kend && !damped<ORDER>(a.dc[2], kbeg - b.kb)) kbeg++;
      while (kend >= kbeg && !damped<ORDER>(a.dc[2], kend - b.kb)) kend--;
      if (kbeg > kend) return;
   }
   const long long npts = b.npts;
   const int col = (i - b.ib) + (int)b.ni * (j - b.jb);
   const double stx = active ? __ldg(a.st[0] + i - b.ib) : 0.0, sty = active ? __ldg(a.st[1] + j - b.jb) : 0.0;
   const double cox = active ? __ldg(a.co[0] + i - b.ib) : 0.0, coy = active ? __ldg(a.co[1] + j - b.jb) : 0.0;

   // The next plane of u and um, loaded one plane ahead: the own point, and with layers
   // along y (x) the rows above and below (the columns beside) the tile by the first warps
   double pu[2][3], pm[2][3];
   const int own = (ty + H) * S::PX + tx + H;
   int pcol[2] = {-1, -1}, pidx[2] = {own, 0};
   {
      int li = -1, lj = -1;
      if (anyy && ty < 2 * H) {
         li = tx + H;
         lj = ty < H ? ty : ty + TY;
      } else if (const int q = tid - 2 * H * TX; anyx && q >= 0 && q < 2 * H * TY) {
         li = q % (2 * H) < H ? q % (2 * H) : q % (2 * H) + TX;
         lj = q / (2 * H) + H;
      }
      const int gi = i0 - H + li, gj = j0 - H + lj;
      if (li >= 0 && gi >= b.ib && gi <= b.ie && gj >= b.jb && gj <= b.je) {
         pidx[1] = lj * S::PX + li;
         pcol[1] = (gi - b.ib) + (int)b.ni * (gj - b.jb);
      }
      if (halo && i >= b.ib && j >= b.jb) pcol[0] = col;
   }
   auto fetch = [&](int kk) {
      const long long plane = b.nij * (long long)(kk - b.kb);
#pragma unroll
      for (int r = 0; r < 2; r++)
         if (pcol[r] >= 0)
#pragma unroll
            for (int c = 0; c < 3; c++) {
               pu[r][c] = __ldg(a.u + plane + pcol[r] + c * npts);
               pm[r][c] = __ldg(a.um + plane + pcol[r] + c * npts);
            }
   };
   // the own column along z: differences and products of the planes behind
   auto diff_z = [&](int kk, int c) {
      const long long q = col + b.nij * (long long)(kk - b.kb) + c * npts;
      return __ldg(a.u + q) - __ldg(a.um + q);
   };
   auto coef_z = [&](int kk) { return __ldg(a.rho + col + b.nij * (long long)(kk - b.kb)) * __ldg(a.dc[2] + kk - b.kb); };
   double dz[3][H], gz[3][LO + 1], ez = 0;
   if (active && anyz) {
      double e[LO + 1];
      if (ORDER == 4) {
         e[0] = coef_z(kbeg - 1);
         e[1] = coef_z(kbeg);
      } else {
         const double e0 = coef_z(kbeg - 2), e1 = coef_z(kbeg - 1), e2 = coef_z(kbeg);
         ez = coef_z(kbeg + 1);
         e[0] = e1 + e0;
         e[1] = e2 + e1;
         e[LO] = ez + e2;
      }
#pragma unroll
      for (int c = 0; c < 3; c++) {
         double w[2 * H];
#pragma unroll
         for (int m = 0; m < 2 * H; m++) w[m] = diff_z(kbeg - H + m, c);
#pragma unroll
         for (int m = 0; m <= LO; m++) gz[c][m] = inner<ORDER>(e[m], w + m + 1, 1);
#pragma unroll
         for (int m = 0; m < H; m++) dz[c][m] = w[H + m];
      }
   }
   int em = 0;
   fetch(kbeg);
   for (int k = kbeg; k <= kend; k++) {
      const long long plane = b.nij * (long long)(k - b.kb), p = plane + col;
      const bool dampz = active && anyz && damped<ORDER>(a.dc[2], k - b.kb);
      if (halo) {
         double(*d)[S::PLANE] = sm.d;
#pragma unroll
         for (int r = 0; r < 2; r++)
            if (pcol[r] >= 0)
#pragma unroll
               for (int c = 0; c < 3; c++) d[c][pidx[r]] = pu[r][c] - pm[r][c];
         __syncthreads();
         if (k < kend) fetch(k + 1);
         // products of the own point and of the halo's: the first warps do the rows beyond
         // the tile, the next threads the columns
         if (anyx && i >= a.i0 - LO && j >= a.j0) {
            const double e = coef_of<ORDER>(a.rho, a.dc[0], p, i - b.ib, 1);
#pragma unroll
            for (int c = 0; c < 3; c++) sm.gx[c][ty * S::GX + tx + LO] = inner<ORDER>(e, &d[c][own], 1);
         }
         if (anyy && i >= a.i0 && j >= a.j0 - LO) {
            const double e = coef_of<ORDER>(a.rho, a.dc[1], p, j - b.jb, b.ni);
#pragma unroll
            for (int c = 0; c < 3; c++) sm.gy[c][(ty + LO) * TX + tx] = inner<ORDER>(e, &d[c][own], S::PX);
         }
         const int xt = tid - (LO + 1) * TX;
         if (anyy && tid < (LO + 1) * TX) {
            const int r = ty < LO ? ty : ty + TY, jj = j0 - LO + r;
            if (i >= a.i0 && jj >= a.j0 - LO) {
               const double e = coef_of<ORDER>(a.rho, a.dc[1], plane + (i - b.ib) + b.ni * (jj - b.jb), jj - b.jb, b.ni);
#pragma unroll
               for (int c = 0; c < 3; c++) sm.gy[c][r * TX + tx] = inner<ORDER>(e, &d[c][(r - LO + H) * S::PX + tx + H], S::PX);
            }
         } else if (anyx && xt >= 0 && xt < (LO + 1) * TY) {
            const int r = xt / (LO + 1), q = xt % (LO + 1), l = q < LO ? q : q + TX, ii = i0 - LO + l;
            if (j0 + r >= a.j0 && ii >= a.i0 - LO) {
               const double e = coef_of<ORDER>(a.rho, a.dc[0], plane + (ii - b.ib) + b.ni * (j0 + r - b.jb), ii - b.ib, 1);
#pragma unroll
               for (int c = 0; c < 3; c++) sm.gx[c][r * S::GX + l] = inner<ORDER>(e, &d[c][(r + H) * S::PX + l - LO + H], 1);
            }
         }
         __syncthreads();
      }
      double sg[3] = {0, 0, 0};
      const double coz = __ldg(a.co[2] + k - b.kb);
      if (dampx) {
         const double w = stx * coy * coz;
#pragma unroll
         for (int c = 0; c < 3; c++) sg[c] = w * outer<ORDER>(&sm.gx[c][ty * S::GX + tx + LO], 1);
      }
      if (dampy) {
         const double w = sty * cox * coz;
#pragma unroll
         for (int c = 0; c < 3; c++) sg[c] += w * outer<ORDER>(&sm.gy[c][(ty + LO) * TX + tx], TX);
      }
      if (active && anyz) {
         const double w = __ldg(a.st[2] + k - b.kb) * cox * coy;
         const double en = coef_z(k + (ORDER == 4 ? 1 : 2)), e = ORDER == 4 ? en : en + ez;
         ez = en;
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const double dn = diff_z(k + H, c);
            double v[H + 1], g[LO + 2];
#pragma unroll
            for (int m = 0; m < H; m++) v[m] = dz[c][m];
            v[H] = dn;
#pragma unroll
            for (int m = 0; m <= LO; m++) g[m] = gz[c][m];
            g[LO + 1] = inner<ORDER>(e, v + 1, 1);
            if (dampz) sg[c] += w * outer<ORDER>(g + LO, 1);
#pragma unroll
            for (int m = 0; m < H; m++) dz[c][m] = v[m + 1];
#pragma unroll
            for (int m = 0; m <= LO; m++) gz[c][m] = g[m + 1];
         }
      }
      if (dampx || dampy || dampz) {
         const double f = a.beta * __ldg(a.irho + p);
#pragma unroll
         for (int c = 0; c < 3; c++) {
            const long long q = p + c * npts;
            const double v = a.out[q] - f * sg[c];
            a.out[q] = v;
            em = max(em, (__double2hiint(v) >> 20) & 0x7ff);
         }
      }
   }
   if (a.emax) {
      em = __reduce_max_sync(0xffffffffu, em);
      if (tx == 0 && em > 0) atomicMax(a.emax, em);
   }
}

}  // namespace

namespace {
// Planes per CTA: 16 on large grids (at 512^3 16 to 32 measure alike, 4 0.6 ms more), down
// to 4 on small ones, where a CTA's march is what the launch waits for (64^3: 4 planes 5 ms
// less over a 20-step gradient than 16).
int layer_chunk(int gx, int gy, int nk) { return std::max(4, std::min(16, (int)((long long)nk * gx * gy / 1500))); }
}  // namespace

int launch_damping_layers(int order, const Box& b, int k1, int k2, const double* u, const double* um, double* out,
                          const double* rho, const double* irho, const double* const dc[3],
                          const double* const st[3], const double* const co[3], double beta, int* emax,
                          cudaStream_t s)
{
   if (beta == 0) return kOk;
   if ((order != 4 && order != 6) || b.cs != b.npts) return kBadArgument;
   const int g = order == 4 ? 2 : 3;
   DampArgs a;
   a.b = b;
   a.i0 = b.ib + g;
   a.i1 = b.ie - g;
   a.j0 = b.jb + g;
   a.j1 = b.je - g;
   a.k0 = std::max(b.kb + g, k1);
   a.k1 = std::min(b.ke - g, k2);
   if (a.i1 < a.i0 || a.j1 < a.j0 || a.k1 < a.k0) return kOk;
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
   const size_t smem = order == 4 ? sizeof(Shape<4>) : sizeof(Shape<6>);
   const void* kern = order == 4 ? (const void*)damping_layers_kernel<4> : (const void*)damping_layers_kernel<6>;
   static std::atomic<int> resident[2][64];
   if (resident_slots(resident[order == 4 ? 0 : 1], kern, kThreads, smem) < 1) return kCudaError;
   const int gx = blocks_for(a.i1 - a.i0 + 1, TX), gy = blocks_for(a.j1 - a.j0 + 1, TY), nk = a.k1 - a.k0 + 1;
   a.kchunk = layer_chunk(gx, gy, nk);
   const dim3 grid(gx, gy, (nk + a.kchunk - 1) / a.kchunk), block(TX, TY);
   if (order == 4)
      damping_layers_kernel<4><<<grid, block, smem, s>>>(a);
   else
      damping_layers_kernel<6><<<grid, block, smem, s>>>(a);
   return launch_status();
}

}  // namespace sw4g

// Poisson negative log-likelihood of ROI images and its gradient on sm_100a (no reference counterpart: the
// reference has no gradient; its nearest relative is DescribePsfCramerRao's central-difference PSF derivatives,
// adapter/inSiliScope/Simulation/PsfGeneratorBridge.cpp:1554-1669).
//
// Model: the reference's Gibson-Lanni/Zernike pupil (ZernikePsf.cpp:188-248) at matched indices and depth 0,
// at a continuous defocus z and position (x, y) per emitter:
//   U[m] = a[m] exp(i phi[m]),  phi = z kz + 2 pi sum_j c_j Z_j - p (kx x + ky y)
//   E = A U A^T  (A[s][m] = exp(i k_m p u_s), u_s = (s + 0.5) / os: the separable DFT to the ROI's sub-pixel samples)
//   mu[i][j] = N kappa sum over pixel (i, j)'s os x os samples of |E|^2 + b_frame
//   NLL = sum mu - k log mu
// and its adjoint: w = 1 - k / mu, G = w N kappa, U_bar = A^H (G o E) conj(A), dNLL/dphi = -2 Im(conj(U_bar) U),
// then the chain through phi (x, y, z, Zernike), dNLL/dN = sum w PSF, dNLL/db = sum w.
//
// One CTA per emitter at a time (a persistent grid): the pupil phase in float64, reduced mod 2 pi, then float32
// sincos; the four products (forward 32x32 -> 32x64 -> 64x64, adjoint back) folded about the ROI's centre, in float32;
// the per-emitter sums in float64. The gradient pass forms the field itself: no per-emitter PSF is stored. The
// Zernike gradient accumulates per CTA in float64 across its emitters and is added once per CTA.

#include "iscu_internal.h"
#include "psf_common.cuh"

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

struct iscu_nll_model
{
   iscu_ctx* ctx = nullptr;
   iscu_nll_spec spec{};
   int M = 0, P = 0, J = 0;
   double kappa = 0.0;
   iscu::DevBuf samples;   // M*M x double4: (p kx, p ky, kz, a)
   iscu::DevBuf basis;     // J x M*M float64: 2 pi Z_j
   iscu::DevBuf cs;        // the folded transform's cosines and sines (NllTables)
   iscu::DevBuf zphase;    // M*M float64: 2 pi sum c_j Z_j of the current evaluation
};

namespace iscu {

namespace {

constexpr int kM = 32, kP = 64, kThreads = 128, kMaxJ = 32;
constexpr int kCtasPerSm = 4;
// The aperture is the samples of |q| <= kQ, q = m - 16 on each axis (dk = 2 kMax / 28 puts its radius at 14 samples).
constexpr int kQ = 14, kR = 2 * kQ + 1, kQuad = (kQ + 1) * (kQ + 1);
constexpr int kT = kP / 2;          // sample pairs per axis
constexpr int kTp = kT + 1;         // row pitch of T in float4 (a row's lanes 4 banks apart: conflict-free)

// Two-lane float32 arithmetic: each lane rounds as the one-lane instruction.
__device__ __forceinline__ uint64_t Dup(float v)
{
   uint64_t d;
   asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "r"(__float_as_uint(v)));
   return d;
}

__device__ __forceinline__ float2 Unpack(uint64_t v)
{
   uint32_t lo, hi;
   asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
   return make_float2(__uint_as_float(lo), __uint_as_float(hi));
}

__device__ __forceinline__ uint64_t Fma2(uint64_t a, uint64_t b, uint64_t c)
{
   uint64_t d;
   asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
   return d;
}

// Sums of NV float64 values over the CTA in one exchange (every thread calls it; every thread gets the sums). red:
// NV x (kThreads / 32) doubles.
template <int NV>
__device__ __forceinline__ void BlockSums(double (&v)[NV], double* red)
{
#pragma unroll
   for (int q = 0; q < NV; ++q)
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
         v[q] += __shfl_xor_sync(0xffffffffu, v[q], d);
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   __syncthreads();
   if (lane == 0)
#pragma unroll
      for (int q = 0; q < NV; ++q)
         red[q * (kThreads / 32) + warp] = v[q];
   __syncthreads();
#pragma unroll
   for (int q = 0; q < NV; ++q)
   {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w)
         t += red[q * (kThreads / 32) + w];
      v[q] = t;
   }
}

// What an evaluation needs before its emitters, in one launch (a copy, four clears and a kernel of their own were half a
// live fit's time on the device): the Zernike phase of every pupil sample, and the accumulated outputs cleared.
struct PrepareArgs
{
   const double* basis;
   int J, MM;
   const double* zernDev;   // nullable: the coefficients are in `zern`
   double zern[kMaxJ];
   double* zphase;
   double* nll;
   int* err;
   double* gBg;             // nullable
   uint32_t nFrames;
   double* gZern;           // nullable
};

__global__ void __launch_bounds__(256) NllPrepareKernel(PrepareArgs a)
{
   __shared__ double z[kMaxJ];
   if (threadIdx.x < kMaxJ)
      z[threadIdx.x] = static_cast<int>(threadIdx.x) >= a.J ? 0.0
                       : a.zernDev                         ? a.zernDev[threadIdx.x]
                                                           : a.zern[threadIdx.x];
   __syncthreads();
   const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
   if (static_cast<int>(i) < a.MM)
   {
      double s = 0.0;
#pragma unroll 8
      for (int j = 0; j < a.J; ++j)
         s += z[j] * a.basis[static_cast<size_t>(j) * a.MM + i];
      a.zphase[i] = s;
   }
   if (i == 0)
   {
      *a.nll = 0.0;
      *a.err = 0;
   }
   if (a.gZern && static_cast<int>(i) < a.J)
      a.gZern[i] = 0.0;
   if (a.gBg && i < a.nFrames)
      a.gBg[i] = 0.0;
}

struct NllArgs
{
   const double4* samples;
   const double* basis;
   const float* cs;          // the folded transform's cosines and sines (NllTables)
   const double* zphase;
   int J, R;
   double kappa;
   uint32_t n;
   const float4* params;     // x, y (ROI px), z (nm), N
   const int32_t* frame;
   uint32_t nFrames;
   const float* bg;
   const float* counts;      // n x R x R
   float* mu;                // nullable
   double* nll;              // accumulated
   float4* gParams;          // nullable: the gradient pass
   double* gBg;
   double* gZern;
   int* err;                 // 1: an emitter names a frame outside the batch
};

// cos / sin of q theta (t + 1/2), theta = dk p / os, laid out as the products read them: fwd[q - 1][w] the cosines then
// the sines of t = 8 w .. 8 w + 7 (q = 1 .. kQ), adj[t][w] those of q = 4 w .. 4 w + 3 (q beyond kQ: zeros).
struct NllTables
{
   float fwd[kQ][4][16];
   float adj[kT][4][8];
};

struct NllSmem
{
   NllTables tab;
   float4 T[kR][kTp];         // T, then its adjoint: row r, sample pair t
   union
   {
      float4 U[kQ + 1][32];   // the folded pupil, then its adjoint: (P.re, P.im, N.re, N.im) of column pair q, row r
      struct
      {
         float4 C[kT / 2][32], S[kT / 2][32];   // half of the weighted field's row sums and differences
      } E;
      double blk[64 + 64];    // ROIs of at most 4 x 4 pixels: the 8 x 8-sample blocks' sums, the pixels' weights
   };
   float4 Uraw[2][kQuad];     // the pupil: (+y +x, +y -x), (-y +x, -y -x) of each quadrant sample
   double dphiSum[4][kQuad];  // the CTA's emitters' dNLL/dphi, summed in float64, for the Zernike gradient
   double red[5 * (kThreads / 32)];
};

// One pixel's likelihood terms from its sample sum: the expected counts, the NLL's term and, for the gradient, the
// sums' terms and the samples' weight.
struct PixelSums
{
   double part = 0.0, gN = 0.0, gB = 0.0;
};

// NP pixels of a thread in stages, so that their float64 chains (the logarithm, the quotient) run side by side.
template <bool kGrad, int NP>
__device__ __forceinline__ void Pixels(const NllArgs& a, uint32_t e, const int (&p)[NP], const bool (&on)[NP],
                                       const float (&sum)[NP], double N, double b, PixelSums& s, float (&G)[NP])
{
   const size_t base = static_cast<size_t>(e) * a.R * a.R;
   float k[NP];
   double mu[NP], lg[NP];
#pragma unroll
   for (int q = 0; q < NP; ++q)
      k[q] = on[q] ? __ldg(a.counts + base + p[q]) : 0.f;
#pragma unroll
   for (int q = 0; q < NP; ++q)
      mu[q] = on[q] ? N * (a.kappa * static_cast<double>(sum[q])) + b : 1.0;
#pragma unroll
   for (int q = 0; q < NP; ++q)
      lg[q] = log(mu[q]);
#pragma unroll
   for (int q = 0; q < NP; ++q)
   {
      const double kk = static_cast<double>(k[q]);
      if (on[q])
      {
         s.part += mu[q] - kk * lg[q];
         if (a.mu)
            a.mu[base + p[q]] = static_cast<float>(mu[q]);
      }
      if (kGrad)
      {
         const double w = on[q] ? 1.0 - kk / mu[q] : 0.0;
         s.gN += w * (a.kappa * static_cast<double>(sum[q]));
         s.gB += w;
         G[q] = static_cast<float>(w * N * a.kappa);
      }
   }
}

// A CTA of four warps takes an emitter at a time; OS: the samples per pixel and axis (1, 2, 4, 8; 0: 16 and more).
//
// Both products are folded. The samples are symmetric about the ROI's centre (their common phase ramp goes into the
// pupil as a shift by half the ROI), so exp(i q theta tau) of +-q and +-tau are one cosine and one sine: a row of U
// is folded into P = U[q] + U[-q] and N = U[q] - U[-q], and C = sum cos P, S = sum sin N give the samples C + i S at
// +tau and C - i S at -tau -- real by complex products of a quarter of the size. With the aperture's 29 of the 32
// samples an emitter's four products take 334 K multiply-adds instead of 1.57 M, exactly the same sums.
//
// What bounds it: shared-memory wavefronts (79 % of the data path with gradients, 62 % without; each product reads its
// constants by broadcast -- a warp's t or q group is the same for its lanes, and such a 16-byte read takes two -- and its
// data once per lane), then the float64 logarithm of each pixel. 128 threads and 55 KB, four CTAs per SM, so that one
// CTA's products run under another's logarithms and barriers. 256,000 emitters of 32 x 32 px, os = 2: likelihood and
// gradients 7.7 ms (unfolded 23.3), the likelihood alone 3.7 (11.6). Constants as kernel parameters were slower (the
// two passes 14.0 ms against 11.7).
template <bool kGrad, int OS>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) NllKernel(NllArgs a)
{
   extern __shared__ __align__(16) unsigned char smemRaw[];
   NllSmem& s = *reinterpret_cast<NllSmem*>(smemRaw);
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   for (int i = tid; i < static_cast<int>(sizeof(NllTables) / sizeof(float)); i += kThreads)
      reinterpret_cast<float*>(&s.tab)[i] = a.cs[i];
   if (kGrad)
      for (int m = tid; m < 4 * kQuad; m += kThreads)
         s.dphiSum[m / kQuad][m % kQuad] = 0.0;
   double nllAcc = 0.0;
   const int R = a.R, RR = R * R;
   for (uint32_t e = blockIdx.x; e < a.n; e += gridDim.x)
   {
      const float4 pr = a.params[e];
      const int f = a.frame[e];
      const bool frameOk = f >= 0 && static_cast<uint32_t>(f) < a.nFrames;
      if (!frameOk && tid == 0)
         atomicExch(a.err, 1);
      const double b = frameOk ? static_cast<double>(a.bg[f]) : 0.0;
      // the position from the ROI's centre: the samples' common ramp
      const double x = static_cast<double>(pr.x) - 0.5 * R, y = static_cast<double>(pr.y) - 0.5 * R, z = pr.z, N = pr.w;
      // the next emitter's counts on their way to L2 while this one computes
      if (e + gridDim.x < a.n && tid * 32 < RR)
         asm volatile("prefetch.global.L2 [%0];" ::"l"(a.counts + static_cast<size_t>(e + gridDim.x) * RR + tid * 32));
      // 1. the pupil, folded: a thread per quadrant sample and its mirrors
      for (int qd = tid; qd < kQuad; qd += kThreads)
      {
         const int qy = qd / (kQ + 1), qx = qd % (kQ + 1), m0 = kM / 2 * kM + kM / 2;
         const double4 sm = a.samples[m0 + qy * kM + qx];
         const double zk = z * sm.z, ax = sm.x * x, ay = sm.y * y;
         const float amp = static_cast<float>(sm.w);
         float2 u[2][2];
#pragma unroll
         for (int iy = 0; iy < 2; ++iy)
#pragma unroll
            for (int ix = 0; ix < 2; ++ix)
            {
               const int m = m0 + (iy ? -qy : qy) * kM + (ix ? -qx : qx);
               // in revolutions, less the whole ones. (The fast sine and cosine, 2^-21 off, were half of the gradients'
               // error; the folded products' own roundings are the other half.)
               const double ph = (zk + a.zphase[m] - ((ix ? -ax : ax) + (iy ? -ay : ay))) * 0.15915494309189533577;
               float sn, cs;
               sincospif(2.f * static_cast<float>(ph - rint(ph)), &sn, &cs);
               const float am = (iy && qy == 0) || (ix && qx == 0) ? 0.f : amp;   // one sample on an axis, not two
               u[iy][ix] = make_float2(am * cs, am * sn);
            }
         if (kGrad)
         {
            s.Uraw[0][qd] = make_float4(u[0][0].x, u[0][0].y, u[0][1].x, u[0][1].y);
            s.Uraw[1][qd] = make_float4(u[1][0].x, u[1][0].y, u[1][1].x, u[1][1].y);
         }
         const float2 p0 = make_float2(u[0][0].x + u[0][1].x, u[0][0].y + u[0][1].y);
         const float2 n0 = make_float2(u[0][0].x - u[0][1].x, u[0][0].y - u[0][1].y);
         const float2 p1 = make_float2(u[1][0].x + u[1][1].x, u[1][0].y + u[1][1].y);
         const float2 n1 = make_float2(u[1][0].x - u[1][1].x, u[1][0].y - u[1][1].y);
         s.U[qx][qy] = make_float4(p0.x + p1.x, p0.y + p1.y, n0.x + n1.x, n0.y + n1.y);
         if (qy)
            s.U[qx][kQ + qy] = make_float4(p0.x - p1.x, p0.y - p1.y, n0.x - n1.x, n0.y - n1.y);
      }
      __syncthreads();
      // 2. T = U A^T over the folded rows: lane = row, a warp's eight t
      {
         const int r = min(lane, kR - 1);
         uint64_t cre[4], cim[4], sre[4], sim[4];
         const float4 u0 = s.U[0][r];
#pragma unroll
         for (int k = 0; k < 4; ++k)
         {
            cre[k] = Dup(u0.x);
            cim[k] = Dup(u0.y);
            sre[k] = sim[k] = 0;
         }
#pragma unroll 2
         for (int q = 1; q <= kQ; ++q)
         {
            const float4 u = s.U[q][r];
            const ulonglong2* t = reinterpret_cast<const ulonglong2*>(s.tab.fwd[q - 1][warp]);
            const ulonglong2 c0 = t[0], c1 = t[1], s0 = t[2], s1 = t[3];
            const uint64_t c[4] = {c0.x, c0.y, c1.x, c1.y}, sn[4] = {s0.x, s0.y, s1.x, s1.y};
            const uint64_t pr2 = Dup(u.x), pi2 = Dup(u.y), nr2 = Dup(u.z), ni2 = Dup(u.w);
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
               cre[k] = Fma2(c[k], pr2, cre[k]);
               cim[k] = Fma2(c[k], pi2, cim[k]);
               sre[k] = Fma2(sn[k], nr2, sre[k]);
               sim[k] = Fma2(sn[k], ni2, sim[k]);
            }
         }
         if (lane < kR)
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
               const float2 cr = Unpack(cre[k]), ci = Unpack(cim[k]), sr = Unpack(sre[k]), si = Unpack(sim[k]);
               s.T[r][8 * warp + 2 * k] = make_float4(cr.x - si.x, ci.x + sr.x, cr.x + si.x, ci.x - sr.x);
               s.T[r][8 * warp + 2 * k + 1] = make_float4(cr.y - si.y, ci.y + sr.y, cr.y + si.y, ci.y - sr.y);
            }
      }
      __syncthreads();
      // 3. E = A T: lane = the column pair +-t, a warp's eight row pairs. E[row sign][column sign][row]
      float2 E[2][2][8];
      {
         uint64_t cre[2][4], cim[2][4], sre[2][4], sim[2][4];
         const float4 t0 = s.T[0][lane];
#pragma unroll
         for (int k = 0; k < 4; ++k)
         {
            cre[0][k] = Dup(t0.x);
            cim[0][k] = Dup(t0.y);
            cre[1][k] = Dup(t0.z);
            cim[1][k] = Dup(t0.w);
            sre[0][k] = sim[0][k] = sre[1][k] = sim[1][k] = 0;
         }
#pragma unroll 2
         for (int q = 1; q <= kQ; ++q)
         {
            const float4 tp = s.T[q][lane], tn = s.T[kQ + q][lane];
            const ulonglong2* t = reinterpret_cast<const ulonglong2*>(s.tab.fwd[q - 1][warp]);
            const ulonglong2 c0 = t[0], c1 = t[1], s0 = t[2], s1 = t[3];
            const uint64_t c[4] = {c0.x, c0.y, c1.x, c1.y}, sn[4] = {s0.x, s0.y, s1.x, s1.y};
            {
               const uint64_t d0 = Dup(tp.x), d1 = Dup(tp.y), d2 = Dup(tp.z), d3 = Dup(tp.w);
#pragma unroll
               for (int k = 0; k < 4; ++k)
               {
                  cre[0][k] = Fma2(c[k], d0, cre[0][k]);
                  cim[0][k] = Fma2(c[k], d1, cim[0][k]);
                  cre[1][k] = Fma2(c[k], d2, cre[1][k]);
                  cim[1][k] = Fma2(c[k], d3, cim[1][k]);
               }
            }
            const uint64_t d0 = Dup(tn.x), d1 = Dup(tn.y), d2 = Dup(tn.z), d3 = Dup(tn.w);
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
               sre[0][k] = Fma2(sn[k], d0, sre[0][k]);
               sim[0][k] = Fma2(sn[k], d1, sim[0][k]);
               sre[1][k] = Fma2(sn[k], d2, sre[1][k]);
               sim[1][k] = Fma2(sn[k], d3, sim[1][k]);
            }
         }
#pragma unroll
         for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
               const float2 cr = Unpack(cre[c][k]), ci = Unpack(cim[c][k]), sr = Unpack(sre[c][k]),
                            si = Unpack(sim[c][k]);
               E[0][c][2 * k] = make_float2(cr.x - si.x, ci.x + sr.x);
               E[1][c][2 * k] = make_float2(cr.x + si.x, ci.x - sr.x);
               E[0][c][2 * k + 1] = make_float2(cr.y - si.y, ci.y + sr.y);
               E[1][c][2 * k + 1] = make_float2(cr.y + si.y, ci.y - sr.y);
            }
      }
      // 4. expected counts and the likelihood. A pixel's samples: OS of a thread's rows by OS neighbouring lanes; the
      // lanes exchange their row sums, each takes its share of the pixels and hands their weights back.
      PixelSums ps;
      constexpr int kOS = OS ? OS : 8, kG = 8 / kOS, kNp = 4 * kG;   // row groups of a thread; pixels of a lane group
      float W[kNp];   // pixel n = (group, row sign, column sign)
#pragma unroll
      for (int n = 0; n < kNp; ++n)
      {
         float v = 0.f;
#pragma unroll
         for (int k = 0; k < kOS; ++k)
         {
            const float2 q = E[(n >> 1) & 1][n & 1][(n >> 2) * kOS + k];
            v = fmaf(q.x, q.x, fmaf(q.y, q.y, v));
         }
#pragma unroll
         for (int d = 1; d < kOS; d <<= 1)
            v += __shfl_xor_sync(0xffffffffu, v, d);
         W[n] = v;
      }
      if (OS)
      {
         constexpr int kBatch = kNp >= 4 * kOS ? 4 : (kNp + kOS - 1) / kOS;   // pixels of a lane per stage
         const int sub = lane % kOS;
         const int rc = R / 2 + lane / kOS, rr = R / 2 + warp * kG;   // the group's +column, the first +row
#pragma unroll
         for (int n0 = 0; n0 < kNp; n0 += kBatch * kOS)
         {
            int p[kBatch];
            bool on[kBatch];
            float sum[kBatch], G[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i)
            {
               sum[i] = 0.f;
               p[i] = 0;
               on[i] = false;
#pragma unroll
               for (int o = 0; o < kOS; ++o)
               {
                  const int n = n0 + i * kOS + o;
                  if (n < kNp && sub == o)
                  {
                     const int row = (n >> 1) & 1 ? R - 1 - (rr + (n >> 2)) : rr + (n >> 2);
                     const int col = n & 1 ? R - 1 - rc : rc;
                     sum[i] = W[n];
                     p[i] = row * R + col;
                     on[i] = true;
                  }
               }
               G[i] = 0.f;
            }
            Pixels<kGrad, kBatch>(a, e, p, on, sum, N, b, ps, G);
            if (kGrad)
#pragma unroll
               for (int i = 0; i < kBatch; ++i)
#pragma unroll
                  for (int o = 0; o < kOS; ++o)
                     if (n0 + i * kOS + o < kNp)
                        W[n0 + i * kOS + o] = kOS == 1 ? G[i]
                                                       : __shfl_sync(0xffffffffu, G[i], (lane & ~(kOS - 1)) | o);
         }
      }
      else
      {
         // 16 samples a pixel and more: the 8 x 8 grid of 8 x 8-sample blocks through shared memory
         double* blk = s.blk;
         const int bc = lane / 8;
         if (lane % 8 == 0)
#pragma unroll
            for (int n = 0; n < 4; ++n)
               blk[((n >> 1) & 1 ? 3 - warp : 4 + warp) * 8 + (n & 1 ? 3 - bc : 4 + bc)] = W[n];
         __syncthreads();
         const int per = 8 / R;   // blocks per pixel and axis
         int p[1] = {tid};
         bool on[1] = {tid < RR};
         float sum[1] = {0.f}, G[1] = {0.f};
         if (on[0])
            for (int by = 0; by < per; ++by)
               for (int bx = 0; bx < per; ++bx)
                  sum[0] += static_cast<float>(blk[(tid / R * per + by) * 8 + tid % R * per + bx]);
         Pixels<kGrad, 1>(a, e, p, on, sum, N, b, ps, G);
         if (kGrad)
         {
            if (on[0])
               blk[64 + tid] = G[0];
            __syncthreads();
#pragma unroll
            for (int n = 0; n < 4; ++n)
               W[n] = static_cast<float>(blk[64 + ((n >> 1) & 1 ? 3 - warp : 4 + warp) / per * R +
                                             (n & 1 ? 3 - bc : 4 + bc) / per]);
            __syncthreads();   // the adjoint's first writes share the memory
         }
      }
      nllAcc += ps.part;
      if (!kGrad)
      {
         if (!OS)
            __syncthreads();   // the blocks share the next pupil's memory
         continue;
      }
      // 5. T_bar = A^H (G o E): lane = the column pair, a warp's four q; the row pairs' sums and differences through
      // shared memory in two halves of every warp's rows
      uint64_t pre[2][2], pim[2][2], nre[2][2], nim[2][2];   // [column sign][q pair]
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
         for (int k = 0; k < 2; ++k)
            pre[c][k] = pim[c][k] = nre[c][k] = nim[c][k] = 0;
#pragma unroll
      for (int half = 0; half < 2; ++half)
      {
         if (half)
            __syncthreads();
#pragma unroll
         for (int k = 0; k < 4; ++k)
         {
            const int row = 4 * half + k, g = 4 * (row / kOS);
            float2 up[2], dn[2];
#pragma unroll
            for (int c = 0; c < 2; ++c)
            {
               const float2 ep = E[0][c][row], em = E[1][c][row];
               const float gp = W[g + c], gm = W[g + 2 + c];
               const float2 wp = make_float2(gp * ep.x, gp * ep.y), wm = make_float2(gm * em.x, gm * em.y);
               up[c] = make_float2(wp.x + wm.x, wp.y + wm.y);
               dn[c] = make_float2(wp.y - wm.y, wm.x - wp.x);   // -i (+ minus -)
            }
            s.E.C[4 * warp + k][lane] = make_float4(up[0].x, up[0].y, up[1].x, up[1].y);
            s.E.S[4 * warp + k][lane] = make_float4(dn[0].x, dn[0].y, dn[1].x, dn[1].y);
         }
         __syncthreads();
#pragma unroll 2
         for (int i = 0; i < kT / 2; ++i)
         {
            const float4 ec = s.E.C[i][lane], es = s.E.S[i][lane];
            const ulonglong2* t =
               reinterpret_cast<const ulonglong2*>(s.tab.adj[8 * (i >> 2) + 4 * half + (i & 3)][warp]);
            const ulonglong2 c2 = t[0], s2 = t[1];
            const uint64_t c[2] = {c2.x, c2.y}, sn[2] = {s2.x, s2.y};
            const uint64_t c0 = Dup(ec.x), c1 = Dup(ec.y), c3 = Dup(ec.z), c4 = Dup(ec.w);
            const uint64_t d0 = Dup(es.x), d1 = Dup(es.y), d3 = Dup(es.z), d4 = Dup(es.w);
#pragma unroll
            for (int k = 0; k < 2; ++k)
            {
               pre[0][k] = Fma2(c[k], c0, pre[0][k]);
               pim[0][k] = Fma2(c[k], c1, pim[0][k]);
               pre[1][k] = Fma2(c[k], c3, pre[1][k]);
               pim[1][k] = Fma2(c[k], c4, pim[1][k]);
               nre[0][k] = Fma2(sn[k], d0, nre[0][k]);
               nim[0][k] = Fma2(sn[k], d1, nim[0][k]);
               nre[1][k] = Fma2(sn[k], d3, nre[1][k]);
               nim[1][k] = Fma2(sn[k], d4, nim[1][k]);
            }
         }
      }
      // the columns folded: (+t plus -t, -i (+t minus -t)) of each row
#pragma unroll
      for (int k = 0; k < 2; ++k)
      {
         const float2 a0 = Unpack(pre[0][k]), a1 = Unpack(pim[0][k]), b0 = Unpack(pre[1][k]), b1 = Unpack(pim[1][k]);
         const float2 e0 = Unpack(nre[0][k]), e1 = Unpack(nim[0][k]), f0 = Unpack(nre[1][k]), f1 = Unpack(nim[1][k]);
         const int q = 4 * warp + 2 * k;
         if (q <= kQ)
            s.T[q][lane] = make_float4(a0.x + b0.x, a1.x + b1.x, a1.x - b1.x, b0.x - a0.x);
         if (q + 1 <= kQ)
            s.T[q + 1][lane] = make_float4(a0.y + b0.y, a1.y + b1.y, a1.y - b1.y, b0.y - a0.y);
         if (q >= 1 && q <= kQ)
            s.T[kQ + q][lane] = make_float4(e0.x + f0.x, e1.x + f1.x, e1.x - f1.x, f0.x - e0.x);
         if (q + 1 <= kQ)
            s.T[kQ + q + 1][lane] = make_float4(e0.y + f0.y, e1.y + f1.y, e1.y - f1.y, f0.y - e0.y);
      }
      __syncthreads();
      // 6. U_bar = T_bar conj(A), folded: lane = row, a warp's four q
      {
         const int r = min(lane, kR - 1);
         uint64_t upr[2] = {0, 0}, upi[2] = {0, 0}, unr[2] = {0, 0}, uni[2] = {0, 0};
#pragma unroll 4
         for (int i = 0; i < kT; ++i)
         {
            const float4 t = s.T[r][i];
            const ulonglong2* tb = reinterpret_cast<const ulonglong2*>(s.tab.adj[i][warp]);
            const ulonglong2 c2 = tb[0], s2 = tb[1];
            const uint64_t c[2] = {c2.x, c2.y}, sn[2] = {s2.x, s2.y};
            const uint64_t cr = Dup(t.x), ci = Dup(t.y), sr = Dup(t.z), si = Dup(t.w);
#pragma unroll
            for (int k = 0; k < 2; ++k)
            {
               upr[k] = Fma2(c[k], cr, upr[k]);
               upi[k] = Fma2(c[k], ci, upi[k]);
               unr[k] = Fma2(sn[k], sr, unr[k]);
               uni[k] = Fma2(sn[k], si, uni[k]);
            }
         }
#pragma unroll
         for (int k = 0; k < 2; ++k)
         {
            const float2 pr2 = Unpack(upr[k]), pi2 = Unpack(upi[k]), nr2 = Unpack(unr[k]), ni2 = Unpack(uni[k]);
            const int q = 4 * warp + 2 * k;
            if (q <= kQ)
               s.U[q][lane] = make_float4(pr2.x, pi2.x, nr2.x, ni2.x);
            if (q + 1 <= kQ)
               s.U[q + 1][lane] = make_float4(pr2.y, pi2.y, nr2.y, ni2.y);
         }
      }
      __syncthreads();
      // 7. dNLL/dphi of each quadrant sample and its mirrors, and the chain through phi
      double sums[5] = {0.0, 0.0, 0.0, ps.gN, ps.gB};
      for (int qd = tid; qd < kQuad; qd += kThreads)
      {
         const int qy = qd / (kQ + 1), qx = qd % (kQ + 1);
         const double4 sm = a.samples[kM / 2 * kM + kM / 2 + qy * kM + qx];
         const float4 p = s.U[qx][qy], u0 = s.Uraw[0][qd], u1 = s.Uraw[1][qd];
         float4 n = make_float4(0.f, 0.f, 0.f, 0.f);
         if (qy)
            n = s.U[qx][kQ + qy];
         // U_bar of (sy, sx) = PP + sy NP + sx (PN + sy NN); -2 Im(conj(U_bar) U) = -2 (Ubar.x u.y - Ubar.y u.x)
         const float2 a0 = make_float2(p.x + n.x, p.y + n.y), a1 = make_float2(p.x - n.x, p.y - n.y);
         const float2 b0 = make_float2(p.z + n.z, p.w + n.w), b1 = make_float2(p.z - n.z, p.w - n.w);
         const float d0 = -2.f * ((a0.x + b0.x) * u0.y - (a0.y + b0.y) * u0.x);
         const float d1 = -2.f * ((a0.x - b0.x) * u0.w - (a0.y - b0.y) * u0.z);
         const float d2 = -2.f * ((a1.x + b1.x) * u1.y - (a1.y + b1.y) * u1.x);
         const float d3 = -2.f * ((a1.x - b1.x) * u1.w - (a1.y - b1.y) * u1.z);
         const double e0 = d0, e1 = d1, e2 = d2, e3 = d3;
         sums[0] -= ((e0 - e1) + (e2 - e3)) * sm.x;
         sums[1] -= ((e0 + e1) - (e2 + e3)) * sm.y;
         sums[2] += ((e0 + e1) + (e2 + e3)) * sm.z;
         s.dphiSum[0][qd] += e0;
         s.dphiSum[1][qd] += e1;
         s.dphiSum[2][qd] += e2;
         s.dphiSum[3][qd] += e3;
      }
      BlockSums<5>(sums, s.red);
      if (tid == 0)
      {
         a.gParams[e] = make_float4(static_cast<float>(sums[0]), static_cast<float>(sums[1]),
                                    static_cast<float>(sums[2]), static_cast<float>(sums[3]));
         if (frameOk)
            atomicAdd(&a.gBg[f], sums[4]);
      }
   }
   // the CTA's sums
   double nllCta[1] = {nllAcc};
   BlockSums<1>(nllCta, s.red);
   if (tid == 0)
      atomicAdd(a.nll, nllCta[0]);
   if (kGrad)
   {
      // warp w projects the summed dphi onto modes j = w, w + 4, ...
      __syncthreads();
      for (int j = warp; j < a.J; j += kThreads / 32)
      {
         const double* Zj = a.basis + static_cast<size_t>(j) * kM * kM + kM / 2 * kM + kM / 2;
         double v = 0.0;
         for (int qd = lane; qd < kQuad; qd += 32)
         {
            const int o = qd / (kQ + 1) * kM, qx = qd % (kQ + 1);
            v += (s.dphiSum[0][qd] * Zj[o + qx] + s.dphiSum[1][qd] * Zj[o - qx]) +
                 (s.dphiSum[2][qd] * Zj[-o + qx] + s.dphiSum[3][qd] * Zj[-o - qx]);
         }
#pragma unroll
         for (int d = 16; d > 0; d >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, d);
         if (lane == 0)
            atomicAdd(&a.gZern[j], v);
      }
   }
}

using NllFn = void (*)(NllArgs);
template <bool kGrad>
NllFn NllOf(int os)
{
   switch (os)
   {
   case 1: return NllKernel<kGrad, 1>;
   case 2: return NllKernel<kGrad, 2>;
   case 4: return NllKernel<kGrad, 4>;
   case 8: return NllKernel<kGrad, 8>;
   default: return NllKernel<kGrad, 0>;
   }
}

// Noll's orthonormal Z_j (n, m from j) at (rho, theta).
void NollNm(int j, int& n, int& m)
{
   n = 0;
   int j1 = j - 1;
   while (j1 > n)
   {
      ++n;
      j1 -= n;
   }
   m = ((j % 2) ? -1 : 1) * ((n % 2) + 2 * ((j1 + ((n + 1) % 2)) / 2));
}

double Factorial(int k)
{
   double f = 1.0;
   for (int i = 2; i <= k; ++i)
      f *= i;
   return f;
}

double ZernikeNoll(int j, double rho, double theta)
{
   int n, m;
   NollNm(j, n, m);
   const int am = m < 0 ? -m : m;
   double r = 0.0;
   for (int s = 0; s <= (n - am) / 2; ++s)
   {
      const double c = ((s % 2) ? -1.0 : 1.0) * Factorial(n - s) /
                       (Factorial(s) * Factorial((n + am) / 2 - s) * Factorial((n - am) / 2 - s));
      r += c * std::pow(rho, n - 2 * s);
   }
   if (m == 0)
      return std::sqrt(n + 1.0) * r;
   return std::sqrt(2.0 * (n + 1)) * r * (m > 0 ? std::cos(am * theta) : std::sin(am * theta));
}

} // namespace

} // namespace iscu

using namespace iscu;

extern "C" {

int iscu_nll_model_create(iscu_ctx* ctx, const iscu_nll_spec* spec, iscu_nll_model** out)
{
   if (!ctx || !spec || !out)
      return Fail(ISCU_ERR_ARG, "null argument");
   *out = nullptr;
   if (spec->pupil != kM || spec->roi * spec->os != kP || spec->roi < 1 || spec->os < 1)
      return Fail(ISCU_ERR_LIMIT, "the gradient model takes a 32 x 32 pupil and roi * os = 64 samples");
   if (spec->n_zern < 0 || spec->n_zern > kMaxJ)
      return Fail(ISCU_ERR_LIMIT, "at most 32 Zernike modes");
   if (!(spec->wavelength_nm > 0.0) || !(spec->na > 0.0) || !(spec->n_imm >= spec->na) || !(spec->pixel_nm > 0.0))
      return Fail(ISCU_ERR_ARG, "wavelength, NA, immersion index >= NA and pixel size must be positive");
   for (int j = 0; j < spec->n_zern; ++j)
      if (spec->noll[j] < 1 || spec->noll[j] > 66)
         return Fail(ISCU_ERR_ARG, "Noll indices 1..66");
   std::lock_guard<std::recursive_mutex> lock(ctx->mu);
   ClearError();
   std::unique_ptr<iscu_nll_model> mdl(new iscu_nll_model());
   mdl->ctx = ctx;
   mdl->spec = *spec;
   const int M = kM, P = kP, J = spec->n_zern, MM = M * M;
   mdl->M = M;
   mdl->P = P;
   mdl->J = J;
   const double pi = 3.14159265358979323846;
   const double kmax = 2.0 * pi * spec->na / spec->wavelength_nm, dk = 2.0 * kmax / (M - 4);
   const double k0n = 2.0 * pi * spec->n_imm / spec->wavelength_nm;
   std::vector<double> samp(4 * static_cast<size_t>(MM)), basis(static_cast<size_t>(J) * MM, 0.0);
   double aSum = 0.0;
   for (int iy = 0; iy < M; ++iy)
      for (int ix = 0; ix < M; ++ix)
      {
         const int m = iy * M + ix;
         const double ky = (iy - M / 2) * dk, kx = (ix - M / 2) * dk, kr2 = kx * kx + ky * ky;
         const bool in = kr2 <= kmax * kmax;
         samp[4 * m + 0] = spec->pixel_nm * kx;
         samp[4 * m + 1] = spec->pixel_nm * ky;
         samp[4 * m + 2] = in ? std::sqrt(std::max(0.0, k0n * k0n - kr2)) : 0.0;
         samp[4 * m + 3] = in ? 1.0 : 0.0;
         aSum += in ? 1.0 : 0.0;
         if (in)
            for (int j = 0; j < J; ++j)
               basis[static_cast<size_t>(j) * MM + m] =
                  2.0 * pi * ZernikeNoll(spec->noll[j], std::sqrt(kr2) / kmax, std::atan2(ky, kx));
      }
   NllTables tab = {};
   for (int t = 0; t < kT; ++t)
      for (int q = 0; q <= kQ; ++q)
      {
         const double ph = q * dk * spec->pixel_nm * ((t + 0.5) / spec->os);
         const float c = static_cast<float>(std::cos(ph)), sn = static_cast<float>(std::sin(ph));
         if (q)
         {
            tab.fwd[q - 1][t / 8][t % 8] = c;
            tab.fwd[q - 1][t / 8][8 + t % 8] = sn;
         }
         tab.adj[t][q / 4][q % 4] = c;
         tab.adj[t][q / 4][4 + q % 4] = sn;
      }
   const double L = 2.0 * pi / dk, px = spec->pixel_nm / spec->os;
   mdl->kappa = px * px / (L * L * aSum);
   ISCU_CK(mdl->samples.Reserve(samp.size() * sizeof(double)));
   ISCU_CK(mdl->basis.Reserve(std::max<size_t>(basis.size(), 1) * sizeof(double)));
   ISCU_CK(mdl->cs.Reserve(sizeof(NllTables)));
   ISCU_CK(mdl->zphase.Reserve(MM * sizeof(double)));
   ISCU_CK(cudaMemcpyAsync(mdl->samples.p, samp.data(), samp.size() * sizeof(double), cudaMemcpyHostToDevice,
                           ctx->stream));
   if (!basis.empty())
      ISCU_CK(cudaMemcpyAsync(mdl->basis.p, basis.data(), basis.size() * sizeof(double), cudaMemcpyHostToDevice,
                              ctx->stream));
   ISCU_CK(cudaMemcpyAsync(mdl->cs.p, &tab, sizeof(tab), cudaMemcpyHostToDevice, ctx->stream));
   ISCU_CK(cudaStreamSynchronize(ctx->stream));
   for (NllFn fn : {NllOf<false>(spec->os), NllOf<true>(spec->os)})
      ISCU_CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(NllSmem))));
   *out = mdl.release();
   return ISCU_OK;
}

void iscu_nll_model_destroy(iscu_nll_model* model)
{
   if (!model)
      return;
   cudaStreamSynchronize(model->ctx->stream);
   delete model;
}

int iscu_nll_model_info(iscu_nll_model* model, double* kappa, int32_t* n_zern)
{
   if (!model)
      return Fail(ISCU_ERR_ARG, "null model");
   if (kappa)
      *kappa = model->kappa;
   if (n_zern)
      *n_zern = model->J;
   return ISCU_OK;
}

int iscu_nll_eval_dev(iscu_nll_model* model, uint32_t n_emitters, const float* params_dev, const int32_t* frame_dev,
                      uint32_t n_frames, const float* bg_dev, const double* zern, const float* counts_dev,
                      float* mu_dev, double* nll_dev, float* grad_params_dev, double* grad_bg_dev,
                      double* grad_zern_dev, int32_t* err_dev)
{
   if (!model || !nll_dev || !err_dev || (n_emitters && (!params_dev || !frame_dev || !counts_dev)) ||
       (n_frames && !bg_dev) || (model->J && !zern))
      return Fail(ISCU_ERR_ARG, "null argument");
   const bool grad = grad_params_dev != nullptr;
   if (grad && ((n_frames && !grad_bg_dev) || (model->J && !grad_zern_dev)))
      return Fail(ISCU_ERR_ARG, "the gradient needs every gradient output");
   iscu_ctx* ctx = model->ctx;
   std::lock_guard<std::recursive_mutex> lock(ctx->mu);
   ClearError();
   PrepareArgs pa = {};
   pa.basis = model->basis.as<double>();
   pa.J = model->J;
   pa.MM = model->M * model->M;
   if (model->J)
   {
      cudaPointerAttributes where = {};
      if (cudaPointerGetAttributes(&where, zern) != cudaSuccess)
         cudaGetLastError();   // not a pointer that CUDA knows: the host's
      if (where.type == cudaMemoryTypeDevice)
      {
         if (where.device != ctx->device)   // (refused by the copy that this was)
            return Fail(ISCU_ERR_ARG, "the Zernike coefficients are on another device");
         pa.zernDev = zern;
      }
      else
         std::copy(zern, zern + model->J, pa.zern);
   }
   pa.zphase = model->zphase.as<double>();
   pa.nll = nll_dev;
   pa.err = err_dev;
   pa.nFrames = n_frames;
   pa.gBg = grad ? grad_bg_dev : nullptr;
   pa.gZern = grad ? grad_zern_dev : nullptr;
   const uint32_t cover = std::max(static_cast<uint32_t>(pa.MM), grad ? n_frames : 0u);
   NllPrepareKernel<<<(cover + 255) / 256, 256, 0, ctx->stream>>>(pa);
   ISCU_CK_LAUNCH(ctx, "NllPrepareKernel");
   if (n_emitters == 0)
      return ISCU_OK;
   NllArgs a;
   a.samples = model->samples.as<double4>();
   a.basis = model->basis.as<double>();
   a.cs = model->cs.as<float>();
   a.zphase = model->zphase.as<double>();
   a.J = model->J;
   a.R = model->spec.roi;
   a.kappa = model->kappa;
   a.n = n_emitters;
   a.params = reinterpret_cast<const float4*>(params_dev);
   a.frame = frame_dev;
   a.nFrames = n_frames;
   a.bg = bg_dev;
   a.counts = counts_dev;
   a.mu = mu_dev;
   a.nll = nll_dev;
   a.gParams = reinterpret_cast<float4*>(grad_params_dev);
   a.gBg = grad_bg_dev;
   a.gZern = grad_zern_dev;
   a.err = err_dev;
   const size_t smem = sizeof(NllSmem);
   int perSm = 0;
   const NllFn fn = grad ? NllOf<true>(model->spec.os) : NllOf<false>(model->spec.os);
   ISCU_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, kThreads, smem));
   const uint32_t grid = std::min<uint32_t>(n_emitters, static_cast<uint32_t>(std::max(1, perSm) * ctx->smCount));
   fn<<<grid, kThreads, smem, ctx->stream>>>(a);
   ISCU_CK_LAUNCH(ctx, "NllKernel");
   return ISCU_OK;
}

} // extern "C"

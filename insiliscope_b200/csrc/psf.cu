// PSF stacks and libraries on sm_100a: the Gibson-Lanni + Zernike (+ double-helix) pupil and its chirp-Z image
// (ComputeZernikePsfPlanes, adapter/inSiliScope/Simulation/ZernikePsf.cpp:160-337).
//
// The reference evaluates out[p] = sum_m in[m] exp(i (kMin + m dk)(x0 + p dx)) per pupil line by Bluestein's
// chirp-Z in float64 (ChirpZ.h:28-142), rows then columns. Here the two passes are the dense products
// E = A U A^T with A[p][m] = exp(i (kMin + m dk)(x0 + p dx)) -- the DFT matrix the CZT factorizes -- so they run as
// matrix multiplications. Float64 is kept where the phases are large: the pupil's OPD phase
// k0 (opd1 + ni (ti - ti0) opd3) + zernike + mask, and the DFT exponent, are formed and reduced mod 2 pi in float64,
// then the unit phasors are rounded to float32.
//
// Kernels:
//  PupilTablesKernel  z-independent pupil tables per request set (aperture, opd1, the opd3 obliquity factor,
//                     Zernike + mask phase), float64 (ZernikePsf.cpp:188-231); the folded transform's cosines and sines
//  DftMatrixKernel    A (P x M) and A^T (M x P) per set, float32 phasors of float64 phases
//  CztFoldKernel      the plain FP32 form: a cluster of CTAs per PSF, both products folded about the plane's centre,
//                     |E|^2, optional sum-1 normalization
//  PupilKernel, CGemmTiledKernel  pupils beyond shared memory: the products through global memory
// The tensor-core form (TF32 split products on tcgen05) is in psf_tc.cu.

#include "iscu_internal.h"
#include "psf_common.cuh"

#include <algorithm>
#include <cooperative_groups.h>
#include <cmath>
#include <cstring>
#include <vector>

namespace iscu {

namespace {

constexpr double kPi = 3.14159265358979323846;

// ------------------------------------------------------------------------------------------ Zernike (device, FP64)
__device__ double LaguerreL(int p, int a, double x)
{
   double lm1 = 0.0, l = 1.0;
   for (int k = 0; k < p; ++k)
   {
      const double next = ((2 * k + 1 + a - x) * l - (k + a) * lm1) / (k + 1);
      lm1 = l;
      l = next;
   }
   return l;
}

// MaskPhase (ZernikePsf.cpp:93-110): the double-helix Gauss-Laguerre superposition's phase.
__device__ double MaskPhase(int maskModes, double maskWaist, double rhoNorm, double phi)
{
   const int n = maskModes > 2 ? maskModes : 2;
   const double w = maskWaist > 0.2 ? maskWaist : 0.2;
   const double u = fmax(0.0, fmin(1.0, rhoNorm)) / w;
   const double u2 = u * u;
   double re = 0.0, im = 0.0;
   for (int p = 0; p < n; ++p)
   {
      const int l = 2 * p + 1;
      const double amp = pow(u, static_cast<double>(l)) * exp(-u2) * LaguerreL(p, l, 2.0 * u2);
      re += amp * cos(l * phi);
      im += amp * sin(l * phi);
   }
   return (re == 0.0 && im == 0.0) ? 0.0 : atan2(im, re);
}

// The folded transform. The pupil's samples k_q = q dk (q = m - M / 2) and the plane's tau dx lie symmetrically about
// 0, so exp(i k_q x_tau) for +-q and +-tau is one cosine and one sine: with P = U[q] + U[-q], N = U[q] - U[-q],
//   C = U[0] + sum cos(q tau) P,  S = sum sin(q tau) N,  the samples at +-tau are C +- i S,
// on each axis: real by complex products of a quarter of the size. The aperture's radius is (M - 4) / 2 samples (dk =
// 2 kMax / (M - 4)), so q <= Q = (M - 4) / 2. tau = t for an odd plane size (t = 0 is one sample, not two), t + 1/2 for
// an even one.
struct Fold
{
   int Q, R, nT;   // the largest q; folded rows (P of q = 0..Q, then N of q = 1..Q); sample pairs
   __host__ __device__ Fold(int M, int P) : Q((M - 4) / 2), R(2 * Q + 1), nT((P + 1) / 2) {}
   __host__ __device__ int Pitch() const { return (nT + 3) / 4 * 4; }        // of the table's rows
   __host__ __device__ int Share(int c) const { return (nT + c - 1) / c; }   // pairs of a CTA of a cluster of c
   size_t Bytes(int c) const
   {
      return sizeof(float4) * (static_cast<size_t>(Q + 1) * R + static_cast<size_t>(R) * (Share(c) | 1));
   }
};

// Entry idx of set s of the folded transform's table: cs[s][q - 1][t] = cos, sin of q dk tau dx, the float64 phase
// reduced mod 2 pi first; zeros beyond the pairs.
__device__ void FoldTable(const SetParams& sp, int M, int P, int idx, int s, float2* __restrict__ cs)
{
   const Fold F(M, P);
   const int pitch = F.Pitch();
   if (idx >= F.Q * pitch)
      return;
   const int q = idx / pitch + 1, t = idx % pitch;
   float2 v = make_float2(0.f, 0.f);
   if (t < F.nT)
   {
      double sn, c;
      sincos(ReduceTwoPi((q * sp.dk) * ((P & 1 ? t : t + 0.5) * sp.dx)), &sn, &c);
      v = make_float2(static_cast<float>(c), static_cast<float>(sn));
   }
   cs[static_cast<size_t>(s) * F.Q * pitch + idx] = v;
}

// ------------------------------------------------------------------------------------------ tables
// tables[s][idx] = (opd1, opd3Factor, zernike + mask phase); opd3Factor < 0 marks a sample outside the aperture.
// cs (nullable): the folded transform's table too, by the blocks beyond the pupil's.
constexpr int kTableThreads = 128;
__global__ void __launch_bounds__(kTableThreads) PupilTablesKernel(const SetParams* __restrict__ sets, int M, int P,
                                                                   double3* __restrict__ tables,
                                                                   float2* __restrict__ cs)
{
   const int s = blockIdx.y;
   // the set's scalars in shared memory: the modes' loop reads them one after the other
   __shared__ SetParams sp;
   static_assert(sizeof(SetParams) % 8 == 0, "copied by 8 bytes");
   for (int i = threadIdx.x; i < static_cast<int>(sizeof(SetParams) / 8); i += kTableThreads)
      reinterpret_cast<uint64_t*>(&sp)[i] = reinterpret_cast<const uint64_t*>(sets + s)[i];
   __syncthreads();
   const int pupilBlocks = (M * M + kTableThreads - 1) / kTableThreads;
   if (static_cast<int>(blockIdx.x) >= pupilBlocks)
   {
      FoldTable(sp, M, P, (blockIdx.x - pupilBlocks) * kTableThreads + threadIdx.x, s, cs);
      return;
   }
   const int idx = blockIdx.x * kTableThreads + threadIdx.x;
   if (idx >= M * M)
      return;
   const int iy = idx / M, ix = idx % M, c0 = M / 2;
   const double ky = (iy - c0) * sp.dk, kx = (ix - c0) * sp.dk;
   // The aperture test decides samples that sit exactly on the circle (M = 64: (30, 0), (18, 24), ...): rounded
   // product by product, as the reference's uncontracted float64 does, so the same samples are in.
   const double kr2 = __dadd_rn(__dmul_rn(kx, kx), __dmul_rn(ky, ky));
   double3 out = make_double3(0.0, -1.0, 0.0);
   if (!(kr2 > __dmul_rn(sp.kMax, sp.kMax)))
   {
      const double kr = sqrt(kr2);
      const double rho = kr / (sp.k0 * sp.na);
      const double s1 = sp.na * rho / sp.ns;
      const double s3 = sp.na * rho / sp.ni;
      out.x = sp.ns * sp.depthM * sqrt(fmax(0.0, 1.0 - s1 * s1));
      out.y = sqrt(fmax(0.0, 1.0 - s3 * s3));
      // ZernikeValue (ZernikePsf.cpp:74-78): R_n^m(rho) cos m phi (l >= 0) or sin m phi, the radial part by Horner in
      // rho^2, the angular one from the powers of (kx + i ky) / kr (phi = 0 at the centre); no pow, atan2 or cos, whose
      // chains made this kernel 20 us at 64 x 64 samples and 12 modes
      double zern = 0.0;
      const double rn = rho / sp.bMax, rn2 = rn * rn;
      const double cphi = kr > 0.0 ? kx / kr : 1.0, sphi = kr > 0.0 ? ky / kr : 0.0;
      for (int t = 0; t < sp.nModes; ++t)
      {
         const int n = sp.modeN[t], m = sp.modeM[t];
         double rad = sp.radial[t][0];
         for (int k = 1; k <= (n - m) / 2; ++k)
            rad = rad * rn2 + sp.radial[t][k];
         double re = 1.0, im = 0.0;
         for (int k = 0; k < m; ++k)
         {
            const double r = re * cphi - im * sphi;
            im = re * sphi + im * cphi;
            re = r;
            rad *= rn;
         }
         zern += rn <= 1.0 ? sp.coeff[t] * rad * (sp.modeL[t] >= 0 ? re : im) : 0.0;
      }
      zern *= 2.0 * kPi;
      const double mask =
         sp.doubleHelix ? MaskPhase(sp.maskModes, sp.maskWaist, rho / sp.bMax, atan2(ky, kx)) : 0.0;
      out.z = zern + mask;
   }
   tables[static_cast<size_t>(s) * M * M + idx] = out;
}

// ------------------------------------------------------------------------------------------ DFT matrices
// A[s][p][m] = exp(i (kMin + m dk)(x0 + p dx)); At[s][m][p] the same value. float64 phase reduced mod 2 pi first.
__global__ void DftMatrixKernel(const SetParams* __restrict__ sets, int M, int P, float2* __restrict__ A,
                                float2* __restrict__ At)
{
   const int s = blockIdx.y;
   const int idx = blockIdx.x * blockDim.x + threadIdx.x;
   if (idx >= P * M)
      return;
   const SetParams& sp = sets[s];
   const int p = idx / M, m = idx % M;
   const double ph = ReduceTwoPi((sp.kMin + m * sp.dk) * (sp.x0 + p * sp.dx));
   double sn, cs;
   sincos(ph, &sn, &cs);
   const float2 v = make_float2(static_cast<float>(cs), static_cast<float>(sn));
   A[static_cast<size_t>(s) * P * M + idx] = v;
   At[static_cast<size_t>(s) * P * M + static_cast<size_t>(m) * P + p] = v;
}

// ------------------------------------------------------------------------------------------ plain FP32 chirp-Z
__device__ __forceinline__ void Cmac(float2& acc, float2 a, float2 b)
{
   acc.x = fmaf(a.x, b.x, acc.x);
   acc.x = fmaf(-a.y, b.y, acc.x);
   acc.y = fmaf(a.x, b.y, acc.y);
   acc.y = fmaf(a.y, b.x, acc.y);
}

// A sum in two doubles (hi + lo, lo what hi's roundings left): the same to 2^-100 in any order, so that a plane's
// normalization does not depend on how many CTAs shared the plane, which the call's number of planes decides.
struct WideSum
{
   double hi = 0.0, lo = 0.0;
   __device__ __forceinline__ void Add(double v)
   {
      const double s = hi + v, b = s - hi;
      lo += (hi - (s - b)) + (v - b);
      hi = s;
   }
   __device__ __forceinline__ void Add(const WideSum& o)
   {
      Add(o.hi);
      lo += o.lo;
   }
   __device__ __forceinline__ double Value() const { return hi + lo; }
};

// The sum over the CTA's threads (thread 0's). red: blockDim.x / 32 entries.
__device__ __forceinline__ WideSum BlockWideSum(WideSum v, double2* red)
{
#pragma unroll
   for (int o = 16; o > 0; o >>= 1)
   {
      WideSum u;
      u.hi = __shfl_down_sync(0xffffffffu, v.hi, o);
      u.lo = __shfl_down_sync(0xffffffffu, v.lo, o);
      v.Add(u);
   }
   if ((threadIdx.x & 31) == 0)
      red[threadIdx.x >> 5] = make_double2(v.hi, v.lo);
   __syncthreads();
   WideSum t;
   if (threadIdx.x == 0)
      for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w)
      {
         WideSum u;
         u.hi = red[w].x;
         u.lo = red[w].y;
         t.Add(u);
      }
   return t;
}

constexpr size_t kPsfScratchKept = 64u << 20;
constexpr int kFoldThreads = 320, kFoldMaxCluster = 8;
constexpr size_t kFoldMaxBytes = 224 * 1024;

// A cluster of C CTAs per PSF (grid: nPsf x C): each takes nT / C of the plane's column pairs through both products,
// which need nothing of the others' columns, and 1/C of the pupil's phasors, written to every CTA of the cluster; the
// plane's sum is exchanged at the end.
//
// What bounds it: at a stack's 49 planes, latency -- a CTA per plane left two thirds of the SMs idle through 36 x the
// arithmetic a plane needs (64-wide blocks over 129 columns; 4.3 x more multiply-adds than the folded products). 49
// planes of 129 x 129 from 64 pupil samples: 26 us (four CTAs a plane) against 218 us the unfolded CTA per plane; the
// call with its tables 51 us against 262, or 950 where cudaMalloc and cudaFree are slow.
__global__ void __launch_bounds__(kFoldThreads, 2) CztFoldKernel(const SetParams* __restrict__ sets,
                                                                 const double3* __restrict__ tables,
                                                                 const float2* __restrict__ cs,
                                                                 const PsfItem* __restrict__ items, int M, int P,
                                                                 int normalize, int split, double2* __restrict__ sums,
                                                                 float* __restrict__ out)
{
   namespace cg = cooperative_groups;
   cg::cluster_group cluster = cg::this_cluster();
   const int C = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
   const int psf = blockIdx.x / (C * split), part = blockIdx.x / C % split, tid = threadIdx.x;
   const Fold F(M, P);
   const int Q = F.Q, R = F.R, nT = F.nT, pitch = F.Pitch(), share = F.Share(C * split), tp = share | 1;
   extern __shared__ __align__(16) unsigned char smem[];
   float4* U = reinterpret_cast<float4*>(smem);         // [q][row]: (P.re, P.im, N.re, N.im) of the column pair q
   float4* T = U + static_cast<size_t>(Q + 1) * R;      // [row][own pair]: the samples at +t and -t
   __shared__ double2 sRed[kFoldThreads / 32], sPart[kFoldMaxCluster];
   const PsfItem it = items[psf];
   const SetParams& sp = sets[it.set];
   const double3* tab = tables + static_cast<size_t>(it.set) * M * M;
   const float2* ct = cs + static_cast<size_t>(it.set) * Q * pitch;
   const int t0 = (part * C + rank) * share, own = max(0, min(share, nT - t0));
   cluster.sync();   // every CTA's shared memory is there to be written
   // the pupil (phase = k0 (opd1 + ni (ti - ti0) opd3F) + zernike + mask, ZernikePsf.cpp:240-248, float64 then reduced),
   // folded on both axes
   for (int i = rank * kFoldThreads + tid; i < (Q + 1) * (Q + 1); i += C * kFoldThreads)
   {
      const int qy = i / (Q + 1), qx = i % (Q + 1), m0 = M / 2 * M + M / 2;
      float2 u[2][2];
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
         for (int x = 0; x < 2; ++x)
         {
            u[y][x] = PupilPhasor(tab[m0 + (y ? -qy : qy) * M + (x ? -qx : qx)], sp, it.dtiM);
            if ((y && qy == 0) || (x && qx == 0))   // one sample on an axis, not two
               u[y][x] = make_float2(0.f, 0.f);
         }
      const float2 p0 = make_float2(u[0][0].x + u[0][1].x, u[0][0].y + u[0][1].y);
      const float2 n0 = make_float2(u[0][0].x - u[0][1].x, u[0][0].y - u[0][1].y);
      const float2 p1 = make_float2(u[1][0].x + u[1][1].x, u[1][0].y + u[1][1].y);
      const float2 n1 = make_float2(u[1][0].x - u[1][1].x, u[1][0].y - u[1][1].y);
      const float4 even = make_float4(p0.x + p1.x, p0.y + p1.y, n0.x + n1.x, n0.y + n1.y);
      const float4 odd = make_float4(p0.x - p1.x, p0.y - p1.y, n0.x - n1.x, n0.y - n1.y);
      for (int c = 0; c < C; ++c)
      {
         float4* to = cluster.map_shared_rank(U, c) + static_cast<size_t>(qx) * R;
         to[qy] = even;
         if (qy)
            to[Q + qy] = odd;
      }
   }
   cluster.sync();
   // T = U A^T over the folded rows: a row and four of the CTA's pairs per thread
   for (int i = tid; i < R * ((own + 3) / 4); i += kFoldThreads)
   {
      const int r = i % R, g = i / R * 4;
      float cr[4], ci[4], sr[4], si[4];
      const float4 u0 = U[r];
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
         cr[k] = u0.x;
         ci[k] = u0.y;
         sr[k] = si[k] = 0.f;
      }
      const float2* c0 = ct + t0 + g;
      int at[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
         at[k] = min(k, own - 1 - g);
#pragma unroll 4
      for (int q = 1; q <= Q; ++q, c0 += pitch)
      {
         const float4 u = U[q * R + r];
#pragma unroll
         for (int k = 0; k < 4; ++k)
         {
            const float2 c = __ldg(c0 + at[k]);
            cr[k] = fmaf(c.x, u.x, cr[k]);
            ci[k] = fmaf(c.x, u.y, ci[k]);
            sr[k] = fmaf(c.y, u.z, sr[k]);
            si[k] = fmaf(c.y, u.w, si[k]);
         }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
         if (g + k < own)
            T[r * tp + g + k] = make_float4(cr[k] - si[k], ci[k] + sr[k], cr[k] + si[k], ci[k] - sr[k]);
   }
   __syncthreads();
   // E = A T, I = |E|^2: a column pair and four row pairs per thread
   float* plane = out + static_cast<size_t>(psf) * P * P;
   const int groups = (nT + 3) / 4, half = P / 2, odd = P & 1;
   WideSum local;
   float I[4][4];   // [row pair][+y +x, +y -x, -y +x, -y -x] of the thread's last item
   const int nItems = own * groups;
   // row y = half + t (+), half - t - 1 + odd (-); columns likewise
   auto store = [&](int i) {
      const int c = t0 + i % own, g = i / own * 4;
      const int xp = half + c, xm = half - c - 1 + odd;
#pragma unroll
      for (int k = 0; k < 4; ++k)
         if (g + k < nT)
         {
            float* yp = plane + static_cast<size_t>(half + g + k) * P;
            float* ym = plane + static_cast<size_t>(half - g - k - 1 + odd) * P;
            yp[xp] = I[k][0];
            yp[xm] = I[k][1];
            ym[xp] = I[k][2];
            ym[xm] = I[k][3];
         }
   };
   for (int i = tid; i < nItems; i += kFoldThreads)
   {
      const int c = i % own, g = i / own * 4;
      float cr[2][4], ci[2][4], sr[2][4], si[2][4];
      const float4 e0 = T[c];
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
         cr[0][k] = e0.x;
         ci[0][k] = e0.y;
         cr[1][k] = e0.z;
         ci[1][k] = e0.w;
         sr[0][k] = si[0][k] = sr[1][k] = si[1][k] = 0.f;
      }
      const float4* c4 = reinterpret_cast<const float4*>(ct + g);
#pragma unroll 2
      for (int q = 1; q <= Q; ++q, c4 += pitch / 2)
      {
         const float4 p = T[q * tp + c], n = T[(Q + q) * tp + c];
         const float4 a = __ldg(c4), b = __ldg(c4 + 1);
         const float co[4] = {a.x, a.z, b.x, b.z}, sn[4] = {a.y, a.w, b.y, b.w};
#pragma unroll
         for (int k = 0; k < 4; ++k)
         {
            cr[0][k] = fmaf(co[k], p.x, cr[0][k]);
            ci[0][k] = fmaf(co[k], p.y, ci[0][k]);
            cr[1][k] = fmaf(co[k], p.z, cr[1][k]);
            ci[1][k] = fmaf(co[k], p.w, ci[1][k]);
            sr[0][k] = fmaf(sn[k], n.x, sr[0][k]);
            si[0][k] = fmaf(sn[k], n.y, si[0][k]);
            sr[1][k] = fmaf(sn[k], n.z, sr[1][k]);
            si[1][k] = fmaf(sn[k], n.w, si[1][k]);
         }
      }
      const bool centreX = odd && t0 + c == 0;
      double item = 0.0;   // (an item's samples are the same however the plane is shared)
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
         const bool centreY = odd && g + k == 0;
#pragma unroll
         for (int x = 0; x < 2; ++x)
         {
            const float pr = cr[x][k] - si[x][k], pi = ci[x][k] + sr[x][k];
            const float mr = cr[x][k] + si[x][k], mi = ci[x][k] - sr[x][k];
            I[k][x] = pr * pr + pi * pi;
            I[k][2 + x] = mr * mr + mi * mi;
            if (g + k < nT && !(x && centreX))
               item += static_cast<double>(I[k][x]) + (centreY ? 0.0 : static_cast<double>(I[k][2 + x]));
         }
      }
      local.Add(item);
      if (!normalize || split > 1 || i + kFoldThreads < nItems)
         store(i);   // the last item stays in registers for its normalization
   }
   if (!normalize)
      return;
   const WideSum mine = BlockWideSum(local, sRed);
   if (split > 1)
   {
      // several clusters' plane: NormalizeFoldKernel goes on
      if (tid == 0)
         sums[blockIdx.x] = make_double2(mine.hi, mine.lo);
      return;
   }
   if (tid == 0)
      for (int c = 0; c < C; ++c)
         cluster.map_shared_rank(sPart, c)[rank] = make_double2(mine.hi, mine.lo);
   cluster.sync();
   WideSum all;
   for (int c = 0; c < C; ++c)
   {
      WideSum u;
      u.hi = sPart[c].x;
      u.lo = sPart[c].y;
      all.Add(u);
   }
   const double sum = all.Value(), inv = sum > 0.0 ? 1.0 / sum : 1.0;
   for (int i = tid; i < nItems; i += kFoldThreads)
   {
      if (i + kFoldThreads < nItems)
      {
         // an earlier item, back from memory (its own thread's writes)
         const int c = t0 + i % own, g = i / own * 4;
         const int xp = half + c, xm = half - c - 1 + odd;
#pragma unroll
         for (int k = 0; k < 4; ++k)
            if (g + k < nT)
            {
               float* yp = plane + static_cast<size_t>(half + g + k) * P;
               float* ym = plane + static_cast<size_t>(half - g - k - 1 + odd) * P;
               const float v[4] = {yp[xp], yp[xm], ym[xp], ym[xm]};
               yp[xp] = static_cast<float>(v[0] * inv);
               yp[xm] = static_cast<float>(v[1] * inv);
               ym[xp] = static_cast<float>(v[2] * inv);
               ym[xm] = static_cast<float>(v[3] * inv);
            }
         continue;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
         for (int j = 0; j < 4; ++j)
            I[k][j] = static_cast<float>(I[k][j] * inv);
      store(i);
   }
}

// The planes that several clusters shared, by the `parts` sums that their CTAs left. grid (any, nPsf).
__global__ void __launch_bounds__(256) NormalizeFoldKernel(float* __restrict__ planes, const double2* __restrict__ sums,
                                                           int parts, int planeElems)
{
   WideSum all;
   for (int c = 0; c < parts; ++c)
   {
      const double2 v = sums[blockIdx.y * parts + c];
      WideSum u;
      u.hi = v.x;
      u.lo = v.y;
      all.Add(u);
   }
   const double sum = all.Value(), inv = sum > 0.0 ? 1.0 / sum : 1.0;
   float* p = planes + static_cast<size_t>(blockIdx.y) * planeElems;
   for (int i = blockIdx.x * 256 + threadIdx.x; i < planeElems; i += gridDim.x * 256)
      p[i] = static_cast<float>(p[i] * inv);
}

// ------------------------------------------------------------------------------------------ large pupils
// When the folded pupil and row pass do not fit a cluster's shared memory (M beyond ~165: a widefield kernel's 512
// samples), the same products go through global memory: the pupil phasors U (nPsf x M x M), then two batched complex
// GEMMs with 64 x 64 output tiles staged 16 deep in shared memory -- T = A U, E = T A^T -- the second one ending in
// |E|^2 and the plane's float64 sum.
__global__ void PupilKernel(const SetParams* __restrict__ sets, const double3* __restrict__ tables,
                            const PsfItem* __restrict__ items, int M, float2* __restrict__ U)
{
   const int b = blockIdx.y;
   const int idx = blockIdx.x * blockDim.x + threadIdx.x;
   if (idx >= M * M)
      return;
   const PsfItem it = items[b];
   U[static_cast<size_t>(b) * M * M + idx] =
      PupilPhasor(tables[static_cast<size_t>(it.set) * M * M + idx], sets[it.set], it.dtiM);
}

// C[b] (rows x cols) = L (rows x K) R (K x cols), L = L0 + set * lSet + b * lBatch, R likewise. kIntensity: writes
// |C|^2 as float and adds the tile's float64 sum to sums[b].
template <bool kIntensity>
__global__ void __launch_bounds__(256) CGemmTiledKernel(const PsfItem* __restrict__ items, const float2* __restrict__ L0,
                                                       size_t lSet, size_t lBatch, const float2* __restrict__ R0,
                                                       size_t rSet, size_t rBatch, int rows, int cols, int K,
                                                       float2* __restrict__ C, float* __restrict__ I,
                                                       double* __restrict__ sums)
{
   __shared__ float2 sL[16][65];
   __shared__ float2 sR[16][64];
   __shared__ double sRed[8];
   const int b = blockIdx.z, set = items[b].set;
   const float2* L = L0 + set * lSet + b * lBatch;
   const float2* R = R0 + set * rSet + b * rBatch;
   const int rb = blockIdx.y * 64, cb = blockIdx.x * 64;
   const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
   float2 acc[4][4];
#pragma unroll
   for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
         acc[i][j] = make_float2(0.f, 0.f);
   for (int k0 = 0; k0 < K; k0 += 16)
   {
#pragma unroll
      for (int e4 = 0; e4 < 4; ++e4)
      {
         const int e = threadIdx.x + 256 * e4;
         const int r = e >> 4, kk = e & 15, kr = e >> 6, c = e & 63;
         sL[kk][r] = (rb + r < rows && k0 + kk < K) ? L[static_cast<size_t>(rb + r) * K + k0 + kk]
                                                    : make_float2(0.f, 0.f);
         sR[kr][c] = (k0 + kr < K && cb + c < cols) ? R[static_cast<size_t>(k0 + kr) * cols + cb + c]
                                                    : make_float2(0.f, 0.f);
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < 16; ++kk)
      {
         float2 l[4], r[4];
#pragma unroll
         for (int i = 0; i < 4; ++i)
         {
            l[i] = sL[kk][ty + 16 * i];
            r[i] = sR[kk][tx + 16 * i];
         }
#pragma unroll
         for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
               Cmac(acc[i][j], l[i], r[j]);
      }
      __syncthreads();
   }
   double local = 0.0;
#pragma unroll
   for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
         const int r = rb + ty + 16 * i, c = cb + tx + 16 * j;
         if (r >= rows || c >= cols)
            continue;
         const size_t o = static_cast<size_t>(b) * rows * cols + static_cast<size_t>(r) * cols + c;
         if (kIntensity)
         {
            const float v = acc[i][j].x * acc[i][j].x + acc[i][j].y * acc[i][j].y;
            I[o] = v;
            local += static_cast<double>(v);
         }
         else
            C[o] = acc[i][j];
      }
   if (kIntensity)
   {
      const double t = BlockSumDouble(local, sRed);
      if (threadIdx.x == 0)
         atomicAdd(sums + b, t);
   }
}

__global__ void NormalizeKernel(float* __restrict__ planes, const double* __restrict__ sums, int planeElems)
{
   const int b = blockIdx.y;
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= planeElems)
      return;
   const double s = sums[b];
   if (s > 0.0)
   {
      float* p = planes + static_cast<size_t>(b) * planeElems;
      p[i] = static_cast<float>(static_cast<double>(p[i]) / s);
   }
}

} // namespace

// The cluster of the folded kernel: a CTA for every SM where the PSFs are few (a stack), eight column pairs a CTA at
// least, and as many as its shared memory needs.
static int FoldCluster(const Fold& F, uint32_t nPsf, int smCount)
{
   int c = 1;
   while (c < kFoldMaxCluster && (F.Bytes(c) > kFoldMaxBytes ||
                                  (static_cast<uint64_t>(nPsf) * c < static_cast<uint64_t>(smCount) && F.nT >= 8 * c)))
      c *= 2;
   return c;
}

// Clusters of kFoldMaxCluster CTAs that share a plane: as many as leave each CTA eight column pairs and take no more than
// three quarters of the SMs (16 clusters of CTAs that fill an SM do not all find eight SMs in one GPC at once: eight
// planes of 513 x 513 from 128 pupil samples 151 us on a cluster each, 174 on two). One plane of 1,001 x 1,001 from 64
// samples, a plan's call: 211 us on one cluster, 75 on seven (90 through global memory, which small plans took).
static int FoldSplit(const Fold& F, int cluster, uint32_t nPsf, int smCount)
{
   if (cluster < kFoldMaxCluster)
      return 1;
   const uint64_t ctas = static_cast<uint64_t>(nPsf) * kFoldMaxCluster;
   return static_cast<int>(std::max<uint64_t>(
      1, std::min<uint64_t>(static_cast<uint64_t>(smCount) * 3 / 4 / ctas,
                            static_cast<uint64_t>(F.nT / (8 * kFoldMaxCluster)))));
}

bool FoldFits(int M, int P) { return Fold(M, P).Bytes(kFoldMaxCluster) <= kFoldMaxBytes; }

// The folded FP32 chirp-Z over its tables (cs).
static int LaunchCztFold(iscu_ctx* ctx, const SetParams* dSets, const double3* dTab, const float2* cs,
                         const PsfItem* dItems, uint32_t nPsf, int M, int P, int normalize, double2* sums, float* out)
{
   const Fold F(M, P);
   const int c = FoldCluster(F, nPsf, ctx->smCount), split = FoldSplit(F, c, nPsf, ctx->smCount);
   ISCU_CK(cudaFuncSetAttribute(CztFoldKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(kFoldMaxBytes)));
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3(nPsf * static_cast<uint32_t>(c * split));
   cfg.blockDim = dim3(kFoldThreads);
   cfg.dynamicSmemBytes = F.Bytes(c * split);
   cfg.stream = ctx->stream;
   cudaLaunchAttribute attr = {};
   attr.id = cudaLaunchAttributeClusterDimension;
   attr.val.clusterDim.x = static_cast<unsigned>(c);
   attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
   cfg.attrs = &attr;
   cfg.numAttrs = 1;
   ISCU_CK(cudaLaunchKernelEx(&cfg, CztFoldKernel, dSets, dTab, cs, dItems, M, P, normalize, split, sums, out));
   ISCU_CK_LAUNCH(ctx, "CztFoldKernel");
   if (split > 1 && normalize)
   {
      NormalizeFoldKernel<<<dim3(std::max<uint32_t>(1, 2 * static_cast<uint32_t>(ctx->smCount) / nPsf), nPsf), 256, 0,
                            ctx->stream>>>(out, sums, c * split, P * P);
      ISCU_CK_LAUNCH(ctx, "NormalizeFoldKernel");
   }
   return ISCU_OK;
}

// The large-pupil FP32 path (global-memory products); temporaries allocated here.
static int LaunchCztGlobalFp32(iscu_ctx* ctx, const SetParams* dSets, const double3* dTab, const float2* dA,
                               const float2* dAt, const PsfItem* dItems, uint32_t nPsf, int M, int P, int normalize,
                               float* out)
{
   DevBuf U, T, S;
   // in batches bounded to ~2 GB of temporaries
   const size_t perPsf = (static_cast<size_t>(M) * M + static_cast<size_t>(P) * M) * sizeof(float2);
   const uint32_t batch = static_cast<uint32_t>(std::max<size_t>(1, std::min<size_t>(nPsf, (2ull << 30) / perPsf)));
   ISCU_CK(U.Reserve(static_cast<size_t>(batch) * M * M * sizeof(float2)));
   ISCU_CK(T.Reserve(static_cast<size_t>(batch) * P * M * sizeof(float2)));
   ISCU_CK(S.Reserve(static_cast<size_t>(nPsf) * sizeof(double)));
   ISCU_CK(cudaMemsetAsync(S.p, 0, static_cast<size_t>(nPsf) * sizeof(double), ctx->stream));
   for (uint32_t b0 = 0; b0 < nPsf; b0 += batch)
   {
      const uint32_t nb = std::min(batch, nPsf - b0);
      PupilKernel<<<dim3((M * M + 255) / 256, nb), 256, 0, ctx->stream>>>(dSets, dTab, dItems + b0, M,
                                                                          U.as<float2>());
      ISCU_CK_LAUNCH(ctx, "PupilKernel");
      CGemmTiledKernel<false><<<dim3((M + 63) / 64, (P + 63) / 64, nb), 256, 0, ctx->stream>>>(
         dItems + b0, dA, static_cast<size_t>(P) * M, 0, U.as<float2>(), 0, static_cast<size_t>(M) * M, P, M, M,
         T.as<float2>(), nullptr, nullptr);
      ISCU_CK_LAUNCH(ctx, "CGemmTiledKernel<product>");
      CGemmTiledKernel<true><<<dim3((P + 63) / 64, (P + 63) / 64, nb), 256, 0, ctx->stream>>>(
         dItems + b0, T.as<float2>(), 0, static_cast<size_t>(P) * M, dAt, static_cast<size_t>(P) * M, 0, P, P, M,
         nullptr, out + static_cast<size_t>(b0) * P * P, S.as<double>() + b0);
      ISCU_CK_LAUNCH(ctx, "CGemmTiledKernel<intensity>");
   }
   if (normalize)
   {
      NormalizeKernel<<<dim3((P * P + 255) / 256, nPsf), 256, 0, ctx->stream>>>(out, S.as<double>(), P * P);
      ISCU_CK_LAUNCH(ctx, "NormalizeKernel");
   }
   ISCU_CK(cudaStreamSynchronize(ctx->stream));
   return ISCU_OK;
}

// ------------------------------------------------------------------------------------------ host side

// GeometryFor + ZernikePupilSamples (ZernikePsf.cpp:118-158).
bool GeometryFor(const iscu_psf_request& r, PsfGeometry& g, std::string& err)
{
   if (!(r.na > 0.0) || !(r.wavelength_nm > 0.0) || !(r.immersion_index > 0.0) || !(r.sample_index > 0.0) ||
       !(r.pixel_size_nm > 0.0) || !(r.z_step_nm > 0.0))
   {
      err = "GibsonLanniZernike PSF: NA, wavelength, refractive indices, pixel size and z step must be > 0.";
      return false;
   }
   g.os = std::max(1, r.oversampling);
   const int camHalf = std::max(1, r.kernel_half_width_px);
   g.halfOv = camHalf * g.os;
   g.size = 2 * g.halfOv + 1;
   const int nzWanted = std::max(3, r.nz);
   g.nz = (nzWanted % 2 == 1) ? nzWanted : nzWanted + 1;
   g.resLateralNm = r.pixel_size_nm / g.os;
   if (r.pupil_samples > 0)
      g.M = std::max(8, std::min(1024, static_cast<int>(r.pupil_samples)));
   else
   {
      const double diagonalUm = 2.0 * std::sqrt(2.0) * camHalf * r.pixel_size_nm / 1000.0;
      const double m = 4.0 + 2.0 * r.na * diagonalUm / (r.wavelength_nm / 1000.0);
      const int need = std::max(64, std::min(512, 4 * static_cast<int>(std::ceil(m / 4.0))));
      int fftLen = 1;
      while (fftLen < need + g.size - 1)
         fftLen <<= 1;
      g.M = std::max(need, std::min(512, (fftLen - g.size + 1) / 4 * 4));
   }
   return true;
}

static double Binomial(int a, int b)
{
   if (b < 0 || b > a)
      return 0.0;
   double r = 1.0;
   for (int i = 0; i < b; ++i)
      r = r * (a - i) / (i + 1);
   return r;
}

// The set parameters of a request for planes of `size` samples (ZernikePsf.cpp:166-223's scalars).
static void MakeSetParams(const iscu_psf_request& r, int M, int size, double resLateralNm, SetParams& sp)
{
   std::memset(&sp, 0, sizeof(sp));
   const double NA = r.na;
   const double lambda = r.wavelength_nm * 1E-9;
   sp.na = NA;
   sp.ni = r.immersion_index;
   sp.ns = r.sample_index;
   sp.depthM = r.sample_depth_nm * 1E-9;
   sp.k0 = 2.0 * kPi / lambda;
   sp.bMax = std::min(1.0, sp.ns / NA);
   sp.kMax = sp.k0 * NA * sp.bMax;
   sp.dk = (2.0 * sp.kMax) / (M - 4);
   sp.kMin = -std::floor(M / 2.0) * sp.dk;
   sp.dx = resLateralNm * 1E-9;
   sp.x0 = -((size - 1) / 2.0) * sp.dx;
   sp.doubleHelix = r.mask_double_helix ? 1 : 0;
   sp.maskModes = r.mask_modes;
   sp.maskWaist = r.mask_waist;
   int n = 0;
   for (int j = 0; j < 28; ++j)
   {
      if (r.zernike[j] == 0.0)
         continue;
      // OSA/ANSI j -> (n, l): j = n(n+1)/2 + k, l = -n + 2k (ZernikePsf.cpp:34-44).
      int nn = 0;
      while ((nn + 1) * (nn + 2) / 2 <= j)
         ++nn;
      const int k = j - nn * (nn + 1) / 2;
      const int l = -nn + 2 * k;
      sp.coeff[n] = r.zernike[j];
      sp.modeN[n] = nn;
      sp.modeL[n] = l;
      sp.modeM[n] = std::abs(l);
      // R_n^m = sum_k (-1)^k C(n - k, k) C(n - 2k, (n - m) / 2 - k) rho^(n - 2k) (ZernikePsf.cpp:58-67)
      const int half = (nn - std::abs(l)) / 2;
      for (int q = 0; q <= half; ++q)
         sp.radial[n][q] = (q % 2 ? -1.0 : 1.0) * Binomial(nn - q, q) * Binomial(nn - 2 * q, half - q);
      ++n;
   }
   sp.nModes = n;
   sp.ti0 = r.working_distance_um * 1E-6;
   sp.focalShift = sp.depthM * (sp.ni / sp.ns);
}

int BuildPsfLibrary(iscu_ctx* ctx, const iscu_psf_request* sets, uint32_t nSets, const uint32_t* setOfPsf,
                    const double* defocusM, uint32_t nPsf, int32_t size, int32_t normalize, int32_t method,
                    float* out)
{
   if (nSets == 0 || nPsf == 0)
      return ISCU_OK;
   std::string err;
   PsfGeometry g0;
   if (!GeometryFor(sets[0], g0, err))
      return Fail(ISCU_ERR_ARG, err);
   const int M = g0.M;
   const int P = size > 0 ? size : g0.size;
   std::vector<SetParams> hs(nSets);
   for (uint32_t s = 0; s < nSets; ++s)
   {
      PsfGeometry g;
      if (!GeometryFor(sets[s], g, err))
         return Fail(ISCU_ERR_ARG, err);
      if (g.M != M)
         return Fail(ISCU_ERR_ARG, "psf library: every set must have the same pupil samples");
      MakeSetParams(sets[s], M, P, g.resLateralNm, hs[s]);
   }
   std::vector<PsfItem> items(nPsf);
   for (uint32_t i = 0; i < nPsf; ++i)
   {
      if (setOfPsf[i] >= nSets)
         return Fail(ISCU_ERR_ARG, "psf library: set index out of range");
      const SetParams& sp = hs[setOfPsf[i]];
      items[i].set = static_cast<int>(setOfPsf[i]);
      // ti - ti0 = (ti0 - focalShift) + defocus - ti0 (ZernikePsf.cpp:237-243).
      const double ti = (sp.ti0 - sp.focalShift) + defocusM[i];
      items[i].dtiM = ti - sp.ti0;
   }
   const size_t tabBytes = static_cast<size_t>(nSets) * M * M * sizeof(double3);
   const size_t matBytes = static_cast<size_t>(nSets) * std::max(P, 2) * M * sizeof(float2);
   const size_t setBytes = (nSets * sizeof(SetParams) + 15) / 16 * 16, itemBytes = nPsf * sizeof(PsfItem);
   const bool split = method == ISCU_CZT_TF32X3 || method == ISCU_CZT_F16X3, folded = !split && FoldFits(M, P);
   // One buffer: the sets and the items (one copy), the tables, the matrices. The context keeps it up to kPsfScratchKept
   // bytes (calls hold the context's lock and end synchronized): five allocations and frees a call took 20 to 500 us.
   const size_t inBytes = (setBytes + itemBytes + 255) / 256 * 256, tabEnd = inBytes + (tabBytes + 255) / 256 * 256;
   const size_t aEnd = tabEnd + (matBytes + 255) / 256 * 256, allBytes = aEnd + (folded ? kFoldSumBytes : matBytes);
   DevBuf own;
   DevBuf& buf = allBytes <= kPsfScratchKept ? ctx->psfScratch : own;
   ISCU_CK(buf.Reserve(allBytes));
   unsigned char* base = buf.as<unsigned char>();
   double3* dTab = reinterpret_cast<double3*>(base + inBytes);
   float2* dA = reinterpret_cast<float2*>(base + tabEnd);
   float2* dAt = folded ? nullptr : reinterpret_cast<float2*>(base + aEnd);
   std::vector<unsigned char> in(setBytes + itemBytes);
   std::memcpy(in.data(), hs.data(), nSets * sizeof(SetParams));
   std::memcpy(in.data() + setBytes, items.data(), itemBytes);
   ISCU_CK(cudaMemcpyAsync(base, in.data(), in.size(), cudaMemcpyHostToDevice, ctx->stream));
   const SetParams* dSets = reinterpret_cast<const SetParams*>(base);
   const PsfItem* dItems = reinterpret_cast<const PsfItem*>(base + setBytes);
   int rc = LaunchPsfTables(ctx, dSets, nSets, M, P, dTab, dA, dAt, folded);
   if (rc == ISCU_OK)
      rc = split ? LaunchCztSplit(ctx, method, dSets, dTab, dA, nSets, dItems, nPsf, M, P, normalize, out)
                 : LaunchCztFp32(ctx, dSets, dTab, dA, dAt, reinterpret_cast<double2*>(base + aEnd), dItems, nPsf, M, P,
                                 normalize, out);
   if (rc != ISCU_OK)
      return rc;
   // The temporaries are another call's, or freed, when this returns; the stream must finish with them first.
   ISCU_CK(cudaStreamSynchronize(ctx->stream));
   return ISCU_OK;
}

// The set parameters of up to maxSets requests into caller memory (no heap): the pupil samples M and plane size P
// they share. Used by the allocation-free entry point (psf_noalloc.cu).
int PrepareSetParams(const iscu_psf_request* sets, uint32_t nSets, int32_t size, uint32_t maxSets, SetParams* out,
                     int* M, int* P)
{
   if (nSets == 0 || nSets > maxSets)
      return Fail(ISCU_ERR_LIMIT, "psf library: 1.." + std::to_string(maxSets) + " request sets");
   std::string err;
   PsfGeometry g0;
   if (!GeometryFor(sets[0], g0, err))
      return Fail(ISCU_ERR_ARG, err);
   *M = g0.M;
   *P = size > 0 ? size : g0.size;
   for (uint32_t s = 0; s < nSets; ++s)
   {
      PsfGeometry g;
      if (!GeometryFor(sets[s], g, err))
         return Fail(ISCU_ERR_ARG, err);
      if (g.M != *M)
         return Fail(ISCU_ERR_ARG, "psf library: every set must have the same pupil samples");
      MakeSetParams(sets[s], *M, *P, g.resLateralNm, out[s]);
   }
   return ISCU_OK;
}

int LaunchPsfTables(iscu_ctx* ctx, const SetParams* dSets, uint32_t nSets, int M, int P, double3* dTab, float2* dA,
                    float2* dAt, bool folded)
{
   const Fold F(M, P);   // (Q x pitch float2 of cs fit max(P, 2) x M)
   const int blocks = (M * M + kTableThreads - 1) / kTableThreads +
                      (folded ? (F.Q * F.Pitch() + kTableThreads - 1) / kTableThreads : 0);
   PupilTablesKernel<<<dim3(blocks, nSets), kTableThreads, 0, ctx->stream>>>(dSets, M, P, dTab, folded ? dA : nullptr);
   ISCU_CK_LAUNCH(ctx, "PupilTablesKernel");
   if (folded)
      return ISCU_OK;
   DftMatrixKernel<<<dim3((P * M + 255) / 256, nSets), 256, 0, ctx->stream>>>(dSets, M, P, dA, dAt);
   ISCU_CK_LAUNCH(ctx, "DftMatrixKernel");
   return ISCU_OK;
}

// The plain FP32 chirp-Z of nPsf items over prepared tables (the folded form where FoldFits, else the global-memory
// form for pupils beyond shared memory).
int LaunchCztFp32(iscu_ctx* ctx, const SetParams* dSets, const double3* dTab, const float2* dA, const float2* dAt,
                  double2* sums, const PsfItem* dItems, uint32_t nPsf, int M, int P, int normalize, float* out)
{
   if (FoldFits(M, P))
      return LaunchCztFold(ctx, dSets, dTab, dA, dItems, nPsf, M, P, normalize, sums, out);
   return LaunchCztGlobalFp32(ctx, dSets, dTab, dA, dAt, dItems, nPsf, M, P, normalize, out);
}

int CheckFp32CztSmem(iscu_ctx* ctx, int M, int P, size_t* smem)
{
   *smem = (static_cast<size_t>(M) * M + static_cast<size_t>(P) * M) * sizeof(float2);
   constexpr size_t kBeside = 64;   // static shared memory that the limit leaves room for
   int optin = 0;
   ISCU_CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
   if (*smem + kBeside > static_cast<size_t>(optin))
      return Fail(ISCU_ERR_LIMIT, "psf library (fp32): the pupil and row pass need (M*M + P*M)*8 = " +
                                     std::to_string(*smem) + " bytes of shared memory beside the kernel's " +
                                     std::to_string(kBeside) + ", over the device's " +
                                     std::to_string(optin) + " per block (M = " + std::to_string(M) + ", P = " +
                                     std::to_string(P) + ")");
   return ISCU_OK;
}

// The plain FP32 pipeline (tables, chirp-Z) on buffers the caller provides.
int LaunchPsfPipelineFp32(iscu_ctx* ctx, const SetParams* dSets, const PsfItem* dItems, double3* dTab, float2* dA,
                          float2* dAt, uint32_t nSets, uint32_t nPsf, int M, int P, int normalize, float* out)
{
   size_t smem = 0;
   int rc = CheckFp32CztSmem(ctx, M, P, &smem);   // (every shape within it folds)
   if (rc == ISCU_OK)
      rc = LaunchPsfTables(ctx, dSets, nSets, M, P, dTab, dA, dAt, true);
   if (rc == ISCU_OK)
      rc = LaunchCztFold(ctx, dSets, dTab, dA, dItems, nPsf, M, P, normalize, nullptr, out);   // (P <= 129: no split)
   return rc;
}

} // namespace iscu

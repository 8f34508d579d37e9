// The binned blink regime on sm_100a (sim::BinnedBlinkRenderer, adapter/inSiliScope/Simulation/BinnedBlinks.h:35-60,
// BinnedBlinks.cpp:150-248): the approximate SMLM render of dense frames.
//
// A frame's emitters (the splat's: photons, position, z plane) are deposited at the nearest cell of a grid of u cells
// per camera pixel, one density per PSF plane, and each plane is convolved with that plane's kernel resampled to the
// cell pitch; the planes' images are summed, clamped at 0 per cell and summed u x u into camera pixels.
// The reference convolves by float FFTs over a grid padded by the kernel radius R (no wrap-around into the frame):
// that is the linear convolution, which this file computes directly -- every cell sums float(photons) x kernel over
// the emitters within R cells, in float64 -- so the result is the FFT's up to its float rounding.
//
// Setup (BinnedBlinkRenderer::Setup, BinnedBlinks.cpp:150-214): u = KernelWidefieldPsf::ValidUpscale (the largest
// divisor of the kernel's oversampling up to the request, WidefieldRender.cpp:262-269); the plane kernels are
// KernelWidefieldPsf::Kernel (WidefieldRender.cpp:300-322), float64 r x r block sums (r = os / u) of the oversampled
// planes; R = KernelWidefieldPsf::Radius (:288-298) capped by the halo cut; or, without a kernel, the normalized
// Gaussian of sigma_px u (BinnedBlinks.cpp:190-212), made on the host with the same std::exp calls.
//
// Render (BinnedBlinks.cpp:216-246; dense frames further down), one CTA per 16 x 16 pixels of one frame, one thread per
// pixel holding its u x u cells: the frame's emitters are examined 256 at a time, those whose cell lies in the padded grid and within R of
// the tile staged in shared memory in event order, and every thread adds each staged emitter to its cells.

#include "iscu_internal.h"

#include <algorithm>
#include <cmath>
#include <vector>

struct iscu_binned
{
   iscu_ctx* ctx = nullptr;
   uint32_t W = 0, H = 0;
   int u = 1, R = 1, nz = 1;
   bool dense = false;     // the dense kernel's shared memory, plane table and number format hold this renderer
   int Pitch();            // sets the pitch from R and nz
   int pitch = 3;          // floats per kernel row: a multiple of 4 (zeros behind the row) where the dense kernel fits
   iscu::DevBuf kernels;   // nz x (2R + 1) x pitch floats
};

namespace iscu {
namespace {

constexpr int kThreads = 256;   // 16 x 16 pixels per CTA
constexpr int kSide = 16;

// KernelWidefieldPsf::Kernel: cell (dx, dy) of plane p = the sum, in float64 and row order, of the oversampled plane
// over [s0 + dy r, +r) x [s0 + dx r, +r) clipped to the plane, rounded to float.
// Rows of `pitch` floats, zeros behind the cells. odd (nullable): set to 1 by a cell that is negative or not finite.
__global__ void CellKernelsKernel(const float* __restrict__ planes, int n, int nz, int r, int s0, int R, int pitch,
                                  float* __restrict__ out, int* __restrict__ odd)
{
   const int D = 2 * R + 1, i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= nz * D * pitch)
      return;
   const int p = i / (D * pitch), c = i - p * D * pitch, dy = c / pitch - R, dx = c % pitch - R;
   if (dx > R)
   {
      out[i] = 0.f;
      return;
   }
   const float* P = planes + static_cast<size_t>(p) * n * n;
   const int ya = s0 + dy * r, yb = min(n, ya + r), xa = s0 + dx * r, xb = min(n, xa + r);
   double acc = 0.0;
   for (int y = max(0, ya); y < yb; ++y)
      for (int x = max(0, xa); x < xb; ++x)
         acc += P[static_cast<size_t>(y) * n + x];
   const float v = static_cast<float>(acc);
   out[i] = v;
   if (odd && __float_as_uint(v) >= 0x7F800000u)
      *odd = 1;
}

} // namespace

int LaunchCellKernels(iscu_ctx* ctx, const float* planes, int n, int nz, int r, int s0, int R, float* out)
{
   const int D = 2 * R + 1, total = nz * D * D;
   CellKernelsKernel<<<(total + 255) / 256, 256, 0, ctx->stream>>>(planes, n, nz, r, s0, R, D, out, nullptr);
   ISCU_CK_LAUNCH(ctx, "CellKernelsKernel");
   return ISCU_OK;
}

namespace {

struct Staged
{
   int cx, cy;   // the emitter's cell (unpadded grid)
   float photons;
   int plane;
};

// grid (ceil(W / 16), ceil(H / 16), frames). Frame k's emitters are emitters[em_start, em_start + em_count) cut at
// nEm. img / alone: frames x H x W, +=. kSparse: frames of denseFrom emitters and more are the dense kernel's (the test in
// every call's kernel made the compiler hold it to 32 registers: 20 frames of 93 x 58 px, 2,010 emitters each, 228 -> 239
// us).
template <int U, bool kSparse>
__global__ void __launch_bounds__(kThreads) BinnedRenderKernel(const iscu_emitter* __restrict__ em, uint32_t nEm,
                                                              const iscu_frame* __restrict__ frames,
                                                              uint32_t denseFrom, const float* __restrict__ K, int nz,
                                                              int R, int pitch, uint32_t W, uint32_t H,
                                                              float* __restrict__ img, float* __restrict__ alone)
{
   __shared__ Staged st[kThreads];
   __shared__ int warpKept[kThreads / 32];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int px = blockIdx.x * kSide + (threadIdx.x & (kSide - 1)), py = blockIdx.y * kSide + (threadIdx.x >> 4);
   const int gw = static_cast<int>(W) * U, gh = static_cast<int>(H) * U, D = 2 * R + 1;
   // the tile's cells, and the cells whose emitters reach them
   const int tx0 = blockIdx.x * kSide * U, ty0 = blockIdx.y * kSide * U;
   const int reachX0 = max(-R, tx0 - R), reachX1 = min(gw + R - 1, tx0 + kSide * U - 1 + R);
   const int reachY0 = max(-R, ty0 - R), reachY1 = min(gh + R - 1, ty0 + kSide * U - 1 + R);
   const iscu_frame fr = frames[blockIdx.z];
   const uint32_t start = min(fr.em_start, nEm), end = min(start + fr.em_count, nEm);
   if (kSparse && end > start && end - start >= denseFrom)
      return;
   const int cx = px * U, cy = py * U;   // this pixel's first cell
   double acc[U][U];
#pragma unroll
   for (int j = 0; j < U; ++j)
#pragma unroll
      for (int i = 0; i < U; ++i)
         acc[j][i] = 0.0;
   for (uint32_t base = start; base < end; base += kThreads)
   {
      Staged s{0, 0, 0.f, 0};
      bool keep = false;
      const uint32_t e = base + threadIdx.x;
      if (e < end)
      {
         const iscu_emitter m = em[e];
         if (m.photons > 0.0 && fabs(m.x_px) < 1e9 && fabs(m.y_px) < 1e9)
         {
            // pixel x spans [x - 0.5, x + 0.5): cell floor((x + 0.5) u)
            s.cx = static_cast<int>(floor((m.x_px + 0.5) * U));
            s.cy = static_cast<int>(floor((m.y_px + 0.5) * U));
            keep = s.cx >= reachX0 && s.cx <= reachX1 && s.cy >= reachY0 && s.cy <= reachY1;
            s.photons = static_cast<float>(m.photons);
            s.plane = min(nz - 1, max(0, m.plane & 0xFFFF));
         }
      }
      // staged in event order: the warps' kept counts, then each lane's rank in its warp
      const unsigned ballot = __ballot_sync(0xFFFFFFFFu, keep);
      if (lane == 0)
         warpKept[warp] = __popc(ballot);
      __syncthreads();
      int offset = 0, total = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w)
      {
         offset += w < warp ? warpKept[w] : 0;
         total += warpKept[w];
      }
      if (keep)
         st[offset + __popc(ballot & ((1u << lane) - 1u))] = s;
      __syncthreads();
      for (int k = 0; k < total; ++k)
      {
         const Staged t = st[k];
         const int dx0 = cx - t.cx, dy0 = cy - t.cy;
         if (dx0 > R || dx0 + U - 1 < -R || dy0 > R || dy0 + U - 1 < -R)
            continue;
         const float* Kp = K + t.plane * D * pitch;
         const double ph = t.photons;
         if (dx0 >= -R && dx0 + U - 1 <= R && dy0 >= -R && dy0 + U - 1 <= R)
         {
            // every cell of the pixel in reach (the common case): no per-cell test
            const float* Kc = Kp + (dy0 + R) * pitch + (dx0 + R);
#pragma unroll
            for (int j = 0; j < U; ++j)
#pragma unroll
               for (int i = 0; i < U; ++i)
                  acc[j][i] += ph * static_cast<double>(__ldg(Kc + j * pitch + i));
            continue;
         }
#pragma unroll
         for (int j = 0; j < U; ++j)
         {
            const int dy = dy0 + j;
            if (dy < -R || dy > R)
               continue;
#pragma unroll
            for (int i = 0; i < U; ++i)
            {
               const int dx = dx0 + i;
               if (dx >= -R && dx <= R)
                  acc[j][i] += ph * static_cast<double>(__ldg(Kp + (dy + R) * pitch + (dx + R)));
            }
         }
      }
      __syncthreads();   // the staging area is rewritten next round
   }
   if (px >= static_cast<int>(W) || py >= static_cast<int>(H))
      return;
   // a cell is the float image's value, clamped at 0; the pixel sums its cells in float64, rows first
   double sum = 0.0;
#pragma unroll
   for (int j = 0; j < U; ++j)
#pragma unroll
      for (int i = 0; i < U; ++i)
      {
         const float v = static_cast<float>(acc[j][i]);
         sum += v > 0.f ? v : 0.f;
      }
   const size_t o = (static_cast<size_t>(blockIdx.z) * H + py) * W + px;
   img[o] += static_cast<float>(sum);
   if (alone)
      alone[o] += static_cast<float>(sum);
}

// ------------------------------------------------------------------------------------------------ dense frames
// The same sums for frames of several emitters per plane, with the plane's kernel in shared memory and a block of
// cells in every thread's registers. A CTA takes 128 x 64 cells of a frame, a warp eight rows of them, a lane 4 x 8
// cells (columns lane, lane + 32, ...). The tile's emitters are sorted by plane (stable: event order within a plane)
// and each plane's kernel is staged once (while the plane before it is added, where two fit), with a margin of zeros
// as wide as a warp's block, so that an emitter costs a block one shared load, two shifts and one float64 multiply-add
// per cell and no test.
//
// The kernel stays float32 in shared memory (half the reads of float64, and a float -> double conversion issues at a
// quarter of the float64 rate): the double with the float's exponent and mantissa bits, hi = b >> 3, lo = b << 29, is
// K 2^-896 for every non-negative finite float, zero and subnormals included, and the photons carry 2^896, so the
// multiply-add rounds as photons x K does. An emitter whose photons are not a normal float is added cell by cell with
// the reach tested instead. Stacks with a negative or non-finite value take the kernel above (200 frames of
// 128 x 128 px, 2,400 emitters a frame, every plane signed: 2.05 ms; 3.76 when such planes were added cell by cell here).
//
// What bounds it: issue and the latency of 16 warps per SM (the accumulators are half the registers), the shared loads
// at 45 %, the float64 pipe at 15 %; 54 % of the multiply-adds lie in an emitter's reach at R = 32. 200 frames of
// 128 x 128 px, 2,400 emitters a frame, u = 2, R = 32: 1.05 ms against 2.03 ms of the kernel above. Slower (with the
// noise, against 1.18): 512 threads of four rows, 32 warps per SM, 1.34; a 64-bit multiply for the two shifts, 1.26.
constexpr int kTileX = 128, kTileY = 64, kRows = 8, kCap = 1024, kMaxPlanes = 512;
constexpr size_t kDenseMaxBytes = 226 * 1024;

struct DenseSmem
{
   uint2 kept[kCap];      // (cell x, y from the tile's corner as 16 + 16 bits, photons)
   uint2 sorted[kCap];
   uint16_t plane[kCap];
   int start[kMaxPlanes + 1], cursor[kMaxPlanes];
   int warpKept[kThreads / 32];
};
constexpr size_t kDenseHead = (sizeof(DenseSmem) + 15) / 16 * 16;

// Shared-memory row pitch (32 zeros, the row, at least 31 zeros) and rows of a staged kernel.
inline int DensePitch(int R) { return 2 * R + 1 + 63 <= 128 ? 128 : 192; }
inline int DenseRows(int R) { return 2 * R + 1 + 2 * (kRows - 1); }
inline size_t DenseKernelBytes(int R) { return sizeof(float) * DensePitch(R) * static_cast<size_t>(DenseRows(R)); }
inline bool DenseFits(int R, int nz) { return 2 * R + 1 + 63 <= 192 && nz <= kMaxPlanes; }
inline int DenseBuffers(int R) { return DensePitch(R) == 128 ? 2 : 1; }
inline size_t DenseBytes(int R)
{
   return kDenseHead + std::max(DenseBuffers(R) * DenseKernelBytes(R), sizeof(float) * kTileX * kTileY);
}

// Cell (gx, gy)'s sum over a frame's emitters [begin, end) in event order, as float (thread 0's). Out of line: it is
// rare, and its variables beside the accumulators took 200 frames of 128 x 128 px, 2,400 emitters a frame, from 1.05 to
// 1.08 ms.
__device__ __noinline__ float EventOrderCell(const iscu_emitter* __restrict__ em, uint32_t begin, uint32_t end,
                                             const float* __restrict__ K, int nz, int R, int U, int gx, int gy,
                                             DenseSmem& s)
{
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, D = 2 * R + 1, pitch = (D + 3) / 4 * 4;
   double* product = reinterpret_cast<double*>(s.plane);
   static_assert(sizeof(s.plane) >= sizeof(double) * kThreads, "a product per thread");
   double sum = 0.0;
   for (uint32_t base = begin; base < end; base += kThreads)
   {
      bool in = false;
      if (base + tid < end)
      {
         const iscu_emitter m = em[base + tid];
         if (m.photons > 0.0 && fabs(m.x_px) < 1e9 && fabs(m.y_px) < 1e9)
         {
            const int dx = gx - static_cast<int>(floor((m.x_px + 0.5) * U));
            const int dy = gy - static_cast<int>(floor((m.y_px + 0.5) * U));
            in = dx >= -R && dx <= R && dy >= -R && dy <= R;
            if (in)
            {
               const size_t row = static_cast<size_t>(min(nz - 1, max(0, m.plane & 0xFFFF))) * D + dy + R;
               product[tid] = static_cast<double>(static_cast<float>(m.photons)) *
                              static_cast<double>(K[row * pitch + dx + R]);
            }
         }
      }
      const unsigned ballot = __ballot_sync(0xFFFFFFFFu, in);
      if (lane == 0)
         s.warpKept[warp] = static_cast<int>(ballot);
      __syncthreads();
      if (tid == 0)
         for (int w = 0; w < kThreads / 32; ++w)
            for (unsigned left = static_cast<unsigned>(s.warpKept[w]); left; left &= left - 1)
               sum += product[32 * w + __ffs(left) - 1];
      __syncthreads();
   }
   return static_cast<float>(sum);
}

// kPitch: the staged row pitch, a constant so that a block's rows are immediate offsets.
template <int kPitch, int kBuffers>
__global__ void __launch_bounds__(kThreads, kBuffers) BinnedDenseKernel(
   const iscu_emitter* __restrict__ em, uint32_t nEm, const iscu_frame* __restrict__ frames, uint32_t denseFrom,
   const float* __restrict__ K, int nz, int R, int U, uint32_t W, uint32_t H, float* __restrict__ img,
   float* __restrict__ alone)
{
   extern __shared__ __align__(16) unsigned char smemRaw[];
   DenseSmem& s = *reinterpret_cast<DenseSmem*>(smemRaw);
   float* sK = reinterpret_cast<float*>(smemRaw + kDenseHead);
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   const int D = 2 * R + 1, rows = D + 2 * (kRows - 1), quads = (D + 3) / 4;
   const int pw = kTileX / U, phh = kTileY / U;   // the tile's pixels
   const int gw = static_cast<int>(W) * U, gh = static_cast<int>(H) * U;
   const int tx0 = blockIdx.x * pw * U, ty0 = blockIdx.y * phh * U;
   const int tx1 = min(tx0 + pw * U, gw) - 1, ty1 = min(ty0 + phh * U, gh) - 1;
   const int reachX0 = max(-R, tx0 - R), reachX1 = min(gw + R - 1, tx1 + R);
   const int reachY0 = max(-R, ty0 - R), reachY1 = min(gh + R - 1, ty1 + R);
   const iscu_frame fr = frames[blockIdx.z];
   const uint32_t begin = min(fr.em_start, nEm), end = min(begin + fr.em_count, nEm);
   if (end <= begin || end - begin < denseFrom)
      return;   // the per-pixel kernel's
   for (int i = tid; i < kBuffers * kPitch * rows; i += kThreads)
      sK[i] = 0.f;
   int total = 0;   // emitters that reach the tile
   double acc[kTileX / 32][kRows];
#pragma unroll
   for (int c = 0; c < kTileX / 32; ++c)
#pragma unroll
      for (int j = 0; j < kRows; ++j)
         acc[c][j] = 0.0;
   // plane p's rows into buffer `buf`, 16 bytes a copy
   const int stepRow = kThreads / quads, stepCol = kThreads % quads;
   auto stage = [&](int p, int buf) {
      const float* src = K + static_cast<size_t>(p) * D * quads * 4;
      float* dst = sK + buf * kPitch * rows + (kRows - 1) * kPitch + 32;
      int y = tid / quads, x = tid % quads;
      while (y < D)
      {
         const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst + y * kPitch + 4 * x));
         asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src + (y * quads + x) * 4) : "memory");
         y += stepRow;
         x += stepCol;
         if (x >= quads)
         {
            x -= quads;
            ++y;
         }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
   };
   for (uint32_t base = begin; base < end;)
   {
      // emitters that reach the tile, in event order, until the buffer could overflow
      int kept = 0;
      for (; base < end && kept <= kCap - kThreads; base += kThreads)
      {
         uint2 e = make_uint2(0, 0);
         int plane = 0;
         bool keep = false;
         if (base + tid < end)
         {
            const iscu_emitter m = em[base + tid];
            if (m.photons > 0.0 && fabs(m.x_px) < 1e9 && fabs(m.y_px) < 1e9)
            {
               const int cx = static_cast<int>(floor((m.x_px + 0.5) * U));
               const int cy = static_cast<int>(floor((m.y_px + 0.5) * U));
               keep = cx >= reachX0 && cx <= reachX1 && cy >= reachY0 && cy <= reachY1;
               const float ph = static_cast<float>(m.photons);
               e = make_uint2((static_cast<uint32_t>(cy - ty0) << 16) | (static_cast<uint32_t>(cx - tx0) & 0xFFFFu),
                              __float_as_uint(ph));
               plane = min(nz - 1, max(0, m.plane & 0xFFFF));
            }
         }
         const unsigned ballot = __ballot_sync(0xFFFFFFFFu, keep);
         if (lane == 0)
            s.warpKept[warp] = __popc(ballot);
         __syncthreads();
         int offset = kept;
#pragma unroll
         for (int w = 0; w < kThreads / 32; ++w)
         {
            offset += w < warp ? s.warpKept[w] : 0;
            kept += s.warpKept[w];
         }
         if (keep)
         {
            offset += __popc(ballot & ((1u << lane) - 1u));
            s.kept[offset] = e;
            s.plane[offset] = static_cast<uint16_t>(plane);
         }
         __syncthreads();
      }
      total += kept;
      // a stable counting sort by plane
      for (int p = tid; p < nz; p += kThreads)
         s.cursor[p] = 0;
      __syncthreads();
      for (int k = tid; k < kept; k += kThreads)
         atomicAdd(&s.cursor[s.plane[k]], 1);
      __syncthreads();
      if (warp == 0)
      {
         int carry = 0;
         for (int p0 = 0; p0 < nz; p0 += 32)
         {
            const int v = p0 + lane < nz ? s.cursor[p0 + lane] : 0;
            int x = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
            {
               const int u = __shfl_up_sync(0xFFFFFFFFu, x, d);
               x += lane >= d ? u : 0;
            }
            if (p0 + lane < nz)
               s.start[p0 + lane] = s.cursor[p0 + lane] = carry + x - v;
            carry += __shfl_sync(0xFFFFFFFFu, x, 31);
         }
         if (lane == 0)
            s.start[nz] = carry;
         __syncwarp();
         for (int k0 = 0; k0 < kept; k0 += 32)
         {
            const bool on = k0 + lane < kept;
            const int k = on ? k0 + lane : k0, plane = s.plane[k];
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, on ? plane : -1);
            const int rank = __popc(peers & ((1u << lane) - 1u));
            const int at = on ? s.cursor[plane] : 0;
            __syncwarp();
            if (on)
            {
               s.sorted[at + rank] = s.kept[k];
               if (rank == 0)
                  s.cursor[plane] = at + __popc(peers);
            }
            __syncwarp();
         }
      }
      __syncthreads();
      auto next = [&](int p) {
         while (p < nz && s.start[p] == s.start[p + 1])
            ++p;
         return p;
      };
      int p = next(0), buf = 0;
      if (kBuffers == 2 && p < nz)
         stage(p, buf);
      while (p < nz)
      {
         const int after = next(p + 1);
         if (kBuffers == 1)
            stage(p, 0);
         asm volatile("cp.async.wait_group 0;" ::: "memory");
         __syncthreads();   // the plane is staged, and the plane before it added by every warp
         if (kBuffers == 2 && after < nz)
            stage(after, buf ^ 1);
         const int k0 = s.start[p], k1 = s.start[p + 1];
         // the kernel's sample for (this warp's first row, this lane's first column) of an emitter in the tile's corner
         const float* Kb = sK + buf * kPitch * rows + (kRows * warp + R + kRows - 1) * kPitch + R + 32 + lane;
         for (int k = k0; k < k1; k += 32)
         {
            // 32 emitters at a time: which reach the warp's rows, and which of its column blocks
            const bool on = k + lane < k1;
            const uint2 e = s.sorted[on ? k + lane : k];
            const int ex = static_cast<int16_t>(e.x & 0xFFFFu), ey = static_cast<int>(e.x) >> 16;
            unsigned reach = __ballot_sync(0xFFFFFFFFu, on && static_cast<unsigned>(kRows * warp - ey + R + kRows - 1) <=
                                                                 static_cast<unsigned>(2 * R + kRows - 1));
            unsigned cols[kTileX / 32];
#pragma unroll
            for (int c = 0; c < kTileX / 32; ++c)
               cols[c] = __ballot_sync(0xFFFFFFFFu, static_cast<unsigned>(32 * c - ex + R + 31) <=
                                                       static_cast<unsigned>(2 * R + 31));
            const int offset = -ey * kPitch - ex;
            unsigned extreme =
               reach & __ballot_sync(0xFFFFFFFFu, e.y - 0x00800000u >= 0x7F000000u);   // not a normal float
            reach &= ~extreme;
            while (reach)
            {
               const int src = __ffs(reach) - 1;
               reach &= reach - 1;
               // photons x 2^896: a normal float's exponent, 896 up
               const unsigned pb = __shfl_sync(0xFFFFFFFFu, e.y, src);
               const double ph =
                  __hiloint2double(static_cast<int>((pb >> 3) + 0x70000000u), static_cast<int>(pb << 29));
               const float* Ke = Kb + __shfl_sync(0xFFFFFFFFu, offset, src);
#pragma unroll
               for (int c = 0; c < kTileX / 32; ++c)
                  if ((cols[c] >> src) & 1u)
                  {
#pragma unroll
                     for (int j = 0; j < kRows; ++j)
                     {
                        const unsigned b = __float_as_uint(Ke[32 * c + j * kPitch]);
                        acc[c][j] = fma(ph, __hiloint2double(static_cast<int>(b >> 3), static_cast<int>(b << 29)),
                                        acc[c][j]);
                     }
                  }
            }
            // the emitters of extreme photons, cell by cell
            while (extreme)
            {
               const int src = __ffs(extreme) - 1;
               extreme &= extreme - 1;
               const double ph = __uint_as_float(__shfl_sync(0xFFFFFFFFu, e.y, src));
               const int r0 = kRows * warp - __shfl_sync(0xFFFFFFFFu, ey, src);
               const int c0 = lane - __shfl_sync(0xFFFFFFFFu, ex, src);
               const float* Ke = Kb + __shfl_sync(0xFFFFFFFFu, offset, src);
#pragma unroll
               for (int c = 0; c < kTileX / 32; ++c)
#pragma unroll
                  for (int j = 0; j < kRows; ++j)
                     if (r0 + j >= -R && r0 + j <= R && c0 + 32 * c >= -R && c0 + 32 * c <= R)
                        acc[c][j] += ph * static_cast<double>(Ke[32 * c + j * kPitch]);
            }
         }
         if (kBuffers == 1)
            __syncthreads();   // the buffer is rewritten
         p = after;
         buf ^= kBuffers - 1;
      }
      __syncthreads();   // the sorted emitters are rewritten
   }
   // A cell is the float image's value, clamped at 0. Its products are exact and not negative, so its sum here and in
   // event order, of `total` terms at most, lie within 2 total + 2 of the sum's last places of each other: they round
   // to the same float unless a boundary is that near (about one cell in 200,000 at 600 emitters). Such a cell is
   // summed again in event order, so that a frame's image does not depend on which kernel its batch took (2 %).
   const unsigned doubt = 2u * min(static_cast<unsigned>(total), 0x08000000u) + 2u;
   uint16_t* again = reinterpret_cast<uint16_t*>(s.kept);   // kept and sorted: a number for every cell of the tile
   static_assert(sizeof(s.kept) + sizeof(s.sorted) >= sizeof(uint16_t) * kTileX * kTileY, "the cells summed again");
   if (tid == 0)
      s.start[0] = 0;
   __syncthreads();
#pragma unroll
   for (int c = 0; c < kTileX / 32; ++c)
#pragma unroll
      for (int j = 0; j < kRows; ++j)
      {
         const double a = acc[c][j];
         const float v = static_cast<float>(a);
         const int x = 32 * c + lane, y = kRows * warp + j;
         sK[y * kTileX + x] = v > 0.f ? v : 0.f;
         bool sure;
         if (v >= 1.17549435e-38f)
            // the 29 bits that the rounding drops, from their midpoint (infinity: 2^28 from it)
            sure = static_cast<unsigned>(abs((__double2loint(a) & 0x1FFFFFFF) - 0x10000000)) > doubt;
         else
         {
            // float's subnormals: in units of the smallest, where a NaN and 0 are sure in any order
            const double u = a * 0x1p149;
            sure = !(fabs(u - floor(u) - 0.5) <= u * (doubt * 0x1p-52));
         }
         if (!sure && x < pw * U && y < phh * U && tx0 + x < gw && ty0 + y < gh)
            again[atomicAdd(&s.start[0], 1)] = static_cast<uint16_t>(y * kTileX + x);
      }
   __syncthreads();
   const int nAgain = s.start[0];
   for (int i = 0; i < nAgain; ++i)
   {
      const int cell = again[i];
      const float v = EventOrderCell(em, begin, end, K, nz, R, U, tx0 + cell % kTileX, ty0 + cell / kTileX, s);
      if (tid == 0)
         sK[cell] = v > 0.f ? v : 0.f;
   }
   __syncthreads();
   for (int i = tid; i < pw * phh; i += kThreads)
   {
      const int x = i % pw, y = i / pw;
      const uint32_t px = blockIdx.x * pw + x, py = blockIdx.y * phh + y;
      if (px >= W || py >= H)
         continue;
      double sum = 0.0;
      for (int j = 0; j < U; ++j)
         for (int k = 0; k < U; ++k)
            sum += sK[(y * U + j) * kTileX + x * U + k];
      const size_t o = (static_cast<size_t>(blockIdx.z) * H + py) * W + px;
      img[o] += static_cast<float>(sum);
      if (alone)
         alone[o] += static_cast<float>(sum);
   }
}

using PixelFn = void (*)(const iscu_emitter*, uint32_t, const iscu_frame*, uint32_t, const float*, int, int, int,
                         uint32_t, uint32_t, float*, float*);
template <bool kSparse>
PixelFn PixelOf(int u)
{
   switch (u)
   {
   case 1: return BinnedRenderKernel<1, kSparse>;
   case 2: return BinnedRenderKernel<2, kSparse>;
   case 3: return BinnedRenderKernel<3, kSparse>;
   case 4: return BinnedRenderKernel<4, kSparse>;
   case 5: return BinnedRenderKernel<5, kSparse>;
   case 6: return BinnedRenderKernel<6, kSparse>;
   case 7: return BinnedRenderKernel<7, kSparse>;
   default: return BinnedRenderKernel<8, kSparse>;
   }
}

using DenseFn = void (*)(const iscu_emitter*, uint32_t, const iscu_frame*, uint32_t, const float*, int, int, int,
                         uint32_t, uint32_t, float*, float*);
DenseFn DenseOf(int R) { return DensePitch(R) == 128 ? BinnedDenseKernel<128, 2> : BinnedDenseKernel<192, 1>; }

// KernelWidefieldPsf::ValidUpscale (WidefieldRender.cpp:262-269).
int ValidUpscale(int oversampling, int requested)
{
   const int os = std::max(1, oversampling);
   for (int u = std::max(1, std::min(requested, os)); u > 1; --u)
      if (os % u == 0)
         return u;
   return 1;
}

// The emitters from which a frame is the dense kernel's in a call of n_emitters over n_frames; 0: no frame. A CTA pays
// for each plane it has an emitter of (the kernel's 17-66 KB staged, a barrier), the kernel above for every emitter and
// pixel: at two emitters of a plane within a tile's reach the two take the same (200 frames of 128 x 128 px, 49 planes,
// u = 2: 200, 400 and 2,400 emitters a frame 0.40, 0.32 (100 frames) and 2.18 ms against 0.44, 0.32 and 1.17, the
// camera's noise included); with one buffer and one CTA per SM (R > 32) at five (u = 4, R = 64, 20 frames of 2,400
// emitters, 5.9 a plane: 0.80 against 0.73 ms; 50 frames of 400: 0.37 against 0.73). Fewer tiles than two per SM leave it
// idle (100 frames of 64 x 64 px at u = 1: 88 against 108 us). The call's average only decides whether the dense kernel is
// launched: each frame goes by its own count, so that sparse frames of a long emitter array stay with the kernel above
// (200 frames of 100 emitters, their array a hundred times as long: 239 us when the average decided for all, 144 so, 138
// with an array of their own; frames of 2,400 emitters 1.05 and 1.08 ms. With one CTA of the kernel above per row of
// tiles beside the dense one 166 us and 1.07 ms).
uint32_t DenseFrom(const iscu_binned* b, uint32_t nEmitters, uint32_t nFrames)
{
   if (!b->dense || nFrames == 0)
      return 0;
   const uint32_t pw = kTileX / b->u, ph = kTileY / b->u;
   const uint64_t tiles = static_cast<uint64_t>((b->W + pw - 1) / pw) * ((b->H + ph - 1) / ph) * nFrames;
   const double reach = 2.0 * b->R, gw = static_cast<double>(b->W) * b->u, gh = static_cast<double>(b->H) * b->u;
   const double part = std::min(1.0, (kTileX + reach) / (gw + reach)) * std::min(1.0, (kTileY + reach) / (gh + reach));
   const double from = (DenseBuffers(b->R) == 2 ? 2.0 : 5.0) * b->nz / part;
   if (tiles < 2ull * static_cast<uint64_t>(b->ctx->smCount) || static_cast<double>(nEmitters) / nFrames < from)
      return 0;
   return static_cast<uint32_t>(std::ceil(from));   // (at least 2, and below nEmitters / nFrames + 1)
}

} // namespace
} // namespace iscu

using namespace iscu;

int iscu_binned::Pitch()
{
   const int D = 2 * R + 1;
   return pitch = DenseFits(R, nz) ? (D + 3) / 4 * 4 : D;
}

extern "C" {

int iscu_binned_create(iscu_ctx* ctx, int32_t slot, double sigma_px, uint32_t width, uint32_t height, int32_t upscale,
                       iscu_binned** out)
{
   if (!ctx || !out)
      return Fail(ISCU_ERR_ARG, "null argument");
   *out = nullptr;
   if (width == 0 || height == 0)
      return Fail(ISCU_ERR_ARG, "binned render: width and height >= 1");
   if (slot >= ISCU_MAX_KERNELS)
      return Fail(ISCU_ERR_ARG, "kernel slot out of range (-1..3)");
   std::lock_guard<std::recursive_mutex> lock(ctx->mu);
   ClearError();
   std::unique_ptr<iscu_binned> b(new iscu_binned());
   b->ctx = ctx;
   b->W = width;
   b->H = height;
   int odd = 0;   // a kernel value is negative or not finite (the Gaussian's are neither)
   if (slot >= 0)
   {
      const KernelSlot& k = ctx->kernels[slot];
      if (!k.valid)
         return Fail(ISCU_ERR_STATE, "no kernel stack in slot " + std::to_string(slot));
      const int os = std::max(1, k.os), n = k.size;
      b->u = ValidUpscale(os, upscale);
      // KernelWidefieldPsf: blocks of r oversampled samples per cell, the cell at offset 0 from s0 (a dye at a cell
      // centre, as SplatSetup places it: tx = kc - r/2 + 0.5 rounded half up)
      const int r = std::max(1, os / b->u);
      const double kc = (n - 1) / 2.0;
      const int s0 = static_cast<int>(std::floor(kc - r / 2.0 + 1.0));
      const int dMin = static_cast<int>(std::ceil((-s0 - r + 1) / static_cast<double>(r)));
      const int dMax = static_cast<int>(std::floor((n - 1 - s0) / static_cast<double>(r)));
      b->R = std::max(1, std::max(-dMin, dMax));
      // the halo cut bounds what the splat draws; the cell kernel stops there too
      if (k.halo && !k.radius2Host.empty())
      {
         const int32_t r2 = *std::max_element(k.radius2Host.begin(), k.radius2Host.end());
         if (r2 >= 0)
            b->R = std::min(b->R, static_cast<int>(std::ceil((std::sqrt(static_cast<double>(r2)) + 1.0) * b->u)));
      }
      b->R = std::max(1, b->R);
      b->nz = std::max(1, k.nz);
      const int D = 2 * b->R + 1, total = b->nz * D * b->Pitch();
      const size_t bytes = static_cast<size_t>(total) * sizeof(float);
      ISCU_CK(b->kernels.Reserve(bytes + sizeof(int)));   // and the flag
      int* flag = reinterpret_cast<int*>(b->kernels.as<unsigned char>() + bytes);
      ISCU_CK(cudaMemsetAsync(flag, 0, sizeof(int), ctx->stream));
      CellKernelsKernel<<<(total + 255) / 256, 256, 0, ctx->stream>>>(k.planes.as<float>(), n, b->nz, r, s0, b->R,
                                                                        b->pitch, b->kernels.as<float>(), flag);
      ISCU_CK_LAUNCH(ctx, "CellKernelsKernel");
      ISCU_CK(cudaMemcpyAsync(&odd, flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      ISCU_CK(cudaStreamSynchronize(ctx->stream));
   }
   else
   {
      if (!(sigma_px > 0.0))
         return Fail(ISCU_ERR_ARG, "binned render: no kernel slot and no Gaussian sigma");
      b->u = std::max(1, std::min(upscale, 8));
      b->R = std::max(1, static_cast<int>(std::ceil(3.0 * sigma_px * b->u)));
      b->nz = 1;
      const int R = b->R, D = 2 * R + 1;
      const double sc = sigma_px * b->u, twoS2 = 2.0 * sc * sc;
      std::vector<double> g(static_cast<size_t>(D) * D);
      double sum = 0.0;
      for (int y = -R; y <= R; ++y)
         for (int x = -R; x <= R; ++x)
         {
            const double v = std::exp(-(static_cast<double>(x) * x + static_cast<double>(y) * y) / twoS2);
            g[static_cast<size_t>(y + R) * D + (x + R)] = v;
            sum += v;
         }
      std::vector<float> gf(static_cast<size_t>(D) * b->Pitch());
      for (size_t i = 0; i < g.size(); ++i)
         gf[i / D * b->pitch + i % D] = static_cast<float>(g[i] / sum);
      ISCU_CK(b->kernels.Reserve(gf.size() * sizeof(float)));
      ISCU_CK(cudaMemcpyAsync(b->kernels.p, gf.data(), gf.size() * sizeof(float), cudaMemcpyHostToDevice,
                              ctx->stream));
   }
   if (b->u > 8)
      return Fail(ISCU_ERR_LIMIT, "binned render: at most 8 cells per pixel");
   if (DenseFits(b->R, b->nz) && !odd)
   {
      ISCU_CK(cudaFuncSetAttribute(DenseOf(b->R), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(kDenseMaxBytes)));
      b->dense = true;
   }
   ISCU_CK(cudaStreamSynchronize(ctx->stream));
   *out = b.release();
   return ISCU_OK;
}

int iscu_binned_info(iscu_binned* b, int32_t* upscale, int32_t* radius_cells, int32_t* planes)
{
   if (!b)
      return Fail(ISCU_ERR_ARG, "null renderer");
   if (upscale)
      *upscale = b->u;
   if (radius_cells)
      *radius_cells = b->R;
   if (planes)
      *planes = b->nz;
   return ISCU_OK;
}

int iscu_binned_dense_from(iscu_binned* b, uint32_t n_emitters, uint32_t n_frames, uint32_t* count)
{
   if (!b || !count)
      return Fail(ISCU_ERR_ARG, "null argument");
   *count = DenseFrom(b, n_emitters, n_frames);
   return ISCU_OK;
}

int iscu_binned_kernels(iscu_binned* b, float* out)
{
   if (!b || !out)
      return Fail(ISCU_ERR_ARG, "null argument");
   std::lock_guard<std::recursive_mutex> lock(b->ctx->mu);
   ClearError();
   const size_t D = 2 * static_cast<size_t>(b->R) + 1;
   ISCU_CK(cudaMemcpy2DAsync(out, D * sizeof(float), b->kernels.p, b->pitch * sizeof(float), D * sizeof(float),
                             b->nz * D, cudaMemcpyDeviceToHost, b->ctx->stream));
   ISCU_CK(cudaStreamSynchronize(b->ctx->stream));
   return ISCU_OK;
}

void iscu_binned_destroy(iscu_binned* b)
{
   if (!b)
      return;
   cudaStreamSynchronize(b->ctx->stream);
   delete b;
}

int iscu_binned_render_dev(iscu_binned* b, const iscu_emitter* emitters_dev, uint32_t n_emitters,
                           const iscu_frame* frames_dev, uint32_t n_frames, float* img_dev, float* alone_dev)
{
   if (!b || (n_frames && (!frames_dev || !img_dev)) || (n_emitters && !emitters_dev))
      return Fail(ISCU_ERR_ARG, "null argument");
   if (n_frames > 65535)
      return Fail(ISCU_ERR_LIMIT, "at most 65535 frames per call");
   iscu_ctx* ctx = b->ctx;
   std::lock_guard<std::recursive_mutex> lock(ctx->mu);
   ClearError();
   if (!n_frames)
      return ISCU_OK;
   const float* K = b->kernels.as<float>();
   const uint32_t denseFrom = DenseFrom(b, n_emitters, n_frames);
   if (denseFrom)
   {
      const uint32_t pw = kTileX / b->u, ph = kTileY / b->u;
      DenseOf(b->R)<<<dim3((b->W + pw - 1) / pw, (b->H + ph - 1) / ph, n_frames), kThreads, DenseBytes(b->R),
                      ctx->stream>>>(emitters_dev, n_emitters, frames_dev, denseFrom, K, b->nz, b->R, b->u, b->W, b->H,
                                     img_dev, alone_dev);
      ISCU_CK_LAUNCH(ctx, "BinnedDenseKernel");
   }
   const dim3 grid((b->W + kSide - 1) / kSide, (b->H + kSide - 1) / kSide, n_frames);
   const PixelFn fn = denseFrom ? PixelOf<true>(b->u) : PixelOf<false>(b->u);
   fn<<<grid, kThreads, 0, ctx->stream>>>(emitters_dev, n_emitters, frames_dev, denseFrom, K, b->nz, b->R, b->pitch,
                                          b->W, b->H, img_dev, alone_dev);
   ISCU_CK_LAUNCH(ctx, "BinnedRenderKernel");
   return ISCU_OK;
}

} // extern "C"

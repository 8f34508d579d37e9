// The two-pass render on sm_100a: the same frames, bit for bit, as the one-pass tile render (render.cu), with the
// float64 tap arithmetic regrouped so that the FP64 pipe, not the tap loads, bounds it.
//
// A splat's value at pixel (dx, dy) of its square is float(photons * sum_j wy[j] (sum_i wx[i] B[r0 + j][c0 + i]))
// (SplatKernel.inl:51-171) with r0 = by + dy os + os - 1, c0 = bx + dx os + os - 1: the block sums it reads depend
// only on the kernel slot, the z plane and the tap origin (bx, by), which takes at most os + 1 values per axis. So:
//
//  1. setup (one thread per emitter): SplatSetup (PsfGeneratorBridge.cpp:1382-1422), and the emitter's group
//     (slot, plane, bx, by) counted;
//  2. the groups' offsets (a scan by the last CTA of the setup) and 3. each emitter listed under its group;
//  4. contributions: a CTA takes a group's block of square pixels and up to 64 of its emitters; each thread loads its
//     pixel's taps into registers once and computes every emitter's float contribution -- the reference's value, from
//     a fused sum where that rounds alike -- into HBM (emitter-major, one float per pixel of the square);
//  5. gather (one CTA per frame tile, or a persistent grid heaviest frame first): every pixel adds, in the frame's
//     emitter order, the contributions of the emitters whose square (and halo cut) covers it -- the same float
//     additions in the same order as RenderPhotonImage (SMLMSimulation.cpp:103-160) -- then the noise chain
//     (ApplyNoiseChain, SMLMNoise.cpp:142-216) in registers.
//
// Compiled with --fmad=false: every float64 multiply and add rounds on its own, as the reference's -ffp-contract=off
// build does.

#include "counter_rng.cuh"
#include "iscu_internal.h"
#include "noise_chain.cuh"
#include "splat_common.cuh"

#include <algorithm>
#include <cstdint>

namespace iscu {

namespace {

constexpr int kE = 64;          // emitters per contribution chunk
// Contribution CTAs: at most kMaxCT computing threads and a staging warp, four per SM (72 registers: the 16 float64 taps
// in registers). A 33 x 33 square is six pixel blocks; 224 x 3, 256 x 3 and 352 x 2 threads measured 1.5 to 6 % more.
constexpr int kMaxCT = 192;
constexpr int kContribPerSm = 4;
constexpr int kGT = 256;        // gather CTA size (one thread per pixel of the tile)
constexpr int kGList = 64;       // a warp's list: worked off when the next 32 emitters may not fit
constexpr int kGChunk = 256;    // gather staging chunk

// The group keys: slot s owns keys [base[s], base[s + 1]); key base[s] + (plane n1 + (by - lo)) n1 + (bx - lo) is the
// group (s, plane, bx, by); the slot's last key collects tap origins outside [lo, lo + n1) (none arise from finite
// positions: SplatSetup keeps by, bx within [kc - os - 1, kc + 1]).
struct KeyMap
{
   int base[ISCU_MAX_KERNELS + 1];
   int lo[ISCU_MAX_KERNELS];
   int n1[ISCU_MAX_KERNELS];
   int side[ISCU_MAX_KERNELS];   // splat square side, 2 camRad + 1
   int pbs[ISCU_MAX_KERNELS];    // pixel blocks of the square: a chunk's work items
};

// The contribution pass's work list (the last CTA of the setup writes it): the items' total, the next item, and each
// slot's first chunk and first item. A slot's keys, so its chunks and items, are consecutive.
struct Work
{
   uint32_t items, next;
   uint32_t chunk[ISCU_MAX_KERNELS], item[ISCU_MAX_KERNELS];
};

__device__ __forceinline__ int TapsOf(const KernelView& kv)
{
   return kv.interp == ISCU_INTERP_CUBIC ? 4 : (kv.interp == ISCU_INTERP_LINEAR ? 2 : 1);
}

// ------------------------------------------------------------------------------------------------ 1. setup
struct SetupArgs
{
   const iscu_emitter* ems;
   uint32_t n;
   Kernels K;
   KeyMap km;
   int* key;          // per emitter; -1: not splatted
   int4* grec;        // per emitter (x0, y0, slot, plane); slot -1: not splatted
   uint32_t* count;   // per key, zero beforehand; then the CTAs done, zero beforehand
   uint32_t* start;   // the offsets (ScanKeys)
   uint32_t* cursor;
   uint32_t* chunkStart;
   Work* work;
};

// An emitter's slot, SplatSetup and key (false: not splatted).
__device__ __forceinline__ bool SetupEmitter(const Kernels& K, const KeyMap& km, const iscu_emitter& em, int& slot,
                                             int& plane, int& key, StagedEmitter& s)
{
   slot = static_cast<int>(static_cast<uint32_t>(em.plane) >> 16);
   plane = em.plane & 0xffff;
   if (!(slot < ISCU_MAX_KERNELS && em.photons > 0.0 && K.k[slot].sums64 && plane < K.k[slot].nz &&
         PositionOk(em.x_px, em.y_px)))
      return false;
   s.x0 = static_cast<int>(RoundHalfUp(em.x_px));
   s.y0 = static_cast<int>(RoundHalfUp(em.y_px));
   SetupWeights(K.k[slot], em.x_px, em.y_px, s);
   const int n1 = km.n1[slot], cy = s.by - km.lo[slot], cx = s.bx - km.lo[slot];
   key = (cy >= 0 && cy < n1 && cx >= 0 && cx < n1) ? km.base[slot] + (plane * n1 + cy) * n1 + cx
                                                    : km.base[slot + 1] - 1;
   return true;
}

// 2. The offsets, by one CTA of kSetupThreads threads, kScanPer consecutive keys a thread and pass: start[k] = cursor[k] =
// exclusive sum of count, chunkStart[k] = exclusive sum of the keys' chunks (ceil(count / kE)); the work list. (The
// chunks' records are written by the scatter: one thread listing all of a key's work in turn took 14 of 26 us on the
// two-colour movie.)
constexpr int kSetupThreads = 512, kScanPer = 8;
__device__ __forceinline__ void ScanKeys(const SetupArgs& a)
{
   constexpr int kWarps = kSetupThreads / 32;
   const int nKeys = a.km.base[ISCU_MAX_KERNELS];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   __shared__ uint32_t sw[2][kWarps], firstChunk[ISCU_MAX_KERNELS + 1];
   uint32_t carryC = 0, carryI = 0;
   for (int k0 = 0; k0 < nKeys; k0 += kSetupThreads * kScanPer)
   {
      const int kb = k0 + static_cast<int>(threadIdx.x) * kScanPer;
      uint32_t c[kScanPer], it[kScanPer], tc = 0, ti = 0;
#pragma unroll
      for (int j = 0; j < kScanPer; ++j)
         c[j] = kb + j < nKeys ? __ldcg(a.count + kb + j) : 0u;
#pragma unroll
      for (int j = 0; j < kScanPer; ++j)
      {
         it[j] = (c[j] + kE - 1) / kE;
         tc += c[j];
         ti += it[j];
      }
      uint32_t xc = tc, xi = ti;   // inclusive warp scans of the threads' totals
#pragma unroll
      for (int d = 1; d < 32; d <<= 1)
      {
         const uint32_t u = __shfl_up_sync(0xffffffffu, xc, d), v = __shfl_up_sync(0xffffffffu, xi, d);
         if (lane >= d)
         {
            xc += u;
            xi += v;
         }
      }
      __syncthreads();   // the pass before has read sw
      if (lane == 31)
      {
         sw[0][warp] = xc;
         sw[1][warp] = xi;
      }
      __syncthreads();
      uint32_t ec = carryC + xc - tc, ei = carryI + xi - ti;
#pragma unroll
      for (int w = 0; w < kWarps; ++w)
      {
         ec += w < warp ? sw[0][w] : 0u;
         ei += w < warp ? sw[1][w] : 0u;
         carryC += sw[0][w];
         carryI += sw[1][w];
      }
#pragma unroll
      for (int j = 0; j < kScanPer; ++j)
      {
         const int k = kb + j;
         if (k < nKeys)
         {
            a.start[k] = ec;
            a.cursor[k] = ec;
            a.chunkStart[k] = ei;
#pragma unroll
            for (int t = 0; t < ISCU_MAX_KERNELS; ++t)
               if (k == a.km.base[t])
                  firstChunk[t] = ei;
         }
         ec += c[j];
         ei += it[j];
      }
   }
   __syncthreads();
   if (threadIdx.x == 0)
   {
      firstChunk[ISCU_MAX_KERNELS] = carryI;
      for (int t = ISCU_MAX_KERNELS; t-- > 0;)
         if (a.km.base[t] == a.km.base[t + 1])
            firstChunk[t] = firstChunk[t + 1];   // a slot without keys
      uint32_t items = 0;
      for (int t = 0; t < ISCU_MAX_KERNELS; ++t)
      {
         a.work->chunk[t] = firstChunk[t];
         a.work->item[t] = items;
         items += (firstChunk[t + 1] - firstChunk[t]) * static_cast<uint32_t>(a.km.pbs[t]);
      }
      a.work->items = items;
      a.work->next = 0;
   }
}

// The emitters' keys, counted; the last CTA to finish works out the keys' offsets (a launch of one CTA for them was 7 us
// on its own).
__global__ void __launch_bounds__(kSetupThreads) ContribSetupKernel(SetupArgs a)
{
   const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
   bool valid = false;
   int key = -1;
   if (g < a.n)
   {
      int slot = 0, plane = 0;
      StagedEmitter s;
      int4 gr = make_int4(0, 0, -1, 0);
      valid = SetupEmitter(a.K, a.km, a.ems[g], slot, plane, key, s);
      if (valid)
         gr = make_int4(s.x0, s.y0, slot, plane);
      a.grec[g] = gr;
      a.key[g] = valid ? key : -1;
   }
   const unsigned vm = __ballot_sync(0xffffffffu, valid);
   if (valid)
   {
      const unsigned peers = __match_any_sync(vm, key);
      if ((threadIdx.x & 31) == __ffs(peers) - 1)
         atomicAdd(&a.count[key], static_cast<uint32_t>(__popc(peers)));
   }
   __shared__ bool last;
   __threadfence();   // the counts before the CTA's arrival
   __syncthreads();
   if (threadIdx.x == 0)
      last = atomicAdd(a.count + a.km.base[ISCU_MAX_KERNELS], 1u) == gridDim.x - 1;
   __syncthreads();
   if (!last)
      return;
   __threadfence();
   ScanKeys(a);
}

// ------------------------------------------------------------------------------------------------ 3. lists
// An emitter as the contribution pass stages it; the lists hold these records in group order.
struct __align__(16) CStage
{
   double wx[4], wp[4];   // the column weights; the row weights times the photons
   uint32_t g;
   float thr;             // 2^-10 x 1.6 photons: below thr x the taps' largest magnitude a sum cancels too much;
                          // infinite (every sum in doubt) where that is no normal float
   int bx, by;
   double photons;
   double wy[4];
   int plane, pad;
};
static_assert(sizeof(CStage) == 128, "8 x 16 bytes");

// Up to kE emitters of one group, with what is the same for the group's pixels: worked out once a chunk (the tap
// offsets' divisions alone were 400 instructions a thread and work item, a third of the contribution pass).
struct __align__(16) CChunk
{
   int off[16];          // tap (j, i)'s offset in the phase layout from a pixel's own word
   const double* base;   // the plane's words of the phase layout
   int first, cnt;       // stage records
   int slot, plane;
   int kind;             // 0 the misc group; 1 tap origins beyond the phase layout; 2 within it
   float invSide;
   int pad[8];
};
static_assert(sizeof(CChunk) == 128, "8 x 16 bytes");

struct ScatterArgs
{
   const iscu_emitter* ems;
   uint32_t n;
   Kernels K;
   KeyMap km;
   const int* key;
   const uint32_t* count;
   const uint32_t* start;
   uint32_t* cursor;
   const uint32_t* chunkStart;
   CStage* stage;
   CChunk* chunk;
};

// Each emitter's record in its group's list; the first emitter of a chunk writes the chunk's.
__global__ void ContribScatterKernel(ScatterArgs a)
{
   const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
   const int key = g < a.n ? a.key[g] : -1;
   const bool valid = key >= 0;
   const unsigned vm = __ballot_sync(0xffffffffu, valid);
   if (!valid)
      return;
   const int lane = threadIdx.x & 31;
   const unsigned peers = __match_any_sync(vm, key);
   const int leader = __ffs(peers) - 1;
   uint32_t base = 0;
   if (lane == leader)
      base = atomicAdd(&a.cursor[key], static_cast<uint32_t>(__popc(peers)));
   base = __shfl_sync(peers, base, leader);
   const uint32_t at = base + __popc(peers & ((1u << lane) - 1u));
   const iscu_emitter em = a.ems[g];
   int slot = 0, plane = 0, k2 = 0;
   StagedEmitter s;
   SetupEmitter(a.K, a.km, em, slot, plane, k2, s);
   CStage c;
#pragma unroll
   for (int k = 0; k < 4; ++k)
   {
      c.wx[k] = s.wx[k];
      c.wy[k] = s.wy[k];
      c.wp[k] = em.photons * s.wy[k];
   }
   c.photons = em.photons;
   c.thr = static_cast<float>(em.photons * (1.6 / 1024.0));
   if (!(c.thr >= 1.17549435e-38f))
      c.thr = __int_as_float(0x7f800000);   // (no float bound of so few photons)
   c.g = g;
   c.bx = s.bx;
   c.by = s.by;
   c.plane = plane;
   c.pad = 0;
   a.stage[at] = c;
   const uint32_t pos = at - a.start[key];
   if (pos % kE != 0)
      return;
   const KernelView& kv = a.K.k[slot];
   const int os = kv.os, nt = TapsOf(kv), ext = kv.nb * os, span = kv.camRad * os, nb2 = kv.nb * kv.nb;
   const int R = s.by + os - 1 + kv.padLo, C = s.bx + os - 1 + kv.padLo;
   const bool misc = key == a.km.base[slot + 1] - 1;
   const bool fits = !misc && kv.phase && R - span >= 0 && R + span + nt - 1 < ext && C - span >= 0 &&
                     C + span + nt - 1 < ext;
   CChunk h;
   int off[2][4];   // each axis' taps: the phase's plane and word
   int row = R / os, ph = R - row * os, col = C / os, cph = C - col * os;
#pragma unroll
   for (int j = 0; j < 4; ++j)
   {
      off[0][j] = ph * os * nb2 + row * kv.nb;
      off[1][j] = cph * nb2 + col;
      ph = ph + 1 == os ? (++row, 0) : ph + 1;
      cph = cph + 1 == os ? (++col, 0) : cph + 1;
   }
#pragma unroll
   for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i)
         h.off[4 * j + i] = fits ? off[0][j] + off[1][i] : 0;
   h.base = kv.phase + static_cast<size_t>(misc ? 0 : plane) * os * os * nb2;
   h.first = static_cast<int>(at);
   h.cnt = static_cast<int>(min(static_cast<uint32_t>(kE), a.count[key] - pos));
   h.slot = slot;
   h.plane = plane;
   h.kind = misc ? 0 : (fits ? 2 : 1);
   h.invSide = 1.f / static_cast<float>(a.km.side[slot]);
   a.chunk[a.chunkStart[key] + pos / kE] = h;
}

// ------------------------------------------------------------------------------------------------ 4. contributions
struct ContribArgs
{
   KeyMap km;
   Kernels K;
   const CChunk* chunk;
   const CStage* stage;  // the emitters in group order
   Work* work;
   float* contrib;       // emitter g's square at contrib[g S ..]
   uint32_t S;
};

// The reference's row = 0; row += wx[i] B; sum += wy[j] row over NT x NT taps held in registers, started from the
// first product (the same values; at most the sign of a zero partial sum differs, which the pixel's float add cannot
// see). Taps outside the bw x bw array are the layout's zero margin where the reference skips them.
template <int NT>
__device__ __forceinline__ double RegisterTaps(const double (&t)[4][4], const CStage& e)
{
   double row[NT];
#pragma unroll
   for (int j = 0; j < NT; ++j)
   {
      double r = e.wx[0] * t[j][0];
#pragma unroll
      for (int i = 1; i < NT; ++i)
         r += e.wx[i] * t[j][i];
      row[j] = r;
   }
   double sum = e.wy[0] * row[0];
#pragma unroll
   for (int j = 1; j < NT; ++j)
      sum += e.wy[j] * row[j];
   return sum;
}

// The same sum with the photons in the row weights and fused multiply-adds: 20 float64 instructions against 36. It and
// photons x RegisterTaps differ by at most 21 roundings of A = sum |wp wx B|, below 2^-48 A.
template <int NT>
__device__ __forceinline__ double FusedTaps(const double (&t)[4][4], const CStage& e)
{
   double sum = 0.0;
#pragma unroll
   for (int j = 0; j < NT; ++j)
   {
      double r = e.wx[0] * t[j][0];
#pragma unroll
      for (int i = 1; i < NT; ++i)
         r = fma(e.wx[i], t[j][i], r);
      sum = j == 0 ? e.wp[0] * r : fma(e.wp[j], r, sum);
   }
   return sum;
}

// The contribution float(photons x sum) of the reference's operation order, from the fused sum c where c rounds to
// the same float surely: A <= 1.5625 photons x the taps' largest magnitude (the weights' magnitudes sum to at most
// 1.25 per axis), so with |c| at least 2^-10 x 1.6 photons x that magnitude the two sums lie within 2^-38 |c| of each
// other, 2^15 of c's last places, and round alike unless a float's midpoint (bit 28 alone of the 29 dropped) is that
// near. In doubt (one in 8,000, and where the taps cancel or the photons are extreme) in the reference's order. `big`:
// the magnitude, at least; `small`: the least |c| taken (-1 where every tap is 0).
template <int NT>
__device__ __forceinline__ bool SureContribution(const double (&t)[4][4], const CStage& e, float big, float small, float& f)
{
   const double c = FusedTaps<NT>(t, e);
   f = static_cast<float>(c);
   const float least = fmaf(e.thr, big, small);
   const unsigned near = static_cast<unsigned>(__double2loint(c)) * 8u + (0x80000000u + (1u << 18));
   return near > (1u << 19) && fabsf(f) >= least && least < 1e30f;
}

template <int NT>
__device__ __forceinline__ float ExactContribution(const double (&t)[4][4], const CStage& e)
{
   return static_cast<float>(e.photons * RegisterTaps<NT>(t, e));
}

// Any tap origin, from the row-major float64 sums with the reference's bounds (the misc group).
__device__ __forceinline__ double BoundedTaps(const KernelView& kv, const CStage& e, int nt, int dx, int dy)
{
   const int os = kv.os, off = os - 1, bw = kv.bw;
   const long long r0 = static_cast<long long>(e.by) + static_cast<long long>(dy) * os + off;
   const long long c0 = static_cast<long long>(e.bx) + static_cast<long long>(dx) * os + off;
   const double* B = kv.sums64 + static_cast<size_t>(e.plane) * bw * bw;
   double sum = 0.0;
   for (int j = 0; j < nt; ++j)
   {
      const long long r = r0 + j;
      if (r < 0 || r >= bw)
         continue;
      double row = 0.0;
      for (int i = 0; i < nt; ++i)
      {
         const long long c = c0 + i;
         if (c >= 0 && c < bw)
            row += e.wx[i] * __ldg(B + static_cast<size_t>(r) * bw + static_cast<size_t>(c));
      }
      sum += e.wy[j] * row;
   }
   return sum;
}

__device__ __forceinline__ bool HaloKeeps(const KernelView& kv, int plane, int dx, int dy)
{
   if (!kv.spanLo)
      return true;
   const int cr = kv.camRad, row = plane * (2 * cr + 1) + dy + cr;
   return dx >= kv.spanLo[row] && dx <= kv.spanHi[row];
}

template <int NT>
__device__ __forceinline__ void GroupContrib(const ContribArgs& a, const KernelView& kv, const CChunk& it,
                                             const CStage* E, int p, int dx, int dy, bool active)
{
   const int cnt = it.cnt;
   if (it.kind == 1)
   {
      for (int k = 0; k < cnt; ++k)
         if (active)
            a.contrib[static_cast<size_t>(E[k].g) * a.S + p] =
               static_cast<float>(E[k].photons * BoundedTaps(kv, E[k], NT, dx, dy));
      return;
   }
   double t[4][4];
   const double* base = it.base + (active ? dy * kv.nb + dx : 0);
#pragma unroll
   for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < NT; ++i)
         t[j][i] = __ldg(base + it.off[4 * j + i]);
   // an upper bound of the taps' magnitudes from their high words
   int hi = 0;
#pragma unroll
   for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < NT; ++i)
         hi = max(hi, __double2hiint(t[j][i]) & 0x7fffffff);
   const float big = hi ? static_cast<float>(__hiloint2double(hi + 1, 0)) : 0.f, small = hi ? 1e-30f : -1.f;
   float* out = a.contrib + p;
   // Where the first emitter is in doubt for a pixel of the warp the others mostly are too (a steep stack's far pixels:
   // a Gaussian falls by more than 2^10 between neighbouring taps): then all in the reference's order at once. (35 M
   // contributions of a Gaussian of 1.2 px in 33 x 33 squares: 200 us with both sums, 138 so; 119 and 115 where few are
   // in doubt.)
   float f;
   const bool sure = SureContribution<NT>(t, E[0], big, small, f);
   if (__any_sync(0xffffffffu, active && !sure))
   {
#pragma unroll 2
      for (int k = 0; k < cnt; ++k)
      {
         const float v = ExactContribution<NT>(t, E[k]);
         if (active)
            out[static_cast<size_t>(E[k].g) * a.S] = v;
      }
      return;
   }
   if (active)
      out[static_cast<size_t>(E[0].g) * a.S] = f;
   int k = 1;
   for (; k + 1 < cnt; k += 2)
   {
      const CStage& e0 = E[k];
      const CStage& e1 = E[k + 1];
      float v0, v1;
      if (!SureContribution<NT>(t, e0, big, small, v0))
         v0 = ExactContribution<NT>(t, e0);
      if (!SureContribution<NT>(t, e1, big, small, v1))
         v1 = ExactContribution<NT>(t, e1);
      if (active)
      {
         out[static_cast<size_t>(e0.g) * a.S] = v0;
         out[static_cast<size_t>(e1.g) * a.S] = v1;
      }
   }
   if (k < cnt && active)
   {
      if (!SureContribution<NT>(t, E[k], big, small, f))
         f = ExactContribution<NT>(t, E[k]);
      out[static_cast<size_t>(E[k].g) * a.S] = f;
   }
}

// All of the CTA's warps, from either role's loop.
__device__ __forceinline__ void RoleBarrier() { asm volatile("bar.sync 0;" ::: "memory"); }

// blockDim.x = computing threads + one staging warp, three buffers: while the others compute item i, the staging warp
// has item i + 1's emitters arriving, issues item i + 2's copy, whose chunk it asked for an item ago, and asks for item
// i + 3's chunk and number i + 4, so that each of these round trips has an item's time. (Fetched one after the other
// within an item they took longer than a short item's work.) An item is one block of computing threads' pixels of a
// chunk, as many a chunk as its own slot's square has (as many as the largest square of all slots, 120,000 emitters of
// 7 x 7 squares beside a stack of 81 x 81 took 205 us instead of 46). The two roles have a loop each: in one loop the
// staging warp's variables made the others spill (35 M contributions 118.8 us, 114.7 without).
//
// What bounds it: the emitter loop, some 84 cycles a warp's contribution and scheduler where its 20 float64 operations
// and the conversion need 56 (a float64 operation issues every 2.35 cycles, a conversion takes 8.5); 54 instructions in
// all, the FP64 pipe at 40 %. Taps, chunk and barriers are 20 % on the dSTORM movie, 9 % on the two-colour one. 35 M
// contributions of the dSTORM movie 133 -> 115 us, 525 M of the two-colour movie 1.44 -> 1.24 ms against unfused sums
// with each thread's own tap offsets. Building the float from the double's bits instead of converting, and two or four
// emitters without a branch between them, measured 5 to 40 % slower (more integer instructions; spilled taps).
__global__ void __launch_bounds__(kMaxCT + 32, kContribPerSm) ContribKernel(ContribArgs a)
{
   __shared__ CStage sE[3][kE];
   __shared__ CChunk sChunk[3];
   __shared__ uint32_t sBlock[3];   // the items' pixel blocks; kNoItem: none is left
   constexpr uint32_t kNoItem = 0xFFFFFFFFu;
   const int nc = static_cast<int>(blockDim.x) - 32;   // computing threads
   const bool stager = static_cast<int>(threadIdx.x) >= nc;
   const int sl = static_cast<int>(threadIdx.x) - nc;  // lane of the staging warp
   const uint32_t items = a.work->items;
   constexpr int kHead = static_cast<int>(sizeof(CChunk) / 16), kRec = static_cast<int>(sizeof(CStage) / 16);
   uint32_t ahead = 0, asked = 0, block = 0;   // lane 0: the number asked for; the item whose chunk is on its way
   int4 head = make_int4(0, 0, 0, 0);  // that chunk's 16 bytes of this lane
   // (a CTA's first three items are its own; the counter hands out the rest)
   auto number = [&] {
      if (sl == 0)
         ahead = 3 * gridDim.x + atomicAdd(&a.work->next, 1u);
   };
   // lane t holds slot t's first item, first chunk and items per chunk
   uint32_t item0 = 0xFFFFFFFFu, chunk0 = 0, per = 1;
   if (stager && sl < ISCU_MAX_KERNELS)
   {
      item0 = a.work->item[sl];
      chunk0 = a.work->chunk[sl];
      per = static_cast<uint32_t>(max(1, a.km.pbs[sl]));
   }
   auto chunk = [&](uint32_t i, uint32_t& block) {
      // the last slot whose items start at or before i (those that share its start have none)
      const int slot = 31 - __clz(static_cast<int>(__ballot_sync(0xffffffffu, i >= item0)));
      const uint32_t in = i - __shfl_sync(0xffffffffu, item0, slot), n = __shfl_sync(0xffffffffu, per, slot);
      const uint32_t c = in / n, at = __shfl_sync(0xffffffffu, chunk0, slot) + c;
      block = in - c * n;
      int4 h = make_int4(0, 0, 0, 0);
      if (i < items && sl < kHead)
         h = __ldg(reinterpret_cast<const int4*>(a.chunk + at) + sl);
      return h;
   };
   auto copy = [&](int buf, uint32_t i, uint32_t block, const int4& h) {
      if (sl == 0)
         sBlock[buf] = i < items ? block : kNoItem;
      if (i < items)
      {
         if (sl < kHead)
            reinterpret_cast<int4*>(&sChunk[buf])[sl] = h;
         __syncwarp();
         const int n = sChunk[buf].cnt * kRec;
         const int4* from = reinterpret_cast<const int4*>(a.stage + sChunk[buf].first);
         const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(sE[buf]));
         for (int t = sl; t < n; t += 32)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16u * t), "l"(from + t) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
   };
   if (stager)
   {
      number();
      const uint32_t i0 = blockIdx.x, i1 = i0 + gridDim.x;
      asked = i1 + gridDim.x;
      uint32_t b0, b1;
      const int4 h0 = chunk(i0, b0), h1 = chunk(i1, b1);
      head = chunk(asked, block);
      copy(0, i0, b0, h0);
      copy(1, i1, b1, h1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      RoleBarrier();
      for (int cur = 0; sBlock[cur] != kNoItem; cur = cur == 2 ? 0 : cur + 1)
      {
         copy(cur == 0 ? 2 : cur - 1, asked, block, head);   // item i + 2 (the buffer of item i - 1, done)
         asked = __shfl_sync(0xffffffffu, ahead, 0);
         head = chunk(asked, block);
         number();
         asm volatile("cp.async.wait_group 1;" ::: "memory");   // item i + 1 is there
         RoleBarrier();
      }
      return;
   }
   RoleBarrier();
   for (int cur = 0;; cur = cur == 2 ? 0 : cur + 1)
   {
      const uint32_t pixels = sBlock[cur];
      if (pixels == kNoItem)
         return;
      const CChunk& it = sChunk[cur];
      const int slot = it.slot;
      const KernelView& kv = a.K.k[slot];
      const int side = a.km.side[slot], cr = kv.camRad;
      const int p = static_cast<int>(pixels) * nc + static_cast<int>(threadIdx.x);
      const bool inSquare = p < side * side;
      // p / side: the quotient's fraction is at least half a 1 / side from a whole number, the float product's error
      // below that for squares of up to 4 M pixels; larger ones divide
      int row = static_cast<int>((static_cast<float>(p) + 0.5f) * it.invSide);
      if (side > 2000)
         row = p / side;
      const int dx = inSquare ? p - row * side - cr : 0, dy = inSquare ? row - cr : 0;
      const int nt = TapsOf(kv);
      const CStage* E = sE[cur];
      if (__any_sync(0xffffffffu, inSquare))
      {
         const bool active = inSquare && (it.kind == 0 || HaloKeeps(kv, it.plane, dx, dy));
         if (it.kind == 0)
         {
            // the misc group: every emitter with its own plane and tap origin
            for (int k = 0; k < it.cnt; ++k)
               if (inSquare && HaloKeeps(kv, E[k].plane, dx, dy))
                  a.contrib[static_cast<size_t>(E[k].g) * a.S + p] =
                     static_cast<float>(E[k].photons * BoundedTaps(kv, E[k], nt, dx, dy));
         }
         else if (nt == 4)
            GroupContrib<4>(a, kv, it, E, p, dx, dy, active);
         else if (nt == 2)
            GroupContrib<2>(a, kv, it, E, p, dx, dy, active);
         else
            GroupContrib<1>(a, kv, it, E, p, dx, dy, active);
      }
      RoleBarrier();
   }
}

// ------------------------------------------------------------------------------------------------ 5. gather
// A staged emitter as one warp adds it: its contribution to the warp's first pixel (counted from the square's pitch, so
// perhaps outside the square), the pitch, and the pixels of the warp's kSub rectangles that its square and halo cut
// cover.
template <int kSub>
struct __align__(16) GEntry
{
   const float* first;
   int side;
   unsigned covers[kSub];
};

struct GatherArgs
{
   const iscu_frame* frames;
   uint32_t nFrames;
   uint32_t nEm;
   const uint32_t* order;    // persistent form: frames, heaviest first
   uint32_t* counter;        // persistent form: the next work item
   const int4* grec;
   const float* contrib;
   uint32_t S;
   Kernels K;
   StaticView st;
   CameraView cam;
   uint32_t seed;
   float* photonsOut;
   uint16_t* aduOut;
};

// Stages one chunk of a frame's emitters whose square reaches the tile, in list order. Every thread calls it.
__device__ __forceinline__ int GatherStage(const GatherArgs& a, uint32_t start, uint32_t count, int tx0, int ty0,
                                           int tx1, int ty1, int4* sG, uint32_t* sId, int* sWarp)
{
   const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
   bool keep = false;
   int4 gr = make_int4(0, 0, -1, 0);
   if (static_cast<uint32_t>(t) < count)
   {
      gr = a.grec[start + t];
      if (gr.z >= 0)
      {
         const int cr = a.K.k[gr.z].camRad;
         keep = gr.x + cr >= tx0 && gr.x - cr <= tx1 && gr.y + cr >= ty0 && gr.y - cr <= ty1;
      }
   }
   const unsigned ballot = __ballot_sync(0xffffffffu, keep);
   if (lane == 0)
      sWarp[warp] = __popc(ballot);
   __syncthreads();
   int base = 0, total = 0;
#pragma unroll
   for (int w = 0; w < kGT / 32; ++w)
   {
      const int c = sWarp[w];
      base += w < warp ? c : 0;
      total += c;
   }
   if (keep)
   {
      base += __popc(ballot & ((1u << lane) - 1u));
      sG[base] = gr;
      sId[base] = start + t;
   }
   __syncthreads();
   return total;
}

// The pixels of the warp's CW x 32 / CW rectangle at (wx0, wy0) that emitter gr's square and halo cut cover, a bit per
// lane.
template <int CW>
__device__ __forceinline__ unsigned Covers(const KernelView& kv, const int4& gr, int wx0, int wy0)
{
   const int cr = kv.camRad, x0 = gr.x - wx0;
   const int lo = max(0, x0 - cr), hi = min(CW - 1, x0 + cr);
   unsigned m = 0;
#pragma unroll
   for (int r = 0; r < 32 / CW; ++r)
   {
      const int dy = wy0 + r - gr.y;
      if (dy < -cr || dy > cr)
         continue;
      int l = lo, h = hi;
      if (kv.spanLo)
      {
         const int at = gr.w * (2 * cr + 1) + dy + cr;
         l = max(l, x0 + kv.spanLo[at]);
         h = min(h, x0 + kv.spanHi[at]);
      }
      if (l <= h)
         m |= ((2u << h) - (1u << l)) << (r * CW & 31);
   }
   return m;
}

// A thread's pixels' adds of the warp's entries, in list order, four entries' loads in flight. The lanes' tests are
// worked out once an entry, a lane per emitter, when the list is made, so that an add is a shared load, a bit test, the
// address and the load, the first and the last two shared by the kSub pixels (TX apart).
template <int TX, int kSub>
__device__ __forceinline__ void GatherAdds(const GEntry<kSub>* list, int n, const unsigned (&bit)[kSub], int lx, int ly,
                                           float (&acc)[kSub])
{
   for (int m = 0; m < n; m += 4)
   {
      float v[4][kSub];
#pragma unroll
      for (int u = 0; u < 4; ++u)
      {
         const GEntry<kSub>& e = list[m + u];   // (the list ends in entries that cover nothing)
         const float* p = e.first + (ly * e.side + lx);
#pragma unroll
         for (int q = 0; q < kSub; ++q)
            v[u][q] = e.covers[q] & bit[q] ? __ldg(p + q * TX) : 0.0f;   // (acc is never -0: adding 0 keeps it)
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
         for (int q = 0; q < kSub; ++q)
            acc[q] += v[u][q];
   }
}

// Every lane of the warp calls it.
template <int TX, int kSub>
__device__ __forceinline__ void GatherFlush(GEntry<kSub>* list, int n, int lane, const unsigned (&bit)[kSub], int lx,
                                            int ly, float (&acc)[kSub])
{
   if (lane < 4 && (n & 3))
      list[n + lane] = GEntry<kSub>{};
   __syncwarp();
   GatherAdds<TX, kSub>(list, n, bit, lx, ly, acc);
   __syncwarp();
}

// kSub: a CTA's tile is kSub tiles of TX x TY side by side, a thread's pixels TX apart: what a CTA does for a chunk of
// emitters (staging, the warps' lists) is half the gather's instructions at 256 x 256 px and 430 emitters a frame, and
// two pixels share it. Six CTAs per SM (40 registers; the noise chain spills a little): the gather's loads and the Knuth
// loops are latency-bound, and the extra warps hide more than the spills cost. Issue-bound (83 %; half of it the noise
// chain): dSTORM movie 139 -> 118 us, two-colour movie 2.85 -> 2.19 ms, against a test of the pixel's distances for each
// emitter and one tile a CTA.
template <int TX, int TY, bool kNoise, bool kPersistent, int kSub>
__global__ void __launch_bounds__(kGT, 6) GatherTilesKernel(GatherArgs a)
{
   static_assert(TX * TY == kGT, "one thread per pixel of the tile");
   static_assert(TX % 32 == 0 || 32 % TX == 0, "a warp covers a rectangle of the tile");
   __shared__ int4 sG[kGChunk];
   __shared__ uint32_t sId[kGChunk];
   __shared__ GEntry<kSub> sList[kGT / 32][kGList];
   __shared__ int sWarp[kGT / 32];
   __shared__ uint32_t sItem;
   const int W = static_cast<int>(a.st.width), H = static_cast<int>(a.st.height);
   constexpr int kTX = kSub * TX;
   const uint32_t tilesX = (W + kTX - 1) / kTX, tilesY = (H + TY - 1) / TY, tilesPerFrame = tilesX * tilesY;
   const uint32_t total = a.nFrames * tilesPerFrame;
   const int warp = threadIdx.x >> 5;
   GEntry<kSub>* list = sList[warp];
   constexpr int CW = TX >= 32 ? 32 : TX;   // a warp's pixels: CW x 32 / CW, kSub times
   const int lane = threadIdx.x & 31, lx = lane % CW, ly = lane / CW;
   const int wcx = TX >= 32 ? (32 * warp) % TX : 0, wry = (32 * warp) / TX;
   for (;;)
   {
      uint32_t f, tile;
      if (kPersistent)
      {
         if (threadIdx.x == 0)
            sItem = atomicAdd(a.counter, 1u);
         __syncthreads();
         const uint32_t item = sItem;
         __syncthreads();
         if (item >= total)
            return;
         f = a.order[item / tilesPerFrame];
         tile = item % tilesPerFrame;
      }
      else
      {
         f = blockIdx.z;
         tile = blockIdx.y * tilesX + blockIdx.x;
      }
      const iscu_frame fr = a.frames[f];
      const uint32_t emCount = fr.em_start < a.nEm ? min(fr.em_count, a.nEm - fr.em_start) : 0u;
      const int tx0 = static_cast<int>(tile % tilesX) * kTX, ty0 = static_cast<int>(tile / tilesX) * TY;
      const int X = tx0 + static_cast<int>(threadIdx.x % TX), Y = ty0 + static_cast<int>(threadIdx.x / TX);
      const int tx1 = min(tx0 + kTX, W) - 1, ty1 = min(ty0 + TY, H) - 1;
      const uint32_t i = static_cast<uint32_t>(Y) * a.st.width + static_cast<uint32_t>(X);
      const int wx0 = tx0 + wcx, wy0 = ty0 + wry;
      float acc[kSub];
      unsigned bit[kSub];
#pragma unroll
      for (int q = 0; q < kSub; ++q)
      {
         const bool inside = X + q * TX < W && Y < H;
         bit[q] = inside ? 1u << lane : 0u;
         acc[q] = inside ? Background(a.st, i + q * TX, fr.bg_scale) : 0.0f;
      }
      int listed = 0;
      for (uint32_t e0 = 0; e0 < emCount; e0 += kGChunk)
      {
         const uint32_t cnt = min(static_cast<uint32_t>(kGChunk), emCount - e0);
         const int kept = GatherStage(a, fr.em_start + e0, cnt, tx0, ty0, tx1, ty1, sG, sId, sWarp);
         for (int k0 = 0; k0 < kept; k0 += 32)
         {
            // the staged emitters that cover a pixel of the warp, a lane per emitter
            GEntry<kSub> e{};
            unsigned any = 0;
            if (k0 + lane < kept)
            {
               const int4 gr = sG[k0 + lane];
               const KernelView& kv = a.K.k[gr.z];
#pragma unroll
               for (int q = 0; q < kSub; ++q)
                  any |= e.covers[q] = Covers<CW>(kv, gr, wx0 + q * TX, wy0);
               e.side = 2 * kv.camRad + 1;
               e.first = a.contrib + static_cast<size_t>(sId[k0 + lane]) * a.S +
                         ((wy0 - gr.y + kv.camRad) * e.side + wx0 - gr.x + kv.camRad);
            }
            const unsigned hit = __ballot_sync(0xffffffffu, any != 0u);
            if (any)
               list[listed + __popc(hit & ((1u << lane) - 1u))] = e;
            listed += __popc(hit);
            __syncwarp();
            if (listed > kGList - 36)   // (32 more, and the entries that end a list)
            {
               GatherFlush<TX, kSub>(list, listed, lane, bit, lx, ly, acc);
               listed = 0;
            }
         }
         if (e0 + kGChunk < emCount)   // (a persistent CTA's next tile starts with barriers)
            __syncthreads();
      }
      GatherFlush<TX, kSub>(list, listed, lane, bit, lx, ly, acc);
      // (one copy of the noise chain, gone through kSub times)
#pragma unroll 1
      for (int q = 0; q < kSub; ++q)
      {
         float v = acc[0];
         unsigned in = bit[0];
#pragma unroll
         for (int r = 1; r < kSub; ++r)
         {
            v = q == r ? acc[r] : v;
            in = q == r ? bit[r] : in;
         }
         if (!in)
            continue;
         const size_t o = static_cast<size_t>(f) * a.st.width * a.st.height + i + q * TX;
         if (a.photonsOut)
            a.photonsOut[o] = v;
         if (kNoise)
         {
            CounterRng u(a.seed, fr.frame);
            a.aduOut[o] = NoisePixel(v, i + q * TX, a.cam, a.st, u);
         }
      }
      if (!kPersistent)
         return;
   }
}

using GatherFn = void (*)(GatherArgs);
template <bool kNoise, bool kPersistent, int kSub>
GatherFn GatherTile(int tile)
{
   switch (tile)
   {
   case 0: return GatherTilesKernel<16, 16, kNoise, kPersistent, kSub>;
   case 1: return GatherTilesKernel<32, 8, kNoise, kPersistent, kSub>;
   default: return GatherTilesKernel<8, 32, kNoise, kPersistent, kSub>;
   }
}
constexpr int kTileW[3] = {16, 32, 8}, kTileH[3] = {16, 8, 32};

} // namespace

namespace {

struct ContribGeometry
{
   KeyMap km = {};
   int nKeys = 0, ct = 32;   // computing threads of a contribution CTA
   size_t S = 1;
};

ContribGeometry GeometryOf(const iscu_ctx* ctx)
{
   ContribGeometry G;
   int maxS2 = 1;
   for (int s = 0; s < ISCU_MAX_KERNELS; ++s)
   {
      G.km.base[s] = G.nKeys;
      const KernelSlot& k = ctx->kernels[s];
      if (!k.valid)
         continue;
      const int cr = k.halfOv / k.os, side = 2 * cr + 1;
      G.km.side[s] = side;
      G.km.n1[s] = k.os + 4;
      G.km.lo[s] = k.halfOv - k.os - 2;
      G.nKeys += k.nz * G.km.n1[s] * G.km.n1[s] + 1;
      maxS2 = std::max(maxS2, side * side);
   }
   G.km.base[ISCU_MAX_KERNELS] = G.nKeys;
   const int blocks = (maxS2 + kMaxCT - 1) / kMaxCT;   // of the largest square
   G.ct = std::min(kMaxCT, ((maxS2 + blocks - 1) / blocks + 31) / 32 * 32);
   for (int s = 0; s < ISCU_MAX_KERNELS; ++s)
      G.km.pbs[s] = (G.km.side[s] * G.km.side[s] + G.ct - 1) / G.ct;
   G.S = static_cast<size_t>(maxS2);
   return G;
}

// An upper bound of the chunks: the full ones and one partial chunk per key, no more than emitters.
size_t MaxChunks(const ContribGeometry& G, uint32_t nEm)
{
   return std::min<size_t>(nEm, static_cast<size_t>(nEm) / kE + static_cast<size_t>(G.nKeys)) + 1;
}

// The scratch of nEm emitters: one buffer's parts, each on 256 bytes.
struct ContribLayout
{
   size_t key = 0, grec, keys, list, chunks, work, contrib, bytes;
   ContribLayout(const ContribGeometry& G, uint32_t nEm)
   {
      const size_t n = std::max<uint32_t>(nEm, 1u);
      const auto after = [](size_t at, size_t size) { return (at + size + 255) / 256 * 256; };
      grec = after(key, n * sizeof(int));
      keys = after(grec, n * sizeof(int4));
      list = after(keys, (4 * static_cast<size_t>(G.nKeys) + 1) * sizeof(uint32_t));
      chunks = after(list, n * sizeof(CStage));
      work = after(chunks, MaxChunks(G, nEm) * sizeof(CChunk));
      contrib = after(work, sizeof(Work));
      bytes = after(contrib, n * G.S * sizeof(float));
   }
};

} // namespace

int ReserveContrib(iscu_ctx* ctx, uint32_t nEm, ContribScratch& sc)
{
   const ContribGeometry G = GeometryOf(ctx);
   if (ctx->contribLimit == 0)
   {
      size_t freeB = 0, totalB = 0;
      ISCU_CK(cudaMemGetInfo(&freeB, &totalB));
      ctx->contribLimit = totalB / 4;
   }
   const size_t contribBytes = static_cast<size_t>(nEm) * G.S * sizeof(float);
   if (contribBytes > ctx->contribLimit)
      return Fail(ISCU_ERR_LIMIT, "two-pass render: contributions of " + std::to_string(nEm) + " emitters need " +
                                     std::to_string(contribBytes >> 20) + " MiB, over the limit");
   if (ContribLayout(G, nEm).bytes <= sc.buf.bytes && sc.buf.p)
      return ISCU_OK;
   // Room for some more emitters than asked for, so that a movie's batches, a few emitters apart, are not each the first
   // pass of a larger buffer (an allocation and a free wait for the device: 0.1 to 5 ms): a 32nd at first, an eighth when
   // it grows, within the limit.
   const uint64_t most = ctx->contribLimit / (G.S * sizeof(float));
   const uint64_t more = std::min<uint64_t>(std::min<uint64_t>(most, 0xFFFFFFFFu), nEm + nEm / (sc.buf.p ? 8u : 32u));
   if (more > nEm)
   {
      if (sc.buf.Reserve(ContribLayout(G, static_cast<uint32_t>(more)).bytes) == cudaSuccess)
         return ISCU_OK;
      cudaGetLastError();   // no room for more than asked for
   }
   ISCU_CK(sc.buf.Reserve(ContribLayout(G, nEm).bytes));
   return ISCU_OK;
}

int LaunchContribRender(iscu_ctx* ctx, int tileConfig, const iscu_emitter* ems, uint32_t nEm,
                        const iscu_frame* frames, uint32_t nFrames, const CameraView* cam, uint32_t seed,
                        float* photons, uint16_t* adu, uint32_t* orderBuf, ContribScratch& sc)
{
   if (nFrames == 0)
      return ISCU_OK;
   const int rcReserve = ReserveContrib(ctx, nEm, sc);
   if (rcReserve != ISCU_OK)
      return rcReserve;
   const ContribGeometry G = GeometryOf(ctx);
   const KeyMap& km = G.km;
   const int nKeys = G.nKeys;
   const size_t S = G.S;
   cudaEvent_t* marks = RenderMarks(ctx);
   if (marks)
      ISCU_CK(cudaEventRecord(marks[0], ctx->stream));
   const ContribLayout L(G, nEm);
   unsigned char* base = sc.buf.as<unsigned char>();
   int* key = reinterpret_cast<int*>(base + L.key);
   int4* grec = reinterpret_cast<int4*>(base + L.grec);
   CStage* list = reinterpret_cast<CStage*>(base + L.list);
   CChunk* chunks = reinterpret_cast<CChunk*>(base + L.chunks);
   Work* work = reinterpret_cast<Work*>(base + L.work);
   float* contrib = reinterpret_cast<float*>(base + L.contrib);
   uint32_t* count = reinterpret_cast<uint32_t*>(base + L.keys);   // and the CTAs done
   uint32_t* start = count + nKeys + 1;
   uint32_t* cursor = start + nKeys;
   uint32_t* chunkStart = cursor + nKeys;
   const Kernels K = KernelsOfCtx(ctx);
   if (nEm > 0)
   {
      ISCU_CK(cudaMemsetAsync(count, 0, (static_cast<size_t>(nKeys) + 1) * sizeof(uint32_t), ctx->stream));
      SetupArgs sa{ems, nEm, K, km, key, grec, count, start, cursor, chunkStart, work};
      ContribSetupKernel<<<(nEm + kSetupThreads - 1) / kSetupThreads, kSetupThreads, 0, ctx->stream>>>(sa);
      ISCU_CK_LAUNCH(ctx, "ContribSetupKernel");
      if (nKeys > 0)
      {
         ScatterArgs xa{ems, nEm, K, km, key, count, start, cursor, chunkStart, list, chunks};
         ContribScatterKernel<<<(nEm + 255) / 256, 256, 0, ctx->stream>>>(xa);
         ISCU_CK_LAUNCH(ctx, "ContribScatterKernel");
         if (marks)
            ISCU_CK(cudaEventRecord(marks[1], ctx->stream));
         ContribArgs ca{km, K, chunks, list, work, contrib, static_cast<uint32_t>(S)};
         ContribKernel<<<kContribPerSm * ctx->smCount, G.ct + 32, 0, ctx->stream>>>(ca);
         ISCU_CK_LAUNCH(ctx, "ContribKernel");
      }
   }
   if (marks)
   {
      if (nEm == 0 || nKeys == 0)
         ISCU_CK(cudaEventRecord(marks[1], ctx->stream));
      ISCU_CK(cudaEventRecord(marks[2], ctx->stream));
   }
   GatherArgs ga;
   ga.frames = frames;
   ga.nFrames = nFrames;
   ga.nEm = nEm;
   ga.grec = grec;
   ga.contrib = contrib;
   ga.S = static_cast<uint32_t>(S);
   ga.K = K;
   ga.st = ctx->Static();
   ga.cam = cam ? *cam : CameraView();
   ga.seed = seed;
   ga.photonsOut = photons;
   ga.aduOut = cam ? adu : nullptr;
   const int tile = tileConfig % 3;
   const bool persistent = tileConfig / 3 == 1;
   // Two tiles a CTA from 12 CTAs an SM on (six run on one): tiles pass of frames of 128 x 128 px, 160 emitters each, at 9
   // a SM 32 us with one and with two, at 17 55 and 52, at 43 124 and 115; 131 x 97 px, 40 emitters, at 9 and 14 23.5 and
   // 23.6, 31.6 and 30.7. Four from 8 on where a frame has more emitters than are staged at once, whose staging four tiles
   // share: frames of 256 x 256 px, 430 emitters, at 4 33.8 us with two and 34.8 with four, at 9 57 and 55, at 87 464 and
   // 429; with 160 emitters the two are within 2 % of each other from 20 to 100 CTAs an SM. Neither where the tile would
   // be wider than the frame (900 frames of 64 x 64 px in tiles of 32: 99 us with two, 112 with four, half of them empty).
   const int th = kTileH[tile];
   const auto tilesOf = [&](int tw) { return (ga.st.width + tw - 1) / tw * ((ga.st.height + th - 1) / th); };
   int sub = 1;
   for (int q = persistent ? 1 : 4; q > 1 && sub == 1; q /= 2)
      if (static_cast<uint32_t>((q - 1) * kTileW[tile]) < ga.st.width &&
          (q == 2 || nEm >= static_cast<uint64_t>(kGChunk) * nFrames) &&
          static_cast<uint64_t>(tilesOf(q * kTileW[tile])) * nFrames >=
             static_cast<uint64_t>(q == 4 ? 8 : 12) * ctx->smCount)
         sub = q;
   const int tw = kTileW[tile] * sub;
   GatherFn fn = nullptr;
   if (persistent)
      fn = cam ? GatherTile<true, true, 1>(tile) : GatherTile<false, true, 1>(tile);
   else if (sub == 4)
      fn = cam ? GatherTile<true, false, 4>(tile) : GatherTile<false, false, 4>(tile);
   else if (sub == 2)
      fn = cam ? GatherTile<true, false, 2>(tile) : GatherTile<false, false, 2>(tile);
   else
      fn = cam ? GatherTile<true, false, 1>(tile) : GatherTile<false, false, 1>(tile);
   if (persistent)
   {
      int rc = LaunchFrameOrder(ctx, frames, nFrames, orderBuf);
      if (rc != ISCU_OK)
         return rc;
      ga.order = orderBuf;
      ga.counter = orderBuf + ((nFrames + 3) & ~3u);
      int perSm = 0;
      ISCU_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, kGT, 0));
      const uint32_t grid = std::min<uint32_t>(static_cast<uint32_t>(std::max(1, perSm) * ctx->smCount),
                                               tilesOf(tw) * nFrames);
      fn<<<grid, kGT, 0, ctx->stream>>>(ga);
   }
   else
   {
      ga.order = nullptr;
      ga.counter = nullptr;
      const dim3 grid((ga.st.width + tw - 1) / tw, (ga.st.height + th - 1) / th, nFrames);
      fn<<<grid, kGT, 0, ctx->stream>>>(ga);
   }
   ISCU_CK_LAUNCH(ctx, "GatherTilesKernel");
   if (marks)
      ISCU_CK(cudaEventRecord(marks[3], ctx->stream));
   return ISCU_OK;
}

} // namespace iscu

// The per-pixel camera noise chain (ApplyNoiseChain, adapter/inSiliScope/Simulation/SMLMNoise.cpp:142-216) as a
// device function, shared by the kernels that end in camera frames (splat_noise.cu, widefield.cu). Every translation
// unit that includes it is compiled with --fmad=false, so its float64 arithmetic rounds as the reference's
// -ffp-contract=off build does.
#pragma once

#include "counter_rng.cuh"
#include "iscu_internal.h"

namespace iscu {

// A pixel's camera values: its maps where set, else the camera scalars (offset 0).
struct PixelCamera
{
   double qe, dark, cic, emGain, maxAdu, readNoise, gain, offset;
   int emccd;
};

// The float64 chain of sensor pixel `pix` of frame `frame`, its roundings and decisions taken from the float32 normal
// where that is sure. Out of line: NoisePixel comes here where its float32 decisions are in doubt. pos: the words of the
// stream that the Poisson draw of `electrons` took, where that draw is sure (kNoDraw: it is not); the chain goes on from
// there, since in a small image the few pixels that come here are the last to end.
constexpr uint32_t kNoDraw = 0xFFFFFFFFu;
static __device__ __noinline__ uint32_t NoisePixelExact(float photonValue, uint32_t pix, uint32_t seed, uint32_t frame,
                                                        PixelCamera cam, float electrons, uint32_t pos)
{
   CounterRng u(seed, frame);
   u.Pixel(pix);
   const double pv = static_cast<double>(photonValue);
   const double photons = pv > 0.0 ? pv : 0.0;   // std::max(0.0, v)
   if (cam.emccd)
   {
      double ne = electrons;
      if (pos == kNoDraw)
         ne = CounterPoisson(photons * cam.qe + cam.dark + cam.cic, u);
      else
      {
         u.ctr = pos >> 2;
         for (uint32_t i = 0; i < (pos & 3u); ++i)
            u.Uniform();
      }
      const double readE = cam.readNoise / cam.emGain, gain = cam.gain, offset = cam.offset;
      // The register's Gamma with float32 decisions (GammaSure), else CounterGamma from the saved stream; then the
      // rounding (before the clamp) from the float32 read-noise normal when no boundary is within the bound of both
      // float32 errors, else the Gamma (if it was not exact) and the normal again in float64 from the saved stream.
      const CounterRng saved = u;
      double out = 0.0, outErr = 0.0;
      bool exact = true;
      if (ne > 0.0)
      {
         exact = !GammaSure(ne, u, out, outErr);
         if (exact)
         {
            u = saved;
            out = CounterGamma(ne, u);
            outErr = 0.0;
         }
      }
      GaussDraw d = DrawGauss(u);
      const double af = offset + (out + readE * static_cast<double>(d.gf)) / gain;
      const double m = (outErr + fabs(readE) * kGaussFastErr) / fabs(gain) + 1e-9 * (1.0 + fabs(af));
      double adu;
      if (!RoundsSurely(af, m, adu))
      {
         if (!exact)
         {
            u = saved;
            out = CounterGamma(ne, u);
            d = DrawGauss(u);
         }
         adu = floor(offset + (out + readE * GaussExact(d)) / gain + 0.5);
      }
      return static_cast<uint16_t>(adu < 0.0 ? 0.0 : (adu > cam.maxAdu ? cam.maxAdu : adu));
   }
   const double ne = CounterPoisson(photons * cam.qe + cam.dark, u);
   const double readNoise = cam.readNoise, gain = cam.gain, offset = cam.offset;
   const GaussDraw d = DrawGauss(u);
   // The ADU from the float32 normal when it is sure: inside (0, 65535) and no rounding boundary within
   // |readNoise / gain| kGaussFastErr of it (the float64 operations' own rounding, ~1e-13, inside the 1e-9 term).
   const double af = offset + (ne + readNoise * static_cast<double>(d.gf)) / gain;
   const double m = fabs(readNoise / gain) * kGaussFastErr + 1e-9 * (1.0 + fabs(af));
   double r;
   if (af > m && af < 65535.0 - m && RoundsSurely(af, m, r))
      return static_cast<uint16_t>(r);
   const double g = GaussExact(d);
   double adu = offset + (ne + readNoise * g) / gain;
   adu = adu < 0.0 ? 0.0 : (adu > 65535.0 ? 65535.0 : adu);
   return static_cast<uint16_t>(floor(adu + 0.5));
}

// ------------------------------------------------------------------------------------------------ the fast chain
// NoisePixel is the same chain with every decision taken in float32 where it is sure, so the ADU are the float64
// chain's bits. What bounds the chain is the issue and integer rate of the Knuth loop's hashes (its trip count is the
// reference's by definition), so the loop carries nothing in float64: 28 instructions a hash against 44, one word of
// the stream selected instead of queued, no float64 exponential, logarithm, quotient or conversion (a conversion
// issues at a quarter of the float64 rate). Error bounds, each stated where it is used, are at least 1.4 times what the
// operations' documented bounds add up to; in doubt (about one pixel in 10^4) the float64 chain decides. Measured: the
// sCMOS noise of 16 frames of 512 x 512 px 159 -> 94 us a call, the EMCCD noise of 64 such frames 0.66 -> 0.35 ms.

__device__ __forceinline__ float Ex2Approx(float x)
{
   float r;
   asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
   return r;
}
__device__ __forceinline__ float Lg2Approx(float x)
{
   float r;
   asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
   return r;
}
__device__ __forceinline__ float RsqrtApprox(float x)
{
   float r;
   asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
   return r;
}
__device__ __forceinline__ float RcpApprox(float x)
{
   float r;
   asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
   return r;
}

// UniformOf's value in float32, exact: 1 + (x >> 9) 2^-23 from the bits, less 1 - 2^-24 (a 24-bit result).
__device__ __forceinline__ float UniformF(uint32_t x)
{
   return __uint_as_float(__funnelshift_r(x, 0x7fu, 9)) - 0.999999940395355224609375f;
}

// The product of the four words' uniforms, two lanes at a time (each rounds as the one-lane instruction).
__device__ __forceinline__ float UniformProduct(const uint32_t (&w)[4])
{
   const uint64_t c = 0xBF7FFFFFBF7FFFFFull;   // -(1 - 2^-24), twice
   uint64_t x, y;
   asm("{.reg .b64 t; mov.b64 t, {%1, %2}; add.rn.f32x2 %0, t, %3;}"
       : "=l"(x)
       : "r"(__funnelshift_r(w[0], 0x7fu, 9)), "r"(__funnelshift_r(w[1], 0x7fu, 9)), "l"(c));
   asm("{.reg .b64 t; mov.b64 t, {%1, %2}; add.rn.f32x2 %0, t, %3;}"
       : "=l"(y)
       : "r"(__funnelshift_r(w[2], 0x7fu, 9)), "r"(__funnelshift_r(w[3], 0x7fu, 9)), "l"(c));
   uint64_t z;
   asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(z) : "l"(x), "l"(y));
   return __uint_as_float(static_cast<uint32_t>(z)) * __uint_as_float(static_cast<uint32_t>(z >> 32));
}

// A pixel's hashes by counter. Before its first exclusive-or the permutation's words d, a and b are linear in the
// counter: a step adds a constant to each.
struct PixelHashes
{
   uint32_t a0, b0, c0, sb;   // the words' constant parts, and b's step per counter

   __device__ __forceinline__ PixelHashes(uint32_t seed, uint32_t frame, uint32_t pix)
   {
      const uint32_t mul = 1664525u, inc = 1013904223u;
      const uint32_t bf = frame * mul + inc;
      c0 = pix * mul + inc;
      a0 = seed * mul + inc + bf * inc;   // a at counter 0, after a += b d
      b0 = bf + c0 * a0;                  // b at counter 0, after b += c a
      sb = c0 * (bf * mul);
   }
   // The counter's words from the linear state (d, a, b at that counter).
   __device__ __forceinline__ void Finish(uint32_t d, uint32_t a, uint32_t b, uint32_t (&w)[4]) const
   {
      uint32_t c = c0 + a * b;
      d += b * c;
      a ^= a >> 16;
      b ^= b >> 16;
      c ^= c >> 16;
      d ^= d >> 16;
      a += b * d;
      b += c * a;
      c += a * b;
      d += b * c;
      w[0] = a;
      w[1] = b;
      w[2] = c;
      w[3] = d;
   }
   __device__ __forceinline__ void At(uint32_t frame, uint32_t ctr, uint32_t (&w)[4]) const
   {
      const uint32_t mul = 1664525u, inc = 1013904223u;
      Finish(inc + ctr * mul, a0 + ctr * ((frame * mul + inc) * mul), b0 + ctr * sb, w);
   }
   // Words pos .. pos + 4 of the stream: always within two hashes.
   __device__ __forceinline__ void Words(uint32_t frame, uint32_t pos, uint32_t (&w)[5]) const
   {
      uint32_t lo[4], hi[4];
      At(frame, pos >> 2, lo);
      At(frame, (pos >> 2) + 1, hi);
      const bool odd = pos & 1, two = pos & 2;
      const uint32_t x[7] = {odd ? lo[1] : lo[0], odd ? lo[2] : lo[1], odd ? lo[3] : lo[2], odd ? hi[0] : lo[3],
                             odd ? hi[1] : hi[0], odd ? hi[2] : hi[1], odd ? hi[3] : hi[2]};
#pragma unroll
      for (int i = 0; i < 5; ++i)
         w[i] = two ? x[i + 2] : x[i];
   }
};

// The stream's normal of the uniform words (radius first, angle second) and a bound of its distance from the float64
// formula's value: lg2.approx is within 2^-22 of log2 on (0.5, 2) and 2^-22 relative elsewhere, so x = -2 ln u1 is
// within 3.4e-7 near 1 and the radius within 3.4e-7 / r; elsewhere the radius and the cosine (__cosf: 2^-21.19 on
// [-pi, pi], its argument rounded) add at most 1.3e-6 r, r <= 5.8. Near u1 = 1 the radius can be NaN; so are its sums.
struct NormalF
{
   float g, e;
};
__device__ __forceinline__ NormalF DrawNormalF(uint32_t w1, uint32_t w2)
{
   const float x = -1.38629436f * Lg2Approx(UniformF(w1));
   const float ir = RsqrtApprox(x), r = x * ir;
   const float h = UniformF(w2) - 0.5f;   // exact; cos(2 pi u2) = -cos(2 pi (u2 - 1/2))
   return {-(r * __cosf(6.28318531f * h)), fmaf(8e-7f, ir, 1.6e-5f)};
}

// floor(v + 0.5) of a v within m of vf (|vf| < 2^22): false when a rounding boundary is within m (or NaN).
__device__ __forceinline__ bool RoundsSurelyF(float vf, float m, float& out)
{
   const float t = vf + 0.5f;
   const float f = floorf(t);
   out = f;
   return fabsf((t - f) - 0.5f) < 0.5f - m;
}

// Pixel i (of the frame; the sensor pixel is i + pixel_base) of a frame whose stream u is keyed by (seed, frame):
// sCMOS or EMCCD, per-pixel maps where set, else the camera scalars (offset 0).
__device__ __forceinline__ uint16_t NoisePixel(float photonValue, uint32_t i, const CameraView& cam,
                                               const StaticView& st, const CounterRng& u)
{
   const uint32_t seed = u.seed, frame = u.frame, pix = i + st.pixelBase;
   const float readF = st.readNoise ? st.readNoise[i] : cam.readF, gainF = st.gain ? st.gain[i] : cam.gainF,
               offF = st.offset ? st.offset[i] : 0.f;
   // lambda within 3 roundings (1.8e-7 relative) of the float64 mean: its terms are not negative. (A camera without
   // float32 bounds: NaN, which no float32 branch below takes -- the Knuth loop for nothing had cost it a third.)
   const float lf = cam.fast ? fmaxf(photonValue, 0.f) * cam.qeF + cam.addF : __int_as_float(0x7fc00000);
   bool ok = cam.fast != 0;
   float ne = 0.f;
   uint32_t pos = 0;          // words of the stream consumed
   uint32_t g1 = 0, g2 = 0;   // the read noise's words
   const PixelHashes H(seed, frame, pix);
   if (lf <= 59.9999f && lf >= 1e-6f)
   {
      // Knuth. L within 1.2e-5 + 4e-6 (lambda's error, the argument's rounding, ex2.approx) of exp(-mean); the
      // product within 2^-24 per factor of the float64 one, 256 factors at most here (1.6e-5), and two more for the
      // block's start below: the margin is 6e-5.
      const float L = Ex2Approx(lf * -1.44269504f), hi = L * 1.00006f, lo = L * 0.99994f;
      const uint32_t mul = 1664525u, inc = 1013904223u, sa = (frame * mul + inc) * mul;
      uint32_t d = inc, a = H.a0, b = H.b0, w[4];
      float p4 = 1.f, prod;
      do
      {
         H.Finish(d, a, b, w);
         prod = UniformProduct(w);
         p4 *= prod;
         d += mul;
         a += sa;
         b += H.sb;
      } while (p4 > hi);   // (each factor is below 1)
      // d is linear in the counter: the blocks drawn, from mul's inverse mod 2^32; the product before the last block
      const uint32_t blocks = (d - inc) * 0xFEE058C5u;
      const float p = p4 * RcpApprox(prod), u0 = UniformF(w[0]), u2 = UniformF(w[2]), p2 = u0 * UniformF(w[1]);
      // the block's first product at or below L: its factor ends the draw
      const float q1 = p * u0, q2 = p * p2, q3 = q2 * u2;
      const bool o1 = q1 > hi, o2 = o1 && q2 > hi, o3 = o2 && q3 > hi;
      const float last = o3 ? p4 : (o2 ? q3 : (o1 ? q2 : q1));
      ok = ok && last < lo && blocks <= 64u && p4 > 1e-36f;   // (a subnormal product has lost its places)
      const int n = o3 ? 3 : (o2 ? 2 : (o1 ? 1 : 0));
      pos = 4 * (blocks - 1) + n;
      ne = static_cast<float>(pos);
      ++pos;
      if (!cam.emccd)
      {
         uint32_t x[4];
         H.Finish(d, a, b, x);
         g1 = o3 ? x[0] : (o2 ? w[3] : (o1 ? w[2] : w[1]));
         g2 = o3 ? x[1] : (o2 ? x[0] : (o1 ? w[3] : w[2]));
      }
   }
   else if (ok)
   {
      uint32_t w[4];
      H.At(frame, 0, w);
      if (lf > 60.0001f && lf < 1e6f)
      {
         // the rounded normal floor(l + sqrt(l) g + 0.5), at least 1 where it is taken here
         pos = 2;
         const NormalF z = DrawNormalF(w[0], w[1]);
         const float s = lf * RsqrtApprox(lf);
         if (!(RoundsSurelyF(fmaf(s, z.g, lf), fmaf(lf, 1.2e-6f, s * z.e), ne) && ne >= 1.f))
         {
            const double ld = static_cast<double>(fmaxf(photonValue, 0.f)) * cam.qe + cam.dark;
            const double l = cam.emccd ? ld + cam.cic : ld;
            double r;
            // the mean in float64, the deviation in float32 (s within 2.8e-7)
            const float dev = s * z.g;
            if (!RoundsSurely(l + static_cast<double>(dev), fmaf(s, z.e, 5e-7f * fabsf(dev)) + 1e-9 * l, r) ||
                !(r >= 1.0))
               r = fmax(0.0, floor(l + sqrt(l) * GaussExact({UniformOf(w[0]), UniformOf(w[1]), 0.f}) + 0.5));
            ne = static_cast<float>(r);
            ok = ok && r < 16777216.0;
         }
         g1 = w[2];
         g2 = w[3];
      }
      else
      {
         // no photons and no dark current: nothing drawn, no electrons
         ok = ok && !(photonValue > 0.f) && (cam.emccd ? cam.dark + cam.cic : cam.dark) == 0.0;
         g1 = w[0];
         g2 = w[1];
      }
   }
   const uint32_t drawn = ok ? pos : kNoDraw;
   const float ig = RcpApprox(gainF), aig = fabsf(ig);
   if (cam.emccd)
   {
      // The register's Gamma (CounterGamma's steps and draws): x within e; t = 1 + c x within dt; v = t^3 within dv;
      // the squeeze and the logarithmic test each within a bound of their terms' errors. From kBright electrons on
      // |c x| <= 0.086: t is positive, and the logarithmic test's right side is its series (bright, below).
      constexpr float kBright = 512.f;
      const bool bright = ne >= kBright;
      const float d = ne - 0.333333333f, c = RsqrtApprox(9.f * d);
      float out = 0.f, outErr = 0.f, x = 0.f, e = 0.f;
      uint32_t w[5];
      if (!(ne > 0.f))
      {
         H.Words(frame, pos, w);
         g1 = w[0];
         g2 = w[1];
      }
      else if (ok)
      {
         ok = false;
         for (int it = 0; it < 16; ++it)
         {
            H.Words(frame, pos, w);
            g1 = w[3];   // the read noise's words, if this draw is taken
            g2 = w[4];
            const NormalF z = DrawNormalF(w[0], w[1]);
            x = z.g;
            e = z.e;
            const float cx = c * x, t = 1.f + cx, dt = fmaf(c, e, fmaf(5e-7f, fabsf(cx), 1.3e-7f));
            const bool negative = !bright && t + dt <= 0.f;   // drawn again before its third uniform
            pos += negative ? 2 : 3;
            if (negative)
               continue;
            const float uw = UniformF(w[2]), x2 = x * x, ax = fabsf(x) + e, ax3 = ax * ax * ax;
            const float s = fmaf(-0.0331f * x2, x2, 1.f);
            const float ds = fmaf(0.14f * ax3, e, fmaf(4e-8f * x2, x2, 4e-7f));
            const float tt = t + dt, v = t * t * t, dv = fmaf(3.f * tt * tt, dt, 2.5e-7f * v);
            out = d * v;
            outErr = fmaf(d, dv, 3.6e-7f * out);
            ok = (bright || t > dt) && uw < s - ds;
            if (ok || !(bright || t > dt) || !(uw >= s + ds))
               break;
            const float lw = 0.693147181f * Lg2Approx(uw), alw = fabsf(lw);
            float rhs, m;
            if (bright)
            {
               // x^2 / 2 + d (1 - v + log v) = 3 d (y^4 / -4 + y^5 / 5 - ...) for y = c x, d = 1 / (9 c^2): the terms up
               // to y^2 have cancelled; what is left out is below 1e-3 of it
               const float c2 = c * c;
               rhs = -(x2 * x2) * (c2 * 0.0833333333f) * fmaf(cx, fmaf(cx, 0.666666667f, -0.8f), 1.f);
               m = fmaf(3e-3f, fabsf(rhs), fmaf(0.4f * ax3 * c2, e, fmaf(1e-6f, alw, 1e-6f)));
            }
            else
            {
               const float lv = 0.693147181f * Lg2Approx(v), iv = RcpApprox(v);
               rhs = fmaf(0.5f, x2, d * (1.f - v + lv));
               m = fmaf(1e-6f, alw, 1e-6f) + fmaf(ax, e, 4e-7f * x2) +
                   d * (fmaf(fabsf(iv - 1.f) + dv * iv, dv, fmaf(1e-6f, fabsf(lv), 1e-6f) + 4e-7f * v));
            }
            ok = lw < rhs - m;
            if (ok || !(lw > rhs + m))
               break;
         }
      }
      if (ok)
      {
         const NormalF z = DrawNormalF(g1, g2);
         const float rn = readF * cam.invEmF, rz = rn * z.g;
         if (bright)
         {
            // float32's own rounding of the Gamma leaves an ADU in doubt for one pixel in 100 at 5,000 electrons (in
            // nearly every warp at 20,000): from the normal on in float64, the square root and the quotient by a Newton
            // step each, so that the normals' bounds are all of the error. EMCCD noise of 16 frames of 512 x 512 px at
            // 300, 1,000, 6,000 and 19,000 electrons 94, 91, 105 and 122 us, and 86, 101, 153 and 242 all in float32: the
            // line is between the first two.
            const double dd = static_cast<double>(ne) - 1.0 / 3.0, c0 = static_cast<double>(c);
            const double cd = c0 * fma(-4.5 * dd * c0, c0, 1.5), td = fma(cd, static_cast<double>(x), 1.0);
            const double gd = st.gain ? static_cast<double>(gainF) : cam.gain, i0 = static_cast<double>(ig);
            const double igd = i0 * fma(-gd, i0, 2.0);
            const double sum = (dd * (td * td * td) + static_cast<double>(rz)) * igd, off = static_cast<double>(offF);
            const double af = off + sum, top = cam.maxAdu;
            // (3 t^2 <= 3.54; 3 d c = sqrt(d))
            const float em = aig * (fmaf(3.9f * d * c, e, fmaf(fabsf(rn), z.e, 4e-7f * fabsf(rz))));
            const double m = static_cast<double>(em) + 1e-9 * (1.0 + fabs(sum) + fabs(off));
            double r;
            if (af > top + m + 0.5)
               return static_cast<uint16_t>(top);
            if (RoundsSurely(af, m, r))
               return static_cast<uint16_t>(r < 0.0 ? 0.0 : (r > top ? top : r));
         }
         else
         {
            const float af = fmaf(out + rz, ig, offF);
            const float m = aig * (outErr + fabsf(rn) * z.e) + 1.2e-6f * fmaf(out + fabsf(rz), aig, fabsf(offF));
            float r;
            if (RoundsSurelyF(af, m, r))   // (m passes 0.5 well before af leaves the float integers)
            {
               const float top = static_cast<float>(cam.maxAdu);
               return static_cast<uint16_t>(fminf(fmaxf(r, 0.f), top));
            }
         }
      }
   }
   else if (ok)
   {
      // the ADU inside (0, 65535): the float32 value within its terms' roundings (eight at most) and the normal's bound
      const NormalF z = DrawNormalF(g1, g2);
      const float rz = readF * z.g, af = fmaf(ne + rz, ig, offF);
      const float m = fabsf(readF * ig) * z.e + 1.2e-6f * fmaf(ne + fabsf(rz), aig, fabsf(offF));
      float r;
      if (RoundsSurelyF(af, m, r) && af > m && af < 65535.f - m)
         return static_cast<uint16_t>(r);
      // in float64 from the same normal, then from the float64 one
      const double rd = st.readNoise ? static_cast<double>(readF) : cam.readNoise,
                   gd = st.gain ? static_cast<double>(gainF) : cam.gain, od = offF, nd = ne;
      double adu = od + (nd + rd * static_cast<double>(z.g)) / gd, rr;
      const double md = fabs(rd / gd) * static_cast<double>(z.e) + 1e-9 * (1.0 + fabs(adu));
      if (adu > md && adu < 65535.0 - md && RoundsSurely(adu, md, rr))
         return static_cast<uint16_t>(rr);
      adu = od + (nd + rd * GaussExact({UniformOf(g1), UniformOf(g2), 0.f})) / gd;
      adu = adu < 0.0 ? 0.0 : (adu > 65535.0 ? 65535.0 : adu);
      return static_cast<uint16_t>(floor(adu + 0.5));
   }
   return static_cast<uint16_t>(NoisePixelExact(
      photonValue, pix, seed, frame,
      {cam.qe, cam.dark, cam.cic, cam.emGain, cam.maxAdu, st.readNoise ? static_cast<double>(readF) : cam.readNoise,
       st.gain ? static_cast<double>(gainF) : cam.gain, static_cast<double>(offF), cam.emccd},
      ne, drawn));
}

} // namespace iscu

// tuned_core.cuh -- per-sample body of the TUNED geometry, shared by the
// single-detector forward (fwd_tuned.cu), the batched multi-detector forward
// (fwd_batched.cu), the adjoint (adjoint_kernels.cuh) and the nearest-lookup
// PLAIN and FP64 forms (fwd_exact.cu), which take the pairs from it and the
// phasor exp(2i chi) to their own precision.
//
// A sample's FP64 set-up -- its disc plan, boresight frame and psi phasors
// (SamplePlan, make_plan) -- is built beforehand by a plan kernel with one
// thread per sample, by one lane per sample of the block's first warp (short
// launches), or by the warp itself; the warp keeps it in its shared memory
// (WarpSmem::plan), so the pair loop's registers hold only the pair geometry.
//
// For one sample, a warp evaluates the HEALPix query_disc rings, one ring per
// lane (place_ring), rounds per-ring small-offset constants to FP32 once
// (RingC, 48 B in shared memory), and strides the disc pairs across lanes; the
// forward takes two neighbouring pixels of a ring per lane and iteration, with
// the geometry of both in packed FP32 instructions, which halves the issue
// slots and the reads of the ring constants (100,000 samples of nside 1024 and
// 3 degrees: 5.2 -> 4.3 ms).  Per pair, FP32 only:
// longitude offset from a per-ring anchor pixel, cancellation-free
// boresight-frame components, the beam grid's polar-cap indices and
// exp(2i chi) as a product of unit phasors.  Any of the three floor decisions
// lying within the margin of an integer, and any pair within 2e-6 rad of the
// boresight, is queued and decided in FP64: by the small-offset form with one
// sine and cosine and one arctangent (quick_pair), or, where that too is close
// to an edge or to the boresight, with the reference's FP64 chain (hpx.cuh
// pair_beam_pixel), so every pair lands on the chain's beam pixel
// (pisco_debug_decisions compares them).
//
// The queue outlives the sample: each entry names a per-warp slot holding its
// sample's FP64 frame and output, and the warp redoes 32 entries at a time,
// whichever samples they came from (a sample queues about four pairs in ten
// thousand, so a per-sample drain would run the FP64 code with a few lanes
// active); what the warps of a block have left at the end the block redoes
// together (flush_block).  The re-evaluated contributions of a sample are added in
// queue order, one lane per sample, into an FP64 sum, and its TOD is written
// (main-pass total + that sum) when its last entry is done: the result does
// not depend on where the drains cut the queue, hence not on the other
// samples of the warp.
//
// Disc edge: per ring, the half width of the disc and the anchor are formed
// in FP32 from split constants (two floats where one loses digits); an edge
// within the error bound of a pixel boundary, and any ring near a pole or a
// full circle, is recomputed with HEALPix's FP64 formula (disc_ring), so the
// disc is HEALPix query_disc's exactly.  With the ring set-up in FP64 it took
// a third of the time at 960 pairs per sample.
//
// Geometry, with the pixel at ring height z (s = sqrt(1 - z^2)), longitude
// offset D from the boresight (z0, s0) and h = 1 - cos D:
//   east  u = s sin D                   north v = sin(dec - dec0) + s z0 h
//   1 - cos(rho) = (1 - cos(dec - dec0)) + s s0 h
//   toward the boresight at the pixel: (s0 sin D, sin(dec0 - dec) + s0 z h)
//   r = sqrt(3) nside_b sqrt(1 - cos rho),  sigma = pi - alpha - psi,
//   alpha = atan2(u, v),  exp(2i chi) = exp(2i beta) exp(2i alpha) exp(2i psi)
// (sphtrigo.cpp:27-54 rewritten in small-offset form).
//
// The per-pair work is handed to an Action (Gather below, Scatter in
// adjoint.cu):
//   kSums                     true: per-sample sums, TOD written per sample
//   void reset(), total(a, b) main-pass sums (kSums)
//   P fetch(int pix)          per-pixel data the action needs (Gather: the sky)
//   void pair(int pix, P fetched, const F8& beam, int bp, float c2, float s2)
//   void pair2(...)           in place of pair with the nearest lookup: two
//                             neighbouring pixels at once
//   void pair_all(...)        in place of pair: every lane calls, with or
//                             without a pair of its own (lanes share the
//                             atomics' sectors)
//   void pair64(...)          optional: the phasor in FP64 or, with a member
//                             type TwoFloat, in two-float arithmetic
//   void stash(Pend&)         per-sample data a queued pair needs later
//   void deferred(const Pend&, int pix, const F8& beam, int bp, float c2, float s2,
//                 float& ta, float& tb)      a re-evaluated pair
//   kStencil                  true: with the bilinear lookup the action gets
//                             the stencil instead of the interpolated value:
//   void pair_stencil(int pix, P fetched, const int px[4], const float w[4], c2, s2)
//   void deferred_stencil(const Pend&, int pix, const int px[4], const float w[4], c2, s2)
// (c2, s2 = cos 2chi, sin 2chi; `beam` is the beam pixel's value, bp its
// index, with the nearest lookup, and the interpolated value, bp = -1, with
// the bilinear one).
// Optional, detected at compile time (the forward and adjoint actions leave
// them out, so they cost nothing there):
//   void outside(int pix, int bp)                a disc pair whose beam pixel
//   void outside_deferred(const Pend&, int pix, int bp)   lies beyond the
//                             stored map (bp; -1: no bilinear stencil pixel in it)
#pragma once

#include <math_constants.h>

#include <type_traits>

#include "hpx.cuh"
#include "internal.h"

// Warps per block of the adjoint's and the diagnostics' kernels, and the
// minimum number of resident blocks per SM requested from the compiler (which
// caps their registers at 65536 / (32 x warps x blocks)); the adjoint's
// planned nearest-lookup instances take 2, 3 or 4 (adjoint_kernels.cuh
// adj_warps_per_sm).
#ifndef PISCO_TUNED_WARPS
#define PISCO_TUNED_WARPS 8
#endif
#ifndef PISCO_TUNED_MINB
#define PISCO_TUNED_MINB 2
#endif

namespace pisco {
namespace tuned {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kQCap = 64;

// Does the action want to hear of disc pairs outside the stored beam map?
template <class A, class = void>
struct HasOutside : std::false_type {};
template <class A>
struct HasOutside<A, std::void_t<decltype(&A::outside)>> : std::true_type {};
// Does the action take the pair's phasor in FP64 (the PLAIN and FP64 forms,
// fwd_exact.cu)?
template <class A, class = void>
struct IsExact : std::false_type {};
template <class A>
struct IsExact<A, std::void_t<decltype(&A::pair64)>> : std::true_type {};
// ... in two-float arithmetic (the PLAIN form, whose products take it rounded
// to FP32)?
template <class A, class = void>
struct IsTwoFloat : std::false_type {};
template <class A>
struct IsTwoFloat<A, std::void_t<typename A::TwoFloat>> : std::true_type {};
// Does the action take the pairs of a warp together (every lane calls
// pair_all, with beam pixel -1 where it has no pair)?
template <class A, class = void>
struct HasPairAll : std::false_type {};
template <class A>
struct HasPairAll<A, std::void_t<decltype(&A::pair_all)>> : std::true_type {};
// Does the action take two pixels per lane?
template <class A, class = void>
struct HasPair2 : std::false_type {};
template <class A>
struct HasPair2<A, std::void_t<decltype(&A::pair2)>> : std::true_type {};
// Decisions whose FP32 value lies within kMarginRel * (r + 2) of an integer (r:
// the pair's ring position; the values are at most r + 1) are redone in FP64
// (about 20 FP32 ulps).  The observed worst case
// over a workload is measured by pisco_tuned_calibrate and must stay well
// below this bound.
constexpr float kMarginRel = 1.2e-6f;
// A ring batch whose longitude offsets all stay within this (radians) takes
// the short series of sin and 1 - cos (short_sin_versin).
constexpr float kShortOffset = 0.125f;
// Pairs with 1 - cos(rho) below this take the reference's degenerate branch
// (rho <= 1e-6, sphtrigo.cpp:40-48) and are done in FP64.
constexpr float kTinyQ = 4.0e-12f;

// One disc ring of the current batch: FP32 offset constants and the pixel
// range, 48 bytes, read with three 16-byte loads.  A broadcast shared-memory
// read costs the L1 pipe a cycle per word all the same, and that pipe is the
// busiest unit of the pair loop, so what a pair can form from the sample's
// own constants (Frame) is not stored per ring.
struct alignas(16) RingC {
    float dc, dphi;  // anchor offset, pixel spacing
    float Ki, s;     // R^2 (1 - cos(dec - dec0)); sin of the colatitude
    float Wz, Di;    // s0 z, sin(dec - dec0)
    int j0;          // ring index of flattened pair t: (j0 + t) mod nr; with two
                     // pixels per lane (j0 + 2 t) mod nr, even
    int kc;          // bits of 1.5 2^23 less the anchor's ring index
    int nr, start;   // ring pixels, first pixel
    int ends;        // ring indices of the range's ends, first | last << 16
    int pad;
};

// The sample's constants of the pair loop: z0, s0, R^2 s0, sin and cos of psi
// (times their common factor).
struct Frame {
    float z0, s0, R2s0, sps, cps;
};

// Samples in flight per warp (a sample keeps its slot until its queued
// pairs are done).
constexpr int kPend = 16;

// A sample whose queued pairs may not all be re-evaluated yet.
struct alignas(16) Pend {
    double ra, dec, psi;     // as given (psi = -pa): the chain's
    double z0, s0, phi;      // the frame in FP64, as the plan has it
    double spsi, cpsi;
    double main_a, main_b;   // main-pass totals
    double fb_a, fb_b;       // re-evaluated pairs, summed in queue order
    const F8* beam;
    void* out_a;
    void* out_b;
    long long idx;           // output index
    float ga, gb;            // adjoint weights
    int nside_beam, npix_beam;
    int left;                // queued entries not yet re-evaluated
    int open;                // main pass still running
    int f64;                 // output type
    int plain;               // the frame does not carry the chain's accuracy
};

// A sample's per-sample geometry: its disc (the rings it touches and the
// edge formula's constants), the boresight frame and the psi phasors.  Built
// by make_plan, either inside the pair kernel (one warp per sample, every
// lane redundantly) or beforehand by plan_kernel with one thread per sample:
// it is FP64 work (some 180 FP64 instructions), which GB300 runs
// at a small fraction of its FP32 rate.  96 bytes.
struct alignas(16) SamplePlan {
    // disc, for disc_ring's exact formula: cos(theta), 1 / sin(theta), longitude
    double z0, xa, phi;
    double spsi, cpsi;        // sin and cos of psi, negated with the frame's flip
    float phi_hi, phi_lo;     // frame: longitude reduced mod 2 pi, latitude,
    float dec_hi, dec_lo;     //   each the sum of two FP32 values
    float z0f, s0f;           // frame: sin and |cos| of the latitude
    float sps, cps;           // the same of psi times a common factor (psi_phasor)
    int ring_lo, ring_hi;     // rings on the edge formula
    int full_lo, full_hi;     // rings touched
    int flags;                // kPlanBad: non-finite pointing; kPlanAllSky; kPlanExact
};
constexpr int kPlanBad = 1;
constexpr int kPlanAllSky = 2;
constexpr int kPlanExact = 4;  // the frame is not the disc's (an ulp from a pole): exact edges

// Per-warp shared state: one ring batch, the samples in flight, the FP64
// re-evaluation queue (sky pixel, slot) and the current sample's plan (read
// from here where needed rather than held in registers across the pair loop).
template <class Real>
struct WarpState {
    SamplePlan plan;
    RingC r[32];
    Pend p[kPend];
    int q[kQCap];
    unsigned char qs[kQCap];
    Real ta[32], tb[32];  // re-evaluated pairs of a drain
};
using WarpSmem = WarpState<float>;

// One disc ring of the current batch in FP64, and the sample's frame: what the
// phasor of an IsExact action is formed from.
struct RingD {
    double dc, dphi;      // anchor offset, pixel spacing
    double s, Zs, Wz, Di; // s, s z0, s0 z, sin(dec - dec0)
};
struct ExactSmem : WarpState<double> {
    RingD rd[32];
    double z0, s0, c2p, s2p;  // sin and |cos| of the latitude, cos and sin of 2 psi
};

// A value as the unevaluated sum of two FP32 values, h the sum rounded (2^-48
// relative), by Dekker's and Knuth's exact sums and products (T. J. Dekker,
// Numer. Math. 18, 224 (1971)).  A product takes 7 FP32 instructions, a sum 8
// to 11, where one FP64 instruction takes as long as 64 FP32 ones.
struct FF {
    float h, l;
};
__device__ __forceinline__ FF ff(double d)
{
    const float h = (float)d;
    return FF{h, (float)(d - (double)h)};
}
__device__ __forceinline__ FF ff_quick(float a, float b)  // a + b, |a| >= |b|
{
    const float h = __fadd_rn(a, b);
    return FF{h, __fsub_rn(b, __fsub_rn(h, a))};
}
__device__ __forceinline__ FF ff_sum(float a, float b)  // a + b, exactly
{
    const float h = __fadd_rn(a, b), t = __fsub_rn(h, a);
    return FF{h, __fadd_rn(__fsub_rn(a, __fsub_rn(h, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ FF operator+(FF a, FF b)
{
    const FF s = ff_sum(a.h, b.h), t = ff_sum(a.l, b.l);
    const FF u = ff_quick(s.h, __fadd_rn(s.l, t.h));
    return ff_quick(u.h, __fadd_rn(u.l, t.l));
}
__device__ __forceinline__ FF operator-(FF a) { return FF{-a.h, -a.l}; }
__device__ __forceinline__ FF operator-(FF a, FF b) { return a + (-b); }
__device__ __forceinline__ FF operator*(FF a, FF b)
{
    const float p = __fmul_rn(a.h, b.h);
    return ff_quick(p, fmaf(a.h, b.l, fmaf(a.l, b.h, fmaf(a.h, b.h, -p))));
}
__device__ __forceinline__ FF operator*(float a, FF b)
{
    const float p = __fmul_rn(a, b.h);
    return ff_quick(p, fmaf(a, b.l, fmaf(a, b.h, -p)));
}
// c + a b for |c| >= |a b| (2^-47 of c; l is not reduced below half an ulp of h)
__device__ __forceinline__ FF ff_horner(FF c, FF a, FF b)
{
    const float p = __fmul_rn(a.h, b.h);
    const FF s = ff_quick(c.h, p);
    return FF{s.h, __fadd_rn(s.l, fmaf(a.h, b.l, fmaf(a.l, b.h, fmaf(a.h, b.h, -p))) + c.l)};
}

// The same of a PLAIN sample: ring constants and frame.
struct RingF {
    FF dc, dphi, s, Zs, Wz, Di;
};
struct PlainSmem : WarpState<double> {
    RingF rd[32];
    FF z0, s0, c2p, s2p;
};
__device__ __forceinline__ void put(double& x, double v) { x = v; }
__device__ __forceinline__ void put(FF& x, double v) { x = ff(v); }

// Warp-uniform queue state, in registers.
struct Queue {
    int n;    // queued entries (< 32 between samples)
    int cur;  // next slot
};

// Where one sample's TOD goes.
struct Out {
    void* a;
    void* b;
    long long idx;
    int f64;
};

// What a checking run (kCheck) finds, per lane: the worst error of an FP32
// decision and of one that quick_pair takes, each in units of its margin; the
// pairs visited, and those whose beam pixel is not the chain's.
struct Check {
    float fp32 = 0.0f, fp64 = 0.0f;
    unsigned long long pairs = 0, differ = 0;
};

__device__ __forceinline__ void store_out(void* out, int f64, long long i, double v)
{
    if (!out) return;
    if (f64) ((double*)out)[i] = v;
    else ((float*)out)[i] = (float)v;
}

__device__ __forceinline__ void finalize(const Pend& P)
{
    store_out(P.out_a, P.f64, P.idx, P.main_a + P.fb_a);
    store_out(P.out_b, P.f64, P.idx, P.main_b + P.fb_b);
}

struct Beam {
    const F8* beam;
    int nside;
    int npix;
    double rho_max;
    double cosr;   // cos(rho_max), evaluated on the device
    float versr;   // 1 - cos(rho_max)
    float rscale;  // sqrt(3) * nside
};

// cos(rho_max) as the disc takes it, and 1 - cos(rho_max): about 100 FP64
// instructions, formed once per block or per detector.
__device__ __forceinline__ void beam_trig(double rho_max, double& cosr, float& versr)
{
    cosr = rho_max >= kPi ? 0.0 : cos(rho_max);
    const double half = sin(0.5 * rho_max);
    versr = (float)(2.0 * half * half);
}

__device__ __forceinline__ Beam make_beam(const F8* beam, int nside, int npix, double rho_max)
{
    Beam b;
    b.beam = beam;
    b.nside = nside;
    b.npix = npix;
    b.rho_max = rho_max;
    beam_trig(rho_max, b.cosr, b.versr);
    b.rscale = (float)(1.7320508075688772 * (double)nside);
    return b;
}

// The beam of a batched launch's detector (its trig formed beforehand).
__device__ __forceinline__ Beam det_beam(const BatchDet& d)
{
    return Beam{d.beam, d.nside_beam, d.npix_beam, d.rho_max, d.cosr, d.versr,
                (float)(1.7320508075688772 * (double)d.nside_beam)};
}

__device__ __forceinline__ void record(unsigned int* err, unsigned int code)
{
    if (err) atomicCAS(err, 0u, code);
}

__device__ __forceinline__ void two_sum(float& s, float& c, float x)
{
    const float t = s + x;
    const float bp = t - s;
    const float e = (s - (t - bp)) + (x - bp);
    s = t;
    c += e;
}

// Two FP32 values in one 64-bit register pair, added and subtracted by one
// instruction each (the packed FP32 forms round every half as the scalar ones
// do; they take one issue slot where two scalar instructions take two).
using F32x2 = unsigned long long;
__device__ __forceinline__ F32x2 pack2(float lo, float hi)
{
    F32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(F32x2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ F32x2 add2(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F32x2 sub2(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F32x2 mul2(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F32x2 fma2(F32x2 a, F32x2 b, F32x2 c)
{
    F32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ F32x2 add2_rd(F32x2 a, F32x2 b)  // rounded down
{
    F32x2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F32x2 both(float x) { return pack2(x, x); }
__device__ __forceinline__ float lo2(F32x2 v)
{
    float a, b;
    unpack2(v, a, b);
    return a;
}
__device__ __forceinline__ float hi2(F32x2 v)
{
    float a, b;
    unpack2(v, a, b);
    return b;
}
// two_sum of both halves
__device__ __forceinline__ void two_sum2(F32x2& s, F32x2& c, F32x2 x)
{
    const F32x2 t = add2(s, x);
    const F32x2 bp = sub2(t, s);
    c = add2(c, add2(sub2(s, sub2(t, bp)), sub2(x, bp)));
    s = t;
}

constexpr float kTwo23 = 8388608.0f;
constexpr int kTwo23Bits = 0x4B000000;  // the bits of 2^23

// floor(x) and its fractional part f = x - floor(x) for 0 <= x < 2^23 by
// FP32 additions: x + 2^23 rounded down is 2^23 + floor(x) exactly (the
// spacing of floats in [2^23, 2^24) is 1), and x - floor(x) is exact
// (Sterbenz).
__device__ __forceinline__ int split_floor(float x, float& f)
{
    const float t = __fadd_rd(x, kTwo23);
    f = x - (t - kTwo23);
    return __float_as_int(t) - kTwo23Bits;
}

// The same with h = floor(x) + 1/2 (exact below 2^22) and f = x - h in
// [-1/2, 1/2]: x lies within m of an integer exactly when |f| > 1/2 - m, one
// comparison for both sides.  Returns the bits of 2^23 + floor(x).
__device__ __forceinline__ int split_half(float x, float& h, float& f)
{
    const float t = __fadd_rd(x, kTwo23);
    h = t - 8388607.5f;
    f = x - h;
    return __float_as_int(t);
}

// (float)k for |k| < 2^22 by FP32 addition: 1.5 * 2^23 + k lies in
// [2^23, 2^24), where floats are the integers and their bits are linear in
// the value, so no conversion instruction is needed (the same value).
__device__ __forceinline__ float small_int_to_float(int k)
{
    return __int_as_float(0x4B400000 + k) - 12582912.0f;
}

// The inverse for an integer-valued float f, |f| < 2^22 (exact, no conversion).
__device__ __forceinline__ int small_float_to_int(float f)
{
    return __float_as_int(f + 12582912.0f) - 0x4B400000;
}

// 1/x by the MUFU reciprocal approximation (relative error below 2^-22).  What
// it decides (sigma in quarter_turns, hence the beam pixel) has that error within
// the margin of the decisions.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 1/sqrt(x) by the MUFU approximation (relative error below 2^-22).
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// One beam pixel, both detectors (32 bytes, one sector): a single 256-bit
// load through the read-only path.  kL1: allocating in L1.  A warp's gather
// of 32 scattered pixels takes the L1 34 cycles when L2 serves it (a sector a
// cycle; 57 from a table of 64 KB, whose few L2 slices are hot) and 19 when L1
// hits, so a kernel whose shared memory leaves L1 150 KB or more keeps beam
// pixels there (20 warps with two pixels per lane: 4.31 ms against 4.93 ms for
// 100,000 samples of a 1.1 MB beam); one that leaves less gives L1 to the
// sky, which neighbouring samples re-read (back-projection at 32 warps per SM: 2.36 ms
// without allocation, 2.47 ms with).
template <bool kL1 = false>
__device__ __forceinline__ F8 load_beam(const F8* p)
{
    F8 r;
    if constexpr (kL1)
        asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y),
              "=f"(r.b.z), "=f"(r.b.w)
            : "l"(p));
    else
        asm("ld.global.nc.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y),
              "=f"(r.b.z), "=f"(r.b.w)
            : "l"(p));
    return r;
}

// Two neighbouring sky pixels, 32-byte aligned.
__device__ __forceinline__ void load_sky2(const float4* p, float4& S0, float4& S1)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(S0.x), "=f"(S0.y), "=f"(S0.z), "=f"(S0.w), "=f"(S1.x), "=f"(S1.y), "=f"(S1.z),
          "=f"(S1.w)
        : "l"(p));
}

// A beam pixel of the bilinear stencil: its four pixels are two pairs of
// ring neighbours, and neighbouring pairs of a sample share stencil pixels,
// so these reads do hit L1; the compiler's own (allocating, 2 x 128-bit)
// loads serve them best (c2 bilinear forward: 331.9 ms, against 348.4 ms
// for one allocating 256-bit load and 368.1 ms without L1 allocation).
// PISCO_BIL_L1 0: no allocation, as the nearest lookup; 1: one allocating
// 256-bit load; 2: the compiler's loads.
#ifndef PISCO_BIL_L1
#define PISCO_BIL_L1 2
#endif
__device__ __forceinline__ F8 load_beam_stencil(const F8* p)
{
#if PISCO_BIL_L1 == 2
    return *p;
#elif PISCO_BIL_L1
    F8 r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y),
          "=f"(r.b.z), "=f"(r.b.w)
        : "l"(p));
    return r;
#else
    return load_beam(p);
#endif
}

// sin(x) and 1 - cos(x): Taylor series for |x| <= 0.5 (truncation below
// 3e-11 relative), CUDA sincosf beyond.
__device__ __forceinline__ void sin_versin(float x, float& sn, float& h)
{
    if (fabsf(x) <= 0.5f) {
        const float x2 = x * x;
        sn = x * fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, 2.75573192e-6f, -1.98412698e-4f),
                                        8.33333333e-3f), -1.66666667e-1f), 1.0f);
        h = x2 * fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, 2.75573192e-7f, -2.48015873e-5f),
                                        1.38888889e-3f), -4.16666667e-2f), 0.5f);
    } else {
        float cs;
        sincosf(x, &sn, &cs);
        h = (cs > 0.0f) ? (sn * sn) / (1.0f + cs) : 1.0f - cs;
    }
}

// The disc's pixels on one ring, as ring indices lo .. lo + n - 1 (0 <= lo <
// npix, wrapping at npix).
struct RingRange {
    int lo, n;
};

// A ring's place under the sample: its latitude offset (sin Di and 1 - cos
// K), and the boresight's longitude in ring pixels, phi npix / 2 pi = at + f +
// e (at an integer, |f| <= 1/2, e what the FP32 product leaves out: f and e are
// kept apart because the anchor's offset can cancel f).
struct RingPlace {
    float Di, K, f, e;
    int at;
};
__device__ __forceinline__ RingPlace place_ring(const SamplePlan& p, const RingT& rt)
{
    RingPlace g;
    // dec - dec0: the difference of the high parts and its exact rounding
    // error, plus the low parts; then sin and 1 - cos at the FP32 value, with
    // a first-order correction for what it leaves out
    const float a = rt.dec_hi - p.dec_hi;
    const float b = a - rt.dec_hi;
    const float e = (rt.dec_hi - (a - b)) - (p.dec_hi + b);
    const float t = e + (rt.dec_lo - p.dec_lo);
    const float df = a + t;
    const float de = t - (df - a);
    float sD, hD;
    sin_versin(df, sD, hD);
    g.Di = fmaf(de, 1.0f - hD, sD);
    g.K = fmaf(de, sD, hD);
    // the product of the two pairs, its rounding error by a fused multiply-add
    const float m = p.phi_hi * rt.fr_hi;
    g.e = fmaf(p.phi_hi, rt.fr_lo, fmaf(p.phi_lo, rt.fr_hi, fmaf(p.phi_hi, rt.fr_hi, -m)));
    const float n = (m + 12582912.0f) - 12582912.0f;  // rint(m), |m| < 2^22
    g.f = __fsub_rn(m, n);  // (not contracted with m's product: e holds its error)
    g.at = small_float_to_int(n);
    return g;
}

// The disc's range on a ring: the edge longitude in FP32 from
//   1 - cos D = (1 - cos radius - (1 - cos(dec - dec0))) / (s s0),
// the exact FP64 HEALPix formula (disc_ring) whenever an edge lies within the
// FP32 angle's error of a pixel boundary.  Same pixels as disc_ring.
//
// The error: with C = 1 - cos radius, H = C / (s s0) and D the edge angle,
// the numerator is off by at most 3.6e-7 C (K to 3e-7, C and the difference
// to half an ulp), 1 - cos D by 7.2e-7 H, D by 7.2e-7 H / sin D + 6e-7 D, and a
// position of fr D pixels by 3e-7 fr D + 2e-7 more (products, sums and f); the
// margin is 1e-6 fr (H / sin D + D) + 3e-7 pixels, at least 1.1 times that.  At
// nside 1024 and 3 degrees it is 6e-5 pixels: two rings in ten thousand take
// the exact formula.
__device__ __forceinline__ RingRange fast_disc_ring(const Hpx& h, const SamplePlan& p,
                                                    double cosr, float versr, int ring,
                                                    const RingT& rt, const RingPlace& g)
{
    RingRange s = {0, 0};
    const int npix = rt.npix2 >> 1;
    if ((p.flags & kPlanAllSky) || ring < p.ring_lo || ring > p.ring_hi) {
        s.n = npix;
        return s;
    }
    const float is = 1.0f / (rt.s * p.s0f);
    const float x = (versr - g.K) * is;  // 1 - cos D
    const float y = sqrtf(x * (2.0f - x));
    const float D = atan2f(y, 1.0f - x);
    const float shift = (rt.npix2 & 1) ? 0.5f : 0.0f;
    const float w = rt.fr_hi * D;
    const float at = (g.f - shift) + g.e;
    const float vlo = at - w, vhi = at + w;
    const float flo = floorf(vlo), fhi = floorf(vhi);
    // y = 0 or a NaN (an edge outside [0, pi]) makes m infinite or a NaN
    const float m = fmaf(1e-6f, rt.fr_hi * (versr * is / y + D), 3e-7f);
    const float rlo = vlo - flo, rhi = vhi - fhi;
    if (!(fminf(rlo, rhi) > m && fmaxf(rlo, rhi) < 1.0f - m) || (p.flags & kPlanExact)) {
        DiscPlan d;
        d.z0 = p.z0;
        d.xa = p.xa;
        d.cosr = cosr;
        d.phi = p.phi;
        d.ring_lo = p.ring_lo;
        d.ring_hi = p.ring_hi;
        d.full_lo = p.full_lo;
        d.full_hi = p.full_hi;
        d.all_sky = (p.flags & kPlanAllSky) != 0;
        const RingSpan e = disc_ring(h, d, ring);
        s.lo = (int)((e.n2 > 0 ? e.start2 : e.start1) - rt.start);
        s.n = (int)(e.n1 + e.n2);
        if (s.n <= 0) s = RingRange{0, 0};
        return s;
    }
    const int lo = g.at + (int)flo + 1, hi = g.at + (int)fhi;
    if (lo > hi) return s;
    s.lo = lo < 0 ? lo + npix : (lo >= npix ? lo - npix : lo);
    s.n = hi - lo + 1;
    return s;
}

// Bilinear beam value of the PLAIN form (HEALPix get_interpol in FP64; the
// weights of stencil pixels outside the stored map are dropped and the rest
// renormalised; the value rounded to float).  false: no stencil pixel lies in
// the map.  Not inlined: only the degenerate boresight pairs take it, and
// inlined its FP64 stencil would spill registers of the main pair loop.
static __device__ __noinline__ bool bilinear_f64(const Hpx& hb, int npb, double rho,
                                                 double sig, const F8* beam, F8& out)
{
    int64_t px[4];
    double w[4];
    get_interpol(hb, rho, sig, px, w);
    double ws = 0.0, va[4] = {0.0, 0.0, 0.0, 0.0}, vb[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (px[i] < 0 || px[i] >= npb) continue;
        ws += w[i];
        const F8 B = beam[px[i]];
        va[0] += B.a.x * w[i]; va[1] += B.a.y * w[i]; va[2] += B.a.z * w[i]; va[3] += B.a.w * w[i];
        vb[0] += B.b.x * w[i]; vb[1] += B.b.y * w[i]; vb[2] += B.b.z * w[i]; vb[3] += B.b.w * w[i];
    }
    if (!(ws > 0.0)) return false;
    out.a = make_float4((float)(va[0] / ws), (float)(va[1] / ws), (float)(va[2] / ws),
                        (float)(va[3] / ws));
    out.b = make_float4((float)(vb[0] / ws), (float)(vb[1] / ws), (float)(vb[2] / ws),
                        (float)(vb[3] / ws));
    return true;
}

// get_interpol's stencil in FP64 with the weights renormalised over the
// pixels inside the stored map (pixels outside get weight 0), rounded to
// float: what a beam-gradient scatter needs.  false: no pixel in the map.
static __device__ __noinline__ bool stencil_f64(const Hpx& hb, int npb, double rho, double sig,
                                                int px[4], float w[4])
{
    int64_t p[4];
    double wd[4];
    get_interpol(hb, rho, sig, p, wd);
    double ws = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (p[i] >= 0 && p[i] < npb) ws += wd[i];
    if (!(ws > 0.0)) return false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool in = p[i] >= 0 && p[i] < npb;
        px[i] = in ? (int)p[i] : 0;
        w[i] = in ? (float)(wd[i] / ws) : 0.0f;
    }
    return true;
}

// (f(a) - f(b)) / (2c (a - b)) for f(x) = 2 asin(c x), the colatitude of ring
// height x (x = nside sqrt(3 (1 - cos theta)), c = 1 / (sqrt(6) nside)), by
// the asin series to c^4 (relative truncation below 1e-8 for theta <= 0.5).
__device__ __forceinline__ float asin_slope(float a, float b, float c2)
{
    const float s2 = fmaf(a, a, fmaf(a, b, b * b));
    const float a2 = a * a, b2 = b * b;
    const float s4 = fmaf(a2, a2, fmaf(a2, a * b, fmaf(a2, b2, fmaf(a * b, b2, b2 * b2))));
    return fmaf(c2 * c2 * 0.075f, s4, fmaf(c2 * (1.0f / 6.0f), s2, 1.0f));
}

#ifndef PISCO_BIL_FASTDIV
#define PISCO_BIL_FASTDIV 1
#endif
// a / b for the stencil weights (b > 0, never an index decision): the MUFU
// reciprocal instead of the IEEE division (c2 bilinear forward: 313.3 ms
// against 332.0 ms; the weights move by about an ulp)
__device__ __forceinline__ float wdiv(float a, float b)
{
#if PISCO_BIL_FASTDIV
    return a * rcp_approx(b);
#else
    return a / b;
#endif
}

// The same stencil in FP32 from the pair's polar-cap coordinates on the beam
// grid: r = nside sqrt(3 (1 - cos rho)) and sigma = (qd + tp) pi/2.  Rings of
// the north cap: ring i holds 4i pixels from 2i(i - 1), half a pixel shifted;
// get_interpol takes the ring above (floor r) and the next one, interpolates
// in longitude on each and linearly in colatitude between them (ring 1 and
// its image across the pole when r < 1).  The weights are continuous across
// every floor decision, so FP32 index choices near a boundary change the
// value only by the FP32 error of r and tp: no FP64 re-evaluation is needed.
__device__ __forceinline__ bool bilinear_f32(const Beam& B, int qd, float tp, float r, F8& out)
{
    const float c = 1.0f / (2.4494897427831781f * (float)B.nside);  // 1 / (sqrt(6) nside)
    const float c2 = c * c;
    float kfr;
    const int k = split_floor(r, kfr);  // ring above (0 above the first ring); r >= 0
    // longitude interpolation on ring i: pixels start + i1, start + i1 + 1
    auto ring = [&](int i, int& p1, int& p2, float& w1, float& w2) {
        const float t = fmaf(tp, small_int_to_float(i), -0.5f);
        const float fl = floorf(t);
        const float f = t - fl;
        int i1 = small_float_to_int(fl) + qd * i, i2 = i1 + 1;
        const int np = 4 * i;
        if (i1 < 0) i1 += np;
        if (i2 >= np) i2 -= np;
        const int start = 2 * i * (i - 1);
        p1 = start + i1;
        p2 = start + i2;
        w1 = 1.0f - f;
        w2 = f;
    };
    // stencil pixels are added as soon as their weight is known, in
    // get_interpol's order; pixels beyond the stored map are dropped
    float ws = 0.0f;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](int p, float w) {
        if (p >= B.npix) return;
        ws += w;
        const F8 v = load_beam_stencil(B.beam + p);
        a.x = fmaf(v.a.x, w, a.x); a.y = fmaf(v.a.y, w, a.y);
        a.z = fmaf(v.a.z, w, a.z); a.w = fmaf(v.a.w, w, a.w);
        b.x = fmaf(v.b.x, w, b.x); b.y = fmaf(v.b.y, w, b.y);
        b.z = fmaf(v.b.z, w, b.z); b.w = fmaf(v.b.w, w, b.w);
    };
    int p1, p2;
    float w1, w2;
    if (k == 0) {
        ring(1, p1, p2, w1, w2);
        const float wt = wdiv(r * asin_slope(r, 0.0f, c2), asin_slope(1.0f, 0.0f, c2));
        const float f = 0.25f * (1.0f - wt);
        add((p1 + 2) & 3, f);
        add((p2 + 2) & 3, f);
        add(p1, fmaf(w1, wt, f));
        add(p2, fmaf(w2, wt, f));
    } else {
        const float kf = small_int_to_float(k);
        const float wt = wdiv((r - kf) * asin_slope(r, kf, c2), asin_slope(kf + 1.0f, kf, c2));
        ring(k, p1, p2, w1, w2);
        add(p1, w1 * (1.0f - wt));
        add(p2, w2 * (1.0f - wt));
        ring(k + 1, p1, p2, w1, w2);
        add(p1, w1 * wt);
        add(p2, w2 * wt);
    }
    if (!(ws > 0.0f)) return false;
    const float iw = wdiv(1.0f, ws);
    out.a = make_float4(a.x * iw, a.y * iw, a.z * iw, a.w * iw);
    out.b = make_float4(b.x * iw, b.y * iw, b.z * iw, b.w * iw);
    return true;
}

// The stencil of bilinear_f32 itself: pixels and weights renormalised over
// the pixels inside the stored map (outside: weight 0), for actions that
// scatter into the beam (Action::kStencil).
__device__ __forceinline__ bool stencil_f32(const Beam& B, int qd, float tp, float r, int px[4],
                                            float w[4])
{
    const float c = 1.0f / (2.4494897427831781f * (float)B.nside);
    const float c2 = c * c;
    float kfr;
    const int k = split_floor(r, kfr);  // r >= 0
    auto ring = [&](int i, int& p1, int& p2, float& w1, float& w2) {
        const float t = fmaf(tp, small_int_to_float(i), -0.5f);
        const float fl = floorf(t);
        const float f = t - fl;
        int i1 = small_float_to_int(fl) + qd * i, i2 = i1 + 1;
        const int np = 4 * i;
        if (i1 < 0) i1 += np;
        if (i2 >= np) i2 -= np;
        const int start = 2 * i * (i - 1);
        p1 = start + i1;
        p2 = start + i2;
        w1 = 1.0f - f;
        w2 = f;
    };
    if (k == 0) {
        ring(1, px[2], px[3], w[2], w[3]);
        const float wt = wdiv(r * asin_slope(r, 0.0f, c2), asin_slope(1.0f, 0.0f, c2));
        const float f = 0.25f * (1.0f - wt);
        w[0] = f;
        w[1] = f;
        w[2] = fmaf(w[2], wt, f);
        w[3] = fmaf(w[3], wt, f);
        px[0] = (px[2] + 2) & 3;
        px[1] = (px[3] + 2) & 3;
    } else {
        ring(k, px[0], px[1], w[0], w[1]);
        ring(k + 1, px[2], px[3], w[2], w[3]);
        const float kf = small_int_to_float(k);
        const float wt = wdiv((r - kf) * asin_slope(r, kf, c2), asin_slope(kf + 1.0f, kf, c2));
        w[0] *= 1.0f - wt;
        w[1] *= 1.0f - wt;
        w[2] *= wt;
        w[3] *= wt;
    }
    float ws = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (px[i] >= B.npix) {
            px[i] = 0;
            w[i] = 0.0f;
        }
        ws += w[i];
    }
    if (!(ws > 0.0f)) return false;
    const float iw = wdiv(1.0f, ws);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] *= iw;
    return true;
}

// The beam pixel and exp(2i chi) of a pair in FP64 without the chain's
// arccosines and the sines and cosines of its angles: one sine and cosine (of
// the longitude offset) and one arctangent, some 200 FP64 instructions against
// 700.  false where the chain itself has to decide: within 1e-3 rad of the
// boresight, a frame near a pole, or a decision within the margin of an integer.
// The chain takes rho as acos(cos rho), which moves it by some 1e-16 / rho and a
// decision by nside_b times as much: on a beam grid of nside 8192 up to 7.6
// margins at 1e-4 rad, 0.22 from 1e-3 on.  (Its degenerate branch lies at 1e-6.)
struct QuickPair {
    long long bp;
    double c2, s2;
    double av, bv, cv, ir, m;  // the decisions (CapPixel) and their margin
};
__device__ __forceinline__ bool quick_pair(const Hpx& hs, const Hpx& hb, const Pend& P, int pix,
                                           QuickPair& q)
{
    if (P.plain) return false;
    double z, phi, s;
    bool have;
    pix2loc(hs, pix, &z, &phi, &s, &have);
    if (!have) s = sqrt((1.0 - z) * (1.0 + z));
    double sd, cd;
    sincos(phi - P.phi, &sd, &cd);
    const double u = s * sd, v = z * P.s0 - s * P.z0 * cd;
    const double nb = P.s0 * sd, db = s * P.z0 - z * P.s0 * cd;
    const double sin2 = fma(u, u, v * v);
    if (!(sin2 > 1e-6)) return false;
    // r = nside sqrt(3 (1 - cos rho)), 1 - cos rho = sin^2 rho / (1 + cos rho)
    const double r = (double)hb.nside * sqrt(3.0 * sin2 / (1.0 + z * P.z0 + s * P.s0 * cd));
    const double X = u * P.spsi - v * P.cpsi, Y = u * P.cpsi + v * P.spsi;
    const double t = atan2(Y, X) * kInvHalfPi;  // quarter turns, in [-2, 2]
    const double tt = t < 0.0 ? t + 4.0 : t;
    const double qd = floor(tt), tp = tt - qd;
    const double av = tp * r, bv = r - av;
    const double fa = floor(av), fb = floor(bv);
    const double ir = fa + fb + 1.0, cv = tp * ir, fc = floor(cv);
    const double m = 1e-9 * (r + 2.0);
    const double ea = av - fa, eb = bv - fb, ec = cv - fc;
    if (!(fmin(fmin(ea, eb), ec) > m && fmax(fmax(ea, eb), ec) < 1.0 - m)) return false;
    q.bp = (long long)(2.0 * ir * (ir - 1.0) + qd * ir + fc);
    q.av = av;
    q.bv = bv;
    q.cv = cv;
    q.ir = ir;
    q.m = m;
    // phasor's w, turned by psi
    const double wr = fma(db, X, nb * Y), wi = fma(nb, X, -(db * Y));
    const double rr = wr * wr, iw = 1.0 / fma(wi, wi, rr);
    q.c2 = fma(-wi, wi, rr) * iw;
    q.s2 = wr * wi * (iw + iw);
    return true;
}

// Compares a pair's decisions with the chain's: the FP32 ones (av, bv, cv of
// ring ir, beam pixel bp) where the pair is not queued, and quick_pair's, which
// a queued pair would take, for every pair that it accepts.  r: the pair's FP32
// ring position (the FP32 margin is kMarginRel (r + 2)).
static __device__ __noinline__ void check_pair(const Hpx& hs, const Hpx& hb, const Pend& P, int pix,
                                               float av, float bv, float cv, int ir, float r, int bp,
                                               bool queued, Check& ck)
{
    double rho, sig, chi;
    const long long want = pair_beam_pixel(hs, hb, pix, P.ra, P.dec, P.psi, &rho, &sig, &chi);
    const double tt = fmodulo(sig * kInvHalfPi, 4.0), tp = tt - floor(tt);
    // nside sqrt(3 (1 - cos rho))
    const double rd = (double)hb.nside * 2.4494897427831781 * sin(0.5 * rho);
    auto worst = [&](double a, double b, double c, double ring) {
        return fmax(fmax(fabs(a - tp * rd), fabs(b - (1.0 - tp) * rd)), fabs(c - tp * ring));
    };
    ++ck.pairs;
    if (!queued) {
        ck.fp32 = fmaxf(ck.fp32, (float)(worst(av, bv, cv, (double)ir) / (kMarginRel * (r + 2.0))));
        ck.differ += bp != want;
    }
    QuickPair q;
    if (quick_pair(hs, hb, P, pix, q)) {
        ck.fp64 = fmaxf(ck.fp64, (float)(worst(q.av, q.bv, q.cv, q.ir) / q.m));
        ck.differ += queued && q.bp != want;
    }
}

// Redoes queued pair e of the warp whose state S is, in FP64: the beam pixel
// and phasor of quick_pair or of the PLAIN form's chain.  kBil: the beam value
// is PLAIN's bilinear one instead of the nearest pixel's.
template <bool kBil, class Smem, class Action, class Real>
__device__ __forceinline__ void redo(const Hpx& hs, const Smem& S, int e, unsigned int* err,
                                     Action& act, Real& ta, Real& tb)
{
    const Pend& P = S.p[S.qs[e]];
    const int pix = S.q[e];
    const Hpx hb = hpx_make(P.nside_beam);
    double rho = 0.0, sig = 0.0;
    QuickPair q;
    if (kBil || !quick_pair(hs, hb, P, pix, q)) {
        double chi;
        q.bp = pair_beam_pixel(hs, hb, pix, P.ra, P.dec, P.psi, &rho, &sig, &chi);
        sincos(2.0 * chi, &q.s2, &q.c2);
    }
    const long long bp = q.bp;
    const double c2 = q.c2, s2 = q.s2;
    if constexpr (kBil && Action::kStencil) {
        int px[4];
        float w[4];
        if (stencil_f64(hb, P.npix_beam, rho, sig, px, w))
            act.deferred_stencil(P, pix, px, w, (float)c2, (float)s2);
        else if constexpr (HasOutside<Action>::value)
            act.outside_deferred(P, pix, -1);
    } else if constexpr (kBil) {
        F8 Bv;
        if (bilinear_f64(hb, P.npix_beam, rho, sig, P.beam, Bv))
            act.deferred(P, pix, Bv, -1, (float)c2, (float)s2, ta, tb);
        else if constexpr (HasOutside<Action>::value)
            act.outside_deferred(P, pix, -1);
    } else if (bp < 0) {
        record(err, kCheckBeamIndex);
    } else if (bp < P.npix_beam) {
        if constexpr (IsExact<Action>::value)
            act.deferred64(pix, (int)bp, c2, s2, ta, tb);
        else
            act.deferred(P, pix, load_beam(P.beam + bp), (int)bp, (float)c2, (float)s2, ta, tb);
    } else if constexpr (HasOutside<Action>::value) {
        act.outside_deferred(P, pix, (int)bp);
    }
}

// Credits the first m redone pairs (S.ta, S.tb) to their samples: serially, in
// queue order, by the first lane of each run of one slot's entries; writes the
// TOD of every sample left with nothing queued.
template <class Action, class Smem>
__device__ __forceinline__ void credit(Smem& S, int m, int lane)
{
    const int slot = lane < m ? S.qs[lane] : -1;
    if (lane < m && (lane == 0 || S.qs[lane - 1] != slot)) {
        Pend& P = S.p[slot];
        int k = lane;
        if (Action::kSums) {
            double a = P.fb_a, b = P.fb_b;
            do {
                a += (double)S.ta[k];
                b += (double)S.tb[k];
                ++k;
            } while (k < m && S.qs[k] == slot);
            P.fb_a = a;
            P.fb_b = b;
        } else {
            do ++k;
            while (k < m && S.qs[k] == slot);
        }
        P.left -= k - lane;
        if (Action::kSums && P.left == 0 && !P.open) finalize(P);
    }
}

// Redoes the first m (<= 32, <= Q.n) queued pairs, one per lane, credits them
// and drops the m entries.
template <bool kBil = false, class Smem, class Action>
__device__ __forceinline__ void drain(const Hpx& hs, int m, Smem& S, Queue& Q, int lane,
                                      unsigned int* err, Action& act)
{
    std::remove_reference_t<decltype(S.ta[0])> ta = 0, tb = 0;
    if (lane < m) redo<kBil>(hs, S, lane, err, act, ta, tb);
    if (Action::kSums) {
        S.ta[lane] = ta;
        S.tb[lane] = tb;
    }
    __syncwarp();
    credit<Action>(S, m, lane);
    // move the rest (<= 32 entries: the queue holds < 64) to the front
    const int rest = Q.n - m;
    int vq = 0, vs = 0;
    if (lane < rest) {
        vq = S.q[m + lane];
        vs = S.qs[m + lane];
    }
    __syncwarp();
    if (lane < rest) {
        S.q[lane] = vq;
        S.qs[lane] = (unsigned char)vs;
    }
    __syncwarp();
    Q.n = rest;
}

// Redoes every queued pair (at a sample boundary, where fewer than 32 are
// queued): all slots are free afterwards.  Called once more before a warp
// leaves the kernel.
template <bool kBil = false, class Smem, class Action>
__device__ __forceinline__ void flush(const Hpx& hs, Smem& S, Queue& Q, int lane,
                                      unsigned int* err, Action& act)
{
    if (Q.n > 0) drain<kBil>(hs, Q.n, S, Q, lane, err, act);
}

// The same for all the warps of a block, when they leave the kernel (every
// thread calls it): their left-over entries are redone together, 32 at a time
// from whichever warp, instead of a long FP64 chain per warp with a few lanes
// active -- what a launch of a few samples per warp spends a tenth of its time
// on.  sm: the block's states; warps: their number.  The bilinear lookup queues
// next to nothing (pairs at the boresight): its warps flush by themselves (2 %
// of its time).
template <bool kBil = false, class Smem, class Action>
__device__ __forceinline__ void flush_block(const Hpx& hs, Smem* sm, int warps, Queue& Q, int lane,
                                            unsigned int* err, Action& act)
{
    const int warp = threadIdx.x >> 5;
    if constexpr (kBil) return flush<kBil>(hs, sm[warp], Q, lane, err, act);
    __shared__ int counts[32];
    if (lane == 0) counts[warp] = Q.n;
    __syncthreads();
    int e = threadIdx.x, w = 0;
    while (w < warps && e >= counts[w]) e -= counts[w++];
    if (w < warps) {
        std::remove_reference_t<decltype(sm->ta[0])> ta = 0, tb = 0;
        redo<kBil>(hs, sm[w], e, err, act, ta, tb);
        if (Action::kSums) {
            sm[w].ta[e] = ta;
            sm[w].tb[e] = tb;
        }
    }
    __syncthreads();
    credit<Action>(sm[warp], Q.n, lane);
    Q.n = 0;
}

// The same for |x| <= kShortOffset, two terms fewer each (truncation below
// 8e-10 relative, an eightieth of an FP32 ulp).
__device__ __forceinline__ void short_sin_versin(float x, float& sn, float& h)
{
    const float x2 = x * x;
    sn = x * fmaf(x2, fmaf(x2, 8.33333333e-3f, -1.66666667e-1f), 1.0f);
    h = x2 * fmaf(x2, fmaf(x2, 1.38888889e-3f, -4.16666667e-2f), 0.5f);
}

// Fraction of the quadrant, atan2(yy, xx) / (pi/2) in [0, 1], of the
// direction (X, Y): yy, xx = |Y|, |X| where the signs agree (quadrants 0 and
// 2) and |X|, |Y| where they differ (1 and 3); sgn is the sign bit of X Y.
// As 1/2 + (2/pi) atan(t), t = (yy - xx) / (yy + xx) in [-1, 1]: no swap of
// numerator and denominator, so no comparison or selection.  The arctangent
// is the minimax polynomial of Abramowitz & Stegun 4.4.49 (|error| <= 2e-8),
// its coefficients times 2/pi; clamped to [0, 1].  X = Y = 0 gives a NaN
// (such pairs are re-done in FP64 anyway).
__device__ __forceinline__ float quarter_turns(float X, float Y, unsigned sgn)
{
    const float d = __uint_as_float(__float_as_uint(fabsf(Y) - fabsf(X)) ^ sgn);
    const float t = d * rcp_approx(fabsf(X) + fabsf(Y));
    const float t2 = t * t;
    constexpr double q = 0.63661977236758134;
    float p = (float)(q * 0.0028662257);
    p = fmaf(p, t2, (float)(q * -0.0161657367));
    p = fmaf(p, t2, (float)(q * 0.0429096138));
    p = fmaf(p, t2, (float)(q * -0.0752896400));
    p = fmaf(p, t2, (float)(q * 0.1065626393));
    p = fmaf(p, t2, (float)(q * -0.1420889944));
    p = fmaf(p, t2, (float)(q * 0.1999355085));
    p = fmaf(p, t2, (float)(q * -0.3333314528));
    p = fmaf(p, t2, (float)q);
    return __saturatef(fmaf(t, p, 0.5f));
}

// A pair's place in the beam's frame: sin D and 1 - cos D of its longitude
// offset, R^2 (1 - cos rho), the rotated components (X, Y), the beam grid's
// polar-cap coordinates (quadrant qd, fraction tp, r = R sqrt(1 - cos rho)).
struct Spot {
    float sn, h, q, X, Y, tp, r;
    int qd;
};

// The pair kf pixels from its ring's anchor, R0 = (dc, dphi, Ki, s) and Di its
// ring's.  East u = s sin D, north v = Di + z0 s (1 - cos D), turned by psi.
__device__ __forceinline__ Spot locate(float kf, const Frame& F, const float4& R0, float Di,
                                       bool narrow)
{
    Spot p;
    const float dl = fmaf(kf, R0.y, R0.x);
    if (narrow) short_sin_versin(dl, p.sn, p.h);
    else sin_versin(dl, p.sn, p.h);
    const float sh = R0.w * p.h, u = R0.w * p.sn;
    const float v = fmaf(F.z0, sh, Di);
    p.q = fmaf(F.R2s0, sh, R0.z);
    p.X = fmaf(u, F.sps, -v * F.cps);
    p.Y = fmaf(u, F.cps, v * F.sps);
    const unsigned sgn = (__float_as_uint(p.X) ^ __float_as_uint(p.Y)) & 0x80000000u;
    p.qd = (int)(2u * (__float_as_uint(p.Y) >> 31) + (sgn >> 31));
    p.tp = quarter_turns(p.X, p.Y, sgn);
    p.r = __fmul_rn(p.q, rsqrt_approx(p.q));
    return p;
}

// exp(2i chi) = w^2 / |w|^2, w = (db + i nb)(X - i Y): the direction to the
// boresight (nb = s0 sin D, db = Wz h - Di) times the rotated beam-frame
// direction (an overall sign drops out).
__device__ __forceinline__ void phasor(const Spot& p, float s0, float Wz, float Di, float& c2,
                                       float& s2)
{
    const float nb = s0 * p.sn;
    const float db = fmaf(Wz, p.h, -Di);
    const float wr = fmaf(db, p.X, nb * p.Y);
    const float wi = fmaf(nb, p.X, -(db * p.Y));
    const float ww = wr * wr;
    const float iw = rcp_approx(fmaf(wi, wi, ww));
    c2 = fmaf(-wi, wi, ww) * iw;
    s2 = wr * wi * (iw + iw);
}

// The nearest beam pixel, ang2pix of the polar cap: jp = floor(tp r), jm =
// floor((1 - tp) r), ring ir = jp + jm + 1, position floor(tp ir) in the
// quadrant.  near: one of the three lies within its margin of an integer, and
// the pair goes to FP64.
struct CapPixel {
    float av, bv, cv;
    int ir, bp;
    bool near;
};
__device__ __forceinline__ CapPixel cap_pixel(const Spot& p)
{
    CapPixel c;
    c.av = __fmul_rn(p.tp, p.r);
    c.bv = __fsub_rn(p.r, c.av);
    float ha, fa, hb, fb, hc, fc;
    const int ja = split_half(c.av, ha, fa), jb = split_half(c.bv, hb, fb);
    const float irf = ha + hb;
    c.cv = __fmul_rn(p.tp, irf);
    const int jc = split_half(c.cv, hc, fc);
    // 1/2 less kMarginRel (r + 2), and r + 1 >= ir
    const float edge = fmaf(-kMarginRel, p.r, 0.5f - 2.0f * kMarginRel);
    c.near = fmaxf(fmaxf(fabsf(fa), fabsf(fb)), fabsf(fc)) > edge;
    c.ir = (ja - kTwo23Bits) + (jb - kTwo23Bits) + 1;
    // 2 ir (ir - 1) + qd ir + position
    c.bp = c.ir * (2 * c.ir - 2 + p.qd) + (jc - kTwo23Bits);
    return c;
}

// Two pairs of one ring, side by side: locate, cap_pixel and phasor with
// every operation that has no ring constant packed, each rounded as the scalar
// form rounds it (whichever form an action takes, a pair's decisions and
// phasor are the same bit for bit).
struct Spot2 {
    float sn0, sn1, h0, h1, q0, q1;
    F32x2 X, Y, tp, r;
    int qd0, qd1;
};
__device__ __forceinline__ unsigned sign_of(float x, float y)
{
    return (__float_as_uint(x) ^ __float_as_uint(y)) & 0x80000000u;
}
__device__ __forceinline__ Spot2 locate2(float kf, const Frame& F, const float4& R0, float Di,
                                         bool narrow)
{
    Spot2 p;
    const float d0 = fmaf(kf, R0.y, R0.x), d1 = fmaf(kf + 1.0f, R0.y, R0.x);
    if (narrow) {
        const F32x2 x = pack2(d0, d1), x2 = mul2(x, x);
        const F32x2 sn = mul2(x, fma2(x2, fma2(x2, both(8.33333333e-3f), both(-1.66666667e-1f)),
                                      both(1.0f)));
        const F32x2 h = mul2(x2, fma2(x2, fma2(x2, both(1.38888889e-3f), both(-4.16666667e-2f)),
                                      both(0.5f)));
        unpack2(sn, p.sn0, p.sn1);
        unpack2(h, p.h0, p.h1);
    } else {
        sin_versin(d0, p.sn0, p.h0);
        sin_versin(d1, p.sn1, p.h1);
    }
    const float g0 = R0.w * p.h0, g1 = R0.w * p.h1;
    const float u0 = R0.w * p.sn0, u1 = R0.w * p.sn1;
    const float w0 = fmaf(F.z0, g0, Di), w1 = fmaf(F.z0, g1, Di);
    p.q0 = fmaf(F.R2s0, g0, R0.z);
    p.q1 = fmaf(F.R2s0, g1, R0.z);
    const float X0 = fmaf(u0, F.sps, -w0 * F.cps), X1 = fmaf(u1, F.sps, -w1 * F.cps);
    const float Y0 = fmaf(u0, F.cps, w0 * F.sps), Y1 = fmaf(u1, F.cps, w1 * F.sps);
    p.X = pack2(X0, X1);
    p.Y = pack2(Y0, Y1);
    const unsigned m0 = sign_of(X0, Y0), m1 = sign_of(X1, Y1);
    p.qd0 = (int)(2u * (__float_as_uint(Y0) >> 31) + (m0 >> 31));
    p.qd1 = (int)(2u * (__float_as_uint(Y1) >> 31) + (m1 >> 31));
    // quarter_turns
    const F32x2 d = pack2(__uint_as_float(__float_as_uint(fabsf(Y0) - fabsf(X0)) ^ m0),
                          __uint_as_float(__float_as_uint(fabsf(Y1) - fabsf(X1)) ^ m1));
    const F32x2 t = mul2(d, pack2(rcp_approx(fabsf(X0) + fabsf(Y0)),
                                  rcp_approx(fabsf(X1) + fabsf(Y1))));
    const F32x2 t2 = mul2(t, t);
    constexpr double q = 0.63661977236758134;
    F32x2 a = both((float)(q * 0.0028662257));
    a = fma2(a, t2, both((float)(q * -0.0161657367)));
    a = fma2(a, t2, both((float)(q * 0.0429096138)));
    a = fma2(a, t2, both((float)(q * -0.0752896400)));
    a = fma2(a, t2, both((float)(q * 0.1065626393)));
    a = fma2(a, t2, both((float)(q * -0.1420889944)));
    a = fma2(a, t2, both((float)(q * 0.1999355085)));
    a = fma2(a, t2, both((float)(q * -0.3333314528)));
    a = fma2(a, t2, both((float)q));
    p.tp = pack2(__saturatef(fmaf(lo2(t), lo2(a), 0.5f)), __saturatef(fmaf(hi2(t), hi2(a), 0.5f)));
    p.r = pack2(__fmul_rn(p.q0, rsqrt_approx(p.q0)), __fmul_rn(p.q1, rsqrt_approx(p.q1)));
    return p;
}
struct CapPixel2 {
    F32x2 av, bv, cv;
    int ir0, ir1, bp0, bp1;
    bool near0, near1;
};
__device__ __forceinline__ CapPixel2 cap_pixel2(const Spot2& p)
{
    CapPixel2 c;
    const F32x2 k23 = both(kTwo23), khalf = both(8388607.5f);
    // (products that sums take are scalar: ptxas fuses a packed product into
    // a packed sum, which the scalar form does not)
    const F32x2 av = pack2(__fmul_rn(lo2(p.tp), lo2(p.r)), __fmul_rn(hi2(p.tp), hi2(p.r)));
    const F32x2 bv = sub2(p.r, av);
    const F32x2 ta = add2_rd(av, k23), tb = add2_rd(bv, k23);
    const F32x2 ha = sub2(ta, khalf), hb = sub2(tb, khalf);
    const F32x2 fa = sub2(av, ha), fb = sub2(bv, hb);
    const F32x2 irf = add2(ha, hb);
    const F32x2 cv = pack2(__fmul_rn(lo2(p.tp), lo2(irf)), __fmul_rn(hi2(p.tp), hi2(irf)));
    const F32x2 tc = add2_rd(cv, k23);
    const F32x2 fc = sub2(cv, sub2(tc, khalf));
    const F32x2 edge = fma2(p.r, both(-kMarginRel), both(0.5f - 2.0f * kMarginRel));
    c.near0 = fmaxf(fmaxf(fabsf(lo2(fa)), fabsf(lo2(fb))), fabsf(lo2(fc))) > lo2(edge);
    c.near1 = fmaxf(fmaxf(fabsf(hi2(fa)), fabsf(hi2(fb))), fabsf(hi2(fc))) > hi2(edge);
    c.ir0 = (__float_as_int(lo2(ta)) - kTwo23Bits) + (__float_as_int(lo2(tb)) - kTwo23Bits) + 1;
    c.ir1 = (__float_as_int(hi2(ta)) - kTwo23Bits) + (__float_as_int(hi2(tb)) - kTwo23Bits) + 1;
    c.bp0 = c.ir0 * (2 * c.ir0 - 2 + p.qd0) + (__float_as_int(lo2(tc)) - kTwo23Bits);
    c.bp1 = c.ir1 * (2 * c.ir1 - 2 + p.qd1) + (__float_as_int(hi2(tc)) - kTwo23Bits);
    c.av = av;
    c.bv = bv;
    c.cv = cv;
    return c;
}
// (the signs of wr and of its factors are turned around: no packed negation)
__device__ __forceinline__ void phasor2(const Spot2& p, float s0, float Wz, float Di, F32x2& c2,
                                        F32x2& s2)
{
    const F32x2 nb = pack2(s0 * p.sn0, s0 * p.sn1), mb = pack2(-s0 * p.sn0, -s0 * p.sn1);
    const F32x2 db = pack2(fmaf(-Wz, p.h0, Di), fmaf(-Wz, p.h1, Di));
    const F32x2 wr = fma2(db, p.X, mul2(mb, p.Y));
    const F32x2 wi = fma2(nb, p.X, mul2(db, p.Y));
    const F32x2 ww = mul2(wr, wr), n = fma2(wi, wi, ww);
    const F32x2 iw = pack2(rcp_approx(lo2(n)), rcp_approx(hi2(n)));
    c2 = mul2(fma2(mul2(wi, both(-1.0f)), wi, ww), iw);
    s2 = mul2(mul2(wr, wi), mul2(iw, both(-2.0f)));
}

// Two pairs: the values loaded for them and their phasors.
struct Unit {
    F8 B0, B1;
    float4 S0, S1;
    F32x2 c, s;  // cos 2chi, sin 2chi
    int pix;     // the first sky pixel
    int bp0, bp1;
    bool in0, in1;
};

// The FP64 ring constants of an IsExact action: ring jc the anchor's index.
__device__ __forceinline__ RingD ring_exact(const Hpx& hs, int ring, int jc, const RingT& rt,
                                            const SamplePlan& p, double z0, double s0)
{
    RingD r;
    const int ns = (int)hs.nside;
    const int north = ring > 2 * ns ? 4 * ns - ring : ring;
    double z;
    if (north < ns) {  // polar caps: z = 1 - t
        const double t = (double)north * (double)north * hs.fact2;
        z = ring == north ? 1.0 - t : t - 1.0;
        r.s = sqrt(t * (2.0 - t));
    } else {
        z = (double)(2 * ns - ring) * hs.fact1;
        r.s = sqrt((1.0 - z) * (1.0 + z));
    }
    const double phi = p.flags & kPlanExact ? (double)p.phi_hi + (double)p.phi_lo : p.phi;
    r.dphi = kTwoPi / (double)(rt.npix2 >> 1);
    r.dc = fma((double)jc + ((rt.npix2 & 1) ? 0.5 : 0.0), r.dphi, -phi);
    r.Zs = r.s * z0;
    r.Wz = s0 * z;
    r.Di = z * s0 - r.s * z0;
    return r;
}

// exp(2i chi) of a pair in FP64 without trigonometric functions of its
// angles: sin D and 1 - cos D by their Taylor series (narrow: |D| <=
// kShortOffset, truncated below 3e-17 relative), then phasor's w, turned by
// psi.  About 45 FP64 instructions, against some 600 of the reference chain's
// arccosines, arctangents, sines and cosines, on a GPU that issues one FP64
// instruction in the time of 64 FP32 ones.
__device__ __forceinline__ void phasor_exact(const RingD& R, double kf, bool narrow, double s0,
                                             double c2p, double s2p, double& c2, double& s2)
{
    const double x = fma(kf, R.dphi, R.dc);
    double sn, h;
    if (narrow) {
        const double x2 = x * x;
        sn = fma(x2, 1.0 / 362880.0, -1.0 / 5040.0);
        sn = fma(x2, sn, 1.0 / 120.0);
        sn = fma(x2, sn, -1.0 / 6.0);
        sn = fma(x * x2, sn, x);
        h = fma(x2, 1.0 / 3628800.0, -1.0 / 40320.0);
        h = fma(x2, h, 1.0 / 720.0);
        h = fma(x2, h, -1.0 / 24.0);
        h = x2 * fma(x2, h, 0.5);
    } else {
        double cs;
        sincos(x, &sn, &cs);
        h = cs > 0.0 ? sn * sn / (1.0 + cs) : 1.0 - cs;
    }
    const double u = R.s * sn, v = fma(R.Zs, h, R.Di);
    const double nb = s0 * sn, db = fma(R.Wz, h, -R.Di);
    const double wr = fma(db, v, -(nb * u)), wi = fma(db, u, nb * v);
    const double rr = wr * wr;
    const double iw = 1.0 / fma(wi, wi, rr);
    const double er = fma(-wi, wi, rr) * iw, ei = wr * wi * (iw + iw);
    c2 = fma(er, c2p, -(ei * s2p));
    s2 = fma(ei, c2p, er * s2p);
}

// ring_exact and phasor_exact in two-float arithmetic.  The anchor's offset is
// near - f - e pixels (RingPlace).
__device__ __forceinline__ RingF ring_two_float(float near, float f, float e, const RingT& rt,
                                                FF z0, FF s0)
{
    RingF r;
    r.dphi = FF{rt.dphi, rt.dphi_lo};
    r.dc = (ff_sum(near, -f) + FF{-e, 0.0f}) * r.dphi;
    r.s = FF{rt.s, rt.s_lo};
    const FF z = FF{rt.z, rt.z_lo};
    r.Zs = r.s * z0;
    r.Wz = s0 * z;
    r.Di = z * s0 - r.Zs;
    return r;
}

// exp(2i chi) rounded to FP32: its error before that rounding, some 1e-12 at
// rho of a degree, is far below what moves the rounded value.  About 240 FP32
// instructions, the time of four FP64 ones; the 45 FP64 instructions of
// phasor_exact took two thirds of a PLAIN launch.  Within 1/8 rad (narrow) and
// within 1/2 (middle) sin x and 1 - cos x are good to 4e-13, by one series whose
// third term takes a second float in the middle range (with one it left 1e-10
// there); beyond, FP64's sincos (20,000 samples at 60 to 74 degrees, 5 degree
// beam: 145 us, 350 with sincos from 1/8 on).
__device__ __forceinline__ void phasor_two_float(const RingF& R, float kf, bool narrow, bool middle,
                                                 FF s0, FF c2p, FF s2p, float& c2, float& s2)
{
    const FF x = kf * R.dphi + R.dc;
    FF sn, h;
    if (narrow || middle) {
        const FF x2 = x * x;
        // sin x = x + x (x2 (-1/6 + x2 (1/120 + x2 p)))
        // 1 - cos x = x2 (1/2 + x2 (-1/24 + x2 (1/720 + x2 q)))
        const float p = fmaf(x2.h, fmaf(x2.h, -2.50521084e-8f, 2.75573192e-6f), -1.98412698e-4f);
        const float q = fmaf(x2.h, fmaf(x2.h, -2.08767570e-9f, 2.75573192e-7f), -2.48015873e-5f);
        FF a, b;
        if (narrow) {
            a = ff_quick(-0.16666667f, fmaf(x2.h, fmaf(x2.h, p, 8.33333333e-3f), 4.9670537e-9f));
            b = ff_quick(-0.041666668f, fmaf(x2.h, fmaf(x2.h, q, 1.38888889e-3f), 1.2417634e-9f));
        } else {
            a = ff_horner(FF{-0.16666667f, 4.9670537e-9f}, x2,
                          ff_quick(8.33333377e-3f, fmaf(x2.h, p, -4.346172e-10f)));
            b = ff_horner(FF{-0.041666668f, 1.2417634e-9f}, x2,
                          ff_quick(1.38888892e-3f, fmaf(x2.h, q, -3.3631094e-11f)));
        }
        sn = ff_horner(x, x, x2 * a);
        h = x2 * ff_horner(FF{0.5f, 0.0f}, x2, b);
    } else {
        double s, c;
        sincos((double)x.h + (double)x.l, &s, &c);
        sn = ff(s);
        h = ff(c > 0.0 ? s * s / (1.0 + c) : 1.0 - c);
    }
    const FF u = R.s * sn, v = R.Zs * h + R.Di;
    const FF nb = s0 * sn, db = R.Wz * h - R.Di;
    const FF wr = db * v - nb * u, wi = db * u + nb * v;
    const FF rr = wr * wr, ii = wi * wi, n = rr + ii;
    // 1 / n: the reciprocal approximation and one Newton step
    const float y = rcp_approx(n.h);
    const float e = fmaf(-n.l, y, fmaf(-n.h, y, 1.0f));
    const FF iw = ff_quick(y, fmaf(e, e * y, e * y));
    const FF er = (rr - ii) * iw, ei = 2.0f * (wr * wi * iw);
    c2 = (er * c2p - ei * s2p).h;
    s2 = (ei * c2p + er * s2p).h;
}

// 1 << x, 0 for x outside [0, 32).
__device__ __forceinline__ unsigned bit_or_0(int x)
{
    unsigned r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(x));
    return r;
}

// (sin psi, cos psi) times a common factor near 1, in FP32, with the angle
// kept to about 2e-9: the rotation by psi multiplies every pair of a sample,
// so the rounding error of its angle is coherent over the sample's sum (an
// FP32 pair rounded once is off by up to 4e-8).  The uses are ratios, so the
// factor drops out.  The larger component runs over eight FP32 values; the
// one whose partner rounds best is kept.
__device__ __forceinline__ void psi_phasor(double s, double c, float& sf, float& cf)
{
    const bool swap = fabs(s) > fabs(c);
    const double big = swap ? s : c, small = swap ? c : s;
    // small / big as the sum of two FP32 values: the trials then run in FP32
    const double ratio = small / big;
    const float rh = (float)ratio, rl = (float)(ratio - (double)rh);
    const float b0 = (float)big;
    float bb = b0, bs = rh * b0, best = 1.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float b = b0 * (1.0f - 0.03125f * (float)i);
        const float r = rh * b;
        const float e = fabsf(fmaf(rl, b, fmaf(rh, b, -r)) * rcp_approx(b));
        if (e < best) {
            best = e;
            bb = b;
            bs = r;
        }
    }
    sf = swap ? bb : bs;
    cf = swap ? bs : bb;
}

__device__ __forceinline__ SamplePlan make_plan(const Hpx& hs, const Beam& B, double ra,
                                                double dec, double pa)
{
    SamplePlan sp;
    const double psi = -pa;
    if (!(isfinite(ra) && isfinite(dec) && isfinite(psi))) {
        sp.flags = kPlanBad;
        sp.full_lo = 1;
        sp.full_hi = 0;
        return sp;
    }
    const DiscPlan P = disc_plan(hs, PD_SUB(kHalfPi, dec), ra, B.rho_max, B.cosr);
    // Boresight frame.  The reference chain (sphtrigo.cpp:29-35) takes dec as
    // given; for cos(dec) < 0 the same point is (pi - dec, ra + pi), and the
    // chain's north direction then points the other way: its alpha is the
    // normalised frame's + pi, hence its sigma is - pi, while beta and
    // exp(2i chi) are unchanged.  So the geometry runs in the normalised frame
    // (s0 >= 0) with (sin psi, cos psi) negated, which adds exactly pi to
    // sigma.  ra is reduced mod 2pi (the anchor longitude of the rings).
    // The frame is disc_plan's (z0 = cos(theta), s0, phi, latitude
    // pi/2 - theta) whenever its reflection agrees with the sign of cos(dec),
    // which decides the flip as in the reference chain; they can differ
    // only within an ulp of the poles, where the frame is rebuilt from dec.
    const bool flip = fabs(dec) < 1.5707963 ? false : cos(dec) < 0.0;
    double z0d, s0d, phi_f, dec0;
    if (flip == P.flip) {
        z0d = P.z0;
        s0d = P.s0;
        phi_f = P.phi;
        dec0 = PD_SUB(kHalfPi, P.theta);
    } else {
        double sdec, cdec;
        sincos(dec, &sdec, &cdec);
        z0d = sdec;
        s0d = fabs(cdec);
        phi_f = fmodulo(flip ? ra + kPi : ra, kTwoPi);
        dec0 = atan2(z0d, s0d);
    }
    sp.phi_hi = (float)phi_f;
    sp.phi_lo = (float)(phi_f - (double)sp.phi_hi);
    sp.dec_hi = (float)dec0;
    sp.dec_lo = (float)(dec0 - (double)sp.dec_hi);
    sp.z0f = (float)z0d;
    sp.s0f = (float)s0d;
    double spsi, cpsi;
    sincos(psi, &spsi, &cpsi);
    sp.spsi = flip ? -spsi : spsi;
    sp.cpsi = flip ? -cpsi : cpsi;
    psi_phasor(sp.spsi, sp.cpsi, sp.sps, sp.cps);
    sp.z0 = P.z0;
    sp.xa = P.xa;
    sp.phi = P.phi;
    sp.ring_lo = (int)P.ring_lo;
    sp.ring_hi = (int)P.ring_hi;
    sp.full_lo = (int)P.full_lo;
    sp.full_hi = (int)P.full_hi;
    sp.flags = (P.all_sky ? kPlanAllSky : 0) | (flip == P.flip ? 0 : kPlanExact);
    return sp;
}

// Processes one sample from its plan.  A non-finite pointing gives NaN TOD
// (kSums) and no pairs.  With kSums the TOD is written to `o` now, or by the
// drain that redoes the sample's last queued pair.  nfall counts queued pairs
// (lane 0 only).  kCheck: the pairs' decisions are compared with the chain's
// (ck).  kBil: bilinear beam lookup (bilinear_f32; only the degenerate pairs are
// queued).
template <bool kCheck, bool kBil = false, class Smem, class Action>
__device__ __forceinline__ void sample_planned(const SamplePlan& SP, const Hpx& hs,
                                               const RingT* rings, const Hpx& hb, const Beam& B,
                                               double ra, double dec, double pa, const Out& o,
                                               Smem& S, Queue& Qs, int lane,
                                               unsigned int* err, Action& act,
                                               unsigned long long& nfall, Check& ck)
{
    RingC* W = S.r;
    const unsigned lt_mask = (1u << lane) - 1u, le_mask = 2u * lt_mask + 1u;
    // two pixels per lane (actions with pair2, nearest lookup)
    constexpr bool kUnits = HasPair2<Action>::value && !kBil;
    if (SP.flags & kPlanBad) {
        if (Action::kSums && lane == 0) {
            store_out(o.a, o.f64, o.idx, CUDART_NAN);
            store_out(o.b, o.f64, o.idx, CUDART_NAN);
        }
        return;
    }
    // claim the next slot; one still waiting on queued pairs is freed by
    // redoing the whole queue
    const int slot = Qs.cur;
    Qs.cur = slot + 1 == kPend ? 0 : slot + 1;
    if (S.p[slot].left > 0) flush<kBil>(hs, S, Qs, lane, err, act);
    if (lane == 0) {
        Pend& Ps = S.p[slot];
        Ps.ra = ra;
        Ps.dec = dec;
        Ps.psi = -pa;
        // a latitude near a pole loses digits in 1 / sin(theta)
        Ps.z0 = SP.z0;
        Ps.s0 = 1.0 / SP.xa;
        Ps.phi = SP.phi;
        Ps.spsi = SP.spsi;
        Ps.cpsi = SP.cpsi;
        Ps.plain = (SP.flags & kPlanExact) != 0 || SP.s0f < 0.01f;
        Ps.nside_beam = (int)hb.nside;
        Ps.fb_a = Ps.fb_b = 0.0;
        Ps.beam = B.beam;
        Ps.out_a = o.a;
        Ps.out_b = o.b;
        Ps.idx = o.idx;
        Ps.npix_beam = B.npix;
        Ps.left = 0;
        Ps.open = 1;
        Ps.f64 = o.f64;
        act.stash(Ps);
    }
    static_assert(sizeof(SamplePlan) == 6 * sizeof(float4), "plan copy");
    if (lane < 6)
        reinterpret_cast<float4*>(&S.plan)[lane] = reinterpret_cast<const float4*>(&SP)[lane];
    __syncwarp();
    if constexpr (Action::kSums) act.reset();
    const SamplePlan& PL = S.plan;
    if constexpr (IsExact<Action>::value) {
        // the frame in FP64; near a pole cos(dec) itself, not 1 / sin(theta)
        double s0 = S.p[slot].s0, z0 = PL.z0;
        if (PL.s0f < 0.5f || (PL.flags & kPlanExact)) {
            sincos(dec, &z0, &s0);
            s0 = fabs(s0);
        }
        if (lane == 0) {
            put(S.z0, z0);
            put(S.s0, s0);
            put(S.c2p, fma(PL.cpsi, PL.cpsi, -(PL.spsi * PL.spsi)));
            put(S.s2p, 2.0 * PL.spsi * PL.cpsi);
        }
        __syncwarp();
    }
    // what the pair loop reads on every pair, in registers
    const float R2 = B.rscale * B.rscale;
    const Frame F{PL.z0f, PL.s0f, R2 * PL.s0f, PL.sps, PL.cps};
    const float tiny = kTinyQ * R2;
    const F8* const beam = B.beam;
    const unsigned npix_beam = (unsigned)B.npix;

    // queues a near-edge pair per lane; redoes them 32 at a time in FP64
    auto queue = [&](bool fb, int pix) {
        const unsigned mk = __ballot_sync(kFull, fb);
        if (!mk) return;
        if (fb) {
            const int at = Qs.n + __popc(mk & lt_mask);
            S.q[at] = pix;
            S.qs[at] = (unsigned char)slot;
        }
        Qs.n += __popc(mk);
        if (lane == 0) {
            nfall += __popc(mk);
            S.p[slot].left += __popc(mk);
        }
        __syncwarp();
        if (Qs.n >= 32) drain<kBil>(hs, 32, S, Qs, lane, err, act);
    };

    for (int r0 = PL.full_lo; r0 <= PL.full_hi; r0 += 32) {
        const int ring = r0 + lane;
        int cnt = 0, items = 0;  // the ring's disc pixels; its lane slots
        bool wide = false;
        [[maybe_unused]] bool beyond = false;
        RingC rc;
        [[maybe_unused]] std::conditional_t<IsTwoFloat<Action>::value, RingF, RingD> rd;
        if (ring <= PL.full_hi) {
            const RingT rt = rings[ring - 1];
            const RingPlace g = place_ring(PL, rt);
            RingRange sp = fast_disc_ring(hs, PL, B.cosr, B.versr, ring, rt, g);
            const int nr = rt.npix2 >> 1;
            // every pixel of the ring's range must lie in the sky map:
            // checked here, once per ring, instead of once per pair
            if (sp.lo < 0 || sp.lo >= nr || sp.n < 0 || sp.n > nr || rt.start < 0 ||
                rt.start + (long long)nr > hs.npix) {
                record(err, kCheckSkyIndex);
                sp = RingRange{0, 0};
            }
            cnt = sp.n;
            if (cnt) {
                // the anchor: the pixel centre nearest to the boresight's longitude
                const float sh = (rt.npix2 & 1) ? 0.5f : 0.0f;
                const float near = floorf(g.f - sh + 0.5f);
                const int jc = g.at + (int)near;
                rc.dc = (((near + sh) - g.f) - g.e) * rt.dphi;
                rc.dphi = rt.dphi;
                rc.Ki = R2 * g.K;
                rc.s = rt.s;
                rc.Wz = F.s0 * rt.z;
                rc.Di = g.Di;
                rc.nr = nr;
                rc.start = rt.start;
                // offsets from the anchor, the range centred on it; a whole
                // ring starts half a turn from it
                if (cnt == nr) {
                    int lo = jc - (nr >> 1);
                    lo += lo < 0 ? nr : 0;
                    sp.lo = lo >= nr ? lo - nr : lo;
                }
                int kk = sp.lo - jc;
                const int mid = kk + (cnt >> 1);
                if (mid >= (nr >> 1) + 1) kk -= nr;
                else if (mid < -(nr >> 1)) kk += nr;
                rc.kc = 0x4B400000 + kk - sp.lo;
                if constexpr (IsTwoFloat<Action>::value)
                    rd = ring_two_float(near + sh, g.f, g.e, rt, S.z0, S.s0);
                else if constexpr (IsExact<Action>::value)
                    rd = ring_exact(hs, ring, jc, rt, PL, S.z0, S.s0);
                const int hi = sp.lo + cnt - 1;  // below 2^16: rings hold at most 2^15 pixels
                rc.ends = sp.lo | hi << 16;
                // two pixels per lane: ring indices 2m and 2m + 1, which are
                // neighbours in memory as well (a ring's pixels and its first
                // pixel are multiples of 4)
                rc.j0 = kUnits ? sp.lo & ~1 : sp.lo;
                items = kUnits ? (hi >> 1) - (sp.lo >> 1) + 1 : cnt;
                // (the anchor is within half a pixel of the boresight's longitude)
                const float far = ((float)max(-kk, kk + cnt - 1) + 0.5f) * rt.dphi;
                wide = far > kShortOffset;
                beyond = far > 0.5f;
            }
        }
        int incl = items;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(kFull, incl, 31);
        // the rings with pixels, packed in order: a lane's ring is then the
        // number of ring starts up to its slot, counted with one warp
        // reduction per iteration instead of a search through shared memory
        const unsigned some = __ballot_sync(kFull, items > 0);
        const int rings_here = __popc(some);
        int first = items > 0 ? incl - items : 0x7fffffff;  // first slot less this iteration's
        if (items > 0) {
            rc.j0 -= (kUnits ? 2 : 1) * first;
            W[__popc(some & lt_mask)] = rc;
            if constexpr (IsExact<Action>::value) S.rd[__popc(some & lt_mask)] = rd;
        }
        const bool narrow = !__any_sync(kFull, wide);
        [[maybe_unused]] bool middle = false;
        if constexpr (IsTwoFloat<Action>::value) middle = !__any_sync(kFull, beyond);
        __syncwarp();
        int k0 = -1;  // ring of the slot before this iteration's
        const int iters = (total + 31) >> 5;
        for (int it = 0; it < iters; ++it, first -= 32) {
            const unsigned starts = __reduce_or_sync(kFull, bit_or_0(first));
            const int k = k0 + __popc(starts & le_mask);
            k0 += __popc(starts);
            const int t = (it << 5) + lane;
            if constexpr (kUnits) {
                // the slots past the end repeat the last one, switched off
                const int tt = min(t, total - 1);
                const RingC& R = W[min(k, rings_here - 1)];
                const float4 R0 = *reinterpret_cast<const float4*>(&R.dc);
                const float4 R1 = *reinterpret_cast<const float4*>(&R.Wz);
                const int4 R3 = *reinterpret_cast<const int4*>(&R.nr);
                const int j = __float_as_int(R1.z) + 2 * tt;  // even, below 2 nr
                const int pix = R3.y + (int)min((unsigned)j, (unsigned)(j - R3.x));
                const float kf = __int_as_float(__float_as_int(R1.w) + j) - 12582912.0f;
                const bool v0 = t < total && j >= (R3.z & 0xffff);
                const bool v1 = t < total && j < (int)((unsigned)R3.z >> 16);
                const Spot2 p = locate2(kf, F, R0, R1.y, narrow);
                const CapPixel2 c = cap_pixel2(p);
                const bool fb0 = v0 && (c.near0 || p.q0 < tiny);
                const bool fb1 = v1 && (c.near1 || p.q1 < tiny);
                if constexpr (kCheck) {
                    const Pend& P = S.p[slot];
                    if (v0)
                        check_pair(hs, hb, P, pix, lo2(c.av), lo2(c.bv), lo2(c.cv), c.ir0, lo2(p.r),
                                   c.bp0, fb0, ck);
                    if (v1)
                        check_pair(hs, hb, P, pix + 1, hi2(c.av), hi2(c.bv), hi2(c.cv), c.ir1,
                                   hi2(p.r), c.bp1, fb1, ck);
                }
                const bool in0 = v0 && !fb0 && (unsigned)c.bp0 < npix_beam;
                const bool in1 = v1 && !fb1 && (unsigned)c.bp1 < npix_beam;
                Unit U;
                U.in0 = in0;
                U.in1 = in1;
                U.pix = pix;
                U.bp0 = in0 ? c.bp0 : 0;
                U.bp1 = in1 ? c.bp1 : 0;
                U.B0 = load_beam<Action::kL1>(beam + U.bp0);
                U.B1 = load_beam<Action::kL1>(beam + U.bp1);
                act.fetch2(pix, U.S0, U.S1);
                phasor2(p, F.s0, R1.x, R1.y, U.c, U.s);
                act.pair2(U);
                if constexpr (HasOutside<Action>::value) {
                    if (v0 && !fb0 && !in0) act.outside(pix, c.bp0);
                    if (v1 && !fb1 && !in1) act.outside(pix + 1, c.bp1);
                }
                if (__any_sync(kFull, fb0 || fb1)) {
#pragma unroll 1
                    for (int e = 0; e < 2; ++e) queue(e ? fb1 : fb0, pix + e);
                }
            } else {
            bool fb = false;
            int pix = 0;
            [[maybe_unused]] int bp = -1;
            [[maybe_unused]] float cos2 = 0.0f, sin2 = 0.0f;
            if (t < total) {
                const float4 R0 = *reinterpret_cast<const float4*>(&W[k].dc);
                const float4 R1 = *reinterpret_cast<const float4*>(&W[k].Wz);
                const int2 R3 = *reinterpret_cast<const int2*>(&W[k].nr);
                const int j = __float_as_int(R1.z) + t;  // ring index, below 2 nr
                pix = R3.y + (int)min((unsigned)j, (unsigned)(j - R3.x));
                const float kf = __int_as_float(__float_as_int(R1.w) + j) - 12582912.0f;
                const Spot p = locate(kf, F, R0, R1.y, narrow);
                fb = p.q < tiny;
                if constexpr (kBil && Action::kStencil) {
                    int px[4];
                    float w[4];
                    if (!fb && stencil_f32(B, p.qd, p.tp, p.r, px, w)) {
                        float c2, s2;
                        phasor(p, F.s0, R1.x, R1.y, c2, s2);
                        act.pair_stencil(pix, act.fetch(pix), px, w, c2, s2);
                    } else if constexpr (HasOutside<Action>::value) {
                        if (!fb) act.outside(pix, -1);
                    }
                } else if constexpr (kBil) {
                    F8 Bv;
                    if (!fb && bilinear_f32(B, p.qd, p.tp, p.r, Bv)) {
                        float c2, s2;
                        phasor(p, F.s0, R1.x, R1.y, c2, s2);
                        act.pair(pix, act.fetch(pix), Bv, -1, c2, s2);
                    } else if constexpr (HasOutside<Action>::value) {
                        if (!fb) act.outside(pix, -1);
                    }
                } else {
                    const CapPixel c = cap_pixel(p);
                    fb |= c.near;
                    if constexpr (kCheck)
                        check_pair(hs, hb, S.p[slot], pix, c.av, c.bv, c.cv, c.ir, p.r, c.bp, fb, ck);
                    if (!fb) {
                        if constexpr (IsExact<Action>::value) {
                            if ((unsigned)c.bp < (unsigned)B.npix) {
                                if constexpr (IsTwoFloat<Action>::value) {
                                    float c2, s2;
                                    phasor_two_float(S.rd[k], kf, narrow, middle, S.s0, S.c2p, S.s2p, c2, s2);
                                    act.pair64(pix, c.bp, c2, s2);
                                } else {
                                    double c2, s2;
                                    phasor_exact(S.rd[k], (double)kf, narrow, S.s0, S.c2p, S.s2p, c2, s2);
                                    act.pair64(pix, c.bp, c2, s2);
                                }
                            }
                        } else if ((unsigned)c.bp < (unsigned)B.npix) {  // 0 <= bp < npix
                            float c2, s2;
                            phasor(p, F.s0, R1.x, R1.y, c2, s2);
                            if constexpr (HasPairAll<Action>::value) {
                                bp = c.bp;
                                cos2 = c2;
                                sin2 = s2;
                            } else {
                                act.pair(pix, act.fetch(pix), load_beam(B.beam + c.bp), c.bp, c2, s2);
                            }
                        } else if constexpr (HasOutside<Action>::value) {
                            act.outside(pix, c.bp);
                        }
                    }
                }
            }
            if constexpr (HasPairAll<Action>::value && !kBil) act.pair_all(pix, bp, cos2, sin2);
            queue(fb, pix);
            }
        }
        __syncwarp();
    }
    if constexpr (Action::kSums) {
        double ta, tb;
        act.total(ta, tb);
        if (lane == 0) {
            Pend& Ps = S.p[slot];
            Ps.main_a = ta;
            Ps.main_b = tb;
            Ps.open = 0;
            if (Ps.left == 0) finalize(Ps);
        }
    } else if (lane == 0) {
        S.p[slot].open = 0;
    }
    __syncwarp();
}

// Processes one sample, its plan built here by the warp.
template <bool kCheck, bool kBil = false, class Smem, class Action>
__device__ __forceinline__ void sample(const Hpx& hs, const RingT* rings, const Hpx& hb,
                                       const Beam& B, double ra, double dec, double pa,
                                       const Out& o, Smem& S, Queue& Qs, int lane,
                                       unsigned int* err, Action& act, unsigned long long& nfall,
                                       Check& ck)
{
    sample_planned<kCheck, kBil>(make_plan(hs, B, ra, dec, pa), hs, rings, hb, B, ra, dec, pa, o,
                                 S, Qs, lane, err, act, nfall, ck);
}

// Adds a lane's findings to *out (every lane of the warp calls).
__device__ __forceinline__ void report(const Check& ck, CheckOut* out)
{
    // both errors are >= 0, so their bits order as they do
    atomicMax(&out->fp32, __float_as_int(ck.fp32));
    atomicMax(&out->fp64, __float_as_int(ck.fp64));
    atomicAdd(&out->pairs, ck.pairs);
    atomicAdd(&out->differ, ck.differ);
}

// Forward action: gather the sky, multiply by the beam, compensated sums of
// both detectors side by side (two_sum2).
template <bool kBeamL1>
struct Gather {
    static constexpr bool kL1 = kBeamL1;  // load_beam
    static constexpr bool kSums = true;
    static constexpr bool kStencil = false;
    const float4* sky;
    bool wide;       // sky is 32-byte aligned
    F32x2 sum, cmp;  // halves: detector a, detector b
    __device__ __forceinline__ void reset() { sum = cmp = pack2(0.0f, 0.0f); }
    __device__ __forceinline__ float4 fetch(int pix) const { return __ldg(&sky[pix]); }
    // the sky's polarisation turned into the beam's frame once for both detectors;
    // I, mostly the largest, comes last, so that a pair is rounded once at its
    // magnitude: with I of 100 and Q, U of 10 at nside 64 and 5 degrees the totals
    // are off by 6.9e-9 of the TOD's spread, with I first 1.15e-8, for 0.3 % of
    // the time (400,000 samples at nside 1024: 16.63 -> 16.68 ms)
    __device__ __forceinline__ static void contrib(const float4& S, const F8& B, float c2, float s2,
                                                  float& ta, float& tb)
    {
        const float q = fmaf(S.y, c2, S.z * s2), u = fmaf(S.z, c2, -(S.y * s2));
        ta = fmaf(S.x, B.a.x, fmaf(q, B.a.y, fmaf(u, B.a.z, S.w * B.a.w)));
        tb = fmaf(S.x, B.b.x, fmaf(-q, B.b.y, fmaf(-u, B.b.z, S.w * B.b.w)));
    }
    __device__ __forceinline__ void pair(int, const float4& S, const F8& B, int, float c2, float s2)
    {
        float ta, tb;
        contrib(S, B, c2, s2, ta, tb);
        two_sum2(sum, cmp, pack2(ta, tb));
    }
    // sky pixels pix (even) and pix + 1: one 256-bit load when the map is
    // 32-byte aligned (a caller's own map need only be 16-byte aligned)
    __device__ __forceinline__ void fetch2(int pix, float4& S0, float4& S1) const
    {
        const float4* p = sky + pix;
        if (wide) {
            load_sky2(p, S0, S1);
        } else {
            S0 = __ldg(p);
            S1 = __ldg(p + 1);
        }
    }
    // two pairs; one that is off adds nothing
    __device__ __forceinline__ void pair2(const Unit& U)
    {
        float a0, b0, a1, b1;
        contrib(U.S0, U.B0, lo2(U.c), lo2(U.s), a0, b0);
        contrib(U.S1, U.B1, hi2(U.c), hi2(U.s), a1, b1);
        if (!U.in0) a0 = b0 = 0.0f;
        if (!U.in1) a1 = b1 = 0.0f;
        two_sum2(sum, cmp, pack2(a0, b0));
        two_sum2(sum, cmp, pack2(a1, b1));
    }
    __device__ __forceinline__ void stash(Pend&) const {}
    __device__ __forceinline__ void deferred(const Pend&, int pix, const F8& B, int, float c2, float s2,
                                            float& ta, float& tb) const
    {
        contrib(fetch(pix), B, c2, s2, ta, tb);
    }
    // warp total (fixed shuffle tree: deterministic)
    __device__ __forceinline__ void total(double& a, double& b) const
    {
        float sa, sb, ca, cb;
        unpack2(sum, sa, sb);
        unpack2(cmp, ca, cb);
        a = (double)sa + (double)ca;
        b = (double)sb + (double)cb;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(kFull, a, o);
            b += __shfl_xor_sync(kFull, b, o);
        }
    }
};

}  // namespace tuned
}  // namespace pisco

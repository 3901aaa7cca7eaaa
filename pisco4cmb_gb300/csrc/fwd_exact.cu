// fwd_exact.cu -- the PLAIN and FP64 forms with the nearest beam lookup, for
// beams in the TUNED geometry's domain.
//
// Same result as the reference chain (convolver.cpp:112-221) pair by pair: the
// disc and the beam pixel of every pair are the chain's (tuned_core.cuh: FP32
// decisions, every one near an edge redone in FP64), and the phasor
// exp(2i chi) is formed from the pair's offsets, for the FP64 form in FP64, for
// PLAIN, which rounds it to float as the reference does, in two-float
// arithmetic.  PLAIN multiplies in FP32, the FP64 form in FP64; both accumulate
// in FP64.
//
// What bounds it: the FP64 pipe, which takes 16 cycles per warp instruction on
// an SM (FP64 form 83 % busy).  plain_kernel (fwd_plain.cu) evaluates the chain's
// ten transcendental functions for every pair, about 600 FP64 instructions; here
// a pair takes about 56 (FP64 form) or, with some 240 FP32 ones, 4 (PLAIN), which
// at 93 pairs per sample has the FP64 pipe 60 % busy and issues in 46 % of the
// cycles.  nside 64, 5 degree beam, PLAIN, 20,000 samples: 2.1 ms in
// plain_kernel, 373 us with the FP64 phasor, 120 us now; nside 2048, 1 degree,
// FP64 form, 6,001 samples: 21.3 -> 2.9 ms.  The bilinear lookup and beams outside
// the domain stay on plain_kernel.
#include "tuned_core.cuh"

namespace pisco {
namespace {

constexpr int kEW = 8;  // warps per block, two blocks per SM

// FP64 accumulation and a fixed shuffle tree (deterministic).
struct GatherSums {
    static constexpr bool kSums = true;
    static constexpr bool kStencil = false;
    double acc_a, acc_b;
    __device__ __forceinline__ void reset() { acc_a = acc_b = 0.0; }
    __device__ __forceinline__ void stash(tuned::Pend&) const {}
    __device__ __forceinline__ void total(double& a, double& b) const
    {
        a = acc_a;
        b = acc_b;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(tuned::kFull, a, o);
            b += __shfl_xor_sync(tuned::kFull, b, o);
        }
    }
};

struct GatherF64 : GatherSums {
    using Smem = tuned::ExactSmem;
    const D4* sky;
    const D8* beam;
    __device__ __forceinline__ explicit GatherF64(const FwdArgs& a) : sky(a.sky64), beam(a.beam64) {}
    __device__ __forceinline__ void deferred64(int pix, int bp, double c2, double s2, double& ta,
                                               double& tb) const
    {
        const D4 S = sky[pix];
        const D8 B = beam[bp];
        const double q = S.y * c2 + S.z * s2, u = S.z * c2 - S.y * s2;
        ta = S.x * B.a.x + q * B.a.y + u * B.a.z + S.w * B.a.w;
        tb = S.x * B.b.x - q * B.b.y - u * B.b.z + S.w * B.b.w;
    }
    __device__ __forceinline__ void pair64(int pix, int bp, double c2, double s2)
    {
        double ta, tb;
        deferred64(pix, bp, c2, s2, ta, tb);
        acc_a += ta;
        acc_b += tb;
    }
};

struct GatherPlain : GatherSums {
    using Smem = tuned::PlainSmem;
    using TwoFloat = void;
    const float4* sky;
    const F8* beam;
    __device__ __forceinline__ explicit GatherPlain(const FwdArgs& a) : sky(a.sky32), beam(a.beam32) {}
    __device__ __forceinline__ void contrib(int pix, int bp, float c2, float s2, float& ta,
                                            float& tb) const
    {
        const float4 S = __ldg(&sky[pix]);
        const F8 B = tuned::load_beam<true>(beam + bp);
        // the rounding of plain_kernel's products, fused as nvcc fuses the
        // reference's expressions there: PLAIN's TOD stays the same
        const float t1 = fmaf(B.a.y, c2, -(B.a.z * s2)), t2 = fmaf(B.a.z, c2, B.a.y * s2);
        const float u1 = fmaf(B.b.z, s2, -(B.b.y * c2)), u2 = fmaf(-B.b.z, c2, -(B.b.y * s2));
        ta = fmaf(S.w, B.a.w, fmaf(S.z, t2, fmaf(S.x, B.a.x, S.y * t1)));
        tb = fmaf(S.w, B.b.w, fmaf(S.z, u2, fmaf(S.x, B.b.x, S.y * u1)));
    }
    __device__ __forceinline__ void deferred64(int pix, int bp, double c2, double s2, double& ta,
                                               double& tb) const
    {
        float a, b;
        contrib(pix, bp, (float)c2, (float)s2, a, b);
        ta = (double)a;
        tb = (double)b;
    }
    __device__ __forceinline__ void pair64(int pix, int bp, float c2, float s2)
    {
        float a, b;
        contrib(pix, bp, c2, s2, a, b);
        acc_a += (double)a;
        acc_b += (double)b;
    }
};

// kPlanned: plans holds the plans of positions [pos0, pos1); otherwise each
// warp builds its own (the same values).
// kCheck: the pairs' decisions are compared with the chain's (*check).
template <class Act, bool kPlanned, bool kCheck>
__global__ void __launch_bounds__(kEW * 32, 2)
    exact_kernel(FwdArgs a, CheckOut* check, const tuned::SamplePlan* __restrict__ plans, long long pos0,
                 long long pos1)
{
    __shared__ typename Act::Smem sm[kEW];
    __shared__ Hpx s_hs, s_hb;
    __shared__ tuned::Beam s_B;
    const int lane = threadIdx.x & 31;
    typename Act::Smem& S = sm[threadIdx.x >> 5];
    if (threadIdx.x == 0) {
        s_hs = hpx_make(a.nside_sky);
        s_hb = hpx_make(a.nside_beam);
        s_B = tuned::make_beam(a.beam32, a.nside_beam, a.npix_beam, a.rho_max);
    }
    __syncthreads();
    unsigned long long nfall = 0;
    tuned::Check ck;
    Act g(a);
    tuned::Queue Q{0, 0};
    const long long gw = (long long)blockIdx.x * kEW + (threadIdx.x >> 5);
    const long long nw = (long long)gridDim.x * kEW;
    for (long long i = pos0 + gw; i < pos1; i += nw) {
        const long long j = a.order ? (long long)a.order[i] : i;  // sample of position i
        const long long s = a.begin + j;
        const tuned::Out o{a.out_a, a.out_b, j, a.out_f64};
        const double ra = a.ra[s], dec = a.dec[s], pa = a.pa[s];
        if constexpr (kPlanned)
            tuned::sample_planned<kCheck>(plans[i - pos0], s_hs, a.rings, s_hb, s_B, ra, dec, pa, o,
                                         S, Q, lane, a.err, g, nfall, ck);
        else
            tuned::sample<kCheck>(s_hs, a.rings, s_hb, s_B, ra, dec, pa, o, S, Q, lane, a.err, g,
                                 nfall, ck);
    }
    tuned::flush_block(s_hs, sm, kEW, Q, lane, a.err, g);
    if constexpr (kCheck) tuned::report(ck, check);
}

template <class Act, bool kPlanned, bool kCheck = false>
void launch_form(const FwdArgs& a, int sm_count, cudaStream_t st, tuned::SamplePlan* plans,
                 long long plan_cap, CheckOut* check = nullptr)
{
    const long long step = kPlanned ? plan_cap : a.n;
    for (long long p0 = 0; p0 < a.n; p0 += step) {
        const long long p1 = p0 + step < a.n ? p0 + step : a.n;
        if (kPlanned) launch_plans(a, plans, p0, p1, st);
        const long long need = (p1 - p0 + kEW - 1) / kEW, most = 2LL * sm_count;
        exact_kernel<Act, kPlanned, kCheck>
            <<<(int)(most < need ? most : need), kEW * 32, 0, st>>>(a, check, plans, p0, p1);
    }
}

}  // namespace

cudaError_t launch_forward_exact(const FwdArgs& a, bool f64, int sm_count, cudaStream_t st,
                                 void* plans, long long plan_cap)
{
    if (a.n <= 0) return cudaSuccess;
    tuned::SamplePlan* p = static_cast<tuned::SamplePlan*>(plans);
    if (p && plan_cap > 0) {
        if (f64) launch_form<GatherF64, true>(a, sm_count, st, p, plan_cap);
        else launch_form<GatherPlain, true>(a, sm_count, st, p, plan_cap);
    } else {
        if (f64) launch_form<GatherF64, false>(a, sm_count, st, nullptr, 0);
        else launch_form<GatherPlain, false>(a, sm_count, st, nullptr, 0);
    }
    return cudaGetLastError();
}

cudaError_t launch_exact_check(const FwdArgs& a, bool f64, int sm_count, cudaStream_t st,
                               CheckOut* check)
{
    if (a.n <= 0) return cudaSuccess;
    if (f64) launch_form<GatherF64, false, true>(a, sm_count, st, nullptr, 0, check);
    else launch_form<GatherPlain, false, true>(a, sm_count, st, nullptr, 0, check);
    return cudaGetLastError();
}

}  // namespace pisco

// fwd_exact.cu -- the PLAIN and FP64 forms with the nearest beam lookup, for
// beams in the TUNED geometry's domain.
//
// Same result as the reference chain (convolver.cpp:112-221) pair by pair: the
// disc and the beam pixel of every pair are the chain's (tuned_core.cuh: FP32
// decisions, every one near an edge redone with the chain itself), and the
// phasor exp(2i chi) is formed in FP64 from the pair's offsets.  PLAIN rounds
// it to float and multiplies in FP32 as the reference does, the FP64 form
// multiplies in FP64; both accumulate in FP64.
//
// What bounds it: the FP64 pipe, which takes 16 cycles per warp instruction on
// an SM.  plain_kernel (fwd_plain.cu) evaluates the chain's ten transcendental
// functions for every pair, about 600 FP64 instructions; here a pair takes
// about 60 (FP64 form) or 50 (PLAIN).  The bilinear lookup and beams outside
// the domain stay on plain_kernel.
#include "tuned_core.cuh"

namespace pisco {
namespace {

constexpr int kEW = 8;  // warps per block, two blocks per SM

template <bool F64>
struct GatherExact {
    static constexpr bool kSums = true;
    static constexpr bool kStencil = false;
    const float4* sky32;
    const D4* sky64;
    const F8* beam32;
    const D8* beam64;
    double acc_a, acc_b;
    __device__ __forceinline__ void reset() { acc_a = acc_b = 0.0; }
    __device__ __forceinline__ void stash(tuned::Pend&) const {}
    __device__ __forceinline__ void contrib(int pix, int bp, double c2d, double s2d, double& ta,
                                            double& tb) const
    {
        if constexpr (F64) {
            const D4 S = sky64[pix];
            const D8 B = beam64[bp];
            const double q = S.y * c2d + S.z * s2d, u = S.z * c2d - S.y * s2d;
            ta = S.x * B.a.x + q * B.a.y + u * B.a.z + S.w * B.a.w;
            tb = S.x * B.b.x - q * B.b.y - u * B.b.z + S.w * B.b.w;
        } else {
            const float4 S = __ldg(&sky32[pix]);
            const F8 B = tuned::load_beam<true>(beam32 + bp);
            const float c2 = (float)c2d, s2 = (float)s2d;
            // the rounding of plain_kernel's products, fused as nvcc fuses the
            // reference's expressions there: PLAIN's TOD stays the same bit for bit
            const float t1 = fmaf(B.a.y, c2, -(B.a.z * s2)), t2 = fmaf(B.a.z, c2, B.a.y * s2);
            const float u1 = fmaf(B.b.z, s2, -(B.b.y * c2)), u2 = fmaf(-B.b.z, c2, -(B.b.y * s2));
            ta = (double)fmaf(S.w, B.a.w, fmaf(S.z, t2, fmaf(S.x, B.a.x, S.y * t1)));
            tb = (double)fmaf(S.w, B.b.w, fmaf(S.z, u2, fmaf(S.x, B.b.x, S.y * u1)));
        }
    }
    __device__ __forceinline__ void pair64(int pix, int bp, double c2, double s2)
    {
        double ta, tb;
        contrib(pix, bp, c2, s2, ta, tb);
        acc_a += ta;
        acc_b += tb;
    }
    __device__ __forceinline__ void deferred64(int pix, int bp, double c2, double s2, double& ta,
                                               double& tb) const
    {
        contrib(pix, bp, c2, s2, ta, tb);
    }
    // warp total (fixed shuffle tree: deterministic)
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

// kPlanned: plans holds the plans of positions [pos0, pos1); otherwise each
// warp builds its own (the same values).
template <bool F64, bool kPlanned>
__global__ void __launch_bounds__(kEW * 32, 2)
    exact_kernel(FwdArgs a, const tuned::SamplePlan* __restrict__ plans, long long pos0,
                 long long pos1)
{
    __shared__ tuned::ExactSmem sm[kEW];
    __shared__ Hpx s_hs, s_hb;
    __shared__ tuned::Beam s_B;
    const int lane = threadIdx.x & 31;
    tuned::ExactSmem& S = sm[threadIdx.x >> 5];
    if (threadIdx.x == 0) {
        s_hs = hpx_make(a.nside_sky);
        s_hb = hpx_make(a.nside_beam);
        s_B = tuned::make_beam(a.beam32, a.nside_beam, a.npix_beam, a.rho_max);
    }
    __syncthreads();
    unsigned long long nfall = 0, npairs = 0;
    float cmax = 0.0f;
    GatherExact<F64> g;
    g.sky32 = a.sky32;
    g.sky64 = a.sky64;
    g.beam32 = a.beam32;
    g.beam64 = a.beam64;
    tuned::Queue Q{0, 0};
    const long long gw = (long long)blockIdx.x * kEW + (threadIdx.x >> 5);
    const long long nw = (long long)gridDim.x * kEW;
    for (long long i = pos0 + gw; i < pos1; i += nw) {
        const long long j = a.order ? (long long)a.order[i] : i;  // sample of position i
        const long long s = a.begin + j;
        const tuned::Out o{a.out_a, a.out_b, j, a.out_f64};
        const double ra = a.ra[s], dec = a.dec[s], pa = a.pa[s];
        if constexpr (kPlanned)
            tuned::sample_planned<false>(plans[i - pos0], s_hs, a.rings, s_hb, s_B, ra, dec, pa, o,
                                         S, Q, lane, a.err, g, nfall, cmax, npairs);
        else
            tuned::sample<false>(s_hs, a.rings, s_hb, s_B, ra, dec, pa, o, S, Q, lane, a.err, g,
                                 nfall, cmax, npairs);
    }
    tuned::flush_block(s_hs, sm, kEW, Q, lane, a.err, g);
}

template <bool F64, bool kPlanned>
void launch_form(const FwdArgs& a, int sm_count, cudaStream_t st, tuned::SamplePlan* plans,
                 long long plan_cap)
{
    const long long step = kPlanned ? plan_cap : a.n;
    for (long long p0 = 0; p0 < a.n; p0 += step) {
        const long long p1 = p0 + step < a.n ? p0 + step : a.n;
        if (kPlanned) launch_plans(a, plans, p0, p1, st);
        const long long need = (p1 - p0 + kEW - 1) / kEW, most = 2LL * sm_count;
        exact_kernel<F64, kPlanned>
            <<<(int)(most < need ? most : need), kEW * 32, 0, st>>>(a, plans, p0, p1);
    }
}

}  // namespace

cudaError_t launch_forward_exact(const FwdArgs& a, bool f64, int sm_count, cudaStream_t st,
                                 void* plans, long long plan_cap)
{
    if (a.n <= 0) return cudaSuccess;
    tuned::SamplePlan* p = static_cast<tuned::SamplePlan*>(plans);
    if (p && plan_cap > 0) {
        if (f64) launch_form<true, true>(a, sm_count, st, p, plan_cap);
        else launch_form<false, true>(a, sm_count, st, p, plan_cap);
    } else {
        if (f64) launch_form<true, false>(a, sm_count, st, nullptr, 0);
        else launch_form<false, false>(a, sm_count, st, nullptr, 0);
    }
    return cudaGetLastError();
}

}  // namespace pisco

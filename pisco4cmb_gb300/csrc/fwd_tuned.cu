// fwd_tuned.cu -- TUNED forward, one detector pair per launch.
//
// Same result as the reference chain (convolver.cpp:112-221) pair by pair,
// with FP32 per-pair geometry; see tuned_core.cuh for the geometry and the
// FP64 re-evaluation of near-edge decisions.  GB300 runs FP64 at a small
// fraction of its FP32 rate, so the reference's per-pair FP64
// transcendentals (about ten per pair) cannot stay on the hot path.
//
// One warp per sample, grid sized to the resident warps of the GPU and
// strided over samples; per-lane compensated FP32 sums, fixed shuffle-tree
// reduction (bit-reproducible).
#include "tuned_core.cuh"

namespace pisco {
namespace {

// Launch shape: the nearest lookup runs one block of 20 warps per SM (register
// cap 96, no spills), two pixels per lane: its pair loop is bound by the L1
// pipe (87 % busy at 1.1 MB of beam: the beam gather, the sky and the rings'
// constants), and 20 warps leave L1 156 KB.  100,000 samples of nside 1024 and
// a 3 degree beam: 16 warps 4.53 ms, 20 warps 4.31 ms, 24 warps (80 registers,
// spilling) 4.47 ms; one pixel per lane at 32 warps of 64 registers took 5.2
// ms.  The warps of a block work on consecutive samples, whose discs overlap,
// so their sky reads share L1.  The bilinear lookup, which needs more
// registers per pair, runs 8 x 2.
#ifndef PISCO_FWD_WARPS
#define PISCO_FWD_WARPS 20
#endif
#ifndef PISCO_BIL_WARPS
#define PISCO_BIL_WARPS 8
#endif

// Where a launch's sample plans come from: each warp builds its own, an array
// built beforehand by plan_kernel, or the block's first warp, one plan per lane
// (a short launch: at most 32 samples per block).
enum Plans { kOwnPlans, kArrayPlans, kBlockPlans };

// kBil: bilinear beam lookup (the PLAIN form's get_interpol stencil in FP32).
// kTW: warps per block (fwd_warps_per_sm / kTW blocks per SM).
// Positions [pos0, pos1) of the launch; plans (kArrayPlans): theirs, index
// position - pos0.
// Warps per SM: 20 for the planned nearest lookup (register cap 96), 16 for
// the others (cap 128).
template <bool kBil, Plans kPlans>
constexpr int fwd_warps_per_sm()
{
    return kPlans != kOwnPlans && !kBil ? PISCO_FWD_WARPS : 16;
}

template <bool kCheck, bool kBil, int kTW, Plans kPlans>
__global__ void __launch_bounds__(kTW * 32, fwd_warps_per_sm<kBil, kPlans>() / kTW)
    tuned_kernel(FwdArgs a, CheckOut* check, const tuned::SamplePlan* __restrict__ plans,
                 long long pos0, long long pos1)
{
    __shared__ tuned::WarpSmem sm[kTW];
    const int lane = threadIdx.x & 31;
    tuned::WarpSmem& S = sm[threadIdx.x >> 5];
    // The grids' and the beam's descriptors are in shared memory, read once
    // per sample rather than held in registers across the pair loop, which
    // leaves those to the pair geometry.  The bilinear lookup, which reads the
    // beam's on every stencil pixel, takes that one from the kernel's arguments
    // (100,003 samples of nside 1024 and 3 degrees: 12.5 ms; copied from shared
    // memory into registers 17.8, the sky's from the arguments too 12.7).
    constexpr bool kDescSmem = !kBil;
    __shared__ Hpx s_hs, s_hb;
    __shared__ tuned::Beam s_B;
    if (threadIdx.x == 0) {
        s_hs = hpx_make(a.nside_sky);
        s_hb = hpx_make(a.nside_beam);
        s_B = tuned::make_beam(a.beam32, a.nside_beam, a.npix_beam, a.rho_max);
    }
    __syncthreads();
    const Hpx rhb = hpx_make(a.nside_beam);
    const tuned::Beam rB{a.beam32, a.nside_beam, a.npix_beam, a.rho_max, s_B.cosr, s_B.versr, s_B.rscale};
    const Hpx& hs = s_hs;
    const Hpx& hb = kDescSmem ? s_hb : rhb;
    const tuned::Beam& B = kDescSmem ? s_B : rB;
    // the warp's positions: first, first + step, ...; a short launch gives each
    // block a contiguous share
    long long first = pos0 + (long long)blockIdx.x * kTW + (threadIdx.x >> 5);
    long long step = (long long)gridDim.x * kTW, end = pos1, lo = 0;
    if constexpr (kPlans == kBlockPlans) {
        const int n = (int)(pos1 - pos0), g = gridDim.x, b = blockIdx.x;
        lo = pos0 + n / g * b + min(b, n % g);
        end = lo + n / g + (b < n % g ? 1 : 0);
        first = lo + (threadIdx.x >> 5);
        step = kTW;
    }
    unsigned long long nfall = 0;
    tuned::Check ck;
    tuned::Gather<true> g;
    g.sky = a.sky32;
    g.wide = (reinterpret_cast<size_t>(a.sky32) & 31) == 0;
    tuned::Queue Q{0, 0};
    __shared__ tuned::SamplePlan s_plans[kPlans == kBlockPlans ? 32 : 1];
    if constexpr (kPlans == kBlockPlans) {
        if (threadIdx.x < 32) {
            const long long i = lo + lane;
            if (i < end) {
                const long long s = a.begin + (a.order ? (long long)a.order[i] : i);
                s_plans[lane] = tuned::make_plan(hs, B, a.ra[s], a.dec[s], a.pa[s]);
            }
        }
        __syncthreads();
    }
    for (long long i = first; i < end; i += step) {
        const long long j = a.order ? (long long)a.order[i] : i;  // sample of position i
        const long long s = a.begin + j;
        const tuned::Out o{a.out_a, a.out_b, j, a.out_f64};
        const double ra = a.ra[s], dec = a.dec[s], pa = a.pa[s];
        if constexpr (kPlans != kOwnPlans)
            tuned::sample_planned<kCheck, kBil>(kPlans == kBlockPlans ? s_plans[i - lo] : plans[i - pos0],
                                                hs, a.rings, hb, B, ra, dec, pa, o,
                                                S, Q, lane, a.err, g, nfall, ck);
        else
            tuned::sample<kCheck, kBil>(hs, a.rings, hb, B, ra, dec, pa, o, S, Q, lane, a.err, g,
                                        nfall, ck);
    }
    tuned::flush_block<kBil>(hs, sm, kTW, Q, lane, a.err, g);
    if (lane == 0 && nfall && a.fallbacks) atomicAdd(a.fallbacks, nfall);
    if constexpr (kCheck) tuned::report(ck, check);
}

// The sample plans of positions [pos0, pos1), one thread per sample.
__global__ void plan_kernel(FwdArgs a, tuned::SamplePlan* __restrict__ plans, long long pos0,
                            long long pos1)
{
    __shared__ Hpx hs;
    __shared__ tuned::Beam B;
    if (threadIdx.x == 0) {
        hs = hpx_make(a.nside_sky);
        B = tuned::make_beam(a.beam32, a.nside_beam, a.npix_beam, a.rho_max);
    }
    __syncthreads();
    for (long long i = pos0 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < pos1;
         i += (long long)gridDim.x * blockDim.x) {
        const long long j = a.order ? (long long)a.order[i] : i;
        const long long s = a.begin + j;
        plans[i - pos0] = tuned::make_plan(hs, B, a.ra[s], a.dec[s], a.pa[s]);
    }
}
static_assert(sizeof(tuned::SamplePlan) == kSamplePlanBytes, "sample plan size");

__global__ void ring_table_kernel(int nside, RingT* rings)
{
    const Hpx h = hpx_make(nside);
    const long long nr = 4LL * nside - 1;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x + 1; r <= nr;
         r += (long long)gridDim.x * blockDim.x) {
        const RingInfo ri = ring_info(h, r);
        const double z = ring2z(h, r);
        const double s = sqrt(PD_MUL(PD_SUB(1.0, z), PD_ADD(1.0, z)));
        RingT t;
        const double dec = atan2(z, s), fr = PD_MUL((double)ri.npix, kInvTwoPi);
        t.dec_hi = (float)dec;
        t.dec_lo = (float)(dec - (double)t.dec_hi);
        t.fr_hi = (float)fr;
        t.fr_lo = (float)(fr - (double)t.fr_hi);
        // near a pole sin(theta) from i^2 / (3 nside^2): 1 - z has lost digits
        const double i = (double)(r <= 2 * h.nside ? r : 4 * h.nside - r), t2 = i * i * h.fact2;
        const double sx = i < (double)h.nside ? sqrt(t2 * (2.0 - t2)) : s;
        const double dphi = PD_DIV(kTwoPi, (double)ri.npix);
        t.s = (float)s;
        t.s_lo = (float)(sx - (double)t.s);
        t.dphi = (float)dphi;
        t.dphi_lo = (float)(dphi - (double)t.dphi);
        t.z = (float)z;
        t.z_lo = (float)(z - (double)t.z);
        t.start = (int)ri.start;
        t.npix2 = (int)(2 * ri.npix + (ri.shifted ? 1 : 0));
        rings[r - 1] = t;
    }
}

constexpr int kShortBlocks = 2;  // a short launch's blocks per SM

}  // namespace

bool tuned_plans_itself(long long n, int sm_count)
{
    return n <= 32LL * kShortBlocks * sm_count;
}

void launch_plans(const FwdArgs& a, tuned::SamplePlan* plans, long long pos0, long long pos1,
                  cudaStream_t st)
{
    // small blocks, so that a short launch's plans spread over the SMs: a plan
    // is a chain of some 180 FP64 instructions, and the warps of an SM queue for
    // its FP64 pipe
    const long long b = (pos1 - pos0 + 127) / 128;
    plan_kernel<<<(int)(b < 65536 ? b : 65536), 128, 0, st>>>(a, plans, pos0, pos1);
}

namespace {

template <class K>
int resident_blocks(K kernel, int threads)
{
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, 0) != cudaSuccess ||
        nb < 1)
        nb = 1;
    return nb;
}

template <bool kCheck, bool kBil, int kTW, Plans kPlans>
void launch_shape(const FwdArgs& a, int sm_count, cudaStream_t st, CheckOut* check,
                  tuned::SamplePlan* plans, long long plan_cap)
{
    const int threads = kTW * 32;
    const long long resident =
        (long long)sm_count * resident_blocks(tuned_kernel<kCheck, kBil, kTW, kPlans>, threads);
    const long long step = kPlans == kArrayPlans ? plan_cap : a.n;
    for (long long p0 = 0; p0 < a.n; p0 += step) {
        const long long p1 = p0 + step < a.n ? p0 + step : a.n;
        if (kPlans == kArrayPlans) launch_plans(a, plans, p0, p1, st);
        long long blocks = (p1 - p0 + kTW - 1) / kTW;
        if (kPlans == kBlockPlans)  // at most 32 samples to a block
            blocks = a.n < kShortBlocks * sm_count ? a.n : kShortBlocks * sm_count;
        else if (resident < blocks)
            blocks = resident;
        tuned_kernel<kCheck, kBil, kTW, kPlans>
            <<<(int)blocks, threads, 0, st>>>(a, check, plans, p0, p1);
    }
}

// kTW: the planned launch's block.  A short launch (tuned_plans_itself: at most
// 64 samples per SM, 32 to a block) gives two blocks per SM an equal share of
// the samples each, and plans in the block (2,003 samples of nside 1024 and 3
// degrees spent 11 us of 178 in plan_kernel and 3 between the launches).  Its
// blocks have 10 warps, all that fit at 96 registers, where that takes fewer
// rounds over a block's samples than 8, or both take one; otherwise 8, which
// have 128 registers and share L1 among fewer.  Times of 10 and 8 warps in us
// (nside 1024, 3 degrees, cold caches; 304 blocks): 2,003 samples 170 and 167,
// 3,040 193 and 254, 4,000 273 and 274, 6,080 324 and 364, 7,000 401 and 385,
// 9,120 452 and 489, 9,728 519 and 494; nside 2048, 1 degree: 4,864 194 and 184,
// 7,296 268 and 234, 9,728 335 and 285.  The bilinear lookup has 8.  Without
// plans the warps build their own (FP64 disc plan in the loop's registers).
template <bool kBil, int kTW>
void launch_lookup(const FwdArgs& a, int sm_count, cudaStream_t st, tuned::SamplePlan* plans,
                   long long plan_cap)
{
    constexpr int kUnplanned = kTW > 16 ? 16 : kTW;
    constexpr int kFew = 8, kMany = PISCO_FWD_WARPS / 2;
    const long long share = (a.n + kShortBlocks * sm_count - 1) / (kShortBlocks * sm_count);
    const bool many = share <= kFew || (share + kMany - 1) / kMany < (share + kFew - 1) / kFew;
    if (tuned_plans_itself(a.n, sm_count) && !kBil && many)
        launch_shape<false, kBil, kMany, kBlockPlans>(a, sm_count, st, nullptr, nullptr, 0);
    else if (tuned_plans_itself(a.n, sm_count))
        launch_shape<false, kBil, kFew, kBlockPlans>(a, sm_count, st, nullptr, nullptr, 0);
    else if (plans && plan_cap > 0)
        launch_shape<false, kBil, kTW, kArrayPlans>(a, sm_count, st, nullptr, plans, plan_cap);
    else
        launch_shape<false, kBil, kUnplanned, kOwnPlans>(a, sm_count, st, nullptr, nullptr, 0);
}

}  // namespace

bool tuned_supported(int nside_beam, int npix_beam, double rho_max)
{
    // The FP32 geometry uses the polar-cap branch of the beam grid's
    // ang2pix: every pair must land in a ring well inside the north cap.
    if (!(rho_max > 0.0) || rho_max > 0.5) return false;
    const double ring = nside_beam * sqrt(3.0 * (1.0 - cos(rho_max)));
    if (ring + 2.0 >= nside_beam) return false;
    const long long ncap = 2LL * nside_beam * (nside_beam - 1);
    return npix_beam <= ncap;
}

cudaError_t launch_ring_table(int nside, RingT* rings, cudaStream_t st)
{
    if (nside < 1 || nside > 8192 || !rings) return cudaErrorInvalidValue;
    const long long nr = 4LL * nside - 1;
    ring_table_kernel<<<(int)((nr + 255) / 256), 256, 0, st>>>(nside, rings);
    return cudaGetLastError();
}

cudaError_t launch_forward_tuned(const FwdArgs& a, int sm_count, cudaStream_t st, void* plans,
                                 long long plan_cap)
{
    if (a.n <= 0) return cudaSuccess;
    tuned::SamplePlan* p = static_cast<tuned::SamplePlan*>(plans);
    if (a.interp == 1) launch_lookup<true, PISCO_BIL_WARPS>(a, sm_count, st, p, plan_cap);
    else launch_lookup<false, PISCO_FWD_WARPS>(a, sm_count, st, p, plan_cap);
    return cudaGetLastError();
}

cudaError_t launch_tuned_check(const FwdArgs& a, int sm_count, cudaStream_t st, CheckOut* check)
{
    if (a.n <= 0) return cudaSuccess;
    launch_shape<true, false, 16, kOwnPlans>(a, sm_count, st, check, nullptr, 0);
    return cudaGetLastError();
}

}  // namespace pisco

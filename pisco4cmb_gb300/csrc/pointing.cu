// pointing.cu -- detector pointing from the array centre's pointing, on the
// GPU: BPoint::focal_plane_to_sky (src/Bpoint/bpoint.cpp:553-674,
// src/Bpoint/BPoint.h:99-103), the step that turns the telescope's boresight
// track into the per-detector (ra, dec, pa) the convolver takes.
//
// It is the part of BPoint that is geometry only: the spherical triangle
// array centre -- detector -- pole (zenith, celestial pole or source).  A
// detector at receiver-frame offsets (dx right, dy up) lies at angular
// distance r = acos(cos dx cos dy) from the array centre, in the direction
// a = atan2(sin dy, sin dx cos dy) from the receiver's x axis; with the
// array centre at latitude y and the receiver's up axis at position angle
// rot (the angle from the pole, counter-clockwise on the sky), the angle
// detector -> array centre -> pole is g = pi/2 - a - rot, and
//   latitude   asin(cos r sin y + sin r cos y cos g)
//   longitude  x -/+ atan2(sin r sin g, cos r cos y - sin r sin y cos g)
//              (Ra/Dec: minus, Az/El: plus)
//   position angle of the detector (of the receiver-frame pole seen from it)
//              atan2(cos y sin rot cos dx - sin y sin dx,
//                    cos y cos rot cos dy - (sin y cos dx + cos y sin rot sin dx) sin dy)
// plus the detector's polarization angle.  BPoint's ephemeris part (SOFA and
// the JPL tables, absent from the reference tree) is not on this path.
//
// FP64 throughout (the pointing feeds the convolver's FP64 per-sample frame);
// outputs [det * nsamples + s].  What bounds it is the FP64 pipe (16 cycles per
// warp instruction on an SM), so the kernel spends as few instructions per
// output as it can: a thread takes one sample and up to 16 detectors, the
// detectors' sines and cosines are formed once per block and the sample's once
// per thread, g needs no angle (sin r cos g = sin dy cos rot + sin dx cos dy sin
// rot, sin r sin g = sin dx cos dy cos rot - sin dy sin rot), and the three
// inverse functions go through one table (atan2_table).  96 detectors x 30,011
// samples: 1.59 ms with everything formed per output, 0.63 ms with this.
#include <cuda_runtime.h>

#include <string>

#include "../../include/pisco_gb300.h"
#include "hpx.cuh"
#include "internal.h"

namespace pisco {
void set_null_ctx_error(const char* msg);  // capi.cu
}

using namespace pisco;

namespace {

constexpr int kThreads = 128;
constexpr int kMostDets = 16;  // detectors of a block

// atan2(y, x) to about an ulp in some 20 FP64 instructions: an FP32 arctangent
// picks the nearest multiple k of pi/64, the vector is turned back by it (tab:
// cos and sin of k pi/64), and the rest, at most 0.0246, comes from the
// arctangent's series to the ninth power (truncated below 1e-17 relative).
__device__ __forceinline__ double atan2_table(double y, double x, const double2* tab)
{
    if (!(fabs(x) + fabs(y) > 1e-30)) return atan2(y, x);  // zeros, NaNs
    const int k = __float2int_rn(atan2f((float)y, (float)x) * 20.371832715762604f);
    const double2 t = tab[k & 127];
    const double d = (y * t.x - x * t.y) / (x * t.x + y * t.y);
    const double d2 = d * d;
    const double p = d2 * fma(d2, fma(d2, fma(d2, 1.0 / 9.0, -1.0 / 7.0), 1.0 / 5.0), -1.0 / 3.0);
    // pi/64 as the sum of two doubles
    const double r = fma((double)k, 1.9135106236677394e-18, fma(d, p, d));
    return fma((double)k, 0.04908738521234052, r);
}

// asin(v); a NaN for |v| > 1.
__device__ __forceinline__ double asin_table(double v, const double2* tab)
{
    return atan2_table(v, sqrt((1.0 - v) * (1.0 + v)), tab);
}

struct DetTrig {
    double sx, cx, sy, cy, a, cr, pol;  // sin, cos of dx and dy; sin dx cos dy; cos dx cos dy
};

// Blocks take (group of `group` detectors, kThreads samples) items in turn.
__global__ void __launch_bounds__(kThreads)
    focal_plane_kernel(int ndets, int group, const double* __restrict__ det_dx,
                       const double* __restrict__ det_dy, const double* __restrict__ det_pol,
                       long long ns, const double* __restrict__ x_ac,
                       const double* __restrict__ y_ac, const double* __restrict__ rot_ac, int flag,
                       double* __restrict__ x_det, double* __restrict__ y_det,
                       double* __restrict__ rot_det)
{
    __shared__ double2 tab[128];
    __shared__ DetTrig det[kMostDets];
    {
        double s, c;
        sincospi((double)threadIdx.x / 64.0, &s, &c);
        tab[threadIdx.x] = make_double2(c, s);
    }
    const long long parts = (ns + kThreads - 1) / kThreads;
    const long long items = parts * ((ndets + group - 1) / group);
    for (long long item = blockIdx.x; item < items; item += gridDim.x) {
        const int d0 = (int)(item / parts) * group;
        const int nd = min(group, ndets - d0);
        __syncthreads();  // tab, and the last item's detectors
        if (threadIdx.x < nd) {
            const int d = d0 + threadIdx.x;
            DetTrig t;
            sincos(det_dx[d], &t.sx, &t.cx);
            sincos(det_dy[d], &t.sy, &t.cy);
            t.a = t.sx * t.cy;
            t.cr = t.cx * t.cy;
            t.pol = det_pol[d];
            det[threadIdx.x] = t;
        }
        __syncthreads();
        const long long s = (item % parts) * kThreads + threadIdx.x;
        if (s >= ns) continue;
        double sl, cl, se, ce;
        const double x = x_ac[s];
        sincos(y_ac[s], &sl, &cl);
        sincos(rot_ac[s], &se, &ce);
        const double cse = cl * se, cce = cl * ce;
        for (int i = 0; i < nd; ++i) {
            const DetTrig& t = det[i];
            const long long k = (long long)(d0 + i) * ns + s;
            const double gc = t.sy * ce + t.a * se;  // sin r cos g
            y_det[k] = asin_table(t.cr * sl + cl * gc, tab);
            const double pa = atan2_table(cse * t.cx - sl * t.sx,
                                          cce * t.cy - (sl * t.cx + cse * t.sx) * t.sy, tab);
            rot_det[k] = pa + t.pol;
            if (flag == 2) {
                x_det[k] = -pa;
            } else {
                const double dl = atan2_table(t.a * ce - t.sy * se, t.cr * cl - sl * gc, tab);
                x_det[k] = flag == 0 ? x + dl : x - dl;
            }
        }
    }
}

pisco_status reject(pisco_status st, const std::string& msg)
{
    set_null_ctx_error(msg.c_str());
    return st;
}

pisco_status check_args(int ndets, long nsamples, int flag, bool ptrs)
{
    if (ndets < 0 || nsamples < 0) return reject(PISCO_ERR_INVALID_ARGUMENT, "focal_plane_to_sky: negative size");
    if ((long long)ndets * nsamples > (1LL << 40))
        return reject(PISCO_ERR_INVALID_ARGUMENT, "focal_plane_to_sky: more than 2^40 outputs");
    if (flag < 0 || flag > 2) return reject(PISCO_ERR_INVALID_ARGUMENT, "focal_plane_to_sky: flag must be 0, 1 or 2");
    if (!ptrs && ndets > 0 && nsamples > 0)
        return reject(PISCO_ERR_INVALID_ARGUMENT, "focal_plane_to_sky: NULL array");
    return PISCO_OK;
}

cudaError_t launch(int ndets, const double* dx, const double* dy, const double* pol, long long ns,
                   const double* x, const double* y, const double* rot, int flag, double* xo,
                   double* yo, double* ro, cudaStream_t st)
{
    if (ndets <= 0 || ns <= 0) return cudaSuccess;
    int device = 0, sms = 1;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    // as many detectors per thread as leave about 16 warps for each SM
    const long long parts = (ns + kThreads - 1) / kThreads;
    long long group = parts * ndets / (sms * 16LL * 32 / kThreads);
    group = group < 1 ? 1 : (group > kMostDets ? kMostDets : group);
    const long long items = parts * ((ndets + group - 1) / group);
    focal_plane_kernel<<<(int)(items < 16384 ? items : 16384), kThreads, 0, st>>>(
        ndets, (int)group, dx, dy, pol, ns, x, y, rot, flag, xo, yo, ro);
    return cudaGetLastError();
}

}  // namespace

extern "C" {

pisco_status pisco_focal_plane_to_sky_device(int ndets, const double* d_det_dx,
                                             const double* d_det_dy, const double* d_det_pol,
                                             long nsamples, const double* d_x_ac,
                                             const double* d_y_ac, const double* d_rot_ac, int flag,
                                             double* d_x_det, double* d_y_det, double* d_rot_det,
                                             void* stream)
{
    set_null_ctx_error("");
    pisco_status st = check_args(ndets, nsamples, flag,
                                 d_det_dx && d_det_dy && d_det_pol && d_x_ac && d_y_ac &&
                                     d_rot_ac && d_x_det && d_y_det && d_rot_det);
    if (st != PISCO_OK) return st;
    const cudaError_t e = launch(ndets, d_det_dx, d_det_dy, d_det_pol, nsamples, d_x_ac, d_y_ac,
                                 d_rot_ac, flag, d_x_det, d_y_det, d_rot_det, (cudaStream_t)stream);
    if (e != cudaSuccess) return reject(PISCO_ERR_CUDA, std::string("focal_plane_to_sky: ") + cudaGetErrorString(e));
    return PISCO_OK;
}

pisco_status pisco_focal_plane_to_sky(int ndets, const double* det_dx, const double* det_dy,
                                      const double* det_pol, long nsamples, const double* x_ac,
                                      const double* y_ac, const double* rot_ac, int flag,
                                      double* x_det, double* y_det, double* rot_det)
{
    set_null_ctx_error("");
    pisco_status st = check_args(ndets, nsamples, flag,
                                 det_dx && det_dy && det_pol && x_ac && y_ac && rot_ac && x_det &&
                                     y_det && rot_det);
    if (st != PISCO_OK || ndets == 0 || nsamples == 0) return st;
    const size_t nd = sizeof(double) * ndets, ns = sizeof(double) * nsamples;
    const size_t no = sizeof(double) * (size_t)ndets * nsamples;
    double* buf = nullptr;
    cudaError_t e = cudaMalloc(&buf, 3 * nd + 3 * ns + 3 * no);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return reject(e == cudaErrorMemoryAllocation ? PISCO_ERR_OUT_OF_MEMORY : PISCO_ERR_CUDA,
                      std::string("focal_plane_to_sky: ") + cudaGetErrorString(e));
    }
    double* d[9];
    d[0] = buf;
    d[1] = d[0] + ndets;
    d[2] = d[1] + ndets;
    d[3] = d[2] + ndets;
    d[4] = d[3] + nsamples;
    d[5] = d[4] + nsamples;
    d[6] = d[5] + nsamples;
    d[7] = d[6] + (size_t)ndets * nsamples;
    d[8] = d[7] + (size_t)ndets * nsamples;
    const double* in[6] = {det_dx, det_dy, det_pol, x_ac, y_ac, rot_ac};
    for (int k = 0; k < 6 && e == cudaSuccess; ++k)
        e = cudaMemcpy(d[k], in[k], k < 3 ? nd : ns, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = launch(ndets, d[0], d[1], d[2], nsamples, d[3], d[4], d[5], flag, d[6], d[7], d[8], 0);
    double* out[3] = {x_det, y_det, rot_det};
    for (int k = 0; k < 3 && e == cudaSuccess; ++k)
        e = cudaMemcpy(out[k], d[6 + k], no, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return reject(PISCO_ERR_CUDA, std::string("focal_plane_to_sky: ") + cudaGetErrorString(e));
    }
    return PISCO_OK;
}

}  // extern "C"

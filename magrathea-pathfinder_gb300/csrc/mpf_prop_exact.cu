// Reference-order (bit-exact) mode.  Must be compiled with -fmad=false.
#include <algorithm>

#include "mpf_exact.cuh"
#include "mpf_internal.h"

namespace mpf {

namespace {

__global__ void k_gather_exact(DevTree T, int kind, const double* __restrict__ xyz, long long n, void* out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    if (kind == 0) {
        ((long long*)out)[i] = locate(T, x, y, z).cell;
        return;
    }
    // kind 1: CIC, 2: TSC, 3: NGP
    Hint hint{-1, 0, {0u, 0u, 0u}};
    const Field7 f = (kind == 1) ? cic_exact<kAllFields, false>(T, x, y, z, hint, nullptr)
                     : (kind == 3) ? ngp(T, x, y, z) : tsc_exact<kAllFields, false>(T, x, y, z, hint, nullptr);
    float* o = (float*)out + 7 * i;
    o[0] = f.rho; o[1] = f.phi; o[2] = f.dx; o[3] = f.dy; o[4] = f.dz; o[5] = f.a; o[6] = f.dt;
}

}  // namespace

template <>
cudaError_t launch_propagate<true>(const DevTree& T, const DevCosmo& C, const PropParams& P, const double* d_launch, long long n,
                                   const PropOut& O, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    // An SM sub-partition's FP64 pipe takes a warp's instruction 64 cycles
    // whatever the number of its lanes (a dependent one waits no longer), so a
    // batch of fewer rays than a warp per sub-partition runs one warp on each
    // (4 an SM), with the lanes left over sharing out the Jacobian's gathers.
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const int rays = (int)std::min<long long>(32, (n + 4 * sms - 1) / (4 * sms));
    const int per_ray = P.jacobian ? rays_to_lanes(rays) : 1;
    const long long warps = (n + rays - 1) / rays;
    const int tpb = (warps < 8ll * sms) ? 32 : 128;
    const unsigned grid = (unsigned)((warps + tpb / 32 - 1) / (tpb / 32));
    if (P.ray_stop) k_propagate<true><<<grid, tpb, 0, stream>>>(T, C, P, d_launch, n, O, rays, per_ray);
    else k_propagate<false><<<grid, tpb, 0, stream>>>(T, C, P, d_launch, n, O, rays, per_ray);
    return cudaGetLastError();
}
cudaError_t launch_gather_exact(const DevTree& T, int kind, const double* d_xyz, long long n, void* d_out, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    const int tpb = 128;
    k_gather_exact<<<(unsigned)((n + tpb - 1) / tpb), tpb, 0, stream>>>(T, kind, d_xyz, n, d_out);
    return cudaGetLastError();
}
}  // namespace mpf

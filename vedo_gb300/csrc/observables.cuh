// observables.cuh - DOWorld::CalculateSystemEnergy (DOWorld.cpp:481-660) over the device state,
// mobile objects only, with fixed-shape tree reductions (deterministic run to run).
#pragma once

#include <cfloat>

#include "dem_common.cuh"

namespace vedo {
namespace obs {
namespace {   // internal linkage: the header is compiled into each engine's translation unit

constexpr int TPB = 256;
constexpr int OBS_A = 16;
// Blocks of the two passes: four per SM, each thread over several objects, so that the shared-memory
// trees (12 FP64 additions per 8 threads and field, 16 cycles each on GB300) run once per block and
// not once per 256 objects, and the last reduction has few partial sums.
inline unsigned obs_blocks(uint32_t n) { return n <= 608u * TPB ? (n + TPB - 1) / TPB + (n == 0) : 608u; }
__global__ void __launch_bounds__(TPB) k_obs_a(uint32_t n, const uint32_t* __restrict__ model_of,
                                               const ModelDev* __restrict__ models, const double4_32a* __restrict__ pos,
                                               const double4_32a* __restrict__ vel, const double4_32a* __restrict__ av,
                                               d3 g, double* __restrict__ part) {
    __shared__ double s[OBS_A][TPB];
    double v[OBS_A];
    for (int q = 0; q < OBS_A; ++q) v[q] = 0.0;
    v[12] = DBL_MAX; v[13] = -DBL_MAX; v[14] = DBL_MAX; v[15] = -DBL_MAX;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ModelDev& m = models[model_of[i]];
        if (m.behavior != BEH_MOBILE) continue;
        const d3 V = ld(vel, i), AV = ld(av, i), P = ld(pos, i);
        const double vl = len(V), al = len(AV);
        const d3 I = mk(m.ix, m.iy, m.iz);
        v[0] -= m.mass * dot(g, P);
        v[1] += 0.5 * m.mass * vl * vl;
        v[2] += 0.5 * (I.x * AV.x * AV.x + I.y * AV.y * AV.y + I.z * AV.z * AV.z);
        const d3 mo = smul(m.mass, V), am = cross(I, AV);
        v[3] += mo.x; v[4] += mo.y; v[5] += mo.z;
        v[6] += am.x; v[7] += am.y; v[8] += am.z;
        v[9] += 1.0;
        v[10] += m.mass;
        v[12] = fmin(v[12], vl); v[13] = fmax(v[13], vl);
        v[14] = fmin(v[14], al); v[15] = fmax(v[15], al);
    }
    for (int q = 0; q < OBS_A; ++q) s[q][threadIdx.x] = v[q];
    __syncthreads();
    for (int w = TPB / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            for (int q = 0; q < 12; ++q) s[q][threadIdx.x] += s[q][threadIdx.x + w];
            s[12][threadIdx.x] = fmin(s[12][threadIdx.x], s[12][threadIdx.x + w]);
            s[13][threadIdx.x] = fmax(s[13][threadIdx.x], s[13][threadIdx.x + w]);
            s[14][threadIdx.x] = fmin(s[14][threadIdx.x], s[14][threadIdx.x + w]);
            s[15][threadIdx.x] = fmax(s[15][threadIdx.x], s[15][threadIdx.x + w]);
        }
        __syncthreads();
    }
    if (threadIdx.x < OBS_A) part[(size_t)blockIdx.x * OBS_A + threadIdx.x] = s[threadIdx.x][0];
}

// One block per field: thread t folds partial sums t, t + 256, ... in order, then a fixed tree over as many
// threads as have one.  (One thread per field, sequential over the blocks, took 0.83 ms at 1954 blocks; the
// tree over all 256 threads 3.7 us for the single partial sum of 64 spheres, 2.8 like this.)
__global__ void __launch_bounds__(TPB) k_obs_reduce(uint32_t nb, int width, const double* __restrict__ part,
                                                    double* __restrict__ res, int nmin_from) {
    __shared__ double s[TPB];
    const int q = blockIdx.x, t = threadIdx.x;
    const bool sum = q < nmin_from, least = !sum && ((q - nmin_from) & 1) == 0;
    auto join = [&](double a, double b) { return sum ? a + b : least ? fmin(a, b) : fmax(a, b); };
    double acc = sum ? 0.0 : least ? DBL_MAX : -DBL_MAX;
    for (uint32_t b = t; b < nb; b += TPB) acc = join(acc, part[(size_t)b * width + q]);
    s[t] = acc;
    __syncthreads();
    int w = TPB / 2;
    while (w > 0 && (uint32_t)w >= nb) w >>= 1;
    for (; w > 0; w >>= 1) {
        if (t < w) s[t] = join(s[t], s[t + w]);
        __syncthreads();
    }
    if (t == 0) res[q] = s[0];
}

__global__ void __launch_bounds__(TPB) k_obs_b(uint32_t n, const uint32_t* __restrict__ model_of,
                                               const ModelDev* __restrict__ models, const double4_32a* __restrict__ pos,
                                               const double4_32a* __restrict__ vel, const double4_32a* __restrict__ av,
                                               const double* __restrict__ res,
                                               const uint8_t* __restrict__ flags, uint32_t np,
                                               double* __restrict__ part) {
    __shared__ double s[6][TPB];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    double v[6] = {0, 0, 0, 0, 0, 0};
    const double cnt = res[9];
    const d3 mmean = smul(1.0 / cnt, mk(res[3], res[4], res[5]));
    const d3 amean = smul(1.0 / cnt, mk(res[6], res[7], res[8]));
    for (uint32_t i = t; i < n; i += nt) {
        const ModelDev& m = models[model_of[i]];
        if (m.behavior != BEH_MOBILE) continue;
        const d3 V = ld(vel, i), AV = ld(av, i), P = ld(pos, i);
        v[0] += len(sub(smul(m.mass, V), mmean));
        v[1] += len(sub(cross(mk(m.ix, m.iy, m.iz), AV), amean));
        v[2] += m.mass * P.x; v[3] += m.mass * P.y; v[4] += m.mass * P.z;
    }
    // the contacts' flag bytes (bit 64), sixteen to a load; the array is 256-byte aligned
    uint32_t hits = 0;
    const uint4* f16 = reinterpret_cast<const uint4*>(flags);
    for (uint32_t k = t; k < np / 16u; k += nt) {
        const uint4 f = f16[k];
        hits += __popc(f.x & 0x40404040u) + __popc(f.y & 0x40404040u) + __popc(f.z & 0x40404040u) +
                __popc(f.w & 0x40404040u);
    }
    for (uint32_t k = (np & ~15u) + t; k < np; k += nt) hits += (flags[k] & 64u) ? 1u : 0u;
    v[5] = (double)hits;
    for (int q = 0; q < 6; ++q) s[q][threadIdx.x] = v[q];
    __syncthreads();
    for (int w = TPB / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int q = 0; q < 6; ++q) s[q][threadIdx.x] += s[q][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 6) part[(size_t)blockIdx.x * 6 + threadIdx.x] = s[threadIdx.x][0];
}


}  // namespace
}  // namespace obs
}  // namespace vedo

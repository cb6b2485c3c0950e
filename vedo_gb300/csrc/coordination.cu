// coordination.cu - the post-processing tool's coordination number (vedo/knight/CalcCoordinateNum.cpp)
// over the device state.
//
// CalcCoordinateNum compares every sphere with every other one (O(N^2) on the host).  Here the
// spheres go into a uniform cell grid whose edge is a little over the largest radius sum, so
// every pair within reach lies in neighbouring cells; one thread per sphere visits the 27 cells
// around its own and decides the reference's FP64 tests (this file is compiled with
// -fmad=false): |p_i - p_j| = sqrt(dx*dx + dy*dy + dz*dz) against r_i + r_j, counting the
// strict test (outputCoordinateNumVTK, :79-126) and the inclusive one (computeAvgCoordinateNum,
// :8-77) in one pass.  The counts are integers, so the result equals the reference's whatever the
// visiting order.
#include "coordination.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dfloat.cuh"
#include "engine_base.h"
#include "prefilter.cuh"
#include "sort_scan.h"

namespace vedo {
namespace {

constexpr int TPB = 256;
inline unsigned nblk(uint64_t n) { return (unsigned)((n + TPB - 1) / TPB); }

// order-preserving map of doubles to unsigned 64-bit integers (exact atomic min/max)
__device__ inline unsigned long long ord64(double d) {
    unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
inline double dbl_of(unsigned long long o) {
    unsigned long long b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}

__device__ inline bool is_sphere(const ModelDev& m) { return m.shape == SHAPE_SPHERE; }
__device__ inline bool finite3(d3 p) { return isfinite(p.x) && isfinite(p.y) && isfinite(p.z); }

// A block's minima/maxima and counts, reduced over its threads before one thread's atomics: an atomic
// per sphere on one address is a serial chain (at 7 per sphere this pass took 2.16 ms for 500,000
// spheres, whose positions are read in 5 us at the copy bandwidth).
__device__ __forceinline__ unsigned long long warp_min64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// bounds of the finite sphere centres ([0..2] min, [3..5] max), the largest radius [6] and the
// number of spheres [7]
__global__ void __launch_bounds__(TPB) k_cn_bounds(uint32_t n, const uint32_t* __restrict__ model_of,
                                                   const ModelDev* __restrict__ models,
                                                   const double4_32a* __restrict__ pos,
                                                   unsigned long long* __restrict__ red) {
    __shared__ unsigned long long s[8][TPB / 32];
    unsigned long long v[8] = {~0ull, ~0ull, ~0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ModelDev& m = models[model_of[i]];
        if (!is_sphere(m)) continue;
        ++v[7];
        const d3 p = ld(pos, i);
        if (!finite3(p)) continue;
        const unsigned long long o[3] = {ord64(p.x), ord64(p.y), ord64(p.z)};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[k] = min(v[k], o[k]);
            v[3 + k] = max(v[3 + k], o[k]);
        }
        v[6] = max(v[6], ord64(m.a0));
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const unsigned long long x = k < 3 ? warp_min64(v[k]) : k < 7 ? warp_max64(v[k]) : warp_sum64(v[k]);
        if (lane == 0) s[k][w] = x;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        const int k = threadIdx.x;
        unsigned long long x = s[k][0];
        for (int q = 1; q < TPB / 32; ++q) x = k < 3 ? min(x, s[k][q]) : k < 7 ? max(x, s[k][q]) : x + s[k][q];
        if (k < 3) atomicMin(&red[k], x);
        else if (k < 7) atomicMax(&red[k], x);
        else atomicAdd(&red[7], x);
    }
}

struct Grid {
    double lo[3], mid[3], inv_h;
    uint32_t dim[3];
    float slack;     // bounds what the FP32 offsets' roundings change in a distance
    float ext;       // largest sum of an offset's magnitudes
};

// (a multiplication by 1/h: within 4e-7 cells of the quotient on a grid of at most 1e9 cells an axis,
// which the cell edge's margin of 1e-6 covers)
__device__ inline uint32_t cell_axis(double x, double lo, double inv_h, uint32_t dim) {
    const double c = floor((x - lo) * inv_h);
    if (!(c >= 0.0)) return 0;                 // below the grid, or not a number
    if (c >= (double)(dim - 1)) return dim - 1;
    return (uint32_t)c;
}

// cell key per sphere (the number of cells for other shapes: sorted last, never visited)
__global__ void __launch_bounds__(TPB) k_cn_keys(uint32_t n, const uint32_t* __restrict__ model_of,
                                                 const ModelDev* __restrict__ models,
                                                 const double4_32a* __restrict__ pos, Grid g, uint32_t ncell,
                                                 uint32_t* __restrict__ key, uint32_t* __restrict__ id) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    id[i] = i;
    if (!is_sphere(models[model_of[i]])) {
        key[i] = ncell;
        return;
    }
    const d3 p = ld(pos, i);
    const uint32_t cx = cell_axis(p.x, g.lo[0], g.inv_h, g.dim[0]), cy = cell_axis(p.y, g.lo[1], g.inv_h, g.dim[1]),
                   cz = cell_axis(p.z, g.lo[2], g.inv_h, g.dim[2]);
    key[i] = cx + g.dim[0] * (cy + g.dim[1] * cz);
}

// [start, end) of every occupied cell in the sorted order, and the spheres' centres (from the grid's
// middle) and radii in that order as double-float pairs: hi (x, y, z, r), lo
__global__ void __launch_bounds__(TPB) k_cn_ranges(uint32_t ns, const uint32_t* __restrict__ key,
                                                   const uint32_t* __restrict__ id,
                                                   const uint32_t* __restrict__ model_of,
                                                   const ModelDev* __restrict__ models,
                                                   const double4_32a* __restrict__ pos, Grid g,
                                                   uint32_t* __restrict__ start, uint32_t* __restrict__ end,
                                                   float4* __restrict__ hi, float4* __restrict__ lo) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ns) return;
    const uint32_t c = key[k], i = id[k];
    if (k == 0 || key[k - 1] != c) start[c] = k;
    if (k + 1 == ns || key[k + 1] != c) end[c] = k + 1;
    const d3 p = ld(pos, i);
    float4 h, l;
    split32(p.x - g.mid[0], h.x, l.x);
    split32(p.y - g.mid[1], h.y, l.y);
    split32(p.z - g.mid[2], h.z, l.z);
    split32(models[model_of[i]].a0, h.w, l.w);
    hi[k] = h;
    lo[k] = l;
}

// One thread per sphere in cell order; a row of three neighbour cells along x is one run of the
// sorted spheres.  FP64 arithmetic on GB300 costs 16 cycles a warp instruction, so the reference's
// test runs only where nothing cheaper decides: FP32 offsets first (all but the spheres at about
// the radius sum), then R^2 - d^2 in double-float for those, put aside so that a warp takes them
// together; within the band around zero that the double-float error cannot leave, the reference's
// FP64 formula.  With the FP64 test of every candidate the count of 500,000 densely packed spheres
// took 1.57 ms; the counts are the same, and with the bounds above and the observables' kernels as
// they were a read of both observables went from 5.84 to 1.77 ms.
constexpr int CN_ASIDE = 16;      // undecided neighbours a thread holds before it settles them
__global__ void __launch_bounds__(TPB) k_cn_count(uint32_t ns, const uint32_t* __restrict__ key,
                                                  const uint32_t* __restrict__ id, const uint32_t* __restrict__ start,
                                                  const uint32_t* __restrict__ end,
                                                  const uint32_t* __restrict__ model_of,
                                                  const ModelDev* __restrict__ models,
                                                  const double4_32a* __restrict__ pos, const float4* __restrict__ hi,
                                                  const float4* __restrict__ lo, Grid g, uint32_t* __restrict__ below,
                                                  uint32_t* __restrict__ touching) {
    __shared__ uint32_t aside[CN_ASIDE][TPB];
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ns) return;
    const uint32_t i = id[k], c = key[k];
    const int cx = (int)(c % g.dim[0]), cy = (int)((c / g.dim[0]) % g.dim[1]), cz = (int)(c / (g.dim[0] * g.dim[1]));
    const float4 hs = hi[k], ls = lo[k];
    uint32_t lt = 0, le = 0, held = 0;
    auto settle = [&]() {
        for (uint32_t t = 0; t < held; ++t) {
            const uint32_t q = aside[t][threadIdx.x];
            const float4 hm = hi[q], lm = lo[q];
            const dfl dx = df_diff(hm.x, lm.x, hs.x, ls.x), dy = df_diff(hm.y, lm.y, hs.y, ls.y),
                      dz = df_diff(hm.z, lm.z, hs.z, ls.z);
            const dfl s2 = df_add(df_add(df_sq(dx), df_sq(dy)), df_sq(dz));
            const dfl R = df_add(dfl{hs.w, ls.w}, dfl{hm.w, lm.w}), R2 = df_sq(R);
            const dfl num = df_add(R2, dfl{-s2.hi, -s2.lo});
            // 1e-9 R^2, and the splits' rounding (2^-48 of an offset): 7 * 2^-48 R ext, rounded up
            const float band = 1e-9f * R2.hi + 1e-13f * R.hi * g.ext;
            if (R.hi > 1e-15f && (num.hi > band || num.hi < -band)) {
                lt += num.hi > 0.0f ? 1u : 0u;
                le += num.hi > 0.0f ? 1u : 0u;
            } else {
                const uint32_t j = id[q];
                const double d = len(sub(ld(pos, i), ld(pos, j)));                   // (m1 - m2).length()
                const double rs = models[model_of[i]].a0 + models[model_of[j]].a0;    // r1 + r2
                lt += d < rs ? 1u : 0u;
                le += d <= rs ? 1u : 0u;
            }
        }
        held = 0;
    };
    for (int z = max(cz - 1, 0); z <= min(cz + 1, (int)g.dim[2] - 1); ++z)
        for (int y = max(cy - 1, 0); y <= min(cy + 1, (int)g.dim[1] - 1); ++y) {
            const uint32_t row = g.dim[0] * ((uint32_t)y + g.dim[1] * (uint32_t)z);
            uint32_t q = 0xffffffffu, e = 0;
            for (int x = max(cx - 1, 0); x <= min(cx + 1, (int)g.dim[0] - 1); ++x) {
                const uint32_t ce = end[row + (uint32_t)x];
                if (ce == 0u) continue;            // an empty cell
                q = min(q, start[row + (uint32_t)x]);
                e = ce;
            }
            for (; q < e; ++q) {
                if (q == k) continue;
                const float4 p = hi[q];
                const float dx = p.x - hs.x, dy = p.y - hs.y, dz = p.z - hs.z;
                const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx)), thr = hs.w + p.w;
                const float far = thr * (1.0f + 4.0f * PF_ARITH_EPS) + g.slack,
                            near = thr * (1.0f - 4.0f * PF_ARITH_EPS) - g.slack;
                if (thr > 1e-15f && d2 > far * far * (1.0f + 4.0f * PF_ARITH_EPS)) continue;
                if (thr > 1e-15f && near > 0.0f && d2 < near * near * (1.0f - 4.0f * PF_ARITH_EPS)) {
                    ++lt;
                    ++le;
                    continue;
                }
                aside[held][threadIdx.x] = q;      // (not a number: decided by the FP64 formula)
                if (++held == CN_ASIDE) settle();
            }
        }
    settle();
    below[i] = lt;
    touching[i] = le;
}

// computeAvgCoordinateNum's selection: centre strictly inside the box widened by the radius
__global__ void __launch_bounds__(TPB) k_cn_average(uint32_t n, const uint32_t* __restrict__ model_of,
                                                    const ModelDev* __restrict__ models,
                                                    const double4_32a* __restrict__ pos,
                                                    const uint32_t* __restrict__ touching, Box6 b,
                                                    unsigned long long* __restrict__ sums) {
    __shared__ unsigned long long s[2][TPB / 32];
    unsigned long long sum = 0, cnt = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ModelDev& m = models[model_of[i]];
        if (!is_sphere(m)) continue;
        const d3 p = ld(pos, i);
        const double r = m.a0;
        if ((p.x < (b.v[1] + r)) && (p.x > (b.v[0] - r)) && (p.y < (b.v[3] + r)) && (p.y > (b.v[2] - r)) &&
            (p.z < (b.v[5] + r)) && (p.z > (b.v[4] - r))) {
            sum += touching[i];
            ++cnt;
        }
    }
    sum = warp_sum64(sum);
    cnt = warp_sum64(cnt);
    if ((threadIdx.x & 31) == 0) {
        s[0][threadIdx.x >> 5] = sum;
        s[1][threadIdx.x >> 5] = cnt;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned long long x = 0;
        for (int q = 0; q < TPB / 32; ++q) x += s[threadIdx.x][q];
        if (x) atomicAdd(&sums[threadIdx.x], x);
    }
}

}  // namespace

// `work`: the caller's workspace of about 80 bytes an object, kept between its calls.  below and touching
// return device arrays inside it, valid until its next use.
static int coordination_device(uint32_t n, const uint32_t* model_of, const ModelDev* models, const double4_32a* pos,
                               uint32_t** below, uint32_t** touching, const double* box, double* average,
                               Scratch& scratch, Scratch& work, cudaStream_t s, std::string& err, uint64_t* launches) {
    uint64_t L = 0;
    auto fail = [&](cudaError_t e) {
        err = std::string("coordination: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? VEDO_ERR_OUT_OF_MEMORY : VEDO_ERR_CUDA;
    };
#define CN_CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return fail(e_); } while (0)
    *below = *touching = nullptr;
    if (n == 0) {
        if (average) *average = NAN;
        return VEDO_OK;
    }
    // the arrays of the workspace, 256-byte aligned: [0] the reductions' results
    const size_t words = ((size_t)n + 63) / 64 * 64;       // n 4-byte words, a multiple of 256 bytes
    const size_t fixed = 256 + 4 * words * (4 + 2 + 8);    // keys and ids twice, two counts, hi and lo
    CN_CK(work.reserve(fixed));
    // bounds of the sphere centres, the largest radius, the sphere count; [8..9]: the average's sums
    const unsigned wide = std::min(nblk(n), 608u);         // a few blocks per SM: few atomics
    unsigned long long init[10];
    for (int k = 0; k < 3; ++k) init[k] = ~0ull;
    for (int k = 3; k < 10; ++k) init[k] = 0ull;
    unsigned long long* red = static_cast<unsigned long long*>(work.ptr);
    CN_CK(cudaMemcpyAsync(red, init, sizeof(init), cudaMemcpyHostToDevice, s));
    k_cn_bounds<<<wide, TPB, 0, s>>>(n, model_of, models, pos, red);
    ++L;
    unsigned long long got[8];
    CN_CK(cudaMemcpyAsync(got, red, sizeof(got), cudaMemcpyDeviceToHost, s));
    CN_CK(cudaStreamSynchronize(s));
    // with no sphere at a finite position no distance test can hold (NaN compares false)
    const bool any = got[6] != 0ull;
    const uint32_t ns = (uint32_t)got[7];
    Grid g{};
    uint32_t ncell = 0;
    if (any) {
        double hi[3];
        for (int k = 0; k < 3; ++k) {
            g.lo[k] = dbl_of(got[k]);
            hi[k] = dbl_of(got[3 + k]);
        }
        const double rmax = dbl_of(got[6]);
        // a pair within reach is at most 2 r_max apart; the margin keeps the floor() of the cell
        // coordinates of two such centres within one of each other despite rounding
        double h = std::max(2.0 * rmax, 1e-300) * (1.0 + 1e-6);
        for (int k = 0; k < 3; ++k) h = std::max(h, (hi[k] - g.lo[k]) * 1e-9);
        const double cap = std::max(64.0, 4.0 * (double)n);
        for (;;) {
            double cells = 1.0;
            for (int k = 0; k < 3; ++k) cells *= std::floor((hi[k] - g.lo[k]) / h) + 1.0;
            if (cells <= cap) break;
            h *= 2.0;
        }
        g.inv_h = 1.0 / h;
        double ext = 0.0;
        for (int k = 0; k < 3; ++k) {
            g.dim[k] = (uint32_t)(std::floor((hi[k] - g.lo[k]) / h) + 1.0);
            g.mid[k] = 0.5 * g.lo[k] + 0.5 * hi[k];
            ext += 0.5 * (hi[k] - g.lo[k]);
        }
        ncell = g.dim[0] * g.dim[1] * g.dim[2];
        g.ext = (float)ext * 1.0001f;
        g.slack = 2.0f * PF_POS_EPS * g.ext;
    }
    CN_CK(work.reserve(fixed + 8 * (size_t)ncell));
    char* w = static_cast<char*>(work.ptr);
    red = reinterpret_cast<unsigned long long*>(w);
    w += 256;
    auto take = [&](size_t bytes) {
        char* p = w;
        w += bytes;
        return p;
    };
    uint32_t* key = reinterpret_cast<uint32_t*>(take(4 * words));
    uint32_t* id = reinterpret_cast<uint32_t*>(take(4 * words));
    uint32_t* key2 = reinterpret_cast<uint32_t*>(take(4 * words));
    uint32_t* id2 = reinterpret_cast<uint32_t*>(take(4 * words));
    uint32_t* nlt = reinterpret_cast<uint32_t*>(take(4 * words));
    uint32_t* nle = reinterpret_cast<uint32_t*>(take(4 * words));
    float4* ph = reinterpret_cast<float4*>(take(16 * words));
    float4* pl = reinterpret_cast<float4*>(take(16 * words));
    uint32_t* cs = reinterpret_cast<uint32_t*>(take(8 * (size_t)ncell));
    uint32_t* ce = cs + ncell;
    *below = nlt;
    *touching = nle;
    CN_CK(cudaMemsetAsync(nlt, 0, 8 * words, s));
    if (any) {
        CN_CK(cudaMemsetAsync(ce, 0, 4 * (size_t)ncell, s));
        int bits = 1;
        while (bits < 32 && (ncell >> bits)) ++bits;
        const bool alt = radix_passes_of(0, bits) & 1;
        k_cn_keys<<<nblk(n), TPB, 0, s>>>(n, model_of, models, pos, g, ncell, alt ? key2 : key, alt ? id2 : id);
        ++L;
        const uint64_t l0 = g_sort_scan_launches;
        CN_CK(radix_sort_u32(key, id, key2, id2, n, 0, bits, scratch, s, alt));
        L += g_sort_scan_launches - l0;
        // the spheres' keys sort before the other shapes': the first ns entries
        if (ns) {
            k_cn_ranges<<<nblk(ns), TPB, 0, s>>>(ns, key, id, model_of, models, pos, g, cs, ce, ph, pl);
            k_cn_count<<<nblk(ns), TPB, 0, s>>>(ns, key, id, cs, ce, model_of, models, pos, ph, pl, g, nlt, nle);
            L += 2;
        }
    }
    if (average) {
        Box6 b;
        for (int k = 0; k < 6; ++k) b.v[k] = box ? box[k] : 0.0;
        CN_CK(cudaMemsetAsync(red + 8, 0, 16, s));
        k_cn_average<<<wide, TPB, 0, s>>>(n, model_of, models, pos, nle, b, red + 8);
        ++L;
        unsigned long long sums[2];
        CN_CK(cudaMemcpyAsync(sums, red + 8, sizeof(sums), cudaMemcpyDeviceToHost, s));
        CN_CK(cudaStreamSynchronize(s));
        // the reference sums in an unsigned 32-bit integer and divides by the selected count
        const uint32_t total = (uint32_t)sums[0];
        *average = total / (double)sums[1];
    }
    CN_CK(cudaGetLastError());
    if (launches) *launches += L;
#undef CN_CK
    return VEDO_OK;
}

}  // namespace vedo

namespace vedo {

int coordination_host(const DeviceObjects& d, uint32_t* below, uint32_t* touching, const double* box,
                      double* average, std::string& err) {
    if (!d.scene || !d.scratch || !d.work) {
        err = "coordination needs a single-scene engine";
        return VEDO_ERR_INVALID_ARGUMENT;
    }
    uint32_t *dlt = nullptr, *dle = nullptr;
    int rc = coordination_device(d.n, d.model_of, d.models, d.pos, &dlt, &dle, box, average, *d.scratch, *d.work,
                                 d.stream, err, d.launches);
    cudaError_t e = cudaSuccess;
    if (rc == VEDO_OK && below && d.n) e = cudaMemcpyAsync(below, dlt, 4 * (size_t)d.n, cudaMemcpyDeviceToHost, d.stream);
    if (rc == VEDO_OK && e == cudaSuccess && touching && d.n)
        e = cudaMemcpyAsync(touching, dle, 4 * (size_t)d.n, cudaMemcpyDeviceToHost, d.stream);
    const cudaError_t es = cudaStreamSynchronize(d.stream);
    if (e == cudaSuccess) e = es;
    if (rc == VEDO_OK && e != cudaSuccess) {
        err = std::string("coordination: ") + cudaGetErrorString(e);
        rc = VEDO_ERR_CUDA;
    }
    return rc;
}

int write_vtk_host(EngineBase* eng, const DeviceObjects& d, const char* path, int with_coordination,
                   std::string& err) {
    if (!path) return VEDO_ERR_INVALID_ARGUMENT;
    if (!d.scene) {
        err = "write_vtk needs a single-scene engine";
        return VEDO_ERR_INVALID_ARGUMENT;
    }
    std::vector<double> pos(3 * (size_t)d.n), vel(3 * (size_t)d.n), av(3 * (size_t)d.n);
    vedo_state_view v{};
    v.position = pos.data();
    v.velocity = vel.data();
    v.angular_velocity = av.data();
    int rc = eng->get_state(v);
    if (rc != VEDO_OK) {
        err = eng->error();
        return rc;
    }
    std::vector<uint32_t> cn;
    if (with_coordination) {
        cn.resize(d.n);
        rc = coordination_host(d, cn.data(), nullptr, nullptr, nullptr, err);
        if (rc != VEDO_OK) return rc;
    }
    if (!write_world_vtk(path, *d.scene, pos.data(), vel.data(), av.data(), with_coordination ? cn.data() : nullptr,
                         err))
        return VEDO_ERR_IO;
    return VEDO_OK;
}

}  // namespace vedo

// engine.cu - FP64 DEM time step and NBS broad phase on the GPU.
//
// Built with -fmad=false: the FP64 arithmetic below reproduces the reference's IEEE
// operation sequence (see dem_physics.cuh).  Per time step (SimMediator::Run,
// SimMediator.cpp:714-842) two kernels run:
//   k_pair  - the FP32 prefilter over every candidate pair, then for the
//             pairs it leaves (in full warps): narrow phase at the current positions (the
//             ContactInfo the reference computed at the end of the previous step) + impact
//             solver + status update; the impulses go to a per-pair output record.
//   k_obj   - one thread per local object: the pair impulses in candidate-list order
//             (the reference's IactContainer order), the field impulse, the external
//             force and DiscreteObject::Response.  Scope-global objects (walls) are
//             summed by one block each (ordered additions, cooperative loads).
// Every UpIact steps the candidate list is rebuilt with NBSConsultant's rule
// (NBSConsultant.cpp:85-374): cell keys, a stable radix sort, cell ranges, then a count
// and a fill pass over (object, neighbour slot) tasks laid out in the reference's
// traversal order, so the new list equals the reference's list element for element.
#include "engine.h"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>

#include "dem_physics.cuh"
#include "prefilter.cuh"
#include "observables.cuh"

namespace vedo {

namespace {

constexpr int TPB = 256;
inline unsigned blocks_for(uint64_t n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }

// Neighbour visiting order of NBSConsultant::Reset (NBSConsultant.cpp:202-270):
// 12 = the cell itself (i < j), 13 = all scope-global objects.
__constant__ int c_slot[15][3] = {{-1, -1, -1}, {-1, -1, 0}, {-1, -1, 1}, {0, -1, -1}, {0, -1, 0},
                                  {0, -1, 1},   {1, -1, -1}, {1, -1, 0},  {1, -1, 1},  {-1, 0, -1},
                                  {-1, 0, 0},   {0, 0, -1},  {0, 0, 0},   {0, 0, 0},   {1, 0, -1}};
constexpr int SLOT_SELF = 12;
constexpr int SLOT_GLOBAL = 13;
constexpr int NSLOT = 15;
// LeapConsultant::subReset (LeapConsultant.h:195-446): the 13 half-shell neighbours, then the
// cell itself (13), then the scope-global objects (14).
__constant__ int c_slot_leap[13][3] = {{-1, -1, -1}, {-1, -1, 0}, {-1, -1, 1}, {0, -1, -1}, {0, -1, 0},
                                       {0, -1, 1},   {1, -1, -1}, {1, -1, 0},  {1, -1, 1},  {-1, 0, -1},
                                       {-1, 0, 0},   {0, 0, -1},  {1, 0, -1}};

// The broad phase's cell-key layout: the axis order of the key (the consultant's comparator:
// NBS and TrirLeX x, y, z; TrirLeY y, x, z; TrirLeZ z, x, y, NBSConsultant.h:62-128), the key's
// extent per axis, the number of zones per axis and, for the Leap consultant, its periodic axes.
struct CellGrid {
    int mode;                  // key order: 0 x, y, z (NBS, TrirLeX); 1 y, x, z (TrirLeY); 2 z, x, y (TrirLeZ)
    uint64_t dim[3];           // key extent per axis (x, y, z)
    uint32_t ncel[3];          // zones per axis (x, y, z): the last zone is ncel - 1
    int leap;                  // 1: LeapConsultant's traversal
    int pbc[3], has_pbc;       // Leap: axes whose neighbours wrap (LeapConsultant.h:146-150)
};
// (fixed indices per mode: the zone coordinates stay in registers)
__host__ __device__ inline uint64_t grid_key(const CellGrid& g, const uint64_t c[3]) {
    if (g.mode == 1) return (c[1] * g.dim[0] + c[0]) * g.dim[2] + c[2];
    if (g.mode == 2) return (c[2] * g.dim[0] + c[0]) * g.dim[1] + c[1];
    return (c[0] * g.dim[1] + c[1]) * g.dim[2] + c[2];
}
__device__ inline void grid_cell(const CellGrid& g, uint64_t key, uint64_t c[3]) {
    if (key <= 0xffffffffull) {        // (nearly always) 32-bit divisions
        const uint32_t k = (uint32_t)key, lo = (uint32_t)(g.mode == 1 ? g.dim[2] : g.mode == 2 ? g.dim[1] : g.dim[2]),
                       mid = (uint32_t)(g.mode == 1 ? g.dim[0] : g.mode == 2 ? g.dim[0] : g.dim[1]);
        if (g.dim[0] <= 0xffffffffull && g.dim[1] <= 0xffffffffull && g.dim[2] <= 0xffffffffull) {
            const uint32_t q = k / lo, first = q / mid, second = q % mid, third = k % lo;
            if (g.mode == 1) { c[1] = first; c[0] = second; c[2] = third; }
            else if (g.mode == 2) { c[2] = first; c[0] = second; c[1] = third; }
            else { c[0] = first; c[1] = second; c[2] = third; }
            return;
        }
    }
    if (g.mode == 1) {
        c[2] = key % g.dim[2]; key /= g.dim[2]; c[0] = key % g.dim[0]; c[1] = key / g.dim[0];
    } else if (g.mode == 2) {
        c[1] = key % g.dim[1]; key /= g.dim[1]; c[0] = key % g.dim[0]; c[2] = key / g.dim[0];
    } else {
        c[2] = key % g.dim[2]; key /= g.dim[2]; c[1] = key % g.dim[1]; c[0] = key / g.dim[1];
    }
}

// order-preserving map of doubles to unsigned 64-bit integers (for exact atomic min/max)
__host__ __device__ inline unsigned long long ord_of(double d) {
    unsigned long long b;
    memcpy(&b, &d, 8);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ inline double dbl_of(unsigned long long o) {
    unsigned long long b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    double d;
    memcpy(&d, &b, 8);
    return d;
}

// ------------------------------------------------------------------------------------
// time step
__device__ __forceinline__ void pair_exact(uint32_t k, const uint2* __restrict__ sm,
                                           const uint32_t* __restrict__ param, const PairParam* __restrict__ params,
                                           const double4_32a* __restrict__ geom, const double4_32a* __restrict__ hole,
                                           const double4_32a* __restrict__ pos,
                                           const double4_32a* __restrict__ vel, const double4_32a* __restrict__ av,
                                           const double4_32a* __restrict__ ox, const double4_32a* __restrict__ oz,
                                           double4_32a* __restrict__ hist, double* __restrict__ v0,
                                           uint8_t* __restrict__ flags, double* __restrict__ out, double dt,
                                           int backup, const Periodic& pb, uint8_t* __restrict__ touched) {
    const uint2 p = sm[k];
    const uint32_t pi = param[k];
    const int cd = params[pi].cd, is = params[pi].is;
    const double4_32a gg = geom[pi];
    PairGeom g{gg.x, gg.y, gg.z, gg.w, 0.0, 0.0, 0.0};
    if (cd == CD_SHP) {
        const double4_32a hh = hole[pi];
        g.hr = hh.x; g.hxo = hh.y; g.hyo = hh.z;
    }
    const d3 Ps = ld(pos, p.x), Pm = ld(pos, p.y);
    double depth;
    d3 n, point;
    detect_pair(cd, g, Ps, Pm, ox, oz, p.y, pb, depth, n, point);
    const bool active = depth > 0.0;
    const uint8_t f0 = flags[k];
    PairStatus st;
    st.f = f0 & (PF_STATUS | PF_NONZERO);
    if (backup) {                                             // ImpactStatus::Backup (ImpactStatus.h:174-178)
        uint8_t s2 = st.f & (uint8_t)~(ST_LAST_CONTACT | ST_LAST_BOND);
        if (st.f & ST_CONTACT) s2 |= ST_LAST_CONTACT;
        if (st.f & ST_BOND) s2 |= ST_LAST_BOND;
        st.f = s2;
    }
    const double* c = params[pi].c;
    const bool bonded = (is == IS_BSDBF || is == IS_BTSDBF || is == IS_BSDB2F) && normal_bond(c[0], c[4], depth);
    if (!active && !bonded) {                                 // ImpactStatus::Clean, nothing added
        if (st.f & PF_NONZERO) {
            hist[k] = make_double4_32a(0.0, 0.0, 0.0, 0.0);
            v0[k] = 0.0;
        }
        if (f0 != 0) flags[k] = 0;
        return;
    }
    if (st.f & PF_NONZERO) {
        double4_32a h = hist[k];
        st.shear = mk(h.x, h.y, h.z);
        st.kn = h.w;
        st.v0 = v0[k];
    } else {
        st.shear = mk(0.0, 0.0, 0.0);
        st.kn = 0.0;
        st.v0 = 0.0;
    }
    const d3 Va = ld(vel, p.x), Vb = ld(vel, p.y), AVa = ld(av, p.x), AVb = ld(av, p.y);
    d3 J, tA, tB;
    const uint8_t app = solve_pair(is, c, active, depth, n, point, Ps, Pm, Va, Vb, AVa, AVb, dt, pb, st, J, tA, tB);
    if (st.f & PF_NONZERO) {
        hist[k] = make_double4_32a(st.shear.x, st.shear.y, st.shear.z, st.kn);
        v0[k] = st.v0;
    }
    flags[k] = st.f | app | (active ? PF_ACTIVE : 0);
    if (app) {
        double* o = out + 9 * (size_t)k;
        o[0] = J.x; o[1] = J.y; o[2] = J.z;
        o[3] = tA.x; o[4] = tA.y; o[5] = tA.z;
        o[6] = tB.x; o[7] = tB.y; o[8] = tB.z;
        touched[p.x] = 1;              // both objects have an impulse to gather this step
        touched[p.y] = 1;
    }
}

// CalculateImpact.  The FP64 pipe issues a warp instruction in 16 cycles however few of its lanes are
// active, and most candidate pairs are apart, so the pairs that need it are evaluated in full warps: the
// blocks resident at once take the list's tiles of 512 candidates in turn, settle them with the FP32
// prefilter (a pair certainly apart that carries no normal bond gets ImpactStatus::Clean and no impulse)
// and put the others aside in shared memory until there is one for every thread; then narrow phase at
// the present positions, impact solver and status update, each pair's operations those of a pass over
// the list (their order does not matter, every pair writes its own records).  While one block waits for
// its gathers the FP64 pipe works on another's.  With tiles of fixed size per block, evaluated alone, a
// list of a few waves lost up to half in the last rounds (us per step, 60,000-sphere hopper, 58,000
// packed, 150,000-sphere drum: 349, 517, 245; 255, 458, 249 like this; 284, 488, 313 with a prefilter
// kernel and a worklist in memory).  Three blocks an SM at 80 registers and a few spills, against two at
// 112: 255 to 263, 458 to 472, 249 to 267.
constexpr int PAIR_TILE = 2;      // candidates a thread settles per tile
__global__ void __launch_bounds__(TPB, 3) k_pair(uint32_t np, const uint2* __restrict__ sm,
                                              const uint32_t* __restrict__ param, const PairParam* __restrict__ params,
                                              const double4_32a* __restrict__ geom,
                                              const double4_32a* __restrict__ hole, const float2* __restrict__ brief,
                                              const double4_32a* __restrict__ pos, const double4_32a* __restrict__ vel,
                                              const double4_32a* __restrict__ av, const double4_32a* __restrict__ ox,
                                              const double4_32a* __restrict__ oz, const float4* __restrict__ pos32,
                                              const float4* __restrict__ wall32, double4_32a* __restrict__ hist,
                                              double* __restrict__ v0, uint8_t* __restrict__ flags,
                                              double* __restrict__ out, double dt, int backup, Periodic pb,
                                              uint8_t* __restrict__ touched) {
    __shared__ uint32_t list[(PAIR_TILE + 1) * TPB];          // fewer than TPB, and a tile's
    __shared__ uint32_t count;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    const uint32_t tiles = (np + PAIR_TILE * TPB - 1u) / (PAIR_TILE * TPB);
    uint32_t t = blockIdx.x, n = 0;                            // n: the pairs put aside (the same in every thread)
    for (;;) {
        while (n < TPB && t < tiles) {
            const uint32_t base = t * (uint32_t)(PAIR_TILE * TPB) + threadIdx.x;
            t += gridDim.x;
            uint2 p[PAIR_TILE];
            uint32_t pi[PAIR_TILE];
#pragma unroll
            for (int r = 0; r < PAIR_TILE; ++r) {              // (the candidates' loads overlap)
                const uint32_t k = base + r * TPB;
                p[r] = k < np ? sm[k] : make_uint2(0u, 0u);
                pi[r] = k < np ? param[k] : 0u;
            }
#pragma unroll
            for (int r = 0; r < PAIR_TILE; ++r) {
                const uint32_t k = base + r * TPB;
                bool near = false;
                if (k < np) {
                    const float2 br = brief[pi[r]];
                    const int cd = __float_as_int(br.y);
                    if (cd && certainly_apart(cd, pos32[p[r].x], pos32[p[r].y], wall32[p[r].y], br.x,
                                              pb.on ? pb.range32 : nullptr)) {
                        const uint8_t f0 = flags[k];
                        if (f0 & PF_NONZERO) {
                            hist[k] = make_double4_32a(0.0, 0.0, 0.0, 0.0);
                            v0[k] = 0.0;
                        }
                        if (f0 != 0) flags[k] = 0;
                    } else {
                        near = true;
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, near);
                uint32_t at = 0;
                if (lane == 0 && m) at = atomicAdd(&count, (uint32_t)__popc(m));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (near) list[at + __popc(m & ((1u << lane) - 1u))] = k;
            }
            __syncthreads();
            n = count;
            __syncthreads();                                   // (before the next tile adds to it)
        }
        if (n == 0) return;
        const uint32_t take = min(n, (uint32_t)TPB);
        const bool mine = threadIdx.x < take;
        const uint32_t k = mine ? list[n - take + threadIdx.x] : 0u;
        n -= take;
        __syncthreads();
        if (threadIdx.x == 0) count = n;
        if (mine)
            pair_exact(k, sm, param, params, geom, hole, pos, vel, av, ox, oz, hist, v0, flags, out, dt, backup, pb,
                       touched);
        __syncthreads();
    }
}

// An entry's share of its object: the slave's A->AddImpact(ImpactA, tA), the master's
// B->AddImpact(-1.0 * ImpactA, tB); a law without torques adds none.
struct Share {
    d3 J, T;
    bool angular;
};
__device__ __forceinline__ Share load_share(uint32_t ent, uint8_t f, const double* __restrict__ out) {
    const double* o = out + 9 * (size_t)(ent >> 1);
    Share s;
    s.J = mk(o[0], o[1], o[2]);
    if (ent & 1) s.J = neg(s.J);
    s.angular = f & PF_ANGULAR;
    const double* t = o + (ent & 1 ? 6 : 3);
    s.T = s.angular ? mk(t[0], t[1], t[2]) : mk(0.0, 0.0, 0.0);
    return s;
}
__device__ __forceinline__ void add_share(const Share& s, d3& J, d3& JA) {
    J = add(J, s.J);
    if (s.angular) JA = add(JA, s.T);
}

// FP32 copies used by the prefilters: position relative to `origin`, and for plates and
// cylinders the unit axis with a validity flag (plates need an orthogonal Ox/Oz frame for
// the plane bound).
__device__ __forceinline__ void write32(uint32_t i, int shape, d3 P, d3 Ox, d3 Oz, d3 origin,
                                        float4* __restrict__ pos32, float4* __restrict__ wall32) {
    pos32[i] = make_float4((float)(P.x - origin.x), (float)(P.y - origin.y), (float)(P.z - origin.z), 0.0f);
    if (shape != SHAPE_SPHERE) {
        const double lz = len(Oz), lx = len(Ox);
        bool ok = lz > 0.0;
        if (shape == SHAPE_PLATE || shape == SHAPE_HOLED) ok = ok && lx > 0.0 && fabs(dot(Ox, Oz)) <= 1e-9 * lx * lz;
        wall32[i] = ok ? make_float4((float)(Oz.x / lz), (float)(Oz.y / lz), (float)(Oz.z / lz), 1.0f)
                       : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

__device__ __forceinline__ void finish_object(uint32_t i, const ModelDev& m, d3 J, d3 JA, double dt, d3 fimp,
                                              double4_32a* __restrict__ pos, double4_32a* __restrict__ vel,
                                              double4_32a* __restrict__ av, double4_32a* __restrict__ ox,
                                              double4_32a* __restrict__ oz, double4_32a* __restrict__ imp,
                                              double4_32a* __restrict__ aimp, int write_imp, d3 origin,
                                              float4* __restrict__ pos32, float4* __restrict__ wall32,
                                              const double* __restrict__ ext_imp, const double* __restrict__ ext_aimp,
                                              const Periodic& pb) {
    J = add(J, muls(fimp, m.sudo));                           // DOContainer::AddFieldImpact (DOContainer.cpp:25)
    J = add(J, smul(dt, mk(m.ext[0], m.ext[1], m.ext[2])));   // DiscreteObject::AddConstrainedImpact (:160-163)
    if (ext_imp) {                 // SimMediator::Run(external impacts): DOContainer::AddImpact (SimMediator.cpp:1015-1018)
        J = add(J, mk(ext_imp[3 * (size_t)i], ext_imp[3 * (size_t)i + 1], ext_imp[3 * (size_t)i + 2]));
        JA = add(JA, mk(ext_aimp[3 * (size_t)i], ext_aimp[3 * (size_t)i + 1], ext_aimp[3 * (size_t)i + 2]));
    }
    if (m.behavior != BEH_FIXED) {
        d3 P = ld(pos, i), V = ld(vel, i), AV = ld(av, i), Ox = ld(ox, i), Oz = ld(oz, i);
        respond_object(m, dt, J, JA, P, V, AV, Ox, Oz);
        if (pb.on) P = wrap_position(pb, P);                 // DOContainer::EnforcePeriodicBoundaryConditions
        st(pos, i, P, 0.0);
        st(ox, i, Ox, 0.0);
        st(oz, i, Oz, 0.0);
        if (m.behavior != BEH_ORBITAL) {
            st(vel, i, V, 0.0);
            st(av, i, AV, 0.0);
        }
        write32(i, m.shape, P, Ox, Oz, origin, pos32, wall32);
    } else if (pb.on) {            // the wrap moves every object, fixed ones included (SimMediator.cpp:746)
        const d3 P = ld(pos, i), W = wrap_position(pb, P);
        if (W.x != P.x || W.y != P.y || W.z != P.z) {
            st(pos, i, W, 0.0);
            write32(i, m.shape, W, ld(ox, i), ld(oz, i), origin, pos32, wall32);
        }
    }
    if (write_imp) {                                          // DiscreteObject::ClearImpact (:141-147)
        st(imp, i, J, 0.0);
        st(aimp, i, JA, 0.0);
    }
}

struct ObjArgs {
    uint32_t n;
    const uint32_t* model_of;
    const ModelDev* models;
    double4_32a *pos, *vel, *av, *ox, *oz, *imp, *aimp;
    const uint32_t *csr_ptr, *csr_ent;
    const uint8_t* flags;
    const double* out;
    double dt;
    d3 fimp;
    int write_imp;
    d3 origin;
    float4 *pos32, *wall32;
    const double *ext_imp, *ext_aimp;
    Periodic pb;
    uint8_t* touched;
    uint32_t nglob;
    const uint32_t* glob;
    uint32_t per;                      // local objects a block takes, a multiple of 32
};

// One block per scope-global object, when its sum is wanted (its impulse is written, or it responds):
// the entries that applied an impulse, added in entry order, which keeps the reference's summation
// order.  Only the additions are serial: seven warps load and compact the next 224 entries into
// shared memory while the first warp adds the present ones, one component a lane, so that an entry
// costs one dependent FP64 addition.  (One warp that did both, with every lane adding all six
// components from shuffles, took 0.91 ms on the walls of 300,000 packed spheres.)
constexpr int GSUM_TILE = TPB - 32;
__device__ __forceinline__ void global_object(const ObjArgs& a, uint32_t i) {
    __shared__ double buf[2][GSUM_TILE][6];
    __shared__ uint32_t cnt[2], warp_cnt[GSUM_TILE / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0 && a.touched[i]) a.touched[i] = 0;
    const ModelDev& m = a.models[a.model_of[i]];
    double sum = 0.0;                          // component `lane` of (J, JA) in the first warp
    if (a.write_imp || m.behavior == BEH_MOBILE || m.behavior == BEH_CONSTRAINED || a.ext_imp) {
        const uint32_t e0 = a.csr_ptr[i], e1 = a.csr_ptr[i + 1];
        const uint32_t tiles = (e1 - e0 + GSUM_TILE - 1) / GSUM_TILE;
        for (uint32_t t = 0; t <= tiles; ++t) {            // load tile t, add tile t - 1
            if (warp > 0 && t < tiles) {
                const uint32_t e = e0 + t * GSUM_TILE + (threadIdx.x - 32);
                uint32_t ent = 0;
                uint8_t f = 0;
                if (e < e1) {
                    ent = a.csr_ent[e];
                    f = a.flags[ent >> 1];
                }
                const bool app = f & PF_APPLIED;
                const unsigned am = __ballot_sync(0xffffffffu, app);
                if (lane == 0) warp_cnt[warp - 1] = (uint32_t)__popc(am);
                asm volatile("bar.sync 1, 224;" ::: "memory");       // the loading warps
                uint32_t at = (uint32_t)__popc(am & ((1u << lane) - 1u)), total = 0;
                for (int w = 0; w < GSUM_TILE / 32; ++w) {
                    if (w < warp - 1) at += warp_cnt[w];
                    total += warp_cnt[w];
                }
                if (threadIdx.x == 32) cnt[t & 1] = total;
                if (app) {
                    const double* o = a.out + 9 * (size_t)(ent >> 1);
                    double* d = buf[t & 1][at];
                    const bool master = ent & 1;           // B->AddImpact(-1.0 * ImpactA, tB), else A->AddImpact(ImpactA, tA)
                    for (int k = 0; k < 3; ++k) d[k] = master ? -o[k] : o[k];
                    // (an impulse without a torque adds +0, which leaves a sum that started at +0 as it is)
                    for (int k = 0; k < 3; ++k) d[3 + k] = f & PF_ANGULAR ? o[(master ? 6 : 3) + k] : 0.0;
                }
            }
            if (warp == 0 && t > 0 && lane < 6) {
                const uint32_t c = cnt[(t - 1) & 1];
#pragma unroll 8
                for (uint32_t k = 0; k < c; ++k) sum = sum + buf[(t - 1) & 1][k][lane];
            }
            __syncthreads();
        }
    }
    if (warp != 0) return;
    d3 J, JA;
    J.x = __shfl_sync(0xffffffffu, sum, 0);
    J.y = __shfl_sync(0xffffffffu, sum, 1);
    J.z = __shfl_sync(0xffffffffu, sum, 2);
    JA.x = __shfl_sync(0xffffffffu, sum, 3);
    JA.y = __shfl_sync(0xffffffffu, sum, 4);
    JA.z = __shfl_sync(0xffffffffu, sum, 5);
    if (lane == 0)
        finish_object(i, m, J, JA, a.dt, a.fimp, a.pos, a.vel, a.av, a.ox, a.oz, a.imp, a.aimp, a.write_imp, a.origin,
                      a.pos32, a.wall32, a.ext_imp, a.ext_aimp, a.pb);
}

// The first nglob blocks take the scope-global objects (no object reads another's state here, so the
// two run side by side in one launch), the others `per` local objects each, one per thread: FP64 work,
// which a short array spreads over as many SMs as it can (20 steps with their rebuild of 8,000 spheres:
// 1260 us in 32 full blocks, the FP64 pipes of 32 SMs, 1182 in 250 blocks of 32 objects).
__global__ void __launch_bounds__(TPB) k_obj(ObjArgs a) {
    if (blockIdx.x < a.nglob) {
        global_object(a, a.glob[blockIdx.x]);
        return;
    }
    const uint32_t i = (blockIdx.x - a.nglob) * a.per + threadIdx.x;
    if (threadIdx.x >= a.per || i >= a.n) return;
    const ModelDev& m = a.models[a.model_of[i]];
    if (m.scope == SCOPE_GLOBAL) return;
    d3 J = mk(0.0, 0.0, 0.0), JA = mk(0.0, 0.0, 0.0);
    // an object no pair applied an impulse to keeps zero sums: its ordered walk adds nothing
    if (a.touched[i]) {
        a.touched[i] = 0;
        const uint32_t e0 = a.csr_ptr[i], e1 = a.csr_ptr[i + 1];
        // the entries that applied an impulse are marked first (integer work), then summed in entry
        // order: a warp issues each FP64 add once per marked entry of its busiest object, not once
        // per candidate entry.  Flags are loaded eight entries at a time and shares two, or each use waits
        // for its own load
        for (uint32_t c0 = e0; c0 < e1; c0 += 64u) {
            const uint32_t c1 = min(e1, c0 + 64u);
            unsigned long long mark = 0ull;
            for (uint32_t e = c0; e < c1; e += 8u) {
                uint32_t ent[8];
                uint8_t f[8];
#pragma unroll
                for (uint32_t u = 0; u < 8u; ++u) ent[u] = e + u < c1 ? a.csr_ent[e + u] : 0u;
#pragma unroll
                for (uint32_t u = 0; u < 8u; ++u) f[u] = e + u < c1 ? a.flags[ent[u] >> 1] : (uint8_t)0;
#pragma unroll
                for (uint32_t u = 0; u < 8u; ++u)
                    mark |= (unsigned long long)(f[u] & PF_APPLIED ? 1u : 0u) << ((e - c0 + u) & 63u);
            }
            while (mark) {
                const uint32_t ea = a.csr_ent[c0 + (uint32_t)(__ffsll((long long)mark) - 1)];
                mark &= mark - 1;
                const bool two = mark != 0ull;
                const uint32_t eb = two ? a.csr_ent[c0 + (uint32_t)(__ffsll((long long)mark) - 1)] : ea;
                mark &= mark - 1;
                const Share sa = load_share(ea, a.flags[ea >> 1], a.out), sb = load_share(eb, a.flags[eb >> 1], a.out);
                add_share(sa, J, JA);
                if (two) add_share(sb, J, JA);
            }
        }
    }
    finish_object(i, m, J, JA, a.dt, a.fimp, a.pos, a.vel, a.av, a.ox, a.oz, a.imp, a.aimp, a.write_imp, a.origin,
                  a.pos32, a.wall32, a.ext_imp, a.ext_aimp, a.pb);
}

// Narrow phase only: PF_ACTIVE of every pair at the current positions (the IsActive()
// that NBSConsultant::RebuildIactRecordTab reads, NBSConsultant.cpp:384).
__global__ void __launch_bounds__(TPB) k_detect_active(uint32_t np, const uint2* __restrict__ sm,
                                                       const uint32_t* __restrict__ param,
                                                       const PairParam* __restrict__ params,
                                                       const double4_32a* __restrict__ geom,
                                                       const double4_32a* __restrict__ hole,
                                                       const float* __restrict__ reach,
                                                       const double4_32a* __restrict__ pos, const double4_32a* __restrict__ ox,
                                                       const double4_32a* __restrict__ oz,
                                                       const float4* __restrict__ pos32,
                                                       const float4* __restrict__ wall32, uint8_t* __restrict__ flags,
                                                       Periodic pb) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= np) return;
    const uint2 p = sm[k];
    const uint32_t pi = param[k];
    const uint8_t f = flags[k];
    double depth = -1.0;
    if (!certainly_apart(params[pi].cd, pos32[p.x], pos32[p.y], wall32[p.y], reach[pi], pb.on ? pb.range32 : nullptr)) {
        const double4_32a gg = geom[pi];
        PairGeom g{gg.x, gg.y, gg.z, gg.w, 0.0, 0.0, 0.0};
        if (params[pi].cd == CD_SHP) {
            const double4_32a hh = hole[pi];
            g.hr = hh.x; g.hxo = hh.y; g.hyo = hh.z;
        }
        d3 n, point;
        detect_pair(params[pi].cd, g, ld(pos, p.x), ld(pos, p.y), ox, oz, p.y, pb, depth, n, point);
    }
    const uint8_t nf = depth > 0.0 ? (uint8_t)(f | PF_ACTIVE) : (uint8_t)(f & ~PF_ACTIVE);
    if (nf != f) flags[k] = nf;
}

// ------------------------------------------------------------------------------------
// broad phase (NBSConsultant::Reset, NBSConsultant.cpp:85-316)
// (A few blocks per SM, each reduced to one set of atomics: eight same-address 64-bit atomics a warp
// took 29 us for 150,000 objects.)
__global__ void __launch_bounds__(TPB) k_safe(uint32_t n, const uint32_t* __restrict__ model_of,
                                              const ModelDev* __restrict__ models, const double4_32a* __restrict__ pos,
                                              const double4_32a* __restrict__ vel, double sf, double dtu, double glen,
                                              double* __restrict__ safe, unsigned long long* __restrict__ red) {
    __shared__ unsigned long long sh[8][TPB / 32];
    unsigned long long v[8] = {~0ull, 0, ~0ull, 0, ~0ull, 0, 0, 0};    // min, max per axis; speed; last local object + 1
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ModelDev& m = models[model_of[i]];
        const double vl = len(ld(vel, i));
        safe[i] = sf * (2.0 * m.range + dtu * vl + 0.5 * dtu * dtu * glen);   // :127-129
        if (m.scope != SCOPE_LOCAL) continue;                                  // :131-141
        const double4_32a p = pos[i];
        const unsigned long long o[3] = {ord_of(p.x), ord_of(p.y), ord_of(p.z)};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            v[2 * q] = min(v[2 * q], o[q]);
            v[2 * q + 1] = max(v[2 * q + 1], o[q]);
        }
        v[6] = max(v[6], ord_of(vl));
        v[7] = max(v[7], (unsigned long long)i + 1);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const bool least = q < 6 && !(q & 1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long x = __shfl_xor_sync(0xffffffffu, v[q], o);
            v[q] = least ? min(v[q], x) : max(v[q], x);
        }
        if ((threadIdx.x & 31) == 0) sh[q][threadIdx.x >> 5] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        const int q = threadIdx.x;
        const bool least = q < 6 && !(q & 1);
        unsigned long long x = sh[q][0];
        for (int w = 1; w < TPB / 32; ++w) x = least ? min(x, sh[q][w]) : max(x, sh[q][w]);
        if (least) atomicMin(&red[q], x);
        else atomicMax(&red[q], x);
    }
}

__global__ void __launch_bounds__(TPB) k_cellkey(uint32_t n, const uint32_t* __restrict__ model_of,
                                                 const ModelDev* __restrict__ models, const double4_32a* __restrict__ pos,
                                                 double xmin, double ymin, double zmin, double zone, CellGrid g,
                                                 uint64_t sentinel, uint64_t* __restrict__ key,
                                                 uint32_t* __restrict__ sid) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t k = sentinel;
    if (models[model_of[i]].scope == SCOPE_LOCAL) {          // NBS :163-178, Leap LeapConsultant.h:160-170
        const double4_32a p = pos[i];
        const uint64_t c[3] = {(uint32_t)((p.x - xmin) / zone), (uint32_t)((p.y - ymin) / zone),
                               (uint32_t)((p.z - zmin) / zone)};
        k = grid_key(g, c);
    }
    key[i] = k;
    sid[i] = i;
}

// One axis of the local objects' positions as sortable keys (others sort last): the Leap
// consultant's spans come from the sorted positions (LeapConsultant.cpp:143-168).
__global__ void __launch_bounds__(TPB) k_axis_key(uint32_t n, const uint32_t* __restrict__ model_of,
                                                  const ModelDev* __restrict__ models,
                                                  const double4_32a* __restrict__ pos, int axis,
                                                  uint64_t* __restrict__ key, uint32_t* __restrict__ sid) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t k = ~0ull;
    if (models[model_of[i]].scope == SCOPE_LOCAL) {
        const double4_32a p = pos[i];
        k = ord_of(axis == 0 ? p.x : axis == 1 ? p.y : p.z);
    }
    key[i] = k;
    sid[i] = i;
}

__global__ void __launch_bounds__(TPB) k_cell_flags(uint32_t nloc, const uint64_t* __restrict__ key,
                                                    uint32_t* __restrict__ flag) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nloc) return;
    flag[p] = (p == 0 || key[p] != key[p - 1]) ? 1u : 0u;
}

// One sphere's part of the distance beyond which a pair of spheres is certainly no candidate: its safe
// length, rounded up, and the rounding of its FP32 position (prefilter.cuh's dist32 bound).
__device__ __forceinline__ float pair_limit(const float4& q, double safe) {
    return (float)safe * (1.0f + 16.0f * PF_ARITH_EPS) + PF_POS_EPS * 1.0001f * l1(q);
}
__global__ void __launch_bounds__(TPB) k_cell_fill(uint32_t nloc, const uint64_t* __restrict__ key,
                                                   const uint32_t* __restrict__ flag_excl,
                                                   uint64_t* __restrict__ cell_key, uint32_t* __restrict__ cell_start,
                                                   uint32_t* __restrict__ cellof, const uint32_t* __restrict__ ncells,
                                                   uint32_t* __restrict__ grid,
                                                   const uint32_t* __restrict__ sid, const uint32_t* __restrict__ model_of,
                                                   const ModelDev* __restrict__ models,
                                                   const float4* __restrict__ pos32, const double* __restrict__ safe,
                                                   float4* __restrict__ rec) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nloc) return;
    const bool head = (p == 0 || key[p] != key[p - 1]);
    const uint32_t c = head ? flag_excl[p] : flag_excl[p] - 1u;   // index of p's cell
    cellof[p] = c;
    if (head) {
        cell_key[c] = key[p];
        cell_start[c] = p;
        if (grid) grid[key[p]] = c;                              // the dense map of a small grid
    }
    if (p == nloc - 1) cell_start[*ncells] = nloc;
    // what the candidate test reads of an object, in cell order: its FP32 position, and its safe length
    // with its share of the test's error allowance (other shapes: no pair with them is settled by it)
    const uint32_t i = sid[p];
    const float4 q = pos32[i];
    rec[p] = make_float4(q.x, q.y, q.z, models[model_of[i]].shape == SHAPE_SPHERE ? pair_limit(q, safe[i]) : __int_as_float(0x7f800000));
}

// Candidate test of BuildIactTab (NBSConsultant.cpp:318-345): DOMap::CalDistance <= safe_i +
// safe_j, decided from FP32 bounds where they are conclusive and in exact FP64 otherwise.
// pb: the Leap consultant's distance takes the boundary's minimum image (nullptr: NBS's does not)
__device__ __forceinline__ bool candidate(const ModelDev& mi, const ModelDev& mj, uint32_t i, uint32_t j, double si,
                                          double sj, float si32, float sj32, const double4_32a* __restrict__ pos,
                                          const double4_32a* __restrict__ ox, const double4_32a* __restrict__ oz,
                                          const float4* __restrict__ pos32, const float4* __restrict__ wall32,
                                          int* __restrict__ err, const Periodic* pb) {
    const float thr = si32 + sj32;                     // float sums of the rounded-to-float safe lengths
    const float tlo = thr * (1.0f - 4.0f * PF_ARITH_EPS), thi = thr * (1.0f + 4.0f * PF_ARITH_EPS);
    if (pb) {
        // periodic: the least distance over the images bounds the detector's from below (the
        // certain-candidate shortcut is not taken: the image the reference picks may be another)
        if (mi.shape == SHAPE_SPHERE && mj.shape == SHAPE_SPHERE) {
            float e;
            const float d = dist32_periodic(pos32[i], pos32[j], pb->range32, e);
            if (d - e > thi) return false;
        }
    } else if (mi.shape == SHAPE_SPHERE && mj.shape == SHAPE_SPHERE) {
        float e;
        const float d = dist32(pos32[i], pos32[j], e);
        if (d - e > thi) return false;
        if (d + e < tlo) return true;
    } else {
        const bool ip = mi.shape != SHAPE_SPHERE;      // the non-sphere member
        const uint32_t w = ip ? i : j, sp = ip ? j : i;
        const int wshape = ip ? mi.shape : mj.shape;
        const float4 wl = wall32[w];
        if (wl.w != 0.0f && (wshape == SHAPE_PLATE || wshape == SHAPE_HOLED || wshape == SHAPE_CYL) &&
            (ip ? mj.shape : mi.shape) == SHAPE_SPHERE) {
            float e;
            const float d = wshape != SHAPE_CYL ? plane_dist32(pos32[sp], pos32[w], wl, e)
                                                  : line_dist32(pos32[sp], pos32[w], wl, e);
            if (d - e > thi) return false;
        } else if (wl.w != 0.0f && wshape == SHAPE_INNER_CYL && (ip ? mj.shape : mi.shape) == SHAPE_SPHERE) {
            // the distance to the shell is at least R minus the axis distance (rim included)
            float e;
            const float d = line_dist32(pos32[sp], pos32[w], wl, e);
            const float R = (float)(ip ? mi.a0 : mj.a0) * (1.0f - 4.0f * PF_ARITH_EPS);
            if (R - (d + e) > thi) return false;
        }
    }
    bool ok;
    const double d = cal_distance(mi, mj, i, j, pos, ox, oz, pb, ok);
    if (!ok) {
        atomicOr(err, ERR_BAD_SHAPE_PAIR);
        return false;
    }
    return !(d > (si + sj));
}

// One thread per (slot, object) task, slot-major so that a warp works on one slot.  Tasks
// are numbered in the reference's traversal order: cell by cell (ix, iy, iz lexicographic),
// within a cell by slot, within a slot by the object's position in the cell (ascending id).
// The count pass leaves which of a task's objects are candidates in a word (tasks of up to 32, nearly
// all), so that the fill pass evaluates no distance again.
template <bool FILL>
__global__ void __launch_bounds__(TPB, 3) k_pairs(uint32_t nloc, const uint32_t* __restrict__ sid,
                                               const uint64_t* __restrict__ cell_key,
                                               const uint32_t* __restrict__ cell_start,
                                               const uint32_t* __restrict__ ncells_p, const uint32_t* __restrict__ cellof,
                                               const uint32_t* __restrict__ grid, uint64_t grid_cells,
                                               const uint32_t* __restrict__ glob, uint32_t nglob,
                                               const uint32_t* __restrict__ model_of, const ModelDev* __restrict__ models,
                                               const int* __restrict__ group_iact, int G,
                                               const double4_32a* __restrict__ pos, const double4_32a* __restrict__ ox,
                                               const double4_32a* __restrict__ oz, const float4* __restrict__ pos32,
                                               const float4* __restrict__ wall32, const double* __restrict__ safe,
                                               const float4* __restrict__ rec,
                                               CellGrid g, Periodic pbv, uint32_t nm, int all_interact,
                                               const uint8_t* __restrict__ refused,
                                               uint32_t* __restrict__ task, uint32_t* __restrict__ picked,
                                               uint32_t* __restrict__ first,
                                               uint32_t* __restrict__ second, int* __restrict__ err) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (uint64_t)nloc * NSLOT) return;
    const int s = (int)(t / nloc);
    const uint32_t P = (uint32_t)(t % nloc);
    const uint32_t c = cellof[P];
    uint64_t cc[3];
    grid_cell(g, cell_key[c], cc);
    const uint32_t cs = cell_start[c], csize = cell_start[c + 1] - cs;
    const uint64_t tid = (uint64_t)cs * NSLOT + (uint64_t)s * csize + (P - cs);
    // the fill pass knows each task's count from the scanned offsets (the next task's offset, or
    // the total after the last one): it stops at its last candidate and skips empty tasks
    const uint32_t off = FILL ? task[tid] : 0u;
    uint32_t want = 0xffffffffu;
    if (FILL) {
        want = ((uint64_t)tid + 1 < (uint64_t)nloc * NSLOT ? task[tid + 1] : ncells_p[1]) - off;
        if (want == 0u) return;
    }
    // NBS: only cells inside the loops are primary (:186-190); Leap visits every zone of its map
    if (!g.leap && (cc[0] >= g.ncel[0] || cc[1] >= g.ncel[1] || cc[2] >= g.ncel[2])) {
        if (!FILL) task[tid] = 0;
        return;
    }
    const int slot_self = g.leap ? 13 : SLOT_SELF, slot_global = g.leap ? 14 : SLOT_GLOBAL;
    const uint32_t* js = nullptr;
    uint32_t jn = 0;
    // the cell whose zone coordinates are w (its index, or none)
    auto find_cell = [&](const uint64_t w[3]) -> uint32_t {
#pragma unroll
        for (int a = 0; a < 3; ++a)
            if (w[a] >= g.dim[a]) return 0xffffffffu;
        const uint64_t nk = grid_key(g, w);
        if (grid) return nk < grid_cells ? grid[nk] : 0xffffffffu;
        const uint32_t nc = *ncells_p;
        uint32_t lo = 0, hi = nc;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (cell_key[mid] < nk) lo = mid + 1; else hi = mid;
        }
        return (lo < nc && cell_key[lo] == nk) ? lo : 0xffffffffu;
    };
    if (s == slot_self) {                                     // BuildIactTab(v), :347-374
        js = sid + P + 1;
        jn = cs + csize - (P + 1);
    } else if (s == slot_global) {                            // BuildIactTab(v, GlobalElement), :266
        js = glob;
        jn = nglob;
    } else if (g.leap || s < NSLOT) {
        int d[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) d[a] = g.leap ? c_slot_leap[s][a] : c_slot[s][a];
        uint32_t c2 = 0xffffffffu;
        if (!((cc[0] == 0 && d[0] < 0) || (cc[1] == 0 && d[1] < 0) || (cc[2] == 0 && d[2] < 0))) {
            const uint64_t w[3] = {cc[0] + d[0], cc[1] + d[1], cc[2] + d[2]};
            c2 = find_cell(w);
        }
        if (c2 == 0xffffffffu && g.leap && g.has_pbc) {
            // the neighbour's periodic image (LeapConsultant.h:199-440): on an axis stepping down
            // from zone 0 (up from the last zone) it wraps when that axis is periodic; ids are
            // _uint_t, and an image that names the opposite neighbour is skipped
            bool at_edge = false, dup = false, valid = true;
            uint64_t w[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const uint32_t ia = (uint32_t)cc[a], mx = g.ncel[a] - 1u;
                uint32_t wa = ia;
                if (d[a] < 0) {
                    at_edge |= ia == 0u;
                    wa = g.pbc[a] ? mx : ia - 1u;
                    dup |= wa == ia + 1u;
                } else if (d[a] > 0) {
                    at_edge |= ia == mx;
                    wa = g.pbc[a] ? 0u : ia + 1u;
                    dup |= wa == ia - 1u;
                }
                valid &= wa != 0xffffffffu;
                w[a] = wa;
            }
            if (at_edge && !dup && valid) c2 = find_cell(w);
        }
        if (c2 != 0xffffffffu) {
            js = sid + cell_start[c2];
            jn = cell_start[c2 + 1] - cell_start[c2];
        }
    }
    const uint32_t i = sid[P];
    uint32_t cnt = 0;
    if (FILL && jn <= 32u) {
        for (uint32_t m = picked[t]; m; m &= m - 1u) {
            const uint32_t j = js[__ffs((int)m) - 1];
            first[off + cnt] = i < j ? i : j;
            second[off + cnt] = i < j ? j : i;
            ++cnt;
        }
        return;
    }
    const uint32_t mdi = model_of[i];
    const ModelDev& mi = models[mdi];
    const double si = safe[i];
    const float si32 = (float)si;
    const int gi = mi.group;
    uint32_t mask = 0u;
    // spheres of a cell against a sphere: the records in cell order settle nearly all that are no
    // candidates from one contiguous load and a squared distance
    const bool quick = s != slot_global && mi.shape == SHAPE_SPHERE && !(g.leap && pbv.on);
    const uint32_t b0 = quick && jn ? (uint32_t)(js - sid) : 0u;
    const float4 pi32 = pos32[i];
    const float mine = pair_limit(pi32, si), slack = 2.1f * PF_POS_EPS * l1(pi32);
    for (uint32_t q = 0; q < jn && cnt < want; ++q) {
        if (quick) {
            const float4 r = rec[b0 + q];
            const float dx = r.x - pi32.x, dy = r.y - pi32.y, dz = r.z - pi32.z, lim = mine + r.w;
            const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            if (d2 > lim * lim * (1.0f + 16.0f * PF_ARITH_EPS)) continue;
            // certainly within: the limits less twice their allowances (an infinite one: not settled here)
            const float in = lim * (1.0f - 64.0f * PF_ARITH_EPS) - slack - 2.1f * PF_POS_EPS * l1(r);
            if (all_interact && lim < 3e38f && in > 0.0f && d2 < in * in * (1.0f - 16.0f * PF_ARITH_EPS)) {
                if (FILL) {
                    const uint32_t j = js[q];
                    first[off + cnt] = i < j ? i : j;
                    second[off + cnt] = i < j ? j : i;
                } else if (q < 32u) {
                    mask |= 1u << q;
                }
                ++cnt;
                continue;
            }
        }
        const uint32_t j = js[q];
        const uint32_t mdj = model_of[j];
        const ModelDev& mj = models[mdj];
        if (group_iact[gi * G + mj.group] < 0) continue;
        const double sj = safe[j];
        if (!candidate(mi, mj, i, j, si, sj, si32, (float)sj, pos, ox, oz, pos32, wall32, err,
                       g.leap && pbv.on ? &pbv : nullptr)) continue;
        if (FILL) {
            first[off + cnt] = i < j ? i : j;
            second[off + cnt] = i < j ? j : i;
        } else {
            if (q < 32u) mask |= 1u << q;
            // no interaction of an object with itself (Assembler.cpp:27-30): the Leap consultant lists such
            // pairs when a periodic axis is one zone wide, and the reference then drops them, leaving its
            // pair table and interactions misaligned; here the list is refused
            if (i == j || refused[i < j ? mdi * nm + mdj : mdj * nm + mdi]) atomicOr(err, ERR_UNSUPPORTED_PAIR);
        }
        ++cnt;
    }
    if (!FILL) picked[t] = mask;
    if (!FILL) task[tid] = cnt;
}

__global__ void __launch_bounds__(TPB) k_refresh32(uint32_t n, const uint32_t* __restrict__ model_of,
                                                   const ModelDev* __restrict__ models,
                                                   const double4_32a* __restrict__ pos,
                                                   const double4_32a* __restrict__ ox,
                                                   const double4_32a* __restrict__ oz, d3 origin,
                                                   float4* __restrict__ pos32, float4* __restrict__ wall32) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    write32(i, models[model_of[i]].shape, ld(pos, i), ld(ox, i), ld(oz, i), origin, pos32, wall32);
}

// What a new pair needs, in one pass over the list: its orientation and model (Assembler::
// CreateInteraction, Assembler.cpp:15-87), its two per-object entries to be sorted, and its history.
// REC: from the IactRecordTab read with the scene (IactRecordTab::GetImpactStatus, IactRecordTab.cpp:20-25;
// records sorted by (first << 32 | second)).  Else carried: the status of the same (first, second) pair of
// the old list when that pair is active at the present positions (RebuildIactRecordTab + Initiate,
// NBSConsultant.cpp:376-395, SimMediator.cpp:690-707), otherwise a default-constructed ImpactStatus.  Only a
// new pair that is active needs the old list, so the narrow phase runs on the pairs near contact here and
// not on every pair of the old list first, and in full warps like k_pair's (150,000-sphere drum: set-up,
// that pass, carry and entries took 211 us, 269 in one pass with a lane each, 187 like this).
constexpr uint32_t SETUP_MAX = 4;     // most rounds of pairs a block takes
struct HistorySource {
    const uint64_t* rkey;              // records
    uint32_t nrec;
    const double4_32a* hist;           // records, or the old list
    const double* v0;
    const uint8_t* flags;
    const uint32_t *ptr, *ent, *first, *second;     // the old list
};
template <bool REC>
__global__ void __launch_bounds__(TPB) k_setup(uint32_t np, uint32_t per, const uint32_t* __restrict__ first,
                                               const uint32_t* __restrict__ second,
                                               const uint32_t* __restrict__ model_of,
                                               const ModelDev* __restrict__ models,
                                               const PairParam* __restrict__ params, uint32_t nm,
                                               const uint8_t* __restrict__ refused,
                                               const double4_32a* __restrict__ geom, const double4_32a* __restrict__ hole,
                                               const float* __restrict__ reach, const double4_32a* __restrict__ pos,
                                               const double4_32a* __restrict__ ox, const double4_32a* __restrict__ oz,
                                               const float4* __restrict__ pos32, const float4* __restrict__ wall32,
                                               Periodic pb, HistorySource src, uint2* __restrict__ sm,
                                               uint32_t* __restrict__ param, uint32_t* __restrict__ ckey,
                                               uint32_t* __restrict__ cval, double4_32a* __restrict__ hist,
                                               double* __restrict__ v0, uint8_t* __restrict__ flags) {
    __shared__ uint32_t list[SETUP_MAX * TPB];
    __shared__ uint32_t count;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    for (uint32_t r = 0; r < per; ++r) {
        const uint32_t k = (blockIdx.x * per + r) * TPB + threadIdx.x;
        bool near = false;
        if (k < np) {
            const uint32_t a = first[k], b = second[k];
            const uint32_t ma = model_of[a], mb = model_of[b];
            const ModelDev& A = models[ma];
            const ModelDev& B = models[mb];
            uint2 p = make_uint2(a, b);
            if (A.shape > B.shape) p = make_uint2(b, a);
            else if (A.shape == B.shape && A.density == 0.0) p = make_uint2(b, a);
            uint32_t pi = p.x == a ? ma * nm + mb : mb * nm + ma;
            if (a == b || refused[ma * nm + mb]) {            // (the list is refused)
                p = make_uint2(a, b);
                pi = 0;
            }
            sm[k] = p;
            param[k] = pi;
            reinterpret_cast<uint2*>(ckey)[k] = p;
            reinterpret_cast<uint2*>(cval)[k] = make_uint2(2 * k, 2 * k + 1);
            uint8_t f = ST_DEFAULT;
            double4_32a h = make_double4_32a(0.0, 0.0, 0.0, 0.0);
            double vv = 0.0;
            if (REC) {
                const uint64_t key = ((uint64_t)a << 32) | b;
                uint32_t lo = 0, hi = src.nrec;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (src.rkey[mid] < key) lo = mid + 1; else hi = mid;
                }
                if (lo < src.nrec && src.rkey[lo] == key) {
                    h = src.hist[lo];
                    vv = src.v0[lo];
                    f = src.flags[lo];
                }
            } else {
                near = params[pi].cd != 0 && !certainly_apart(params[pi].cd, pos32[p.x], pos32[p.y], wall32[p.y],
                                                              reach[pi], pb.on ? pb.range32 : nullptr);
            }
            hist[k] = h;
            v0[k] = vv;
            flags[k] = f;
        }
        if (REC) continue;
        const unsigned m = __ballot_sync(0xffffffffu, near);
        uint32_t at = 0;
        if (lane == 0 && m) at = atomicAdd(&count, (uint32_t)__popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (near) list[at + __popc(m & ((1u << lane) - 1u))] = k;
    }
    if (REC) return;
    __syncthreads();
    const uint32_t nw = count;
    for (uint32_t q = threadIdx.x; q < nw; q += TPB) {         // the FP64 narrow phase in full warps
        const uint32_t k = list[q], pi = param[k];
        const uint2 p = sm[k];
        const double4_32a gg = geom[pi];
        PairGeom g{gg.x, gg.y, gg.z, gg.w, 0.0, 0.0, 0.0};
        if (params[pi].cd == CD_SHP) {
            const double4_32a hh = hole[pi];
            g.hr = hh.x; g.hxo = hh.y; g.hyo = hh.z;
        }
        double depth;
        d3 n, point;
        detect_pair(params[pi].cd, g, ld(pos, p.x), ld(pos, p.y), ox, oz, p.y, pb, depth, n, point);
        if (!(depth > 0.0)) continue;
        const uint32_t a = first[k], b = second[k], e1 = src.ptr[a + 1];
        for (uint32_t e = src.ptr[a]; e < e1; ++e) {
            const uint32_t ko = src.ent[e] >> 1;
            if (src.first[ko] != a || src.second[ko] != b) continue;
            const uint8_t of = src.flags[ko];
            if (of & PF_NONZERO) {
                hist[k] = src.hist[ko];
                v0[k] = src.v0[ko];
            }
            flags[k] = of & (PF_STATUS | PF_NONZERO);
            break;
        }
    }
}

// Where each object's entries begin in the sorted keys.  BY_KEY: a thread per entry marks the objects
// between its key and the one before it (with fewer entries than objects, or above a million, a thread
// per object searches; 8,000 objects of 34 entries: 9.6 us searched, 3.2 marked; 150,000 of 44: 13, 18).
template <bool BY_KEY>
__global__ void __launch_bounds__(TPB) k_csr_ptr(uint32_t n, const uint32_t* __restrict__ key, uint32_t m,
                                                 uint32_t* __restrict__ ptr) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (BY_KEY) {
        uint32_t q0 = 1u, q1 = 0u;                             // objects [q0, q1] begin at entry i
        if (i <= m) {
            q0 = i ? key[i - 1] + 1u : 0u;
            q1 = i < m ? key[i] : n;
        }
        const bool wide = q0 + 32u < q1;                        // a long gap: the warp fills it
        if (!wide)
            for (uint32_t q = q0; q <= q1; ++q) ptr[q] = i;
        for (unsigned w = __ballot_sync(0xffffffffu, wide); w; w &= w - 1u) {
            const int l = __ffs((int)w) - 1;
            const uint32_t a = __shfl_sync(0xffffffffu, q0, l), b = __shfl_sync(0xffffffffu, q1, l),
                           at = __shfl_sync(0xffffffffu, i, l);
            for (uint32_t q = a + (threadIdx.x & 31u); q <= b; q += 32u) ptr[q] = at;
        }
        return;
    }
    if (i > n) return;
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (key[mid] < i) lo = mid + 1; else hi = mid;
    }
    ptr[i] = lo;
}

}  // namespace

// ====================================================================================
#define CK(call)                                                  \
    do {                                                          \
        cudaError_t _e = (call);                                  \
        if (_e != cudaSuccess) return cuda_fail(_e, #call);       \
    } while (0)

int Engine::cuda_fail(cudaError_t e, const char* where) {
    err_ = std::string("CUDA error ") + cudaGetErrorString(e) + " at " + where;
    return e == cudaErrorMemoryAllocation ? VEDO_ERR_OUT_OF_MEMORY : VEDO_ERR_CUDA;
}

template <class T>
static cudaError_t dalloc(T** p, size_t count) {
    *p = nullptr;
    if (count == 0) count = 1;
    return cudaMalloc((void**)p, sizeof(T) * count);
}

void Engine::free_list(PairList& L) {
    cudaFree(L.first); cudaFree(L.second); cudaFree(L.sm); cudaFree(L.param); cudaFree(L.hist); cudaFree(L.v0);
    cudaFree(L.flags); cudaFree(L.out); cudaFree(L.csr_ent); cudaFree(L.csr_ptr);
    L = PairList{};
}

int Engine::ensure_list(PairList& L, uint32_t cap) {
    if (L.csr_ptr == nullptr) CK(dalloc(&L.csr_ptr, (size_t)n_ + 1));
    if (cap <= L.cap && L.first) return VEDO_OK;
    uint32_t* ptr = L.csr_ptr;
    L.csr_ptr = nullptr;
    free_list(L);
    L.csr_ptr = ptr;
    uint64_t c = std::max<uint64_t>(1024, (uint64_t)cap + cap / 4);
    if (c > 0x7fffffffull) c = 0x7fffffffull;
    L.cap = (uint32_t)c;
    CK(dalloc(&L.first, c)); CK(dalloc(&L.second, c)); CK(dalloc(&L.sm, c)); CK(dalloc(&L.param, c));
    CK(dalloc(&L.hist, c)); CK(dalloc(&L.v0, c)); CK(dalloc(&L.flags, c)); CK(dalloc(&L.out, 9 * c));
    CK(dalloc(&L.csr_ent, 2 * c));
    return VEDO_OK;
}

Engine::~Engine() {
    if (status_) std::fclose(status_);
    if (stream_) cudaStreamSynchronize(stream_);
    free_list(cur_);
    free_list(old_);
    void* ptrs[] = {d_models_, d_params_, d_geom_, d_group_iact_, d_model_of_, d_refused_, d_picked_, d_bp_, d_brief_, d_pos_, d_vel_, d_av_, d_ox_,
                    d_oz_, d_imp_, d_aimp_, d_global_, d_safe_, d_red_, d_key_, d_key_alt_, d_cell_key_, d_sid_,
                    d_sid_alt_, d_cell_start_, d_cellof_, d_flag_, d_task_, d_total_, d_ck_, d_cv_, d_ck_alt_,
                    d_cv_alt_, d_cnt_, d_rec_key_, d_rec_hist_, d_rec_v0_, d_rec_flags_, d_obs_, d_stage_,
                    d_pos32_, d_wall32_, d_reach_, d_grid_, d_ext_, d_hole_, d_touched_};
    for (void* p : ptrs) if (p) cudaFree(p);
    for (auto& e : ev_) if (e) cudaEventDestroy(e);
    if (stream_) cudaStreamDestroy(stream_);
}

static void upload3(std::vector<double4_32a>& tmp, const std::vector<double>& v, uint32_t n) {
    tmp.resize(n);
    for (uint32_t i = 0; i < n; ++i) tmp[i] = make_double4_32a(v[3 * i], v[3 * i + 1], v[3 * i + 2], 0.0);
}

int Engine::init(const HScene& scene, const vedo_engine_opts& opts) {
    host_ = scene;
    opts_ = opts;
    if (opts_.up_iact == 0) opts_.up_iact = 1;
    if (opts_.consultant > 1) return fail(VEDO_ERR_INVALID_ARGUMENT, "unknown consultant");
    leap_ = opts_.consultant == 1;
    out_prefix_ = opts.output_prefix ? opts.output_prefix : "";
    std::string msg;
    int rc = build_tables(host_, tab_, msg);
    if (rc != VEDO_OK) return fail(rc, msg);
    zoi_on_ = host_.zoi_switch[0] || host_.zoi_switch[1] || host_.zoi_switch[2];
    n_ = host_.n;
    nm_ = (uint32_t)tab_.models.size();
    dt_ = host_.time_interval;
    t_ = host_.time_current;
    t_stop_ = host_.time_stop;
    sf_ = host_.safety_factor;
    for (int k = 0; k < 3; ++k) g_[k] = host_.g[k];
    device_ = opts.device;
    CK(cudaSetDevice(device_));
    CK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    for (auto& e : ev_) CK(cudaEventCreate(&e));
    // constant tables
    CK(dalloc(&d_models_, nm_));
    CK(cudaMemcpy(d_models_, tab_.models.data(), sizeof(ModelDev) * nm_, cudaMemcpyHostToDevice));
    CK(dalloc(&d_params_, (size_t)nm_ * nm_));
    CK(cudaMemcpy(d_params_, tab_.params.data(), sizeof(PairParam) * nm_ * nm_, cudaMemcpyHostToDevice));
    std::vector<double4_32a> geo((size_t)nm_ * nm_);
    for (size_t q = 0; q < geo.size(); ++q)
        geo[q] = make_double4_32a(tab_.geom[4 * q], tab_.geom[4 * q + 1], tab_.geom[4 * q + 2], tab_.geom[4 * q + 3]);
    CK(dalloc(&d_geom_, geo.size()));
    CK(cudaMemcpy(d_geom_, geo.data(), sizeof(double4_32a) * geo.size(), cudaMemcpyHostToDevice));
    for (size_t q = 0; q < geo.size(); ++q)
        geo[q] = make_double4_32a(tab_.hole[4 * q], tab_.hole[4 * q + 1], tab_.hole[4 * q + 2], 0.0);
    CK(dalloc(&d_hole_, geo.size()));
    CK(cudaMemcpy(d_hole_, geo.data(), sizeof(double4_32a) * geo.size(), cudaMemcpyHostToDevice));
    const int G = tab_.ngroups;
    CK(dalloc(&d_group_iact_, (size_t)G * G));
    CK(cudaMemcpy(d_group_iact_, tab_.group_iact.data(), sizeof(int) * G * G, cudaMemcpyHostToDevice));
    CK(dalloc(&d_model_of_, n_));
    CK(cudaMemcpy(d_model_of_, host_.model_of.data(), sizeof(uint32_t) * n_, cudaMemcpyHostToDevice));
    // pairs of models the Assembler makes no interaction of (Assembler.cpp:27-87), by the models of the
    // lower and the higher object
    std::vector<uint8_t> refused((size_t)nm_ * nm_);
    for (uint32_t a = 0; a < nm_; ++a)
        for (uint32_t b = 0; b < nm_; ++b) {
            const ModelDev &A = tab_.models[a], &B = tab_.models[b];
            bool swap = false;                                 // the higher object is the slave
            if (A.shape > B.shape) swap = true;
            else if (A.shape == B.shape) swap = A.density == 0.0;
            refused[(size_t)a * nm_ + b] = A.density < 0.0 || B.density < 0.0 || (A.density == 0.0 && B.density == 0.0) ||
                                           tab_.params[swap ? (size_t)b * nm_ + a : (size_t)a * nm_ + b].cd == 0;
        }
    // whether every two sphere models interact: the candidate test then needs no look at the models
    all_interact_ = 1;
    for (uint32_t a = 0; a < nm_; ++a)
        for (uint32_t b = 0; b < nm_; ++b)
            if (tab_.models[a].shape == SHAPE_SPHERE && tab_.models[b].shape == SHAPE_SPHERE &&
                (refused[(size_t)a * nm_ + b] ||
                 tab_.group_iact[(size_t)tab_.models[a].group * tab_.ngroups + tab_.models[b].group] < 0))
                all_interact_ = 0;
    CK(dalloc(&d_refused_, refused.size()));
    CK(cudaMemcpy(d_refused_, refused.data(), refused.size(), cudaMemcpyHostToDevice));
    // objects
    std::vector<double4_32a> tmp;
    double4_32a** dst[] = {&d_pos_, &d_vel_, &d_av_, &d_ox_, &d_oz_, &d_imp_, &d_aimp_};
    const std::vector<double>* src[] = {&host_.pos, &host_.vel, &host_.av, &host_.ox, &host_.oz, &host_.imp, &host_.aimp};
    for (int k = 0; k < 7; ++k) {
        CK(dalloc(dst[k], n_));
        upload3(tmp, *src[k], n_);
        CK(cudaMemcpy(*dst[k], tmp.data(), sizeof(double4_32a) * n_, cudaMemcpyHostToDevice));
    }
    for (uint32_t i = 0; i < n_; ++i)
        if (tab_.models[host_.model_of[i]].scope != SCOPE_LOCAL) global_ids_.push_back(i);
        else leap_rmax_ = std::max(leap_rmax_, tab_.models[host_.model_of[i]].range);
    if (leap_ && global_ids_.size() == n_)           // the reference indexes an empty vector
        return fail(VEDO_ERR_INVALID_SCENE, "the Leap consultant needs a local object");
    // FP32 prefilter copies: origin at the centre of the initial bounding box
    {
        double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
        for (uint32_t i = 0; i < n_; ++i)
            for (int k = 0; k < 3; ++k) {
                lo[k] = std::min(lo[k], host_.pos[3 * i + k]);
                hi[k] = std::max(hi[k], host_.pos[3 * i + k]);
            }
        for (int k = 0; k < 3; ++k) origin_[k] = 0.5 * (lo[k] + hi[k]);
        CK(dalloc(&d_pos32_, n_));
        CK(dalloc(&d_wall32_, n_));
        CK(dalloc(&d_touched_, n_));
        CK(cudaMemset(d_touched_, 0, n_));
        CK(cudaMemset(d_wall32_, 0, sizeof(float4) * n_));
        std::vector<float> reach((size_t)nm_ * nm_, 0.0f);
        for (size_t q = 0; q < reach.size(); ++q) {
            const double* gq = &tab_.geom[4 * q];   // ra, b0, b1, b2
            double r = 0.0;
            if (tab_.params[q].cd == CD_SS) r = gq[0] + gq[1];
            else if (cd_plane(tab_.params[q].cd) == CD_SP) r = gq[0] + 0.5 * gq[2];
            else if (tab_.params[q].cd == CD_SC) r = gq[0] + gq[1];
            // inside a hollow cylinder: -(R - r), its magnitude rounded down (prefilter.cuh)
            if (tab_.params[q].cd == CD_SIC) reach[q] = (float)(gq[0] - gq[1]) * (1.0f - 1e-6f);
            else reach[q] = (float)r * (1.0f + 1e-6f);
        }
        // what k_pair's prefilter reads of a pair's models: reach and detector, no detector (the pair is
        // always evaluated) where the law may bond
        std::vector<float2> brief(reach.size());
        for (size_t q = 0; q < reach.size(); ++q) {
            const PairParam& P = tab_.params[q];
            const bool bondable = (P.is == IS_BSDBF || P.is == IS_BTSDBF || P.is == IS_BSDB2F) && P.c[4] != 0.0;
            const int cd = bondable ? 0 : P.cd;
            float w;
            memcpy(&w, &cd, 4);
            brief[q] = make_float2(reach[q], w);
        }
        CK(dalloc(&d_brief_, brief.size()));
        CK(cudaMemcpy(d_brief_, brief.data(), sizeof(float2) * brief.size(), cudaMemcpyHostToDevice));
        CK(dalloc(&d_reach_, reach.size()));
        CK(cudaMemcpy(d_reach_, reach.data(), sizeof(float) * reach.size(), cudaMemcpyHostToDevice));
        k_refresh32<<<blocks_for(n_), TPB>>>(n_, d_model_of_, d_models_, d_pos_, d_ox_, d_oz_,
                                             mk(origin_[0], origin_[1], origin_[2]), d_pos32_, d_wall32_);
        CK(cudaGetLastError());
        CK(cudaDeviceSynchronize());
    }
    CK(dalloc(&d_global_, global_ids_.size()));
    if (!global_ids_.empty())
        CK(cudaMemcpy(d_global_, global_ids_.data(), sizeof(uint32_t) * global_ids_.size(), cudaMemcpyHostToDevice));
    // broad-phase scratch
    CK(dalloc(&d_safe_, n_)); CK(dalloc(&d_red_, 8)); CK(dalloc(&d_key_, n_)); CK(dalloc(&d_key_alt_, n_));
    CK(dalloc(&d_cell_key_, n_)); CK(dalloc(&d_sid_, n_)); CK(dalloc(&d_sid_alt_, n_));
    CK(dalloc(&d_bp_, n_));
    CK(dalloc(&d_cell_start_, (size_t)n_ + 1)); CK(dalloc(&d_cellof_, n_)); CK(dalloc(&d_flag_, n_));
    CK(dalloc(&d_total_, 4));
    CK(dalloc(&d_obs_, (size_t)(blocks_for(n_) + 2) * 16 + 64));
    // IDO records, sorted by key, first of equal keys kept (std::map::insert)
    const HRecords& R = host_.rec;
    if (R.size()) {
        std::vector<uint32_t> ord(R.size());
        for (uint32_t q = 0; q < ord.size(); ++q) ord[q] = q;
        auto key = [&](uint32_t q) { return ((uint64_t)R.first[q] << 32) | R.second[q]; };
        std::stable_sort(ord.begin(), ord.end(), [&](uint32_t a, uint32_t b) { return key(a) < key(b); });
        std::vector<uint64_t> rk;
        std::vector<double4_32a> rh;
        std::vector<double> rv;
        std::vector<uint8_t> rf;
        for (uint32_t q : ord) {
            if (!rk.empty() && rk.back() == key(q)) continue;
            rk.push_back(key(q));
            rh.push_back(make_double4_32a(R.shear[3 * q], R.shear[3 * q + 1], R.shear[3 * q + 2], R.kn[q]));
            rv.push_back(R.v0[q]);
            // default-constructed ImpactStatus + setters (IactRecordTab.cpp:432-530)
            rf.push_back((uint8_t)(ST_DEFAULT | (R.contact[q] ? ST_CONTACT : 0) | (R.bond[q] ? ST_BOND : 0) | PF_NONZERO));
        }
        rc = upload_records(rk, rh, rv, rf);
        if (rc != VEDO_OK) return rc;
    }
    // first candidate list (NBSConsultant constructor) + Initiate
    rc = rebuild(true);
    if (rc != VEDO_OK) return rc;
    CK(cudaStreamSynchronize(stream_));
    backup_pending_ = false;
    if (!out_prefix_.empty()) {
        // SimMediator's constructor (SimMediator.cpp:103-123): the SystemStatus.csv header, then
        // CalculateSystemEnergy with the IactRecordTab read from the file
        std::string dir = out_prefix_;
        const size_t slash = dir.find_last_of('/');
        dir = slash == std::string::npos ? std::string() : dir.substr(0, slash + 1);
        status_ = std::fopen((dir + "SystemStatus.csv").c_str(), "w");
        if (!status_) return fail(VEDO_ERR_IO, "cannot write " + dir + "SystemStatus.csv");
        std::fprintf(status_, "Simulated time, number of elements, number of interactions, Number of contacts, "
                              "System energy, Potential energy, Kinetic energy, Kinetic energy (translation), "
                              "Kinetic energy (rotation), Minimal velocity, Maximal velocity, "
                              "Minimal angular velocity, Maximal angular velocity, Norm of momentum, "
                              "Norm of angular momentum");
        for (uint32_t u = 0; u < 2 * host_.num_udd_impact; ++u) std::fprintf(status_, ", User-defined Value %u", u + 1);
        std::fprintf(status_, "\n");
        uint64_t contacts = 0;
        for (size_t q = 0; q < host_.rec.first.size(); ++q) contacts += host_.rec.contact[q] ? 1u : 0u;
        rc = status_row(host_.rec.first.size(), contacts);
        if (rc != VEDO_OK) return rc;
    }
    return VEDO_OK;
}

// The records the next list takes its history from (sorted by key).
int Engine::upload_records(const std::vector<uint64_t>& rk, const std::vector<double4_32a>& rh,
                           const std::vector<double>& rv, const std::vector<uint8_t>& rf) {
    for (void** p : {(void**)&d_rec_key_, (void**)&d_rec_hist_, (void**)&d_rec_v0_, (void**)&d_rec_flags_}) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
    nrec_ = (uint32_t)rk.size();
    if (!nrec_) return VEDO_OK;
    CK(dalloc(&d_rec_key_, nrec_)); CK(dalloc(&d_rec_hist_, nrec_)); CK(dalloc(&d_rec_v0_, nrec_));
    CK(dalloc(&d_rec_flags_, nrec_));
    CK(cudaMemcpy(d_rec_key_, rk.data(), 8 * nrec_, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(d_rec_hist_, rh.data(), sizeof(double4_32a) * nrec_, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(d_rec_v0_, rv.data(), 8 * nrec_, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(d_rec_flags_, rf.data(), nrec_, cudaMemcpyHostToDevice));
    return VEDO_OK;
}

// LeapConsultant::NextStep at a reset (LeapConsultant.cpp:61-68): SyncWorld,
// RebuildIactRecordTab, then Consultant::CleanUp (Consultant.cpp:264-319).  The mobile objects
// outside the zone of interest are erased and the others renumbered (their order kept); the
// records of the interactions active at the current positions -- their statuses as the carry of
// an ordinary reset takes them -- are re-keyed as IactRecordTab::ModifyPair does, and become the
// records the reset's list takes its history from.  Host work, run only when an object leaves.
int Engine::leap_cleanup(bool* erased_any) {
    *erased_any = false;
    int rc = sync_host_state();
    if (rc != VEDO_OK) return rc;
    std::vector<uint32_t> jump;
    const std::vector<uint32_t> erased = zoi_outside(host_, jump);
    if (erased.empty()) return VEDO_OK;
    const uint32_t np = cur_.np;
    std::vector<uint32_t> fa(np), fb(np);
    std::vector<uint8_t> fl(np);
    std::vector<double4_32a> hh(np);
    std::vector<double> vv(np);
    if (np) {
        k_detect_active<<<blocks_for(np), TPB, 0, stream_>>>(np, cur_.sm, cur_.param, d_params_, d_geom_, d_hole_,
                                                             d_reach_, d_pos_, d_ox_, d_oz_, d_pos32_, d_wall32_,
                                                             cur_.flags, tab_.pbc);
        ++launches_;
        CK(cudaMemcpyAsync(fa.data(), cur_.first, 4 * (size_t)np, cudaMemcpyDeviceToHost, stream_));
        CK(cudaMemcpyAsync(fb.data(), cur_.second, 4 * (size_t)np, cudaMemcpyDeviceToHost, stream_));
        CK(cudaMemcpyAsync(fl.data(), cur_.flags, np, cudaMemcpyDeviceToHost, stream_));
        CK(cudaMemcpyAsync(hh.data(), cur_.hist, sizeof(double4_32a) * np, cudaMemcpyDeviceToHost, stream_));
        CK(cudaMemcpyAsync(vv.data(), cur_.v0, 8 * (size_t)np, cudaMemcpyDeviceToHost, stream_));
        CK(cudaStreamSynchronize(stream_));
    }
    std::vector<std::pair<uint32_t, uint32_t>> keys;
    std::vector<uint32_t> src;
    for (uint32_t k = 0; k < np; ++k)
        if (fl[k] & PF_ACTIVE) {
            keys.push_back({fa[k], fb[k]});
            src.push_back(k);
        }
    std::vector<uint64_t> rk;
    std::vector<double4_32a> rh;
    std::vector<double> rv;
    std::vector<uint8_t> rf;
    for (const auto& kv : modify_pair(keys, jump)) {
        const uint32_t k = src[kv.second];
        const bool nz = fl[k] & PF_NONZERO;
        rk.push_back(((uint64_t)kv.first.first << 32) | kv.first.second);
        rh.push_back(nz ? hh[k] : make_double4_32a(0.0, 0.0, 0.0, 0.0));
        rv.push_back(nz ? vv[k] : 0.0);
        rf.push_back((uint8_t)(fl[k] & (PF_STATUS | PF_NONZERO)));
    }
    erase_objects(host_, erased);
    n_ = host_.n;
    // the survivors' state and models (the buffers keep their larger capacity)
    std::vector<double4_32a> tmp;
    double4_32a* dst[] = {d_pos_, d_vel_, d_av_, d_ox_, d_oz_, d_imp_, d_aimp_};
    const std::vector<double>* srcv[] = {&host_.pos, &host_.vel, &host_.av, &host_.ox, &host_.oz, &host_.imp,
                                         &host_.aimp};
    for (int k = 0; k < 7; ++k) {
        upload3(tmp, *srcv[k], n_);
        CK(cudaMemcpy(dst[k], tmp.data(), sizeof(double4_32a) * n_, cudaMemcpyHostToDevice));
    }
    CK(cudaMemcpy(d_model_of_, host_.model_of.data(), sizeof(uint32_t) * n_, cudaMemcpyHostToDevice));
    global_ids_.clear();
    leap_rmax_ = 0.0;                      // LeapConsultant::Reset takes the largest range anew
    for (uint32_t i = 0; i < n_; ++i)
        if (tab_.models[host_.model_of[i]].scope != SCOPE_LOCAL) global_ids_.push_back(i);
        else leap_rmax_ = std::max(leap_rmax_, tab_.models[host_.model_of[i]].range);
    if (global_ids_.size() == n_) return fail(VEDO_ERR_INVALID_SCENE, "the zone of interest erased every local object");
    if (!global_ids_.empty())
        CK(cudaMemcpy(d_global_, global_ids_.data(), sizeof(uint32_t) * global_ids_.size(), cudaMemcpyHostToDevice));
    k_refresh32<<<blocks_for(n_), TPB, 0, stream_>>>(n_, d_model_of_, d_models_, d_pos_, d_ox_, d_oz_,
                                                     mk(origin_[0], origin_[1], origin_[2]), d_pos32_, d_wall32_);
    ++launches_;
    CK(cudaMemsetAsync(d_touched_, 0, n_, stream_));
    CK(cudaStreamSynchronize(stream_));
    rc = upload_records(rk, rh, rv, rf);
    if (rc != VEDO_OK) return rc;
    *erased_any = true;
    return VEDO_OK;
}

// One line of SystemStatus.csv (SimMediator::CalculateSystemEnergy, SimMediator.cpp:46-81):
// time, object count, IactRecordTab size and contact count, then the energies and extrema of
// DOWorld::CalculateSystemEnergy, as the reference's ostream writes them (6 significant
// digits).  The user-defined impact values, which the engine does not carry, are written as 0.
int Engine::status_row(uint64_t records, uint64_t contacts) {
    double o[13];
    const int rc = get_observables(o);
    if (rc != VEDO_OK) return rc;
    std::fprintf(status_, "%g, %u, %llu, %llu, %g, %g, %g, %g, %g, %g, %g, %g, %g, %g, %g", t_, n_,
                 (unsigned long long)records, (unsigned long long)contacts, o[0] + o[1] + o[2], o[0], o[1] + o[2],
                 o[1], o[2], o[3], o[4], o[5], o[6], o[7], o[8]);
    for (uint32_t u = 0; u < 2 * host_.num_udd_impact; ++u) std::fprintf(status_, ", 0");
    std::fprintf(status_, "\n");
    std::fflush(status_);
    return VEDO_OK;
}

// The line SimMediator::Run writes at a reset or record step: the record table rebuilt from the
// interactions that are active at the new positions (NBSConsultant::RebuildIactRecordTab,
// NBSConsultant.cpp:376-389), and among them those whose status holds a contact.
int Engine::status_row_now() {
    uint64_t active = 0, contacts = 0;
    if (cur_.np) {
        k_detect_active<<<blocks_for(cur_.np), TPB, 0, stream_>>>(cur_.np, cur_.sm, cur_.param, d_params_, d_geom_,
                                                                  d_hole_, d_reach_, d_pos_, d_ox_, d_oz_, d_pos32_,
                                                                  d_wall32_, cur_.flags, tab_.pbc);
        std::vector<uint8_t> f(cur_.np);
        CK(cudaMemcpyAsync(f.data(), cur_.flags, cur_.np, cudaMemcpyDeviceToHost, stream_));
        CK(cudaStreamSynchronize(stream_));
        for (uint8_t b : f)
            if (b & PF_ACTIVE) {
                ++active;
                contacts += (b & ST_CONTACT) ? 1u : 0u;
            }
    }
    return status_row(active, contacts);
}

int Engine::rebuild(bool from_records) {
    const uint64_t l0 = g_sort_scan_launches;
    uint64_t own = 0;
    std::swap(cur_, old_);
    // 1. safe lengths and bounds (:120-146)
    const double dtu = (double)opts_.up_iact * dt_;
    const double glen = len(mk(g_[0], g_[1], g_[2]));
    unsigned long long red0[8] = {ord_of(DBL_MAX), ord_of(DBL_MIN), ord_of(DBL_MAX), ord_of(DBL_MIN),
                                  ord_of(DBL_MAX), ord_of(DBL_MIN), ord_of(0.0), 0ull};
    CK(cudaMemcpyAsync(d_red_, red0, sizeof(red0), cudaMemcpyHostToDevice, stream_));
    k_safe<<<std::min(blocks_for(n_), 608u), TPB, 0, stream_>>>(n_, d_model_of_, d_models_, d_pos_, d_vel_, sf_, dtu, glen, d_safe_,
                                                d_red_);
    ++own;
    unsigned long long red[8];
    CK(cudaMemcpyAsync(red, d_red_, sizeof(red), cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    const double xmin = dbl_of(red[0]), xmax = dbl_of(red[1]), ymin = dbl_of(red[2]), ymax = dbl_of(red[3]);
    const double zmin = dbl_of(red[4]), zmax = dbl_of(red[5]), vmax = dbl_of(red[6]);
    const uint32_t nloc = n_ - (uint32_t)global_ids_.size();
    double rmax = 0.0;
    CellGrid g{};
    g.mode = 0;
    if (leap_) {
        // LeapConsultant::Reset (LeapConsultant.cpp:108-195): the largest range of the local
        // objects, and the comparator from the spans between the 2 % and 98 % quantiles of the
        // local positions per axis (sorted on the device)
        rmax = leap_rmax_;
        const double keep = 1.0 - 0.02, hi_d = keep * nloc - 1, lo_d = 0.02 * nloc;
        const uint32_t ih = hi_d < 0.0 ? 0u : (uint32_t)hi_d, il = (uint32_t)lo_d;
        double span[3];
        for (int a = 0; a < 3; ++a) {
            k_axis_key<<<blocks_for(n_), TPB, 0, stream_>>>(n_, d_model_of_, d_models_, d_pos_, a, d_key_, d_sid_);
            ++own;
            CK(radix_sort_u64(d_key_, d_sid_, d_key_alt_, d_sid_alt_, n_, 0, 64, scratch_, stream_));
            unsigned long long q[2];
            CK(cudaMemcpyAsync(&q[0], d_key_ + ih, 8, cudaMemcpyDeviceToHost, stream_));
            CK(cudaMemcpyAsync(&q[1], d_key_ + il, 8, cudaMemcpyDeviceToHost, stream_));
            CK(cudaStreamSynchronize(stream_));
            span[a] = dbl_of(q[0]) - dbl_of(q[1]);
        }
        g.mode = span[0] >= span[1] ? (span[0] >= span[2] ? 0 : 2) : (span[1] >= span[2] ? 1 : 2);
    } else if (red[7]) {
        rmax = tab_.models[host_.model_of[red[7] - 1]].range;              // the last local DO (:140)
    }
    const double zone = sf_ * (2.0 * rmax + dtu * vmax + 0.5 * dtu * dtu * glen);   // :146, Leap :138
    auto ncel = [&](double lo, double hi) {
        uint32_t c = (uint32_t)std::ceil((hi - lo) / zone);
        return std::max(c, (uint32_t)1);
    };
    const uint32_t ncx = ncel(xmin, xmax), ncy = ncel(ymin, ymax), ncz = ncel(zmin, zmax);
    g.ncel[0] = ncx; g.ncel[1] = ncy; g.ncel[2] = ncz;
    g.leap = leap_ ? 1 : 0;
    // key extents: zone ids reach ncel (a span that is a whole number of zones); Leap visits every
    // zone, so its neighbours reach ncel + 1
    const uint64_t pad = leap_ ? 2 : 1;
    g.dim[0] = (uint64_t)ncx + pad; g.dim[1] = (uint64_t)ncy + pad; g.dim[2] = (uint64_t)ncz + pad;
    if (leap_) {
        const double lo3[3] = {xmin, ymin, zmin}, hi3[3] = {xmax, ymax, zmax};
        for (int a = 0; a < 3; ++a) {                                      // LeapConsultant.h:146-150
            g.pbc[a] = tab_.pbc.sw[a] && (hi3[a] - lo3[a]) >= 0.5 * tab_.pbc.range[a];
            g.has_pbc |= g.pbc[a];
        }
    }
    const uint64_t sentinel = g.dim[0] * g.dim[1] * g.dim[2];
    int bits = 1;
    while (bits < 64 && (sentinel >> bits)) ++bits;
    // 2. cell keys, stable sort (locals by cell in the comparator's order, ids ascending within a cell)
    const bool kalt = radix_passes_of(0, bits) & 1;
    k_cellkey<<<blocks_for(n_), TPB, 0, stream_>>>(n_, d_model_of_, d_models_, d_pos_, xmin, ymin, zmin, zone, g,
                                                   sentinel, kalt ? d_key_alt_ : d_key_, kalt ? d_sid_alt_ : d_sid_);
    ++own;
    CK(radix_sort_u64(d_key_, d_sid_, d_key_alt_, d_sid_alt_, n_, 0, bits, scratch_, stream_, kalt));
    // 3. cell ranges
    uint32_t np = 0;
    int herr = 0;
    if (nloc) {
        // dense cell map when the grid is small compared with the object count
        uint32_t* grid = nullptr;
        const uint64_t gcells = sentinel;
        if (gcells <= std::max<uint64_t>(8ull * n_, 1ull << 22) && gcells < (1ull << 31)) {
            if (gcells > grid_cap_) {
                if (d_grid_) cudaFree(d_grid_);
                d_grid_ = nullptr;
                grid_cap_ = gcells + gcells / 4;
                CK(dalloc(&d_grid_, grid_cap_));
            }
            CK(cudaMemsetAsync(d_grid_, 0xff, sizeof(uint32_t) * gcells, stream_));
            grid = d_grid_;
        }
        k_cell_flags<<<blocks_for(nloc), TPB, 0, stream_>>>(nloc, d_key_, d_flag_);
        CK(exclusive_scan_u32(d_flag_, d_flag_, nloc, d_total_, scratch_, stream_));
        k_cell_fill<<<blocks_for(nloc), TPB, 0, stream_>>>(nloc, d_key_, d_flag_, d_cell_key_, d_cell_start_,
                                                           d_cellof_, d_total_, grid, d_sid_, d_model_of_, d_models_, d_pos32_,
                                                           d_safe_, d_bp_);
        own += 2;
        // 4. count pass over (object, slot) tasks, scan, fill pass
        const uint64_t ntask = (uint64_t)nloc * NSLOT;
        if (ntask + 1 > task_cap_) {
            if (d_task_) cudaFree(d_task_);
            if (d_picked_) cudaFree(d_picked_);
            d_task_ = d_picked_ = nullptr;
            task_cap_ = (uint32_t)(ntask + 1);
            CK(dalloc(&d_task_, task_cap_));
            CK(dalloc(&d_picked_, task_cap_));
        }
        int* err = reinterpret_cast<int*>(d_total_ + 2);
        CK(cudaMemsetAsync(err, 0, sizeof(int), stream_));
        k_pairs<false><<<blocks_for(ntask), TPB, 0, stream_>>>(
            nloc, d_sid_, d_cell_key_, d_cell_start_, d_total_, d_cellof_, grid, gcells, d_global_,
            (uint32_t)global_ids_.size(), d_model_of_, d_models_, d_group_iact_, tab_.ngroups, d_pos_, d_ox_, d_oz_,
            d_pos32_, d_wall32_, d_safe_, d_bp_, g, tab_.pbc, nm_, all_interact_, d_refused_, d_task_, d_picked_, nullptr, nullptr, err);
        ++own;
        CK(exclusive_scan_u32(d_task_, d_task_, (uint32_t)ntask, d_total_ + 1, scratch_, stream_));
        uint32_t got[2];
        CK(cudaMemcpyAsync(got, d_total_ + 1, sizeof(got), cudaMemcpyDeviceToHost, stream_));
        CK(cudaStreamSynchronize(stream_));
        np = got[0];
        herr = (int)got[1];
        int rc = ensure_list(cur_, np);
        if (rc != VEDO_OK) return rc;
        k_pairs<true><<<blocks_for(ntask), TPB, 0, stream_>>>(
            nloc, d_sid_, d_cell_key_, d_cell_start_, d_total_, d_cellof_, grid, gcells, d_global_,
            (uint32_t)global_ids_.size(), d_model_of_, d_models_, d_group_iact_, tab_.ngroups, d_pos_, d_ox_, d_oz_,
            d_pos32_, d_wall32_, d_safe_, d_bp_, g, tab_.pbc, nm_, all_interact_, d_refused_, d_task_, d_picked_, cur_.first, cur_.second, err);
        ++own;
    } else {
        int rc = ensure_list(cur_, 0);
        if (rc != VEDO_OK) return rc;
    }
    cur_.np = np;
    // 5. interactions: orientation, model, history; 6. per-object contact entries in ascending pair
    // index (stable radix sort by object)
    const uint32_t m = 2 * np;
    if (m > csr_cap_) {
        for (uint32_t** p : {&d_ck_, &d_ck_alt_, &d_cv_alt_}) {
            if (*p) cudaFree(*p);
            *p = nullptr;
        }
        csr_cap_ = std::max<uint32_t>(m + m / 4, 2048);
        CK(dalloc(&d_ck_, csr_cap_)); CK(dalloc(&d_ck_alt_, csr_cap_)); CK(dalloc(&d_cv_alt_, csr_cap_));
    }
    if (np) {
        int obits = 1;
        while (obits < 32 && ((n_ - 1) >> obits)) ++obits;
        const bool calt = radix_passes_of(0, obits) & 1;
        const HistorySource src = from_records ? HistorySource{d_rec_key_, nrec_, d_rec_hist_, d_rec_v0_, d_rec_flags_,
                                                               nullptr, nullptr, nullptr, nullptr}
                                               : HistorySource{nullptr, 0, old_.hist, old_.v0, old_.flags, old_.csr_ptr,
                                                               old_.csr_ent, old_.first, old_.second};
        auto k = from_records ? k_setup<true> : k_setup<false>;
        const uint32_t per = np >= SETUP_MAX * TPB * 304u ? SETUP_MAX : 1u;    // a block for every SM first
        k<<<blocks_for(np, (int)(per * TPB)), TPB, 0, stream_>>>(np, per, cur_.first, cur_.second, d_model_of_, d_models_, d_params_, nm_,
                                               d_refused_, d_geom_, d_hole_, d_reach_, d_pos_, d_ox_, d_oz_, d_pos32_,
                                               d_wall32_, tab_.pbc, src, cur_.sm, cur_.param, calt ? d_ck_alt_ : d_ck_,
                                               calt ? d_cv_alt_ : cur_.csr_ent, cur_.hist, cur_.v0, cur_.flags);
        ++own;
        CK(radix_sort_u32(d_ck_, cur_.csr_ent, d_ck_alt_, d_cv_alt_, m, 0, obits, scratch_, stream_, calt));
    }
    if (m >= n_ && m <= (1u << 20)) k_csr_ptr<true><<<blocks_for((uint64_t)m + 1), TPB, 0, stream_>>>(n_, d_ck_, m, cur_.csr_ptr);
    else k_csr_ptr<false><<<blocks_for((uint64_t)n_ + 1), TPB, 0, stream_>>>(n_, d_ck_, m, cur_.csr_ptr);
    ++own;
    CK(cudaGetLastError());
    launches_ += own + (g_sort_scan_launches - l0);
    if (herr & ERR_BAD_SHAPE_PAIR)
        return fail(VEDO_ERR_UNSUPPORTED_MODEL, "broad phase met a shape pair DOMap::CalDistance does not handle");
    if (herr & ERR_UNSUPPORTED_PAIR)
        return fail(VEDO_ERR_UNSUPPORTED_MODEL,
                    "a candidate pair has no detector/solver (the reference would drop it and misalign its "
                    "interaction records)");
    backup_pending_ = false;
    return VEDO_OK;
}

int Engine::step_once(bool write_impulses) {
    const double dt = dt_;
    const bool prof = profiling_;
    // CalculateImpact
    if (prof) CK(cudaEventRecord(ev_[0], stream_));
    if (cur_.np) {
        if (!pair_grid_) {                         // the blocks resident at once
            int blocks = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_pair, TPB, 0) != cudaSuccess || blocks < 1) blocks = 1;
            int sms = 1;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, opts_.device);
            pair_grid_ = (unsigned)(blocks * std::max(sms, 1));
        }
        k_pair<<<std::min(pair_grid_, blocks_for(cur_.np, PAIR_TILE * TPB)), TPB, 0, stream_>>>(
            cur_.np, cur_.sm, cur_.param, d_params_, d_geom_, d_hole_, d_brief_, d_pos_, d_vel_, d_av_, d_ox_, d_oz_,
            d_pos32_, d_wall32_, cur_.hist, cur_.v0, cur_.flags, cur_.out, dt, backup_pending_ ? 1 : 0, tab_.pbc,
            d_touched_);
        ++launches_;
    }
    if (prof) CK(cudaEventRecord(ev_[1], stream_));
    // AddFieldImpact + AddConstrainedImpact + Response (+ CheckContactStatus in the next k_pair)
    const d3 fimp = muls(mk(g_[0], g_[1], g_[2]), dt);    // csp->GetFieldAcceleration() * dt (SimMediator.cpp:738)
    const d3 org = mk(origin_[0], origin_[1], origin_[2]);
    ObjArgs oa;
    oa.n = n_;
    oa.model_of = d_model_of_;
    oa.models = d_models_;
    oa.pos = d_pos_; oa.vel = d_vel_; oa.av = d_av_; oa.ox = d_ox_; oa.oz = d_oz_; oa.imp = d_imp_; oa.aimp = d_aimp_;
    oa.csr_ptr = cur_.csr_ptr;
    oa.csr_ent = cur_.csr_ent;
    oa.flags = cur_.flags;
    oa.out = cur_.out;
    oa.dt = dt;
    oa.fimp = fimp;
    oa.write_imp = write_impulses ? 1 : 0;
    oa.origin = org;
    oa.pos32 = d_pos32_;
    oa.wall32 = d_wall32_;
    oa.ext_imp = ext_imp_;
    oa.ext_aimp = ext_aimp_;
    oa.pb = tab_.pbc;
    oa.touched = d_touched_;
    oa.nglob = (uint32_t)global_ids_.size();
    oa.glob = d_global_;
    oa.per = std::min<uint32_t>(TPB, std::max(32u, (n_ / 608u + 31u) / 32u * 32u));   // four blocks an SM
    k_obj<<<oa.nglob + blocks_for(n_, (int)oa.per), TPB, 0, stream_>>>(oa);
    ++launches_;
    if (prof) CK(cudaEventRecord(ev_[2], stream_));
    backup_pending_ = true;
    // NBSConsultant::NextStep (NBSConsultant.cpp:35-78)
    ++round_;
    t_ += dt;                                              // SystemParameter::NextStep (SystemParameter.h:113-116)
    if (round_ % opts_.up_iact == 0) {
        if (prof) CK(cudaEventRecord(ev_[3], stream_));
        bool erased = false;
        if (leap_ && zoi_on_) {                            // LeapConsultant.cpp:61-68
            int rc = leap_cleanup(&erased);
            if (rc != VEDO_OK) return rc;
        }
        int rc = rebuild(erased);                          // after an erasure, from the re-keyed records
        if (rc != VEDO_OK) return rc;
        if (prof) {
            CK(cudaEventRecord(ev_[4], stream_));
            CK(cudaEventSynchronize(ev_[4]));
            float ms = 0;
            cudaEventElapsedTime(&ms, ev_[3], ev_[4]);
            prof_ms_[2] += ms;
        }
    }
    if (prof) {
        float a = 0, b = 0;
        CK(cudaEventSynchronize(ev_[2]));
        cudaEventElapsedTime(&a, ev_[0], ev_[1]);
        cudaEventElapsedTime(&b, ev_[1], ev_[2]);
        prof_ms_[0] += a;
        prof_ms_[1] += b;
    }
    if (opts_.record && round_ % opts_.record == 0 && !out_prefix_.empty()) {
        int rc = record_ido();
        if (rc != VEDO_OK) return rc;
    }
    if (status_ && (round_ % opts_.up_iact == 0 || (opts_.record && round_ % opts_.record == 0))) {
        int rc = status_row_now();                         // SimMediator.cpp:784-792
        if (rc != VEDO_OK) return rc;
    }
    if (t_ >= t_stop_ && !out_prefix_.empty()) {         // NBSConsultant.cpp:65-76
        std::string dir = out_prefix_;
        size_t slash = dir.find_last_of('/');
        dir = slash == std::string::npos ? std::string() : dir.substr(0, slash + 1);
        int rc = write_ido((dir + "terminate.ido").c_str());
        if (rc != VEDO_OK) return rc;
    }
    return VEDO_OK;
}

int Engine::run(uint32_t nsteps, int* keep_running) {
    prof_ms_[0] = prof_ms_[1] = prof_ms_[2] = prof_ms_[3] = 0;
    launches_ = 0;
    CK(cudaSetDevice(device_));
    CK(cudaEventRecord(ev_[5], stream_));
    for (uint32_t s = 0; s < nsteps; ++s) {
        int rc = step_once(s + 1 == nsteps);
        if (rc != VEDO_OK) return rc;
    }
    CK(cudaEventRecord(ev_[6], stream_));
    CK(cudaStreamSynchronize(stream_));
    CK(cudaGetLastError());
    float tot = 0;
    cudaEventElapsedTime(&tot, ev_[5], ev_[6]);
    prof_ms_[3] = tot;
    if (keep_running) *keep_running = t_ < t_stop_ ? 1 : 0;   // SimMediator.cpp:839-841
    return VEDO_OK;
}

// One step with per-object external impulses (SimMediator::Run(external impacts),
// SimMediator.cpp:987-1119): host [n][3] arrays, NULL adds zeros as the reference adds them.
int Engine::run_with_impulses(const double* impulse, const double* angular_impulse, int* keep_running) {
    CK(cudaSetDevice(device_));
    if (!d_ext_) CK(cudaMalloc(&d_ext_, 2 * 24 * (size_t)n_));
    const double* src[2] = {impulse, angular_impulse};
    for (int k = 0; k < 2; ++k) {
        double* dst = d_ext_ + (size_t)k * 3 * n_;
        if (src[k]) CK(cudaMemcpyAsync(dst, src[k], 24 * (size_t)n_, cudaMemcpyHostToDevice, stream_));
        else CK(cudaMemsetAsync(dst, 0, 24 * (size_t)n_, stream_));
    }
    ext_imp_ = d_ext_;
    ext_aimp_ = d_ext_ + 3 * (size_t)n_;
    const int rc = run(1, keep_running);
    ext_imp_ = ext_aimp_ = nullptr;
    return rc;
}

uint64_t Engine::last_profile(double out[4]) const {
    for (int k = 0; k < 4; ++k) out[k] = prof_ms_[k];
    return launches_;
}

// ------------------------------------------------------------------------------------
// state I/O: host [n][3] arrays <-> device double4 (x, y, z, pad); the repacking runs on the
// device, the host side is one contiguous copy per array.
namespace {
__global__ void k_pack3(uint32_t n, const double* __restrict__ src, double4_32a* __restrict__ dst) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = make_double4_32a(src[3 * (size_t)i], src[3 * (size_t)i + 1], src[3 * (size_t)i + 2], 0.0);
}
// Every array asked for in one launch (blockIdx.y), as a call of a few dozen objects is made of its
// launches.  The table stays in the parameters' constant bank: without __grid_constant__ its indexing
// by blockIdx.y made every thread copy it to its stack, 112 B (a read of the positions of 200,000
// spheres: 64 us, 56 like this).
struct Fields {
    const double4_32a* src[7];
    double* dst[7];
};
__global__ void k_unpack3(uint32_t n, const __grid_constant__ Fields f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const double4_32a v = f.src[blockIdx.y][i];
        double* dst = f.dst[blockIdx.y];
        dst[3 * (size_t)i] = v.x;
        dst[3 * (size_t)i + 1] = v.y;
        dst[3 * (size_t)i + 2] = v.z;
    }
}
}  // namespace

int Engine::ensure_stage() {
    if (d_stage_) return VEDO_OK;
    CK(dalloc(&d_stage_, 7 * 3 * (size_t)n_));
    return VEDO_OK;
}

int Engine::get_state(const vedo_state_view& v) {
    int rc = ensure_stage();
    if (rc != VEDO_OK) return rc;
    double* dst[] = {v.position, v.velocity, v.angular_velocity, v.orientation_x, v.orientation_z, v.impact,
                     v.angular_impact};
    const double4_32a* src[] = {d_pos_, d_vel_, d_av_, d_ox_, d_oz_, d_imp_, d_aimp_};
    Fields f{};
    int nf = 0;
    for (int k = 0; k < 7; ++k) {
        if (!dst[k]) continue;
        f.src[nf] = src[k];
        f.dst[nf++] = d_stage_ + (size_t)k * 3 * n_;
    }
    if (nf) k_unpack3<<<dim3(blocks_for(n_), (unsigned)nf), TPB, 0, stream_>>>(n_, f);
    for (int k = 0; k < 7; ++k)
        if (dst[k])
            CK(cudaMemcpyAsync(dst[k], d_stage_ + (size_t)k * 3 * n_, 24 * (size_t)n_, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    CK(cudaGetLastError());
    return VEDO_OK;
}

int Engine::set_state(const vedo_state_view& v) {
    int rc = ensure_stage();
    if (rc != VEDO_OK) return rc;
    const double* srcs[] = {v.position, v.velocity, v.angular_velocity, v.orientation_x, v.orientation_z, v.impact,
                            v.angular_impact};
    double4_32a* dst[] = {d_pos_, d_vel_, d_av_, d_ox_, d_oz_, d_imp_, d_aimp_};
    for (int k = 0; k < 7; ++k) {
        if (!srcs[k]) continue;
        double* st = d_stage_ + (size_t)k * 3 * n_;
        CK(cudaMemcpyAsync(st, srcs[k], 24 * (size_t)n_, cudaMemcpyHostToDevice, stream_));
        k_pack3<<<blocks_for(n_), TPB, 0, stream_>>>(n_, st, dst[k]);
    }
    k_refresh32<<<blocks_for(n_), TPB, 0, stream_>>>(n_, d_model_of_, d_models_, d_pos_, d_ox_, d_oz_,
                                                     mk(origin_[0], origin_[1], origin_[2]), d_pos32_, d_wall32_);
    CK(cudaStreamSynchronize(stream_));
    CK(cudaGetLastError());
    return VEDO_OK;
}

int Engine::num_interactions(uint32_t* n) {
    *n = cur_.np;
    return VEDO_OK;
}

int Engine::get_interactions(const vedo_contact_view& v) {
    const uint32_t np = cur_.np;
    if (!np) return VEDO_OK;
    // ContactInfo::bActive of the last narrow phase = detection at the current positions
    k_detect_active<<<blocks_for(np), TPB, 0, stream_>>>(np, cur_.sm, cur_.param, d_params_, d_geom_, d_hole_, d_reach_,
                                                         d_pos_, d_ox_, d_oz_, d_pos32_, d_wall32_, cur_.flags, tab_.pbc);
    std::vector<uint2> sm(np);
    std::vector<uint8_t> fl(np);
    std::vector<double4_32a> h(np);
    if (v.first) CK(cudaMemcpyAsync(v.first, cur_.first, 4 * np, cudaMemcpyDeviceToHost, stream_));
    if (v.second) CK(cudaMemcpyAsync(v.second, cur_.second, 4 * np, cudaMemcpyDeviceToHost, stream_));
    CK(cudaMemcpyAsync(sm.data(), cur_.sm, sizeof(uint2) * np, cudaMemcpyDeviceToHost, stream_));
    CK(cudaMemcpyAsync(fl.data(), cur_.flags, np, cudaMemcpyDeviceToHost, stream_));
    CK(cudaMemcpyAsync(h.data(), cur_.hist, sizeof(double4_32a) * np, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    for (uint32_t k = 0; k < np; ++k) {
        const bool nz = fl[k] & PF_NONZERO;
        if (v.slave) v.slave[k] = sm[k].x;
        if (v.master) v.master[k] = sm[k].y;
        if (v.active) v.active[k] = (fl[k] & PF_ACTIVE) ? 1 : 0;
        if (v.contact) v.contact[k] = (fl[k] & ST_CONTACT) ? 1 : 0;
        if (v.kn) v.kn[k] = nz ? h[k].w : 0.0;
        if (v.shear) {
            v.shear[3 * k] = nz ? h[k].x : 0.0;
            v.shear[3 * k + 1] = nz ? h[k].y : 0.0;
            v.shear[3 * k + 2] = nz ? h[k].z : 0.0;
        }
    }
    return VEDO_OK;
}

int Engine::get_observables(double out[13]) {
    const unsigned nb = obs::obs_blocks(n_);
    double* part = d_obs_;
    double* res = d_obs_ + (size_t)nb * 16 + 16;
    const d3 g = mk(g_[0], g_[1], g_[2]);
    obs::k_obs_a<<<nb, TPB, 0, stream_>>>(n_, d_model_of_, d_models_, d_pos_, d_vel_, d_av_, g, part);
    obs::k_obs_reduce<<<16, TPB, 0, stream_>>>(nb, 16, part, res, 12);
    if (cur_.np)
        k_detect_active<<<blocks_for(cur_.np), TPB, 0, stream_>>>(cur_.np, cur_.sm, cur_.param, d_params_, d_geom_,
                                                                  d_hole_, d_reach_, d_pos_, d_ox_, d_oz_, d_pos32_,
                                                                  d_wall32_, cur_.flags, tab_.pbc);
    obs::k_obs_b<<<nb, TPB, 0, stream_>>>(n_, d_model_of_, d_models_, d_pos_, d_vel_, d_av_, res, cur_.flags, cur_.np,
                                          part);
    obs::k_obs_reduce<<<6, TPB, 0, stream_>>>(nb, 6, part, res + 16, 6);
    double r[22];
    CK(cudaMemcpyAsync(r, res, sizeof(r), cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    const bool any = r[9] > 0;
    out[0] = r[0]; out[1] = r[1]; out[2] = r[2];
    out[3] = any ? r[12] : 0.0; out[4] = any ? r[13] : 0.0; out[5] = any ? r[14] : 0.0; out[6] = any ? r[15] : 0.0;
    out[7] = r[16]; out[8] = r[17];
    out[9] = r[21];
    const double msum = r[10];
    out[10] = msum > 0 ? r[18] / msum : 0.0;
    out[11] = msum > 0 ? r[19] / msum : 0.0;
    out[12] = msum > 0 ? r[20] / msum : 0.0;
    return VEDO_OK;
}

int Engine::sync_host_state() {
    vedo_state_view v{host_.pos.data(), host_.vel.data(), host_.av.data(), host_.ox.data(), host_.oz.data(),
                      host_.imp.data(), host_.aimp.data()};
    return get_state(v);
}

int Engine::coordination(uint32_t* below, uint32_t* touching, const double* box, double* average) {
    DeviceObjects d;
    d.n = n_; d.model_of = d_model_of_; d.models = d_models_; d.pos = d_pos_;
    d.stream = stream_; d.scratch = &scratch_; d.work = &cn_; d.scene = &host_; d.launches = &launches_;
    std::string m;
    const int rc = coordination_host(d, below, touching, box, average, m);
    return rc == VEDO_OK ? rc : fail(rc, m);
}

int Engine::write_vtk(const char* path, int with_coordination) {
    DeviceObjects d;
    d.n = n_; d.model_of = d_model_of_; d.models = d_models_; d.pos = d_pos_;
    d.stream = stream_; d.scratch = &scratch_; d.work = &cn_; d.scene = &host_; d.launches = &launches_;
    std::string m;
    const int rc = write_vtk_host(this, d, path, with_coordination, m);
    return rc == VEDO_OK ? rc : fail(rc, m);
}

int Engine::write_ido(const char* path) {
    int rc = sync_host_state();
    if (rc != VEDO_OK) return rc;
    host_.time_current = t_;
    // IactRecordTab = the active interactions (NBSConsultant::RebuildIactRecordTab)
    const uint32_t np = cur_.np;
    std::vector<uint32_t> a(np), b(np);
    std::vector<uint8_t> act(np), con(np);
    std::vector<double> sh(3 * (size_t)np), kn(np);
    vedo_contact_view cv{a.data(), b.data(), nullptr, nullptr, act.data(), sh.data(), kn.data(), con.data()};
    rc = get_interactions(cv);
    if (rc != VEDO_OK) return rc;
    std::vector<double> v0(np);
    if (np) {
        CK(cudaMemcpyAsync(v0.data(), cur_.v0, 8 * np, cudaMemcpyDeviceToHost, stream_));
        CK(cudaStreamSynchronize(stream_));
    }
    HRecords R;
    std::vector<uint32_t> idx;
    for (uint32_t k = 0; k < np; ++k)
        if (act[k]) idx.push_back(k);
    std::sort(idx.begin(), idx.end(), [&](uint32_t x, uint32_t y) {
        return a[x] != a[y] ? a[x] < a[y] : b[x] < b[y];
    });
    for (uint32_t k : idx) {
        R.first.push_back(a[k]); R.second.push_back(b[k]);
        R.contact.push_back(con[k]); R.bond.push_back(0);
        R.kn.push_back(kn[k]); R.v0.push_back(v0[k]);
        for (int q = 0; q < 3; ++q) {
            R.shear.push_back(sh[3 * k + q]);
            R.point.push_back(0.0); R.dirn.push_back(0.0); R.imp.push_back(0.0); R.aimp.push_back(0.0);
        }
        R.overlap.push_back(0.0);
    }
    HScene copy_rec = host_;
    copy_rec.rec = R;
    std::string msg;
    if (!vedo::write_ido(path, copy_rec, msg)) return fail(VEDO_ERR_IO, msg);
    return VEDO_OK;
}

int Engine::record_ido() {                                 // Consultant::RecordIDO (Consultant.cpp:217-230)
    char num[32];
    snprintf(num, sizeof(num), "%d", (int)(10000001 + record_count_));
    std::string file = out_prefix_ + "_" + (record_count_ < 11000001 ? std::string(num + 2) : std::string(num)) + ".ido";
    ++record_count_;
    return write_ido(file.c_str());
}

EngineBase* make_fp64_engine() { return new (std::nothrow) Engine(); }

}  // namespace vedo

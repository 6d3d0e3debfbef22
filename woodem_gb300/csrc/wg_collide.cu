// Broad phase: the full run of InsertionSortCollider (pkg/dem/InsertionSortCollider.cpp:445-646).
//
// The reference maintains three insertion-sorted bound arrays; every min/max inversion
// creates a potential contact when the closed 3-axis AABB test passes (:52-58, :63-98) or
// removes a non-real contact when the boxes separate. After each full run its contact set
// is therefore
//     { (i,j) : closed AABB overlap of i and j, Collider::mayCollide(i,j) }  U  { real contacts },
// and pending (law-removed) contacts survive only while their boxes overlap
// (ContactContainer::removePending, ContactContainer.hpp:78-93). This file computes exactly
// that set on the GPU:
//   1. Bo1 functors + verlet enlargement per particle            (k_aabb)
//   2. spheres bucketed into a uniform grid whose cell is at least the largest sphere box, by a counting
//      sort on the cell of the box minimum                        (k_make_grids, k_cellkey .. )
//   3. half-shell sweep over the sorted cells: every candidate pair is tested once with the
//      reference's closed-interval comparisons                   (k_pairs_ss)
//   4. facets query the cells their box covers; walls (infinite boxes) test every sphere
//   5. the new pair keys are radix-sorted and merged with the real contacts of the previous
//      set, carrying their persistent state                      (k_mark_orphans .. k_gather)
//   6. CSR incidence for the deterministic force sum              (k_lo_start, hi sort, k_hi_start)
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "wg_internal.h"
#include "wg_math.cuh"
#include "wg_ends.cuh"
#include "wg_geom.cuh"

namespace wg {

struct PeriBox;
// The counts of a full run; the host reads them twice, after the sweep and at the end.
struct CollideTotals {
    unsigned long long pairs;  // pairs found (past the buffer's capacity too)
    unsigned long long real, kept;  // real contacts before the merge, and those of them found among the new pairs
    unsigned long long act, actReal;  // totals of the work-list scans
    int32_t heavy, heavyFree;
    int32_t bad;  // a sphere's box is not finite
    int32_t far;  // some grid is far from zero (Grid::far)
};
struct CollideWork {
    // sphere and "large" (non-sphere) id lists, built at upload
    int32_t* sphereIds = nullptr;
    int nSph = 0;
    int32_t* largeIds = nullptr;   // facets with finite boxes (cell query)
    int nLarge = 0;
    int32_t* globalIds = nullptr;  // walls and oversized boxes (tested against every sphere)
    int nGlobal = 0;
    bool largeLargePossible = false;
    std::vector<int32_t> hLarge, hGlobal;
    // grid scratch
    uint32_t* cellKey = nullptr;  // cell of each sphere of sphereIds, and its place within the cell
    int32_t* cellRank = nullptr;
    uint32_t* skey = nullptr;     // cells of the spheres in cell order
    PeriBox* speri = nullptr;     // periodic: the boxes in cell order, in fractions of the cell
    float4* smnf = nullptr;       // box min rounded down, mask in w (cell order)
    float4* smxf = nullptr;       // box max rounded up, particle id in w
    int32_t* newLo = nullptr;     // first index of each lo id in the sorted new pairs
    int32_t* oldLo = nullptr;     // the same in the previous contact keys
    int64_t newLoCap = 0, oldLoCap = 0;
    bool oldLoValid = false;
    int32_t* cellOff = nullptr;   // first sphere of each cell
    int64_t cellOffCap = 0;
    long long* red = nullptr;     // reduction partials
    std::vector<int32_t> hChunk;      // grid-reduction chunks of sphereIds (never across scenes)
    std::vector<int32_t> hSceneChunk; // chunks of scene k: [hSceneChunk[k], hSceneChunk[k+1])
    std::vector<int64_t> hSceneSph;   // spheres of scene k: sphereIds[hSceneSph[k] .. hSceneSph[k+1])
    int32_t* dChunk = nullptr;
    Grid* dGrids = nullptr;
    int32_t* dSceneChunk = nullptr;   // chunks of scene k on the device
    bool chunksDirty = true;
    int32_t* gStart = nullptr;        // walls of scene k in globalIds (batches)
    // pairs
    uint64_t* pairs = nullptr;
    uint64_t* pairsSorted = nullptr;
    int64_t pairCap = 0;
    int32_t* pairCd = nullptr;        // periodic: cell distance of each new pair
    int32_t* pairCdSorted = nullptr;
    int32_t* newCd = nullptr;         // periodic: cell distance per merged contact
    CollideTotals* tot = nullptr;     // counts a run makes on the device
    CollideTotals* hTot = nullptr;    // pinned
    // merge scratch
    int32_t* orph = nullptr;      // flags then exclusive scan
    uint64_t* orphKey = nullptr;
    int32_t* orphSrc = nullptr;
    int32_t* src = nullptr;
    int64_t mergeCap = 0, orphCap = 0, srcCap = 0;
    // FP32-force mode, aperiodic: the packed state of the next set, and where each contact of this and the
    // next one is packed (plain active contacts alone)
    DevPackedSS Kb{};
    int32_t *packIdx = nullptr, *packIdxB = nullptr;
    int64_t packIdxCap = 0, packIdxCapB = 0;
    uint64_t* act = nullptr;      // exclusive scan of the active contacts (low half) and the plain ones of them (high)
    uint64_t* actReal = nullptr;  // FP64 mode: the same of the real contacts
    uint32_t* hiKeys = nullptr;
    uint32_t* hiKeysSorted = nullptr;
    int32_t* hiVals = nullptr;
    int64_t hiCap = 0;
    void* cubTmp = nullptr;
    size_t cubBytes = 0;
};

static const int BS = 256;
// spheres per block of the grid-bounds reduction: four loads a thread in flight, and a block for every
// SM from 150 000 spheres on
constexpr int64_t kGridChunk = 1024;

// ---------------------------------------------------------------- Bo1 functors + verlet
// Bo1_Sphere_Aabb::go pkg/dem/Sphere.cpp:50-79, Bo1_Wall_Aabb::go pkg/dem/Wall.cpp:24-33,
// Bo1_Facet_Aabb::go pkg/dem/Facet.cpp:177-200; enlargement by verletDist and nodeLastPos
// bookkeeping of updateBboxes_doFullRun pkg/dem/InsertionSortCollider.cpp:386-414.
__global__ void k_aabb(DevNodes N, DevParticles P, const ScenePar* __restrict__ spp, int* __restrict__ dErr) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P.n) return;
    const ScenePar& sp = spp[sceneOfP(P, p)];
    const int sh = P.shape[p];
    D3 mn, mx;
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    if (sh == WG_SHAPE_SPHERE) {
        const double4_32a pr = N.posr[p];
        const double f = (sp.bo1DistFactor > 0 ? sp.bo1DistFactor : 1.) * pr.w;
        D3 h{f, f, f};
        const D3 pos{pr.x, pr.y, pr.z};
        if (!sp.periodic) {
            mn = pos - h;
            mx = pos + h;
        } else {
            if (sp.hasShear) {
                const D3 perp = h;
                for (int ax = 0; ax < 3; ax++) {
                    const int ax1 = (ax + 1) % 3, ax2 = (ax + 2) % 3;
                    setComp(h, ax1, comp(h, ax1) + .5 * comp(perp, ax1) * (1 / sp.cellCos[ax] - 1));
                    setComp(h, ax2, comp(h, ax2) + .5 * comp(perp, ax2) * (1 / sp.cellCos[ax] - 1));
                }
            }
            DM3 U;
            for (int k = 0; k < 9; k++) U.m[k] = sp.unshear[k];
            const D3 u = mul(U, pos);
            mn = u - h;
            mx = u + h;
        }
        N.lastPos[p] = make_double4_32a(pr.x, pr.y, pr.z, 0.);
        if (N.lh) {
            N.lh[p] = N.mir[p].ph;
            N.ll[p] = N.mir[p].pl;
        }
    } else if (sh == WG_SHAPE_WALL) {
        const int ax = P.aux[p].x;
        const double4_32a pr = N.posr[p];
        mn = D3{-inf, -inf, -inf};
        mx = D3{inf, inf, inf};
        setComp(mn, ax, comp(D3{pr.x, pr.y, pr.z}, ax));
        setComp(mx, ax, comp(D3{pr.x, pr.y, pr.z}, ax));
        N.lastPos[p] = make_double4_32a(pr.x, pr.y, pr.z, 0.);
        if (N.lh) {
            N.lh[p] = N.mir[p].ph;
            N.ll[p] = N.mir[p].pl;
        }
    } else {
        const int4 fn = P.aux[p];
        const double ht = P.facet[p].w;
        const D3 htv{ht, ht, ht};
        const int nn[3] = {fn.x, fn.y, fn.z};
        for (int k = 0; k < 3; k++) {
            const double4_32a pr = N.posr[nn[k]];
            D3 v{pr.x, pr.y, pr.z};
            if (sp.periodic) {
                DM3 U;
                for (int q = 0; q < 9; q++) U.m[q] = sp.unshear[q];
                v = mul(U, v);
            }
            const D3 a = v - htv, b = v + htv;
            if (k == 0) {
                mn = a;
                mx = b;
            } else {
                mn = D3{smin(mn.x, a.x), smin(mn.y, a.y), smin(mn.z, a.z)};
                mx = D3{smax(mx.x, b.x), smax(mx.y, b.y), smax(mx.z, b.z)};
            }
            N.lastPos[nn[k]] = make_double4_32a(pr.x, pr.y, pr.z, 0.);
            if (N.lh) {
                N.lh[nn[k]] = N.mir[nn[k]].ph;
                N.ll[nn[k]] = N.mir[nn[k]].pl;
            }
        }
        N.lastPos[p] = N.posr[p];
        if (N.lh) {
            N.lh[p] = N.mir[p].ph;
            N.ll[p] = N.mir[p].pl;
        }
    }
    if (sp.verletDist > 0) {
        const D3 vd{sp.verletDist, sp.verletDist, sp.verletDist};
        mx = mx + vd;
        mn = mn - vd;
    }
    // a NaN coordinate would silently drop the particle from every pair test: stop the run instead
    if (isnan(mn.x) || isnan(mn.y) || isnan(mn.z) || isnan(mx.x) || isnan(mx.y) || isnan(mx.z)) atomicCAS(dErr, 0, 102);
    P.mn[p] = make_double4_32a(mn.x, mn.y, mn.z, 0.);
    P.mx[p] = make_double4_32a(mx.x, mx.y, mx.z, 0.);
}

// the next FP32 number above f
__device__ __forceinline__ float nextUp(float f) {
    const int u = __float_as_int(f);
    return f == 0.f ? __int_as_float(1) : __int_as_float(f > 0.f ? u + 1 : u - 1);
}

// An integer that orders FP64 numbers as they are (the same function takes it back). Minima and maxima of
// doubles would occupy the FP64 pipe, which those of integers do not.
__device__ __forceinline__ long long orderOf(long long bits) { return bits ^ ((bits >> 63) & 0x7fffffffffffffffLL); }

// ---------------------------------------------------------------- grid bounds over spheres
// partial[b] = {min mn.x, min mn.y, min mn.z, max mn.x, max mn.y, max mn.z, max extent} over the
// spheres ids[chunk[b] .. chunk[b+1]) (chunks never span two scenes of a batch), in FP64: rounded to FP32 where
// they stand, boxes of 1 cm at coordinates of 1e6 m would make the cells ten times too long. As orderOf().
__global__ void k_grid_reduce(DevParticles P, const int32_t* __restrict__ ids, const int32_t* __restrict__ chunk,
                              long long* __restrict__ partial) {
    __shared__ long long s[7][BS / 32];
    const unsigned FULL = 0xffffffffu;
    const long long INF = 0x7ff0000000000000LL, most = orderOf(INF), least = orderOf(INF | (1LL << 63));
    long long v[7] = {most, most, most, least, least, least, 0};
    bool bad = false;  // an edge that is not finite: a NaN or infinite position
    for (int i = chunk[blockIdx.x] + threadIdx.x; i < chunk[blockIdx.x + 1]; i += blockDim.x) {
        const int p = ids[i];
        const double4_32a a = P.mn[p], b = P.mx[p];
        const double lo[3] = {a.x, a.y, a.z}, hi[3] = {b.x, b.y, b.z};
        for (int q = 0; q < 3; q++) {
            const long long u = orderOf(__double_as_longlong(lo[q])), e = __double_as_longlong(hi[q] - lo[q]);
            bad = bad || (e & INF) == INF;
            v[q] = min(v[q], u);
            v[3 + q] = max(v[3 + q], u);
            v[6] = max(v[6], e);
        }
    }
    if (bad) v[6] = INF;
    for (int o = 16; o > 0; o >>= 1) {
        for (int q = 0; q < 3; q++) v[q] = min(v[q], __shfl_down_sync(FULL, v[q], o));
        for (int q = 3; q < 7; q++) v[q] = max(v[q], __shfl_down_sync(FULL, v[q], o));
    }
    if ((threadIdx.x & 31) == 0)
        for (int q = 0; q < 7; q++) s[q][threadIdx.x >> 5] = v[q];
    __syncthreads();
    if (threadIdx.x < 7) {
        const int q = threadIdx.x;
        long long m = s[q][0];
        for (int w = 1; w < BS / 32; w++) m = q < 3 ? min(m, s[q][w]) : max(m, s[q][w]);
        partial[blockIdx.x * 7 + q] = m;
    }
}

// The grid of each scene from the partial bounds of its chunks: cells slightly larger than the largest
// sphere box, so that boxes that overlap sit in adjacent cells, and no more than cellBound() of them.
// A warp per scene, all warps of the block for a single one, then the first cell keys in scene order. A bound that is not
// finite sets tot->bad.
__host__ __device__ __forceinline__ int64_t cellBound(int64_t spheres, int scenes) {
    const int64_t least = scenes > 1 ? 64 : 1 << 16;
    return 8 * spheres > least ? 8 * spheres : least;
}
constexpr double kCellMargin = 2e-6;
__global__ void __launch_bounds__(1024) k_make_grids(int K, const int32_t* __restrict__ chunk, const int32_t* __restrict__ sceneChunk,
                                                     const long long* __restrict__ partial, const ScenePar* __restrict__ spp, int peri,
                                                     Grid* __restrict__ out, CollideTotals* __restrict__ tot) {
    __shared__ long long s[32][7];
    const unsigned FULL = 0xffffffffu;
    const long long INF = 0x7ff0000000000000LL, most0 = orderOf(INF), least0 = orderOf(INF | (1LL << 63));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = blockDim.x >> 5, each = K == 1 ? warps : 1, part = K == 1 ? warp : 0;  // warps of a scene
    for (int k = K == 1 ? 0 : warp; k < K; k += K == 1 ? 1 : warps) {
        const int c0 = sceneChunk[k], c1 = sceneChunk[k + 1];
        long long u[7] = {most0, most0, most0, least0, least0, least0, 0};
        auto across = [&]() {  // to the first lane
            for (int o = 16; o > 0; o >>= 1) {
                for (int q = 0; q < 3; q++) u[q] = min(u[q], __shfl_down_sync(FULL, u[q], o));
                for (int q = 3; q < 7; q++) u[q] = max(u[q], __shfl_down_sync(FULL, u[q], o));
            }
        };
        for (int b = c0 + 32 * part + lane; b < c1; b += 32 * each) {
            for (int q = 0; q < 3; q++) u[q] = min(u[q], partial[7 * b + q]);
            for (int q = 3; q < 7; q++) u[q] = max(u[q], partial[7 * b + q]);
        }
        across();
        if (K == 1) {
            if (lane == 0)
                for (int q = 0; q < 7; q++) s[warp][q] = u[q];
            __syncthreads();
            if (warp) continue;
            if (lane < warps)
                for (int q = 0; q < 7; q++) u[q] = s[lane][q];
            across();
        }
        if (lane) continue;
        double v[7];
        for (int q = 0; q < 7; q++) v[q] = __longlong_as_double(orderOf(u[q]));
        Grid g{0, 0, 0, 1, 1, 1, 1, 1, 1, 0, 0};
        if (c0 != c1) {
            bool fine = true;
            for (int q = 0; q < 7; q++) fine = fine && isfinite(v[q]);
            if (!fine) tot->bad = 1;
            else {
                const int64_t most = cellBound((int64_t)chunk[c1] - chunk[c0], K);
                double h = v[6] * (1 + kCellMargin) + 1e-300;
                const double ext[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
                int64_t dims[3];
                for (;;) {
                    for (int q = 0; q < 3; q++) {
                        // the periodic cell [0, size) per axis (unsheared coordinates), or the bounds
                        const double d = peri ? floor(spp->cellSize[q] / h) : floor(ext[q] / h) + 1;
                        dims[q] = d < 1. ? 1 : (d > 1e9 ? (int64_t)1000000000 : (int64_t)d);
                    }
                    if ((double)dims[0] * (double)dims[1] * (double)dims[2] <= (double)most) break;
                    h *= 1.25;
                }
                g.ox = v[0]; g.oy = v[1]; g.oz = v[2]; g.h = h;
                g.rh = 1. / h;
                g.nx = (int32_t)dims[0]; g.ny = (int32_t)dims[1]; g.nz = (int32_t)dims[2];
                g.ncell = dims[0] * dims[1] * dims[2];
                // coordinates that FP32 numbers resolve badly, compared with a cell: the boxes in cell order are
                // kept relative to the grid's origin
                for (int q = 0; q < 6; q++)
                    if (fabs(v[q]) > 4096. * h) g.far = tot->far = 1;
                if (peri)
                    for (int q = 0; q < 3; q++)
                        if (!(h <= 0.49 * spp->cellSize[q])) g.exact = 1;
            }
        }
        out[k] = g;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    int64_t base = 0;
    for (int k0 = 0; k0 < K; k0 += 32) {
        const int k = k0 + lane;
        const int64_t mine = k < K ? out[k].ncell : 0;
        int64_t upTo = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t w = __shfl_up_sync(FULL, upTo, o);
            if (lane >= o) upTo += w;
        }
        if (k < K) out[k].base = base + upTo - mine;
        base += __shfl_sync(FULL, upTo, 31);
    }
}

// rh = 1/h: over 2^31 cells the product is off by less than half the margin that h has over the largest box
__device__ __forceinline__ int cellCoord(double v, double o, double rh, int n) {
    const int ci = __double2int_rd((v - o) * rh);
    return ci < 0 ? 0 : (ci >= n ? n - 1 : ci);
}

// The cell of each sphere and its place within it (count: spheres per cell, zero before). The places
// depend on the atomics' order; the pairs found, sorted afterwards, do not.
__global__ void k_cellkey(DevParticles P, const int32_t* __restrict__ ids, int n, const Grid* __restrict__ Gs,
                          uint32_t* __restrict__ key, int32_t* __restrict__ rank, int32_t* __restrict__ count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int p = ids[i];
    const Grid G = Gs[sceneOfP(P, p)];
    const double4_32a a = P.mn[p];
    const int cx = cellCoord(a.x, G.ox, G.rh, G.nx), cy = cellCoord(a.y, G.oy, G.rh, G.ny), cz = cellCoord(a.z, G.oz, G.rh, G.nz);
    const uint32_t k = (uint32_t)(G.base + ((int64_t)cz * G.ny + cy) * G.nx + cx);
    key[i] = k;
    rank[i] = atomicAdd(count + k, 1);
}

__device__ __forceinline__ int64_t lowerBound32(const uint32_t* a, int64_t n, uint32_t k) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        int64_t m = (lo + hi) >> 1;
        if (a[m] < k) lo = m + 1; else hi = m;
    }
    return lo;
}
__device__ __forceinline__ int64_t lowerBound64(const uint64_t* a, int64_t n, uint64_t k) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        int64_t m = (lo + hi) >> 1;
        if (a[m] < k) lo = m + 1; else hi = m;
    }
    return lo;
}

// the spheres' boxes in cell order, rounded outward to FP32 (of a grid far from zero, relative to its origin: the
// subtraction keeps their order, and so what overlapF and overlapOuter conclude from it)
__global__ void k_gather_sorted(DevParticles P, const int32_t* __restrict__ ids, int n, const Grid* __restrict__ Gs, const int* __restrict__ far,
                                const uint32_t* __restrict__ key,
                                const int32_t* __restrict__ rank, const int32_t* __restrict__ off, uint32_t* __restrict__ skey,
                                float4* __restrict__ smnf, float4* __restrict__ smxf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int anyFar = *far;
    const int p = ids[i];
    double4_32a a = P.mn[p], b = P.mx[p];
    if (anyFar) {
        const Grid& G = Gs[sceneOfP(P, p)];
        if (G.far) {
            a = make_double4_32a(a.x - G.ox, a.y - G.oy, a.z - G.oz, 0.);
            b = make_double4_32a(b.x - G.ox, b.y - G.oy, b.z - G.oz, 0.);
        }
    }
    const int at = off[key[i]] + rank[i];
    skey[at] = key[i];
    smnf[at] = make_float4(__double2float_rd(a.x), __double2float_rd(a.y), __double2float_rd(a.z), __uint_as_float(P.mask[p]));
    smxf[at] = make_float4(__double2float_ru(b.x), __double2float_ru(b.y), __double2float_ru(b.z), __int_as_float(p));
}

// Collider::mayCollide pkg/dem/Collision.cpp:19-41 for particles that share no nodes
__device__ __forceinline__ bool maskOk(uint32_t a, uint32_t b, uint32_t lone) { return (a & b) != 0 && (a & b & lone) == 0; }

// a pair as it is sorted: the lo id above the hi id, `bits` bits each (the fewest that hold an id)
__device__ __forceinline__ uint64_t pairKey(int a, int b, int bits) {
    const int lo = a < b ? a : b, hi = a < b ? b : a;
    return ((uint64_t)(uint32_t)lo << bits) | (uint32_t)hi;
}
__device__ __forceinline__ void emitPair(int a, int b, int bits, uint64_t* pairs, int64_t cap, unsigned long long* counter) {
    const unsigned long long idx = atomicAdd(counter, 1ull);
    if ((int64_t)idx < cap) pairs[idx] = pairKey(a, b, bits);
}

// Outward-rounded FP32 boxes overlap whenever the FP64 boxes do, so the FP32 test rejects most
// candidates exactly. One FP32 number inward of each outward bound lies within the FP64 box, so boxes
// shrunk to those overlap only if the FP64 boxes do, and accept most of the rest exactly; the FP64 test
// (InsertionSortCollider::spatialOverlap) decides the cases in between.
__device__ __forceinline__ bool overlapF(const float4& mn1, const float4& mx1, const float4& mn2, const float4& mx2) {
    return (mn1.x <= mx2.x) && (mx1.x >= mn2.x) && (mn1.y <= mx2.y) && (mx1.y >= mn2.y) && (mn1.z <= mx2.z) && (mx1.z >= mn2.z);
}
__device__ __forceinline__ float nextDown(float f) { return -nextUp(-f); }
__device__ __forceinline__ float4 upOf(const float4& f) { return make_float4(nextUp(f.x), nextUp(f.y), nextUp(f.z), 0.f); }
__device__ __forceinline__ float4 downOf(const float4& f) { return make_float4(nextDown(f.x), nextDown(f.y), nextDown(f.z), 0.f); }
// the FP64 closed overlap of particles p and q whose outward-rounded boxes (mn, mx) overlap
__device__ __forceinline__ bool overlapOuter(const DevParticles& P, int p, int q, const float4& mn1, const float4& mx1, const float4& mn2,
                                             const float4& mx2) {
    if (overlapF(upOf(mn1), downOf(mx1), upOf(mn2), downOf(mx2))) return true;
    return overlap3(P.mn[p], P.mx[p], P.mn[q], P.mx[q]);
}

// Pairs found by the lanes of a warp are written with one atomic per warp: each lane keeps up to
// kPairBuf pairs in registers, the warp reserves room for all of them at once (the single counter
// would otherwise serialise millions of atomics in L2), and a lane whose buffer fills flushes it
// the same way. Must be called by all lanes of the warp together.
constexpr int kPairBuf = 8;
__device__ __forceinline__ void flushPairs(uint64_t (&buf)[kPairBuf], int& nb, uint64_t* pairs, int64_t cap,
                                           unsigned long long* counter) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int incl = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total > 0) base = atomicAdd(counter, (unsigned long long)total);
    base = __shfl_sync(FULL, base, 31);
    const unsigned long long at = base + (unsigned long long)(incl - nb);
#pragma unroll
    for (int q = 0; q < kPairBuf; q++)
        if (q < nb && (int64_t)(at + q) < cap) pairs[at + q] = buf[q];
    nb = 0;
}

// Appends key to the lane's pair buffer (register-resident: the slot is chosen by unrolled
// comparisons, never by a runtime index).
__device__ __forceinline__ void pushPair(uint64_t (&buf)[kPairBuf], int& nb, uint64_t key) {
#pragma unroll
    for (int q = 0; q < kPairBuf; q++)
        if (q == nb) buf[q] = key;
    nb++;
}

// Half-shell sweep: particle i tests the rest of its own cell, the next cell in x, and the
// three-cell x-runs of the rows (dy,dz) in {(1,0),(-1,1),(0,1),(1,1)}; each pair is met once.
// The candidate ranges of a lane are walked as one sequence, kSweepBatch candidates at a time
// (their boxes are loaded together), so that the warp can flush together.
constexpr int kSweepBatch = 2;
__global__ void __launch_bounds__(256, 4) k_pairs_ss(DevParticles P, const uint32_t* __restrict__ skey, const float4* __restrict__ smnf,
                                                     const float4* __restrict__ smxf, int n, const Grid* __restrict__ Gs,
                                                     const int32_t* __restrict__ off, uint32_t lone, int bits, const int* __restrict__ bad,
                                                     uint64_t* __restrict__ pairs, int64_t cap, unsigned long long* __restrict__ counter) {
    if (*bad) return;
    const unsigned FULL = 0xffffffffu;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    // the five ranges [b_r, b_r + len_r) of sorted indices, as starts and cumulative lengths
    int b0 = 0, b1 = 0, b2 = 0, b3 = 0, b4 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0, total = 0;
    float4 fn1 = make_float4(0.f, 0.f, 0.f, 0.f), fx1 = fn1;
    uint32_t m1 = 0;
    int pi = 0;
    if (valid) {
        fn1 = smnf[i];
        fx1 = smxf[i];
        m1 = __float_as_uint(fn1.w);
        pi = __float_as_int(fx1.w);
        const Grid G = Gs[sceneOfP(P, pi)];
        const uint32_t k = (uint32_t)((int64_t)skey[i] - G.base);
        const int cx = (int)(k % (uint32_t)G.nx);
        const int cy = (int)((k / (uint32_t)G.nx) % (uint32_t)G.ny);
        const int cz = (int)(k / ((uint32_t)G.nx * (uint32_t)G.ny));
        const int cx1 = cx + 1 < G.nx ? cx + 1 : cx;
        const int x0 = cx > 0 ? cx - 1 : 0;
        int rb[4], re[4];
        const int DY[4] = {1, -1, 0, 1}, DZ[4] = {0, 1, 1, 1};
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int y = cy + DY[r], z = cz + DZ[r];
            rb[r] = re[r] = 0;
            if (y < 0 || y >= G.ny || z >= G.nz) continue;
            const int64_t rowBase = G.base + ((int64_t)z * G.ny + y) * G.nx;
            rb[r] = off[rowBase + x0];
            re[r] = off[rowBase + cx1 + 1];
        }
        b0 = i + 1;
        c1 = off[G.base + ((int64_t)cz * G.ny + cy) * G.nx + cx1 + 1] - b0;
        b1 = rb[0];
        c2 = c1 + (re[0] - rb[0]);
        b2 = rb[1];
        c3 = c2 + (re[1] - rb[1]);
        b3 = rb[2];
        c4 = c3 + (re[2] - rb[2]);
        b4 = rb[3];
        total = c4 + (re[3] - rb[3]);
    }
    uint64_t buf[kPairBuf];
    int nb = 0;
    for (int v0 = 0; __any_sync(FULL, v0 < total); v0 += kSweepBatch) {
        int jj[kSweepBatch];
        float4 a[kSweepBatch], c[kSweepBatch];
#pragma unroll
        for (int u = 0; u < kSweepBatch; u++) {
            const int v = v0 + u;
            jj[u] = v >= total ? -1
                               : (v < c1 ? b0 + v : (v < c2 ? b1 + (v - c1) : (v < c3 ? b2 + (v - c2) : (v < c4 ? b3 + (v - c3) : b4 + (v - c4)))));
            if (jj[u] >= 0) {
                a[u] = smnf[jj[u]];
                c[u] = smxf[jj[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kSweepBatch; u++)
            if (jj[u] >= 0 && overlapF(fn1, fx1, a[u], c[u]) && maskOk(m1, __float_as_uint(a[u].w), lone) &&
                overlapOuter(P, pi, __float_as_int(c[u].w), fn1, fx1, a[u], c[u]))
                pushPair(buf, nb, pairKey(pi, __float_as_int(c[u].w), bits));
        if (__any_sync(FULL, nb > kPairBuf - kSweepBatch)) flushPairs(buf, nb, pairs, cap, counter);
    }
    flushPairs(buf, nb, pairs, cap, counter);
}

// A box relative to its grid's origin (out of line: inlined, the subtractions become predicated FP64 instructions of
// every warp).
static __device__ __noinline__ void makeRelative(const Grid& G, double4_32a& a, double4_32a& b) {
    a = make_double4_32a(a.x - G.ox, a.y - G.oy, a.z - G.oz, 0.);
    b = make_double4_32a(b.x - G.ox, b.y - G.oy, b.z - G.oz, 0.);
}
// A facet (finite box) against the spheres of the cells its box can reach: a sphere j that
// overlaps it has mn_j in [mn_f - h, mx_f] on every axis. One warp per facet; its lanes split
// each x-run of cells.
__global__ void k_pairs_local(DevParticles P, const int32_t* __restrict__ lids, int nl, const float4* __restrict__ smnf,
                              const float4* __restrict__ smxf, const Grid* __restrict__ Gs, const int32_t* __restrict__ off, uint32_t lone,
                              int bits, const int* __restrict__ bad, uint64_t* __restrict__ pairs, int64_t cap,
                              unsigned long long* __restrict__ counter) {
    if (*bad) return;
    const unsigned FULL = 0xffffffffu;
    const int t = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= nl) return;  // warp-uniform
    const int p = lids[t];
    const Grid G = Gs[sceneOfP(P, p)];
    const double4_32a mn1 = P.mn[p], mx1 = P.mx[p];
    double4_32a rn = mn1, rx = mx1;
    if (G.far) makeRelative(G, rn, rx);
    const float4 fn1 = make_float4(__double2float_rd(rn.x), __double2float_rd(rn.y), __double2float_rd(rn.z), 0.f);
    const float4 fx1 = make_float4(__double2float_ru(rx.x), __double2float_ru(rx.y), __double2float_ru(rx.z), 0.f);
    const uint32_t m1 = P.mask[p];
    const int x0 = cellCoord(mn1.x - G.h, G.ox, G.rh, G.nx), x1 = cellCoord(mx1.x, G.ox, G.rh, G.nx);
    const int y0 = cellCoord(mn1.y - G.h, G.oy, G.rh, G.ny), y1 = cellCoord(mx1.y, G.oy, G.rh, G.ny);
    const int z0 = cellCoord(mn1.z - G.h, G.oz, G.rh, G.nz), z1 = cellCoord(mx1.z, G.oz, G.rh, G.nz);
    uint64_t buf[kPairBuf];
    int nb = 0;
    for (int z = z0; z <= z1; z++)
        for (int y = y0; y <= y1; y++) {
            const int64_t rowBase = G.base + ((int64_t)z * G.ny + y) * G.nx;
            const int beg = off[rowBase + x0], end = off[rowBase + x1 + 1];
            for (int j0 = beg; j0 < end; j0 += 32) {
                const int j = j0 + lane;
                if (j < end) {
                    const float4 fn2 = smnf[j], fx2 = smxf[j];
                    const int q = __float_as_int(fx2.w);
                    if (q != p && overlapF(fn1, fx1, fn2, fx2) && maskOk(m1, __float_as_uint(fn2.w), lone) &&
                        overlapOuter(P, p, q, fn1, fx1, fn2, fx2))
                        pushPair(buf, nb, pairKey(p, q, bits));
                }
                if (__any_sync(FULL, nb == kPairBuf)) flushPairs(buf, nb, pairs, cap, counter);
            }
        }
    flushPairs(buf, nb, pairs, cap, counter);
}

// ---------------------------------------------------------------- periodic cell
__global__ void k_cellkey_peri(DevParticles P, const int32_t* __restrict__ ids, int n, const Grid* __restrict__ Gs,
                               const ScenePar* __restrict__ spp, uint32_t* __restrict__ key, int32_t* __restrict__ rank,
                               int32_t* __restrict__ count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ScenePar& sp = *spp;
    const Grid G = *Gs;
    const int p = ids[i];
    const double4_32a a = P.mn[p];
    const double w[3] = {cellWrapRelD(a.x, 0., sp.cellSize[0]), cellWrapRelD(a.y, 0., sp.cellSize[1]),
                         cellWrapRelD(a.z, 0., sp.cellSize[2])};
    const int nn[3] = {G.nx, G.ny, G.nz};
    int c[3];
    for (int k = 0; k < 3; k++) {
        const int ci = (int)floor(w[k] / (sp.cellSize[k] / nn[k]));
        c[k] = ci < 0 ? 0 : (ci >= nn[k] ? nn[k] - 1 : ci);
    }
    const uint32_t k = (uint32_t)(((int64_t)c[2] * G.ny + c[1]) * G.nx + c[0]);
    key[i] = k;
    rank[i] = atomicAdd(count + k, 1);
}
// Pairs emitted with their cell distance (periods of the lo particle minus those of the hi one).
__device__ __forceinline__ void flushPairsCd(uint64_t (&buf)[kPairBuf], int32_t (&cbuf)[kPairBuf], int& nb, uint64_t* pairs,
                                             int32_t* cds, int64_t cap, unsigned long long* counter) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int incl = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total > 0) base = atomicAdd(counter, (unsigned long long)total);
    base = __shfl_sync(FULL, base, 31);
    const unsigned long long at = base + (unsigned long long)(incl - nb);
#pragma unroll
    for (int q = 0; q < kPairBuf; q++)
        if (q < nb && (int64_t)(at + q) < cap) {
            pairs[at + q] = buf[q];
            cds[at + q] = cbuf[q];
        }
    nb = 0;
}
// A sphere's box in the periodic sweep, in sorted order: the box minimum as a fraction of the cell in
// [0, 1) with its period taken off, and the box's edges as fractions.
struct PeriBox {
    float4 u;  // fraction per axis, mask in w
    float4 l;  // edges per axis
    int4 p;    // periods per axis, particle id in w
};
// How far the FP32 fractions above may be from the exact ones: below 3 roundings of 2^-24 each with
// those of the FP64 quotients behind them; ten times that is decided in FP64.
constexpr float kPeriEps = 2e-6f;
__global__ void k_gather_peri(DevParticles P, const int32_t* __restrict__ ids, int n, const uint32_t* __restrict__ key,
                              const int32_t* __restrict__ rank, const int32_t* __restrict__ off, const ScenePar* __restrict__ spp,
                              uint32_t* __restrict__ skey, PeriBox* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int q = ids[i], at = off[key[i]] + rank[i];
    skey[at] = key[i];
    const double4_32a a = P.mn[q], b = P.mx[q];
    const double m[3] = {a.x, a.y, a.z}, x[3] = {b.x, b.y, b.z};
    float u[3], l[3];
    int p[3];
    for (int k = 0; k < 3; k++) {
        const double d = 1. / spp->cellSize[k], f = m[k] * d, fl = floor(f);
        p[k] = (int)fl;
        u[k] = (float)(f - fl);
        l[k] = (float)((x[k] - m[k]) * d);
    }
    out[at].u = make_float4(u[0], u[1], u[2], __uint_as_float(P.mask[q]));
    out[at].l = make_float4(l[0], l[1], l[2], 0.f);
    out[at].p = make_int4(p[0], p[1], p[2], q);
}
// out of line: a few pairs in ten thousand come here
static __device__ __noinline__ int overlapPeriExact(const DevParticles& P, int lo, int hi, const ScenePar* __restrict__ spp, int* per) {
    return overlapPeri(P.mn[lo], P.mx[lo], P.mn[hi], P.mx[hi], spp->cellSize, per);
}
// One axis of the periodic overlap of boxes i and j in fractions of the cell: d, the distance from i's
// minimum to the nearest image of j's, taken modulo 1; r the period taken off. The boxes overlap where
// the one that starts later starts within the other (boxes shorter than half the cell). Returns the
// gap (negative: overlap).
__device__ __forceinline__ float periGap(float ui, float li, float uj, float lj, float& d, int& r) {
    d = uj - ui;
    const float f = rintf(d);
    r = (int)f;
    d -= f;
    return d >= 0.f ? d - li : -d - lj;
}
// Periodic sweep: particle i tests the spheres of higher id in the (up to 27, wrapped, distinct)
// cells around its own; each pair is met once, from its lo id.
// The exact test (overlapPeri: 18 FP64 divisions a pair) decides only the pairs with a gap or a
// distance within kPeriEps of zero; every other one is rejected, or accepted with its periods, from
// the FP32 fractions:
//   the origin of overlapPeri's wrap is the box that starts first (d > 0: i's, d < 0: j's), so that
//   the periods are p_i - p_j - r either way, and the overlap is a gap of zero or less.
// G.exact: some box is about half the cell or longer on an axis, where overlapPeri raises an error;
// every candidate then goes through it.
// Bound by instruction issue over about 85 candidates a sphere. With the exact test on every candidate
// the sweep took nearly all of a full run of 200 000 spheres: 9.0 -> 0.48 ms.
__global__ void __launch_bounds__(128) k_pairs_ss_peri(DevParticles P, const uint32_t* __restrict__ skey, const PeriBox* __restrict__ box,
                                                       int n, const Grid* __restrict__ Gs, const int32_t* __restrict__ off, uint32_t lone,
                                                       int bits, const int* __restrict__ bad, const ScenePar* __restrict__ spp,
                                                       uint64_t* __restrict__ pairs, int32_t* __restrict__ cds, int64_t cap,
                                                       unsigned long long* __restrict__ counter, int* __restrict__ dErr) {
    if (*bad) return;
    const Grid G = *Gs;
    const int exactOnly = G.exact;
    const unsigned FULL = 0xffffffffu;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    const int nx = G.nx, ny = G.ny, nz = G.nz;
    int cx = 0, cy = 0, cz = 0;
    PeriBox me{};
    if (valid) {
        const uint32_t k = skey[i];
        cx = (int)(k % (uint32_t)nx);
        cy = (int)((k / (uint32_t)nx) % (uint32_t)ny);
        cz = (int)(k / ((uint32_t)nx * (uint32_t)ny));
        me = box[i];
    }
    const uint32_t m1 = __float_as_uint(me.u.w);
    const int pi = me.p.w;
    // distinct wrapped rows; along x the cells cx-1 .. cx+1 as one run of sorted spheres, and the cell
    // across the boundary as a second one
    const int oy = ny >= 3 ? 3 : ny, oz = nz >= 3 ? 3 : nz;
    const int xa = nx >= 3 ? max(cx - 1, 0) : 0, xb = nx >= 3 ? min(cx + 1, nx - 1) : nx - 1;
    const int xw = nx >= 3 ? (cx == 0 ? nx - 1 : (cx == nx - 1 ? 0 : -1)) : -1;
    uint64_t buf[kPairBuf];
    int32_t cbuf[kPairBuf];
    int nb = 0;
    for (int q = 0; q < 2 * oy * oz; q++) {
        const int row = q >> 1;
        const int dy = row % oy - (oy == 3 ? 1 : 0), dz = row / oy - (oz == 3 ? 1 : 0);
        int y = cy + dy, z = cz + dz;
        y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
        z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
        const int64_t rowBase = ((int64_t)z * ny + y) * nx;
        int j = 0, end = 0;
        if (valid) {
            if (!(q & 1)) {
                j = off[rowBase + xa];
                end = off[rowBase + xb + 1];
            } else if (xw >= 0) {
                j = off[rowBase + xw];
                end = off[rowBase + xw + 1];
            }
        }
        for (; __any_sync(FULL, j < end); j++) {
            if (j < end) {
                const float4 u = box[j].u, l = box[j].l;
                float dx, dyy, dzz;
                int rx, ry, rz;
                const float gx = periGap(me.u.x, me.l.x, u.x, l.x, dx, rx), gy = periGap(me.u.y, me.l.y, u.y, l.y, dyy, ry),
                            gz = periGap(me.u.z, me.l.z, u.z, l.z, dzz, rz);
                const float gap = fmaxf(fmaxf(gx, gy), gz);
                if (gap <= kPeriEps || exactOnly) {
                    const int4 p = box[j].p;
                    const int pj = p.w;
                    if (pj > pi && maskOk(m1, __float_as_uint(u.w), lone)) {
                        int per[3] = {me.p.x - p.x - rx, me.p.y - p.y - ry, me.p.z - p.z - rz};
                        int r = 1;
                        if (exactOnly || gap >= -kPeriEps || fminf(fminf(fabsf(dx), fabsf(dyy)), fabsf(dzz)) <= kPeriEps)
                            r = overlapPeriExact(P, pi, pj, spp, per);
                        if (r < 0) atomicCAS(dErr, 0, 103);
                        else if (r > 0) {
                            const uint64_t key = pairKey(pi, pj, bits);
                            const int32_t cd = packCellDist(per[0], per[1], per[2]);
#pragma unroll
                            for (int v = 0; v < kPairBuf; v++)
                                if (v == nb) {
                                    buf[v] = key;
                                    cbuf[v] = cd;
                                }
                            nb++;
                        }
                    }
                }
            }
            if (__any_sync(FULL, nb == kPairBuf)) flushPairsCd(buf, cbuf, nb, pairs, cds, cap, counter);
        }
    }
    flushPairsCd(buf, cbuf, nb, pairs, cds, cap, counter);
}
// Walls against every sphere with the periodic overlap test (pair oriented lo, hi).
__global__ void k_pairs_global_peri(DevParticles P, const int32_t* __restrict__ gids, int ng, const int32_t* __restrict__ sph, int ns,
                                    uint32_t lone, int bits, const ScenePar* __restrict__ spp, uint64_t* __restrict__ pairs,
                                    int32_t* __restrict__ cds, int64_t cap, unsigned long long* __restrict__ counter,
                                    int* __restrict__ dErr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    const int s = sph[i];
    for (int g = 0; g < ng; g++) {
        const int w = gids[g];
        if (w == s || !maskOk(P.mask[s], P.mask[w], lone)) continue;
        const int lo = s < w ? s : w, hi = s < w ? w : s;
        int per[3];
        const int r = overlapPeri(P.mn[lo], P.mx[lo], P.mn[hi], P.mx[hi], spp->cellSize, per);
        if (r < 0) atomicCAS(dErr, 0, 103);
        else if (r > 0) {
            const unsigned long long idx = atomicAdd(counter, 1ull);
            if ((int64_t)idx < cap) {
                pairs[idx] = pairKey(lo, hi, bits);
                cds[idx] = packCellDist(per[0], per[1], per[2]);
            }
        }
    }
}

// Walls (and any box too large for the grid) against every sphere.
// gids are grouped by scene: the walls of scene k are gids[gStart[k] .. gStart[k+1]) (gStart null:
// one scene, all of gids)
__global__ void k_pairs_global(DevParticles P, const int32_t* __restrict__ gids, int ng, const int32_t* __restrict__ gStart,
                               const int32_t* __restrict__ sph, int ns, uint32_t lone, int bits, uint64_t* __restrict__ pairs, int64_t cap,
                               unsigned long long* __restrict__ counter) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    const int s = sph[i];
    const double4_32a mn1 = P.mn[s], mx1 = P.mx[s];
    const uint32_t m1 = P.mask[s];
    const int sc = sceneOfP(P, s);
    const int g0 = gStart ? gStart[sc] : 0, g1 = gStart ? gStart[sc + 1] : ng;
    for (int g = g0; g < g1; g++) {
        const int w = gids[g];
        if (w == s) continue;
        if (overlap3(mn1, mx1, P.mn[w], P.mx[w]) && maskOk(m1, P.mask[w], lone)) emitPair(s, w, bits, pairs, cap, counter);
    }
}

// Pairs among non-spheres (only launched when their masks allow contact at all).
__global__ void k_pairs_large_large(DevParticles P, const int32_t* __restrict__ ids, int n, uint32_t lone, int bits,
                                    uint64_t* __restrict__ pairs, int64_t cap, unsigned long long* __restrict__ counter) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * n) return;
    const int a = (int)(t / n), b = (int)(t % n);
    if (b <= a) return;
    const int pa = ids[a], pb = ids[b];
    if (sceneOfP(P, pa) != sceneOfP(P, pb)) return;  // the scenes of a batch never interact
    // facets sharing a node may not collide (Collision.cpp:27-31)
    if (P.shape[pa] == WG_SHAPE_FACET && P.shape[pb] == WG_SHAPE_FACET) {
        const int4 x = P.aux[pa], y = P.aux[pb];
        const int xa[3] = {x.x, x.y, x.z}, ya[3] = {y.x, y.y, y.z};
        for (int u = 0; u < 3; u++)
            for (int v = 0; v < 3; v++)
                if (xa[u] == ya[v]) return;
    }
    if (overlap3(P.mn[pa], P.mx[pa], P.mn[pb], P.mx[pb]) && maskOk(P.mask[pa], P.mask[pb], lone)) emitPair(pa, pb, bits, pairs, cap, counter);
}

// ---------------------------------------------------------------- merge with previous contacts
// a contact of a particle that was (re)loaded or parked since the last full run does not survive
__device__ __forceinline__ bool freshPair(const uint8_t* fresh, uint64_t k) {
    return fresh && (fresh[(int)(k >> 32)] || fresh[(int)(k & 0xffffffffu)]);
}
// start[p] = first index of key array (sorted ascending, key = lo << 32 | hi) whose lo is >= p,
// for p in [0, nPar]; one thread per index fills the ids between its lo and its predecessor's.
__global__ void k_lo_bounds(const uint64_t* __restrict__ key, int64_t n, int nPar, int32_t* __restrict__ start) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    const int cur = (i < n) ? (int)(key[i] >> 32) : nPar;
    const int prev = (i > 0) ? (int)(key[i - 1] >> 32) : -1;
    for (int q = prev + 1; q <= cur && q <= nPar; q++) start[q] = (int32_t)i;
}
// position of k in the sorted key array, searched within the range of its lo id (a few entries
// for a sphere, thousands for a wall), or -1
__device__ __forceinline__ int64_t findInRange(const uint64_t* __restrict__ key, const int32_t* __restrict__ start, uint64_t k) {
    const int lo = (int)(k >> 32);
    int64_t a = start[lo], b = start[lo + 1];
    while (a < b) {
        const int64_t m = (a + b) >> 1;
        if (key[m] < k) a = m + 1;
        else b = m;
    }
    return (a < start[lo + 1] && key[a] == k) ? a : -1;
}
// the sorted pairs (lo << bits | hi) as contact keys (lo << 32 | hi), with k_lo_bounds of them
__global__ void k_unpack_keys(const uint64_t* __restrict__ in, int64_t n, int bits, int nPar, uint64_t* __restrict__ out,
                              int32_t* __restrict__ start) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    const int prev = i > 0 ? (int)(in[i - 1] >> bits) : -1;
    int cur = nPar;
    if (i < n) {
        const uint64_t k = in[i];
        cur = (int)(k >> bits);
        out[i] = ((uint64_t)(uint32_t)cur << 32) | (k & ((1ull << bits) - 1));
    }
    for (int q = prev + 1; q <= cur && q <= nPar; q++) start[q] = (int32_t)i;
}
__global__ void k_mark_orphans(DevContacts C, const uint64_t* __restrict__ nk, const int32_t* __restrict__ newLo,
                               int32_t* __restrict__ orph, const uint8_t* __restrict__ fresh) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= C.n) return;
    int32_t o = 0;
    if ((C.flags[j] & C_REAL) && !freshPair(fresh, C.key[j])) o = findInRange(nk, newLo, C.key[j]) < 0 ? 1 : 0;
    orph[j] = o;
}
__global__ void k_compact_orphans(DevContacts C, const int32_t* __restrict__ orphFlag, const int32_t* __restrict__ orphScan,
                                  uint64_t* __restrict__ okey, int32_t* __restrict__ osrc) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= C.n) return;
    if (orphFlag[j]) {
        const int32_t o = orphScan[j];
        okey[o] = C.key[j];
        osrc[o] = (int32_t)j;
    }
}
// The place of every new pair in the merged set and the old contact it continues. tot (null: not
// wanted): the real contacts of the old set, and those of them among the new pairs; where the two differ
// some real contact lost its overlap.
__global__ void k_place_new(const uint64_t* __restrict__ nk, int64_t nn, const uint64_t* __restrict__ okey, int64_t no, DevContacts Cold,
                            const int32_t* __restrict__ oldLo, uint64_t* __restrict__ outKey, int32_t* __restrict__ src,
                            const int32_t* __restrict__ nkCd, int32_t* __restrict__ outCd, const uint8_t* __restrict__ fresh,
                            CollideTotals* __restrict__ tot) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool real = false, kept = false;
    if (i < nn) {
        const uint64_t k = nk[i];
        const int64_t out = i + (no > 0 ? lowerBound64(okey, no, k) : 0);
        int64_t pos = Cold.n > 0 ? findInRange(Cold.key, oldLo, k) : -1;
        if (pos >= 0 && freshPair(fresh, k)) pos = -1;
        kept = tot && pos >= 0 && (Cold.flags[pos] & C_REAL);
        outKey[out] = k;
        src[out] = (int32_t)pos;
        if (nkCd) outCd[out] = nkCd[i];
    }
    if (!tot) return;
    if (i < Cold.n) real = (Cold.flags[i] & C_REAL) && !freshPair(fresh, Cold.key[i]);
    const int a = __syncthreads_count(real), b = __syncthreads_count(kept);
    if (threadIdx.x == 0) {
        if (a) atomicAdd(&tot->real, (unsigned long long)a);
        if (b) atomicAdd(&tot->kept, (unsigned long long)b);
    }
}
__global__ void k_place_orph(const uint64_t* __restrict__ nk, int64_t nn, const uint64_t* __restrict__ okey,
                             const int32_t* __restrict__ osrc, int64_t no, uint64_t* __restrict__ outKey, int32_t* __restrict__ src) {
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= no) return;
    const uint64_t k = okey[o];
    const int64_t out = o + lowerBound64(nk, nn, k);
    outKey[out] = k;
    src[out] = osrc[o];
}
// Dormant contacts. Between two full runs no node moves farther than verletDist from the position
// it had at the first of them (the verlet test of Leapfrog triggers the next full run before that),
// so a pair that is not real and whose surfaces are more than 2*verletDist apart now cannot touch
// before the next full run: the geometry functor would reject it at every step until then. Such
// contacts stay in the container (they are potential contacts of the reference) but the contact
// kernels skip them. The bounds are taken with a relative margin of 1e-9, and only for aperiodic
// scenes (a periodic cell moves the images of the particles by itself).
// The FP64 tests of dormantPair (sphere-sphere without mirrors, wall-sphere, facet-sphere), out of
// line: inlined, they become predicated FP64 instructions in the warps of mirror-tested pairs.
__device__ __noinline__ bool dormantFarFP64(const DevNodes& N, const DevParticles& P, const ScenePar* __restrict__ spp, int scene,
                                            uint32_t ty, int A, int B) {
    const ScenePar& sp = spp[scene];
    const double m2 = 2 * sp.verletDist;
    bool far;
    const double4_32a pb = N.posr[B];
    if (ty == CT_SS) {
        const double4_32a pa = N.posr[A];
        const double dx = pb.x - pa.x, dy = pb.y - pa.y, dz = pb.z - pa.z;
        const double reach = (fabs(sp.ssDistFactor) * (pa.w + pb.w) + m2) * (1 + 1e-9);
        far = dx * dx + dy * dy + dz * dz > reach * reach;
    } else if (ty == CT_WS) {
        const int4 ax = P.aux[A];
        const double4_32a pw = N.posr[A];
        const double d = (ax.x == 0 ? pb.x - pw.x : (ax.x == 1 ? pb.y - pw.y : pb.z - pw.z));
        far = fabs(d) > (pb.w + m2) * (1 + 1e-9);
    } else {
        // distance from the sphere centre to the triangle: to its plane when the projection falls
        // inside, else to the nearest edge; it bounds from below the distance the functor tests
        // (Facet.cpp:247-259), and every point of the triangle moves at most verletDist since its
        // vertices do
        const int4 nd = P.aux[A];
        const D3 p0 = ld3(N.posr[nd.x]), p1 = ld3(N.posr[nd.y]), p2 = ld3(N.posr[nd.z]);
        const D3 sC = ld3(pb);
        const D3 nn = cross(p1 - p0, p2 - p0);
        const double nl = sqrt(sqn(nn));
        far = false;
        if (nl > 0) {
            const D3 fN = nn / nl;
            const double planeDist = dot(sC - p0, fN);
            const D3 fC = sC - planeDist * fN;
            const bool inside = dot(cross(p1 - p0, nn), fC - p0) <= 0 && dot(cross(p2 - p1, nn), fC - p1) <= 0 &&
                                dot(cross(p0 - p2, nn), fC - p2) <= 0;
            double d2;
            if (inside) d2 = planeDist * planeDist;
            else {
                d2 = sqn(sC - closestSegmentPt(sC, p0, p1));
                d2 = fmin(d2, sqn(sC - closestSegmentPt(sC, p1, p2)));
                d2 = fmin(d2, sqn(sC - closestSegmentPt(sC, p2, p0)));
            }
            const double reach = (pb.w + P.facet[A].w + m2) * (1 + 1e-9);
            far = d2 > reach * reach;
        }
    }
    return far;
}
// whether contact k (flags fl, not real) is dormant
__device__ __forceinline__ bool dormantPair(const DevNodes& N, const DevParticles& P, const ScenePar* __restrict__ spp, uint64_t k, uint32_t fl) {
    const uint32_t ty = ctype(fl);
    if (ty == CT_NONE) return false;
    const int lo = (int)(k >> 32), hi = (int)(k & 0xffffffffu);
    const int A = (fl & C_SWAP) ? hi : lo, B = (fl & C_SWAP) ? lo : hi;
    const int scene = sceneOfP(P, B);
    if (!(ty == CT_SS && N.mir)) return dormantFarFP64(N, P, spp, scene, ty, A, B);
    // FP32-force mode: the double-float mirrors of the positions, FP32 arithmetic; the
    // relative position carries ~47 bits and the squares and sums ~2^-22 relative error
    const ScenePar& sp = spp[scene];
    const float4 ha = N.mir[A].ph, la = N.mir[A].pl, hb = N.mir[B].ph, lb = N.mir[B].pl;
    float sx, tx, sy, ty_, sz, tz;
    dfDiff(ha.x, la.x, hb.x, lb.x, sx, tx);
    dfDiff(ha.y, la.y, hb.y, lb.y, sy, ty_);
    dfDiff(ha.z, la.z, hb.z, lb.z, sz, tz);
    const float dx = sx + tx, dy = sy + ty_, dz = sz + tz;
    const float reach = (sp.ssDfAbsF * (ha.w + hb.w) + sp.reach2F) * (1.f + 1e-5f);
    return dx * dx + dy * dy + dz * dz > reach * reach;
}

// carry persistent state of surviving contacts; new contacts get their functor type and orientation
// (CGeomDispatcher functor order: Facet/Wall first, ContactLoop.cpp:145-152); in an aperiodic scene those
// that are not real are marked dormant where they are. packedState: the state of sphere-sphere contacts
// goes from the old packed state to the new one (k_pack_ss)
__global__ void k_gather(DevContacts Cold, DevContacts Cnew, const int32_t* __restrict__ src, DevNodes N, DevParticles P,
                         const ScenePar* __restrict__ spp, const long long* __restrict__ dStep, const int32_t* __restrict__ newCd,
                         int peri, int packedState) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Cnew.n) return;
    const int32_t s0 = src[i];
    const uint64_t k = Cnew.key[i];
    const uint32_t fo = s0 >= 0 ? Cold.flags[s0] : (uint32_t)C_REMOVED;
    // a contact removed since the last full run comes back as a new one
    const int32_t s = (fo & C_REMOVED) ? -1 : s0;
    // FP32-force mode carries the state of real contacts only (a contact that is not real has no
    // state any kernel reads; the listing reports zeros for it)
    const bool fp32 = Cnew.fcol[0] != nullptr;
    uint32_t fl = 0;
    if (s >= 0) {
        fl = fo & ~(C_PENDING | C_DORMANT);
        Cnew.step0[i] = Cold.step0[s];
        Cnew.cdist[i] = Cold.cdist[s];
        if (!fp32 || ((fo & C_REAL) && !(packedState && ctype(fo) == CT_SS))) {
#pragma unroll
            for (int q = 0; q < CC_NCOL; q++)
                if (Cnew.col[q]) Cnew.col[q][i] = Cold.col[q][s];
#pragma unroll
            for (int q = 0; q < CF_NCOL; q++)
                if (Cnew.fcol[q]) Cnew.fcol[q][i] = Cold.fcol[q][s];
        }
    } else {
        const int lo = (int)(k >> 32), hi = (int)(k & 0xffffffffu);
        const int tl = P.shape[lo], th = P.shape[hi];
        uint32_t ty = CT_NONE;
        const int a = (tl == WG_SHAPE_SPHERE) ? th : tl;
        const bool sphLo = (tl == WG_SHAPE_SPHERE), sphHi = (th == WG_SHAPE_SPHERE);
        if (sphLo && sphHi) ty = CT_SS;
        else if (sphLo || sphHi) {
            if (a == WG_SHAPE_FACET) ty = CT_FS;
            else if (a == WG_SHAPE_WALL) ty = CT_WS;
            if (sphLo) fl |= C_SWAP;  // the non-sphere (hi) becomes pA
        }
        fl |= ty << 2;
        Cnew.step0[i] = (int32_t)(*dStep);
        Cnew.cdist[i] = newCd ? newCd[i] : packCellDist(0, 0, 0);
        if (!fp32) {
#pragma unroll
            for (int q = 0; q < CC_NCOL; q++)
                if (Cnew.col[q]) Cnew.col[q][i] = 0.;
        }
    }
    if (!peri && !(fl & C_REAL) && dormantPair(N, P, spp, k, fl)) fl |= C_DORMANT;
    Cnew.flags[i] = fl;
}

// ---------------------------------------------------------------- CSR incidence
// Only active contacts (a functor applies and the pair is not dormant) own end slots.
__device__ __forceinline__ bool activeContact(uint32_t fl) { return ctype(fl) != CT_NONE && !(fl & C_DORMANT); }
// a plain contact joins two spheres of the same period
__device__ __forceinline__ bool plainContact(uint32_t fl, int32_t cd) { return ctype(fl) == CT_SS && cd == packCellDist(0, 0, 0); }
// What one contact adds to the running counts that place the active contacts in the work list: 1 in
// the low half, and 1 in the high half if it is plain; with `real`, real contacts alone.
struct WorkClass {
    const uint32_t* flags;
    const int32_t* cdist;
    int64_t n;
    uint32_t real;
    __device__ __forceinline__ uint64_t operator()(int64_t c) const {
        if (c >= n) return 0;
        const uint32_t fl = flags[c];
        if (!activeContact(fl) || (fl & real) != real) return 0;
        return 1ull | (plainContact(fl, cdist[c]) ? 1ull << 32 : 0ull);
    }
};
// loStart[p] = active contacts with lo < p; first[p]: the first contact with a lo id of p or more
__global__ void k_lo_start(const int32_t* __restrict__ first, int nPar, const uint64_t* __restrict__ act, int32_t* __restrict__ loStart) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p <= nPar) loStart[p] = (int32_t)(uint32_t)act[first[p]];
}
// hi id of the active contacts, nPar for the others (sorted past every particle)
__global__ void k_hi_keys(const uint64_t* __restrict__ key, const uint32_t* __restrict__ flags, int64_t n, uint32_t nPar,
                          uint32_t* __restrict__ hk, int32_t* __restrict__ hv) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    hk[c] = activeContact(flags[c]) ? (uint32_t)(key[c] & 0xffffffffu) : nPar;
    hv[c] = (int32_t)c;
}
__global__ void k_hi_start(const uint32_t* __restrict__ hks, int64_t n, int nPar, int32_t* __restrict__ hiStart) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > nPar) return;
    hiStart[p] = (int32_t)lowerBound32(hks, n, (uint32_t)p);
}
__device__ __forceinline__ void clearEnd(const DevIncidence& I, int64_t e) {
    if (I.endA) {
        I.endA[e] = make_double4_32a(0., 0., 0., 0.);
        I.endB[e] = make_double2(0., 0.);
    } else {
        I.endAf[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        I.endBf[e] = make_float2(0.f, 0.f);
    }
}
// Room that a run has before the host knows what the new set needs: for so many active contacts and plain ones
// (act < 0: nothing is to be cleared). tot: the real contacts are counted, and none must be missing.
struct Room {
    int64_t act = -1, plain = -1;
    const CollideTotals* tot = nullptr;
    // whether the set whose active contacts and plain ones are counted in act (low and high half) is the new one
    __device__ __forceinline__ bool suffices(uint64_t n) const {
        return (int64_t)(uint32_t)n <= act && (int64_t)(n >> 32) <= plain && !(tot && tot->real != tot->kept);
    }
};
// Up to so many contacts the kernel that gives out the slots clears the ends (a launch less: 10 000 spheres 245 -> 238 us
// a run); beyond, a kernel of its own does, which writes them in order (1M drum: 76 us for both, 121 in one).
constexpr int64_t kClearInSlots = 1 << 19;
// end slots: active contact c with hi==p sits at loStart[p] + (its index k in hiList); with lo==p
// at hiStart[p+1] + (active contacts before c) (see DevIncidence); inactive contacts have no slot (-1).
// The work list holds the nOther active contacts that are not plain (walls, facets, spheres of
// different periods) and then the plain ones, each group in ascending contact order. In the FP64 mode
// (actReal) the real contacts of a group come before its others: a warp of the contact kernel then tests contacts
// of one kind, and most that are real pass it by. Before the kernel sorted what is left to do (contactsOfBlock),
// this order alone took the contact loop of a drum of 250 000 from 0.70 to 0.49 ms a step; with both it takes
// 0.46. A periodic scene in the FP32-force mode, whose contacts are gathered from the contact arrays either
// way, has it too (200 000: 0.12 -> 0.11 ms). The packed FP32 kernel is bound by the gathered mirror
// records, which neighbours in contact order share: there the real ones come first within tiles of
// contacts only (k_pack_ss; 1M drum: split over the whole list, the step took 0.168 ms instead of 0.161).
// The ends start without a contribution, once nothing can call the old set back.
template <bool CLEAR>
__global__ void k_slots(const uint64_t* __restrict__ key, const uint32_t* __restrict__ flags, const int32_t* __restrict__ cdist, int64_t n,
                        const uint64_t* __restrict__ act, const uint64_t* __restrict__ actReal, DevIncidence I, Room room) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint64_t tot = act[n], totReal = actReal ? actReal[n] : 0;  // over all contacts
    const int nAct = (int)(uint32_t)tot, nPlain = (int)(tot >> 32);
    const bool clear = CLEAR && room.suffices(tot);
    if (k < nAct) {
        const int32_t ch = I.hiList[k];
        const int hiP = (int)(key[ch] & 0xffffffffu);
        const int32_t slot = I.loStart[hiP] + (int32_t)k;
        I.slotHi[ch] = slot;
        if (clear) clearEnd(I, slot);
    }
    const uint32_t fl = flags[k];
    if (activeContact(fl)) {
        const uint64_t a = act[k];
        const int all = (int)(uint32_t)a, plain = (int)(a >> 32);
        const int loP = (int)(key[k] >> 32), hiP = (int)(key[k] & 0xffffffffu);
        const int32_t slot = I.hiStart[loP + 1] + all;
        I.slotLo[k] = slot;
        if (clear) clearEnd(I, slot);
        const bool isPlain = plainContact(fl, cdist[k]);
        int w = isPlain ? plain : all - plain;  // place within the group
        if (actReal) {
            const uint64_t r = actReal[k];
            const int rAll = (int)(uint32_t)r, rPlain = (int)(r >> 32);
            const int before = isPlain ? rPlain : rAll - rPlain;  // real ones of the group before this contact
            const int real = isPlain ? (int)(totReal >> 32) : (int)(uint32_t)totReal - (int)(totReal >> 32);
            w = (fl & C_REAL) ? before : real + (w - before);
        }
        if (isPlain) w += nAct - nPlain;
        I.work[w] = (fl & C_SWAP) ? make_int4((int)k, hiP, loP, (int)(fl & 0xeu)) : make_int4((int)k, loP, hiP, (int)(fl & 0xeu));
    } else {
        I.slotLo[k] = -1;
        I.slotHi[k] = -1;
    }
}

// Particles summed by the block tree; the ones whose node has a free DOF are also summed before
// every Leapfrog (the others only when the forces are reported).
__global__ void k_heavy(DevIncidence I, DevParticles P, const uint32_t* __restrict__ nodeFlags, int threshold,
                        CollideTotals* __restrict__ tot, const uint64_t* __restrict__ act, const uint64_t* __restrict__ actReal, int64_t n) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) {  // the totals of the work-list scans, for the host
        tot->act = act[n];
        tot->actReal = actReal ? actReal[n] : 0;
    }
    if (p >= P.n) return;
    if (P.shape[p] == WG_SHAPE_FACET) return;
    const int d = (I.hiStart[p + 1] - I.hiStart[p]) + (I.loStart[p + 1] - I.loStart[p]);
    if (d > threshold) {
        const int q = atomicAdd(&tot->heavy, 1);
        I.heavy[q] = p;
        if ((nodeFlags[p] & F_DOF_ALL) != F_DOF_ALL) I.heavyFree[atomicAdd(&tot->heavyFree, 1)] = p;
    }
}
// every end of the active contacts (counted in the low half of *act) starts without a contribution
__global__ void k_zero_ends(DevIncidence I, const uint64_t* __restrict__ act, Room room) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < 2 * (int64_t)(uint32_t)*act && room.suffices(*act)) clearEnd(I, e);
}

// the packed state K back into the contact arrays of its set, contact c from idx[c] (whatever the work list holds)
__global__ void k_unpack_set(DevContacts C, DevPackedSS K, const int32_t* __restrict__ idx, int copyFt) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C.n) return;
    const uint32_t fl = C.flags[c];
    if (!activeContact(fl) || !plainContact(fl, C.cdist[c])) return;
    const int64_t j = idx[c];
    C.flags[c] = K.flags[j] & 0xffu;
#pragma unroll
    for (int q = 0; q < CF_NCOL; q++) C.fcol[q][c] = K.col[q][j];
    if (copyFt) {
        C.col[CC_FT1][c] = K.ft[0][j];
        C.col[CC_FT2][c] = K.ft[1][j];
    }
}

// ---------------------------------------------------------------- counting
// Contacts whose lo id is in [p0, p1): out[0] those not removed, out[1] the real ones. packed: the plain
// active contacts have their flags in the packed state and are counted there.
__device__ __forceinline__ void addCounts(bool there, bool real, unsigned long long* __restrict__ out) {
    const int a = __syncthreads_count(there), r = __syncthreads_count(real);
    if (threadIdx.x == 0) {
        if (a) atomicAdd(out, (unsigned long long)a);
        if (r) atomicAdd(out + 1, (unsigned long long)r);
    }
}
__global__ void k_count(DevContacts C, int packed, int64_t p0, int64_t p1, unsigned long long* __restrict__ out) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t fl = C_REMOVED;
    if (c < C.n) {
        const int64_t lo = (int64_t)(C.key[c] >> 32);
        fl = C.flags[c];
        if (lo < p0 || lo >= p1 || (packed && activeContact(fl) && plainContact(fl, C.cdist[c]))) fl = C_REMOVED;
    }
    addCounts(!(fl & C_REMOVED), (fl & C_REAL) && !(fl & C_REMOVED), out);
}
__global__ void k_count_packed(DevPackedSS K, int64_t p0, int64_t p1, unsigned long long* __restrict__ out) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t fl = C_REMOVED;
    if (j < K.n) {
        const int4 it = K.item[j];
        const int lo = min(it.x, it.y);
        fl = lo >= p0 && lo < p1 ? K.flags[j] : (uint32_t)C_REMOVED;
    }
    addCounts(!(fl & C_REMOVED), (fl & C_REAL) && !(fl & C_REMOVED), out);
}
int read_grid(Sim& S, int k, Grid& g) {
    if (!S.cw || !S.cw->dGrids) return S.fail(WG_ERR_STATE, "no grid before the first full run");
    WG_CUDA_TRY(cudaSetDevice(S.device));
    WG_CUDA_TRY(cudaMemcpyAsync(&g, S.cw->dGrids + k, sizeof g, cudaMemcpyDeviceToHost, S.stream));
    WG_CUDA_TRY(cudaStreamSynchronize(S.stream));
    return 0;
}
int count_contacts(Sim& S, int64_t p0, int64_t p1, int64_t out[2]) {
    out[0] = out[1] = 0;
    if (!S.uploaded || S.C.n == 0) return 0;
    WG_CUDA_TRY(cudaSetDevice(S.device));
    if (!S.dCount) {
        S.dCount = (unsigned long long*)S.dalloc(2 * sizeof(unsigned long long));
        if (!S.dCount) return S.fail(WG_ERR_CUDA, "out of device memory (counts)");
    }
    const bool packed = S.packDirty && S.K.n > 0;
    unsigned long long h[2];
    WG_CUDA_TRY(cudaMemsetAsync(S.dCount, 0, sizeof(h), S.stream));
    k_count<<<(unsigned)((S.C.n + 255) / 256), 256, 0, S.stream>>>(S.C, packed ? 1 : 0, p0, p1, S.dCount);
    if (packed) k_count_packed<<<(unsigned)((S.K.n + 255) / 256), 256, 0, S.stream>>>(S.K, p0, p1, S.dCount);
    WG_CUDA_TRY(cudaGetLastError());
    WG_CUDA_TRY(cudaMemcpyAsync(h, S.dCount, sizeof(h), cudaMemcpyDeviceToHost, S.stream));
    WG_CUDA_TRY(cudaStreamSynchronize(S.stream));
    out[0] = (int64_t)h[0];
    out[1] = (int64_t)h[1];
    return 0;
}

// ---------------------------------------------------------------- host orchestration
// Larger arrays in place of others, all of them or none: where one cannot be had, the old ones stay.
class Larger {
    Sim& S;
    std::vector<std::pair<void*, void*>> fresh;  // where the pointer is kept, and the new array
    bool ok = true;

public:
    explicit Larger(Sim& s) : S(s) {}
    ~Larger() {
        for (auto& f : fresh) S.dfree(f.second);
    }
    template <class T>
    void add(T*& p, int64_t n) {
        void* const q = S.dalloc(sizeof(T) * n);
        ok = ok && q;
        if (q) fresh.push_back({&p, q});
    }
    bool put() {
        if (!ok) return false;
        for (auto& f : fresh) {
            void* old;
            std::memcpy(&old, f.first, sizeof old);
            std::memcpy(f.first, &f.second, sizeof old);
            S.dfree(old);
        }
        fresh.clear();
        return true;
    }
};

static int ensureCub(Sim& S, size_t bytes) {
    CollideWork& W = *S.cw;
    if (bytes <= W.cubBytes) return 0;
    Larger L(S);
    char* tmp = (char*)W.cubTmp;
    const size_t want = bytes * 3 / 2 + 1024;
    L.add(tmp, (int64_t)want);
    if (!L.put()) return S.fail(WG_ERR_CUDA, "out of device memory (collider scratch)");
    W.cubTmp = tmp;
    W.cubBytes = want;
    return 0;
}

// Scratch of one capacity whose contents need not last: given up before the larger one is asked for, all of it
// or none (cap is 0 then). False: out of device memory.
template <class... T>
static bool scratch(Sim& S, int64_t& cap, int64_t need, T*&... p) {
    if (need <= cap) return true;
    const int64_t want = std::max<int64_t>(need, cap * 3 / 2 + 1024);
    ((S.dfree(p), p = nullptr), ...);
    ((p = (T*)S.dalloc(sizeof(T) * want)), ...);
    cap = want;
    if ((... && (p != nullptr))) return true;
    ((S.dfree(p), p = nullptr), ...);
    cap = 0;
    return false;
}

static int buildLists(Sim& S) {
    CollideWork& W = *S.cw;
    std::vector<int32_t> sph, large, glob;
    for (int64_t p = 0; p < S.nPar; p++) {
        if (!S.hParked.empty() && S.hParked[p]) continue;  // empty part of a serving slot
        if (S.hShape[p] == WG_SHAPE_SPHERE) sph.push_back((int32_t)p);
        else if (S.hShape[p] == WG_SHAPE_WALL) glob.push_back((int32_t)p);
        else large.push_back((int32_t)p);
    }
    W.nSph = (int)sph.size();
    // per-scene sphere ranges and grid-reduction chunks (particles of a batch are grouped by scene)
    const int K = S.nScenes;
    W.hSceneSph.assign(K + 1, 0);
    for (int32_t p : sph) W.hSceneSph[(S.hSceneOfPar.empty() ? 0 : S.hSceneOfPar[p]) + 1]++;
    for (int k = 0; k < K; k++) W.hSceneSph[k + 1] += W.hSceneSph[k];
    W.chunksDirty = true;
    W.hChunk.assign(1, 0);
    W.hSceneChunk.assign(1, 0);
    const int64_t CH = kGridChunk;
    for (int k = 0; k < K; k++) {
        for (int64_t b = W.hSceneSph[k]; b < W.hSceneSph[k + 1]; b += CH) W.hChunk.push_back((int32_t)std::min(b + CH, W.hSceneSph[k + 1]));
        W.hSceneChunk.push_back((int32_t)W.hChunk.size() - 1);
    }
    W.hLarge = large;
    W.hGlobal = glob;
    // capacity for every particle: the lists are rebuilt when serving slots change
    if (!W.sphereIds) {
        Larger L(S);
        L.add(W.sphereIds, S.nPar);
        L.add(W.largeIds, S.nPar);
        L.add(W.globalIds, S.nPar);
        L.add(W.gStart, S.nScenes + 1);
        if (!L.put()) return S.fail(WG_ERR_CUDA, "out of device memory");
    }
    W.nLarge = W.nGlobal = 0;
    if (!sph.empty()) WG_CUDA_TRY(cudaMemcpyAsync(W.sphereIds, sph.data(), sizeof(int32_t) * sph.size(), cudaMemcpyHostToDevice, S.stream));
    // non-sphere pairs are possible only if some pair of them shares a mask bit outside loneMask
    bool ll = false;
    std::vector<int32_t> nonSph(large);
    nonSph.insert(nonSph.end(), glob.begin(), glob.end());
    {
        uint32_t seen = 0;  // OR of masks
        // exact test on distinct mask values
        std::vector<uint32_t> masks;
        for (int32_t p : nonSph) masks.push_back(S.hMask[p]);
        std::sort(masks.begin(), masks.end());
        masks.erase(std::unique(masks.begin(), masks.end()), masks.end());
        for (size_t a = 0; a < masks.size() && !ll; a++)
            for (size_t b = a; b < masks.size() && !ll; b++)
                if ((masks[a] & masks[b]) != 0 && (masks[a] & masks[b] & S.cfg.lone_mask) == 0) ll = true;
        (void)seen;
    }
    W.largeLargePossible = ll && nonSph.size() > 1;
    return 0;
}

// ---------------------------------------------------------------- the second half of a run, over a set of n contacts
static int hiKeyBits(const Sim& S) {  // bits of the largest hi key, nPar
    int bits = 1;
    while ((int64_t(1) << bits) <= S.nPar) bits++;
    return bits;
}
// Room for the incidence of n contacts; the arrays in use stay until all of the larger ones are there.
static int incidenceRoom(Sim& S, int64_t n) {
    CollideWork& W = *S.cw;
    const bool realFirst = S.prec == WG_PREC_FP64 || S.cfg.periodic;  // see k_slots
    if (W.hiCap < std::max<int64_t>(n, 1)) {
        const int64_t cap = std::max<int64_t>(n, 1) * 3 / 2 + 1024;
        Larger L(S);
        L.add(W.hiKeys, cap);
        L.add(W.hiKeysSorted, cap);
        L.add(W.hiVals, cap);
        L.add(S.I.hiList, cap);
        L.add(S.I.slotLo, cap);
        L.add(S.I.slotHi, cap);
        L.add(W.act, cap + 1);
        if (realFirst) L.add(W.actReal, cap + 1);
        L.add(S.I.work, cap);
        if (!L.put()) return S.fail(WG_ERR_CUDA, "out of device memory (incidence)");
        W.hiCap = cap;
    }
    size_t a = 0, b = 0;
    const auto in = thrust::make_transform_iterator(thrust::counting_iterator<int64_t>(0), WorkClass{S.C.flags, S.C.cdist, n, 0});
    cub::DeviceScan::ExclusiveSum(nullptr, a, in, W.act, (int)(n + 1), S.stream);
    if (n > 0) cub::DeviceRadixSort::SortPairs(nullptr, b, W.hiKeys, W.hiKeysSorted, W.hiVals, S.I.hiList, n, 0, hiKeyBits(S), S.stream);
    return ensureCub(S, std::max(a, b));
}
// CSR incidence and work list of the n contacts of S.C; first: the first contact of every lo id. The room is there.
// The host does not know the number of active contacts before the end; the ends are cleared as far as room says.
static int incidence(Sim& S, int64_t n, const int32_t* first, const Room& room) {
    CollideWork& W = *S.cw;
    cudaStream_t st = S.stream;
    const unsigned gn = (unsigned)((n + BS - 1) / BS);
    auto scan = [&](uint32_t real, uint64_t* out) -> int {
        const auto in = thrust::make_transform_iterator(thrust::counting_iterator<int64_t>(0), WorkClass{S.C.flags, S.C.cdist, n, real});
        size_t tb = W.cubBytes;
        WG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(W.cubTmp, tb, in, out, (int)(n + 1), st));
        return 0;
    };
    int r = scan(0, W.act);
    if (!r && W.actReal) r = scan(C_REAL, W.actReal);
    if (r) return r;
    k_lo_start<<<(unsigned)((S.nPar + 1 + BS - 1) / BS), BS, 0, st>>>(first, (int)S.nPar, W.act, S.I.loStart);
    if (n > 0) {
        k_hi_keys<<<gn, BS, 0, st>>>(S.C.key, S.C.flags, n, (uint32_t)S.nPar, W.hiKeys, W.hiVals);
        size_t tb = W.cubBytes;
        WG_CUDA_TRY(cub::DeviceRadixSort::SortPairs(W.cubTmp, tb, W.hiKeys, W.hiKeysSorted, W.hiVals, S.I.hiList, n, 0, hiKeyBits(S), st));
    }
    k_hi_start<<<(unsigned)((S.nPar + 1 + BS - 1) / BS), BS, 0, st>>>(W.hiKeysSorted, n, (int)S.nPar, S.I.hiStart);
    if (n > 0 && room.act >= 0) k_slots<true><<<gn, BS, 0, st>>>(S.C.key, S.C.flags, S.C.cdist, n, W.act, W.actReal, S.I, room);
    else if (n > 0) k_slots<false><<<gn, BS, 0, st>>>(S.C.key, S.C.flags, S.C.cdist, n, W.act, W.actReal, S.I, room);
    k_heavy<<<(unsigned)((S.nPar + BS - 1) / BS), BS, 0, st>>>(S.I, S.P, S.N.flags, kHeavyThreshold, W.tot, W.act, W.actReal, n);
    return 0;
}
// Room for the ends of nAct contacts; the old ends stay until the new ones are there.
static int endRoom(Sim& S, int64_t nAct) {
    if (S.I.endCap >= 2 * std::max<int64_t>(nAct, 1)) return 0;
    const int64_t cap = 2 * std::max<int64_t>(nAct, 1) * 5 / 4 + 2048;
    Larger L(S);
    if (S.prec == WG_PREC_FP32) {
        L.add(S.I.endAf, cap);
        L.add(S.I.endBf, cap);
    } else {
        L.add(S.I.endA, cap);
        L.add(S.I.endB, cap);
    }
    if (!L.put()) return S.fail(WG_ERR_CUDA, "out of device memory (contact ends)");
    S.I.endCap = cap;
    return 0;
}
// Room in Q, whose contents need not last, for n packed contacts, in one block of memory. ft: with the IdealElPl
// shear force.
static int packRoom(Sim& S, DevPackedSS& Q, int64_t n, bool ft) {
    if (Q.cap >= n && (Q.ft[0] || !ft)) return 0;
    S.dfree(Q.item);
    Q = DevPackedSS{};
    const int64_t cap = (n * 5 / 4 + 4096) / 64 * 64;  // every column is aligned
    char* p = (char*)S.dalloc((size_t)cap * (sizeof(int4) + (ft ? 2 * sizeof(double) : 0) + sizeof(uint32_t) + CF_NCOL * sizeof(float)));
    if (!p) return S.fail(WG_ERR_CUDA, "out of device memory (packed contacts)");
    auto take = [&](size_t bytes) {
        void* const at = p;
        p += bytes * cap;
        return at;
    };
    Q.item = (int4*)take(sizeof(int4));
    for (int q = 0; ft && q < 2; q++) Q.ft[q] = (double*)take(sizeof(double));
    Q.flags = (uint32_t*)take(sizeof(uint32_t));
    for (int q = 0; q < CF_NCOL; q++) Q.col[q] = (float*)take(sizeof(float));
    Q.cap = cap;
    return 0;
}

// A run that ends early after room for the incidence of the new set was made: the old set, from its keys and flags, takes
// its incidence and work list again (the ends and the packed state are still those of the old set).
struct Undo {
    Sim& S;
    const bool packedState;
    bool swapped = false, incidence = false, off = false;
    Undo(Sim& s, bool p) : S(s), packedState(p) {}
    void swap() {
        std::swap(S.C, S.Cb);
        swapped = !swapped;
    }
    ~Undo() {
        if (off) return;
        if (swapped) swap();
        if (!incidence) return;
        const std::string why = S.err;  // what the run failed for
        if (restore()) S.K.n = 0;       // the device is gone
        S.err = why;
    }
    int restore() {
        CollideWork& W = *S.cw;
        const int64_t n = S.C.n;
        if (S.contactsReplaced) {  // set from outside and never run: it has no forces to list
            if (!W.hiCap) return 0;
            WG_CUDA_TRY(cudaMemsetAsync(S.I.slotLo, 0xff, sizeof(int32_t) * W.hiCap, S.stream));
            WG_CUDA_TRY(cudaMemsetAsync(S.I.slotHi, 0xff, sizeof(int32_t) * W.hiCap, S.stream));
            return 0;
        }
        if (packedState && n > 0) k_unpack_set<<<(unsigned)((n + BS - 1) / BS), BS, 0, S.stream>>>(S.C, S.K, W.packIdx, S.K.ftLive ? 1 : 0);
        k_lo_bounds<<<(unsigned)((n + 1 + BS - 1) / BS), BS, 0, S.stream>>>(S.C.key, n, (int)S.nPar, W.oldLo);
        WG_CUDA_TRY(cudaMemsetAsync(&W.tot->heavy, 0, 2 * sizeof(int32_t), S.stream));
        int r = incidenceRoom(S, n);
        if (!r) r = wg::incidence(S, n, W.oldLo, Room{});
        if (r) return r;
        launch_pack_ss(S.stream, S.C, S.I, S.P, S.K, S.K, nullptr, nullptr, W.packIdx, W.act + n, S.K.n);
        S.packDirty = false;
        WG_CUDA_TRY(cudaGetLastError());
        return 0;
    }
};

static int fullRun(Sim& S) {
    cudaStream_t st = S.stream;
    if (!S.cw) {
        S.cw = new CollideWork();
        S.listsDirty = true;
    }
    if (S.listsDirty) {
        int r = buildLists(S);
        if (r) return r;
        S.listsDirty = false;
    }
    CollideWork& W = *S.cw;
    // The packed sphere-sphere state goes from the old set to the new one; the contact arrays take back its
    // flags alone. Until the new set is in place the packed state stays that of the old one.
    const bool packed = S.prec == WG_PREC_FP32 && !S.cfg.periodic;
    const bool packedState = S.K.n > 0;  // none where the contact arrays were set from outside
    if (packedState && S.packDirty) launch_unpack_ss(st, S.C, S.I, S.K, S.nMixed, true);
    const uint32_t lone = S.cfg.lone_mask;
    if (S.cfg.periodic && S.hPar.hasShear && !W.hGlobal.empty())
        return S.fail(WG_ERR_UNSUPPORTED, "Walls not supported in skewed (Scene.cell.trsf is not diagonal) periodic boundary conditions.");
    // 1. boxes
    if (S.nPar > 0) k_aabb<<<(unsigned)((S.nPar + BS - 1) / BS), BS, 0, st>>>(S.N, S.P, S.dPar, S.dFlags + 1);
    // lastPos for node slots not owned by a particle box computation (dummy slots) stays stale:
    // they never move (blocked, zero velocity) and are never tested against a stale reference.
    // 2. grid over spheres, one per scene of a batch (keys of scene k start at its grid's base). The grids
    // are made on the device, so that the host need not wait for the bounds; it knows how many cells there
    // can be.
    const int K = S.nScenes;
    const int ns = W.nSph;
    const bool peri = S.cfg.periodic != 0;
    if (!W.hTot) WG_CUDA_TRY(cudaMallocHost(&W.hTot, sizeof(CollideTotals)));
    if (!W.tot && !(W.tot = (CollideTotals*)S.dalloc(sizeof(CollideTotals)))) return S.fail(WG_ERR_CUDA, "out of device memory (counts)");
    WG_CUDA_TRY(cudaMemsetAsync(W.tot, 0, sizeof(CollideTotals), st));
    int* const bad = &W.tot->bad;
    if (ns > 0) {
        const int nb = (int)W.hChunk.size() - 1;
        if (!W.dGrids) {
            // capacity for the most chunks the particles can form (one per scene plus the full ones)
            const int cap = (int)(S.nPar / kGridChunk + S.nScenes + 2);
            const int64_t sph = S.nPar;  // every particle could be an active sphere
            Larger L(S);
            L.add(W.red, 7 * (int64_t)cap);
            L.add(W.dChunk, cap + 1);
            L.add(W.dSceneChunk, K + 1);
            L.add(W.dGrids, K);
            L.add(W.cellKey, sph);
            L.add(W.cellRank, sph);
            L.add(W.skey, sph);
            if (peri) L.add(W.speri, sph);
            else {
                L.add(W.smnf, sph);
                L.add(W.smxf, sph);
            }
            if (!L.put()) return S.fail(WG_ERR_CUDA, "out of device memory (grid)");
        }
        if (W.chunksDirty) {
            WG_CUDA_TRY(cudaMemcpyAsync(W.dChunk, W.hChunk.data(), sizeof(int32_t) * (nb + 1), cudaMemcpyHostToDevice, st));
            WG_CUDA_TRY(cudaMemcpyAsync(W.dSceneChunk, W.hSceneChunk.data(), sizeof(int32_t) * (K + 1), cudaMemcpyHostToDevice, st));
            W.chunksDirty = false;
        }
        int64_t ncell = 0;
        for (int k = 0; k < K; k++) ncell += cellBound(W.hSceneSph[k + 1] - W.hSceneSph[k], K);
        if (ncell >= (int64_t(1) << 31) - 2) return S.fail(WG_ERR_CAPACITY, "too many broad-phase cells in the batch");
        if (!scratch(S, W.cellOffCap, ncell + 1, W.cellOff)) return S.fail(WG_ERR_CUDA, "out of device memory (grid)");
        const unsigned gs = (unsigned)((ns + BS - 1) / BS);
        k_grid_reduce<<<nb, BS, 0, st>>>(S.P, W.sphereIds, W.dChunk, W.red);
        k_make_grids<<<1, K == 1 ? 1024 : 32 * std::min(K, 32), 0, st>>>(K, W.dChunk, W.dSceneChunk, W.red, S.dPar, peri ? 1 : 0, W.dGrids, W.tot);
        // spheres in cell order: their number per cell, its running sum, then each to its place
        WG_CUDA_TRY(cudaMemsetAsync(W.cellOff, 0, sizeof(int32_t) * (ncell + 1), st));
        if (peri) k_cellkey_peri<<<gs, BS, 0, st>>>(S.P, W.sphereIds, ns, W.dGrids, S.dPar, W.cellKey, W.cellRank, W.cellOff);
        else k_cellkey<<<gs, BS, 0, st>>>(S.P, W.sphereIds, ns, W.dGrids, W.cellKey, W.cellRank, W.cellOff);
        size_t tb = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb, W.cellOff, W.cellOff, (int)(ncell + 1), st);
        if (ensureCub(S, tb)) return WG_ERR_CUDA;
        tb = W.cubBytes;
        WG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(W.cubTmp, tb, W.cellOff, W.cellOff, (int)(ncell + 1), st));
        if (peri) k_gather_peri<<<gs, BS, 0, st>>>(S.P, W.sphereIds, ns, W.cellKey, W.cellRank, W.cellOff, S.dPar, W.skey, W.speri);
        else k_gather_sorted<<<gs, BS, 0, st>>>(S.P, W.sphereIds, ns, W.dGrids, &W.tot->far, W.cellKey, W.cellRank, W.cellOff, W.skey, W.smnf, W.smxf);
    }
    // lists of large particles: facets with boxes spanning a few cells use the grid, the rest are global
    {
        // decide on the host from the facet sizes measured at the previous full run would need a copy;
        // facet boxes are static in the supported scenes, so classify them once by size here
        if (W.nLarge == 0 && W.nGlobal == 0 && (!W.hLarge.empty() || !W.hGlobal.empty())) {
            std::vector<double4_32a> mn, mx;
            std::vector<Grid> hG(K, Grid{0, 0, 0, 1, 1, 1, 1, 1, 1, 0, 0});
            if (!W.hLarge.empty()) {
                mn.resize(S.nPar);
                mx.resize(S.nPar);
                WG_CUDA_TRY(cudaMemcpyAsync(mn.data(), S.P.mn, sizeof(double4_32a) * S.nPar, cudaMemcpyDeviceToHost, st));
                WG_CUDA_TRY(cudaMemcpyAsync(mx.data(), S.P.mx, sizeof(double4_32a) * S.nPar, cudaMemcpyDeviceToHost, st));
                if (ns > 0) WG_CUDA_TRY(cudaMemcpyAsync(hG.data(), W.dGrids, sizeof(Grid) * K, cudaMemcpyDeviceToHost, st));
                WG_CUDA_TRY(cudaStreamSynchronize(st));
            }
            std::vector<int32_t> loc, glo = W.hGlobal;
            for (int32_t p : W.hLarge) {
                double e = std::max({mx[p].x - mn[p].x, mx[p].y - mn[p].y, mx[p].z - mn[p].z});
                const double hk = hG[S.hSceneOfPar.empty() ? 0 : S.hSceneOfPar[p]].h;
                if (ns > 0 && std::isfinite(e) && e <= 8 * hk) loc.push_back(p);
                else glo.push_back(p);
            }
            std::sort(glo.begin(), glo.end());  // grouped by scene (particles of a batch are)
            W.nLarge = (int)loc.size();
            W.nGlobal = (int)glo.size();
            if (W.nLarge) WG_CUDA_TRY(cudaMemcpyAsync(W.largeIds, loc.data(), sizeof(int32_t) * loc.size(), cudaMemcpyHostToDevice, S.stream));
            if (W.nGlobal) WG_CUDA_TRY(cudaMemcpyAsync(W.globalIds, glo.data(), sizeof(int32_t) * glo.size(), cudaMemcpyHostToDevice, S.stream));
            if (K > 1) {
                std::vector<int32_t> gs(K + 1, 0);
                for (int32_t p : glo) gs[S.hSceneOfPar[p] + 1]++;
                for (int k = 0; k < K; k++) gs[k + 1] += gs[k];
                WG_CUDA_TRY(cudaMemcpyAsync(W.gStart, gs.data(), sizeof(int32_t) * (K + 1), cudaMemcpyHostToDevice, S.stream));
            }
        }
    }
    // 3-4. pair generation with a capacity retry
    auto pairRoom = [&](int64_t need) {
        return peri ? scratch(S, W.pairCap, need, W.pairs, W.pairsSorted, W.pairCd, W.pairCdSorted)
                    : scratch(S, W.pairCap, need, W.pairs, W.pairsSorted);
    };
    if (!pairRoom(std::max<int64_t>(1 << 16, 8 * S.nPar))) return S.fail(WG_ERR_CUDA, "out of device memory (pairs)");
    int idBits = 1;  // bits of an id
    while ((int64_t(1) << idBits) < S.nPar) idBits++;
    unsigned long long* const counter = &W.tot->pairs;
    int64_t nNew = 0;
    for (int attempt = 0; attempt < 3; attempt++) {
        if (attempt > 0) WG_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
        if (peri) {
            if (ns > 0)
                k_pairs_ss_peri<<<(ns + 127) / 128, 128, 0, st>>>(S.P, W.skey, W.speri, ns, W.dGrids, W.cellOff, lone, idBits, bad, S.dPar,
                                                                  W.pairs, W.pairCd, W.pairCap, counter, S.dFlags + FL_ERR);
            if (ns > 0 && W.nGlobal > 0)
                k_pairs_global_peri<<<(ns + BS - 1) / BS, BS, 0, st>>>(S.P, W.globalIds, W.nGlobal, W.sphereIds, ns, lone, idBits, S.dPar,
                                                                     W.pairs, W.pairCd, W.pairCap, counter, S.dFlags + FL_ERR);
        } else if (ns > 0) {
            k_pairs_ss<<<(ns + BS - 1) / BS, BS, 0, st>>>(S.P, W.skey, W.smnf, W.smxf, ns, W.dGrids, W.cellOff, lone, idBits, bad, W.pairs,
                                                        W.pairCap, counter);
            if (W.nLarge > 0)
                k_pairs_local<<<(unsigned)(((int64_t)W.nLarge * 32 + BS - 1) / BS), BS, 0, st>>>(
                    S.P, W.largeIds, W.nLarge, W.smnf, W.smxf, W.dGrids, W.cellOff, lone, idBits, bad, W.pairs, W.pairCap, counter);
            if (W.nGlobal > 0)
                k_pairs_global<<<(ns + BS - 1) / BS, BS, 0, st>>>(S.P, W.globalIds, W.nGlobal, K > 1 ? W.gStart : nullptr, W.sphereIds, ns,
                                                                lone, idBits, W.pairs, W.pairCap, counter);
        }
        if (W.largeLargePossible && !peri) {
            // all non-spheres against each other
            int nn = W.nLarge + W.nGlobal;
            std::vector<int32_t> all;
            (void)all;
            int32_t* ids = W.globalIds;
            if (W.nLarge > 0) {
                // concatenate: globalIds has room for every non-sphere
                WG_CUDA_TRY(cudaMemcpyAsync(W.globalIds + W.nGlobal, W.largeIds, sizeof(int32_t) * W.nLarge, cudaMemcpyDeviceToDevice, st));
            }
            int64_t tot = (int64_t)nn * nn;
            k_pairs_large_large<<<(unsigned)((tot + BS - 1) / BS), BS, 0, st>>>(S.P, ids, nn, lone, idBits, W.pairs, W.pairCap, counter);
        }
        WG_CUDA_TRY(cudaMemcpyAsync(W.hTot, W.tot, sizeof(CollideTotals), cudaMemcpyDeviceToHost, st));
        WG_CUDA_TRY(cudaStreamSynchronize(st));
        if (W.hTot->bad) return S.fail(WG_ERR_NAN, "InsertionSortCollider: non-finite sphere bounding box (NaN or infinite position)");
        nNew = (int64_t)W.hTot->pairs;
        if (nNew <= W.pairCap) break;
        if (!pairRoom(nNew + nNew / 4)) return S.fail(WG_ERR_CUDA, "out of device memory (pairs)");
    }
    // sort the pairs, (lo << idBits | hi)
    if (nNew > 0) {
        size_t tb = 0;
        if (peri) cub::DeviceRadixSort::SortPairs(nullptr, tb, W.pairs, W.pairsSorted, W.pairCd, W.pairCdSorted, nNew, 0, 2 * idBits, st);
        else cub::DeviceRadixSort::SortKeys(nullptr, tb, W.pairs, W.pairsSorted, nNew, 0, 2 * idBits, st);
        if (ensureCub(S, tb)) return WG_ERR_CUDA;
        tb = W.cubBytes;
        if (peri)
            WG_CUDA_TRY(cub::DeviceRadixSort::SortPairs(W.cubTmp, tb, W.pairs, W.pairsSorted, W.pairCd, W.pairCdSorted, nNew, 0, 2 * idBits,
                                                        st));
        else WG_CUDA_TRY(cub::DeviceRadixSort::SortKeys(W.cubTmp, tb, W.pairs, W.pairsSorted, nNew, 0, 2 * idBits, st));
    }
    // 5. merge with the previous contact set. Real contacts without an overlap (a law that keeps separated
    // contacts, or no verletDist) stay: they are looked for first where they can occur, which costs a
    // scan and a wait; elsewhere the merge counts whether every real contact was among the new pairs, and is
    // done again with them if the host finds that one was not.
    const int64_t nOld = S.C.n;
    if (!scratch(S, W.newLoCap, S.nPar + 2, W.newLo) || !scratch(S, W.oldLoCap, S.nPar + 2, W.oldLo))
        return S.fail(WG_ERR_CUDA, "out of device memory (merge)");
    // W.pairs takes the sorted pairs back as contact keys
    const uint64_t* const nk = W.pairs;
    k_unpack_keys<<<(unsigned)((nNew + 1 + BS - 1) / BS), BS, 0, st>>>(W.pairsSorted, nNew, idBits, (int)S.nPar, W.pairs, W.newLo);
    if (nOld > 0 && (!W.oldLoValid || S.contactsReplaced))
        k_lo_bounds<<<(unsigned)((nOld + 1 + BS - 1) / BS), BS, 0, st>>>(S.C.key, nOld, (int)S.nPar, W.oldLo);
    bool lookForOrphans = false;
    for (int k = 0; k < K; k++) {
        const wg_config& c = K > 1 ? S.cfgs[k] : S.cfg;
        lookForOrphans = lookForOrphans || !((K > 1 ? S.hPars[k] : S.hPar).verletDist > 0) || (c.law == 0 && c.no_break);
    }
    bool law0 = S.cfg.law == 0;
    for (const wg_config& c : S.cfgs) law0 = law0 || c.law == 0;
    Undo undo(S, packedState);
    for (;;) {
        int64_t nOrph = 0;
        if (nOld > 0 && lookForOrphans) {
            if (!scratch(S, W.mergeCap, nOld * 2 + 2, W.orph)) return S.fail(WG_ERR_CUDA, "out of device memory (merge)");
            int32_t* flagsArr = W.orph;
            int32_t* scanArr = W.orph + (nOld + 1);
            k_mark_orphans<<<(unsigned)((nOld + BS - 1) / BS), BS, 0, st>>>(S.C, nk, W.newLo, flagsArr, S.P.fresh);
            size_t tb = 0;
            cub::DeviceScan::ExclusiveSum(nullptr, tb, flagsArr, scanArr, (int)nOld, st);
            if (ensureCub(S, tb)) return WG_ERR_CUDA;
            tb = W.cubBytes;
            WG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(W.cubTmp, tb, flagsArr, scanArr, (int)nOld, st));
            int32_t last[2];
            WG_CUDA_TRY(cudaMemcpyAsync(&last[0], flagsArr + nOld - 1, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
            WG_CUDA_TRY(cudaMemcpyAsync(&last[1], scanArr + nOld - 1, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
            WG_CUDA_TRY(cudaStreamSynchronize(st));
            nOrph = (int64_t)last[0] + last[1];
            if (nOrph > 0) {
                if (!scratch(S, W.orphCap, nOrph, W.orphKey, W.orphSrc)) return S.fail(WG_ERR_CUDA, "out of device memory (merge)");
                k_compact_orphans<<<(unsigned)((nOld + BS - 1) / BS), BS, 0, st>>>(S.C, flagsArr, scanArr, W.orphKey, W.orphSrc);
            }
        }
        const int64_t n = nNew + nOrph;
        int r = S.ensureContactCapacity(n);
        if (r) return r;
        if (!(peri ? scratch(S, W.srcCap, std::max<int64_t>(n, 1), W.src, W.newCd) : scratch(S, W.srcCap, std::max<int64_t>(n, 1), W.src)))
            return S.fail(WG_ERR_CUDA, "out of device memory (merge)");
        undo.incidence = true;  // the arrays that are in use may be others from here on
        r = incidenceRoom(S, n);
        if (r) return r;
        S.Cb.n = n;
        const unsigned gn = (unsigned)((n + BS - 1) / BS);
        const int64_t places = std::max<int64_t>(nNew, lookForOrphans ? 0 : nOld);
        if (places > 0)
            k_place_new<<<(unsigned)((places + BS - 1) / BS), BS, 0, st>>>(nk, nNew, W.orphKey, nOrph, S.C, W.oldLo, S.Cb.key, W.src,
                                                                          peri ? W.pairCdSorted : nullptr, W.newCd, S.P.fresh,
                                                                          lookForOrphans ? nullptr : W.tot);
        if (nOrph > 0)
            k_place_orph<<<(unsigned)((nOrph + BS - 1) / BS), BS, 0, st>>>(nk, nNew, W.orphKey, W.orphSrc, nOrph, S.Cb.key, W.src);
        if (n > 0) k_gather<<<gn, BS, 0, st>>>(S.C, S.Cb, W.src, S.N, S.P, S.dPar, S.dStep, peri ? W.newCd : nullptr, peri ? 1 : 0,
                                             packedState ? 1 : 0);
        undo.swap();
        if (nOrph > 0)  // the first index of every lo id in the merged set; without orphans that of the new pairs
            k_lo_bounds<<<(unsigned)((n + 1 + BS - 1) / BS), BS, 0, st>>>(S.C.key, n, (int)S.nPar, W.newLo);
        // 6. CSR incidence over the active contacts
        DevPackedSS& Q = W.Kb;
        auto pack = [&](int64_t most) {
            Q.ftLive = law0;
            launch_pack_ss(st, S.C, S.I, S.P, S.K, Q, packedState ? W.packIdx : nullptr, W.src, W.packIdxB, W.act + n, most);
        };
        // The ends are cleared and the packed state is made before the host knows the numbers, where the room that
        // is there suffices
        const bool ft = law0 || S.P.fresh;  // a serving slot may take a job with that law at any time
        Room room;
        room.act = S.I.endCap ? S.I.endCap / 2 : -1;
        room.plain = !packed ? n : (Q.ft[0] || !ft ? Q.cap : -1);
        room.tot = lookForOrphans ? nullptr : W.tot;
        if (packed && !scratch(S, W.packIdxCapB, n, W.packIdxB)) return S.fail(WG_ERR_CUDA, "out of device memory (packed contacts)");
        auto zero = [&](const Room& rm) {
            const int64_t most = 2 * std::min(rm.act, n);
            if (most > 0) k_zero_ends<<<(unsigned)((most + BS - 1) / BS), BS, 0, st>>>(S.I, W.act + n, rm);
        };
        r = incidence(S, n, W.newLo, n <= kClearInSlots ? room : Room{});
        if (r) return r;
        if (n > kClearInSlots) zero(room);
        if (packed) pack(std::min(n, room.plain));
        WG_CUDA_TRY(cudaMemcpyAsync(W.hTot, W.tot, sizeof(CollideTotals), cudaMemcpyDeviceToHost, st));
        WG_CUDA_TRY(cudaStreamSynchronize(st));
        const CollideTotals& T = *W.hTot;
        if (!lookForOrphans && T.real != T.kept) {
            // again, with the real contacts that have no overlap any more: the old set is in the spare arrays
            lookForOrphans = true;
            undo.swap();
            WG_CUDA_TRY(cudaMemsetAsync(&W.tot->heavy, 0, 2 * sizeof(int32_t), st));
            continue;
        }
        const int64_t nAct = (int64_t)(uint32_t)T.act, nSS = (int64_t)(T.act >> 32);
        // the new set takes the old one's place, after what takes more memory
        if (nAct > room.act || nSS > room.plain) {
            r = packed ? packRoom(S, Q, nSS, ft) : 0;
            if (!r) r = endRoom(S, nAct);  // last: the old ends are gone then
            if (r) return r;
            if (packed && nSS > room.plain) pack(nSS);
            zero(Room{nAct, nSS, nullptr});
        }
        undo.off = true;
        if (packed) {
            Q.n = nSS;
            std::swap(S.K, W.Kb);
            std::swap(W.packIdx, W.packIdxB);
            std::swap(W.packIdxCap, W.packIdxCapB);
        }
        S.I.nAct = nAct;
        S.nMixed = nAct - nSS;
        S.packDirty = packedState && nSS > 0;  // the contact arrays hold no state of those contacts then
        S.I.nHeavy = S.cfg.apply_forces ? T.heavy : 0;
        S.I.nHeavyFree = S.cfg.apply_forces ? T.heavyFree : 0;
        S.contactsReplaced = false;
        break;
    }
    std::swap(W.newLo, W.oldLo);
    std::swap(W.newLoCap, W.oldLoCap);
    W.oldLoValid = true;
    if (S.P.fresh) WG_CUDA_TRY(cudaMemsetAsync(S.P.fresh, 0, S.nPar, st));
    WG_CUDA_TRY(cudaGetLastError());
    S.nFullRuns++;
    return 0;
}

// A run that fails leaves the contacts, their state and their forces as they were; the boxes and the verlet
// reference positions are those of the failed run, so that the next step starts with a full run.
int collide_full_run(Sim& S) {
    const int r = fullRun(S);
    if (r) S.forceFull = true;
    return r;
}

void collide_free(Sim& S) {
    if (!S.cw) return;
    if (S.cw->hTot) cudaFreeHost(S.cw->hTot);
    delete S.cw;
    S.cw = nullptr;
}

}  // namespace wg

// Random sequential insertion of non-overlapping spheres on the device (scene generation).
//
// The device counterpart of wg_pack_rsa (wg_pack.cpp), which plays the role of
// SpherePack::makeCloud (lib/sphere-pack/SpherePack.hpp:75) for the regions of the benchmark
// scenes. The host version places sphere i (in the given order) at the first of up to
// max_attempts uniform candidate centres that overlaps no sphere placed before it. Here the
// spheres are inserted in rounds over a window of the lowest-indexed unplaced spheres (1/64 of
// the spheres, at least 256 and at most 32768):
//   1. every sphere of the window draws its next candidate centre (a counter-based hash of the
//      seed, the sphere index and the attempt number, so the result does not depend on the
//      launch shape) and tests it against the spheres placed in earlier rounds;
//   2. a candidate that is clear of them is accepted unless it overlaps the clear candidate of
//      a lower-indexed sphere of the same round;
//   3. accepted spheres join the placed set; the others draw again in the next round.
// Accepted spheres never overlap, and every sphere still gets max_attempts candidates. The
// order of acceptance follows the index order only within a window (a sphere may be placed a
// round before a lower-indexed one), so the packing is not the host version's sphere for
// sphere; its statistics (count, solid fraction, uniformity) are those of sequential insertion.
// As in the host version, the result is the prefix of spheres before the first one that found
// no place; spheres after it that were placed are dropped.
//
// A window moves on every kRounds rounds, so most of the time it holds a few stragglers whose place is
// found once in hundreds of attempts, and a round of three small kernels tests one attempt of
// each. With at most kSpec unplaced spheres in the window the kRounds attempts of all of them are
// therefore tested against the placed set at once, one warp per attempt and one cell of the
// neighbourhood per lane (k_spec_test), and one block then goes through the rounds in order over
// the few that are clear: against the spheres accepted in earlier rounds of the batch, against
// the clear candidates of lower index, and on to the next window (k_spec_resolve). The rounds, and
// so the packing, are the same; the host waits once in kBatches of them. What bounds it now is
// the latency of the two kernels of a batch. 30 000 spheres at 0.35: 907 -> 57 ms.
//
// Neighbour search: a uniform grid of edge 2 r_max over the region; placed spheres and the
// clear candidates of a round are kept in per-cell linked lists (a head per cell, a next link
// per sphere, pushed with atomicExch). The order of a list depends on the atomics, but every
// test is over the whole list, so the result does not.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace {

struct PackGrid {
    double lo[3], L[3], cw[3];
    int nc[3];
    int kind;  // 0 box, 1 cylinder along x, 2 periodic box
    double cyl[4];
};

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
// the k-th uniform double in [0, 1) of attempt a of sphere i
__device__ __forceinline__ double uni(uint64_t seed, int64_t i, int64_t a, int k) {
    const uint64_t h = mix64(seed ^ mix64((uint64_t)i * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull) ^
                             mix64((uint64_t)a * 0xD1B54A32D192ED03ull + (uint64_t)k * 0x8CB92BA72F3D8DD7ull + 1));
    return (double)(h >> 11) * (1.0 / 9007199254740992.0);
}

__device__ __forceinline__ int cellOf(const PackGrid& G, const double c[3], int ci[3]) {
    for (int k = 0; k < 3; k++) {
        int q = (int)floor((c[k] - G.lo[k]) / G.cw[k]);
        ci[k] = q < 0 ? 0 : (q >= G.nc[k] ? G.nc[k] - 1 : q);
    }
    return (ci[2] * G.nc[1] + ci[1]) * G.nc[0] + ci[0];
}

// whether centres c (radius r) and p (radius q) overlap
__device__ __forceinline__ bool clash(const PackGrid& G, const double c[3], double r, const double* __restrict__ p, double q) {
    const bool peri = G.kind == 2;
    double d2 = 0;
    for (int k = 0; k < 3; k++) {
        double d = c[k] - p[k];
        if (peri) d -= G.L[k] * rint(d / G.L[k]);
        d2 += d * d;
    }
    const double rr = r + q;
    return d2 < rr * rr;
}
// whether centre c of radius r overlaps a sphere of the list of the cell at offset (dx, dy, dz) from ci
// (only entries below `below` count when below >= 0)
__device__ __forceinline__ bool clashCell(const PackGrid& G, const double c[3], double r, const int ci[3], int dx, int dy, int dz,
                                          const int32_t* __restrict__ head, const int32_t* __restrict__ next,
                                          const double* __restrict__ pos, const double* __restrict__ radii, int64_t below) {
    const bool peri = G.kind == 2;
    int q[3] = {ci[0] + dx, ci[1] + dy, ci[2] + dz};
    for (int k = 0; k < 3; k++)
        if (q[k] < 0 || q[k] >= G.nc[k]) {
            if (!peri) return false;
            q[k] = (q[k] + G.nc[k]) % G.nc[k];
        }
    for (int32_t j = head[(q[2] * G.nc[1] + q[1]) * G.nc[0] + q[0]]; j >= 0; j = next[j]) {
        if (below >= 0 && j >= below) continue;
        if (clash(G, c, r, pos + 3 * (int64_t)j, radii[j])) return true;
    }
    return false;
}
// the same over the 27 cells around ci
__device__ bool clashList(const PackGrid& G, const double c[3], double r, const int ci[3], const int32_t* __restrict__ head,
                          const int32_t* __restrict__ next, const double* __restrict__ pos, const double* __restrict__ radii,
                          int64_t below) {
    for (int dz = -1; dz <= 1; dz++)
        for (int dy = -1; dy <= 1; dy++)
            for (int dx = -1; dx <= 1; dx++)
                if (clashCell(G, c, r, ci, dx, dy, dz, head, next, pos, radii, below)) return true;
    return false;
}
// the candidate centre of attempt a of sphere i (radius r); false if it lies outside the region
__device__ __forceinline__ bool candidate(const PackGrid& G, uint64_t seed, int64_t i, int64_t a, double r, double c[3]) {
    const bool peri = G.kind == 2;
    for (int k = 0; k < 3; k++) {
        const double m = peri ? 0. : r;
        c[k] = G.lo[k] + m + uni(seed, i, a, k) * (G.L[k] - 2 * m);
    }
    if (G.kind == 1) {
        const double dy = c[1] - G.cyl[0], dz = c[2] - G.cyl[1];
        if (sqrt(dy * dy + dz * dz) > G.cyl[2] - r) return false;
        if (c[2] + r > G.cyl[3]) return false;
    }
    return true;
}

// round step 1: candidates of the unplaced spheres in [w0, w1), tested against the placed set;
// clear ones are pushed on the round lists
__global__ void k_rsa_draw(PackGrid G, int64_t w0, int64_t w1, const double* __restrict__ radii, uint64_t seed,
                           const int32_t* __restrict__ state, const int64_t* __restrict__ attempt, double* __restrict__ cand,
                           int32_t* __restrict__ clear, const int32_t* __restrict__ headP, const int32_t* __restrict__ nextP,
                           const double* __restrict__ pos, int32_t* __restrict__ headR, int32_t* __restrict__ nextR) {
    const int64_t i = w0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w1) return;
    clear[i] = 0;
    if (state[i] != 0) return;  // placed or failed
    const double r = radii[i];
    double c[3];
    const bool inside = candidate(G, seed, i, attempt[i], r, c);
    for (int k = 0; k < 3; k++) cand[3 * i + k] = c[k];
    if (!inside) return;
    int ci[3];
    const int cell = cellOf(G, c, ci);
    if (clashList(G, c, r, ci, headP, nextP, pos, radii, -1)) return;
    clear[i] = 1;
    nextR[i] = atomicExch(headR + cell, (int32_t)i);
}

// round step 2: a clear candidate is accepted unless it overlaps the clear candidate of a
// lower-indexed sphere; rejected and unclear ones move to their next attempt
__global__ void k_rsa_resolve(PackGrid G, int64_t w0, int64_t w1, const double* __restrict__ radii, int64_t maxAttempts,
                              int32_t* __restrict__ state, int64_t* __restrict__ attempt, const double* __restrict__ cand,
                              const int32_t* __restrict__ clear, const int32_t* __restrict__ headR, const int32_t* __restrict__ nextR,
                              int32_t* __restrict__ accepted) {
    const int64_t i = w0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w1) return;
    accepted[i] = 0;
    if (state[i] != 0) return;
    bool ok = false;
    if (clear[i]) {
        const double c[3] = {cand[3 * i], cand[3 * i + 1], cand[3 * i + 2]};
        int ci[3];
        cellOf(G, c, ci);
        ok = !clashList(G, c, radii[i], ci, headR, nextR, cand, radii, i);
    }
    if (ok) {
        accepted[i] = 1;
        return;
    }
    const int64_t a = attempt[i] + 1;
    attempt[i] = a;
    if (a >= maxAttempts) state[i] = 2;  // no place found
}

// round step 3: accepted spheres join the placed set (their round-list links are dead after
// the round; the placed set keeps its own links)
__global__ void k_rsa_commit(PackGrid G, int64_t w0, int64_t w1, int32_t* __restrict__ state, const double* __restrict__ cand,
                             const int32_t* __restrict__ clear, const int32_t* __restrict__ accepted, double* __restrict__ pos,
                             int32_t* __restrict__ headP, int32_t* __restrict__ nextP, int32_t* __restrict__ headR) {
    const int64_t i = w0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w1 || !clear[i]) return;
    const double c[3] = {cand[3 * i], cand[3 * i + 1], cand[3 * i + 2]};
    int ci[3];
    const int cell = cellOf(G, c, ci);
    headR[cell] = -1;  // the round lists end with the round (every clear candidate clears its cell)
    if (!accepted[i]) return;
    for (int k = 0; k < 3; k++) pos[3 * i + k] = c[k];
    nextP[i] = atomicExch(headP + cell, (int32_t)i);
    state[i] = 1;
}

// ---- batches of kRounds rounds for a window with at most kSpec unplaced spheres
constexpr int kRounds = 16;   // rounds between two moves of the window
constexpr int kSpec = 1024;   // one thread of the resolving block each
constexpr int kBatches = 32;  // batches queued per host wait
struct Window {
    int64_t w0, w1;   // the window
    int64_t prefix;   // the result, once done
    int32_t nU;       // its unplaced spheres that have attempts left
    int32_t done;
};

__global__ void __launch_bounds__(256) k_spec_test(PackGrid G, const Window* __restrict__ win, const int32_t* __restrict__ list,
                                                   const double* __restrict__ radii, uint64_t seed, int64_t maxAttempts,
                                                   const int64_t* __restrict__ attempt, const int32_t* __restrict__ headP,
                                                   const int32_t* __restrict__ nextP, const double* __restrict__ pos,
                                                   uint8_t* __restrict__ clear) {
    const int nU = win->nU;
    if (win->done || nU > kSpec) return;
    const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nU * kRounds; t += warps) {
        const int u = t % nU, round = t / nU;
        const int64_t i = list[u], a = attempt[i] + round;
        const double r = radii[i];
        double c[3];
        bool ok = a < maxAttempts && candidate(G, seed, i, a, r, c);  // the same for the whole warp
        if (ok) {
            int ci[3];
            cellOf(G, c, ci);
            const bool hit = lane < 27 && clashCell(G, c, r, ci, lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1, headP, nextP, pos, radii, -1);
            ok = !__any_sync(0xffffffffu, hit);
        }
        if (lane == 0) clear[round * kSpec + u] = ok ? 1 : 0;
    }
}

// A centre in shared memory, exact and rounded to FP32 for a first test.
struct Centre {
    double p[3], r;
    float f[3], fr;
};
__device__ __forceinline__ void setCentre(Centre& C, const PackGrid& G, const double c[3], double r) {
    for (int k = 0; k < 3; k++) {
        C.p[k] = c[k];
        C.f[k] = (float)(c[k] - G.lo[k]);
    }
    C.r = r;
    C.fr = (float)r;
}
__device__ __forceinline__ bool clashCentre(const PackGrid& G, const float L[3], const Centre& A, const Centre& B) {
    const float rr = (A.fr + B.fr) * 1.00001f;
    for (int k = 0; k < 3; k++) {
        float d = fabsf(A.f[k] - B.f[k]);
        if (G.kind == 2) d = fminf(d, fabsf(L[k] - d));
        if (d > rr + 1e-6f * L[k]) return false;  // farther apart on one axis than the FP32 coordinates' rounding explains
    }
    return clash(G, A.p, A.r, B.p, B.r);
}

// Moves the window past its placed prefix and lists its unplaced spheres in ascending order (one block
// of kSpec threads; sh: 34 ints). The block itself may just have written the states: they are read past L1.
__device__ void moveWindow(Window* win, int64_t n, int64_t W, const int32_t* state, int32_t* __restrict__ list, int* sh) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int64_t w0 = win->w0;
    // the first sphere that is not placed
    for (;;) {
        const int64_t i = w0 + t;
        const bool stop = i >= n || __ldcg(state + i) != 1;
        if (t == 0) sh[33] = kSpec;
        __syncthreads();
        if (stop) atomicMin(sh + 33, t);
        __syncthreads();
        const int first = sh[33];
        __syncthreads();
        w0 += first;
        if (first < kSpec) break;
    }
    const int64_t w1 = w0 + W < n ? w0 + W : n;
    if (w0 >= n || __ldcg(state + w0) == 2) {  // everything placed, or the next sphere found no place
        if (t == 0) {
            win->prefix = w0 < n ? w0 : n;
            win->done = 1;
        }
        return;
    }
    int total = 0;
    for (int64_t b = w0; b < w1; b += kSpec) {
        const int64_t i = b + t;
        const bool un = i < w1 && __ldcg(state + i) == 0;
        const unsigned m = __ballot_sync(0xffffffffu, un);
        if (lane == 0) sh[warp] = __popc(m);
        __syncthreads();
        int before = total;
        for (int w = 0; w < warp; w++) before += sh[w];
        const int at = before + __popc(m & ((1u << lane) - 1u));
        if (un && at < kSpec) list[at] = (int32_t)i;
        for (int w = 0; w < kSpec / 32; w++) total += sh[w];
        __syncthreads();
    }
    if (t == 0) {
        win->w0 = w0;
        win->w1 = w1;
        win->nU = total;
    }
}
__global__ void __launch_bounds__(kSpec) k_move_window(Window* win, int64_t n, int64_t W, const int32_t* __restrict__ state,
                                                       int32_t* __restrict__ list) {
    __shared__ int sh[34];
    if (win->done) return;
    moveWindow(win, n, W, state, list, sh);
}

__global__ void __launch_bounds__(kSpec) k_spec_resolve(PackGrid G, Window* win, int64_t n, int64_t W, int32_t* __restrict__ list,
                                                        const double* __restrict__ radii, uint64_t seed, int64_t maxAttempts,
                                                        int32_t* __restrict__ state, int64_t* __restrict__ attempt,
                                                        int32_t* __restrict__ headP, int32_t* __restrict__ nextP,
                                                        double* __restrict__ pos, const uint8_t* __restrict__ clear) {
    extern __shared__ Centre smem[];
    Centre* acc = smem;          // accepted in this batch
    Centre* cur = smem + kSpec;  // clear candidates of the round, ascending
    __shared__ int sh[34], nAcc;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nU = win->nU;
    if (win->done || nU > kSpec) return;
    const bool in = t < nU;
    const int64_t i = in ? list[t] : 0;
    const double r = in ? radii[i] : 0.;
    const int64_t a0 = in ? attempt[i] : 0;
    const float L[3] = {(float)G.L[0], (float)G.L[1], (float)G.L[2]};
    unsigned mask = 0;
    if (in)
        for (int q = 0; q < kRounds; q++) mask |= (unsigned)clear[q * kSpec + t] << q;
    bool placed = false;
    double mine[3] = {0., 0., 0.};
    if (t == 0) nAcc = 0;
    __syncthreads();
    for (int q = 0; q < kRounds; q++) {
        const int have = nAcc;
        bool ok = !placed && ((mask >> q) & 1u);
        Centre me;
        if (ok) {
            double c[3];
            candidate(G, seed, i, a0 + q, r, c);
            setCentre(me, G, c, r);
            for (int k = 0; k < have && ok; k++) ok = !clashCentre(G, L, me, acc[k]);
        }
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) sh[warp] = __popc(m);
        __syncthreads();
        int rank = __popc(m & ((1u << lane) - 1u));
        for (int w = 0; w < warp; w++) rank += sh[w];
        if (ok) cur[rank] = me;
        __syncthreads();
        if (ok) {
            for (int k = 0; k < rank && ok; k++) ok = !clashCentre(G, L, me, cur[k]);
            if (ok) {
                placed = true;
                for (int k = 0; k < 3; k++) mine[k] = me.p[k];
                acc[atomicAdd(&nAcc, 1)] = me;
            }
        }
        __syncthreads();
    }
    if (in) {
        if (placed) {
            int ci[3];
            const int cell = cellOf(G, mine, ci);
            for (int k = 0; k < 3; k++) pos[3 * i + k] = mine[k];
            nextP[i] = atomicExch(headP + cell, (int32_t)i);
            state[i] = 1;
        } else {
            const int64_t a = a0 + kRounds < maxAttempts ? a0 + kRounds : maxAttempts;
            attempt[i] = a;
            if (a >= maxAttempts) state[i] = 2;
        }
    }
    __syncthreads();
    moveWindow(win, n, W, state, list, sh);
}

// stream-ordered scratch (no device-wide synchronisation when it is freed, so that a packer
// running beside simulations on other streams does not wait for their work)
struct Scratch {
    cudaStream_t st = nullptr;
    std::vector<void*> ptrs;
    ~Scratch() {
        for (void* p : ptrs) cudaFreeAsync(p, st);
        if (st) {
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
    }
    template <class T>
    T* get(size_t count) {
        void* p = nullptr;
        if (cudaMallocAsync(&p, sizeof(T) * count, st) != cudaSuccess) return nullptr;
        ptrs.push_back(p);
        return (T*)p;
    }
};

}  // namespace

extern "C" {

/* The device packer; arguments and result as wg_pack_rsa (wg_pack.cpp). Negative result: a CUDA
   error (-1) or an argument error (-2). */
int64_t wg_pack_rsa_device(int64_t n, const double* radii, const double* lo, const double* hi, int32_t region_kind,
                           const double* params, uint64_t seed, int64_t max_attempts, double* centers) {
    if (n <= 0) return 0;
    if (!radii || !lo || !hi || !centers || region_kind < 0 || region_kind > 2 || max_attempts < 1 || n >= (int64_t(1) << 31) - 1)
        return -2;
    if (region_kind == 1 && !params) return -2;
    double rmax = 0;
    for (int64_t i = 0; i < n; i++) {
        if (!(radii[i] > 0) || !std::isfinite(radii[i])) return -2;
        rmax = std::fmax(rmax, radii[i]);
    }
    PackGrid G{};
    G.kind = region_kind;
    const double cs = 2 * rmax;
    int64_t ncell = 1;
    for (int k = 0; k < 3; k++) {
        G.lo[k] = lo[k];
        G.L[k] = hi[k] - lo[k];
        if (!(G.L[k] > 0) || !std::isfinite(G.L[k])) return -2;
        const int64_t q = std::max<int64_t>(1, (int64_t)std::floor(G.L[k] / cs));
        if (q > (1 << 20)) return -2;
        G.nc[k] = (int)q;
        G.cw[k] = G.L[k] / (double)q;
        ncell *= q;
    }
    if (ncell > (int64_t(1) << 30)) return -2;
    if (region_kind == 1)
        for (int k = 0; k < 4; k++) G.cyl[k] = params[k];
    // device arrays, on a stream of the call's own
    Scratch X;
    if (cudaStreamCreateWithFlags(&X.st, cudaStreamNonBlocking) != cudaSuccess) {
        X.st = nullptr;
        return -1;
    }
    cudaStream_t st = X.st;
    double* dRad = X.get<double>(n);
    double* dPos = X.get<double>(3 * n);
    double* dCand = X.get<double>(3 * n);
    int32_t* dState = X.get<int32_t>(n);
    int64_t* dAtt = X.get<int64_t>(n);
    int32_t* dClear = X.get<int32_t>(n);
    int32_t* dAcc = X.get<int32_t>(n);
    int32_t* dHeadP = X.get<int32_t>(ncell);
    int32_t* dNextP = X.get<int32_t>(n);
    int32_t* dHeadR = X.get<int32_t>(ncell);
    int32_t* dNextR = X.get<int32_t>(n);
    if (!dRad || !dPos || !dCand || !dState || !dAtt || !dClear || !dAcc || !dHeadP || !dNextP || !dHeadR || !dNextR) return -1;
    bool ok = cudaMemcpyAsync(dRad, radii, sizeof(double) * n, cudaMemcpyHostToDevice, st) == cudaSuccess &&
              cudaMemsetAsync(dState, 0, sizeof(int32_t) * n, st) == cudaSuccess &&
              cudaMemsetAsync(dAtt, 0, sizeof(int64_t) * n, st) == cudaSuccess &&
              cudaMemsetAsync(dHeadP, 0xff, sizeof(int32_t) * ncell, st) == cudaSuccess &&
              cudaMemsetAsync(dHeadR, 0xff, sizeof(int32_t) * ncell, st) == cudaSuccess;
    if (!ok) return -1;
    // the window: the unplaced spheres of [w0, w1), w1 - w0 at most W, a small fraction of the
    // spheres so that the window holds spheres of similar rank (the insertion order puts the
    // largest first: a window of all spheres would let small ones fill the gaps the large ones
    // need); after every kRounds rounds w0 moves past the placed prefix; the first sphere that found no
    // place ends the insertion
    const int64_t W = std::min<int64_t>(32768, std::max<int64_t>(256, n / 64));
    Window* dWin = X.get<Window>(1);
    int32_t* dList = X.get<int32_t>(kSpec);
    uint8_t* dSpec = X.get<uint8_t>((size_t)kSpec * kRounds);
    const size_t shm = 2 * sizeof(Centre) * kSpec;
    Window win{};
    if (!dWin || !dList || !dSpec ||
        cudaFuncSetAttribute(k_spec_resolve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm) != cudaSuccess ||
        cudaMemsetAsync(dWin, 0, sizeof(Window), st) != cudaSuccess)
        return -1;
    k_move_window<<<1, kSpec, 0, st>>>(dWin, n, W, dState, dList);
    for (;;) {
        // a launch that was refused would leave the window where it is for good
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(&win, dWin, sizeof(Window), cudaMemcpyDeviceToHost, st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess)
            return -1;
        if (win.done) break;
        if (win.nU <= kSpec) {
            for (int q = 0; q < kBatches; q++) {
                k_spec_test<<<304, 256, 0, st>>>(G, dWin, dList, dRad, seed, max_attempts, dAtt, dHeadP, dNextP, dPos, dSpec);
                k_spec_resolve<<<1, kSpec, shm, st>>>(G, dWin, n, W, dList, dRad, seed, max_attempts, dState, dAtt, dHeadP, dNextP, dPos,
                                                      dSpec);
            }
            continue;
        }
        // a window of many unplaced spheres (over 65 536 spheres in all): round by round, one thread each
        const unsigned g = (unsigned)((win.w1 - win.w0 + 255) / 256);
        for (int round = 0; round < kRounds; round++) {
            k_rsa_draw<<<g, 256, 0, st>>>(G, win.w0, win.w1, dRad, seed, dState, dAtt, dCand, dClear, dHeadP, dNextP, dPos, dHeadR, dNextR);
            k_rsa_resolve<<<g, 256, 0, st>>>(G, win.w0, win.w1, dRad, max_attempts, dState, dAtt, dCand, dClear, dHeadR, dNextR, dAcc);
            k_rsa_commit<<<g, 256, 0, st>>>(G, win.w0, win.w1, dState, dCand, dClear, dAcc, dPos, dHeadP, dNextP, dHeadR);
        }
        k_move_window<<<1, kSpec, 0, st>>>(dWin, n, W, dState, dList);
    }
    const int64_t prefix = win.prefix;
    if (prefix > 0 && (cudaMemcpyAsync(centers, dPos, sizeof(double) * 3 * prefix, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                       cudaStreamSynchronize(st) != cudaSuccess))
        return -1;
    if (cudaGetLastError() != cudaSuccess) return -1;
    return prefix;
}

}  // extern "C"

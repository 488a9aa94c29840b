// se_realspace.cu -- the real-space and self terms of the Ewald sum beside
// the k-space solve: SE3P_direct_real_rc (SE_direct.c:464-506),
// SE3P_direct_real (:508-549) and SE3P_direct_self (:551-562), plus the
// real-space force (the gradient of the same sum; the reference has none).
//
// Two algorithms, chosen by the cutoff:
//   all pairs   any rc and layers: one thread per target, the sources in
//               tiles of 128 through shared memory, the images in the
//               reference's (p0, p1, p2) order -- the reference's summation
//               order for every target;
//   cell list   0 < rc <= L/2 with at least 3 cells of edge >= rc per axis:
//               particles sorted by cell (the library's stable sort), one
//               warp per target (in cell order), or one thread for many
//               targets of few neighbours, over the 27 neighbour cells.
//               Each particle keeps its position wrapped into the box and the
//               number of boxes it was moved by, so the image of a pair is
//               recovered exactly and the reference's limit |p| <= layers on
//               it holds for positions anywhere.
// Scratch memory of the cell list is taken from a stream-ordered pool
// (ScratchPool) and returned on the same stream.
#include <cmath>
#include <mutex>

#include "se_internal.h"

namespace se {
namespace {

constexpr int RS_THREADS = 128;
constexpr double RS_PI = 3.14159265358979323846;

struct RsParams {
    int N, layers;
    double L, xi, rc, rc2, g;   // g = 2 xi / sqrt(pi)
};

// One pair term at separation d (|d|^2 = rr): potential and force weights.
template <bool FORCE>
__device__ __forceinline__ void pair_term(const RsParams& S, double qn, const double d[3],
                                          double rr, double& phi, double f[3])
{
    const double r = sqrt(rr);
    const double e = erfc(S.xi * r) / r;
    phi += qn * e;
    if (FORCE) {
        const double s = qn * (e + S.g * exp(-S.xi * S.xi * rr)) / rr;
        f[0] += s * d[0];
        f[1] += s * d[1];
        f[2] += s * d[2];
    }
}

template <bool FORCE>
__global__ void __launch_bounds__(RS_THREADS) k_real_allpairs(
    RsParams S, const double* __restrict__ x, const double* __restrict__ q,
    double* __restrict__ phi, double* __restrict__ force)
{
    __shared__ double4 src[RS_THREADS];
    const int N = S.N;
    const int m = blockIdx.x * RS_THREADS + threadIdx.x;
    double xm[3] = {0, 0, 0};
    if (m < N) {
        xm[0] = x[m];
        xm[1] = x[m + N];
        xm[2] = x[m + 2 * N];
    }
    double acc = 0, f[3] = {0, 0, 0};
    const int l = S.layers;
    for (int t0 = 0; t0 < N; t0 += RS_THREADS) {
        const int n = t0 + threadIdx.x;
        __syncthreads();
        if (n < N) src[threadIdx.x] = make_double4(x[n], x[n + N], x[n + 2 * N], q[n]);
        __syncthreads();
        if (m >= N) continue;
        const int cnt = min(RS_THREADS, N - t0);
        for (int j = 0; j < cnt; j++) {
            const double4 s = src[j];
            const double r0 = xm[0] - s.x, r1 = xm[1] - s.y, r2 = xm[2] - s.z;
            for (int p0 = -l; p0 <= l; p0++)
                for (int p1 = -l; p1 <= l; p1++)
                    for (int p2 = -l; p2 <= l; p2++) {
                        if (m == t0 + j && p0 == 0 && p1 == 0 && p2 == 0) continue;
                        const double d[3] = {r0 + p0 * S.L, r1 + p1 * S.L, r2 + p2 * S.L};
                        const double rr = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
                        if (S.rc > 0 && rr > S.rc2) continue;
                        pair_term<FORCE>(S, s.w, d, rr, acc, f);
                    }
        }
    }
    if (m >= N) return;
    if (phi) phi[m] += acc;
    if (FORCE) {
        const double qm = q[m];
        force[m] += qm * f[0];
        force[m + N] += qm * f[1];
        force[m + 2 * N] += qm * f[2];
    }
}

// Cell of every particle (edge cs = L / nc >= rc), from its position wrapped
// into [0, L); the number of boxes it was moved by, packed per axis.
__global__ void k_real_keys(RsParams S, int nc, const double* __restrict__ x,
                            int* __restrict__ key)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= S.N) return;
    int c[3];
    for (int a = 0; a < 3; a++) {
        const double v = x[n + (long long)a * S.N];
        const double w = v - S.L * floor(v / S.L);
        c[a] = min((int)(w * nc / S.L), nc - 1);
    }
    key[n] = (c[0] * nc + c[1]) * nc + c[2];
}

// The groups of 32 targets left to k_real_cells_crowded, and its next target.
struct RsCrowded {
    int groups, next;
};

// Sorted records: wrapped position and charge, and the box shifts k_a =
// floor(x_a / L) (each within +-511).
__global__ void k_real_gather(RsParams S, const int* __restrict__ perm,
                              const double* __restrict__ x, const double* __restrict__ q,
                              double4* __restrict__ rec, int* __restrict__ kbox,
                              RsCrowded* __restrict__ crowded)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0 && crowded) *crowded = {};
    if (s >= S.N) return;
    const int n = perm[s];
    double w[3];
    int k[3];
    for (int a = 0; a < 3; a++) {
        const double v = x[n + (long long)a * S.N];
        const double fl = floor(v / S.L);
        w[a] = v - S.L * fl;
        k[a] = (int)fl;
    }
    rec[s] = make_double4(w[0], w[1], w[2], q[n]);
    kbox[s] = ((k[0] + 512) & 1023) | (((k[1] + 512) & 1023) << 10) | (((k[2] + 512) & 1023) << 20);
}

__device__ __forceinline__ int kbox_of(int pk, int a) { return ((pk >> (10 * a)) & 1023) - 512; }

// The candidates of a target in cell c are 18 runs of the sorted particles: run u
// holds the z cells c[2] - 1 to c[2] + 1 of neighbour row u / 2 (u even), or the one of
// them past the box's end (u odd, else empty).  shift: the run's box shifts + 1, 2
// bits an axis.
__device__ __forceinline__ void neighbour_run(int u, const int c[3], int nc, const int* __restrict__ cell_off,
                                              int& beg, int& end, int& shift)
{
    const int cx = c[0] + u / 6 - 1, cy = c[1] + u / 2 % 3 - 1;
    const int sh0 = cx < 0 ? -1 : (cx >= nc ? 1 : 0);
    const int sh1 = cy < 0 ? -1 : (cy >= nc ? 1 : 0);
    const int row = ((cx - sh0 * nc) * nc + cy - sh1 * nc) * nc;
    int z0 = max(c[2] - 1, 0), z1 = min(c[2] + 1, nc - 1);
    int sh2 = 0;
    if (u & 1) {
        sh2 = c[2] == 0 ? -1 : (c[2] == nc - 1 ? 1 : 0);
        z0 = c[2] == 0 ? nc - 1 : 0;
        z1 = sh2 ? z0 : z0 - 1;
    }
    beg = cell_off[row + z0];
    end = cell_off[row + z1 + 1];
    shift = (sh0 + 1) | (sh1 + 1) << 2 | (sh2 + 1) << 4;
}

// Separation of the target at xm from particle o of a run, and its square.
__device__ __forceinline__ double separation(const RsParams& S, const double xm[3], const double4& o, int shift,
                                             double (&d)[3])
{
    d[0] = xm[0] - (o.x + ((shift & 3) - 1) * S.L);
    d[1] = xm[1] - (o.y + ((shift >> 2 & 3) - 1) * S.L);
    d[2] = xm[2] - (o.z + ((shift >> 4 & 3) - 1) * S.L);
    return d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
}

// The term of a pair inside the cutoff, e: the particle and its run's shifts.
template <bool FORCE>
__device__ __forceinline__ void queued_pair(const RsParams& S, const double xm[3], int km,
                                            const double4* __restrict__ rec, const int* __restrict__ kbox, int2 e,
                                            double& acc, double (&f)[3])
{
    const double4 o = rec[e.x];
    const int kt = kbox[e.x];
    double d[3];
    const double rr = separation(S, xm, o, e.y, d);
    bool in = true;   // the image index of the pair in raw coordinates
    for (int a = 0; a < 3; a++) {
        const int p = kbox_of(kt, a) - kbox_of(km, a) - ((e.y >> 2 * a & 3) - 1);
        in = in && p >= -S.layers && p <= S.layers;
    }
    if (in) pair_term<FORCE>(S, o.w, d, rr, acc, f);
}

// One warp per target s (in cell order).  The lanes test 32 candidates of the
// neighbour cells at a time and queue the pairs inside the cutoff; 32 queued pairs
// are then evaluated together, one per lane.  About one candidate in eight is a pair,
// and a pair costs some ten times a test (erfc, exp, two divisions): with a target per
// thread, its pairs evaluated as they are found, most lanes sat out every evaluation
// (50,000 particles, about 100 neighbours each, force: 548 -> 205 us; the FP64
// pipe 35% and the issue slots 65% busy; with the separations queued instead
// of the particles, 246 us).
// A lane sums its pairs in queue order and the lanes' sums are added in a
// fixed order, so results are deterministic.
template <bool FORCE>
__device__ __forceinline__ void target_by_warp(const RsParams& S, int nc, const double4* __restrict__ rec,
                                               const int* __restrict__ kbox, const int* __restrict__ perm,
                                               const int* __restrict__ cell_off, double* __restrict__ phi,
                                               double* __restrict__ force, int s, int2* que)
{
    const int lane = threadIdx.x & 31;
    const double4 me = rec[s];
    const int km = kbox[s];
    const double xm[3] = {me.x, me.y, me.z};
    int c[3];
    for (int a = 0; a < 3; a++) c[a] = min((int)(xm[a] * nc / S.L), nc - 1);
    // lane l < 18: run l and its box shifts
    int beg = 0, end = 0, shift = 0;
    if (lane < 18) neighbour_run(lane, c, nc, cell_off, beg, end, shift);
    double acc = 0, f[3] = {0, 0, 0};
    auto pair = [&](int2 e) { queued_pair<FORCE>(S, xm, km, rec, kbox, e, acc, f); };
    int queued = 0;
    for (int run = 0; run < 18; run++) {
        const int b = __shfl_sync(0xffffffffu, beg, run), e = __shfl_sync(0xffffffffu, end, run);
        if (b >= e) continue;
        const int sh = __shfl_sync(0xffffffffu, shift, run);
        for (int t0 = b; t0 < e; t0 += 32) {
            const int t = t0 + lane;
            double d[3];
            // (a particle is in one cell, so t = s is the pair with itself)
            const bool in = t < e && t != s && !(separation(S, xm, rec[min(t, e - 1)], sh, d) > S.rc2);
            const unsigned hit = __ballot_sync(0xffffffffu, in);
            if (in) que[queued + __popc(hit & ((1u << lane) - 1u))] = make_int2(t, sh);
            queued += __popc(hit);
            if (queued >= 32) {
                __syncwarp();
                pair(que[lane]);
                queued -= 32;
                const int2 rest = que[32 + lane];
                __syncwarp();
                if (lane < queued) que[lane] = rest;
            }
        }
    }
    __syncwarp();
    if (lane < queued) pair(que[lane]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (FORCE)
            for (int a = 0; a < 3; a++) f[a] += __shfl_xor_sync(0xffffffffu, f[a], o);
    }
    if (lane != 0) return;
    const int m = perm[s];
    if (phi) phi[m] += acc;
    if (FORCE) {
        force[m] += me.w * f[0];
        force[m + S.N] += me.w * f[1];
        force[m + 2 * S.N] += me.w * f[2];
    }
}

template <bool FORCE>
__global__ void __launch_bounds__(RS_THREADS) k_real_cells(
    RsParams S, int nc, const double4* __restrict__ rec, const int* __restrict__ kbox,
    const int* __restrict__ perm, const int* __restrict__ cell_off, double* __restrict__ phi,
    double* __restrict__ force)
{
    __shared__ int2 queue[RS_THREADS / 32][64];   // particle, box shifts + 1 (2 bits an axis)
    const int warp = threadIdx.x >> 5, s = blockIdx.x * (RS_THREADS / 32) + warp;
    if (s < S.N) target_by_warp<FORCE>(S, nc, rec, kbox, perm, cell_off, phi, force, s, queue[warp]);
}

// One thread per target, for many targets of few candidates each.  A lane queues its
// own pairs inside the cutoff and the lanes of a warp evaluate theirs together,
// when some lane's queue is full (straight from the test, a warp pays for a pair
// whenever one lane has one).  A warp with a target of more than RS_CROWDED candidates
// leaves its targets to k_real_cells_crowded.
constexpr int RS_QUEUE = 16;
constexpr int RS_CROWDED = 224;
constexpr int RS_CROWDED_CTAS = 148 * 12;   // (as many as are resident, and more)

template <bool FORCE>
__global__ void __launch_bounds__(RS_THREADS) k_real_cells_sparse(
    RsParams S, int nc, const double4* __restrict__ rec, const int* __restrict__ kbox,
    const int* __restrict__ perm, const int* __restrict__ cell_off, double* __restrict__ phi,
    double* __restrict__ force, RsCrowded* __restrict__ crowded, int* __restrict__ group)
{
    __shared__ int2 queue[RS_THREADS / 32][RS_QUEUE][32];
    int2(*que)[32] = queue[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int s = blockIdx.x * RS_THREADS + threadIdx.x;
    const bool on = s < S.N;   // (the other lanes of the last warp have no candidates)
    const double4 me = rec[on ? s : 0];
    const int km = kbox[on ? s : 0];
    const double xm[3] = {me.x, me.y, me.z};
    int c[3];
    for (int a = 0; a < 3; a++) c[a] = min((int)(xm[a] * nc / S.L), nc - 1);
    int candidates = 0;
    if (on)
        for (int run = 0; run < 18; run++) {
            int beg, end, shift;
            neighbour_run(run, c, nc, cell_off, beg, end, shift);
            candidates += end - beg;
        }
    if (__any_sync(0xffffffffu, candidates > RS_CROWDED)) {
        if (lane == 0) group[atomicAdd(&crowded->groups, 1)] = s >> 5;
        return;
    }
    double acc = 0, f[3] = {0, 0, 0};
    int queued = 0;
    auto flush = [&] {
        for (int i = 0; __any_sync(0xffffffffu, i < queued); i++)
            if (i < queued) queued_pair<FORCE>(S, xm, km, rec, kbox, que[i][lane], acc, f);
        queued = 0;
    };
    for (int run = 0; run < 18; run++) {
        int beg = 0, end = 0, shift = 0;
        if (on) neighbour_run(run, c, nc, cell_off, beg, end, shift);
        for (int t0 = beg; __any_sync(0xffffffffu, t0 < end); t0 += 2) {
            double4 o[2];   // (two loads in flight)
#pragma unroll
            for (int j = 0; j < 2; j++)
                if (t0 + j < end) o[j] = rec[t0 + j];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int t = t0 + j;
                double d[3];
                if (t < end && t != s && !(separation(S, xm, o[j], shift, d) > S.rc2))
                    que[queued++][lane] = make_int2(t, shift);
            }
            if (__any_sync(0xffffffffu, queued > RS_QUEUE - 2)) flush();
        }
    }
    flush();
    if (!on) return;
    const int m = perm[s];
    if (phi) phi[m] += acc;
    if (FORCE) {
        force[m] += me.w * f[0];
        force[m + S.N] += me.w * f[1];
        force[m + 2 * S.N] += me.w * f[2];
    }
}

// The targets of the listed groups, a warp each, as the warps get free.
template <bool FORCE>
__global__ void __launch_bounds__(RS_THREADS) k_real_cells_crowded(
    RsParams S, int nc, const double4* __restrict__ rec, const int* __restrict__ kbox,
    const int* __restrict__ perm, const int* __restrict__ cell_off, double* __restrict__ phi,
    double* __restrict__ force, RsCrowded* __restrict__ crowded, const int* __restrict__ group)
{
    __shared__ int2 queue[RS_THREADS / 32][64];
    const int groups = crowded->groups;
    for (;;) {
        int t = 0;
        if ((threadIdx.x & 31) == 0) t = atomicAdd(&crowded->next, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >> 5 >= groups) return;
        const int s = 32 * group[t >> 5] + (t & 31);
        if (s < S.N) target_by_warp<FORCE>(S, nc, rec, kbox, perm, cell_off, phi, force, s, queue[threadIdx.x >> 5]);
        __syncwarp();   // its queue is used again
    }
}

__global__ void k_self(const double* __restrict__ q, int N, double c, double* __restrict__ phi)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < N) phi[m] -= c * q[m];
}

// Cells per axis of the cell-list form, or 0 when the all-pairs form applies.
int cells_per_axis(double L, double rc)
{
    if (!(rc > 0) || 2 * rc > L) return 0;
    const double nc = floor(L / rc);
    return (nc >= 3 && nc <= 256) ? (int)nc : 0;
}

// Whether the targets go a thread each (k_real_cells_sparse) where they are not
// crowded: from 2^18 particles on and up to 160 candidates on average.  A warp and a
// thread per target, force, us: 2M uniform particles with 1, 6, 15 and 25
// neighbours (6 to 160 candidates) 3331, 4021, 4157, 4133 and 735, 1006, 1709, 2490;
// 300,000 with 1, 15 and 50 600, 716, 880 and 245, 438, 902; 30,000 with 1 and 10
// 150, 142 and 127, 141, 3,000 with 1 86 and 98.  1M clustered (16 Gaussians of sigma
// 0.03; 5 neighbours on average, most targets left to k_real_cells_crowded) 6649
// and 6609, potentials alone 5297 and 5932; with 140,000 of them the warps left to the
// thread kernel are its whole time: 385 and 570.
static bool sparse_targets(int N, int ncell)
{
    return N >= 1 << 18 && 27.0 * N <= 160.0 * ncell;
}

// Scratch of a call, ordered on its stream: from a pool of this library's own
// that keeps up to KEEP bytes between calls (the device's default pool gives
// everything back at the next synchronisation, and taking it again cost a call
// that was waited for 0.5 ms); inside a stream capture from the default pool.
struct ScratchPool {
    static constexpr unsigned long long KEEP = 256ull << 20;
    static constexpr int MAX_DEVICES = 64;
    std::mutex mu;
    cudaMemPool_t pool[MAX_DEVICES] = {};

    int alloc(void** p, size_t bytes, cudaStream_t st)
    {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        int dev = 0;
        SE_CUDA(cudaGetDevice(&dev));
        const bool plain = cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone;
        if (!plain || dev >= MAX_DEVICES) {
            cudaGetLastError();
            SE_CUDA(cudaMallocAsync(p, bytes, st));
            return SE_OK;
        }
        cudaMemPool_t mp;
        {
            std::lock_guard<std::mutex> lock(mu);
            if (!pool[dev]) {
                cudaMemPoolProps props = {};
                props.allocType = cudaMemAllocationTypePinned;
                props.location.type = cudaMemLocationTypeDevice;
                props.location.id = dev;
                SE_CUDA(cudaMemPoolCreate(&pool[dev], &props));
                unsigned long long keep = KEEP;
                SE_CUDA(cudaMemPoolSetAttribute(pool[dev], cudaMemPoolAttrReleaseThreshold, &keep));
            }
            mp = pool[dev];
        }
        SE_CUDA(cudaMallocFromPoolAsync(p, bytes, mp, st));
        return SE_OK;
    }
};

ScratchPool& scratch_pool()
{
    static ScratchPool* p = new ScratchPool();
    return *p;
}

int real_space(const double* x, const double* q, int N, double L, double xi, int layers,
               double rc, double* phi, double* force, cudaStream_t st)
{
    RsParams S;
    S.N = N;
    S.layers = layers;
    S.L = L;
    S.xi = xi;
    S.rc = rc > 0 ? rc : 0.0;
    S.rc2 = S.rc * S.rc;
    S.g = 2.0 * xi / sqrt(RS_PI);
    const int nc = cells_per_axis(L, rc);
    const unsigned nb = ceil_div(N, RS_THREADS);
    if (nc == 0) {
        if (force) k_real_allpairs<true><<<nb, RS_THREADS, 0, st>>>(S, x, q, phi, force);
        else k_real_allpairs<false><<<nb, RS_THREADS, 0, st>>>(S, x, q, phi, nullptr);
        SE_CUDA(cudaGetLastError());
        return SE_OK;
    }
    const int ncell = nc * nc * nc;
    const size_t sb = sort_scratch_bytes(N, ncell);
    const size_t nbytes = 256 * ((sizeof(int) * N + 255) / 256);
    const size_t rbytes = 256 * ((sizeof(double4) * N + 255) / 256);
    const size_t obytes = 256 * ((sizeof(int) * (ncell + 1) + 255) / 256);
    const size_t total = 3 * nbytes + rbytes + obytes + sb;
    char* base = nullptr;
    SE_TRY(scratch_pool().alloc((void**)&base, total, st));
    int* key = reinterpret_cast<int*>(base);
    int* perm = reinterpret_cast<int*>(base + nbytes);
    int* kbox = reinterpret_cast<int*>(base + 2 * nbytes);
    double4* rec = reinterpret_cast<double4*>(base + 3 * nbytes);
    int* off = reinterpret_cast<int*>(base + 3 * nbytes + rbytes);
    void* scratch = base + 3 * nbytes + rbytes + obytes;
    int r = SE_OK;
    k_real_keys<<<ceil_div(N, 256), 256, 0, st>>>(S, nc, x, key);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        r = stable_sort(key, nullptr, N, ncell, perm, nullptr, off, scratch, sb, st, nullptr);
        if (r == SE_OK) {
            // (the keys are of no more use: the crowded groups' list in their place)
            const bool sparse = sparse_targets(N, ncell);
            RsCrowded* crowded = sparse ? reinterpret_cast<RsCrowded*>(key) : nullptr;
            int* group = key + sizeof(RsCrowded) / sizeof(int);
            k_real_gather<<<ceil_div(N, 256), 256, 0, st>>>(S, perm, x, q, rec, kbox, crowded);
            if (sparse) {
                (force ? k_real_cells_sparse<true> : k_real_cells_sparse<false>)<<<nb, RS_THREADS, 0, st>>>(
                    S, nc, rec, kbox, perm, off, phi, force, crowded, group);
                (force ? k_real_cells_crowded<true> : k_real_cells_crowded<false>)<<<RS_CROWDED_CTAS, RS_THREADS, 0, st>>>(
                    S, nc, rec, kbox, perm, off, phi, force, crowded, group);
            } else {
                (force ? k_real_cells<true> : k_real_cells<false>)<<<ceil_div(N, RS_THREADS / 32), RS_THREADS, 0, st>>>(
                    S, nc, rec, kbox, perm, off, phi, force);
            }
            e = cudaGetLastError();
        }
    }
    cudaFreeAsync(base, st);
    if (e != cudaSuccess) return cuda_fail(e, "real-space kernels", __FILE__, __LINE__);
    return r;
}

}  // namespace
}  // namespace se

extern "C" int se_real_space(const double* x, const double* q, int N, double L, double xi,
                             int layers, double rc, double* phi, double* force, void* stream)
{
    if (N < 0 || !(L > 0) || !(xi > 0) || layers < 0 || layers > 64 || (!phi && !force) ||
        (N > 0 && (!x || !q)))
        return SE_ERR_INVALID;
    if (N == 0) return SE_OK;
    return se::real_space(x, q, N, L, xi, layers, rc, phi, force, se::as_stream(stream));
}

extern "C" int se_self_term(const double* q, int N, double xi, double* phi, void* stream)
{
    if (N < 0 || !(xi > 0) || (N > 0 && (!q || !phi))) return SE_ERR_INVALID;
    if (N == 0) return SE_OK;
    se::k_self<<<se::ceil_div(N, 256), 256, 0, se::as_stream(stream)>>>(
        q, N, 2.0 * xi / sqrt(se::RS_PI), phi);
    SE_CUDA(cudaGetLastError());
    return SE_OK;
}

// se_interp3.cuh -- interpolation (SE_FGG_int / SE_FGG_int_force,
// SE_fgg.c:968-1100) with the periodic unfold (SE_FGG_extend_fcn,
// SE_fgg.c:417-443) fused, on FP64 matrix instructions, for any grid and
// stencil.  Included inside namespace se by se_solve.cu after se_interp2.cuh.
//
// The particles of a fine bin (8^3 stencil corners) share a window of P + 7
// grid cells per axis.  For a group of 8 of them the sum over y is a matrix
// product: U[z][particle] = sum_y H[x][y][z] wy[y][particle], 8 z cells by 8
// particles by 4 y per instruction, with the y weights zero outside each
// stencil; forces take a second product with the y force weights.  U is
// weighted with wx (and the force weights) and summed over the x planes in
// the accumulators' own layout, then with wz.
//
// One CTA of 4 independent warps per bin (and per `chunk` further particles
// of a crowded one, launch_interp3); a warp takes a group at a time.  H comes straight from
// the grid through L1: a window in shared memory (102 KB at P = 16, two CTAs
// per SM) left the matrix unit idle while it was copied.  The operand tile is
// laid so that its 8 rows are neighbouring z: a load touches 4 grid rows, and
// two z tiles share 16-byte loads (the load wavefronts were the bound: 8 per
// 8-byte load).  Forces load the next planes' operands into the registers of
// the ones just used; potentials, with half the products per operand, do
// better with more warps and no lookahead.
//
// The groups hold particles of neighbouring x offset, so they walk about P + 2
// planes instead of P + 7.  A sum that is not finite is taken again over the
// particle's own stencil: outside it the weights are zero, but zero times an
// infinity of the caller's grid is not.
//
// B200, FP64, interpolation stage before (windows in shared memory, FP64
// FMAs) and after: 100,000 particles, M = 128, P = 16 force 0.322 -> 0.257 ms,
// potential 0.275 -> 0.190 ms; 20,000 particles, M = 100, P = 20, force 0.606
// -> 0.139 ms; 2M clustered, M = 256, P = 12, force 3.34 -> 2.14 ms; 250,000,
// M = 192, P = 12, potential 0.385 -> 0.305 ms; 1M, M = 256, P = 12, force 1.53
// -> 1.55 ms, P = 8 potential 0.81 -> 0.49 ms.  At P = 16 the matrix unit is
// 54% busy (its instructions alone take 0.126 ms), the L1 wavefronts 70%; the warps
// in flight matter most (potentials with 4, 5 and 7 CTAs per SM at 250,000, P =
// 12: 0.449, 0.315 and 0.305 ms; forces keep 128 registers, with fewer they
// spill).  The weights are explicit FMAs, which every instantiation rounds alike (the
// same products left to the compiler: 0.256 ms for 0.258 here, 0.104 for 0.101 at M =
// 100, P = 12, and other last bits at P = 31 and 32 with shared groups).

constexpr int I3_WARPS = 4;
constexpr int I3_PART = 256;   // particles of a bin a CTA takes at most
// from this many particles on they are grouped by whether they reach the last
// z tile (with fewer, groups of 8 stay partly empty: 30 per bin, P = 12, 1.61
// -> 1.78 ms)
constexpr int I3_BY_TILE = 64;

// depth of the y contraction in steps of 4 cells over the window of a bin's
// stencils, FB + P - 1 cells
__host__ __device__ constexpr int interp3_nk(int P) { return (FB + P + 2) / 4; }

// x planes a warp contracts together with nt z tiles (independent chains)
__host__ __device__ constexpr int interp3_nx(bool force, int nt) { return force ? 2 / nt : 4 / nt; }

// factor of cell w of a bin's window on axis a, for sorted particle p whose
// stencil starts at cell r: from the tile-aligned rows, in which the window
// starts at entry hw, or from the P-wide rows
template <bool TILED, typename T>
__device__ __forceinline__ double interp3_factor(const T* __restrict__ fac, int PS, int P, int p, int a, int w,
                                                 int r, int hw)
{
    if constexpr (TILED) {
        return (hw + w) < 32 ? (double)fac[(long long)p * 96 + 32 * a + hw + w] : 0.0;
    } else {
        const int i = w - r;
        return (unsigned)i < (unsigned)P ? (double)fac[((long long)p * 3 + a) * PS + i] : 0.0;
    }
}

// The same sum over particle p's own stencil alone, one cell after the other:
// value q (potential, fx, fy, fz).
template <bool TILED, typename T>
__device__ __noinline__ double interp3_direct(const SysDev& S, const double* __restrict__ gs,
                                              const T* __restrict__ fac, int PS, int p, int pk, double4 rc, int q)
{
    const int P = S.P, M = S.M;
    auto weight = [&](int a, int i) -> double {
        const double f = TILED ? (double)fac[(long long)p * 96 + 32 * a + (g_of(pk, a) & 15) + i]
                               : (double)fac[((long long)p * 3 + a) * PS + i];
        const double u = a == 0 ? rc.x : (a == 1 ? rc.y : rc.z);
        return q == a + 1 ? f * (-S.c * (u - (S.lo + i) * S.h)) : f;
    };
    double sum = 0.0;
    for (int i = 0; i < P; i++) {
        double sx = 0.0;
        for (int j = 0; j < P; j++) {
            const double* row =
                gs + ((long long)((g_of(pk, 0) + i) % M) * M + (g_of(pk, 1) + j) % M) * M;
            double sy = 0.0;
            for (int k = 0; k < P; k++) sy += row[(g_of(pk, 2) + k) % M] * weight(2, k);
            sx += sy * weight(1, j);
        }
        sum += sx * weight(0, i);
    }
    return sum;
}

// CTAs per SM the kernel is compiled for: potentials of deep contractions do better with
// the registers (200,000 particles, M = 100, potential, 7 and 5 CTAs: P = 20 482 and
// 486 us, P = 24 618 and 587, P = 32 1137 and 1095; force, 4 and 3: P = 24 960 and 984)
__host__ __device__ constexpr int interp3_ctas(int NK, bool force) { return force ? 4 : (NK >= 8 ? 5 : 7); }

// SHARE (launches of few groups, in chunks of 8): the z tiles of one or two groups go
// over all the warps
template <int NK, bool FORCE, bool TILED, bool SHARE, typename T>
__global__ void __launch_bounds__(I3_WARPS * 32, interp3_ctas(NK, FORCE)) k_interp3(
    const SysDev* __restrict__ sys, const int* __restrict__ part_prefix, int nsys, const int* __restrict__ tab,
    int units, int chunk, int P, const double4* __restrict__ srec, const int* __restrict__ sg,
    const int* __restrict__ sperm, const T* __restrict__ fac, int PS,
    const int* __restrict__ boff, const double* __restrict__ grid, double* __restrict__ out,
    double* __restrict__ phi_out)
{
    constexpr int XE = 4 * NK + 2 * interp3_nx(FORCE, 1);
    __shared__ unsigned char order[I3_PART];
    __shared__ int start[2 * FB + 1];
    __shared__ int xoff[XE];
    __shared__ __align__(16) double wtab[I3_WARPS][FORCE ? 2 : 1][XE][8];   // the warps' x weights
    // the tiles' sums of every lane of shared groups
    __shared__ double part[SHARE ? 2 : 1][SHARE ? (NK + 1) / 2 : 1][FORCE ? 6 : 2][32];
    // ---- the CTA's particles [c0, c0 + n) of one bin, at most `chunk`
    const int unit = blockIdx.x;
    int c0, n, sysi, bin;
    if (unit < units) {   // the first of unit's bin
        bin = __ldg(tab + units + unit);
        sysi = __ldg(tab + unit);
        c0 = boff[bin];
        n = min(chunk, boff[bin + 1] - c0);
    } else {   // of the sorted particles [s0, s0 + chunk) those past the
               // first `chunk` of the bin that holds s0
        const int s0 = (unit - units) * chunk;
        sysi = find_sys(part_prefix, nsys, sperm[s0]);
        const SysDev& S = sys[sysi];
        if (S.P != P || S.mode != (FORCE ? SE_FORCE : SE_POTENTIAL) ||
            ((S.path & PATH_PAIR_INTERP) != 0) != TILED || !S.interp3)
            return;   // another launch's system, or another kernel's
        const int pk = sg[s0];
        bin = S.bin_base + (g_of(pk, 0) / FB * S.nf[1] + g_of(pk, 1) / FB) * S.nf[2] + g_of(pk, 2) / FB;
        c0 = max(boff[bin] + chunk, s0);
        n = min(boff[bin + 1], s0 + chunk) - c0;
    }
    if (n <= 0) return;
    const SysDev& S = sys[sysi];
    const int lb = bin - S.bin_base, M = S.M;
    const int o0 = (lb / (S.nf[1] * S.nf[2])) * FB, o1 = ((lb / S.nf[2]) % S.nf[1]) * FB,
              o2 = (lb % S.nf[2]) * FB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const double* gs = grid + S.grid_off;
    auto wrap = [&](int i) { return TILED ? (i >= M ? i - M : i) : i % M; };
    for (int x = threadIdx.x; x < XE; x += blockDim.x) xoff[x] = wrap(o0 + x) * M * M;
    int yoff[NK];
#pragma unroll
    for (int k = 0; k < NK; k++) yoff[k] = wrap(o1 + 4 * k + t) * M;
    const double c = S.c, h = S.h;
    const int hx = o0 & 8, hy = o1 & 8, hz = o2 & 8;
    const int nz = (FB + P + 6) / 8;
    double(*wx)[8] = wtab[warp][0], (*fx)[8] = wtab[warp][FORCE ? 1 : 0];

    // ---- the particles ordered by whether their stencil reaches the last z
    // tile and by x offset: the groups of 8 then span few x and often leave
    // that tile out (any order does: a particle's sums do not depend on its
    // group)
    const bool by_tile = n >= I3_BY_TILE && 8 * (nz - 1) - P >= 2;
    auto rank = [&](int i) {
        const int pk = sg[c0 + i];
        return (by_tile && g_of(pk, 2) - o2 + P > 8 * (nz - 1) ? FB : 0) + g_of(pk, 0) - o0;
    };
    if (n > 8) {
        if (threadIdx.x <= 2 * FB) start[threadIdx.x] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&start[rank(i) + 1], 1);
        __syncthreads();
        if (threadIdx.x == 0)
            for (int i = 1; i < 2 * FB; i++) start[i] += start[i - 1];
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) order[atomicAdd(&start[rank(i)], 1)] = (unsigned char)i;
    } else if (threadIdx.x < n) {
        order[threadIdx.x] = threadIdx.x;
    }
    __syncthreads();
    {
        const int share = !SHARE ? 1 : (n <= 8 ? I3_WARPS : (n <= 16 ? I3_WARPS / 2 : 1));
        for (int g0 = 8 * (warp / share); g0 < n; g0 += 8 * I3_WARPS / share) {
            // ---- the group's weights.  Lane (g, t): y weights of particle g
            // at y = 4 k + t; x weights in shared memory; z weights of
            // particles 2 t, 2 t + 1 at z = 8 i + g (below)
            const bool valid = g0 + g < n;
            const int p = c0 + order[min(g0 + g, n - 1)];
            const int pk = sg[p];
            const double4 rc = srec[p];
            const int rx = g_of(pk, 0) - o0, ry = g_of(pk, 1) - o1, rz = g_of(pk, 2) - o2;
            double by[NK], fy[FORCE ? NK : 1];
            const double uy = fma(-(double)(S.lo - ry), h, rc.y);
#pragma unroll
            for (int k = 0; k < NK; k++) {
                by[k] = valid ? interp3_factor<TILED>(fac, PS, P, p, 1, 4 * k + t, ry, hy) : 0.0;
                if (FORCE) fy[k] = by[k] * (-c * fma(-(double)(4 * k + t), h, uy));
            }
            int xlo = rx, xhi = rx + P;
            {
                const int src = (lane & 7) * 4;
                const int pn = __shfl_sync(0xffffffffu, p, src);
                const int rn = __shfl_sync(0xffffffffu, rx, src);
                const double ux = fma(-(double)(S.lo - rn), h, __shfl_sync(0xffffffffu, rc.x, src));
                for (int x = lane >> 3; x < XE; x += 4) {
                    const double w = x < 4 * NK ? interp3_factor<TILED>(fac, PS, P, pn, 0, x, rn, hx) : 0.0;
                    wx[x][lane & 7] = w;
                    if (FORCE) fx[x][lane & 7] = w * (-c * fma(-(double)x, h, ux));
                }
                xlo = __reduce_min_sync(0xffffffffu, xlo);
                xhi = __reduce_max_sync(0xffffffffu, xhi);
            }
            int pz[2], rzn[2];
            double uz[2];
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const int src = (2 * t + b) * 4;
                pz[b] = __shfl_sync(0xffffffffu, p, src);
                rzn[b] = __shfl_sync(0xffffffffu, rz, src);
                uz[b] = fma(-(double)(S.lo - rzn[b]), h, __shfl_sync(0xffffffffu, rc.z, src));
            }
            __syncwarp();
            const int ztop = __reduce_max_sync(0xffffffffu, rz) + P;
            double s[2][4] = {};
            // the sums over x at the lane's cell z of a tile, with the z weights
            auto add_tile = [&](int z, const double (&ap)[2], const double (&ax)[2], const double (&ay)[2]) {
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    const double wz = interp3_factor<TILED>(fac, PS, P, pz[b], 2, z, rzn[b], hz);
                    s[b][0] = fma(wz, ap[b], s[b][0]);
                    if (FORCE) {
                        s[b][1] = fma(wz, ax[b], s[b][1]);
                        s[b][2] = fma(wz, ay[b], s[b][2]);
                        s[b][3] = fma(wz * (-c * fma(-(double)z, h, uz[b])), ap[b], s[b][3]);
                    }
                }
            };
            // U[z][particle] = sum_y H[x][y][z] wy of NX planes x and NT z
            // tiles, then the sums over x with the x weights.  Two tiles
            // share 16-byte loads: the rows of the first are the even z of
            // their 16, those of the second the odd ones
            auto tiles = [&](int i, auto nt) {
                constexpr int NT = decltype(nt)::value, NX = interp3_nx(FORCE, NT);
                const double* col = gs + wrap(o2 + 8 * i + NT * g);
                double ap[NT][2] = {}, ax[NT][2] = {}, ay[NT][2] = {};
                double a[NX][NK][NT];
                auto load = [&](int x, int j, int k) {
                    const double* cell = col + xoff[x + j] + yoff[k];
                    if constexpr (NT == 2) {
                        const double2 w = __ldg(reinterpret_cast<const double2*>(cell));
                        a[j][k][0] = w.x;
                        a[j][k][1] = w.y;
                    } else {
                        a[j][k][0] = __ldg(cell);
                    }
                };
                auto load_all = [&](int x) {
#pragma unroll
                    for (int k = 0; k < NK; k++)
#pragma unroll
                        for (int j = 0; j < NX; j++) load(x, j, k);
                };
                if (FORCE) load_all(xlo);
#pragma unroll 1
                for (int x = xlo; x < xhi; x += NX) {
                    if (!FORCE) load_all(x);
                    double u[NX][NT][2] = {}, v[FORCE ? NX : 1][NT][2] = {};
#pragma unroll
                    for (int k = 0; k < NK; k++) {
#pragma unroll
                        for (int j = 0; j < NX; j++) {
#pragma unroll
                            for (int m = 0; m < NT; m++) {
                                mma_f64(u[j][m][0], u[j][m][1], a[j][k][m], by[k]);
                                if (FORCE) mma_f64(v[j][m][0], v[j][m][1], a[j][k][m], fy[k]);
                            }
                        }
                        // the operands of the next planes take their place
                        // (past the window: read, not used)
                        if (FORCE) {
#pragma unroll
                            for (int j = 0; j < NX; j++) load(x + NX, j, k);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < NX; j++) {
                        const double2 w = *reinterpret_cast<const double2*>(&wx[x + j][2 * t]);
                        double2 f = make_double2(0.0, 0.0);
                        if (FORCE) f = *reinterpret_cast<const double2*>(&fx[x + j][2 * t]);
#pragma unroll
                        for (int m = 0; m < NT; m++) {
                            ap[m][0] = fma(w.x, u[j][m][0], ap[m][0]);
                            ap[m][1] = fma(w.y, u[j][m][1], ap[m][1]);
                            if (FORCE) {
                                ax[m][0] = fma(f.x, u[j][m][0], ax[m][0]);
                                ax[m][1] = fma(f.y, u[j][m][1], ax[m][1]);
                                ay[m][0] = fma(w.x, v[j][m][0], ay[m][0]);
                                ay[m][1] = fma(w.y, v[j][m][1], ay[m][1]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < NT; m++) {
                    if (share == 1) {
                        add_tile(8 * i + NT * g + m, ap[m], ax[m], ay[m]);
                        continue;
                    }
                    double(*pt)[32] = part[SHARE ? g0 / 8 : 0][SHARE ? i + m : 0];
                    pt[0][lane] = ap[m][0];
                    pt[1][lane] = ap[m][1];
                    if (FORCE) {
                        pt[2][lane] = ax[m][0];
                        pt[3][lane] = ax[m][1];
                        pt[4][lane] = ay[m][0];
                        pt[5][lane] = ay[m][1];
                    }
                }
            };
            // the tiles two at a time where rows are 16-byte aligned and do
            // not wrap inside a pair of cells (even M), the last of an odd
            // number alone; those that no stencil of the group reaches add
            // nothing and are left out
            const int pairs = M % 2 == 0 ? nz / 2 : 0;
            for (int i = warp % share; i < nz - pairs; i += share) {
                if (i < pairs) {
                    if (16 * i < ztop) tiles(2 * i, std::integral_constant<int, 2>());
                } else if (8 * (pairs + i) < ztop) {
                    tiles(pairs + i, std::integral_constant<int, 1>());
                }
            }
            if (share > 1) {   // the group's first warp adds the tiles, in order
                __syncthreads();   // (one round: every warp gets here once)
                if (warp % share != 0) continue;
                for (int i = 0; i < nz; i++) {
                    const bool paired = i < 2 * pairs;
                    if (8 * (paired ? i & ~1 : i) >= ztop) break;
                    const double(*pt)[32] = part[SHARE ? g0 / 8 : 0][SHARE ? i : 0];
                    const double ap[2] = {pt[0][lane], pt[1][lane]};
                    double ax[2] = {0, 0}, ay[2] = {0, 0};
                    if (FORCE) {
                        ax[0] = pt[2][lane];
                        ax[1] = pt[3][lane];
                        ay[0] = pt[4][lane];
                        ay[1] = pt[5][lane];
                    }
                    add_tile(paired ? 16 * (i / 2) + 2 * g + i % 2 : 8 * i + g, ap, ax, ay);
                }
            }
            // ---- the sums over the 8 lanes of each particle pair, by halving:
            // lane (g, t) ends with value g & 3 (potential, fx, fy, fz) of
            // particle 2 t + (g >> 2)
            const bool g2 = g & 4, g1 = g & 2, g0b = g & 1;
            double r[4];
#pragma unroll
            for (int q = 0; q < (FORCE ? 4 : 1); q++)
                r[q] = (g2 ? s[1][q] : s[0][q]) + __shfl_xor_sync(0xffffffffu, g2 ? s[0][q] : s[1][q], 16);
            double val;
            if (FORCE) {
                const double m0 = (g1 ? r[2] : r[0]) + __shfl_xor_sync(0xffffffffu, g1 ? r[0] : r[2], 8);
                const double m1 = (g1 ? r[3] : r[1]) + __shfl_xor_sync(0xffffffffu, g1 ? r[1] : r[3], 8);
                val = (g0b ? m1 : m0) + __shfl_xor_sync(0xffffffffu, g0b ? m0 : m1, 4);
            } else {
                val = r[0] + __shfl_xor_sync(0xffffffffu, r[0], 8);
                val += __shfl_xor_sync(0xffffffffu, val, 4);
            }
            const int ip = 2 * t + (g >> 2), q = FORCE ? g & 3 : 0;
            if (g0 + ip < n && (FORCE || (g & 3) == 0)) {
                const int pm = c0 + order[g0 + ip];
                const int loc = sperm[pm] - S.part_off;
                const double scale = S.h3 * S.d;
                if (!isfinite(val)) val = interp3_direct<TILED>(S, gs, fac, PS, pm, sg[pm], srec[pm], q);
                if (q == 0) {
                    double* dst = FORCE ? phi_out : out;
                    if (dst) dst[(FORCE ? S.part_off : S.out_off) + loc] = scale * val;
                } else {
                    out[S.out_off + loc + (long long)(q - 1) * S.N] = srec[pm].w / S.d * scale * val;
                }
            }
            __syncwarp();   // the x weights are read before the next group's
        }
    }
}

// The same sums, a particle per warp: in sparse bins the groups above hold one or two
// particles and cost as much as with 8.  A lane takes a z cell of the stencil and
// walks its y and x cells in k_interp3's order (the cells it leaves out have zero
// weights), so the results are the same bits.  Bound by the latency of its loads, 8
// in flight: 2,300 particles, M = 250, P = 21, potential 123 us (the cells past a
// multiple of 8 one after the other 169); with 16, four planes at a time, 10,000, M =
// 100, P = 24 176 for 140.
template <bool FORCE, bool TILED, typename T>
__global__ void __launch_bounds__(I3_WARPS * 32) k_interp3_sparse(
    const SysDev* __restrict__ sys, const int* __restrict__ part_prefix, int nsys, int ntot, int P,
    const double4* __restrict__ srec, const int* __restrict__ sg, const int* __restrict__ sperm,
    const T* __restrict__ fac, int PS, const double* __restrict__ grid, double* __restrict__ out,
    double* __restrict__ phi_out)
{
    constexpr int E = 40;   // cells of the widest window, whole z tiles
    __shared__ double2 wxs[I3_WARPS][32], wys[I3_WARPS][32];   // weights, force weights
    __shared__ int yos[I3_WARPS][32], xos[I3_WARPS][32];
    __shared__ double sums[I3_WARPS][FORCE ? 3 : 1][E];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * I3_WARPS + warp;
    if (p >= ntot) return;
    const int orig = sperm[p];
    const SysDev& S = sys[find_sys(part_prefix, nsys, orig)];
    if (S.P != P || S.mode != (FORCE ? SE_FORCE : SE_POTENTIAL) || ((S.path & PATH_PAIR_INTERP) != 0) != TILED ||
        !S.interp3)
        return;
    const int M = S.M, pk = sg[p];
    const double4 rc = srec[p];
    const double c = S.c, h = S.h;
    const double* gs = grid + S.grid_off;
    // the stencil's first cell in the bin's window, per axis
    const int rx = g_of(pk, 0) % FB, ry = g_of(pk, 1) % FB, rz = g_of(pk, 2) % FB;
    const int hx = g_of(pk, 0) - rx & 8, hy = g_of(pk, 1) - ry & 8, hz = g_of(pk, 2) - rz & 8;
    if (lane < P) {
        const int x = rx + lane, y = ry + lane;
        const double wx = interp3_factor<TILED>(fac, PS, P, p, 0, x, rx, hx);
        const double wy = interp3_factor<TILED>(fac, PS, P, p, 1, y, ry, hy);
        const double ux = fma(-(double)(S.lo - rx), h, rc.x), uy = fma(-(double)(S.lo - ry), h, rc.y);
        wxs[warp][lane] = make_double2(wx, wx * (-c * fma(-(double)x, h, ux)));
        wys[warp][lane] = make_double2(wy, wy * (-c * fma(-(double)y, h, uy)));
        xos[warp][lane] = (g_of(pk, 0) + lane) % M * M * M;
        yos[warp][lane] = (g_of(pk, 1) + lane) % M * M;
    } else {
        wys[warp][lane] = make_double2(0.0, 0.0);
    }
    for (int z = lane; z < E; z += 32)
        for (int q = 0; q < (FORCE ? 3 : 1); q++) sums[warp][q][z] = 0.0;
    __syncwarp();
    if (lane < P) {
        const double* col = gs + (g_of(pk, 2) + lane) % M;
        double ap = 0, ax = 0, ay = 0;
        for (int x = 0; x < P; x++) {
            const double* plane = col + xos[warp][x];
            double u = 0, v = 0;
            for (int y0 = 0; y0 < P; y0 += 8) {
                double cell[8];
#pragma unroll
                for (int k = 0; k < 8; k++) cell[k] = y0 + k < P ? __ldg(plane + yos[warp][y0 + k]) : 0.0;
#pragma unroll
                for (int k = 0; k < 8; k++) {   // (past the stencil: zero times zero)
                    const double2 w = wys[warp][y0 + k];
                    u = fma(cell[k], w.x, u);
                    if (FORCE) v = fma(cell[k], w.y, v);
                }
            }
            const double2 w = wxs[warp][x];
            ap = fma(w.x, u, ap);
            if (FORCE) {
                ax = fma(w.y, u, ax);
                ay = fma(w.x, v, ay);
            }
        }
        sums[warp][0][rz + lane] = ap;
        if (FORCE) {
            sums[warp][FORCE ? 1 : 0][rz + lane] = ax;
            sums[warp][FORCE ? 2 : 0][rz + lane] = ay;
        }
    }
    __syncwarp();
    // the sums over z: lane g < 8 the cells that k_interp3's lanes (g, t) hold, then the
    // same halving
    const int g = lane & 7, nz = (FB + P + 6) / 8, pairs = M % 2 == 0 ? nz / 2 : 0;
    const double uz = fma(-(double)(S.lo - rz), h, rc.z);
    double s[4] = {};
    for (int i = 0; i < nz; i++) {
        const int z = i < 2 * pairs ? 16 * (i / 2) + 2 * g + i % 2 : 8 * i + g;
        const double wz = interp3_factor<TILED>(fac, PS, P, p, 2, z, rz, hz);
        s[0] = fma(wz, sums[warp][0][z], s[0]);
        if (FORCE) {
            s[1] = fma(wz, sums[warp][FORCE ? 1 : 0][z], s[1]);
            s[2] = fma(wz, sums[warp][FORCE ? 2 : 0][z], s[2]);
            s[3] = fma(wz * (-c * fma(-(double)z, h, uz)), sums[warp][0][z], s[3]);
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < (FORCE ? 4 : 1); q++) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
    if (lane < (FORCE ? 4 : 1)) {
        double val = lane == 0 ? s[0] : (lane == 1 ? s[1] : (lane == 2 ? s[2] : s[3]));
        if (!isfinite(val)) val = interp3_direct<TILED>(S, gs, fac, PS, p, pk, rc, lane);
        const int loc = orig - S.part_off;
        const double scale = S.h3 * S.d;
        if (lane == 0) {
            double* dst = FORCE ? phi_out : out;
            if (dst) dst[(FORCE ? S.part_off : S.out_off) + loc] = scale * val;
        } else {
            out[S.out_off + loc + (long long)(lane - 1) * S.N] = rc.w / S.d * scale * val;
        }
    }
}

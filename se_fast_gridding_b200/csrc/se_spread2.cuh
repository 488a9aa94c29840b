// se_spread2.cuh -- the spread (SE_FGG_grid, SE_fgg.c:3866-4028) with the
// periodic fold (SE_FGG_wrap_fcn, SE_fgg.c:327-352) fused, for the systems
// whose grid is cut into whole 16^3 tiles (M a multiple of 16, M >= 32) and
// whose stencil fits two tiles (P <= 16), and, on P-wide factor rows (GEN, at
// the kernel), for all others but the smallest grids.  Included inside namespace se by
// se_solve.cu after se_spread.cuh (whose bin-range helpers it uses).
//
// Factor rows aligned to tiles.  k_factors writes, per particle and axis, a
// 32-entry row R[j] = f[j - s] (zero outside the stencil), where s = g mod 16
// is the stencil's start inside its home tile g / 16.  A stencil covers at
// most the home tile and the next one (periodically), and the row of tile
// home + h is R[16h .. 16h + 15]: one aligned 64-byte copy, no wrap logic.
//
// One CTA of 4 warps owns one 16^3 tile; warp w = 2 wy + wz owns the
// 16 x 8 x 8 block of y in 8 wy + [0, 8) and z in 8 wz + [0, 8), and the
// warps run independently, with no CTA barrier.  A warp lists the bin
// segments whose particles may reach its block (the tile's 16 x cells, its
// own 8 y and 8 z: at most 5 x 4 x 2 segments), walks their candidates in
// order, keeps the particles whose stencil meets the block and sorts them
// into three x classes -- the particle's x row in the tile meets both 8-cell
// halves, the low half only or the high half only -- one list ring each.
// Whenever a class holds a group the warp streams it
// through two shared-memory stages that cp.async fills from the factor rows
// while the warp works on the other: the x tile row (of a one-half class,
// that half), the warp's 8 y and 8 z entries and the charge, consecutive lanes
// copying consecutive pieces of a row; the next 32 candidates' corners are
// loaded meanwhile.  (With a particle's pieces copied by one lane, and the
// corners loaded when they were needed, a group's set-up took as long as its
// sums: 100,000 particles, M = 128, P = 16, stage 0.130 -> 0.116 ms; 16M
// clustered, M = 512, P = 12, 11.0 -> 10.1 ms; 256 systems of M = 64 2.37 ->
// 2.10 ms.)  A one-half group costs half the FMAs of a full one, and a particle
// is a one-half particle in about half of the tiles it meets at P = 16 (more at
// smaller P).  Every cell belongs to one lane of one CTA: no atomics and a fixed
// order of summation (the groups' order, which depends only on the block's
// candidate list).
// FP32: each lane adds px[x] * (q py[y] pz[z]) into the 16 x 2 cells of its
// (y, z) and (y, z + 1), or the 8 x 2 of the class's half, with packed FP32 pair
// FMAs, and after every 512 of the warp's particles the FP32 sums are added into
// the FP64 grid in place (the first time stored), which the lane alone reads
// and writes.
// FP64: matrix instructions, 4 particles onto 8 x by 8 z cells of one y, with
// the cells' sums in the accumulators (64 registers).  They run at the rate of
// scalar FP64 FMAs but need a fraction of the instructions and shared-memory
// loads: 100,000 particles, M = 128, P = 16 0.240 -> 0.142 ms (the matrix unit's
// share 0.066 ms, 0.094 with the products that feed it); 1M, M = 256, P = 12 1.10
// -> 0.63 ms, P = 8 0.59 -> 0.33 ms; 2M clustered 3.49 -> 2.23 ms.  (For FP32 the
// same products on FP64 units, 0.145 ms, or on BF16 units with 24 bits in three
// parts, 0.148 ms, lose to packed FMAs: splitting the operands costs more
// instructions than the FMAs.)
//
// Crowded tiles are split.  Each warp's candidate list is cut into parts of
// at most S2_CAP candidates (split_cap); k_tile_parts counts the candidates of each
// tile's most crowded block and scans the part counts, and k_spread2 runs
// one CTA per part, whose warps take part s of their own lists.  Part 0
// writes the tile into the grid as above; part s >= 1 writes its sums into
// slab slot (extra parts of the tiles before it) + s - 1, 16^3 FP64 cells;
// the part that finishes last (a per-tile counter) adds the slabs into the
// grid in the order s = 1, 2, ...  A tile's parts and their sums depend only
// on its own candidates, so results stay deterministic and a batched
// system's grid equals its single solve's.  Uniform inputs at the
// configurations' densities have far fewer than S2_CAP candidates per block
// and are never split.

#ifndef SE_S2_CAP
#define SE_S2_CAP 8192
#endif
#ifndef SE_S2_UNROLL
#define SE_S2_UNROLL 16
#endif
constexpr int S2_CAP = SE_S2_CAP;   // candidates per part of a warp's list
// ... and of a system of N particles: at least `least`, and as many as make at most
// `most` parts of all of them.  Off the whole tiles, where a particle is a candidate
// of up to 4^3 tiles, 512 parts bound the slabs.  Where every block sees every
// particle (M <= P + 15: at most 27 tiles, which leave the chip idle) parts of 512
// from 1,025 particles on, or of N / 64: M = 32, P = 21, FP64 spread, 5,100 particles
// 0.467 -> 0.122 ms; 1,024 (not split) 0.105, 1,088 0.098 (with parts of 1,024 0.128)
struct SplitRule {
    int least, most;   // most <= least
};
__host__ __device__ inline SplitRule split_rule(int path, int M, int P, int N)
{
    if (path & PATH_TILE_SPREAD) return {S2_CAP, 0};   // any number of parts
    return M <= P + 15 && N > 1024 ? SplitRule{512, 64} : SplitRule{S2_CAP, 512};
}
__host__ __device__ inline int split_cap(int path, int M, int P, int N)
{
    const SplitRule r = split_rule(path, M, P, N);
    const int even = r.most ? N / r.most : 0;
    return even < r.least ? r.least : even;
}
constexpr int S2_WARPS = 4;   // warp blocks per tile
// warps per CTA: a tile's four warp blocks run as S2_WARPS / CW CTAs (the warps
// are independent), so that the SMs share out the blocks more evenly: one warp
// in FP32 (against two: 1M uniform, M = 256, P = 12 0.548 -> 0.529 ms, 256
// systems of M = 64 2.10 -> 2.05 ms, 16M clustered no difference), two in FP64
// (2M clustered 2.28 -> 2.23 ms)
template <typename F, bool GEN>
constexpr bool s2_fp32_sums() { return sizeof(F) == 4 && !GEN; }
template <typename F, bool GEN>
constexpr int s2_cta_warps() { return s2_fp32_sums<F, GEN>() ? 1 : 2; }
constexpr int S2_LIST = 64;    // per-class list ring: >= group - 1 + 32
// bin segments reaching a warp's block: <= 5 x 4 x 2 on whole tiles (P <= 16),
// <= 8 x 7 x 2 otherwise (P <= 32, the last bin of an axis cut)
template <bool GEN>
constexpr int s2_segs() { return GEN ? 112 : 40; }
constexpr int S2_FOLD = 512;   // FP32 partial sums cover this many of a warp's particles
// x classes of a particle in a tile: its x row meets both 8-cell halves,
// the low half only, the high half only
constexpr int S2_CLASSES = 3;
constexpr int S2_UNROLL = SE_S2_UNROLL;   // particles per unrolled pass of a group
// FP32 CTAs per SM the kernel is compiled for: 5 (96 registers) where the
// tiles outnumber 4 CTAs per SM, 4 (128 registers) where all of them are
// resident at once either way; FP64 sums: 4
constexpr int S2_BLOCKS_MANY = 5, S2_BLOCKS_FEW = 4, S2_BLOCKS_FP64 = 4;

// particles a warp stages at once: one per lane (FP32 sums), half a warp (FP64)
template <typename F, bool GEN>
constexpr int s2_group() { return s2_fp32_sums<F, GEN>() ? 32 : 16; }

template <typename F, bool GEN>
struct Spread2Stage {
    F px[s2_group<F, GEN>()][16];
    F pz[s2_group<F, GEN>()][8];
    F py[s2_group<F, GEN>()][8];
    double q[s2_group<F, GEN>()];
};

// Where entry x of staged particle k's x row and entry z of its y and z rows
// lie in the row: for the matrix instructions moved (whole 32-byte groups) so that
// a warp's operand loads, 8 entries of 4 consecutive particles, fall in distinct
// banks.
template <typename F, bool GEN>
__device__ __forceinline__ int s2_px(int k, int x)
{
    if (sizeof(F) == 4) return GEN ? x ^ (((k >> 1) & 1) << 3) : x;
    return x ^ ((k & 3) << 2);
}

template <typename F>
__device__ __forceinline__ int s2_pz(int k, int z)
{
    return sizeof(F) == 4 ? z : z ^ (((k >> 1) & 1) << 2);
}

// A listed particle: 8 particle + 4 hx + 2 hy + hz, the halves of its
// tile-aligned rows; on the P-wide rows (GEN) the particle and its stencil's
// entries at the first x of both 8-cell halves and the block's first y and z, plus
// 8, a byte each.
template <bool GEN>
struct Spread2Entry {
    using Type = unsigned;
};
template <>
struct Spread2Entry<true> {
    using Type = uint2;
};

template <typename F, int CW, bool GEN>
struct Spread2Smem {
    Spread2Stage<F, GEN> stage[CW][2];
    typename Spread2Entry<GEN>::Type list[CW][S2_CLASSES][S2_LIST];
    int seg_beg[CW][s2_segs<GEN>()];
    int seg_pre[CW][s2_segs<GEN>()];
};

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc) : "memory");
}

__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gsrc) : "memory");
}

// 16 bytes, or 16 zero bytes where !on (gsrc is then not read)
__device__ __forceinline__ void cp_async16_or_zero(void* sdst, const void* gsrc, bool on)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gsrc), "r"(on ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_async_one_or_zero(float* sdst, const float* gsrc, bool on)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(gsrc), "r"(on ? 4 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_async8_or_zero(void* sdst, const void* gsrc, bool on)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(gsrc), "r"(on ? 8 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_async_one_or_zero(double* sdst, const double* gsrc, bool on)
{
    cp_async8_or_zero(sdst, gsrc, on);
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// A warp's sums: 16 x 8 x 8 cells, 32 per lane.
template <typename Acc>
struct Spread2Accum;

// FP32: 16 x for z and for z + 1.
template <>
struct Spread2Accum<float> {
    float2 a[8], b[8];   // packed x pairs for z and z + 1
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int m = 0; m < 8; m++) a[m] = b[m] = make_float2(0.f, 0.f);
    }
    __device__ __forceinline__ void add(const float* px, float c0, float c1)
    {
        const float2 k0 = f32x2(c0, c0), k1 = f32x2(c1, c1);
        const float4* p4 = reinterpret_cast<const float4*>(px);
#pragma unroll
        for (int m = 0; m < 4; m++) {
            float2 lo, hi;
            f32x2_split(p4[m], lo, hi);
            a[2 * m] = ffma2(lo, k0, a[2 * m]);
            a[2 * m + 1] = ffma2(hi, k0, a[2 * m + 1]);
            b[2 * m] = ffma2(lo, k1, b[2 * m]);
            b[2 * m + 1] = ffma2(hi, k1, b[2 * m + 1]);
        }
    }
    // x in [8 H, 8 H + 8) only (the row is zero on the other half)
    template <int H>
    __device__ __forceinline__ void add_half(const float* px, float c0, float c1)
    {
        const float2 k0 = f32x2(c0, c0), k1 = f32x2(c1, c1);
        const float4* p4 = reinterpret_cast<const float4*>(px);
#pragma unroll
        for (int m = 2 * H; m < 2 * H + 2; m++) {
            float2 lo, hi;
            f32x2_split(p4[m], lo, hi);
            a[2 * m] = ffma2(lo, k0, a[2 * m]);
            a[2 * m + 1] = ffma2(hi, k0, a[2 * m + 1]);
            b[2 * m] = ffma2(lo, k1, b[2 * m]);
            b[2 * m + 1] = ffma2(hi, k1, b[2 * m + 1]);
        }
    }
    // cell (x, z + zz) at cell0 + x * plane + zz: the FP64 grid value plus
    // this lane's FP32 partial sums (or the sums alone the first time)
    __device__ __forceinline__ void fold(double* cell0, long long plane, bool first)
    {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            double2 old[8];
#pragma unroll
            for (int k = 0; k < 8; k++)
                old[k] = first ? make_double2(0.0, 0.0)
                               : *reinterpret_cast<const double2*>(cell0 + (8 * h + k) * plane);
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const int m = 4 * h + k / 2;
                const float2 u = a[m], v = b[m];
                *reinterpret_cast<double2*>(cell0 + (8 * h + k) * plane) =
                    make_double2(old[k].x + (double)u.x, old[k].y + (double)v.x);
                *reinterpret_cast<double2*>(cell0 + (8 * h + k + 1) * plane) =
                    make_double2(old[k + 1].x + (double)u.y, old[k + 1].y + (double)v.y);
                a[m] = b[m] = make_float2(0.f, 0.f);
            }
        }
    }
};

// The cells of a block that lie on the grid: x < nx from the lane's first
// cell on, y < ny and z < nz (nothing outside is stored).
struct BlockBounds {
    int nx, ny, nz;
};

// FP64: the cells of the warp's block as the matrix instructions spread them
// over a warp: with g = lane / 4 and t = lane % 4, x in {g, g + 8}, every y, z in
// {2 t, 2 t + 1}.  One instruction adds 4 particles to 8 x by 8 z cells of one y:
// D[x][z] += px[x] (py[y] (q pz[z])).
template <>
struct Spread2Accum<double> {
    double v[8][4];   // [y][x = g: z, z + 1; x = g + 8: z, z + 1]
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int y = 0; y < 8; y++)
#pragma unroll
            for (int k = 0; k < 4; k++) v[y][k] = 0.0;
    }
    // staged particles i .. i + 3, particle i + t the contraction's element t;
    // HALVES bit 0: x in [0, 8), bit 1: x in [8, 16)
    template <int HALVES, typename F, bool GEN>
    __device__ __forceinline__ void add(const Spread2Stage<F, GEN>& st, int i, int g, int t)
    {
        const int k = i + t;
        const double a0 = (HALVES & 1) ? (double)st.px[k][s2_px<F, GEN>(t, g)] : 0.0;
        const double a1 = (HALVES & 2) ? (double)st.px[k][s2_px<F, GEN>(t, g + 8)] : 0.0;
        const double pz = st.q[k] * (double)st.pz[k][s2_pz<F>(t, g)];
#pragma unroll
        for (int y = 0; y < 8; y += 2) {
            const auto py = *reinterpret_cast<const std::conditional_t<sizeof(F) == 4, float2, double2>*>(&st.py[k][s2_pz<F>(t, y)]);
            const double b0 = (double)py.x * pz, b1 = (double)py.y * pz;
            if (HALVES & 1) mma_f64(v[y][0], v[y][1], a0, b0);
            if (HALVES & 2) mma_f64(v[y][2], v[y][3], a1, b0);
            if (HALVES & 1) mma_f64(v[y + 1][0], v[y + 1][1], a0, b1);
            if (HALVES & 2) mma_f64(v[y + 1][2], v[y + 1][3], a1, b1);
        }
    }
    // the first n particles of the stage (zero rows up to a multiple of 4)
    template <int HALVES, typename F, bool GEN>
    __device__ __forceinline__ void add_group(const Spread2Stage<F, GEN>& st, int n, int g, int t)
    {
        constexpr int G = s2_group<F, GEN>();
        if (n == G) {
#pragma unroll
            for (int i = 0; i < G; i += 4) add<HALVES>(st, i, g, t);
        } else {
#pragma unroll 1
            for (int i = 0; i < n; i += 4) add<HALVES>(st, i, g, t);
        }
    }
    // cell (x, y, z) at cell0 + x plane + y row + z, cell0 that of the lane's
    // first x and z
    __device__ __forceinline__ void store(double* cell0, long long plane, int row) const
    {
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int y = 0; y < 8; y++)
                *reinterpret_cast<double2*>(cell0 + 8 * h * plane + y * row) =
                    make_double2(v[y][2 * h], v[y][2 * h + 1]);
    }
    // the same on a grid that may end inside the block; of an odd one (row) the rows
    // have any alignment, of an even one a lane's z and z + 1 are both on it or neither
    __device__ __forceinline__ void store(double* cell0, long long plane, int row, const BlockBounds& in) const
    {
        const bool even = row % 2 == 0;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int y = 0; y < 8; y++) {
                double* c = cell0 + 8 * h * plane + y * row;
                if (8 * h >= in.nx || y >= in.ny || in.nz <= 0) continue;
                if (even) {
                    *reinterpret_cast<double2*>(c) = make_double2(v[y][2 * h], v[y][2 * h + 1]);
                } else {
                    c[0] = v[y][2 * h];
                    if (in.nz > 1) c[1] = v[y][2 * h + 1];
                }
            }
    }
};

// The bins whose particles may reach block (wy, wz) of a tile at corner
// (x0, y0, z0) -- x: the tile's 16 cells, y and z: the block's 8 -- as
// segments (x bin, y bin, z run) numbered x-major; a z run is a contiguous
// range of bins, so a segment is a contiguous range of the sorted particles.
struct BlockBins {
    BinRanges rx, ry, rz;
    int nx, ny;
    __device__ __forceinline__ BlockBins(const SysDev& S, int x0, int y0, int z0)
        : rx(bins_reaching(x0, 16, S.M, S.P, S.nf[0])),
          ry(bins_reaching(y0, 8, S.M, S.P, S.nf[1])),
          rz(bins_reaching(z0, 8, S.M, S.P, S.nf[2])),
          nx(range_count(rx)), ny(range_count(ry))
    {
    }
    __device__ __forceinline__ int segments() const { return nx * ny * 2; }
    // the particles [beg, beg + len) of segment u
    __device__ __forceinline__ void segment(const SysDev& S, const int* __restrict__ boff, int u,
                                            int& beg, int& len) const
    {
        const int zr = u & 1, iy = (u >> 1) % ny, ix = (u >> 1) / ny;
        const int bz0 = zr ? rz.b0 : rz.a0, bz1 = zr ? rz.b1 : rz.a1;
        beg = 0;
        len = 0;
        if (bz0 <= bz1) {
            const int kb = S.bin_base + (range_at(rx, ix) * S.nf[1] + range_at(ry, iy)) * S.nf[2];
            beg = boff[kb + bz0];
            len = boff[kb + bz1 + 1] - beg;
        }
    }
};

// The number of candidates (the particles of the bin segments that reach
// it) of warp block w of tile lt of system S; every lane gets it.
__device__ __forceinline__ int block_candidates(const SysDev& S, int lt, int w,
                                                const int* __restrict__ boff, int lane)
{
    const int nt = S.nt[0];
    const int tix = lt / (nt * nt), tiy = (lt / nt) % nt, tiz = lt % nt;
    if (tiy * 16 + 8 * (w >> 1) >= S.M || tiz * 16 + 8 * (w & 1) >= S.M) return 0;
    const BlockBins B(S, tix * 16, tiy * 16 + 8 * (w >> 1), tiz * 16 + 8 * (w & 1));
    int sum = 0;
    for (int u = lane; u < B.segments(); u += 32) {
        int beg, len;
        B.segment(S, boff, u, beg, len);
        sum += len;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// Parts per tile (one warp per warp block, two tiles per CTA:
// max(1, ceil(candidates of the most crowded block / split_cap)) for the
// k_spread2 systems, 1 for the others), then, in the block that finishes
// last, their exclusive scan in place: parts[t] = the first part of tile t,
// parts[ntiles] = the number of parts, and part_tile[s] = the tile of part s.
// More parts than the launch bound (which no input reaches: split_slots) set
// bit 2 of err.  The block counter is left at zero for the next
// launch.
constexpr int TP_WARPS = 8;
constexpr int TP_TILES = TP_WARPS / S2_WARPS;   // tiles per CTA

__global__ void __launch_bounds__(TP_WARPS * 32) k_tile_parts(
    const SysDev* __restrict__ sys, const int* __restrict__ tile_prefix, int nsys, int ntiles,
    const int* __restrict__ boff, int* parts, unsigned* counter, int bound, int* err,
    int* __restrict__ part_tile)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x * TP_TILES + warp / S2_WARPS, wb = warp % S2_WARPS;
    __shared__ int cand[TP_WARPS];
    int c = 0, cap = S2_CAP;
    if (tile < ntiles) {
        const SysDev& S = sys[find_sys(tile_prefix, nsys, tile)];
        cap = split_cap(S.path, S.M, S.P, S.N);
        if ((S.path & PATH_TILE_SPREAD) || spread2_general(S.path, S.M, S.P))
            c = block_candidates(S, tile - S.tile_base, wb, boff, lane);
    }
    if (lane == 0) cand[warp] = c;
    __syncthreads();
    if (wb == 0 && lane == 0 && tile < ntiles) {
        int most = 0;
#pragma unroll
        for (int k = 0; k < S2_WARPS; k++) most = max(most, cand[warp + k]);
        parts[tile] = max(1, (most + cap - 1) / cap);
    }
    __shared__ int last;
    __shared__ int wsum[TP_WARPS];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    int carry = 0;
    for (int t0 = 0; t0 < ntiles; t0 += TP_WARPS * 32 * 4) {
        const int idx = t0 + threadIdx.x * 4;
        int v[4], sum = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[i] = idx + i < ntiles ? __ldcg(parts + idx + i) : 0;
            sum += v[i];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int before = 0, tot = 0;
#pragma unroll
        for (int w = 0; w < TP_WARPS; w++) {
            before += w < warp ? wsum[w] : 0;
            tot += wsum[w];
        }
        int run = carry + before + incl - sum;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (idx + i < ntiles) parts[idx + i] = run;
            run += v[i];
        }
        carry += tot;
        __syncthreads();   // wsum is reused
    }
    if (threadIdx.x == 0) {
        parts[ntiles] = carry;
        if (carry > bound) atomicOr(err, 2);
        *counter = 0u;
    }
    // every part's tile, for k_spread2 (the first `bound` parts)
    __syncthreads();
    for (int t = threadIdx.x; t < ntiles; t += blockDim.x) {
        const int a = __ldcg(parts + t), b = min(__ldcg(parts + t + 1), bound);
        for (int s = a; s < b; s++) part_tile[s] = t;
    }
}

// CW warps per CTA (S2_WARPS / CW CTAs per part of a tile); tile_parts null: no
// tile has a second part.  GEN: the systems of spread2_general, with rows the
// P-wide factor rows (PS entries apart), copied one entry at a time, tiles that may
// reach past the grid's end, and FP64 sums of FP32 factors too: as fast there as
// FP32 sums (58,600 particles, M = 100, P = 12: 0.115 ms both) and closer (a
// third of the error or less).  Against k_spread, which builds each chunk's rows
// per CTA, B200, FP64 spread stage: 58,600 particles, M = 100, P = 8 0.142 ->
// 0.069 ms, P = 12 0.292 -> 0.110, P = 24 0.837 -> 0.379; 3,900, P = 8 0.023 ->
// 0.016; 122,000, M = 250, P = 12 0.483 -> 0.183; 41,000, M = 128, P = 21 0.391 ->
// 0.142.  FP32 0.131 -> 0.071, 0.238 -> 0.115, 0.627 -> 0.396, 0.021 -> 0.016,
// 0.265 -> 0.185, 0.215 -> 0.146.  5,100, M = 32, P = 21 FP64 0.770 -> 0.467 (in parts
// 0.122).  Spread calls (sort and launches in them) of few particles: 53, M = 32, P =
// 24 39 -> 41 us, 12, M = 281, P = 28 FP32 105 -> 110, FP64 123 -> 111.
template <typename F, int BLOCKS, bool GEN = false, int CW = s2_cta_warps<F, GEN>()>
__global__ void __launch_bounds__(CW * 32, BLOCKS * (S2_WARPS / CW)) k_spread2(
    const SysDev* __restrict__ sys, const int* __restrict__ tile_sys,
    const double4* __restrict__ srec, const int* __restrict__ sg,
    const F* __restrict__ rows, int PS, const int* __restrict__ boff, double* __restrict__ grid,
    const int* __restrict__ tile_parts, const int* __restrict__ part_tile, int ntiles,
    int* __restrict__ tile_done, double* __restrict__ slab, int slab_slots,
    int* __restrict__ err)
{
    constexpr bool FOLD = s2_fp32_sums<F, GEN>();
    using Acc = std::conditional_t<FOLD, float, double>;
    constexpr int G = s2_group<F, GEN>();
    constexpr int V = 16 / sizeof(F);   // entries per 16-byte copy
    constexpr int S2_CTA_SPLIT = S2_WARPS / CW, S2_THREADS = CW * 32;
    __shared__ __align__(16) Spread2Smem<F, CW, GEN> sm;
    __shared__ int folds;   // this CTA finished its tile's parts last

    // ---- the part this CTA sums and its tile (k_tile_parts' part_tile; warp
    // blocks sub CW + [0, CW) of it), and the tile's system
    const int item = blockIdx.x / S2_CTA_SPLIT, sub = blockIdx.x % S2_CTA_SPLIT;
    int tile = item;
    if (tile_parts) {
        const int nall = tile_parts[ntiles];
        tile = part_tile[item];   // (the grid holds at most `bound` parts)
        if (item >= nall) return;
    }
    if ((unsigned)tile >= (unsigned)ntiles) {   // cannot happen: flagged, nothing summed
        if (threadIdx.x == 0) atomicOr(err, 2);
        return;
    }
    const int first = tile_parts ? tile_parts[tile] : tile;
    const int ipart = item - first;
    const int nparts = tile_parts ? tile_parts[tile + 1] - first : 1;
    const SysDev& S = sys[tile_sys[tile]];
    // the other variant or k_spread covers the other systems
    if (!(GEN ? spread2_general(S.path, S.M, S.P) : (S.path & PATH_TILE_SPREAD) != 0)) return;
    const int slot0 = first - tile;   // slab slot of part 1
    if (ipart > 0 && slot0 + ipart - 1 >= slab_slots) {   // cannot happen: see k_tile_parts
        if (threadIdx.x == 0) atomicOr(err, 2);
        return;
    }
    const int nt = S.nt[0], P = S.P, M = S.M;
    const int lt = tile - S.tile_base;
    const int tix = lt / (nt * nt), tiy = (lt / nt) % nt, tiz = lt % nt;
    const int x0 = tix * 16, y0 = tiy * 16, z0 = tiz * 16;
    const int t = threadIdx.x, lw = t >> 5, lane = t & 31;
    const int warp = sub * CW + lw;   // the warp block of the tile
    const int wy = warp >> 1, wz = warp & 1;
    const int ly = lane >> 2, lz = (lane & 3) * 2;

    // ---- the bin segments reaching this warp's block (at most 5 x 4 x 2) and
    // their prefix: the warp's own candidate list, in segment order
    const bool outside = GEN && (y0 + 8 * wy >= M || z0 + 8 * wz >= M);   // no cell of the block is on the grid
    const BlockBins B(S, x0, outside ? 0 : y0 + 8 * wy, outside ? 0 : z0 + 8 * wz);
    int nseg = outside ? 0 : B.segments();
    if (nseg > s2_segs<GEN>()) {   // cannot happen: flagged, the block sums nothing
        if (lane == 0) atomicOr(err, 2);
        nseg = 0;
    }
    int* seg_beg = sm.seg_beg[lw];
    int* seg_pre = sm.seg_pre[lw];
    int total = 0;
    auto scan = [&](int u, int beg, int len) {
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (u < nseg) {
            seg_beg[u] = beg;
            seg_pre[u] = total + incl - len;
        }
        total += __shfl_sync(0xffffffffu, incl, 31);
    };
    if constexpr (GEN) {
        constexpr int R = (s2_segs<GEN>() + 31) / 32;
        int beg[R], len[R], any = 0;
#pragma unroll
        for (int r = 0; r < R; r++) {   // (every load first)
            beg[r] = len[r] = 0;
            if (32 * r + lane < nseg) B.segment(S, boff, 32 * r + lane, beg[r], len[r]);
            any |= len[r];
        }
        if (!__any_sync(0xffffffffu, any)) nseg = 0;
        else
#pragma unroll
            for (int r = 0; r < R; r++) scan(32 * r + lane, beg[r], len[r]);
    } else {
        for (int u0 = 0; u0 < nseg; u0 += 32) {
            int beg = 0, len = 0;
            if (u0 + lane < nseg) B.segment(S, boff, u0 + lane, beg, len);
            scan(u0 + lane, beg, len);
        }
    }
    __syncwarp();   // the warps are independent from here on

    const unsigned lanes_before = (1u << lane) - 1u;
    double* gs = grid + S.grid_off;
    const long long gplane = (long long)M * M;
    // part 0 sums into the grid, the others into their slab slot (cells
    // [x][y][z] of the tile, 16^3); cell0: the lane's first cell
    const long long plane = ipart == 0 ? gplane : 256;
    const int row = ipart == 0 ? M : 16;
    double* cell0 = (ipart == 0 ? gs + (long long)x0 * gplane + (long long)y0 * M + z0
                                : slab + (long long)(slot0 + ipart - 1) * 4096) +
                    (long long)(8 * wy) * row + 8 * wz + lz + (FOLD ? (long long)ly * row : ly * plane);
    // this part's candidates: [cbeg, cend) of the warp's list
    const int cap = GEN ? split_cap(S.path, S.M, S.P, S.N) : S2_CAP;   // (ipart cap < N + cap)
    const int cbeg = ipart * cap, cend = min(total, cbeg + cap);

    Spread2Accum<Acc> acc;
    acc.zero();
    // one ring per x class: byte c of cnt holds the entries of class c
    // listed and not yet staged (< 64), byte c of ring the slot of the first
    unsigned cnt = 0u, ring = 0u;
    // a class holds a group when its count has a bit of value >= G
    constexpr unsigned FULL = (G == 32 ? 0x20u : 0x30u) * 0x010101u;
    int cpos = cbeg, buf = 0, pending = 0, pcls = 0, since_fold = 0;
    int seg = 0;   // the segment holding candidate cpos
    while (seg + 1 < nseg && seg_pre[seg + 1] <= cpos) seg++;
    // the lane's candidate of the 32 at cpos, loaded one round ahead
    int part = 0, pk = 0;
    auto fetch = [&] {
        const int pos = cpos + lane;
        int sl = seg;   // this lane's segment, found forward
        if (pos < cend) {
            while (sl + 1 < nseg && seg_pre[sl + 1] <= pos) sl++;
            part = seg_beg[sl] + (pos - seg_pre[sl]);
            pk = sg[part];
        }
        seg = __reduce_max_sync(0xffffffffu, sl);
    };
    fetch();
    bool written = false;
    for (;;) {
        // ---- list until some class holds a group (or every remaining
        // candidate is listed), each class in candidate order
        while (!(cnt & FULL) && cpos < cend) {
            int cls = -1;
            typename Spread2Entry<GEN>::Type entry = {};
            if (cpos + lane < cend) {
                // 8 cells from entry e on meet the stencil's entries [0, P)
                auto meets = [&](int e) { return (unsigned)(e + 7) < (unsigned)(P + 7); };
                bool lo, hi, yz;
                if constexpr (GEN) {
                    // the stencil's entry at the first cell of 8: the corner lies
                    // among them or less than M - 7 before them
                    auto entry_at = [&](int first, int axis) {
                        const int e = first - g_of(pk, axis);
                        return e < -7 ? e + M : e;
                    };
                    const int el = entry_at(x0, 0), eh = entry_at(x0 + 8, 0);
                    const int ey = entry_at(y0 + 8 * wy, 1), ez = entry_at(z0 + 8 * wz, 2);
                    lo = meets(el);
                    hi = meets(eh);
                    yz = meets(ey) && meets(ez);
                    // (an entry that meets nothing is not used, or >= P in its byte)
                    const auto byte = [](int e) { return (unsigned)min(e + 8, 255); };
                    entry = make_uint2((unsigned)part, byte(el) | byte(eh) << 8 | byte(ey) << 16 | byte(ez) << 24);
                } else {
                    // per axis: which tile after the home tile this one is, and
                    // the stencil's entry at the tile's (block's) first cell
                    int hx = tix - (g_of(pk, 0) >> 4), hy = tiy - (g_of(pk, 1) >> 4), hz = tiz - (g_of(pk, 2) >> 4);
                    hx += hx < 0 ? nt : 0;
                    hy += hy < 0 ? nt : 0;
                    hz += hz < 0 ? nt : 0;
                    const int ex = 16 * hx - (g_of(pk, 0) & 15);
                    const int ey = 16 * hy - (g_of(pk, 1) & 15) + 8 * wy, ez = 16 * hz - (g_of(pk, 2) & 15) + 8 * wz;
                    lo = meets(ex);
                    hi = meets(ex + 8);
                    yz = meets(ey) && meets(ez);
                    entry = ((unsigned)part << 3) | (hx << 2) | (hy << 1) | hz;
                }
                if (yz) cls = lo ? (hi ? 0 : 1) : (hi ? 2 : -1);
            }
            const unsigned k0 = __ballot_sync(0xffffffffu, cls == 0);
            const unsigned k1 = __ballot_sync(0xffffffffu, cls == 1);
            const unsigned k2 = __ballot_sync(0xffffffffu, cls == 2);
            if (cls >= 0) {
                const unsigned kc = cls == 0 ? k0 : (cls == 1 ? k1 : k2);
                const int sh = 8 * cls;
                sm.list[lw][cls][((ring >> sh) + (cnt >> sh) + __popc(kc & lanes_before)) &
                                   (S2_LIST - 1)] = entry;
            }
            cnt += __popc(k0) | (__popc(k1) << 8) | (__popc(k2) << 16);
            cpos += 32;
            fetch();
        }
        __syncwarp();   // list entries visible to the warp
        // ---- the class to stage: a full group if some class has one (the
        // first such class), else the first class with entries left
        const unsigned pick = (cnt & FULL) ? (cnt & FULL) : cnt;
        const int cls = pick ? (__ffs(pick) - 1) >> 3 : 0;
        const int sh = 8 * cls;
        const int avail = (cnt >> sh) & 0xFF;
        const int head = (ring >> sh) & (S2_LIST - 1);
        const auto* list = sm.list[lw][cls];
        // ---- stage the next group of the class: the x tile rows (of a
        // one-half class, that half), the block's 8 y and 8 z entries and the
        // charges, zeros past the group's n particles; consecutive lanes copy
        // consecutive 16-byte pieces of a row
        const int n = min(G, avail);
        if (n > 0) {
            Spread2Stage<F, GEN>& st = sm.stage[lw][buf];
            if constexpr (GEN) {
                // entry by entry, zeros outside the stencil
                auto copy = [&](F* dst, int i, int a, int k, int shift) {
                    const uint2 e = i < n ? list[(head + i) & (S2_LIST - 1)] : make_uint2(0u, 0u);
                    const int j = (int)(e.y >> shift & 255u) - 8 + k;
                    const bool on = i < n && (unsigned)j < (unsigned)P;
                    cp_async_one_or_zero(dst, rows + ((long long)e.x * 3 + a) * PS + (on ? j : 0), on);
                };
                // (of a short group no more rows than its sums take, a multiple of 4)
                auto stage = [&](auto rows_used) {
                    if (cls == 0) {
#pragma unroll 4
                        for (int i = lane >> 4; i < rows_used; i += 2)
                            copy(&st.px[i][s2_px<F, GEN>(i, lane & 15)], i, 0, lane & 7, lane & 8);
                    } else {
                        const int k = 8 * (cls - 1) + (lane & 7);
#pragma unroll 4
                        for (int i = lane >> 3; i < rows_used; i += 4) copy(&st.px[i][s2_px<F, GEN>(i, k)], i, 0, lane & 7, 8 * (cls - 1));
                    }
#pragma unroll 4
                    for (int i = lane >> 3; i < rows_used; i += 4) {
                        copy(&st.py[i][s2_pz<F>(i, lane & 7)], i, 1, lane & 7, 16);
                        copy(&st.pz[i][s2_pz<F>(i, lane & 7)], i, 2, lane & 7, 24);
                    }
                    if (lane < rows_used) {
                        const unsigned p = lane < n ? list[(head + lane) & (S2_LIST - 1)].x : 0u;
                        cp_async8_or_zero(&st.q[lane], &srec[p].w, lane < n);
                    }
                };
                if (n == G) stage(std::integral_constant<int, G>());
                else stage((n + 3) & ~3);
            } else {
                constexpr int C8 = 8 / V, C16 = 16 / V;   // pieces per 8 and 16 entries
                if (cls == 0) {
#pragma unroll
                    for (int i0 = 0; i0 < G; i0 += 32 / C16) {
                        const int i = i0 + lane / C16, k = V * (lane % C16);
                        const unsigned e = i < n ? list[(head + i) & (S2_LIST - 1)] : 0u;
                        cp_async16_or_zero(&st.px[i][s2_px<F, GEN>(i, k)],
                                           rows + (long long)(e >> 3) * 96 + 4 * (e & 4) + k, i < n);
                    }
                }
#pragma unroll
                for (int i0 = 0; i0 < G; i0 += 32 / C8) {
                    const int i = i0 + lane / C8, k = V * (lane % C8);
                    const unsigned e = i < n ? list[(head + i) & (S2_LIST - 1)] : 0u;
                    const Acc* r = rows + (long long)(e >> 3) * 96 + k;
                    if (cls != 0) {
                        const int o = 8 * (cls - 1);
                        cp_async16_or_zero(&st.px[i][s2_px<F, GEN>(i, o + k)], r + 4 * (e & 4) + o, i < n);
                    }
                    cp_async16_or_zero(&st.py[i][s2_pz<F>(i, k)], r + 32 + 8 * (e & 2) + 8 * wy, i < n);
                    cp_async16_or_zero(&st.pz[i][s2_pz<F>(i, k)], r + 64 + 16 * (e & 1) + 8 * wz, i < n);
                    if (k == 0) cp_async8_or_zero(&st.q[i], &srec[e >> 3].w, i < n);
                }
            }
            cp_async_commit();
            cnt -= (unsigned)n << sh;
            ring = (ring & ~(0xFFu << sh)) | ((unsigned)((head + n) & (S2_LIST - 1)) << sh);
        }
        __syncwarp();   // the staged entries are read before the list refills over them
        // ---- the previous group, while this one lands
        if (pending > 0) {
            if (n > 0) cp_async_wait<1>();
            else cp_async_wait<0>();
            __syncwarp();
            Spread2Stage<F, GEN>& st = sm.stage[lw][buf ^ 1];
            if constexpr (FOLD) {
                // lane i scales its particle's 8 y entries by the charge, once
                if (lane < pending) {
                    const Acc qv = (Acc)st.q[lane];
#pragma unroll
                    for (int k = 0; k < 8; k++) st.py[lane][k] = st.py[lane][k] * qv;
                }
                __syncwarp();
                // every group holds G rows (a short one padded with zeros, which
                // add exact zeros): one unrolled pass per class with constant
                // offsets; a one-half class touches the lane's 8 x 2 cells of its half
                if (pcls == 0) {
#pragma unroll S2_UNROLL
                    for (int i = 0; i < G; i++) {
                        const Acc y = st.py[i][ly];
                        acc.add(st.px[i], y * st.pz[i][lz], y * st.pz[i][lz + 1]);
                    }
                } else if (pcls == 1) {
#pragma unroll S2_UNROLL
                    for (int i = 0; i < G; i++) {
                        const Acc y = st.py[i][ly];
                        acc.template add_half<0>(st.px[i], y * st.pz[i][lz], y * st.pz[i][lz + 1]);
                    }
                } else {
#pragma unroll S2_UNROLL
                    for (int i = 0; i < G; i++) {
                        const Acc y = st.py[i][ly];
                        acc.template add_half<1>(st.px[i], y * st.pz[i][lz], y * st.pz[i][lz + 1]);
                    }
                }
            } else {
                const int t4 = lane & 3;
                if (pcls == 0) acc.template add_group<3>(st, pending, ly, t4);
                else if (pcls == 1) acc.template add_group<1>(st, pending, ly, t4);
                else acc.template add_group<2>(st, pending, ly, t4);
            }
            if constexpr (FOLD) {
                since_fold += pending;
                if (since_fold >= S2_FOLD) {
                    acc.fold(cell0, plane, !written);
                    written = true;
                    since_fold = 0;
                }
            }
            __syncwarp();   // the stage is read before it is refilled
        }
        if (n == 0) break;
        pending = n;
        pcls = cls;
        buf ^= 1;
    }

    // ---- the lane's cells
    if constexpr (FOLD) {
        if (since_fold > 0 || !written) acc.fold(cell0, plane, !written);
    } else if (GEN && total == 0 && ipart == 0) {
        // a block without candidates: zeros, 4 rows of 8 cells at a time (on an
        // almost empty grid the stores are the spread)
        const int nx = min(16, M - x0), ny = min(8, M - y0 - 8 * wy), nz = min(8, M - z0 - 8 * wz);
        double* block = gs + (long long)x0 * gplane + (long long)(y0 + 8 * wy) * M + z0 + 8 * wz;
        for (int r = lane >> 3; r < 128; r += 4)
            if (r >> 3 < nx && (r & 7) < ny && (lane & 7) < nz) block[(r >> 3) * gplane + (r & 7) * M + (lane & 7)] = 0.0;
    } else if (GEN) {
        // (a slab holds whole tiles)
        const int end = ipart == 0 ? M : nt * 16;
        acc.store(cell0, plane, row, {end - x0 - ly, end - y0 - 8 * wy, end - z0 - 8 * wz - lz});
    } else {
        acc.store(cell0, plane, row);
    }

    // ---- a split tile: the part that finishes last adds the slabs into the
    // grid, in part order
    if (nparts > 1) {
        __threadfence();
        __syncthreads();
        if (t == 0) folds = atomicAdd(&tile_done[tile], 1) == nparts * S2_CTA_SPLIT - 1;
        __syncthreads();
        if (folds) {
            __threadfence();
            // (8 cells of a thread side by side: the loads' latency is the time)
            for (int c0 = t; c0 < 4096; c0 += 8 * S2_THREADS) {
                double v[8];
                auto cell = [&](int j) -> double* {
                    const int c = c0 + j * S2_THREADS, x = c >> 8, y = (c >> 4) & 15, z = c & 15;
                    if (GEN && (x0 + x >= M || y0 + y >= M || z0 + z >= M)) return nullptr;
                    return gs + (long long)(x0 + x) * gplane + (long long)(y0 + y) * M + z0 + z;
                };
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const double* gp = cell(j);
                    v[j] = gp ? __ldcg(gp) : 0.0;
                }
                const double* sp = slab + (long long)slot0 * 4096 + c0;
                for (int k = 0; k < nparts - 1; k++, sp += 4096)
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] += __ldcg(sp + j * S2_THREADS);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (double* gp = cell(j)) *gp = v[j];
            }
            if (t == 0) tile_done[tile] = 0;
        }
    }
}

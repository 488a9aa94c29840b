// se_device.cuh -- definitions shared by the device-resident kernels
// (included inside namespace se by se_solve.cu).
#pragma once

constexpr int FB = 8;                     // fine bin edge, in stencil corners
constexpr int TX = 16, TY = 16, TZ = 16;  // spread tile (output cells)
constexpr int WY = 4, WZ = 8;             // one warp's lane block: 4 y x 8 z
constexpr int SPREAD_WARPS = (TY / WY) * (TZ / WZ);
constexpr int SPREAD_THREADS = SPREAD_WARPS * 32;
// particles staged per spread round
template <typename Acc>
constexpr int spread_chunk() { return 64; }

// Packed FP32 pairs (sm_100a): one FFMA2 (__ffma2_rn) does two FP32 FMAs,
// each rounded to nearest.
__device__ __forceinline__ float2 f32x2(float lo, float hi) { return make_float2(lo, hi); }

__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// The two packed pairs in 16 bytes of FP32 values.
__device__ __forceinline__ void f32x2_split(const float4& v, float2& lo, float2& hi)
{
    lo = make_float2(v.x, v.y);
    hi = make_float2(v.z, v.w);
}

// D += A B on an 8 x 8 tile of FP64 sums, 4 deep: with g = lane / 4 and
// t = lane % 4, a = A[g][t], b = B[t][g], d0 and d1 = D[g][2 t], D[g][2 t + 1].
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// The tile-aligned kernels (k_spread2, k_interp2 on tile-aligned factor rows)
// apply when a system's grid is cut into whole 16^3 tiles and its stencil
// fits two tiles.
__host__ __device__ inline bool spread2_eligible(int M, int P)
{
    return M % 16 == 0 && M >= 32 && P <= 16;
}

// A system's kernel path (SysDev::path): which spread and interpolation run.
constexpr int PATH_TILE_SPREAD = 1;    // k_spread2 on tile-aligned rows
constexpr int PATH_PAIR_INTERP = 2;    // k_interp2 or k_interp3 on tile-aligned rows
constexpr int PATH_RUNTIME_P = 4;      // interpolation without the P-unrolled variants
constexpr int PATH_RADIX_SORT = 8;     // the batch sorts with the radix passes (se_sort.cu)
constexpr int PATH_FFT3 = 16;          // the batch's FP64 FFTs through se_fft.cuh (not cuFFT)
constexpr int PATH_BIN_WINDOWS = 32;   // k_interp2 stages one window per bin (not per z pair)

// Whether a system off the whole tiles spreads by k_spread2 on its P-wide
// factor rows: where a run of 8 cells meets a stencil in one piece (M >= P + 7);
// k_spread serves the smaller grids.
__host__ __device__ inline bool spread2_general(int path, int M, int P)
{
    return !(path & PATH_TILE_SPREAD) && M >= P + 7;
}

// Whether k_interp3 serves a system (else k_interp2 on the path with
// PATH_PAIR_INTERP, k_interp without).  Measured on B200, interpolation stage:
// - FP64 on tile-aligned rows: from M = 128 on, forces of P = 10 to 12 from M =
//   192 on (M = 192, 1 to 80 particles per bin: 1.2 to 2.4x faster at P = 8 and
//   16, potentials at P = 12 1.2 to 1.7x, forces at P = 12 0.96 to 1.1x; M = 128 to
//   176, P = 8, 12 and 16, 0.5 to 40 per bin: no call slower); on
//   smaller grids its warps are too few for their latency (M = 64: 0.7 to 1.1x);
// - on other grids not for P <= 8 below M = 64 (M = 36, 1 to 18 per bin: 0.75
//   to 1x, 4 us of a solve of 85, with chunks of 256 particles; as its work is cut
//   now, 4,500, M = 54, P = 8, force 48 and 52 us, crowded bins would gain);
// - else FP64: always (M = 36 to 150, 1 to 120 per bin: 0.9 to 8x);
// - else FP32: where the window kernel has no compiled-in stencil or,
//   for potentials, gains nothing by it (P = 8 1.03 to 1.5x, P = 15 1.4 to 3x,
//   P = 20 1.8 to 4.5x, potentials at P = 12 and 16 0.97 to 2x, forces there
//   0.75 (120 per bin) to 1.5x (4 per bin)).
inline bool interp3_better(int path, int precision, int M, int P, int mode)
{
    if (path & PATH_PAIR_INTERP)
        return precision == SE_FP64 && M >= (mode == SE_FORCE && P >= 10 && P <= 12 ? 192 : 128);
    if (P <= 8 && M < 64) return false;
    return precision == SE_FP64 || mode == SE_POTENTIAL || (P != 12 && P != 16);
}

// The default path: the tile-aligned spread wherever it applies, and the
// window-pair interpolation from P = 8 on (for shorter stencils its
// per-particle set-up and z-pair padding cost more than they save: the timed
// choice picks the general interpolation there on B200).
__host__ __device__ inline int default_path(int M, int P)
{
    if (!spread2_eligible(M, P)) return 0;
    return PATH_TILE_SPREAD | (P >= 8 ? PATH_PAIR_INTERP : 0);
}

constexpr int MAX_SEG = 96;               // bin segments reaching one tile
constexpr int INTERP_WARPS = 8;
constexpr int MAX_P = 32;
constexpr double PI_D = 3.14159265358979323846;

// Per-system parameters and offsets of a batch (one entry per system).
struct SysDev {
    int N, M, P, lo, mode;
    int path;         // PATH_* bits
    int interp3;      // k_interp3 serves the system (interp3_better)
    int part_off, out_off;
    long long grid_off, spec_off;
    int nf[3];        // fine bins per axis
    int bin_base;     // first global fine-bin id
    int nt[3];        // spread tiles per axis
    int tile_base;    // first global spread-tile id
    double h, c, d, h3;
    double rho;       // exp(-2 c h^2)
    double kfac;      // 2 pi / L
    double scalar;    // -(1 - eta) / (4 xi^2)
    double dnorm;     // 4 pi / M^3
};

// largest s with prefix[s] <= v
__device__ __forceinline__ int find_sys(const int* __restrict__ prefix, int nsys, int v)
{
    int lo = 0, hi = nsys - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= v) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// periodic index in [0, n) for any int i (SE_fgg.c:17-25 vmod)
__host__ __device__ __forceinline__ int pmod(int i, int n)
{
    const int r = i % n;
    return r < 0 ? r + n : r;
}

// i in (-n, 2n) to [0, n) without a division
__device__ __forceinline__ int wrap1(int i, int n)
{
    i = i < 0 ? i + n : i;
    return i >= n ? i - n : i;
}

__device__ __forceinline__ int pack_g(int gx, int gy, int gz) { return gx | (gy << 10) | (gz << 20); }
__device__ __forceinline__ int g_of(int pk, int a) { return (pk >> (10 * a)) & 1023; }

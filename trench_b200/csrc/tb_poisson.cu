// Geometric-multigrid-preconditioned CG for the staircase Poisson operator.
//
// Replaces the reference's SuperLU factorisation (trench_charging_2d.py:297-309,
// 378-392).  The operator is the SPD form L = -dx^2 * A of the reference's
// 5-point finite-volume matrix A (trench_charging_2d.py:252-294): per cell a
// diagonal d > 0 and non-negative couplings kE (to the east neighbour, x
// periodic) and kN (to the north neighbour).  Cells marked fixed are Dirichlet
// zero (identity rows, couplings into them removed) -- a driven or, with the
// superposition done by the caller, a floating conductor.
//
// Precision: FP32 V-cycles inside an FP32 PCG, wrapped in FP64 iterative
// refinement (residual r = b - L x in FP64, normalised before each FP32 solve).
//
// Hierarchy: cell-centred 2x2 aggregation; the coarse operator is one half of
// the Galerkin product P^T L P for piecewise-constant P restricted to free
// cells (the scaling that makes aggregation consistent with rediscretisation).
// Smoother: multicolour (red-black) Gauss-Seidel, forward before and reversed
// after the coarse correction, so the V-cycle is a symmetric preconditioner.
//
// Many right-hand sides are solved together: vectors are (nrhs, cells) and
// every kernel covers all of them in one launch (blockIdx.y = rhs).  Dot products
// are per-block partial sums added in block order, so a solve is deterministic.
//
// Launches: a small grid's solve is bound by latency -- a level's smoothing colour,
// residual, restriction and prolongation are one short dependent pass each, about a
// hundred to a V-cycle.
//  * The levels whose vectors and operator fit in one CTA's shared memory (the bottom)
//    run in one CTA per right-hand side with barriers between the passes, the coarsest
//    level in one warp.
//  * A grid whose columns fit in the shared memory of a cluster (cluster_fit: a CTA's columns,
//    4 ceil(ceil(nx / 4) / 8) of them, hold at most 3584 cells) is solved whole by one launch
//    (k_solve_cluster): FP64 residual, convergence test, PCG and V-cycles.  Each right-hand
//    side stops at its own convergence, and the host waits once.
//  * Larger grids keep one launch per pass over all right-hand sides (their passes are
//    long enough), with the bottom as one launch.
#include <cooperative_groups.h>
#include <math.h>

#include <float.h>

#include <algorithm>
#include <vector>

#include "tb_internal.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int PT = 256;  // threads per block
constexpr int CTA_THREADS = 1024;       // threads of the one-CTA bottom
constexpr int GATHER = 2;               // cells whose loads are in flight together in a thread
// Shared memory of the bottom: 28 bytes a cell (the four couplings, x, b and the diagonal).
constexpr int BOTTOM_BYTES = 200 * 1024;
constexpr int BOTTOM_CELL = 28;
constexpr int COARSEST_WARP_CELLS = 128;   // a coarsest level this small is swept by one warp

struct Level {
    int nx = 0, ny = 0;
    int n = 0;
    float *d = nullptr, *ke = nullptr, *kn = nullptr;
    uint8_t *fixed = nullptr;
    float *x = nullptr, *b = nullptr, *r = nullptr;  // (max_rhs, n)
    unsigned inv_ny = 0, inv_half = 0;               // c / ny and c / ((ny + 1) / 2) by __umulhi (inverse_of)
    float4 *k4 = nullptr;                            // couplings to E, W, N, S (the one-CTA kernels)
    float *df = nullptr;                             // diagonal, infinite on fixed cells (s / df = 0)
};

}  // namespace

struct tb_poisson {
    int max_rhs = 0;
    std::vector<Level> lev;
    double *d64 = nullptr, *ke64 = nullptr, *kn64 = nullptr;
    double *r64 = nullptr;                     // (max_rhs, n)
    float *e = nullptr, *pr = nullptr, *pz = nullptr, *pp = nullptr, *pq = nullptr;  // PCG vectors
    double *scal = nullptr;                    // (max_rhs, 8) per-rhs scalars
    double *part = nullptr;                    // (max_rhs, blocks, PART) per-block partial sums
    int part_blocks = 0;
    int pre = 1, post = 1, coarse_sweeps = 16;
    int bottom = -1;                           // first level kept in one CTA's shared memory
    int bottom_bytes = 0;                      // its shared memory
    int cluster_bytes[2] = {0, 0};             // shared memory of the one-launch solve of 1 and 2 sides; 0 = does not fit
    std::vector<float> cd, cke, ckn;           // the coarsest level
    std::vector<uint8_t> cfx;
    float *d_coarse = nullptr;                 // its sweeps as a matrix, by columns (one-launch solve)
    Level *d_lev = nullptr;                    // device copy of lev
};

namespace {

enum { S_RR = 0, S_BB = 1, S_AA = 2, S_RZ = 3, S_PQ = 4, S_RZ_NEW = 5, S_OUTER = 6 };
constexpr int PART = 3;  // doubles per (right-hand side, block) in the partial-sums buffer

__device__ __forceinline__ int wrapx(int i, int nx) { return i < 0 ? i + nx : (i >= nx ? i - nx : i); }

// y = L x at one cell (FP32 or FP64 operator)
template <typename T, typename V>
__device__ __forceinline__ V apply_at(const T *d, const T *ke, const T *kn, const V *x, int nx, int ny, int c) {
    const int ix = c / ny, iy = c - ix * ny;
    const int w = wrapx(ix - 1, nx) * ny + iy, e = wrapx(ix + 1, nx) * ny + iy;
    V s = (V)d[c] * x[c] - (V)ke[c] * x[e] - (V)ke[w] * x[w];
    if (iy + 1 < ny) s -= (V)kn[c] * x[c + 1];
    if (iy > 0) s -= (V)kn[c - 1] * x[c - 1];
    return s;
}

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double sh[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;
}

// Sum of the magnitudes of the terms of (L x)[c]: the scale of the rounding error of
// the residual at that cell.
__device__ __forceinline__ double apply_abs_at(const double *d, const double *ke, const double *kn, const double *x,
                                               int nx, int ny, int c) {
    const int ix = c / ny, iy = c - ix * ny;
    const int w = wrapx(ix - 1, nx) * ny + iy, e = wrapx(ix + 1, nx) * ny + iy;
    double s = fabs(d[c] * x[c]) + fabs(ke[c] * x[e]) + fabs(ke[w] * x[w]);
    if (iy + 1 < ny) s += fabs(kn[c] * x[c + 1]);
    if (iy > 0) s += fabs(kn[c - 1] * x[c - 1]);
    return s;
}

// r64 = b - L x (FP64); per-block partial sums of |r|^2, |b|^2 and |a|^2 into part, a the
// cell-wise magnitude |b| + sum |terms of L x| that bounds the residual's own rounding
__global__ void k_resid64(int nx, int ny, const double *d, const double *ke, const double *kn, const double *x,
                          const double *b, double *r, double *part) {
    const int n = nx * ny, rhs = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const double *xr = x + (size_t)rhs * n;
    double rr = 0, bb = 0, aa = 0;
    if (c < n) {
        const double bv = b[(size_t)rhs * n + c];
        const double v = bv - apply_at(d, ke, kn, xr, nx, ny, c);
        r[(size_t)rhs * n + c] = v;
        rr = v * v;
        bb = bv * bv;
        const double a = fabs(bv) + apply_abs_at(d, ke, kn, xr, nx, ny, c);
        aa = a * a;
    }
    rr = block_sum(rr);
    bb = block_sum(bb);
    aa = block_sum(aa);
    if (threadIdx.x == 0) {
        double *pp = part + ((size_t)rhs * gridDim.x + blockIdx.x) * PART;
        pp[0] = rr;
        pp[1] = bb;
        pp[2] = aa;
    }
}

// scal[rhs][slot0 + j] = sum over blocks of part[rhs][block][j], in block order (deterministic)
__global__ void k_sum_partials(int nrhs, int nblk, int nslot, const double *part, double *scal, int slot0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrhs * nslot) return;
    const int rhs = i / nslot, j = i - rhs * nslot;
    double t = 0;
    for (int b = 0; b < nblk; ++b) t += part[((size_t)rhs * nblk + b) * PART + j];
    scal[rhs * 8 + slot0 + j] = t;
}

// r32 = r64 / |r64| ; e = 0
__global__ void k_normalise(int n, const double *r64, float *r32, float *e, double *scal) {
    const int rhs = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double nr = sqrt(scal[rhs * 8 + S_RR]);
    const double inv = nr > 0 ? 1.0 / nr : 0.0;
    r32[(size_t)rhs * n + c] = (float)(r64[(size_t)rhs * n + c] * inv);
    e[(size_t)rhs * n + c] = 0.f;
}

// x64 += |r64| * e
__global__ void k_correct(int n, const float *e, double *x, const double *scal) {
    const int rhs = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double nr = sqrt(scal[rhs * 8 + S_RR]);
    x[(size_t)rhs * n + c] += nr * (double)e[(size_t)rhs * n + c];
}

// Gauss-Seidel sweep over one colour (x updated in place).  Colours 0/1 are the
// red-black checkerboard; with odd nx the periodic wrap would put columns nx-1 and
// 0 side by side in one colour, so column nx-1 gets colours 2/3 (by row parity) and
// no two neighbours ever share a colour.
__device__ __forceinline__ void smooth_at(const Level &L, int rhs, int c, int color) {
    const int nx = L.nx, ny = L.ny, n = L.n;
    const int ix = c / ny, iy = c - ix * ny;
    const int col = ((nx & 1) && ix == nx - 1) ? 2 + (iy & 1) : ((ix + iy) & 1);
    if (col != color || L.fixed[c]) return;
    float *xr = L.x + (size_t)rhs * n;
    const float *ke = L.ke, *kn = L.kn;
    const int w = wrapx(ix - 1, nx) * ny + iy, e = wrapx(ix + 1, nx) * ny + iy;
    float s = L.b[(size_t)rhs * n + c] + ke[c] * xr[e] + ke[w] * xr[w];
    if (iy + 1 < ny) s += kn[c] * xr[c + 1];
    if (iy > 0) s += kn[c - 1] * xr[c - 1];
    xr[c] = s / L.d[c];
}

__global__ void k_smooth(const Level L, int color) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < L.n) smooth_at(L, blockIdx.y, c, color);
}

__global__ void k_zero(size_t n, float *x) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = 0.f;
}

__device__ __forceinline__ void resid_at(const Level &L, int rhs, int c) {
    const size_t o = (size_t)rhs * L.n;
    L.r[o + c] = L.fixed[c] ? 0.f : L.b[o + c] - apply_at(L.d, L.ke, L.kn, L.x + o, L.nx, L.ny, c);
}

__global__ void k_resid32(const Level L) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < L.n) resid_at(L, blockIdx.y, c);
}

// coarse b = sum of the free fine residuals of the 2x2 aggregate
__device__ __forceinline__ void restrict_at(const Level &F, const Level &C, int rhs, int c) {
    const int fnx = F.nx, fny = F.ny, cny = C.ny;
    const int I = c / cny, J = c - I * cny;
    float s = 0.f;
    for (int a = 0; a < 2; ++a) {
        const int i = 2 * I + a;
        if (i >= fnx) break;
        for (int q = 0; q < 2; ++q) {
            const int j = 2 * J + q;
            if (j >= fny) break;
            const int f = i * fny + j;
            if (!F.fixed[f]) s += F.r[(size_t)rhs * F.n + f];
        }
    }
    C.b[(size_t)rhs * C.n + c] = s;
}

__global__ void k_restrict(const Level F, const Level C) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < C.n) restrict_at(F, C, blockIdx.y, c);
}

__device__ __forceinline__ void prolong_at(const Level &F, const Level &C, int rhs, int f) {
    if (F.fixed[f]) return;
    const int i = f / F.ny, j = f - i * F.ny;
    F.x[(size_t)rhs * F.n + f] += C.x[(size_t)rhs * C.n + (i >> 1) * C.ny + (j >> 1)];
}

__global__ void k_prolong(const Level F, const Level C) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f < F.n) prolong_at(F, C, blockIdx.y, f);
}

// ---- one-CTA kernels -------------------------------------------------------------------

// Bytes of one bottom level in shared memory (kept a multiple of 16).
__host__ __device__ __forceinline__ int bottom_level_bytes(int n) { return (BOTTOM_CELL * n + 15) & ~15; }

// One level as the one-CTA kernels see it; the pointers lead to shared or global memory.
struct LevelView {
    int nx, ny, n;
    unsigned inv_ny, inv_half;   // see inverse_of; the 64-bit division itself costs more than a pass
    const float4 *k;        // couplings to E, W, N, S
    float *x, *b;
    const float *d;         // diagonal, infinite on fixed cells
};

// c / k = (c inverse_of(k)) >> 32 for c k < 2^32 and k > 1.
__host__ __device__ __forceinline__ unsigned inverse_of(int k) { return (unsigned)(0x100000000ULL / (unsigned)k) + 1u; }
__device__ __forceinline__ int quotient(int c, int k, unsigned inv) { return k == 1 ? c : (int)__umulhi((unsigned)c, inv); }
__device__ __forceinline__ int column_of(const LevelView &L, int c) { return quotient(c, L.ny, L.inv_ny); }

// Neighbours E, W, N, S of a cell; beyond the top or bottom row the cell itself, whose
// coupling there is zero.
__device__ __forceinline__ int4 neighbours(const LevelView &L, int ix, int iy, int c) {
    return make_int4(ix == L.nx - 1 ? iy : c + L.ny, ix == 0 ? c + (L.nx - 1) * L.ny : c - L.ny,
                     iy + 1 < L.ny ? c + 1 : c, iy > 0 ? c - 1 : c);
}
// Sum of the couplings times the neighbours' values.
template <typename V>
__device__ __forceinline__ float coupled(const float4 k, const V *x, const int4 a) {
    return fmaf(k.w, x[a.w], fmaf(k.z, x[a.z], fmaf(k.y, x[a.y], k.x * x[a.x])));
}
__device__ __forceinline__ bool is_free(float d) { return d < FLT_MAX; }
// s / d rounded to the nearest, 0 on fixed cells (whose d is infinite): the reciprocal with one
// Newton step, and the quotient corrected by its exact remainder (Markstein, IBM J. Res. Dev. 34,
// 1990; divisors with every mantissa bit set may be one ulp off).  Straight-line: the general
// division's range check made a solve 1051 instead of 925 us (60 x 250 cells).
__device__ __forceinline__ float relaxed(float s, float d) {
    const float f = is_free(d) ? d : 1.f;
    float y = __fdividef(1.f, f);
    y = fmaf(y, fmaf(-f, y, 1.f), y);
    const float q = s * y;
    const float v = fmaf(fmaf(-f, q, s), y, q);
    return is_free(d) ? v : 0.f;
}

// The bottom levels' shared memory: per level the couplings, x, b and the diagonal.
__device__ __forceinline__ LevelView bottom_view(unsigned char *sm, const Level *lev, int first, int l) {
    for (int k = first; k < l; ++k) sm += bottom_level_bytes(lev[k].n);
    LevelView V;
    V.nx = lev[l].nx;
    V.ny = lev[l].ny;
    V.n = lev[l].n;
    V.inv_ny = lev[l].inv_ny;
    V.inv_half = lev[l].inv_half;
    V.k = reinterpret_cast<const float4 *>(sm);
    float *f = reinterpret_cast<float *>(sm) + 4 * V.n;
    V.x = f;
    V.b = f + V.n;
    V.d = f + 2 * V.n;
    return V;
}

__device__ void bottom_load(unsigned char *sm, const Level *lev, int first, int nlev) {
    for (int l = first; l < nlev; ++l) {
        const LevelView V = bottom_view(sm, lev, first, l);
        const Level L = lev[l];
        for (int c = threadIdx.x; c < V.n; c += blockDim.x) {
            const_cast<float4 *>(V.k)[c] = L.k4[c];
            const_cast<float *>(V.d)[c] = L.df[c];
        }
    }
}

// One Gauss-Seidel colour by `count` threads (this one is number `i`); the colours of smooth_at
// (the checkerboard, with the last column of an odd grid in colours 2 and 3 by row parity), and its
// division.  Every loop of
// these kernels gathers several cells before it stores any, so that their loads are in flight
// together: one cell at a time a pass cost 5 us, the latency of fifteen gathers in a row.
template <int G>
__device__ __forceinline__ void smooth_colour(const LevelView &L, int color, int i, int count) {
    const int half = (L.ny + 1) >> 1;
    const int m = color < 2 ? ((L.nx & 1) ? L.nx - 1 : L.nx) * half : half;
    for (int k0 = i; k0 < m; k0 += G * count) {
        float v[G];
        int at[G];
#pragma unroll
        for (int j = 0; j < G; ++j) {
            const int k = min(k0 + j * count, m - 1);
            int ix, iy;
            if (color < 2) {
                ix = quotient(k, half, L.inv_half);
                iy = 2 * (k - ix * half) + ((ix + color) & 1);
            } else {
                ix = L.nx - 1;
                iy = 2 * k + color - 2;
            }
            const bool valid = k0 + j * count < m && iy < L.ny;
            iy = min(iy, L.ny - 1);
            const int c = ix * L.ny + iy;
            v[j] = relaxed(L.b[c] + coupled(L.k[c], L.x, neighbours(L, ix, iy, c)), L.d[c]);
            at[j] = valid ? c : -1;
        }
#pragma unroll
        for (int j = 0; j < G; ++j)
            if (at[j] >= 0) L.x[at[j]] = v[j];
    }
}

// x = the first colour's sweep of x = 0, for one cell.
__device__ __forceinline__ float first_colour(const LevelView &L, int c, float b) {
    const int ix = column_of(L, c), iy = c - ix * L.ny;
    const bool first = ((ix + iy) & 1) == 0 && !((L.nx & 1) && ix == L.nx - 1);
    return first ? relaxed(b, L.d[c]) : 0.f;
}
__device__ __forceinline__ void smooth_start(const LevelView &L) {
#pragma unroll GATHER
    for (int c = threadIdx.x; c < L.n; c += CTA_THREADS) L.x[c] = first_colour(L, c, L.b[c]);
}

// Coarse right-hand side: the free residuals of each 2x2 aggregate, summed.
__device__ __forceinline__ void restrict_residual(const LevelView &F, const LevelView &C, int i, int count) {
    for (int c = i; c < C.n; c += count) {
        const int I = column_of(C, c), J = c - I * C.ny;
        float r[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int ix = min(2 * I + (a >> 1), F.nx - 1), iy = min(2 * J + (a & 1), F.ny - 1);
            const int f = ix * F.ny + iy;
            const float d = F.d[f];
            const bool counts = is_free(d) && 2 * I + (a >> 1) < F.nx && 2 * J + (a & 1) < F.ny;
            const float v = F.b[f] - ((is_free(d) ? d : 0.f) * F.x[f] - coupled(F.k[f], F.x, neighbours(F, ix, iy, f)));
            r[a] = counts ? v : 0.f;
        }
        C.b[c] = (r[0] + r[1]) + (r[2] + r[3]);
    }
}

template <int G>
__device__ __forceinline__ void prolong(const LevelView &F, const LevelView &C, int i, int count) {
    for (int f0 = i; f0 < F.n; f0 += G * count) {
        float v[G];
#pragma unroll
        for (int j = 0; j < G; ++j) {
            const int f = min(f0 + j * count, F.n - 1);
            const int ix = column_of(F, f), iy = f - ix * F.ny;
            v[j] = F.x[f] + (is_free(F.d[f]) ? C.x[(ix >> 1) * C.ny + (iy >> 1)] : 0.f);
        }
#pragma unroll
        for (int j = 0; j < G; ++j)
            if (f0 + j * count < F.n) F.x[f0 + j * count] = v[j];
    }
}

__device__ __forceinline__ int colours(const LevelView &L) { return (L.nx & 1) ? 4 : 2; }

// The pre-smoothing of a level after its first colour (already in x), and its post-smoothing.
__device__ __forceinline__ void pre_smooth(const LevelView &L, int pre) {
    const int nc = colours(L);
    for (int k = 0; k < pre; ++k)
        for (int c = k == 0 ? 1 : 0; c < nc; ++c) {
            smooth_colour<GATHER>(L, c, threadIdx.x, blockDim.x);
            __syncthreads();
        }
}
__device__ __forceinline__ void post_smooth(const LevelView &L, int post) {
    const int nc = colours(L);
    for (int k = 0; k < post; ++k)
        for (int c = nc - 1; c >= 0; --c) {
            smooth_colour<GATHER>(L, c, threadIdx.x, blockDim.x);
            __syncthreads();
        }
}

// The V-cycle from level `first` (its right-hand side in place, in shared memory) down to the
// coarsest and back.  Every thread of the CTA calls it; it ends with a barrier.
__device__ __forceinline__ void bottom_cycle(unsigned char *sm, const Level *lev, int first, int nlev, int pre, int post,
                                             int coarse_sweeps) {
    const int t = threadIdx.x, T = blockDim.x;
    for (int l = first; l + 1 < nlev; ++l) {
        const LevelView L = bottom_view(sm, lev, first, l), C = bottom_view(sm, lev, first, l + 1);
        smooth_start(L);
        __syncthreads();
        pre_smooth(L, pre);
        restrict_residual(L, C, t, T);
        __syncthreads();
    }
    const LevelView L = bottom_view(sm, lev, first, nlev - 1);
    const int nc = colours(L);
    if (L.n > COARSEST_WARP_CELLS) {
        // a coarsest level that is long and one or two cells wide
        for (int c = t; c < L.n; c += T) L.x[c] = 0.f;
        __syncthreads();
        for (int dir = 0; dir < 2; ++dir)
            for (int k = 0; k < coarse_sweeps; ++k)
                for (int q = 0; q < nc; ++q) {
                    smooth_colour<GATHER>(L, dir == 0 ? q : nc - 1 - q, t, T);
                    __syncthreads();
                }
    } else if (t < 32) {
        // a cell or two a lane: one warp, no block barriers
        for (int c = t; c < L.n; c += 32) L.x[c] = 0.f;
        __syncwarp();
        for (int dir = 0; dir < 2; ++dir)
            for (int k = 0; k < coarse_sweeps; ++k)
                for (int q = 0; q < nc; ++q) {
                    smooth_colour<1>(L, dir == 0 ? q : nc - 1 - q, t, 32);
                    __syncwarp();
                }
    }
    __syncthreads();
    for (int l = nlev - 2; l >= first; --l) {
        const LevelView L = bottom_view(sm, lev, first, l), C = bottom_view(sm, lev, first, l + 1);
        prolong<GATHER>(L, C, t, T);
        __syncthreads();
        post_smooth(L, post);
    }
}

// The bottom of a V-cycle for grids solved with one launch per pass: one CTA per right-hand side.
__global__ void __launch_bounds__(CTA_THREADS) k_vcycle_bottom(const Level *lev, int first, int nlev, int pre,
                                                               int post, int coarse_sweeps) {
    extern __shared__ __align__(16) unsigned char sm[];
    const LevelView V = bottom_view(sm, lev, first, first);
    const size_t o = (size_t)blockIdx.x * V.n;
    bottom_load(sm, lev, first, nlev);
    for (int c = threadIdx.x; c < V.n; c += blockDim.x) V.b[c] = lev[first].b[o + c];
    __syncthreads();
    bottom_cycle(sm, lev, first, nlev, pre, post, coarse_sweeps);
    for (int c = threadIdx.x; c < V.n; c += blockDim.x) lev[first].x[o + c] = V.x[c];
}

// ---- the whole solve in one launch: one cluster per right-hand side (or two) --------------
//
// A pass over one right-hand side of a small grid is far too short for the whole GPU and far too
// long for one SM (15,000 cells in one CTA: 8,400 cycles for half of them, bound by the SM's loads).
// Here a cluster of CLUSTER CTAs holds it in shared memory: every CTA owns a block of columns of
// level 0 and the same columns of level 1 -- couplings, diagonal, x, b and the search direction
// -- with one halo column on each side, which the owner writes through distributed shared
// memory when it changes its own edge.  Level 2 and below (a sixteenth of the cells) are CTA 0's.
// A pass is a few cells a thread between two cluster barriers.  60 x 250, one right-hand side:
// 0.71 ms (36 PCG iterations of 19 us) against 3.6 ms of kernels and 1.4 ms of gaps between
// 540 launches; 300 right-hand sides, two to a cluster: 10.6 ms against 15.8 ms.
constexpr int CLUSTER = 8;
constexpr int CL_THREADS = 512;
constexpr int CL_CELLS = 7;             // cells of level 0 a thread owns at most
constexpr int CL_COARSEST = 64;         // the coarsest level's sweeps as one matrix of at most this size
constexpr int CL_MAX_LEVELS = 12;
constexpr int CL_SMEM = 224 * 1024;
// More sides than this of a grid of fewer cells than this are quicker in launches, which take all
// of them in every pass.  us in one launch and in launches, 100, 200 and 300 sides: 12 x 70 cells 2240
// and 2746, 4165 and 3913, 5565 and 4931; 33 x 120 cells 3720 and 3740, 6101 and 5718, 9556 and
// 7757; 44 x 120 cells 2872 and 3894, 4663 and 6121, 6543 and 8289.
constexpr int CL_SIDES = 120, CL_FEW_CELLS = 4500;

struct ClusterSolve {
    const Level *lev;
    int nlev, pre, post, max_outer, inner, nrhs;
    const double *d64, *ke64, *kn64, *b;
    double *x, *scal;
    double rtol;
    const float *coarse;                // (n, n) of the coarsest level, by columns
};

// Columns of level l owned by a CTA, from the columns of level 2 it owns.
struct Columns {
    int x0, w;
};
__host__ __device__ __forceinline__ Columns columns_of(int rank, int l, int nx_l, int nx2) {
    const int per = (nx2 + CLUSTER - 1) / CLUSTER;
    Columns c;
    const int a = rank * per < nx2 ? rank * per : nx2, b = (rank + 1) * per < nx2 ? (rank + 1) * per : nx2;
    const int sh = 2 - l;
    const int lo = (a << sh) < nx_l ? (a << sh) : nx_l, hi = (b << sh) < nx_l ? (b << sh) : nx_l;
    c.x0 = lo;
    c.w = hi - lo;
    return c;
}

// Shared memory layout in bytes: the same offsets in every CTA (sized for the widest block).
struct ClusterLayout {
    int k0, d0, k1, d1;                 // couplings and diagonals of levels 0 and 1
    int x0, p0, r0, x1, b1, per_rhs;    // of right-hand side 0; the next one's are per_rhs further
    int kd[CL_MAX_LEVELS], xb[CL_MAX_LEVELS];   // levels 2..: couplings + diagonal; x and b of right-hand side 0
    int coarse, sums, bytes;
};
__host__ __device__ __forceinline__ int align16(int v) { return (v + 15) & ~15; }
__host__ __device__ inline ClusterLayout cluster_layout(const int *nx, const int *ny, int nlev, int R) {
    ClusterLayout L;
    const Columns c0 = columns_of(0, 0, nx[0], nx[2]), c1 = columns_of(0, 1, nx[1], nx[2]);
    int o = 0;
    auto take = [&](int bytes) {
        const int at = o;
        o += align16(bytes);
        return at;
    };
    L.k0 = take(16 * c0.w * ny[0]);
    L.d0 = take(4 * c0.w * ny[0]);
    L.k1 = take(16 * c1.w * ny[1]);
    L.d1 = take(4 * c1.w * ny[1]);
    for (int l = 2; l < nlev; ++l) L.kd[l] = take(20 * nx[l] * ny[l]);
    const int nc = nx[nlev - 1] * ny[nlev - 1];
    L.coarse = take(4 * nc * nc);
    L.sums = take(2 * CLUSTER * 4 * R * 8);
    const int first = o;
    L.x0 = take(4 * (c0.w + 2) * ny[0]);
    L.p0 = take(4 * (c0.w + 2) * ny[0]);
    L.r0 = take(4 * c0.w * ny[0]);
    L.x1 = take(4 * (c1.w + 2) * ny[1]);
    L.b1 = take(4 * c1.w * ny[1]);
    for (int l = 2; l < nlev; ++l) L.xb[l] = take(8 * nx[l] * ny[l]);
    L.per_rhs = o - first;
    L.bytes = first + R * L.per_rhs;
    return L;
}

// A level's own columns with their halo: local column lc = 1..w is global column x0 + lc - 1;
// x is (w + 2, ny), b, k and d are (w, ny).
struct Block {
    int nx, ny, x0, w;
    unsigned inv_ny, inv_half;
    float *x, *b;
    const float4 *k;
    const float *d;
    float *left, *right;                // the neighbours' halo columns of x (distributed shared memory)
};

// Writes x of local column lc, row iy, and the neighbour's halo copy if it is an edge column.
__device__ __forceinline__ void put(const Block &B, float *x, float *left, float *right, int lc, int iy, float v) {
    x[lc * B.ny + iy] = v;
    if (lc == 1) left[iy] = v;
    if (lc == B.w) right[iy] = v;
}

__device__ __forceinline__ float gather4(const float4 k, const float *x, int at, int ny, int iy) {
    const int n = iy + 1 < ny ? at + 1 : at, s = iy > 0 ? at - 1 : at;
    return fmaf(k.w, x[s], fmaf(k.z, x[n], fmaf(k.y, x[at - ny], k.x * x[at + ny])));
}

__device__ __forceinline__ void block_colour(const Block &B, int color) {
    const bool odd = B.nx & 1;
    const int half = (B.ny + 1) >> 1;
    // columns of the checkerboard colours (all but the last of an odd grid) among the own ones
    const int w = odd ? min(B.w, B.nx - 1 - B.x0) : B.w;
    const int last = odd && B.x0 + B.w == B.nx && B.w > 0 ? B.w : 0;     // local index of the last column
    const int m = color < 2 ? max(w, 0) * half : (last ? half : 0);
    for (int k = threadIdx.x; k < m; k += CL_THREADS) {
        int lc, iy;
        if (color < 2) {
            const int col = quotient(k, half, B.inv_half);
            lc = col + 1;
            iy = 2 * (k - col * half) + ((B.x0 + col + color) & 1);
        } else {
            lc = last;
            iy = 2 * k + color - 2;
        }
        if (iy >= B.ny) continue;
        const int at = lc * B.ny + iy, c = at - B.ny;
        put(B, B.x, B.left, B.right, lc, iy, relaxed(B.b[c] + gather4(B.k[c], B.x, at, B.ny, iy), B.d[c]));
    }
}

// x = the first colour's sweep of x = 0.
__device__ __forceinline__ float start_value(const Block &B, int ix, int iy, float b, float d) {
    const bool first = ((ix + iy) & 1) == 0 && !((B.nx & 1) && ix == B.nx - 1);
    return first ? relaxed(b, d) : 0.f;
}

// Free residual of one fine cell (local column lc).
__device__ __forceinline__ float block_residual(const Block &F, int lc, int iy) {
    const int at = lc * F.ny + iy, c = at - F.ny;
    const float d = F.d[c];
    return is_free(d) ? F.b[c] - (d * F.x[at] - gather4(F.k[c], F.x, at, F.ny, iy)) : 0.f;
}
__device__ __forceinline__ float aggregate_residual(const Block &F, int I, int J) {
    // coarse column I (from the block's first), row J
    float r[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int col = 2 * I + (a >> 1), iy = 2 * J + (a & 1);
        r[a] = col < F.w && iy < F.ny ? block_residual(F, col + 1, iy) : 0.f;
    }
    return (r[0] + r[1]) + (r[2] + r[3]);
}

// Sums of v[0..N) over the cluster, in every thread; added in rank order.  `buf`: 2 x CLUSTER x
// N doubles in every CTA, by call parity.  One cluster barrier.
template <int N>
__device__ __forceinline__ void cluster_sum(cg::cluster_group &cl, double (&v)[N], double *buf, int &parity) {
    __shared__ double sh[N][CL_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rank = (int)cl.block_rank();
#pragma unroll
    for (int k = 0; k < N; ++k) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (lane == 0) sh[k][w] = v[k];
    }
    __syncthreads();
    double *at = buf + parity * CLUSTER * N;
    parity ^= 1;
    if (threadIdx.x < CLUSTER * N) {
        const int r = threadIdx.x / N, k = threadIdx.x - r * N;
        double s = 0.0;
        for (int i = 0; i < CL_THREADS / 32; ++i) s += sh[k][i];
        cl.map_shared_rank(at, r)[rank * N + k] = s;
    }
    cl.sync();
#pragma unroll
    for (int k = 0; k < N; ++k) {
        v[k] = 0.0;
        for (int r = 0; r < CLUSTER; ++r) v[k] += at[r * N + k];
    }
}

// Levels 2 and below of CTA 0 (their right-hand sides in place): R right-hand sides side by
// side, CL_THREADS / R threads each.
template <int R>
__device__ __forceinline__ void deep_cycle(unsigned char *sm, const ClusterLayout &Y, const ClusterSolve &A,
                                           const int *nx, const int *ny, const unsigned *inv_ny,
                                           const unsigned *inv_half) {
    constexpr int T = CL_THREADS / R;
    const int rhs = threadIdx.x / T, i = threadIdx.x - rhs * T;
    auto view = [&](int l) {
        LevelView V;
        V.nx = nx[l];
        V.ny = ny[l];
        V.n = nx[l] * ny[l];
        V.inv_ny = inv_ny[l];
        V.inv_half = inv_half[l];
        V.k = reinterpret_cast<const float4 *>(sm + Y.kd[l]);
        V.d = reinterpret_cast<const float *>(sm + Y.kd[l]) + 4 * V.n;
        V.x = reinterpret_cast<float *>(sm + Y.xb[l] + rhs * Y.per_rhs);
        V.b = V.x + V.n;
        return V;
    };
    for (int l = 2; l + 1 < A.nlev; ++l) {
        const LevelView L = view(l), C = view(l + 1);
        for (int c = i; c < L.n; c += T) L.x[c] = first_colour(L, c, L.b[c]);
        __syncthreads();
        const int nc = colours(L);
        for (int k = 0; k < A.pre; ++k)
            for (int c = k == 0 ? 1 : 0; c < nc; ++c) {
                smooth_colour<1>(L, c, i, T);
                __syncthreads();
            }
        restrict_residual(L, C, i, T);
        __syncthreads();
    }
    {
        const LevelView L = view(A.nlev - 1);
        const float *M = reinterpret_cast<const float *>(sm + Y.coarse);
        for (int row = i; row < L.n; row += T) {
            float s0 = 0.f, s1 = 0.f;
            int c = 0;
            for (; c + 1 < L.n; c += 2) {
                s0 = fmaf(M[c * L.n + row], L.b[c], s0);
                s1 = fmaf(M[(c + 1) * L.n + row], L.b[c + 1], s1);
            }
            if (c < L.n) s0 = fmaf(M[c * L.n + row], L.b[c], s0);
            L.x[row] = s0 + s1;
        }
        __syncthreads();
    }
    for (int l = A.nlev - 2; l >= 2; --l) {
        const LevelView L = view(l), C = view(l + 1);
        prolong<2>(L, C, i, T);
        __syncthreads();
        const int nc = colours(L);
        for (int k = 0; k < A.post; ++k)
            for (int c = nc - 1; c >= 0; --c) {
                smooth_colour<1>(L, c, i, T);
                __syncthreads();
            }
    }
}

// FP64 residual and convergence test, FP32 PCG with V-cycles, FP64 correction, repeated (the steps
// of tb_poisson_solve's launch loop), for R right-hand sides.  They stop together; one that has
// converged is left as it is.
template <int R>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(CL_THREADS, 1) k_solve_cluster(const ClusterSolve A) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int nx[CL_MAX_LEVELS], ny[CL_MAX_LEVELS];
    __shared__ unsigned inv_ny[CL_MAX_LEVELS], inv_half[CL_MAX_LEVELS];
    __shared__ ClusterLayout Y;
    cg::cluster_group cl = cg::this_cluster();
    const int t = threadIdx.x, rank = (int)cl.block_rank();
    if (t < A.nlev) {
        nx[t] = A.lev[t].nx;
        ny[t] = A.lev[t].ny;
        inv_ny[t] = A.lev[t].inv_ny;
        inv_half[t] = A.lev[t].inv_half;
    }
    __syncthreads();
    if (t == 0) Y = cluster_layout(nx, ny, A.nlev, R);
    __syncthreads();
    const int active = (nx[2] + (nx[2] + CLUSTER - 1) / CLUSTER - 1) / ((nx[2] + CLUSTER - 1) / CLUSTER);
    const int lrank = rank == 0 ? active - 1 : rank - 1, rrank = rank + 1 >= active ? 0 : rank + 1;
    auto block = [&](int l, int r) {
        Block B;
        const Columns c = columns_of(rank, l, nx[l], nx[2]), cleft = columns_of(lrank, l, nx[l], nx[2]);
        B.nx = nx[l];
        B.ny = ny[l];
        B.inv_ny = inv_ny[l];
        B.inv_half = inv_half[l];
        B.x0 = c.x0;
        B.w = c.w;
        B.x = reinterpret_cast<float *>(sm + (l == 0 ? Y.x0 : Y.x1) + r * Y.per_rhs);
        B.b = reinterpret_cast<float *>(sm + (l == 0 ? Y.r0 : Y.b1) + r * Y.per_rhs);
        B.k = reinterpret_cast<const float4 *>(sm + (l == 0 ? Y.k0 : Y.k1));
        B.d = reinterpret_cast<const float *>(sm + (l == 0 ? Y.d0 : Y.d1));
        B.left = cl.map_shared_rank(B.x, rank < active ? lrank : rank) + (cleft.w + 1) * B.ny;
        B.right = cl.map_shared_rank(B.x, rank < active ? rrank : rank);
        return B;
    };
    // the operator
    for (int l = 0; l < 2; ++l) {
        const Block B = block(l, 0);
        const int o = B.x0 * B.ny;
        for (int c = t; c < B.w * B.ny; c += CL_THREADS) {
            const_cast<float4 *>(B.k)[c] = A.lev[l].k4[o + c];
            const_cast<float *>(B.d)[c] = A.lev[l].df[o + c];
        }
    }
    if (rank == 0) {
        for (int l = 2; l < A.nlev; ++l) {
            const int n = nx[l] * ny[l];
            float4 *k = reinterpret_cast<float4 *>(sm + Y.kd[l]);
            float *d = reinterpret_cast<float *>(k) + 4 * n;
            for (int c = t; c < n; c += CL_THREADS) {
                k[c] = A.lev[l].k4[c];
                d[c] = A.lev[l].df[c];
            }
        }
        const int nc = nx[A.nlev - 1] * ny[A.nlev - 1];
        for (int c = t; c < nc * nc; c += CL_THREADS) reinterpret_cast<float *>(sm + Y.coarse)[c] = A.coarse[c];
    }
    double *sums = reinterpret_cast<double *>(sm + Y.sums);
    int parity = 0;
    cl.sync();   // every CTA has started: its shared memory may be written from here on

    const Block F0 = block(0, 0), C0 = block(1, 0);
    const int FY = F0.ny, own = F0.w * FY, n = nx[0] * FY;
    const unsigned inv_fy = F0.inv_ny;
    const int left_halo = (columns_of(lrank, 0, nx[0], nx[2]).w + 1) * FY;
    // the cells this thread owns: local column and row of cell t + j CL_THREADS of the block
    auto place = [&](int j, int *lc, int *iy) {
        const int c = t + j * CL_THREADS;
        if (c >= own) return -1;
        const int col = quotient(c, FY, inv_fy);
        *lc = col + 1;
        *iy = c - col * FY;
        return c;
    };
    const int rhs0 = blockIdx.x / CLUSTER * R;
    int outer = 0;
    double nr[R], bb[R], aa[R], last[R];
    int count[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        last[r] = INFINITY;
        count[r] = 0;
    }
    for (;;) {
        // r64 = b - L x and the magnitudes its rounding is measured by
        double v64[R][CL_CELLS], sum[3 * R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            sum[3 * r] = sum[3 * r + 1] = sum[3 * r + 2] = 0.0;
            const bool there = rhs0 + r < A.nrhs;
            const double *x = A.x + (size_t)(there ? rhs0 + r : 0) * n, *b = A.b + (size_t)(there ? rhs0 + r : 0) * n;
#pragma unroll
            for (int j = 0; j < CL_CELLS; ++j) {
                int lc, iy;
                v64[r][j] = 0.0;
                if (place(j, &lc, &iy) < 0 || !there) continue;
                const int ix = F0.x0 + lc - 1, c = ix * FY + iy;
                const int w = (ix == 0 ? nx[0] - 1 : ix - 1) * FY + iy, e = (ix == nx[0] - 1 ? 0 : ix + 1) * FY + iy;
                const double t0 = A.d64[c] * x[c], t1 = A.ke64[c] * x[e], t2 = A.ke64[w] * x[w];
                const double t3 = iy + 1 < FY ? A.kn64[c] * x[c + 1] : 0.0, t4 = iy > 0 ? A.kn64[c - 1] * x[c - 1] : 0.0;
                const double bv = b[c], v = bv - (t0 - t1 - t2 - t3 - t4);
                const double a = fabs(bv) + fabs(t0) + fabs(t1) + fabs(t2) + fabs(t3) + fabs(t4);
                v64[r][j] = v;
                sum[3 * r] += v * v;
                sum[3 * r + 1] += bv * bv;
                sum[3 * r + 2] += a * a;
            }
        }
        cluster_sum<3 * R>(cl, sum, sums, parity);
        // A guess within the tolerance stays as it is.  Otherwise refined to a tenth of the tolerance
        // (the launches refine every side as long as the worst needs it, most of them further than
        // the tolerance), or to the residual's own rounding floor (see tb_poisson_solve); once within
        // the tolerance, no further than it still falls.
        bool go[R], any = false;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            nr[r] = sqrt(sum[3 * r]);
            bb[r] = sqrt(sum[3 * r + 1]);
            aa[r] = sqrt(sum[3 * r + 2]);
            const double rel = bb[r] > 0 ? nr[r] / bb[r] : nr[r];
            go[r] = count[r] == outer && rhs0 + r < A.nrhs &&
                    !(rel <= (outer == 0 ? A.rtol : 0.1 * A.rtol) || nr[r] <= 32.0 * DBL_EPSILON * aa[r] || outer >= A.max_outer ||
                      (rel <= A.rtol && rel > 0.5 * last[r]));
            last[r] = rel;
            any = any || go[r];
            if (go[r]) ++count[r];
        }
        if (!any) break;
        ++outer;
        float e[R][CL_CELLS], q[R][CL_CELLS];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const Block F = block(0, r);
            const double inv = nr[r] > 0 ? 1.0 / nr[r] : 0.0;
#pragma unroll
            for (int j = 0; j < CL_CELLS; ++j) {
                int lc, iy;
                const int c = place(j, &lc, &iy);
                e[r][j] = q[r][j] = 0.f;
                if (c < 0) continue;
                const float v = (float)(v64[r][j] * inv);
                F.b[c] = v;
                put(F, F.x, F.left, F.right, lc, iy, start_value(F, F.x0 + lc - 1, iy, v, F.d[c]));
            }
        }
        cl.sync();
        double rz_old[R];
#pragma unroll
        for (int r = 0; r < R; ++r) rz_old[r] = 0.0;
        const int nc0 = (nx[0] & 1) ? 4 : 2, nc1 = (nx[1] & 1) ? 4 : 2;
        for (int it = 0; it < A.inner; ++it) {
            // z = M r: one symmetric V-cycle (its first colour was smoothed with r)
            for (int k = 0; k < A.pre; ++k)
                for (int c = k == 0 ? 1 : 0; c < nc0; ++c) {
#pragma unroll
                    for (int r = 0; r < R; ++r) block_colour(block(0, r), c);
                    cl.sync();
                }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block F = block(0, r), C = block(1, r);
                for (int c = t; c < C.w * C.ny; c += CL_THREADS) {
                    const int I = quotient(c, C.ny, C.inv_ny), J = c - I * C.ny;
                    const float v = aggregate_residual(F, I, J);
                    C.b[c] = v;
                    put(C, C.x, C.left, C.right, I + 1, J, start_value(C, C.x0 + I, J, v, C.d[c]));
                }
            }
            cl.sync();
            for (int k = 0; k < A.pre; ++k)
                for (int c = k == 0 ? 1 : 0; c < nc1; ++c) {
#pragma unroll
                    for (int r = 0; r < R; ++r) block_colour(block(1, r), c);
                    cl.sync();
                }
            // level 2's right-hand side, into CTA 0
            const int per2 = (nx[2] + CLUSTER - 1) / CLUSTER, a2 = min(rank * per2, nx[2]);
            const int w2 = min((rank + 1) * per2, nx[2]) - a2;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block C = block(1, r);
                float *b2 = reinterpret_cast<float *>(sm + Y.xb[2] + r * Y.per_rhs) + nx[2] * ny[2];
                float *to = cl.map_shared_rank(b2, 0) + a2 * ny[2];
                for (int c = t; c < w2 * ny[2]; c += CL_THREADS) {
                    const int I = quotient(c, ny[2], inv_ny[2]), J = c - I * ny[2];
                    to[c] = aggregate_residual(C, I, J);
                }
            }
            cl.sync();
            if (rank == 0) deep_cycle<R>(sm, Y, A, nx, ny, inv_ny, inv_half);
            cl.sync();
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block C = block(1, r);
                const float *x2 = cl.map_shared_rank(reinterpret_cast<float *>(sm + Y.xb[2] + r * Y.per_rhs), 0);
                for (int c = t; c < C.w * C.ny; c += CL_THREADS) {
                    const int I = quotient(c, C.ny, C.inv_ny), J = c - I * C.ny;
                    const float up = is_free(C.d[c]) ? x2[((C.x0 + I) >> 1) * ny[2] + (J >> 1)] : 0.f;
                    put(C, C.x, C.left, C.right, I + 1, J, C.x[c + C.ny] + up);
                }
            }
            cl.sync();
            for (int k = 0; k < A.post; ++k)
                for (int c = nc1 - 1; c >= 0; --c) {
#pragma unroll
                    for (int r = 0; r < R; ++r) block_colour(block(1, r), c);
                    cl.sync();
                }
            // (the last colour's barrier above also lets the fine columns read level 1: they are the same CTA's)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block F = block(0, r), C = block(1, r);
#pragma unroll
                for (int j = 0; j < CL_CELLS; ++j) {
                    int lc, iy;
                    const int c = place(j, &lc, &iy);
                    if (c < 0) continue;
                    const float up = is_free(F.d[c]) ? C.x[(((lc - 1) >> 1) + 1) * C.ny + (iy >> 1)] : 0.f;
                    put(F, F.x, F.left, F.right, lc, iy, F.x[c + FY] + up);
                }
            }
            cl.sync();
            for (int k = 0; k < A.post; ++k)
                for (int c = nc0 - 1; c >= 0; --c) {
#pragma unroll
                    for (int r = 0; r < R; ++r) block_colour(block(0, r), c);
                    if (k + 1 < A.post || c > 0) cl.sync();
                    else __syncthreads();       // what follows reads own columns only, up to the next barrier
                }
            double rz[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block F = block(0, r);
                rz[r] = 0.0;
#pragma unroll
                for (int j = 0; j < CL_CELLS; ++j) {
                    int lc, iy;
                    const int c = place(j, &lc, &iy);
                    if (c >= 0) rz[r] += (double)F.b[c] * (double)F.x[c + FY];
                }
            }
            cluster_sum<R>(cl, rz, sums, parity);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block F = block(0, r);
                const float beta = it > 0 && rz_old[r] > 0 ? (float)(rz[r] / rz_old[r]) : 0.f;
                float *p = reinterpret_cast<float *>(sm + Y.p0 + r * Y.per_rhs);
                float *pl = cl.map_shared_rank(p, rank < active ? lrank : rank) + left_halo;
                float *pr = cl.map_shared_rank(p, rank < active ? rrank : rank);
#pragma unroll
                for (int j = 0; j < CL_CELLS; ++j) {
                    int lc, iy;
                    const int c = place(j, &lc, &iy);
                    if (c < 0) continue;
                    const float z = F.x[c + FY];
                    put(F, p, pl, pr, lc, iy, it > 0 ? z + beta * p[c + FY] : z);
                }
            }
            cl.sync();
            double pq[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block F = block(0, r);
                const float *p = reinterpret_cast<const float *>(sm + Y.p0 + r * Y.per_rhs);
                pq[r] = 0.0;
#pragma unroll
                for (int j = 0; j < CL_CELLS; ++j) {
                    int lc, iy;
                    const int c = place(j, &lc, &iy);
                    if (c < 0) continue;
                    const float d = F.d[c], pc = p[c + FY];
                    q[r][j] = is_free(d) ? d * pc - gather4(F.k[c], p, c + FY, FY, iy) : 0.f;
                    pq[r] += (double)q[r][j] * (double)pc;
                }
            }
            cluster_sum<R>(cl, pq, sums, parity);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const Block F = block(0, r);
                const float *p = reinterpret_cast<const float *>(sm + Y.p0 + r * Y.per_rhs);
                const float alpha = (pq[r] > 0 && rz[r] > 0) ? (float)(rz[r] / pq[r]) : 0.f;
                rz_old[r] = rz[r];
#pragma unroll
                for (int j = 0; j < CL_CELLS; ++j) {
                    int lc, iy;
                    const int c = place(j, &lc, &iy);
                    if (c < 0) continue;
                    e[r][j] += alpha * p[c + FY];
                    const float v = F.b[c] - alpha * q[r][j];
                    F.b[c] = v;
                    put(F, F.x, F.left, F.right, lc, iy, start_value(F, F.x0 + lc - 1, iy, v, F.d[c]));
                }
            }
            cl.sync();
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!go[r]) continue;
            double *x = A.x + (size_t)(rhs0 + r) * n;
#pragma unroll
            for (int j = 0; j < CL_CELLS; ++j) {
                int lc, iy;
                if (place(j, &lc, &iy) >= 0) x[(F0.x0 + lc - 1) * FY + iy] += nr[r] * (double)e[r][j];
            }
        }
        cl.sync();
    }
    if (rank == 0 && t < R && rhs0 + t < A.nrhs) {
        double *sc = A.scal + (size_t)(rhs0 + t) * 8;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r == t) {
                sc[S_RR] = nr[r] * nr[r];
                sc[S_BB] = bb[r] * bb[r];
                sc[S_AA] = aa[r] * aa[r];
                sc[S_OUTER] = (double)count[r];
            }
    }
    cl.sync();   // no CTA leaves while another may still write to its shared memory
}

// q = L p (FP32, fine level); per-block partial sums of p.q into part
__global__ void k_matvec_dot(int nx, int ny, const float *d, const float *ke, const float *kn, const uint8_t *fixed,
                             const float *p, float *q, double *part) {
    const int n = nx * ny, rhs = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    double acc = 0;
    if (c < n) {
        const size_t o = (size_t)rhs * n;
        const float v = fixed[c] ? 0.f : apply_at(d, ke, kn, p + o, nx, ny, c);
        q[o + c] = v;
        acc = (double)v * (double)p[o + c];
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part[((size_t)rhs * gridDim.x + blockIdx.x) * PART] = acc;
}

// x += a p ; r -= a q with a = rz / pq
__global__ void k_axpy(int n, const float *p, const float *q, float *x, float *r, const double *scal) {
    const int rhs = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double pq = scal[rhs * 8 + S_PQ], rz = scal[rhs * 8 + S_RZ];
    const float a = (pq > 0 && rz > 0) ? (float)(rz / pq) : 0.f;
    const size_t o = (size_t)rhs * n + c;
    x[o] += a * p[o];
    r[o] -= a * q[o];
}

// per-block partial sums of r.z into part
__global__ void k_dot(int n, const float *r, const float *z, double *part) {
    const int rhs = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    double acc = 0;
    if (c < n) {
        const size_t o = (size_t)rhs * n + c;
        acc = (double)r[o] * (double)z[o];
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part[((size_t)rhs * gridDim.x + blockIdx.x) * PART] = acc;
}

// p = z + b p with b = rz_new / rz (p = z when first)
__global__ void k_update_p(int n, const float *z, float *p, const double *scal, int first) {
    const int rhs = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const size_t o = (size_t)rhs * n + c;
    if (first) { p[o] = z[o]; return; }
    const double rz = scal[rhs * 8 + S_RZ], rzn = scal[rhs * 8 + S_RZ_NEW];
    const float beta = rz > 0 ? (float)(rzn / rz) : 0.f;
    p[o] = z[o] + beta * p[o];
}

// per-rhs scalar bookkeeping between PCG steps
__global__ void k_shift_rz(int nrhs, double *scal) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrhs) return;
    scal[i * 8 + S_RZ] = scal[i * 8 + S_RZ_NEW];
    scal[i * 8 + S_RZ_NEW] = 0;
    scal[i * 8 + S_PQ] = 0;
}

__global__ void k_clear_slots(int nrhs, double *scal, int first, int count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrhs) return;
    for (int k = first; k < first + count; ++k) scal[i * 8 + k] = 0;
}

dim3 grid_for(int n, int nrhs) { return dim3((n + PT - 1) / PT, nrhs); }

// One colour-ordered Gauss-Seidel sweep, forward (0, 1, 2, 3) or backward.
void sweep(const Level &L, int nrhs, bool forward, cudaStream_t s) {
    const dim3 g = grid_for(L.n, nrhs);
    const int ncol = (L.nx & 1) ? 4 : 2;
    for (int k = 0; k < ncol; ++k) {
        const int color = forward ? k : ncol - 1 - k;
        k_smooth<<<g, PT, 0, s>>>(L, color);
    }
}

// z = M r on the fine level (one symmetric V-cycle); r lives in lev[0].b.
void vcycle(tb_poisson *ps, int l, int nrhs, cudaStream_t s) {
    Level &L = ps->lev[l];
    if (l == ps->bottom) {
        k_vcycle_bottom<<<nrhs, CTA_THREADS, ps->bottom_bytes, s>>>(ps->d_lev, l, (int)ps->lev.size(), ps->pre,
                                                                    ps->post, ps->coarse_sweeps);
        return;
    }
    const size_t tot = (size_t)nrhs * L.n;
    k_zero<<<(unsigned)((tot + PT - 1) / PT), PT, 0, s>>>(tot, L.x);
    const dim3 g = grid_for(L.n, nrhs);
    if (l + 1 == (int)ps->lev.size()) {
        for (int k = 0; k < ps->coarse_sweeps; ++k) sweep(L, nrhs, true, s);
        for (int k = 0; k < ps->coarse_sweeps; ++k) sweep(L, nrhs, false, s);
        return;
    }
    for (int k = 0; k < ps->pre; ++k) sweep(L, nrhs, true, s);
    k_resid32<<<g, PT, 0, s>>>(L);
    Level &C = ps->lev[l + 1];
    k_restrict<<<grid_for(C.n, nrhs), PT, 0, s>>>(L, C);
    vcycle(ps, l + 1, nrhs, s);
    k_prolong<<<g, PT, 0, s>>>(L, C);
    for (int k = 0; k < ps->post; ++k) sweep(L, nrhs, false, s);
}

// z = M r : copies r into the level-0 right-hand side, runs the V-cycle, copies x out.
void precondition(tb_poisson *ps, int nrhs, const float *r, float *z, cudaStream_t s) {
    Level &L = ps->lev[0];
    const size_t bytes = (size_t)nrhs * L.n * sizeof(float);
    cudaMemcpyAsync(L.b, r, bytes, cudaMemcpyDeviceToDevice, s);
    vcycle(ps, 0, nrhs, s);
    cudaMemcpyAsync(z, L.x, bytes, cudaMemcpyDeviceToDevice, s);
}

// Builds the coarse operator of level f into c (host arrays).
void coarsen(int fnx, int fny, const std::vector<float> &d, const std::vector<float> &ke,
             const std::vector<float> &kn, const std::vector<uint8_t> &fx, int &cnx, int &cny,
             std::vector<float> &cd, std::vector<float> &cke, std::vector<float> &ckn, std::vector<uint8_t> &cfx) {
    cnx = (fnx + 1) / 2;
    cny = (fny + 1) / 2;
    const int cn = cnx * cny;
    std::vector<double> sd(cn, 0.0), se(cn, 0.0), sn(cn, 0.0);
    std::vector<int> nfree(cn, 0);
    auto agg = [&](int i, int j) { return (i >> 1) * cny + (j >> 1); };
    for (int i = 0; i < fnx; ++i) {
        for (int j = 0; j < fny; ++j) {
            const int f = i * fny + j;
            if (fx[f]) continue;
            const int a = agg(i, j);
            nfree[a]++;
            sd[a] += d[f];
            // east coupling
            const int ie = i + 1 == fnx ? 0 : i + 1;
            const int fe = ie * fny + j;
            if (!fx[fe] && ke[f] != 0.f) {
                const int b = agg(ie, j);
                if (b == a) sd[a] -= 2.0 * ke[f];
                else if (b == (((i >> 1) + 1) == cnx ? 0 : (i >> 1) + 1) * cny + (j >> 1)) se[a] += ke[f];
            }
            if (j + 1 < fny && !fx[f + 1] && kn[f] != 0.f) {
                const int b = agg(i, j + 1);
                if (b == a) sd[a] -= 2.0 * kn[f];
                else sn[a] += kn[f];
            }
        }
    }
    cd.assign(cn, 1.f);
    cke.assign(cn, 0.f);
    ckn.assign(cn, 0.f);
    cfx.assign(cn, 1);
    for (int a = 0; a < cn; ++a) {
        if (!nfree[a]) continue;
        cfx[a] = 0;
        cd[a] = (float)(0.5 * sd[a]);
        cke[a] = (float)(0.5 * se[a]);
        ckn[a] = (float)(0.5 * sn[a]);
    }
    // couplings into fixed coarse cells are dropped
    for (int I = 0; I < cnx; ++I)
        for (int J = 0; J < cny; ++J) {
            const int a = I * cny + J;
            const int e = (I + 1 == cnx ? 0 : I + 1) * cny + J;
            if (cfx[a] || cfx[e]) cke[a] = 0.f;
            if (J + 1 >= cny || cfx[a] || cfx[a + 1]) ckn[a] = 0.f;
        }
}

// Whether level number `count` (from 1) of lnx x lny cells is the last of the hierarchy.
bool is_coarsest(int lnx, int lny, int count) { return lnx * lny <= 64 || lnx <= 2 || lny <= 2 || count >= 16; }

// Shared memory of the one-launch solve with 1 and 2 right-hand sides to a cluster, 0 where the
// grid does not fit: at least three levels, a coarsest one of at most CL_COARSEST cells, the
// blocks' cells within the threads' and the layout within an SM.
void cluster_fit(int nx, int ny, int bytes[2]) {
    int lx[CL_MAX_LEVELS], ly[CL_MAX_LEVELS], n = 0;
    bytes[0] = bytes[1] = 0;
    for (;;) {
        if (n == CL_MAX_LEVELS) return;
        lx[n] = nx;
        ly[n++] = ny;
        if (is_coarsest(nx, ny, n)) break;
        nx = (nx + 1) / 2;
        ny = (ny + 1) / 2;
    }
    if (n < 3 || nx * ny > CL_COARSEST || (long long)lx[0] * ly[0] > CLUSTER * CL_CELLS * CL_THREADS ||
        columns_of(0, 0, lx[0], lx[2]).w * ly[0] > CL_CELLS * CL_THREADS)
        return;
    for (int R = 1; R <= 2; ++R) {
        const int b = cluster_layout(lx, ly, n, R).bytes;
        if (b <= CL_SMEM) bytes[R - 1] = b;
    }
}

// Whether `sides` right-hand sides of n cells are solved by a launch per pass.
bool launches_solve(const tb_poisson *ps, int n, int sides) {
    return ps->cluster_bytes[0] == 0 || (sides > CL_SIDES && n < CL_FEW_CELLS);
}

// The coarsest level's sweeps of the V-cycle (from x = 0, `sweeps` forward then backward) as a
// matrix, by columns: x = C b.
std::vector<float> coarsest_matrix(int nx, int ny, const std::vector<float> &d, const std::vector<float> &ke,
                                   const std::vector<float> &kn, const std::vector<uint8_t> &fx, int sweeps) {
    const int n = nx * ny, nc = (nx & 1) ? 4 : 2;
    std::vector<float> M((size_t)n * n);
    std::vector<double> x(n);
    for (int col = 0; col < n; ++col) {
        std::fill(x.begin(), x.end(), 0.0);
        for (int k = 0; k < 2 * sweeps; ++k)
            for (int q = 0; q < nc; ++q) {
                const int color = k < sweeps ? q : nc - 1 - q;
                for (int ix = 0; ix < nx; ++ix)
                    for (int iy = 0; iy < ny; ++iy) {
                        const int c = ix * ny + iy;
                        const int own = ((nx & 1) && ix == nx - 1) ? 2 + (iy & 1) : ((ix + iy) & 1);
                        if (own != color || fx[c]) continue;
                        const int w = (ix == 0 ? nx - 1 : ix - 1) * ny + iy, e = (ix == nx - 1 ? 0 : ix + 1) * ny + iy;
                        double s = (c == col ? 1.0 : 0.0) + (double)ke[c] * x[e] + (double)ke[w] * x[w];
                        if (iy + 1 < ny) s += (double)kn[c] * x[c + 1];
                        if (iy > 0) s += (double)kn[c - 1] * x[c - 1];
                        x[c] = s / d[c];
                    }
            }
        for (int r = 0; r < n; ++r) M[(size_t)col * n + r] = (float)x[r];
    }
    return M;
}

template <typename T>
int upload(tb_ctx *ctx, T **dst, const T *src, size_t n) {
    if (n == 0) return TB_OK;
    TB_CUDA(ctx, cudaMalloc(dst, n * sizeof(T)));
    if (src) TB_CUDA(ctx, cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice));
    return TB_OK;
}

}  // namespace

void tb_poisson_free(tb_poisson *ps) {
    if (!ps) return;
    for (Level &L : ps->lev) {
        cudaFree(L.d); cudaFree(L.ke); cudaFree(L.kn); cudaFree(L.fixed);
        cudaFree(L.x); cudaFree(L.b); cudaFree(L.r);
        cudaFree(L.k4); cudaFree(L.df);
    }
    cudaFree(ps->d64); cudaFree(ps->ke64); cudaFree(ps->kn64); cudaFree(ps->r64);
    cudaFree(ps->e); cudaFree(ps->pr); cudaFree(ps->pz); cudaFree(ps->pp); cudaFree(ps->pq);
    cudaFree(ps->scal);
    cudaFree(ps->part);
    cudaFree(ps->d_lev);
    cudaFree(ps->d_coarse);
    delete ps;
}

extern "C" int tb_poisson_setup(tb_ctx *ctx, const double *h_diag, const double *h_ke, const double *h_kn,
                                const uint8_t *h_fixed, int max_rhs) {
    if (!ctx) return TB_ERR_ARG;
    if (!h_diag || !h_ke || !h_kn || !h_fixed || max_rhs < 1)
        return tb_fail(ctx, TB_ERR_ARG, "tb_poisson_setup: missing operator arrays or max_rhs < 1");
    TB_CUDA(ctx, cudaSetDevice(ctx->device));
    const int nx = ctx->nx, ny = ctx->ny, n = nx * ny;
    for (int c = 0; c < n; ++c) {
        if (!h_fixed[c] && !(h_diag[c] > 0))
            return tb_fail(ctx, TB_ERR_ARG, "tb_poisson_setup: diagonal must be positive on free cells (cell %d)", c);
        if (h_ke[c] < 0 || h_kn[c] < 0)
            return tb_fail(ctx, TB_ERR_ARG, "tb_poisson_setup: couplings must be non-negative (cell %d)", c);
    }
    if (ctx->poisson) { tb_poisson_free(ctx->poisson); ctx->poisson = nullptr; }
    tb_poisson *ps = new tb_poisson();
    ps->max_rhs = max_rhs;
    // fine level: couplings into fixed cells removed, fixed rows identity
    std::vector<float> d(n), ke(n), kn(n);
    std::vector<uint8_t> fx(h_fixed, h_fixed + n);
    std::vector<double> d64(n), ke64(n), kn64(n);
    for (int ix = 0; ix < nx; ++ix)
        for (int iy = 0; iy < ny; ++iy) {
            const int c = ix * ny + iy;
            const int e = (ix + 1 == nx ? 0 : ix + 1) * ny + iy;
            d64[c] = fx[c] ? 1.0 : h_diag[c];
            ke64[c] = (fx[c] || fx[e]) ? 0.0 : h_ke[c];
            kn64[c] = (iy + 1 >= ny || fx[c] || fx[c + 1]) ? 0.0 : h_kn[c];
            d[c] = (float)d64[c]; ke[c] = (float)ke64[c]; kn[c] = (float)kn64[c];
        }
    int rc = TB_OK;
    if ((rc = upload(ctx, &ps->d64, d64.data(), n)) || (rc = upload(ctx, &ps->ke64, ke64.data(), n)) ||
        (rc = upload(ctx, &ps->kn64, kn64.data(), n))) {
        tb_poisson_free(ps);
        return rc;
    }
    cudaError_t ae = cudaFuncSetAttribute(k_vcycle_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize, BOTTOM_BYTES);
    if (ae == cudaSuccess)
        ae = cudaFuncSetAttribute(k_solve_cluster<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, CL_SMEM);
    if (ae == cudaSuccess)
        ae = cudaFuncSetAttribute(k_solve_cluster<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, CL_SMEM);
    if (ae != cudaSuccess) {
        tb_poisson_free(ps);
        return tb_cuda_check(ctx, ae, "cudaFuncSetAttribute");
    }
    cluster_fit(nx, ny, ps->cluster_bytes);
    if (ps->cluster_bytes[0] > 0) {
        // where the device cannot run such a cluster the launches keep their work vectors
        if (tb_active_clusters(k_solve_cluster<1>, CLUSTER, CL_THREADS, ps->cluster_bytes[0]) < 1)
            ps->cluster_bytes[0] = ps->cluster_bytes[1] = 0;
        else if (ps->cluster_bytes[1] > 0 &&
                 tb_active_clusters(k_solve_cluster<2>, CLUSTER, CL_THREADS, ps->cluster_bytes[1]) < 1)
            ps->cluster_bytes[1] = 0;
    }
    // the one-launch solve keeps its vectors in shared memory
    const size_t sides = launches_solve(ps, n, max_rhs) ? (size_t)max_rhs : 0;
    int lnx = nx, lny = ny;
    for (;;) {
        Level L;
        L.nx = lnx; L.ny = lny; L.n = lnx * lny;
        L.inv_ny = inverse_of(lny);
        L.inv_half = inverse_of((lny + 1) / 2);
        const size_t vec = sides * L.n;
        std::vector<float4> k4(L.n);
        std::vector<float> df(L.n);
        for (int ix = 0; ix < lnx; ++ix)
            for (int iy = 0; iy < lny; ++iy) {
                const int c = ix * lny + iy, w = (ix == 0 ? lnx - 1 : ix - 1) * lny + iy;
                k4[c] = make_float4(ke[c], ke[w], iy + 1 < lny ? kn[c] : 0.f, iy > 0 ? kn[c - 1] : 0.f);
                df[c] = fx[c] ? INFINITY : d[c];
            }
        if ((rc = upload(ctx, &L.k4, k4.data(), L.n)) || (rc = upload(ctx, &L.df, df.data(), L.n)) ||
            (rc = upload(ctx, &L.d, d.data(), L.n)) || (rc = upload(ctx, &L.ke, ke.data(), L.n)) ||
            (rc = upload(ctx, &L.kn, kn.data(), L.n)) || (rc = upload(ctx, &L.fixed, fx.data(), L.n)) ||
            (rc = upload<float>(ctx, &L.x, nullptr, vec)) || (rc = upload<float>(ctx, &L.b, nullptr, vec)) ||
            (rc = upload<float>(ctx, &L.r, nullptr, vec))) {
            ps->lev.push_back(L);
            tb_poisson_free(ps);
            return rc;
        }
        ps->lev.push_back(L);
        if (is_coarsest(lnx, lny, (int)ps->lev.size())) {
            ps->cd = d;
            ps->cke = ke;
            ps->ckn = kn;
            ps->cfx = fx;
            break;
        }
        std::vector<float> cd, cke, ckn;
        std::vector<uint8_t> cfx;
        int cnx, cny;
        coarsen(lnx, lny, d, ke, kn, fx, cnx, cny, cd, cke, ckn, cfx);
        d.swap(cd); ke.swap(cke); kn.swap(ckn); fx.swap(cfx);
        lnx = cnx; lny = cny;
    }
    const size_t vec = sides * n;
    if ((rc = upload<double>(ctx, &ps->r64, nullptr, vec)) || (rc = upload<float>(ctx, &ps->e, nullptr, vec)) ||
        (rc = upload<float>(ctx, &ps->pr, nullptr, vec)) || (rc = upload<float>(ctx, &ps->pz, nullptr, vec)) ||
        (rc = upload<float>(ctx, &ps->pp, nullptr, vec)) || (rc = upload<float>(ctx, &ps->pq, nullptr, vec)) ||
        (rc = upload<double>(ctx, &ps->scal, nullptr, (size_t)max_rhs * 8)) ||
        (rc = upload<double>(ctx, &ps->part, nullptr, sides * ((n + PT - 1) / PT) * PART)) ||
        (rc = upload<Level>(ctx, &ps->d_lev, ps->lev.data(), ps->lev.size()))) {
        tb_poisson_free(ps);
        return rc;
    }
    // the bottom: the first level whose vectors and operator, with those below it, fit in shared memory
    for (int l = (int)ps->lev.size() - 1, bytes = 0; l >= 0; --l) {
        bytes += bottom_level_bytes(ps->lev[l].n);
        if (bytes > BOTTOM_BYTES) break;
        ps->bottom = l;
        ps->bottom_bytes = bytes;
    }
    if (ps->cluster_bytes[0] > 0) {
        const Level &last = ps->lev.back();
        const std::vector<float> M = coarsest_matrix(last.nx, last.ny, ps->cd, ps->cke, ps->ckn, ps->cfx,
                                                     ps->coarse_sweeps);
        if ((rc = upload(ctx, &ps->d_coarse, M.data(), M.size()))) {
            tb_poisson_free(ps);
            return rc;
        }
    }
    ctx->poisson = ps;
    return TB_OK;
}

extern "C" int tb_poisson_schedule(tb_ctx *ctx, int pre, int post, int coarse_sweeps) {
    if (!ctx) return TB_ERR_ARG;
    if (!ctx->poisson) return tb_fail(ctx, TB_ERR_ARG, "tb_poisson_schedule: call tb_poisson_setup first");
    if (pre < 1 || pre > 8 || post < 1 || post > 8 || coarse_sweeps < 1 || coarse_sweeps > 256)
        return tb_fail(ctx, TB_ERR_ARG, "tb_poisson_schedule: sweeps out of range");
    ctx->poisson->pre = pre;
    ctx->poisson->post = post;
    tb_poisson *ps = ctx->poisson;
    if (ps->d_coarse && ps->coarse_sweeps != coarse_sweeps) {
        const Level &last = ps->lev.back();
        const std::vector<float> M = coarsest_matrix(last.nx, last.ny, ps->cd, ps->cke, ps->ckn, ps->cfx, coarse_sweeps);
        TB_CUDA(ctx, cudaSetDevice(ctx->device));
        TB_CUDA(ctx, cudaDeviceSynchronize());   // no solve still reads the old one
        TB_CUDA(ctx, cudaMemcpy(ps->d_coarse, M.data(), M.size() * sizeof(float), cudaMemcpyHostToDevice));
    }
    ps->coarse_sweeps = coarse_sweeps;
    return TB_OK;
}

extern "C" int tb_poisson_levels(const tb_ctx *ctx) {
    return (ctx && ctx->poisson) ? (int)ctx->poisson->lev.size() : 0;
}

extern "C" int64_t tb_poisson_side_bytes(const tb_ctx *ctx) {
    if (!ctx || !ctx->poisson) return 0;
    const tb_poisson *ps = ctx->poisson;
    long long bytes = 8 * sizeof(double);                       // scal
    const long long n = ps->lev[0].n;
    if (!launches_solve(ps, (int)n, ps->max_rhs)) return bytes;
    for (const Level &L : ps->lev) bytes += 3LL * L.n * (long long)sizeof(float);
    bytes += n * (long long)(sizeof(double) + 5 * sizeof(float));   // r64; e, pr, pz, pp, pq
    return bytes + (n + PT - 1) / PT * PART * (long long)sizeof(double);
}

extern "C" int tb_poisson_solve(tb_ctx *ctx, int nrhs, const double *d_b, double *d_x, double rtol, int max_outer,
                                int inner, int *iters, double *h_resid, void *stream) {
    if (!ctx) return TB_ERR_ARG;
    tb_poisson *ps = ctx->poisson;
    if (!ps) return tb_fail(ctx, TB_ERR_ARG, "tb_poisson_solve: call tb_poisson_setup first");
    if (nrhs < 1 || nrhs > ps->max_rhs || !d_b || !d_x || !(rtol > 0) || max_outer < 1 || inner < 1)
        return tb_fail(ctx, TB_ERR_ARG, "tb_poisson_solve: invalid arguments (nrhs=%d, max_rhs=%d)", nrhs,
                       ps->max_rhs);
    TB_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = (cudaStream_t)stream;
    const Level &F = ps->lev[0];
    const int n = F.n;
    const dim3 g = grid_for(n, nrhs);
    const unsigned sb = (unsigned)((nrhs + PT - 1) / PT);
    std::vector<double> sc((size_t)nrhs * 8);
    int outer = 0;
    double worst = 0;
    const bool small = !launches_solve(ps, n, nrhs);
    if (small) {
        ClusterSolve A;
        A.lev = ps->d_lev;
        A.nlev = (int)ps->lev.size();
        A.pre = ps->pre;
        A.post = ps->post;
        A.max_outer = max_outer;
        A.inner = inner;
        A.nrhs = nrhs;
        A.d64 = ps->d64;
        A.ke64 = ps->ke64;
        A.kn64 = ps->kn64;
        A.b = d_b;
        A.x = d_x;
        A.scal = ps->scal;
        A.rtol = rtol;
        A.coarse = ps->d_coarse;
        // two right-hand sides to a cluster share its barriers once there are more than run side by
        // side, 16 of 8 SMs: 16 sides of 33 x 120 cells take 919 us one to a cluster, 1346 two to one
        if (nrhs > 16 && ps->cluster_bytes[1] > 0)
            k_solve_cluster<2><<<(nrhs + 1) / 2 * CLUSTER, CL_THREADS, ps->cluster_bytes[1], s>>>(A);
        else
            k_solve_cluster<1><<<nrhs * CLUSTER, CL_THREADS, ps->cluster_bytes[0], s>>>(A);
        TB_CUDA(ctx, cudaGetLastError());
        TB_CUDA(ctx, cudaMemcpyAsync(sc.data(), ps->scal, sc.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        TB_CUDA(ctx, cudaStreamSynchronize(s));
        for (int k = 0; k < nrhs; ++k) {
            const double rr = sqrt(sc[k * 8 + S_RR]), bb = sqrt(sc[k * 8 + S_BB]);
            worst = fmax(worst, bb > 0 ? rr / bb : rr);
            outer = (int)fmax((double)outer, sc[k * 8 + S_OUTER]);
        }
    }
    while (!small) {
        k_clear_slots<<<sb, PT, 0, s>>>(nrhs, ps->scal, 0, 8);
        k_resid64<<<g, PT, 0, s>>>(F.nx, F.ny, ps->d64, ps->ke64, ps->kn64, d_x, d_b, ps->r64, ps->part);
        k_sum_partials<<<(3 * nrhs + PT - 1) / PT, PT, 0, s>>>(nrhs, g.x, 3, ps->part, ps->scal, S_RR);
        TB_CUDA(ctx, cudaMemcpyAsync(sc.data(), ps->scal, sc.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        TB_CUDA(ctx, cudaStreamSynchronize(s));
        worst = 0;
        bool done = true;
        for (int k = 0; k < nrhs; ++k) {
            const double rr = sqrt(sc[k * 8 + S_RR]), bb = sqrt(sc[k * 8 + S_BB]), aa = sqrt(sc[k * 8 + S_AA]);
            const double rel = bb > 0 ? rr / bb : rr;
            if (rel > worst) worst = rel;
            // converged: the relative residual reaches rtol, or the residual is as small as
            // its own FP64 rounding allows (a backward error of 32 eps against the magnitudes
            // of b and of the terms of L x, which on a charged grid, where x is large where b
            // is zero, can lie above rtol |b|)
            if (!(rel <= rtol || rr <= 32.0 * DBL_EPSILON * aa)) done = false;
        }
        if (done || outer >= max_outer) break;
        ++outer;
        // FP32 PCG on L e = r / |r|
        k_normalise<<<g, PT, 0, s>>>(n, ps->r64, ps->pr, ps->e, ps->scal);
        for (int it = 0; it < inner; ++it) {
            precondition(ps, nrhs, ps->pr, ps->pz, s);
            k_dot<<<g, PT, 0, s>>>(n, ps->pr, ps->pz, ps->part);
            k_sum_partials<<<(nrhs + PT - 1) / PT, PT, 0, s>>>(nrhs, g.x, 1, ps->part, ps->scal, S_RZ_NEW);
            k_update_p<<<g, PT, 0, s>>>(n, ps->pz, ps->pp, ps->scal, it == 0);
            k_shift_rz<<<sb, PT, 0, s>>>(nrhs, ps->scal);
            k_matvec_dot<<<g, PT, 0, s>>>(F.nx, F.ny, F.d, F.ke, F.kn, F.fixed, ps->pp, ps->pq, ps->part);
            k_sum_partials<<<(nrhs + PT - 1) / PT, PT, 0, s>>>(nrhs, g.x, 1, ps->part, ps->scal, S_PQ);
            k_axpy<<<g, PT, 0, s>>>(n, ps->pp, ps->pq, ps->e, ps->pr, ps->scal);
        }
        k_correct<<<g, PT, 0, s>>>(n, ps->e, d_x, ps->scal);
        TB_CUDA(ctx, cudaGetLastError());
    }
    if (iters) *iters = outer;
    if (h_resid) *h_resid = worst;
    bool ok = true;
    for (int k = 0; k < nrhs; ++k) {
        const double rr = sqrt(sc[k * 8 + S_RR]), bb = sqrt(sc[k * 8 + S_BB]), aa = sqrt(sc[k * 8 + S_AA]);
        ok = ok && ((bb > 0 ? rr / bb : rr) <= rtol || rr <= 32.0 * DBL_EPSILON * aa);
    }
    if (!ok)
        return tb_fail(ctx, TB_ERR_CONVERGENCE, "Poisson solve reached %d refinement steps at relative residual %.3e",
                       outer, worst);
    return TB_OK;
}

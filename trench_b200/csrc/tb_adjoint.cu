// Adjoint of the charging loop: history tallies, the surrogate recurrence over the
// stored histories, and its reverse sweep.
//
// Likelihood-ratio reweighting.  Ion energies and angles are drawn from histogram
// tables with bin probabilities p_k.  Changing them to r_k p_k reweights every
// traced ion by r(bin); with the trajectories held fixed, the expected ion deposit
// of batch b on surface slot s becomes
//     ci_b[s](r) = Ni_b[s] + sum_k (rE_k - 1) TE_b[k][s] + sum_l (rA_l - 1) TA_b[l][s]
// (first order in r - 1; at r = 1 it is the traced count), TE/TA the per-bin
// tallies of the absorbed ions.  d ci_b / d r_k = T_b[k] is the score-function
// (likelihood-ratio) estimator of the deposit's sensitivity to the bin weight.
//
// The charge update over those deposits is the recurrence of tb_step_charge
// (trench_charging_2d.py:1239-1266: deposit, leakage, driven or floating
// conductor), same arithmetic, so at r = 1 it reproduces the traced run's surface
// charge (to the rounding of the real-valued sums, which tb_step_charge may add in
// another order).  Its adjoint, per batch in reverse, with
// lambda = dJ / d rho_{b+1}:
//   floating conductor  rho_{b+1} = r' + e_c C (dV - drift) / dx^2,
//                       drift = dx^2 sum_s g_s (r'_s - rho_b,s), dV = f(ni, ne, drift)
//     => lambda'_s = lambda_s + kappa g_s, kappa = lambda_c C (df/dx_i - 1),
//        dJ/d ni = lambda_c (q / dx^2) df/dx_i, dJ/d ne = lambda_c (q / dx^2) df/dx_e,
//        and -kappa g_s flows to rho_b
//   driven conductor    lambda'_s = 0 on conductor slots
//   leakage             r' = M (r dx^2 + h) / dx^2  =>  u = M^T lambda'
//   deposit             r = rho_b + (ci - ce) q / dx^2 (0 on conductors)
//     => lambda_b = u - kappa g,  mu_s = dJ/d ci_s = u_s q / dx^2 (+ dJ/d ni on the
//        conductor, + dJ/d bottom_b on bottom slots)
//   parameters          dJ/d r_k += sum_s T_b[k][s] mu_s.
// Field feedback (optional): the traced deposits themselves depend on rho_b through
// the field.  With their response measured along orthonormal surface-charge modes V
// (ci(rho) ~ ci + Ui V^T (rho - rho_b), ce likewise with Ue),
//     lambda_b += V (Ui^T mu + Ue^T mu_e),  mu_e_s = dJ/d ce_s
// (-u_s q / dx^2 off the conductor, dJ/d ne on it).
// f is the semi-implicit conductor step (trench_charging_2d.py:815-830):
//   x_i = q ni / C + drift, x_e = q ne / C, k = x_i / Te, frac = (1 - e^-k) / k,
//   f = -Te logaddexp(-k, L), L = log(x_e frac / Te);
//   df/dx_i = s1 - s2 (1/(e^k - 1) - 1/k), df/dx_e = -Te s2 / x_e,
//   s1 = 1 / (1 + e^(k + L)), s2 = 1 - s1 (the weights of logaddexp's arguments).
//
// Compiled with -fmad=false, like the step kernels it mirrors.
#include <cooperative_groups.h>
#include <math.h>

#include "tb_internal.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int ONE_BLOCK = 1024;

__device__ double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
    __syncthreads();
    return t;  // valid in thread 0
}

__device__ double logaddexp(double x, double y) {
    if (x == y) return x + 0.693147180559945309417232121458176568;
    const double t = x - y;
    if (t > 0) return x + log1p(exp(-t));
    if (t <= 0) return y + log1p(exp(t));
    return t;  // NaN
}

__device__ double conductor_step(double n_i, double n_e, double q, double C, double Te, double drift) {
    const double x_i = q * n_i / C + drift, x_e = q * n_e / C;
    if (n_e == 0) return x_i;
    const double k = x_i / Te;
    const double frac = k != 0 ? -expm1(-k) / k : 1.0;
    return -Te * logaddexp(-k, log(x_e / Te * frac));
}

// d(conductor_step)/d x_i (= d/d drift) and d/d x_e.  With no electron deposit the
// step is x_i itself.
__device__ void conductor_partials(double n_i, double n_e, double q, double C, double Te, double drift,
                                   double *f_xi, double *f_xe) {
    if (n_e == 0) { *f_xi = 1.0; *f_xe = 0.0; return; }
    const double x_i = q * n_i / C + drift, x_e = q * n_e / C;
    const double k = x_i / Te;
    const double frac = k != 0 ? -expm1(-k) / k : 1.0;
    const double L = log(x_e / Te * frac);
    const double s1 = 1.0 / (1.0 + exp(k + L)), s2 = 1.0 / (1.0 + exp(-(k + L)));
    // d log(frac) / dk = 1/(e^k - 1) - 1/k; Laurent series near k = 0
    const double k2 = k * k;
    const double dlf = fabs(k) < 1e-2 ? -0.5 + k * (1.0 / 12.0 - k2 * (1.0 / 720.0 - k2 / 30240.0))
                                      : 1.0 / expm1(k) - 1.0 / k;
    *f_xi = s1 - s2 * dlf;
    *f_xe = -Te * s2 / x_e;
}

__global__ void k_tally(const tb_tally_args a, int ncell, int *err) {
    const long long n = a.n_species;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * n || a.d_status[i] != 1) return;
    const int c = a.d_hit[i];
    const int s = (c >= 0 && c < ncell) ? a.d_slot[c] : -1;
    if (s < 0 || s >= a.m) { atomicCAS(err, TB_DERR_NONE, TB_DERR_OFF_SURFACE); return; }
    const int ne = a.n_energy, na = a.n_angle;
    if (i < n) {
        const int be = a.d_bin_e ? a.d_bin_e[i] : 0, ba = a.d_bin_a ? a.d_bin_a[i] : 0;
        if ((ne > 0 && be >= ne) || (na > 0 && ba >= na)) { atomicCAS(err, TB_DERR_NONE, TB_DERR_BAD_CELL); return; }
        if (ne > 0) atomicAdd(&a.d_table[(size_t)be * a.m + s], 1);
        if (na > 0) atomicAdd(&a.d_table[(size_t)(ne + ba) * a.m + s], 1);
        atomicAdd(&a.d_table[(size_t)(ne + na) * a.m + s], 1);
    } else {
        atomicAdd(&a.d_table[(size_t)(ne + na + 1) * a.m + s], 1);
    }
}

// Reweighted ion deposit on slot s of one table.
__device__ double ion_deposit(const tb_adjoint_args &a, const int32_t *T, int m, int s) {
    const int ne = a.n_energy, na = a.n_angle;
    double ci = (double)T[(size_t)(ne + na) * m + s];
    if (a.d_rE)
        for (int k = 0; k < ne; ++k) ci += (a.d_rE[k] - 1.0) * (double)T[(size_t)k * m + s];
    if (a.d_rA)
        for (int l = 0; l < na; ++l) ci += (a.d_rA[l] - 1.0) * (double)T[(size_t)(ne + l) * m + s];
    return ci;
}

// Forward 1/2: deposit and leakage input (tb_step.cu k_deposit, over table deposits).
__global__ void __launch_bounds__(ONE_BLOCK) k_fwd_deposit(const tb_step_desc d, const tb_adjoint_args a, int b) {
    __shared__ double sh[32];
    const int m = d.m;
    const int32_t *T = a.d_tables + (size_t)b * (a.n_energy + a.n_angle + 2) * m;
    const double dx2 = d.dx * d.dx;
    double ni = 0, ne = 0, bi = 0;
    for (int s = threadIdx.x; s < m; s += blockDim.x) {
        const double ci = ion_deposit(a, T, m, s);
        const double ce = (double)T[(size_t)(a.n_energy + a.n_angle + 1) * m + s];
        const uint8_t f = d.d_sflag[s];
        const double rp = a.d_rho[s];
        d.d_rho_prev[s] = rp;
        double drho = ((ci - ce) * d.q_macro) / dx2;
        if (f & TB_SFLAG_COND) drho = 0.0;
        const double r = rp + drho;
        a.d_rho[s] = r;
        const double qs = r * dx2;
        d.d_work[s] = d.d_leak_h ? qs + d.d_leak_h[s] : qs;
        if (f & TB_SFLAG_COND) { ni += ci; ne += ce; }
        if (f & TB_SFLAG_BOTTOM) bi += ci;
    }
    ni = block_sum(ni, sh);
    ne = block_sum(ne, sh);
    bi = block_sum(bi, sh);
    if (threadIdx.x == 0) {
        a.d_scal[4 * b + 0] = ni;
        a.d_scal[4 * b + 1] = ne;
        a.d_bottom[b] = bi;
    }
}

// y = A x, A row-major (rows, cols), one warp per row; with acc != 0, y += A x.
template <typename T>
__global__ void k_gemv(int rows, int cols, const T *A, const double *x, double *y, int acc) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rows) return;
    const T *r = A + (size_t)warp * cols;
    double s = 0.0;
    for (int c = lane; c < cols; c += 32) s += (double)r[c] * x[c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) y[warp] = acc ? y[warp] + s : s;
}

// Forward 2/2: leakage result, driven conductor, floating-conductor step (k_finish).
__global__ void __launch_bounds__(ONE_BLOCK) k_fwd_finish(const tb_step_desc d, const tb_adjoint_args a, int b) {
    __shared__ double sh[32];
    const double dx2 = d.dx * d.dx;
    const bool leak = d.d_leak_M != nullptr;
    double drift = 0;
    for (int s = threadIdx.x; s < d.m; s += blockDim.x) {
        const uint8_t f = d.d_sflag[s];
        double r = a.d_rho[s];
        if (leak) r = d.d_work[d.m + s] / dx2;
        if (d.driven && (f & TB_SFLAG_COND)) r = 0.0;
        a.d_rho[s] = r;
        if (d.floating) drift += (r - d.d_rho_prev[s]) * d.d_g_s[s];
    }
    drift = block_sum(drift, sh);
    if (threadIdx.x == 0) {
        double dr = 0.0;
        if (d.floating && d.c_slot >= 0) {
            dr = drift * dx2;
            const double ni = a.d_scal[4 * b + 0], ne = a.d_scal[4 * b + 1];
            const double dV = conductor_step(ni, ne, d.q_macro, d.C_cond, d.Te, dr);
            a.d_rho[d.c_slot] += d.C_cond * (dV - dr) / dx2;
        }
        a.d_scal[4 * b + 2] = dr;
    }
}

// Scratch layout of the reverse sweep: [0, m) mu (ion deposits), [m, 2m) mu_e
// (electron deposits), 2m kappa, 2m + 1 dJ/d ni, 2m + 2 dJ/d ne, [2m + 4, ...) the
// feedback coefficients.

// Reverse 1/3: through the conductor step; lambda' into work[0, m).
__global__ void __launch_bounds__(ONE_BLOCK) k_rev_conductor(const tb_step_desc d, const tb_adjoint_args a, int b,
                                                             const double *lambda, double *scratch) {
    __shared__ double kap_sh;
    if (threadIdx.x == 0) {
        double kap = 0.0, jni = 0.0, jne = 0.0;
        if (d.floating && d.c_slot >= 0) {
            double f_xi, f_xe;
            conductor_partials(a.d_scal[4 * b + 0], a.d_scal[4 * b + 1], d.q_macro, d.C_cond, d.Te,
                               a.d_scal[4 * b + 2], &f_xi, &f_xe);
            const double lc = lambda[d.c_slot];
            kap = lc * d.C_cond * (f_xi - 1.0);
            jni = lc * f_xi * d.q_macro / (d.dx * d.dx);
            jne = lc * f_xe * d.q_macro / (d.dx * d.dx);
        }
        kap_sh = kap;
        scratch[2 * d.m] = kap;
        scratch[2 * d.m + 1] = jni;
        scratch[2 * d.m + 2] = jne;
    }
    __syncthreads();
    const double kap = kap_sh;
    for (int s = threadIdx.x; s < d.m; s += blockDim.x) {
        double l = lambda[s];
        if (d.floating) l += kap * d.d_g_s[s];
        if (d.driven && (d.d_sflag[s] & TB_SFLAG_COND)) l = 0.0;
        d.d_work[s] = l;
    }
}

// Reverse 2/3: through the deposit; lambda <- dJ/d rho_b, mu and mu_e into scratch.
__global__ void __launch_bounds__(ONE_BLOCK) k_rev_deposit(const tb_step_desc d, const tb_adjoint_args a, int b,
                                                           double *lambda, const double *gbottom, double *scratch) {
    const double dx2 = d.dx * d.dx;
    const bool leak = d.d_leak_M != nullptr;
    const double kap = scratch[2 * d.m], jni = scratch[2 * d.m + 1], jne = scratch[2 * d.m + 2];
    const double gb = gbottom ? gbottom[b] : 0.0;
    for (int s = threadIdx.x; s < d.m; s += blockDim.x) {
        const uint8_t f = d.d_sflag[s];
        const double u = leak ? d.d_work[d.m + s] : d.d_work[s];
        const bool cond = f & TB_SFLAG_COND;
        double mu = cond ? (d.floating ? jni : 0.0) : u * d.q_macro / dx2;
        if (f & TB_SFLAG_BOTTOM) mu += gb;
        scratch[s] = mu;
        scratch[d.m + s] = cond ? (d.floating ? jne : 0.0) : -(u * d.q_macro / dx2);
        lambda[s] = d.floating ? u - kap * d.d_g_s[s] : u;
    }
}

// Reverse 3/3 (field feedback): lambda += V (Ui^T mu + Ue^T mu_e) with the batch's
// response set; one warp per mode for the coefficients.
__global__ void __launch_bounds__(ONE_BLOCK) k_rev_feedback(const tb_step_desc d, const tb_adjoint_args a, int b,
                                                            double *lambda, double *scratch) {
    const int set = a.d_resp_index[b];
    if (set < 0) return;
    const int m = d.m, K = a.n_basis;
    const double *Ui = a.d_resp_i + (size_t)set * m * K, *Ue = a.d_resp_e + (size_t)set * m * K;
    double *coef = scratch + 2 * m + 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int j = warp; j < K; j += warps) {
        double c = 0.0;
        for (int s = lane; s < m; s += 32)
            c += Ui[(size_t)s * K + j] * scratch[s] + Ue[(size_t)s * K + j] * scratch[m + s];
        for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
        if (lane == 0) coef[j] = c;
    }
    __syncthreads();
    for (int s = threadIdx.x; s < m; s += blockDim.x) {
        double add = 0.0;
        for (int j = 0; j < K; ++j) add += a.d_basis[(size_t)s * K + j] * coef[j];
        lambda[s] += add;
    }
}

// ---- the sweeps of up to FUSED_MAX_M slots: one launch, one cluster ----------------------
//
// The recurrence is a serial chain of small steps (m = 300: a 300 x 300 product and a few
// vectors a batch), so one launch per step is bound by launch latency (five launches a batch in
// the reverse sweep).  Here one cluster of FUSED_CTAS CTAs walks all batches of a call: each CTA owns a
// contiguous range of slots and their rows of M (kept in shared memory across the batches
// when they fit), vectors that every row needs are written to every CTA through distributed
// shared memory, and a batch takes two cluster barriers.  Sums over CTAs are added in rank
// order by every CTA, so all of them hold the same bits and the result does not depend on
// scheduling.  Larger m keeps one launch per step over the whole GPU: there the product
// itself (8 m^2 bytes) outweighs the launches.  A sweep of 50 batches with its copies, 98 table
// rows, us in one launch and in launches: m = 300, 32 modes: forward 830 and 1491, reverse 805 and
// 2091; m = 440: 950, 1751, 913, 2695 (the operator's rows no longer fit shared memory); m = 760:
// 1549, 2008, 1408, 3764; m = 1000: 2185, 2131, 1965, 4688; without modes 2135, 2228, 1577, 1830.
constexpr int FUSED_CTAS = 8;
constexpr int FUSED_MAX_M = 1024;
constexpr int FUSED_THREADS = 1024;
constexpr int FUSED_SMEM = 200 * 1024;
constexpr int FUSED_MAX_BASIS = 256;
constexpr int FUSED_MAX_ROWS = 1024;      // table rows of the reverse sweep
constexpr int FUSED_MAX_BATCHES = 1024;   // batches of a reverse call

struct Slots {
    int m, per, s0, s1;    // all slots; slots of a CTA at most; this CTA's
};
__device__ __forceinline__ Slots slots_of(int m, int rank) {
    Slots r;
    r.m = m;
    r.per = (m + FUSED_CTAS - 1) / FUSED_CTAS;
    r.s0 = min(m, rank * r.per);
    r.s1 = min(m, r.s0 + r.per);
    return r;
}

// Sums of v[0..N) over the CTA, in every thread.
template <int N>
__device__ __forceinline__ void cta_sum(double (&v)[N]) {
    __shared__ double sh[N][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (lane == 0) sh[k][w] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) {
        v[k] = sh[k][lane];
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    __syncthreads();
}

// Row . x for the CTA's row r of the operator (shared memory if M_s is given), one warp.
__device__ __forceinline__ double row_product(const double *M_s, const double *M, int row, int local, int m,
                                              const double *x) {
    const double *a = M_s ? M_s + (size_t)local * m : M + (size_t)row * m;
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    for (int c = lane; c < m; c += 32) s += a[c] * x[c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Shared memory of the sweeps: the operator's rows first (rows = 0: not kept), then doubles.
__host__ __device__ __forceinline__ size_t fused_rows_bytes(int m) {
    return (size_t)((m + FUSED_CTAS - 1) / FUSED_CTAS) * m * sizeof(double);
}

__global__ void __cluster_dims__(FUSED_CTAS, 1, 1) __launch_bounds__(FUSED_THREADS)
    k_fwd_fused(const tb_step_desc d, const tb_adjoint_args a, int keep_rows) {
    extern __shared__ __align__(16) double smem[];
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), t = threadIdx.x, lane = t & 31, w = t >> 5, W = blockDim.x >> 5;
    const Slots S = slots_of(d.m, rank);
    const int m = S.m, ns = S.s1 - S.s0;
    double *M_s = keep_rows ? smem : nullptr;
    double *qs = smem + (keep_rows ? (size_t)S.per * m : 0);    // 2 x m: the leakage input, by batch parity
    double *part = qs + 2 * m;                                  // 2 x FUSED_CTAS x 4: the CTAs' sums
    double *rho = part + 2 * FUSED_CTAS * 4;                    // own slots: charge, and before the batch
    double *prev = rho + S.per, *ce_s = prev + S.per;
    double *wsum = ce_s + S.per;                                // W x per partial deposits
    const bool leak = d.d_leak_M != nullptr;
    const double dx2 = d.dx * d.dx;
    const int ne = a.n_energy, na = a.n_angle, rows = ne + na + 2;
    if (keep_rows && leak)
        for (int i = t; i < ns * m; i += blockDim.x) M_s[i] = d.d_leak_M[(size_t)S.s0 * m + i];
    for (int i = t; i < ns; i += blockDim.x) rho[i] = a.d_rho[S.s0 + i];
    cl.sync();   // every CTA has started: its shared memory may be written from here on
    for (int b = 0; b < a.n_batches; ++b) {
        const int32_t *T = a.d_tables + (size_t)b * rows * m;
        double *qb = qs + (b & 1) * m, *pb = part + (b & 1) * FUSED_CTAS * 4;
        // reweighted deposits: 128 threads' rows by eight slots (a sector of a table row), the rows
        // of a warp summed by shuffles and the warps' sums in warp order
        const int sub = t & 7;
#pragma unroll 4
        for (int i0 = 0; i0 < ns; i0 += 8) {
            const int i = min(i0 + sub, ns - 1);
            double ci = 0.0;
            for (int k = t >> 3; k < rows; k += blockDim.x >> 3) {
                const double v = (double)T[(size_t)k * m + S.s0 + i];
                if (k < ne) ci += a.d_rE ? (a.d_rE[k] - 1.0) * v : 0.0;
                else if (k < ne + na) ci += a.d_rA ? (a.d_rA[k - ne] - 1.0) * v : 0.0;
                else if (k == ne + na) ci += v;
                else ce_s[i] = v;
            }
            ci += __shfl_xor_sync(0xffffffffu, ci, 8);
            ci += __shfl_xor_sync(0xffffffffu, ci, 16);
            if (lane < 8 && i0 + sub < ns) wsum[w * S.per + i0 + sub] = ci;
        }
        __syncthreads();
        double sum[4] = {0.0, 0.0, 0.0, 0.0};   // ni, ne, bottom deposit, drift
        for (int i = t; i < ns; i += blockDim.x) {
            const int s = S.s0 + i;
            const uint8_t f = d.d_sflag[s];
            double ci = 0.0;
            for (int v = 0; v < W; ++v) ci += wsum[v * S.per + i];
            const double ce = ce_s[i], rp = rho[i];
            prev[i] = rp;
            double drho = ((ci - ce) * d.q_macro) / dx2;
            if (f & TB_SFLAG_COND) drho = 0.0;
            const double r = rp + drho;
            rho[i] = r;
            if (leak) {
                const double q = r * dx2;
                const double v = d.d_leak_h ? q + d.d_leak_h[s] : q;
                for (int c = 0; c < FUSED_CTAS; ++c) cl.map_shared_rank(qb, c)[s] = v;
            }
            if (f & TB_SFLAG_COND) { sum[0] += ci; sum[1] += ce; }
            if (f & TB_SFLAG_BOTTOM) sum[2] += ci;
        }
        if (leak) {
            cl.sync();
            for (int i = w; i < ns; i += W) {
                const double v = row_product(M_s, d.d_leak_M, S.s0 + i, i, m, qb);
                if (lane == 0) rho[i] = v / dx2;
            }
        }
        __syncthreads();
        for (int i = t; i < ns; i += blockDim.x) {
            const int s = S.s0 + i;
            if (d.driven && (d.d_sflag[s] & TB_SFLAG_COND)) rho[i] = 0.0;
            if (d.floating) sum[3] += (rho[i] - prev[i]) * d.d_g_s[s];
        }
        cta_sum(sum);
        if (t < FUSED_CTAS)
            for (int k = 0; k < 4; ++k) cl.map_shared_rank(pb, t)[rank * 4 + k] = sum[k];
        cl.sync();
        double tot[4] = {0.0, 0.0, 0.0, 0.0};
        for (int c = 0; c < FUSED_CTAS; ++c)
            for (int k = 0; k < 4; ++k) tot[k] += pb[c * 4 + k];
        const bool step = d.floating && d.c_slot >= 0;
        const double dr = step ? tot[3] * dx2 : 0.0;
        if (t == 0 && step && d.c_slot >= S.s0 && d.c_slot < S.s1) {
            const double dV = conductor_step(tot[0], tot[1], d.q_macro, d.C_cond, d.Te, dr);
            rho[d.c_slot - S.s0] += d.C_cond * (dV - dr) / dx2;
        }
        if (rank == 0 && t == 0) {
            a.d_scal[4 * b + 0] = tot[0];
            a.d_scal[4 * b + 1] = tot[1];
            a.d_scal[4 * b + 2] = dr;
            a.d_bottom[b] = tot[2];
        }
        __syncthreads();
    }
    for (int i = t; i < ns; i += blockDim.x) a.d_rho[S.s0 + i] = rho[i];
    cl.sync();   // no CTA leaves while another may still write to its shared memory
}

__global__ void __cluster_dims__(FUSED_CTAS, 1, 1) __launch_bounds__(FUSED_THREADS)
    k_rev_fused(const tb_step_desc d, const tb_adjoint_args a, double *lambda, const double *gbottom, double *grad,
                int keep_rows) {
    extern __shared__ __align__(16) double smem[];
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), t = threadIdx.x, lane = t & 31, w = t >> 5, W = blockDim.x >> 5;
    const Slots S = slots_of(d.m, rank);
    const int m = S.m, ns = S.s1 - S.s0, K = a.n_basis;
    double *M_s = keep_rows ? smem : nullptr;
    double *lam = smem + (keep_rows ? (size_t)S.per * m : 0);   // 2 x m: lambda before the batch, by parity
    double *l = lam + 2 * m;                                    // m: lambda through the conductor step
    double *coef = l + m;                                       // 2 x FUSED_CTAS x K: the CTAs' shares of the coefficients
    double *mu = coef + 2 * FUSED_CTAS * K, *mu_e = mu + S.per, *u = mu_e + S.per;
    double *wsum = u + S.per;                                   // W x K
    double *gacc = wsum + W * K;                                // table rows: the CTA's share of the gradient
    double *fx = gacc + a.n_energy + a.n_angle;                 // 2 x batches: the conductor step's partials
    const bool leak = d.d_leak_M != nullptr;
    const double dx2 = d.dx * d.dx;
    const int nrow = a.n_energy + a.n_angle;
    const size_t per_table = (size_t)(nrow + 2) * m;
    if (keep_rows && leak)
        for (int i = t; i < ns * m; i += blockDim.x) M_s[i] = a.d_leak_MT[(size_t)S.s0 * m + i];
    int par = 0;
    for (int s = t; s < m; s += blockDim.x) lam[s] = lambda[s];
    for (int k = t; k < nrow; k += blockDim.x) gacc[k] = 0.0;
    const bool step = d.floating && d.c_slot >= 0;
    if (step)
        for (int b = t; b < a.n_batches; b += blockDim.x)
            conductor_partials(a.d_scal[4 * b + 0], a.d_scal[4 * b + 1], d.q_macro, d.C_cond, d.Te, a.d_scal[4 * b + 2],
                               &fx[2 * b], &fx[2 * b + 1]);
    __syncthreads();
    cl.sync();   // every CTA has started: its shared memory may be written from here on
    for (int b = a.n_batches - 1; b >= 0; --b) {
        const double *lb = lam + par * m;
        // through the conductor step
        double kap = 0.0, jni = 0.0, jne = 0.0;
        if (step) {
            const double f_xi = fx[2 * b], f_xe = fx[2 * b + 1];
            const double lc = lb[d.c_slot];
            kap = lc * d.C_cond * (f_xi - 1.0);
            jni = lc * f_xi * d.q_macro / dx2;
            jne = lc * f_xe * d.q_macro / dx2;
        }
        for (int s = t; s < m; s += blockDim.x) {
            double v = lb[s];
            if (d.floating) v += kap * d.d_g_s[s];
            if (d.driven && (d.d_sflag[s] & TB_SFLAG_COND)) v = 0.0;
            l[s] = v;
        }
        __syncthreads();
        for (int i = w; i < ns; i += W) {
            const double v = leak ? row_product(M_s, a.d_leak_MT, S.s0 + i, i, m, l) : l[S.s0 + i];
            if (lane == 0) u[i] = v;
        }
        __syncthreads();
        // through the deposit
        const double gb = gbottom ? gbottom[b] : 0.0;
        for (int i = t; i < ns; i += blockDim.x) {
            const int s = S.s0 + i;
            const uint8_t f = d.d_sflag[s];
            const bool cond = f & TB_SFLAG_COND;
            double v = cond ? (d.floating ? jni : 0.0) : u[i] * d.q_macro / dx2;
            if (f & TB_SFLAG_BOTTOM) v += gb;
            mu[i] = v;
            mu_e[i] = cond ? (d.floating ? jne : 0.0) : -(u[i] * d.q_macro / dx2);
            if (d.floating) u[i] -= kap * d.d_g_s[s];
        }
        __syncthreads();
        // field feedback: lambda += V (Ui^T mu + Ue^T mu_e), a lane per mode
        const int set = K > 0 ? a.d_resp_index[b] : -1;
        if (set >= 0) {
            const double *Ui = a.d_resp_i + (size_t)set * m * K, *Ue = a.d_resp_e + (size_t)set * m * K;
            double *cb = coef + par * FUSED_CTAS * K;
            for (int j0 = 0; j0 < K; j0 += 32) {
                const int j = j0 + lane;
                double c = 0.0;
                if (j < K)
                    for (int i = w; i < ns; i += W)
                        c += Ui[(size_t)(S.s0 + i) * K + j] * mu[i] + Ue[(size_t)(S.s0 + i) * K + j] * mu_e[i];
                if (j < K) wsum[w * K + j] = c;
            }
            __syncthreads();
            for (int j = t; j < K; j += blockDim.x) {
                double c = 0.0;
                for (int v = 0; v < W; ++v) c += wsum[v * K + j];
                for (int r = 0; r < FUSED_CTAS; ++r) cl.map_shared_rank(cb, r)[rank * K + j] = c;
            }
            cl.sync();
            for (int j = t; j < K; j += blockDim.x) {
                double c = 0.0;
                for (int r = 0; r < FUSED_CTAS; ++r) c += cb[r * K + j];
                wsum[j] = c;
            }
            __syncthreads();
            for (int i = w; i < ns; i += W) {
                double v = 0.0;
                for (int j = lane; j < K; j += 32) v += a.d_basis[(size_t)(S.s0 + i) * K + j] * wsum[j];
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) u[i] += v;
            }
            __syncthreads();
        }
        // dJ/d lambda before the batch, to every CTA
        par ^= 1;
        for (int i = t; i < ns * FUSED_CTAS; i += blockDim.x) {
            const int c = i / ns, k = i - c * ns;
            cl.map_shared_rank(lam + par * m, c)[S.s0 + k] = u[k];
        }
        // parameters: dJ/d r_k += sum_s T[k][s] mu_s over the CTA's slots, a warp per row
        const int32_t *T = a.d_tables + (size_t)b * per_table;
        for (int k = w; k < nrow; k += W) {
            double g = 0.0;
            for (int i = lane; i < ns; i += 32) g += (double)T[(size_t)k * m + S.s0 + i] * mu[i];
            for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
            if (lane == 0) gacc[k] += g;
        }
        cl.sync();
    }
    if (rank == 0) {
        for (int s = t; s < m; s += blockDim.x) lambda[s] = lam[par * m + s];
        for (int k = t; k < nrow; k += blockDim.x) {
            double g = 0.0;
            for (int c = 0; c < FUSED_CTAS; ++c) g += cl.map_shared_rank(gacc, c)[k];
            grad[k] += g;
        }
    }
    cl.sync();   // no CTA leaves while another may still write to its shared memory
}


// Dynamic shared memory of the sweeps without the operator's rows, in bytes.
size_t fwd_bytes(int m) {
    const size_t per = (m + FUSED_CTAS - 1) / FUSED_CTAS;
    return (2 * (size_t)m + 2 * FUSED_CTAS * 4 + 3 * per + (FUSED_THREADS / 32) * per) * sizeof(double);
}
size_t rev_bytes(int m, int K, int rows, int batches) {
    const size_t per = (m + FUSED_CTAS - 1) / FUSED_CTAS;
    return (3 * (size_t)m + 2 * FUSED_CTAS * (size_t)K + 3 * per + (FUSED_THREADS / 32) * (size_t)K + rows +
            2 * (size_t)batches) * sizeof(double);
}

// Whether the device runs the sweeps' clusters at their largest; asked once per context.
int ask_clusters(tb_ctx *ctx) {
    if (ctx->adjoint_clusters >= 0) return TB_OK;
    TB_CUDA(ctx, cudaFuncSetAttribute(k_fwd_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_SMEM));
    TB_CUDA(ctx, cudaFuncSetAttribute(k_rev_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_SMEM));
    const int f = tb_active_clusters(k_fwd_fused, FUSED_CTAS, FUSED_THREADS, FUSED_SMEM);
    const int r = tb_active_clusters(k_rev_fused, FUSED_CTAS, FUSED_THREADS, FUSED_SMEM);
    ctx->adjoint_clusters = f < r ? f : r;
    return TB_OK;
}

int check_step(tb_ctx *ctx, const tb_step_desc *d, const tb_adjoint_args *a, const char *who) {
    if (d->m < 1 || !d->d_sflag || !d->d_rho_prev || !d->d_work || !(d->dx > 0))
        return tb_fail(ctx, TB_ERR_ARG, "%s: incomplete step descriptor", who);
    if (d->floating && (!d->d_g_s || !(d->C_cond > 0)))
        return tb_fail(ctx, TB_ERR_ARG, "%s: floating conductor needs g_s and C_cond", who);
    if (a->n_batches < 1 || a->n_energy < 0 || a->n_angle < 0 || !a->d_tables || !a->d_rho || !a->d_scal ||
        !a->d_bottom)
        return tb_fail(ctx, TB_ERR_ARG, "%s: incomplete adjoint arguments", who);
    if ((a->d_rE && a->n_energy < 1) || (a->d_rA && a->n_angle < 1))
        return tb_fail(ctx, TB_ERR_ARG, "%s: reweighting factors for an empty table", who);
    if (a->n_basis < 0 || (a->n_basis > 0 && (!a->d_basis || !a->d_resp_i || !a->d_resp_e || !a->d_resp_index)))
        return tb_fail(ctx, TB_ERR_ARG, "%s: incomplete field-feedback arguments", who);
    return TB_OK;
}

}  // namespace

extern "C" int tb_tally(tb_ctx *ctx, const tb_tally_args *a, void *stream) {
    if (!ctx || !a) return TB_ERR_ARG;
    if (a->n_species < 0 || a->m < 1 || a->n_energy < 0 || a->n_angle < 0 || !a->d_table || !a->d_slot)
        return tb_fail(ctx, TB_ERR_ARG, "tb_tally: invalid arguments");
    if (a->n_species == 0) return TB_OK;
    if (!a->d_status || !a->d_hit || (a->n_energy > 0 && !a->d_bin_e) || (a->n_angle > 0 && !a->d_bin_a))
        return tb_fail(ctx, TB_ERR_ARG, "tb_tally: a particle array is missing");
    TB_CUDA(ctx, cudaSetDevice(ctx->device));
    const long long total = 2 * a->n_species;
    k_tally<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*a, ctx->nx * ctx->ny, ctx->d_err);
    TB_CUDA(ctx, cudaGetLastError());
    return TB_OK;
}

extern "C" int tb_adjoint_forward(tb_ctx *ctx, const tb_step_desc *d, const tb_adjoint_args *a, void *stream) {
    if (!ctx || !d || !a) return TB_ERR_ARG;
    int rc = check_step(ctx, d, a, "tb_adjoint_forward");
    if (rc != TB_OK) return rc;
    TB_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = (cudaStream_t)stream;
    if ((rc = ask_clusters(ctx)) != TB_OK) return rc;
    size_t bytes = fwd_bytes(d->m);
    const int keep = d->d_leak_M && bytes + fused_rows_bytes(d->m) <= (size_t)FUSED_SMEM;
    if (keep) bytes += fused_rows_bytes(d->m);
    if (d->m <= FUSED_MAX_M && ctx->adjoint_clusters > 0) {
        k_fwd_fused<<<FUSED_CTAS, FUSED_THREADS, bytes, s>>>(*d, *a, keep);
        TB_CUDA(ctx, cudaGetLastError());
        return TB_OK;
    }
    const int wpb = 8, blocks = (d->m + wpb - 1) / wpb;
    for (int b = 0; b < a->n_batches; ++b) {
        k_fwd_deposit<<<1, ONE_BLOCK, 0, s>>>(*d, *a, b);
        if (d->d_leak_M)
            k_gemv<double><<<blocks, 32 * wpb, 0, s>>>(d->m, d->m, d->d_leak_M, d->d_work, d->d_work + d->m, 0);
        k_fwd_finish<<<1, ONE_BLOCK, 0, s>>>(*d, *a, b);
    }
    TB_CUDA(ctx, cudaGetLastError());
    return TB_OK;
}

extern "C" int tb_adjoint_reverse(tb_ctx *ctx, const tb_step_desc *d, const tb_adjoint_args *a, double *d_lambda,
                                  const double *d_gbottom, double *d_grad, double *d_scratch, void *stream) {
    if (!ctx || !d || !a) return TB_ERR_ARG;
    int rc = check_step(ctx, d, a, "tb_adjoint_reverse");
    if (rc != TB_OK) return rc;
    if (!d_lambda || !d_scratch || (a->n_energy + a->n_angle > 0 && !d_grad))
        return tb_fail(ctx, TB_ERR_ARG, "tb_adjoint_reverse: lambda, grad and scratch are required");
    if (d->d_leak_M && !a->d_leak_MT)
        return tb_fail(ctx, TB_ERR_ARG, "tb_adjoint_reverse: leakage needs the transposed operator");
    TB_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = (cudaStream_t)stream;
    const int wpb = 8, blocks = (d->m + wpb - 1) / wpb;
    const int rows = a->n_energy + a->n_angle;
    if ((rc = ask_clusters(ctx)) != TB_OK) return rc;
    size_t bytes = rev_bytes(d->m, a->n_basis, rows, a->n_batches);
    const int keep = d->d_leak_M && bytes + fused_rows_bytes(d->m) <= (size_t)FUSED_SMEM;
    if (keep) bytes += fused_rows_bytes(d->m);
    if (d->m <= FUSED_MAX_M && a->n_basis <= FUSED_MAX_BASIS && rows <= FUSED_MAX_ROWS &&
        a->n_batches <= FUSED_MAX_BATCHES && ctx->adjoint_clusters > 0) {
        k_rev_fused<<<FUSED_CTAS, FUSED_THREADS, bytes, s>>>(*d, *a, d_lambda, d_gbottom, d_grad, keep);
        TB_CUDA(ctx, cudaGetLastError());
        return TB_OK;
    }
    const size_t per = (size_t)(rows + 2) * d->m;
    for (int b = a->n_batches - 1; b >= 0; --b) {
        k_rev_conductor<<<1, ONE_BLOCK, 0, s>>>(*d, *a, b, d_lambda, d_scratch);
        if (d->d_leak_M)
            k_gemv<double><<<blocks, 32 * wpb, 0, s>>>(d->m, d->m, a->d_leak_MT, d->d_work, d->d_work + d->m, 0);
        k_rev_deposit<<<1, ONE_BLOCK, 0, s>>>(*d, *a, b, d_lambda, d_gbottom, d_scratch);
        if (a->n_basis > 0) k_rev_feedback<<<1, ONE_BLOCK, 0, s>>>(*d, *a, b, d_lambda, d_scratch);
        if (rows > 0)
            k_gemv<int32_t><<<(rows + wpb - 1) / wpb, 32 * wpb, 0, s>>>(rows, d->m, a->d_tables + (size_t)b * per,
                                                                        d_scratch, d_grad, 1);
    }
    TB_CUDA(ctx, cudaGetLastError());
    return TB_OK;
}

// ugks_lo.cuh -- device-side state of one Couette domain and the second-order (Van-Leer UGKS)
// kernels' parameter blocks.
#pragma once
#include <algorithm>
#include <cmath>

#include "../../include/ugks_b200.h"
#include "ugks_device.cuh"

namespace ugks {

constexpr int kMaxVel = 5 * 512;  // largest velocity set one CTA row covers (5 velocities x 512 threads)
constexpr int kRedSlots = 40;    // max values reduced together in one block_reduce
constexpr int kNDiag = 13;       // per-cell explicit residual-norm contributions

struct LoParams {
    int nx, ny, nvel, ck;
    double dx, dy, area, gm1, pr, omega, mu_ref, cfl, umax, vmax;
    double wall_ux[2];       // bottom, top wall speed (WallUx(3:4))
    double wall_lam[2];      // 1/Tw per wall
    double fixed_dt;         // > 0: Time_global_fixed
    double inv_dx, inv_dy;   // 1/dx, 1/dy for the slope stencils
    double inv_area;         // 1/area when area is a power of two (then x/area == x*inv_area exactly), else 0
    // the research S2CN2 wall variants (ugks_params): kinetic walls, W1T midpoint walls, W1D, W2R
    int s2_kinetic, s2_midpoint, s2_face_time, s2_shared;
    // a tensor-product velocity table (tensor_table): its abscissae per axis, nvel = tnu tnv; 0: none
    int tnu, tnv;
};

// x / area, as a multiplication when that is exact (area a power of two: both operations round the
// same real number x * 2^-e once)
__device__ __forceinline__ double div_area(double x, const LoParams& P) {
    return P.inv_area != 0.0 ? x * P.inv_area : x / P.area;
}

struct LoBuffers {
    const double* u;         // [nvel] velocity table, k = i + j*Nu
    const double* v;
    const double* w;
    const double* tab;       // [8][64] the axes of a tensor table (LoParams::tnu > 0): u, wx, v, wy, then wx for u >= 0,
                             // u < 0 and wy for v >= 0, v < 0
    double* h;               // [nc][nvel] state, cell c = j*nx + i
    double* b;
    double* W;               // [nc][4] conservative variables
    double* sxh;             // [nc][nvel] Van-Leer slopes of h, b in x and y (Interpolation)
    double* syh;
    double* sxb;
    double* syb;
    double* fxh;             // [ny][nx][nvel] x-face micro flux (face i is between cells i-1 and i)
    double* fxb;
    double* fxw;             // [ny][nx][4] x-face macro flux
    double* fyh;             // [ny+1][nx][nvel] y-face micro flux (row 0 / ny are the walls)
    double* fyb;
    double* fyw;             // [ny+1][nx][4]
    double* res_w;           // [nc][4]   res_macro_flux_store
    double* res_h;           // [nc][nvel] res_h_flux_store (moment-projected stream * dt)
    double* res_b;
    double* peq_h;           // [nc][nvel] physical equilibrium (implicit paths)
    double* peq_b;
    double* pcol_h;          // [nc][nvel] physical collision
    double* pcol_b;
    double* dtl;             // [nc] dt_local of the next TimeStep
    double* dt;              // [2] dt_global of the next step; [1] dt of the last completed update
    double* cell_diag;       // [nc][kNDiag]
    double* diag;            // [kNDiag] reduced over cells by the last CTA
    double* wall_aero;       // [2][nx][3] local-frame pnn, pnt, qn per wall face
    unsigned* counter;       // [1] last-CTA counter (self-resetting)
    unsigned* status;        // [1] error bits
    const double* eval;      // [2] {valid, dt}: when valid and dt == dt[0], the slopes, fluxes and rates
                             // of the current state are already in place and the evaluation returns
                             // at entry (nullptr: always evaluate)
    const unsigned* halt;    // [1] nonzero after a rejected step of a multi-step launch sequence.  With
                             // halt set, a kernel returns at entry once this flag or any status bit
                             // is set, so a failure anywhere in a step ends the sequence there
                             // (nullptr: never halted)
};

__device__ __forceinline__ bool halted(const LoBuffers& B) {
    return B.halt != nullptr && (*B.halt != 0u || *B.status != 0u);
}

// true when the evaluation kernels have nothing to do: the cached evaluation is current, or the
// launch sequence has halted
__device__ __forceinline__ bool eval_cached(const LoBuffers& B) {
    return halted(B) || (B.eval != nullptr && B.eval[0] != 0.0 && B.eval[1] == B.dt[0]);
}

__device__ __forceinline__ int wrapx(int i, int nx) { return i < 0 ? i + nx : (i >= nx ? i - nx : i); }

// Velocity slot r of this thread: k, clamped index kk, and whether it is a real velocity.  Velocity
// loops are branch-free: a slot beyond nvel reads a valid velocity with weight 0 and skips stores.
struct Slot {
    int k, kk;
    bool ok;
};
__device__ __forceinline__ Slot slot(int r, int nv) {
    Slot s;
    s.k = threadIdx.x + r * blockDim.x;
    s.ok = s.k < nv;
    s.kk = s.ok ? s.k : nv - 1;
    return s;
}

// Whether (u, v, w) is the tensor product of two rules of at most 64 abscissae each, k = i + j nu
// (InitVelocityFromStructuredFile, mod_InitializeFlow.f90:480-509): u[k] = u_i and v[k] = v_j exactly, and
// w[k] = wx_i wy_j to within 4 units in the last place, the rounding of a product whose factors are
// themselves recovered from the products (the S2 closures use the factors: a table of rounded decimal weights that
// misses this keeps the general kernels).  On success tab holds u, wx, v, wy, each padded to 64 with its last
// abscissa and weight 0, and the weights of the axes' halves (LoBuffers::tab).  tensor_table on the host and the scan of
// the allocation-free entry point on the device apply one rule with one arithmetic, so that a table takes the same
// kernels through both: the factors, up to their common scale, are two alternations of means of the ratios, each
// weight's rounding averaged out, the sums compensated so that a factor is right to about an ulp.
constexpr int kTensorTab = 8 * 64;
// the factor of one abscissa: the mean of its n weights (stride apart) over the other axis's factors
__host__ __device__ inline double tensor_factor(const double* w, int n, int stride, const double* other) {
    double t = 0.0, c = 0.0;
    for (int k = 0; k < n; ++k) comp_add(t, c, w[(size_t)k * stride] / other[k]);
    return (t + c) / (double)n;
}
// whether the weight is its factors' product, rounded (never a fused product and difference), to 4 units in the last place
__host__ __device__ inline bool tensor_weight(double fx, double fy, double w) {
#ifdef __CUDA_ARCH__
    const double p = __dmul_rn(fx, fy), d = __dsub_rn(p, w);
#else
    const double p = fx * fy, d = p - w;
#endif
    return fabs(d) <= 4.0 * 2.220446049250313e-16 * w;
}
inline bool tensor_table(int nv, const double* u, const double* v, const double* w, int* nu_out, int* nv_out,
                         double tab[kTensorTab]) {
    int nu = 1;
    while (nu < nv && v[nu] == v[0]) ++nu;
    if (nv % nu != 0) return false;
    const int nj = nv / nu;
    if (nu < 2 || nj < 2 || nu > 64 || nj > 64) return false;
    for (int k = 0; k < nv; ++k) {
        if (!(u[k] == u[k % nu] && v[k] == v[k - k % nu])) return false;
        if (!(w[k] > 0.0) || !std::isfinite(w[k]) || !std::isfinite(u[k]) || !std::isfinite(v[k])) return false;
    }
    double fx[64], fy[64];
    for (int j = 0; j < nj; ++j) fy[j] = w[(size_t)j * nu] / w[0];
    for (int it = 0; it < 2; ++it) {
        for (int i = 0; i < nu; ++i) fx[i] = tensor_factor(w + i, nj, nu, fy);
        for (int j = 0; j < nj; ++j) fy[j] = tensor_factor(w + (size_t)j * nu, nu, 1, fx);
    }
    for (int a = 0; a < 64; ++a) {
        tab[a] = u[std::min(a, nu - 1)];
        tab[64 + a] = a < nu ? fx[a] : 0.0;
        tab[128 + a] = v[(size_t)std::min(a, nj - 1) * nu];
        tab[192 + a] = a < nj ? fy[a] : 0.0;
        tab[256 + a] = tab[a] >= 0.0 ? tab[64 + a] : 0.0;
        tab[320 + a] = tab[a] >= 0.0 ? 0.0 : tab[64 + a];
        tab[384 + a] = tab[128 + a] >= 0.0 ? tab[192 + a] : 0.0;
        tab[448 + a] = tab[128 + a] >= 0.0 ? 0.0 : tab[192 + a];
    }
    for (int k = 0; k < nv; ++k)
        if (!tensor_weight(fx[k % nu], fy[k / nu], w[k])) return false;
    *nu_out = nu;
    *nv_out = nj;
    return true;
}

// The kernels' parameter block of a domain described by the C ABI's ugks_params, with U_MAX / V_MAX
// of its velocity table (InitVelocityFromStructuredFile, mod_InitializeFlow.f90:508).  Host only;
// shared by the context path and the allocation-free entry point so that both derive the same block.
inline LoParams make_lo_params(const ugks_params& p, double umax, double vmax) {
    LoParams P{};
    P.nx = p.nx; P.ny = p.ny; P.nvel = p.nvel; P.ck = p.ck;
    P.dx = p.dx; P.dy = p.dy;
    P.area = std::fabs((-p.dx) * (-p.dy) - (p.dx) * (-p.dy)) * 0.5;
    {
        int e2 = 0;
        const double m2 = std::frexp(P.area, &e2);
        P.inv_area = (m2 == 0.5 && std::isfinite(P.area)) ? std::ldexp(1.0, 1 - e2) : 0.0;
    }
    P.gm1 = (double)(p.ck + 4) / (double)(p.ck + 2) - 1.0;
    P.pr = p.pr; P.omega = p.omega; P.mu_ref = p.mu_ref; P.cfl = p.cfl;
    P.umax = umax; P.vmax = vmax;
    for (int s = 0; s < 2; ++s) { P.wall_ux[s] = p.wall_ux[s]; P.wall_lam[s] = 1.0 / p.wall_tnative[s]; }
    P.fixed_dt = p.fixed_dt;
    P.inv_dx = 1.0 / p.dx;
    P.inv_dy = 1.0 / p.dy;
    P.s2_kinetic = p.s2_kinetic_wall != 0;
    P.s2_midpoint = p.s2_time_centered != 0;
    P.s2_face_time = p.s2_face_time != 0;
    P.s2_shared = p.s2_shared_predictor != 0;
    return P;
}

// The residual vector `res` of ApplyExplicitUpdate (mod_TimeIntegrator.f90:108-127) from the cell-reduced
// sums dg[kNDiag] (sum of squared rates [0..3], of |W| [4..7], of area^2 [8]).  Host only.
inline void finish_explicit_res(int nx, int ny, const double* dg, double* res) {
    const double SMV = 1.1754943508222875e-38;
    const double ncell = (double)nx * (double)ny;
    const double ords = std::fmax(std::fmax(dg[4], dg[7]), SMV);
    for (int m = 0; m < 4; ++m) {
        const double rel = std::sqrt(ncell * dg[m]) / (dg[4 + m] + SMV);
        const double ab = std::sqrt(dg[m] / std::fmax(dg[8], SMV));
        const bool near0 = dg[4 + m] <= std::sqrt(2.220446049250313e-16) * std::fmax(ords, 2.2250738585072014e-308);
        res[m] = near0 ? ab : rel;
    }
}

// Per-cell TimeStep (mod_Solve.f90:386-405): dt_local = CFL*area/(dy*max(U_MAX,|U|+c)+dx*max(V_MAX,|V|+c))
__device__ __forceinline__ double cell_dt(const LoParams& P, const double w[4], bool& ok) {
    Prim p;
    ok = get_primary(P.gm1, w, p);
    if (!ok) return 0.0;
    const double sos = sqrt(0.5 * (P.gm1 + 1.0) / p.L);
    const double a = fmax(P.umax, fabs(p.U) + sos), bq = fmax(P.vmax, fabs(p.V) + sos);
    return P.cfl * P.area / (P.dy * a + P.dx * bq);
}

// Last-CTA epilogue: dt_global = min(dt_local) (MPI_AllReduce MIN, mod_Solve.f90:409-418) and
// the residual-norm sums (mod_TimeIntegrator.f90:102-106), reduced in a fixed order.
__device__ __forceinline__ void last_cta_epilogue(const LoParams& P, const LoBuffers& B, bool write_dt, bool write_diag,
                                  double* red, double* rout) {
    __shared__ unsigned s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(B.counter, 1u) == (unsigned)(gridDim.x - 1)) ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int nc = P.nx * P.ny;
    double acc[14];
#pragma unroll
    for (int m = 0; m < 13; ++m) acc[m] = 0.0;
    acc[13] = -INFINITY;   // max of -dt_local == -min(dt_local)
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
        if (write_dt) acc[13] = fmax(acc[13], -__ldcg(B.dtl + c));
        if (write_diag) {
#pragma unroll
            for (int m = 0; m < 9; ++m) acc[m] += __ldcg(B.cell_diag + (size_t)c * kNDiag + m);
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[9 + m] = fmax(acc[9 + m], __ldcg(B.cell_diag + (size_t)c * kNDiag + 9 + m));
        }
    }
    block_reduce<9, 5>(acc, red, rout);
    if (threadIdx.x == 0) {
        if (write_diag) {
            for (int m = 0; m < 13; ++m) B.diag[m] = acc[m];
        }
        if (write_dt) {
            B.dt[1] = B.dt[0];   // dt_global of the step that just completed
            B.dt[0] = P.fixed_dt > 0.0 ? P.fixed_dt : -acc[13];
        }
        *B.counter = 0u;
    }
}

}  // namespace ugks

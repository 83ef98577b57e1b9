// ugks_s2_tensor.cuh -- the discrete closure and make_mke on tensor-product velocity tables.
//
// A structured velocity table (k = i + j Nu, u depending on i alone, v on j alone, weight = wx_i wy_j) makes
// the closure Maxwellian a product, exp(-cx^2 / T) exp(-cy^2 / T), so every velocity sum of it times a
// polynomial is a combination of products of 1-D sums: about 2 (Nu + Nv) terms and 2 exponential rows instead of
// Nu Nv terms with one exponential each.  The sums are taken about the Maxwellian's (or the state's) mean,
// so no term cancels against another of larger size.  Eight lanes own one node (four nodes a warp): each
// lane takes every eighth abscissa of both axes, the sums are joined by a butterfly, and the node's scalar
// logic runs on the group's lanes alike, except where several right-hand sides of one 4x4 system are
// wanted: there each lane solves its own.
#pragma once
#include "ugks_s2_math.cuh"

namespace ugks {
namespace {

constexpr int kTG = 8;   // lanes per node

// xor-butterfly sums over the node's lanes: every lane returns the same totals
template <int N>
__device__ __forceinline__ void t_sum(double* v) {
#pragma unroll
    for (int o = kTG / 2; o > 0; o >>= 1)
#pragma unroll
        for (int m = 0; m < N; ++m) v[m] += __shfl_xor_sync(0xffffffffu, v[m], o);
}
__device__ __forceinline__ double t_min(double v) {
#pragma unroll
    for (int o = kTG / 2; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// lane `src` of the node's group
__device__ __forceinline__ double t_get(double v, int src) {
    return __shfl_sync(0xffffffffu, v, ((threadIdx.x & 31) & ~(kTG - 1)) + src);
}

// The 1-D sums of both axes: x[a] = sum_i w_i c_i^a exp(-(x_i - mean)^2 itw), c_i = x_i - center, for a = 0..5, over the
// abscissae (pos) and weights (wt) of an axis of the table (LoBuffers::tab: rows of 64, padded with weight 0), and
// the smallest exponential of each.  R >= abscissae / 8.  A function of its own, as is t_solve: a node runs through it
// six to eight times, and in line the nodes' kernels spent more time fetching instructions than waiting on them
// (stalls 3.0 against 2.1 an issue; 1 % of an S2CN2 step).
struct TAxes {
    double x[6], y[6], ex, ey;
};
template <int R>
__device__ __noinline__ void t_sums(const double* __restrict__ tu, const double* __restrict__ wu, const double* __restrict__ tv,
                                    const double* __restrict__ wv, double mu, double mv, double itw, double cu, double cv,
                                    TAxes* out) {
    const int gl = threadIdx.x & (kTG - 1);
    double s[12], ex = INFINITY, ey = INFINITY;
#pragma unroll
    for (int a = 0; a < 12; ++a) s[a] = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const double xu = __ldg(tu + gl + kTG * r), xv = __ldg(tv + gl + kTG * r);
        const double du = xu - mu, dv = xv - mv, pu = xu - cu, pv = xv - cv;
        const double eu = exp(-(du * du) * itw), ev = exp(-(dv * dv) * itw);
        ex = fmin(ex, eu);
        ey = fmin(ey, ev);
        double a = __ldg(wu + gl + kTG * r) * eu, b = __ldg(wv + gl + kTG * r) * ev;
        s[0] += a;
        s[6] += b;
#pragma unroll
        for (int m = 1; m < 6; ++m) { a = a * pu; b = b * pv; s[m] += a; s[6 + m] += b; }
    }
    t_sum<12>(s);
#pragma unroll
    for (int a = 0; a < 6; ++a) { out->x[a] = s[a]; out->y[a] = s[6 + a]; }
    out->ex = t_min(ex);
    out->ey = t_min(ey);
}

// solve_dense_4x4 (mod_CorrectedWF2DClosure.f90:631-661) as s2_solve4, the pivots' divisions taken as one reciprocal each;
// `least`: the largest pivot that counts as none
__device__ __noinline__ bool t_solve(const double* m, const double* rhs, double* out, double least = 100.0 * DBL_MIN) {
    double a[4][5], x[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int c = 0; c < 4; ++c) a[r][c] = m[r * 4 + c];
        a[r][4] = rhs[r];
    }
    double ip[4];
    bool ok = true;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        int row = p;
        double best = fabs(a[p][p]);
#pragma unroll
        for (int i = p + 1; i < 4; ++i) if (fabs(a[i][p]) > best) { best = fabs(a[i][p]); row = i; }
        ok = ok && best > least && isfinite(best);
#pragma unroll
        for (int i = p + 1; i < 4; ++i) {
            const bool sw = row == i;
#pragma unroll
            for (int c = p; c < 5; ++c) {
                const double t = a[p][c];
                a[p][c] = sw ? a[i][c] : t;
                a[i][c] = sw ? t : a[i][c];
            }
        }
        ip[p] = 1.0 / a[p][p];
#pragma unroll
        for (int i = p + 1; i < 4; ++i) {
            const double f = a[i][p] * ip[p];
#pragma unroll
            for (int c = p + 1; c < 5; ++c) a[i][c] = a[i][c] - f * a[p][c];
        }
    }
#pragma unroll
    for (int i = 3; i >= 0; --i) {
        double v = a[i][4];
#pragma unroll
        for (int c = i + 1; c < 4; ++c) v = v - a[i][c] * x[c];
        x[i] = v * ip[i];
        ok = ok && isfinite(x[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = ok ? x[i] : 0.0;
    return ok;
}

struct TClosure {
    double th[4];   // converged (rho, u, v, T_native)
    double res;     // scaled residual of the moments at th (make_mke's gate)
    double* jac;    // [16] moment Jacobian at th, row-major, in the group's slice of shared memory
};

// w_newton_next with t_solve
__device__ __forceinline__ int t_newton_next(bool new_iter, const WClosure& C, const double res[4], double norm, int iter,
                                             double step[4], double& alpha, double trial[4]) {
    const double tol = 5.0e-13, floor_a = 9.5367431640625e-07;   // 2^-20
    if (new_iter) {
        if (norm <= tol) return W_DONE;
        if (iter > 12) return W_FAIL;
        const double mr[4] = {-res[0], -res[1], -res[2], -res[3]};
        if (!t_solve(C.jac, mr, step)) return W_FAIL;
        alpha = 1.0;
    }
    while (alpha >= floor_a) {
        double nt[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) nt[m] = C.th[m] + alpha * step[m];
        if (nt[0] > 0.0 && nt[3] > 0.0 && isfinite(nt[0]) && isfinite(nt[1]) && isfinite(nt[2]) && isfinite(nt[3])) {
#pragma unroll
            for (int m = 0; m < 4; ++m) trial[m] = nt[m];
            return W_TRIAL;
        }
        alpha = 0.5 * alpha;
    }
    return W_FAIL;
}

// solve_q_first (mod_CorrectedWF2DClosure.f90:331-426) for the target moments w: the accept / backtrack / stop
// logic of w_closure on the 1-D sums.  Every lane of the warp calls it; a group whose `act` is false
// (no node) or whose iteration has ended idles through the others' evaluations.
template <int R>
__device__ bool t_closure(const LoParams& P, const LoBuffers& B, const double w[4], bool act, TClosure& C) {
    const int ck = P.ck;
    const bool lead = (threadIdx.x & (kTG - 1)) == 0;
    double trial[4];
    bool done = !act, ok = false;
    {   // primitive_from_conserved_2d (mod_CorrectedWF2DEquilibrium.f90:25-41)
        const double u = w[1] / w[0], v = w[2] / w[0];
        const double kin = 0.5 * (u * u + v * v), ein = w[3] / w[0] - kin;
        const double temp = 4.0 * ein / (double)(ck + 2);
        if (!(isfinite(w[0]) && isfinite(w[1]) && isfinite(w[2]) && isfinite(w[3]) && w[0] > 0.0 && isfinite(u) &&
              isfinite(v) && isfinite(temp) && temp > 0.0))
            done = true;
        trial[0] = done ? 1.0 : w[0]; trial[1] = done ? 0.0 : u; trial[2] = done ? 0.0 : v; trial[3] = done ? 1.0 : temp;
    }
    WClosure Cw;   // th and the Jacobian slice w_newton_next works on
    Cw.jac = C.jac;
#pragma unroll
    for (int m = 0; m < 4; ++m) Cw.th[m] = trial[m];
    double res[4] = {0.0, 0.0, 0.0, 0.0}, step[4] = {0.0, 0.0, 0.0, 0.0}, alpha = 1.0, norm = 0.0;
    int iter = 0;
    bool first = true;
    for (int guard = 0; guard < 1024; ++guard) {
        if (__all_sync(0xffffffffu, done)) break;
        TAxes ax;   // sum wx cx^a e_x, sum wy cy^b e_y
        const S2Th t = s2_th(trial, ck);
        t_sums<R>(B.tab, B.tab + 64, B.tab + 128, B.tab + 192, t.u, t.v, t.itw, t.u, t.v, &ax);
        auto S = [&](int a, int b) { return t.pref * ax.x[a] * ax.y[b]; };
        const double s00 = S(0, 0), s10 = S(1, 0), s01 = S(0, 1), s11 = S(1, 1), s20 = S(2, 0), s02 = S(0, 2);
        const double c20 = s20 + s02;                          // sums of c^2, c^2 cx, c^2 cy, c^4
        const double c30 = S(3, 0) + S(1, 2), c03 = S(2, 1) + S(0, 3);
        const double c40 = S(4, 0) + 2.0 * S(2, 2) + S(0, 4);
        const double u2 = 0.5 * (t.u * t.u + t.v * t.v), hb = 0.5 * t.ckh;
        // moments (1, u, v, |c|^2 / 2 + b) of q f from f's sums with 1, cx, cy, c^2 and the b part
        auto mom = [&](double f0, double fx, double fy, double f2, double fb, double* m, int st) {
            m[0] = f0;
            m[st] = t.u * f0 + fx;
            m[2 * st] = t.v * f0 + fy;
            m[3 * st] = u2 * f0 + t.u * fx + t.v * fy + 0.5 * f2 + hb * fb;
        };
        double J[16], q[4];
        const double i1 = t.itw, i2 = t.itw * t.itw, d1 = 2.0 * t.itw;
        mom(s00, s10, s01, c20, s00, q, 1);
        mom(t.ir * s00, t.ir * s10, t.ir * s01, t.ir * c20, t.ir * s00, J, 4);
        mom(d1 * s10, d1 * s20, d1 * s11, d1 * c30, d1 * s10, J + 1, 4);
        mom(d1 * s01, d1 * s11, d1 * s02, d1 * c03, d1 * s01, J + 2, 4);
        mom(i2 * c20 - i1 * s00, i2 * c30 - i1 * s10, i2 * c03 - i1 * s01, i2 * c40 - i1 * c20, i2 * c20, J + 3, 4);
        double nres[4], all = 0.0;   // finite if every sum is (magnitudes, so that nothing cancels)
#pragma unroll
        for (int m = 0; m < 16; ++m) all += fabs(J[m]);
#pragma unroll
        for (int m = 0; m < 4; ++m) { all += fabs(q[m]); nres[m] = q[m] - w[m]; }
        const bool fin = isfinite(all);
        // the Maxwellian is positive at every velocity (its smallest value is the product of the axes' smallest)
        const double qmin = t.pref * ax.ex * ax.ey;
        const bool pos = qmin > 0.0 && t.ckh * qmin > 0.0;
        const double nn = fin ? s2_scaled(nres, w) : INFINITY;
        const bool accept = !done && (first ? fin : (fin && (nn < norm || nn <= 5.0e-13)));
        if (accept && lead)
#pragma unroll
            for (int m = 0; m < 16; ++m) C.jac[m] = J[m];
        __syncwarp();
        if (!done) {
            int a;
            if (accept) {
#pragma unroll
                for (int m = 0; m < 4; ++m) { Cw.th[m] = trial[m]; res[m] = nres[m]; }
                norm = nn;
                iter = first ? 1 : iter + 1;
                a = t_newton_next(true, Cw, res, norm, iter, step, alpha, trial);
                if (a == W_DONE && !pos) a = W_FAIL;
            } else if (first) {
                a = W_FAIL;
            } else {
                alpha = 0.5 * alpha;
                a = t_newton_next(false, Cw, res, norm, iter, step, alpha, trial);
            }
            first = false;
            if (a != W_TRIAL) { done = true; ok = a == W_DONE; }
        }
        __syncwarp();
    }
    double rs = 0.0, sc = 1.0;   // make_mke's gate on the moments of M
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        C.th[m] = Cw.th[m];
        rs = fmax(rs, fabs(res[m]));
        sc = fmax(sc, fabs(w[m]));
    }
    C.res = rs / sc;
    return ok;
}

// moments of a closure direction td (s2_dq over the velocities) by the 1-D sums about (ux, vy): a sum of its own, about
// another centre than the Jacobian's, so a gate on it tests the Jacobian and the solve
__device__ __noinline__ void t_direction(const TAxes* ax, const S2Th* th, double ux, double vy, const double* td, double* m) {
    const S2Th& t = *th;
    const double dx = ux - t.u, dy = vy - t.v, ab = td[3] * t.itw, p3 = ab * t.itw;
    const double a1 = 2.0 * t.itw * td[1], a2 = 2.0 * t.itw * td[2];
    const double p0 = td[0] * t.ir - ab + a1 * dx + a2 * dy + p3 * (dx * dx + dy * dy), p1 = a1 + 2.0 * p3 * dx, p2 = a2 + 2.0 * p3 * dy;
    auto S = [&](int a, int b) { return ax->x[a] * ax->y[b]; };
    const double s00 = S(0, 0), s10 = S(1, 0), s01 = S(0, 1), s11 = S(1, 1), s20 = S(2, 0), s02 = S(0, 2);
    const double c20 = s20 + s02, c30 = S(3, 0) + S(1, 2), c03 = S(2, 1) + S(0, 3), c40 = S(4, 0) + 2.0 * S(2, 2) + S(0, 4);
    const double m0 = p0 * s00 + p1 * s10 + p2 * s01 + p3 * c20, mx = p0 * s10 + p1 * s20 + p2 * s11 + p3 * c30;
    const double my = p0 * s01 + p1 * s11 + p2 * s02 + p3 * c03, m2 = p0 * c20 + p1 * c30 + p2 * c03 + p3 * c40;
    m[0] = t.pref * m0;
    m[1] = t.pref * (ux * m0 + mx);
    m[2] = t.pref * (vy * m0 + my);
    m[3] = t.pref * (0.5 * (ux * ux + vy * vy) * m0 + ux * mx + vy * my + 0.5 * m2 + 0.5 * t.ckh * (m0 + ab * s00));
}

// make_mke_prepared (mod_S2D1.f90:111-151) at the closure C of w: the primitive scalars and the closure
// directions of the raw Shakhov terms, whose moments come from 1-D sums about the state's mean.  Lane 0
// of the group solves for K_x, lane 1 (the axes exchanged) for K_y; lanes 2..4 solve for three further
// right-hand sides extra[0..11] when given (the macro slopes of a face node) and return their own solution
// in td.  Returns the gates: M's moments equal w, the moments that every direction leaves, summed anew, are below 2e-12
// (K's as they stand, the others relative to theirs), all finite.
template <int R>
__device__ bool t_mke(const LoParams& P, const LoBuffers& B, const double w[4], const TClosure& C, WMke& M,
                      const double* extra, double td[4]) {
    const int ck = P.ck, gl = threadIdx.x & (kTG - 1);
    double rho, th;
    const bool pok = s2_primitive(w, ck, rho, M.ux, M.vy, th);
    M.lam = 0.5 / th;
    M.coeff = 0.8 * (1.0 - P.pr) * M.lam * M.lam / rho;
    const S2Th t = s2_th(C.th, ck);
    TAxes ax;
    t_sums<R>(B.tab, B.tab + 64, B.tab + 128, B.tab + 192, t.u, t.v, t.itw, M.ux, M.vy, &ax);
    const bool sw = gl & 1;   // the axis of K is the first of (N, O)
    double N[6], O[6];
#pragma unroll
    for (int a = 0; a < 6; ++a) { N[a] = sw ? ax.y[a] : ax.x[a]; O[a] = sw ? ax.x[a] : ax.y[a]; }
    const double un = sw ? M.vy : M.ux, uo = sw ? M.ux : M.vy, l2 = 2.0 * M.lam, pc = t.pref * M.coeff;
    // f = cn (2 lam c^2 - 4): its sums with 1, cn, co, c^2; b adds (2 / ck) cn
    const double s10 = N[1] * O[0];
    const double m0 = l2 * (N[3] * O[0] + N[1] * O[2]) - 4.0 * s10;
    const double mn = l2 * (N[4] * O[0] + N[2] * O[2]) - 4.0 * (N[2] * O[0]);
    const double mo = l2 * (N[3] * O[1] + N[1] * O[3]) - 4.0 * (N[1] * O[1]);
    const double m2 = l2 * (N[5] * O[0] + 2.0 * (N[3] * O[2]) + N[1] * O[4]) - 4.0 * (N[3] * O[0] + N[1] * O[2]);
    const double cn = pc * (un * m0 + mn), co = pc * (uo * m0 + mo);
    double rhs[4];
    rhs[0] = pc * m0;
    rhs[1] = sw ? co : cn;
    rhs[2] = sw ? cn : co;
    rhs[3] = pc * (0.5 * (un * un + uo * uo) * m0 + un * mn + uo * mo + 0.5 * m2 +
                   0.5 * t.ckh * (m0 + 2.0 / (double)ck * s10));
    const bool mine = extra != nullptr && gl >= 2 && gl < 5;
    if (mine)
#pragma unroll
        for (int m = 0; m < 4; ++m) rhs[m] = extra[(gl - 2) * 4 + m];
    bool ok = t_solve(C.jac, rhs, td);
    double sc = 1.0;
    if (mine)
#pragma unroll
        for (int m = 0; m < 4; ++m) sc = fmax(sc, fabs(rhs[m]));
    double mom[4], left = 0.0;
    t_direction(&ax, &t, M.ux, M.vy, td, mom);
#pragma unroll
    for (int m = 0; m < 4; ++m) { left = fmax(left, fabs(rhs[m] - mom[m])); ok = ok && isfinite(mom[m]); }
    ok = ok && left / sc <= 2.0e-12;
#pragma unroll
    for (int m = 0; m < 4; ++m) { M.tdx[m] = t_get(td[m], 0); M.tdy[m] = t_get(td[m], 1); }
    const unsigned grp = 0xffu << ((threadIdx.x & 31) & ~(kTG - 1));
    ok = (__ballot_sync(0xffffffffu, !ok) & grp) == 0u;
    return pok && ok && C.res <= 2.0e-12;
}

// build_targets' sums (mod_S2D1.f90:1246-1300) of one cell in shared memory: its 9 nodes' Maxwellians as products of two
// rows of exponentials (the Gauss weight and rho / (pi T) folded into the x row), and M, K_x, K_y the product times a
// cubic in the velocity whose coefficients are the node's.
// make_mke's gate on the moments of K_x and K_y (2e-12) is taken here on the sums over the nodes, by the kernels that form
// them, with every velocity's own rounding; each node's is t_mke's, by 1-D sums.  Per node and velocity it cost 4 % of an S2CN2
// step more.
constexpr double kTGate = 2.0e-12;
struct STargetNode {   // mean of theta, mean of the state, ck T / 2, the cubic's coefficients
    double u, v, ux, vy, ckh, sl, s0, kb;   // Shakhov factor sl c^2 - s0; kb = 2 coeff / ck
    double x[5], y[5];                      // direction polynomial 1, cx, cy, c^2 of K_x and K_y, and its b part
};
struct STargets {
    double ex[9][64], ey[9][64];
    STargetNode n[9];
    // by the whole CTA, from the node scalars; followed by a barrier
    __device__ __forceinline__ void fill(const LoParams& P, const LoBuffers& B, const S2Buffers& SB, int cc) {
        const int nu = P.tnu, nw = P.tnv, tid = threadIdx.x;
        const double gw[3] = {5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0};
        if (tid < 9) {
            double th[4];
            WMke M;
            w_load_scalars(SB.tscal + ((size_t)cc * 9 + tid) * kS2TScal, th, M);
            const S2Th t = s2_th(th, P.ck);
            STargetNode& c = n[tid];
            c.u = t.u; c.v = t.v; c.ux = M.ux; c.vy = M.vy; c.ckh = t.ckh;
            c.sl = 2.0 * M.lam * M.coeff; c.s0 = 4.0 * M.coeff; c.kb = 2.0 / (double)P.ck * M.coeff;
            const double i2 = t.itw * t.itw;
#pragma unroll
            for (int d = 0; d < 2; ++d) {
                const double* td = d ? M.tdy : M.tdx;
                double* p = d ? c.y : c.x;
                p[0] = td[0] * t.ir - td[3] * t.itw;
                p[1] = 2.0 * t.itw * td[1];
                p[2] = 2.0 * t.itw * td[2];
                p[3] = td[3] * i2;
                p[4] = td[3] * t.itw;
            }
        }
        for (int q = tid; q < 9 * (nu + nw); q += blockDim.x) {
            const int p = q / (nu + nw), a = q - p * (nu + nw);
            const double* o = SB.tscal + ((size_t)cc * 9 + p) * kS2TScal;
            const double itw = 1.0 / o[3];
            if (a < nu) {
                const double d = B.tab[a] - o[1];
                ex[p][a] = gw[p % 3] * gw[p / 3] * (o[0] / (kPi * o[3])) * exp(-(d * d) * itw);
            } else {
                const double d = B.tab[128 + a - nu] - o[2];
                ey[p][a - nu] = exp(-(d * d) * itw);
            }
        }
    }
    // M, K_x, K_y (h and b each) of the velocities k0, k0 + step, ... (those past the table take its last one)
    template <int VPT>
    __device__ __forceinline__ void at(const LoParams& P, const LoBuffers& B, int k0, int step, double a[VPT][6]) const {
        const int nu = P.tnu;
        double uk[VPT], vk[VPT];
        int iu[VPT], iv[VPT];
#pragma unroll
        for (int r = 0; r < VPT; ++r) {
            const int k = min(k0 + r * step, P.nvel - 1);
            iv[r] = k / nu;
            iu[r] = k - iv[r] * nu;
            uk[r] = B.tab[iu[r]];
            vk[r] = B.tab[128 + iv[r]];
#pragma unroll
            for (int m = 0; m < 6; ++m) a[r][m] = 0.0;
        }
#pragma unroll 1
        for (int p = 0; p < 9; ++p) {
            const STargetNode& c = n[p];
#pragma unroll
            for (int r = 0; r < VPT; ++r) {
                const double q = ex[p][iu[r]] * ey[p][iv[r]], qb = c.ckh * q;
                const double cx = uk[r] - c.u, cy = vk[r] - c.v, px = uk[r] - c.ux, py = vk[r] - c.vy;
                const double c2 = cx * cx + cy * cy, sh = c.sl * (px * px + py * py) - c.s0;
                const double kx = px * sh - (c.x[0] + c.x[1] * cx + c.x[2] * cy + c.x[3] * c2);
                const double ky = py * sh - (c.y[0] + c.y[1] * cx + c.y[2] * cy + c.y[3] * c2);
                a[r][0] += q;
                a[r][1] += qb;
                a[r][2] += q * kx;
                a[r][3] += qb * (kx + c.kb * px - c.x[4]);
                a[r][4] += q * ky;
                a[r][5] += qb * (ky + c.kb * py - c.y[4]);
            }
        }
    }
};

}  // namespace
}  // namespace ugks

// ugks_lo_tensor.cu -- the second-order Explicit step on tensor-product velocity tables (LoParams::tnu > 0), sm_100a, FP64.
//
//   k_lo_fluxes_t : Interpolation, the interior faces and the moving walls of one evaluation (k_lo_slopes, k_lo_faces*,
//                   k_lo_walls) in one launch, one CTA a face
//   k_lo_cells_t  : ComputeResidual + ApplyExplicitUpdate (k_lo_cells), one CTA a cell
//
// The kernels of ugks_lo.cu take every velocity sum as a block reduction, five to seven a CTA, each with its barriers
// and a scalar phase behind it, take an exponential a velocity and equilibrium, and read the distribution and its stored
// slopes twice.  Here all sums of the distribution's own are taken in one reduction over one reading of it (the slopes formed
// on the way), about a mean known beforehand.  Then one warp runs the scalar chain while the others take the
// equilibria's sums, whose exponentials are products of two rows on a tensor table.  The equilibria are projected
// (mod_ImplicitCommon.f90:42-82) in the basis 1, cx, cy, c^2 / 2 about their mean, which spans the same corrections with
// the same weights, max(|E|, eps max(1, max |E|)), and gated as there: by the pivots of the Gram matrix in the
// basis 1, u, v, |v|^2 / 2 and by the moments of the projected distribution summed over the velocities.
// ImplicitSteady keeps the kernels of ugks_lo.cu: its gate step is decided by their rounding.
//
// Bound by the latency of its phases (barriers, the scalar chain), by issue, and by spills: the long unrolled loops read
// their scalars from shared memory anew for each velocity (lo_reread), and the cells the old distribution from L2 (13x51x48^2:
// faces 176 -> 163 us, cells 153 -> 136).  The step takes 83 us at 8x64x32^2 and 287 at 13x51x48^2 (the kernels of ugks_lo.cu 117
// and 387).  128 threads a CTA with the table's velocities spread over them, four CTAs an SM; above 1024 velocities 256 threads
// with 10 each, two CTAs an SM (faces 512 with 5: 190 us instead of 175, 320 with 8: 174; cells 512 with 5: 135, 320 with 8:
// 135, 384 with 7: 132 instead of 133).
#include "ugks_s2_tensor.cuh"

namespace ugks {

namespace {

// The CTA's division of labour after its reduction: warp 0 runs the scalar chain, the other warps the equilibria's sums.
// `sync` joins the workers.
struct LoCrew {
    int n, id;      // workers and this thread's place among them
    bool scalar, worker;
    __device__ __forceinline__ LoCrew() {
        scalar = threadIdx.x < 32;
        worker = !scalar;
        n = (int)blockDim.x - 32;
        id = (int)threadIdx.x - 32;
    }
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }
    // the workers' per-thread sums v to their warps' partials red[warp][32] (N <= 32 sums, column m)
    template <int N>
    __device__ __forceinline__ void partial(const double* v, double* red) const {
        constexpr int sh = 5 - ilog2(pow2_ceil(N));
        const double t = warp_halving<N, false>(v);
        const int lane = threadIdx.x & 31;
        if ((lane & ((1 << sh) - 1)) == 0) red[(id >> 5) * 32 + (lane >> sh)] = t;
    }
    __device__ __forceinline__ double total(const double* red, int m) const {
        double t = red[m];
        for (int w = 1; w < n / 32; ++w) t += red[w * 32 + m];
        return t;
    }
};
// the Maxwellian's two rows of exponentials about (U, V) by the workers: ex (times pref), ey
__device__ __forceinline__ void lo_rows_of(const LoCrew& C, const LoParams& P, const double* __restrict__ tab, double U, double V,
                                           double L, double pref, double* ex, double* ey) {
    for (int q = C.id; q < P.tnu + P.tnv; q += C.n) {
        const double d = q < P.tnu ? tab[q] - U : tab[128 + q - P.tnu] - V, e = exp(-L * (d * d));
        if (q < P.tnu) ex[q] = pref * e;
        else ey[q - P.tnu] = e;
    }
}
// the largest product of the two rows
__device__ __forceinline__ double lo_peak(const LoParams& P, const double* ex, const double* ey) {
    double a = 0.0, b = 0.0;
    for (int q = threadIdx.x & 31; q < P.tnu; q += 32) a = fmax(a, ex[q]);
    for (int q = threadIdx.x & 31; q < P.tnv; q += 32) b = fmax(b, ey[q]);
    double v[2] = {a, b};
    warp_max_all<2>(v);
    return v[0] * v[1];
}

// the scalars in shared memory are read again after it: held in registers across an unrolled loop they spilled its state
__device__ __forceinline__ void lo_reread() { asm volatile("" ::: "memory"); }

// Projections (ProjectToConservedMoments, mod_ImplicitCommon.f90:42-82).  Two gates, as the kernels of ugks_lo.cu have them:
// the pivots of the Gram matrix in the basis 1, u, v, |v|^2 / 2 (solve_dense4's rule, which refuses a mean far
// outside the thermal width however well the centred system can be solved), and, in the kernels' last pass, the moments of the
// projected distribution summed over the velocities.
constexpr double kGate = 1.0e-10;
__device__ __forceinline__ double lo_scale(const double w[4]) {
    return fmax(fmax(fmax(fabs(w[0]), fabs(w[1])), fmax(fabs(w[2]), fabs(w[3]))), 1.0);
}
// a projection's targets and what its moments may miss each of them by; a lane a moment compares
struct LoTarget {
    double w[4], tol;
    __device__ __forceinline__ void set(const double t[4]) {
#pragma unroll
        for (int m = 0; m < 4; ++m) w[m] = t[m];
        tol = kGate * lo_scale(t);
    }
    __device__ __forceinline__ bool missed(int m, double moment) const { return !(fabs(moment - w[m]) <= tol); }
};
__device__ __forceinline__ double lo_least(const double G[16]) {
    double ps = DBL_MIN;
#pragma unroll
    for (int m = 0; m < 16; ++m) ps = fmax(ps, fabs(G[m]));
    return 1000.0 * kEps * ps;
}
// lam of a projection from its 14 sums f (moments of the equilibrium and Gram matrix in the basis 1, cx, cy, c^2 / 2 about
// (U, V)) onto the conserved moments tg.  `plain`: the lane takes the system in the basis 1, u, v, |v|^2 / 2 instead, for its
// pivots; a warp's lanes of both kinds run through one solve.
__device__ __forceinline__ bool lo_lambda(const double f[14], double U, double V, const double tg[4], bool plain, double lam[4]) {
    const double K = 0.5 * (U * U + V * V);
    double G[16], least = 100.0 * DBL_MIN;
    gram_expand(f + 4, G);
    double rhs[4] = {tg[0] - f[0], (tg[1] - U * tg[0]) - f[1], (tg[2] - V * tg[0]) - f[2],
                     (tg[3] - U * tg[1] - V * tg[2] + K * tg[0]) - f[3]};
    if (plain) {   // rows, then columns: u = cx + U, v = cy + V, |v|^2 / 2 = c^2 / 2 + U cx + V cy + K
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            G[12 + c] += U * G[4 + c] + V * G[8 + c] + K * G[c];
            G[4 + c] += U * G[c];
            G[8 + c] += V * G[c];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            double* g = G + 4 * r;
            g[3] += U * g[1] + V * g[2] + K * g[0];
            g[1] += U * g[0];
            g[2] += V * g[0];
        }
        rhs[3] += U * rhs[1] + V * rhs[2] + K * rhs[0];
        rhs[1] += U * rhs[0];
        rhs[2] += V * rhs[0];
        least = lo_least(G);
    }
    return t_solve(G, rhs, lam, least);
}

// a microscopic slope (1, vn, vt, |v|^2/2) of a face (dir 0: vn = u, vt = v; 1: vn = v, vt = -u) as a polynomial in the
// velocity about (U, V): p0 + p1 cx + p2 cy + p3 c^2
__device__ __forceinline__ void lo_centred(int dir, const double X[4], double U, double V, double* p) {
    const double gx = dir == 0 ? X[1] : -X[2], gy = dir == 0 ? X[2] : X[1];
    p[0] = X[0] + gx * U + gy * V + 0.5 * X[3] * (U * U + V * V);
    p[1] = gx + X[3] * U;
    p[2] = gy + X[3] * V;
    p[3] = 0.5 * X[3];
}

struct LoFluxC {
    double U, V, l2, kq, qx, qy, lam[4], bf, fh, fb, mxi2, mt[5];   // mean, 2 L, Shakhov factor, heat, lam, ck/(2L), floors
    double a[2][4], b[4], T[4];   // slopes along the normal (left / right, or a wall's), tangential, in time
    LoTarget tg[2];               // the projection's, and a wall's unit shape's
};

// values and slopes of h and b at cell c, velocity k (Interpolation, mod_Interpolation.f90:26-170).  The four limiters
// (sign a + sign b) |a| |b| / (|a| + |b| + tiny), halved above and below, take one reciprocal a field, of the product of its
// two denominators: each is at least 5e-39, and the product leaves the range above no sooner than the numerators do, so the
// slopes last as long as by divisions of their own and a difference of one field that is not finite stays out of the
// other's.  One reciprocal of all four, 3 % faster at 13x51x48^2 (274 against 282 us a step), lost them from
// differences of 1e77 on.  The cell sizes multiply the limited differences.
struct LoVal {
    double h, b, hx, hy, bx, by;
};
__device__ __forceinline__ LoVal lo_val(const LoParams& P, const LoBuffers& B, int c, int i, int j, int k) {
    const int nx = P.nx, nv = P.nvel;
    const size_t q = (size_t)c * nv + k;
    const size_t xm = (size_t)(c - i + wrapx(i - 1, nx)) * nv + k, xp = (size_t)(c - i + wrapx(i + 1, nx)) * nv + k;
    const bool lo = j == 0, up = j == P.ny - 1;   // one-sided slopes on the wall rows
    const size_t row = (size_t)nx * nv, ym = lo ? q : q - row, yp = up ? q : q + row;
    LoVal r;
    r.h = B.h[q];
    r.b = B.b[q];
    const double d[8] = {r.h - B.h[xm], B.h[xp] - r.h, r.h - B.h[ym], B.h[yp] - r.h,
                         r.b - B.b[xm], B.b[xp] - r.b, r.b - B.b[ym], B.b[yp] - r.b};
    double den[4], num[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const double x = d[2 * t], y = d[2 * t + 1], p = x * y;
        den[t] = 0.5 * (fabs(x) + fabs(y) + kSMV);
        num[t] = p > 0.0 ? copysign(p, x) : 0.0;
    }
    const double ih = 1.0 / (den[0] * den[1]), ib = 1.0 / (den[2] * den[3]);
    r.hx = num[0] * (den[1] * ih) * P.inv_dx;
    r.hy = (lo ? d[3] : (up ? d[2] : num[1] * (den[0] * ih))) * P.inv_dy;
    r.bx = num[2] * (den[3] * ib) * P.inv_dx;
    r.by = (lo ? d[7] : (up ? d[6] : num[3] * (den[2] * ib))) * P.inv_dy;
    return r;
}
// the row k / nu of velocity k < 2560, nu <= 64, by a float reciprocal: (k + 1/2) / nu is at least 1/128 off an integer
__device__ __forceinline__ int lo_row(int k, float inv_nu) { return (int)(((float)k + 0.5f) * inv_nu); }

// the projected equilibrium (H, Bq) of the Maxwellian value H0, and its part of the flux (mod_Evolution.f90:396-453 without
// the face values'): Mt1 (equilibrium + Shakhov) + Mt2 (normal and tangential slopes) + Mt3 time slope
__device__ __forceinline__ void lo_equilibrium(const LoFluxC& c, double H0, double cx, double cy, double c2, double& H, double& Bq) {
    const double b0 = H0 * c.bf;
    H = H0 + fmax(H0, c.fh) * (c.lam[0] + c.lam[1] * cx + c.lam[2] * cy + c.lam[3] * (0.5 * c2));
    Bq = b0 + 0.5 * fmax(b0, c.fb) * c.lam[3];
}
__device__ __forceinline__ void lo_poly(const LoFluxC& c, const double* d, double H0, double cx, double cy, double vn, double vt,
                                        double c2ck, double& H, double& Bq, double& gh, double& gb) {
    const double c2 = cx * cx + cy * cy, qd = c.kq * (cx * c.qx + cy * c.qy), sh = 1.0 + qd * (c.l2 * c2 - 4.0);
    lo_equilibrium(c, H0, cx, cy, c2, H, Bq);
    const double pn = d[0] + d[1] * cx + d[2] * cy + d[3] * c2, pt = c.b[0] + c.b[1] * cx + c.b[2] * cy + c.b[3] * c2;
    const double pT = c.T[0] + c.T[1] * cx + c.T[2] * cy + c.T[3] * c2;
    const double Z = c.mt[1] * (vn * pn + vt * pt) + c.mt[2] * pT;
    const double z3 = c.mt[1] * (vn * d[3] + vt * c.b[3]) + c.mt[2] * c.T[3];
    gh = H * (c.mt[0] * sh + Z) + Bq * z3;
    gb = Bq * (c.mt[0] * (sh + qd * c2ck) + Z) + c.mxi2 * H * z3;
}

// the projected unit-density wall Maxwellian of the value Hw (s_w: lam, floors)
__device__ __forceinline__ void lo_shape(double Hw, double bfac, const double* s_w, double cx, double cy, double& h, double& b) {
    const double bw = Hw * bfac;
    h = Hw + fmax(Hw, s_w[4]) * (s_w[0] + s_w[1] * cx + s_w[2] * cy + s_w[3] * (0.5 * (cx * cx + cy * cy)));
    b = bw + 0.5 * fmax(bw, s_w[5]) * s_w[3];
}

template <int VPT>
__device__ __forceinline__ void lo_wall_t(const LoParams& P, const LoBuffers& B, int wf, double dt, double* red,
                                          double* rout, double* ex, double* ey, LoFluxC& sc, double* s_w) {
    const int nx = P.nx, nv = P.nvel, nu = P.tnu, tid = threadIdx.x, lane = tid & 31;
    const int iw = wf >= nx ? 1 : 0, i = wf - iw * nx, j = iw ? P.ny - 1 : 0, cell = j * nx + i;
    const double side = iw ? 1.0 : -1.0, ux = P.wall_ux[iw], L = P.wall_lam[iw], hl = side * 0.5 * P.dy;
    const double* Wc = B.W + cell * 4;
    const float inu = 1.0f / (float)nu;
    double hv[VPT], bv[VPT], ph[VPT], pb[VPT], acc[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) acc[m] = 0.0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const double u = B.u[s.kk], v = B.v[s.kk], w = s.ok ? B.w[s.kk] : 0.0;
        const LoVal q = lo_val(P, B, cell, i, j, s.kk);
        hv[r] = q.h + hl * q.hy;
        bv[r] = q.b + hl * q.by;
        ph[r] = u * q.hx + v * q.hy;
        pb[r] = u * q.bx + v * q.by;
        const double th = w * -q.hx, cx = u - ux, e = 0.5 * w * ((cx * cx + v * v) * hv[r] + bv[r]);
        acc[0] += th;            // tangential slope moments in the wall's frame vn = v, vt = -u
        acc[1] += v * th;
        acc[2] -= u * th;
        acc[3] += 0.5 * ((u * u + v * v) * th - w * q.bx);
        acc[4] += cx * e;        // heat of the face values about the wall's velocity
        acc[5] += v * e;
    }
    block_reduce_smem<6, 0>(acc, red, rout);
    const LoCrew C;
    Prim pc;
    const bool ok = get_primary(P.gm1, Wc, pc);
    if (!ok) { pc.r = 1.0; pc.L = 1.0; }
    const Prim pg{pc.r / pc.L * L, 0.0, -ux, L};   // the cell's pressure at the wall's temperature (:2027)
    const double bfac = (double)P.ck / (2.0 * L), irho = 1.0 / pg.r;
    if (C.worker) {   // the wall equilibrium and its unit-density shape: moments and Gram matrices about (ux, 0)
        lo_rows_of(C, P, B.tab, ux, 0.0, L, pg.r * (L / kPi), ex, ey);
        C.sync();
        const double peak = lo_peak(P, ex, ey);
        const double fgh = kEps * fmax(peak, 1.0), fgb = kEps * fmax(peak * bfac, 1.0);
        const double fwh = kEps * fmax(peak * irho, 1.0), fwb = kEps * fmax(peak * irho * bfac, 1.0);
        double a[28];
#pragma unroll
        for (int m = 0; m < 28; ++m) a[m] = 0.0;
        for (int k = C.id; k < nv; k += C.n) {
            const int jv = lo_row(k, inu);
            const double w = B.w[k], cx = B.u[k] - ux, v = B.v[k], H = ex[k - jv * nu] * ey[jv], Hw = H * irho;
            moment_add(w, cx, v, H, H * bfac, a);
            gram_add(w, fmax(H, fgh), fmax(H * bfac, fgb), cx, v, a + 4);
            moment_add(w, cx, v, Hw, Hw * bfac, a + 14);
            gram_add(w, fmax(Hw, fwh), fmax(Hw * bfac, fwb), cx, v, a + 18);
        }
        C.partial<28>(a, red);
        if (C.id == 0) { sc.fh = fgh; sc.fb = fgb; s_w[4] = fwh; s_w[5] = fwb; }
    }
    if (C.scalar) {
        double tau = 1.0, Mt[5], cg[4], sw[4], a[4], an[4], at[4], aT[4], m1[4], m2[4];
        const bool tok = get_tau(P.mu_ref, P.omega, pg, tau);
        if (!tok) tau = 1.0;
        time_coeffs(dt, tau, Mt);
        get_conserved(P.gm1, pg, cg);
        const double wl[4] = {Wc[0], Wc[2], -Wc[1], Wc[3]};
#pragma unroll
        for (int m = 0; m < 4; ++m) sw[m] = lane == 0 ? (cg[m] - wl[m]) / (side * 0.5 * P.dy) : rout[m];
        micro_slope(P.ck, pg, sw, a);   // lane 0: normal, the others: tangential
        // CalcMoment's full moments: 1 and the mean, then its recurrence
        const double iL = 1.0 / L;
        double Mu[6], Mv[6], Mx[3] = {1.0, 0.5 * (double)P.ck * iL, (double)P.ck * ((double)P.ck + 2.0) * 0.25 * (iL * iL)};
        Mu[0] = Mv[0] = 1.0;
        Mu[1] = pg.U;
        Mv[1] = pg.V;
#pragma unroll
        for (int m = 2; m < 6; ++m) {
            const double k = 0.5 * (double)(m - 1) * iL;
            Mu[m] = pg.U * Mu[m - 1] + k * Mu[m - 2];
            Mv[m] = pg.V * Mv[m - 1] + k * Mv[m - 2];
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) { an[m] = __shfl_sync(0xffffffffu, a[m], 0); at[m] = __shfl_sync(0xffffffffu, a[m], 1); }
        moment_auvxi(an, Mu, Mv, Mx, 1, 0, m1);
        moment_auvxi(at, Mu, Mv, Mx, 0, 1, m2);
#pragma unroll
        for (int m = 0; m < 4; ++m) sw[m] = -pg.r * (m1[m] + m2[m]);
        micro_slope(P.ck, pg, sw, aT);
        if (lane == 0) {
            sc.U = ux; sc.V = 0.0; sc.l2 = 2.0 * L; sc.kq = 0.8 * (1.0 - P.pr) * L * L / pg.r;
            sc.qx = rout[4]; sc.qy = rout[5]; sc.mxi2 = Mx[2]; sc.bf = bfac;
#pragma unroll
            for (int m = 0; m < 5; ++m) sc.mt[m] = Mt[m];
            lo_centred(1, an, ux, 0.0, sc.a[0]);
            lo_centred(1, at, ux, 0.0, sc.b);
            lo_centred(1, aT, ux, 0.0, sc.T);
            if (!ok) set_status(B.status, ST_GETPRIMARY);
            if (ok && !tok) set_status(B.status, ST_TAU);
        }
    }
    __syncthreads();
    if (tid < 32) {   // lane 0: the equilibrium's projection, lane 1: the shape's, lanes 2 and 3: their pivots
        double f[14], tg[4], lam[4];
        const int o = lane & 1 ? 14 : 0;
#pragma unroll
        for (int m = 0; m < 14; ++m) f[m] = C.total(red, o + m);
        const Prim pq{lane & 1 ? 1.0 : pg.r, ux, 0.0, L};
        get_conserved(P.gm1, pq, tg);
        const bool pok = lo_lambda(f, ux, 0.0, tg, lane & 2, lam);
        if (lane < 2) {
            double* q = lane == 0 ? sc.lam : s_w;
#pragma unroll
            for (int m = 0; m < 4; ++m) q[m] = lam[m];
            sc.tg[lane].set(tg);
        }
        if (!pok && lane < 4) set_status(B.status, ST_FACE_PROJECTION);
    }
    __syncthreads();
    // toward the wall: the incident flux; away from it: the unit wall Maxwellian, its density from zero net mass (:2166)
    const double c2ck = 2.0 / (double)P.ck;
    acc[0] = acc[1] = 0.0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const int jv = lo_row(s.kk, inu);
        const double u = B.u[s.kk], v = B.v[s.kk], wv = (s.ok ? B.w[s.kk] : 0.0) * v, H0 = ex[s.kk - jv * nu] * ey[jv];
        const double cx = u - ux;
        if ((copysign(1.0, v) > 0.0) == (iw == 1)) {
            double H, Bq, gh, gb;
            lo_poly(sc, sc.a[0], H0, cx, v, v, -u, c2ck, H, Bq, gh, gb);
            hv[r] = gh + sc.mt[3] * hv[r] - sc.mt[4] * ph[r];
            bv[r] = gb + sc.mt[3] * bv[r] - sc.mt[4] * pb[r];
            acc[0] += wv * hv[r];
        } else {
            lo_shape(H0 * irho, bfac, s_w, cx, v, hv[r], bv[r]);
            acc[1] += wv * hv[r];
        }
    }
    // the gates of both projections, over all velocities, in a loop of their own: a domain has few wall faces
    double mom[10] = {acc[0], acc[1], 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int k = tid; k < nv; k += (int)blockDim.x) {
        const int jv = lo_row(k, inu);
        const double w = B.w[k], u = B.u[k], v = B.v[k], cx = u - ux, H0 = ex[k - jv * nu] * ey[jv];
        double h, b;
        lo_equilibrium(sc, H0, cx, v, cx * cx + v * v, h, b);
        moment_add(w, u, v, h, b, mom + 2);
        lo_shape(H0 * irho, bfac, s_w, cx, v, h, b);
        moment_add(w, u, v, h, b, mom + 6);
    }
    block_reduce_smem<10, 0>(mom, red, rout);
    if (tid >= 2 && tid < 10 && sc.tg[(tid - 2) >> 2].missed((tid - 2) & 3, rout[tid])) set_status(B.status, ST_FACE_PROJECTION);
    const double rhow = -rout[0] / (dt * rout[1]), flen = P.dx;
    const size_t o = (size_t)((iw ? P.ny : 0) * nx + i);
#pragma unroll
    for (int m = 0; m < 4; ++m) acc[m] = 0.0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const double u = B.u[s.kk], v = B.v[s.kk], w = s.ok ? B.w[s.kk] : 0.0;
        const double f = (copysign(1.0, v) > 0.0) == (iw == 1) ? v : dt * v * rhow;
        const double hk = f * hv[r], bk = f * bv[r];
        if (s.ok) { B.fyh[o * nv + s.k] = flen * hk; B.fyb[o * nv + s.k] = flen * bk; }
        moment_add(w, v, -u, hk, bk, acc);
    }
    block_reduce_smem<4, 0>(acc, red, rout);
    if (tid == 0) {
        double* aero = B.wall_aero + (iw * nx + i) * 3;
        aero[0] = rout[1] / dt;
        aero[1] = rout[2] / dt;
        aero[2] = rout[3] / dt + ux * rout[2] / dt;
        // GlobalFrame with cosx = -0, cosy = 1: (f1, f2, f3, f4) -> (f1, -f3, f2, f4), times the face length
        double* Fw = B.fyw + o * 4;
        Fw[0] = flen * rout[0];
        Fw[1] = flen * (-rout[2]);
        Fw[2] = flen * rout[1];
        Fw[3] = flen * rout[3];
        if (!(isfinite(rout[0]) && isfinite(rout[1]) && isfinite(rout[2]) && isfinite(rout[3])))
            set_status(B.status, ST_NONFINITE_FLUX);
    }
}

template <int VPT>
__device__ __forceinline__ void lo_face_t(const LoParams& P, const LoBuffers& B, int fi, double dt, double* red,
                                          double* rout, double* ex, double* ey, LoFluxC& sc) {
    const int nx = P.nx, nv = P.nvel, nu = P.tnu, tid = threadIdx.x, lane = tid & 31;
    const int dir = fi < nx * P.ny ? 0 : 1, g = dir == 0 ? fi : fi - nx * P.ny;
    const int i = g % nx, j = (dir == 0 ? 0 : 1) + g / nx;              // the upper cell
    const int il = dir == 0 ? wrapx(i - 1, nx) : i, jl = dir == 0 ? j : j - 1;
    const int cR = j * nx + i, cL = jl * nx + il;
    const double hl = 0.5 * (dir == 0 ? P.dx : P.dy), flen = dir == 0 ? P.dy : P.dx;
    const double ur = B.W[cL * 4 + 1] / B.W[cL * 4], vr = B.W[cL * 4 + 2] / B.W[cL * 4];
    const float inu = 1.0f / (float)nu;
    double hv[VPT], bv[VPT], ph[VPT], pb[VPT], acc[13];
#pragma unroll
    for (int m = 0; m < 13; ++m) acc[m] = 0.0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const double u = B.u[s.kk], v = B.v[s.kk], w = s.ok ? B.w[s.kk] : 0.0;
        const bool left = copysign(1.0, dir == 0 ? u : v) > 0.0;
        const double sg = left ? hl : -hl;
        const LoVal q = lo_val(P, B, left ? cL : cR, left ? il : i, left ? jl : j, s.kk);
        hv[r] = q.h + sg * (dir == 0 ? q.hx : q.hy);
        bv[r] = q.b + sg * (dir == 0 ? q.bx : q.by);
        ph[r] = u * q.hx + v * q.hy;
        pb[r] = u * q.bx + v * q.by;
        // the face values about the lower cell's velocity, and the tangential slope (t = -x on horizontal faces)
        const double cx = u - ur, cy = v - vr, xx = cx * cx, yy = cy * cy, wh = w * hv[r], wb = w * bv[r], e = (xx + yy) * wh + wb;
        const double th = w * (dir == 0 ? q.hy : -q.hx), tb = w * (dir == 0 ? q.by : -q.bx);
        acc[0] += wh;
        acc[1] += cx * wh;
        acc[2] += cy * wh;
        acc[3] += xx * wh;
        acc[4] += cx * cy * wh;
        acc[5] += yy * wh;
        acc[6] += wb;
        acc[7] += cx * e;
        acc[8] += cy * e;
        acc[9] += th;
        acc[10] += u * th;
        acc[11] += v * th;
        acc[12] += 0.5 * ((u * u + v * v) * th + tb);
    }
    block_reduce_smem<13, 0>(acc, red, rout);
    const LoCrew C;
    const double* f = rout;
    const double wg[4] = {f[0], ur * f[0] + f[1], vr * f[0] + f[2],
                          0.5 * (ur * ur + vr * vr) * f[0] + ur * f[1] + vr * f[2] + 0.5 * (f[3] + f[5] + f[6])};
    const double cv[4] = {wg[0], dir == 0 ? wg[1] : wg[2], dir == 0 ? wg[2] : -wg[1], wg[3]};
    Prim pf;
    const bool ok = get_primary(P.gm1, cv, pf);
    if (!ok) { pf.r = 1.0; pf.U = 0.0; pf.V = 0.0; pf.L = 1.0; }
    const double U = dir == 0 ? pf.U : -pf.V, V = dir == 0 ? pf.V : pf.U;   // in the grid's frame
    const double bfac = (double)P.ck / (2.0 * pf.L);
    if (C.worker) {   // the face equilibrium's moments and Gram matrix about (U, V)
        lo_rows_of(C, P, B.tab, U, V, pf.L, pf.r * (pf.L / kPi), ex, ey);
        C.sync();
        const double peak = lo_peak(P, ex, ey), fh = kEps * fmax(peak, 1.0), fb = kEps * fmax(peak * bfac, 1.0);
        double a[14];
#pragma unroll
        for (int m = 0; m < 14; ++m) a[m] = 0.0;
#pragma unroll 2
        for (int k = C.id; k < nv; k += C.n) {
            const int jv = lo_row(k, inu);
            const double w = B.w[k], cx = B.u[k] - U, cy = B.v[k] - V, H = ex[k - jv * nu] * ey[jv];
            moment_add(w, cx, cy, H, H * bfac, a);
            gram_add(w, fmax(H, fh), fmax(H * bfac, fb), cx, cy, a + 4);
        }
        C.partial<14>(a, red);
        if (C.id < 32) {   // GetTau and Mt by the first worker warp, beside the scalar chain
            double tau = 1.0, Mt[5];
            const bool tok = get_tau(P.mu_ref, P.omega, pf, tau);
            if (!tok) tau = 1.0;
            time_coeffs(dt, tau, Mt);
            if (C.id == 0) {
                sc.fh = fh;
                sc.fb = fb;
#pragma unroll
                for (int m = 0; m < 5; ++m) sc.mt[m] = Mt[m];
                if (ok && !tok) set_status(B.status, ST_TAU);
            }
        }
    }
    if (C.scalar) {   // the face's scalar chain (GetPrimary, MicroSlope x4, CalcMoment, GetTau, Mt)
        // lane 0: aL from (W_face - W_L) / (dx/2), lane 1: aR from (W_R - W_face) / (dx/2), the others: tangential
        double sw[4], a[4], aL[4], aR[4], bs[4], aT[4], o4[4];
        {
            const double* Wc = B.W + (lane == 0 ? cL : cR) * 4;
            const double wc[4] = {Wc[0], dir == 0 ? Wc[1] : Wc[2], dir == 0 ? Wc[2] : -Wc[1], Wc[3]};
            const double ts[4] = {f[9], dir == 0 ? f[10] : f[11], dir == 0 ? f[11] : -f[10], f[12]};
#pragma unroll
            for (int m = 0; m < 4; ++m) sw[m] = lane == 0 ? (cv[m] - wc[m]) / hl : (lane == 1 ? (wc[m] - cv[m]) / hl : ts[m]);
        }
        micro_slope(P.ck, pf, sw, a);
        // CalcMoment and Moment_auvxi (mod_Evolution.f90:1810-1885) of aL (u^1, u > 0 half), aR (u^1, u < 0 half) and b (v^1,
        // all u), each on its lane: its half's recurrence from its zeroth and first moment (1 and U for all u)
        const double iL = 1.0 / pf.L;
        double Mx[3] = {1.0, 0.5 * (double)P.ck * iL, (double)P.ck * ((double)P.ck + 2.0) * 0.25 * (iL * iL)};
        {
            const double x = sqrt(pf.L) * pf.U, e = 0.5 * exp(-pf.L * pf.U * pf.U) / sqrt(kPi * pf.L);
            const double h = 0.5 * erfc(lane == 0 ? -x : x);
            double mu[6], mv[6], Mu[5], Mv[5];
            mu[0] = lane < 2 ? h : 1.0;
            mu[1] = pf.U * mu[0] + (lane == 0 ? e : (lane == 1 ? -e : 0.0));
            mv[0] = 1.0;
            mv[1] = pf.V;
#pragma unroll
            for (int m = 2; m < 6; ++m) {
                const double k = 0.5 * (double)(m - 1) * iL;
                mu[m] = pf.U * mu[m - 1] + k * mu[m - 2];
                mv[m] = pf.V * mv[m - 1] + k * mv[m - 2];
            }
#pragma unroll
            for (int m = 0; m < 5; ++m) { Mu[m] = lane < 2 ? mu[m + 1] : mu[m]; Mv[m] = lane < 2 ? mv[m] : mv[m + 1]; }
            moment_auvxi(a, Mu, Mv, Mx, 0, 0, o4);
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            sw[m] = -pf.r * (__shfl_sync(0xffffffffu, o4[m], 0) + __shfl_sync(0xffffffffu, o4[m], 1) +
                             __shfl_sync(0xffffffffu, o4[m], 2));
            aL[m] = __shfl_sync(0xffffffffu, a[m], 0);
            aR[m] = __shfl_sync(0xffffffffu, a[m], 1);
            bs[m] = __shfl_sync(0xffffffffu, a[m], 2);
        }
        micro_slope(P.ck, pf, sw, aT);
        if (lane == 0) {
            // heat flux of the face values, shifted from (ur, vr) to the face's velocity
            const double dx = U - ur, dy = V - vr, d2 = dx * dx + dy * dy, e2 = f[3] + f[5] + f[6], dp = dx * f[1] + dy * f[2];
            sc.qx = 0.5 * (f[7] - dx * e2 + d2 * f[1] - d2 * dx * f[0]) - (dx * f[3] + dy * f[4]) + dx * dp;
            sc.qy = 0.5 * (f[8] - dy * e2 + d2 * f[2] - d2 * dy * f[0]) - (dx * f[4] + dy * f[5]) + dy * dp;
            sc.U = U; sc.V = V; sc.l2 = 2.0 * pf.L; sc.kq = 0.8 * (1.0 - P.pr) * pf.L * pf.L / pf.r;
            sc.mxi2 = Mx[2]; sc.bf = bfac;
            lo_centred(dir, aL, U, V, sc.a[0]);
            lo_centred(dir, aR, U, V, sc.a[1]);
            lo_centred(dir, bs, U, V, sc.b);
            lo_centred(dir, aT, U, V, sc.T);
            if (!ok) set_status(B.status, ST_GETPRIMARY);
        }
    }
    __syncthreads();
    if (tid < 32) {   // lane 0: the projection, lane 1: its pivots
        double t[14], tg[4], lam[4];
#pragma unroll
        for (int m = 0; m < 14; ++m) t[m] = C.total(red, m);
        const Prim pq{pf.r, U, V, pf.L};
        get_conserved(P.gm1, pq, tg);
        const bool pok = lo_lambda(t, U, V, tg, lane & 1, lam);
        if (lane == 0)
#pragma unroll
            for (int m = 0; m < 4; ++m) sc.lam[m] = lam[m];
        if (lane == 0) sc.tg[0].set(tg);
        if (!pok && lane < 2) set_status(B.status, ST_FACE_PROJECTION);
    }
    __syncthreads();
    // the micro flux (mod_Evolution.f90:396-453) times the face length
    const double c2ck = 2.0 / (double)P.ck;
    const size_t o = (size_t)(j * nx + i);
    double* Fh = (dir == 0 ? B.fxh : B.fyh) + o * nv;
    double* Fb = (dir == 0 ? B.fxb : B.fyb) + o * nv;
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m] = 0.0;   // the flux's moments, the projected equilibrium's
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const int jv = lo_row(s.kk, inu);
        const double u = B.u[s.kk], v = B.v[s.kk], w = s.ok ? B.w[s.kk] : 0.0, H0 = ex[s.kk - jv * nu] * ey[jv];
        lo_reread();
        const double vn = dir == 0 ? u : v, vt = dir == 0 ? v : -u, cx = u - sc.U, cy = v - sc.V;
        double H, Bq, gh, gb;
        lo_poly(sc, sc.a[copysign(1.0, vn) > 0.0 ? 0 : 1], H0, cx, cy, vn, vt, c2ck, H, Bq, gh, gb);
        moment_add(w, u, v, H, Bq, acc + 4);
        const double fh = flen * (vn * (gh + sc.mt[3] * hv[r] - sc.mt[4] * ph[r]));
        const double fb = flen * (vn * (gb + sc.mt[3] * bv[r] - sc.mt[4] * pb[r]));
        if (s.ok) { Fh[s.k] = fh; Fb[s.k] = fb; }
        moment_add(w, u, v, fh, fb, acc);   // MomentConserved in the global frame (:470-473)
    }
    block_reduce_smem<8, 0>(acc, red, rout);
    if (tid < 4) {
        ((dir == 0 ? B.fxw : B.fyw) + o * 4)[tid] = rout[tid];
        if (!isfinite(rout[tid])) set_status(B.status, ST_NONFINITE_FLUX);
    }
    if (tid >= 4 && tid < 8 && sc.tg[0].missed(tid - 4, rout[tid])) set_status(B.status, ST_FACE_PROJECTION);
}

template <int VPT, int NTMAX>
__global__ void __launch_bounds__(NTMAX, 512 / NTMAX) k_lo_fluxes_t(LoParams P, LoBuffers B) {
    if (eval_cached(B)) return;
    __shared__ double red[16 * 32], rout[kRedSlots], ex[64], ey[64], s_w[6];
    __shared__ LoFluxC sc;
    const double dt = B.dt[0];
    const int id = blockIdx.x;
    if (id < 2 * P.nx) lo_wall_t<VPT>(P, B, id, dt, red, rout, ex, ey, sc, s_w);
    else lo_face_t<VPT>(P, B, id - 2 * P.nx, dt, red, rout, ex, ey, sc);
}

// One cell: the reduction of the distribution's sums (stream moments, the stream projection's Gram matrix, the old heat
// flux); by warp 0 the macro update and the stream projection, by the others the sums of the old and new equilibria
// (mod_TimeIntegrator.f90:235-293); their projections; the update.  MODE as k_lo_cells.
enum { MODE_RESIDUAL = 1, MODE_UPDATE = 2 };
struct LoCellC {
    double U, V, l2, kx, ky, bf, fh, fb, lam[4];   // mean, 2 L, coeff q, ck/(2L), floors, lam
    LoTarget tg;
    // equilibrium + Shakhov of the Maxwellian value H
    __device__ __forceinline__ void at(double H, double cx, double cy, double c2, double c2ck, double& E, double& F) const {
        const double qd = kx * cx + ky * cy, sh = 1.0 + qd * (l2 * c2 - 4.0);
        E = H * sh;
        F = bf * H * (sh + qd * c2ck);
    }
};
// The stream projection's Gram sums again, into rout[4..13], for a cell (hc, bc) whose maximum of |h| or |b| passes 1, and its
// floors.  Out of line and on the stored distribution, so that the kernel holds nothing for it: a state near the
// reference's units (density 1, T = 2: h up to 0.16) never comes here.
__device__ __noinline__ void lo_dense_stream(const double* __restrict__ hc, const double* __restrict__ bc,
                                             const double* __restrict__ u, const double* __restrict__ v,
                                             const double* __restrict__ w, int nv, double* red, double* rout, double* floors) {
    __shared__ double s_max[2], s_gram[10];
    double acc[10], mx[2] = {0.0, 0.0};
    for (int k = threadIdx.x; k < nv; k += blockDim.x) { mx[0] = fmax(mx[0], fabs(hc[k])); mx[1] = fmax(mx[1], fabs(bc[k])); }
    block_reduce_smem<0, 2>(mx, red, s_max);
    const double fh = kEps * fmax(s_max[0], 1.0), fb = kEps * fmax(s_max[1], 1.0);
#pragma unroll
    for (int m = 0; m < 10; ++m) acc[m] = 0.0;
    for (int k = threadIdx.x; k < nv; k += blockDim.x) gram_add(w[k], fmax(fabs(hc[k]), fh), fmax(fabs(bc[k]), fb), u[k], v[k], acc);
    block_reduce_smem<10, 0>(acc, red, s_gram);
    if (threadIdx.x < 10) rout[4 + threadIdx.x] = s_gram[threadIdx.x];
    if (threadIdx.x == 0) { floors[0] = fh; floors[1] = fb; }
    __syncthreads();
}

template <int VPT, int NTMAX, int MODE>
__global__ void __launch_bounds__(NTMAX, 512 / NTMAX) k_lo_cells_t(LoParams P, LoBuffers B) {
    __shared__ double red[16 * 32], rout[kRedSlots], ex[2][64], ey[2][64], s_lam[4], s_tau[2], s_mx[16][4], s_floor[2];
    __shared__ LoCellC sc[2];
    __shared__ LoTarget s_rate;
    const int nv = P.nvel, nu = P.tnu, tid = threadIdx.x, nx = P.nx, lane = tid & 31;
    const int c = blockIdx.x, i = c % nx, j = c / nx;
    const double dt = B.dt[0], dti = 1.0 / dt, c2ck = 2.0 / (double)P.ck;
    const double* Wo = B.W + c * 4;
    const size_t fl = (size_t)(j * nx + i), fr = (size_t)(j * nx + wrapx(i + 1, nx)), gr = (size_t)((j + 1) * nx + i);
    const double uo = Wo[1] / Wo[0], vo = Wo[2] / Wo[0], scale = 1.0 / (P.area * dt);
    const float inu = 1.0f / (float)nu;
    double *hc = B.h + (size_t)c * nv, *bc = B.b + (size_t)c * nv;
    double rh[VPT], rb[VPT], acc[17];
#pragma unroll
    for (int m = 0; m < 17; ++m) acc[m] = 0.0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const int k = s.kk;
        if (MODE & MODE_RESIDUAL) {   // AssembleMicroFluxResidual (mod_Residual.f90:60-95)
            rh[r] = (B.fxh[fl * nv + k] - B.fxh[fr * nv + k] + B.fyh[fl * nv + k] - B.fyh[gr * nv + k]) * scale;
            rb[r] = (B.fxb[fl * nv + k] - B.fxb[fr * nv + k] + B.fyb[fl * nv + k] - B.fyb[gr * nv + k]) * scale;
        } else {
            rh[r] = B.res_h[(size_t)c * nv + k];
            rb[r] = B.res_b[(size_t)c * nv + k];
        }
    }
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const double u = B.u[s.kk], v = B.v[s.kk], w = s.ok ? B.w[s.kk] : 0.0, hr = hc[s.kk], br = bc[s.kk];
        if (MODE & MODE_RESIDUAL) {
            moment_add(w, u, v, rh[r], rb[r], acc);
            gram_add(w, fmax(fabs(hr), kEps), fmax(fabs(br), kEps), u, v, acc + 4);
            acc[16] = fmax(acc[16], fmax(fabs(hr), fabs(br)));   // a slot past the table repeats its last velocity
        }
        if (MODE & MODE_UPDATE) {   // GetHeatFlux_Vec of the old state
            const double cx = u - uo, cy = v - vo, t = 0.5 * w * ((cx * cx + cy * cy) * hr + br);
            acc[14] += t * cx;
            acc[15] += t * cy;
        }
    }
    block_reduce_smem<16, 1>(acc, red, rout);
    // the stream projection's weights are max(|h|, eps max(1, max |h|)): those above stand unless a maximum passes 1
    if ((MODE & MODE_RESIDUAL) && rout[16] > 1.0)
        lo_dense_stream(hc, bc, B.u, B.v, B.w, nv, red, rout, s_floor);
    else if (tid == 0) s_floor[0] = s_floor[1] = kEps;
    double resw[4], Wn[4];   // AssembleMacroResidual (mod_Residual.f90:30-54)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        resw[m] = MODE & MODE_RESIDUAL ? (B.fxw[fl * 4 + m] - B.fxw[fr * 4 + m] + B.fyw[fl * 4 + m] - B.fyw[gr * 4 + m]) / P.area
                                       : B.res_w[c * 4 + m];
        Wn[m] = Wo[m] + resw[m];
    }
    const LoCrew C;
    Prim po{1.0, 0.0, 0.0, 1.0}, pn{1.0, 0.0, 0.0, 1.0};
    bool pok = true;
    if (MODE & MODE_UPDATE) {
        const double w4[4] = {Wo[0], Wo[1], Wo[2], Wo[3]};
        pok = get_primary(P.gm1, w4, po);
        if (!pok) { po.r = 1.0; po.U = po.V = 0.0; po.L = 1.0; }
        const bool nok = get_primary(P.gm1, Wn, pn);
        if (!nok) { pn.r = 1.0; pn.U = pn.V = 0.0; pn.L = 1.0; }
        pok = pok && nok;
    }
    if ((MODE & MODE_UPDATE) && C.worker) {
        const double q0 = rout[14], q1 = rout[15];
        if (C.id < 2) {
            const Prim& p = C.id ? pn : po;
            const double cf = 0.8 * (1.0 - P.pr) * p.L * p.L / p.r;
            LoCellC& s = sc[C.id];
            s.U = p.U; s.V = p.V; s.l2 = 2.0 * p.L; s.kx = cf * q0; s.ky = cf * q1; s.bf = (double)P.ck / (2.0 * p.L);
        }
        lo_rows_of(C, P, B.tab, po.U, po.V, po.L, po.r * (po.L / kPi), ex[0], ey[0]);
        lo_rows_of(C, P, B.tab, pn.U, pn.V, pn.L, pn.r * (pn.L / kPi), ex[1], ey[1]);
        C.sync();
        // the floors' max(1, max |E|): |E| <= pref (1 + coeff |q| sup c (2 L c^2 + 4) exp(-L c^2)), the supremum at most
        // 2.3 / sqrt(L) (2.3 + 0.43 (2 / ck) for F); only where that bound passes 1 is the maximum taken
        double fl[4] = {kEps, kEps, kEps, kEps};
        bool need = false;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const Prim& p = t ? pn : po;
            const double pre = p.r * (p.L / kPi), m = (fabs(sc[t].kx) + fabs(sc[t].ky)) / sqrt(p.L);
            need = need || !(pre * (1.0 + 2.3 * m) <= 1.0) || !(sc[t].bf * pre * (1.0 + (2.3 + 0.43 * c2ck) * m) <= 1.0);
        }
        auto equil = [&](int t, int k, double& E, double& F, double& cx, double& cy) {
            const int jv = lo_row(k, inu);
            const LoCellC& s = sc[t];
            cx = B.u[k] - s.U;
            cy = B.v[k] - s.V;
            s.at(ex[t][k - jv * nu] * ey[t][jv], cx, cy, cx * cx + cy * cy, c2ck, E, F);
        };
        if (need) {
            double mx[4] = {0.0, 0.0, 0.0, 0.0};
            for (int k = C.id; k < nv; k += C.n)
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    double E, F, cx, cy;
                    equil(t, k, E, F, cx, cy);
                    mx[2 * t] = fmax(mx[2 * t], fabs(E));
                    mx[2 * t + 1] = fmax(mx[2 * t + 1], fabs(F));
                }
            warp_max_all<4>(mx);
            if (lane == 0)
#pragma unroll
                for (int m = 0; m < 4; ++m) s_mx[C.id >> 5][m] = mx[m];
            C.sync();
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                double x = 1.0;
                for (int w = 0; w < C.n / 32; ++w) x = fmax(x, s_mx[w][m]);
                fl[m] = kEps * x;
            }
        }
        if (C.id == 0) { sc[0].fh = fl[0]; sc[0].fb = fl[1]; sc[1].fh = fl[2]; sc[1].fb = fl[3]; }
        double a[28];
#pragma unroll
        for (int m = 0; m < 28; ++m) a[m] = 0.0;
        for (int k = C.id; k < nv; k += C.n) {
            const double w = B.w[k];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                double E, F, cx, cy;
                equil(t, k, E, F, cx, cy);
                moment_add(w, cx, cy, E, F, a + 14 * t);
                gram_add(w, fmax(fabs(E), fl[2 * t]), fmax(fabs(F), fl[2 * t + 1]), cx, cy, a + 14 * t + 4);
            }
        }
        C.partial<28>(a, red);
    }
    if (C.scalar) {
        if (MODE & MODE_UPDATE) {   // lane 0: tau of the old state, lane 1: of the new
            double tau = 1.0;
            const bool ok = get_tau(P.mu_ref, P.omega, lane == 1 ? pn : po, tau);
            if (lane < 2) {
                s_tau[lane] = ok ? tau : 1.0;
                if (!ok || !pok) set_status(B.status, ST_GETPRIMARY);
            }
        }
        if (MODE & MODE_RESIDUAL) {   // EnforceStreamingMomentCompatibility (mod_ImplicitMicro.f90:293-306)
            double G[16], rhs[4], lam[4];
            gram_expand(rout + 4, G);
#pragma unroll
            for (int m = 0; m < 4; ++m) rhs[m] = resw[m] * dti - rout[m];
            const bool ok = t_solve(G, rhs, lam, lo_least(G));
            if (lane == 0) {
                const double rate[4] = {resw[0] * dti, resw[1] * dti, resw[2] * dti, resw[3] * dti};
                s_rate.set(rate);
#pragma unroll
                for (int m = 0; m < 4; ++m) s_lam[m] = lam[m];
                if (!ok) set_status(B.status, ST_PROJECTION);
            }
        }
    }
    __syncthreads();
    if (MODE & MODE_UPDATE) {
        if (tid < 32) {   // lane 0: the old equilibrium onto W_old's moments, lane 1: the new one onto W_new, lanes 2, 3: pivots
            const bool nw = lane & 1;
            double f[14], tg[4], lam[4];
            const int o = nw ? 14 : 0;
#pragma unroll
            for (int m = 0; m < 14; ++m) f[m] = C.total(red, o + m);
            get_conserved(P.gm1, po, tg);
            if (nw)
#pragma unroll
                for (int m = 0; m < 4; ++m) tg[m] = Wn[m];
            const bool ok = lo_lambda(f, nw ? pn.U : po.U, nw ? pn.V : po.V, tg, lane & 2, lam);
            if (lane < 2)
#pragma unroll
                for (int m = 0; m < 4; ++m) sc[lane].lam[m] = lam[m];
            if (lane < 2) sc[lane].tg.set(tg);
            if (!ok && lane < 4) set_status(B.status, ST_PROJECTION);
        }
        __syncthreads();
    }
    // the moments of the projected stream and equilibria, for the gates: a warp's totals, then a lane of the second warp each,
    // beside the first thread's norms
    auto put = [&](int g, const double* m) {
        const double t = warp_halving<4, false>(m);
        if ((lane & 7) == 0) red[(tid >> 5) * 12 + 4 * g + (lane >> 3)] = t;
    };
    if (MODE & MODE_RESIDUAL) {   // res_h_flux_store = stream_h * dt (mod_Residual.f90:114-115)
        double mom[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int r = 0; r < VPT; ++r) {
            const Slot s = slot(r, nv);
            lo_reread();
            const double u = B.u[s.kk], v = B.v[s.kk], c2 = u * u + v * v;
            // (no read past the table's end of an element that its own thread may have updated)
            const double hr = s.ok ? hc[s.kk] : 0.0, br = s.ok ? bc[s.kk] : 0.0;
            const double sh = rh[r] + fmax(fabs(hr), s_floor[0]) * (s_lam[0] + u * s_lam[1] + v * s_lam[2] + 0.5 * c2 * s_lam[3]);
            const double sb = rb[r] + 0.5 * fmax(fabs(br), s_floor[1]) * s_lam[3];
            moment_add(s.ok ? B.w[s.kk] : 0.0, u, v, sh, sb, mom);
            rh[r] = dt * sh;
            rb[r] = dt * sb;
            if (MODE == MODE_RESIDUAL && s.ok) {
                B.res_h[(size_t)c * nv + s.k] = rh[r];
                B.res_b[(size_t)c * nv + s.k] = rb[r];
            }
        }
        put(2, mom);
    }
    if (MODE & MODE_UPDATE) {   // ApplyExplicitUpdate (mod_TimeIntegrator.f90:16-134, 235-293)
        const double ito = 0.5 * dt / s_tau[0], itn = 0.5 * dt / s_tau[1], inv = 1.0 / (1.0 + itn);
        double mq[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
#pragma unroll
        for (int r = 0; r < VPT; ++r) {
            const Slot s = slot(r, nv);
            const int jv = lo_row(s.kk, inu), iv = s.kk - jv * nu;
            const double u = B.u[s.kk], v = B.v[s.kk], w = s.ok ? B.w[s.kk] : 0.0;
            const double hr = s.ok ? hc[s.kk] : 0.0, br = s.ok ? bc[s.kk] : 0.0;
            lo_reread();
            double E[2], F[2];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const LoCellC& q = sc[t];
                const double cx = u - q.U, cy = v - q.V, c2 = cx * cx + cy * cy;
                q.at(ex[t][iv] * ey[t][jv], cx, cy, c2, c2ck, E[t], F[t]);
                E[t] = E[t] + fmax(fabs(E[t]), q.fh) * (q.lam[0] + q.lam[1] * cx + q.lam[2] * cy + q.lam[3] * (0.5 * c2));
                F[t] = F[t] + 0.5 * fmax(fabs(F[t]), q.fb) * q.lam[3];
                moment_add(w, u, v, E[t], F[t], mq[t]);
            }
            if (s.ok) {
                hc[s.k] = (hr + rh[r] + (itn * E[1] + ito * (E[0] - hr))) * inv;
                bc[s.k] = (br + rb[r] + (itn * F[1] + ito * (F[0] - br))) * inv;
            }
        }
        put(0, mq[0]);
        put(1, mq[1]);
    }
    __syncthreads();
    {
        const int m = tid - 32, first = MODE & MODE_UPDATE ? 0 : 8, last = MODE & MODE_RESIDUAL ? 12 : 8;
        if (m >= first && m < last) {
            double t = red[m];
            for (int q = 1; q < (int)blockDim.x / 32; ++q) t += red[q * 12 + m];
            if ((m < 8 ? sc[m >> 2].tg : s_rate).missed(m & 3, t)) set_status(B.status, ST_PROJECTION);
        }
    }
    if (MODE == MODE_RESIDUAL) {
        if (tid == 0)
#pragma unroll
            for (int m = 0; m < 4; ++m) B.res_w[c * 4 + m] = resw[m];
        return;
    }
    if (tid == 0) {
        bool fin = true, dok;
        double Wp[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) { Wp[m] = Wo[m]; fin = fin && isfinite(Wn[m]); }
        if (!fin) set_status(B.status, ST_NONFINITE_STATE);
        // residual-norm contributions (AccumulateMacroResidualNorm, mod_TimeIntegrator.f90:163-191)
        double* dg = B.cell_diag + (size_t)c * kNDiag;
        for (int m = 0; m < 4; ++m) {
            const double d = (Wp[m] - Wn[m]) * P.area / dt;
            dg[m] = d * d;
            dg[4 + m] = fabs(Wn[m]) * P.area;
            dg[9 + m] = fabs(d);
        }
        dg[8] = P.area * P.area;
        B.dtl[c] = cell_dt(P, Wn, dok);
#pragma unroll
        for (int m = 0; m < 4; ++m) B.W[c * 4 + m] = Wn[m];   // every thread has read W_old before the barrier above
    }
    last_cta_epilogue(P, B, true, true, red, rout);
}

}  // namespace

// 128 threads a CTA, as many velocities each as the table needs; above 1024 velocities 256 threads with 10 each
cudaError_t launch_lo_fluxes_t(const LoParams& P, const LoBuffers& B, cudaStream_t s) {
    const int n = 2 * P.nx + P.nx * P.ny + P.nx * (P.ny - 1);
    if (P.nvel <= 128) k_lo_fluxes_t<1, 128><<<n, 128, 0, s>>>(P, B);
    else if (P.nvel <= 256) k_lo_fluxes_t<2, 128><<<n, 128, 0, s>>>(P, B);
    else if (P.nvel <= 512) k_lo_fluxes_t<4, 128><<<n, 128, 0, s>>>(P, B);
    else if (P.nvel <= 1024) k_lo_fluxes_t<8, 128><<<n, 128, 0, s>>>(P, B);
    else k_lo_fluxes_t<10, 256><<<n, 256, 0, s>>>(P, B);
    return cudaGetLastError();
}

template <int VPT, int NT>
static void cells_t(const LoParams& P, const LoBuffers& B, int mode, cudaStream_t s) {
    const int nc = P.nx * P.ny;
    if (mode == 3) k_lo_cells_t<VPT, NT, 3><<<nc, NT, 0, s>>>(P, B);
    else if (mode == 2) k_lo_cells_t<VPT, NT, 2><<<nc, NT, 0, s>>>(P, B);
    else k_lo_cells_t<VPT, NT, 1><<<nc, NT, 0, s>>>(P, B);
}
cudaError_t launch_lo_cells_t(const LoParams& P, const LoBuffers& B, int mode, cudaStream_t s) {
    if (P.nvel <= 128) cells_t<1, 128>(P, B, mode, s);
    else if (P.nvel <= 256) cells_t<2, 128>(P, B, mode, s);
    else if (P.nvel <= 512) cells_t<4, 128>(P, B, mode, s);
    else if (P.nvel <= 1024) cells_t<8, 128>(P, B, mode, s);
    else cells_t<10, 256>(P, B, mode, s);
    return cudaGetLastError();
}

}  // namespace ugks

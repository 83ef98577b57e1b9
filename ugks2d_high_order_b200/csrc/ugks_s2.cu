// ugks_s2.cu -- the high-order "S2" evolution of HighOrderImplicit and S2CN2 on sm_100a (FP64).
//
//   k_s2_init         : S2 cold start, h, b := discrete closure Maxwellian of W (S2NativeInitializeState,
//                       mod_S2NativeAdapter.f90:192-445 with make_mke).  One warp per cell.
//   k_s2_macro        : macro WENO of W: the normal / tangential slopes of every interior face at its 3
//                       Gauss nodes (compute_flux :803-808,849-854) and the 9 mean-shifted volume node
//                       states of every cell (build_targets, mod_S2D1.f90:1246-1300).
//   k_s2_recon1/2     : tensor WENO-AO(5,3) reconstruction with one-sided wall quartics and the
//                       positivity limiter (mod_S2D1Reconstruction.f90, limit_cell_outputs
//                       mod_S2D1.f90:315-345): the shared first layer, then per cell the second-layer
//                       templates and the limiter; writes the face cache.
// then, on tensor-product velocity tables (LoParams::tnu > 0; ugks_s2_tensor.cuh),
//   k_s2_target_nodes_t : build_targets' closures by 1-D sums: eight lanes per (cell, volume node) -> node scalars.
//   k_s2_target_sum_t   : the Gauss-weighted targets M, K_x, K_y per (cell, velocity) from those scalars
//                         (S2CN2's collision forms them itself).
//   k_s2_face_moments   : the velocity sums of a face's three nodes over the upwind face values, one CTA a face.
//   k_s2_face_nodes_t   : ugks_node (mod_S2D1.f90:421-521) at one Gauss node by eight lanes: closure, directions and time
//                         coefficients -> node scalars.
//   k_s2_face_flux_t    : the three nodes' micro fluxes, Gauss-weighted, into the face arrays, one CTA a face.
//   k_s2_walls_t        : the multiscale diffuse wall (s2w2_wall_node, mod_S2MultiscaleWall.f90:45-184), one CTA a wall
//                         face: its three nodes, their flux and the wall diagnostics.
// and on other tables, and where a wall variant wants the nodes' fluxes or coefficients,
//   k_s2_target_nodes, k_s2_target_sum, k_s2_face_nodes, k_s2_face_flux (one CTA per face node), k_s2_wall_nodes, and
//   k_s2_combine      : the Gauss-weighted node fluxes times the face length into the face arrays.
//
// In the latter the discrete closure (solve_q_first, mod_CorrectedWF2DClosure.f90:331-426) runs on one warp: its
// lanes stride over the velocities, every moment sum is a per-lane sum and a fixed butterfly whose
// totals every lane receives, and every lane runs the reference's accept / backtrack / stop logic on
// those identical totals.  Per-velocity closure quantities (the Maxwellian, the Shakhov directions,
// the slope directions) are recomputed from the closure's few scalars in each pass instead of being
// stored.
#include "ugks_s2_tensor.cuh"

namespace ugks {

// ------------------------------------------------------------------------------------------
// reconstruction + limiter in two passes into the face cache (rec_cell / rec_wall, ugks_s2.cuh; sides: x left, x right,
// y bottom, y top).
//
// k_s2_recon1, the first layer (prepare_first_layer_plane, mod_S2D1Reconstruction.f90:501-578):
// per (cell, velocity, field) the 1-D WENO along x of the cell's own row -- values and derivatives
// at xi = -1/2, +1/2 and values at the 3 Gauss nodes -- and, for rows away from the walls, along y
// of the cell's own column -- values and derivatives at -1/2, +1/2.  These are the first-layer
// results the tensor templates of the 5 neighbouring cells share.  l1[cell][field*11 + q][nvel]:
// q 0..3 = x value/derivative at -1/2, +1/2; 4..6 = x Gauss values; 7..10 = y value/derivative.
// CTA: 4 warps (field, direction) over 32 velocities of one cell.
__global__ void __launch_bounds__(128) k_s2_recon1(LoParams P, LoBuffers B, S2Buffers S) {
    if (eval_cached(B)) return;
    const int nv = P.nvel, nx = P.nx, ny = P.ny, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f = warp >> 1, dir = warp & 1;
    const int k0 = blockIdx.x * 32 + lane;
    const bool kok = k0 < nv;
    const int k = kok ? k0 : nv - 1;
    const int cc = blockIdx.y, i = cc % nx, j = cc / nx;
    if (dir == 1 && s2_near_wall(j, ny)) return;   // walls use one-sided quartics instead
    const S2Field F{(f == 0 ? B.h : B.b) + k, nv, nx, ny};
    double q[5], fw[4], c[5];
#pragma unroll
    for (int s = -2; s <= 2; ++s) q[s + 2] = dir == 0 ? F.at(i + s, j) : F.at(i, j + s);
    const S2Diff d = s2_diff(q);
    s2_weights(q, d, fw);
    s2_power(q[2], d, fw, c);
    double* o = S.l1 + ((size_t)cc * 22 + f * 11 + (dir == 0 ? 0 : 7)) * nv + k;
    const double e = c[0] + (0.25 * c[2] + 0.0625 * c[4]), odd = 0.5 * c[1] + 0.125 * c[3];
    const double de = c[1] + 0.75 * c[3], dodd = c[2] + 0.5 * c[4];
    if (kok) {
        o[0] = e - odd; o[(size_t)nv] = de - dodd; o[2 * (size_t)nv] = e + odd; o[3 * (size_t)nv] = de + dodd;
        if (dir == 0) {
            double v[3];
            s2_gauss_values(c, v);
#pragma unroll
            for (int a = 0; a < 3; ++a) o[(size_t)(4 + a) * nv] = v[a];
        }
        if (!(isfinite(e) && isfinite(odd) && isfinite(de) && isfinite(dodd))) set_status(B.status, ST_NONFINITE_FLUX);
    }
}

// k_s2_recon2, the second layer (tensor_velocity_tile, :723-792; reconstruct_wall_tile, :918-971) and
// limit_cell_outputs (mod_S2D1.f90:315-345).  A cell has four face sides (x left, x right, y bottom, y top) at 3 Gauss
// nodes with value, normal and tangential derivative, and three volume Gauss rows, for h and b; the
// positivity factor theta is the minimum over all their values.  The face cache keeps, per velocity, the sides it
// leaves the cell through, so along each axis only that side needs its derivatives: the other side's
// values enter theta alone.
//
// Cells away from the walls: a thread takes one field of one velocity through both axes and the three rows; CTA = 4
// warps, warp pairs (h, b) over 2 x 32 velocities.  Each side is stored as soon as it is known, as if
// theta were 1, and drawn towards the mean afterwards where the limiter acts, so no result waits in registers.
// Cells in the three rows next to a wall (one-sided quartics across y; the wall sides for every velocity): CTA = 4
// warps (field, axis) over 32 velocities, both sides of the axis held until theta is known.
// Bound by FP64 arithmetic and issue slots (about 930 FP64 operations a thread, two threads a cell-velocity;
// 56 % and 63 % busy).  Residency pays: eight CTAs an SM, although 64 registers spill 412 / 388 bytes a thread, beat five to
// seven.  104 us at 8x64x32^2 against 214 for all four sides in the tables' form, k_s2_recon1 34 against 42 (ncu, cold).
// The limiter's candidate of a sample x < 0, (1 - margin) m / (m - x), falls with x (m > 0; theta is 0 otherwise): the
// smallest sample gives the smallest candidate.
__device__ __forceinline__ double s2_limit(double xmin, double mf) {
    return xmin < 0.0 ? fmin(1.0, (1.0 - 64.0 * kEps) * mf / (mf - xmin)) : 1.0;
}
__device__ __forceinline__ double s2_min(double a, double b) { return b < a ? b : a; }

__device__ __forceinline__ void s2_recon2_wall(const LoParams& P, const LoBuffers& B, const S2Buffers& S, int cc, int kgroup,
                                               double (*s_th)[32]) {
    const int nv = P.nvel, nx = P.nx, ny = P.ny, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f = warp >> 1, axis = warp & 1;
    const int k0 = kgroup * 32 + lane;
    const bool kok = k0 < nv;
    const int k = kok ? k0 : nv - 1;
    const int i = cc % nx, j = cc / nx;
    const int first = s2_wall_first(j, ny);   // rows of the x first layer
    const double* L1 = S.l1 + (size_t)f * 11 * nv + k;
    auto X = [&](int r, int q) { return L1[((size_t)((first + r) * nx + i) * 22 + q) * nv]; };
    const double hm = B.h[(size_t)cc * nv + k], bm = B.b[(size_t)cc * nv + k];
    const double mf = f == 0 ? hm : bm;
    double face[2][3], dn[2][3], dt[2][3], xmin = 0.0, sum = 0.0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        double a5[5], b5[5], dummy;
        if (axis == 0) {
#pragma unroll
            for (int r = 0; r < 5; ++r) { a5[r] = X(r, 2 * s); b5[r] = X(r, 2 * s + 1); }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                s2_wall_eval(a5, j, ny, c_s2.gnode[a], face[s][a], dt[s][a]);
                s2_wall_eval(b5, j, ny, c_s2.gnode[a], dn[s][a], dummy);
            }
        } else {
            const S2Field F{(f == 0 ? B.h : B.b) + k, nv, nx, ny};
#pragma unroll
            for (int r = -2; r <= 2; ++r) {
                double q[5];
#pragma unroll
                for (int t = 0; t < 5; ++t) q[t] = F.at(i + r, first + t);
                s2_wall_eval(q, j, ny, s == 0 ? -0.5 : 0.5, a5[r + 2], b5[r + 2]);
            }
            s2_power_companion3(a5, b5, face[s], dt[s], dn[s]);
        }
        const int row = axis == 0 ? s : 2;   // volume Gauss rows 0, 1 by the x warp, 2 by the y warp
        if (axis == 0 || s == 0) {
#pragma unroll
            for (int r = 0; r < 5; ++r) a5[r] = X(r, 4 + row);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                double vol;
                s2_wall_eval(a5, j, ny, c_s2.gnode[b], vol, dummy);
                xmin = s2_min(xmin, vol);
                sum += vol;
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            xmin = s2_min(xmin, face[s][a]);
            sum += face[s][a] + dn[s][a] + dt[s][a];
        }
    }
    s_th[warp][lane] = s2_limit(xmin, mf);
    __syncthreads();
    double theta = fmin(fmin(s_th[0][lane], s_th[1][lane]), fmin(s_th[2][lane], s_th[3][lane]));
    theta = (hm <= 0.0 || bm <= 0.0) ? 0.0 : fmax(0.0, fmin(1.0, theta));
    // the derivatives are divided by the cell sizes (limit_cell_outputs): multiplied by the reciprocals
    // here, exact when dx and dy are powers of two (the delivered meshes), within an ulp otherwise
    const double ind = 1.0 / (axis == 0 ? P.dx : P.dy), itd = 1.0 / (axis == 0 ? P.dy : P.dx);
    const int fv = f == 0 ? 0 : 1, fn = f == 0 ? 2 : 4, ft = f == 0 ? 3 : 5;
    const double uk = B.u[k], vk = B.v[k];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const bool store = kok && rec_leaves(2 * axis + s, uk, vk);
        const bool wall = kok && axis == 1 && ((s == 0 && j == 0) || (s == 1 && j == ny - 1));
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double v = mf + theta * (face[s][a] - mf), n = theta * dn[s][a] * ind, t = theta * dt[s][a] * itd;
            if (store) {
                S.rec[rec_cell(cc, axis, f, a, nv) + k] = v;
                S.rec[rec_cell(cc, axis, 2 + f, a, nv) + k] = axis == 0 ? uk * n + vk * t : vk * n + uk * t;
            }
            if (wall) {
                S.rec[rec_wall(nx, ny, s, i, fv, a, nv) + k] = v;
                S.rec[rec_wall(nx, ny, s, i, fn, a, nv) + k] = n;
                S.rec[rec_wall(nx, ny, s, i, ft, a, nv) + k] = t;
            }
        }
    }
    if (kok && !(isfinite(sum) && isfinite(theta))) set_status(B.status, ST_NONFINITE_FLUX);
}

constexpr int kRecon2Threads = 128;
__global__ void __launch_bounds__(kRecon2Threads, 8) k_s2_recon2(LoParams P, LoBuffers B, S2Buffers S) {
    if (eval_cached(B)) return;
    __shared__ double s_th[kRecon2Threads / 32][32];
    const int nv = P.nvel, nx = P.nx, ny = P.ny, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // CTAs: the wall rows' (row, i, 32 velocities), then the other cells' (cell, 2 x 32 velocities)
    const int ng = (nv + 31) >> 5, nq = (ng + 1) >> 1, wrows = min(ny, 6), nwall = wrows * nx * ng;
    int id = (int)blockIdx.x;
    if (id < nwall) {
        const int c = id / ng, row = c / nx;
        s2_recon2_wall(P, B, S, (row < 3 ? row : ny - wrows + row) * nx + c % nx, id % ng, s_th);
        return;
    }
    id -= nwall;
    const int c0 = id / nq, i = c0 % nx, j = 3 + c0 / nx, cc = j * nx + i, f = warp & 1;
    const int k0 = ((id % nq) * 2 + (warp >> 1)) * 32 + lane;
    const bool kok = k0 < nv;
    const int k = kok ? k0 : nv - 1;
    const size_t st = (size_t)22 * nv, rowst = st * nx;
    const double* L1 = S.l1 + (size_t)f * 11 * nv + k + (size_t)cc * st;
    const double hm = B.h[(size_t)cc * nv + k], bm = B.b[(size_t)cc * nv + k], mf = f == 0 ? hm : bm;
    double xmin = 0.0, sum = 0.0;   // sum: a value of every template with all its coefficients, for their finiteness
#pragma unroll
    for (int axis = 0; axis < 2; ++axis) {
        const double vn = axis == 0 ? B.u[k] : B.v[k], vt = axis == 0 ? B.v[k] : B.u[k];
        const bool hi = vn >= 0.0;   // the upper side is the leaving one
        const double* L = L1 + (size_t)(axis == 0 ? 0 : 7) * nv;
        const double *Lv = L + (size_t)(hi ? 2 : 0) * nv, *Lo = L + (size_t)(hi ? 0 : 2) * nv;
        double a5[5], b5[5], o5[5], face[3], dn[3], dt[3], ov[3];
#pragma unroll
        for (int r = 0; r < 5; ++r) {
            const long long off = axis == 0 ? (long long)(r - 2) * (long long)rowst
                                            : (long long)(wrapx(i + r - 2, nx) - i) * (long long)st;
            a5[r] = Lv[off];
            b5[r] = Lv[off + nv];
            o5[r] = Lo[off];
        }
        s2_power_companion3(a5, b5, face, dt, dn);
        s2_power_values3(o5, ov);
        // the derivatives are divided by the cell sizes (limit_cell_outputs): multiplied by the reciprocals
        // here, exact when dx and dy are powers of two (the delivered meshes), within an ulp otherwise
        const double in = vn * (1.0 / (axis == 0 ? P.dx : P.dy)), it = vt * (1.0 / (axis == 0 ? P.dy : P.dx));
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            xmin = s2_min(s2_min(xmin, face[a]), ov[a]);
            const double path = in * dn[a] + it * dt[a];
            if (a == 2) sum += (face[a] + path) + ov[a];
            if (kok) {   // unlimited: theta is 1 but for a few cells and velocities
                S.rec[rec_cell(cc, axis, f, a, nv) + k] = face[a];
                S.rec[rec_cell(cc, axis, 2 + f, a, nv) + k] = path;
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {   // volume Gauss row p
        double a5[5], vol[3];
#pragma unroll
        for (int r = 0; r < 5; ++r) a5[r] = L1[(long long)(r - 2) * (long long)rowst + (size_t)(4 + p) * nv];
        s2_power_values3(a5, vol);
#pragma unroll
        for (int a = 0; a < 3; ++a) xmin = s2_min(xmin, vol[a]);
        sum += vol[2];
    }
    const double cand = s2_limit(xmin, mf);
    s_th[warp][lane] = cand;
    __syncthreads();
    double theta = fmin(cand, s_th[warp ^ 1][lane]);
    theta = (hm <= 0.0 || bm <= 0.0) ? 0.0 : fmax(0.0, fmin(1.0, theta));
    if (!kok) return;
    if (theta < 1.0) {   // the limiter acts: the values this thread stored, drawn towards the mean
#pragma unroll 1
        for (int axis = 0; axis < 2; ++axis)
#pragma unroll 1
            for (int a = 0; a < 3; ++a) {
                double* v = S.rec + rec_cell(cc, axis, f, a, nv) + k;
                *v = mf + theta * (*v - mf);
                S.rec[rec_cell(cc, axis, 2 + f, a, nv) + k] *= theta;
            }
    }
    if (!isfinite(sum)) set_status(B.status, ST_NONFINITE_FLUX);
}

// first and second layer of all cells
static cudaError_t launch_recon(const LoParams& P, const LoBuffers& B, const S2Buffers& S, cudaStream_t s) {
    const int ng = (P.nvel + 31) / 32, inner = P.ny > 6 ? P.ny - 6 : 0, wall = P.ny - inner;
    k_s2_recon1<<<dim3((unsigned)ng, (unsigned)(P.nx * P.ny)), 128, 0, s>>>(P, B, S);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_s2_recon2<<<(unsigned)(P.nx * (wall * ng + inner * ((ng + 1) / 2))), kRecon2Threads, 0, s>>>(P, B, S);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------
// S2 cold start: one warp per cell, h, b := the discrete closure Maxwellian of W
__global__ void __launch_bounds__(256, 2) k_s2_init(LoParams P, LoBuffers B, S2Buffers SB) {
    const int nv = P.nvel, nc = P.nx * P.ny, lane = threadIdx.x & 31, nr = (nv + 31) >> 5;
    const int cc = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (cc >= nc) return;
    __shared__ double s_jac[8][16];
    double w[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) w[m] = B.W[cc * 4 + m];
    WClosure C;
    C.jac = s_jac[threadIdx.x >> 5];
    WMke M;
    const bool ok = w_closure(P, B, w, C) && w_make_mke(P, B, w, C, M);
    const S2Th tt = s2_th(C.th, P.ck);
    if (ok)
        for (int r = 0; r < nr; ++r) {
            const WVel s = wvel(B, nv, r);
            const S2Q q = s2_q(tt, s.u, s.v);
            if (s.ok) { B.h[(size_t)cc * nv + s.k] = q.qh; B.b[(size_t)cc * nv + s.k] = q.qb; }
        }
    if (!ok && lane == 0) set_status(B.status, ST_PROJECTION);
}

// macro WENO of W: per interior face and component the normal slopes of both sides and the
// tangential slope at the 3 Gauss nodes (s2d1_face3, compute_flux :803-808,849-854), and per cell
// and component the 3x3 Gauss values and the mean-shifted volume node states (build_targets
// :1270-1279).  Faces: 2 warps per face, an 8-lane group per (component, side); cells: one warp per
// cell, an 8-lane group per component.
__global__ void __launch_bounds__(128) k_s2_macro(LoParams P, LoBuffers B, S2Buffers SB, int faces, int cells) {
    if (eval_cached(B)) return;
    const int nx = P.nx, ny = P.ny, nfx = nx * ny, nf = nfx + nx * (ny - 1), nc = nx * ny;
    int wid = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31, grp = lane >> 3, gl = lane & 7;
    const int nfw = faces ? nf * 2 : 0;
    if (wid < nfw) {
        const int fi = wid >> 1, m = (wid & 1) * 2 + (grp >> 1), right = grp & 1;
        const int axis = fi < nfx ? 0 : 1, f = axis == 0 ? fi : fi - nfx;
        const int i = f % nx, j = f / nx;
        const S2Field F{B.W + m, 4, nx, ny};
        double dn[3] = {0.0, 0.0, 0.0}, dt[3] = {0.0, 0.0, 0.0};
        bool ok;
        if (axis == 0) ok = s2_side3_group(F, 0, right ? (i + 1) % nx : i, j, right ? -0.5 : 0.5, gl, dn, dt);
        else ok = s2_side3_group(F, 1, right ? j + 1 : j, i, right ? -0.5 : 0.5, gl, dn, dt);
        // the right side's tangential derivatives to the left side's lane 0
        double tr[3];
#pragma unroll
        for (int g = 0; g < 3; ++g) tr[g] = __shfl_down_sync(0xffffffffu, dt[g], 8);
        if (gl == 0) {
            if (!ok) set_status(B.status, ST_NONFINITE_FLUX);
            const double dnrm = axis == 0 ? P.dx : P.dy, dtg = axis == 0 ? P.dy : P.dx;
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                double* o = SB.mac + (size_t)(fi * 3 + g) * 12;
                o[(right ? 4 : 0) + m] = dn[g] / dnrm;
                if (!right) o[8 + m] = 0.5 * (dt[g] + tr[g]) / dtg;
            }
        }
        return;
    }
    wid -= nfw;
    if (!cells || wid >= nc) return;
    const int cc = wid, m = grp, i = cc % nx, j = cc / nx;
    const S2Field F{B.W + m, 4, nx, ny};
    double vol[3] = {0.0, 0.0, 0.0};
    const bool ok = s2_cell9_group(F, i, j, gl, vol);
    if (__any_sync(0xffffffffu, !ok) && lane == 0) set_status(B.status, ST_PROJECTION);
    // nodes[a][c] = vol of lane a, entry c; the mean over the 9 nodes in the reference's order
    const int base = lane & ~7;
    double nodes[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) nodes[a][c] = __shfl_sync(0xffffffffu, vol[c], base + a);
    const double gw[3] = {5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0};
    double avg = 0.0;
    for (int c = 0; c < 3; ++c)
        for (int a = 0; a < 3; ++a) avg = avg + gw[a] * gw[c] * nodes[a][c];
    const double wc = B.W[cc * 4 + m];
    if (gl < 3)
        for (int c = 0; c < 3; ++c) SB.wq[((size_t)cc * 9 + c * 3 + gl) * 4 + m] = nodes[gl][c] + wc - avg;
}

// The face-node closure kernel comes in two CTA shapes.  A single instance runs it in 128-thread
// CTAs, three per SM: up to 170 registers a thread (no spills) at 12 warps per SM, faster per step
// than two 256-thread CTAs per SM capped at 128 registers (which spill the closure's state).  Many
// instances on concurrent streams (S2Buffers::concurrent) gain more from the 16 resident warps of
// the 256-thread shape, which they keep.  The volume-node kernel is fastest in the 256-thread shape
// in both cases.
constexpr int kS2NodeThreads = 128;

// build_targets, closure part: one warp per (cell, volume node) -> the node scalars
__global__ void __launch_bounds__(256, 2) k_s2_target_nodes(LoParams P, LoBuffers B, S2Buffers SB, int qrec) {
    if (eval_cached(B)) return;
    extern __shared__ double s_qrec[];
    const int nc = P.nx * P.ny, lane = threadIdx.x & 31;
    const int wid = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (wid >= nc * 9) return;
    __shared__ double s_jac[8][16];
    double w[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) w[m] = SB.wq[(size_t)wid * 4 + m];
    WClosure C;
    C.jac = s_jac[threadIdx.x >> 5];
    WMke M;
    const WQRec qr{qrec ? s_qrec + (threadIdx.x >> 5) * (((P.nvel + 31) >> 5) * 32) : nullptr};
    const bool ok = w_closure(P, B, w, C, qr) && w_make_mke(P, B, w, C, M, qr);
    if (lane == 0) {
        if (ok) w_store_scalars(SB.tscal + (size_t)wid * kS2TScal, C, M);
        else set_status(B.status, ST_PROJECTION);
    }
}

// build_targets, sum part: per (cell, velocity) the Gauss-weighted M, K_x, K_y of the 9 nodes
__global__ void __launch_bounds__(256) k_s2_target_sum(LoParams P, LoBuffers B, S2Buffers SB) {
    if (eval_cached(B)) return;
    const int nv = P.nvel, cc = blockIdx.y;
    const int k = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= nv) return;
    const double uk = B.u[k], vk = B.v[k];
    const double gw[3] = {5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0};
    double amh = 0.0, amb = 0.0, akxh = 0.0, akxb = 0.0, akyh = 0.0, akyb = 0.0;
    for (int p = 0; p < 9; ++p) {
        double th[4];
        WMke M;
        w_load_scalars(SB.tscal + ((size_t)cc * 9 + p) * kS2TScal, th, M);
        S2Q q;
        double mh, mb, kxh, kxb, kyh, kyb;
        w_mke_at(s2_th(th, P.ck), M, P.ck, uk, vk, q, mh, mb, kxh, kxb, kyh, kyb);
        const double wt2 = gw[p % 3] * gw[p / 3];
        amh = amh + wt2 * mh; amb = amb + wt2 * mb;
        akxh = akxh + wt2 * kxh; akxb = akxb + wt2 * kxb;
        akyh = akyh + wt2 * kyh; akyb = akyb + wt2 * kyb;
    }
    const size_t q = (size_t)cc * nv + k;
    SB.mh[q] = amh; SB.mb[q] = amb; SB.kxh[q] = akxh; SB.kxb[q] = akxb; SB.kyh[q] = akyh; SB.kyb[q] = akyb;
}

// build_targets on a tensor-product velocity table (LoParams::tnu > 0): the closures by 1-D sums, eight lanes a
// (cell, volume node), four nodes a warp -> the same node scalars.  Bound by the latency of the Newton
// chain (two exponentials, a butterfly, a 4x4 solve an evaluation): 16 us at 8x64x32^2 and 27 for the sums below, against 165
// and 49 for the kernels above (ncu, cold).  Eight lanes a
// node share the uniform scalar work four ways a warp and still fill the chip with 1152 warps at that size.
// A table that is no tensor product (tensor_table) takes the kernels above.
template <int R>
__global__ void __launch_bounds__(128, 3) k_s2_target_nodes_t(LoParams P, LoBuffers B, S2Buffers SB) {
    if (eval_cached(B)) return;
    __shared__ double s_jac[128 / kTG][17];
    const int nn = P.nx * P.ny * 9, gl = threadIdx.x & (kTG - 1);
    const int id = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kTG), node = min(id, nn - 1);
    double w[4], td[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) w[m] = SB.wq[(size_t)node * 4 + m];
    TClosure C;
    C.jac = s_jac[threadIdx.x / kTG];
    WMke M;
    bool ok = t_closure<R>(P, B, w, id < nn, C);
    ok = t_mke<R>(P, B, w, C, M, nullptr, td) && ok;
    if (id >= nn) return;
    if (!ok) {
        if (gl == 0) set_status(B.status, ST_PROJECTION);
        return;
    }
    double* o = SB.tscal + (size_t)node * kS2TScal;
    if (gl == 0) {
#pragma unroll
        for (int m = 0; m < 4; ++m) { o[m] = C.th[m]; o[4 + m] = M.tdx[m]; o[8 + m] = M.tdy[m]; }
        o[12] = M.ux; o[13] = M.vy; o[14] = M.lam; o[15] = M.coeff;
    }
    o[16 + gl] = C.jac[gl];
    o[24 + gl] = C.jac[8 + gl];
}

// build_targets, sum part, on a tensor table: one CTA per cell (STargets, ugks_s2_tensor.cuh)
__global__ void __launch_bounds__(256, 2) k_s2_target_sum_t(LoParams P, LoBuffers B, S2Buffers SB) {
    if (eval_cached(B)) return;
    __shared__ STargets st;
    __shared__ double red[8 * 8], rout[kRedSlots];
    const int nv = P.nvel, cc = blockIdx.x, tid = threadIdx.x, nt = (int)blockDim.x;
    st.fill(P, B, SB, cc);
    __syncthreads();
    double* out[6] = {SB.mh, SB.mb, SB.kxh, SB.kxb, SB.kyh, SB.kyb};
    double mom[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) mom[m] = 0.0;
    for (int k0 = tid; k0 < nv; k0 += 4 * nt) {
        double a[4][6];
        st.at<4>(P, B, k0, nt, a);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = k0 + r * nt;
            if (k < nv) {
                moment_add(B.w[k], B.u[k], B.v[k], a[r][2], a[r][3], mom);
                moment_add(B.w[k], B.u[k], B.v[k], a[r][4], a[r][5], mom + 4);
#pragma unroll
                for (int m = 0; m < 6; ++m) out[m][(size_t)cc * nv + k] = a[r][m];
            }
        }
    }
    block_reduce_smem<8, 0>(mom, red, rout);
    if (tid < 8 && !(fabs(rout[tid]) <= kTGate)) set_status(B.status, ST_PROJECTION);
}

// ------------------------------------------------------------------------------------------
// interior face nodes (ugks_node, mod_S2D1.f90:421-521), scalar part: one warp per (face, Gauss
// node) -- the right x face of every cell, then the top y face of every cell below the last row --
// computes W0, the closure, make_mke, q0, the slope and time directions and Mt, and stores them as
// the node's scalars (SB.fscal) for k_s2_face_flux.
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_s2_face_nodes(LoParams P, LoBuffers B, S2Buffers SB, int qrec) {
    if (eval_cached(B)) return;
    extern __shared__ double s_qrec[];
    const int nv = P.nvel, nx = P.nx, ny = P.ny, ck = P.ck, lane = threadIdx.x & 31, nr = (nv + 31) >> 5;
    const int nfx = nx * ny, nf = nfx + nx * (ny - 1);
    const int wid = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (wid >= nf * 3) return;
    const int fi = wid / 3, g = wid % 3;
    const int axis = fi < nfx ? 0 : 1, f = axis == 0 ? fi : fi - nfx;
    const int cl = f, i = cl % nx, j = cl / nx;
    const int cr = axis == 0 ? j * nx + (i + 1) % nx : (j + 1) * nx + i;
    const double dt = B.dt[0];
    const double* mac = SB.mac + (size_t)wid * 12;   // [nl | nr | t][component] of this node
    auto upwind = [&](const WVel& s, int field) {
        const double vn = axis == 0 ? s.u : s.v;
        const bool left = vn >= 0.0;
        return SB.rec[rec_cell(left ? cl : cr, axis, field, g, nv) + s.k];
    };
    // W0: moments of the upwind face values
    double acc[16];
#pragma unroll
    for (int m = 0; m < 4; ++m) acc[m] = 0.0;
    for (int r = 0; r < nr; ++r) {
        const WVel s = wvel(B, nv, r);
        moment_add(s.w, s.u, s.v, upwind(s, 0), upwind(s, 1), acc);
    }
    warp_sum_all<4>(acc);
    const double w0[4] = {acc[0], acc[1], acc[2], acc[3]};
    __shared__ double s_jac[NT / 32][16];
    WClosure C;
    C.jac = s_jac[threadIdx.x >> 5];
    WMke M;
    const WQRec qr{qrec ? s_qrec + (threadIdx.x >> 5) * (nr * 32) : nullptr};
    bool ok = w_closure(P, B, w0, C, qr) && w_make_mke(P, B, w0, C, M, qr);
    double q0x = 0.0, q0y = 0.0, tdl[4], tdr[4], tdt[4], tdm[4], wt[4], mt[5], tau = 0.0;
    if (ok) {   // q0 = heat(w0, f0 - analytic Maxwellian of w0)
        const double nrho = w0[0], nu = w0[1] / w0[0], nvv = w0[2] / w0[0];
        const double temp = 4.0 * (w0[3] / w0[0] - 0.5 * (nu * nu + nvv * nvv)) / (double)(ck + 2);
        const double lamn = 1.0 / temp;
        // directions of the macro normal slopes (left, right) and the tangential slope
        const bool okd = s2_solve4(C.jac, mac, tdl) & s2_solve4(C.jac, mac + 4, tdr) & s2_solve4(C.jac, mac + 8, tdt);
        if (!okd)
#pragma unroll
            for (int m = 0; m < 4; ++m) tdl[m] = tdr[m] = tdt[m] = NAN;
        // one pass over the velocities for q0 (qacc) and the direction moments (acc): two independent
        // chains per velocity, each summed in velocity order and reduced on its own
        double qacc[2] = {0.0, 0.0};
#pragma unroll
        for (int m = 0; m < 16; ++m) acc[m] = 0.0;
        const S2Th tt = s2_th(C.th, ck);
        for (int r = 0; r < nr; ++r) {
            const WVel s = wvel(B, nv, r);
            {
                const double du = s.u - nu, dv = s.v - nvv;
                const double eah = nrho * lamn / kPi * exp(-lamn * (du * du + dv * dv));
                const double eab = 0.5 * (double)ck * temp * eah;
                const double cx = s.u - M.ux, cy = s.v - M.vy, c2 = cx * cx + cy * cy;
                const double dh = upwind(s, 0) - eah, db = upwind(s, 1) - eab;
                qacc[0] += 0.5 * s.w * cx * (c2 * dh + db);
                qacc[1] += 0.5 * s.w * cy * (c2 * dh + db);
            }
            const S2Q q = qr.at(tt, s, r);
            double dlh, dlb, drh, drb, dth, dtb;
            s2_dq(q, tdl, dlh, dlb);
            s2_dq(q, tdr, drh, drb);
            s2_dq(q, tdt, dth, dtb);
            moment_add(s.w, s.u, s.v, dlh, dlb, acc);
            moment_add(s.w, s.u, s.v, drh, drb, acc + 4);
            moment_add(s.w, s.u, s.v, dth, dtb, acc + 8);
            const double vn = axis == 0 ? s.u : s.v, vt = axis == 0 ? s.v : s.u;
            const double fh = vn * (vn >= 0.0 ? dlh : drh) + vt * dth;
            const double fb = vn * (vn >= 0.0 ? dlb : drb) + vt * dtb;
            moment_add(s.w, s.u, s.v, fh, fb, acc + 12);
        }
        warp_sum_all<2>(qacc);
        q0x = qacc[0];
        q0y = qacc[1];
        warp_sum_all<16>(acc);
        for (int d = 0; d < 3; ++d) {   // gates of the three directions
            double mx = 0.0, sc = 1.0;
            for (int m = 0; m < 4; ++m) {
                mx = fmax(mx, fabs(acc[4 * d + m] - mac[4 * d + m]));
                sc = fmax(sc, fabs(mac[4 * d + m]));
            }
            ok = ok && mx / sc <= 2.0e-12;
        }
        // the time direction and the time coefficients Mt (mod_Evolution.f90:346-350)
#pragma unroll
        for (int m = 0; m < 4; ++m) wt[m] = -acc[12 + m];
        ok = ok && s2_solve4(C.jac, wt, tdm);
        ok = ok && s2_tau(P, w0, tau);
        const double ex = exp(-dt / tau);
        mt[3] = tau * (1.0 - ex);
        mt[4] = -tau * dt * ex + tau * mt[3];
        mt[0] = dt - mt[3];
        mt[1] = -tau * mt[0] + mt[4];
        mt[2] = 0.5 * dt * dt - tau * mt[0];
    }
    // the node scalars of the flux pass (k_s2_face_flux)
    if (lane == 0) {
        double* o = SB.fscal + (size_t)wid * kS2FScal;
        o[0] = ok ? 1.0 : 0.0;
        if (ok) {
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                o[1 + m] = C.th[m]; o[5 + m] = M.tdx[m]; o[9 + m] = M.tdy[m];
                o[19 + m] = tdl[m]; o[23 + m] = tdr[m]; o[27 + m] = tdt[m]; o[31 + m] = tdm[m]; o[40 + m] = wt[m];
            }
            o[13] = M.ux; o[14] = M.vy; o[15] = M.lam; o[16] = M.coeff; o[17] = q0x; o[18] = q0y;
#pragma unroll
            for (int m = 0; m < 5; ++m) o[35 + m] = mt[m];
#pragma unroll
            for (int m = 0; m < 16; ++m) o[44 + m] = C.jac[m];
            o[60] = tau;
        } else {
            set_status(B.status, ST_NONFINITE_FLUX);
        }
    }
}

// ugks_node's flux at one face Gauss node (mod_S2D1.f90:486-507): one CTA per (face, node), VPT
// velocities per thread, from the node scalars; the node micro flux goes to SB.node, its moments to
// SB.nodew, and the time-direction moment gate (2e-12) is checked on the block-reduced moments.
// Three CTAs per SM (80 registers, small spills): the kernel waits on its face-cache loads, and 24
// resident warps hide that better than 16.
template <int VPT>
__global__ void __launch_bounds__(256, 3) k_s2_face_flux(LoParams P, LoBuffers B, S2Buffers SB) {
    if (eval_cached(B)) return;
    __shared__ double sc[kS2FScal];
    __shared__ double red[8 * 8];
    __shared__ double rout[kRedSlots];
    const int nv = P.nvel, nx = P.nx, ny = P.ny, ck = P.ck;
    const int nfx = nx * ny;
    const int wid = blockIdx.x, fi = wid / 3, g = wid % 3;
    const int axis = fi < nfx ? 0 : 1, f = axis == 0 ? fi : fi - nfx;
    const int cl = f, i = cl % nx, j = cl / nx;
    const int cr = axis == 0 ? j * nx + (i + 1) % nx : (j + 1) * nx + i;
    if (threadIdx.x < kS2FScal) sc[threadIdx.x] = SB.fscal[(size_t)wid * kS2FScal + threadIdx.x];
    __syncthreads();
    if (sc[0] == 0.0) return;   // the scalars kernel failed (status set there)
    double th[4], tdl[4], tdr[4], tdt[4], tdm[4], mt[5];
    WMke M;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        th[m] = sc[1 + m]; M.tdx[m] = sc[5 + m]; M.tdy[m] = sc[9 + m];
        tdl[m] = sc[19 + m]; tdr[m] = sc[23 + m]; tdt[m] = sc[27 + m]; tdm[m] = sc[31 + m];
    }
    M.ux = sc[13]; M.vy = sc[14]; M.lam = sc[15]; M.coeff = sc[16];
    const double q0x = sc[17], q0y = sc[18];
#pragma unroll
    for (int m = 0; m < 5; ++m) mt[m] = sc[35 + m];
    const S2Th tt = s2_th(th, ck);
    double* outh = SB.node + (size_t)wid * 2 * nv;
    double* outb = outh + nv;
    double acc[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m] = 0.0;
    int bad = 0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot sl_ = slot(r, nv);
        const int k = sl_.kk;
        const double uk = B.u[k], vk = B.v[k], wk = sl_.ok ? B.w[k] : 0.0;
        S2Q q;
        double mh, mb, kxh, kxb, kyh, kyb;
        w_mke_at(tt, M, ck, uk, vk, q, mh, mb, kxh, kxb, kyh, kyb);
        const double s0h = mh + kxh * q0x + kyh * q0y;
        const double s0b = mb + kxb * q0x + kyb * q0y;
        double dlh, dlb, drh, drb, dth, dtb, mth, mtb;
        s2_dq(q, tdl, dlh, dlb);
        s2_dq(q, tdr, drh, drb);
        s2_dq(q, tdt, dth, dtb);
        s2_dq(q, tdm, mth, mtb);
        moment_add(wk, uk, vk, mth, mtb, acc);
        const double vn = axis == 0 ? uk : vk, vt = axis == 0 ? vk : uk;
        const bool left = vn >= 0.0;
        const double* rc = SB.rec + rec_cell(left ? cl : cr, axis, 0, g, nv) + k;   // fields 3 nv apart
        const double f0h = rc[0], f0b = rc[(size_t)3 * nv], ph = rc[(size_t)6 * nv], pb = rc[(size_t)9 * nv];
        const double sh = vn * (left ? dlh : drh) + vt * dth;
        const double sb = vn * (left ? dlb : drb) + vt * dtb;
        const double fhv = vn * (mt[0] * s0h + mt[1] * sh + mt[2] * mth + mt[3] * f0h - mt[4] * ph);
        const double fbv = vn * (mt[0] * s0b + mt[1] * sb + mt[2] * mtb + mt[3] * f0b - mt[4] * pb);
        moment_add(wk, uk, vk, fhv, fbv, acc + 4);
        if (sl_.ok) {
            outh[sl_.k] = fhv;
            outb[sl_.k] = fbv;
            if (!(isfinite(fhv) && isfinite(fbv))) bad = 1;
            if (SB.coef) {   // ugks_node's f0_h, f0_b, k_h, k_b (mod_S2D1.f90:501-505)
                double* cf = SB.coef + (size_t)wid * 4 * nv + sl_.k;
                const double tau = sc[60];
                cf[0] = vn * f0h;
                cf[(size_t)nv] = vn * f0b;
                cf[2 * (size_t)nv] = vn * ((s0h - f0h) / tau - ph);
                cf[3 * (size_t)nv] = vn * ((s0b - f0b) / tau - pb);
            }
        }
    }
    block_reduce_smem<8, 0>(acc, red, rout);
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        double mx = 0.0, scl = 1.0;
#pragma unroll
        for (int m = 0; m < 4; ++m) { mx = fmax(mx, fabs(rout[m] - sc[40 + m])); scl = fmax(scl, fabs(sc[40 + m])); }
#pragma unroll
        for (int m = 0; m < 4; ++m) SB.nodew[(size_t)wid * 4 + m] = rout[4 + m];
        if (bad || !(mx / scl <= 2.0e-12)) set_status(B.status, ST_NONFINITE_FLUX);
    }
}

// ------------------------------------------------------------------------------------------
// interior faces on a tensor-product velocity table, in three kernels:
//   k_s2_face_moments : one CTA a face, the sums of the upwind face values that W0 and q0 of its three nodes need,
//                       taken about the lower cell's velocity -> fscal[1..9] (the only pass over the velocities
//                       that the node's scalars need; bound by the latency of the face cache's values, 48 KB
//                       a face at 32^2: 12 loads in flight a thread, 20 us; 6 in flight or one warp a node cost the step
//                       10 to 16 us more)
//   k_s2_face_nodes_t : eight lanes a node, W0's closure, make_mke, q0, the directions and Mt by 1-D sums
//                       -> the node scalars of k_s2_face_nodes
//   k_s2_face_flux_t  : one CTA a face, its three nodes' micro fluxes and their Gauss sum -> the face arrays
// 20 + 26 + 69 us at 8x64x32^2 against 220 + 63 + 13 for k_s2_face_nodes, k_s2_face_flux and k_s2_combine (ncu, cold), which
// other tables and the wall variants' coefficient outputs keep.
__global__ void __launch_bounds__(128) k_s2_face_moments(LoParams P, LoBuffers B, S2Buffers SB) {
    if (eval_cached(B)) return;
    __shared__ double red[4][32];
    const int nv = P.nvel, nx = P.nx, ny = P.ny, tid = threadIdx.x;
    const int nfx = nx * ny, fi = blockIdx.x;
    const int axis = fi < nfx ? 0 : 1, cl = axis == 0 ? fi : fi - nfx;
    const int i = cl % nx, j = cl / nx;
    const int cr = axis == 0 ? j * nx + (i + 1) % nx : (j + 1) * nx + i;
    const double iw = 1.0 / B.W[cl * 4], ur = B.W[cl * 4 + 1] * iw, vr = B.W[cl * 4 + 2] * iw;
    const double* rl = SB.rec + rec_cell(cl, axis, 0, 0, nv);   // [field][node][nvel]
    const double* rr = SB.rec + rec_cell(cr, axis, 0, 0, nv);
    double a[27];
#pragma unroll
    for (int m = 0; m < 27; ++m) a[m] = 0.0;
#pragma unroll 2
    for (int k = tid; k < nv; k += 128) {
        const double uk = B.u[k], vk = B.v[k], wk = B.w[k];
        const double* rc = ((axis == 0 ? uk : vk) >= 0.0 ? rl : rr) + k;
        const double cx = uk - ur, cy = vk - vr, xx = cx * cx, yy = cy * cy, xy = cx * cy, c2 = xx + yy;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const double h = wk * rc[(size_t)g * nv], b = wk * rc[(size_t)(3 + g) * nv], e = c2 * h + b;
            a[9 * g] += h;
            a[9 * g + 1] += cx * h;
            a[9 * g + 2] += cy * h;
            a[9 * g + 3] += xx * h;
            a[9 * g + 4] += xy * h;
            a[9 * g + 5] += yy * h;
            a[9 * g + 6] += b;
            a[9 * g + 7] += cx * e;
            a[9 * g + 8] += cy * e;
        }
    }
    red[tid >> 5][tid & 31] = warp_halving<27, false>(a);   // lane m: the warp's total of sum m
    __syncthreads();
    if (tid < 27) SB.fscal[((size_t)fi * 3 + tid / 9) * kS2FScal + 1 + tid % 9] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
}

template <int R>
__global__ void __launch_bounds__(128, 3) k_s2_face_nodes_t(LoParams P, LoBuffers B, S2Buffers SB) {
    if (eval_cached(B)) return;
    __shared__ double s_jac[128 / kTG][17];
    const int nx = P.nx, ny = P.ny, ck = P.ck, gl = threadIdx.x & (kTG - 1);
    const int nfx = nx * ny, nn = (nfx + nx * (ny - 1)) * 3;
    const int id = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kTG), node = min(id, nn - 1);
    const int fi = node / 3, axis = fi < nfx ? 0 : 1, cl = axis == 0 ? fi : fi - nfx;
    const double dt = B.dt[0];
    const double* mac = SB.mac + (size_t)node * 12;   // [nl | nr | t][component] of this node
    double* o = SB.fscal + (size_t)node * kS2FScal;
    // W0: the moments of the upwind face values, from the sums about the lower cell's velocity (ur, vr)
    const double iw = 1.0 / B.W[cl * 4], ur = B.W[cl * 4 + 1] * iw, vr = B.W[cl * 4 + 2] * iw;
    double f[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) f[m] = o[1 + m];
    const double w0[4] = {f[0], ur * f[0] + f[1], vr * f[0] + f[2],
                          0.5 * (ur * ur + vr * vr) * f[0] + ur * f[1] + vr * f[2] + 0.5 * (f[3] + f[5] + f[6])};
    TClosure C;
    C.jac = s_jac[threadIdx.x / kTG];
    WMke M;
    double td[4];
    bool ok = t_closure<R>(P, B, w0, id < nn, C);
    ok = t_mke<R>(P, B, w0, C, M, mac, td) && ok;
    // q0 = heat(w0, f0 - analytic Maxwellian of w0) about (ux, vy): f0's part shifted from (ur, vr)
    double q0x, q0y;
    {
        const double temp = 4.0 * (w0[3] / w0[0] - 0.5 * (M.ux * M.ux + M.vy * M.vy)) / (double)(ck + 2), lamn = 1.0 / temp;
        const double dx = M.ux - ur, dy = M.vy - vr, d2 = dx * dx + dy * dy, e2 = f[3] + f[5], dp = dx * f[1] + dy * f[2];
        const double hx = 0.5 * (f[7] - dx * (e2 + f[6]) + d2 * f[1] - d2 * dx * f[0]) - (dx * f[3] + dy * f[4]) + dx * dp;
        const double hy = 0.5 * (f[8] - dy * (e2 + f[6]) + d2 * f[2] - d2 * dy * f[0]) - (dx * f[4] + dy * f[5]) + dy * dp;
        TAxes ax;
        t_sums<R>(B.tab, B.tab + 64, B.tab + 128, B.tab + 192, M.ux, M.vy, lamn, M.ux, M.vy, &ax);
        const double pr = 0.5 * w0[0] * lamn / kPi, cb = 0.5 * (double)ck * temp;
        q0x = hx - pr * (ax.x[3] * ax.y[0] + ax.x[1] * ax.y[2] + cb * ax.x[1] * ax.y[0]);
        q0y = hy - pr * (ax.y[3] * ax.x[0] + ax.y[1] * ax.x[2] + cb * ax.y[1] * ax.x[0]);
    }
    // wt = -moments of vn (left ? dl : dr) + vt dt: lane 2 sums the left half of the normal axis with the left
    // direction, lane 3 the right half with the right one, lane 4 the other axis with the tangential one
    const S2Th t = s2_th(C.th, ck);
    double wt[4], tdm[4];
    {
        const double* tn = B.tab + (axis == 0 ? 0 : 128);
        const double* to = B.tab + (axis == 0 ? 128 : 0);
        const double un0 = axis == 0 ? t.u : t.v, uo0 = axis == 0 ? t.v : t.u;
        const double* h = B.tab + (axis == 0 ? 256 : 384);   // weights of the normal axis's halves
        TAxes l, rt;   // (normal half vn >= 0, other axis), (normal half vn < 0, other axis)
        t_sums<R>(tn, h, to, to + 64, un0, uo0, t.itw, un0, uo0, &l);
        t_sums<R>(tn, h + 64, to, to + 64, un0, uo0, t.itw, un0, uo0, &rt);
        double N[6], O[5];
#pragma unroll
        for (int a = 0; a < 6; ++a) N[a] = gl == 4 ? l.y[a] : (gl == 3 ? rt.x[a] : l.x[a]);
#pragma unroll
        for (int a = 0; a < 5; ++a) O[a] = gl == 4 ? l.x[a] + rt.x[a] : l.y[a];
        const bool nisx = (axis == 0) != (gl == 4);   // this lane's normal component is x
        const double un = gl == 4 ? uo0 : un0, uo = gl == 4 ? un0 : uo0;
        const double d0 = td[0] * t.ir - td[3] * t.itw, d3 = td[3] * t.itw * t.itw, db = td[3] * t.itw;
        const double dn = 2.0 * t.itw * (nisx ? td[1] : td[2]), dco = 2.0 * t.itw * (nisx ? td[2] : td[1]);
        // f = (un + cn)(d0 + dn cn + do co + d3 c^2): its sums with 1, cn, co, c^2 by rows of equal cn power
        const double p00 = un * d0, p10 = d0 + un * dn, p20 = dn + un * d3, p01 = un * dco, p02 = un * d3;
        double F[4][3];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            F[0][b] = p00 * O[b] + p01 * O[b + 1] + p02 * O[b + 2];
            F[1][b] = p10 * O[b] + dco * O[b + 1] + d3 * O[b + 2];
            F[2][b] = p20 * O[b];
            F[3][b] = d3 * O[b];
        }
        double m0 = 0.0, mn = 0.0, mo = 0.0, m2 = 0.0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            m0 += N[a] * F[a][0];
            mn += N[a + 1] * F[a][0];
            mo += N[a] * F[a][1];
            m2 += N[a + 2] * F[a][0] + N[a] * F[a][2];
        }
        const double mb = m0 + db * O[0] * (un * N[0] + N[1]);
        const double cn = t.pref * (un * m0 + mn), co = t.pref * (uo * m0 + mo);
        double c[4] = {t.pref * m0, nisx ? cn : co, nisx ? co : cn,
                       t.pref * (0.5 * (un * un + uo * uo) * m0 + un * mn + uo * mo + 0.5 * m2 + 0.5 * t.ckh * mb)};
#pragma unroll
        for (int m = 0; m < 4; ++m) wt[m] = -(t_get(c[m], 2) + t_get(c[m], 3) + t_get(c[m], 4));
        ok = t_solve(C.jac, wt, tdm) && ok;   // its moments are gated in k_s2_face_flux_t
    }
    double tau = 0.0, mt[5];
    ok = ok && s2_tau(P, w0, tau) && isfinite(q0x) && isfinite(q0y);
    const double ex = exp(-dt / tau);   // Mt (mod_Evolution.f90:346-350)
    mt[3] = tau * (1.0 - ex);
    mt[4] = -tau * dt * ex + tau * mt[3];
    mt[0] = dt - mt[3];
    mt[1] = -tau * mt[0] + mt[4];
    mt[2] = 0.5 * dt * dt - tau * mt[0];
    if (id >= nn) return;
    if (!ok) {
        if (gl == 0) { o[0] = 0.0; set_status(B.status, ST_NONFINITE_FLUX); }
        return;
    }
    if (gl == 0) {
        o[0] = 1.0;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            o[1 + m] = C.th[m]; o[5 + m] = M.tdx[m]; o[9 + m] = M.tdy[m]; o[31 + m] = tdm[m]; o[40 + m] = wt[m];
        }
        o[13] = M.ux; o[14] = M.vy; o[15] = M.lam; o[16] = M.coeff; o[17] = q0x; o[18] = q0y;
#pragma unroll
        for (int m = 0; m < 5; ++m) o[35 + m] = mt[m];
        o[60] = tau;
    } else if (gl >= 2 && gl < 5) {
#pragma unroll
        for (int m = 0; m < 4; ++m) o[19 + (gl - 2) * 4 + m] = td[m];
    }
    o[44 + gl] = C.jac[gl];
    o[52 + gl] = C.jac[8 + gl];
}

// The flux of a face: at each node, per velocity, the Maxwellian (a product of two rows of exponentials in
// shared memory) times a cubic in the velocity, whose coefficients join s0, the slope and the time directions
// with their Mt, plus the face values' part (ugks_node, mod_S2D1.f90:486-507).  The three nodes' Gauss sum
// goes straight to the face arrays and its velocity moments are the face's macro flux, so no node flux is
// stored.  The moments of each node's time direction are summed on the way and gated as in k_s2_face_flux (6 us of 69).
// Bound by the latency of the face cache's 12 values a (face, velocity), 100 MB at 8x64x32^2.  The nodes unrolled wait on
// instruction fetch (30 to 60 us more a step).
struct S2FluxC {
    double u, v, ux, vy, ckh, l2, kq, kb, qx, qy, mt0, mt3, mt4;   // means, ck T / 2, 2 lam, mt0 coeff, kq 2 / ck, q0, Mt
    double e[5], t[5], d[2][5];   // polynomials 1, cx, cy, c^2 and b part: mt2 dm - mt0 K dirs; mt1 tangential; mt1 left, right
    double m[5];                  // dm, the time direction
};
__global__ void __launch_bounds__(256, 2) k_s2_face_flux_t(LoParams P, LoBuffers B, S2Buffers SB) {
    if (eval_cached(B)) return;
    __shared__ double ex[3][64], ey[3][64];
    __shared__ S2FluxC sc[3];
    __shared__ double red[8 * 8], rout[kRedSlots], s_time[8][12];   // s_time: the warps' moments of the nodes' time directions
    const int nv = P.nvel, nu = P.tnu, nw = P.tnv, nx = P.nx, ny = P.ny, nfx = nx * ny, tid = threadIdx.x;
    const int fi = blockIdx.x, axis = fi < nfx ? 0 : 1, cl = axis == 0 ? fi : fi - nfx, i = cl % nx, j = cl / nx;
    const int cr = axis == 0 ? j * nx + (i + 1) % nx : (j + 1) * nx + i;
    const double* fs = SB.fscal + (size_t)fi * 3 * kS2FScal;
    if (fs[0] == 0.0 || fs[kS2FScal] == 0.0 || fs[2 * kS2FScal] == 0.0) return;   // a failed node (status set there)
    if (tid < 3) {
        const double* o = fs + tid * kS2FScal;
        const double th[4] = {o[1], o[2], o[3], o[4]};
        const S2Th t = s2_th(th, P.ck);
        S2FluxC& c = sc[tid];
        c.u = t.u; c.v = t.v; c.ux = o[13]; c.vy = o[14]; c.ckh = t.ckh; c.l2 = 2.0 * o[15];
        c.qx = o[17]; c.qy = o[18]; c.mt0 = o[35]; c.mt3 = o[38]; c.mt4 = o[39];
        c.kq = o[35] * o[16]; c.kb = c.kq * (2.0 / (double)P.ck);
        auto poly = [&](const double* td, double* p) {
            p[0] = td[0] * t.ir - td[3] * t.itw;
            p[1] = 2.0 * t.itw * td[1];
            p[2] = 2.0 * t.itw * td[2];
            p[3] = td[3] * (t.itw * t.itw);
            p[4] = td[3] * t.itw;
        };
        double x[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = o[37] * o[31 + m] - o[35] * (o[17] * o[5 + m] + o[18] * o[9 + m]);
        poly(x, c.e);
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = o[36] * o[27 + m];
        poly(x, c.t);
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = o[36] * o[19 + m];
        poly(x, c.d[0]);
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = o[36] * o[23 + m];
        poly(x, c.d[1]);
        poly(o + 31, c.m);
    }
    if (tid < 96) s_time[tid / 12][tid % 12] = 0.0;
    for (int q = tid; q < 3 * (nu + nw); q += blockDim.x) {
        const int g = q / (nu + nw), a = q - g * (nu + nw);
        const double* o = fs + g * kS2FScal + 1;
        const double itw = 1.0 / o[3];
        if (a < nu) {
            const double d = B.tab[a] - o[1];
            ex[g][a] = o[0] / (kPi * o[3]) * exp(-(d * d) * itw);
        } else {
            const double d = B.tab[128 + a - nu] - o[2];
            ey[g][a - nu] = exp(-(d * d) * itw);
        }
    }
    __syncthreads();
    const double gw[3] = {5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0};
    const double len = axis == 0 ? P.dy : P.dx;
    const size_t out = axis == 0 ? (size_t)j * nx + (i + 1) % nx : (size_t)(j + 1) * nx + i;
    double* Fh = (axis == 0 ? B.fxh : B.fyh) + out * nv;
    double* Fb = (axis == 0 ? B.fxb : B.fyb) + out * nv;
    double* Fw = (axis == 0 ? B.fxw : B.fyw) + out * 4;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    int bad = 0;
    for (int kb = 0; kb < nv; kb += 4 * (int)blockDim.x) {   // every lane, for the warps' sums
        const int k0 = kb + tid;
        double fh[4], fb[4], uk[4], vk[4];
        int iu[4], iv[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = min(k0 + r * (int)blockDim.x, nv - 1);
            iv[r] = k / nu;
            iu[r] = k - iv[r] * nu;
            uk[r] = B.tab[iu[r]];
            vk[r] = B.tab[128 + iv[r]];
            fh[r] = fb[r] = 0.0;
        }
#pragma unroll 1
        for (int g = 0; g < 3; ++g) {
            const S2FluxC& c = sc[g];
            double mt[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const double vn = axis == 0 ? uk[r] : vk[r], vt = axis == 0 ? vk[r] : uk[r];
                const bool left = vn >= 0.0;
                const double* rc = SB.rec + rec_cell(left ? cl : cr, axis, 0, g, nv) + min(k0 + r * (int)blockDim.x, nv - 1);
                const double f0h = rc[0], f0b = rc[(size_t)3 * nv], ph = rc[(size_t)6 * nv], pb = rc[(size_t)9 * nv];
                const double* d = c.d[left ? 0 : 1];
                const double q = ex[g][iu[r]] * ey[g][iv[r]];
                const double cx = uk[r] - c.u, cy = vk[r] - c.v, px = uk[r] - c.ux, py = vk[r] - c.vy;
                const double c2 = cx * cx + cy * cy, qd = c.qx * px + c.qy * py;
                const double pe = c.e[0] + c.e[1] * cx + c.e[2] * cy + c.e[3] * c2;
                const double pd = d[0] + d[1] * cx + d[2] * cy + d[3] * c2;
                const double pt = c.t[0] + c.t[1] * cx + c.t[2] * cy + c.t[3] * c2;
                const double vh = c.mt0 + c.kq * qd * (c.l2 * (px * px + py * py) - 4.0) + pe + vn * pd + vt * pt;
                const double vb = vh + c.kb * qd + c.e[4] + vn * d[4] + vt * c.t[4];
                const double wn = gw[g] * vn;
                fh[r] += wn * (q * vh + c.mt3 * f0h - c.mt4 * ph);
                fb[r] += wn * (c.ckh * q * vb + c.mt3 * f0b - c.mt4 * pb);
                asm volatile("" ::: "memory");   // the node's scalars are read again: held across the velocities they spilled
                const int k = k0 + r * (int)blockDim.x;
                const double pm = c.m[0] + c.m[1] * cx + c.m[2] * cy + c.m[3] * c2;
                moment_add(k < nv ? B.w[k] : 0.0, uk[r], vk[r], q * pm, c.ckh * q * (pm + c.m[4]), mt);
            }
            const double t = warp_halving<4, false>(mt);
            if ((tid & 7) == 0) s_time[tid >> 5][4 * g + ((tid & 31) >> 3)] += t;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = k0 + r * (int)blockDim.x;
            if (k < nv) {
                fh[r] = fh[r] * len;
                fb[r] = fb[r] * len;
                Fh[k] = fh[r];
                Fb[k] = fb[r];
                moment_add(B.w[k], uk[r], vk[r], fh[r], fb[r], acc);
                if (!(isfinite(fh[r]) && isfinite(fb[r]))) bad = 1;
            }
        }
    }
    block_reduce_smem<4, 0>(acc, red, rout);
    if (tid < 12) {   // the time directions' gate, as in k_s2_face_flux
        const double* wt = fs + (tid >> 2) * kS2FScal + 40;
        double t = s_time[0][tid];
        for (int w = 1; w < (int)blockDim.x / 32; ++w) t += s_time[w][tid];
        const double scl = fmax(fmax(fmax(fabs(wt[0]), fabs(wt[1])), fmax(fabs(wt[2]), fabs(wt[3]))), 1.0);
        if (!(fabs(t - wt[tid & 3]) / scl <= 2.0e-12)) bad = 1;
    }
    bad = __syncthreads_or(bad);
    if (tid < 4) Fw[tid] = rout[tid];
    if (tid == 0 && bad) set_status(B.status, ST_NONFINITE_FLUX);
}

// wall face nodes (s2w2_wall_node, mod_S2MultiscaleWall.f90:45-184): one warp per (wall face,
// Gauss node); bottom faces of row 0, then top faces of row ny-1.  Node fluxes go to the node
// buffers after the interior faces.
__global__ void __launch_bounds__(256, 2) k_s2_wall_nodes(LoParams P, LoBuffers B, S2Buffers SB, int qrec) {
    if (eval_cached(B)) return;
    extern __shared__ double s_qrec[];
    const int nv = P.nvel, nx = P.nx, ny = P.ny, ck = P.ck, lane = threadIdx.x & 31, nr = (nv + 31) >> 5;
    const int nf = nx * ny + nx * (ny - 1);
    const int wid = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (wid >= 2 * nx * 3) return;
    const int wf = wid / 3, g = wid % 3;
    const int top = wf >= nx ? 1 : 0, i = wf - top * nx;
    const int cc = top ? (ny - 1) * nx + i : i;
    const size_t node = (size_t)(nf + wf) * 3 + g;
    const double side = top ? 1.0 : -1.0;
    const double ux = P.wall_ux[top], theta = 0.5 / P.wall_lam[top];
    const double dt = B.dt[0];
    const double* wcell = B.W + cc * 4;
    const double pp = (2.0 / (double)(ck + 2)) * (wcell[3] - 0.5 * (wcell[1] * wcell[1] + wcell[2] * wcell[2]) / wcell[0]);
    const double lambda = 0.5 / theta;
    const double prim_g[4] = {pp / theta, 0.0, -ux, lambda};
    const double wc[4] = {wcell[0], wcell[2], -wcell[1], wcell[3]};
    const double wg[4] = {prim_g[0], 0.0, -prim_g[0] * ux, prim_g[0] * ((double)(ck + 2) / (4.0 * lambda) + 0.5 * ux * ux)};
    // wall_equilibrium: the discrete closure of the wall state
    const double wwall[4] = {prim_g[0], prim_g[0] * ux, 0.0, prim_g[0] * ((double)(ck + 2) * theta / 2.0 + ux * ux / 2.0)};
    __shared__ double s_jac[8][16];
    WClosure C;
    C.jac = s_jac[threadIdx.x >> 5];
    const WQRec qr{qrec ? s_qrec + (threadIdx.x >> 5) * (nr * 32) : nullptr};
    bool ok = pp > 0.0 && isfinite(pp) && w_closure(P, B, wwall, C, qr);
    auto rec = [&](const WVel& s, int field) {
        return SB.rec[rec_wall(nx, ny, top, i, field, g, nv) + s.k];
    };
    double acc[8];
    double an[4], at[4], atime[4], mt[5], mxi2 = 0.0, coeff = 0.0, hlx = 0.0, hly = 0.0, tau_wall = 0.0;
    if (ok) {
#pragma unroll
        for (int m = 0; m < 6; ++m) acc[m] = 0.0;
        for (int r = 0; r < nr; ++r) {
            const WVel s = wvel(B, nv, r);
            const double hin = rec(s, 0), bin = rec(s, 1), ht = rec(s, 3), bt = rec(s, 5);
            const double vn = s.v, vt = -s.u, v2 = vn * vn + vt * vt;
            acc[0] += s.w * (-ht);
            acc[1] += s.w * (-(vn * ht));
            acc[2] += s.w * (-(vt * ht));
            acc[3] += s.w * (-(0.5 * (v2 * ht + bt)));
            const double vt2 = -s.u + ux, w2 = vn * vn + vt2 * vt2;
            acc[4] += 0.5 * s.w * vn * (w2 * hin + bin);
            acc[5] += 0.5 * s.w * vt2 * (w2 * hin + bin);
        }
        warp_sum_all<6>(acc);
        double sw[4], sw_t[4], Mu[7], Mv[6], Mxi[3], m1[4], m2[4];
        for (int m = 0; m < 4; ++m) { sw[m] = (wg[m] - wc[m]) / (side * 0.5 * P.dy); sw_t[m] = acc[m]; }
        s2w_micro_slope(ck, prim_g, sw, an);
        s2w_micro_slope(ck, prim_g, sw_t, at);
        s2w_moments(ck, prim_g, Mu, Mv, Mxi);
        s2w_auvxi(an, Mu, Mv, Mxi, 1, 0, m1);
        s2w_auvxi(at, Mu, Mv, Mxi, 0, 1, m2);
        for (int m = 0; m < 4; ++m) sw[m] = -prim_g[0] * (m1[m] + m2[m]);
        s2w_micro_slope(ck, prim_g, sw, atime);
        const double wgg[4] = {wg[0], -wg[2], wg[1], wg[3]};
        ok = s2_tau(P, wgg, tau_wall);
        s2w_time_coeffs(dt, tau_wall, mt);
        coeff = P.pr != 1.0 ? 0.8 * (1.0 - P.pr) * lambda * lambda / prim_g[0] : 0.0;
        mxi2 = Mxi[2];
        hlx = acc[4];
        hly = acc[5];
    }
    // the incident micro flux g_in and the reflected wall Maxwellian of one velocity
    const S2Th tt = s2_th(C.th, ck);
    auto gin = [&](const WVel& s, int r, double& ginh, double& ginb, double& wallh, double& wallb, double& mh,
                   double& mb, double& corrh, double& corrb) {
        const S2Q q = qr.at(tt, s, r);
        mh = q.qh;
        mb = q.qb;
        wallh = mh / prim_g[0];
        wallb = mb / prim_g[0];
        corrh = 0.0;
        corrb = 0.0;
        if (P.pr != 1.0) {
            const double vn = s.v, vt = -s.u + ux, v2 = vn * vn + vt * vt;
            const double qdot = vn * hlx + vt * hly, shh = 2.0 * lambda * v2 - 4.0;
            corrh = coeff * qdot * shh * mh;
            corrb = coeff * qdot * (shh + 2.0 / (double)ck) * mb;
        }
        const double vn = s.v, vt = -s.u, v2 = vn * vn + vt * vt;
        const double Han = (an[0] + an[1] * vn + an[2] * vt) * mh + 0.5 * an[3] * (v2 * mh + mb);
        const double Hatan = (at[0] + at[1] * vn + at[2] * vt) * mh + 0.5 * at[3] * (v2 * mh + mb);
        const double Hatime = (atime[0] + atime[1] * vn + atime[2] * vt) * mh + 0.5 * atime[3] * (v2 * mh + mb);
        const double Ban = (an[0] + an[1] * vn + an[2] * vt) * mb + 0.5 * an[3] * (v2 * mb + mxi2 * mh);
        const double Batan = (at[0] + at[1] * vn + at[2] * vt) * mb + 0.5 * at[3] * (v2 * mb + mxi2 * mh);
        const double Batime = (atime[0] + atime[1] * vn + atime[2] * vt) * mb + 0.5 * atime[3] * (v2 * mb + mxi2 * mh);
        ginh = mt[0] * mh + mt[1] * (vn * Han + vt * Hatan) + mt[2] * Hatime + mt[3] * rec(s, 0) -
               mt[4] * (vn * rec(s, 2) + s.u * rec(s, 3));
        ginb = mt[0] * mb + mt[1] * (vn * Ban + vt * Batan) + mt[2] * Batime + mt[3] * rec(s, 1) -
               mt[4] * (vn * rec(s, 4) + s.u * rec(s, 5));
        ginh = ginh + mt[0] * corrh;
        ginb = ginb + mt[0] * corrb;
    };
    double inc = 0.0, rhow = 0.0;
    if (ok) {   // incidence and reflection -> wall density
        acc[0] = acc[1] = 0.0;
        for (int r = 0; r < nr; ++r) {
            const WVel s = wvel(B, nv, r);
            double ginh, ginb, wallh, wallb, mh, mb, ch, cb;
            gin(s, r, ginh, ginb, wallh, wallb, mh, mb, ch, cb);
            if (side * s.v > 0.0) acc[0] += s.w * s.v * ginh;
            else acc[1] += dt * s.w * s.v * wallh;
        }
        warp_sum_all<2>(acc);
        inc = acc[0];
        const double refl = acc[1];
        rhow = -inc / refl;
        ok = isfinite(refl) && fabs(refl) > DBL_MIN && isfinite(rhow) && rhow > 0.0;
    }
    if (ok) {
        double* outh = SB.node + node * 2 * nv;
        double* outb = outh + nv;
#pragma unroll
        for (int m = 0; m < 4; ++m) acc[m] = 0.0;
        for (int r = 0; r < nr; ++r) {
            const WVel s = wvel(B, nv, r);
            double ginh, ginb, wallh, wallb, mh, mb, ch, cb, fh, fb;
            gin(s, r, ginh, ginb, wallh, wallb, mh, mb, ch, cb);
            if (side * s.v > 0.0) { fh = s.v * ginh; fb = s.v * ginb; }
            else { fh = dt * s.v * rhow * wallh; fb = dt * s.v * rhow * wallb; }
            acc[0] += s.w * fh; acc[1] += s.w * (s.u * fh); acc[2] += s.w * (s.v * fh);
            acc[3] += s.w * (0.5 * ((s.u * s.u + s.v * s.v) * fh + fb));
            if (s.ok) {
                outh[s.k] = fh;
                outb[s.k] = fb;
                ok = ok && isfinite(fh) && isfinite(fb);
            }
        }
        warp_sum_all<4>(acc);
        ok = ok && isfinite(acc[0]) && fabs(acc[0]) <= 2.0e-12 * fmax(1.0, fabs(inc));
        if (lane < 4) SB.nodew[node * 4 + lane] = lane == 0 ? acc[0] : (lane == 1 ? acc[1] : (lane == 2 ? acc[2] : acc[3]));
    }
    ok = __all_sync(0xffffffffu, ok);
    if (ok && SB.coef) {   // the optional f0_h, f0_b, k_h, k_b outputs (mod_S2MultiscaleWall.f90:155-177)
        auto qk = [&](const WVel& s, double m, double corr, int fv, int fn, int ft) {
            return (m + corr - rec(s, fv)) / tau_wall - s.v * rec(s, fn) - s.u * rec(s, ft);
        };
        acc[0] = acc[1] = acc[2] = 0.0;
        for (int r = 0; r < nr; ++r) {
            const WVel s = wvel(B, nv, r);
            double ginh, ginb, wallh, wallb, mh, mb, ch, cb;
            gin(s, r, ginh, ginb, wallh, wallb, mh, mb, ch, cb);
            if (side * s.v > 0.0) {
                acc[0] += s.w * s.v * rec(s, 0);
                acc[1] += s.w * s.v * qk(s, mh, ch, 0, 2, 3);
            } else {
                acc[2] += s.w * s.v * wallh;
            }
        }
        warp_sum_all<3>(acc);
        const double r0 = -acc[0] / acc[2], r1 = -acc[1] / acc[2];
        ok = isfinite(r0) && isfinite(r1) && r0 > 0.0;
        double* cf = SB.coef + node * 4 * nv;
        acc[0] = acc[1] = 0.0;
        for (int r = 0; r < nr && ok; ++r) {
            const WVel s = wvel(B, nv, r);
            double ginh, ginb, wallh, wallb, mh, mb, ch, cb, c0, c1, c2, c3;
            gin(s, r, ginh, ginb, wallh, wallb, mh, mb, ch, cb);
            if (side * s.v > 0.0) {
                c0 = s.v * rec(s, 0);
                c1 = s.v * rec(s, 1);
                c2 = s.v * qk(s, mh, ch, 0, 2, 3);
                c3 = s.v * qk(s, mb, cb, 1, 4, 5);
            } else {
                c0 = s.v * r0 * wallh;
                c1 = s.v * r0 * wallb;
                c2 = s.v * r1 * wallh;
                c3 = s.v * r1 * wallb;
            }
            acc[0] += s.w * c0;
            acc[1] += s.w * c2;
            if (s.ok) {
                cf[s.k] = c0;
                cf[(size_t)nv + s.k] = c1;
                cf[2 * (size_t)nv + s.k] = c2;
                cf[3 * (size_t)nv + s.k] = c3;
            }
        }
        if (ok) {
            warp_sum_all<2>(acc);
            ok = fabs(acc[0]) <= 2.0e-12 && fabs(acc[1]) <= 2.0e-12;
        }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) set_status(B.status, ST_NONFINITE_FLUX);
}

// The multiscale wall on a tensor-product velocity table: one CTA per wall face, its three Gauss nodes at once.
// The nodes share the wall state, so one closure (warp 0, by 1-D sums) serves them while the other warps
// sum the incident state's moments; three lanes then form the nodes' slopes, and each velocity's
// incident flux is taken once, kept in registers until the wall density is known, and summed over the nodes
// into the face arrays (no node flux is stored; nodew keeps the nodes' macro fluxes).  16 CTAs at nx = 8, beside
// the interior faces on the side stream: bound by the chain closure -> slopes -> two block reductions (50 us at 8x64x32^2,
// 136 us for k_s2_wall_nodes, one warp a node; ncu, cold).  254 registers a thread keep an SM to itself, which costs a batch, whose
// other instances hid the walls, 0.6 %.  Above 1024 velocities 512 threads with 5 each spill 776 / 916 bytes a thread,
// in 2 nx CTAs.
struct S2WallC {
    double n[4], t[4], m[4], hx, hy;   // normal, tangential, time slopes (half of the energy slope last); heat of the incident state
};
template <int VPT, int NT>
__global__ void __launch_bounds__(NT) k_s2_walls_t(LoParams P, LoBuffers B, S2Buffers SB, int rows) {
    if (eval_cached(B)) return;
    __shared__ double red[(NT / 32) * 32], rout[kRedSlots];
    __shared__ double ex[64], ey[64], s_jac[4][17], s_th[4];
    __shared__ S2WallC sc[3];
    __shared__ double s_mt[5];
    __shared__ int s_ok;
    const int nv = P.nvel, nu = P.tnu, nw = P.tnv, nx = P.nx, ny = P.ny, ck = P.ck, tid = threadIdx.x;
    const int wf = blockIdx.x, top = wf >= nx ? 1 : 0, i = wf - top * nx, cc = top ? (ny - 1) * nx + i : i;
    const double side = top ? 1.0 : -1.0, ux = P.wall_ux[top], theta = 0.5 / P.wall_lam[top], dt = B.dt[0];
    const double* wcell = B.W + cc * 4;
    const double pp = (2.0 / (double)(ck + 2)) * (wcell[3] - 0.5 * (wcell[1] * wcell[1] + wcell[2] * wcell[2]) / wcell[0]);
    const double lambda = 0.5 / theta, rho = pp / theta;
    const double* rec = SB.rec + rec_wall(nx, ny, top, i, 0, 0, nv);   // [field][node][nvel]
    auto at = [&](int field, int g, int k) { return rec[((size_t)field * 3 + g) * nv + k]; };
    if (tid < 32) {   // wall_equilibrium: the discrete closure of the wall state
        const double wwall[4] = {rho, rho * ux, 0.0, rho * ((double)(ck + 2) * theta / 2.0 + ux * ux / 2.0)};
        TClosure C;
        C.jac = s_jac[tid / kTG];
        bool ok;
        switch (rows) {
            case 3: ok = t_closure<3>(P, B, wwall, true, C); break;
            case 4: ok = t_closure<4>(P, B, wwall, true, C); break;
            case 6: ok = t_closure<6>(P, B, wwall, true, C); break;
            default: ok = t_closure<8>(P, B, wwall, true, C); break;
        }
        if (tid == 0) {
            s_ok = ok && pp > 0.0 && isfinite(pp);
#pragma unroll
            for (int m = 0; m < 4; ++m) s_th[m] = C.th[m];
        }
    } else {   // the tangential slope's moments and the heat of the incident state, per node
        double a[18];
#pragma unroll
        for (int m = 0; m < 18; ++m) a[m] = 0.0;
        for (int k = tid - 32; k < nv; k += NT - 32) {
            const double wk = B.w[k], vn = B.v[k], vt = -B.u[k], v2 = vn * vn + vt * vt, vt2 = vt + ux, w2 = vn * vn + vt2 * vt2;
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                const double ht = wk * at(3, g, k), q = 0.5 * wk * (w2 * at(0, g, k) + at(1, g, k));
                a[6 * g] -= ht;
                a[6 * g + 1] -= vn * ht;
                a[6 * g + 2] -= vt * ht;
                a[6 * g + 3] -= 0.5 * (v2 * ht + wk * at(5, g, k));
                a[6 * g + 4] += vn * q;
                a[6 * g + 5] += vt2 * q;
            }
        }
        red[(tid >> 5) * 32 + (tid & 31)] = warp_halving<18, false>(a);   // lane m: the warp's total of sum m
    }
    __syncthreads();
    if (tid < 3) {   // the slopes of node tid and the time coefficients
        const double prim_g[4] = {rho, 0.0, -ux, lambda};
        const double wc[4] = {wcell[0], wcell[2], -wcell[1], wcell[3]};
        const double wg[4] = {rho, 0.0, -rho * ux, rho * ((double)(ck + 2) / (4.0 * lambda) + 0.5 * ux * ux)};
        double a[6], sw[4], an[4], atn[4], am[4], Mu[7], Mv[6], Mxi[3], m1[4], m2[4], mt[5], tau = 1.0;
        for (int m = 0; m < 6; ++m) {
            a[m] = 0.0;
            for (int w = 1; w < NT / 32; ++w) a[m] += red[w * 32 + 6 * tid + m];
        }
        for (int m = 0; m < 4; ++m) sw[m] = (wg[m] - wc[m]) / (side * 0.5 * P.dy);
        s2w_micro_slope(ck, prim_g, sw, an);
        s2w_micro_slope(ck, prim_g, a, atn);
        s2w_moments(ck, prim_g, Mu, Mv, Mxi);
        s2w_auvxi(an, Mu, Mv, Mxi, 1, 0, m1);
        s2w_auvxi(atn, Mu, Mv, Mxi, 0, 1, m2);
        for (int m = 0; m < 4; ++m) sw[m] = -rho * (m1[m] + m2[m]);
        s2w_micro_slope(ck, prim_g, sw, am);
        const double wgg[4] = {wg[0], -wg[2], wg[1], wg[3]};
        const bool ok = s2_tau(P, wgg, tau);
        s2w_time_coeffs(dt, tau, mt);
        S2WallC& c = sc[tid];
        for (int m = 0; m < 4; ++m) { const double f = m < 3 ? 1.0 : 0.5; c.n[m] = f * an[m]; c.t[m] = f * atn[m]; c.m[m] = f * am[m]; }
        c.hx = a[4];
        c.hy = a[5];
        if (tid == 0) {
            for (int m = 0; m < 5; ++m) s_mt[m] = mt[m];
            if (!ok) s_ok = 0;
        }
    }
    const S2Th t = s2_th(s_th, ck);
    for (int q = tid - 32; q >= 0 && q < nu + nw; q += NT - 32) {
        const double d = q < nu ? B.tab[q] - t.u : B.tab[128 + q - nu] - t.v;
        const double e = exp(-(d * d) * t.itw);
        if (q < nu) ex[q] = t.pref * e;
        else ey[q - nu] = e;
    }
    __syncthreads();
    if (!s_ok) {
        if (tid == 0) set_status(B.status, ST_NONFINITE_FLUX);
        return;
    }
    const double coeff = P.pr != 1.0 ? 0.8 * (1.0 - P.pr) * lambda * lambda / rho : 0.0;
    const double mxi2 = (double)ck * ((double)ck + 2.0) / (4.0 * (lambda * lambda)), c2ck = 2.0 / (double)ck, irho = 1.0 / rho;
    const double mt0 = s_mt[0], mt1 = s_mt[1], mt2 = s_mt[2], mt3 = s_mt[3], mt4 = s_mt[4];
    double fh[3][VPT], fb[3][VPT], acc[12];   // toward the wall: v times the incident flux; away: dt v times the unit wall Maxwellian
#pragma unroll
    for (int m = 0; m < 6; ++m) acc[m] = 0.0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const int k = s.kk, jv = k / nu;
        const double u = B.u[k], v = B.v[k], wk = s.ok ? B.w[k] : 0.0, mh = ex[k - jv * nu] * ey[jv], mb = t.ckh * mh;
        const bool toward = side * v > 0.0;
        const double vn = v, vt = -u, v2 = vn * vn + vt * vt, vt2 = vt + ux, sh = 2.0 * lambda * (vn * vn + vt2 * vt2) - 4.0;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const S2WallC& c = sc[g];
            const double qd = coeff * (vn * c.hx + vt2 * c.hy);
            const double ln = c.n[0] + c.n[1] * vn + c.n[2] * vt + c.n[3] * v2, lt = c.t[0] + c.t[1] * vn + c.t[2] * vt + c.t[3] * v2;
            const double lm = c.m[0] + c.m[1] * vn + c.m[2] * vt + c.m[3] * v2;
            const double L = mt1 * (vn * ln + vt * lt) + mt2 * lm, E = mt1 * (vn * c.n[3] + vt * c.t[3]) + mt2 * c.m[3];
            const double gh = mh * (mt0 * (1.0 + qd * sh) + L + t.ckh * E) + mt3 * at(0, g, k) - mt4 * (vn * at(2, g, k) + u * at(3, g, k));
            const double gb = mh * (t.ckh * (mt0 * (1.0 + qd * (sh + c2ck)) + L) + mxi2 * E) + mt3 * at(1, g, k) -
                              mt4 * (vn * at(4, g, k) + u * at(5, g, k));
            fh[g][r] = toward ? v * gh : dt * v * (mh * irho);
            fb[g][r] = toward ? v * gb : dt * v * (mb * irho);
            acc[2 * g] += toward ? wk * fh[g][r] : 0.0;
            acc[2 * g + 1] += toward ? 0.0 : wk * fh[g][r];
        }
    }
    block_reduce<6, 0>(acc, red, rout);   // incidence and reflection of the nodes -> wall densities
    double rw[3], inc[3];
    bool ok = true;
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        inc[g] = acc[2 * g];
        const double refl = acc[2 * g + 1];
        rw[g] = -inc[g] / refl;
        ok = ok && isfinite(refl) && fabs(refl) > DBL_MIN && isfinite(rw[g]) && rw[g] > 0.0;
    }
    const double gw[3] = {5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0};
    const size_t o = top ? (size_t)ny * nx + i : (size_t)i;
#pragma unroll
    for (int m = 0; m < 12; ++m) acc[m] = 0.0;
#pragma unroll
    for (int r = 0; r < VPT; ++r) {
        const Slot s = slot(r, nv);
        const double u = B.u[s.kk], v = B.v[s.kk], wk = s.ok ? B.w[s.kk] : 0.0;
        const bool toward = side * v > 0.0;
        double ah = 0.0, ab = 0.0;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const double f = toward ? 1.0 : rw[g], h = f * fh[g][r], b = f * fb[g][r];
            moment_add(wk, u, v, h, b, acc + 4 * g);
            ah += gw[g] * h;
            ab += gw[g] * b;
        }
        if (s.ok) {
            B.fyh[o * nv + s.k] = ah * P.dx;
            B.fyb[o * nv + s.k] = ab * P.dx;
            ok = ok && isfinite(ah) && isfinite(ab);
        }
    }
    block_reduce_smem<12, 0>(acc, red, rout);
    const int bad = __syncthreads_or(!ok);
    if (tid == 0) {
        bool fine = !bad;
        double rate[4] = {0.0, 0.0, 0.0, 0.0};
        const size_t node = (size_t)(nx * ny + nx * (ny - 1) + wf) * 3;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const double mass = rout[4 * g];
            fine = fine && isfinite(mass) && fabs(mass) <= 2.0e-12 * fmax(1.0, fabs(inc[g]));
#pragma unroll
            for (int m = 0; m < 4; ++m) { SB.nodew[(node + g) * 4 + m] = rout[4 * g + m]; rate[m] += gw[g] * rout[4 * g + m]; }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            B.fyw[o * 4 + m] = rate[m] * P.dx;
            if (SB.wall_raw != nullptr) SB.wall_raw[(size_t)wf * 4 + m] = rate[m];
            rate[m] = rate[m] / dt;
        }
        // PublishWallDiagnostics (mod_S2NativeAdapter.f90:1075-1097): native frame n = +y, t = -x; the heat removes
        // the moving wall's mechanical work
        double* a = B.wall_aero + (size_t)wf * 3;
        a[0] = rate[2];
        a[1] = -rate[1];
        a[2] = rate[3] - ux * rate[1];
        if (!fine) set_status(B.status, ST_NONFINITE_FLUX);
    }
}

// Gauss-weighted sum of the node fluxes of every face (interior, then the walls) times the face
// length, into the face arrays ComputeResidual reads; the walls' macro fluxes also unscaled into
// SB.wall_raw, and the walls' (pnn, pnt, qn) into B.wall_aero.  One thread per (face, velocity);
// threads k < 4 also do the macro flux.
__global__ void __launch_bounds__(256) k_s2_combine(LoParams P, LoBuffers B, S2Buffers SB, int f0) {
    if (eval_cached(B)) return;
    const int nv = P.nvel, nx = P.nx, ny = P.ny, nfx = nx * ny, nf = nfx + nx * (ny - 1);
    const int fi = f0 + (int)blockIdx.y;
    const int k = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= nv) return;
    const double gw[3] = {5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0};
    size_t o;
    double len, *Fh, *Fb, *Fw;
    int wall = -1;
    if (fi < nfx) {
        const int i = fi % nx, j = fi / nx;
        o = (size_t)j * nx + (i + 1) % nx; len = P.dy; Fh = B.fxh; Fb = B.fxb; Fw = B.fxw;
    } else if (fi < nf) {
        const int f = fi - nfx, i = f % nx, j = f / nx;
        o = (size_t)(j + 1) * nx + i; len = P.dx; Fh = B.fyh; Fb = B.fyb; Fw = B.fyw;
    } else {
        wall = fi - nf;
        const int top = wall >= nx ? 1 : 0, i = wall - top * nx;
        o = top ? (size_t)ny * nx + i : (size_t)i; len = P.dx; Fh = B.fyh; Fb = B.fyb; Fw = B.fyw;
    }
    const double* nd = SB.node + (size_t)fi * 3 * 2 * nv;
    double afh = 0.0, afb = 0.0;
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        afh = afh + gw[g] * nd[(size_t)(2 * g) * nv + k];
        afb = afb + gw[g] * nd[(size_t)(2 * g + 1) * nv + k];
    }
    Fh[o * nv + k] = afh * len;
    Fb[o * nv + k] = afb * len;
    if (k < 4) {
        double afw = 0.0;
#pragma unroll
        for (int g = 0; g < 3; ++g) afw = afw + gw[g] * SB.nodew[((size_t)fi * 3 + g) * 4 + k];
        Fw[o * 4 + k] = afw * len;
        if (wall >= 0 && SB.wall_raw != nullptr) SB.wall_raw[(size_t)wall * 4 + k] = afw;
    }
    if (wall >= 0 && k == 0) {   // PublishWallDiagnostics (mod_S2NativeAdapter.f90:1075-1097)
        const int top = wall >= nx ? 1 : 0;
        const double measure = B.dt[0] * len;
        double rate[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            double afw = 0.0;
#pragma unroll
            for (int g = 0; g < 3; ++g) afw = afw + gw[g] * SB.nodew[((size_t)fi * 3 + g) * 4 + m];
            rate[m] = afw * len / measure;
        }
        // native frame n = +y, t = -x; the heat removes the moving wall's mechanical work
        double* a = B.wall_aero + (size_t)wall * 3;
        a[0] = rate[2];
        a[1] = -rate[1];
        a[2] = rate[3] - P.wall_ux[top] * rate[1];
    }
}


// Shared memory for the closure kernels' Maxwellian records (WQRec): one record of the velocity set
// per warp, used when it fits these caps.  The caps keep the kernels' resident CTAs per SM: three
// 128-thread face-node CTAs (up to 2304 = 48^2 velocities), two 256-thread target- and face-node CTAs
// (up to 1760 velocities).  The wall-node kernel has only 6 nx warps: one CTA per SM will do.
constexpr int kQRecCap128x3 = 72 * 1024, kQRecCap256x2 = 110 * 1024, kQRecCapWall = 200 * 1024;

cudaError_t prepare_s2() {
    cudaError_t e = s2_upload_tables();
    const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_s2_face_nodes<kS2NodeThreads, 3>, dyn, kQRecCap128x3);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_s2_face_nodes<256, 2>, dyn, kQRecCap256x2);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_s2_target_nodes, dyn, kQRecCap256x2);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_s2_wall_nodes, dyn, kQRecCapWall);
    return e;
}

// bytes of the Maxwellian records of a CTA of `threads` threads, 0 (no records) above `cap`.  Many
// instances on concurrent streams (S2Buffers::concurrent) take none: their kernels share SMs with other
// instances' kernels, and the records' shared-memory carve-out cost the batch more than it saved it
// (7.47e8 -> 7.44e8 updates/s for the 256-instance distribution, same GPU); the values are the same
// either way.
static int qrec_bytes(const S2Buffers& S, int nv, int threads, int cap) {
    const long long b = (long long)(threads / 32) * ((nv + 31) / 32) * 32 * (long long)sizeof(double);
    return !S.concurrent && b <= cap ? (int)b : 0;
}


// which 0: the S2 cold start; 1: the S2 Evolution of one pseudo-step (targets, reconstruction,
// faces, walls); 2: the Evolution with the targets kept (S2CN2); 3: the targets of B.W only; 5: their node scalars alone
cudaError_t s2_enqueue(int which, const LoParams& P, const LoBuffers& B, const S2Buffers& S, cudaStream_t s,
                       cudaStream_t s2, cudaEvent_t fork, cudaEvent_t join) {
    const int nx = P.nx, ny = P.ny, nv = P.nvel, nc = nx * ny, nf = nx * ny + nx * (ny - 1);
    auto warps = [](long long n) { return (unsigned)((n * 32 + 255) / 256); };
    auto node_ctas = [](long long n) { return (unsigned)((n * 32 + kS2NodeThreads - 1) / kS2NodeThreads); };
    if (which == 0) {
        k_s2_init<<<warps(nc), 256, 0, s>>>(P, B, S);
        return cudaGetLastError();
    }
    if (which == 4) {
        return launch_recon(P, B, S, s);
    }
    const int faces = which < 3, targets = which != 2;
    const long long nmacw = (faces ? (long long)nf * 2 : 0) + (targets ? (long long)nc : 0);   // warps
    // The macro pass feeds the targets and the face nodes, the reconstruction neither of them: with an evolution it runs on
    // the side stream beside the reconstruction (9 us), followed there by the targets of which 1 (first read after the face
    // arrays) and, after the reconstruction, the wall nodes; which 3 and 5: everything on the main stream
    cudaStream_t ts = faces ? s2 : s;
    cudaError_t e = cudaSuccess;
    if (faces) {
        e = cudaEventRecord(fork, s);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s2, fork, 0);
    }
    if (e == cudaSuccess) {
        k_s2_macro<<<(unsigned)((nmacw * 32 + 127) / 128), 128, 0, ts>>>(P, B, S, faces, targets);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && faces) e = cudaEventRecord(join, s2);
    if (e == cudaSuccess && targets) {
        if (P.tnu > 0) {
            const unsigned g = (unsigned)((nc * 9 * kTG + 127) / 128);
            const int n = P.tnu > P.tnv ? P.tnu : P.tnv;
            if (n <= 24) k_s2_target_nodes_t<3><<<g, 128, 0, ts>>>(P, B, S);
            else if (n <= 32) k_s2_target_nodes_t<4><<<g, 128, 0, ts>>>(P, B, S);
            else if (n <= 48) k_s2_target_nodes_t<6><<<g, 128, 0, ts>>>(P, B, S);
            else k_s2_target_nodes_t<8><<<g, 128, 0, ts>>>(P, B, S);
            const int nt = std::min(256, (nv + 127) / 128 * 32);
            if (which != 5) k_s2_target_sum_t<<<(unsigned)nc, nt, 0, ts>>>(P, B, S);
            e = cudaGetLastError();
        } else {
            const int qb = qrec_bytes(S, nv, 256, kQRecCap256x2);
            k_s2_target_nodes<<<warps((long long)nc * 9), 256, qb, ts>>>(P, B, S, qb > 0);
            e = cudaGetLastError();
            if (e == cudaSuccess) {
                k_s2_target_sum<<<dim3((unsigned)((nv + 255) / 256), (unsigned)nc), 256, 0, ts>>>(P, B, S);
                e = cudaGetLastError();
            }
        }
    }
    if (e != cudaSuccess || !faces) return e;
    // a tensor table's faces and walls: the fused fluxes, unless a wall variant wants the nodes' fluxes and coefficients
    const bool tensor = P.tnu > 0, fused = tensor && S.coef == nullptr;
    e = launch_recon(P, B, S, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, join, 0);   // the macro pass
    if (e == cudaSuccess) e = cudaEventRecord(fork, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s2, fork, 0);
    if (e == cudaSuccess) {
        if (P.s2_kinetic) e = launch_s2_w1_walls(P, B, S, s2);
        else if (fused) {
            const int n = P.tnu > P.tnv ? P.tnu : P.tnv, rows = n <= 24 ? 3 : n <= 32 ? 4 : n <= 48 ? 6 : 8;
            if (nv <= 1024) k_s2_walls_t<4, 256><<<2 * nx, 256, 0, s2>>>(P, B, S, rows);
            else k_s2_walls_t<5, 512><<<2 * nx, 512, 0, s2>>>(P, B, S, rows);
            e = cudaGetLastError();
        } else {
            const int qb = qrec_bytes(S, nv, 256, kQRecCapWall);
            k_s2_wall_nodes<<<warps(2LL * nx * 3), 256, qb, s2>>>(P, B, S, qb > 0);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaEventRecord(join, s2);
    if (e == cudaSuccess && tensor) {
        const unsigned g = (unsigned)((nf * 3 * kTG + 127) / 128);
        const int n = P.tnu > P.tnv ? P.tnu : P.tnv;
        k_s2_face_moments<<<(unsigned)nf, 128, 0, s>>>(P, B, S);
        if (n <= 24) k_s2_face_nodes_t<3><<<g, 128, 0, s>>>(P, B, S);
        else if (n <= 32) k_s2_face_nodes_t<4><<<g, 128, 0, s>>>(P, B, S);
        else if (n <= 48) k_s2_face_nodes_t<6><<<g, 128, 0, s>>>(P, B, S);
        else k_s2_face_nodes_t<8><<<g, 128, 0, s>>>(P, B, S);
        if (fused) k_s2_face_flux_t<<<(unsigned)nf, std::min(256, (nv + 127) / 128 * 32), 0, s>>>(P, B, S);
        e = cudaGetLastError();
    } else if (e == cudaSuccess) {
        if (S.concurrent) {
            const int qb = qrec_bytes(S, nv, 256, kQRecCap256x2);
            k_s2_face_nodes<256, 2><<<warps((long long)nf * 3), 256, qb, s>>>(P, B, S, qb > 0);
        } else {
            const int qb = qrec_bytes(S, nv, kS2NodeThreads, kQRecCap128x3);
            k_s2_face_nodes<kS2NodeThreads, 3><<<node_ctas((long long)nf * 3), kS2NodeThreads, qb, s>>>(P, B, S, qb > 0);
        }
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && !fused) {
        if (nv <= 1024) k_s2_face_flux<4><<<(unsigned)(nf * 3), 256, 0, s>>>(P, B, S);
        else k_s2_face_flux<10><<<(unsigned)(nf * 3), 256, 0, s>>>(P, B, S);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, join, 0);
    // the node fluxes that were stored: all faces', or a kinetic wall's alone
    if (e == cudaSuccess && !fused) e = launch_s2_combine(P, B, S, 0, nf + 2 * nx, s);
    else if (e == cudaSuccess && P.s2_kinetic) e = launch_s2_combine(P, B, S, nf, 2 * nx, s);
    return e;
}

cudaError_t launch_s2_combine(const LoParams& P, const LoBuffers& B, const S2Buffers& S, int f0, int nfaces,
                              cudaStream_t s) {
    k_s2_combine<<<dim3((unsigned)((P.nvel + 255) / 256), (unsigned)nfaces), 256, 0, s>>>(P, B, S, f0);
    return cudaGetLastError();
}

}  // namespace ugks

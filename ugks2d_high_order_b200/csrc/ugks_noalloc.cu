// ugks_noalloc.cu -- an Explicit-step entry point that allocates no memory at all.
//
// Who needs it: host codes that manage every byte of device memory themselves (a Fortran or
// C driver with its own pre-sized device pool, or an application running under a memory cap
// where a later cudaMalloc may fail) and latency-critical loops where cudaMalloc/cudaFree would
// implicitly synchronise the device.  Such callers cannot create a ugks_ctx, because
// ugks_ctx_create allocates the working arrays.  This entry point takes the caller's own device
// arrays for the inputs and outputs and keeps all of its working arrays (Van-Leer slopes, face
// fluxes, per-cell reductions, the status word) in one file-scope __device__ array of fixed size.
//
// Limits and behaviour (also stated in include/ugks_b200.h):
//   * The scratch array is kNoAllocBytes = 36 MiB.  A call whose working set does not fit is
//     rejected with UGKS_EINVAL before any GPU work; the reference's delivered case (8x64 cells,
//     32x32 velocities) needs 33.8 MB.  The array belongs to this file's device module.  Under
//     CUDA's lazy module loading (the default) that module, and with it the 36 MiB, is loaded on a
//     device at the first call there, so a caller that sizes its own device pool or runs under a
//     memory cap makes one call on each device before it does so.  The array then stays until the
//     process exits.
//   * The first call on a device looks the array's device address up (cudaGetSymbolAddress) with
//     that device current.
//   * Every call synchronises its stream twice: once after scanning the velocity table (U_MAX / V_MAX set the
//     time step, its structure the kernels) and once after reading the status and the outputs.  The
//     call therefore cannot be captured in a CUDA graph.
//   * Every call uses the same array and it keeps the previous call's contents; this call clears
//     what must start at zero (the last-CTA counter and the status word).  Calls that overlap on
//     the GPU (other streams, other host threads driving the same device) race on the array and
//     must be serialised by the caller.  Host threads that drive different devices use different
//     arrays and share no host state.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "../../include/ugks_b200.h"
#include "ugks_lo.cuh"

namespace ugks {
cudaError_t launch_lo_slopes(const LoParams& P, const LoBuffers& B, cudaStream_t s);
cudaError_t launch_lo_faces(const LoParams& P, const LoBuffers& B, cudaStream_t s);
cudaError_t launch_lo_walls(const LoParams& P, const LoBuffers& B, cudaStream_t s);
cudaError_t launch_lo_cells(const LoParams& P, const LoBuffers& B, int mode, bool collision, cudaStream_t s);
cudaError_t launch_lo_timestep(const LoParams& P, const LoBuffers& B, cudaStream_t s);
cudaError_t launch_lo_fluxes_t(const LoParams& P, const LoBuffers& B, cudaStream_t s);
cudaError_t launch_lo_cells_t(const LoParams& P, const LoBuffers& B, int mode, cudaStream_t s);
}  // namespace ugks

using namespace ugks;

namespace {

constexpr size_t kNoAllocBytes = (size_t)36 << 20;
constexpr size_t kNoAllocDoubles = kNoAllocBytes / sizeof(double);
constexpr int kMaxDevices = 64;

// The scratch.  Host code must not use this name as an address: in host code it names a
// host-side shadow, so only the address returned by cudaGetSymbolAddress is passed to kernels.
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];
// the axes of a tensor-product velocity table (LoBuffers::tab), beside the working set, whose limit stays as it was
static __device__ __align__(256) double g_noalloc_tab[kTensorTab];

// Device address of the scratch per device, filled on the first call on that device.  Every lookup of
// one device yields the same address, so two host threads filling one entry at once store the same
// value; the entries are atomic so that such a store is well defined.
std::atomic<double*> g_scratch_addr[kMaxDevices];

struct Plan {
    size_t flags, dt, dg, scan, sxh, syh, sxb, syb, fxh, fxb, fxw, fyh, fyb, fyw, dtl, cd, wa, total;
};

Plan plan_for(int nx, int ny, int nv) {
    Plan p{};
    size_t off = 0;
    auto take = [&](size_t n) { size_t o = off; off += (n + 31) / 32 * 32; return o; };   // 256-byte aligned
    const size_t nc = (size_t)nx * ny, S = nc * nv, SY = (size_t)(ny + 1) * nx * nv;
    p.flags = take(4); p.dt = take(2); p.dg = take(kNDiag);   // read back together
    p.scan = 0;   // the table scan's result, in the words the steps then use: read before they start
    p.sxh = take(S); p.syh = take(S); p.sxb = take(S); p.syb = take(S);
    p.fxh = take(S); p.fxb = take(S); p.fxw = take(nc * 4);
    p.fyh = take(SY); p.fyb = take(SY); p.fyw = take((size_t)(ny + 1) * nx * 4);
    p.dtl = take(nc); p.cd = take(nc * kNDiag);
    p.wa = take((size_t)2 * nx * 3);
    p.total = off;
    return p;
}

// One CTA over the velocity table: U_MAX and V_MAX (InitVelocityFromStructuredFile, mod_InitializeFlow.f90:508), and
// whether it is a tensor product, by tensor_table's rule and arithmetic: then out[2], out[3] are its abscissae per axis and
// tab its axes.  One launch and one small copy instead of two copies of the table.
constexpr int kScanThreads = 256;
__global__ void __launch_bounds__(kScanThreads) k_table_scan(const double* u, const double* v, const double* w, int nv, double* out,
                                                             double* tab) {
    __shared__ double mx[2][kScanThreads / 32], fx[64], fy[64];
    __shared__ int s_nu, s_bad;
    const int tid = threadIdx.x;
    if (tid == 0) { s_nu = nv; s_bad = 0; }
    __syncthreads();
    double m[2] = {-INFINITY, -INFINITY};
    for (int k = tid; k < nv; k += kScanThreads) {
        m[0] = fmax(m[0], u[k]);
        m[1] = fmax(m[1], v[k]);
        if (k > 0 && !(v[k] == v[0])) atomicMin(&s_nu, k);   // (v[0] itself may compare unequal: not a number)
    }
    warp_max_all<2>(m);
    if ((tid & 31) == 0) { mx[0][tid >> 5] = m[0]; mx[1][tid >> 5] = m[1]; }
    __syncthreads();
    const int nu = s_nu, nj = nv / nu;
    bool ok = nv % nu == 0 && nu >= 2 && nj >= 2 && nu <= 64 && nj <= 64;
    if (ok) {   // uniform over the CTA
        for (int k = tid; k < nv; k += kScanThreads) {
            const int i = k % nu;
            if (!(u[k] == u[i] && v[k] == v[k - i] && w[k] > 0.0 && isfinite(w[k]) && isfinite(u[k]) && isfinite(v[k]))) s_bad = 1;
        }
        if (tid < nj) fy[tid] = w[tid * nu] / w[0];
        for (int it = 0; it < 2; ++it) {
            __syncthreads();
            if (tid < nu) fx[tid] = tensor_factor(w + tid, nj, nu, fy);
            __syncthreads();
            if (tid < nj) fy[tid] = tensor_factor(w + tid * nu, nu, 1, fx);
        }
        __syncthreads();
        for (int k = tid; k < nv; k += kScanThreads)
            if (!tensor_weight(fx[k % nu], fy[k / nu], w[k])) s_bad = 1;
        if (tid < 64) {
            const double xu = u[min(tid, nu - 1)], xv = v[min(tid, nj - 1) * nu], a = tid < nu ? fx[tid] : 0.0, b = tid < nj ? fy[tid] : 0.0;
            tab[tid] = xu; tab[64 + tid] = a; tab[128 + tid] = xv; tab[192 + tid] = b;
            tab[256 + tid] = xu >= 0.0 ? a : 0.0; tab[320 + tid] = xu >= 0.0 ? 0.0 : a;
            tab[384 + tid] = xv >= 0.0 ? b : 0.0; tab[448 + tid] = xv >= 0.0 ? 0.0 : b;
        }
        __syncthreads();
        ok = s_bad == 0;
    }
    if (tid == 0) {
        for (int t = 1; t < kScanThreads / 32; ++t) { mx[0][0] = fmax(mx[0][0], mx[0][t]); mx[1][0] = fmax(mx[1][0], mx[1][t]); }
        out[0] = mx[0][0];
        out[1] = mx[1][0];
        out[2] = ok ? (double)nu : 0.0;
        out[3] = ok ? (double)nj : 0.0;
    }
}

int fail(cudaError_t e) {
    std::fprintf(stderr, "ugks_step_explicit_noalloc: CUDA error %s\n", cudaGetErrorString(e));
    return UGKS_ECUDA;
}

}  // namespace

extern "C" int ugks_step_explicit_noalloc(const ugks_params* prm, const double* u, const double* v, const double* w,
                                          double* h, double* b, double* W, int nsteps, void* stream,
                                          double* dt_out, double* res_out) {
    if (!prm || !u || !v || !w || !h || !b || !W || nsteps < 0) return UGKS_EINVAL;
    if (prm->method != UGKS_METHOD_EXPLICIT) return UGKS_EUNSUPPORTED;
    const int nx = prm->nx, ny = prm->ny, nv = prm->nvel;
    if (nx < 1 || ny < 3 || nv < 1 || nv > kMaxVel || !(prm->dx > 0) || !(prm->dy > 0) || prm->ck < 1)
        return UGKS_EINVAL;
    const Plan pl = plan_for(nx, ny, nv);
    if (pl.total > kNoAllocDoubles) {
        std::fprintf(stderr,
                     "ugks_step_explicit_noalloc: %dx%d cells x %d velocities need %zu bytes of scratch, "
                     "more than the fixed %zu-byte array\n",
                     nx, ny, nv, pl.total * sizeof(double), kNoAllocBytes);
        return UGKS_EINVAL;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(e);
    if (dev < 0 || dev >= kMaxDevices) return UGKS_EINVAL;
    double* base = g_scratch_addr[dev].load(std::memory_order_acquire);
    if (!base) {   // once per device, with that device current
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e != cudaSuccess) return fail(e);
        base = static_cast<double*>(ptr);
        g_scratch_addr[dev].store(base, std::memory_order_release);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    // U_MAX, V_MAX of the table and its axes when it is a tensor product; the host reads four numbers
    void* tab = nullptr;
    e = cudaGetSymbolAddress(&tab, g_noalloc_tab);
    if (e != cudaSuccess) return fail(e);
    k_table_scan<<<1, kScanThreads, 0, s>>>(u, v, w, nv, base + pl.scan, static_cast<double*>(tab));
    double scan[4];
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(scan, base + pl.scan, sizeof scan, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(e);
    LoParams P = make_lo_params(*prm, scan[0], scan[1]);
    P.tnu = (int)scan[2];
    P.tnv = (int)scan[3];

    LoBuffers B{};
    B.u = u; B.v = v; B.w = w; B.tab = static_cast<double*>(tab); B.h = h; B.b = b; B.W = W;
    B.sxh = base + pl.sxh; B.syh = base + pl.syh; B.sxb = base + pl.sxb; B.syb = base + pl.syb;
    B.fxh = base + pl.fxh; B.fxb = base + pl.fxb; B.fxw = base + pl.fxw;
    B.fyh = base + pl.fyh; B.fyb = base + pl.fyb; B.fyw = base + pl.fyw;
    B.dtl = base + pl.dtl; B.dt = base + pl.dt; B.cell_diag = base + pl.cd; B.diag = base + pl.dg;
    B.wall_aero = base + pl.wa;
    B.counter = reinterpret_cast<unsigned*>(base + pl.flags);
    B.status = B.counter + 1;
    // the fused explicit step reads no residual cache and no collision arrays
    B.res_w = B.res_h = B.res_b = nullptr;
    B.peq_h = B.peq_b = B.pcol_h = B.pcol_b = nullptr;

    // the counter and the status word must start at zero; the previous call left its values
    e = cudaMemsetAsync(base + pl.flags, 0, 4 * sizeof(double), s);
    if (e == cudaSuccess) e = launch_lo_timestep(P, B, s);
    for (int k = 0; k < nsteps && e == cudaSuccess; ++k) {
        if (P.tnu > 0) {
            e = launch_lo_fluxes_t(P, B, s);
            if (e == cudaSuccess) e = launch_lo_cells_t(P, B, 3, s);
            continue;
        }
        e = launch_lo_slopes(P, B, s);
        if (e == cudaSuccess) e = launch_lo_faces(P, B, s);
        if (e == cudaSuccess) e = launch_lo_walls(P, B, s);
        if (e == cudaSuccess) e = launch_lo_cells(P, B, 3, false, s);
    }
    if (e != cudaSuccess) return fail(e);
    double back[96];   // status word, dt and norms, one copy
    static_assert(kNDiag <= 32, "flags, dt and dg are the scratch's first three blocks of 32 doubles");
    e = cudaMemcpyAsync(back, base + pl.flags, sizeof back, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(e);
    unsigned words[2];
    std::memcpy(words, back, sizeof words);
    const unsigned status = words[1];
    const double *dt2 = back + (pl.dt - pl.flags), *dg = back + (pl.dg - pl.flags);
    if (dt_out) *dt_out = nsteps > 0 ? dt2[1] : dt2[0];
    if (res_out && nsteps > 0) finish_explicit_res(nx, ny, dg, res_out);
    return status ? UGKS_ENUMERIC : UGKS_OK;
}

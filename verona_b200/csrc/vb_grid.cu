// Grid-level entry points that mirror the reference's kernels one at a time,
// on caller-owned device arrays in the reference layout (FP64 AoS, variable
// fastest, padded extents n+6 on the active axes). They are the fine-grained
// seam for a caller that replaces single kernels of HARM_HLL; the time loop
// itself is the fused vb_step. FP64, built with -fmad=false: bit-identical to
// the oracle's k_fluxes / k_update / k_utop / k_ptou / k_limit.
//   vb_grid_fluxes     function_Fluxes of one axis, src/3dim/algos.jl:14-176
//                      (2D: src/2dim/algos.jl:11-168)
//   vb_grid_update     function_Update, src/3dim/algos.jl:178-200
//   vb_grid_con2prim   function_UtoP, src/3dim/structs.jl:218-628
//                      (2D: src/2dim/structs.jl:249-330; 1D: src/1dim/structs.jl:78-105)
//   vb_grid_prim2con   kernel_PtoU, src/3dim/structs.jl:66-81
//   vb_grid_limit      function_Limit, src/3dim/algos.jl:5-12
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/verona_b200.h"
#include "vb_aos.cuh"
#include "vb_con2prim.cuh"
#include "vb_internal.h"

namespace vb {

struct GridAoS {
    int dims, nv;
    int np[3];  // padded extents (1 on inactive axes)
    long long st[3];
    long long ncell;
};

static inline bool grid_aos(int dims, int nx, int ny, int nz, GridAoS& g) {
    if (dims < 1 || dims > 3 || nx < 1 || (dims > 1 && ny < 1) || (dims > 2 && nz < 1)) return false;
    g.dims = dims;
    g.nv = 2 + dims;
    const int n[3] = {nx, ny, nz};
    for (int a = 0; a < 3; ++a) g.np[a] = a < dims ? n[a] + 2 * NG : 1;
    g.st[0] = 1;
    g.st[1] = g.np[0];
    g.st[2] = (long long)g.np[0] * g.np[1];
    g.ncell = (long long)g.np[0] * g.np[1] * g.np[2];
    return true;
}

// a / b, a >= 0: the 64-bit division, an emulated sequence, only where a needs it
__device__ __forceinline__ long long quo(long long a, int b) {
    return a <= 0xFFFFFFFFll ? (long long)((uint32_t)a / (uint32_t)b) : a / b;
}

__device__ __forceinline__ void cell_ijk(const GridAoS& g, long long c, int& i, int& j, int& k) {
    const long long row = quo(c, g.np[0]), pl = quo(row, g.np[1]);
    i = (int)(c - row * g.np[0]);
    j = (int)(row - pl * g.np[1]);
    k = (int)pl;
}

// true if (i, j, k) lies in [lo, np - hi) on every active axis
__device__ __forceinline__ bool in_range(const GridAoS& g, int i, int j, int k, int lo, int hi) {
    const int x[3] = {i, j, k};
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (a < g.dims) ok = ok && x[a] >= lo && x[a] < g.np[a] - hi;
    return ok;
}

// Fluxes along one axis: faces i + 1/2 for every index in [2, n - 4] on all
// active axes. Each cell is reconstructed once, not once per adjoining face.
//
// Axis x: a warp takes 32 consecutive cells of a row (31 faces); the state right
// of a face is the next lane's.
template <int DIM, int REC, int RS>
__global__ void __launch_bounds__(256) k_grid_fluxes_x(GridAoS g, const double* __restrict__ P, double gamma, double fl,
                                                       double* __restrict__ F) {
    constexpr int NV = 2 + DIM;
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
    const int n0 = g.np[0], segs = (n0 - 5 + 30) / 31;  // faces 2 .. n0 - 4
    const int r1 = DIM > 1 ? g.np[1] - 5 : 1, r2 = DIM > 2 ? g.np[2] - 5 : 1;
    const long long tot = (long long)segs * r1 * r2;
    for (long long w = warp; w < tot; w += nwarp) {
        const long long row = quo(w, segs), pl = quo(row, r1);
        const int i = 2 + 31 * (int)(w - row * segs) + lane;
        const int j = DIM > 1 ? 2 + (int)(row - pl * r1) : 0, k = DIM > 2 ? 2 + (int)pl : 0;
        const int ic = min(i, n0 - 3);  // lanes past the row reconstruct its last cell
        const long long c = ic + (long long)j * g.st[1] + (long long)k * g.st[2];
        const double* q = P + NV * c;
        double qr[NV], ql[NV], PR[NV], Fo[NV];
        recon_n<REC, NV, double>([&](int v, int o) { return q[NV * o + v]; }, qr, ql);
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            qr[v] = jmax(fl, qr[v]);
            ql[v] = jmax(fl, ql[v]);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) PR[v] = __shfl_down_sync(0xffffffffu, qr[v], 1);
        if (lane < 31 && i <= n0 - 4) {
            face_flux<DIM, RS>(0, gamma, ql, PR, Fo);
#pragma unroll
            for (int v = 0; v < NV; ++v) F[NV * c + v] = Fo[v];
        }
    }
}
// Axes y, z: a thread marches a run of faces of one column, lanes along x; the
// state left of the next face stays in its registers. The stencil's cells are
// read again at each face, from L1: kept in registers (50 of them for five
// variables) they left 8 warps per SM.
template <int DIM, int REC, int RS>
__global__ void __launch_bounds__(128, 4) k_grid_fluxes_m(GridAoS g, const double* __restrict__ P, double gamma,
                                                          double fl, int d, int run, double* __restrict__ F) {
    constexpr int NV = 2 + DIM;
    const int nd = d == 1 ? g.np[1] : g.np[2], no = DIM < 3 ? 1 : (d == 1 ? g.np[2] : g.np[1]) - 5;
    const long long sd = NV * (d == 1 ? g.st[1] : g.st[2]), so = d == 1 ? g.st[2] : g.st[1];
    const int nx = g.np[0] - 5, runs = (nd - 5 + run - 1) / run;
    const long long tot = (long long)nx * no * runs;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
        const long long a = quo(t, nx), b = quo(a, no);
        const int i = 2 + (int)(t - a * nx), o = (int)(a - b * no), f0 = 2 + (int)b * run;
        const int f1 = min(f0 + run, nd - 3);  // faces f0 .. f1 - 1
        const long long base = NV * (i + (DIM < 3 ? 0 : (2 + o) * so));
        double qr[NV], ql[NV], PL[NV], Fo[NV];
        auto cell = [&](const double* q) {
            recon_n<REC, NV, double>([&](int v, int m) { return q[m * sd + v]; }, qr, ql);
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                qr[v] = jmax(fl, qr[v]);
                ql[v] = jmax(fl, ql[v]);
            }
        };
        const double* q = P + base + f0 * sd;
        double* out = F + base + f0 * sd;
        cell(q);
#pragma unroll 1
        for (int f = f0; f < f1; ++f) {
#pragma unroll
            for (int v = 0; v < NV; ++v) PL[v] = ql[v];
            q += sd;
            cell(q);
            face_flux<DIM, RS>(d, gamma, PL, qr, Fo);
#pragma unroll
            for (int v = 0; v < NV; ++v) out[v] = Fo[v];
            out += sd;
        }
    }
}

// Per value, not per cell: consecutive threads take consecutive doubles of a row.
// c: dt / dx_d (the reference's (dt / dx) * difference)
template <int DIM>
__global__ void __launch_bounds__(256) k_grid_update(GridAoS g, const double* __restrict__ U,
                                                     const double* __restrict__ Fx, const double* __restrict__ Fy,
                                                     const double* __restrict__ Fz, double cx, double cy, double cz,
                                                     double* __restrict__ Uo) {
    constexpr int NV = 2 + DIM;
    const int nrow = NV * (g.np[0] - 6), r1 = DIM > 1 ? g.np[1] - 6 : 1, r2 = DIM > 2 ? g.np[2] - 6 : 1;
    const long long rows = (long long)r1 * r2;
    for (long long row = blockIdx.y; row < rows; row += gridDim.y) {
        const long long pl = quo(row, r1), j = DIM > 1 ? 3 + row - pl * r1 : 0, k = DIM > 2 ? 3 + pl : 0;
        const long long base = NV * (3 + j * g.st[1] + k * g.st[2]);
        for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < nrow; x += gridDim.x * blockDim.x) {
            const long long e = base + x;
            double r = U[e];
            r = r - cx * (Fx[e] - Fx[e - NV]);
            if (DIM > 1) r = r - cy * (Fy[e] - Fy[e - NV * g.st[1]]);
            if (DIM > 2) r = r - cz * (Fz[e] - Fz[e - NV * g.st[2]]);
            Uo[e] = r;
        }
    }
}

// NT cells of the padded array per CTA, through shared memory; interior cells solved
constexpr int GC_NT = 128;
template <int DIM>
__global__ void __launch_bounds__(GC_NT, DIM == 2 ? 6 : 8) k_grid_con2prim(GridAoS g, const double* __restrict__ U,
                                                                          double gamma, int n_iter, double tol,
                                                                          double* __restrict__ P,
                                                                          unsigned long long* failures) {
    constexpr int NV = 2 + DIM;
    __shared__ double sU[NV * GC_NT], sP[NV * GC_NT];
    __shared__ unsigned char inside[GC_NT];
    unsigned long long nf = 0;
    for (long long c0 = (long long)blockIdx.x * GC_NT; c0 < g.ncell; c0 += (long long)gridDim.x * GC_NT) {
        const int n = (int)min((long long)GC_NT, g.ncell - c0), t = threadIdx.x;
        int i, j, k;
        cell_ijk(g, c0 + t, i, j, k);
        const bool in = t < n && in_range(g, i, j, k, 3, 3);
        if (!__syncthreads_or(in)) continue;
        inside[t] = in;
        aos_in<NV, GC_NT>(U, c0, n, sU);
        aos_in<NV, GC_NT>(P, c0, n, sP);
        __syncthreads();
        if (in) {
            double u[NV], p[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                u[v] = sU[t * NV + v];
                p[v] = sP[t * NV + v];
            }
            int r;
            if (DIM == 1)
                r = c2p_1d(gamma, n_iter, tol, u, p);
            else if (DIM == 2)
                r = c2p_2d(gamma, n_iter, tol, u, p);
            else
                r = c2p_3d(gamma, n_iter, tol, u, p);
            nf += (r < 0);
#pragma unroll
            for (int v = 0; v < NV; ++v) sP[t * NV + v] = p[v];
        }
        __syncthreads();
        for (int e = t; e < n * NV; e += GC_NT)
            if (inside[e / NV]) P[c0 * NV + e] = sP[e];
        __syncthreads();
    }
    if (failures && nf) atomicAdd(failures, nf);
}

constexpr int GP_NT = 256;
template <int DIM>
__global__ void __launch_bounds__(GP_NT) k_grid_prim2con(GridAoS g, const double* __restrict__ P, double gamma,
                                                         double* __restrict__ U) {
    constexpr int NV = 2 + DIM;
    __shared__ double s[NV * GP_NT];
    for (long long c0 = (long long)blockIdx.x * GP_NT; c0 < g.ncell; c0 += (long long)gridDim.x * GP_NT) {
        const int n = (int)min((long long)GP_NT, g.ncell - c0);
        aos_in<NV, GP_NT>(P, c0, n, s);
        __syncthreads();
        double p[NV], u[NV];
        if ((int)threadIdx.x < n) {
#pragma unroll
            for (int v = 0; v < NV; ++v) p[v] = s[threadIdx.x * NV + v];
            prim2con<DIM>(gamma, p, u);
#pragma unroll
            for (int v = 0; v < NV; ++v) s[threadIdx.x * NV + v] = u[v];
        }
        __syncthreads();
        aos_out<NV, GP_NT>(U, c0, n, s);
        __syncthreads();
    }
}

__global__ void k_grid_limit(GridAoS g, double* __restrict__ P, double fl) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < g.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        P[g.nv * c + 0] = jmax(P[g.nv * c + 0], fl);
        P[g.nv * c + 1] = jmax(P[g.nv * c + 1], fl);
    }
}

static int blocks_for(long long n) {
    long long b = (n + 255) / 256;
    return (int)(b < 148 * 32 ? (b > 0 ? b : 1) : 148 * 32);
}

}  // namespace vb

using namespace vb;

static thread_local std::string g_grid_err;

static int gfail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_grid_err = buf;
    return code;
}

static int gdone(const char* what) {
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VB_OK : gfail(VB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

// faces per marching run: short enough that the runs fill the GPU (148 SMs at 512
// threads), long enough that the one extra reconstruction of each is small
static int march_run(long long columns, int faces) {
    const long long want = (148LL * 512 + columns - 1) / columns;  // runs per column
    const long long run = (faces + want - 1) / want;
    return (int)(run < 4 ? 4 : run);
}

template <int DIM, int REC, int RS>
static void launch_fluxes_t(const GridAoS& g, const double* P, double gamma, double fl, int axis, double* F,
                            cudaStream_t s) {
    const long long nx = g.np[0] - 5;
    if (axis == 0) {
        const long long rows = (DIM > 1 ? g.np[1] - 5 : 1) * (long long)(DIM > 2 ? g.np[2] - 5 : 1);
        const int nb = blocks_for(rows * ((nx + 30) / 31) * 32);
        k_grid_fluxes_x<DIM, REC, RS><<<nb, 256, 0, s>>>(g, P, gamma, fl, F);
    } else if constexpr (DIM > 1) {
        const int faces = g.np[axis] - 5;
        const long long cols = nx * (DIM > 2 ? g.np[3 - axis] - 5 : 1);
        const int run = march_run(cols, faces);
        const int nb = blocks_for(2 * cols * ((faces + run - 1) / run));  // blocks of 128
        k_grid_fluxes_m<DIM, REC, RS><<<nb, 128, 0, s>>>(g, P, gamma, fl, axis, run, F);
    }
}
template <int DIM>
static void launch_fluxes(const GridAoS& g, int rec, int rs, const double* P, double gamma, double fl, int axis,
                          double* F, cudaStream_t s) {
#define VB_GF(RC, RSC) \
    if (rec == RC && rs == RSC) return launch_fluxes_t<DIM, RC, RSC>(g, P, gamma, fl, axis, F, s);
    VB_GF(REC_MINMOD, RS_HLL)
    VB_GF(REC_MINMOD, RS_HLLC)
    VB_GF(REC_PPM, RS_HLL)
    VB_GF(REC_PPM, RS_HLLC)
    VB_GF(REC_WENOZ, RS_HLL)
    VB_GF(REC_WENOZ, RS_HLLC)
#undef VB_GF
}

extern "C" {

const char* vb_grid_last_error(void) { return g_grid_err.c_str(); }

int vb_grid_fluxes(int dims, int nx, int ny, int nz, const double* P_aos, double gamma, double floor_, int axis,
                   int recon, int riemann, double* F_aos, void* stream) {
    GridAoS g;
    if (!grid_aos(dims, nx, ny, nz, g)) return gfail(VB_ERR_ARG, "vb_grid_fluxes: dims %d size %d %d %d", dims, nx, ny, nz);
    if (!P_aos || !F_aos) return gfail(VB_ERR_ARG, "vb_grid_fluxes: null array");
    if (axis < 0 || axis >= dims) return gfail(VB_ERR_ARG, "vb_grid_fluxes: axis %d of a %dD grid", axis, dims);
    if (recon < VB_RECON_MINMOD || recon > VB_RECON_WENOZ || (riemann != VB_RIEMANN_HLL && riemann != VB_RIEMANN_HLLC))
        return gfail(VB_ERR_ARG, "vb_grid_fluxes: recon %d riemann %d", recon, riemann);
    cudaStream_t s = (cudaStream_t)stream;
    if (dims == 1) launch_fluxes<1>(g, recon, riemann, P_aos, gamma, floor_, axis, F_aos, s);
    else if (dims == 2) launch_fluxes<2>(g, recon, riemann, P_aos, gamma, floor_, axis, F_aos, s);
    else launch_fluxes<3>(g, recon, riemann, P_aos, gamma, floor_, axis, F_aos, s);
    return gdone("vb_grid_fluxes");
}

int vb_grid_update(int dims, int nx, int ny, int nz, const double* U_aos, const double* Fx, const double* Fy,
                   const double* Fz, double dt, double dx, double dy, double dz, double* Uout_aos, void* stream) {
    GridAoS g;
    if (!grid_aos(dims, nx, ny, nz, g)) return gfail(VB_ERR_ARG, "vb_grid_update: dims %d size %d %d %d", dims, nx, ny, nz);
    if (!U_aos || !Uout_aos || !Fx || (dims > 1 && !Fy) || (dims > 2 && !Fz))
        return gfail(VB_ERR_ARG, "vb_grid_update: null array");
    cudaStream_t s = (cudaStream_t)stream;
    const int nrow = g.nv * nx;
    const long long rows = (dims > 1 ? ny : 1) * (long long)(dims > 2 ? nz : 1);
    const dim3 nb((nrow + 255) / 256, (unsigned)(rows < 65535 ? rows : 65535));
    const double cx = dt / dx, cy = dims > 1 ? dt / dy : 0.0, cz = dims > 2 ? dt / dz : 0.0;
    if (dims == 1) k_grid_update<1><<<nb, 256, 0, s>>>(g, U_aos, Fx, Fy, Fz, cx, cy, cz, Uout_aos);
    else if (dims == 2) k_grid_update<2><<<nb, 256, 0, s>>>(g, U_aos, Fx, Fy, Fz, cx, cy, cz, Uout_aos);
    else k_grid_update<3><<<nb, 256, 0, s>>>(g, U_aos, Fx, Fy, Fz, cx, cy, cz, Uout_aos);
    return gdone("vb_grid_update");
}

int vb_grid_con2prim(int dims, int nx, int ny, int nz, const double* U_aos, double gamma, int n_iter, double tol,
                     double* P_aos, uint64_t* failures_dev, void* stream) {
    GridAoS g;
    if (!grid_aos(dims, nx, ny, nz, g)) return gfail(VB_ERR_ARG, "vb_grid_con2prim: dims %d size %d %d %d", dims, nx, ny, nz);
    if (!U_aos || !P_aos || n_iter < 1) return gfail(VB_ERR_ARG, "vb_grid_con2prim: null array or n_iter %d", n_iter);
    cudaStream_t s = (cudaStream_t)stream;
    const int nb = blocks_for(2 * g.ncell);
    unsigned long long* f = reinterpret_cast<unsigned long long*>(failures_dev);
    if (dims == 1) k_grid_con2prim<1><<<nb, GC_NT, 0, s>>>(g, U_aos, gamma, n_iter, tol, P_aos, f);
    else if (dims == 2) k_grid_con2prim<2><<<nb, GC_NT, 0, s>>>(g, U_aos, gamma, n_iter, tol, P_aos, f);
    else k_grid_con2prim<3><<<nb, GC_NT, 0, s>>>(g, U_aos, gamma, n_iter, tol, P_aos, f);
    return gdone("vb_grid_con2prim");
}

int vb_grid_prim2con(int dims, int nx, int ny, int nz, const double* P_aos, double gamma, double* U_aos,
                     void* stream) {
    GridAoS g;
    if (!grid_aos(dims, nx, ny, nz, g)) return gfail(VB_ERR_ARG, "vb_grid_prim2con: dims %d size %d %d %d", dims, nx, ny, nz);
    if (!P_aos || !U_aos) return gfail(VB_ERR_ARG, "vb_grid_prim2con: null array");
    cudaStream_t s = (cudaStream_t)stream;
    const int nb = blocks_for(g.ncell);
    if (dims == 1) k_grid_prim2con<1><<<nb, 256, 0, s>>>(g, P_aos, gamma, U_aos);
    else if (dims == 2) k_grid_prim2con<2><<<nb, 256, 0, s>>>(g, P_aos, gamma, U_aos);
    else k_grid_prim2con<3><<<nb, 256, 0, s>>>(g, P_aos, gamma, U_aos);
    return gdone("vb_grid_prim2con");
}

int vb_grid_limit(int dims, int nx, int ny, int nz, double* P_aos, double floor_, void* stream) {
    GridAoS g;
    if (!grid_aos(dims, nx, ny, nz, g)) return gfail(VB_ERR_ARG, "vb_grid_limit: dims %d size %d %d %d", dims, nx, ny, nz);
    if (!P_aos) return gfail(VB_ERR_ARG, "vb_grid_limit: null array");
    k_grid_limit<<<blocks_for(g.ncell), 256, 0, (cudaStream_t)stream>>>(g, P_aos, floor_);
    return gdone("vb_grid_limit");
}

}  // extern "C"

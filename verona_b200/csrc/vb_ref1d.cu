// The reference's 1D solver, Verona1D.HARM_HLL (src/1dim/algos.jl:58-315),
// FP64, as one thread-block cluster that runs every step of a call: the N cells
// are divided among the cluster's CTAs, each of which does a whole RK stage of
// its cells (reconstruction, HLL, update, con2prim) from shared memory, and the
// cluster meets once per stage, so a whole shock-tube run is a single launch.
//
// What bounds it is the serial FP64 chain of a stage, and on one SM its FP64
// rate too: one CTA of 1024 threads, with block barriers between the phases and
// the arrays in global memory, took 26.5 us a step at N = 1024; 16 CTAs of 64
// cells take 8.9 us. Neighbours exchange P through L2 (stores, then the
// cluster barrier's release and acquire, then loads past L1).
//
// The reference keeps state between stages that this kernel keeps too: the
// face arrays PL/PR start as copies of P and are only refreshed on the ranges
// the Julia loops write (src/1dim/algos.jl:91-117), so the edge faces keep
// their t = 0 values; cells 1, N-1, N (1-based) of U are never updated.
// Compiled with -fmad=false: bit-identical to the oracle restatement.
#include <algorithm>

#include "vb_cluster.cuh"
#include "vb_con2prim.cuh"
#include "vb_internal.h"

namespace vb {

constexpr int R1_MAXT = 480;     // threads per CTA: cells of a tile + 2 (46 KB of shared memory)

__device__ __forceinline__ void ref1d_cons(double g, double p1, double p2, double p3, double* U) {
    double gamma = sqrt(sq(p3) + 1.0);
    double pressure = (g - 1.0) * p2;
    U[0] = p1 * gamma;
    U[1] = -(p2 + pressure + p1) * sq(gamma) + pressure;
    U[2] = (p2 + pressure + p1) * gamma * p3;
}

__device__ __forceinline__ void ref1d_flux(double g, double p1, double p2, double p3, double* F) {
    double gamma = sqrt(sq(p3) + 1.0);
    double pressure = (g - 1.0) * p2;
    F[0] = p1 * p3;
    F[1] = -(p2 + pressure + p1) * gamma * p3;
    F[2] = pressure + (p2 + pressure + p1) * sq(p3);
}

// HLL flux of one face, the expressions of the Julia loop (:233-282)
static __device__ __noinline__ void ref1d_hll_general(double g, const double* pl, const double* pr, double* F) {
    double UL[3], UR[3], FL[3], FR[3];
    ref1d_cons(g, pr[0], pr[1], pr[2], UR);
    ref1d_flux(g, pr[0], pr[1], pr[2], FR);
    ref1d_cons(g, pl[0], pl[1], pl[2], UL);
    ref1d_flux(g, pl[0], pl[1], pl[2], FL);
    double vL = pl[2] / sqrt(sq(pl[2]) + 1.0);
    double vR = pr[2] / sqrt(sq(pr[2]) + 1.0);
    double CL = sound_speed(pl[0], pl[1], g);
    double CR = sound_speed(pr[0], pr[1], g);
    double sL = sq(CL) / ((sq(pl[2]) + 1.0) * (1.0 - sq(CL)));
    double sR = sq(CR) / ((sq(pr[2]) + 1.0) * (1.0 - sq(CR)));
    double Cmax = jmax((vL + sqrt(sL * (1.0 - sq(vL) + sL))) / (1.0 + sL),
                       (vR + sqrt(sR * (1.0 - sq(vR) + sR))) / (1.0 + sR));
    double Cmin = -jmin((vL - sqrt(sL * (1.0 - sq(vL) + sL))) / (1.0 + sL),
                        (vR - sqrt(sR * (1.0 - sq(vR) + sR))) / (1.0 + sR));
    for (int v = 0; v < 3; ++v) {
        if (Cmax < 0)
            F[v] = FR[v];
        else if (Cmin < 0)
            F[v] = FL[v];
        else
            F[v] = (FR[v] * Cmin + FL[v] * Cmax - Cmax * Cmin * (UR[v] - UL[v])) / (Cmax + Cmin);
    }
}

// the same on the branch-free divide and square root (vb_fp64.cuh, with the
// range test of the grid kernels' faces)
struct Ref1DSide {
    double U[3], F[3], lp, lm;
    __device__ __forceinline__ bool make(double g, const double* p) {
        const double gamma = d64::root(sq(p[2]) + 1.0);
        const double pressure = (g - 1.0) * p[1];
        const double w = p[1] + pressure + p[0];
        U[0] = p[0] * gamma;
        U[1] = -w * sq(gamma) + pressure;
        U[2] = w * gamma * p[2];
        F[0] = p[0] * p[2];
        F[1] = -w * gamma * p[2];
        F[2] = pressure + w * sq(p[2]);
        const double v = d64::quot_s(p[2], d64::divisor(gamma));
        const double C = d64::root(d64::quot((g * (g - 1.0) * p[1]), d64::divisor(p[0] + g * p[1])));
        const double c1 = 1.0 - sq(C);
        const double s = d64::quot(sq(C), d64::divisor((sq(p[2]) + 1.0) * c1));
        const double r2 = s * (1.0 - sq(v) + s);
        const double r = d64::root(r2);
        const d64::Div is = d64::divisor(1.0 + s);
        lp = d64::quot_s(v + r, is);
        lm = d64::quot_s(v - r, is);
        return face_in_range<1>(p) && d64::pos_in<-60, 60>(c1) && d64::pos_in<-900, 900>(r2);
    }
};
__device__ __forceinline__ void ref1d_hll(double g, const double* pl, const double* pr, double* F) {
    Ref1DSide L, R;
    bool ok = R.make(g, pr);
    ok &= L.make(g, pl);
    const double Cmax = jmax(L.lp, R.lp), Cmin = -jmin(L.lm, R.lm), sum = Cmax + Cmin;
    const d64::Div is = d64::divisor(sum);
    const bool use_R = Cmax < 0, use_L = !use_R && Cmin < 0;
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        const double h = d64::quot_s(R.F[v] * Cmin + L.F[v] * Cmax - Cmax * Cmin * (R.U[v] - L.U[v]), is);
        F[v] = use_R ? R.F[v] : (use_L ? L.F[v] : h);
    }
    if (!(ok && (use_R || use_L || d64::pos_in<-300, 300>(sum)))) {
        const double l[3] = {pl[0], pl[1], pl[2]}, r[3] = {pr[0], pr[1], pr[2]};
        double f[3];
        ref1d_hll_general(g, l, r, f);
#pragma unroll
        for (int v = 0; v < 3; ++v) F[v] = f[v];
    }
}

// One RK stage of cells [a, b): face states and fluxes of P (faces a-1 .. b-1),
// Uo = Ub - coef dF on the cells the reference updates, then Pout = con2prim(Uo)
// on every cell from the guess G (P at the start of the step).
template <int REC>
__device__ void ref1d_stage(const Ref1DState& st, int a, int b, const double* P, const double* Ub, double* Uo,
                            const double* G, double* Pout, double coef, double g, int n_iter, double tol) {
    __shared__ double sP[3][R1_MAXT + 4], sL[3][R1_MAXT], sR[3][R1_MAXT], sF[3][R1_MAXT];
    const int N = st.N, tid = threadIdx.x, T = blockDim.x;
    const int reach = REC == REC_MINMOD ? 1 : 2;  // cells reach .. N-1-reach are reconstructed (src/1dim/algos.jl:91-117)
    for (int c0 = a; c0 < b; c0 += T - 2) {
        const int n = min(T - 2, b - c0);
        // cells c0-3 .. c0+n+2
        for (int e = tid; e < n + 6; e += T) {
            const int i = c0 - 3 + e;
            if (i >= 0 && i < N)
#pragma unroll
                for (int v = 0; v < 3; ++v) sP[v][e] = __ldcg(P + v * N + i);
        }
        __syncthreads();
        // slot t: cell c0 - 1 + t, its face values; the right one belongs to face c0 - 1 + t
        // (left state), the left one to face c0 - 2 + t (right state)
        const int i = c0 - 1 + tid;
        if (tid < n + 2 && i >= 0 && i < N) {
            double qr[3], ql[3];
            if (i >= reach && i <= N - 1 - reach) {
                recon_n<REC, 3, double>([&](int v, int o) { return sP[v][tid + 2 + o]; }, qr, ql);
            } else {
#pragma unroll
                for (int v = 0; v < 3; ++v) {  // never refreshed: the values of t = 0
                    ql[v] = st.PL[v * N + i];
                    qr[v] = i > 0 ? st.PR[v * N + i - 1] : 0.0;
                }
            }
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                sL[v][tid] = ql[v];
                sR[v][tid] = qr[v];
            }
        }
        __syncthreads();
        // face c0 - 1 + t, t = 0 .. n: left state of slot t, right state of slot t + 1
        if (tid <= n && i >= 0 && i < N) {
            double pl[3], pr[3], F[3];
            const bool last = i + 1 >= N;  // face N - 1 has no cell to its right
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                pl[v] = sL[v][tid];
                pr[v] = last ? st.PR[v * N + i] : sR[v][tid + 1];
            }
            ref1d_hll(g, pl, pr, F);
#pragma unroll
            for (int v = 0; v < 3; ++v) sF[v][tid] = F[v];
        }
        __syncthreads();
        if (tid < n) {
            const int c = c0 + tid;
            double u[3], p[3];
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                u[v] = Ub[v * N + c];
                p[v] = G[v * N + c];
            }
            if (c >= 1 && c <= N - 3) {  // i = 2:(N-2) (:284-288, :409-413)
#pragma unroll
                for (int v = 0; v < 3; ++v) u[v] = u[v] - coef * (sF[v][tid + 1] - sF[v][tid]);
            } else {
#pragma unroll
                for (int v = 0; v < 3; ++v) u[v] = Uo[v * N + c];
            }
            c2p_1d(g, n_iter, tol, u, p);
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                Uo[v * N + c] = u[v];
                Pout[v * N + c] = p[v];
            }
        }
        __syncthreads();
    }
    cluster_meet();
}

template <int REC>
__global__ void __launch_bounds__(R1_MAXT) k_ref1d_steps(Ref1DState st, double g, int n_iter, double tol, double dt,
                                                         double dx, int nsteps) {
    const int N = st.N, m = (N + (int)gridDim.x - 1) / (int)gridDim.x;
    const int a = min(N, (int)blockIdx.x * m), b = min(N, a + m);
    const double c1 = 0.5 * dt / dx, c2 = dt / dx;
    for (int n = 0; n < nsteps; ++n) {
        // both con2prims start from the P of the step's start (Phalf = deepcopy(P))
        ref1d_stage<REC>(st, a, b, st.P, st.U, st.Uh, st.P, st.Ph, c1, g, n_iter, tol);
        ref1d_stage<REC>(st, a, b, st.Ph, st.U, st.U, st.P, st.P, c2, g, n_iter, tol);
    }
}

__global__ void k_ref1d_init(Ref1DState st, const double* __restrict__ Pa, double g) {
    const int N = st.N;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        double p[3] = {Pa[3 * i], Pa[3 * i + 1], Pa[3 * i + 2]};
        double U[3];
        ref1d_cons(g, p[0], p[1], p[2], U);  // PtoU, src/1dim/structs.jl:58-66
        for (int v = 0; v < 3; ++v) {
            st.P[v * N + i] = p[v];
            st.Ph[v * N + i] = p[v];
            st.PL[v * N + i] = p[v];
            st.PR[v * N + i] = p[v];
            st.U[v * N + i] = U[v];
            st.Uh[v * N + i] = U[v];
        }
    }
}

__global__ void k_ref1d_store(Ref1DState st, double* __restrict__ Pa) {
    const int N = st.N;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
        for (int v = 0; v < 3; ++v) Pa[3 * i + v] = st.P[v * N + i];
}

cudaError_t launch_ref1d_init(const Ref1DState& st, const double* Pa, double g, cudaStream_t s) {
    k_ref1d_init<<<(st.N + 255) / 256, 256, 0, s>>>(st, Pa, g);
    return cudaGetLastError();
}

template <int REC>
static cudaError_t launch_ref1d_rec(const Ref1DState& st, double g, int n_iter, double tol, double dt, double dx,
                                    int nsteps, cudaStream_t s) {
    auto kern = k_ref1d_steps<REC>;
    static int widest[64] = {0};
    const int wide = widest_cluster(kern, R1_MAXT, 0, widest);
    // at least 32 cells per CTA
    int c = 1;
    while (c < wide && 64 * c <= st.N) c *= 2;
    const int m = (st.N + c - 1) / c;
    const int t = std::min(R1_MAXT, (m + 2 + 31) / 32 * 32);
    return launch_cluster(kern, c, t, 0, s, st, g, n_iter, tol, dt, dx, nsteps);
}

cudaError_t launch_ref1d_steps(const Ref1DState& st, double g, int rec, int n_iter, double tol, double dt,
                               double dx, int nsteps, cudaStream_t s) {
    if (nsteps <= 0) return cudaSuccess;
    if (rec == REC_MINMOD) return launch_ref1d_rec<REC_MINMOD>(st, g, n_iter, tol, dt, dx, nsteps, s);
    if (rec == REC_PPM) return launch_ref1d_rec<REC_PPM>(st, g, n_iter, tol, dt, dx, nsteps, s);
    return launch_ref1d_rec<REC_WENOZ>(st, g, n_iter, tol, dt, dx, nsteps, s);
}

cudaError_t launch_ref1d_store(const Ref1DState& st, double* Pa, cudaStream_t s) {
    k_ref1d_store<<<(st.N + 255) / 256, 256, 0, s>>>(st, Pa);
    return cudaGetLastError();
}

}  // namespace vb

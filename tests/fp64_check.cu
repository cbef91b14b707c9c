// The branch-free FP64 divide and square root (vb_fp64.cuh) and the
// reconstructions, face fluxes and con2prim built on them, against the IEEE
// operations and the general forms, bit for bit (NaN compares as NaN).
//   operands: random mantissas, a quarter each of almost all zeros and almost
//     all ones, exponents over the documented ranges (the divide proper only
//     on the device: on the host it is the IEEE operation);
//   states: ordinary ones, and ones with exact and signed zeros, tiny, huge,
//     subnormal, infinite and NaN components, which must take the general form.
// Run on the host by default, on the device with the argument "device".
// Prints "ok" or the counts of mismatches.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "vb_con2prim.cuh"

using namespace vb;

#define HD __host__ __device__ inline
HD unsigned long long mix(unsigned long long x) {  // splitmix64
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
struct Rng {
    unsigned long long s;
    HD unsigned long long bits() { return mix(s++); }
    HD double unit() { return (double)(bits() >> 11) * 0x1.0p-53; }
};
HD double from_bits(unsigned long long u) {
    double x;
    memcpy(&x, &u, 8);
    return x;
}
HD bool same(double x, double y) {
    unsigned long long a, b;
    memcpy(&a, &x, 8);
    memcpy(&b, &y, 8);
    return a == b || (x != x && y != y);
}
HD double operand(Rng& r, int emin, int emax, bool neg) {
    const unsigned long long k = r.bits(), t = r.bits();
    unsigned long long m = r.bits() & 0xfffffffffffffull;
    if (k % 4 == 1) m = t & 0x3;
    if (k % 4 == 2) m = 0xfffffffffffffull - (t & 0x3);
    const unsigned long long e = 1023 + emin + (t >> 8) % (unsigned long long)(emax - emin);
    return from_bits((neg && (k >> 60 & 1) ? 1ull << 63 : 0) | e << 52 | m);
}
// a factor for a state: mostly 1, sometimes something awkward
HD double awkward(Rng& r) {
    const double v[] = {0.0, -0.0, 1e-38, -1e-80, 1e-95, 1e-200, 5e-324, 1e20, 1e60, 1e200, INFINITY, NAN};
    const unsigned long long k = r.bits();
    return k % 16 ? 1.0 : v[(k >> 8) % 12];
}

enum { N_KINDS = 12 };
// one trial; bad[k] counts mismatches of kind k
HD void trial(unsigned long long id, unsigned* bad) {
    Rng r{id * 1000003ull};
    {
        const double b = operand(r, -900, 900, true), a = operand(r, -80, 80, true) * b;  // quotient near 2^+-80
        if (d64::abs_in<-900, 900>(a) && !same(d64::quot_s(a, d64::divisor(b)), a / b)) ++bad[0];
        const double w = operand(r, -900, 900, false);
        if (!same(d64::root(w), sqrt(w))) ++bad[1];
        const double x = operand(r, -800, 800, true);
        if (!same(d64::sixth(x), x / 6.0)) ++bad[2];
        const double p = operand(r, -3, 3, true), q = operand(r, -3, 3, true);
        if (!same(d64::quot_s(p, d64::divisor(q)), p / q)) ++bad[0];
        if (!same(d64::quot_s(-0.0, d64::divisor(q)), -0.0 / q)) ++bad[0];
    }
    {
        double q[5], base = 10.0 * (r.unit() - 0.5), step = (r.bits() % 4 == 0) ? 0.0 : r.unit();
        const double f = awkward(r);
        for (int k = 0; k < 5; ++k) {
            q[k] = base + step * (r.unit() - 0.5);
            if (r.bits() % 8 == 0) q[k] = 0.0;
            q[k] *= r.bits() % 4 ? f : awkward(r);
        }
        double a, b, c, d;
        recon_n<REC_WENOZ, 1, double>([&](int, int o) { return q[2 + o]; }, &a, &b);
        recon<REC_WENOZ>(q[0], q[1], q[2], q[3], q[4], c, d);
        if (!same(a, c) || !same(b, d)) ++bad[3];
        recon_n<REC_PPM, 1, double>([&](int, int o) { return q[2 + o]; }, &a, &b);
        recon<REC_PPM>(q[0], q[1], q[2], q[3], q[4], c, d);
        if (!same(a, c) || !same(b, d)) ++bad[4];
    }
    const double g = 1.05 + 0.93 * r.unit();
    double P[2][5];
    const double lor = exp(4.0 * r.unit());
    for (int s = 0; s < 2; ++s) {
        P[s][0] = exp(8.0 * (r.unit() - 0.5)) * fabs(awkward(r));
        P[s][1] = exp(12.0 * (r.unit() - 0.7)) * fabs(awkward(r));
        for (int m = 0; m < 3; ++m)
            P[s][2 + m] = (r.bits() % 4 ? 1.0 : 0.0) * lor * (r.unit() - 0.5) * awkward(r);
    }
    for (int m = 0; m < 5; ++m)
        if (r.bits() % 4 == 0) P[1][m] = P[0][m];
    double F[5], H[5];
    const int ax = (int)(r.bits() % 3);
    auto cmp = [&](int n, int kind) {
        for (int v = 0; v < n; ++v)
            if (!same(F[v], H[v])) {
                ++bad[kind];
                return;
            }
    };
    face_flux<3, RS_HLL>(ax, g, P[0], P[1], F);
    face_flux_ieee<3, RS_HLL>(ax, g, P[0], P[1], H);
    cmp(5, 5);
    face_flux<3, RS_HLLC>(ax, g, P[0], P[1], F);
    face_flux_ieee<3, RS_HLLC>(ax, g, P[0], P[1], H);
    cmp(5, 6);
    face_flux<2, RS_HLLC>(ax % 2, g, P[0], P[1], F);
    face_flux_ieee<2, RS_HLLC>(ax % 2, g, P[0], P[1], H);
    cmp(4, 7);
    face_flux<1, RS_HLL>(0, g, P[0], P[1], F);
    face_flux_ieee<1, RS_HLL>(0, g, P[0], P[1], H);
    cmp(3, 8);
    // con2prim of state 0 from a guess up to 30 % off (or from state 1)
    const int n_iter = r.bits() % 8 ? 50 : 3;
    double U[5];
    for (int dim = 1; dim <= 3; ++dim) {
        double G[5];
        for (int v = 0; v < 5; ++v) G[v] = r.bits() % 8 ? P[0][v] * (0.7 + 0.6 * r.unit()) : P[1][v];
        for (int v = 0; v < 5; ++v) F[v] = H[v] = G[v];
        int a, b;
        if (dim == 1) {
            prim2con<1>(g, P[0], U);
            a = c2p_1d(g, n_iter, 1e-12, U, F);
            b = c2p_1d_general(g, n_iter, 1e-12, U, H);
        } else if (dim == 2) {
            prim2con<2>(g, P[0], U);
            a = c2p_2d(g, n_iter, 1e-12, U, F);
            b = c2p_2d_general(g, n_iter, 1e-12, U, H);
        } else {
            prim2con<3>(g, P[0], U);
            a = c2p_3d(g, n_iter, 1e-12, U, F);
            b = c2p_3d_general(g, n_iter, 1e-12, U, H);
        }
        if (a != b) ++bad[8 + dim];
        cmp(2 + dim, 8 + dim);
    }
}

__global__ void k_check(unsigned long long n, unsigned* bad) {
    unsigned b[N_KINDS] = {};
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x)
        trial(i, b);
    for (int k = 0; k < N_KINDS; ++k)
        if (b[k]) atomicAdd(bad + k, b[k]);
}

int main(int argc, char** argv) {
    unsigned bad[N_KINDS] = {};
    if (argc > 1 && !strcmp(argv[1], "device")) {
        unsigned* d = nullptr;
        if (cudaMalloc(&d, sizeof bad) != cudaSuccess || cudaMemset(d, 0, sizeof bad) != cudaSuccess) return 2;
        k_check<<<148 * 4, 128>>>(40000000ull, d);
        if (cudaMemcpy(bad, d, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
        cudaFree(d);
    } else {
        for (unsigned long long i = 0; i < 200000; ++i) trial(i, bad);
    }
    int any = 0;
    for (int k = 0; k < N_KINDS; ++k)
        if (bad[k]) any = 1, printf("kind %d: %u mismatches\n", k, bad[k]);
    if (!any) printf("ok\n");
    return any;
}

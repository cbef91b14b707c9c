// The branch-free FP64 divide and square root (vb_fp64.cuh) on the device over all
// of the operands that its callers admit, against the IEEE operations.
//   ranges: dividend, divisor and quotient with independent exponents in
//     [2^-900, 2^900], the ends often, and dividends up to the largest number
//     (WENOZ tests the quotient and the divisor only); roots of [2^-900, 2^900].
//     Bit for bit: of random operands one pair in 2^50 lies within 2^-51 ulp of a
//     middle, where the two may differ.
//   middles: a / b = M - r / B and sqrt(a) = sqrt(M^2 - r) for integers M halfway
//     between two FP64 numbers and small r, at |r| / (2 B) ulp and |r| / (4 M) ulp from
//     that middle. Bit for bit from 2^-51 ulp on, at most one ulp away nearer to it.
// Argument: the number of trials. Prints "ok" or the mismatches; the count of
// differences nearer than 2^-51 ulp goes to stderr.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "vb_fp64.cuh"

using namespace vb;
typedef unsigned long long u64;
typedef unsigned __int128 u128;

#define HD __host__ __device__ inline
HD u64 mix(u64 x) {  // splitmix64
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
struct Rng {
    u64 s;
    HD u64 bits() { return mix(s++); }
    HD int in(int lo, int hi) { return lo + (int)(bits() % (u64)(hi - lo + 1)); }
};
HD u64 to_bits(double x) {
    u64 u;
    memcpy(&u, &x, 8);
    return u;
}
HD double from_bits(u64 u) {
    double x;
    memcpy(&x, &u, 8);
    return x;
}
HD bool one_ulp(double x, double y) {
    const long long d = (long long)to_bits(x) - (long long)to_bits(y);
    return d >= -1 && d <= 1;
}
// exponent in [lo, hi - 1], a quarter of the draws within two of an end
HD int expo(Rng& r, int lo, int hi) {
    const u64 k = r.bits();
    if (k % 8 == 0) return lo + (int)(k >> 8) % 2;
    if (k % 8 == 1) return hi - 1 - (int)(k >> 8) % 2;
    return r.in(lo, hi - 1);
}
HD double number(Rng& r, int lo, int hi, bool sign) {
    const u64 k = r.bits();
    u64 m = r.bits() & 0xfffffffffffffull;
    if (k % 4 == 1) m = (k >> 8) & 7;
    if (k % 4 == 2) m = 0xfffffffffffffull - ((k >> 8) & 7);
    return from_bits((sign && k >> 63 ? 1ull << 63 : 0) | (u64)(1023 + expo(r, lo, hi)) << 52 | m);
}

enum { QUOT, QUOT_BIG, ROOT, QUOT_MID, QUOT_NEAR, ROOT_MID, ROOT_NEAR, DIFFER, N_KINDS };
__device__ void check_quot(double a, double b, unsigned* bad, int kind, bool near) {
    const double q = d64::quot_s(a, d64::divisor(b)), e = a / b;
    if (to_bits(q) == to_bits(e)) return;
    if (!near || !one_ulp(q, e)) ++bad[kind];
    if (near) ++bad[DIFFER];
}
__device__ void check_root(double a, unsigned* bad, int kind, bool near) {
    const double q = d64::root(a), e = sqrt(a);
    if (to_bits(q) == to_bits(e)) return;
    if (!near || !one_ulp(q, e)) ++bad[kind];
    if (near) ++bad[DIFFER];
}
// the odd x below 2^56 with x^2 = r mod 2^56, r = 1 mod 8
__device__ u64 root_mod(u64 r) {
    u64 x = 1;
    for (int i = 3; i < 57; ++i)
        if ((x * x - r) >> i & 1) x += 1ull << (i - 1);
    return x;
}
__device__ void trial(u64 id, unsigned* bad) {
    Rng r{id * 1000003ull};
    {
        const double a = number(r, -900, 900, true), b = number(r, -900, 900, true), q = a / b;
        if (d64::abs_in<-900, 900>(q)) check_quot(a, b, bad, QUOT, false);
        const double big = number(r, 890, 1024, true), c = number(r, 2, 890, true), p = big / c;
        if (d64::abs_in<-900, 900>(p)) check_quot(big, c, bad, QUOT_BIG, false);
        check_root(number(r, -900, 900, false), bad, ROOT, false);
    }
    {
        const u64 k = r.bits();
        u64 B = 1ull << 52 | (r.bits() & 0xfffffffffffffull) | 1;
        if (k % 8 == 0) B = (1ull << 53) - 1 - 2 * ((k >> 8) % 64);  // mantissas of almost all ones
        if (k % 8 == 1) B = (1ull << 52) + 1 + 2 * ((k >> 8) % 64);
        const int odd = 2 * r.in(0, k & 64 ? 4 : 4000) + 1, rr = k & 128 ? odd : -odd;
        u64 inv = B;
        for (int i = 0; i < 6; ++i) inv *= 2 - B * inv;  // 1 / B mod 2^64
        const u64 M = ((u64)(long long)rr * inv) & ((1ull << 54) - 1);
        if (M >> 53) {  // halfway: 54 bits, odd
            const u128 A = ((u128)M * B - (u128)(__int128)rr) >> 54;
            const int eb = r.in(-800, 700), ea = eb + r.in(-60, 60);
            // |r| / (2 B) >= 2^-51, B < 2^53
            check_quot(ldexp((double)(u64)A, ea), ldexp((double)B, eb), bad, odd >= 9 ? QUOT_MID : QUOT_NEAR, odd < 9);
        }
    }
    {
        const u64 k = r.bits();
        const int lim = k & 64 ? 4 : 4000, rr = 8 * r.in(-lim, lim) + 1, mag = rr < 0 ? -rr : rr;
        u64 M = root_mod((u64)(long long)rr);
        if (k & 1) M = 0 - M;
        M = (M + (k & 2 ? 1ull << 53 : 0)) & ((1ull << 54) - 1);
        if (M >> 53) {
            u128 v = (u128)M * M - (u128)(__int128)rr;
            int tz = 0;
            while (!(u64)(v & 1)) v >>= 1, ++tz;
            if (v >> 53 == 0) {  // an FP64 number: M^2 - r = v 2^tz
                const int e = 2 * r.in(-400, 350);
                // |r| / (4 M) >= 2^-51, M < 2^54
                check_root(ldexp((double)(u64)v, tz + e), bad, mag >= 32 ? ROOT_MID : ROOT_NEAR, mag < 32);
            }
        }
    }
}
__global__ void k_check(u64 n, unsigned* bad) {
    unsigned b[N_KINDS] = {};
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) trial(i, b);
    for (int k = 0; k < N_KINDS; ++k)
        if (b[k]) atomicAdd(bad + k, b[k]);
}

int main(int argc, char** argv) {
    const u64 n = argc > 1 ? strtoull(argv[1], nullptr, 10) : 100000000ull;
    unsigned bad[N_KINDS] = {}, *d = nullptr;
    if (cudaMalloc(&d, sizeof bad) != cudaSuccess || cudaMemset(d, 0, sizeof bad) != cudaSuccess) return 2;
    k_check<<<148 * 8, 128>>>(n, d);
    if (cudaMemcpy(bad, d, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    cudaFree(d);
    fprintf(stderr, "%llu trials, %u differences within 2^-51 ulp of a middle\n", n, bad[DIFFER]);
    int any = 0;
    for (int k = 0; k < DIFFER; ++k)
        if (bad[k]) any = 1, printf("kind %d: %u mismatches\n", k, bad[k]);
    if (!any) printf("ok\n");
    return any;
}

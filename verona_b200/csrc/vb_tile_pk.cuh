// The box tile's stage body (stage_tile, vb_stage.cuh) in the FP32-bulk form on
// packed pairs, for the batch kernel: reconstruction and face fluxes advance two
// cells or faces per instruction (vb_stage_zp.cuh, namespace pk), a cell and the
// one half a tile further, two face indices half the list apart, the two halo
// layers of an axis. Flux differences, RK combination and con2prim are stage_tile's,
// in FP64 on the FP32 fluxes; the FP64 accumulators wait in shared memory, so the
// packed phases keep their registers. 36 tubes and 12 quadrant problems (4.2 M cells,
// two steps) in tiles of 32 x 8: 3.6 ms, against 5.95 ms one cell per thread.
#pragma once
#include "vb_ns.h"

#include "vb_stage_zp.cuh"

namespace VB_NS {

template <int DIM, int TX, int TY, int NT> struct PkTile {
    using G = TileGeom<DIM, TX, TY, 1>;
    static constexpr int TC = TX * TY, CPT = (TC + NT - 1) / NT;
    static constexpr size_t smem_bytes() {
        return 8 * (size_t)G::NV * TC + 4 * (size_t)G::NV * (G::EXTMAX + 2 * G::FACEMAX);
    }
};

// one axis: stage the tile with its halo along D, face states, fluxes, differences into sA
template <int DIM, int D, int REC, int RS, int TX, int TY, int NT, typename Halo>
__device__ __forceinline__ void pk_axis(const StageParams& p, const float* Pin, const int* org, const int* vt,
                                        double* sA, float* sP, float* sL, float* sR, const Halo& halo) {
    using namespace pk;
    constexpr int NV = 2 + DIM, TC = TX * TY;
    constexpr int EX = TX + (D == 0 ? 6 : 0), EY = TY + (D == 1 ? 6 : 0), EXT = EX * EY;
    constexpr int FX = TX + (D == 0), NF = FX * (TY + (D == 1));
    constexpr int SD = D == 0 ? 1 : EX, FS = D == 0 ? 1 : FX;  // steps along D: staged cell, face
    constexpr int TD = D == 0 ? TX : TY, HL = TC / TD;          // tile extent along D, cells of a halo layer
    const int tid = threadIdx.x;
    const f2 fl = S2((float)p.floor_), g = S2((float)p.gamma), gm1 = S2((float)(p.gamma - 1.0));
    const int ox = org[0] - (D == 0 ? NG : 0), oy = org[1] - (D == 1 ? NG : 0);
    __syncthreads();
    for (int e = tid; e < NV * EXT; e += NT) {
        const int v = e / EXT, r = e - v * EXT, gi = ox + r % EX, gj = oy + r / EX;
        sP[e] = gi < p.n[0] && gj < p.n[1] ? __ldcg(Pin + v * p.vs + gi + p.sy * gj) : 0.0f;
    }
    __syncthreads();
    halo(D, sP);
    // the tile's own cells: (lx, ly) with (lx, ly + TY / 2), in 1D lx with lx + TX / 2
    {
        constexpr int DX = DIM == 1 ? TX / 2 : 0, DY = DIM == 1 ? 0 : TY / 2;
        constexpr int OFF = DX + EX * DY, FOFF = DX + FX * DY;
        for (int e = tid; e < TC / 2; e += NT) {
            const int lx = e % TX, ly = e / TX;
            const float* q = sP + lx + (D == 0 ? NG : 0) + EX * (ly + (D == 1 ? NG : 0));
            const int fR = lx + FX * ly;
#pragma unroll
            for (int v = 0; v < NV; ++v, q += EXT) {
                f2 qr, ql;
                recon2<REC>(P2(q[-2 * SD], q[OFF - 2 * SD]), P2(q[-SD], q[OFF - SD]), P2(q[0], q[OFF]),
                            P2(q[SD], q[OFF + SD]), P2(q[2 * SD], q[OFF + 2 * SD]), qr, ql);
                if (v < 2) {
                    qr = vmax(fl, qr);
                    ql = vmax(fl, ql);
                }
                sR[v * NF + fR] = qr.x;
                sR[v * NF + fR + FOFF] = qr.y;
                sL[v * NF + fR + FS] = ql.x;
                sL[v * NF + fR + FOFF + FS] = ql.y;
            }
        }
    }
    // halo cells -1 (its right state, of face 0) and vt[D] (its left state, of face vt[D]): the
    // face vt[D] of a partial tile is written by the cell vt[D] of the tile's own cells above
    for (int e = tid; e < HL * NV; e += NT) {
        const int v = e / HL, k = e - v * HL;
        const int f0 = D == 0 ? FX * k : k;
        const float* q = sP + v * EXT + (D == 0 ? EX * k + NG - 1 : k + EX * (NG - 1));
        constexpr int OFF = (TD + 1) * SD;
        f2 qr, ql;
        recon2<REC>(P2(q[-2 * SD], q[OFF - 2 * SD]), P2(q[-SD], q[OFF - SD]), P2(q[0], q[OFF]), P2(q[SD], q[OFF + SD]),
                    P2(q[2 * SD], q[OFF + 2 * SD]), qr, ql);
        sL[v * NF + f0] = v < 2 ? maxn(fl.x, ql.x) : ql.x;
        sR[v * NF + f0 + TD * FS] = v < 2 ? maxn(fl.x, qr.y) : qr.y;
    }
    __syncthreads();
    // fluxes over the left states; faces beyond the valid cells compute on zeros and are not used
    {
        constexpr int H = (NF + 1) / 2;
        for (int e = tid; e < H; e += NT) {
            const int e2 = e + H < NF ? e + H : e;
            f2 PL[NV], PR[NV], F[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                PL[v] = P2(sL[v * NF + e], sL[v * NF + e2]);
                PR[v] = P2(sR[v * NF + e], sR[v * NF + e2]);
            }
            pk::face_flux<D, RS, DIM>(g, gm1, PL, PR, F);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                sL[v * NF + e] = F[v].x;
                if (e + H < NF) sL[v * NF + e + H] = F[v].y;
            }
        }
    }
    __syncthreads();
    const double cdt = p.dtdx[D];
    for (int cell = tid; cell < TC; cell += NT) {
        const int lx = cell % TX, ly = cell / TX;
        if (lx >= vt[0] || ly >= vt[1]) continue;
        const int f = lx + FX * ly;
#pragma unroll
        for (int v = 0; v < NV; ++v)
            sA[v * TC + cell] = sA[v * TC + cell] - cdt * ((double)sL[v * NF + f + FS] - (double)sL[v * NF + f]);
    }
}

// halo: called with the tile staged for each axis
template <int DIM, int REC, int RS, int TX, int TY, int NT, typename Halo>
__device__ __forceinline__ void stage_tile_pk(const StageParams& p, const StageBufs<float>& b, int bx, int by,
                                              unsigned char* smem_raw, const Halo& halo) {
    using T = PkTile<DIM, TX, TY, NT>;
    constexpr int NV = 2 + DIM, TC = T::TC;
    double* sA = reinterpret_cast<double*>(smem_raw);
    float* sP = reinterpret_cast<float*>(sA + NV * TC);
    float *sL = sP + NV * T::G::EXTMAX, *sR = sL + NV * T::G::FACEMAX;
    const int tid = threadIdx.x;
    const int org[2] = {NG + bx * TX, DIM > 1 ? NG + by * TY : 0};
    const int vt[2] = {min(TX, p.n[0] - NG - org[0]), DIM > 1 ? min(TY, p.n[1] - NG - org[1]) : 1};
    auto index = [&](int cell, long long& c) -> bool {
        const int lx = cell % TX, ly = cell / TX;
        c = (org[0] + lx) + p.sy * (org[1] + ly);
        return lx < vt[0] && ly < vt[1];
    };
    // each thread reads and writes sA for its own cells only
    for (int cell = tid; cell < TC; cell += NT) {
        long long c;
        if (index(cell, c))
#pragma unroll
            for (int v = 0; v < NV; ++v) sA[v * TC + cell] = __ldcg(b.Us + v * p.vs + c);
    }
    pk_axis<DIM, 0, REC, RS, TX, TY, NT>(p, b.Pin, org, vt, sA, sP, sL, sR, halo);
    if constexpr (DIM > 1) pk_axis<DIM, 1, REC, RS, TX, TY, NT>(p, b.Pin, org, vt, sA, sP, sL, sR, halo);
    unsigned long long n_fail = 0, n_fb = 0, n_it = 0, n_cells = 0;
    for (int cell = tid; cell < TC; cell += NT) {
        long long c;
        if (!index(cell, c)) continue;
        double U[NV], P[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            double u = sA[v * TC + cell];
            if (p.rk_a != 0.0) u = p.rk_a * __ldcg(b.U0 + v * p.vs + c) + p.rk_b * u;
            U[v] = u;
            b.Uo[v * p.vs + c] = u;
            P[v] = (double)__ldcg(b.Pin + v * p.vs + c);
        }
        int fb;
        const int r = solve_cell<DIM, 0, true>(p, U, P, c, fb);
        n_fail += (r < 0);
        n_fb += fb;
        n_it += (r < 0 ? -r : r);
        n_cells += 1;
        P[0] = jmax(P[0], p.floor_);
        P[1] = jmax(P[1], p.floor_);
#pragma unroll
        for (int v = 0; v < NV; ++v) b.Pout[v * p.vs + c] = (float)P[v];
    }
    if (n_fail) count_add(p.counters, CNT_C2P_FAIL, n_fail);
    if (p.stats) {
        for (int o = 16; o > 0; o >>= 1) {
            n_fb += __shfl_xor_sync(0xffffffffu, n_fb, o);
            n_it += __shfl_xor_sync(0xffffffffu, n_it, o);
            n_cells += __shfl_xor_sync(0xffffffffu, n_cells, o);
        }
        if ((tid & 31) == 0) {
            count_add(p.counters, CNT_C2P_FALLBACK, n_fb);
            count_add(p.counters, CNT_C2P_ITERS, n_it);
            count_add(p.counters, CNT_C2P_CELLS, n_cells);
        }
    } else if (n_fb) {
        count_add(p.counters, CNT_C2P_FALLBACK, n_fb);
    }
}

}  // namespace vb

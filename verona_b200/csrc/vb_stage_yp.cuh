// Y-marching 2D stage kernel of the FP32-bulk form: the packed pairs of the
// z-pair kernel (vb_stage_zp.cuh) on a 2D grid, one warp working by itself.
//
// A warp owns a strip of 30 columns and marches ly rows in y, two rows (j, j+1)
// at a time, each lane one column with both rows as one float2. Lanes 0 and 31
// are the strip's neighbours: all 32 lanes reconstruct along x, the left state
// of a face comes from the lane to the left and the flux of a cell's right face
// from the lane to the right by shuffle, so lanes 1..30 get both faces and no
// state or flux goes through shared memory. Along y the flux of the face below
// and the left state of the face above stay in the lane. A warp therefore
// waits for no other: the box kernel (k_stage, one cell per thread, scalar
// FP32, three barriers per axis) was bound by instruction issue and those
// barriers. Its price is 32 lanes' work for 30 columns.
//
// Rows arrive in a ring of eight per warp, [4 variables][40 columns] each: by
// TMA (one box per row, two rows ahead; the box starts at the 16-byte boundary
// at or before the strip), or by 4-byte asynchronous copies (tma_tiles = 0).
// The kernel writes U = rk_a U0 + rk_b (Us - div) with the flux differences of the
// FP32 fluxes and their sum in FP64, as the box kernel does: a face's flux leaves
// one cell and enters the next with the same FP64 factor, so sums of U over the grid
// keep to FP64 rounding. con2prim follows in k_c2p_2d. Scheme: src/2dim/algos.jl:11-189.
//
// 2047 x 1021, WENOZ + HLLC: 102 us a stage against 239 us of the box kernel, both
// without con2prim (con2prim apart: 51 us); 4096 x 4096: 0.67 ms. With the divergence
// summed in FP32 it took 92 us: the FP64 sums are 28 conversions, an eighth of
// the FP32 rate each, for 8 values.
#pragma once
#include "vb_ns.h"
#include <cuda.h>  // CUtensorMap

#include "vb_stage_zp.cuh"

namespace VB_NS {

struct YpGeom {
    static constexpr int NV = 4, COLS = 30, BXW = 40, RR = 8;  // RR rows in the ring: j-1 .. j+6
    static constexpr int WARPS = 4, NT = 32 * WARPS;
    static constexpr int ROWF = NV * BXW;       // floats per row slot (640 bytes: 128-byte aligned slots)
    static constexpr int ROW_BYTES = 4 * ROWF;
    static constexpr int U_BYTES = 8 * 2 * 2 * NV * 32;  // Us and U0 of two rows, [array][row][variable][lane]
    static constexpr int WARP_BYTES = RR * ROW_BYTES + 128 + U_BYTES;  // rows, mbarriers, U
};
static_assert(YpGeom::ROW_BYTES % 128 == 0 && YpGeom::BXW >= YpGeom::COLS + 6 + 2 && YpGeom::BXW % 4 == 0, "row box");
static_assert(YpGeom::RR * 8 <= 128, "mbarriers");
constexpr uint32_t YP_MAX_POLLS = 1u << 22;  // bounded waits for a TMA row

template <int REC, int RS, bool TMA, int MINB>
__global__ void __launch_bounds__(YpGeom::NT, MINB)
    k_stage_yp(StageParams p, StageBufs<float> b, int ly, const __grid_constant__ CUtensorMap tm) {
    using namespace pk;
    using G = YpGeom;
    constexpr int NV = G::NV, RR = G::RR, BXW = G::BXW;
    __shared__ __align__(128) unsigned char smem[G::WARPS * G::WARP_BYTES];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int strip = (int)blockIdx.x * G::WARPS + warp;
    const int n0 = p.n[0], n1 = p.n[1];
    const int xs = strip * G::COLS;  // padded x of the strip's first stencil cell: its first column - 3
    if (xs >= n0 - 2 * NG) return;   // no block-wide barrier below
    float* ring = reinterpret_cast<float*>(smem + warp * G::WARP_BYTES);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + warp * G::WARP_BYTES + RR * G::ROW_BYTES);
    double* ubuf = reinterpret_cast<double*>(smem + warp * G::WARP_BYTES + RR * G::ROW_BYTES + 128) + lane;
    const int bx0 = xs & ~3;                  // box start, 16-byte aligned
    const int o = xs - bx0 + 2 + lane;        // this lane's cell in a row: x = xs + 2 + lane
    const int y0 = NG + (int)blockIdx.y * ly;
    const int yend = min(y0 + ly, n1 - NG);
    const long long sy = p.sy, vs = p.vs;
    const int x = xs + 2 + lane;
    const bool mine = lane >= 1 && lane <= G::COLS && x < n0 - NG;
    const f2 fl = S2((float)p.floor_);
    const f2 g = S2((float)p.gamma), gm1 = S2((float)(p.gamma - 1.0));

    auto row = [&](int r) -> const float* { return ring + (r & (RR - 1)) * G::ROWF; };
    // row r -> its slot; r is the ((r - y0 + 3) / RR)-th load of the slot
    auto issue = [&](int r) {
        if constexpr (TMA) {
            if (lane == 0) {
                uint64_t* q = &bar[r & (RR - 1)];
                tc::mbar_arrive_expect_tx(q, G::ROW_BYTES);
                tc::tma_load_3d(ring + (r & (RR - 1)) * G::ROWF, &tm, bx0, r, 0, q);
            }
        } else {
            const int rc = min(r, n1 - 1);
            float* d = ring + (r & (RR - 1)) * G::ROWF;
#pragma unroll
            for (int e = lane; e < G::ROWF; e += 32) {
                const int v = e / BXW, c = min(bx0 + e % BXW, n0 - 1);
                cp_async4(d + e, b.Pin + v * vs + c + sy * rc);
            }
        }
    };
    auto wait = [&](int r) -> bool {
        const uint32_t parity = (uint32_t)((r - y0 + NG) / RR) & 1u;
        return tc::mbar_wait(&bar[r & (RR - 1)], parity, nullptr, YP_MAX_POLLS);
    };
    // reconstruct rows (c, c+1) along y, floored
    auto yrecon = [&](int c, f2* qr, f2* ql) {
        const float *r0 = row(c - 2) + o, *r1 = row(c - 1) + o, *r2 = row(c) + o, *r3 = row(c + 1) + o,
                    *r4 = row(c + 2) + o, *r5 = row(c + 3) + o;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int k = v * BXW;
            const float s1 = r1[k], s2 = r2[k], s3 = r3[k], s4 = r4[k];
            recon2<REC>(P2(r0[k], s1), P2(s1, s2), P2(s2, s3), P2(s3, s4), P2(s4, r5[k]), qr[v], ql[v]);
            if (v < 2) {
                qr[v] = vmax(fl, qr[v]);
                ql[v] = vmax(fl, ql[v]);
            }
        }
    };

    bool ok = true;
    if constexpr (TMA) {
        if (lane == 0) {
            for (int s = 0; s < RR; ++s) tc::mbar_init(&bar[s], 1);
            tc::fence_mbar_init();
        }
        __syncwarp();
    }
    int issued = y0 + 4;  // last row issued
    for (int r = y0 - 3; r <= y0 + 4; ++r) issue(r);
    if constexpr (TMA) {
        for (int r = y0 - 3; r <= y0 + 4; ++r) ok = wait(r) && ok;
    } else {
        cp_async_wait_all();
        __syncwarp();
    }
    float qly[NV], Fym[NV];  // left state of face j + 1/2, flux of face j - 1/2
    {
        f2 qr[NV], ql[NV], L[NV], R[NV], F[NV];
        yrecon(y0 - 1, qr, ql);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            L[v] = S2(ql[v].x);
            R[v] = S2(qr[v].y);
            qly[v] = ql[v].y;
        }
        face_flux<1, RS, 2>(g, gm1, L, R, F);
#pragma unroll
        for (int v = 0; v < NV; ++v) Fym[v] = F[v].x;
    }

#pragma unroll 1
    for (int j = y0; j < yend; j += 2) {
        const bool two = j + 1 < yend;
        // every lane is past the previous pair: rows j+5, j+6 replace j-3, j-2
        if (!__all_sync(0xffffffffu, ok)) break;
        if (j + 2 < yend) {
            if constexpr (TMA) tc::fence_proxy_async();
            issue(j + 5);
            issue(j + 6);
            issued = j + 6;
        }
        // this pair's Us and U0 for the end of the step, past the registers: loaded
        // there they held the warp for 58 % of its cycles (2047 x 1021: 124 against 93 us)
        if (mine) {
            const long long c = x + sy * j;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (q == 1 && !two) break;
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    cp_async8(ubuf + (q * NV + v) * 32, b.Us + v * vs + c + q * sy);
                    if (p.rk_a != 0.0) cp_async8(ubuf + ((2 + q) * NV + v) * 32, b.U0 + v * vs + c + q * sy);
                }
            }
        }
        // fluxes of the faces left of the cell (x) and, below, above it (y); their
        // differences wait for the end of the step, where no state is live
        f2 Fx[NV], Fy[NV];
        {  // x
            const float *ra = row(j) + o, *rb = row(j + 1) + o;
            f2 qr[NV], L[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const int k = v * BXW;
                f2 ql;
                recon2<REC>(P2(ra[k - 2], rb[k - 2]), P2(ra[k - 1], rb[k - 1]), P2(ra[k], rb[k]),
                            P2(ra[k + 1], rb[k + 1]), P2(ra[k + 2], rb[k + 2]), qr[v], ql);
                if (v < 2) {
                    qr[v] = vmax(fl, qr[v]);
                    ql = vmax(fl, ql);
                }
                L[v] = P2(__shfl_up_sync(0xffffffffu, ql.x, 1), __shfl_up_sync(0xffffffffu, ql.y, 1));
            }
            face_flux<0, RS, 2>(g, gm1, L, qr, Fx);
        }
        {  // y: rows j+1, j+2 from the rows j-1 .. j+4; faces j+1/2, j+3/2
            f2 qr[NV], ql[NV], L[NV];
            yrecon(j + 1, qr, ql);
#pragma unroll
            for (int v = 0; v < NV; ++v) L[v] = P2(qly[v], ql[v].x);
            face_flux<1, RS, 2>(g, gm1, L, qr, Fy);
#pragma unroll
            for (int v = 0; v < NV; ++v) qly[v] = ql[v].y;
        }
        cp_async_wait_all();
        const double cx = p.dtdx[0], cy = p.dtdx[1];
        double* out = b.Uo + (x + sy * j);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const float rx = __shfl_down_sync(0xffffffffu, Fx[v].x, 1), ry = __shfl_down_sync(0xffffffffu, Fx[v].y, 1);
            if (mine) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q == 1 && !two) break;
                    double u = ubuf[(q * NV + v) * 32];
                    u = u - cx * ((double)(q ? ry : rx) - (double)(q ? Fx[v].y : Fx[v].x));
                    u = u - cy * ((double)(q ? Fy[v].y : Fy[v].x) - (double)(q ? Fy[v].x : Fym[v]));
                    if (p.rk_a != 0.0) u = p.rk_a * ubuf[((2 + q) * NV + v) * 32] + p.rk_b * u;
                    out[v * vs + q * sy] = u;
                }
            }
            Fym[v] = Fy[v].y;
        }
        if (j + 2 < yend) {
            if constexpr (TMA) {
                ok = wait(j + 5) && ok;
                ok = wait(j + 6) && ok;
            } else {
                __syncwarp();  // the rows' copies were waited for with U's
            }
        }
    }
    if constexpr (TMA) {
        // every row issued was waited for unless a wait ran out: then wait
        // (bounded) for the newest load of each slot before the CTA can end
        if (!__all_sync(0xffffffffu, ok)) {
            for (int r = issued - RR + 1; r <= issued; ++r) wait(r);
            if (lane == 0) count_add(p.counters, CNT_TIMEOUT, 1);
        }
    }
}

// tensor map of a 2D FP32 state array for k_stage_yp: dims (x, y, variable), one row of every variable
inline bool encode_yp_tmap(void* out, const float* P, const Grid& g) {
    if (g.dims != 2 || g.nv != YpGeom::NV) return false;
    const cuuint64_t dim[3] = {(cuuint64_t)g.n[0], (cuuint64_t)g.n[1], (cuuint64_t)YpGeom::NV};
    const cuuint64_t stride[2] = {(cuuint64_t)g.sy * 4, (cuuint64_t)g.vs * 4};
    const cuuint32_t box[3] = {(cuuint32_t)YpGeom::BXW, 1, (cuuint32_t)YpGeom::NV};
    return encode_tmap(out, P, 4, 3, dim, stride, box);
}

constexpr int YP_MINB = 4;  // 16 warps per SM at 128 registers
template <int REC, int RS, bool TMA>
cudaError_t launch_stage_yp_t(const StageParams& p, const StageBufs<float>& b, cudaStream_t s) {
    const int nx = p.n[0] - 2 * NG, ny = p.n[1] - 2 * NG;
    const int strips = (nx + YpGeom::COLS - 1) / YpGeom::COLS, bx = (strips + YpGeom::WARPS - 1) / YpGeom::WARPS;
    const int ly = z_range(bx, ny, YP_MINB * sm_count(), 2);
    CUtensorMap tm;
    if (TMA)
        tm = *static_cast<const CUtensorMap*>(p.tmap_row);
    else
        memset(&tm, 0, sizeof tm);
    k_stage_yp<REC, RS, TMA, YP_MINB><<<dim3(bx, (ny + ly - 1) / ly), YpGeom::NT, 0, s>>>(p, b, ly, tm);
    return cudaGetLastError();
}
template <int REC, int RS>
cudaError_t launch_stage_yp_rs(const StageParams& p, const StageBufs<float>& b, cudaStream_t s) {
    return p.tmap_row ? launch_stage_yp_t<REC, RS, true>(p, b, s) : launch_stage_yp_t<REC, RS, false>(p, b, s);
}
template <int REC> cudaError_t launch_stage_yp_rec(int rs, const StageParams& p, const StageBufs<float>& b, cudaStream_t s) {
    return rs == RS_HLLC ? launch_stage_yp_rs<REC, RS_HLLC>(p, b, s) : launch_stage_yp_rs<REC, RS_HLL>(p, b, s);
}
inline cudaError_t dispatch_stage_yp(int rec, int rs, const StageParams& p, const StageBufs<float>& b, cudaStream_t s) {
    if (rec == REC_MINMOD) return launch_stage_yp_rec<REC_MINMOD>(rs, p, b, s);
    if (rec == REC_PPM) return launch_stage_yp_rec<REC_PPM>(rs, p, b, s);
    return launch_stage_yp_rec<REC_WENOZ>(rs, p, b, s);
}

}  // namespace vb

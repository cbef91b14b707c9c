// Ghosted 1D grids of up to 2048 cells, FP64: every step of a call in one launch
// of a thread-block cluster. One CTA per 128-cell tile runs the box tile's stage
// body (stage_tile, vb_stage.cuh) with its loads past L1, the ghosts are filled
// and floored as in the batch kernel (BatchHalo, batch_ghosts), and the cluster
// meets once per stage. The kernels of one stage take about as long to launch as
// to run at this size: a step of MINMOD + HLLC, RK2 (WENOZ, RK3) takes 15.6 (25.3) us
// here and 24.6 (35.9) us in separate launches, the same from 256 to 2048 cells.
// 2048 cells are one tile for each CTA of the widest cluster; longer grids keep the
// separate launches (24.6 us at 2049, 24.0 at 8192). Built with -fmad=false: the same arithmetic as those kernels, bit for bit.
#include <algorithm>
#include <cstring>

#include "vb_batch.cuh"
#include "vb_cluster.cuh"
#include "vb_tube.h"

namespace vb {

constexpr int TUBE_TX = 128;

template <int REC, int RS>
__global__ void __launch_bounds__(TUBE_TX) k_tube(TubeRun r, const __grid_constant__ BatchProb pr, StageParams q) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double t = r.t0;
    int c = r.cur;
    const int stages = r.rk == 3 ? 3 : 2;
    for (int n = 0; n < r.nsteps; ++n, t += r.dt) {
        double *Pc = r.P[c], *Pn = r.P[1 - c];
        for (int st = 0; st < stages; ++st) {
            StageBufs<double> b;
            b.Pin = (st & 1) ? Pn : Pc;
            b.Pout = (st & 1) ? Pc : Pn;
            b.U0 = r.U0;
            q.dtdx[0] = r.rk == 2 && st == 0 ? r.half_dtdx : r.dtdx;
            if (r.rk == 3) {  // SSP-RK3
                q.rk_a = st == 0 ? 0.0 : (st == 1 ? 0.75 : 1.0 / 3.0);
                q.rk_b = st == 0 ? 1.0 : (st == 1 ? 0.25 : 2.0 / 3.0);
                b.Us = st == 0 ? r.U0 : r.U1;
                b.Uo = st == 2 ? r.U0 : r.U1;
            } else {  // midpoint RK2
                q.rk_a = 0.0;
                q.rk_b = 1.0;
                b.Us = r.U0;
                b.Uo = st ? r.U0 : r.U1;
            }
            const int tile = (int)blockIdx.x;
            if (tile < pr.ntx) {
                batch_ghosts<double>(q, pr, b.Pin, b.Pout, tile, 0, TUBE_TX, 1, st == 0, t);
                BatchHalo<double> halo;
                halo.init(pr, b.Pin, tile, 0, TUBE_TX, 1, st == 0, t);
                stage_tile<1, REC, RS, double, TUBE_TX, 1, 1, TUBE_TX, true>(q, b, tile, 0, 0, smem_raw, nullptr, halo);
            }
            cluster_meet();
        }
        if (r.rk == 3) c ^= 1;  // an odd number of buffer swaps
    }
}

bool tube_fits(int cells) { return cells <= TUBE_TX * CLUSTER_MAX; }

template <int REC, int RS>
static cudaError_t launch_tube_t(const TubeRun& r, const BatchProb& pr, const StageParams& q, cudaStream_t s) {
    auto kern = k_tube<REC, RS>;
    constexpr size_t smem = TileGeom<1, TUBE_TX, 1, 1>::smem_bytes<double>();
    static int widest[64] = {0};
    int c = 1;
    while (c < pr.ntx) c *= 2;
    if (c > widest_cluster(kern, TUBE_TX, smem, widest)) return cudaErrorNotSupported;  // the caller takes the separate kernels
    return launch_cluster(kern, c, TUBE_TX, smem, s, r, pr, q);
}

cudaError_t launch_tube(int rec, int rs, const TubeRun& r, const int* bc_kind, const double (*bc_par)[16],
                        const StageParams& p, cudaStream_t s) {
    BatchProb pr{};
    pr.dims = 1;
    pr.n0 = p.n[0];
    pr.n1 = 1;
    pr.vs = p.vs;
    pr.ntx = (p.n[0] - 2 * NG + TUBE_TX - 1) / TUBE_TX;
    pr.nty = 1;
    for (int f = 0; f < 2; ++f) {
        pr.bc_kind[f] = bc_kind[f];
        for (int k = 0; k < 8; ++k) pr.bc_par[f][k] = bc_par[f][k];
    }
#define VB_CASE(RC, RSC) \
    if (rec == RC && rs == RSC) return launch_tube_t<RC, RSC>(r, pr, p, s);
    VB_CASE(REC_MINMOD, RS_HLL)
    VB_CASE(REC_MINMOD, RS_HLLC)
    VB_CASE(REC_PPM, RS_HLL)
    VB_CASE(REC_PPM, RS_HLLC)
    VB_CASE(REC_WENOZ, RS_HLL)
    VB_CASE(REC_WENOZ, RS_HLLC)
#undef VB_CASE
    return cudaErrorInvalidValue;
}

}  // namespace vb

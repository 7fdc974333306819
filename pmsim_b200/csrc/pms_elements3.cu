// pms_elements3.cu -- fused element kernel for 3D cells of few nodes (Hex8, Tet4), several cells per
// warp: strain -> return map -> F_e and the upper node-pair blocks of K_e for the gather assembly.
//
// One warp per cell leaves most lanes idle where a lane owns an integration point (8 of 32 for Hex8, 4
// for Tet4).  Here slot h of a warp owns cell CPW*group + h, CPW = 32/LPC: lane p < ngauss of the slot owns
// integration point p (phase 1), lane m < NN node m (F_e), and lane t tile t of 2x2 node pairs of the
// upper triangle (K_e).  Phase 1 leaves the gradients g and, at plastic points, h = S g of every node
// in shared memory, so the pairs read both with 16-byte loads and no barrier.
//
// Bounds: the shared-memory data path (LSU data pipe busy 83% on 40x40x40 Hex8, FP64 pipe 34%) at 12 warps (36
// Hex8 or 96 Tet4 cells) per SM; 16 warps spill.  Element kernel of a
// fused step: 40x40x40 Hex8 326 us with a warp per cell, 147 us here (2 blocks per SM 166, 4 blocks 165);
// 30x30x30 Tet4 squares (162,000 cells) 378 and 132 us.  Larger cells (Tet10: 15 tiles, Hex20) stay with
// a warp per cell, and so do rules with more points than lanes per cell (Hex8 with 27).
#include <algorithm>

#include "../../include/pms.h"
#include "pms_element.cuh"
#include "pms_gather.h"

using namespace pms;

namespace {

constexpr int WPB3 = 4;  // warps per block

template <int NN> struct Tile3 {
    static constexpr int NG = (NN + 1) / 2;        // node groups of two
    static constexpr int NT = NG * (NG + 1) / 2;  // tiles of the upper triangle
    static constexpr int LPC = NT > NN ? NT : NN;  // lanes per cell (and the most points a rule may have)
};

// Shared memory (doubles): the block's table dN[m*3 + j][LT], w[LT] with LT = LPC points; per cell X[3*NN],
// dU[3*NN], G[ng][GS], H[ng][GS], TC[ng][4] (alpha, gamma, beta), CS[ng][6].  The cell area also stages the
// upper blocks of K_e for the write-out.
__host__ __device__ constexpr int gs3(int nn) { return 3 * nn + 2; }  // row stride: even, lanes spread over the banks
__host__ __device__ constexpr int table3_doubles(int nn, int lt) { return (3 * nn * lt + lt + 1) & ~1; }
__host__ __device__ constexpr int cell3_doubles(int nn, int ng) {
    const int work = 6 * nn + 2 * ng * gs3(nn) + 10 * ng, stage = nn * (nn + 1) / 2 * 9;
    return ((work > stage ? work : stage) + 1) & ~1;
}
__host__ __device__ constexpr int smem3_bytes(int nn, int ng, int lpc) {
    return (table3_doubles(nn, lpc) + WPB3 * (32 / lpc) * cell3_doubles(nn, ng)) * 8;
}

template <int NN, int UPD, bool DOF, bool DOK>
__global__ void __launch_bounds__(WPB3 * 32, 3) element3_kernel(ElemArgs A) {
    using TL = Tile3<NN>;
    constexpr int LPC = TL::LPC, CPW = 32 / LPC, GS = gs3(NN), NU = NN * (NN + 1) / 2;
    extern __shared__ __align__(16) double smem3[];
    const int ng = A.ngauss;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // the lanes past CPW*LPC join the last slot with hl >= LPC, so they own no node, point or tile
    const int slot = min(lane / LPC, CPW - 1), hl = lane - slot * LPC;
    const int cd = cell3_doubles(NN, ng);
    double* dNs = smem3;               // [m*3+j][LPC]
    double* ws = dNs + 3 * NN * LPC;  // [LPC]
    double* warp_area = smem3 + table3_doubles(NN, LPC) + CPW * wid * cd;
    double* Xs = warp_area + slot * cd;
    double* Us = Xs + 3 * NN;
    double* G = Us + 3 * NN;    // [p][GS]
    double* H = G + ng * GS;    // [p][GS]
    double* TC = H + ng * GS;   // [p][4]
    double* CS = TC + ng * 4;   // [p][6]
    for (int i = threadIdx.x; i < ng * 3 * NN; i += blockDim.x) {
        const int p = i / (3 * NN), r = i - p * 3 * NN;
        dNs[r * LPC + p] = A.tab[i];
    }
    for (int i = threadIdx.x; i < ng; i += blockDim.x) ws[i] = A.tab[ng * 3 * NN + i];
    __syncthreads();
    wait_for_previous();

    int ti = -1, tj = -1;  // this lane's tile (ti <= tj), row-major over the node groups
    {
        int k = 0;
#pragma unroll
        for (int i = 0; i < TL::NG; i++)
#pragma unroll
            for (int j = i; j < TL::NG; j++) {
                if (k == hl) ti = i, tj = j;
                k++;
            }
    }
    constexpr bool ODD = (NN & 1) != 0;  // the last group has one node
    static_assert(!ODD, "the 3D kinds have an even number of nodes");
    constexpr bool do_update = UPD != UPD_NONE;

    const int64_t ngroup = (A.ncell + CPW - 1) / CPW;
    for (int64_t grp = (int64_t)blockIdx.x * WPB3 + wid; grp < ngroup; grp += (int64_t)gridDim.x * WPB3) {
        __syncwarp();  // the previous group's write-out is done with the cells' shared memory
        // a slot without a cell (the ragged end) repeats the group's first cell and writes nothing
        const int64_t first = A.cell0 + grp * CPW;
        const bool active = grp * CPW + slot < A.ncell;
        const int64_t cell = active ? first + slot : first;
        const MatConst mc = A.mats[A.cmat ? A.cmat[cell] : 0];

        // the IP state first, so that its latency overlaps the node staging
        const int64_t ip0 = cell * ng;
        const bool has_ip = hl < ng;
        double sig[6], z = 0.0, lam = 0.0;
        int el = 1;
#pragma unroll
        for (int c = 0; c < 6; c++) sig[c] = 0.0;
        if (has_ip) {
            const double* ssrc = UPD == UPD_BACKUP ? A.sig_src : A.sig;
            const double* zsrc = UPD == UPD_BACKUP ? A.z_src : A.z;
            const double* lsrc = UPD == UPD_BACKUP ? A.lam_src : A.lam;
            const uint8_t* esrc = UPD == UPD_BACKUP ? A.el_src : A.el;
#pragma unroll
            for (int c = 0; c < 6; c++) sig[c] = ssrc[(int64_t)c * A.nip + ip0 + hl];
            z = zsrc[ip0 + hl];
            lam = lsrc[ip0 + hl];
            el = esrc[ip0 + hl];
        }
        if (hl < NN) {
            const int pt = A.conn[cell * NN + hl];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                Xs[hl * 3 + i] = A.coords[(int64_t)pt * 3 + i];
                if (do_update) Us[hl * 3 + i] = A.ddu[(int64_t)pt * 3 + i];
            }
        }
        __syncwarp();

        // ---------------- phase 1: lane p of the slot owns integration point p ----------------
        int err = OK, err_t = OK;  // stress-update (and geometry) error, tangent error
        if (has_ip) {
            const int p = hl;
            double J[9];
#pragma unroll
            for (int k = 0; k < 9; k++) J[k] = 0.0;
#pragma unroll
            for (int m = 0; m < NN; m++)
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) J[i * 3 + j] = fma(Xs[m * 3 + i], dNs[(m * 3 + j) * LPC + p], J[i * 3 + j]);
            double Ji[9];
            const double det = inv_jacobian<3>(J, Ji);
            if (!(det > 0.0)) err = E_JACOBIAN;
            const double coef = det * ws[p] * A.thickness;
            double D[9];  // displacement gradient: sum of u_i g_j
#pragma unroll
            for (int k = 0; k < 9; k++) D[k] = 0.0;
            double* Gp = G + p * GS;
#pragma unroll
            for (int m = 0; m < NN; m++) {
                double g[3];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    double v = 0.0;
#pragma unroll
                    for (int j = 0; j < 3; j++) v = fma(dNs[(m * 3 + j) * LPC + p], Ji[j * 3 + i], v);
                    g[i] = v;
                    Gp[m * 3 + i] = v;
                }
                if (do_update) {
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) D[i * 3 + j] = fma(Us[m * 3 + i], g[j], D[i * 3 + j]);
                }
            }
            if (do_update) {  // Mandel components: sqrt(2) (D_ij + D_ji)/2
                const double eps[6] = {D[0], D[4], D[8], (D[1] + D[3]) * INV_SQRT2, (D[5] + D[7]) * INV_SQRT2,
                                       (D[2] + D[6]) * INV_SQRT2};
                const int st = ip_update<6>(mc, mc.hh, sig, z, lam, el, eps);
                if (st != OK && err == OK) err = st;
            }
            if (DOF) {  // coef * sigma: xx, yy, xy, zz, yz, xz
                double2* c6 = reinterpret_cast<double2*>(CS + p * 6);
                c6[0] = make_double2(coef * sig[0], coef * sig[1]);
                c6[1] = make_double2(coef * sig[3] * INV_SQRT2, coef * sig[2]);
                c6[2] = make_double2(coef * sig[4] * INV_SQRT2, coef * sig[5] * INV_SQRT2);
            }
            if (DOK) {
                double a, b, s[6];
                err_t = tangent_coefs<6>(mc, mc.hh, sig, lam, el, a, b, s);
                const double be = coef * b;
                double2* t = reinterpret_cast<double2*>(TC + p * 4);
                // alpha; kappa = gamma - c alpha (see the node pairs below); beta
                const double cvol = (mc.kk - 2.0 * mc.gg / 3.0) / mc.gg;
                const double al = coef * 0.5 * a;
                t[0] = make_double2(al, coef * (mc.kk - a / 3.0) - cvol * al);
                TC[p * 4 + 2] = be;
                if (be != 0.0) {
                    const double sxy = s[3] * INV_SQRT2, syz = s[4] * INV_SQRT2, sxz = s[5] * INV_SQRT2;
                    double* Hp = H + p * GS;
#pragma unroll
                    for (int m = 0; m < NN; m++) {
                        const double g0 = Gp[m * 3], g1 = Gp[m * 3 + 1], g2 = Gp[m * 3 + 2];
                        Hp[m * 3] = fma(sxz, g2, fma(sxy, g1, s[0] * g0));
                        Hp[m * 3 + 1] = fma(syz, g2, fma(s[1], g1, sxy * g0));
                        Hp[m * 3 + 2] = fma(s[2], g2, fma(syz, g1, sxz * g0));
                    }
                }
            }
        }
        // first failing IP of each cell (lowest p): an update error if any, else a tangent error
        {
            const unsigned bad = __ballot_sync(FULL, err != OK);
            const unsigned bad_t = __ballot_sync(FULL, err_t != OK);
            if (bad | bad_t) {
                const unsigned mask = LPC == 32 ? FULL : ((1u << LPC) - 1u);
                const unsigned mine = (bad >> (LPC * slot)) & mask, mine_t = (bad_t >> (LPC * slot)) & mask;
                const int f = mine ? __ffs(mine) - 1 : 0, ft = mine_t ? __ffs(mine_t) - 1 : 0;
                const int code = __shfl_sync(FULL, err, LPC * slot + f);
                const int code_t = __shfl_sync(FULL, err_t, LPC * slot + ft);
                if (active && hl == 0) {
                    if (mine) report(A, do_update ? RANK_UPDATE : RANK_TANGENT, code, cell, f);
                    else if (mine_t) report(A, RANK_TANGENT, code_t, cell, ft);
                }
            }
        }
        if (active && do_update && has_ip) {
#pragma unroll
            for (int c = 0; c < 6; c++) A.sig[(int64_t)c * A.nip + ip0 + hl] = sig[c];
            A.z[ip0 + hl] = z;
            A.lam[ip0 + hl] = lam;
            A.el[ip0 + hl] = (uint8_t)el;
        }
        __syncwarp();

        // ---------------- F_int: lane m of the slot owns node m ----------------
        if (DOF && hl < NN) {
            double f0 = 0.0, f1 = 0.0, f2 = 0.0;
            for (int p = 0; p < ng; p++) {
                const double2* c6 = reinterpret_cast<const double2*>(CS + p * 6);
                const double2 d = c6[0], o = c6[1], q = c6[2];  // (xx, yy), (xy, zz), (yz, xz)
                const double* g = G + p * GS + hl * 3;
                const double g0 = g[0], g1 = g[1], g2 = g[2];
                f0 += d.x * g0 + o.x * g1 + q.y * g2;
                f1 += o.x * g0 + d.y * g1 + q.x * g2;
                f2 += q.y * g0 + q.x * g1 + o.y * g2;
            }
            if (active) {
                double* fe = A.fe + ((cell - A.ke_cell0) * NN + hl) * 3;
                fe[0] = f0;
                fe[1] = f1;
                fe[2] = f2;
            }
        }

        // ---------------- node pairs: the lane owns a tile of 2x2 blocks ----------------
        // X_ab = sum_p alpha_p g_a g_b^T over every point, K_ab = X_ab^T + tr(X_ab) 1 + c X_ab, then kappa_p g_a g_b^T +
        // beta_p h_a h_b^T at the plastic points (c = lambda/G, kappa = gamma - c alpha; an elastic point has
        // gamma = c alpha)
        if (DOK) {
            double acc[2][2][3][3];
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) acc[r][c][i][j] = 0.0;
            if (ti >= 0) {
                auto load6 = [](const double* v, double (&o)[2][3]) {  // two nodes, 16-byte aligned
                    const double2* d = reinterpret_cast<const double2*>(v);
                    const double2 x = d[0], y = d[1], w = d[2];
                    o[0][0] = x.x; o[0][1] = x.y; o[0][2] = y.x;
                    o[1][0] = y.y; o[1][1] = w.x; o[1][2] = w.y;
                };
                for (int p = 0; p < ng; p++) {
                    const double al = TC[p * 4];
                    const double* Gp = G + p * GS;
                    double gr[2][3], gb[2][3];
                    load6(Gp + 6 * ti, gr);
                    load6(Gp + 6 * tj, gb);
#pragma unroll
                    for (int r = 0; r < 2; r++)
#pragma unroll
                        for (int i = 0; i < 3; i++) gr[r][i] *= al;
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int r = 0; r < 2; r++)
#pragma unroll
                            for (int i = 0; i < 3; i++)
#pragma unroll
                                for (int j = 0; j < 3; j++) acc[r][c][i][j] = fma(gr[r][i], gb[c][j], acc[r][c][i][j]);
                }
                const double cvol = (mc.kk - 2.0 * mc.gg / 3.0) / mc.gg;
#pragma unroll
                for (int r = 0; r < 2; r++)
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        double (&x)[3][3] = acc[r][c];
                        const double tr = x[0][0] + x[1][1] + x[2][2];
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            x[i][i] = fma(cvol, x[i][i], x[i][i]) + tr;
#pragma unroll
                            for (int j = i + 1; j < 3; j++) {
                                const double u = x[i][j], l = x[j][i];
                                x[i][j] = fma(cvol, u, l);
                                x[j][i] = fma(cvol, l, u);
                            }
                        }
                    }
                for (int p = 0; p < ng; p++) {
                    const double be = TC[p * 4 + 2];
                    if (be == 0.0) continue;  // elastic point: same value on every lane of the slot
                    const double kap = TC[p * 4 + 1];
                    double gr[2][3], gb[2][3];
                    load6(G + p * GS + 6 * ti, gr);
                    load6(G + p * GS + 6 * tj, gb);
#pragma unroll
                    for (int r = 0; r < 2; r++)
#pragma unroll
                        for (int i = 0; i < 3; i++) gr[r][i] *= kap;
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int r = 0; r < 2; r++)
#pragma unroll
                            for (int i = 0; i < 3; i++)
#pragma unroll
                                for (int j = 0; j < 3; j++) acc[r][c][i][j] = fma(gr[r][i], gb[c][j], acc[r][c][i][j]);
                    load6(H + p * GS + 6 * ti, gr);
                    load6(H + p * GS + 6 * tj, gb);
#pragma unroll
                    for (int r = 0; r < 2; r++)
#pragma unroll
                        for (int i = 0; i < 3; i++) gr[r][i] *= be;
#pragma unroll
                    for (int c = 0; c < 2; c++)
#pragma unroll
                        for (int r = 0; r < 2; r++)
#pragma unroll
                            for (int i = 0; i < 3; i++)
#pragma unroll
                                for (int j = 0; j < 3; j++) acc[r][c][i][j] = fma(gr[r][i], gb[c][j], acc[r][c][i][j]);
                }
            }
            __syncwarp();  // every slot is done reading the areas that the staging overwrites
            if (ti >= 0) {
#pragma unroll
                for (int r = 0; r < 2; r++)
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        const int a = 2 * ti + r, b = 2 * tj + c;
                        if (a > b) continue;
                        double* dst = Xs + 9 * upper_block(NN, a, b);
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = 0; j < 3; j++) dst[i * 3 + j] = acc[r][c][i][j];
                    }
            }
            __syncwarp();
            // the group's cells follow one another in memory: one run of 16-byte stores
            constexpr int NQ = NU * 9 / 2;
            static_assert(NU * 9 % 2 == 0, "a cell's blocks fill whole 16-byte words");
            const int n = NQ * (int)min((int64_t)CPW, A.ncell - grp * CPW);
            double2* dst = reinterpret_cast<double2*>(A.ke + (first - A.ke_cell0) * (int64_t)(NU * 9));
            for (int t = lane; t < n; t += 32) {
                const int c = t / NQ;
                dst[t] = reinterpret_cast<const double2*>(warp_area + c * cd)[t - c * NQ];
            }
        }
    }
}

template <int NN, int UPD, bool DOF, bool DOK>
void launch_t(pms_elements* h, const ElemArgs& a, cudaStream_t stream) {
    constexpr int LPC = Tile3<NN>::LPC, CPW = 32 / LPC;
    auto kern = element3_kernel<NN, UPD, DOF, DOK>;
    const int smem = smem3_bytes(NN, a.ngauss, LPC);
    const int64_t groups = (a.ncell + CPW - 1) / CPW;
    const int64_t blocks = std::min<int64_t>((groups + WPB3 - 1) / WPB3, launch_plan(h, (const void*)kern, smem, WPB3 * 32));
    void* args[] = {(void*)&a};
    if (a.grid) *a.grid = blocks;
    launch_overlapped(a.overlap, (const void*)kern, std::max<int64_t>(blocks, 1), WPB3 * 32, smem, stream, args);
}

template <int NN>
bool launch_nn(pms_elements* h, const ElemArgs& a, int upd, bool dof, bool dok, cudaStream_t st) {
    if (a.ngauss > Tile3<NN>::LPC) return false;
    if (!dof && !dok) {
        if (upd == UPD_CURRENT) launch_t<NN, UPD_CURRENT, false, false>(h, a, st);
        else launch_t<NN, UPD_BACKUP, false, false>(h, a, st);
    } else if (upd == UPD_BACKUP) {
        if (dok) launch_t<NN, UPD_BACKUP, true, true>(h, a, st);
        else launch_t<NN, UPD_BACKUP, true, false>(h, a, st);
    } else if (dof && dok) {
        launch_t<NN, UPD_NONE, true, true>(h, a, st);
    } else if (dof) {
        launch_t<NN, UPD_NONE, true, false>(h, a, st);
    } else {
        launch_t<NN, UPD_NONE, false, true>(h, a, st);
    }
    return true;
}

}  // namespace

namespace pms {

bool launch_elements3(pms_elements* h, int kind, const ElemArgs& a, int upd, bool dof, bool dok, cudaStream_t stream) {
    switch (kind) {
    case PMS_TET4: return launch_nn<4>(h, a, upd, dof, dok, stream);
    case PMS_HEX8: return launch_nn<8>(h, a, upd, dof, dok, stream);
    default: return false;
    }
}

}  // namespace pms

// pms_gather.cu -- gather assembly: the rows of K and R summed over the cells' element matrices.
#include <algorithm>

#include "../../include/pms.h"
#include "pms_gather.h"

using namespace pms;

namespace {

constexpr unsigned FULL = 0xffffffffu;
// One group of lanes per block row A of K.  For each incidence k of A (cell c, local node a) the group adds
// the NN node-pair blocks (a, b) of c's element matrix -- kept as its upper blocks, so block (b, a) is
// read transposed where b < a -- at column slot[k*NN + b] of the row's buffer in shared memory, and
// writes the row once, coalesced.  The incidences go in ascending (= cell) order, so every entry of
// K is the fixed-order sum over its cells: bit-identical on every run.  The same pass forms R (row A
// sums its cells' F_e).  ke and fe are read by ordinary loads: a launch that overlaps the element kernel
// is resident while they are written, and the read-only path (__ldg) is for memory that stays as it is from
// the kernel's start to its end; the maps of the mesh do.
//
// Bounds: 64x64x32 Hex20 moves 4.2 GB (0.65 ms at 6.5 TB/s) and takes 1.54 ms, a lane per 3x3 block took 1.57:
// the LSU data pipe (each 8-byte value is loaded, added in shared memory and written out; busy 72% on 32x32x16
// Hex20, 84% on 40x40x40 Hex8, 83% on 350x350 Qua8, 66% on 24x23x21 Tet4) and the row's chain of dependent
// loads (long scoreboard: 39, 44, 68 and 52% of the cycles between a warp's instructions).  The other kinds gained: 40x40x40 Hex8 136 -> 116 us (lower
// triangle 136 -> 114), 701x350 Qua8 231 -> 176, 24x23x21 Tet4 60 -> 50, 400x300 Tri6 151 -> 110,
// 20x10 Qua8 15 -> 8.6 us (F_int and K in one launch).  Measured slower: ranges and incidences loaded a
// row or two ahead (Hex20 1.9 ms, 701x350 Qua8 0.46 ms: fewer warps, spills), source lists per block of K with the
// sums in registers (2.4 ms, 0.32 ms), upper rows only with the lower part stored transposed (2.7 ms:
// scattered 24-byte stores), the largest shared-memory carveout (Qua8 +40%: L1 holds the slots and
// the sectors that two loads share).
constexpr int GATHER_WARPS = 8;         // warps per block, at most (fewer where the row buffers are large)
constexpr int GATHER_SMEM = 72 * 1024;  // row buffers of a block (one warp's may need more)

// Where entry (i, c) of a block row goes in the triangle storages, relative to tbase[A]: row i holds,
// lower, c = 0 .. ND*dp + i (from i*ND*dp + i(i+1)/2 on), upper, c = dp*ND + i .. ND*nba - 1 (from
// i*ND*(nba - dp) - i(i-1)/2 on); -1: outside the triangle.
template <int ND>
__device__ __forceinline__ int triangle_place(bool lower, int nba, int dp, int i, int c) {
    if (lower) return c <= ND * dp + i ? i * ND * dp + i * (i + 1) / 2 + c : -1;
    const int r = c - ND * dp - i;
    return r >= 0 ? i * ND * (nba - dp) - i * (i - 1) / 2 + r : -1;
}

// 3D: lane e = (i, j) of nine lanes carries entry (i, j) of its blocks, so a group of nine lanes reads a
// block's 72 bytes together and the addresses of the NN blocks differ by constants.  The warp's 27
// lanes are three rows of one group each (ROWS = 3), or one row with three blocks at a time for the cells
// whose rows are long and of uneven length (ROWS = 1: Hex20, 8 or 4 cells a row).  The buffer keeps a
// block's nine entries together (few bank conflicts); the write-out reads it by scalar rows.
template <int NN> struct Gather3 {
    static constexpr int ROWS = NN >= 13 ? 1 : 3;
    static constexpr int BPI = 3 / ROWS;              // blocks at a time
    static constexpr int NIT = (NN + BPI - 1) / BPI;  // blocks per lane and incidence
    static constexpr bool FEW = NN < 10;              // has a kernel for few rows
    static constexpr int CL = ROWS == 1 ? 27 : 9;     // lanes that hold a row's incidences
};

// NB incidences are loaded before they are added: two with one row a warp, one with three rows (the registers
// of two cost a third of the warps: 40x40x40 Hex8 255 us a step with one, 266 with two; Tet4, with half the blocks a
// lane, was not measured beyond few rows).  Where the call's rows are all in flight at once anyway (FEW), the chain of
// a row's loads is the time: the warps get more registers and load two incidences ahead (four for Tet4, whose rows are
// up to 24 cells long).  K in calls that follow one another, us: Hex8 5x5x5 14.5 -> 13.1, 9x8x8 15.6 -> 14.1, 13x13x12
// 17.9 -> 16.6, 17x18x15 22.8 and 22.8; Tet4 6x6x6 21.3 -> 16.7, 13x13x12 25.9 -> 21.0, 18x18x18 38.9 -> 36.0.  Hex20
// gains nothing (6x6x6 21.0 and 21.0), Tet10 was not measured.  Four incidences for Hex8 gave the same as two.
template <int NN, bool TRI, bool FEW>
__global__ void __launch_bounds__(GATHER_WARPS * 32, FEW ? 2 : 3) gather3_kernel(GatherArgs P) {
    constexpr int NU = NN * (NN + 1) / 2;
    using GS = Gather3<NN>;
    constexpr int ROWS = GS::ROWS, BPI = GS::BPI, NIT = GS::NIT, CL = GS::CL;
    constexpr int NB = ROWS == 1 ? 2 : !FEW ? 1 : NN > 4 ? 2 : 4;
    extern __shared__ double rowbuf[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int e = lane % 9, sub = lane / 9;  // lanes 27..31: sub = 3, no blocks
    const int et = 3 * (e % 3) + e / 3;
    const int q = ROWS == 3 ? min(sub, 2) : 0, b0 = ROWS == 3 ? 0 : sub;
    const int c0 = ROWS == 3 ? 9 * q : 0;  // first lane of the row's incidences
    const int cl = lane - c0;              // this lane's incidence in a run of CL
    double* buf = rowbuf + (int64_t)(wid * ROWS + q) * P.nbmax * 9;
    const int64_t step = (int64_t)gridDim.x * wpb * ROWS;
    int64_t r = ((int64_t)blockIdx.x * wpb + wid) * ROWS;  // first row of the warp (of nrow)
    if (r >= P.nrow) return;
    wait_for_previous();
    let_next_start(P.signal);
    const bool mine = sub < 3;
    for (; r < P.nrow; r += step) {
        const int64_t A = P.node0 + r + q;
        const bool row_on = r + q < P.nrow;
        int64_t k0 = 0, ba = 0;
        int nba = 0, ninc = 0;
        if (row_on) {
            k0 = P.inc_ptr[A];
            ba = P.bptr[A];
            ninc = (int)(P.inc_ptr[A + 1] - k0);
            nba = (int)(P.bptr[A + 1] - ba);
        }
        int32_t code = (cl < CL && cl < ninc) ? __ldg(P.inc + k0 + cl) : 0;
        int dp = 0;
        int64_t tb = 0;
        if constexpr (TRI) {
            if (row_on) {
                dp = __ldg(P.kdiag + A);
                tb = __ldg(P.tbase + A);
            }
        }
        const int nmax = ROWS == 1 ? ninc : __reduce_max_sync(FULL, ninc);
        const bool acc_f = P.ff && row_on && mine && b0 == 0 && e < 3;
        double f = 0.0;
        bool zeroed = false;
        for (int n0 = 0; n0 < nmax; n0 += NB) {
            double v[NB][NIT], fv[NB];
            int pos[NB][NIT];
#pragma unroll
            for (int t = 0; t < NB; t++) {
                const int n = n0 + t;
                if (n > 0 && n % CL == 0) {  // the next run of incidences
                    code = (cl < CL && n + cl < ninc) ? __ldg(P.inc + k0 + n + cl) : 0;
                }
                const int32_t cd = __shfl_sync(FULL, code, c0 + n % CL);
                const bool on = n < ninc && mine;
                const int cell = cd / NN, a = cd - cell * NN;
                // block (a, b), b >= a: 9*upper_block(a, b) + e = up + 9*b; else the transpose of (b, a):
                // 9*upper_block(b, a) + et = lo + 9*(upper_block(b, b) - b)
                const double* kc = P.ke + (int64_t)cell * (NU * 9);
                const double* up = kc + 9 * (upper_block(NN, a, a) - a) + e;
                const double* lo = kc + 9 * a + et;
                const int16_t* sl = P.slot + (k0 + n) * NN;
                fv[t] = (acc_f && on) ? P.fe[(int64_t)cd * 3 + e] : 0.0;
#pragma unroll
                for (int u = 0; u < NIT; u++) {
                    const int b = u * BPI + b0;
                    const bool have = on && (NIT * BPI == NN || b < NN);
                    pos[t][u] = have ? (int)__ldg(sl + b) : -1;
                    v[t][u] = have ? *(b >= a ? up + 9 * b : lo + 9 * (upper_block(NN, b, b) - b)) : 0.0;
                }
            }
            if (!zeroed) {  // while the first loads are under way
                for (int x = ROWS == 3 ? e : lane; x < nba * 9 && (ROWS == 1 || mine); x += ROWS == 3 ? 9 : 32) buf[x] = 0.0;
                zeroed = true;
            }
#pragma unroll
            for (int t = 0; t < NB; t++) {
                // three blocks of one row at a time: an entry's next contribution may come from other lanes
                if (ROWS == 1 || t == 0) __syncwarp();
#pragma unroll
                for (int u = 0; u < NIT; u++)
                    if (pos[t][u] >= 0) buf[9 * pos[t][u] + e] += v[t][u];
                f += fv[t];
            }
        }
        if (acc_f) P.ff[A * 3 + e] = f;
        __syncwarp();
        // write-out: all lanes, one row of the warp after another; entry (i, c) from block c/3
#pragma unroll
        for (int g = 0; g < ROWS; g++) {
            const int nb = __shfl_sync(FULL, nba, 9 * g);
            const double* src = rowbuf + (int64_t)(wid * ROWS + g) * P.nbmax * 9;
            const int nrow = 3 * nb;
            double* dst;
            int dg = 0;
            if constexpr (TRI) {
                dst = P.csr + __shfl_sync(FULL, tb, 9 * g);
                dg = __shfl_sync(FULL, dp, 9 * g);
            } else {
                dst = P.csr + 9 * __shfl_sync(FULL, ba, 9 * g);
            }
            for (int x = lane; x < 9 * nb; x += 32) {
                const int i = (x >= nrow) + (x >= 2 * nrow), c = x - i * nrow, p = c / 3;
                const double val = src[9 * p + 3 * i + (c - 3 * p)];
                if constexpr (TRI) {
                    const int at = triangle_place<3>(P.sym == PMS_SYM_LOWER, nb, dg, i, c);
                    if (at >= 0) dst[at] = val;
                } else {
                    dst[x] = val;
                }
            }
        }
        __syncwarp();
    }
}

// 2D: a group of NN lanes per row, G = 32/NN rows per warp; lane b carries the whole 2x2 block (a, b), 32
// contiguous bytes (one sector) in two 16-byte loads, transposed in registers where it is stored as
// (b, a).
template <int NN, bool TRI>
__global__ void __launch_bounds__(GATHER_WARPS * 32, 5) gather2_kernel(GatherArgs P) {
    constexpr int NU = NN * (NN + 1) / 2, G = 32 / NN;
    extern __shared__ __align__(16) double rowbuf2[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    double* buf = rowbuf2 + (int64_t)wid * G * P.nbmax * 4;
    const int g = min(lane / NN, G - 1), b = lane - g * NN;  // the lanes past G*NN: b >= NN, no blocks
    const int64_t step = (int64_t)gridDim.x * wpb * G;
    int64_t r = ((int64_t)blockIdx.x * wpb + wid) * G;  // first row of the warp (of nrow)
    if (r >= P.nrow) return;
    wait_for_previous();
    let_next_start(P.signal);
    const bool aligned = ((uintptr_t)P.csr & 15) == 0;  // the caller's values may start on an odd 8 bytes
    for (; r < P.nrow; r += step) {
        const int64_t A = P.node0 + r + g;
        const bool row_on = r + g < P.nrow, on = row_on && b < NN;
        int64_t k0 = 0, ba = 0;
        int nba = 0, ninc = 0;
        if (row_on) {
            k0 = P.inc_ptr[A];
            ba = P.bptr[A];
            ninc = (int)(P.inc_ptr[A + 1] - k0);
            nba = (int)(P.bptr[A + 1] - ba);
        }
        int32_t code = (b < NN && b < ninc) ? __ldg(P.inc + k0 + b) : 0;
        int dp = 0;
        int64_t tb = 0;
        if constexpr (TRI) {
            if (row_on) {
                dp = __ldg(P.kdiag + A);
                tb = __ldg(P.tbase + A);
            }
        }
        // the rows of the warp are consecutive, so their buffers lie back to back in CSR order
        const int64_t bfirst = __shfl_sync(FULL, ba, 0);
        const int off = row_on ? (int)(ba - bfirst) : 0;
        const int total = __reduce_max_sync(FULL, off + nba);
        const int nmax = __reduce_max_sync(FULL, ninc);
        double2* r0 = reinterpret_cast<double2*>(buf + 4 * off);  // scalar rows 0 and 1 of the block row
        double2* r1 = r0 + nba;
        double f = 0.0;
        const bool acc_f = P.ff && on && b < 2;
        for (int n = 0; n < nmax; n++) {
            if (n > 0 && n % NN == 0)  // the next run of incidences
                code = (b < NN && n + b < ninc) ? __ldg(P.inc + k0 + n + b) : 0;
            const int32_t cd = __shfl_sync(FULL, code, g * NN + n % NN);
            double2 u = make_double2(0.0, 0.0), v = u;
            double fv = 0.0;
            int pos = -1;
            if (on && n < ninc) {
                const int cell = cd / NN, a = cd - cell * NN;
                const bool upper = a <= b;
                const double2* src = reinterpret_cast<const double2*>(
                    P.ke + 4 * ((int64_t)cell * NU + upper_block(NN, upper ? a : b, upper ? b : a)));
                u = src[0];
                v = src[1];
                pos = __ldg(P.slot + (k0 + n) * NN + b);
                if (acc_f) fv = P.fe[(int64_t)cd * 2 + b];
                if (!upper) {
                    const double x = u.y;
                    u.y = v.x;
                    v.x = x;
                }
            }
            if (n == 0) {  // while the first loads are under way
                for (int x = lane; x < total * 2; x += 32) reinterpret_cast<double2*>(buf)[x] = make_double2(0.0, 0.0);
            }
            __syncwarp();  // the previous incidence is added
            if (pos >= 0) {
                const double2 x = r0[pos], y = r1[pos];
                r0[pos] = make_double2(x.x + u.x, x.y + u.y);
                r1[pos] = make_double2(y.x + v.x, y.y + v.y);
            }
            f += fv;
        }
        if (acc_f) P.ff[A * 2 + b] = f;
        __syncwarp();
        if constexpr (TRI) {
            if (on) {
                double* dst = P.csr + tb;
                const double* src = buf + 4 * off;
                for (int x = b; x < 4 * nba; x += NN) {
                    const int i = x >= 2 * nba;
                    const int at = triangle_place<2>(P.sym == PMS_SYM_LOWER, nba, dp, i, x - i * 2 * nba);
                    if (at >= 0) dst[at] = src[x];
                }
            }
        } else {
            double* dst = P.csr + 4 * bfirst;
            if (aligned) {
                for (int x = lane; x < total * 2; x += 32)
                    reinterpret_cast<double2*>(dst)[x] = reinterpret_cast<const double2*>(buf)[x];
            } else {
                for (int x = lane; x < total * 4; x += 32) dst[x] = buf[x];
            }
        }
        __syncwarp();
    }
}

template <int ND, int NN>
GatherShape shape_t(bool tri, bool few, int nbmax) {
    GatherShape s;
    if constexpr (ND == 3) {
        s.kern = tri ? (const void*)gather3_kernel<NN, true, false> : (const void*)gather3_kernel<NN, false, false>;
        if constexpr (Gather3<NN>::FEW)
            if (few) s.kern = tri ? (const void*)gather3_kernel<NN, true, true> : (const void*)gather3_kernel<NN, false, true>;
        s.rows = Gather3<NN>::ROWS;
    } else {
        s.kern = tri ? (const void*)gather2_kernel<NN, true> : (const void*)gather2_kernel<NN, false>;
        s.rows = 32 / NN;
    }
    const int warp_bytes = s.rows * std::max(nbmax, 1) * ND * ND * 8;
    s.wpb = std::max(1, std::min(GATHER_WARPS, GATHER_SMEM / warp_bytes));
    s.smem = s.wpb * warp_bytes;
    return s;
}

}  // namespace

namespace pms {

GatherShape gather_shape(int kind, bool triangle, bool few, int nbmax) {
    switch (kind) {
    case PMS_TRI3: return shape_t<2, 3>(triangle, few, nbmax);
    case PMS_TRI6: return shape_t<2, 6>(triangle, few, nbmax);
    case PMS_QUA4: return shape_t<2, 4>(triangle, few, nbmax);
    case PMS_QUA8: return shape_t<2, 8>(triangle, few, nbmax);
    case PMS_QUA9: return shape_t<2, 9>(triangle, few, nbmax);
    case PMS_TRI10: return shape_t<2, 10>(triangle, few, nbmax);
    case PMS_TRI15: return shape_t<2, 15>(triangle, few, nbmax);
    case PMS_TET4: return shape_t<3, 4>(triangle, few, nbmax);
    case PMS_TET10: return shape_t<3, 10>(triangle, few, nbmax);
    case PMS_HEX8: return shape_t<3, 8>(triangle, few, nbmax);
    default: return shape_t<3, 20>(triangle, few, nbmax);
    }
}

}  // namespace pms

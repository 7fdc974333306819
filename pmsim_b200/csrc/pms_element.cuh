// pms_element.cuh -- what the element kernels share: their arguments, the error keys and the inverse of
// the Jacobian matrix.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "pms_device.cuh"

struct pms_elements;

namespace pms {

constexpr unsigned FULL = 0xffffffffu;

// Modes of the element kernel
// UPD_MODE: the mode comes at run time from the cell's problem (batched solver):
//   0 = inactive (cell skipped), 1 = step start: assemble from the current state with lambda = 0
//   and copy it to the backup, 2 = update from the backup with ddu, then assemble.
enum { UPD_NONE = 0, UPD_CURRENT = 1, UPD_BACKUP = 2, UPD_MODE = 3 };

struct ElemArgs {
    int64_t ncell;     // cells in this launch
    int64_t cell0;     // first cell of this launch
    int axisym = 0;    // 2D axisymmetric idealization (x = radius)
    bool overlap = false;  // host side: launch beside the end of the previous kernel (launch_overlapped)
    int64_t* grid = nullptr;  // host side: receives the blocks launched
    int64_t nip;       // total IPs of the mesh (SoA stride)
    int ngauss;
    double thickness;
    const double* coords;   // npoint*nd
    const int32_t* conn;    // ncell_total*nn
    const int32_t* cmat;    // per-cell material (nullable)
    const MatConst* mats;
    const double* ddu;      // ndof
    const double* tab;      // dN[ngauss][nn][nd], then w[ngauss], then N[ngauss][nn] (axisymmetric)
    // IP state, SoA with stride nip: sig[c*nip + ip]
    const double* sig_src; const double* z_src; const double* lam_src; const uint8_t* el_src;
    double* sig; double* z; double* lam; uint8_t* el;
    double* fe;   // [cell][nn][nd]
    double* ke;   // [cell][NE][NE] dense element matrices
    unsigned long long* errkey;  // error key of the failing IP the reference would report (0: none)
    unsigned long long* prob_err = nullptr;  // UPD_MODE (nullable): the same key per problem
    const int32_t* cell_prob = nullptr;  // UPD_MODE: problem of each cell
    const uint8_t* pmode = nullptr;      // UPD_MODE: mode of each problem
    // work queue (nq > 0): the launch covers ncell queued cells, range k from q_first[k]
    int32_t nq = 0;
    const int64_t* q_off = nullptr;
    const int64_t* q_first = nullptr;
    // dense outputs (no CSR): the fe / ke rows of cell c are c - ke_cell0
    int64_t ke_cell0 = 0;
    // ke layout: 0 = full row-major NE x NE (per-cell calls); 1 = the upper node-pair blocks (a <= b)
    // only, row by row, each ND x ND block contiguous (upper_entry): NN(NN+1)/2 blocks per cell (the
    // gather assembly)
    int ke_upper = 0;
    // direct assembly (CSR kernels): cell c adds its node-row slab a into block row A = conn[c][a]
    // and its F_int share into R once ticket[A] equals c's rank among A's cells (crank), then
    // advances the ticket; cells are taken in ascending order from the counter `next`
    const int64_t* bptr = nullptr;       // block-row pointers [npoint + 1]
    const int16_t* cslot = nullptr;      // [cell][a][b]: column slot of node b in block row conn[a]
    const int32_t* crank = nullptr;      // [cell][a]: rank (bits 0..29), last-cell flag (bit 30)
    const uint32_t* cfirst = nullptr;    // [cell][a] bit b: first contribution to block (conn[a], conn[b])
    const int32_t* order = nullptr;      // direct assembly: the k-th dequeued position takes cell order[k]
    int32_t* ticket = nullptr;           // [npoint]: slabs of this launch already added to the row
    unsigned long long* next = nullptr;  // in-order work counter, zero at launch
    double* csr = nullptr;               // CSR values of K (DOK)
    double* ff = nullptr;                // R = F_int (DOF)
};

// Which failing IP is reported.  The reference stops at the first error of its loops: the stress
// update of every cell (Elements::update_secondary_values) runs before any tangent
// (Elements::assemble_kke), and each loop goes through the cells and their IPs in ascending order
// (src/fem/elements.rs:156-181).  A failing IP offers the key
//   rank << 56 | (2^40 - 1 - cell) << 16 | (255 - ip) << 8 | code
// (rank 2: update error, 1: tangent/assembly error) and atomicMax keeps the one the reference
// would return: update errors first, then the lowest cell, then its lowest IP.
constexpr int RANK_ORDER = 3, RANK_UPDATE = 2, RANK_TANGENT = 1;
__host__ __device__ constexpr unsigned long long error_key(int rank, int64_t cell, int ip, int code) {
    return ((unsigned long long)rank << 56) | ((((1ull << 40) - 1) - (unsigned long long)cell) << 16) |
           ((unsigned long long)(255 - ip) << 8) | (unsigned long long)(code & 0xff);
}
__device__ __forceinline__ void report(const ElemArgs& A, int rank, int code, int64_t cell, int ip) {
    if (code == OK) return;
    const unsigned long long k = error_key(rank, cell, ip, code);
    atomicMax(A.errkey, k);
    if (A.prob_err && A.cell_prob) atomicMax(A.prob_err + A.cell_prob[cell], k);
}

template <int ND>
__device__ __forceinline__ double inv_jacobian(const double* J, double* Ji) {
    if (ND == 2) {
        double det = J[0] * J[3] - J[1] * J[2];
        double id = 1.0 / det;
        Ji[0] = J[3] * id;
        Ji[1] = -J[1] * id;
        Ji[2] = -J[2] * id;
        Ji[3] = J[0] * id;
        return det;
    } else {
        double c0 = J[4] * J[8] - J[5] * J[7];
        double c1 = J[5] * J[6] - J[3] * J[8];
        double c2 = J[3] * J[7] - J[4] * J[6];
        double det = J[0] * c0 + J[1] * c1 + J[2] * c2;
        double id = 1.0 / det;
        Ji[0] = c0 * id;
        Ji[1] = (J[2] * J[7] - J[1] * J[8]) * id;
        Ji[2] = (J[1] * J[5] - J[2] * J[4]) * id;
        Ji[3] = c1 * id;
        Ji[4] = (J[0] * J[8] - J[2] * J[6]) * id;
        Ji[5] = (J[2] * J[3] - J[0] * J[5]) * id;
        Ji[6] = c2 * id;
        Ji[7] = (J[1] * J[6] - J[0] * J[7]) * id;
        Ji[8] = (J[0] * J[4] - J[1] * J[3]) * id;
        return det;
    }
}

// Blocks of a kernel that the GPU holds at once with `smem` bytes of shared memory a block, looked up (and
// the kernel's attributes set) once per handle, kernel and size (pms_elements.cu).
int64_t launch_plan(pms_elements* h, const void* kern, int smem, int threads, bool max_shared = true);

// 3D cells of few nodes, several to a warp, into the upper layout of the gather assembly
// (pms_elements3.cu).  Returns false where the kind or its rule does not fit; upd: UPD_NONE,
// UPD_CURRENT or UPD_BACKUP.
bool launch_elements3(pms_elements* h, int kind, const ElemArgs& a, int upd, bool dof, bool dok, cudaStream_t stream);

}  // namespace pms

// pms_gather.h -- row gather of the element matrices into the CSR values of K and into R
// (pms_gather.cu), and the layout of the element matrices it reads.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pms {

// Programmatic dependent launch: the kernels of a batched call (element kernel, then gather) let the
// next one's blocks start as soon as their own have, and wait for the previous kernel to finish
// before they touch its results, so that launch and start-up overlap its end.  What they read of them
// they read by ordinary loads (no __ldg, no const __restrict__).  Both are no-ops after an ordinary launch.  Only where the gather is one wave (launch_overlapped's `overlap`): 20x10 Qua8
// step 16.4 -> 11.6 us, 87x48 Qua9 23.8 -> 20.1, 12x10x6 Hex20 51 -> 45; on larger meshes the early gather
// blocks run at the element kernel's shared-memory carveout, where they miss in L1 (701x350 Qua8 526 ->
// 864 us).
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

inline cudaError_t launch_overlapped(bool overlap, const void* kern, int64_t blocks, int threads, int smem,
                                     cudaStream_t stream, void** args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelExC(&cfg, kern, args);
}

// Number of node-pair blocks (a', b'), a' <= b', before block (a, b) of the upper layout.
__host__ __device__ constexpr int upper_block(int nn, int a, int b) { return a * nn - a * (a - 1) / 2 + (b - a); }
// Upper layout of an element matrix: entry (i, j) of block (a, b), a <= b, at
// BB*upper_block(a, b) + i*ND + j.  A block's entries are contiguous, so the row gather reads block
// (a, b) and the transpose of block (b, a) alike: whole runs of blocks on the one side, 72 (32 in 2D)
// contiguous bytes on the other.
template <int NN, int ND>
__host__ __device__ constexpr int upper_entry(int a, int b, int i, int j) {
    return ND * ND * upper_block(NN, a, b) + i * ND + j;
}

struct GatherArgs {
    int64_t node0, nrow;  // block rows [node0, node0 + nrow)
    int nbmax;            // largest block row
    const int64_t* bptr;
    const int64_t* inc_ptr;
    const int32_t* inc;   // incidences of a node, ascending cells: cell*nn + local node
    const int16_t* slot;  // [k*nn + b]: column slot of local node b of incidence k in the block row
    const double* ke;     // [cell][upper layout]
    const double* fe;     // [cell][node][ND]
    double* csr;
    double* ff;  // nullable: no R
    // triangle storages (sym = PMS_SYM_LOWER: columns <= row, PMS_SYM_UPPER: columns >= row;
    // src/base/assembly.rs:92-122): the other entries are not written out, and row (A, i) starts at
    // tbase[A] plus the lengths of rows (A, 0..i-1); kdiag[A] = A's own position in its block row
    int sym;
    const int32_t* kdiag;
    const int64_t* tbase;
};

// Kernel and launch shape of an element kind's gather; few: the kernel for calls whose rows are all in
// flight at once, where the kind has one (Tet4, Hex8, Hex20).
struct GatherShape {
    const void* kern;
    int rows;  // block rows per warp
    int wpb;   // warps per block
    int smem;  // bytes per block
};
GatherShape gather_shape(int kind, bool triangle, bool few, int nbmax);

}  // namespace pms

// pms_gather.h -- row gather of the element matrices into the CSR values of K and into R
// (pms_gather.cu), and the layout of the element matrices it reads.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pms {

// Programmatic dependent launch: the kernels of a batched call (element kernel, then gather) may start up beside
// the end of the one before and wait for it to finish before they touch its results, so that launch and start-up
// overlap its end.  What they read of them they read by ordinary loads (no __ldg, no const __restrict__).  The
// wait and the signal are no-ops after an ordinary launch.  Where the gather is one wave (launch_overlapped's
// `overlap`; the slabs of a host-array call each by its own size).
//
// When the next kernel may start: an element kernel gives no signal, so its gather starts as its last blocks leave;
// a gather signals once its own wait is over, and only where its blocks and the element kernel's fit the SMs side by
// side (GatherArgs::signal).  A signal before the wait lets a row of future calls settle on the SMs: they take the slots of
// the running kernel unevenly, and gathers among them run at the element kernel's shared-memory carveout, where they miss in
// L1.  Calls in a row, us, plain launches | signals before the waits | here: step of 20x10 Qua8 16.5 | 11.6 | 11.0, 60x45
// 18.5 | 20.0 | 13.9; 9x8x8 Hex20 39.1 | 45.0 | 35.2; 9x8x8 Hex8 22.6 | 21.6 | 18.0, 11x10x10 22.6 | 28.7 | 18.4; 16x15x15
// Tet4 43.1 | 46.4 | 39.1, without K 25.9 | 43.0 | 21.5.  A gather's signal above that line: 9x8x8 Hex20 43.1 in place of
// 35.2, 60x45 Qua8 16.8 and 13.9; none below it: 4x3x3 Hex20 30.4 in place of 28.2, 20x10 Qua8 11.5 and 11.0.
// (predicated, not a branch, and no memory clobber: the signal publishes nothing, and either would keep the compiler from
// scheduling the loads around it, 1 us of a 2D step)
__device__ __forceinline__ void let_next_start(int signal) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p griddepcontrol.launch_dependents;\n\t}" ::"r"(signal));
}
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
    int signal;  // let the next kernel's blocks start beside this one's
    // triangle storages (sym = PMS_SYM_LOWER: columns <= row, PMS_SYM_UPPER: columns >= row;
    // src/base/assembly.rs:92-122): the other entries are not written out, and row (A, i) starts at
    // tbase[A] plus the lengths of rows (A, 0..i-1); kdiag[A] = A's own position in its block row
    int sym;
    const int32_t* kdiag;
    const int64_t* tbase;
};

// Kernel and launch shape of an element kind's gather; few: the kernel for calls whose rows are all in
// flight at once, where the kind has one (Tet4, Hex8).
struct GatherShape {
    const void* kern;
    int rows;  // block rows per warp
    int wpb;   // warps per block
    int smem;  // bytes per block
};
GatherShape gather_shape(int kind, bool triangle, bool few, int nbmax);

}  // namespace pms

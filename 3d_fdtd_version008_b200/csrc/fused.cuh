// fused.cuh -- one launch per time step: H and E of every cell in one pass over the grid.
//
// FP32 and FP64 solves of a size that gains from it (Solver's rule) take this step.  The two sweeps
// (kernels.cuh) read and write E and H in place, so a step reads E and H from
// memory twice.  Here a step reads the fields from one copy and writes them to another: a block
// can then recompute the H it needs of its neighbours' cells (the row below, the column to the
// left, the plane below) from values nobody overwrites, and E and H are read once and written
// once per step.  The second copy is shared by the handles of a device (IdleCopies in solver.cu).
//
// A block owns TY rows of a tile of u vectors in x and marches in +z through a chunk of planes.
// Warp w holds row j0 - 1 + w: warp 0 the row below the tile (H only), warps 1 .. TY the owned
// rows.  Lane l holds vector (tile's first vector) + l - 1: lane 0 recomputes H of the column to the
// left, the lane after the owned vectors only lends its E to the x-difference.  Planes arrive by
// TMA: position m of a ring of NS stages holds E of plane k0 + m and H of plane k0 + m - 1, three
// components in one box each, zero-filled outside the grid.  In each plane
//   H:  every warp computes H^{n+1/2} of its row from the staged planes, keeps it in registers
//       and puts Hx and Hz into the stage in place of the old ones, where the next row's warp
//       reads them;
//   E:  once the row below is ready (an mbarrier per row; no block barrier), the owning warps
//       compute E^{n+1} from H in registers, the row below's from the stage, the column's by
//       shuffle, the plane's from the previous iteration.
// Warp 0 refills a stage when every warp has read it.
//
// What bounds it: 24 (FP32) bytes are read and 24 written per cell and step, so HBM is the floor; the
// copies in flight (two blocks of 26 KB stages, two planes ahead) and the 16 warps' instruction
// latencies keep it at 0.81 (FP64) and 0.73 (FP32) of the measured copy bandwidth on 536^3.  Hence everything
// a plane waits for comes from shared memory (coefficients, material rows) or is asked for
// one plane ahead (psi, row numbers: L2 prefetch), FP32 arithmetic runs on pairs of cells, and
// the kernel has to fit 128 registers exactly: with the shared memory in use L1 holds next to
// nothing, and a spilled value costs an L2 trip (a build with 100 spilled bytes ran 15 - 30 % slower).
// Against the two sweeps it is measured, size by size, at Solver's rule (setup_fused in solver.cu).
//
// psi_H is needed by the blocks that recompute a neighbour's H too, so it also alternates
// between two copies; psi_E, P (two slots already), Nu and Ng are touched by their owner alone.
#pragma once

#include "kernels.cuh"

#include <cuda.h>

namespace fdtdk {

struct FusedGeom {
    int u;       // vectors a tile owns in x
    int gx, gy;  // tiles in x, in y
    int kc;      // planes per chunk
    int nrow;    // material rows
    unsigned wait_ns;  // bound on one wait in the kernel, below 2^31
    int hold;    // 1: the row-ready barriers never complete, so that the waits on them run out
};

template <typename T>
struct FusedShape {
    static constexpr int W = Vec<T>::W;
    // Owned rows per block: with the row below 8 warps, two blocks of which leave 128 registers
    // per thread (9 warps: 96, as a scheduler then holds up to 5 of the 18).
    static constexpr int TY = 7;
    static constexpr int NS = 4;          // stages
    static constexpr int kMaxKc = 64;     // planes per chunk: at most
    static constexpr int kRows = sizeof(T) == 8 ? 64 : 128;  // material rows held in shared memory: at most
    static constexpr int LH = 1;       // lanes before the owned ones
    static constexpr int kMaxU = 30;   // owned vectors: at most 32 - LH - 1, and
    static constexpr int kAlignU = 2;  // whole 32-byte sectors
    static constexpr int XW = 32 * W;                     // elements of a staged row
    static constexpr unsigned EB = 3 * (TY + 2) * XW * sizeof(T);
    static constexpr unsigned HB = 3 * (TY + 1) * XW * sizeof(T);
    static constexpr unsigned STAGE = EB + HB;
    static constexpr int kWarps = TY + 1;
    static constexpr int kThreads = 32 * kWarps;
    static constexpr unsigned XCO = 6 * XW * sizeof(T);  // coefficients along x
    static constexpr size_t bytes() { return size_t(NS) * STAGE + XCO + (6 * (TY + 2 + kMaxKc + 1) + 4 * kRows) * sizeof(T); }
    static_assert(EB % 128 == 0 && HB % 128 == 0, "TMA destinations start on 128 bytes");
};

// The psi_H arrays of the copy being read.
template <typename T>
struct PsiOld {
    const T* p[6];
};

template <typename T>
using FusedKernel = void (*)(const CUtensorMap, const CUtensorMap, const StepArgs<T, T>, const PsiOld<T>, const FusedGeom,
                             const ESrc, unsigned*);
// The fused step in FP32 or FP64, with or without plane-wave sheets.  Instantiated in fused.cu.
template <typename T>
FusedKernel<T> fused_kernel(bool sheets);

}  // namespace fdtdk

// Arguments and launch of the persistent incompressible loop (nsi_loop.cu).
#pragma once

#include "loop.cuh"
#include "nsi_ops.cuh"

namespace gb {

// One cell per thread.  Up to kNsiWide threads per block all of a cell's
// neighbours are gathered at once and its face normals stay in shared memory.
constexpr int kNsiWide = 256;
constexpr int kNsiMax = 512;

struct NsiLoopArgs : LoopArgs {
    MeshDev m;
    const float4* ghost_off;              // per ghost: its face centre - its centroid
    float* p[2];
    float4* u[2];
    float* err;
    NsiGhostTable ghosts;
    NsiParams par;
    int limited;
    TagRec* state[2];                     // 2 per cell and buffer: (p, u, v), (w)
    TagRec* grad;                         // 6 per cell: gradients of p, u, v, w; with limiters (p, u, v), (w)
};

constexpr int kNsiGradRecs = 6;

// shared memory of a block (bytes)
constexpr int nsi_loop_smem(int max_faces, int threads) {
    return threads * ((threads <= kNsiWide ? 56 : 40) * max_faces + 28);
}

cudaError_t launch_nsi_loop(NsiLoopArgs& a, int max_faces, int threads, cudaStream_t s);

}  // namespace gb

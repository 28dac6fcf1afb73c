// Arguments and launch of the persistent Euler loop (euler_loop.cu).
#pragma once

#include "loop.cuh"

namespace gb {

struct EulerLoopArgs : LoopArgs {
    MeshDev m;
    const float4* ghost_off;              // per ghost: its face centre - its centroid
    float* rho[2];
    float4* rhou[2];
    float* rhoe[2];
    float* rec_rho;
    float4* rec_rhou;
    float* err;
    GhostBcTable ghosts;
    float cfl;
    TagRec* state[2];                     // 2 per cell and buffer: (rho, u, v), (w, E)
    TagRec* rec;                          // 2 per entry: (rho, u, v), (w, E)
};

// One instance of a batch in the batched loop: its own workers and reducer,
// and what k_batch_reduce keeps of it.
struct BatchLoopInst : EulerLoopArgs {
    int first_block;                      // workers [first_block, first_block + n_blocks), then the reducer
    int max_iter;
    double res0_fixed;
    int *cur, *status, *n_iters;
    double *res0, *ratio, *history;       // history may be null
};

void launch_ghost_off(const DevMesh& d, float4* ghost_off, cudaStream_t s);
// form: loop_form(max_faces, threads)
cudaError_t launch_euler_loop(EulerLoopArgs& a, LoopForm form, int max_faces, int threads, bool transposed,
                              cudaStream_t s);
// blocks: of the grid; inst_of_block: the instance of each.  WIDE or NARROW.
cudaError_t launch_batch_loop(const BatchLoopInst* insts, const int* inst_of_block, int blocks, LoopForm form,
                              int max_faces, int threads, bool transposed, cudaStream_t s);

MeshDev mesh_dev(const DevMesh& m);

}  // namespace gb

// The scans behind ssm_scan, gated_scan and delta_scan that run as register-tiled walks (see scan_walk.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace dlmk {

enum WalkMode : int { WALK_HEAD = 0, WALK_CHANNEL = 1, WALK_DELTA = 2, WALK_REMOVE = 3 };

// Rows of q, k, v, ... are `ld*` floats apart.  q and k hold the heads / q_div query heads of N entries side by side, v and o
// the heads of P entries; `dec` is a number a head (WALK_HEAD, WALK_DELTA) or N numbers a head (WALK_CHANNEL, WALK_REMOVE).
struct WalkParams {
    const float* q; int ldq;
    const float* k; int ldk;
    const float* v; int ldv;
    const float* dec; int ldd;
    const float* beta; int ldb;          // WALK_DELTA: raw write strength a head
    const float* rate; int ldr;          // WALK_REMOVE: raw removal rate, N numbers a head
    const float* rate_bias;              // WALK_REMOVE: [heads * N]
    const float* A_log; const float* dec_bias; const float* D; const float* fixed_decay;     // [heads] or nullptr
    float* state;                        // [slots, heads, N, P]
    const int32_t* cu_q; const int32_t* state_slot;
    float* o; int ldo;
    int heads, q_div, N, P;
    int silu_inputs, unit;
    float unit_eps, q_scale, inv_tau, decay_coef;
    int longest;                         // tokens of the step's longest request, or a bound of it; 0: not known
    int wide, wide_v, state_vec, walkers, tile;      // filled in by scan_walk: 16-byte copies are possible (of the vectors, of
                                         // v), a lane's columns of the state come as one access; warps that walk; tokens a tile
};

// False when the sizes are not its: the caller takes the kernel it has for any size.
bool scan_walk(int mode, WalkParams p, int R, cudaStream_t stream);

}  // namespace dlmk

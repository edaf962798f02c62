// Batched routed-expert GEMMs on the 5th-generation tensor cores (tcgen05, accumulators in tensor memory).
//
// For every expert e with its n_e tokens (pairs sorted by expert, "slots"):
//   up   : G[h, t] = W1_e[h, :] . x_t,  U[h, t] = W3_e[h, :] . x_t,  mid[slot, h] = silu(G) * U
//   down : y[slot, o] = w_pair * W2_e[o, :] . mid[slot, :]
// Weights are the MMA's A operand, tokens its B operand, so a weight tile is read from HBM once for all tokens of the tile.
#pragma once

#include "moe_prep.cuh"
#include "stream_ring.cuh"
#include "tc05.cuh"

#include <cuda.h>

namespace dsv4 {

}  // namespace dsv4

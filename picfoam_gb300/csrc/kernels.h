// kernels.h -- host-side declarations of the kernel launchers.
#pragma once

#include "common.cuh"

namespace pgd {

cudaError_t move_fp64_set_tables(const TetConst& t, const PatchConst& p);
void launch_move_fp64(const MoveParams& P, int sms, cudaStream_t s);
// Blocks per SM of the FP32 mover outside of graphs, three rounds of the five
// that are resident: the chunks differ in their faces crossed, and with one
// round the SMs idled 11 % of the time at its end.  26 million parcels: 549 us a
// step with 5, 522 with 15 (and a deposit window of 512 cells, not 768: a
// third of the chunk); 3.3 million that cross many cells: 965 and 812 us.
constexpr int kMoveBlocks32 = 15;
// Returns the number of kernels launched (in-cell mover + crossing tracker, or
// the general kernel).
int launch_move_fp32(const MoveParams& P, int grid, cudaStream_t s);
// Velocity push of every live particle by tt without tracking (FP64 or FP32 store).
void launch_push_only(const MoveParams& P, bool fp32, double tt, int grid, cudaStream_t s);

}  // namespace pgd

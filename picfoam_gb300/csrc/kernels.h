// kernels.h -- host-side declarations of the kernel launchers.
#pragma once

#include "common.cuh"

namespace pgd {

cudaError_t move_fp64_set_tables(const TetConst& t);
void launch_move_fp64(const MoveParams& P, int sms, cudaStream_t s);
// Blocks per SM of the FP32 mover outside of graphs: 5, which are resident, or
// three rounds of them.  The chunks differ in the faces that their parcels
// cross, and with one round the SMs idle at its end; but each block clears and
// flushes its deposit window once more.  Three rounds pay from some 11 million
// parcels on (72,000 per SM), and for fewer where they cross many faces: `faces`
// are those of this species' last step, 0 when there is none.  A pass of ten
// steps with 5 and 15 blocks, 0.22 faces per parcel: 1.0 million 801 and 911 us
// (16 per cell), 3.0 million 1915 and 2117 (8 per cell), 12 million 6654 and
// 6369, 26 million 7115 and 6985 (100 per cell).  One million with 5.7 faces
// each 595 and 619 us in 5 steps, with 21 822 and 774; 0.3 million with 21 399
// and 431, with 83 617 and 619.
int move_blocks32(long parcels, double faces, int sms);
// Returns the number of kernels launched (in-cell mover + crossing tracker, or
// the general kernel).
int launch_move_fp32(const MoveParams& P, int grid, cudaStream_t s);
// Velocity push of every live particle by tt without tracking (FP64 or FP32 store).
void launch_push_only(const MoveParams& P, bool fp32, double tt, int grid, cudaStream_t s);

}  // namespace pgd

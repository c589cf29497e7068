// move_fp64.cu -- FP64 (exact) form of the fused push + track + deposit.
// Built with --fmad=false: every product and sum rounds on its own, in the
// evaluation order of the CPU oracle, so the two agree bit for bit.
#include <algorithm>

#include "kernels.h"
#include "move_impl.cuh"

namespace pgd {

__constant__ TetConst c_tet64;

// An FP64 warp instruction holds its quarter of an SM for 64 cycles whether one
// lane needs it or all, so the mover is bound by the number of FP64 warp
// instructions.  A warp therefore takes chunks of up to kMoveChunk particles
// through three passes of full warps: push (velocities written back), track,
// deposit.  In the track pass a lane whose particle has arrived takes the next
// one of the chunk; with one particle per lane from push to deposit 18 of 32
// lanes tracked on average (electrons of a 25 x 23 x 21 plasma).  Compares,
// sign tests and the choice of the face are done on the integer pipe.
// Four steps of 2 x 483,000 particles with the Vay pusher: 3.7 ms, 4.5 ms with
// one particle per lane and four divisions per tet step; the FP64 pipe is the
// bound, half of it in the pusher's roots and divisions.
constexpr int kMoveWarps = 4;        // per block
constexpr int kMoveBlocks = 3;       // per SM
constexpr int kMoveChunk = 512;      // particles of a warp per round at most
constexpr int kRefill = 6;           // idle lanes that make a warp fetch particles

// The smallest double whose square root rounds to c or above.
constexpr double kSpeedLimit = 0x1.3f4d4eacdd756p+56;

__device__ __forceinline__ unsigned long long bits(double x) {
    return (unsigned long long)__double_as_longlong(x);
}

// About y / |d| in FP32, good to 2^-18 for normal operands; 0 where y or d is
// subnormal or y is not positive, below 2^-98 where the quotient is below
// 2^-99, at least 1.9 where it is above 4.
__device__ __forceinline__ float rough_ratio(double y, double d) {
    const int hy = __double2hiint(y), hd = __double2hiint(d) & 0x7fffffff;
    const int ey = hy >> 20, ed = hd >> 20;
    const float my = __int_as_float(0x3f800000 | (hy & 0xfffff) << 3);
    const float md = __int_as_float(0x3f800000 | (hd & 0xfffff) << 3);
    const float q = __fdividef(my, md) * __int_as_float((127 + min(max(ey - ed, -100), 2)) << 23);
    return (ey > 0 && ed > 0) ? q : 0.f;
}

// The first barycentric coordinate to reach zero along dy: the smallest
// -y[i] / dy[i] < 1 over dy[i] < thr, the lowest i among equals; -1 if none.
// FP32 quotients leave the one or two faces that can be it, so a step costs
// one FP64 division instead of up to four (some 600 cycles each).
__device__ __forceinline__ int first_face(const double (&y)[4], const double (&dy)[4], double thr, double* lam_out) {
    float q[4];
    unsigned cand = 0;
    float cut = 1.f;
    // thr = -1e-12 S is negative (or -0), so dy < thr is an unsigned compare
    // of the bits, unless S is NaN: then nothing is below it
    const bool number = (bits(thr) << 1) <= 0xffe0000000000000ull;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        q[i] = 4.f;
        if (number && bits(dy[i]) > bits(thr)) {
            q[i] = rough_ratio(y[i], dy[i]);
            cut = fminf(cut, q[i]);
            cand |= 1u << i;
        }
    }
    cut = cut * (1.f + 0x1p-16f) + 0x1p-97f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (!(q[i] <= cut)) cand &= ~(1u << i);
    double lam = 1.0;
    int hit = -1;
    while (cand) {
        const int i = __ffs(cand) - 1;
        cand &= cand - 1;
        const double yi = i < 2 ? (i == 0 ? y[0] : y[1]) : (i == 2 ? y[2] : y[3]);
        const double di = i < 2 ? (i == 0 ? dy[0] : dy[1]) : (i == 2 ? dy[2] : dy[3]);
        const double l = -yi / di;
        if (l < lam) {
            lam = l;
            hit = i;
        }
    }
    *lam_out = lam;
    return hit;
}

// One tet step: barycentric displacement, first coordinate to reach zero,
// clamp and renormalise.  Returns the hit tet face or -1.
__device__ __forceinline__ int tet_step(const MoveParams& P, PState<double>& s, const double (&dx)[3],
                                        double* lam_out) {
    const double* inv = P.m.tetinv + (size_t(P.m.cell_class[s.cell]) * 12 + s.tet) * 9;
    double dy[4];
    dy[1] = inv[0] * dx[0] + inv[1] * dx[1] + inv[2] * dx[2];
    dy[2] = inv[3] * dx[0] + inv[4] * dx[1] + inv[5] * dx[2];
    dy[3] = inv[6] * dx[0] + inv[7] * dx[1] + inv[8] * dx[2];
    dy[0] = -(dy[1] + dy[2] + dy[3]);
    const double S = fabs(dy[0]) + fabs(dy[1]) + fabs(dy[2]) + fabs(dy[3]);
    double lam;
    const int hit = first_face(s.y, dy, -1e-12 * S, &lam);
    double y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double v = s.y[i] + lam * dy[i];
        // max(v, 0), 0 for a NaN
        y[i] = i != hit && bits(v) - 1 < 0x7ff0000000000000ull ? v : 0.0;
    }
    const double r = 1.0 / (y[0] + y[1] + y[2] + y[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) s.y[i] = y[i] * r;
    *lam_out = lam;
    return hit;
}

__device__ __forceinline__ void sync_velocity(const MoveParams& P, const TetConst& T, PState<double>& s,
                                              double fraction) {
    if (P.sync && P.charged && s.zf != 0.0) push(P, T, s, fraction * P.dt);
}

// PICParcel::hitPatch (PICParcel.C:153-184) for the patch models in scope.
// False: the parcel is removed.  *resync: its velocity was taken to the time
// of the hit.
__device__ __forceinline__ bool hit_patch(const MoveParams& P, const TetConst& T, PState<double>& s, int patch,
                                          double sf, unsigned* walls, bool* resync) {
    const int kind = P.m.patches->kind[patch];
    if (kind == PICGPU_PATCH_ABSORB) return false;
    // FloatingPotential deletes every parcel; a circuit electrode
    // (circuitRLC.C:268-288) deletes charged parcels and reflects neutral ones
    if (kind == PICGPU_PATCH_FLOATING || (kind == PICGPU_PATCH_CIRCUIT && P.q != 0.0)) {
        atomicAdd(P.qconv + patch, P.p.nw ? s.nw * (P.q * s.zf) : P.weight * P.q);
        return false;
    }
    const int f = s.tet / 2;
    const double* n = P.m.fnormal + size_t(P.m.cell_class[s.cell]) * 18 + 3 * f;
    if (kind == PICGPU_PATCH_WALL || kind == PICGPU_PATCH_CIRCUIT) {
        sync_velocity(P, T, s, sf - 0.5);
        (*walls)++;
        *resync = true;
    }
    const double Un = s.U[0] * n[0] + s.U[1] * n[1] + s.U[2] * n[2];
    if (Un > 0.0) {
        const double t = 2.0 * Un;
        s.U[0] = s.U[0] - t * n[0];
        s.U[1] = s.U[1] - t * n[1];
        s.U[2] = s.U[2] - t * n[2];
    }
    return true;
}

__device__ __forceinline__ void deposit_add(const MoveParams& P, double* dst64, long long* dstfix, size_t idx,
                                            double v) {
    if (P.deposit_mode == PICGPU_DEPOSIT_FIXED_POINT) {
        const long long q = __double2ll_rn(v * P.fix_scale);
        atomicAdd(reinterpret_cast<unsigned long long*>(dstfix + idx), (unsigned long long)q);
    } else {
        atomicAdd(dst64 + idx, v);
    }
}

// ChargeDistribution::add for one particle at its end-of-step position.
__device__ __forceinline__ void deposit(const MoveParams& P, const TetConst& T, const PState<double>& s) {
    // charge x nParticle of the parcel (VolumeWeighting.C:114)
    const double value = P.p.nw ? P.q * s.zf * s.nw : P.value;
    if (value == 0.0) return;
    if (P.charge_distribution == PICGPU_WEIGHTING_CELL_AVERAGE) {
        deposit_add(P, P.cc_data, P.cc_fix, s.cell, value);
        return;
    }
    const int* cp = P.m.cell_pt + 8 * size_t(s.cell);
    deposit_add(P, P.cc_data, P.cc_fix, s.cell, s.y[0] * value);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        deposit_add(P, P.vtx_data, P.vtx_fix, cp[T.tri[s.tet][i]], s.y[i + 1] * value);
}

__device__ __forceinline__ void load_place(const MoveParams& P, int i, int tetg, PState<double>& s) {
    s.cell = tetg / 12;
    s.tet = tetg - 12 * s.cell;
#pragma unroll
    for (int a = 0; a < 3; ++a) s.y[1 + a] = P.p.y64[a][i];
}

__device__ __forceinline__ void load_velocity(const MoveParams& P, int i, PState<double>& s) {
#pragma unroll
    for (int a = 0; a < 3; ++a) s.U[a] = P.p.u64[a][i];
}

__device__ __forceinline__ void store_velocity(const MoveParams& P, int i, const PState<double>& s) {
#pragma unroll
    for (int a = 0; a < 3; ++a) P.p.u64[a][i] = s.U[a];
}

// The displacement left at the step fraction sf: PICParcel::move's dt (1 - sf) U
// with the solved directions only and the way back to the mesh's centre plane
// on empty ones.  Returns 1 - sf.
__device__ __forceinline__ double leg(const MoveParams& P, const TetConst& T, const PState<double>& s, double sf,
                                      double (&disp)[3]) {
    double Ut[3] = {s.U[0], s.U[1], s.U[2]};
    double dev[3] = {0.0, 0.0, 0.0};
    if (P.m.any_empty) {
        const double* off = P.m.offset + size_t(P.m.cell_class[s.cell]) * 24;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (!P.m.empty[a]) continue;
            Ut[a] = 0.0;
            const double x = P.m.cc[3 * size_t(s.cell) + a] + s.y[1] * off[3 * T.tri[s.tet][0] + a] +
                             s.y[2] * off[3 * T.tri[s.tet][1] + a] + s.y[3] * off[3 * T.tri[s.tet][2] + a];
            dev[a] = x - P.m.mesh_centre[a];
        }
    }
    const double f = 1.0 - sf;
    const double fdt = f * P.dt;
#pragma unroll
    for (int a = 0; a < 3; ++a) disp[a] = fdt * Ut[a] - dev[a];
    return f;
}

__global__ void __launch_bounds__(32 * kMoveWarps, kMoveBlocks) move_kernel_fp64(MoveParams P, int rounds) {
    __shared__ TetConst T;
    __shared__ double y0[kMoveWarps][kMoveChunk];   // the coordinate that the store leaves out
    for (unsigned k = threadIdx.x; k < sizeof(TetConst); k += blockDim.x)
        reinterpret_cast<char*>(&T)[k] = reinterpret_cast<const char*>(&c_tet64)[k];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* const own_y0 = y0[warp];
    unsigned steps = 0, faces = 0, walls = 0, absorbed = 0;

    // the rows of 32 dealt out evenly: share k of all gets rows [k R / all, (k + 1) R / all)
    const long rows = (long(P.n) - P.first + 31) / 32, all = long(gridDim.x) * kMoveWarps * rounds;
    for (int round = 0; round < rounds; ++round) {
        const long share = (long(round) * gridDim.x + blockIdx.x) * kMoveWarps + warp;
        const int begin = P.first + int(share * rows / all) * 32;
        const int end = min(P.n, P.first + int((share + 1) * rows / all) * 32);

        // push
        for (int i = begin + lane; i < end; i += 32) {
            const int tetg = P.p.tet[i];
            if (tetg < 0) continue;
            PState<double> s;
            load_place(P, i, tetg, s);
            s.y[0] = 1.0 - s.y[1] - s.y[2] - s.y[3];
            own_y0[i - begin] = s.y[0];
            if (!P.solve_movement) continue;
            load_velocity(P, i, s);
            load_attributes(P, i, s);
            // PICParcel::move pushes charged parcels only (PICParcel.C:55)
            if (P.charged && s.zf != 0.0) {
                push(P, T, s, P.dt);
                store_velocity(P, i, s);
            }
            // sqrt(U.U) < c; false for a NaN
            if (bits(dot3(s.U, s.U)) >= bits(kSpeedLimit)) {
                P.p.tet[i] = -1;
                absorbed++;
                atomicMax(&P.counters->error, int(PICGPU_SPEED_OF_LIGHT));
            }
        }
        __syncwarp();

        // track
        if (P.solve_movement) {
            PState<double> s;
            double disp[3], f = 0.0, sf = 0.0, rem = 0.0;
            int i = -1, budget = 0, resyncs = 0, next = begin;
            bool new_leg = false;
            for (;;) {
                const unsigned idle = __ballot_sync(0xffffffffu, i < 0);
                if (idle == 0xffffffffu && next >= end) break;
                if (next < end && __popc(idle) >= kRefill) {
                    if (i < 0) {
                        const int k = next + __popc(idle & ((1u << lane) - 1));
                        const int tetg = k < end ? P.p.tet[k] : -1;
                        if (tetg >= 0) {
                            i = k;
                            load_place(P, i, tetg, s);
                            s.y[0] = own_y0[i - begin];
                            load_velocity(P, i, s);
                            load_attributes(P, i, s);
                            sf = 0.0;
                            resyncs = 0;
                            budget = P.max_steps;
                            new_leg = true;
                        }
                    }
                    next += __popc(idle);
                }
                if (i >= 0) {
                    if (new_leg) {
                        f = leg(P, T, s, sf, disp);
                        rem = 1.0;
                        new_leg = false;
                    }
                    bool keep = true, done = false;
                    if (--budget < 0) {
                        keep = false;
                        atomicMax(&P.counters->error, int(PICGPU_TRACK_LOOP_CAP));
                    } else {
                        const double dx[3] = {rem * disp[0], rem * disp[1], rem * disp[2]};
                        double lam;
                        const int hit = tet_step(P, s, dx, &lam);
                        steps++;
                        done = hit < 0;
                        if (!done) {
                            sf = sf + (f * rem) * lam;
                            int nb = 0;
                            if (hit == 0) {
                                faces++;
                                nb = P.m.nbr[6 * size_t(s.cell) + s.tet / 2];
                            } else {
                                rem = rem * (1.0 - lam);
                            }
                            if (nb >= 0) {
                                // into the next tet of the cell, or the one across the face
                                const int8_t* src = hit == 0 ? T.cross_src[s.tet] : T.inner_src[s.tet][hit];
                                double y[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const int q = src[j];   // negative: zero
                                    y[j] = q < 0 ? 0.0 : q < 2 ? (q == 0 ? s.y[0] : s.y[1]) : (q == 2 ? s.y[2] : s.y[3]);
                                }
                                if (hit == 0) {
                                    y[0] = 0.0;
                                    s.tet = T.cross_next[s.tet];
                                    s.cell = nb;
                                } else {
                                    s.tet = T.inner_next[s.tet][hit];
                                }
#pragma unroll
                                for (int j = 0; j < 4; ++j) s.y[j] = y[j];
                            } else {
                                bool resync = false;
                                keep = hit_patch(P, T, s, -nb - 1, sf, &walls, &resync);
                                if (keep && resync && ++resyncs == 1) sync_velocity(P, T, s, 0.5 - sf);
                                if (keep) store_velocity(P, i, s);
                            }
                            if (hit == 0) {
                                new_leg = true;
                                done = !(sf < 1.0);
                            }
                        }
                    }
                    if (!keep) {
                        P.p.tet[i] = -1;
                        absorbed++;
                        i = -1;
                    } else if (done) {
                        P.p.tet[i] = 12 * s.cell + s.tet;
#pragma unroll
                        for (int a = 0; a < 3; ++a) P.p.y64[a][i] = s.y[1 + a];
                        own_y0[i - begin] = s.y[0];
                        i = -1;
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();

        // deposit
        for (int i = begin + lane; i < end; i += 32) {
            const int tetg = P.p.tet[i];
            if (tetg < 0) continue;
            PState<double> s;
            load_place(P, i, tetg, s);
            s.y[0] = own_y0[i - begin];
            load_attributes(P, i, s);
            deposit(P, T, s);
        }
        __syncwarp();
    }
    warp_add_counter<double>(&P.counters->tet_steps, steps);
    warp_add_counter<double>(&P.counters->faces, faces);
    warp_add_counter<double>(&P.counters->walls, walls);
    warp_add_counter<double>(&P.counters->absorbed, absorbed);
}

// Push only, no tracking, of slots [first, n): initalizeLeapFrog
// (picInitialise.C:219-227) calls the pusher's updateVelocity(p, -dt/2) on
// every parcel, moving or not; an emitted parcel is synchronised the same way
// (ParticleEmitter.C:401, PICParcel.C:220-227).
template <class Real>
__global__ void __launch_bounds__(256) push_only_kernel(MoveParams P, Real tt) {
    for (int i = P.first + blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x) {
        const int tetg = P.p.tet[i];
        if (tetg < 0) continue;
        PState<Real> s;
        s.cell = tetg / 12;
        s.tet = tetg - 12 * s.cell;
        s.y[1] = ybuf<Real>(P.p, 0)[i];
        s.y[2] = ybuf<Real>(P.p, 1)[i];
        s.y[3] = ybuf<Real>(P.p, 2)[i];
        s.y[0] = Real(1) - s.y[1] - s.y[2] - s.y[3];
        s.U[0] = ubuf<Real>(P.p, 0)[i];
        s.U[1] = ubuf<Real>(P.p, 1)[i];
        s.U[2] = ubuf<Real>(P.p, 2)[i];
        load_attributes(P, i, s);
        push<Real>(P, c_tet64, s, tt);
        ubuf<Real>(P.p, 0)[i] = s.U[0];
        ubuf<Real>(P.p, 1)[i] = s.U[1];
        ubuf<Real>(P.p, 2)[i] = s.U[2];
    }
}

void launch_push_only(const MoveParams& P, bool fp32, double tt, int grid, cudaStream_t s) {
    if (fp32) push_only_kernel<float><<<grid, 256, 0, s>>>(P, float(tt));
    else push_only_kernel<double><<<grid, 256, 0, s>>>(P, tt);
}

cudaError_t move_fp64_set_tables(const TetConst& t) { return cudaMemcpyToSymbol(c_tet64, &t, sizeof t); }

void launch_move_fp64(const MoveParams& P, int sms, cudaStream_t s) {
    // as many warps as the chip holds, each with an equal share of the rows of
    // 32, in as many rounds as keep a share within a chunk
    const long rows = (std::max(0L, long(P.n) - P.first) + 31) / 32;
    const long blocks = std::max(1L, std::min((rows + kMoveWarps - 1) / kMoveWarps, long(sms) * kMoveBlocks));
    const long per_round = blocks * kMoveWarps * (kMoveChunk / 32);
    move_kernel_fp64<<<unsigned(blocks), 32 * kMoveWarps, 0, s>>>(P, int((rows + per_round - 1) / per_round));
}

}  // namespace pgd

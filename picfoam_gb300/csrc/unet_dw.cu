// unet_dw.cu -- weight gradients of the warm-start U-Net's 3x3x3 convolutions
// on the 5th-generation tensor cores.
//
//   dW[t][co][ci] += sum_v h[v][co] x[v + off_t][ci]
//
// is a GEMM per tap t with K = voxels: A = h (rows co), B = x shifted by the
// tap (columns ci), FP32 accumulators in TMEM (column blocks dx, then the
// (dz, dy) pairs, then ci).  Both operands are channels-last, i.e. MN-major: an 8-channel group
// of one voxel is one 16-byte row of a core matrix.
//
// The voxels are numbered with one pad column per row and one pad row per
// plane, pos = x + (X + 1) y + (X + 1)(Y + 1) z, where h and x are zero on the
// pads and outside.  A tap is then a constant shift of pos for every voxel,
// and a K-tile of kTile positions needs one staged run of x per (dz, dy) pair
// (kTile + 2 positions); its three dx taps are the same run read one 16-byte
// row apart, which the descriptor's start address expresses.  Rows of A past
// COUT read other staged data and go to accumulator lanes that nobody reads.
//
// FP32 operands (the network input of the first layer, the loss gradient of
// the last) are staged as three BF16 parts whose sum is the FP32 value
// exactly, as channels of their own; the products' sums then meet in FP32 as
// before.
//
// The tensor core truncates when it adds to an accumulator, so a long chain
// drifts: 2.5e-6 of the result over 340 accumulations, 7.5e-6 over 900, where
// the CUDA-core kernel this replaces was 1e-7 to 6e-7 off.  A chain therefore
// ends after kChain tiles (16 accumulations); the warps that can read
// the rows' TMEM lanes add it to FP32 sums in shared memory, rounded to
// nearest.  Measured against 64-bit sums of the same operands, relative error
// here and of the CUDA-core kernel: 16 -> 16 at 64^3 2.2e-7 (6.0e-7), at 128^3
// 2.4e-7 (5.5e-7), 48 -> 16 2.0e-7 (5.7e-7), 64 -> 64 at 16^3 0.9e-7 (1.3e-7),
// 16 -> 1 2.7e-7 (6.4e-7), 2 -> 16 2.8e-7 (5.3e-7).
//
// What bounds it: the loaders' instructions and the MMAs (each reads 4 KB of A
// from shared memory, whatever its N) about equally; x comes 9 times through
// L2.  At 64^3 voxels, against the CUDA-core kernel (which staged both
// operands 27 times): 16 -> 16 46 us (1046), 48 -> 16 125 us (3012), 16 -> 1
// 46 us (544), 2 -> 16 50 us (158); 64 -> 64 at 16^3 18 us (1114).
//
// Loader warps (cp.async, zero-filled on the pads), one MMA warp and the
// draining warps meet at mbarriers; every wait is bounded, and on a timeout
// the kernel raises *err, frees its TMEM and returns.
#include <cuda_bf16.h>

#include <algorithm>

#include "tc.cuh"
#include "unet.h"

namespace pgd {
namespace {

constexpr int kTile = 128;                       // positions per K-tile
constexpr int kRun = kTile + 2;                  // staged positions of one (dz, dy) pair
constexpr int kChain = 2;                        // tiles accumulated in TMEM before they are drained
constexpr int kWarps = 13;
constexpr int kMmaWarp = 12;
constexpr uint32_t kASbo = kTile * 16, kBSbo = kRun * 16, kLbo = 128;

template <int CIN, int COUT>
struct DwShape {
    static_assert(CIN % 16 == 0 && COUT % 8 == 0 && COUT <= 64, "unsupported channel counts");
    // (dz, dy) pairs per CTA: as many as TMEM's 512 columns, and with 64 rows
    // the sums in shared memory, hold
    static constexpr int kFit = COUT > 32 ? 96 / CIN : 512 / (3 * CIN);
    static constexpr int kPairs = kFit < 9 ? kFit : 9;
    static constexpr int kGroups = (9 + kPairs - 1) / kPairs;
    static constexpr int kCols = 3 * kPairs * CIN;
    static constexpr int kABytes = COUT / 8 * int(kASbo);
    static constexpr int kPairBytes = CIN / 8 * int(kBSbo);
    static constexpr int kStage = kABytes + kPairs * kPairBytes;
    // A's 16 channel groups (those past COUT are staged data of no meaning)
    // end within the stage
    static_assert(kStage >= 16 * int(kASbo), "A reads past the stage");
    static constexpr int kAccStride = COUT + 1;
    static constexpr int kBytes = 2 * kStage + kCols * kAccStride * 4;
    // above half of an SM's shared memory: a CTA takes all TMEM columns
    static constexpr int kSmem = kBytes > 120 * 1024 ? kBytes : 120 * 1024;
    static_assert(kSmem <= 227 * 1024, "shared memory");
    // warps w with w % 4 < kQuarters can read the rows' TMEM lanes: they
    // drain; the others, but the MMA warp, load
    static constexpr int kQuarters = COUT > 32 ? 2 : 1;
    static constexpr int kDrainers = 32 * 3 * kQuarters;
    static constexpr int kLoaders = 32 * (kWarps - 1 - 3 * kQuarters);
};

struct DwArgs {
    ConvGrid g;
    const __nv_bfloat16* h;      // [V][COUT] (BF16 form)
    const float* h32;            // [V] (split form)
    ConvSrc s1, s2;              // BF16 input, concatenated
    const float* x32;            // [V][2] (split form)
    float* dw;
    int* err;
};

// v = p[0] + p[1] + p[2], exactly (24 mantissa bits in three BF16 parts).
__device__ __forceinline__ void split3(float v, __nv_bfloat16* p) {
    p[0] = __float2bfloat16_rn(v);
    const float r = v - __bfloat162float(p[0]);
    p[1] = __float2bfloat16_rn(r);
    p[2] = __float2bfloat16_rn(r - __bfloat162float(p[1]));
}

// Voxel of a padded position and its coordinates; -1 on a pad, -2 outside.
__device__ __forceinline__ long voxel_of(int pos, const ConvGrid& g, int R, int P, int total, int* x, int* y, int* z) {
    *x = *y = *z = 0;
    if (pos < 0 || pos >= total) return -2;
    *z = int(unsigned(pos) / unsigned(P));
    const int q = pos - *z * P;
    *y = int(unsigned(q) / unsigned(R));
    *x = q - *y * R;
    if (*x >= g.X || *y >= g.Y) return -1;
    return (long(*z) * g.Y + *y) * g.X + *x;
}

// 16 bytes global -> shared without registers; zeros (the source, a valid
// address all the same, is not read) unless ok.
__device__ __forceinline__ void copy16(void* dst, const __nv_bfloat16* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_addr(dst)), "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}

// XF / HF: the FP32 forms (2 input channels as 6 + 10 zeros; 1 output channel
// as 3 + 5 zeros).
template <int CIN, int COUT, bool XF, bool HF>
__global__ void __launch_bounds__(32 * kWarps) dw_tc_kernel(DwArgs a, int tiles, int per_cta) {
    using S = DwShape<CIN, COUT>;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[2], empty[2], chain_done, drained;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = a.g.X + 1, P = R * (a.g.Y + 1), total = P * a.g.Z;
    const int first = blockIdx.x * per_cta, last = min(tiles, first + per_cta);
    const int pair0 = blockIdx.y * S::kPairs, pairs = min(9 - pair0, S::kPairs);
    if (first >= last) return;   // block-uniform
    const int count = last - first, chains = (count + kChain - 1) / kChain;
    float* const acc = reinterpret_cast<float*>(smem + 2 * S::kStage);   // [column][row]

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(&full[s], S::kLoaders);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(&chain_done, 1);
        tc::mbar_init(&drained, S::kDrainers);
        abort_flag = 0;
        tc::mbar_init_fence();
    }
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    volatile int* aborted = &abort_flag;

    if (warp == kMmaWarp) {
        const uint32_t idesc = tc::idesc_bf16_f32(128, pairs * CIN) | tc::kMnMajorAB;
        for (int i = 0; i < count && lane == 0; ++i) {
            const int s = i & 1, in_chain = i % kChain;
            // the last chain's sums have left TMEM
            if (*aborted || (in_chain == 0 && i > 0 && !tc::mbar_wait(&drained, uint32_t(i / kChain - 1) & 1u)) ||
                !tc::mbar_wait(&full[s], uint32_t(i >> 1) & 1u)) {
                *aborted = 1;
                break;
            }
            tc::fence_after_sync();
            const uint32_t a0 = tc::smem_addr(smem + s * S::kStage), b0 = a0 + S::kABytes;
            // the pairs' channel groups are equally spaced: one MMA per dx
            // and K-step covers them all
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                for (int ks = 0; ks < kTile / 16; ++ks) {
                    const uint64_t ad = tc::smem_desc(a0 + 256u * ks, kLbo, kASbo);
                    const uint64_t bd = tc::smem_desc(b0 + 16u * (16 * ks + dx), kLbo, kBSbo);
                    tc::mma_bf16(tmem + uint32_t(dx * pairs * CIN), ad, bd, idesc, (in_chain > 0 || ks > 0) ? 1u : 0u);
                }
            tc::commit(&empty[s]);
            if (in_chain == kChain - 1 || i == count - 1) tc::commit(&chain_done);
        }
        __syncwarp();
    } else if (warp % 4 < S::kQuarters) {
        // rows 32 (warp % 4) + lane; three warps share the columns
        const int row = 32 * (warp % 4) + lane;
        const uint32_t lane_base = tmem + (uint32_t(32 * (warp % 4)) << 16);
        for (int c = 0; c < chains; ++c) {
            if (!tc::mbar_wait(&chain_done, uint32_t(c) & 1u)) *aborted = 1;
            __syncwarp();
            if (*aborted) break;
            tc::fence_after_sync();
            for (int b = warp / 4; b < 3 * pairs * CIN / 16; b += 3) {
                float v[16];
                tc::tmem_ld16(lane_base + uint32_t(16 * b), v);
                if (row < COUT) {
                    float* p = acc + 16 * b * S::kAccStride + row;
#pragma unroll
                    for (int j = 0; j < 16; ++j) p[j * S::kAccStride] = c == 0 ? v[j] : p[j * S::kAccStride] + v[j];
                }
            }
            tc::fence_before_sync();
            tc::mbar_arrive(&drained);
        }
    } else {
        const int id = ((warp / 4) * (4 - S::kQuarters) + warp % 4 - S::kQuarters) * 32 + lane;
        for (int i = 0; i < count && !*aborted; ++i) {
            const int s = i & 1;
            if (i >= 2 && !tc::mbar_wait(&empty[s], uint32_t((i >> 1) - 1) & 1u)) {
                *aborted = 1;
                break;
            }
            uint8_t* A = smem + s * S::kStage;
            uint8_t* B = A + S::kABytes;
            const int k0 = (first + i) * kTile;
            int x, y, z;
            for (int e = id; e < kTile * (COUT / 8); e += S::kLoaders) {
                const int p = e / (COUT / 8), j = e % (COUT / 8);
                const long v = voxel_of(k0 + p, a.g, R, P, total, &x, &y, &z);
                uint8_t* dst = A + j * kASbo + p * 16;
                if (HF) {
                    __align__(16) __nv_bfloat16 h[8] = {};
                    if (v >= 0) split3(__ldg(a.h32 + v), h);
                    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(h);
                } else {
                    copy16(dst, a.h + (v >= 0 ? v : 0) * COUT + 8 * j, v >= 0);
                }
            }
            // two threads per position, each every other channel group; a
            // pair shifts y and z only (positions whose h is zero may read
            // anything finite)
            for (int e = id; e < 2 * kRun; e += S::kLoaders) {
                const int p = e >> 1;
                const bool in = voxel_of(k0 - 1 + p, a.g, R, P, total, &x, &y, &z) >= -1 && x < a.g.X;
                uint8_t* dst = B + p * 16;
                for (int pr = 0; pr < pairs; ++pr, dst += S::kPairBytes) {
                    const int zz = z + (pair0 + pr) / 3 - 1, yy = y + (pair0 + pr) % 3 - 1;
                    const bool ok = in && unsigned(zz) < unsigned(a.g.Z) && unsigned(yy) < unsigned(a.g.Y);
                    const long v = ok ? (long(zz) * a.g.Y + yy) * a.g.X + x : 0;
                    if (XF) {
                        __align__(16) __nv_bfloat16 h[8] = {};
                        if (ok && !(e & 1)) {
                            const float2 f = __ldg(reinterpret_cast<const float2*>(a.x32) + v);
                            split3(f.x, h);
                            split3(f.y, h + 3);
                        }
                        *reinterpret_cast<uint4*>(dst + (e & 1) * kBSbo) = *reinterpret_cast<uint4*>(h);
                        continue;
                    }
                    const long c =
                        ok && a.s1.up ? (long(zz >> 1) * (a.g.Y >> 1) + (yy >> 1)) * (a.g.X >> 1) + (x >> 1) : v;
#pragma unroll
                    for (int k = 0; k < CIN / 16; ++k) {
                        const int j = 2 * k + (e & 1);
                        const __nv_bfloat16* src = 8 * j < a.s1.C ? a.s1.p + (c * a.s1.C + 8 * j)
                                                                  : a.s2.p + (v * a.s2.C + (8 * j - a.s1.C));
                        copy16(dst + j * kBSbo, src, ok);
                    }
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            tc::fence_async_smem();
            tc::mbar_arrive(&full[s]);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (!*aborted) {
        for (int e = tid; e < 3 * pairs * (XF ? 2 * COUT : HF ? CIN : CIN * COUT); e += 32 * kWarps) {
            // CTAs start at different taps, so that their adds spread
            const int per = XF ? 2 * COUT : HF ? CIN : CIN * COUT;
            const int t = (e / per + blockIdx.x) % (3 * pairs), q = e % per;
            const float* c = acc + (t % 3 * pairs + t / 3) * CIN * S::kAccStride;
            float* out = a.dw + size_t(3 * pair0 + t) * per + q;
            if (XF) {
                const float* p = c + 3 * (q & 1) * S::kAccStride + (q >> 1);
                atomicAdd(out, p[0] + p[S::kAccStride] + p[2 * S::kAccStride]);
            } else if (HF) {
                const float* p = c + q * S::kAccStride;
                atomicAdd(out, p[0] + p[1] + p[2]);
            } else {
                atomicAdd(out, c[(q % CIN) * S::kAccStride + q / CIN]);
            }
        }
    } else if (tid == 0) {
        atomicExch(a.err, 1);
    }
    if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

template <int CIN, int COUT, bool XF, bool HF>
cudaError_t launch(const DwArgs& a, int sm_count, cudaStream_t st) {
    using S = DwShape<CIN, COUT>;
    auto k = dw_tc_kernel<CIN, COUT, XF, HF>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
    if (e != cudaSuccess) return e;
    const long total = long(a.g.X + 1) * (a.g.Y + 1) * a.g.Z;
    const int tiles = int((total + kTile - 1) / kTile);
    // one CTA per SM over (position ranges) x (groups of (dz, dy) pairs)
    const int per = (tiles + sm_count / S::kGroups - 1) / std::max(1, sm_count / S::kGroups);
    k<<<dim3((tiles + per - 1) / per, S::kGroups), 32 * kWarps, S::kSmem, st>>>(a, tiles, per);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_dw_tc(int cin, int cout, const ConvGrid& g, const __nv_bfloat16* h, const float* h32,
                         const ConvSrc& s1, const ConvSrc& s2, const float* x32, float* dw, int* err,
                         cudaStream_t st) {
    // padded positions and the shifts of a tap are 32-bit
    if (long(g.X + 1) * (g.Y + 1) * (g.Z + 2) > (1L << 30)) return cudaErrorInvalidValue;
    int dev = 0, sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const DwArgs a{g, h, h32, s1, s2, x32, dw, err};
    if (x32) return cin == 2 && cout == 16 ? launch<16, 16, true, false>(a, sm, st) : cudaErrorInvalidValue;
    if (s1.C + s2.C != cin || s1.C % 8 || s2.C % 8) return cudaErrorInvalidValue;
    if (h32) return cin == 16 && cout == 1 ? launch<16, 8, false, true>(a, sm, st) : cudaErrorInvalidValue;
#define PGD_DW(CI, CO) \
    if (cin == CI && cout == CO) return launch<CI, CO, false, false>(a, sm, st);
    PGD_DW(16, 16) PGD_DW(16, 32) PGD_DW(32, 32) PGD_DW(32, 64) PGD_DW(64, 64) PGD_DW(96, 32) PGD_DW(48, 16)
#undef PGD_DW
    return cudaErrorInvalidValue;
}

}  // namespace pgd

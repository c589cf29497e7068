// pcg.cu -- the Jacobi-preconditioned Poisson PCG as one persistent kernel
// (solve(fvm::laplacian(phiE) + rhoCharge/epsilon0), ElectroStaticSolver.C:61-64).
//
// Built with --fmad=false: the kernel evaluates in the order of the CPU
// oracle, and every sum runs in the fixed tree order of reduce.cuh (a chunk
// of kChunk cells has 256 sums of kItems strided cells each; lane l of one
// warp adds sums l, l+32, ..., l+224, then an xor-tree; the chunk sums are
// combined in the same order), so a solve is bit-reproducible and matches the
// oracle bit for bit.
//
// The PCG runs in the Chronopoulos-Gear form (one reduction point per
// iteration): with u = D^-1 r, w = M u, s = M p,
//   p = u + beta p,  s = w + beta s,  x += alpha p,  r -= alpha s,  u = D^-1 r
//   w = M u,  gamma = r.u,  delta = w.u,  beta = gamma / gamma_old,
//   alpha = gamma / (delta - beta gamma / alpha_old).
// It is the same Krylov iteration as the textbook PCG of lduMatrix (the
// iterates agree in exact arithmetic).  The vector updates, the SpMV and the
// dot products use explicit fused multiply-adds (the oracle calls std::fma at
// the same places).
//
// What bounds it: on this part one FP64 warp instruction holds its quarter of
// the SM for 64 cycles (a dependent chain costs the same, a division 580), so
// a chunk's iteration keeps one SM busy for 8192 cycles, and on small meshes
// the chain "all u written - SpMV - sum of delta - one division - update"
// with its two waits for all blocks counts.  Hence
//   * one cooperative launch per solve: r, p, s, w, u of a cell stay with its
//     thread (registers; shared memory when a block has several chunks) and
//     only u and the chunk sums pass through L2;
//   * a cluster of 2 to 8 blocks shares a chunk when the chunks alone would
//     leave SMs idle, one cell per thread so that all four quarters of an SM
//     work; the chunk's tree reads its sums through distributed shared memory;
//   * three further warps per block hold everything that is not per cell:
//     one forms gamma, beta and beta gamma / alpha_old (two of the three
//     divisions), one r.r, while the others run the SpMV; the third waits for
//     the other blocks and closes the iteration with delta and alpha;
//   * x, p and s are updated while delta is summed.
// Per iteration on GB300, against the two-kernel iteration of fields.cu in a
// CUDA graph: 128 cells 2 (11.5) us, 5917 cells 6.6 (18.6), 27,000 cells
// 6.8 (19), 91,125 cells 9.5 (19.5), 262,144 cells 16.0 (21).
#include "fields.h"
#include "reduce.cuh"

#include <cooperative_groups.h>

namespace pgd {

namespace cg = cooperative_groups;

namespace {

constexpr int kScalarThreads = 96;          // warps G, R, D
constexpr unsigned kSpinLimit = 1u << 22;   // polls of one wait, about a second
// Where a block keeps r, p, s, w, u of its cells: registers (one chunk per
// block) or shared memory (up to kSmemChunks).
constexpr int kReg = 0, kSmem = 1;
constexpr int kSmemChunks = 4;
constexpr int kVecs = 5;
constexpr int kSums = 6;                    // sets of thread sums of a chunk
enum { kR, kP, kS, kW, kU };

struct PcgArgs {
    DMesh m;
    const double* __restrict__ b;
    double* x;
    double* u;          // exchanged between blocks
    double* part;       // gamma, r.r, delta, b.b sums of the chunks
    PcgState* st;
    double tol;
    int maxit;
    int chunks;
};

constexpr int threads_of(int I, int S) { return (I == 1 && S > 1 ? kChunk / S : 256) + kScalarThreads; }

template <int Mode, int I>
struct Store {   // kReg
    double v[kVecs][I];
    double xv[I];
    __device__ double& at(int k, int, int j) { return v[k][j]; }
    __device__ double& x(int j, long) { return xv[j]; }
};
template <int I>
struct Store<kSmem, I> {
    double* base;
    double* xg;
    __device__ double& at(int k, int lc, int j) {
        return base[((lc * kVecs + k) * kItems + j) * 256 + int(threadIdx.x)];
    }
    __device__ double& x(int, long c) { return xg[c]; }
};

__device__ __forceinline__ void arrive(unsigned* bar) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}

// Waits until the counter has passed `target`; false when the poll limit ran out.
__device__ __forceinline__ bool wait(const unsigned* bar, unsigned target) {
    for (unsigned i = 0; i < kSpinLimit; ++i) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        if (int(v - target) >= 0) return true;
    }
    return false;
}

// One warp: the sum over nb chunk sums in the order of final_sum +
// block_tree, without the additions of zeros (which change nothing); valid in
// every lane.
__device__ __forceinline__ double warp_final_sum(const double* part, int nb) {
    const int lane = threadIdx.x & 31;
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 0.0;
    for (int i0 = 0; i0 < nb; i0 += 256) {
        double p[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int i = i0 + 32 * k + lane;
            p[k] = i < nb ? __ldcg(part + i) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (i0 == 0) v[k] = p[k];
            else if (i0 + 32 * k < nb) v[k] = v[k] + p[k];
    }
    double r = v[0];
#pragma unroll
    for (int k = 1; k < 8; ++k)
        if (32 * k < nb) r = r + v[k];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
        if (off < nb) r = r + __shfl_xor_sync(0xffffffffu, r, off);
    return __shfl_sync(0xffffffffu, r, 0);
}

// One warp: a chunk's sum from its thread sums, in the order of block_tree;
// they lie in the S blocks of the cluster, 256 / S each, and those from
// `count` on are zero.
template <int S>
__device__ __forceinline__ double warp_chunk_sum(double* tv, int count, const cg::cluster_group& cl) {
    constexpr int per = 256 / S;
    const int lane = threadIdx.x & 31;
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int t = 32 * k + lane;
        v[k] = 0.0;
        if (32 * k < count) v[k] = S == 1 ? tv[t] : *cl.map_shared_rank(tv + t % per, 32 * k / per);
    }
    double r = v[0];
#pragma unroll
    for (int k = 1; k < 8; ++k)
        if (32 * k < count) r = r + v[k];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) r = r + __shfl_xor_sync(0xffffffffu, r, off);
    return r;
}

// y = M x in the row of cell c: on a uniform block mesh every coupled face in
// direction f carries the same coefficient (the host checks every face), so
// the per-face array is not read.  xn holds x at the neighbours, anything
// where there is none (the loads carry no branch, so a thread's are all in
// flight together).
template <bool Uniform>
__device__ __forceinline__ double row(const DMesh& m, double diag, double xc, const int* nb, long c,
                                      const double* xn) {
    double s = diag * xc;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        const double v = fma(Uniform ? m.lap_coef[f] : m.Moff[6 * c + f], xn[f], s);
        s = nb[f] >= 0 ? v : s;
    }
    return s;
}

struct Scalars {
    double g, rr, bb, beta, t, alpha, rz, lim;
    int fail;
};

// Named barriers (0 is __syncthreads).
enum { kBarU = 1, kBarW = 2, kBarT = 3, kBarBeta = 4, kBarMain = 5 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// S blocks (a cluster) per chunk; I cells per thread: kItems when a block has
// whole chunks, 1 when it shares one or is alone with at most 256 cells.
// Threads [0, M) own the block's cells; warps G, R and D the scalars.
template <bool Uniform, int Mode, int I, int S>
__global__ void __launch_bounds__(threads_of(I, S)) pcg_kernel(PcgArgs A) {
    extern __shared__ double dyn[];   // sums; then kSmem: the vectors, I = 1: r, u, w of the block
    __shared__ Scalars sc;
    const cg::cluster_group cl = cg::this_cluster();
    constexpr bool alone = I == 1 && S == 1;   // one block, at most 256 cells
    constexpr int per = 256 / S;
    const int M = alone ? int(blockDim.x) - kScalarThreads : threads_of(I, S) - kScalarThreads;
    const int tid = threadIdx.x;
    const bool mine = tid < M;
    const int lane = tid & 31, role = (tid - M) >> 5;   // 0: G, 1: R, 2: D
    const int rank = S == 1 ? 0 : int(cl.block_rank());
    const int cluster = blockIdx.x / S, clusters = gridDim.x / S;
    const int slots = (A.chunks + clusters - 1) / clusters;   // chunks per block, at most
    const int nb = A.chunks, n = A.m.n_cells;
    const bool single = alone || clusters == 1;
    unsigned ph = 0;                                     // passes begun: waits per counter
    // sums of quantity q (0 gamma, 1 r.r, 2 delta, 3 b.b) of the block's chunk
    // lc; gamma and r.r in two sets, as warps G and R of another block may
    // still read one while the next is written
    auto tv = [&](int q, int lc, unsigned pass) {
        return dyn + ((q < 2 ? 2 * q + int(pass & 1u) : q + 2) * slots + lc) * per;
    };
    double* const vals = dyn + kSums * slots * per;   // I = 1: kItems x per values of r, u, w (b)
    // cell of item j of this thread in chunk ch
    auto cell = [&](int ch, int j) {
        return long(ch) * kChunk + (I == 1 ? rank * per + tid % per + 256 * (tid / per) : tid + 256 * j);
    };
    PcgState* st = A.st;

    Store<Mode, I> V;
    if constexpr (Mode == kSmem) {
        V.base = vals;
        V.xg = A.x;
    }
    double dinv[I], diag[I];
    int nbr[I][6];
#pragma unroll
    for (int j = 0; j < I; ++j)
#pragma unroll
        for (int f = 0; f < 6; ++f) nbr[j][f] = -1;
    if (tid == 0) sc.fail = 0;
    auto load_cell = [&](long c, int j) {
        dinv[j] = A.m.dinv[c];
        diag[j] = A.m.Mdiag[c];
#pragma unroll
        for (int f = 0; f < 6; ++f) nbr[j][f] = A.m.nbr[6 * c + f];
    };
    auto put_u = [&](long c, int j, double v) {
        if (alone) vals[M + c] = v;
        else __stcg(A.u + c, v);
    };
    auto get_u = [&](long i) { return alone ? vals[M + i] : __ldcg(A.u + i); };
    constexpr int kNext = alone ? 0 : per / 32;   // first warp of the next chain
    // I = 1: sum q of strided cells t, t + 256, ... from the block's values
    // a and b, by the warps starting at `first`
    auto chain = [&](int q, const double* a, const double* b, int first) {
        const int t = tid - 32 * first;
        if (t < 0 || t >= per) return;
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            if (!(alone && j > 0) && long(cluster) * kChunk + rank * per + t + 256 * j < n)
                v = fma(a[j * per + t], b[j * per + t], v);
        tv(q, 0, ph)[t] = v;
    };
    auto sync_all = [&]() {
        if (S == 1) __syncthreads();
        else cl.sync();
    };
    auto failed = [&]() {
        // every block of the cluster learns of it before its next sync_all
        for (int q = 0; q < S; ++q) *(S == 1 ? &sc.fail : cl.map_shared_rank(&sc.fail, q)) = 1;
        atomicMax(&st->fail, 1);
    };
    // the chunk sums of quantity q, by the calling warp
    auto publish = [&](int q, double* out, unsigned pass) {
        if (rank != 0) return;
        int lc = 0;
        for (int ch = cluster; ch < nb; ch += clusters, ++lc) {
            const double v = warp_chunk_sum<S>(tv(q, lc, pass), min(n - ch * kChunk, 256), cl);
            if (lane == 0) out[ch] = v;
        }
    };
    // waits until every cluster has arrived at counter b (`target` arrivals)
    auto meet = [&](int b, unsigned target) {
        __syncwarp();
        if (lane == 0) {
            if (rank == 0) arrive(&st->bar[b]);
            if (!wait(&st->bar[b], target)) failed();
        }
        __syncwarp();
    };
    // the sum of quantity q over all chunks; one cluster reads its thread
    // sums directly, ordered by the cluster's own barriers
    auto total = [&](int q, unsigned pass) {
        return single ? warp_chunk_sum<S>(tv(q, 0, pass), min(n, 256), cl) : warp_final_sum(A.part + q * nb, nb);
    };
    sync_all();

    // ---- r = b - M x, u = D^-1 r ----
    if (mine) {
        int lc = 0;
        for (int ch = cluster; ch < nb; ch += clusters, ++lc) {
            double sg = 0.0, srr = 0.0, sbb = 0.0;
#pragma unroll
            for (int j = 0; j < I; ++j) {
                const long c = cell(ch, j);
                if (c >= n) continue;
                load_cell(c, j);
                const double xc = A.x[c], bc = A.b[c];
                double xn[6];
#pragma unroll
                for (int f = 0; f < 6; ++f) xn[f] = A.x[nbr[j][f] >= 0 ? nbr[j][f] : c];
                const double ri = bc - row<Uniform>(A.m, diag[j], xc, nbr[j], c, xn);
                const double ui = dinv[j] * ri;
                if (Mode == kReg) V.x(j, c) = xc;
                V.at(kR, lc, j) = ri;
                V.at(kU, lc, j) = ui;
                put_u(c, j, ui);
                if (I == 1) {
                    vals[tid] = ri;
                    vals[M + tid] = ui;
                    vals[2 * M + tid] = bc;
                } else {
                    sg = fma(ri, ui, sg);
                    srr = fma(ri, ri, srr);
                    sbb = fma(bc, bc, sbb);
                }
            }
            if (I > 1) {
                tv(0, lc, ph)[tid] = sg;
                tv(1, lc, ph)[tid] = srr;
                tv(3, lc, ph)[tid] = sbb;
            }
        }
        if (I == 1) {
            bar_sync(kBarMain, M);
            chain(0, vals, vals + M, 0);
            chain(1, vals, vals, kNext);
            chain(3, vals + 2 * M, vals + 2 * M, 2 * kNext);
        }
    }
    int k = -1, done = 0, converged = 0;
    double alpha = 0.0;
    while (true) {
        sync_all();
        if (sc.fail) break;
        ++ph;
        if (mine) {
            // ---- w = M u ----
            if (!single) bar_sync(kBarU, M + 32);
            int lc = 0;
            for (int ch = cluster; ch < nb; ch += clusters, ++lc) {
                double sd = 0.0;
                double un[I][6];
#pragma unroll
                for (int j = 0; j < I; ++j) {
                    const long c = min(cell(ch, j), long(n) - 1);
                    if (Mode != kReg) load_cell(c, j);
#pragma unroll
                    for (int f = 0; f < 6; ++f) un[j][f] = get_u(nbr[j][f] >= 0 ? nbr[j][f] : c);
                }
#pragma unroll
                for (int j = 0; j < I; ++j) {
                    const long c = cell(ch, j);
                    if (c >= n) continue;
                    const double uc = V.at(kU, lc, j);
                    const double wc = row<Uniform>(A.m, diag[j], uc, nbr[j], c, un[j]);
                    V.at(kW, lc, j) = wc;
                    if (I == 1) vals[2 * M + tid] = wc;
                    else sd = fma(wc, uc, sd);
                }
                if (I > 1) tv(2, lc, ph)[tid] = sd;
            }
            if (I == 1) {
                bar_sync(kBarMain, M);
                chain(2, vals + 2 * M, vals + M, 0);
            }
            if (S > 1) {
                cl.sync();
            } else if (single) {
                bar_arrive(kBarW, M + 32);
            } else {
                // a warp per chunk forms its sum
                bar_sync(kBarMain, M);
                const int w = tid >> 5, ch = cluster + w * clusters;
                if (w < slots && ch < nb) {
                    const double v = warp_chunk_sum<S>(tv(2, w, ph), min(n - ch * kChunk, 256), cl);
                    if (lane == 0) A.part[2 * nb + ch] = v;
                }
                bar_arrive(kBarW, M + 32);
            }
            // ---- while delta is summed: x += alpha p of the last direction,
            //      p = u + beta p, s = w + beta s (p = u, s = w at the start) ----
            const bool start = k < 0;
            if (!start) {
                lc = 0;
                for (int ch = cluster; ch < nb; ch += clusters, ++lc)
#pragma unroll
                    for (int j = 0; j < I; ++j) {
                        const long c = cell(ch, j);
                        if (c < n) V.x(j, c) = fma(alpha, V.at(kP, lc, j), V.x(j, c));
                    }
            }
            bar_sync(kBarBeta, M + 32);
            const double beta = sc.beta;
            lc = 0;
            for (int ch = cluster; ch < nb; ch += clusters, ++lc)
#pragma unroll
                for (int j = 0; j < I; ++j) {
                    if (cell(ch, j) >= n) continue;
                    const double u0 = V.at(kU, lc, j), w0 = V.at(kW, lc, j);
                    V.at(kP, lc, j) = start ? u0 : fma(beta, V.at(kP, lc, j), u0);
                    V.at(kS, lc, j) = start ? w0 : fma(beta, V.at(kS, lc, j), w0);
                }
        } else if (role == 2) {
            // D: u of every block, then delta and alpha
            if (!single) {
                meet(0, ph * unsigned(clusters));
                bar_arrive(kBarU, M + 32);
            }
            if (S == 1) bar_sync(kBarW, M + 32);
            else cl.sync();
            if (!single) {
                if (S > 1) publish(2, A.part + 2 * nb, ph);
                meet(2, ph * unsigned(clusters));
            }
            const double d = total(2, ph);
            bar_sync(kBarT, 64);
            if (lane == 0) {
                const double g = sc.g;
                sc.alpha = k < 0 ? g / d : g / (d - sc.t);
            }
        } else {
            // G: gamma (and b.b at the start), beta; R: r.r
            if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            if (!single) {
                publish(role, A.part + role * nb, ph - 1);
                if (k < 0 && role == 0) publish(3, A.part + 3 * nb, 0);
                meet(1, ph * 2u * unsigned(clusters));
            }
            const double v = total(role, ph - 1);
            if (role == 0) {
                const double bb = k < 0 ? total(3, 0) : 0.0;
                const double be = k < 0 ? 0.0 : v / sc.rz;
                if (lane == 0) {
                    sc.beta = be;
                    if (k < 0) {
                        sc.bb = bb;
                        sc.lim = (A.tol * A.tol) * bb;
                    }
                }
                __syncwarp();
                bar_arrive(kBarBeta, M + 32);
                if (lane == 0) {
                    sc.t = k < 0 ? 0.0 : be * v / sc.alpha;
                    sc.g = v;
                    sc.rz = v;
                }
                __syncwarp();
                bar_arrive(kBarT, 64);
            } else if (lane == 0) {
                sc.rr = v;
            }
            if (S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        __syncthreads();
        alpha = sc.alpha;
        if (k < 0 && blockIdx.x == 0 && tid == 0) {
            st->rr0 = sc.rr;
            st->bb = sc.bb;
            st->lim = sc.lim;
        }
        ++k;
        if (sc.rr <= sc.lim) {
            done = converged = 1;
            break;
        }
        if (k > 0 && k >= A.maxit) {
            done = 1;
            break;
        }
        // ---- r -= alpha s, u = D^-1 r ----
        if (mine) {
            int lc = 0;
            for (int ch = cluster; ch < nb; ch += clusters, ++lc) {
                double sg = 0.0, srr = 0.0;
#pragma unroll
                for (int j = 0; j < I; ++j) {
                    const long c = cell(ch, j);
                    if (c >= n) continue;
                    const double di = Mode == kReg ? dinv[j] : A.m.dinv[c];
                    const double ri = fma(-alpha, V.at(kS, lc, j), V.at(kR, lc, j));
                    const double ui = di * ri;
                    V.at(kR, lc, j) = ri;
                    V.at(kU, lc, j) = ui;
                    put_u(c, j, ui);
                    if (I == 1) {
                        vals[tid] = ri;
                        vals[M + tid] = ui;
                    } else {
                        sg = fma(ri, ui, sg);
                        srr = fma(ri, ri, srr);
                    }
                }
                if (I > 1) {
                    tv(0, lc, ph)[tid] = sg;
                    tv(1, lc, ph)[tid] = srr;
                }
            }
            if (I == 1) {
                bar_sync(kBarMain, M);
                chain(0, vals, vals + M, 0);
                chain(1, vals, vals, kNext);
            }
        }
    }
    // ---- results ----
    if (Mode == kReg && mine) {
#pragma unroll
        for (int j = 0; j < I; ++j) {
            const long c = cell(cluster, j);
            if (c < n) A.x[c] = V.x(j, c);
        }
    }
    if (tid == 0) {
        if (blockIdx.x == 0) {
            st->rr = sc.rr;
            st->k = st->iters = k;
            st->done = done;
            st->converged = converged;
        }
        // the last block out clears the counters for the next solve
        __threadfence();
        if (atomicAdd(&st->exits, 1u) == gridDim.x - 1) {
            st->bar[0] = st->bar[1] = st->bar[2] = 0u;
            st->exits = 0u;
        }
    }
    if (S > 1) cl.sync();
}

using Kernel = void (*)(PcgArgs);

template <bool Uniform>
Kernel kernel_of(const PcgPlan& p) {
    switch (p.split) {
        case 8: return pcg_kernel<Uniform, kReg, 1, 8>;
        case 4: return pcg_kernel<Uniform, kReg, 1, 4>;
        case 2: return pcg_kernel<Uniform, kReg, 1, 2>;
        default: break;
    }
    if (p.alone) return pcg_kernel<Uniform, kReg, 1, 1>;
    return p.clusters >= p.chunks ? pcg_kernel<Uniform, kReg, kItems, 1> : pcg_kernel<Uniform, kSmem, kItems, 1>;
}

Kernel kernel_of(const PcgPlan& p, bool uniform) { return uniform ? kernel_of<true>(p) : kernel_of<false>(p); }

void configure(const PcgPlan& p, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(p.clusters * p.split);
    cfg->blockDim = dim3(p.alone ? (p.cells + 31) / 32 * 32 + kScalarThreads
                                 : threads_of(p.split > 1 ? 1 : kItems, p.split));
    cfg->dynamicSmemBytes = p.smem;
    cfg->attrs = attr;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg->numAttrs = p.split > 1 ? 2 : 1;
}

cudaError_t prepare(PcgPlan* plan, int sm_count, bool uniform) {
    const int slots = (plan->chunks + plan->clusters - 1) / plan->clusters, per = 256 / plan->split;
    int doubles = kSums * slots * per;
    if (slots > 1) doubles += slots * kVecs * kChunk;
    else if (plan->split > 1) doubles += 3 * kItems * per;
    else if (plan->alone) doubles += 3 * 256;
    plan->smem = doubles * int(sizeof(double));
    const Kernel k = kernel_of(*plan, uniform);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, plan->smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure(*plan, &cfg, attr);
    int fit = 0;
    if (plan->split > 1) {
        e = cudaOccupancyMaxActiveClusters(&fit, k, &cfg);
    } else {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k, int(cfg.blockDim.x), plan->smem);
        fit *= sm_count;
    }
    plan->fits = e == cudaSuccess && fit >= plan->clusters;
    return e;
}

}  // namespace

// The launch shape for n cells.  Up to 256 cells: one block, which waits for
// nobody.  Otherwise a chunk is split over the largest cluster
// that leaves every block an SM of its own (FP64 issue is the bound and is
// per SM); more chunks than SMs go round the blocks in shared memory, up to
// kSmemChunks each.  plan->fits stays false beyond that: there the
// two-kernel iteration of fields.cu streams its vectors and FP64 issue hides
// its launches.
cudaError_t pcg_make_plan(int n, bool uniform, PcgPlan* plan) {
    int dev = 0, sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    *plan = PcgPlan{};
    plan->cells = n;
    plan->chunks = pcg_blocks(n);
    const int slots = (plan->chunks + sm - 1) / sm;
    if (slots > kSmemChunks) return cudaSuccess;
    plan->clusters = (plan->chunks + slots - 1) / slots;
    plan->alone = n <= 256;
    for (int split = plan->alone ? 1 : 8; split >= 1 && !plan->fits; split >>= 1) {
        if (split > 1 && plan->chunks * split > sm) continue;
        plan->split = split;
        if ((e = prepare(plan, sm, uniform)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_pcg_solve(const DMesh& m, const PcgPlan& plan, const double* b, double* x, double* u, double* part,
                             PcgState* st, double tol, int maxit, cudaStream_t s) {
    PcgArgs A{};
    A.m = m;
    A.b = b;
    A.x = x;
    A.u = u;
    A.part = part;
    A.st = st;
    A.tol = tol;
    A.maxit = maxit;
    A.chunks = plan.chunks;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure(plan, &cfg, attr);
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, kernel_of(plan, m.lap_uniform != 0), A);
}

}  // namespace pgd

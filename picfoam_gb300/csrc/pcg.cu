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
// the chain "u of the neighbours - SpMV - sum of delta - one division - update"
// counts, which goes through L2 twice (a store seen by a load elsewhere: some
// 1400 cycles).  Hence
//   * one cooperative launch per solve: r, p, s, w, u of a cell stay with its
//     thread (registers; shared memory when a block has several chunks) and
//     only u and the chunk sums pass through L2;
//   * blocks do not meet: a value that passes through L2 carries the number of
//     its pass (PcgSlot), and who needs it reads it until the number is right.
//     Counting arrivals instead (all written, fence, atomic, poll, then the
//     load of the value) took three trips more per iteration.  Two sets of
//     slots, used in turn: a set is written again two passes later, when the
//     sums of the pass between, to which every block adds after its reads,
//     are known;
//   * a cluster of 2 to 8 blocks shares a chunk when the chunks alone would
//     leave SMs idle, one cell per thread so that all four quarters of an SM
//     work; the blocks send their thread sums to the block that adds them up
//     (st.async into its shared memory, counted by an mbarrier);
//   * three further warps per block hold everything that is not per cell:
//     one forms gamma, beta and beta gamma / alpha_old (two of the three
//     divisions), one r.r, while the others run the SpMV; the third closes the
//     iteration with delta and alpha;
//   * x, p and s are updated while delta is summed.
// A block with whole chunks has 6144 neighbours to read per chunk, which as
// slots are twice the bytes: there u is exchanged as it is behind an arrival
// counter, and with one chunk per block, where the registers are full, so are
// the sums of the chunks.
// Per iteration on GB300 (before: with arrival counters throughout, and as the
// two-kernel iteration of fields.cu in a CUDA graph): 5917 cells 4.2 us (6.4,
// 18.6; 4.0 with its end in leave()), 27,000 cells 5.5 (7.2, 19), 64,000 cells 6.9 (8.1), 91,125 cells 9.0
// (9.3, 19.5; 10.0 with slots), 262,144 cells 15.8 (15.7, 21; 18.4 with slots
// for u), 512,000 cells 25.3 (27.4); one block of 128 cells 2 us (2, 11.5).
#include "fields.h"
#include "reduce.cuh"

#include <cooperative_groups.h>

namespace pgd {

namespace cg = cooperative_groups;

namespace {

constexpr int kScalarThreads = 96;          // warps G, R, D
// Polls of one wait before it gives up (8 times as many of an mbarrier): a poll
// of a slot or counter is a load from L2, some 700 cycles, so this is seconds.
// Tests run the kernels with waits that look once.
constexpr unsigned kPolls = 1u << 22, kLookOnce = 2;
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
    PcgSlot* u;         // exchanged between blocks: two sets of n
    PcgSlot* part;      // gamma, r.r, delta, b.b sums of the chunks, two sets each
    PcgState* st;
    double tol;
    int maxit;
    int chunks;
    int ranks;          // blocks per cluster that the plan counts on
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

using u64 = unsigned long long;

// A slot's two words each hold half of the value and the pass number, so each
// is valid by itself whatever order the words arrive in.
__device__ __forceinline__ void put_slot(PcgSlot* p, double v, unsigned pass) {
    const u64 b = u64(__double_as_longlong(v)), e = u64(pass) << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"((b & 0xffffffffull) | e), "l"((b >> 32) | e)
                 : "memory");
}
__device__ __forceinline__ bool get_slot(const PcgSlot* p, unsigned pass, double* v) {
    u64 lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    *v = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
    return unsigned(lo >> 32) == pass && unsigned(hi >> 32) == pass;
}

__device__ __forceinline__ bool get(const PcgSlot* p, unsigned pass, double* v) { return get_slot(p, pass, v); }
__device__ __forceinline__ bool get(const double* p, unsigned, double* v) {
    *v = __ldcg(p);
    return true;
}

// Repeats ready() (uniform over the warp) until it holds; false when the limit
// (2 or more) ran out or another block gave up.
template <class F>
__device__ __forceinline__ bool wait_for(F ready, unsigned limit, const int* fail) {
    for (unsigned i = 1; i < limit; ++i) {
        if (ready()) return true;
        if ((i & 1023u) == 0 && *static_cast<const volatile int*>(fail)) break;
    }
    return false;
}

__device__ __forceinline__ bool phase_done(unsigned bar, unsigned parity) {
    unsigned there;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(there)
        : "r"(bar), "r"(parity)
        : "memory");
    return there != 0u;
}

__device__ __forceinline__ unsigned smem(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ unsigned peer(unsigned addr, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// Chunk sums that a lane reads at once, and so the chunks of a split plan.
constexpr int sums_per_lane(int S) { return S == 8 ? 1 : S == 4 ? 2 : S == 2 ? 3 : 8; }

// One warp: the sum over nb chunk sums in the order of final_sum +
// block_tree, without the additions of zeros (which change nothing); valid in
// every lane.  *ok turns false when a sum did not come.
template <int K, unsigned Polls, class Part>
__device__ __forceinline__ double warp_final_sum(const Part* part, int nb, unsigned pass, const int* fail, bool* ok) {
    const int lane = threadIdx.x & 31;
    double v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = 0.0;
    for (int i0 = 0; i0 < nb; i0 += 256) {
        double p[K];
        *ok = *ok && wait_for(
                         [&] {
                             bool all = true;
#pragma unroll
                             for (int k = 0; k < K; ++k) {
                                 const int i = i0 + 32 * k + lane;
                                 p[k] = 0.0;
                                 if (i < nb) all = get(part + i, pass, &p[k]) && all;
                             }
                             return sizeof(Part) == sizeof(double) || __all_sync(0xffffffffu, all);
                         },
                         Polls, fail);
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (i0 == 0) v[k] = p[k];
            else if (i0 + 32 * k < nb) v[k] = v[k] + p[k];
    }
    double r = v[0];
#pragma unroll
    for (int k = 1; k < K; ++k)
        if (32 * k < nb) r = r + v[k];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
        if (off < nb) r = r + __shfl_xor_sync(0xffffffffu, r, off);
    return __shfl_sync(0xffffffffu, r, 0);
}

// One warp: a chunk's sum from its 256 thread sums, in the order of
// block_tree; those from `count` on are zero.
__device__ __forceinline__ double warp_chunk_sum(const double* tv, int count) {
    const int lane = threadIdx.x & 31;
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = 32 * k < count ? tv[32 * k + lane] : 0.0;
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

// The end of a cluster's block: it leaves when no other can still send to it.
// After a wait that ran out, copies may be on their way that nobody waited for;
// a thread per barrier of a block that receives then waits for them.  How many
// there are follows from the pass in which each block stopped: it had sent its
// sums of gamma and r.r in the passes before it, of delta up to it and of b.b
// once.  A block is at most a pass ahead of another, so at most one phase per
// barrier is open, and it is armed; the bytes that nobody sent are counted off.
// (Not inlined: the kernel's registers then are what they were without it; as a
// part of its body it cost 27,000 cells 3 % of an iteration.)
template <int S>
__device__ __noinline__ void leave(u64 (*bars)[2], unsigned* last_pass, unsigned* drain, unsigned pass, bool done,
                                   bool receives) {
    constexpr unsigned kPhase = 256u * 8u;
    const cg::cluster_group cl = cg::this_cluster();
    const unsigned tid = threadIdx.x;
    if (tid == 0) *last_pass = pass;
    if (!done && tid < S) *cl.map_shared_rank(drain, int(tid)) = 1u;
    cl.sync();
    if (!*drain) return;
    if (tid < 8 && receives) {
        const unsigned q = tid >> 1, odd = tid & 1u, bar = smem(&bars[q][odd]);
        auto sent = [&](unsigned last) {
            return q == 3u ? 1u - odd : ((q == 2u) == (odd != 0u) ? last + 1u : last) / 2u;
        };
        unsigned used = sent(pass);   // phases that this block waited for
        if (used > 0u && !phase_done(bar, (used - 1u) & 1u)) --used;
        unsigned bytes = 0u;
        for (int r = 0; r < S; ++r) bytes += kPhase / S * sent(*cl.map_shared_rank(last_pass, r));
        bytes -= kPhase * used;
        if (bytes > 0u) {
            if (bytes < kPhase)
                asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(bar),
                             "r"(kPhase - bytes)
                             : "memory");
            for (unsigned i = 0; i < kPolls && !phase_done(bar, used & 1u); ++i) {}
        }
    }
    cl.sync();
}

struct Scalars {
    double g, rr, beta, t, alpha;
};

// Named barriers (0 is __syncthreads).
enum { kBarG = 1, kBarW = 2, kBarT = 3, kBarBeta = 4, kBarMain = 5, kBarU = 6 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// S blocks (a cluster) per chunk; I cells per thread: kItems when a block has
// whole chunks, 1 when it shares one or is alone with at most 256 cells.
// Threads [0, M) own the block's cells; warps G, R and D the scalars.
template <bool Uniform, int Mode, int I, int S, unsigned Polls>
__device__ __forceinline__ void pcg_body(const PcgArgs& A) {
    extern __shared__ double dyn[];   // sums; then kSmem: the vectors, I = 1: r, u, w of the block
    __shared__ Scalars scalars[2];    // in turn: a warp may still read one pass's while the next one's are written
    __shared__ double sc_rz, sc_bb, sc_lim;
    __shared__ __align__(8) u64 bars[4][2];   // S > 1: bytes received, per quantity, odd and even passes
    __shared__ unsigned last_pass, drain;     // S > 1: see leave()
    const cg::cluster_group cl = cg::this_cluster();
    // Every address of a peer below counts on S blocks per cluster.  A launch
    // that formed other ones (a tool between this library and the driver that
    // repeats the launch without its cluster) is given back untouched.
    if (S > 1 && (cl.num_blocks() != unsigned(S) || A.ranks != S)) {
        if (threadIdx.x == 0) atomicMax(&A.st->fail, kPcgShape);
        return;
    }
    constexpr bool alone = I == 1 && S == 1;   // one block, at most 256 cells
    // whole chunks per block: u as it is, an arrival counter instead of slots
    constexpr bool counted = I > 1;
    // one chunk per block, in registers: so are the chunks' sums
    constexpr bool counted_sums = counted && Mode == kReg;
    constexpr int kWarpsG = counted ? 96 : 64;   // threads that wait for the block's u, gamma and r.r sums
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
    PcgState* st = A.st;
    const unsigned pass0 = st->pass;    // number of the last solve's last pass
    unsigned ph = 0;                    // passes begun
    bool bad = false;                   // a wait of this thread ran out
    // thread sums of quantity q (0 gamma, 1 r.r, 2 delta, 3 b.b) of the block's
    // chunk lc; S > 1: what the blocks of the cluster sent.  In two sets where
    // one may still be read while the next is written
    auto tv = [&](int q, int lc, unsigned pass) {
        return S > 1 ? dyn + 256 * (2 * q + int(pass & 1u))
                     : dyn + ((q < 2 ? 2 * q + int(pass & 1u) : q + 2) * slots + lc) * 256;
    };
    double* const vals = dyn + (S > 1 ? 8 : kSums * slots) * 256;   // I = 1: kItems x per values of r, u, w (b)
    // cell of item j of this thread in chunk ch
    auto cell = [&](int ch, int j) {
        return long(ch) * kChunk + (I == 1 ? rank * per + tid % per + 256 * (tid / per) : tid + 256 * j);
    };

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
    // arms the barrier of quantity q and the pass's parity
    auto expect = [&](int q, unsigned pass) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem(&bars[q][pass & 1u])),
                     "r"(256 * 8)
                     : "memory");
    };
    if (S > 1) {
        if (tid == 0) drain = 0u;
        if (tid < 8) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem(&bars[tid / 2][tid % 2])) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            expect(tid / 2, unsigned(tid));
        }
        cl.sync();
    }
    auto load_cell = [&](long c, int j) {
        dinv[j] = A.m.dinv[c];
        diag[j] = A.m.Mdiag[c];
#pragma unroll
        for (int f = 0; f < 6; ++f) nbr[j][f] = A.m.nbr[6 * c + f];
    };
    // u of the pass ph + 1
    auto put_u = [&](long c, int j, double v) {
        if (alone) vals[M + c] = v;
        else if (counted) __stcg(reinterpret_cast<double*>(A.u) + c, v);
        else put_slot(A.u + long((ph + 1) & 1u) * n + c, v, pass0 + ph + 1);
    };
    constexpr int kNext = alone ? 0 : per / 32;   // first warp of the next chain
    // I = 1: sum q of strided cells t, t + 256, ... from the block's values
    // a and b, by the warps starting at `first`; S > 1: sent to the block that
    // adds the chunk up, or to all of them when there is no other chunk
    auto chain = [&](int q, const double* a, const double* b, int first) {
        const int t = tid - 32 * first;
        if (t < 0 || t >= per) return;
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            if (!(alone && j > 0) && long(cluster) * kChunk + rank * per + t + 256 * j < n)
                v = fma(a[j * per + t], b[j * per + t], v);
        if constexpr (S == 1) {
            tv(q, 0, ph)[t] = v;
        } else {
            const unsigned to = smem(tv(q, 0, ph) + rank * per + t), bar = smem(&bars[q][ph & 1u]);
            for (int r = 0; r < (single ? S : 1); ++r)
                asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                                 peer(to, r)),
                             "l"(__double_as_longlong(v)), "r"(peer(bar, r))
                             : "memory");
        }
    };
    auto failed = [&]() {
        bad = true;
        if (lane == 0) atomicMax(&st->fail, kPcgWait);
    };
    // S > 1, the calling warp: the pass's sums of quantity q are there.  Its
    // barrier is armed again at once, for two passes later: no block sends
    // those before every block has sent the sums of delta of the pass between,
    // which this one does after the __syncthreads that follows.
    auto received = [&](int q, unsigned pass) {
        if (S == 1) return;
        const unsigned bar = smem(&bars[q][pass & 1u]), phase = (q == 2 ? pass - 1 : pass) >> 1;
        const bool ok = wait_for([&] { return bool(__all_sync(0xffffffffu, phase_done(bar, phase & 1u))); },
                                 8 * Polls, &st->fail);
        if (!ok) failed();
        else if (lane == 0) expect(q, pass);
    };
    // waits until every block has added to counter b in this pass
    auto meet = [&](int b) {
        __syncwarp();
        if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->bar[b]) : "memory");
        const bool ok = wait_for(
            [&] {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&st->bar[b]) : "memory");
                return bool(__all_sync(0xffffffffu, int(v - ph * unsigned(clusters)) >= 0));
            },
            Polls, &st->fail);
        if (!ok) failed();
    };
    auto put_part = [&](int q, int ch, double v) {
        const long i = long(2 * q + int(ph & 1u)) * nb + ch;
        if (counted_sums) __stcg(reinterpret_cast<double*>(A.part) + i, v);
        else put_slot(A.part + i, v, pass0 + ph);
    };
    // the calling warp: quantity q summed over all chunks; `pass`: whose thread
    // sums.  One warp of each cluster publishes its chunks' sums (of delta,
    // with S == 1, the warps that own the cells did).
    auto total = [&](int q, unsigned pass) {
        if (single) {
            received(q, pass);
            return __shfl_sync(0xffffffffu, warp_chunk_sum(tv(q, 0, pass), min(n, 256)), 0);
        }
        if (rank == 0 && (S > 1 || q != 2)) {
            received(q, pass);
            int lc = 0;
            for (int ch = cluster; ch < nb; ch += clusters, ++lc) {
                const double v = warp_chunk_sum(tv(q, lc, pass), min(n - ch * kChunk, 256));
                if (lane == 0) put_part(q, ch, v);
            }
        }
        if (counted_sums) meet(q);
        bool ok = true;
        const long set = long(2 * q + int(ph & 1u)) * nb;
        const double v =
            counted_sums
                ? warp_final_sum<8, Polls>(reinterpret_cast<const double*>(A.part) + set, nb, 0u, &st->fail, &ok)
                : warp_final_sum<sums_per_lane(S), Polls>(A.part + set, nb, pass0 + ph, &st->fail, &ok);
        if (!ok) failed();
        return v;
    };

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
            bar_sync(kBarMain, M);   // vals + 2 M holds w from now on
        }
        if (S == 1) bar_arrive(kBarG, M + kWarpsG);
    }
    int k = -1, done = 0, converged = 0;
    double alpha = 0.0;
    while (true) {
        ++ph;
        Scalars& sc = scalars[ph & 1u];
        if (mine) {
            // ---- w = M u ----
            if (counted) bar_sync(kBarU, M + 32);
            const PcgSlot* const u = A.u + long(ph & 1u) * n;
            int lc = 0;
            for (int ch = cluster; ch < nb; ch += clusters, ++lc) {
                double sd = 0.0;
                if (Mode != kReg) {
#pragma unroll
                    for (int j = 0; j < I; ++j) load_cell(min(cell(ch, j), long(n) - 1), j);
                }
                double un[I][6];
                if constexpr (alone || counted) {
                    const double* const ud = alone ? vals + M : reinterpret_cast<const double*>(A.u);
#pragma unroll
                    for (int j = 0; j < I; ++j) {
                        const long c = min(cell(ch, j), long(n) - 1);
#pragma unroll
                        for (int f = 0; f < 6; ++f) {
                            const long i = nbr[j][f] >= 0 ? nbr[j][f] : c;
                            un[j][f] = alone ? ud[i] : __ldcg(ud + i);
                        }
                    }
                } else {
                    const bool ok = wait_for(
                        [&] {
                            bool all = true;
#pragma unroll
                            for (int f = 0; f < 6; ++f) {
                                un[0][f] = 0.0;
                                if (nbr[0][f] >= 0) all = get_slot(u + nbr[0][f], pass0 + ph, &un[0][f]) && all;
                            }
                            return bool(__all_sync(0xffffffffu, all));
                        },
                        Polls, &st->fail);
                    if (!ok) failed();
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
            if (S == 1 && single) {
                bar_arrive(kBarW, M + 32);
            } else if (S == 1) {
                // a warp per chunk forms its sum
                bar_sync(kBarMain, M);
                const int w = tid >> 5, ch = cluster + w * clusters;
                if (w < slots && ch < nb) {
                    const double v = warp_chunk_sum(tv(2, w, ph), min(n - ch * kChunk, 256));
                    if (lane == 0) put_part(2, ch, v);
                }
                if (counted_sums) bar_arrive(kBarW, M + 32);
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
            if (counted) {
                bar_sync(kBarG, M + kWarpsG);
                if (!single) meet(4);
                bar_arrive(kBarU, M + 32);
            }
            if (S == 1 && (single || counted_sums)) bar_sync(kBarW, M + 32);
            const double d = total(2, ph);
            bar_sync(kBarT, 64);
            if (lane == 0) sc.alpha = k < 0 ? sc.g / d : sc.g / (d - sc.t);
        } else {
            // G: gamma (and b.b at the start), beta; R: r.r
            if (S == 1) bar_sync(kBarG, M + kWarpsG);
            const double v = total(role, ph - 1);
            if (role == 0) {
                const double be = k < 0 ? 0.0 : v / sc_rz;
                if (k < 0) {
                    const double bb = total(3, 0);
                    if (lane == 0) {
                        sc_bb = bb;
                        sc_lim = (A.tol * A.tol) * bb;
                    }
                }
                if (lane == 0) sc.beta = be;
                __syncwarp();
                bar_arrive(kBarBeta, M + 32);
                if (lane == 0) {
                    sc.t = k < 0 ? 0.0 : be * v / scalars[(ph - 1) & 1u].alpha;
                    sc.g = v;
                    sc_rz = v;
                }
                __syncwarp();
                bar_arrive(kBarT, 64);
            } else if (lane == 0) {
                sc.rr = v;
            }
        }
        if (__syncthreads_or(bad)) break;
        alpha = sc.alpha;
        if (k < 0 && blockIdx.x == 0 && tid == 0) {
            st->rr0 = sc.rr;
            st->bb = sc_bb;
            st->lim = sc_lim;
        }
        ++k;
        if (sc.rr <= sc_lim) {
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
            if (S == 1) bar_arrive(kBarG, M + kWarpsG);
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
            st->rr = scalars[ph & 1u].rr;
            st->k = st->iters = k;
            st->done = done;
            st->converged = converged;
        }
        // the last block out numbers the passes of the next solve on (with
        // room for blocks a pass apart when one gave up)
        __threadfence();
        if (atomicAdd(&st->exits, 1u) == gridDim.x - 1) {
            st->pass = pass0 + ph + 4;
            for (unsigned& b : st->bar) b = 0u;
            st->exits = 0u;
        }
    }
    if (S > 1) leave<S>(bars, &last_pass, &drain, ph, done != 0, single || rank == 0);
}

template <bool Uniform, int Mode, int I, unsigned Polls = kPolls>
__global__ void __launch_bounds__(threads_of(I, 1)) pcg_kernel(PcgArgs A) {
    pcg_body<Uniform, Mode, I, 1, Polls>(A);
}

// The cluster's size belongs to the kernel, so no launch can be without it.
template <bool Uniform, int S, unsigned Polls = kPolls>
__global__ void __cluster_dims__(S, 1, 1) __launch_bounds__(threads_of(1, S)) pcg_cluster_kernel(PcgArgs A) {
    pcg_body<Uniform, kReg, 1, S, Polls>(A);
}

using Kernel = void (*)(PcgArgs);

template <bool Uniform>
Kernel kernel_of(const PcgPlan& p) {
    switch (p.split) {
        case 8: return pcg_cluster_kernel<Uniform, 8>;
        case 4: return pcg_cluster_kernel<Uniform, 4>;
        case 2: return pcg_cluster_kernel<Uniform, 2>;
        default: break;
    }
    if (p.alone) return pcg_kernel<Uniform, kReg, 1>;
    return p.clusters >= p.chunks ? pcg_kernel<Uniform, kReg, kItems> : pcg_kernel<Uniform, kSmem, kItems>;
}

// The forms whose blocks wait for one another, with waits that look once.
Kernel look_once(const PcgPlan& p) {
    switch (p.split) {
        case 8: return pcg_cluster_kernel<false, 8, kLookOnce>;
        case 4: return pcg_cluster_kernel<false, 4, kLookOnce>;
        case 2: return pcg_cluster_kernel<false, 2, kLookOnce>;
        default: break;
    }
    return p.clusters >= p.chunks ? pcg_kernel<false, kReg, kItems, kLookOnce>
                                  : pcg_kernel<false, kSmem, kItems, kLookOnce>;
}

Kernel kernel_of(const PcgPlan& p, bool uniform) {
    if (p.look_once && !p.alone) return look_once(p);
    return uniform ? kernel_of<true>(p) : kernel_of<false>(p);
}

void configure(const PcgPlan& p, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(p.clusters * p.split);
    cfg->blockDim = dim3(p.alone ? (p.cells + 31) / 32 * 32 + kScalarThreads
                                 : threads_of(p.split > 1 ? 1 : kItems, p.split));
    cfg->dynamicSmemBytes = p.smem;
    cfg->attrs = attr;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg->numAttrs = 1;
}

// Dynamic shared memory of a block with `slots` chunks of its own (kSmem).
constexpr int smem_bytes(int slots) { return slots * (kSums * 256 + kVecs * kChunk) * int(sizeof(double)); }

cudaError_t prepare(PcgPlan* plan, int sm_count, bool uniform) {
    const int slots = (plan->chunks + plan->clusters - 1) / plan->clusters, per = 256 / plan->split;
    int doubles = plan->split > 1 ? 8 * 256 : kSums * 256;
    if (plan->split > 1) doubles += 3 * kItems * per;
    else if (plan->alone) doubles += 3 * 256;
    plan->smem = slots > 1 ? smem_bytes(slots) : doubles * int(sizeof(double));
    const Kernel k = kernel_of(*plan, uniform);
    cudaError_t e = cudaSuccess;
    // the limit belongs to the function, not to this plan: always the largest
    // plan's, so that a smaller one does not take it from a context in use
    if (slots > 1)
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(kSmemChunks));
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
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
        if (split > 1 && (plan->chunks * split > sm || plan->chunks > 32 * sums_per_lane(split))) continue;
        plan->split = plan->ranks = split;
        if ((e = prepare(plan, sm, uniform)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_pcg_solve(const DMesh& m, const PcgPlan& plan, const double* b, double* x, PcgSlot* slots,
                             PcgState* st, double tol, int maxit, cudaStream_t s) {
    PcgArgs A{};
    A.m = m;
    A.b = b;
    A.x = x;
    A.u = slots;
    A.part = slots + 2 * long(plan.cells);
    A.st = st;
    A.tol = tol;
    A.maxit = maxit;
    A.chunks = plan.chunks;
    A.ranks = plan.ranks;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    configure(plan, &cfg, attr);
    cfg.stream = s;
    const Kernel k = kernel_of(plan, m.lap_uniform != 0);
    if (plan.look_once)   // a kernel that prepare() has not seen
        if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 smem_bytes(kSmemChunks)))
            return e;
    return cudaLaunchKernelEx(&cfg, k, A);
}

}  // namespace pgd

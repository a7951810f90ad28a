// pcg_common.cuh - what the FP64 and the FP32-form PCG kernels share (k_pcg.cu,
// k_pcg32.cu): status words, team barrier, halo words, bulk copies, the job
// record and the team tables of a batched launch.
#pragma once
#include "ifl_device.cuh"

namespace ifl {

// Dynamic shared memory of the PCG kernel, addressed through this symbol so
// that every ring and halo access compiles to a shared-space instruction.
extern __shared__ __align__(128) char g_smem[];

// Default polls of a halo-word or barrier wait (about a second); the host may
// set another limit per solve (PcgConfig::wait_limit).  The mbarrier waits of
// the bulk-copy rings keep their own fixed limit: they wait for copies this
// warp issued from this GPU's memory, which always complete, and a timed-out
// sweep still waits for every copy it issued before it leaves.
constexpr long long kWaitLimit = 1ll << 22;
constexpr long long kMbarWaitLimit = 1ll << 20;  // try_wait suspends between polls
constexpr double kTau = 0.97, kSigma = 0.25, kTol = 1e-5;
constexpr unsigned long long kSentinel = ~0ull;
constexpr unsigned FULL = 0xffffffffu;

// Status words a wait checks: the scene's own and one shared by every scene
// of a batched launch (the same word for a single-scene launch).  A timed-out
// wait marks both, so every later wait of the launch stops waiting.
struct Flags {
    unsigned *scene, *all;
    long long limit;  // polls of one halo or barrier wait before it gives up
};

// The blocks that solve one scene: ranks 0..size-1, their barrier counter and
// the per-block partial sums.  A single-scene launch is one team of the whole
// grid.
struct Team {
    int rank, size;
    unsigned *barrier;  // arrival counter
    unsigned goal;      // arrivals the last barrier waited for
};

template <typename F>
struct PcgArgs {
    SDIdx sd;
    const F *adiag, *ax, *ay;
    double *pc;
    F *mic;  // MIC(0) apply operands, five or six values per slot (pcg_ring.cuh)
    const uint8_t *nb;
    double *r, *p, *as;
    F *rf;  // r in storage precision for the substitutions (== r when F is double)
    F *z, *sa, *sb;
    double *partials;
    unsigned *barrier;
    Flags fl;
    unsigned long long *halo;  // [2][S][D]: [0] rows handed upward, [1] rows handed downward (pcg_halo_words in all)
    PcgOut *out;
    unsigned long long *iter_total;
    int mode, limit, pinned;
    int K, stages;
    int rowsum_zero;  // 1: pressure matrix (rows sum to zero), 0: heat matrix
    int all_red;      // 1: every cell takes part in the dot products and AXPYs (unmasked solves)
    int ref;          // FP64: 1: the reference's own arithmetic (k_pcg64.cu)
};

// ------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// Asks for global memory to be in L2 (16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void prefetch_l2(const void *p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// 1-D bulk copy global -> shared (16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool timed_out(const Flags &f) {
    return (ld_volatile(f.scene) | ld_volatile(f.all)) & FLAG_TIMEOUT;
}
__device__ __forceinline__ void set_timeout(const Flags &f) {
    atomicOr(f.scene, FLAG_TIMEOUT);
    if (f.all != f.scene) atomicOr(f.all, FLAG_TIMEOUT);
}

// Team barrier: one arrival counter that only grows (zero at launch) and the
// count this barrier waits for, bounded wait.  A team of one block needs only
// the block barrier.  An arrival releases this block's writes and the poll
// acquires the others', so no separate fences and no second word that the last
// arrival has to publish: 2 100 cycles on GB300 for 2 to 152 blocks, against
// 4 300 for an arrival counter with a generation word behind it.
static __device__ void team_barrier(Team &T, const Flags &fl) {
    __syncthreads();
    if (T.size == 1) return;
    T.goal += (unsigned)T.size;
    if (threadIdx.x == 0) {
        unsigned seen;
        asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(seen) : "l"(T.barrier) : "memory");
        seen++;
        long long n = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(T.barrier) : "memory");
            if ((int)(seen - T.goal) >= 0) break;
            if (++n > fl.limit || timed_out(fl)) {
                set_timeout(fl);
                break;
            }
        }
    }
    __syncthreads();
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o);
    return v;
}

// ------------------------------------------------------------ halo words
__device__ __forceinline__ unsigned long long henc(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ double hdec(unsigned long long w) { return __longlong_as_double((long long)w); }

// Halo rows: shared memory between warps of one block, global memory between
// blocks.  A channel holds the row's generic address, so one instruction
// serves both spaces (relaxed, GPU scope; stronger than a shared row needs).
// One 8-byte access is single-copy atomic, so a reader sees either the
// sentinel or the whole word.  A halo word carries its value itself, so no
// other memory access has to be ordered around it: the asm statements are
// volatile (kept, in program order) but do not clobber memory.  Loads and
// stores are predicated inside the asm: a sweep step never branches around a
// halo access.
struct Chan {
    unsigned long long *row;  // generic address of the row (word x at row + x)
    bool valid;
};
__device__ __forceinline__ unsigned long long hload(const Chan &c, int x) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.u64 %0, [%1];" : "=l"(v) : "l"(c.row + x));
    return v;
}
// The word at x where p holds, else `other`.
__device__ __forceinline__ unsigned long long hload_if(const Chan &c, int x, bool p, unsigned long long other) {
    unsigned long long v = other;
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q ld.relaxed.gpu.u64 %0, [%1];\n}\n"
                 : "+l"(v)
                 : "l"(c.row + x), "r"((unsigned)p));
    return v;
}
__device__ __forceinline__ void hstore_if(const Chan &c, int x, unsigned long long v, bool p) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.relaxed.gpu.u64 [%0], %1;\n}\n" ::"l"(c.row + x),
                 "l"(v), "r"((unsigned)p));
}

// Halo words of one sub-block: lane l < n needs the word at column xs[l]
// (need), prefetched in w.  Lanes whose word is still the sentinel poll it
// (bounded; the whole warp loops together, only in this slow path); then the
// sentinel goes back for the next sweep.  A timed-out wait yields 0.
__device__ __forceinline__ unsigned long long halo_take_warp(const Chan &c, int x, bool need, unsigned long long w,
                                                             const Flags &flags) {
    if (__any_sync(FULL, need && w == kSentinel)) {
        long long n = 0;
        bool given_up = false;
        for (;;) {
            const bool wait = need && w == kSentinel && !given_up;
            if (!__any_sync(FULL, wait)) break;
            if (wait) {
                w = hload(c, x);
                if (w == kSentinel && (++n > flags.limit || timed_out(flags))) {
                    set_timeout(flags);
                    given_up = true;
                }
            }
        }
        if (given_up) w = 0ull;
    }
    hstore_if(c, x, kSentinel, need);
    return w;
}

// ------------------------------------------------------------ batched solves
// Many independent scenes in one cooperative launch.  The grid is cut into
// teams; a team of g blocks solves scenes of up to g*K strips.  Teams of one
// size form a class and take that class's scenes from a shared queue (largest
// estimated work first), so a team that finishes early takes the next scene.
struct BatchTeams {
    const int2 *block_team;   // per block: {team, rank in team}
    const int2 *team;         // per team: {blocks, class}
    const int2 *class_range;  // per class: {offset, count} into class_jobs
    const int *class_jobs;    // job indices, each class in queue order
    int *class_next;          // queue heads (zero at launch)
    int *team_job;            // job taken by each team
    unsigned *team_bar;       // barrier counter of each team, kBarStride words apart (zero at launch)
    unsigned *all;            // launch-wide status word
    const int4 *ctl;          // per job: {pinned pressure, pinned heat, limit pressure, limit heat}
    // Placement of teams across SMs: the hardware puts consecutive blocks of a
    // launch on the same few SMs, so a team of consecutive block indices would
    // share those SMs' pipes.  Each block instead takes the slot
    // (its rank on its SM) x nsm + (its SM's dense index), and teams are built
    // from consecutive slots, i.e. from blocks on different SMs.
    const short *sm_dense;    // %smid -> dense SM index (-1: unknown); 1024 entries
    int *sm_fill;             // blocks placed per SM (zero at launch)
    unsigned *grid_bar;       // barrier counter over the whole grid (zero at launch)
    unsigned *remap_fail;     // set when a block could not be placed (zero at launch)
    int nsm, per, remap;
    long long wait_limit;     // polls of one halo or barrier wait
};
constexpr int kBarStride = 8;  // words between the teams' barrier counters (a 32-byte sector each)

// The team and rank of this block (s_slot: a shared word of the block).
static __device__ int2 batch_slot(const BatchTeams &B, int *s_slot) {
    const Flags fl{B.all, B.all, B.wait_limit};
    if (threadIdx.x == 0) {
        int slot = (int)blockIdx.x;
        if (B.remap) {
            unsigned smid;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
            const int d = smid < 1024u ? B.sm_dense[smid] : -1;
            const int k = d >= 0 ? atomicAdd(B.sm_fill + d, 1) : B.per;
            if (d >= 0 && k < B.per) slot = k * B.nsm + d;
            else atomicOr(B.remap_fail, 1u);
        }
        *s_slot = slot;
    }
    if (B.remap) {
        // every block learns whether all of them were placed, then all follow the same rule
        Team G{(int)blockIdx.x, (int)gridDim.x, B.grid_bar, 0u};
        team_barrier(G, fl);
        if (threadIdx.x == 0 && ld_volatile(B.remap_fail)) *s_slot = (int)blockIdx.x;
    }
    __syncthreads();
    return B.block_team[*s_slot];
}

// The team's next job into sA (shared by the block); false when the queue of
// its class is empty.  After a barrier that timed out the team's word may still be
// an earlier job's or -1 (its value at creation), and may change: one thread reads
// it for the block.
template <typename F>
__device__ bool batch_take(const BatchTeams &B, Team &T, int team, int cls, const PcgArgs<F> *jobs, PcgArgs<F> &sA,
                           int mode, int heat, int pinned, int K, int stages) {
    const Flags fl{B.all, B.all, B.wait_limit};
    if (T.rank == 0 && threadIdx.x == 0) {
        const int2 cr = B.class_range[cls];
        const int k = atomicAdd(B.class_next + cls, 1);
        *(volatile int *)(B.team_job + team) = k < cr.y ? B.class_jobs[cr.x + k] : -1;
    }
    team_barrier(T, fl);
    __shared__ int s_job;
    if (threadIdx.x == 0) s_job = *(volatile int *)(B.team_job + team);
    __syncthreads();
    const int j = s_job;
    if (j < 0) return false;
    for (int k = threadIdx.x; k < (int)(sizeof(PcgArgs<F>) / 4); k += blockDim.x)
        ((unsigned *)&sA)[k] = ((const unsigned *)(jobs + j))[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        const int4 c = B.ctl[j];
        sA.mode = mode;
        sA.limit = heat ? c.w : c.z;
        sA.pinned = pinned >= -1 ? pinned : (heat ? c.y : c.x);
        sA.K = K;
        sA.stages = stages;
        sA.fl.all = B.all;
        sA.fl.limit = B.wait_limit;
    }
    __syncthreads();
    return true;
}

}  // namespace ifl

// pcg_job.cuh - one solve by a team of blocks, the kernels for one scene and for
// a batch, and their launch.  Included after the form's own passes: sweep_strip,
// prepare_strip, matvec, axpy and start for PcgArgs<F>.
#pragma once
#include "pcg_ring.cuh"

namespace ifl {

namespace {

// Shared-memory layout of a block: ring mbarriers (of each strip) | the halo rows
// between its strips, K-1 upward and K-1 downward (apart, since each direction
// leaves words behind that it never reads) | the rings.
__host__ __device__ __forceinline__ unsigned halo_offset(int K) { return 8u * Ring<float>::KINDS * kMaxStages * K; }
__host__ __device__ __forceinline__ unsigned ring_offset(int K, int D) {
    const size_t nh = 2 * (size_t)(K > 1 ? K - 1 : 0) * (D + kHaloPad);
    return (unsigned)(((halo_offset(K) + nh * 8 + 127) / 128) * 128);
}

// Sweep of all strips of this block: warps 0..K-1 sweep, K..2K-1 load for them,
// 2K..3K-1 prepare, 3K..4K-1 take the halo words.  The team's T.size*K sweeping warps take the strips
// round-robin: warp `base` sweeps strips base, base + P, base + 2P,
// ... (P = T.size*K), in increasing order for the forward solve and in
// decreasing order for the backward solve, so that every strip waits only on a
// strip that is swept earlier by its own warp or by another warp in the same or
// an earlier round (no cycle).  When every warp has a single strip, the halo
// rows between the warps of one block live in shared memory; otherwise every
// strip hands its boundary row over through its own global row (a shared row
// would be reused by the next round while its reader may still need it).
template <typename F, bool REF, bool BWD>
__device__ void sweep_all(const PcgArgs<F> &A, const Team &T, Ring<F> &R) {
    const int role = (threadIdx.x >> 5) / A.K, w = (threadIdx.x >> 5) % A.K;
    const SDIdx sd = A.sd;
    int nstrips_blk = sd.S - T.rank * A.K;
    nstrips_blk = nstrips_blk > A.K ? A.K : nstrips_blk;
    if (role >= kRoles || w >= nstrips_blk) return;
    const int P = T.size * A.K;
    const int base = T.rank * A.K + w;
    const size_t row = pcg_halo_row(sd);
    unsigned long long *up = A.halo, *down = A.halo + (size_t)sd.S * row;
    auto smem_row = [&](int k) {
        const unsigned at = (unsigned)(((BWD ? A.K - 1 : 0) + k) * row);
        return Chan{(unsigned long long *)(g_smem + halo_offset(A.K) + 8u * at), true};
    };
    auto glob_row = [&](unsigned long long *r) { return Chan{r, true}; };
    const bool one_round = sd.S <= P;
    const int nmine = (sd.S - base + P - 1) / P;  // strips of this warp
    for (int j0 = 0; j0 < nmine; j0++) {
        const int s = base + (BWD ? nmine - 1 - j0 : j0) * P;
        Chan in{nullptr, false}, out{nullptr, false};
        if (!BWD) {  // rows travel upward: strip s takes from s-1, gives to s+1
            if (s > 0) in = (one_round && w > 0) ? smem_row(w - 1) : glob_row(up + (size_t)(s - 1) * row);
            if (s + 1 < sd.S)
                out = (one_round && w + 1 < nstrips_blk) ? smem_row(w) : glob_row(up + (size_t)s * row);
        } else {     // downward: strip s takes from s+1, gives to s-1
            if (s + 1 < sd.S)
                in = (one_round && w + 1 < nstrips_blk) ? smem_row(w) : glob_row(down + (size_t)(s + 1) * row);
            if (s > 0) out = (one_round && w > 0) ? smem_row(w - 1) : glob_row(down + (size_t)s * row);
        }
        if (role == 0) {
            // FP32: the halo words are folded into the operands (put_halo)
            if (sizeof(F) == 8 && in.valid) sweep_strip<REF, BWD, sizeof(F) == 8>(A, s, R, out);
            else sweep_strip<REF, BWD, false>(A, s, R, out);
        } else if (role == 1) {
            load_strip<F, REF, BWD>(A, s, R, in.valid);
        } else if (role == 2 && BWD && !REF) {
            prepare_strip(A, s, R, in.valid);
        } else if (role == 3 && in.valid) {
            take_strip<F, REF, BWD>(A, R, in);
        } else {
            R.skip(sd.D / Lay<F>::kSteps);
        }
    }
}

// One complete solve (factor and/or PCG, by A.mode) of one scene by team T.
// The halo words must hold the sentinel on entry; those that a sweep waits for
// hold it again on exit (every word that is waited for is taken).
// The elementwise passes work on chunks of pcg_chunk_diags(sd) diagonals,
// dealt out to the team's warps in turn.  Every reduction is summed per chunk
// (per strip for sigma), then over the partials in a fixed order, so the result
// depends on the scene alone, not on the number of blocks or warps that solve
// it: a scene gives bit-identical results in a single-scene launch, in any
// batch and with any launch shape.
// REF: the reference's own arithmetic in the triangular solves, the matvec and
// the AXPYs, sigma by a pass over z and r, and sums in an order of their own
// (k_pcg64.cu says where and why).
// Otherwise sigma = z.r is taken as y.(dd y), y the forward solve's result: z.r =
// (L^-T D L^-1 r).r = (L^-1 r).D(L^-1 r) exactly, and in floating point within
// the rounding of the two triangular solves.  Cells outside the masked MIC(0)
// work have dd = 0 and add nothing.
template <typename F, bool REF>
__device__ void pcg_job(const PcgArgs<F> &A, Team &T, Ring<F> &R, double *sm) {
    const int warps = blockDim.x >> 5;
    const SDIdx sd = A.sd;
    const int warp = threadIdx.x >> 5;
    const int kc = pcg_chunk_diags(sd);
    const int nchunk = (int)pcg_chunks(sd);
    const int nwarps = T.size * warps;
    // chunks c_begin, c_begin + nwarps, ...: every SM quarter gets as many, few or many
    const int c_begin = warp * T.size + T.rank, c_end = nchunk;
    R.buf = ring_offset(A.K, sd.D) + (unsigned)(warp % A.K) * A.stages * kStageBytes<F>;
    const bool masked = !A.all_red, pressure = A.rowsum_zero;
    const double *part = A.partials;

    if (A.mode & PCG_FACTOR) {
        const int nq = (sd.H + 31) / 32;
        for (int q = warp * T.size + T.rank; q < nq; q += nwarps) {
            const Chan in{A.halo + (size_t)(q > 0 ? q - 1 : 0) * sd.W, q > 0}, out{A.halo + (size_t)q * sd.W, q + 1 < nq};
            if (q > 0) factor_rows<F, true>(A, q, in, out);
            else factor_rows<F, false>(A, q, in, out);
        }
        team_barrier(T, A.fl);
        coefs<F, REF>(A, c_begin, c_end, nwarps, kc);  // used after start()'s barrier
    }
    if (!(A.mode & PCG_SOLVE)) return;

    if (masked) start<true>(A, c_begin, c_end, nwarps, kc);
    else start<false>(A, c_begin, c_end, nwarps, kc);
    team_barrier(T, A.fl);
    // The forward sweep, and meanwhile the maximum norm of r from its partials, by a
    // warp that has nothing to do in this sweep (on its own it is 2.5 to 6.5 K cycles
    // of every iteration).
    auto forward = [&]() -> double {
        sweep_all<F, REF, false>(A, T, R);
        if (warp == 2 * A.K) max_of(part, nchunk, sm);
        team_barrier(T, A.fl);
        return sm[0];
    };
    // z = M^-1 r  (:351)
    double maxError = forward();
    sweep_all<F, REF, true>(A, T, R);
    team_barrier(T, A.fl);

    // dot product and sigma from their partials
    auto dot_of = [&]() -> double {
        if constexpr (REF) return ref_total(part + nchunk, ref_chunks(sd), sm + kSums);
        else return total_of(part + nchunk, nchunk, sm + kSums);
    };
    auto sigma_of = [&]() -> double {
        if constexpr (REF) {
            ref_dot_zr(A, T);
            team_barrier(T, A.fl);
            return ref_total(part + 2 * nchunk, ref_chunks(sd), sm + 2 * kSums);
        } else {
            return total_of(part + 2 * nchunk, sd.S, sm + 2 * kSums);
        }
    };
    double sigma = sigma_of();
    int iterations = 0, status;
    if (A.pinned >= 0 ? A.pinned == 0 : maxError < kTol) {
        status = 1;
    } else {
        status = 2;
        double beta = 0.0;
        // the search direction alternates between sa and sb (the matvec reads one
        // and writes the other): iteration k writes sb when k is even
        for (int iter = 0; iter < A.limit; iter++) {
            // block-uniform: every thread of the block leaves together
            if ((iter & 15) == 0 && __syncthreads_or(threadIdx.x == 0 && timed_out(A.fl))) break;
            if constexpr (REF) ref_matvec(A, T, iter, beta);
            else if (sizeof(F) == 8 || !pressure) matvec<false>(A, iter, (F)beta, c_begin, c_end, nwarps, kc);
            else matvec<true>(A, iter, (F)beta, c_begin, c_end, nwarps, kc);
            team_barrier(T, A.fl);
            const double alpha = sigma / dot_of();
            constexpr bool kRowsum = sizeof(F) == 4;  // FP64 passes are the same for every matrix
            if (!pressure) axpy<REF, false, true>(A, iter, alpha, c_begin, c_end, nwarps, kc);
            else if (masked) axpy<REF, kRowsum, true>(A, iter, alpha, c_begin, c_end, nwarps, kc);
            else axpy<REF, kRowsum, false>(A, iter, alpha, c_begin, c_end, nwarps, kc);
            team_barrier(T, A.fl);
            iterations = iter + 1;
            // z = M^-1 r; sigmaNew = z.r  (:372-376); a solve that has converged has
            // swept forward once too often, which changes neither p nor r
            maxError = forward();
            if (A.pinned >= 0 ? iterations >= A.pinned : maxError < kTol) {
                status = 0;
                break;
            }
            sweep_all<F, REF, true>(A, T, R);
            team_barrier(T, A.fl);
            const double sigmaNew = sigma_of();
            beta = sigmaNew / sigma;
            sigma = sigmaNew;
        }
        if (status == 2) iterations = A.limit;
    }
    if (T.rank == 0 && threadIdx.x == 0) {
        A.out->iterations = iterations;
        A.out->status = status;
        A.out->max_error = maxError;
        atomicAdd(A.iter_total, (unsigned long long)iterations);
    }
}

// The form of the solve: see k_pcg64.cu.
template <typename F>
__device__ __forceinline__ void pcg_solve(const PcgArgs<F> &A, Team &T, Ring<F> &R, double *sm) {
    if constexpr (sizeof(F) == 4) {
        pcg_job<F, false>(A, T, R, sm);
    } else {
        if (A.ref) pcg_job<F, true>(A, T, R, sm);
        else pcg_job<F, false>(A, T, R, sm);
    }
}

// Ring state of this warp (its role's position); the mbarriers are initialised
// once per launch.
template <typename F>
__device__ void ring_init(Ring<F> &R, int K, int stages) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    R.buf = 0u;
    R.bars = 8u * Ring<F>::KINDS * kMaxStages * (warp % K);
    R.stages = stages;
    R.st = 0;
    R.parity = 0u;
    R.dead = false;
    if (lane == 0 && warp < K) {
        for (int k = 0; k < stages; k++) {
            mbar_init(R.bar(Ring<F>::COPIED, k), 1);
            mbar_init(R.bar(Ring<F>::PREPARED, k), 1);
            mbar_init(R.bar(Ring<F>::READY, k), 1);
            mbar_init(R.bar(Ring<F>::FREE, k), 1);
        }
        fence_mbar_init();
    }
}

template <typename F>
__global__ void __launch_bounds__(kMaxThreads<F>, 1) pcg_kernel(PcgArgs<F> A) {
    __shared__ double sm[3 * kSums];
    Team T{(int)blockIdx.x, (int)gridDim.x, A.barrier, 0u};
    Ring<F> R;
    ring_init(R, A.K, A.stages);
    const size_t nh = 2 * (size_t)(A.K > 1 ? A.K - 1 : 0) * pcg_halo_row(A.sd);
    for (size_t k = threadIdx.x; k < nh; k += blockDim.x)
        ((unsigned long long *)(g_smem + halo_offset(A.K)))[k] = kSentinel;
    __syncthreads();
    pcg_solve(A, T, R, sm);
}

// Many independent scenes in one cooperative launch (see BatchTeams).
template <typename F>
__global__ void __launch_bounds__(kBatchThreads, 1)
    pcg_batch_kernel(const PcgArgs<F> *jobs, BatchTeams B, int mode, int heat, int pinned, int K, int stages) {
    __shared__ double sm[3 * kSums];
    __shared__ PcgArgs<F> sA;
    __shared__ int s_slot;
    const int2 bt = batch_slot(B, &s_slot);
    const int2 tm = B.team[bt.x];
    Team T{bt.y, tm.x, B.team_bar + kBarStride * bt.x, 0u};
    Ring<F> R;
    ring_init(R, K, stages);
    __syncthreads();
    while (batch_take<F>(B, T, bt.x, tm.y, jobs, sA, mode, heat, pinned, K, stages)) {
        // halo rows start at the sentinel: the shared rows of this block
        // (their length changes with the scene) and the scene's global rows
        const size_t nh = 2 * (size_t)(K > 1 ? K - 1 : 0) * pcg_halo_row(sA.sd);
        for (size_t k = threadIdx.x; k < nh; k += blockDim.x)
            ((unsigned long long *)(g_smem + halo_offset(K)))[k] = kSentinel;
        const size_t ng = pcg_halo_words(sA.sd);
        for (size_t k = (size_t)T.rank * blockDim.x + threadIdx.x; k < ng; k += (size_t)T.size * blockDim.x)
            sA.halo[k] = kSentinel;
        team_barrier(T, sA.fl);
        pcg_solve(sA, T, R, sm);
    }
}

constexpr int kSingleThreads = 256, kSingleStages = 8;

template <typename F>
size_t pcg_smem(int K, int D, int stages) { return ring_offset(K, D) + (size_t)K * stages * kStageBytes<F>; }

// What a shape {threads, strips per block, stages} comes to: at least a strip's
// four warps per strip, as many strips and stages as threads and shared memory
// allow (smem: bytes of a block).
template <typename F>
void pcg_shape(int threads, int D, size_t smem_max, int *block, int *K, int *stages) {
    *K = std::min(*K, kBatchThreads / (32 * kRoles));
    while (*stages > 2 && pcg_smem<F>(*K, D, *stages) > smem_max) (*stages)--;
    while (*K > 1 && pcg_smem<F>(*K, D, *stages) > smem_max) (*K)--;
    *block = std::max(threads, 32 * kRoles * *K);
}

template <typename F>
cudaError_t launch_single(PcgArgs<F> A, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
                          int *blocks_used) {
    const SDIdx &sd = A.sd;
    A.mode = cfg.mode;
    A.limit = cfg.limit;
    A.pinned = cfg.pinned;
    // A strip per SM: two would hand over through its shared memory, but in the
    // backward sweep they also share its bandwidth (copies, preparer and sweep
    // move 11 KB per step, 86 cycles).
    A.K = 1;
    A.stages = kSingleStages;
    A.fl.limit = cfg.wait_limit > 0 ? cfg.wait_limit : kWaitLimit;
    const size_t smem = pcg_smem<F>(A.K, sd.D, A.stages);
    const void *fn = (const void *)pcg_kernel<F>;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // one block per SM; small scenes: as many blocks as give every chunk an SM
    // quarter (FP64 instructions of one quarter do not overlap)
    const int want = std::max((sd.S + A.K - 1) / A.K, (int)((pcg_chunks(sd) + 3) / 4));
    const int G = std::max(1, std::min(std::min(sms, X.max_blocks), want));
    if (blocks_used) *blocks_used = G;
    e = cudaMemsetAsync(X.barrier, 0, sizeof(unsigned), st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(X.halo, 0xff, pcg_halo_words(sd) * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    // FP32 grids with more chunks than the warps of 256-thread blocks (above about
    // 550^2): twice the warps for the elementwise passes.  Cycles per iteration of
    // matvec and AXPYs, without their barriers, 256 and 512 threads: 768^2 33K and 28K,
    // 1536^2 88K and 58K (clock counters of a scratch copy); smaller grids only have more warps at the barriers.
    const int threads = sizeof(F) == 4 && pcg_chunks(sd) > (size_t)sms * kSingleThreads / 32 ? kMaxThreads<F> : kSingleThreads;
    void *args[] = {&A};
    return cudaLaunchCooperativeKernel(fn, dim3(G), dim3(threads), args, smem, st);
}

}  // namespace

}  // namespace ifl

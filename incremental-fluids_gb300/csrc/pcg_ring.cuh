// pcg_ring.cuh - the parts of the PCG kernels that do not depend on what a lane
// does in a step of a sweep: the ring that feeds a sweeping warp, the MIC(0)
// factor, fixed-order sums (k_pcg64.cu, k_pcg32.cu).
#pragma once
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "pcg_common.cuh"

namespace ifl {

namespace {

// The order of the sums that scenes with bodies keep in FP64 (k_pcg64.cu): chunks
// of kRefChunk diagonals, in which each lane adds its cells in the order of the
// diagonals and the lanes follow a shuffle tree; then lane l of one warp adds the
// chunks l, l + 32, ... and the lanes follow the same tree.
constexpr int kRefChunk = 16;
__device__ __forceinline__ int ref_chunks(const SDIdx &sd) { return sd.S * sd.D / kRefChunk; }
__device__ __forceinline__ double ref_total(const double *pt, int n, double *sm) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        double acc = 0.0;
        for (int c0 = lane; c0 < n; c0 += 32 * 8) {
            double v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = c0 + 32 * j < n ? __ldcg(pt + c0 + 32 * j) : 0.0;
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (c0 + 32 * j < n) acc = acc + v[j];
        }
        acc = warp_sum(acc);
        if (lane == 0) sm[0] = acc;
    }
    __syncthreads();
    return sm[0];
}

// Steps of a ring block, and cells of a diagonal (see SDIdx).
template <typename F> struct Lay;
template <> struct Lay<double> { static constexpr int kSteps = 8, kCells = 32; };
template <> struct Lay<float> { static constexpr int kSteps = kTileBlock, kCells = 256; };
template <typename F> constexpr unsigned kVecBytes = Lay<F>::kSteps * Lay<F>::kCells * sizeof(F);  // a block of one array
template <typename F> constexpr unsigned kHaloAt = 4u * kVecBytes<F>;       // its halo words, behind four arrays
template <typename F> constexpr unsigned kStageBytes = kHaloAt<F> + 128u;   // a ring stage
constexpr int kMaxStages = 8;
// Threads of a block at most.  The batched passes are bound by how many 128-thread
// blocks an SM holds, three at 160 registers and four at 128 (512 FP32 scenes of 64^2
// to 768^2: 381 and 316 ms; 256 FP64 scenes to 512^2: 427 and 375 ms); the FP64
// form's single solves have a block per SM and would only spill.
constexpr int kBatchThreads = 512;
template <typename F> constexpr int kMaxThreads = sizeof(F) == 4 ? 512 : 384;
constexpr int kRoles = 4;   // warps that work on one strip: sweep, load, prepare, take
constexpr int kSums = 16;   // partial sums of a reduction (see total_of)

// ---------------------------------------------------------- conversions
// float <-> double on the integer pipe.  A conversion instruction takes an FP64
// slot (19 cycles per warp and SM on this part), these take about eight integer
// instructions (2 cycles).  Zeros and normal numbers here; subnormals,
// infinities and NaN take the instruction.
__device__ __forceinline__ double to_f64(float f) {
    const unsigned u = __float_as_uint(f), t = u & 0x7fffffffu;
    unsigned hi = (t >> 3) + 0x38000000u, lo = u << 29;
    if (t - 0x00800000u >= 0x7f000000u) {  // zero, subnormal, infinity, NaN
        if (t != 0u) return (double)f;
        hi = 0u;
        lo = 0u;
    }
    return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)lo);
}
// Round to nearest even, as the instruction.
__device__ __forceinline__ float to_f32(double d) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d), t = hi & 0x7fffffffu;
    if (t - 0x38100000u >= 0x0fe00000u) {  // outside [2^-126, 2^128): zero, subnormal result, overflow, NaN
        if ((t | lo) != 0u) return (float)d;
        return __uint_as_float(hi & 0x80000000u);
    }
    unsigned m = ((t - 0x38000000u) << 3) | (lo >> 29);
    const unsigned rest = lo & 0x1fffffffu;
    m += (rest > 0x10000000u || (rest == 0x10000000u && (m & 1u))) ? 1u : 0u;
    return __uint_as_float(m | (hi & 0x80000000u));
}

template <typename F> __device__ __forceinline__ F from_f64(double d);
template <> __device__ __forceinline__ double from_f64<double>(double d) { return d; }
template <> __device__ __forceinline__ float from_f64<float>(double d) { return to_f32(d); }
__device__ __forceinline__ double to_f64(double d) { return d; }

// The MIC(0) coefficients lie as the sweeps read them, a diagonal's arrays side by
// side: those of the forward sweep, then, behind them all, those of the backward
// sweep.  In the L D L^T form -al, -bd and dd, -a, -b (k_pcg32.cu); in the
// reference's own form (REF, see k_pcg64.cu) lx of the left cell, ly of the lower
// cell, pc and lx, ly, pc, with lx = aPlusX pc and ly = aPlusY pc.  FP64: a cell's
// two neighbour coefficients side by side (one 16-byte load of the sweep).
template <bool REF, bool BWD> constexpr int kCoefs = REF || BWD ? 3 : 2;
enum { C_LEFT = 0, C_DOWN = 1, C_RIGHT = 1, C_UP = 2, C_DD = 0, R_RIGHT = 0, R_UP = 1, R_PC = 2 };
// Array `arr` of the cell with slot k.
template <bool REF, bool BWD, typename F>
__device__ __forceinline__ F *coef(const PcgArgs<F> &A, size_t k, int arr) {
    constexpr int n = Lay<F>::kCells, c = kCoefs<REF, BWD>, pair = BWD && !REF ? 1 : 0;
    F *row = A.mic + (BWD ? kCoefs<REF, false> * A.sd.total() : 0) + (k / n) * (c * n);
    if (sizeof(F) == 8 && (arr == pair || arr == pair + 1)) return row + pair * n + (k % n) * 2 + arr - pair;
    return row + arr * n + k % n;
}

// --------------------------------------------------------------- sweeps
// A strip's ring in shared memory: `stages` buffers of kSteps diagonals,
//   [r][al, bd per diagonal] (forward) or [y][dd, a, b per diagonal] (backward),
//   then the halo words of the block's steps.
// Four warps share it, each with its own running position (stage, mbarrier
// parity):
//  * the loader waits for a free stage and starts two bulk copies into it;
//  * the preparer (backward, L D L^T form) waits for the copies, multiplies y by
//    dd in place and adds up sigma;
//  * the taker (where the strip has a neighbour to take from) puts the halo words
//    to the operands as they arrive;
//  * the sweeping warp waits until all that is done (`ready`), stores its results
//    and hands its boundary row on, and frees the stage.
// Every wait is bounded.  A timeout elsewhere in the launch does not shorten the
// mbarrier waits: the copies were issued from this GPU's memory and complete,
// and the taker's halo polls give up by themselves, so a timed-out sweep still
// consumes every block it issued and no bulk copy is left behind in shared memory.
// A ring is `dead` once an mbarrier wait ran out all the same: its warp then
// waits and issues no more.
template <typename F>
struct Ring {
    unsigned buf;   // byte offset of the stages in g_smem
    unsigned bars;  // byte offset of the mbarriers, kMaxStages of each kind
    int stages, st;
    unsigned parity;
    bool dead;
    enum { COPIED = 0, PREPARED = 1, READY = 2, FREE = 3, KINDS = 4 };
    __device__ __forceinline__ uint64_t *bar(int kind, int at) const {
        return (uint64_t *)(g_smem + bars) + kind * kMaxStages + at;
    }
    __device__ __forceinline__ unsigned stage(int at) const { return buf + (unsigned)at * kStageBytes<F>; }
    __device__ __forceinline__ void next() {
        st = st + 1 == stages ? 0 : st + 1;
        parity ^= st == 0 ? 1u : 0u;
    }
    __device__ __forceinline__ void skip(int n) {  // n blocks that this warp has no part in
        const int at = st + n;
        st = at % stages;
        parity ^= (unsigned)(at / stages) & 1u;
    }
};
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Whether a phase is complete, without waiting for it (try_wait suspends).
__device__ __forceinline__ bool mbar_test(uint64_t *bar, unsigned parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// This lane: phase `parity` of a barrier, tested earlier with the result `done`.
template <typename F>
__device__ __forceinline__ void ring_wait_lane(Ring<F> &R, uint64_t *bar, unsigned parity, bool done, const Flags &flags) {
    if (done) return;
    long long n = 0;
    while (!R.dead && !mbar_try_wait(bar, parity)) {
        if (++n > kMbarWaitLimit + flags.limit) {
            set_timeout(flags);
            R.dead = true;
        }
    }
}
// Whole warp: the phase `parity` of a barrier.
template <typename F>
__device__ __forceinline__ void ring_wait(Ring<F> &R, uint64_t *bar, unsigned parity, const Flags &flags) {
    if (__all_sync(FULL, R.dead || mbar_try_wait(bar, parity))) return;
    long long n = 0;
    while (!__all_sync(FULL, mbar_try_wait(bar, parity))) {
        if (++n > kMbarWaitLimit + flags.limit) {
            set_timeout(flags);
            R.dead = true;
            break;
        }
    }
}

// The halo word of step j of a block, into its stage.  FP64: behind the operands,
// as the reference's order of operations is kept (k_pcg64.cu).  FP32: folded into
// the edge lane's operands, r (or dd y) += b * word, and b = 0, so that the sweep
// needs no word of its own (reading and selecting it took 6 cycles per step).
template <typename F, bool BWD>
__device__ __forceinline__ void put_halo(char *stage, int j, unsigned long long w) {
    if constexpr (sizeof(F) == 8) {
        *(volatile unsigned long long *)(stage + kHaloAt<F> + 8 * j) = w;
    } else {
        constexpr int kC = kCoefs<false, BWD>, kEdge = BWD ? 31 * 16 + 12 : 0;  // element w of lane 31, x of lane 0
        const int jj = BWD ? Lay<F>::kSteps - 1 - j : j;
        float *r = (float *)(stage + jj * 1024 + kEdge);
        float *b = (float *)(stage + kVecBytes<F> + (jj * kC + kC - 1) * 1024 + kEdge);
#pragma unroll
        for (int e = 0; e < 2; e++) {  // the tile's columns, 512 bytes apart
            r[128 * e] = fmaf(b[128 * e], __uint_as_float((unsigned)(w >> (32 * e))), r[128 * e]);
            b[128 * e] = 0.f;
        }
    }
}

// The loader's part of one strip: the bulk copies, as stages become free.
template <typename F, bool REF, bool BWD>
__device__ __noinline__ void load_strip(const PcgArgs<F> &A, int s, Ring<F> &ring, bool in) {
    constexpr int kC = kCoefs<REF, BWD>;  // coefficient arrays
    constexpr bool kPrepared = BWD && !REF;  // the preparer stands between the copies and the sweep
    constexpr int kT = Lay<F>::kSteps, kCells = Lay<F>::kCells;
    constexpr unsigned kVec = kVecBytes<F>;
    if (ring.dead) return;
    Ring<F> R = ring;
    const Flags flags = A.fl;
    const int D = A.sd.D, nblk = D / kT;
    const size_t row0 = (size_t)s * D + (BWD ? D - kT : 0);  // first diagonal of the first block
    const F *vec = (BWD ? A.z : A.rf) + row0 * kCells;
    const F *cf = coef<REF, BWD>(A, row0 * kCells, 0);
    fence_proxy_async_global();  // generic-proxy writes before this sweep -> bulk copies
    for (int blk = 0; blk < nblk; blk++) {
        if (!__all_sync(FULL, mbar_try_wait(R.bar(Ring<F>::FREE, R.st), R.parity ^ 1u))) {
            ring_wait(R, R.bar(Ring<F>::FREE, R.st), R.parity ^ 1u, flags);
            if (R.dead) break;
        }
        if ((threadIdx.x & 31) == 0) {
            // without preparer and halo words the sweeping warp itself waits for the
            // copies; the barriers that nobody waits for keep pace
            uint64_t *ready = R.bar(Ring<F>::READY, R.st), *copied = R.bar(Ring<F>::COPIED, R.st);
            uint64_t *tx = kPrepared || in ? copied : ready;
            char *dst = g_smem + R.stage(R.st);
            fence_proxy_async_shared();  // what was written into the stage by hand -> bulk copies
            mbar_expect_tx(tx, (1u + kC) * kVec);
            bulk_g2s(dst, vec, kVec, tx);
            bulk_g2s(dst + kVec, cf, kC * kVec, tx);
            if (!kPrepared) mbar_arrive(R.bar(Ring<F>::PREPARED, R.st));
            if (!kPrepared && !in) mbar_arrive(copied);
        }
        vec += BWD ? -kT * kCells : kT * kCells;
        cf += (BWD ? -kT * kCells : kT * kCells) * kC;
        R.next();
    }
    ring = R;
    __syncwarp();
}

// The taker's part of one strip: the halo words.  At step t the edge lane needs the
// boundary value of one column (a double, or the two floats of a tile's columns)
// in one 8-byte word of the neighbour's row (t <= D - 32; beyond, the coefficient
// is zero).  Lane i polls the word of the i-th step from the first block that
// waits for words, so one round of loads (about 700 cycles) serves up to eight
// blocks.  A warp of its own: with the copies in the same loop a round served
// little more than a block in the time that the sweep takes for one (640 cycles),
// and every strip behind another fell back further at every block.
template <typename F, bool REF, bool BWD>
__device__ __noinline__ void take_strip(const PcgArgs<F> &A, Ring<F> &ring, const Chan in) {
    constexpr bool kPrepared = BWD && !REF;
    constexpr int kT = Lay<F>::kSteps;
    Ring<F> R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31, D = A.sd.D, nblk = D / kT;
    unsigned long long w = kSentinel;
    bool given_up = false;
    long long polls = 0;
    for (int ready = 0; ready < nblk;) {  // blocks whose words are in place
        const int t = ready * kT + lane;
        const bool need = t <= D - 32;
        unsigned long long *word = in.row + (BWD ? D - 32 - t : t + 32);
        // poll when the next block lacks a word, for all that are missing
        const bool missing = need && w == kSentinel && !given_up;
        if ((__ballot_sync(FULL, missing) & ((1u << kT) - 1u)) != 0u && missing) {
            asm volatile("ld.relaxed.gpu.u64 %0, [%1];" : "=l"(w) : "l"(word));
            if (w != kSentinel) asm volatile("st.relaxed.gpu.u64 [%0], %1;" ::"l"(word), "l"(kSentinel));
        }
        if (!need) w = 0ull;
        // the operands, which the words are put behind or folded into, of the blocks that fit the ring
        const int q = lane / kT;
        const bool wrapped = R.st + q >= R.stages;
        const int st = R.st + q - (wrapped ? R.stages : 0);
        bool there = (w != kSentinel || given_up) && q < R.stages;
        if (there)
            there = R.dead || mbar_test(R.bar(kPrepared ? Ring<F>::PREPARED : Ring<F>::COPIED, st), R.parity ^ (wrapped ? 1u : 0u));
        const unsigned have = __ballot_sync(FULL, there);
        // blocks that have all they need
        const int k = min((have == FULL ? 32 : __ffs(~have) - 1) / kT, nblk - ready);
        if (k > 0) {
            polls = 0;
            if (q < k) put_halo<F, BWD>(g_smem + R.stage(st), lane % kT, given_up && w == kSentinel ? 0ull : w);
            __syncwarp();
            if (lane < k) {
                int at = R.st + lane;
                at -= at >= R.stages ? R.stages : 0;
                mbar_arrive(R.bar(Ring<F>::READY, at));
            }
            w = __shfl_down_sync(FULL, w, (k * kT) & 31);
            if (lane >= 32 - k * kT) w = kSentinel;
            ready += k;
            R.skip(k);
        } else if (++polls > flags.limit || ((polls & 15) == 0 && __any_sync(FULL, timed_out(flags)))) {
            if (!given_up) set_timeout(flags);
            given_up = true;
            R.dead = polls > kMbarWaitLimit + flags.limit;
        }
    }
    ring = R;
    __syncwarp();
}

// --------------------------------------------------------------- factor
// buildPreconditioner (3-conjugate-gradients/Fluid.cpp:253-269): FP64
// arithmetic in the reference's order (the factor is bit-identical), so the
// step's FP64 instructions at 64 cycles each (one warp of an SM quarter), most of
// them in the square root and the division, are what it costs: rows, not tiles,
// are spread over the warps - lane l of a warp walks row 32 q + l, one column
// behind lane l - 1 - and the step does nothing that need not be in the chain: the
// sweeps' coefficients are formed from the factor afterwards (coefs), everywhere
// at once.  A cell forms the terms that its right and upper neighbours subtract
// from their diagonals (the same products the reference forms there).  The upper
// term of row 32 q - 1 arrives through a halo row of W words.
template <typename F, bool IN>
__device__ __noinline__ void factor_rows(const PcgArgs<F> &A, int q, const Chan in, const Chan out) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int W = sd.W, H = sd.H, y = 32 * q + lane;
    const bool rowok = y < H;
    const size_t base = sd.slot(0, rowok ? y : 0);
    auto at = [](size_t row, int x) { return sizeof(F) == 8 ? row + (size_t)x * 32 : row + (size_t)(x >> 1) * 256 + (x & 1) * 128; };
    // operands of the step after the current one
    F ndiag = F(0), nax = F(0), nay = F(0);
    unsigned nbits = 0u;
    unsigned long long nword = kSentinel;
    auto prefetch = [&](int t) {
        const int x = t - lane;
        if (rowok && x >= 0 && x < W) {
            const size_t k = at(base, x);
            ndiag = A.adiag[k];
            nax = A.ax[k];
            nay = A.ay[k];
            nbits = A.nb[k];
        }
        if constexpr (IN) nword = hload_if(in, t, lane == 0 && t < W, kSentinel);
    };
    double left = 0.0, upper = 0.0;  // terms for the right and the upper neighbour of the previous cell
    prefetch(0);
    for (int t = 0; t < W + 31; t++) {
        const int x = t - lane;
        const bool active = rowok && x >= 0 && x < W;
        const double diag = to_f64(ndiag), ax = to_f64(nax), ay = to_f64(nay);
        const unsigned b = active ? nbits : 0u;
        double down = __shfl_up_sync(FULL, upper, 1);
        if constexpr (IN) {
            const bool need = lane == 0 && t < W;
            const unsigned long long w = halo_take_warp(in, t, need, nword, A.fl);
            if (need) down = hdec(w);
        }
        if (t + 1 < W + 31) prefetch(t + 1);
        double ev = diag;
        if (b & NB_LEFT) ev = ev - left;
        if (b & NB_DOWN) ev = ev - down;
        if (ev < kSigma * diag) ev = diag;
        const double pcv = 1.0 / sqrt(ev);
        const double px = ax * pcv, py = ay * pcv, txy = kTau * px * py;
        left = px * px + txy;
        upper = py * py + txy;
        if (b & NB_SELF) A.pc[at(base, x)] = pcv;
        hstore_if(out, x, henc(upper), out.valid && lane == 31 && active);
    }
}

// The sweeps' coefficients of this warp's chunks, from the factor.  A cell writes
// its own backward ones and the forward ones of its right and upper neighbours.
template <typename F, bool REF>
__device__ __noinline__ void coefs(const PcgArgs<F> &A, int c_begin, int c_end, int c_step, int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    for (int row = c_begin * kc; row < c_end * kc; row += (row + 1) % kc ? 1 : (c_step - 1) * kc + 1) {
        const int s = row / sd.D, d = row - s * sd.D;
#pragma unroll
        for (int i = 0; i < Lay<F>::kCells / 32; i++) {
            const int idx = 32 * i + lane, l = sizeof(F) == 8 ? idx : (idx >> 2) & 31;
            const int x = sizeof(F) == 8 ? d - l : 2 * (d - l) + (idx >> 7);
            const int y = sizeof(F) == 8 ? 32 * s + l : 4 * (32 * s + l) + (idx & 3);
            if (x < 0 || x >= sd.W || y >= sd.H) continue;
            const size_t k = (size_t)row * Lay<F>::kCells + idx;
            const double pcv = A.pc[k], p2 = !(A.nb[k] & NB_SELF) ? 0.0 : REF ? pcv : pcv * pcv;
            const F sign = REF ? F(1) : F(-1), dd = from_f64<F>(p2);
            // A neighbour that does not exist has a zero coefficient, whatever the matrix
            // holds there: lane 31 (0) of a strip without one sees its own previous value.
            const bool right = x + 1 < sd.W, upper = y + 1 < sd.H;
            const F va = sign * from_f64<F>(right ? to_f64(A.ax[k]) * p2 : 0.0),
                    vb = sign * from_f64<F>(upper ? to_f64(A.ay[k]) * p2 : 0.0);
            *coef<REF, true>(A, k, REF ? R_RIGHT : C_RIGHT) = va;
            *coef<REF, true>(A, k, REF ? R_UP : C_UP) = vb;
            *coef<REF, true>(A, k, REF ? R_PC : C_DD) = dd;
            if (REF) *coef<REF, false>(A, k, R_PC) = dd;
            if (right) *coef<REF, false>(A, sd.slot(x + 1, y), C_LEFT) = va;
            if (upper) *coef<REF, false>(A, sd.slot(x, y + 1), C_DOWN) = vb;
        }
    }
}

// Sum of n partials in a fixed order that depends on n alone:
// virtual warp v < kSums adds the partials v*32 + lane + 512 k in order of k,
// its lanes follow a fixed shuffle tree, and so do the kSums results.  Every
// block forms the same bits, whatever its number of warps.
__device__ __forceinline__ double total_of(const double *pt, int n, double *sm) {
    const int warps = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (n <= 32) {  // every warp for itself
        double acc = lane < n ? __ldcg(pt + lane) : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            if (o >= n) continue;
            const double w = __shfl_down_sync(FULL, acc, o);
            acc = acc + w;
        }
        return __shfl_sync(FULL, acc, 0);
    }
    for (int v = warp; v < kSums; v += warps) {
        double acc = 0.0;
        if (v * 32 < n) {
            for (int i0 = v * 32 + lane; i0 < n; i0 += 4 * 32 * kSums) {
                double w[4];
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = i0 + j * 32 * kSums < n ? __ldcg(pt + i0 + j * 32 * kSums) : 0.0;
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (i0 + j * 32 * kSums < n) acc = acc + w[j];
            }
            acc = warp_sum(acc);
        }
        if (lane == 0) sm[v] = acc;
    }
    __syncthreads();
    double acc = sm[lane & (kSums - 1)];
    const int used = (n + 31) / 32;  // sums beyond are zero
    for (int o = kSums / 2; o > 0; o >>= 1) {
        if (o >= used) continue;
        const double w = __shfl_xor_sync(FULL, acc, o);
        acc = acc + w;
    }
    return __shfl_sync(FULL, acc, 0);
}

// std::max(maxError, |r|) on the bit patterns: non-negative doubles order as
// unsigned integers; a NaN (above +inf) is skipped, as (maxError < NaN) is false.
__device__ __forceinline__ void max_bits(unsigned long long &mx, double r) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
    if (b <= 0x7ff0000000000000ull && b > mx) mx = b;
}
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(FULL, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// Maximum of n partials that max_bits formed, by one warp, into sm[0].
__device__ __forceinline__ void max_of(const double *pt, int n, double *sm) {
    unsigned long long mx = 0ull;
    for (int c0 = threadIdx.x & 31; c0 < n; c0 += 32 * 8) {
        double v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = c0 + 32 * j < n ? __ldcg(pt + c0 + 32 * j) : 0.0;
#pragma unroll
        for (int j = 0; j < 8; j++) max_bits(mx, v[j]);
    }
    mx = warp_max_bits(mx);
    if ((threadIdx.x & 31) == 0) sm[0] = __longlong_as_double((long long)mx);
}

}  // namespace

}  // namespace ifl

// k_pcg32.cu - the FP32 form's MIC(0)-preconditioned conjugate gradients as one
// persistent cooperative kernel per solve, or per batch of solves (sm_103a).
//
// Reference: FluidSolver::project (3-conjugate-gradients/Fluid.cpp:349-380),
// buildPreconditioner (:247-272), applyPreconditioner (:275-304),
// matrixVectorProduct (:315-332), dotProduct/scaledAdd/infinityNorm (:307-346);
// masked forms in 4-solid-boundaries/Fluid.cpp:656-721 and
// 6-heat/Fluid.cpp:781-826.
//
// Data: the arrays of the pressure system lie in the tile form of the
// strip-diagonal layout (SDIdx with ts = 1): a lane owns tiles of 2 columns x 4
// rows, a strip is 32 tile rows (128 cells) and is stored tile diagonal by tile
// diagonal, each as the lanes' first columns (a float4 of 4 rows per lane), then
// their second columns.  Slots outside the grid hold zeros in every array and
// stay zero: a neighbour that does not exist has a zero coefficient, so no pass
// needs neighbour tests.
//
// The MIC(0) preconditioner is applied in its L D L^T form.  With pc the
// reference's factor, the reference's two substitutions
//     q = (r - aPlusX_l pc_l q_l - aPlusY_d pc_d q_d) pc
//     z = (q - aPlusX pc z_r - aPlusY pc z_u) pc
// become, with y = q / pc,
//     y = r - al y_l - bd y_d,          z = dd y - a z_r - b z_u,
//     a = aPlusX pc^2, b = aPlusY pc^2, dd = pc^2, al = a of the left cell,
//     bd = b of the lower cell:
// one fused multiply-add per neighbour on the dependency chain where the
// reference's order needs a multiply, two subtractions and another multiply,
// and 12 (16) bytes of operands per cell where {q, MIC(0) record} took 20.
//
// What bounds the sweeps: one warp walks a strip, and a lone warp pays two to
// four cycles for every instruction, beside a dependency chain per wavefront
// step of a shuffle (25 cycles) and six fused multiply-adds (5 each).  So a step
// does eight cells of every lane, nothing in it depends on the position in the
// grid (the padding is computed along), and two more warps per strip take from
// the sweeping warp what is not on the chain: a loader fills a ring in shared
// memory and takes the neighbouring strip's boundary row, and in the backward
// sweep a preparer forms dd y and sigma.  What is left per step is 6 loads of 16
// bytes from shared memory, 16 fused multiply-adds, two shuffles and three
// stores: 150 cycles, of which the multiply-adds are 63, the loads 45, the
// stores 30 (timed with each left out).
//
// r and p are FP64; the matvec is FP32 (its results are stored as they are
// formed), dot products, the maximum norm, alpha and beta are FP64.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "pcg_common.cuh"

namespace ifl {

namespace {

constexpr int kT = kTileBlock;                    // tile diagonals per block of a ring
constexpr int kDepth = 2;                         // steps whose operands are in registers (divides kT)
constexpr unsigned kVecBytes = kT * 1024u;        // a block of one array
constexpr unsigned kHaloAt = 4u * kVecBytes;      // halo words of a block behind the operands of the backward sweep
constexpr unsigned kStageBytes = kHaloAt + 128u;  // a ring stage
constexpr int kMaxStages = 8;
constexpr int kRoles = 3;                         // warps that work on one strip: sweep, load, prepare
constexpr int kSums = 16;                         // partial sums of a reduction (see total32)

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

// Float-float numbers (hi + lo, |lo| <= ulp(hi)/2): an exact product of two
// floats and a sum with an error-free two-sum of the high parts (Knuth's
// TwoSum; the library is compiled without contraction, so these stay exact).
struct FF {
    float hi, lo;
};
__device__ __forceinline__ FF ff_prod(float a, float b) {
    const float p = a * b;
    return FF{p, fmaf(a, b, -p)};
}
__device__ __forceinline__ FF ff_add(FF x, FF y) {
    const float s = x.hi + y.hi;
    const float bb = s - x.hi;
    const float err = (x.hi - (s - bb)) + (y.hi - bb);
    const float lo = err + x.lo + y.lo;
    const float hi = s + lo;
    return FF{hi, lo - (hi - s)};
}

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float lo2(unsigned long long w) { return __uint_as_float((unsigned)w); }
__device__ __forceinline__ float hi2(unsigned long long w) { return __uint_as_float((unsigned)(w >> 32)); }
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// a*b + c, element by element.
__device__ __forceinline__ float4 fma4(const float4 &a, const float4 &b, const float4 &c) {
    return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w));
}
__device__ __forceinline__ float4 mul4(const float4 &a, const float4 &b) {
    return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w);
}

// The MIC(0) coefficients lie as the sweeps read them, a tile diagonal's arrays
// side by side, one base address for all: -al and -bd for the forward sweep (512
// floats per tile diagonal), then, behind them all, dd, -a and -b for the
// backward sweep (768 floats).  k: the cell's slot.
enum { C_AL = 0, C_BD = 1, C_DD = 0, C_A = 1, C_B = 2 };
__device__ __forceinline__ float *fwd_coef(const PcgArgs<float> &A, size_t k, int arr) {
    return A.mic + (k >> 8) * 512 + arr * 256 + (k & 255);
}
__device__ __forceinline__ float *bwd_coef(const PcgArgs<float> &A, size_t k, int arr) {
    return A.mic + 2 * A.sd.total() + (k >> 8) * 768 + arr * 256 + (k & 255);
}

// --------------------------------------------------------------- sweeps
// A strip's ring in shared memory: `stages` buffers of kT tile diagonals,
//   [r][al, bd per diagonal] (forward) or [y][dd, a, b per diagonal] (backward),
//   then the kT halo words of the block.
// Three warps share it, each with its own running position (stage, mbarrier
// parity):
//  * the loader waits for a free stage, starts two bulk copies into it, takes the
//    block's halo words as they arrive and puts them behind the operands;
//  * the preparer (backward) waits for the copies, multiplies y by dd in place and
//    adds up sigma;
//  * the sweeping warp waits for both (`ready`), stores its results and hands its
//    boundary row on, and frees the stage.
// Every wait is bounded.  A timeout elsewhere in the launch does not shorten the
// mbarrier waits: the copies were issued from this GPU's memory and complete,
// and the loader's halo polls give up by themselves, so a timed-out sweep still
// consumes every block it issued and no bulk copy is left behind in shared memory.
// A ring is `dead` once an mbarrier wait ran out all the same: its warp then
// waits and issues no more.
struct Ring32 {
    unsigned buf;   // byte offset of the stages in g_smem
    unsigned bars;  // byte offset of the mbarriers, kMaxStages of each kind
    int stages, st;
    unsigned parity;
    bool dead;
    enum { COPIED = 0, READY = 1, FREE = 2, KINDS = 3 };
    __device__ __forceinline__ uint64_t *bar(int kind, int at) const {
        return (uint64_t *)(g_smem + bars) + kind * kMaxStages + at;
    }
    __device__ __forceinline__ unsigned stage(int at) const { return buf + (unsigned)at * kStageBytes; }
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
// Whole warp: the phase `parity` of a barrier.
__device__ __forceinline__ void ring32_wait(Ring32 &R, uint64_t *bar, unsigned parity, const Flags &flags) {
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

// The loader's part of one strip.  Halo words: at step t the waiting lane needs
// the boundary values of one tile column, two floats in one 8-byte word, at
// in_word(t) of the neighbour's row (t <= D - 32; beyond, the coefficient is
// zero).  Lane i polls the word of the i-th step from the first block that waits
// for words, so one round of loads (about 700 cycles) serves up to eight blocks.
template <bool BWD, bool IN>
__device__ __noinline__ void load32_strip(const PcgArgs<float> &A, int s, Ring32 &ring, const Chan in) {
    constexpr int kC = BWD ? 3 : 2;  // coefficient arrays
    Ring32 R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31;
    const int D = A.sd.D, nblk = D / kT;
    const size_t row0 = (size_t)s * D + (BWD ? D - kT : 0);  // first tile diagonal of the first block
    const float *vec = (BWD ? A.z : A.rf) + row0 * 256;
    const float *cf = BWD ? bwd_coef(A, row0 * 256, C_DD) : fwd_coef(A, row0 * 256, C_AL);
    fence_proxy_async_global();  // generic-proxy writes before this sweep -> bulk copies
    int issued = 0, ready = 0;   // blocks whose copies are started, whose halo words are in place
    int rst = R.st;              // stage of block `ready`
    unsigned long long w = kSentinel;
    bool given_up = false;
    long long polls = 0;
    while (ready < nblk) {
        // start copies into free stages; wait for one only when there is nothing else to do
        while (issued < nblk && issued < ready + R.stages) {
            uint64_t *fr = R.bar(Ring32::FREE, R.st);
            if (!__all_sync(FULL, R.dead || mbar_test(fr, R.parity ^ 1u))) {
                if (issued > ready) break;
                ring32_wait(R, fr, R.parity ^ 1u, flags);
            }
            if (lane == 0) {
                // forward, the sweeping warp itself waits for the copies; `copied` keeps pace
                uint64_t *ready_bar = R.bar(Ring32::READY, R.st), *copied = R.bar(Ring32::COPIED, R.st);
                uint64_t *tx = BWD ? copied : ready_bar;
                char *dst = g_smem + R.stage(R.st);
                mbar_expect_tx(tx, (1u + kC) * kVecBytes);
                bulk_g2s(dst, vec, kVecBytes, tx);
                bulk_g2s(dst + kVecBytes, cf, kC * kVecBytes, tx);
                if (!BWD) mbar_arrive(copied);
                if (!IN) mbar_arrive(ready_bar);
            }
            vec += BWD ? -kT * 256 : kT * 256;
            cf += (BWD ? -kT * 256 : kT * 256) * kC;
            R.next();
            issued++;
            if (!IN) ready++;
        }
        if constexpr (IN) {
            const int t = ready * kT + lane;
            const bool need = t <= D - 32;
            unsigned long long *word = in.row + (BWD ? D - 32 - t : t + 32);
            if (need && w == kSentinel && !given_up) {
                asm volatile("ld.relaxed.gpu.u64 %0, [%1];" : "=l"(w) : "l"(word));
                if (w != kSentinel) asm volatile("st.relaxed.gpu.u64 [%0], %1;" ::"l"(word), "l"(kSentinel));
            }
            if (!need) w = 0ull;
            const unsigned have = __ballot_sync(FULL, w != kSentinel || given_up);
            // blocks from `ready` on whose words are all there
            int k = min(__ffs(~have) - 1 < 0 ? 32 : __ffs(~have) - 1, (issued - ready) * kT) / kT;
            if (k > 0) {
                polls = 0;
                const int q = lane / kT;
                int st = rst + q;
                st -= st >= R.stages ? R.stages : 0;
                if (q < k)
                    *(volatile unsigned long long *)(g_smem + R.stage(st) + kHaloAt + 8 * (lane % kT)) = given_up && w == kSentinel ? 0ull : w;
                __syncwarp();
                if (lane < k) {
                    int at = rst + lane;
                    at -= at >= R.stages ? R.stages : 0;
                    mbar_arrive(R.bar(Ring32::READY, at));
                }
                w = __shfl_down_sync(FULL, w, k * kT);
                if (lane >= 32 - k * kT) w = kSentinel;
                ready += k;
                rst += k;
                rst -= rst >= R.stages ? R.stages : 0;
            } else if (++polls > flags.limit || ((polls & 15) == 0 && __any_sync(FULL, timed_out(flags)))) {
                if (!given_up) set_timeout(flags);
                given_up = true;
            }
        }
    }
    ring = R;
    __syncwarp();
}

// The preparer's part of one backward strip: y becomes dd y, and sigma = z.r =
// sum of dd y^2 (see pcg32_job) is added up: sums of two fused FP32 products per
// row of the tiles and step, over a block, then FP64.
__device__ __noinline__ void prepare32_strip(const PcgArgs<float> &A, int s, Ring32 &ring) {
    Ring32 R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31, nblk = A.sd.D / kT;
    double qq = 0.0;
    for (int blk = 0; blk < nblk; blk++) {
        ring32_wait(R, R.bar(Ring32::COPIED, R.st), R.parity, flags);
        char *g = g_smem + R.stage(R.st) + lane * 16;
        float4 qs = zero4();
#pragma unroll
        for (int j = kT - 1; j >= 0; j--) {
            float4 *y = (float4 *)(g + j * 1024);
            const float4 *dd = (const float4 *)(g + kVecBytes + j * 3 * 1024);
            const float4 y0 = y[0], y1 = y[32], q0 = mul4(dd[0], y0), q1 = mul4(dd[32], y1);
            y[0] = q0;
            y[32] = q1;
            qs = fma4(q1, y1, fma4(q0, y0, qs));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(R.bar(Ring32::READY, R.st));
        qq += to_f64((qs.x + qs.y) + (qs.z + qs.w));
        R.next();
    }
    // the strip's partial: lanes by a fixed shuffle tree (independent of which
    // warp of which team works on the strip)
    qq = warp_sum(qq);
    if (lane == 0) A.partials[2 * pcg_chunks(A.sd) + s] = qq;
    ring = R;
    __syncwarp();
}

// One strip of a sweep.  At step t lane l works on tile diagonal t (backward:
// D-1-t), one tile behind lane l-1 (l+1), whose boundary row arrives by two
// shuffles; lane 0 (31) takes it from the block's halo words (IN: whether the
// strip has a neighbour to take from), and lane 31 (0) hands this strip's on
// through `out` as soon as it is formed: a word of two floats per tile column X,
// at X + 32 of the row (forward; the lane starts at X = -31) or at X (backward).
// Words of columns that no step waits for are written along and never read.
// Functions of their own: inlined, the solve's registers spill into their steps.
template <bool BWD, bool IN>
__device__ __noinline__ void sweep32_strip(const PcgArgs<float> &A, int s, Ring32 &ring, const Chan out) {
    // the vector operand (r, or dd y) and two coefficient arrays behind it (backward: a and b, after dd)
    constexpr int kC = BWD ? 3 : 2, kSkip = BWD ? 1 : 0;
    Ring32 R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int nblk = sd.D / kT;
    const bool edge = lane == (BWD ? 31 : 0), hands = out.valid && lane == (BWD ? 0 : 31);
    float4 *zp = (float4 *)A.z + ((size_t)s * sd.D + (BWD ? sd.D - kT : 0)) * 64 + lane;
    unsigned long long *op = out.row + (BWD ? sd.D - 1 : 1);  // word of this lane's first step
    float4 o0[kDepth][3], o1[kDepth][3];  // operands of kDepth steps, columns 0 and 1
    char *g = nullptr;  // this lane's column of the current block
    // operands of step j of the block into buffer j % kDepth
    auto load = [&](int j) {
        const int i = j % kDepth, jj = BWD ? kT - 1 - j : j;
        const char *v = g + jj * 1024, *c = g + kVecBytes + (jj * kC + kSkip) * 1024;
        o0[i][0] = *(const float4 *)v;
        o1[i][0] = *(const float4 *)(v + 512);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            o0[i][k + 1] = *(const float4 *)(c + k * 1024);
            o1[i][k + 1] = *(const float4 *)(c + k * 1024 + 512);
        }
    };
    float4 n = zero4();        // the previous tile's column next to this one
    float g0 = 0.f, g1 = 0.f;  // boundary row of the previous lane (columns 0, 1)
    for (int blk = 0; blk < nblk; blk++) {
        ring32_wait(R, R.bar(Ring32::READY, R.st), R.parity, flags);
        g = g_smem + R.stage(R.st) + lane * 16;
#pragma unroll
        for (int j = 0; j < kDepth; j++) load(j);
        float2 halo[kT];  // all of the block's halo words at once: no step waits for its own
        if constexpr (IN) {
            const float2 *h = (const float2 *)(g - lane * 16 + kHaloAt);
#pragma unroll
            for (int j = 0; j < kT; j++) halo[j] = h[j];
        }
#pragma unroll
        for (int j = 0; j < kT; j++) {
            if constexpr (IN) {
                g0 = edge ? halo[j].x : g0;
                g1 = edge ? halo[j].y : g1;
            }
            const int i = j % kDepth;
            float4 v0, v1;
            float h0, h1;
            if constexpr (!BWD) {  // r, -al, -bd; columns left to right, rows upward
                auto up = [](float4 t, const float4 &b, float g) {
                    t.x = fmaf(b.x, g, t.x);
                    t.y = fmaf(b.y, t.x, t.y);
                    t.z = fmaf(b.z, t.y, t.z);
                    t.w = fmaf(b.w, t.z, t.w);
                    return t;
                };
                v0 = up(fma4(o0[i][1], n, o0[i][0]), o0[i][2], g0);
                h0 = __shfl_up_sync(FULL, v0.w, 1);
                v1 = up(fma4(o1[i][1], v0, o1[i][0]), o1[i][2], g1);
                h1 = __shfl_up_sync(FULL, v1.w, 1);
                n = v1;
            } else {  // dd y, -a, -b; columns right to left, rows downward
                auto down = [](float4 t, const float4 &b, float g) {
                    t.w = fmaf(b.w, g, t.w);
                    t.z = fmaf(b.z, t.w, t.z);
                    t.y = fmaf(b.y, t.z, t.y);
                    t.x = fmaf(b.x, t.y, t.x);
                    return t;
                };
                v1 = down(fma4(o1[i][1], n, o1[i][0]), o1[i][2], g1);
                h1 = __shfl_down_sync(FULL, v1.x, 1);
                v0 = down(fma4(o0[i][1], v1, o0[i][0]), o0[i][2], g0);
                h0 = __shfl_down_sync(FULL, v0.x, 1);
                n = v0;
            }
            if (j + kDepth < kT) load(j + kDepth);
            hstore_if(Chan{op, true}, BWD ? -j : j, BWD ? pack2(v0.x, v1.x) : pack2(v0.w, v1.w), hands);
            zp[(BWD ? kT - 1 - j : j) * 64] = v0;
            zp[(BWD ? kT - 1 - j : j) * 64 + 32] = v1;
            g0 = h0;
            g1 = h1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(R.bar(Ring32::FREE, R.st));
        R.next();
        zp += BWD ? -kT * 64 : kT * 64;
        op += BWD ? -kT : kT;
    }
    ring = R;
    __syncwarp();
}

// Shared-memory layout of a block: ring mbarriers (of each strip) | the halo rows
// between its strips, K-1 upward and K-1 downward (apart, since each direction
// leaves words behind that it never reads) | the rings.
__host__ __device__ __forceinline__ unsigned halo32_offset(int K) { return 8u * Ring32::KINDS * kMaxStages * K; }
__host__ __device__ __forceinline__ unsigned ring32_offset(int K, int D) {
    const size_t nh = 2 * (size_t)(K > 1 ? K - 1 : 0) * (D + kHaloPad);
    return (unsigned)(((halo32_offset(K) + nh * 8 + 127) / 128) * 128);
}

// Sweep of all strips of this block: warps 0..K-1 sweep, K..2K-1 load for them,
// 2K..3K-1 prepare.  The team's T.size*K sweeping warps take
// the strips round-robin: warp `base` sweeps strips base, base + P, base + 2P,
// ... (P = T.size*K), in increasing order for the forward solve and in
// decreasing order for the backward solve, so that every strip waits only on a
// strip that is swept earlier by its own warp or by another warp in the same or
// an earlier round (no cycle).  When every warp has a single strip, the halo
// rows between the warps of one block live in shared memory; otherwise every
// strip hands its boundary row over through its own global row (a shared row
// would be reused by the next round while its reader may still need it).
template <bool BWD>
__device__ void sweep32(const PcgArgs<float> &A, const Team &T, Ring32 &R) {
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
        return Chan{(unsigned long long *)(g_smem + halo32_offset(A.K) + 8u * at), true};
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
            if (in.valid) sweep32_strip<BWD, true>(A, s, R, out);
            else sweep32_strip<BWD, false>(A, s, R, out);
        } else if (role == 1) {
            if (in.valid) load32_strip<BWD, true>(A, s, R, in);
            else load32_strip<BWD, false>(A, s, R, in);
        } else if (BWD) {
            prepare32_strip(A, s, R);
        } else {
            R.skip(sd.D / kT);
        }
    }
}

// --------------------------------------------------------------- factor
// buildPreconditioner (3-conjugate-gradients/Fluid.cpp:253-269): FP64
// arithmetic in the reference's order (the factor is bit-identical), so the
// step's ~35 FP64 instructions at 64 cycles each (one warp of an SM quarter)
// are what it costs: rows, not tiles, are spread over the warps - lane l of a
// warp walks row 32 q + l, one column behind lane l - 1 - and the scattered
// accesses to the tile layout hide behind them.  A cell forms the terms that
// its right and upper neighbours subtract from their diagonals (the same
// products the reference forms there) and writes their al and bd.  The upper
// term of row 32 q - 1 arrives through a halo row of W words.
template <bool IN>
__device__ __noinline__ void factor32_rows(const PcgArgs<float> &A, int q, const Chan in, const Chan out) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int W = sd.W, H = sd.H, y = 32 * q + lane;
    const bool rowok = y < H;
    const size_t base = sd.slot(0, rowok ? y : 0), above = sd.slot(0, y + 1 < H ? y + 1 : 0);
    auto at = [](size_t row, int x) { return row + (size_t)(x >> 1) * 256 + (x & 1) * 128; };
    // operands of the step after the current one
    float ndiag = 0.f, nax = 0.f, nay = 0.f;
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
            if (need) down = hdec<double>(w);
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
        const bool self = b & NB_SELF;
        const double p2 = self ? pcv * pcv : 0.0;
        const float va = to_f32(ax * p2), vb = to_f32(ay * p2);
        if (active) {
            const size_t k = at(base, x);
            if (self) A.pc[k] = pcv;
            *bwd_coef(A, k, C_A) = -va;
            *bwd_coef(A, k, C_B) = -vb;
            *bwd_coef(A, k, C_DD) = to_f32(p2);
            if (x + 1 < W) *fwd_coef(A, at(base, x + 1), C_AL) = -va;
            if (y + 1 < H) *fwd_coef(A, at(above, x), C_BD) = -vb;
        }
        hstore_if(out, x, henc(upper), out.valid && lane == 31 && active);
    }
}

// ------------------------------------------------------------------ solve
// Sum (or maximum) of n partials in a fixed order that depends on n alone:
// virtual warp v < kSums adds the partials v*32 + lane + 512 k in order of k,
// its lanes follow a fixed shuffle tree, and so do the kSums results.  Every
// block forms the same bits, whatever its number of warps.
__device__ __forceinline__ double total32(const double *pt, int n, bool is_max, double *sm) {
    const int warps = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (n <= 32) {  // every warp for itself
        double acc = lane < n ? __ldcg(pt + lane) : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            if (o >= n) continue;
            const double w = __shfl_down_sync(FULL, acc, o);
            acc = is_max ? smax(acc, w) : acc + w;
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
                    if (i0 + j * 32 * kSums < n) acc = is_max ? smax(acc, w[j]) : acc + w[j];
            }
            acc = is_max ? warp_max(acc) : warp_sum(acc);
        }
        if (lane == 0) sm[v] = acc;
    }
    __syncthreads();
    double acc = sm[lane & (kSums - 1)];
    const int used = (n + 31) / 32;  // sums beyond are zero
    for (int o = kSums / 2; o > 0; o >>= 1) {
        if (o >= used) continue;
        const double w = __shfl_xor_sync(FULL, acc, o);
        acc = is_max ? smax(acc, w) : acc + w;
    }
    return __shfl_sync(FULL, acc, 0);
}

// What a lane needs to find its tile: (strip, lane) and the tile grid.
struct Tiles {
    int s, lane, Wt;
    bool rowok;
    size_t base;  // float4 index of tile diagonal 0, column 0
    __device__ __forceinline__ Tiles(const SDIdx &sd, int strip, int l)
        : s(strip), lane(l), Wt(sd.tw()), rowok(strip * 32 + l < sd.th()), base((size_t)strip * sd.D * 64 + l) {}
    __device__ __forceinline__ bool in(int d) const { return rowok && d >= lane && d < lane + Wt; }
    __device__ __forceinline__ size_t at(int d) const { return base + (size_t)d * 64; }
};

// s = z + beta*s (first iteration: s = z), then z' = A s and z'.s over this
// warp's chunks (3-conjugate-gradients/Fluid.cpp:361-362, 375, 315-332).  A lane
// forms the new s of its tile, of the column left of it and of the column right
// of it, and of two cells for each of its neighbour lanes (the lower lane's top
// row belongs to diagonal d-1, the upper lane's bottom row to d+1), which
// arrive by shuffle; lanes 0 and 31 take theirs from the adjacent strips.  All
// of it is loaded straight into registers at once (64 words): a warp's load is
// 512 bytes, and tiles outside the grid are not fetched.
// ROWSUM (pressure: the reference's rows sum to zero: aDiag = sum of the face
// factors, each off-diagonal = -factor): the form sum_j a_ij (s_j - s_i) in
// FP32 fused multiply-adds.  It keeps the zero row sums exactly (with the
// FP32-rounded aDiag the plain form left a tiny, non-zero eigenvalue that made
// CG stagnate on some scenes, up to the 2000-iteration cap), and its terms
// carry no cancellation between the diagonal and the neighbours.  Heat
// matrices: a float-float sum of the exact products.
template <bool ROWSUM>
__device__ __noinline__ void matvec32(const PcgArgs<float> &A, int iter, float beta, int c_begin, int c_end, int c_step, int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int D = sd.D;
    const float *so = (iter & 1) ? A.sb : A.sa;
    float4 *sn = (float4 *)((iter & 1) ? A.sa : A.sb);
    const bool first = iter == 0;
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / D, d0 = c * kc - s * D;  // a chunk lies inside one strip
        const Tiles T(sd, s, lane);
        double dacc = 0.0;
        for (int u = 0; u < kc; u++) {
            const int d = d0 + u;
            const bool in = T.in(d), inL = T.in(d - 1), inR = T.in(d + 1);
            const size_t k = T.at(d);
            const float4 *z4 = (const float4 *)A.z + k, *s4 = (const float4 *)so + k, *x4 = (const float4 *)A.ax + k,
                         *y4 = (const float4 *)A.ay + k;
            float4 zc0 = zero4(), zc1 = zero4(), zl = zero4(), zr = zero4(), sc0 = zero4(), sc1 = zero4(), sl = zero4(),
                   sr = zero4(), x0 = zero4(), x1 = zero4(), xl = zero4(), y0 = zero4(), y1 = zero4(), a0 = zero4(),
                   a1 = zero4();
            // for the neighbour lanes: top row of tile d-1 (columns 0, 1) with its aPlusY, bottom row of tile d+1
            float tz0 = 0.f, tz1 = 0.f, ts0 = 0.f, ts1 = 0.f, ty0 = 0.f, ty1 = 0.f, bz1 = 0.f, bs1 = 0.f;
            // across the strip's edges (lanes 0 and 31)
            float ez0 = 0.f, ez1 = 0.f, es0 = 0.f, es1 = 0.f, ey0 = 0.f, ey1 = 0.f;
            if (in) {
                zc0 = z4[0];
                zc1 = z4[32];
                x0 = x4[0];
                x1 = x4[32];
                y0 = y4[0];
                y1 = y4[32];
                if (!ROWSUM) {
                    a0 = ((const float4 *)A.adiag)[k];
                    a1 = ((const float4 *)A.adiag)[k + 32];
                }
            }
            if (inL) {
                zl = z4[-32];
                xl = x4[-32];
                tz0 = z4[-64].w;
                ty0 = y4[-64].w;
                ty1 = y4[-32].w;
            }
            if (inR) {
                zr = z4[64];
                bz1 = z4[96].x;
            }
            // lane 0 of strip s continues below in lane 31 of strip s-1, tile
            // diagonal d+31; lane 31 above in lane 0 of strip s+1, diagonal d-31
            const bool dn = lane == 0 && s > 0 && in, up = lane == 31 && in && (s + 1) * 32 < sd.th();
            const size_t ke = dn ? (((size_t)(s - 1) * D + d + 31) * 64 + 31) * 4 + 3
                                 : (((size_t)(s + 1) * D + d - 31) * 64) * 4;
            if (dn || up) {
                ez0 = A.z[ke];
                ez1 = A.z[ke + 128];
                if (dn) {
                    ey0 = A.ay[ke];
                    ey1 = A.ay[ke + 128];
                }
            }
            if (!first) {
                if (in) {
                    sc0 = s4[0];
                    sc1 = s4[32];
                }
                if (inL) {
                    sl = s4[-32];
                    ts0 = s4[-64].w;
                }
                if (inR) {
                    sr = s4[64];
                    bs1 = s4[96].x;
                }
                if (dn || up) {
                    es0 = so[ke];
                    es1 = so[ke + 128];
                }
            }
            auto mix = [&](float z, float v) { return first ? z : fmaf(v, beta, z); };
            auto mix4 = [&](const float4 &z, const float4 &v) {
                return make_float4(mix(z.x, v.x), mix(z.y, v.y), mix(z.z, v.z), mix(z.w, v.w));
            };
            const float4 C0 = mix4(zc0, sc0), C1 = mix4(zc1, sc1), L = mix4(zl, sl), Rr = mix4(zr, sr);
            tz1 = zl.w;
            ts1 = sl.w;
            const float t0 = mix(tz0, ts0), t1 = mix(tz1, ts1), b0 = Rr.x, b1 = mix(bz1, bs1);
            float dn0 = __shfl_up_sync(FULL, t0, 1), dn1 = __shfl_up_sync(FULL, t1, 1);
            float yd0 = __shfl_up_sync(FULL, ty0, 1), yd1 = __shfl_up_sync(FULL, ty1, 1);
            float up0 = __shfl_down_sync(FULL, b0, 1), up1 = __shfl_down_sync(FULL, b1, 1);
            if (lane == 0) {
                dn0 = mix(ez0, es0);
                dn1 = mix(ez1, es1);
                yd0 = ey0;
                yd1 = ey1;
            }
            if (lane == 31) {
                up0 = mix(ez0, es0);
                up1 = mix(ez1, es1);
            }
            if (!in) continue;
            sn[k] = C0;
            sn[k + 32] = C1;
            // per cell: left, lower, right, upper neighbour and their matrix entries
            const float cv[2][4] = {{C0.x, C0.y, C0.z, C0.w}, {C1.x, C1.y, C1.z, C1.w}};
            const float lv[2][4] = {{L.x, L.y, L.z, L.w}, {C0.x, C0.y, C0.z, C0.w}};
            const float rv[2][4] = {{C1.x, C1.y, C1.z, C1.w}, {Rr.x, Rr.y, Rr.z, Rr.w}};
            const float la[2][4] = {{xl.x, xl.y, xl.z, xl.w}, {x0.x, x0.y, x0.z, x0.w}};
            const float ra[2][4] = {{x0.x, x0.y, x0.z, x0.w}, {x1.x, x1.y, x1.z, x1.w}};
            const float ya[2][4] = {{y0.x, y0.y, y0.z, y0.w}, {y1.x, y1.y, y1.z, y1.w}};
            const float ad[2][4] = {{a0.x, a0.y, a0.z, a0.w}, {a1.x, a1.y, a1.z, a1.w}};
            const float dnv[2] = {dn0, dn1}, upv[2] = {up0, up1}, yd[2] = {yd0, yd1};
#pragma unroll
            for (int e = 0; e < 2; e++) {
                float t[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float sc = cv[e][j], lo = j > 0 ? cv[e][j - 1] : dnv[e], hi = j < 3 ? cv[e][j + 1] : upv[e];
                    const float alo = j > 0 ? ya[e][j - 1] : yd[e];
                    if constexpr (ROWSUM) {
                        t[j] = la[e][j] * (lv[e][j] - sc);
                        t[j] = fmaf(alo, lo - sc, t[j]);
                        t[j] = fmaf(ra[e][j], rv[e][j] - sc, t[j]);
                        t[j] = fmaf(ya[e][j], hi - sc, t[j]);
                        dacc = fma(to_f64(t[j]), to_f64(sc), dacc);
                    } else {
                        FF acc = ff_add(ff_prod(ad[e][j], sc), ff_prod(la[e][j], lv[e][j]));
                        acc = ff_add(acc, ff_prod(alo, lo));
                        acc = ff_add(acc, ff_prod(ra[e][j], rv[e][j]));
                        acc = ff_add(acc, ff_prod(ya[e][j], hi));
                        const double td = (double)acc.hi + (double)acc.lo;
                        A.as[4 * (k + 32 * e) + j] = td;
                        dacc = fma(td, to_f64(sc), dacc);
                    }
                }
                if constexpr (ROWSUM) ((float4 *)A.as)[k + 32 * e] = make_float4(t[0], t[1], t[2], t[3]);
            }
        }
        dacc = warp_sum(dacc);
        if (lane == 0) A.partials[pcg_chunks(sd) + c] = dacc;
    }
}

// Cells of a tile's column e that take part in the AXPYs and the maximum norm,
// as a bit mask: in the masked variants the red cells, otherwise the grid's.
template <bool MASKED>
__device__ __forceinline__ unsigned live4(const PcgArgs<float> &A, const SDIdx &sd, const Tiles &T, int d, int e) {
    if constexpr (MASKED) {
        const unsigned nb = ((const unsigned *)A.nb)[T.at(d) + 32 * e];
        return ((nb >> 5) & 1u) | ((nb >> 12) & 2u) | ((nb >> 19) & 4u) | ((nb >> 26) & 8u);
    } else {
        const int rows = sd.H - 4 * (T.s * 32 + T.lane);
        return 2 * (d - T.lane) + e < sd.W ? (rows >= 4 ? 15u : (1u << rows) - 1u) : 0u;
    }
}
static_assert(NB_RED == 32, "live4 picks bit 5 of each cell's byte");

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

// p += alpha s; r -= alpha z'; maxError = |r|_inf  (:363-366)
template <bool ROWSUM, bool MASKED>
__device__ __noinline__ void axpy32(const PcgArgs<float> &A, int iter, double alpha, int c_begin, int c_end, int c_step, int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int D = sd.D;
    const float4 *sp = (const float4 *)((iter & 1) ? A.sa : A.sb);  // the s this iteration's matvec wrote
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / D, d0 = c * kc - s * D;
        const Tiles T(sd, s, lane);
        unsigned long long mx = 0ull;  // bits of the largest |r| so far
        for (int u = 0; u < kc; u++) {
            const int d = d0 + u;
            if (!T.in(d)) continue;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const size_t k = T.at(d) + 32 * e;
                const unsigned live = live4<MASKED>(A, sd, T, d, e);
                double2 *pp = (double2 *)A.p + 2 * k, *rp = (double2 *)A.r + 2 * k;
                const float4 sv = sp[k];
                const double2 p0 = pp[0], p1 = pp[1], r0 = rp[0], r1 = rp[1];
                double p[4] = {p0.x, p0.y, p1.x, p1.y}, r[4] = {r0.x, r0.y, r1.x, r1.y}, a[4];
                if constexpr (ROWSUM) {
                    const float4 t = ((const float4 *)A.as)[k];
                    a[0] = to_f64(t.x);
                    a[1] = to_f64(t.y);
                    a[2] = to_f64(t.z);
                    a[3] = to_f64(t.w);
                } else {
                    const double2 a0 = ((const double2 *)A.as)[2 * k], a1 = ((const double2 *)A.as)[2 * k + 1];
                    a[0] = a0.x;
                    a[1] = a0.y;
                    a[2] = a1.x;
                    a[3] = a1.y;
                }
                const float sf[4] = {sv.x, sv.y, sv.z, sv.w};
                float rf[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double pn = fma(to_f64(sf[q]), alpha, p[q]), rn = fma(a[q], -alpha, r[q]);
                    if (live >> q & 1u) {
                        p[q] = pn;
                        r[q] = rn;
                        max_bits(mx, rn);
                    }
                    rf[q] = to_f32(r[q]);
                }
                pp[0] = make_double2(p[0], p[1]);
                pp[1] = make_double2(p[2], p[3]);
                rp[0] = make_double2(r[0], r[1]);
                rp[1] = make_double2(r[2], r[3]);
                ((float4 *)A.rf)[k] = make_float4(rf[0], rf[1], rf[2], rf[3]);
            }
        }
        mx = warp_max_bits(mx);
        if (lane == 0) A.partials[c] = __longlong_as_double((long long)mx);
    }
}

// p = 0; maxError = |r|_inf (3-conjugate-gradients/Fluid.cpp:350, 354); FP32 copy of r.
template <bool MASKED>
__device__ __noinline__ void start32(const PcgArgs<float> &A, int c_begin, int c_end, int c_step, int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / sd.D, d0 = c * kc - s * sd.D;
        const Tiles T(sd, s, lane);
        unsigned long long mx = 0ull;
        for (int u = 0; u < kc; u++) {
            const int d = d0 + u;
            if (!T.in(d)) continue;
            for (int e = 0; e < 2; e++) {
                const size_t k = T.at(d) + 32 * e;
                const unsigned live = live4<MASKED>(A, sd, T, d, e);
                const double2 r0 = ((const double2 *)A.r)[2 * k], r1 = ((const double2 *)A.r)[2 * k + 1];
                const double r[4] = {r0.x, r0.y, r1.x, r1.y};
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (live >> q & 1u) max_bits(mx, r[q]);
                ((double2 *)A.p)[2 * k] = make_double2(0.0, 0.0);
                ((double2 *)A.p)[2 * k + 1] = make_double2(0.0, 0.0);
                ((float4 *)A.rf)[k] = make_float4(to_f32(r[0]), to_f32(r[1]), to_f32(r[2]), to_f32(r[3]));
            }
        }
        mx = warp_max_bits(mx);
        if (lane == 0) A.partials[c] = __longlong_as_double((long long)mx);
    }
}

// One complete solve (factor and/or PCG, by A.mode) of one scene by team T.
// The halo words must hold the sentinel on entry; those that a sweep waits for
// hold it again on exit (every word that is waited for is taken).
// The elementwise passes work on chunks of pcg_chunk_diags(sd) tile diagonals,
// dealt out to the team's warps in turn.  Every reduction is summed per chunk
// (per strip for sigma), then over the partials in a fixed order, so the result
// depends on the scene alone, not on the number of blocks or warps that solve
// it: a scene gives bit-identical results in a single-scene launch, in any
// batch and with any launch shape.
// sigma = z.r is taken as y.(dd y), y the forward solve's result: z.r =
// (L^-T D L^-1 r).r = (L^-1 r).D(L^-1 r) exactly, and in floating point within
// the rounding of the two triangular solves.  Cells outside the masked MIC(0)
// work have dd = 0 and add nothing.
__device__ void pcg32_job(const PcgArgs<float> &A, Team &T, Ring32 &R, double *sm) {
    const int warps = blockDim.x >> 5;
    const SDIdx sd = A.sd;
    const int warp = threadIdx.x >> 5;
    const int kc = pcg_chunk_diags(sd);
    const int nchunk = (int)pcg_chunks(sd);
    const int nwarps = T.size * warps;
    // chunks c_begin, c_begin + nwarps, ...: every SM quarter gets as many, few or many
    const int c_begin = warp * T.size + T.rank, c_end = nchunk;
    R.buf = ring32_offset(A.K, sd.D) + (unsigned)(warp % A.K) * A.stages * kStageBytes;
    const bool masked = !A.all_red, pressure = A.rowsum_zero;
    const double *part = A.partials;

    if (A.mode & PCG_FACTOR) {
        const int nq = (sd.H + 31) / 32;
        for (int q = warp * T.size + T.rank; q < nq; q += nwarps) {
            const Chan in{A.halo + (size_t)(q > 0 ? q - 1 : 0) * sd.W, q > 0}, out{A.halo + (size_t)q * sd.W, q + 1 < nq};
            if (q > 0) factor32_rows<true>(A, q, in, out);
            else factor32_rows<false>(A, q, in, out);
        }
        team_barrier(T, A.fl);
    }
    if (!(A.mode & PCG_SOLVE)) return;

    if (masked) start32<true>(A, c_begin, c_end, nwarps, kc);
    else start32<false>(A, c_begin, c_end, nwarps, kc);
    team_barrier(T, A.fl);
    // z = M^-1 r  (:351)
    sweep32<false>(A, T, R);
    team_barrier(T, A.fl);
    sweep32<true>(A, T, R);
    team_barrier(T, A.fl);

    double maxError = total32(part, nchunk, true, sm);
    double sigma = total32(part + 2 * nchunk, sd.S, false, sm + 2 * kSums);
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
            if (pressure) matvec32<true>(A, iter, (float)beta, c_begin, c_end, nwarps, kc);
            else matvec32<false>(A, iter, (float)beta, c_begin, c_end, nwarps, kc);
            team_barrier(T, A.fl);
            const double alpha = sigma / total32(part + nchunk, nchunk, false, sm + kSums);
            if (!pressure) axpy32<false, true>(A, iter, alpha, c_begin, c_end, nwarps, kc);
            else if (masked) axpy32<true, true>(A, iter, alpha, c_begin, c_end, nwarps, kc);
            else axpy32<true, false>(A, iter, alpha, c_begin, c_end, nwarps, kc);
            team_barrier(T, A.fl);
            maxError = total32(part, nchunk, true, sm);
            iterations = iter + 1;
            if (A.pinned >= 0 ? iterations >= A.pinned : maxError < kTol) {
                status = 0;
                break;
            }
            // z = M^-1 r; sigmaNew = z.r  (:372-376)
            sweep32<false>(A, T, R);
            team_barrier(T, A.fl);
            sweep32<true>(A, T, R);
            team_barrier(T, A.fl);
            const double sigmaNew = total32(part + 2 * nchunk, sd.S, false, sm + 2 * kSums);
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

// Ring state of this warp (its role's position); the mbarriers are initialised
// once per launch.
__device__ void ring32_init(Ring32 &R, int K, int stages) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    R.buf = 0u;
    R.bars = 8u * Ring32::KINDS * kMaxStages * (warp % K);
    R.stages = stages;
    R.st = 0;
    R.parity = 0u;
    R.dead = false;
    if (lane == 0 && warp < K) {
        for (int k = 0; k < stages; k++) {
            mbar_init(R.bar(Ring32::COPIED, k), 1);
            mbar_init(R.bar(Ring32::READY, k), 2);
            mbar_init(R.bar(Ring32::FREE, k), 1);
        }
        fence_mbar_init();
    }
}

// 168 registers per thread.
constexpr int kMaxThreads32 = 384;

__global__ void __launch_bounds__(kMaxThreads32, 1) pcg32_kernel(PcgArgs<float> A) {
    __shared__ double sm[3 * kSums];
    Team T{(int)blockIdx.x, (int)gridDim.x, A.barrier, 0u};
    Ring32 R;
    ring32_init(R, A.K, A.stages);
    const size_t nh = 2 * (size_t)(A.K > 1 ? A.K - 1 : 0) * pcg_halo_row(A.sd);
    for (size_t k = threadIdx.x; k < nh; k += blockDim.x)
        ((unsigned long long *)(g_smem + halo32_offset(A.K)))[k] = kSentinel;
    __syncthreads();
    pcg32_job(A, T, R, sm);
}

// Many independent scenes in one cooperative launch (see BatchTeams).
__global__ void __launch_bounds__(kMaxThreads32, 1)
    pcg32_batch_kernel(const PcgArgs<float> *jobs, BatchTeams B, int mode, int heat, int pinned, int K, int stages) {
    __shared__ double sm[3 * kSums];
    __shared__ PcgArgs<float> sA;
    __shared__ int s_slot;
    const int2 bt = batch_slot(B, &s_slot);
    const int2 tm = B.team[bt.x];
    Team T{bt.y, tm.x, B.team_bar + kBarStride * bt.x, 0u};
    Ring32 R;
    ring32_init(R, K, stages);
    __syncthreads();
    while (batch_take<float>(B, T, bt.x, tm.y, jobs, sA, mode, heat, pinned, K, stages)) {
        // halo rows start at the sentinel: the shared rows of this block
        // (their length changes with the scene) and the scene's global rows
        const size_t nh = 2 * (size_t)(K > 1 ? K - 1 : 0) * pcg_halo_row(sA.sd);
        for (size_t k = threadIdx.x; k < nh; k += blockDim.x)
            ((unsigned long long *)(g_smem + halo32_offset(K)))[k] = kSentinel;
        const size_t ng = pcg_halo_words(sA.sd);
        for (size_t k = (size_t)T.rank * blockDim.x + threadIdx.x; k < ng; k += (size_t)T.size * blockDim.x)
            sA.halo[k] = kSentinel;
        team_barrier(T, sA.fl);
        pcg32_job(sA, T, R, sm);
    }
}

constexpr int kSingleThreads = 256, kSingleStages = 6;

}  // namespace

size_t pcg32_smem(int K, int D, int stages) { return ring32_offset(K, D) + (size_t)K * stages * kStageBytes; }

const void *pcg32_batch_fn() { return (const void *)pcg32_batch_kernel; }
// What a shape {threads, strips per block, stages} comes to: at least a strip's
// three warps per strip, as many strips and stages as threads and shared memory
// allow (smem: bytes of a block).
void pcg32_shape(int threads, int D, size_t smem_max, int *block, int *K, int *stages) {
    *K = std::min(*K, kMaxThreads32 / (32 * kRoles));
    while (*stages > 2 && pcg32_smem(*K, D, *stages) > smem_max) (*stages)--;
    while (*K > 1 && pcg32_smem(*K, D, *stages) > smem_max) (*K)--;
    *block = std::max(threads, 32 * kRoles * *K);
}

cudaError_t launch_pcg32(PcgArgs<float> A, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
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
    const size_t smem = pcg32_smem(A.K, sd.D, A.stages);
    const void *fn = (const void *)pcg32_kernel;
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
    void *args[] = {&A};
    return cudaLaunchCooperativeKernel(fn, dim3(G), dim3(kSingleThreads), args, smem, st);
}

}  // namespace ifl

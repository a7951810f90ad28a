// k_gs.cu - the Gauss-Seidel pressure solve of tutorial steps 1-2 (sm_103a).
//
// project() of 1-matrixless/Fluid.cpp:192-240 (the same in
// 2-better-advection): lexicographic Gauss-Seidel sweeps over the implicit
// five-point stencil with solid walls, p kept from the previous step, until
// the largest change of a sweep is below 1e-5 or 600 sweeps.
//
// What bounds it: a cell is a chain of FP64 operations, each 64 cycles of its
// warp on this part, and a sweep on its own is a recurrence along W + H
// diagonals.  But sweep k + 1 needs only the values that sweep k left two
// diagonals ahead of it, so many sweeps run at a time, each on a warp of its
// own, and 600 sweeps take about 600 x 4 diagonal steps instead of 600 x (W + 31).
// Every value, and so the sweep count, is that of the sequential loop.
//
// Worker (s, j) is one warp: strip s (32 rows), sweeps j, j + J, j + 2J, ...
// Lane l is on row 32s + l; step d visits the cell x = d - l of every lane (one
// contiguous strip-diagonal line).  The left value is the lane's own previous
// result, the lower one lane l - 1's by shuffle; the right one is the previous
// sweep's value of the own row, the upper one lane l + 1's right one.  Lane 0
// takes its lower value from strip s - 1's worker of the same sweep, lane 31 its
// upper one from strip s + 1's worker of the previous sweep.
//
// Hand-over: sweep k writes ring buffer (k + 1) mod B.  An entry is 16 bytes, the
// value and the value xor the sweep's tag.  A reader that finds its tag in the two
// words has the value, with no counter or fence behind it, even if the words of
// the entry before and of this one came mixed: with this sweep's check word the
// tag comes out only for this sweep's value, and an older check word can only
// give it by chance beside this sweep's value.  A worker loads the entries of a
// step one step ahead (a step is about the L2's latency) and loads again those
// that had not come.
//
// Convergence: the strips of a sweep pass its largest change on, the last strip
// decides (`verdict`: the first converged sweep so far), and sweep k starts once
// the verdict of sweep k - L is in and open.  So up to L - 1 sweeps run ahead of
// the decision; their buffers are dropped.  B = L + 1 buffers: sweep k + B starts
// after sweep k + 1 is complete (nobody reads sweep k any more) and found not
// converged (sweep k is not the result).  A worker that has no sweep left to ask
// before waits for an entry of its own (`decided`): the last sweeps, and with
// them their verdicts, do not exist if an earlier one converged.
//
// 600 sweeps at 128 x 128: 1.9 ms; 111 ms with one sweep and the head of the next in
// flight, a hand-over with a fence every four diagonals and a division per cell.
//
// Every wait is bounded; a timeout sets the status word and an abort word that
// releases every other wait.
#include <algorithm>

#include "ifl_device.cuh"

namespace ifl {

namespace {

constexpr double kGsTol = 1e-5;
constexpr int kBlockWarps = 4;  // workers per block at most: one for each quarter of an SM
constexpr unsigned FULL = 0xffffffffu;

// A value and its check word, the value's bits xor the sweep's tag (sweep + 2; the
// initial p counts as sweep -1; an empty entry has tag 0).
struct __align__(16) Entry {
    unsigned long long v, check;
};

struct GsArgs {
    const double *r;
    double *p;
    SDIdx sd;
    double scale;  // timestep / (density * hx * hx)
    int limit, pinned;
    long long spin_limit;  // polls of one wait before the solve gives up
    PcgOut *out;
    unsigned *flags;
    unsigned long long *iter_total;
    int J, L;              // sweeps in flight per strip; sweeps that may run ahead of a verdict
    Entry *ring;           // L + 1 buffers of p
    Entry *down, *up;      // -scale p of every strip's last and first row, by buffer, strip and column
    Entry *change;         // L + 1 x S: largest change of a sweep up to strip s
    Entry *verdict;        // L + 1: first converged sweep + 1, or 0 (as bits of v)
    Entry *decided;        // the same for the whole solve, written once
    unsigned long long *abort;
};

// ------------------------------------------------------------- hand-over
__device__ __forceinline__ Entry ld_entry(const Entry *e) {
    Entry r;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(r.v), "=l"(r.check) : "l"(e) : "memory");
    return r;
}
__device__ __forceinline__ void st_entry_if(Entry *e, double v, unsigned long long tag, bool p) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %3, 0;\n @q st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n}\n" ::"l"(e),
                 "l"(b), "l"(b ^ tag), "r"((unsigned)p)
                 : "memory");
}
__device__ __forceinline__ void st_entry(Entry *e, double v, unsigned long long tag) { st_entry_if(e, v, tag, true); }
__device__ __forceinline__ double value_of(const Entry &e) { return __longlong_as_double((long long)e.v); }
__device__ __forceinline__ unsigned long long tag_of(const Entry &e) { return e.v ^ e.check; }
__device__ __forceinline__ bool gs_aborted(const GsArgs &A) {
    return *(const volatile unsigned long long *)A.abort != 0ull;
}
__device__ __forceinline__ void gs_abort(const GsArgs &A) {
    atomicOr(A.flags, FLAG_TIMEOUT);
    *(volatile unsigned long long *)A.abort = 1ull;
}
// Whole warp: the entry with this tag, and what its writer did before (acquire).
__device__ __forceinline__ double gs_wait(const GsArgs &A, const Entry *e, unsigned long long tag) {
    Entry c = ld_entry(e);
    long long spins = 0;
    while (__any_sync(FULL, tag_of(c) != tag)) {
        if (++spins > A.spin_limit) gs_abort(A);
        if (gs_aborted(A)) break;
        c = ld_entry(e);
    }
    __threadfence();
    return __shfl_sync(FULL, value_of(c), 0);
}
// Whole warp, after its loads and stores: hands an entry on with them (release).
__device__ __forceinline__ void gs_publish(Entry *e, double v, unsigned long long tag) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        __threadfence();
        st_entry(e, v, tag);
    }
    __syncwarp();
}

// -------------------------------------------------------------- division
// x / d, rounded as the division instruction sequence rounds it, for a divisor
// known in advance (four FP64 operations; the division takes nine times one, 562
// cycles): q = x (zh + zl) with zh + zl = 1/d to twice the precision is within an
// ulp of the quotient (N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating
// correctly rounded floating-point division when the divisor is known in
// advance", IEEE Trans. Computers 53, 2004), so its remainder is exact and
// one step with zh = RN(1/d) rounds correctly (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
// 34, 1990).  Holds where nothing underflows or overflows: 2^-100 <= d <= 2^100
// and 2^-800 <= |x| < 2^800.  A zero divides to itself.
struct Divisor {
    double d, zh, zl;
    __device__ __forceinline__ void set(double v) {
        d = v;
        zh = 1.0 / v;
        zl = fma(-v, zh, 1.0) / v;
    }
};
__device__ __forceinline__ unsigned biased_exponent(double x) { return ((unsigned)__double2hiint(x) >> 20) & 0x7ffu; }
__device__ __forceinline__ bool is_zero(double x) { return (((unsigned)__double2hiint(x) << 1) | (unsigned)__double2loint(x)) == 0u; }

// Out of line: inline, the compiler divides first and selects after.
__device__ __noinline__ double divide(double x, double d) { return x / d; }

__global__ void __launch_bounds__(32 * kBlockWarps) gs_kernel(GsArgs A) {
    extern __shared__ unsigned char spread[];  // spreads the workers over the SMs; never touched
    (void)spread;
    const int lane = threadIdx.x & 31, worker = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int S = A.sd.S, s = worker % S, j = worker / S;
    if (j >= A.J) return;
    const int w = A.sd.W, h = A.sd.H, D = A.sd.D, B = A.L + 1;
    const int y = s * 32 + lane;
    const bool row = y < h;
    const int steps = w + 31;  // diagonals of one strip per sweep
    const double scale = A.scale;
    // diag of the reference: scale added once per existing neighbour, in order
    Divisor d2, d3, d4;
    d2.set(scale + scale);
    d3.set((scale + scale) + scale);
    d4.set(((scale + scale) + scale) + scale);
    const unsigned ed = biased_exponent(d2.d);
    const bool plain = ed < 1023u - 98u || ed > 1023u + 98u || !(scale > 0.0);  // divisors out of range: divide
    const size_t own = (size_t)s * D * 32 + lane, cells = A.sd.total();
    const bool below = s > 0, above = s + 1 < S;
    // lane 0 reads the last row of the strip below and hands its own up, lane 31 the
    // first row of the strip above and hands its own down
    const bool edge = (lane == 0 && below) || (lane == 31 && above);
    const int nsweeps = A.pinned >= 0 ? min(A.limit, A.pinned) : A.limit;
    // divisors of an inner column and of the first and last one, which in a grid of
    // one column are the same one
    const int around = 2 + (y > 0) + (y < h - 1), fewer = around - (w > 1 ? 1 : 2);
    const Divisor inner = around == 4 ? d4 : around == 3 ? d3 : d2, at_side = fewer == 4 ? d4 : fewer == 3 ? d3 : d2;
    const unsigned columns = row ? (unsigned)w : 0u;

    // the initial p is sweep -1, buffer 0
    for (int d = j; d < steps && nsweeps > 0; d += A.J) {
        const int x = d - lane;
        if (!row || x < 0 || x >= w) continue;
        const double v = A.p[own + (size_t)d * 32];
        st_entry(A.ring + own + (size_t)d * 32, v, 1ull);
        if (lane == 0 && below) st_entry(A.up + (size_t)s * w + x, fma(-scale, v, 0.0), 1ull);
    }

    int stop = 0;  // first converged sweep + 1
    bool dead = false;
    for (int k = j; k < nsweeps; k += A.J) {
        if (k >= A.L) {
            stop = (int)__double_as_longlong(gs_wait(A, A.verdict + (k - A.L) % B, (unsigned long long)(k - A.L) + 2));
            if (stop != 0) break;
        }
        dead = __any_sync(FULL, gs_aborted(A));
        if (dead) break;
        const unsigned long long tag = (unsigned long long)k + 2;  // this sweep's; the previous sweep's is tag - 1
        const int b_old = k % B, b_new = (k + 1) % B;
        // Operands of a step: the previous sweep's right value, the edge lane's neighbour
        // row and the right-hand side.  Lanes at a column outside the grid load what lies
        // there and ignore it.  Two sets in turn, pointers that move on by two steps.
        struct Operands {
            Entry right, side;
            double rr;
        } two[2] = {};
        const Entry *old_right = A.ring + (size_t)b_old * cells + own + 32;  // column of the step + 1
        // the row that lane 0 / lane 31 reads (column d / d - 31 at step d), and hands on
        const Entry *halo = lane == 0 && below  ? A.down + ((size_t)b_new * S + s - 1) * w
                            : lane == 31 && above ? A.up + ((size_t)b_old * S + s + 1) * w - 31
                                                  : A.ring + 1;
        Entry *hand = lane == 0 ? A.up + ((size_t)b_new * S + s) * w : A.down + ((size_t)b_new * S + s) * w - 31;
        Entry *result = A.ring + (size_t)b_new * cells + own;
        const double *rhs = A.r + own;
        const unsigned long long halo_tag = lane == 0 ? tag : tag - 1;
        unsigned long long mx = 0ull;  // bits of the largest change
        double ql = 0.0;               // -scale * (this lane's previous value)
        double pold = 0.0;             // the previous sweep's value of the cell
        int x = -lane;                 // column of an even step
        // operands of step u after the even step that the pointers are at
        auto load = [&](Operands &o, int u) {
            o.right = ld_entry(old_right + u * 32);
            o.side = ld_entry(halo + u);
            o.rr = *((unsigned)(x + u) < columns ? rhs + u * 32 : A.r + own + (size_t)lane * 32);
        };
        // the entries of that step, loaded again until they are there
        auto settle = [&](Operands &o, int u) {
            const bool need = (unsigned)(x + u + 1) < columns, needs = edge && (unsigned)(x + u) < columns;
            long long spins = 0;
            while (__any_sync(FULL, (need && tag_of(o.right) != tag - 1) || (needs && tag_of(o.side) != halo_tag))) {
                if (++spins > A.spin_limit) gs_abort(A);
                if ((spins & 15) == 0 || spins > A.spin_limit) {
                    if (__any_sync(FULL, gs_aborted(A))) return false;
                }
                if (need && tag_of(o.right) != tag - 1) o.right = ld_entry(old_right + u * 32);
                if (needs && tag_of(o.side) != halo_tag) o.side = ld_entry(halo + u);
            }
            return true;
        };
        auto step = [&](Operands &o, Operands &next, int u) {
            if (!settle(o, u)) return false;
            const int col = x + u;
            const bool act = (unsigned)col < columns;
            const double right = (unsigned)(col + 1) < columns ? value_of(o.right) : 0.0;
            const double side = act && edge ? value_of(o.side) : 0.0, rr = o.rr;
            load(next, u + 1);
            // 0 - scale * value, as the reference's first subtraction leaves it; 0 for a
            // neighbour that does not exist (subtracting scale * value and adding this
            // give the same bits: the running sum is never -0)
            const double qr = fma(-scale, right, 0.0);
            double qd = __shfl_up_sync(FULL, ql, 1);
            double qu = __shfl_down_sync(FULL, qr, 1);
            if (lane == 0) qd = side;
            if (lane == 31) qu = side;
            const double num = rr - (((ql + qd) + qr) + qu);
            const bool side_col = col == 0 || col == w - 1;
            const double dv = side_col ? at_side.d : inner.d, zh = side_col ? at_side.zh : inner.zh,
                         zl = side_col ? at_side.zl : inner.zl;
            const double q = fma(num, zh, num * zl);
            double np = fma(fma(-q, dv, num), zh, q);
            if (is_zero(num)) np = num;
            const bool range = biased_exponent(num) - (1023u - 800u) < 1600u || is_zero(num);
            if (__any_sync(FULL, act && (plain || !range))) np = divide(num, dv);
            const unsigned long long c = (unsigned long long)__double_as_longlong(pold - np) & 0x7fffffffffffffffull;
            const double qn = fma(-scale, np, 0.0);
            // maxDelta = std::max(maxDelta, |change|): a NaN is skipped
            if (act && c <= 0x7ff0000000000000ull && c > mx) mx = c;
            st_entry_if(result + u * 32, np, tag, act);
            st_entry_if(hand + u, qn, tag, act && edge);
            ql = act ? qn : 0.0;
            pold = right;
            return true;
        };
        two[1].right = ld_entry(old_right - 32);  // column 0, lane 0
        dead = !settle(two[1], -1);
        if (dead) break;
        pold = lane == 0 && row ? value_of(two[1].right) : 0.0;
        load(two[0], 0);
        for (int d = 0; d < steps && !dead; d += 2) {
            dead = !step(two[0], two[1], 0);
            if (!dead && d + 1 < steps) dead = !step(two[1], two[0], 1);
            old_right += 64;
            halo += 2;
            rhs += 64;
            result += 64;
            hand += 2;
            x += 2;
        }
        if (dead) break;
        // the sweep's largest change up to this strip; the last strip decides
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(FULL, mx, o);
            mx = other > mx ? other : mx;
        }
        const int b = k % B;
        if (below) {
            const unsigned long long m = (unsigned long long)__double_as_longlong(gs_wait(A, A.change + (size_t)b * S + s - 1, tag));
            mx = m > mx ? m : mx;
        }
        const double change = __longlong_as_double((long long)mx);
        gs_publish(A.change + (size_t)b * S + s, change, tag);
        if (!above) {
            int v = k > 0 ? (int)__double_as_longlong(gs_wait(A, A.verdict + (k - 1) % B, tag - 1)) : 0;
            const bool open = v == 0;
            if (open && A.pinned < 0 && change < kGsTol) v = k + 1;
            if (open && (v != 0 || k == nsweeps - 1)) gs_publish(A.decided, __longlong_as_double((long long)v), 1ull);
            gs_publish(A.verdict + b, __longlong_as_double((long long)v), tag);
        }
    }
    int final_sweeps = nsweeps;
    double maxDelta = 0.0;
    if (nsweeps > 0 && !dead) {
        if (stop == 0) stop = (int)__double_as_longlong(gs_wait(A, A.decided, 1ull));
        if (stop != 0) final_sweeps = stop;
        maxDelta = gs_wait(A, A.change + (size_t)((final_sweeps - 1) % B) * S + S - 1, (unsigned long long)final_sweeps + 1);
        dead = __any_sync(FULL, gs_aborted(A));
    }
    // the result is in buffer `final`; move it to p (this strip's own cells)
    for (int d = j; d < steps && final_sweeps > 0 && !dead; d += A.J) {
        const int x = d - lane;
        if (row && x >= 0 && x < w)
            A.p[own + (size_t)d * 32] = value_of(ld_entry(A.ring + (size_t)(final_sweeps % B) * cells + own + (size_t)d * 32));
    }
    if (s == 0 && j == 0 && lane == 0) {
        A.out->iterations = final_sweeps;
        A.out->status = stop != 0 && !dead ? 0 : 2;
        A.out->max_error = maxDelta;
        atomicAdd(A.iter_total, (unsigned long long)final_sweeps);
    }
}

size_t ring_words(const SDIdx &sd, int L) {
    // (64 entries more: loads beyond a row's or a strip's last column, which are ignored; `decided`, `abort`)
    return ((size_t)(L + 1) * (sd.total() + 2 * (size_t)sd.S * sd.W + sd.S + 1) + 64 + 1) * 2 + 2;
}

// Sweeps in flight (J) and the lead over the verdict (L).  A sweep follows the one
// before it by three to four steps (one of dependence, one of loading ahead, the
// hand-over): at 128 x 128, with 159 steps of about 1500 cycles, 600 sweeps took
// 4.4 million cycles with 40 sweeps in flight per strip, 3.9 with 56, 3.5 with 76
// and 3.2 with 120, so half as many as steps; and no more than four workers per SM:
// an FP64 instruction takes 64 cycles of a warp with one worker on an SM and 76
// with four.  The verdict of a sweep comes after the last strip's last step (36
// steps per strip: 32 rows and the hand-over).  The ring is kept below kRingBytes
// with fewer sweeps in flight, but not below the three buffers of 16-byte entries
// that one sweep and its successor need: 0.9 GB at 4096^2, 55 GB at 32768^2, where
// a handle has fewer arrays for it (solver.cu).
constexpr size_t kRingBytes = (size_t)512 << 20;
void gs_plan(const SDIdx &sd, int sms, int *J, int *L) {
    const long steps = sd.W + 31, until = steps + 36L * (sd.S - 1) + 8;
    *J = (int)std::max(1L, std::min(4L * sms / sd.S, (steps + 1) / 2));
    auto lead = [&](int n) { return (int)((n * until + steps - 1) / steps) + 2; };
    *L = lead(*J);
    while (*J > 1 && ring_words(sd, *L) * 8 > kRingBytes) *L = lead(--*J);
    while (*L > 2 && ring_words(sd, *L) * 8 > kRingBytes) --*L;
}

}  // namespace

size_t gs_words(const SDIdx &sd, int sms) {
    int J, L;
    gs_plan(sd, sms, &J, &L);
    return ring_words(sd, L);
}

template <typename F>
cudaError_t launch_gs(const Scene<F> &S, const PcgScratch &X, double dt, int limit, int pinned, cudaStream_t st,
                      long long wait_limit) {
    const SDIdx &sd = S.sd;
    int dev = 0, sms = 0, per_sm = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    GsArgs A;
    gs_plan(sd, sms, &A.J, &A.L);
    // blocks of as many workers as seat them all with one block per SM, up to one
    // for each of its quarters (single-warp blocks share a quarter: 1.6 times the
    // time per step with two workers on an SM)
    const int share = (sd.S * A.J + sms - 1) / sms;
    const int warps = std::min(share, kBlockWarps), smem = share > kBlockWarps ? 0 : std::min(optin, 120 * 1024);
    if (smem) {
        e = cudaFuncSetAttribute(gs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gs_kernel, 32 * warps, smem);
    if (e != cudaSuccess) return e;
    if ((long)per_sm * sms * warps < (long)sd.S * A.J) A.J = (int)((long)per_sm * sms * warps / sd.S);
    if (A.J < 1) return cudaErrorCooperativeLaunchTooLarge;
    A.r = S.r;
    A.p = S.p;
    A.sd = sd;
    A.scale = dt / (S.rho_air * S.hx * S.hx);
    A.limit = limit;
    A.pinned = pinned;
    A.spin_limit = wait_limit > 0 ? wait_limit : kSpinLimit;
    A.out = X.out;
    A.flags = S.flags;
    A.iter_total = X.iter_total;
    const size_t rows = (size_t)(A.L + 1) * sd.S * sd.W;
    A.ring = (Entry *)X.gs;
    A.down = A.ring + (size_t)(A.L + 1) * sd.total();
    A.up = A.down + rows;
    A.change = A.up + rows;
    A.verdict = A.change + (size_t)(A.L + 1) * sd.S;
    A.decided = A.verdict + A.L + 1 + 64;
    A.abort = (unsigned long long *)(A.decided + 1);
    // every tag back to `empty`: the whole of it, 47 MB at 128 x 128 (10 us)
    e = cudaMemsetAsync(X.gs, 0, ring_words(sd, A.L) * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    void *args[] = {&A};
    return cudaLaunchCooperativeKernel((const void *)gs_kernel, dim3((sd.S * A.J + warps - 1) / warps), dim3(32 * warps), args, (size_t)smem, st);
}

template cudaError_t launch_gs<double>(const Scene<double> &, const PcgScratch &, double, int, int, cudaStream_t,
                                       long long);
template cudaError_t launch_gs<float>(const Scene<float> &, const PcgScratch &, double, int, int, cudaStream_t,
                                      long long);

}  // namespace ifl

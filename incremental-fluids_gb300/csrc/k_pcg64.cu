// k_pcg64.cu - the FP64 form's MIC(0)-preconditioned conjugate gradients as one
// persistent cooperative kernel per solve, or per batch of solves (sm_103a).
// References: see k_pcg32.cu; the same solve with FP64 operands throughout.
//
// What bounds it: GB300 issues an FP64 instruction of a warp once in 64 cycles,
// whatever its lanes do and however independent it is (19 cycles per warp with
// all four quarters of an SM at work).  So everything here counts FP64
// instructions per warp:
//  * a wavefront step of a strip (32 rows, a lane per row) is two fused
//    multiply-adds in the L D L^T form of the MIC(0) apply (k_pcg32.cu), where
//    the reference's order takes five multiplications and subtractions; shuffles,
//    loads and stores run in their shadow;
//  * the preparer warp forms dd y and sigma on another SM quarter;
//  * the matvec forms each neighbour's new s with one multiply-add and its dot
//    product with another: 10 instructions per 32 cells where there were 21;
//  * the elementwise passes deal diagonals out to every SM quarter of the GPU.
// That form serves the plain step (3) and ifl_pcg_solve_noalloc: its pressure is
// 1e-15 off the reference's.  The solves of scenes with bodies (steps 4-8) keep
// the reference's own arithmetic and the order of sums that this form has always
// had (REF): for some placements of the bodies their conjugate gradients amplify
// a last-bit difference, even of the order of a sum, by up to 1e8 (24 seeded
// scenes of steps 5-7: velocities up to 1e-8 off; a 48 x 66 scene of step 7 in
// one step 2e-8 off the oracle's).  Bit for bit the reference's are the factor and
// each application of the preconditioner; the order of the sums, and with it the last
// bits of alpha and beta, is this form's own.
#include "pcg_ring.cuh"

namespace ifl {

namespace {

constexpr int kT = Lay<double>::kSteps;  // diagonals per block of a ring
constexpr unsigned kVec = kVecBytes<double>;

// c + a*b, rounded once, or twice as the reference does (REF).
template <bool REF>
__device__ __forceinline__ double madd(double a, double b, double c) {
    return REF ? c + a * b : fma(a, b, c);
}

// The preparer's part of one backward strip: y becomes dd y, and sigma = z.r =
// sum of dd y^2 (see pcg_job) is added up.
__device__ __noinline__ void prepare_strip(const PcgArgs<double> &A, int s, Ring<double> &ring, bool in) {
    Ring<double> R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31, nblk = A.sd.D / kT;
    double qq = 0.0;
    for (int blk = 0; blk < nblk; blk++) {
        ring_wait(R, R.bar(Ring<double>::COPIED, R.st), R.parity, flags);
        char *g = g_smem + R.stage(R.st) + lane * 8;
#pragma unroll
        for (int j = kT - 1; j >= 0; j--) {
            double *y = (double *)(g + j * 256);
            const double y0 = *y, q = *(const double *)(g + kVec + j * 768) * y0;
            *y = q;
            qq = fma(q, y0, qq);
        }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(R.bar(Ring<double>::PREPARED, R.st));
            if (!in) mbar_arrive(R.bar(Ring<double>::READY, R.st));  // else the taker's, with the halo words
        }
        R.next();
    }
    qq = warp_sum(qq);
    if (lane == 0) A.partials[2 * pcg_chunks(A.sd) + s] = qq;
    ring = R;
    __syncwarp();
}

// One strip of a sweep.  At step t lane l works on diagonal t (backward: D-1-t),
// one column behind lane l-1 (l+1), whose value arrives by shuffle; lane 0 (31)
// takes it from the block's halo words (IN: whether the strip has a neighbour to
// take from), and lane 31 (0) hands this strip's on through `out`: the word of
// column x at x + 32 of the row (forward; the lane starts at x = -31) or at x
// (backward).  Words of columns that no step waits for are written along and
// never read.  The multiply-add with the lane's own previous value comes first:
// the shuffle arrives while it runs.
// REF: q = ((r - lx_l q_l) - ly_d q_d) pc and z = ((q - lx z_r) - ly z_u) pc, each
// operation rounded, as the reference forms them.
template <bool REF, bool BWD, bool IN>
__device__ __noinline__ void sweep_strip(const PcgArgs<double> &A, int s, Ring<double> &ring, const Chan out) {
    // the vector operand (r, dd y or q) and the coefficient arrays behind it (backward L D L^T: a and b, after dd)
    constexpr int kC = kCoefs<REF, BWD>, kSkip = BWD && !REF ? 1 : 0, kO = REF ? 4 : 3;
    Ring<double> R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int nblk = sd.D / kT;
    const bool edge = lane == (BWD ? 31 : 0), hands = out.valid && lane == (BWD ? 0 : 31);
    double *zp = A.z + ((size_t)s * sd.D + (BWD ? sd.D - kT : 0)) * 32 + lane;
    unsigned long long *op = out.row + (BWD ? sd.D - 1 : 1);  // word of this lane's first step
    double n = 0.0, h = 0.0;  // this lane's previous value, the previous lane's
    bool next_ready = false;
    for (int blk = 0; blk < nblk; blk++) {
        ring_wait_lane(R, R.bar(Ring<double>::READY, R.st), R.parity, next_ready, flags);
        const char *g = g_smem + R.stage(R.st);
        double o[kT][kO], halo[kT];
#pragma unroll
        for (int j = 0; j < kT; j++) {
            const int jj = BWD ? kT - 1 - j : j;
            const char *c = g + kVec + (jj * kC + kSkip) * 256;
            const double2 pair = *(const double2 *)(c + lane * 16);
            o[j][0] = *(const double *)(g + jj * 256 + lane * 8);
            o[j][1] = pair.x;
            o[j][2] = pair.y;
            if constexpr (REF) o[j][3] = *(const double *)(c + 512 + lane * 8);
            if (IN && (j & 1) == 0) {
                const double2 word = *(const double2 *)(g + kHaloAt<double> + 8 * j);
                halo[j] = word.x;
                halo[j + 1] = word.y;
            }
        }
#pragma unroll
        for (int j = 0; j < kT; j++) {
            if (j == kT - 2) {
                Ring<double> N = R;
                N.next();
                next_ready = mbar_test(N.bar(Ring<double>::READY, N.st), N.parity);
            }
            const double t = REF ? o[j][0] - o[j][1] * n : fma(o[j][1], n, o[j][0]);
            if constexpr (IN) h = edge ? halo[j] : h;
            if constexpr (REF) n = (t - o[j][2] * h) * o[j][3];
            else n = fma(o[j][2], h, t);
            h = BWD ? __shfl_down_sync(FULL, n, 1) : __shfl_up_sync(FULL, n, 1);
            hstore_if(Chan{op, true}, BWD ? -j : j, henc(n), hands);
            zp[(BWD ? kT - 1 - j : j) * 32] = n;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(R.bar(Ring<double>::FREE, R.st));
        R.next();
        zp += BWD ? -kT * 32 : kT * 32;
        op += BWD ? -kT : kT;
    }
    ring = R;
    __syncwarp();
}

// What a lane needs to find its cells: (strip, lane) and the grid.
struct Cells {
    int lane, W;
    bool rowok;
    size_t base;  // slot on diagonal 0
    __device__ __forceinline__ Cells(const SDIdx &sd, int strip, int l)
        : lane(l), W(sd.W), rowok(strip * 32 + l < sd.H), base((size_t)strip * sd.D * 32 + l) {}
    __device__ __forceinline__ bool in(int d) const { return rowok && d >= lane && d < lane + W; }
    __device__ __forceinline__ size_t at(int d) const { return base + (size_t)d * 32; }
};

// s = z + beta*s (first iteration: s = z) and z' = A s on diagonal d
// (3-conjugate-gradients/Fluid.cpp:361-362, 375, 315-332); returns this lane's z'
// and in *sv its s.  A lane forms the new s of its cell and of the cells left and
// right of it; the lower neighbour is lane-1's left cell and the upper one
// lane+1's right cell, which arrive by shuffle; lanes 0 and 31 take theirs from
// the adjacent strips.  A neighbour that does not exist has a zero coefficient.
template <bool REF>
__device__ __forceinline__ double matvec_row(const PcgArgs<double> &A, const Cells &T, int s, int d, int iter, double beta,
                                             double *sv) {
    const int lane = T.lane, D = A.sd.D;
    const double *so = (iter & 1) ? A.sb : A.sa;
    double *sn = (iter & 1) ? A.sa : A.sb;
    const bool first = iter == 0, in = T.in(d), inL = T.in(d - 1), inR = T.in(d + 1);
    const size_t k = T.at(d);
    double zc = 0.0, zl = 0.0, zr = 0.0, ze = 0.0, sc = 0.0, sl = 0.0, sr = 0.0, se = 0.0;
    double ad = 0.0, ax = 0.0, ay = 0.0, axl = 0.0, ayl = 0.0, aye = 0.0;
    if (in) {
        zc = A.z[k];
        ad = A.adiag[k];
        ax = A.ax[k];
        ay = A.ay[k];
    }
    if (inL) {
        zl = A.z[k - 32];
        axl = A.ax[k - 32];
        ayl = A.ay[k - 32];
    }
    if (inR) zr = A.z[k + 32];
    // lane 0 of strip s continues below in lane 31 of strip s-1, diagonal d+31;
    // lane 31 above in lane 0 of strip s+1, diagonal d-31
    const bool dn = lane == 0 && s > 0 && in, up = lane == 31 && in && (s + 1) * 32 < A.sd.H;
    const size_t ke = dn ? ((size_t)(s - 1) * D + d + 31) * 32 + 31 : ((size_t)(s + 1) * D + d - 31) * 32;
    if (dn || up) ze = A.z[ke];
    if (dn) aye = A.ay[ke];
    if (!first) {
        if (in) sc = so[k];
        if (inL) sl = so[k - 32];
        if (inR) sr = so[k + 32];
        if (dn || up) se = so[ke];
    }
    auto mix = [&](double z, double v) { return first ? z : madd<REF>(v, beta, z); };
    const double C = mix(zc, sc), L = mix(zl, sl), Rr = mix(zr, sr), E = mix(ze, se);
    double lo = __shfl_up_sync(FULL, L, 1), alo = __shfl_up_sync(FULL, ayl, 1);
    double hi = __shfl_down_sync(FULL, Rr, 1);
    if (lane == 0) {
        lo = E;
        alo = aye;
    }
    if (lane == 31) hi = E;
    // cell, left, lower, right, upper
    double t = ad * C;
    t = madd<REF>(axl, L, t);
    t = madd<REF>(alo, lo, t);
    t = madd<REF>(ax, Rr, t);
    t = madd<REF>(ay, hi, t);
    if (in) {
        sn[k] = C;
        A.as[k] = t;
    }
    *sv = in ? C : 0.0;
    return in ? t : 0.0;
}

// The matvec and z'.s over this warp's chunks.
template <bool ROWSUM>  // the FP32 form's: always false here
__device__ __noinline__ void matvec(const PcgArgs<double> &A, int iter, double beta, int c_begin, int c_end, int c_step,
                                    int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / sd.D, d0 = c * kc - s * sd.D;  // a chunk lies inside one strip
        const Cells T(sd, s, lane);
        double dacc = 0.0;
        for (int u = 0; u < kc; u++) {
            double v;
            const double t = matvec_row<false>(A, T, s, d0 + u, iter, beta, &v);
            dacc = fma(t, v, dacc);
        }
        dacc = warp_sum(dacc);
        if (lane == 0) A.partials[pcg_chunks(sd) + c] = dacc;
    }
}

// ---- the reference's arithmetic, with sums over chunks of kRefChunk diagonals

// Dot product of two operands by the chunk.  Where every warp of the team has one, a
// warp takes its chunks start to end.  Otherwise the warps of a block form a chunk's
// products, a diagonal each in turn, and leave them in shared memory, and one warp
// adds them in order: a quarter of the time for a team with warps to spare (203x150
// alone: 11.6K instead of 20.0K cycles for the matvec), but the others wait for the
// sum.
template <typename Product>
__device__ __forceinline__ void ref_dot(const PcgArgs<double> &A, const Team &T, double *partials, Product product) {
    __shared__ double prod[kRefChunk][32];
    const SDIdx sd = A.sd;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, n = ref_chunks(sd);
    if (n >= T.size * warps) {
        for (int c = warp * T.size + T.rank; c < n; c += T.size * warps) {
            const int s = c * kRefChunk / sd.D, d0 = c * kRefChunk - s * sd.D;
            const Cells C(sd, s, lane);
            double acc = 0.0;
            for (int u = 0; u < kRefChunk; u++) acc = acc + product(C, s, d0 + u);
            acc = warp_sum(acc);
            if (lane == 0) partials[c] = acc;
        }
        return;
    }
    for (int c = T.rank; c < n; c += T.size) {
        const int s = c * kRefChunk / sd.D, d0 = c * kRefChunk - s * sd.D;  // a chunk lies inside one strip
        const Cells C(sd, s, lane);
        for (int u = warp; u < kRefChunk; u += warps) prod[u][lane] = product(C, s, d0 + u);
        __syncthreads();
        if (warp == 0) {
            double acc = 0.0;
#pragma unroll
            for (int u = 0; u < kRefChunk; u++) acc = acc + prod[u][lane];
            acc = warp_sum(acc);
            if (lane == 0) partials[c] = acc;
        }
        __syncthreads();
    }
}
__device__ __noinline__ void ref_matvec(const PcgArgs<double> &A, const Team &T, int iter, double beta) {
    ref_dot(A, T, A.partials + pcg_chunks(A.sd), [&](const Cells &C, int s, int d) {
        double v;
        const double t = matvec_row<true>(A, C, s, d, iter, beta, &v);
        return t * v;
    });
}
// sigma = z.r over the red cells (3-conjugate-gradients/Fluid.cpp:356, 376); z is
// zero outside the masked MIC(0) work.
__device__ __noinline__ void ref_dot_zr(const PcgArgs<double> &A, const Team &T) {
    ref_dot(A, T, A.partials + 2 * pcg_chunks(A.sd),
            [&](const Cells &C, int, int d) { return C.in(d) ? A.z[C.at(d)] * A.r[C.at(d)] : 0.0; });
}

// p += alpha s; r -= alpha z'; maxError = |r|_inf  (:363-366).  MASKED: only the
// red cells take part.
template <bool REF, bool ROWSUM, bool MASKED>
__device__ __noinline__ void axpy(const PcgArgs<double> &A, int iter, double alpha, int c_begin, int c_end, int c_step,
                                  int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const double *sp = (iter & 1) ? A.sa : A.sb;  // the s this iteration's matvec wrote
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / sd.D, d0 = c * kc - s * sd.D;
        const Cells T(sd, s, lane);
        unsigned long long mx = 0ull;  // bits of the largest |r| so far
        for (int u = 0; u < kc; u++) {
            const size_t k = T.at(d0 + u);
            if (T.in(d0 + u) && (!MASKED || (A.nb[k] & NB_RED))) {
                A.p[k] = madd<REF>(sp[k], alpha, A.p[k]);
                const double rn = madd<REF>(A.as[k], -alpha, A.r[k]);
                A.r[k] = rn;
                max_bits(mx, rn);
            }
        }
        mx = warp_max_bits(mx);
        if (lane == 0) A.partials[c] = __longlong_as_double((long long)mx);
    }
}

// p = 0; maxError = |r|_inf (3-conjugate-gradients/Fluid.cpp:350, 354).
template <bool MASKED>
__device__ __noinline__ void start(const PcgArgs<double> &A, int c_begin, int c_end, int c_step, int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / sd.D, d0 = c * kc - s * sd.D;
        const Cells T(sd, s, lane);
        unsigned long long mx = 0ull;
        for (int u = 0; u < kc; u++) {
            const size_t k = T.at(d0 + u);
            if (!T.in(d0 + u)) continue;
            A.p[k] = 0.0;
            if (!MASKED || (A.nb[k] & NB_RED)) max_bits(mx, A.r[k]);
        }
        mx = warp_max_bits(mx);
        if (lane == 0) A.partials[c] = __longlong_as_double((long long)mx);
    }
}

}  // namespace

}  // namespace ifl

#include "pcg_job.cuh"

namespace ifl {

size_t pcg64_smem(int K, int D, int stages) { return pcg_smem<double>(K, D, stages); }
const void *pcg64_batch_fn() { return (const void *)pcg_batch_kernel<double>; }
void pcg64_shape(int threads, int D, size_t smem_max, int *block, int *K, int *stages) {
    pcg_shape<double>(threads, D, smem_max, block, K, stages);
}
cudaError_t launch_pcg64(PcgArgs<double> A, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
                         int *blocks_used) {
    return launch_single<double>(A, X, cfg, st, blocks_used);
}

}  // namespace ifl

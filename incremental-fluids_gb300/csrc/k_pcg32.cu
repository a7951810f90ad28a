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
// grid (the padding is computed along), and three more warps per strip take from
// the sweeping warp what is not on the chain: a loader fills a ring in shared
// memory, a taker folds the neighbouring strip's boundary row into the operands,
// and in the backward sweep a preparer forms dd y and sigma.  What is left per step is 6 loads of 16
// bytes from shared memory, 16 fused multiply-adds, two shuffles and three
// stores: 150 cycles, of which the multiply-adds are 63, the loads 45, the
// stores 30 (timed in a scratch copy with each left out).
//
// r and p are FP64; the matvec is FP32 (its results are stored as they are
// formed), dot products, the maximum norm, alpha and beta are FP64.
#include "pcg_ring.cuh"

namespace ifl {

namespace {

constexpr int kT = Lay<float>::kSteps;            // tile diagonals per block of a ring
constexpr unsigned kVec = kVecBytes<float>;
constexpr int kDepth = 2;                         // steps whose operands are in registers (divides kT)

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
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// a*b + c, element by element.
__device__ __forceinline__ float4 fma4(const float4 &a, const float4 &b, const float4 &c) {
    return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w));
}
__device__ __forceinline__ float4 mul4(const float4 &a, const float4 &b) {
    return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w);
}

// The preparer's part of one backward strip: y becomes dd y, and sigma = z.r =
// sum of dd y^2 (see pcg_job) is added up: sums of two fused FP32 products per
// row of the tiles and step, over a block, then FP64.
__device__ __noinline__ void prepare_strip(const PcgArgs<float> &A, int s, Ring<float> &ring, bool in) {
    Ring<float> R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31, nblk = A.sd.D / kT;
    double qq = 0.0;
    for (int blk = 0; blk < nblk; blk++) {
        ring_wait(R, R.bar(Ring<float>::COPIED, R.st), R.parity, flags);
        char *g = g_smem + R.stage(R.st) + lane * 16;
        float4 qs = zero4();
#pragma unroll
        for (int j = kT - 1; j >= 0; j--) {
            float4 *y = (float4 *)(g + j * 1024);
            const float4 *dd = (const float4 *)(g + kVec + j * 3 * 1024);
            const float4 y0 = y[0], y1 = y[32], q0 = mul4(dd[0], y0), q1 = mul4(dd[32], y1);
            y[0] = q0;
            y[32] = q1;
            qs = fma4(q1, y1, fma4(q0, y0, qs));
        }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(R.bar(Ring<float>::PREPARED, R.st));
            if (!in) mbar_arrive(R.bar(Ring<float>::READY, R.st));  // else the taker's, with the halo words
        }
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
// shuffles; lane 0 (31) has its neighbour strip's folded into its operands
// (put_halo), and lane 31 (0) hands this strip's on through `out` as soon as it is
// formed: a word of two floats per tile column X,
// at X + 32 of the row (forward; the lane starts at X = -31) or at X (backward).
// Words of columns that no step waits for are written along and never read.
// Functions of their own: inlined, the solve's registers spill into their steps.
template <bool REF, bool BWD, bool IN>
__device__ __noinline__ void sweep_strip(const PcgArgs<float> &A, int s, Ring<float> &ring, const Chan out) {
    // the vector operand (r, or dd y) and two coefficient arrays behind it (backward: a and b, after dd)
    constexpr int kC = BWD ? 3 : 2, kSkip = BWD ? 1 : 0;
    Ring<float> R = ring;
    const Flags flags = A.fl;
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int nblk = sd.D / kT;
    const bool hands = out.valid && lane == (BWD ? 0 : 31);
    float4 *zp = (float4 *)A.z + ((size_t)s * sd.D + (BWD ? sd.D - kT : 0)) * 64 + lane;
    unsigned long long *op = out.row + (BWD ? sd.D - 1 : 1);  // word of this lane's first step
    float4 o0[kDepth][3], o1[kDepth][3];  // operands of kDepth steps, columns 0 and 1
    char *g = nullptr;  // this lane's column of the current block
    // operands of step j of the block into buffer j % kDepth
    auto load = [&](int j) {
        const int i = j % kDepth, jj = BWD ? kT - 1 - j : j;
        const char *v = g + jj * 1024, *c = g + kVec + (jj * kC + kSkip) * 1024;
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
    bool next_ready = false;
    for (int blk = 0; blk < nblk; blk++) {
        ring_wait_lane(R, R.bar(Ring<float>::READY, R.st), R.parity, next_ready, flags);
        g = g_smem + R.stage(R.st) + lane * 16;
#pragma unroll
        for (int j = 0; j < kDepth; j++) load(j);
#pragma unroll
        for (int j = 0; j < kT; j++) {
            // asked for two steps ahead: waiting for a barrier that is complete takes 90 cycles too
            if (j == kT - 2) {
                Ring<float> N = R;
                N.next();
                next_ready = mbar_test(N.bar(Ring<float>::READY, N.st), N.parity);
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
        if (lane == 0) mbar_arrive(R.bar(Ring<float>::FREE, R.st));
        R.next();
        zp += BWD ? -kT * 64 : kT * 64;
        op += BWD ? -kT : kT;
    }
    ring = R;
    __syncwarp();
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

// The operands of this warp's next chunk on their way from HBM to L2: the scenes of
// a batch do not fit there together, and a warp has no more loads in flight than
// its registers hold.
template <typename T>
__device__ __forceinline__ void prefetch_chunk(const T *p, int c, int c_end, int kc) {
    if (c < c_end && (threadIdx.x & 31) == 0) prefetch_l2(p + (size_t)c * kc * 256, kc * 256 * sizeof(T));
}

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
__device__ __noinline__ void matvec(const PcgArgs<float> &A, int iter, float beta, int c_begin, int c_end, int c_step, int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int D = sd.D;
    const float *so = (iter & 1) ? A.sb : A.sa;
    float4 *sn = (float4 *)((iter & 1) ? A.sa : A.sb);
    const bool first = iter == 0;
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / D, d0 = c * kc - s * D;  // a chunk lies inside one strip
        const Tiles T(sd, s, lane);
        prefetch_chunk(A.z, c + c_step, c_end, kc);
        prefetch_chunk(so, c + c_step, c_end, kc);
        prefetch_chunk(A.ax, c + c_step, c_end, kc);
        prefetch_chunk(A.ay, c + c_step, c_end, kc);
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

// p += alpha s; r -= alpha z'; maxError = |r|_inf  (:363-366)
template <bool REF, bool ROWSUM, bool MASKED>
__device__ __noinline__ void axpy(const PcgArgs<float> &A, int iter, double alpha, int c_begin, int c_end, int c_step, int kc) {
    const int lane = threadIdx.x & 31;
    const SDIdx sd = A.sd;
    const int D = sd.D;
    const float4 *sp = (const float4 *)((iter & 1) ? A.sa : A.sb);  // the s this iteration's matvec wrote
    for (int c = c_begin; c < c_end; c += c_step) {
        const int s = (c * kc) / D, d0 = c * kc - s * D;
        const Tiles T(sd, s, lane);
        prefetch_chunk((const float *)sp, c + c_step, c_end, kc);
        if (ROWSUM) prefetch_chunk((const float *)A.as, c + c_step, c_end, kc);
        else prefetch_chunk(A.as, c + c_step, c_end, kc);
        prefetch_chunk(A.p, c + c_step, c_end, kc);
        prefetch_chunk(A.r, c + c_step, c_end, kc);
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
__device__ __noinline__ void start(const PcgArgs<float> &A, int c_begin, int c_end, int c_step, int kc) {
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

}  // namespace

}  // namespace ifl

#include "pcg_job.cuh"

namespace ifl {

size_t pcg32_smem(int K, int D, int stages) { return pcg_smem<float>(K, D, stages); }
const void *pcg32_batch_fn() { return (const void *)pcg_batch_kernel<float>; }
void pcg32_shape(int threads, int D, size_t smem_max, int *block, int *K, int *stages) {
    pcg_shape<float>(threads, D, smem_max, block, K, stages);
}
cudaError_t launch_pcg32(PcgArgs<float> A, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
                         int *blocks_used) {
    return launch_single<float>(A, X, cfg, st, blocks_used);
}

}  // namespace ifl

// k_pcg.cu - host side of the PCG solves: job records, single launches, and the
// plan of a batched launch (teams, queues and their tables).  The kernels are in
// k_pcg32.cu and k_pcg64.cu, which say what they compute and what bounds them.
#include <algorithm>
#include <functional>
#include <cstring>
#include <type_traits>
#include <vector>

#include "pcg_common.cuh"

namespace ifl {

// k_pcg32.cu, k_pcg64.cu
size_t pcg32_smem(int K, int D, int stages);
size_t pcg64_smem(int K, int D, int stages);
const void *pcg32_batch_fn();
const void *pcg64_batch_fn();
void pcg32_shape(int threads, int D, size_t smem_max, int *block, int *K, int *stages);
void pcg64_shape(int threads, int D, size_t smem_max, int *block, int *K, int *stages);
cudaError_t launch_pcg32(PcgArgs<float> A, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
                         int *blocks_used);
cudaError_t launch_pcg64(PcgArgs<double> A, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
                         int *blocks_used);

template <typename F>
int pcg_max_blocks() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return 2 * sms;
}

namespace {
template <typename F>
PcgArgs<F> make_args(const Scene<F> &S, const PcgScratch &X, int heat) {
    PcgArgs<F> A;
    std::memset(&A, 0, sizeof A);
    A.sd = S.sd;
    A.adiag = S.adiag;
    A.ax = S.ax;
    A.ay = S.ay;
    A.pc = S.pc;
    A.mic = S.mic;
    A.nb = S.nb;
    A.r = S.r;
    A.p = S.p;
    A.as = S.as;
    A.rf = S.rf;
    A.z = S.z;
    A.sa = S.sa;
    A.sb = S.sb;
    A.partials = X.partials;
    A.barrier = X.barrier;
    A.halo = X.halo;
    A.fl = Flags{S.flags, S.flags};
    A.out = X.out + (heat ? 1 : 0);
    A.iter_total = X.iter_total;
    A.rowsum_zero = heat ? 0 : 1;
    A.all_red = (!heat && S.variant < 6) ? 1 : 0;
    A.ref = S.variant >= 4 ? 1 : 0;
    return A;
}
}  // namespace

namespace {
// FP32-form work arrays of an FP64 scene, and the conversion of its matrix.
PcgArgs<float> make_args_f32(const Scene<double> &S, const PcgF32 &M, const PcgScratch &X, int heat) {
    PcgArgs<float> A;
    std::memset(&A, 0, sizeof A);
    A.sd = S.sd;
    A.adiag = M.adiag;
    A.ax = M.ax;
    A.ay = M.ay;
    A.pc = S.pc;
    A.mic = M.mic;
    A.nb = S.nb;
    A.r = S.r;
    A.p = S.p;
    A.as = S.as;
    A.rf = M.rf;
    A.z = M.z;
    A.sa = M.sa;
    A.sb = M.sb;
    A.partials = X.partials;
    A.barrier = X.barrier;
    A.halo = X.halo;
    A.fl = Flags{S.flags, S.flags};
    A.out = X.out + (heat ? 1 : 0);
    A.iter_total = X.iter_total;
    A.rowsum_zero = heat ? 0 : 1;
    A.all_red = (!heat && S.variant < 6) ? 1 : 0;
    A.ref = S.variant >= 4 ? 1 : 0;
    return A;
}
__global__ void matrix_to_f32_kernel(const double *a, const double *b, const double *c, float *fa, float *fb,
                                     float *fc, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        fa[i] = (float)a[i];
        fb[i] = (float)b[i];
        fc[i] = (float)c[i];
    }
}
}  // namespace

template <>
cudaError_t launch_pcg<double>(const Scene<double> &S, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
                               int *blocks_used) {
    return launch_pcg64(make_args(S, X, cfg.heat), X, cfg, st, blocks_used);
}
template <>
cudaError_t launch_pcg<float>(const Scene<float> &S, const PcgScratch &X, const PcgConfig &cfg, cudaStream_t st,
                              int *blocks_used) {
    return launch_pcg32(make_args(S, X, cfg.heat), X, cfg, st, blocks_used);
}

cudaError_t launch_pcg_f32(const Scene<double> &S, const PcgF32 &M, const PcgScratch &X, const PcgConfig &cfg,
                           cudaStream_t st, int *blocks_used) {
    if (cfg.mode & PCG_FACTOR) {  // the FP32 form stores the matrix in FP32 (rounded once)
        const size_t n = S.sd.total();
        matrix_to_f32_kernel<<<(int)std::min<size_t>((n + 255) / 256, 152 * 8), 256, 0, st>>>(
            S.adiag, S.ax, S.ay, M.adiag, M.ax, M.ay, n);
    }
    return launch_pcg32(make_args_f32(S, M, X, cfg.heat), X, cfg, st, blocks_used);
}

// ------------------------------------------------------- batched solves, host
struct PcgBatchPlan {
    int precision = 0;  // sizeof(F)
    int n = 0;
    PcgShape shape{};
    int grid = 0;      // co-resident blocks of the launch
    int block = 0, K = 0, stages = 0;  // threads, strips and ring stages of a block
    int max_team = 128;  // largest team the planner may form
    size_t smem = 0;
    std::vector<int> strips, diags, cells;
    // device: [jobs pressure][jobs heat][block_team][team][class_range][class_jobs][team_job]
    //         [zeroed at launch: class_next | team_bar | all]
    char *dev = nullptr;
    size_t dev_bytes = 0;
    void *jobs[2] = {nullptr, nullptr};
    int4 *ctl = nullptr;
    BatchTeams B{};
    size_t tab_off = 0, tab_bytes = 0;  // host-built tables copied each schedule
    size_t zero_off = 0, zero_bytes = 0;
    char *host = nullptr;  // pinned staging of the tables
    cudaEvent_t uploaded = nullptr;
    int nclass = 0;
};

namespace {
constexpr int kMaxClasses = 8;  // team sizes 1, 2, 4, ... 128 blocks; class kMaxClasses: idle blocks
constexpr int kMaxSmid = 1024;

// Which %smid values this device's blocks run on.
__global__ void smid_probe_kernel(int *seen) {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    if (threadIdx.x == 0 && smid < (unsigned)kMaxSmid) seen[smid] = 1;
}
size_t al256(size_t v) { return (v + 255) / 256 * 256; }

template <typename F>
const void *batch_fn() {
    return sizeof(F) == 4 ? pcg32_batch_fn() : pcg64_batch_fn();
}
}  // namespace

template <typename F>
PcgBatchPlan *pcg_batch_create(const Scene<F> *const *scenes, const PcgScratch *const *scratch, int n,
                               const PcgShape &shape, std::string *err) {
    auto fail = [&](const std::string &m) -> PcgBatchPlan * {
        if (err) *err = m;
        return nullptr;
    };
    if (n <= 0) return fail("empty batch");
    if ((shape.threads != 32 && shape.threads != 64 && shape.threads != 128 && shape.threads != 256) || shape.K < 1 ||
        shape.K > shape.threads / 32 ||
        shape.stages < 2 || shape.stages > 4)
        return fail("unsupported batched PCG shape");
    int dmax = 0;
    for (int i = 0; i < n; i++) dmax = std::max(dmax, scenes[i]->sd.D);
    const void *fn = batch_fn<F>();
    int dev = 0, sms = 0, per = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) {
        cudaGetLastError();
        return fail("the batched PCG kernel is not available");
    }
    const size_t smem_max = (size_t)optin - fa.sharedSizeBytes;
    int block = shape.threads, K = shape.K, stages = shape.stages;
    (sizeof(F) == 4 ? pcg32_shape : pcg64_shape)(shape.threads, dmax, smem_max, &block, &K, &stages);
    const size_t smem = (sizeof(F) == 4 ? pcg32_smem : pcg64_smem)(K, dmax, stages);
    // the attribute stays at the device maximum, so a launch (or a graph
    // replay) of any plan is valid whatever plan was created last
    if (smem > smem_max ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max) != cudaSuccess) {
        cudaGetLastError();
        return fail("shared memory per block exceeds the device limit");
    }
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, block, smem);
    const int grid = sms * per;
    if (grid < 1) return fail("too few co-resident blocks for the batched PCG shape");

    PcgBatchPlan *P = new PcgBatchPlan;
    P->precision = (int)sizeof(F);
    P->n = n;
    P->shape = shape;
    P->grid = grid;
    P->block = block;
    P->K = K;
    P->stages = stages;
    P->smem = smem;
    for (int i = 0; i < n; i++) {
        P->strips.push_back(scenes[i]->sd.S);
        P->diags.push_back(scenes[i]->sd.D);
        P->cells.push_back(scenes[i]->w * scenes[i]->h);
    }
    size_t off = 0;
    const size_t o_jobs0 = off;
    off = al256(off + n * sizeof(PcgArgs<F>));
    const size_t o_jobs1 = off;
    off = al256(off + n * sizeof(PcgArgs<F>));
    P->tab_off = off;
    const size_t o_bt = off;
    off = al256(off + grid * sizeof(int2));
    const size_t o_team = off;
    off = al256(off + grid * sizeof(int2));
    const size_t o_cr = off;
    off = al256(off + (kMaxClasses + 1) * sizeof(int2));
    const size_t o_cj = off;
    off = al256(off + n * sizeof(int));
    P->tab_bytes = off - P->tab_off;
    const size_t o_ctl = off;
    off = al256(off + n * sizeof(int4));
    const size_t o_tj = off;
    off = al256(off + grid * sizeof(int));
    P->zero_off = off;
    const size_t o_cn = off;
    off += (kMaxClasses + 1) * sizeof(int);
    const size_t o_tb = off;
    off += kBarStride * grid * sizeof(unsigned);
    const size_t o_all = off;
    off += sizeof(unsigned);
    const size_t o_fill = off;
    off += sms * sizeof(int);
    const size_t o_gbar = off;
    off += sizeof(unsigned);
    const size_t o_rfail = off;
    off += sizeof(unsigned);
    P->zero_bytes = off - P->zero_off;
    off = al256(off);
    const size_t o_dense = off;
    off += kMaxSmid * sizeof(short);
    P->dev_bytes = al256(off);
    if (cudaMalloc(&P->dev, P->dev_bytes) != cudaSuccess ||
        cudaMallocHost(&P->host, P->tab_bytes) != cudaSuccess ||
        cudaEventCreateWithFlags(&P->uploaded, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        pcg_batch_destroy(P);
        return fail("device allocation for the batched PCG tables failed");
    }
    if (cudaMemset(P->dev + o_tj, 0xff, grid * sizeof(int)) != cudaSuccess) {  // no job yet: -1
        cudaGetLastError();
        pcg_batch_destroy(P);
        return fail("initialising the batched PCG tables failed");
    }
    P->jobs[0] = P->dev + o_jobs0;
    P->jobs[1] = P->dev + o_jobs1;
    P->B.block_team = (const int2 *)(P->dev + o_bt);
    P->B.team = (const int2 *)(P->dev + o_team);
    P->B.class_range = (const int2 *)(P->dev + o_cr);
    P->B.class_jobs = (const int *)(P->dev + o_cj);
    P->B.team_job = (int *)(P->dev + o_tj);
    P->B.class_next = (int *)(P->dev + o_cn);
    P->B.team_bar = (unsigned *)(P->dev + o_tb);
    P->B.all = (unsigned *)(P->dev + o_all);
    P->ctl = (int4 *)(P->dev + o_ctl);
    P->B.ctl = P->ctl;
    P->B.sm_fill = (int *)(P->dev + o_fill);
    P->B.grid_bar = (unsigned *)(P->dev + o_gbar);
    P->B.remap_fail = (unsigned *)(P->dev + o_rfail);
    P->B.sm_dense = (const short *)(P->dev + o_dense);
    P->B.nsm = sms;
    P->B.per = per;
    P->B.remap = 0;
    {
        // dense SM indices from a probe launch with many small blocks
        int *seen = (int *)(P->dev + o_fill);  // scratch before first use
        std::vector<int> hs(kMaxSmid, 0);
        std::vector<short> dense(kMaxSmid, -1);
        int *dseen = nullptr;
        if (cudaMalloc(&dseen, kMaxSmid * sizeof(int)) == cudaSuccess &&
            cudaMemset(dseen, 0, kMaxSmid * sizeof(int)) == cudaSuccess) {
            smid_probe_kernel<<<sms * 16, 32>>>(dseen);
            if (cudaMemcpy(hs.data(), dseen, kMaxSmid * sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess) {
                int n = 0;
                for (int i = 0; i < kMaxSmid; i++)
                    if (hs[i]) dense[i] = (short)n++;
                if (n == sms) P->B.remap = 1;
            }
        }
        cudaGetLastError();
        if (dseen) cudaFree(dseen);
        (void)seen;
        if (cudaMemcpy((void *)P->B.sm_dense, dense.data(), kMaxSmid * sizeof(short), cudaMemcpyHostToDevice) !=
            cudaSuccess) {
            cudaGetLastError();
            P->B.remap = 0;
        }
    }
    std::vector<PcgArgs<F>> a0(n), a1(n);
    for (int i = 0; i < n; i++) {
        a0[i] = make_args(*scenes[i], *scratch[i], 0);
        a1[i] = make_args(*scenes[i], *scratch[i], 1);
    }
    if (cudaMemcpy(P->jobs[0], a0.data(), n * sizeof(PcgArgs<F>), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(P->jobs[1], a1.data(), n * sizeof(PcgArgs<F>), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        pcg_batch_destroy(P);
        return fail("upload of the batched PCG jobs failed");
    }
    return P;
}

void pcg_batch_destroy(PcgBatchPlan *P) {
    if (!P) return;
    if (P->uploaded) {
        cudaEventSynchronize(P->uploaded);
        cudaEventDestroy(P->uploaded);
    }
    if (P->host) cudaFreeHost(P->host);
    if (P->dev) cudaFree(P->dev);
    delete P;
}

int pcg_batch_grid(const PcgBatchPlan *P) { return P->grid; }
int pcg_batch_block(const PcgBatchPlan *P) { return P->block; }
int pcg_batch_strips(const PcgBatchPlan *P) { return P->K; }
size_t pcg_batch_table_bytes(const PcgBatchPlan *P) { return P->tab_bytes; }
void pcg_batch_set_max_team(PcgBatchPlan *P, int blocks) { P->max_team = blocks > 0 ? blocks : 128; }

// Teams and queues from a cost model: work(i, g) = estimated time of scene i's
// solves on a team of g blocks.  Scene i starts in class first_class[i] (teams
// of 2^c blocks).  Every non-empty class gets one team; then, while blocks are
// left, the class with the latest estimated finish (its queue, largest scene
// first, handed to whichever of its teams frees first) gets one more team or
// teams twice as large (up to max_team blocks), whichever shortens that
// finish most per block spent, as long as it improves.  Each queue is ordered by work, largest first.
// teams[c] and tsize[c] give the teams of class c; returns the blocks in
// teams, or -1 when the classes' first teams alone exceed the grid.
int pcg_plan_teams_fn(int grid, int n, const int *first_class, const PlanWork &work, int *teams, int *tsize,
                      std::vector<std::vector<int>> *queues, int max_team) {
    std::vector<std::vector<int>> members(kMaxClasses);
    for (int i = 0; i < n; i++) {
        const int c = first_class[i];
        if (c < 0 || c >= kMaxClasses) return -1;
        members[c].push_back(i);
    }
    int size[kMaxClasses];
    // Finish time of a class: its queue (largest first) served by `nt` teams of
    // g blocks, each job taken by the team that frees first.
    std::vector<double> loads;  // min-heap of the teams' busy times
    auto finish = [&](int c, int nt, int g) {
        loads.assign(std::min<size_t>(nt, members[c].size()), 0.0);
        double fin = 0.0;
        for (int i : members[c]) {
            std::pop_heap(loads.begin(), loads.end(), std::greater<double>());
            loads.back() += work(i, g);
            fin = std::max(fin, loads.back());
            std::push_heap(loads.begin(), loads.end(), std::greater<double>());
        }
        return fin;
    };
    double fin[kMaxClasses];
    for (int c = 0; c < kMaxClasses; c++) {
        size[c] = 1 << c;
        std::stable_sort(members[c].begin(), members[c].end(),
                         [&](int a, int b) { return work(a, 1 << c) > work(b, 1 << c); });
    }
    int left = grid;
    for (int c = 0; c < kMaxClasses; c++) {
        teams[c] = members[c].empty() ? 0 : 1;
        left -= teams[c] << c;
        fin[c] = members[c].empty() ? 0.0 : finish(c, 1, size[c]);
    }
    if (left < 0) return -1;
    for (;;) {
        int best = -1;
        double bt = -1.0;
        for (int c = 0; c < kMaxClasses; c++) {
            if (!members[c].empty() && fin[c] > bt) {
                bt = fin[c];
                best = c;
            }
        }
        if (best < 0) break;
        const int c = best, sz = size[c];
        // more teams of the current size: the fewest that shorten the finish
        // (with jobs of equal size one more team may not)
        int add = 0;
        double fin_add = bt;
        for (int k = 1; teams[c] + k <= (int)members[c].size() && k * sz <= left; k++) {
            fin_add = finish(c, teams[c] + k, sz);
            if (fin_add < bt) {
                add = k;
                break;
            }
        }
        const bool can_add = add > 0;
        // every team of the class twice as large
        const bool can_grow = sz * 2 <= max_team && teams[c] * sz <= left;
        const double fin_grow = can_grow ? finish(c, teams[c], 2 * sz) : bt;
        // the option that shortens the finish most per block spent
        const double gain_add = can_add ? (bt - fin_add) / ((double)add * sz) : 0.0;
        const double gain_grow = can_grow ? (bt - fin_grow) / ((double)teams[c] * sz) : 0.0;
        if (gain_add > 0.0 && gain_add >= gain_grow) {
            teams[c] += add;
            left -= add * sz;
            fin[c] = fin_add;
        } else if (gain_grow > 0.0) {
            left -= teams[c] * sz;
            size[c] = 2 * sz;
            fin[c] = fin_grow;
        } else {
            break;
        }
    }
    for (int c = 0; c < kMaxClasses; c++) tsize[c] = size[c];
    if (queues) *queues = std::move(members);
    return grid - left;
}

// Host preview and the original model: scenes go to the class of the
// smallest power-of-two team that covers their strips (one sweeping warp per
// strip); work = work_sweep (the wavefront part, which more blocks do not
// shorten) + work_elem (the elementwise part at that smallest team, which
// shrinks with the team).
int pcg_plan_teams(int grid, int K, int n, const int *strips, const double *work_sweep,
                   const double *work_elem, int *teams, int *tsize, std::vector<std::vector<int>> *queues,
                   int max_team) {
    std::vector<int> cls(n);
    for (int i = 0; i < n; i++) {
        const int need = (strips[i] + K - 1) / K;
        int c = 0;
        while ((1 << c) < need) c++;
        if (c >= kMaxClasses) return -1;
        cls[i] = c;
    }
    const PlanWork w = [&](int i, int g) {
        return work_sweep[i] + (work_elem ? work_elem[i] * (double)(1 << cls[i]) / g : 0.0);
    };
    return pcg_plan_teams_fn(grid, n, cls.data(), w, teams, tsize, queues, max_team);
}

int pcg_batch_schedule(PcgBatchPlan *P, const int *first_class, const PlanWork &work, cudaStream_t st) {
    int teams[kMaxClasses], tsize[kMaxClasses];
    std::vector<std::vector<int>> members;
    if (pcg_plan_teams_fn(P->grid, P->n, first_class, work, teams, tsize, &members, P->max_team) < 0) return -1;
    // host tables
    if (cudaEventSynchronize(P->uploaded) != cudaSuccess) return -2;  // staging free again
    char *h = P->host;
    const size_t base = P->tab_off;
    auto at = [&](const void *devp) { return h + ((const char *)devp - (P->dev + base)); };
    int2 *bt = (int2 *)at(P->B.block_team);
    int2 *tm = (int2 *)at(P->B.team);
    int2 *cr = (int2 *)at(P->B.class_range);
    int *cj = (int *)at(P->B.class_jobs);
    int blk = 0, team = 0, pos = 0;
    for (int c = 0; c < kMaxClasses; c++) {
        cr[c] = make_int2(pos, (int)members[c].size());
        for (int i : members[c]) cj[pos++] = i;
        for (int t = 0; t < teams[c]; t++, team++) {
            tm[team] = make_int2(tsize[c], c);
            for (int r = 0; r < tsize[c]; r++) bt[blk++] = make_int2(team, r);
        }
    }
    // blocks left over form one-block teams of the empty idle class
    cr[kMaxClasses] = make_int2(pos, 0);
    for (; blk < P->grid; blk++, team++) {
        tm[team] = make_int2(1, kMaxClasses);
        bt[blk] = make_int2(team, 0);
    }
    if (cudaMemcpyAsync(P->dev + base, h, P->tab_bytes, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaEventRecord(P->uploaded, st) != cudaSuccess)
        return -2;
    return 0;
}

int4 *pcg_batch_ctl(PcgBatchPlan *P) { return P->ctl; }

// cfg.pinned >= -1 applies to every scene; -2 takes each scene's entry of the
// control table (cfg.limit is unused: limits come from the table).
template <typename F>
cudaError_t launch_pcg_batch(PcgBatchPlan *P, const PcgConfig &cfg, cudaStream_t st) {
    if (P->precision != (int)sizeof(F)) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(P->dev + P->zero_off, 0, P->zero_bytes, st);
    if (e != cudaSuccess) return e;
    const PcgArgs<F> *jobs = (const PcgArgs<F> *)P->jobs[cfg.heat ? 1 : 0];
    BatchTeams B = P->B;
    B.wait_limit = cfg.wait_limit > 0 ? cfg.wait_limit : kWaitLimit;
    int mode = cfg.mode, heat = cfg.heat, pinned = cfg.pinned, K = P->K, stages = P->stages;
    void *args[] = {&jobs, &B, &mode, &heat, &pinned, &K, &stages};
    return cudaLaunchCooperativeKernel(batch_fn<F>(), dim3(P->grid), dim3(P->block), args,
                                       P->smem, st);
}

template PcgBatchPlan *pcg_batch_create<double>(const Scene<double> *const *, const PcgScratch *const *, int,
                                                const PcgShape &, std::string *);
template PcgBatchPlan *pcg_batch_create<float>(const Scene<float> *const *, const PcgScratch *const *, int,
                                               const PcgShape &, std::string *);
template cudaError_t launch_pcg_batch<double>(PcgBatchPlan *, const PcgConfig &, cudaStream_t);
template cudaError_t launch_pcg_batch<float>(PcgBatchPlan *, const PcgConfig &, cudaStream_t);

template int pcg_max_blocks<double>();
template int pcg_max_blocks<float>();

}  // namespace ifl

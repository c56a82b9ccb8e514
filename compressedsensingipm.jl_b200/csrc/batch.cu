// C ABI (include/csipm.h), part 5: batched interior-point solves.
//
// csipm_solve_batch advances many recoveries of uneven sizes together, one
// kernel launch per step for all of them.  Each recovery is an ordinary
// handle (csipm_create: its plans, twiddles, mask, spectrum, A^T z0,
// reduction workspace and control block).  The batch writes an instance
// table to device memory — per instance its vector pointers (the offsets of
// its data), size, lambda, reduction workspace, control block and the
// PassArgs of its FFT passes (run-time plans: any length) — and launches
// every element kernel and every FFT pass once with gridDim.y = instances.
// Block (x, y) works on instance y; reductions complete per instance
// (RedWorkspace::xonly); the run-time-plan passes walk each instance's
// tiles with the same gridDim.x blocks.  An instance that has stopped
// (converged, max_iter, non-finite) returns at once from every kernel (its
// control block's status, or its CG scalars' done flag inside a CG loop).
//
// The method is csipm_solve's FP64 path — the same kernel bodies, the same
// device stop test and forcing term — in the reference packing, so each
// instance takes csipm_solve's iterates up to the order of floating-point
// sums (the FFT passes are the run-time-plan kernels (passes.cuh), not the two-level ones).
// The reference has no counterpart: it solves one recovery per call
// (src/CompressedSensingIPM.jl:31-36).
#include <chrono>

#include "internal.h"

namespace csipm_internal {

// CG iterations of one lockstep loop at most (csipm_solve's graph cap)
constexpr int BATCH_CG_CAP = 2000;

// ------------------------------------------------------------------ instance table
struct BInst {
    long long n;
    double lam;
    int precond;
    int pad;
    const double* b;     // A^T z0, reference order
    double *beta, *s1, *s2, *z1, *z2, *Qb, *Db, *Minv, *dba, *db, *r, *p, *q, *c;
    double* slots;
    double* partials;
    unsigned int* ticket;
    IpmCtl* ctl;
    CgScalars* cgs;
    __device__ __forceinline__ RedWorkspace ws(double* out) const { return RedWorkspace{partials, ticket, out, 1}; }
    __device__ __forceinline__ bool running() const { return ctl->status == IPM_RUNNING; }
};

// One FFT pass of one instance: its arguments, source and epilogue.
// P and Q are those of the 1D passes.
template <class Epi>
struct BPass {
    PassArgs<double> a;
    const double* src;
    Epi epi;
    const double2* twN;
    int P, Q;
};

// ------------------------------------------------------------------ element kernels
// Every wrapper reads its instance (blockIdx.y) and calls the kernel body
// csipm_solve launches; an instance that has stopped returns at once (all
// its blocks alike, so no reduction waits on it).
__global__ void __launch_bounds__(EW_THREADS) bk_init1(const BInst* __restrict__ I) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    ipm_init1_kernel_body(q.n, q.b, q.lam, q.beta, q.ws(q.slots + SL_MAXB));
}

__global__ void __launch_bounds__(EW_THREADS) bk_init2(const BInst* __restrict__ I) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    ipm_init2_kernel_body(q.n, q.b, q.Qb, q.lam, q.beta, q.slots + SL_MAXB, q.s1, q.s2, q.z1, q.z2);
}

// control blocks take ||z0||^2 and the KKT scale from the slots (one thread per instance)
__global__ void bk_ctl_start(const BInst* __restrict__ I, int count) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const BInst& q = I[k];
    q.ctl->z0sq = q.slots[SL_Z0SQ];
    q.ctl->kkt_scale = fmax(1.0, q.slots[SL_MAXB + 1]);
}

__global__ void __launch_bounds__(EW_THREADS, 3) bk_resid(const BInst* __restrict__ I, int step) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    if (!q.running()) return;
    // also starts the predictor's CG at the next iteration's tolerance
    ipm_resdiag_kernel_body<float, double, double>(q.n, q.b, q.Qb, q.lam, q.beta, q.s1, q.s2, q.z1, q.z2,
                                                   step ? q.dba : nullptr, step ? q.db : nullptr, q.slots + SL_SIGMU,
                                                   q.slots + SL_ALPHA, q.Db, q.Minv, (float*)nullptr, (float*)nullptr,
                                                   q.precond, q.ws(q.slots + SL_RED), q.r, q.p, q.cgs,
                                                   DevScalar(0.0, &q.ctl->rt_next));
}

// stop test per instance; a stopped instance also closes its CG scalars so
// the CG loops of the step skip it
__global__ void bk_stop(const BInst* __restrict__ I, int count) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const BInst& q = I[k];
    if (!q.running()) return;
    ipm_stop_kernel_body(q.slots + SL_RED, q.ctl, 0, 0);
    if (q.ctl->status != IPM_RUNNING) q.cgs->done = 1;
}

__global__ void __launch_bounds__(EW_THREADS) bk_cg_update(const BInst* __restrict__ I, int it, int which) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    // only an instance still running has a start of its own to copy
    if (!q.running()) return;
    cg_update_kernel_body<double, double, true>(q.n, it, which ? q.db : q.dba, which ? q.dba : nullptr, q.r, q.p, q.q,
                                                q.precond ? q.Minv : nullptr, q.ws(q.slots + SL_DUMMY), q.cgs);
}

__global__ void __launch_bounds__(EW_THREADS) bk_cg_pupdate(const BInst* __restrict__ I, int it) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    cg_pupdate_kernel_body<double>(q.n, it, q.r, q.precond ? q.Minv : nullptr, q.p, q.cgs);
}

// after a CG loop: count its iterations; a breakdown stops the instance
// (csipm_solve reports it as non-finite); one thread per instance
__global__ void bk_cg_post(const BInst* __restrict__ I, int count) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const BInst& q = I[k];
    if (!q.running()) return;
    q.ctl->cg_iter += q.cgs->iters;
    if (q.cgs->breakdown) q.ctl->status = IPM_NONFINITE;
}

// instances still iterating a CG loop (done clear) -> *out
__global__ void bk_cg_active(const BInst* __restrict__ I, int count, int* __restrict__ out) {
    pdl_enter();
    __shared__ int s;
    if (threadIdx.x == 0) s = 0;
    __syncthreads();
    int c = 0;
    for (int k = threadIdx.x; k < count; k += blockDim.x) c += (I[k].running() && !I[k].cgs->done) ? 1 : 0;
    atomicAdd(&s, c);
    __syncthreads();
    if (threadIdx.x == 0) *out = s;
}

__global__ void bk_running(const BInst* __restrict__ I, int count, int* __restrict__ out) {
    pdl_enter();
    __shared__ int s;
    if (threadIdx.x == 0) s = 0;
    __syncthreads();
    int c = 0;
    for (int k = threadIdx.x; k < count; k += blockDim.x) c += I[k].running() ? 1 : 0;
    atomicAdd(&s, c);
    __syncthreads();
    if (threadIdx.x == 0) *out = s;
}

__global__ void __launch_bounds__(EW_THREADS, 3) bk_stepstats(const BInst* __restrict__ I, int corrector) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    if (!q.running()) return;
    ipm_stepstats_kernel_body<double>(q.n, q.lam, q.s1, q.s2, q.z1, q.z2, corrector ? q.dba : nullptr,
                                      corrector ? q.slots + SL_SIGMU : nullptr, corrector ? q.db : q.dba,
                                      q.ws(q.slots + SL_SS));
}

__global__ void bk_sigma(const BInst* __restrict__ I, int count) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const BInst& q = I[k];
    if (!q.running()) return;
    ipm_sigma_kernel_body(q.slots + SL_SS, q.ctl, q.slots + SL_SIGMU);
}

__global__ void bk_alpha(const BInst* __restrict__ I, int count) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const BInst& q = I[k];
    if (!q.running()) return;
    ipm_alpha_kernel_body(q.slots + SL_SS, q.ctl, q.slots + SL_ALPHA);
}

// start of the corrector's CG from the predictor's residual, at the warm start dba
__global__ void __launch_bounds__(EW_THREADS, 3) bk_corr(const BInst* __restrict__ I) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    if (!q.running()) return;
    ipm_corr_kernel_body<double, double, double>(q.n, q.lam, q.s1, q.s2, q.z1, q.z2, (const double*)q.dba,
                                                 q.slots + SL_SIGMU, (const double*)q.r, q.r, q.p,
                                                 q.precond ? (const double*)q.Minv : nullptr, q.cgs,
                                                 q.ws(q.slots + SL_DUMMY), DevScalar(0.0, &q.ctl->rt));
}

__global__ void __launch_bounds__(EW_THREADS) bk_beta_step(const BInst* __restrict__ I) {
    pdl_enter();
    const BInst& q = I[blockIdx.y];
    if (!q.running()) return;
    ipm_beta_step_kernel_body<double>(q.n, q.beta, q.db, q.slots + SL_ALPHA);
}

// ------------------------------------------------------------------ FFT pass kernels
// One block size for all instances of a batch (each brings its own plan and
// tile layout).
constexpr int BATCH_THREADS = 256;

template <bool INV, int IN, int OUT, class Epi>
__global__ void __launch_bounds__(BATCH_THREADS) bk_strided(const BPass<Epi>* __restrict__ B) {
    pdl_enter();
    const BPass<Epi>& e = B[blockIdx.y];
    const PassArgs<double>& a = e.a;
    strided_pass_kernel_body<double, INV, IN, OUT, double, Epi>(a, e.src, e.epi);
}

template <bool MASK, class Epi>
__global__ void __launch_bounds__(BATCH_THREADS) bk_row(const BPass<Epi>* __restrict__ B) {
    pdl_enter();
    const PassArgs<double>& a = B[blockIdx.y].a;
    row_pass_kernel_body<double, IN_SPEC, OUT_SPEC, MASK>(a);
}

template <class Epi>
__global__ void __launch_bounds__(BATCH_THREADS) bk_l1d_first(const BPass<Epi>* __restrict__ B) {
    pdl_enter();
    const BPass<Epi>& e = B[blockIdx.y];
    const PassArgs<double>& a = e.a;
    l1d_first_kernel_body<double, double>(a, e.src, e.twN, e.P);
}

template <bool MASK, class Epi>
__global__ void __launch_bounds__(BATCH_THREADS) bk_l1d_row(const BPass<Epi>* __restrict__ B) {
    pdl_enter();
    const BPass<Epi>& e = B[blockIdx.y];
    const PassArgs<double>& a = e.a;
    l1d_row_kernel_body<double, IN_SPEC, OUT_SPEC, MASK>(a, e.twN, e.P, e.Q);
}

template <class Epi>
__global__ void __launch_bounds__(BATCH_THREADS) bk_l1d_last(const BPass<Epi>* __restrict__ B) {
    pdl_enter();
    const BPass<Epi>& e = B[blockIdx.y];
    const PassArgs<double>& a = e.a;
    l1d_last_kernel_body<double, Epi>(a, e.twN, e.P, e.Q, e.epi);
}

// ------------------------------------------------------------------ host side
// The pass sequence of one A'A product for the batch's pipeline kind, over
// tables of per-instance pass arguments (one table per pass, built once).
enum { PK_1D = 0, PK_1DL = 1, PK_2D = 2, PK_3D = 3 };

template <class Epi>
struct BProduct {
    int kind = 0;
    bool mask = false;
    int count = 0;
    // device tables, one per pass (up to 5)
    BPass<Epi>* tab[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    // launch shapes
    size_t smem[5] = {0, 0, 0, 0, 0};
    int gx[5] = {0, 0, 0, 0, 0};
    int npass = 0;
};

struct BatchState {
    int count = 0;
    cudaStream_t st = nullptr;
    cudaMemPool_t pool = nullptr;
    std::vector<void*> allocs;
    BInst* inst = nullptr;        // device table
    int* flag = nullptr;          // device counter (active CG loops / running instances)
    int* hflag = nullptr;         // pinned mirror
    BProduct<EpiStore<double>> pq;   // Qb = A'A beta
    BProduct<EpiCG<double>> pc;      // q = A'A p + Db p, p.q
    int gx_elem = 1;
    long long launches = 0;
    char* hstage = nullptr;       // pinned staging of the tables' uploads
    size_t hstage_bytes = 0, hstage_used = 0;
    ~BatchState() {
        for (void* p : allocs) cudaFreeAsync(p, st);
        if (hflag) pinned_put(hflag, 64);
        if (hstage) {
            cudaStreamSynchronize(st);   // the uploads from it have completed
            pinned_put(hstage, hstage_bytes);
        }
    }
    // host -> device copy through the pinned staging buffer (asynchronous);
    // pageable once the buffer is full
    cudaError_t upload(void* dst, const void* src, size_t bytes) {
        const size_t at = (hstage_used + 15) & ~(size_t)15;
        if (hstage && at + bytes <= hstage_bytes) {
            std::memcpy(hstage + at, src, bytes);
            hstage_used = at + bytes;
            return cudaMemcpyAsync(dst, hstage + at, bytes, cudaMemcpyHostToDevice, st);
        }
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    }
    template <typename P>
    bool alloc(P** p, size_t count_) {
        void* q = nullptr;
        if (cudaMallocFromPoolAsync(&q, sizeof(P) * count_, pool, st) != cudaSuccess) return false;
        allocs.push_back(q);
        *p = reinterpret_cast<P*>(q);
        return true;
    }
};

int batch_kind(csipm_handle h) {
    if (h->g.dim == 3) return PK_3D;
    if (h->g.dim == 2) return PK_2D;
    // both run the same three passes; the two classes stay apart as csipm.h says
    return h->g.m1 > L1D_MIN_M ? PK_1DL : PK_1D;
}

// Persistent-pass grid: the batch shares one wave of the kernel's CTAs
template <typename K>
int batch_grid(K kernel, int threads, size_t smem, int count, int max_tiles) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)kernel, threads, smem) != cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    const int wave = std::max(1, sms) * per_sm;
    const int g = std::max(1, (wave + count - 1) / count);
    return std::max(1, std::min(g, max_tiles));
}

// Builds the pass tables of one product kind.  x: per-instance source
// vectors (beta or p); epi: per-instance epilogues; skip: per-instance flags.
template <class Epi>
int build_product(BatchState& B, BProduct<Epi>& P, const std::vector<csipm_handle>& hs, const std::vector<const double*>& x,
                  const std::vector<Epi>& epi, const std::vector<const int*>& skip) {
    const int K = (int)hs.size();
    P.count = K;
    P.kind = batch_kind(hs[0]);
    P.mask = hs[0]->op64.maskw != nullptr;
    std::vector<std::vector<BPass<Epi>>> t;
    // an instance's pass: its tile at the handle's lines (or rows) per CTA,
    // laid out for the batch's block size (csipm_solve_batch has refused
    // in-place rows)
    auto add = [&](int pass, const FftOperator<double>& op, PassArgs<double> a, const PassCfg& cfg, PassKind kind,
                   const double* src, const Epi& e, const int* sk) -> bool {
        if ((int)t.size() <= pass) t.resize(pass + 1);
        PassCfg c;
        const int n = cfg.tiles * cfg.tb;
        for (int tb = cfg.tb; tb >= 1; tb /= 2) {
            lay_pass(a.pl, a.Ltab, tb, n, kind, BATCH_THREADS, sizeof(double2), &c);
            if (c.smem <= FftOperator<double>::smem_limit()) break;
        }
        FftOperator<double>::tile_args(c, &a);
        a.skip = sk;
        BPass<Epi> bp{};
        bp.a = a;
        bp.src = src;
        bp.epi = e;
        bp.twN = op.tw1;
        bp.P = op.l1P;
        bp.Q = op.l1Q;
        t[pass].push_back(bp);
        P.smem[pass] = std::max(P.smem[pass], c.smem);
        P.gx[pass] = std::max(P.gx[pass], c.tiles);
        return c.smem <= FftOperator<double>::smem_limit();
    };
    for (int k = 0; k < K; ++k) {
        FftOperator<double>& op = hs[k]->op64;
        const double sc = 1.0 / (2.0 * (double)op.g.N);
        const int* sk = skip[k];
        bool ok = true;
        if (op.g.dim == 1) {
            ok = add(0, op, l1d_args(op, 0, 1.0, sk), op.f_cfg, PASS_LINES, x[k], epi[k], sk) &&
                 add(1, op, l1d_args(op, 1, sc, sk), op.p_cfg, PASS_PAIRS, nullptr, epi[k], sk) &&
                 add(2, op, l1d_args(op, 2, 1.0, sk), op.q_cfg, PASS_PAIRS, nullptr, epi[k], sk);
        } else {
            const PassArgs<double> a2 = op.strided_args(2), ra = op.row_args(sc, nullptr, nullptr);
            int pass = 0;
            ok = add(pass++, op, a2, op.s2_cfg, PASS_LINES, x[k], epi[k], sk);   // gather + inverse dim 2
            if (P.kind == PK_3D) ok = add(pass++, op, op.strided_args(3), op.s3_cfg, PASS_LINES, nullptr, epi[k], sk) && ok;
            ok = add(pass++, op, ra, op.row_cfg, PASS_ROWS, nullptr, epi[k], sk) && ok;   // rows
            if (P.kind == PK_3D) ok = add(pass++, op, op.strided_args(3), op.s3_cfg, PASS_LINES, nullptr, epi[k], sk) && ok;
            ok = add(pass++, op, a2, op.s2_cfg, PASS_LINES, nullptr, epi[k], sk) && ok;   // forward dim 2 + scatter
        }
        if (!ok) return CSIPM_ERR_UNSUPPORTED;
    }
    P.npass = (int)t.size();
    for (int pass = 0; pass < P.npass; ++pass) {
        if (!B.alloc(&P.tab[pass], t[pass].size())) return CSIPM_ERR_OOM;
        if (B.upload(P.tab[pass], t[pass].data(), sizeof(BPass<Epi>) * t[pass].size()) != cudaSuccess)
            return CSIPM_ERR_CUDA;
    }
    return CSIPM_OK;
}

template <typename K, class Epi>
cudaError_t launch_bpass(K kernel, const BProduct<Epi>& P, int pass, cudaStream_t st) {
    const cudaError_t e = smem_optin(kernel, P.smem[pass]);
    if (e != cudaSuccess) return e;
    const int gx = batch_grid(kernel, BATCH_THREADS, P.smem[pass], P.count, P.gx[pass]);
    launch_pdl(true, kernel, dim3(gx, P.count), BATCH_THREADS, P.smem[pass], st, P.tab[pass]);
    return cudaGetLastError();
}

// One A'A product for every instance of the batch.
template <class Epi>
cudaError_t batch_product(BatchState& B, const BProduct<Epi>& P) {
    cudaStream_t st = B.st;
    cudaError_t e = cudaSuccess;
    B.launches += P.npass;
    if (P.kind == PK_1D || P.kind == PK_1DL) {
        if ((e = launch_bpass(bk_l1d_first<Epi>, P, 0, st)) != cudaSuccess) return e;
        e = P.mask ? launch_bpass(bk_l1d_row<true, Epi>, P, 1, st) : launch_bpass(bk_l1d_row<false, Epi>, P, 1, st);
        if (e != cudaSuccess) return e;
        return launch_bpass(bk_l1d_last<Epi>, P, 2, st);
    }
    int pass = 0;
    if ((e = launch_bpass(bk_strided<true, IN_GATHER, OUT_SPEC, Epi>, P, pass++, st)) != cudaSuccess) return e;
    if (P.kind == PK_3D && (e = launch_bpass(bk_strided<true, IN_SPEC, OUT_SPEC, Epi>, P, pass++, st)) != cudaSuccess)
        return e;
    e = P.mask ? launch_bpass(bk_row<true, Epi>, P, pass, st) : launch_bpass(bk_row<false, Epi>, P, pass, st);
    if (e != cudaSuccess) return e;
    ++pass;
    if (P.kind == PK_3D && (e = launch_bpass(bk_strided<false, IN_SPEC, OUT_SPEC, Epi>, P, pass++, st)) != cudaSuccess)
        return e;
    return launch_bpass(bk_strided<false, IN_SPEC, OUT_SCATTER, Epi>, P, pass, st);
}

int read_flag(BatchState& B) {
    if (cudaMemcpyAsync(B.hflag, B.flag, sizeof(int), cudaMemcpyDeviceToHost, B.st) != cudaSuccess ||
        cudaStreamSynchronize(B.st) != cudaSuccess)
        return -1;
    return *B.hflag;
}

// One Newton solve's CG loop for every running instance, in lockstep: the
// product skips instances whose loop is done, the updates return for them.
// which: 0 predictor (iterate dba), 1 corrector (db).
int batch_cg_loop(BatchState& B, int which) {
    const dim3 ge(B.gx_elem, B.count);
    int since = 0, chunk = 2;
    for (int it = 0; it < BATCH_CG_CAP; ++it) {
        cudaError_t e = batch_product(B, B.pc);
        if (e != cudaSuccess) return fail(nullptr, CSIPM_ERR_CUDA, std::string("batch CG product: ") + cudaGetErrorString(e));
        launch_pdl(true, bk_cg_update, ge, EW_THREADS, 0, B.st, B.inst, it, which);
        launch_pdl(true, bk_cg_pupdate, ge, EW_THREADS, 0, B.st, B.inst, it);
        B.launches += 2;
        if (++since >= chunk) {
            since = 0;
            if (chunk < 8) chunk *= 2;
            launch_pdl(true, bk_cg_active, 1, 256, 0, B.st, B.inst, B.count, B.flag);
            B.launches += 1;
            const int active = read_flag(B);
            if (active < 0) return fail(nullptr, CSIPM_ERR_CUDA, std::string("batch CG loop: ") + cudaGetErrorString(cudaGetLastError()));
            if (active == 0) break;
        }
    }
    launch_pdl(true, bk_cg_post, (B.count + 127) / 128, 128, 0, B.st, B.inst, B.count);
    B.launches += 1;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CSIPM_OK : fail(nullptr, CSIPM_ERR_CUDA, std::string("batch CG loop: ") + cudaGetErrorString(e));
}

}  // namespace csipm_internal

extern "C" {

int csipm_solve_batch(csipm_handle* hs_in, int count, double* const* beta_out, csipm_stats* stats) {
    using namespace csipm_internal;
    if (!hs_in || !beta_out || count < 1) return fail(nullptr, CSIPM_ERR_INVALID, "null argument or empty batch");
    std::vector<csipm_handle> hs(hs_in, hs_in + count);
    for (int k = 0; k < count; ++k) {
        if (!hs[k] || !beta_out[k]) return fail(nullptr, CSIPM_ERR_INVALID, "null handle or output in the batch");
        if (hs[k]->device != hs[0]->device) return fail(nullptr, CSIPM_ERR_INVALID, "the batch spans devices");
        if (batch_kind(hs[k]) != batch_kind(hs[0]) || (hs[k]->op64.maskw != nullptr) != (hs[0]->op64.maskw != nullptr))
            return fail(nullptr, CSIPM_ERR_INVALID,
                        "a batch shares the dimension count, the long-row 1D passes and the presence of missing samples");
        // rows longer than a tile run in place, in a kernel and with plans of
        // their own that a batch's passes do not take
        if (hs[k]->g.dim >= 2 && !hs[k]->op64.row_cfg.pp)
            return fail(nullptr, CSIPM_ERR_UNSUPPORTED,
                        "dimension 1 of an instance is too long for the batch's row pass; solve it alone");
        for (int j = 0; j < k; ++j)
            if (hs[j] == hs[k]) return fail(nullptr, CSIPM_ERR_INVALID, "a handle appears twice in the batch");
    }
    for (csipm_handle h : hs) {
        const int r = ensure_ipm_buffers(h);
        if (r) return r;
    }
    BatchState B;
    B.count = count;
    B.st = hs[0]->stream;
    B.pool = hs[0]->pool;
    cudaStream_t st = B.st;
    // the handles' own streams hand over to the batch's
    cudaEvent_t ev = nullptr;
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return fail(nullptr, CSIPM_ERR_CUDA, "event");
    for (csipm_handle h : hs)
        if (h->stream != st) {
            cudaEventRecord(ev, h->stream);
            cudaStreamWaitEvent(st, ev, 0);
        }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    auto done = [&](int status) {
        cudaEventDestroy(ev);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        return status;
    };
    // ---- instance table and control blocks
    std::vector<BInst> I(count);
    long long nmax = 1;
    for (int k = 0; k < count; ++k) {
        csipm_handle h = hs[k];
        BInst& q = I[k];
        q.n = h->N;
        q.lam = h->lambda;
        q.precond = h->opt.preconditioner ? 1 : 0;
        q.b = h->b;
        q.beta = h->beta; q.s1 = h->s1; q.s2 = h->s2; q.z1 = h->z1; q.z2 = h->z2; q.Qb = h->Qb;
        q.Db = h->Db; q.Minv = h->Minv; q.dba = h->dba; q.db = h->db;
        q.r = h->cg_r; q.p = h->cg_p; q.q = h->cg_q; q.c = h->c;
        q.slots = h->slots;
        q.partials = h->partials;
        q.ticket = h->ticket;
        q.ctl = h->ctl;
        q.cgs = h->cgs;
        nmax = std::max(nmax, h->N);
        IpmCtl& c = *h->hctl;
        std::memset(&c, 0, sizeof(IpmCtl));
        const csipm_options& o = h->opt;
        c.tol = o.tol;
        c.rt_opt = o.ipm_cg_rtol;
        c.forcing = o.ipm_cg_forcing;
        c.rt_floor = CG_FORCING_FLOOR;
        c.rin_floor = CG_FORCING_FLOOR;
        c.lam = h->lambda;
        c.two_n = 2.0 * (double)h->N;
        c.max_iter = o.max_iter;
        c.k = -1;
        c.rt_next = o.ipm_cg_rtol;
        c.rin_next = o.ipm_cg_rtol;
        c.status = IPM_RUNNING;
        if (cudaMemcpyAsync(h->ctl, h->hctl, sizeof(IpmCtl), cudaMemcpyHostToDevice, st) != cudaSuccess)
            return done(fail(nullptr, CSIPM_ERR_CUDA, "control block upload failed"));
    }
    if (!B.alloc(&B.inst, count) || !B.alloc(&B.flag, 1)) return done(fail(nullptr, CSIPM_ERR_OOM, "out of device memory"));
    B.hflag = (int*)pinned_get(64);
    if (!B.hflag) return done(fail(nullptr, CSIPM_ERR_OOM, "pinned host allocation failed"));
    {
        const size_t need = sizeof(BInst) * count + 10 * sizeof(BPass<EpiCG<double>>) * count + 16 * 12;
        size_t pb = 1 << 16;
        while (pb < need) pb <<= 1;
        if ((B.hstage = (char*)pinned_get(pb)) != nullptr) B.hstage_bytes = pb;
    }
    if (B.upload(B.inst, I.data(), sizeof(BInst) * count) != cudaSuccess)
        return done(fail(nullptr, CSIPM_ERR_CUDA, "instance table upload failed"));
    {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)bk_resid, EW_THREADS, 0);
        const long long wave = (long long)std::max(1, sms) * std::max(1, per_sm);
        B.gx_elem = (int)std::max(1LL, std::min((nmax + EW_THREADS - 1) / EW_THREADS,
                                                std::max(1LL, (wave + count - 1) / count)));
    }
    // ---- product tables: Qb = A'A beta (skips stopped instances), the CG's q = A'A p + Db p
    {
        std::vector<const double*> xb(count), xp(count);
        std::vector<EpiStore<double>> es(count);
        std::vector<EpiCG<double>> ec(count);
        std::vector<const int*> sk_ipm(count), sk_cg(count);
        for (int k = 0; k < count; ++k) {
            csipm_handle h = hs[k];
            xb[k] = h->beta;
            xp[k] = h->cg_p;
            es[k] = EpiStore<double>{h->Qb};
            RedWorkspace w{h->partials, h->ticket, &h->cgs->pq, 1};
            ec[k] = EpiCG<double>{h->cg_p, h->Db, h->cg_q, w, 0.0};
            sk_ipm[k] = &h->ctl->status;
            sk_cg[k] = &h->cgs->done;
        }
        int r = build_product(B, B.pq, hs, xb, es, sk_ipm);
        if (!r) r = build_product(B, B.pc, hs, xp, ec, sk_cg);
        if (r) return done(fail(nullptr, r, "batch pass tables failed"));
    }
    const dim3 ge(B.gx_elem, count);
    const int g1 = (count + 127) / 128;
    // ---- initial point (as csipm_solve)
    launch_pdl(true, bk_init1, ge, EW_THREADS, 0, st, B.inst);
    {
        const cudaError_t e = batch_product(B, B.pq);
        if (e != cudaSuccess) return done(fail(nullptr, CSIPM_ERR_CUDA, std::string("batch product: ") + cudaGetErrorString(e)));
    }
    launch_pdl(true, bk_init2, ge, EW_THREADS, 0, st, B.inst);
    launch_pdl(true, bk_ctl_start, g1, 128, 0, st, B.inst, count);
    B.launches += 3;
    int status = CSIPM_OK;
    bool pending = false;
    for (int iter = 0;; ++iter) {
        if (iter > 0) {
            const cudaError_t e = batch_product(B, B.pq);
            if (e != cudaSuccess) {
                status = fail(nullptr, CSIPM_ERR_CUDA, std::string("batch product: ") + cudaGetErrorString(e));
                break;
            }
        }
        launch_pdl(true, bk_resid, ge, EW_THREADS, 0, st, B.inst, pending ? 1 : 0);
        launch_pdl(true, bk_stop, g1, 128, 0, st, B.inst, count);
        launch_pdl(true, bk_running, 1, 256, 0, st, B.inst, count, B.flag);
        B.launches += 3;
        const int running = read_flag(B);
        if (running < 0) { status = fail(nullptr, CSIPM_ERR_CUDA, "batch synchronisation failed"); break; }
        if (running == 0) break;
        // predictor from zero (the residual pass started its CG)
        if ((status = batch_cg_loop(B, 0)) != CSIPM_OK) break;
        // centring target and corrector, warm-started at dba
        launch_pdl(true, bk_stepstats, ge, EW_THREADS, 0, st, B.inst, 0);
        launch_pdl(true, bk_sigma, g1, 128, 0, st, B.inst, count);
        launch_pdl(true, bk_corr, ge, EW_THREADS, 0, st, B.inst);
        B.launches += 3;
        if ((status = batch_cg_loop(B, 1)) != CSIPM_OK) break;
        // step
        launch_pdl(true, bk_stepstats, ge, EW_THREADS, 0, st, B.inst, 1);
        launch_pdl(true, bk_alpha, g1, 128, 0, st, B.inst, count);
        launch_pdl(true, bk_beta_step, ge, EW_THREADS, 0, st, B.inst);
        B.launches += 3;
        {
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) {
                status = fail(nullptr, CSIPM_ERR_CUDA, std::string("batch launch: ") + cudaGetErrorString(e));
                break;
            }
        }
        pending = true;
    }
    // ---- results
    for (int k = 0; k < count; ++k) {
        csipm_handle h = hs[k];
        if (cudaMemcpyAsync(beta_out[k], h->beta, sizeof(double) * h->N, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
            cudaMemcpyAsync(h->hctl, h->ctl, sizeof(IpmCtl), cudaMemcpyDeviceToHost, st) != cudaSuccess) {
            status = fail(nullptr, CSIPM_ERR_CUDA, "batch result copy failed");
            break;
        }
    }
    cudaEventRecord(e1, st);
    if (cudaEventSynchronize(e1) != cudaSuccess) return done(fail(nullptr, CSIPM_ERR_CUDA, "batch synchronisation failed"));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    int first_bad = CSIPM_OK;
    for (int k = 0; k < count; ++k) {
        csipm_handle h = hs[k];
        const IpmCtl& C = *h->hctl;
        csipm_stats S{};
        S.status = status != CSIPM_OK ? status
                   : C.status == IPM_CONVERGED ? CSIPM_OK
                   : C.status == IPM_NONFINITE ? CSIPM_ERR_NONFINITE : CSIPM_ERR_IPM_MAXITER;
        S.ipm_iter = C.k;
        S.cg_iter = C.cg_iter;
        S.matvecs = C.cg_iter + C.k + 1;
        S.gap = C.gap;
        S.obj = C.obj;
        S.lasso_obj = C.F;
        S.mu = C.mu;
        S.dual_inf = C.dual_inf;
        S.solve_ms = ms;
        S.launches = B.launches;
        if (S.status != CSIPM_OK) {
            h->err = status != CSIPM_OK                  ? std::string(get_last_error())
                     : S.status == CSIPM_ERR_NONFINITE ? "non-finite iterate or CG breakdown"
                                                        : "IPM reached max_iter before the tolerance";
            if (first_bad == CSIPM_OK) first_bad = S.status;
        }
        if (stats) stats[k] = S;
    }
    if (first_bad != CSIPM_OK && status == CSIPM_OK) {
        status = first_bad;
        set_last_error("an instance of the batch did not converge (see its csipm_stats.status)");
    }
    return done(status);
}

}  // extern "C"

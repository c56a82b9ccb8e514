// 1D: the real FFT of length N1 = 2M runs its length-M complex FFT as
// M = P*Q (four-step) over many CTAs.
//
// Spectrum index k = k1 + P*k2 (k1 < P, k2 < Q), spatial index n = n2 + Q*n1.
// With W = exp(+2 pi i / M) for the inverse transform:
//     z[n2 + Q n1] = sum_k1 W_P^{n1 k1} W^{n2 k1} sum_k2 Z[k1 + P k2] W_Q^{n2 k2}
// and the forward transform is the same factorisation run backwards.  The
// half spectrum buffer (M+1 complex) holds every intermediate in place:
//
//   first:  lines k1 (Q values, stride P): gather beta -> X[k], X[M-k] ->
//           C2R pre-processing -> inverse DFT_Q -> twiddle conj(w_M^{n2 k1})
//           -> spec[k1 + P n2]
//   row:    rows n2 (P contiguous values): inverse DFT_P -> z[n2 + Q n1]
//           scaled and masked -> (A: store the real samples) or forward
//           DFT_P -> twiddle w_M^{n2 k1} -> spec[k1 + P n2]
//           (A^T: the row starts from the real samples instead)
//   last:   lines k1 and their mirrors P - k1 together: forward DFT_Q along
//           k2, then Z[k] and Z[M-k] are both in the tile: R2C
//           post-processing -> scatter to beta with the epilogue
//
// w_M^e = exp(-2 pi i e / M) is read from the N1-th root table (index 2e).
//
// The passes are bound by latency, not bandwidth (1D vectors of the serving
// range sit in L2), so what counts is launches and the chain inside one:
// three launches where four kernels ran (a plain lines pass, then the post-
// processing over all k), one for short rows (l1d_one_kernel), and register-radix stages (fft_device.cuh) with
// loads and stores attached to the first and last stage.  Epilogues with many
// operands on long vectors take the post-processing out of the last pass again
// (l1d_last).
#pragma once
#include "passes.cuh"

namespace csipm {

// beta of spectrum position k (0 <= k <= M), 1D packing
template <typename T, typename TS>
__device__ __forceinline__ cplx_t<T> gather1(const TS* __restrict__ src, int M, int k) {
    const bool vert = k == 0 || k == M;
    const T a = (T)src[k == 0 ? 0 : (k == M ? 1 : k + 1)], b = (T)src[vert ? 0 : M + k];
    const T r = (T)0.7071067811865476;
    return vert ? mk(a, (T)0) : mk(a * r, b * r);
}

// ---------------------------------------------------------------- first pass
template <typename T, typename TS>
struct L1dFirst {
    using C = cplx_t<T>;
    const TS* src;
    C* spec;
    const C* twN;
    int M, P, k1;
    __device__ __forceinline__ C one(int x, int) const {
        if (k1 >= P) return mk((T)0, (T)0);
        const int k = k1 + P * x;
        return c2r_pre(gather1<T>(src, M, k), gather1<T>(src, M, M - k), twN[k]);
    }
    __device__ __forceinline__ void one(int x, int, C v) const {
        if (k1 >= P) return;
        const int ex = x * k1;   // < M
        spec[k1 + (size_t)P * x] = ex ? cmulc(v, twN[2 * ex]) : v;
    }
    template <int R> __device__ __forceinline__ void load(C* v, int u, int m, int b) const {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = one(u + r * m, b);
    }
    template <int R> __device__ __forceinline__ void store(const C* v, int u, int Ns, int b) const {
#pragma unroll
        for (int r = 0; r < R; ++r) one(u + r * Ns, b, v[r]);
    }
};

template <typename T, typename TS>
__device__ __forceinline__ void l1d_first_kernel_body(const PassArgs<T>& a, const TS* __restrict__ src,
                                                      const cplx_t<T>* __restrict__ twN, int P) {
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FftTile<cplx_t<T>> t = make_tile(a, smem_raw);
    const int b = threadIdx.x & ((1 << a.lay.lg) - 1);
    for (int i0 = blockIdx.x << a.lay.lg; i0 < P; i0 += gridDim.x << a.lay.lg) {
        L1dFirst<T, TS> io{src, a.spec, twN, a.g.m1, P, i0 + b};
        fft_through<T, true>(t, io, io);
        __syncthreads();
    }
}
template <typename T, typename TS>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas<T>())
l1d_first_kernel(const __grid_constant__ PassArgs<T> a, const TS* __restrict__ src, const cplx_t<T>* __restrict__ twN, int P) {
    pdl_enter();
    l1d_first_kernel_body<T, TS>(a, src, twN, P);
}

// ------------------------------------------------------------------ row pass
// one row n2: P contiguous spectrum values, or the real samples n2 + Q n1
template <typename T, bool MASK>
struct L1dRow {
    using C = cplx_t<T>;
    C* spec;             // of this row
    const T* in;
    T* out;
    const uint32_t* mask;
    const C* twN;
    int n2, Q;
    T sc;
    bool live;
    __device__ __forceinline__ C keep(int n1, C y) const {
        y.x *= sc;
        y.y *= sc;
        if (MASK && live) {
            const int n = n2 + Q * n1;
            const uint32_t w = mask[n >> 4];
            const int sh = (2 * n) & 31;
            if (!((w >> sh) & 1u)) y.x = (T)0;
            if (!((w >> (sh + 1)) & 1u)) y.y = (T)0;
        }
        return y;
    }
};
template <typename T, bool MASK>
struct L1dRowSpec : L1dRow<T, MASK> {   // spectrum in, twiddled spectrum out
    using C = cplx_t<T>;
    __device__ __forceinline__ C one(int k1, int) const { return this->live ? this->spec[k1] : mk((T)0, (T)0); }
    __device__ __forceinline__ void one(int k1, int, C v) const {
        if (!this->live) return;
        const int ex = this->n2 * k1;   // < M
        this->spec[k1] = ex ? cmul(v, this->twN[2 * ex]) : v;
    }
    template <int R> __device__ __forceinline__ void load(C* v, int u, int m, int b) const {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = one(u + r * m, b);
    }
    template <int R> __device__ __forceinline__ void store(const C* v, int u, int Ns, int b) const {
#pragma unroll
        for (int r = 0; r < R; ++r) one(u + r * Ns, b, v[r]);
    }
};
template <typename T, bool MASK>
struct L1dRowReal : L1dRow<T, MASK> {   // real samples
    using C = cplx_t<T>;
    __device__ __forceinline__ C one(int n1, int) const {
        if (!this->live) return mk((T)0, (T)0);
        return this->keep(n1, *reinterpret_cast<const C*>(this->in + 2 * ((size_t)this->n2 + (size_t)this->Q * n1)));
    }
    __device__ __forceinline__ void one(int n1, int, C v) const {
        if (this->live) *reinterpret_cast<C*>(this->out + 2 * ((size_t)this->n2 + (size_t)this->Q * n1)) = this->keep(n1, v);
    }
    template <int R> __device__ __forceinline__ void load(C* v, int u, int m, int b) const {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = one(u + r * m, b);
    }
    template <int R> __device__ __forceinline__ void store(const C* v, int u, int Ns, int b) const {
#pragma unroll
        for (int r = 0; r < R; ++r) one(u + r * Ns, b, v[r]);
    }
};

template <typename T, int IN, int OUT, bool MASK>
__device__ __forceinline__ void l1d_row_kernel_body(const PassArgs<T>& a, const cplx_t<T>* __restrict__ twN, int P,
                                                    int Q) {
    using C = cplx_t<T>;
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FftTile<C> t = make_tile(a, smem_raw);
    const int b = threadIdx.x & ((1 << a.lay.lg) - 1);
    for (int r0 = blockIdx.x << a.lay.lg; r0 < Q; r0 += gridDim.x << a.lay.lg) {
        const int n2 = r0 + b;
        const L1dRow<T, MASK> base{a.spec + (size_t)P * n2, a.real_in, a.real_out, a.maskw, twN, n2, Q, (T)a.scale,
                                   n2 < Q};
        L1dRowSpec<T, MASK> sp{base};
        L1dRowReal<T, MASK> re{base};
        if (IN == IN_REAL) {
            first_stage<T, false>(t, re);
        } else {
            t.st = a.inv;
            first_stage<T, true>(t, sp);
            mid_stages<T, true>(t, 1, t.nst - 1);
            if (OUT == OUT_REAL) {
                last_stage<T, true>(t, re);
                __syncthreads();
                continue;
            }
            chain_stage<T>(t, [&](int n1, int, C z) { return base.keep(n1, z); });
            t.st = a.fwd;
        }
        mid_stages<T, false>(t, 1, t.nst - 1);
        last_stage<T, false>(t, sp);
        __syncthreads();
    }
}
template <typename T, int IN, int OUT, bool MASK>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas<T>())
l1d_row_kernel(const __grid_constant__ PassArgs<T> a, const cplx_t<T>* __restrict__ twN, int P, int Q) {
    pdl_enter();
    l1d_row_kernel_body<T, IN, OUT, MASK>(a, twN, P, Q);
}

// ----------------------------------------------------------------- last pass
// Lanes b < TB/2 hold line i0 + b, the others the mirror P - (i0 + b - TB/2);
// the lines 0 and P/2 are their own mirrors (their second lane idles).
template <typename T>
struct L1dLast {
    using C = cplx_t<T>;
    const C* spec;
    int P, k1;           // k1 < 0: idle lane
    __device__ __forceinline__ C one(int x, int) const {
        return k1 >= 0 ? spec[k1 + (size_t)P * x] : mk((T)0, (T)0);
    }
    template <int R> __device__ __forceinline__ void load(C* v, int u, int m, int) const {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = one(u + r * m, 0);
    }
};

template <typename T, class Epi>
__device__ __forceinline__ void scatter1(int M, int k, cplx_t<T> v, Epi& ep) {
    scatter_one<T>(MapEntry{k == 0 ? 0 : (k == M ? 1 : k + 1), M + k, (k == 0 || k == M) ? KIND_VERT : KIND_PLUS, 1}, v, ep);
}

template <typename T, class Epi>
__device__ __forceinline__ void l1d_last_kernel_body(const PassArgs<T>& a, const cplx_t<T>* __restrict__ twN, int P,
                                                     int Q, const Epi& epi) {
    using C = cplx_t<T>;
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FftTile<C> t = make_tile(a, smem_raw);
    const int M = a.g.m1;
    const int lh = a.lay.lg - 1, TH = 1 << lh;   // pairs per tile
    const int npair = P / 2 + 1;
    const int b = threadIdx.x & (2 * TH - 1);
    Epi ep = epi;
    for (int i0 = blockIdx.x << lh; i0 < npair; i0 += gridDim.x << lh) {
        const int ib = i0 + (b & (TH - 1));
        const bool self = ib == 0 || 2 * ib == P;
        L1dLast<T> ld{a.spec, P, ib >= npair ? -1 : (b < TH ? ib : (self ? -1 : P - ib))};
        first_stage<T, false>(t, ld);
        mid_stages<T, false>(t, 1, t.nst);
        for (int w = threadIdx.x; w < Q << lh; w += blockDim.x) {
            const int c = w & (TH - 1), k2 = w >> lh, i = i0 + c;
            if (i >= npair) continue;
            const int k = i + P * k2;
            const C zk = t.buf[t.cur + t.lay.at(k2, c)];
            if (k == 0) {
                scatter1<T>(M, 0, r2c_post(zk, zk, twN[0]), ep);
                scatter1<T>(M, M, mk((T)2 * (zk.x - zk.y), (T)0), ep);
            } else if (i == 0 || 2 * i == P) {
                const C zm = t.buf[t.cur + t.lay.at(i == 0 ? Q - k2 : Q - 1 - k2, c)];
                scatter1<T>(M, k, r2c_post(zk, zm, twN[k]), ep);
            } else {
                const C zm = t.buf[t.cur + t.lay.at(Q - 1 - k2, TH + c)];
                scatter1<T>(M, k, r2c_post(zk, zm, twN[k]), ep);
                scatter1<T>(M, M - k, r2c_post(zm, zk, twN[M - k]), ep);
            }
        }
        __syncthreads();
    }
    ep.finish();
}
template <typename T, class Epi>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas<T>())
l1d_last_kernel(const __grid_constant__ PassArgs<T> a, const cplx_t<T>* __restrict__ twN, int P, int Q, Epi epi) {
    pdl_enter();
    l1d_last_kernel_body<T, Epi>(a, twN, P, Q, epi);
}

// ------------------------------------------------- post-processing of a pair
// R2C post-processing and epilogue of positions k and M-k (0 <= 2k <= M) from
// Z[k] and Z[M-k], which z(k) reads.
template <typename T, class Epi, class Z>
__device__ __forceinline__ void l1d_post_pair(int M, int k, Z&& z, const cplx_t<T>* __restrict__ twN, Epi& ep) {
    using C = cplx_t<T>;
    const C zk = z(k);
    if (k == 0) {
        scatter1<T>(M, 0, r2c_post(zk, zk, twN[0]), ep);
        scatter1<T>(M, M, mk((T)2 * (zk.x - zk.y), (T)0), ep);
    } else if (2 * k == M) {
        scatter1<T>(M, k, r2c_post(zk, zk, twN[k]), ep);
    } else {
        // the operands of both entries of a position before either is stored
        const C zm = z(M - k);
        const C v[2] = {r2c_post(zk, zm, twN[k]), r2c_post(zm, zk, twN[M - k])};
        const int at[2] = {k, M - k};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const typename Epi::Pre pr = ep.pre(at[q] + 1), pi = ep.pre(M + at[q]);
            ep.put(at[q] + 1, SQRT2_D * (double)v[q].x, pr);
            ep.put(M + at[q], SQRT2_D * (double)v[q].y, pi);
        }
    }
}

// Post pass: one thread a pair of positions, Z from the spectrum.  The last pass
// of the plugins' epilogues on long vectors (l1d_last says when).
template <typename T, class Epi>
__global__ void __launch_bounds__(256) l1d_post_kernel(const __grid_constant__ PassArgs<T> a, const cplx_t<T>* __restrict__ twN,
                                                       Epi epi) {
    pdl_enter();
    if (a.skip && *a.skip) return;
    const int M = a.g.m1;
    Epi ep = epi;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; 2 * k <= M; k += gridDim.x * blockDim.x)
        l1d_post_pair<T>(M, k, [&](int x) { return a.spec[x]; }, twN, ep);
    ep.finish();
}

// ------------------------------------------------------- short rows, one launch
// A whole product of a row of up to L1D_ONE_N samples in one CTA: the row plan
// of M from the gather (or the real samples) to the scatter (or the samples),
// with the C2R and R2C steps at its ends and no spectrum in HBM.
template <typename T, int IN, int OUT, bool MASK, typename TS, class Epi>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas<T>())
l1d_one_kernel(const __grid_constant__ PassArgs<T> a, const TS* __restrict__ src, Epi epi) {
    pdl_enter();
    using C = cplx_t<T>;
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FftTile<C> t = make_tile(a, smem_raw);
    const int M = a.g.m1;
    const L1dRow<T, MASK> base{nullptr, a.real_in, a.real_out, a.maskw, nullptr, 0, 1, (T)a.scale, true};
    L1dRowReal<T, MASK> re{base};
    if constexpr (IN == IN_REAL) {
        first_stage<T, false>(t, re);
    } else {
        t.st = a.inv;
        L1dFirst<T, TS> in{src, nullptr, a.tw, M, 1, 0};
        first_stage<T, true>(t, in);
        mid_stages<T, true>(t, 1, t.nst - 1);
        if constexpr (OUT == OUT_REAL) {
            last_stage<T, true>(t, re);
        } else {
            chain_stage<T>(t, [&](int n, int, C z) { return base.keep(n, z); });
            t.st = a.fwd;
        }
    }
    if constexpr (OUT == OUT_SCATTER) {
        mid_stages<T, false>(t, 1, t.nst);
        Epi ep = epi;
        for (int k = threadIdx.x; 2 * k <= M; k += blockDim.x)
            l1d_post_pair<T>(M, k, [&](int x) { return t.buf[t.cur + t.lay.at(x, 0)]; }, a.tw, ep);
        ep.finish();
    }
}

// ---------------------------------------------------------------- launchers
// pass: 0 first, 1 row, 2 last
template <typename T>
PassArgs<T> l1d_args(const FftOperator<T>& op, int pass, double scale, const int* skip) {
    PassArgs<T> a{};
    a.g = op.g;
    a.spec = op.spec;
    a.pl = pass == 1 ? op.planP : op.planQ;
    a.tw = pass == 1 ? op.twP : op.twQ;
    a.Ltab = pass == 1 ? op.l1P : op.l1Q;
    FftOperator<T>::tile_args(pass == 0 ? op.f_cfg : (pass == 1 ? op.p_cfg : op.q_cfg), &a);
    a.maskw = op.maskw;
    a.wpr = op.wpr;
    a.scale = scale;
    a.skip = skip;
    return a;
}

template <typename T, typename TS>
cudaError_t l1d_first(const FftOperator<T>& op, const TS* src, const int* skip, cudaStream_t st) {
    auto k = l1d_first_kernel<T, TS>;
    const PassCfg& c = op.f_cfg;
    const cudaError_t e = smem_optin(k, c.smem);
    if (e != cudaSuccess) return e;
    launch_pdl(pdl_pays(1, op.g.N), k, c.tiles, c.threads, c.smem, st, l1d_args(op, 0, 1.0, skip), src, op.tw1, op.l1P);
    return cudaGetLastError();
}

template <typename T, int IN, int OUT, bool MASK>
cudaError_t l1d_row(const FftOperator<T>& op, double scale, const T* real_in, T* real_out, const int* skip,
                    cudaStream_t st) {
    auto k = l1d_row_kernel<T, IN, OUT, MASK>;
    const PassCfg& c = op.p_cfg;
    const cudaError_t e = smem_optin(k, c.smem);
    if (e != cudaSuccess) return e;
    PassArgs<T> a = l1d_args(op, 1, scale, skip);
    a.real_in = real_in;
    a.real_out = real_out;
    launch_pdl(pdl_pays(1, op.g.N), k, c.tiles, c.threads, c.smem, st, a, op.tw1, op.l1P, op.l1Q);
    return cudaGetLastError();
}

// The last pass.  An epilogue with many operands (the KKT plugins': 4 to 12
// values an entry) meets a tile of two to eight lines badly: every operand is
// read 8 to 32 bytes at a time, a few hundred threads wait for them, and long
// vectors have only tiles of two lines.  From L1D_POST_N samples such an epilogue
// takes a pass of its own, after the lines went through in place.  Measured on
// B200, in the last pass -> in its own, us waited for: condensed product 16384
// 29.4 -> 31.6, 32768 32.9 -> 32.4, 65536 39.2 -> 33.0, 262144 62.8 -> 38.2,
// 777600 102 -> 59; the plugin's 6N product 16384 31.4 -> 32.7, 32768 36.9 ->
// 33.9, 262144 89.5 -> 41.3; 20 CG iterations on 2N vectors 16384 776 -> 780,
// 32768 802 -> 791, 262144 1251 -> 1038.
constexpr long long L1D_POST_N = 1LL << 15;
template <typename T, class Epi>
cudaError_t l1d_last(const FftOperator<T>& op, const Epi& epi, const int* skip, cudaStream_t st) {
    if constexpr (sizeof(typename Epi::Pre) > 2 * sizeof(double)) {
        if (op.g.N >= L1D_POST_N) {
            PassArgs<T> a = l1d_args(op, 0, 1.0, skip);
            a.n_lines = a.sx = op.l1P;
            a.n_outer = 1;
            cudaError_t e = launch_strided<T, false, IN_SPEC, OUT_SPEC>(op.f_cfg, a, (const double*)nullptr,
                                                                       EpiStore<double>{nullptr}, st);
            if (e != cudaSuccess) return e;
            const int blocks = std::min(1024, op.g.m1 / 512 + 1);
            launch_pdl(pdl_pays(1, op.g.N), l1d_post_kernel<T, Epi>, blocks, 256, 0, st, a, op.tw1, epi);
            return cudaGetLastError();
        }
    }
    auto k = l1d_last_kernel<T, Epi>;
    const PassCfg& c = op.q_cfg;
    const cudaError_t e = smem_optin(k, c.smem);
    if (e != cudaSuccess) return e;
    launch_pdl(pdl_pays(1, op.g.N), k, c.tiles, c.threads, c.smem, st, l1d_args(op, 2, 1.0, skip), op.tw1, op.l1P, op.l1Q, epi);
    return cudaGetLastError();
}

// A whole product of a short row (op.l1_one).
template <typename T, int IN, int OUT, bool MASK, typename TS, class Epi>
cudaError_t l1d_one(const FftOperator<T>& op, const TS* src, const Epi& epi, double scale, const T* real_in, T* real_out,
                    const int* skip, cudaStream_t st) {
    auto k = l1d_one_kernel<T, IN, OUT, MASK, TS, Epi>;
    const PassCfg& c = op.row_cfg;
    const cudaError_t e = smem_optin(k, c.smem);
    if (e != cudaSuccess) return e;
    PassArgs<T> a = op.row_args(scale, real_in, real_out);
    a.skip = skip;
    launch_pdl(pdl_pays(1, op.g.N), k, 1, c.threads, c.smem, st, a, src, epi);
    return cudaGetLastError();
}

// compiled once (passes_r*.cu): the kernels of one precision, and the last
// pass's epilogues
#define CSIPM_1D_LIST64(X) X(double, EpiStore<double>, EpiCG<double>)
#define CSIPM_1D_LIST32(X) X(float, EpiCG<float>, EpiStore<float>)
#define CSIPM_PASS_1D_ROW(EXT, T, IN, OUT, MASK)                                                                      \
    EXT template cudaError_t l1d_row<T, IN, OUT, MASK>(const FftOperator<T>&, double, const T*, T*, const int*,        \
                                                       cudaStream_t);
#define CSIPM_PASS_1D_ONE(EXT, T, IN, OUT, MASK, EPI)                                                                 \
    EXT template cudaError_t l1d_one<T, IN, OUT, MASK, T, EPI>(const FftOperator<T>&, const T*, const EPI&, double,    \
                                                               const T*, T*, const int*, cudaStream_t);
#define CSIPM_PASS_1D(EXT, T, EPI1, EPI2)                                                                              \
    CSIPM_PASS_1D_ONE(EXT, T, IN_GATHER, OUT_SCATTER, true, EPI1)                                                      \
    CSIPM_PASS_1D_ONE(EXT, T, IN_GATHER, OUT_SCATTER, false, EPI1)                                                     \
    CSIPM_PASS_1D_ONE(EXT, T, IN_GATHER, OUT_SCATTER, true, EPI2)                                                      \
    CSIPM_PASS_1D_ONE(EXT, T, IN_GATHER, OUT_SCATTER, false, EPI2)                                                     \
    EXT template cudaError_t l1d_first<T, T>(const FftOperator<T>&, const T*, const int*, cudaStream_t);               \
    CSIPM_PASS_1D_ROW(EXT, T, IN_SPEC, OUT_SPEC, true)                                                                 \
    CSIPM_PASS_1D_ROW(EXT, T, IN_SPEC, OUT_SPEC, false)                                                                \
    CSIPM_PASS_1D_ROW(EXT, T, IN_SPEC, OUT_REAL, true)                                                                 \
    CSIPM_PASS_1D_ROW(EXT, T, IN_SPEC, OUT_REAL, false)                                                                \
    CSIPM_PASS_1D_ROW(EXT, T, IN_REAL, OUT_SPEC, false)                                                                \
    EXT template cudaError_t l1d_last<T, EPI1>(const FftOperator<T>&, const EPI1&, const int*, cudaStream_t);          \
    EXT template cudaError_t l1d_last<T, EPI2>(const FftOperator<T>&, const EPI2&, const int*, cudaStream_t);
#ifndef CSIPM_PASSES_HERE
#define CSIPM_X(...) CSIPM_PASS_1D(extern, __VA_ARGS__)
CSIPM_1D_LIST64(CSIPM_X)
CSIPM_1D_LIST32(CSIPM_X)
#undef CSIPM_X
#endif

}  // namespace csipm

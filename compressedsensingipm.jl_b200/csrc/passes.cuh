// The operator's passes with run-time plans (any even size), their tiles and
// launchers, and the operator itself (FftOperator).
//
// They serve every reference-order gather and scatter, the 1D passes, batches,
// and the lines and rows for which the autotuner finds them faster than a
// two-level kernel (fft2.cuh) or for which there is none.  What bounds them is
// instruction issue and shared-memory latency at 512 (FP64) threads per SM,
// then HBM.  Measured on B200 against the former passes (radices up to 8,
// every stage and load through shared memory, run-time index division, primes
// as direct sums), queued one after another in FP64: A'A 310 x 410 x 410 (primes
// 31 and 41) 10.64 -> 1.96 ms, the synthesis and analysis of a 1024^2 image 85 ->
// 46 us, A'A 1D 777600 137 -> 58 us; condensed KKT product at 256^3 1.40 -> 0.63
// ms; a batch of 16 images of sides 128-256 11.7 -> 7.4 ms.
// 80 registers (768 threads per SM) measured 8-21% slower on the 1D and 2D
// passes than 128 (512 threads).
#pragma once
#include "fft_device.cuh"
#include "operator.cuh"
#include "plan.h"

namespace csipm {

// The tile of a pass in dynamic shared memory: one or two buffers, then the
// tables of its prime stages (a barrier follows them; without primes there is none).
template <typename T>
__device__ __forceinline__ FftTile<cplx_t<T>> make_tile(const PassArgs<T>& a, unsigned char* smem) {
    using C = cplx_t<T>;
    FftTile<C> t;
    t.lay = a.lay;
    t.st = a.fwd;
    t.nst = a.pl.nst;
    t.L = a.pl.L;
    t.tw = a.tw;
    t.buf = reinterpret_cast<C*>(smem);
    t.cur = 0;
    t.oth = a.two ? a.span : 0;
    C* cs = t.buf + t.oth + a.span;
    t.cs = cs;
    if (a.primes) {
        prime_tables(a.fwd, a.pl.nst, a.tw, a.Ltab, cs);
        __syncthreads();
    }
    return t;
}

// ------------------------------------------------------------ strided pass
// A tile is TB consecutive dim-1 positions x one full line along the axis;
// each CTA walks tiles t = blockIdx.x, blockIdx.x + gridDim.x, ...
// The loads of a tile are issued by its first stage straight into registers
// and several CTAs share an SM, so there is no staging buffer.
template <typename T, bool INV, int IN, int OUT, typename TS, class Epi>
__device__ __forceinline__ void strided_pass_kernel_body(const PassArgs<T>& a, const TS* __restrict__ src, const Epi& epi) {
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FftTile<cplx_t<T>> t = make_tile(a, smem_raw);
    const int TB = 1 << a.lay.lg;
    const int tiles_x = (a.n_lines + TB - 1) >> a.lay.lg;
    const int ntiles = tiles_x * a.n_outer;
    const int b = threadIdx.x & (TB - 1);
    Epi ep = epi;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int o = tile / tiles_x, ii = ((tile - o * tiles_x) << a.lay.lg) + b;
        const bool live = ii < a.n_lines;
        SpecLine<T> sp{a.spec + ii + (long long)o * a.so, a.sx, live};
        constexpr bool GIN = IN == IN_GATHER || IN == IN_SGATHER;
        constexpr bool SOUT = OUT == OUT_SCATTER || OUT == OUT_SSCATTER;
        if constexpr (GIN) {
            GatherLine<T, TS, IN == IN_SGATHER> gl;
            gl.set(a.g, src, ii, a.jk_mode == 1 ? o : 0, live);
            fft_through<T, INV>(t, gl, sp);
        } else if constexpr (SOUT) {
            ScatterLine<T, Epi, OUT == OUT_SSCATTER> sl;
            sl.set(a.g, &ep, ii, a.jk_mode == 1 ? o : 0, live);
            fft_through<T, INV>(t, sp, sl);
        } else {
            fft_through<T, INV>(t, sp, sp);
        }
        __syncthreads();
    }
    if (OUT == OUT_SCATTER || OUT == OUT_SSCATTER) ep.finish();
}

// Threads per CTA at most, and the CTAs per SM the register allocation must
// allow: a radix-10 butterfly holds 40 (FP64) or 20 (FP32) registers of data and as
// many of twiddles.  FP32 at 64 registers (2 CTAs; 24-72 bytes of stack in the
// strided kernels) against 128 (1 CTA), mixed recoveries on B200, ms: 442x494
// 2.35 / 2.26, 598x758 5.21 / 4.45, 1000x1022 3.66 / 3.50, 94^3 3.61 / 3.52, 100^3
// 2.57 / 2.57, 130^3 6.30 / 6.41, 1D 777600 3.45 / 3.51: the border between them
// lies with the lengths and is not drawn.
constexpr int PASS_THREADS = 512;
template <typename T> constexpr int pass_min_ctas() { return sizeof(T) == 8 ? 1 : 2; }

template <typename T, bool INV, int IN, int OUT, typename TS, class Epi>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas<T>())
strided_pass_kernel(const __grid_constant__ PassArgs<T> a, const TS* __restrict__ src, Epi epi) {
    pdl_enter();
    strided_pass_kernel_body<T, INV, IN, OUT, TS, Epi>(a, src, epi);
}

// ---------------------------------------------------------------- row pass
// a row of the half spectrum staged in shared memory, C2R pre-processed
// (x = 0..M-1)
template <typename T>
struct C2rRow {
    using C = cplx_t<T>;
    const C* p;      // the staged tile
    TileLay lay;
    const C* tw;     // N1-th roots
    int M;
    __device__ __forceinline__ C one(int x, int b) const {
        return c2r_pre(p[lay.at(x, b)], p[lay.at(M - x, b)], tw[x]);
    }
    template <int R> __device__ __forceinline__ void load(C* v, int u, int m, int b) const {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = one(u + r * m, b);
    }
};

// a row of real samples as complex pairs, scaled and (MASK) with the missing
// samples cleared
template <typename T, bool MASK>
struct RealRow {
    using C = cplx_t<T>;
    const T* in;
    T* out;
    const uint32_t* mask;    // of this row
    T sc;
    bool live;
    __device__ __forceinline__ C keep(int n, C y) const {
        y.x *= sc;
        y.y *= sc;
        if (MASK && live) {
            const uint32_t w = mask[n >> 4];
            const int sh = (2 * n) & 31;
            if (!((w >> sh) & 1u)) y.x = (T)0;
            if (!((w >> (sh + 1)) & 1u)) y.y = (T)0;
        }
        return y;
    }
    __device__ __forceinline__ C one(int n, int) const {
        return live ? keep(n, *reinterpret_cast<const C*>(in + 2 * (size_t)n)) : mk((T)0, (T)0);
    }
    __device__ __forceinline__ void one(int n, int, C v) const {
        if (live) *reinterpret_cast<C*>(out + 2 * (size_t)n) = keep(n, v);
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

// Last inverse stage, scale + mask, first forward stage: with the forward
// plan the inverse one reversed, the outputs x = u + r*M/R of the one are the
// inputs of the other, so the real samples never leave the registers.
// keep(n, b, z) scales and masks.  The tile is in t.cur before and after; ends
// with a barrier.
template <typename T, class Keep>
__device__ __forceinline__ void chain_stage(FftTile<cplx_t<T>>& t, Keep&& keep) {
    using C = cplx_t<T>;
    const FftStage s = t.st[t.nst - 1];
    const TileLay lay = t.lay;
    const int n = s.m << lay.lg, mask = (1 << lay.lg) - 1;
    for (int w = threadIdx.x; w < n; w += blockDim.x) {
        const int b = w & mask, u = w >> lay.lg;
        switch (s.R) {
#define CSIPM_CHAIN(RR)                                                                   \
            case RR: {                                                                    \
                C v[RR];                                                                  \
                bfly_load<T, RR, true>(v, t.buf + t.cur, lay, s, t.tw, u, u, b);          \
                _Pragma("unroll") for (int r = 0; r < RR; ++r) v[r] = keep(u + r * s.m, b, v[r]); \
                Dft<RR, false, T>::run(v);                                                \
                bfly_put<T, RR>(v, t.buf + t.oth, lay, u * RR, 1, b);                     \
            } break;
            CSIPM_RADICES(CSIPM_CHAIN)
#undef CSIPM_CHAIN
        }   // row plans start with a register radix (make_row_plan)
    }
    t.swap();
    __syncthreads();
}

// Rows along dim 1 (rows = (j, k) pairs), RB a tile, each M+1 half-spectrum
// values.  SPEC -> SPEC: C2R, inverse, scale + mask, forward, R2C; the
// inverse runs the plan's stages reversed, the forward in order.
template <typename T, int IN, int OUT, bool MASK>
__device__ __forceinline__ void row_pass_kernel_body(const PassArgs<T>& a) {
    using C = cplx_t<T>;
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FftTile<C> t = make_tile(a, smem_raw);
    const int M = a.g.m1, RB = 1 << a.lay.lg;
    const int ntiles = (a.nrows + RB - 1) >> a.lay.lg;
    const unsigned mag = 0xffffffffu / (unsigned)(M + 1) + 1u;
    const int b = threadIdx.x & (RB - 1);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int r0 = tile << a.lay.lg, row = r0 + b;
        const bool live = row < a.nrows;
        RealRow<T, MASK> rr{IN == IN_REAL ? a.real_in + (size_t)row * a.g.n1 : nullptr,
                            OUT == OUT_REAL ? a.real_out + (size_t)row * a.g.n1 : nullptr,
                            MASK ? a.maskw + (size_t)row * a.wpr : nullptr, (T)a.scale, live};
        const int total = (M + 1) << a.lay.lg;
        if (IN == IN_REAL) {
            first_stage<T, false>(t, rr);
        } else {
            // whole rows, coalesced, into the second buffer; C2R and the first
            // inverse stage read them there (read in place from global memory,
            // x and M - x of eight rows at a time thrashed the L1: 3x the time)
            C* raw = t.buf + t.oth;
#pragma unroll 4
            for (int e = threadIdx.x; e < total; e += blockDim.x) {
                const int rb = quot(e, M + 1, mag), k = e - rb * (M + 1);
                if (r0 + rb < a.nrows) raw[t.lay.at(k, rb)] = a.spec[(size_t)(r0 + rb) * a.g.ld1 + k];
            }
            __syncthreads();
            C2rRow<T> cr{raw, t.lay, a.tw, M};
            t.st = a.inv;
            first_stage<T, true>(t, cr);
            mid_stages<T, true>(t, 1, t.nst - 1);
            if (OUT == OUT_REAL) {
                last_stage<T, true>(t, rr);
                __syncthreads();
                continue;
            }
            chain_stage<T>(t, [&](int n, int, C z) { return rr.keep(n, z); });
            t.st = a.fwd;
        }
        mid_stages<T, false>(t, 1, t.nst);
        // R2C post-processing of the natural-order transform, whole rows coalesced
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            const int rb = quot(e, M + 1, mag), k = e - rb * (M + 1);
            if (r0 + rb >= a.nrows) break;
            C v;
            if (k == 0 || k == M) {
                const C z0 = t.buf[t.cur + t.lay.at(0, rb)];
                v = k == 0 ? r2c_post(z0, z0, a.tw[0]) : mk((T)2 * (z0.x - z0.y), (T)0);
            } else {
                v = r2c_post(t.buf[t.cur + t.lay.at(k, rb)], t.buf[t.cur + t.lay.at(M - k, rb)], a.tw[k]);
            }
            a.spec[(size_t)(r0 + rb) * a.g.ld1 + k] = v;
        }
        __syncthreads();
    }
}
template <typename T, int IN, int OUT, bool MASK>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas<T>()) row_pass_kernel(const __grid_constant__ PassArgs<T> a) {
    pdl_enter();
    row_pass_kernel_body<T, IN, OUT, MASK>(a);
}

// In-place row pass for rows whose two tile buffers do not fit on chip (2D
// with N1 above about 12000): one row a CTA, register-staged stages.
template <typename T, int IN, int OUT, bool MASK>
__global__ void __launch_bounds__(1024) row_pass_ip_kernel(PassArgs<T> a) {
    // no early placement of the next pass: its tiles take the L1 that this
    // kernel's spills live in (A'A on 13122 x 4 samples, queued: 200 us, so 101)
    pdl_wait();
    using C = cplx_t<T>;
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* buf = reinterpret_cast<C*>(smem_raw);
    const int M = a.g.m1;
    // One row a CTA.  The layout comes in at run time: with RB = TBP = 1 known to
    // the compiler it unrolled the engine's stages into twice the spills at the
    // 64 registers that 1024 threads leave (5888 bytes for 3392): A'A on
    // 12804 x 4 samples (rows of 2 3 11 97) 1310 us, so 720.
    const int RB = 1 << a.lay.lg, TBP = a.lay.tbp;
    __shared__ int s_rad[FFT_MAX_STAGES];
    load_radices(a.pl, s_rad);
    const C* tw = a.tw;
    const int r0 = blockIdx.x * RB;
    const int nr = min(RB, a.nrows - r0);
    const C zero = mk((T)0, (T)0);

    // ---- load
    if (IN == IN_REAL) {
        for (int e = threadIdx.x; e < M * RB; e += blockDim.x) {
            const int b = e / M, n = e % M;
            C val = zero;
            if (b < nr) val = *reinterpret_cast<const C*>(a.real_in + (size_t)(r0 + b) * a.g.n1 + 2 * n);
            buf[n * TBP + b] = val;
        }
    } else {
        for (int e = threadIdx.x; e < (M + 1) * RB; e += blockDim.x) {
            const int b = e / (M + 1), n = e % (M + 1);
            C val = zero;
            if (b < nr) {
                val = a.spec[(size_t)(r0 + b) * a.g.ld1 + n];
            }
            buf[n * TBP + b] = val;
        }
    }
    __syncthreads();
    const int half = M / 2;
    if (IN != IN_REAL) {
        for (int e = threadIdx.x; e < (half + 1) * RB; e += blockDim.x) {
            const int b = e % RB, k = e / RB;
            if (k == 0) {
                const C x0 = buf[b], xm = buf[M * TBP + b];
                buf[b] = c2r_pre(x0, xm, tw[0]);
            } else if (2 * k == M) {
                const C xk = buf[k * TBP + b];
                buf[k * TBP + b] = c2r_pre(xk, xk, tw[k]);
            } else {
                const C xk = buf[k * TBP + b], xm = buf[(M - k) * TBP + b];
                buf[k * TBP + b] = c2r_pre(xk, xm, tw[k]);
                buf[(M - k) * TBP + b] = c2r_pre(xm, xk, tw[M - k]);
            }
        }
        __syncthreads();
        fft_lines_ip<T, true>(buf, s_rad, a.pl.nst, M, RB, TBP, tw, a.Ltab);
    }
    // ---- middle: scale and mask the real samples (x[2n], x[2n+1]) = (Re z[n], Im z[n])
    const T sc = (T)a.scale;
    for (int e = threadIdx.x; e < M * RB; e += blockDim.x) {
        const int b = e / M, n = e % M;
        if (b < nr) {
            C y = buf[n * TBP + b];
            y.x *= sc;
            y.y *= sc;
            if (MASK) {
                const uint32_t w = a.maskw[(size_t)(r0 + b) * a.wpr + (n >> 4)];
                const int sh = (2 * n) & 31;
                if (!((w >> sh) & 1u)) y.x = (T)0;
                if (!((w >> (sh + 1)) & 1u)) y.y = (T)0;
            }
            if (OUT == OUT_REAL) *reinterpret_cast<C*>(a.real_out + (size_t)(r0 + b) * a.g.n1 + 2 * n) = y;
            else buf[n * TBP + b] = y;
        }
    }
    if (OUT == OUT_REAL) return;
    __syncthreads();
    fft_lines_ip<T, false>(buf, s_rad, a.pl.nst, M, RB, TBP, tw, a.Ltab);
    for (int e = threadIdx.x; e < (half + 1) * RB; e += blockDim.x) {
        const int b = e % RB, k = e / RB;
        if (k == 0) {
            const C z0 = buf[b];
            buf[b] = r2c_post(z0, z0, tw[0]);
            buf[M * TBP + b] = mk((T)2 * (z0.x - z0.y), (T)0);
        } else if (2 * k == M) {
            const C zk = buf[k * TBP + b];
            buf[k * TBP + b] = r2c_post(zk, zk, tw[k]);
        } else {
            const C zk = buf[k * TBP + b], zm = buf[(M - k) * TBP + b];
            buf[k * TBP + b] = r2c_post(zk, zm, tw[k]);
            buf[(M - k) * TBP + b] = r2c_post(zm, zk, tw[M - k]);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < (M + 1) * RB; e += blockDim.x) {
        const int b = e / (M + 1), n = e % (M + 1);
        if (b < nr) a.spec[(size_t)(r0 + b) * a.g.ld1 + n] = buf[n * TBP + b];
    }
}

// ------------------------------------------------------------ host side
struct PassCfg {
    int tb = 0;          // lines per CTA (strided) / rows per CTA (row pass), a power of two
    int threads = 0;
    size_t smem = 0;
    int pp = 1;          // 1: run-time-plan pass (TileLay fields below); 0: in-place row kernel
    TileLay lay{0, 1};
    int span = 0, two = 0, primes = 0;
    FftStage fwd[PASS_STAGES], inv[PASS_STAGES];
    int tiles = 0;       // number of tiles of the pass
    dim3 grid;           // one CTA per tile (persistent grids are capped at launch)
};

// What a pass keeps in shared memory besides the stages' exchange.
enum PassKind { PASS_LINES, PASS_ROWS, PASS_PAIRS };   // strided; rows of the half spectrum; 1D mirrored lines

// Tile layout, threads and shared memory of a run-time-plan pass over `lines`
// (a power of two) lines per CTA, `n` of them in all.  threads: 0 to choose,
// else given.  csize: bytes of a complex value.
constexpr size_t PASS_SMEM = 200 * 1024;   // dynamic shared memory of a CTA at most (B200: 227 KB with the static part)
inline void lay_pass(const FftPlanDev& pl, int Ltab, int lines, int n, PassKind kind, int threads, size_t csize,
                     PassCfg* c) {
    c->tb = lines;
    c->pp = 1;
    // Refused before its stages are written: a line longer than a tile (16 bits
    // may not hold it) and a plan of more stages than the arguments carry (the
    // in-place rows' plans, radices up to 8, have up to 8 for lengths of a tile).
    if (pl.L * csize > PASS_SMEM || pl.nst > PASS_STAGES) {
        c->smem = ~(size_t)0;
        return;
    }
    TileLay l;
    l.lg = 0;
    while ((1 << l.lg) < lines) ++l.lg;
    // rows are read and written along the row, so their pitch is odd; 1D pairs
    // are read like strided lines (padded by one they met 2-way bank conflicts:
    // last pass of 777600, 27.5 -> 26.0 us)
    l.tbp = kind == PASS_ROWS && lines > 1 ? lines + 1 : lines;
    c->lay = l;
    c->span = (kind == PASS_ROWS ? pl.L + 1 : pl.L) * l.tbp;   // a staged row has M+1 values
    c->tiles = (n + lines - 1) / lines;
    const int table = prime_table_size(pl);
    c->primes = table > 0;
    fill_stages(pl, Ltab, false, c->fwd);
    fill_stages(pl, Ltab, true, c->inv);
    // a second buffer where a stage goes from shared memory to shared memory
    // (rows and 1D pairs: nearly always; a line of two register stages never)
    c->two = kind == PASS_ROWS || pl.nst > 2 || (kind == PASS_PAIRS && pl.nst > 1);
    for (int s = 0; s + 1 < pl.nst || (s < pl.nst && kind != PASS_LINES); ++s)
        if (!reg_radix(pl.rad[s])) c->two = 1;
    c->smem = ((size_t)c->span * (1 + c->two) + table) * csize;
    if (threads == 0) {
        // the threads that keep the most lanes of an SM busy: resident threads
        // (registers, shared memory, and the
        // tiles an SM gets) times the share of them the stages occupy
        const int regs = PASS_THREADS * (csize >= 16 ? pass_min_ctas<double>() : pass_min_ctas<float>());
        const int per_sm = (c->tiles + 147) / 148;
        double best = -1.0;
        for (int t = std::max(64, lines); t <= PASS_THREADS; t += 32) {
            double need = 0, spent = 0;
            for (int s = 0; s < pl.nst; ++s) {
                const double w = reg_radix(pl.rad[s]) ? pl.rad[s] + 4 : PRIME_K * (pl.rad[s] / 2);
                const int it = stage_items(pl.rad[s], pl.L, l.lg);
                need += it * w;
                spent += (double)((it + t - 1) / t) * t * w;
            }
            const int ctas = std::max(1, std::min({regs / t, (int)(220 * 1024 / (c->smem + 1024)), per_sm}));
            const double score = need / spent * std::min(ctas * t, regs);
            if (score > best * 1.001) {
                best = score;
                threads = t;
            }
        }
    }
    c->threads = threads;
}

// ------------------------------------------------------------ mask
// Observed-sample mask, one bit per real sample, rows of N1 bits padded to
// 32-bit words: every in-row bit set, padding clear; then the missing
// samples' bits cleared (duplicates are harmless).
static __global__ void mask_init_kernel(size_t words, int wpr, int n1, uint32_t* __restrict__ w) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < words; t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t % wpr);
        const int nb = min(32, n1 - 32 * c);
        w[t] = nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u);
    }
}

static __global__ void mask_clear_kernel(const int64_t* __restrict__ idx, int64_t n, int n1, int wpr,
                                         uint32_t* __restrict__ w) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = idx[t];
        const int64_t r = v / n1;
        const int i = (int)(v - r * n1);
        atomicAnd(&w[r * wpr + (i >> 5)], ~(1u << (i & 31)));
    }
}

inline unsigned mask_blocks(long long n) { return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 4096)); }

// 1D (long1d.cuh): a row of M complex values runs as M = P*Q over many CTAs.
constexpr int L1D_MIN_M = 2048;     // above: rows whose split must have Q >= 2
constexpr int L1D_MAX_P = 4096;     // row length of the four-step row kernel
constexpr int L1D_MAX_Q = 768;      // line length of the first and last passes

// Rows of up to this many samples run their products in one launch of one CTA
// (l1d_one_kernel): three launches cost more than the idle SMs.  FP64 on B200,
// three launches -> one, us waited for: A'A 64 18.2 -> 13.0, 500 23.7 -> 14.3,
// 2048 23.2 -> 17.2, 4096 25.5 -> 21.4, 6000 26.6 -> 24.6, 8192 27.0 -> 32.5; the
// plugin's 6N product 500 25.6 -> 17.5, 4096 28.3 -> 28.0, 6000 30.1 -> 33.3;
// recovery 500 1034 -> 771, 4096 1428 -> 1289, 8192 1151 -> 1315.
constexpr int L1D_ONE_N = 4096;

// M = P*Q with Q the largest divisor of M not above sqrt(M) (nor L1D_MAX_Q),
// P = M/Q; false when P exceeds L1D_MAX_P.  Q = 1 (M prime) up to L1D_MIN_M.
inline bool l1d_split(int M, int* P, int* Q) {
    int best = M <= L1D_MIN_M ? 1 : 0;
    for (int q = 2; (long long)q * q <= M && q <= L1D_MAX_Q; ++q)
        if (M % q == 0) best = q;
    if (!best || M / best > L1D_MAX_P) return false;
    *Q = best;
    *P = M / best;
    return true;
}

// W^e = exp(-2 pi i e / L), built on the device from the first octant with
// the exact symmetries of the roots of unity (sign changes and swaps only):
//   e in (L/2, L):    W^e = conj W^(L-e)                       (conjugation)
//   e in [L/4, L/2]:  W^e = -i W^(e-L/4)                       (quarter turn, 4 | L)
//   e in (L/8, L/4):  W^e = (-Im W^(L/4-e), -Re W^(L/4-e))     (reflection, 8 | L)
// What remains is computed directly as sincospi(2e/L) (2e/L is one rounding
// of an exact ratio; for 8 | L it lies in [0, 1/4]).  The table is symmetric
// bit for bit, as the real-input passes assume.
__device__ __forceinline__ double2 root_of_unity(long long e, long long L) {
    bool conj = false, rot = false, refl = false;
    if (2 * e > L) { e = L - e; conj = true; }
    if (L % 4 == 0 && 4 * e >= L) { e -= L / 4; rot = true; }
    if (L % 8 == 0 && 8 * e > L && 4 * e < L) { e = L / 4 - e; refl = true; }
    double sn, cs;
    sincospi((double)(2 * e) / (double)L, &sn, &cs);
    double re = cs, im = -sn;
    if (refl) { const double r2 = -im; im = -re; re = r2; }
    if (rot) { const double r2 = im; im = -re; re = r2; }
    if (conj) im = -im;
    return make_double2(re, im);
}

__device__ __forceinline__ void put_root(double2* o, double2 w) { *o = w; }
__device__ __forceinline__ void put_root(float2* o, double2 w) { *o = make_float2((float)w.x, (float)w.y); }

template <typename C>
__global__ void twiddle_kernel(int L, C* __restrict__ out) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < L; e += gridDim.x * blockDim.x)
        put_root(out + e, root_of_unity(e, L));
}

template <typename C>
inline cudaError_t launch_twiddles(int L, C* dst, cudaStream_t st) {
    const int blocks = std::max(1, std::min((L + 255) / 256, 1024));
    twiddle_kernel<C><<<blocks, 256, 0, st>>>(L, dst);
    return cudaGetLastError();
}

template <typename T>
class FftOperator {
public:
    using C = cplx_t<T>;
    Geom g{};
    cudaStream_t stream = nullptr;
    C* spec = nullptr;              // (m1+1) x n2 x n3, pitch ld1
    uint32_t* maskw = nullptr;      // nullptr: no missing samples
    int wpr = 0;
    FftPlanDev plan1{}, plan2{}, plan3{};
    C* tw1 = nullptr;               // n1-th roots (row pass)
    C* tw2 = nullptr;
    C* tw3 = nullptr;
    PassCfg row_cfg, s2_cfg, s3_cfg;
    // two-level register passes (fft2.cuh): factor pairs, 0 when not used
    int s2_A = 0, s2_B = 0, s3_A = 0, s3_B = 0, r_A = 0, r_B = 0;
    size_t bytes = 0;
    bool owns = true;               // false: buffers belong to someone else; release() frees nothing
    // 1D: M = l1P * l1Q
    int l1P = 0, l1Q = 0;
    FftPlanDev planP{}, planQ{};
    C* twP = nullptr;
    C* twQ = nullptr;
    PassCfg f_cfg, p_cfg, q_cfg;    // first lines, rows, last lines (pairs)
    bool l1_one = false;            // a short row: products in one launch (plan1, row_cfg)

    // stream-ordered allocations from this pool on `stream` when set (the
    // handle's), else plain cudaMalloc/cudaFree
    cudaMemPool_t pool = nullptr;

    ~FftOperator() { release(); }

    template <typename P>
    cudaError_t dalloc(P** p, size_t count) {
        void* q = nullptr;
        const cudaError_t e = pool ? cudaMallocFromPoolAsync(&q, sizeof(P) * count, pool, stream)
                                   : cudaMalloc(&q, sizeof(P) * count);
        *p = reinterpret_cast<P*>(q);
        return e;
    }
    void dfree(void* p) {
        if (!p) return;
        if (pool) cudaFreeAsync(p, stream);
        else cudaFree(p);
    }

    void release() {
        if (!owns) return;
        dfree(spec); spec = nullptr;
        dfree(maskw); maskw = nullptr;
        dfree(tw1); tw1 = nullptr;
        dfree(tw2); tw2 = nullptr;
        dfree(tw3); tw3 = nullptr;
        dfree(twP); twP = nullptr;
        dfree(twQ); twQ = nullptr;
    }

    // twiddle table of L entries, written on the device (stream-ordered: no
    // host computation, no copy)
    bool upload_table(int L, C** dst, std::string* err) {
        if (dalloc(dst, L) != cudaSuccess) { *err = "out of device memory (twiddles)"; return false; }
        if (launch_twiddles(L, *dst, stream) != cudaSuccess) { *err = "twiddle kernel launch failed"; return false; }
        return true;
    }

    static size_t smem_limit() { return PASS_SMEM; }

    static constexpr int FULL_TB = sizeof(T) == 8 ? 8 : 16;   // lines of a 128-byte access

    // Strided configuration with tb lines per CTA; false when the tile is too large.
    static bool strided_cfg(const FftPlanDev& pl, int n_lines, int n_outer, int tb, size_t most, PassCfg* cfg) {
        const int tiles = ((n_lines + tb - 1) / tb) * n_outer;
        lay_pass(pl, pl.L, tb, tiles * tb, PASS_LINES, 0, sizeof(C), cfg);
        if (cfg->smem > most) return false;
        cfg->grid = dim3(cfg->tiles, 1, 1);
        return true;
    }
    // Row configuration with rb rows per CTA.
    static bool rows_cfg(const FftPlanDev& pl, int nrows, int rb, size_t most, PassCfg* cfg) {
        if (rb > 1 && rb > nrows) return false;
        lay_pass(pl, 2 * pl.L, rb, nrows, PASS_ROWS, 0, sizeof(C), cfg);   // N1-th roots
        if (cfg->smem > most) return false;
        cfg->grid = dim3(cfg->tiles, 1, 1);
        return true;
    }

    // Strided passes: 128-byte accesses while a tile takes 72 KB at most (three
    // CTAs per SM) and the pass has a tile for every SM, narrower ones else.
    bool choose_strided(const FftPlanDev& pl, int n_lines, int n_outer, PassCfg* cfg, std::string* err) {
        if (6 * (size_t)pl.L * sizeof(C) > smem_limit()) {
            *err = "transform length too large for the on-chip strided pass";
            return false;
        }
        for (int tb = FULL_TB; tb >= 2; tb /= 2) {
            const bool last = tb == 2;
            if (strided_cfg(pl, n_lines, n_outer, tb, last ? smem_limit() : 72 * 1024, cfg) &&
                (last || cfg->tiles >= 148))
                return true;
        }
        *err = "transform length too large for the on-chip strided pass";
        return false;
    }

    // Row passes: rows per CTA as for the strided lines; the in-place kernel
    // for rows whose tile does not fit.
    bool choose_row(int nrows, PassCfg* cfg, std::string* err) {
        const int M = g.m1;
        for (int rb = 8; rb >= 1; rb /= 2) {
            if (rows_cfg(plan1, nrows, rb, rb == 1 ? smem_limit() : 72 * 1024, cfg) && (rb == 1 || cfg->tiles >= 148))
                return true;
        }
        // in place: the register-staged engine takes radices <= 8
        if (!make_fft_plan_ip(M, &plan1, err)) return false;
        const size_t o1 = (size_t)(M + 1) * sizeof(C);
        int thr = std::max(64, std::min(1024, ((M + 7) / 8 + 31) / 32 * 32));
        while (thr < 1024 && !plan_fits(plan1, 1, thr)) thr += 32;
        if (o1 > smem_limit() || !plan_fits(plan1, 1, thr)) {
            *err = "dimension 1 too large for the on-chip row pass";
            return false;
        }
        cfg->pp = 0;
        cfg->tb = 1;
        cfg->lay = TileLay{0, 1};
        cfg->threads = thr;
        cfg->smem = o1;
        cfg->tiles = nrows;
        cfg->grid = dim3(nrows, 1, 1);
        return true;
    }

    // 1D tiles: a long row has only P and Q lines (a few hundred to a few
    // thousand), so they are as wide as still gives about one CTA per SM.
    bool choose_1d(std::string* err) {
        auto widest = [&](const FftPlanDev& pl, int n, PassKind kind, int least, PassCfg* c) {
            for (int w = 8; w >= least; w /= 2) {
                lay_pass(pl, pl.L, w, n, kind, 0, sizeof(C), c);
                if (c->smem <= smem_limit() && (c->tiles >= 148 || w <= 2)) return true;
            }
            return false;
        };
        const bool ok = widest(planQ, l1P, PASS_LINES, 2, &f_cfg) && widest(planP, l1Q, PASS_PAIRS, 1, &p_cfg) &&
                        widest(planQ, 2 * (l1P / 2 + 1), PASS_PAIRS, 2, &q_cfg);
        if (!ok) *err = "1D length too large for the on-chip passes";
        return ok;
    }

    // Use the two-level register passes where the line length factors into an
    // instantiated pair (FP64, 2D/3D).
    void choose_two_level();

    // plans and tiles of every pass
    bool make_plans(std::string* err) {
        if (g.dim == 1) {
            if (!l1d_split(g.m1, &l1P, &l1Q)) {
                *err = "1D length has no split M = P*Q with P <= 4096, Q <= 768";
                return false;
            }
            plan1 = FftPlanDev{};
            std::string none;
            l1_one = g.n1 <= L1D_ONE_N && make_row_plan(g.m1, &plan1, &none) && rows_cfg(plan1, 1, 1, PASS_SMEM, &row_cfg);
            return make_row_plan(l1P, &planP, err) && make_fft_plan(l1Q, &planQ, err) && choose_1d(err);
        }
        if (!make_row_plan(g.m1, &plan1, err) || !choose_row(g.n2 * g.n3, &row_cfg, err)) return false;
        if (!make_fft_plan(g.n2, &plan2, err) ||
            !choose_strided(plan2, g.m1 + 1, g.dim == 3 ? g.n3 : 1, &s2_cfg, err))
            return false;
        return g.dim < 3 || (make_fft_plan(g.n3, &plan3, err) && choose_strided(plan3, g.m1 + 1, g.n2, &s3_cfg, err));
    }

    // dev_missing: n_missing 0-based linear indices of missing samples in
    // device memory (validated by the caller), or n_missing == 0 for no mask
    bool init(const Geom& geom, const int64_t* dev_missing, int64_t n_missing, cudaStream_t st, std::string* err) {
        g = geom;
        stream = st;
        const int nrows = g.n2 * g.n3;
        if (!make_plans(err)) return false;
        if (g.dim == 1 && (!upload_table(l1P, &twP, err) || !upload_table(l1Q, &twQ, err))) return false;
        choose_two_level();
        if (!upload_table(g.n1, &tw1, err)) return false;
        if (g.dim >= 2 && !upload_table(g.n2, &tw2, err)) return false;
        if (g.dim >= 3 && !upload_table(g.n3, &tw3, err)) return false;
        const size_t spec_elems = (size_t)g.ld1 * g.n2 * g.n3;
        if (dalloc(&spec, spec_elems) != cudaSuccess) { *err = "out of device memory (spectrum)"; return false; }
        bytes += sizeof(C) * spec_elems;
        if (n_missing > 0) {
            wpr = (g.n1 + 31) / 32;
            const size_t words = (size_t)wpr * nrows;
            if (dalloc(&maskw, words) != cudaSuccess) { *err = "out of device memory (mask)"; return false; }
            bytes += sizeof(uint32_t) * words;
            mask_init_kernel<<<mask_blocks(words), 256, 0, stream>>>(words, wpr, g.n1, maskw);
            mask_clear_kernel<<<mask_blocks(n_missing), 256, 0, stream>>>(dev_missing, n_missing, g.n1, wpr, maskw);
            if (cudaGetLastError() != cudaSuccess) { *err = "mask construction failed"; return false; }
        }
        return true;
    }

    static void tile_args(const PassCfg& c, PassArgs<T>* a) {
        a->lay = c.lay;
        a->span = c.span;
        a->two = c.two;
        a->primes = c.primes;
        std::copy(c.fwd, c.fwd + PASS_STAGES, a->fwd);
        std::copy(c.inv, c.inv + PASS_STAGES, a->inv);
    }
    PassArgs<T> row_args(double scale, const T* real_in, T* real_out) const {
        PassArgs<T> a{};
        a.g = g; a.pl = plan1; a.tw = tw1; a.Ltab = g.n1;
        a.spec = spec; a.nrows = g.n2 * g.n3;
        tile_args(row_cfg, &a);
        a.maskw = maskw; a.wpr = wpr; a.scale = scale; a.real_in = real_in; a.real_out = real_out;
        return a;
    }
    // axis 2 or 3
    PassArgs<T> strided_args(int axis) const {
        PassArgs<T> a{};
        a.g = g;
        a.spec = spec;
        a.n_lines = g.m1 + 1;
        if (axis == 3) {
            a.pl = plan3; a.tw = tw3; a.Ltab = g.n3;
            tile_args(s3_cfg, &a);
            a.so = g.ld1; a.sx = (long long)g.ld1 * g.n2; a.jk_mode = 0; a.n_outer = g.n2;
        } else {
            a.pl = plan2; a.tw = tw2; a.Ltab = g.n2;
            tile_args(s2_cfg, &a);
            a.so = (long long)g.ld1 * g.n2; a.sx = g.ld1; a.jk_mode = g.dim == 3 ? 1 : 2; a.n_outer = g.dim == 3 ? g.n3 : 1;
        }
        return a;
    }
};

// CTAs of a run-time-plan pass: one per tile up to WAVES waves of resident
// CTAs (later tiles are walked by the same CTAs).
inline int pass_grid(const void* fn, const PassCfg& c) {
    constexpr int WAVES = 16;
    return std::min(c.tiles, WAVES * persistent_grid(fn, c.threads, c.smem, c.tiles));
}

template <typename T, bool INV, int IN, int OUT, typename TS, class Epi>
cudaError_t launch_strided(const PassCfg& c, const PassArgs<T>& a, const TS* src, const Epi& epi, cudaStream_t st) {
    auto k = strided_pass_kernel<T, INV, IN, OUT, TS, Epi>;
    const cudaError_t e = smem_optin(k, c.smem);
    if (e != cudaSuccess) return e;
    launch_pdl(pdl_pays(a.g.dim, a.g.N), k, pass_grid((const void*)k, c), c.threads, c.smem, st, a, src, epi);
    return cudaGetLastError();
}

template <typename T, int IN, int OUT, bool MASK>
cudaError_t launch_row(const PassCfg& c, const PassArgs<T>& a, cudaStream_t st) {
    if (c.pp) {
        auto k = row_pass_kernel<T, IN, OUT, MASK>;
        const cudaError_t e = smem_optin(k, c.smem);
        if (e != cudaSuccess) return e;
        launch_pdl(pdl_pays(a.g.dim, a.g.N), k, pass_grid((const void*)k, c), c.threads, c.smem, st, a);
    } else {
        auto k = row_pass_ip_kernel<T, IN, OUT, MASK>;
        const cudaError_t e = smem_optin(k, c.smem);
        if (e != cudaSuccess) return e;
        launch_pdl(pdl_pays(a.g.dim, a.g.N), k, c.grid, c.threads, c.smem, st, a);
    }
    return cudaGetLastError();
}

// The launches compiled once (passes_*.cu): (T, INV, IN, OUT, TS, Epi) and
// (T, IN, OUT, MASK); the plugins' epilogues are compiled where they are used.
#define CSIPM_STRIDED_LIST64(X)                                       \
    X(double, true, IN_GATHER, OUT_SPEC, double, EpiStore<double>)    \
    X(double, true, IN_SPEC, OUT_SPEC, double, EpiStore<double>)      \
    X(double, false, IN_SPEC, OUT_SPEC, double, EpiStore<double>)     \
    X(double, false, IN_SPEC, OUT_SCATTER, double, EpiStore<double>)  \
    X(double, false, IN_SPEC, OUT_SCATTER, double, EpiCG<double>)     \
    X(double, true, IN_SGATHER, OUT_SPEC, double, EpiStore<double>)   \
    X(double, false, IN_SPEC, OUT_SSCATTER, double, EpiStore<double>) \
    X(double, false, IN_SPEC, OUT_SSCATTER, double, EpiCG<double>)
#define CSIPM_STRIDED_LIST32(X)                                      \
    X(float, true, IN_GATHER, OUT_SPEC, float, EpiStore<double>)     \
    X(float, true, IN_SGATHER, OUT_SPEC, float, EpiStore<double>)    \
    X(float, true, IN_SPEC, OUT_SPEC, double, EpiStore<double>)      \
    X(float, false, IN_SPEC, OUT_SPEC, double, EpiStore<double>)     \
    X(float, false, IN_SPEC, OUT_SCATTER, double, EpiCG<float>)      \
    X(float, false, IN_SPEC, OUT_SSCATTER, double, EpiCG<float>)
#define CSIPM_ROW_LIST64(X)              \
    X(double, IN_SPEC, OUT_SPEC, true)   \
    X(double, IN_SPEC, OUT_SPEC, false)  \
    X(double, IN_SPEC, OUT_REAL, true)   \
    X(double, IN_SPEC, OUT_REAL, false)  \
    X(double, IN_REAL, OUT_SPEC, false)
#define CSIPM_ROW_LIST32(X)              \
    X(float, IN_SPEC, OUT_SPEC, true)    \
    X(float, IN_SPEC, OUT_SPEC, false)
#define CSIPM_PASS_S(EXT, T, INV, IN, OUT, TS, EPI)                                                          \
    EXT template cudaError_t launch_strided<T, INV, IN, OUT, TS, EPI>(const PassCfg&, const PassArgs<T>&,    \
                                                                      const TS*, const EPI&, cudaStream_t);
#define CSIPM_PASS_R(EXT, T, IN, OUT, MASK) \
    EXT template cudaError_t launch_row<T, IN, OUT, MASK>(const PassCfg&, const PassArgs<T>&, cudaStream_t);
#ifndef CSIPM_PASSES_HERE
#define CSIPM_X(...) CSIPM_PASS_S(extern, __VA_ARGS__)
CSIPM_STRIDED_LIST64(CSIPM_X)
CSIPM_STRIDED_LIST32(CSIPM_X)
#undef CSIPM_X
#define CSIPM_X(...) CSIPM_PASS_R(extern, __VA_ARGS__)
CSIPM_ROW_LIST64(CSIPM_X)
CSIPM_ROW_LIST32(CSIPM_X)
#undef CSIPM_X
#endif

}  // namespace csipm

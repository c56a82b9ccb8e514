// Mixed-radix Stockham FFT over a tile of TB interleaved lines of length L,
// with the radices of a run-time plan.
//
// Stage s with radix R and Ns = product of the radices before it maps
// butterfly u of line b to
//   inputs  x = u + r*(L/R)                       (r = 0..R-1)
//   outputs x = (u - u%Ns)*R + u%Ns + r*Ns
// with twiddle W_{Ns*R}^{(u%Ns)*r} on input r, giving natural order after the
// last stage.  Twiddles come from a table of Ltab-th roots of unity
// W^e = exp(-2*pi*i*e/Ltab) (Ltab a multiple of L); the inverse transform uses
// their conjugates.
//
// Radices up to 10 are register butterflies: the first stage's inputs come
// straight from the pass's source and the last stage's outputs go straight to
// its destination, so a line of two stages (up to 100 points) crosses shared
// memory once.  Primes above 7 are one stage each, computed from the sums
// and differences of mirrored inputs (prime_stage).  The former engine
// (radices up to 8, every stage through shared memory, primes as direct
// sums with a table look-up per product) spent its time on shared-memory
// traffic and run-time index division.
//
// Rows too long for two tile buffers use the in-place engine at the end of
// this file (radices up to 8, register-staged).
#pragma once
#include "cplx.cuh"
#include "dft.cuh"
#include "plan_dev.h"

namespace csipm {

// ------------------------------------------------------------------- stages
// x/d for 0 <= x < 2^16, d < 2^16 from mag = floor((2^32 - 1)/d) + 1 (exact in
// that range); d == 1 is the one divisor whose reciprocal does not fit
__device__ __forceinline__ int quot(int x, int d, unsigned mag) { return d == 1 ? x : (int)__umulhi((unsigned)x, mag); }

// One butterfly of a stage: inputs v, twiddled and transformed.
template <int R, bool INV, typename T>
__device__ __forceinline__ void twiddle_dft(cplx_t<T>* v, int k, const FftStage& s, const cplx_t<T>* __restrict__ tw) {
    if (R > 1 && s.Ns > 1) {
        const int e = k * s.step;
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = twmul<INV>(v[r], tw[r * e]);
    }
    Dft<R, INV, T>::run(v);
}

#define CSIPM_RADICES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)

// Butterfly w of a smem -> smem stage: load<R> and transform, then put<R>.
template <typename T, int R, bool INV>
__device__ __forceinline__ void bfly_load(cplx_t<T>* v, const cplx_t<T>* in, const TileLay& lay, const FftStage& s,
                                          const cplx_t<T>* __restrict__ tw, int u, int k, int b) {
    const cplx_t<T>* p = in + lay.at(u, b);
    const int d = s.m * lay.tbp;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[r * d];
    twiddle_dft<R, INV, T>(v, k, s, tw);
}
template <typename T, int R>
__device__ __forceinline__ void bfly_put(const cplx_t<T>* v, cplx_t<T>* out, const TileLay& lay, int o, int Ns, int b) {
    cplx_t<T>* p = out + lay.at(o, b);
    const int d = Ns * lay.tbp;
#pragma unroll
    for (int r = 0; r < R; ++r) p[r * d] = v[r];
}

// ---- prime stages
// A radix p without a register butterfly: with t_j = x_j + x_{p-j} and
// d_j = x_j - x_{p-j} (j = 1..h, h = (p-1)/2) of the twiddled inputs,
//   X_k, X_{p-k} = (x_0 + sum_j cos(2 pi j k/p) t_j) -+ i sum_j sin(2 pi j k/p) d_j,
// (p-1)^2 real multiply-adds a butterfly instead of 4 p^2, and each
// thread takes PRIME_K pairs (k, p-k), so a value read from shared memory
// serves 2*PRIME_K of them.  Up to PRIME_MAT the cosines and sines of all
// (j, k) lie in shared memory, PRIME_K neighbours at a time (a broadcast read
// at a fixed offset each; one table of p roots with the index j k mod p kept
// by additions spent more instructions on indices than on arithmetic); larger
// primes use the table of roots.  Five pairs a thread divide those of 11, 31 and
// 41; a last group that is not full computes the rest for nothing.  A'A in FP64 on
// B200 with 3 / 4 / 5 / 6 pairs, us: 310x410x410 (31, 41) 2190 / 2099 / 1946 / 2040,
// 984^2 (41) 59 / 54 / 54 / 59, 952^2 (17) 49 / 45 / 46 / 48, 988^2 (19) 56 / 58 / 55 /
// 53, 936^2 (13) 49 / 50 / 51 / 45, 130^3 (13) 81 / 86 / 102 / 85.
constexpr int PRIME_K = 5;
constexpr int PRIME_MAT = 64;

__host__ __device__ constexpr int prime_groups(int p) { return ((p - 1) / 2 + PRIME_K - 1) / PRIME_K; }
__host__ __device__ constexpr int prime_table(int p) {
    return p <= PRIME_MAT ? (p - 1) / 2 * prime_groups(p) * PRIME_K : p;
}

// the tables (cos, -sin) of every prime stage, each at its cs
template <typename C>
__device__ __forceinline__ void prime_tables(const FftStage* st, int nst, const C* __restrict__ tw, int Ltab, C* cs) {
    for (int s = 0; s < nst; ++s) {
        const int p = st[s].R;
        if (reg_radix(p)) continue;
        C* t = cs + st[s].cs;
        const int unit = Ltab / p;
        if (p > PRIME_MAT) {
            for (int e = threadIdx.x; e < p; e += blockDim.x) t[e] = tw[e * unit];
        } else {
            const int nk = prime_groups(p) * PRIME_K;
            for (int e = threadIdx.x; e < (p - 1) / 2 * nk; e += blockDim.x)
                t[e] = tw[((e / nk + 1) * (e % nk + 1)) % p * unit];
        }
    }
}

// t_j at position j, d_j at position p - j of buf, from ld(x, b) (the source
// of a first stage, or buf itself: one thread owns both positions).
template <typename T, bool INV, class Ld>
__device__ __forceinline__ void prime_combine(cplx_t<T>* buf, const TileLay& lay, const FftStage& s, bool first,
                                              const cplx_t<T>* __restrict__ tw, Ld&& ld) {
    using C = cplx_t<T>;
    const int p = s.R, h = (p - 1) / 2, mask = (1 << lay.lg) - 1;
    const int n = (s.m * (h + 1)) << lay.lg;
    for (int w = threadIdx.x; w < n; w += blockDim.x) {
        const int b = w & mask, rest = w >> lay.lg;
        const int j = quot(rest, s.m, s.mag_m), u = rest - j * s.m;
        if (j == 0) {
            if (first) buf[lay.at(u, b)] = ld(u, b);
            continue;
        }
        const int x1 = u + j * s.m, x2 = u + (p - j) * s.m;
        C a = ld(x1, b), c = ld(x2, b);
        if (s.Ns > 1) {
            const int k = u - s.Ns * quot(u, s.Ns, s.mag_ns);
            a = twmul<INV>(a, tw[k * j * s.step]);
            c = twmul<INV>(c, tw[k * (p - j) * s.step]);
        }
        buf[lay.at(x1, b)] = cadd(a, c);
        buf[lay.at(x2, b)] = csub(a, c);
    }
}

// The sums of one thread's PRIME_K pairs; put(x, b, value) receives the
// outputs (never into buf).
template <typename T, bool INV, class Put>
__device__ __forceinline__ void prime_sums(const cplx_t<T>* buf, const TileLay& lay, const FftStage& s,
                                           const cplx_t<T>* cs, Put&& put) {
    using C = cplx_t<T>;
    const int p = s.R, h = (p - 1) / 2, mask = (1 << lay.lg) - 1;
    const int ng = prime_groups(p);
    const int n = (s.m * ng) << lay.lg;
    for (int w = threadIdx.x; w < n; w += blockDim.x) {
        const int b = w & mask, rest = w >> lay.lg;
        const int g = quot(rest, s.m, s.mag_m), u = rest - g * s.m;
        const C x0 = buf[lay.at(u, b)];
        C e[PRIME_K], f[PRIME_K], sum = x0;
#pragma unroll
        for (int q = 0; q < PRIME_K; ++q) {
            e[q] = x0;
            f[q] = mk((T)0, (T)0);
        }
        auto add = [&](int q, C r, C t, C d) {   // r = (cos, -sin)
            e[q].x += r.x * t.x;
            e[q].y += r.x * t.y;
            f[q].x -= r.y * d.x;
            f[q].y -= r.y * d.y;
        };
        const int step = s.m * lay.tbp;
        const C *pt = buf + lay.at(u, b), *pd = pt + p * step;   // t_j, d_j
        if (p <= PRIME_MAT) {
            const C* row = cs + g * PRIME_K;
#pragma unroll 1
            for (int j = 1; j <= h; ++j, row += ng * PRIME_K) {
                const C t = *(pt += step), d = *(pd -= step);
                sum = cadd(sum, t);
#pragma unroll
                for (int q = 0; q < PRIME_K; ++q) add(q, row[q], t, d);
            }
        } else {
            int idx[PRIME_K];
#pragma unroll
            for (int q = 0; q < PRIME_K; ++q) idx[q] = 0;
#pragma unroll 1
            for (int j = 1; j <= h; ++j) {
                const C t = *(pt += step), d = *(pd -= step);
                sum = cadd(sum, t);
#pragma unroll
                for (int q = 0; q < PRIME_K; ++q) {
                    idx[q] += min(g * PRIME_K + q + 1, h);
                    if (idx[q] >= p) idx[q] -= p;
                    add(q, cs[idx[q]], t, d);
                }
            }
        }
        const int k0 = u - s.Ns * quot(u, s.Ns, s.mag_ns);
        const int o = (u - k0) * p + k0;
        if (g == 0) put(o, b, sum);
#pragma unroll
        for (int q = 0; q < PRIME_K; ++q) {
            const int k = g * PRIME_K + q + 1;
            if (k <= h) {
                const C jf = cmul_i(f[q]);
                put(o + k * s.Ns, b, INV ? cadd(e[q], jf) : csub(e[q], jf));
                put(o + (p - k) * s.Ns, b, INV ? csub(e[q], jf) : cadd(e[q], jf));
            }
        }
    }
}

// Items of a stage: what one thread takes at a time.
__host__ __device__ __forceinline__ int stage_items(int R, int L, int lg) {
    return reg_radix(R) ? (L / R) << lg : ((L / R) * prime_groups(R)) << lg;
}

// A tile's buffers and tables.
template <typename C>
struct FftTile {
    TileLay lay;
    const FftStage* st;
    int nst, L;
    const C* tw;
    const C* cs;      // prime roots of st
    C* buf;           // shared memory; the tile between stages is at buf + cur,
    int cur, oth;     // the second buffer (only touched by stages from shared to shared memory) at buf + oth
    __device__ __forceinline__ void swap() { const int t = cur; cur = oth; oth = t; }
};

// Stages s0..s1-1, smem -> smem from one buffer to the other (the tile in
// t.cur before and after); ends with a barrier.  There is no barrier inside a
// radix's branch: the compiler cannot prove the branch uniform and spills what
// lives across one.
template <typename T, bool INV>
__device__ __forceinline__ void mid_stages(FftTile<cplx_t<T>>& t, int s0, int s1) {
    using C = cplx_t<T>;
    const TileLay lay = t.lay;
    const int mask = (1 << lay.lg) - 1;
#pragma unroll 1
    for (int q = s0; q < s1; ++q) {
        const FftStage s = t.st[q];
        const int n = s.m << lay.lg;
        if (reg_radix(s.R)) {
            for (int w = threadIdx.x; w < n; w += blockDim.x) {
                const int b = w & mask, u = w >> lay.lg;
                const int k = u - s.Ns * quot(u, s.Ns, s.mag_ns);
                const int o = (u - k) * s.R + k;
                switch (s.R) {
#define CSIPM_MID(RR)                                                       \
                    case RR: {                                              \
                        C v[RR];                                            \
                        bfly_load<T, RR, INV>(v, t.buf + t.cur, lay, s, t.tw, u, k, b); \
                        bfly_put<T, RR>(v, t.buf + t.oth, lay, o, s.Ns, b); \
                    } break;
                    CSIPM_RADICES(CSIPM_MID)
#undef CSIPM_MID
                }
            }
        } else {
            C* buf = t.buf + t.cur;
            prime_combine<T, INV>(buf, lay, s, false, t.tw, [&](int x, int c) { return buf[lay.at(x, c)]; });
            __syncthreads();
            C* out = t.buf + t.oth;
            prime_sums<T, INV>(buf, lay, s, t.cs + s.cs, [&](int x, int c, C w) { out[lay.at(x, c)] = w; });
        }
        t.swap();
        __syncthreads();
    }
}

// First stage: ld.load<R>(v, u, m, b) brings the inputs u + r*m of line b
// (ld.one(x, b) a single one), the results go to t.cur; ends with a barrier.
template <typename T, bool INV, class Ld>
__device__ __forceinline__ void first_stage(FftTile<cplx_t<T>>& t, Ld& ld) {
    using C = cplx_t<T>;
    const FftStage s = t.st[0];
    const int mask = (1 << t.lay.lg) - 1;
    switch (s.R) {
#define CSIPM_FIRST(RR)                                                                   \
        case RR:                                                                          \
            for (int w = threadIdx.x; w < s.m << t.lay.lg; w += blockDim.x) {             \
                const int b = w & mask, u = w >> t.lay.lg;                                \
                C v[RR];                                                                  \
                ld.template load<RR>(v, u, s.m, b);                                       \
                Dft<RR, INV, T>::run(v);                                                  \
                bfly_put<T, RR>(v, t.buf + t.cur, t.lay, u * RR, 1, b);                  \
            }                                                                             \
            break;
        CSIPM_RADICES(CSIPM_FIRST)
#undef CSIPM_FIRST
        default: {
            C* out = t.buf + t.oth;
            const TileLay lay = t.lay;
            prime_combine<T, INV>(t.buf + t.cur, lay, s, true, t.tw, [&](int x, int b) { return ld.one(x, b); });
            __syncthreads();
            prime_sums<T, INV>(t.buf + t.cur, lay, s, t.cs + s.cs, [&](int x, int b, C v) { out[lay.at(x, b)] = v; });
            t.swap();
        } break;
    }
    __syncthreads();
}

// Last stage: outputs x = u + r*Ns of line b go to out.store<R>(v, u, Ns, b)
// (out.one(x, b, v) a single one).
template <typename T, bool INV, class St>
__device__ __forceinline__ void last_stage(FftTile<cplx_t<T>>& t, St& out) {
    using C = cplx_t<T>;
    const FftStage s = t.st[t.nst - 1];
    const int mask = (1 << t.lay.lg) - 1;
    const TileLay lay = t.lay;
    switch (s.R) {
#define CSIPM_LAST(RR)                                                                    \
        case RR:                                                                          \
            for (int w = threadIdx.x; w < s.m << lay.lg; w += blockDim.x) {               \
                const int b = w & mask, u = w >> lay.lg;                                  \
                C v[RR];                                                                  \
                bfly_load<T, RR, INV>(v, t.buf + t.cur, lay, s, t.tw, u, u, b);           \
                out.template store<RR>(v, u, s.Ns, b);                                    \
            }                                                                             \
            break;
        CSIPM_RADICES(CSIPM_LAST)
#undef CSIPM_LAST
        default: {
            C* buf = t.buf + t.cur;
            prime_combine<T, INV>(buf, lay, s, false, t.tw, [&](int x, int b) { return buf[lay.at(x, b)]; });
            __syncthreads();
            prime_sums<T, INV>(buf, lay, s, t.cs + s.cs,
                               [&](int x, int b, C v) { out.one(x, b, v); });
        } break;
    }
}

// A whole transform from ld to out.  Every thread of the block calls it (it
// contains barriers); the caller synchronises before the buffers are reused.
template <typename T, bool INV, class Ld, class St>
__device__ __forceinline__ void fft_through(FftTile<cplx_t<T>>& t, Ld& ld, St& out) {
    using C = cplx_t<T>;
    if (t.nst == 1) {   // one radix: no exchange (a prime goes through shared memory)
        const FftStage s = t.st[0];
        const int mask = (1 << t.lay.lg) - 1;
        switch (s.R) {
#define CSIPM_ONE(RR)                                                     \
            case RR:                                                      \
                for (int w = threadIdx.x; w < 1 << t.lay.lg; w += blockDim.x) { \
                    C v[RR];                                              \
                    ld.template load<RR>(v, 0, 1, w & mask);              \
                    Dft<RR, INV, T>::run(v);                              \
                    out.template store<RR>(v, 0, 1, w & mask);            \
                }                                                         \
                break;
            CSIPM_RADICES(CSIPM_ONE)
#undef CSIPM_ONE
            default:
                prime_combine<T, INV>(t.buf + t.cur, t.lay, s, true, t.tw, [&](int x, int b) { return ld.one(x, b); });
                __syncthreads();
                prime_sums<T, INV>(t.buf + t.cur, t.lay, s, t.cs + s.cs, [&](int x, int b, C v) { out.one(x, b, v); });
                break;
        }
        return;
    }
    first_stage<T, INV>(t, ld);
    mid_stages<T, INV>(t, 1, t.nst - 1);
    last_stage<T, INV>(t, out);
}

// ------------------------------------------------- in-place engine (very long rows)
// per-thread register budget: about 8 complex values per stage
template <int R> struct MaxItems { static constexpr int v = (8 + R - 1) / R; };
constexpr int GENERIC_MAX_ITEMS = 8;

template <typename T, int R, bool INV>
__device__ __forceinline__ void stage_ip(cplx_t<T>* __restrict__ buf, int L, int TB, int TBP, int Ns,
                                      const cplx_t<T>* __restrict__ tw, int step) {
    using C = cplx_t<T>;
    constexpr int MI = MaxItems<R>::v;
    const int m = L / R;
    const int nitems = TB * m;
    const int tid = threadIdx.x, nthr = blockDim.x;
    C v[MI][R];
    int oidx[MI];
#pragma unroll
    for (int it = 0; it < MI; ++it) {
        const int w = tid + it * nthr;
        oidx[it] = -1;
        if (w < nitems) {
            const int b = w % TB, u = w / TB, k = u % Ns;
#pragma unroll
            for (int r = 0; r < R; ++r) v[it][r] = buf[(u + r * m) * TBP + b];
            if (Ns > 1) {
#pragma unroll
                for (int r = 1; r < R; ++r) v[it][r] = twmul<INV>(v[it][r], tw[k * r * step]);
            }
            Dft<R, INV, T>::run(v[it]);
            oidx[it] = ((u - k) * R + k) * TBP + b;
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < MI; ++it) {
        if (oidx[it] >= 0) {
#pragma unroll
            for (int r = 0; r < R; ++r) buf[oidx[it] + r * Ns * TBP] = v[it][r];
        }
    }
    __syncthreads();
}

template <typename T, bool INV>
__device__ __forceinline__ void stage_generic_ip(cplx_t<T>* __restrict__ buf, int L, int TB, int TBP, int Ns, int p,
                                              const cplx_t<T>* __restrict__ tw, int step, int Ltab) {
    using C = cplx_t<T>;
    const int m = L / p;
    const int nitems = TB * L;
    const int tid = threadIdx.x, nthr = blockDim.x;
    C res[GENERIC_MAX_ITEMS];
    int oidx[GENERIC_MAX_ITEMS];
#pragma unroll
    for (int it = 0; it < GENERIC_MAX_ITEMS; ++it) {
        const int w = tid + it * nthr;
        oidx[it] = -1;
        if (w < nitems) {
            const int b = w % TB, rest = w / TB;
            const int u = rest % m, ro = rest / m, k = u % Ns;
            const int e0 = (int)(((long long)step * (k + ro * Ns)) % Ltab);
            C acc = mk((T)0, (T)0);
            int e = 0;
            for (int t = 0; t < p; ++t) {
                acc = cadd(acc, twmul<INV>(buf[(u + t * m) * TBP + b], tw[e]));
                e += e0;
                if (e >= Ltab) e -= Ltab;
            }
            res[it] = acc;
            oidx[it] = ((u - k) * p + k + ro * Ns) * TBP + b;
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < GENERIC_MAX_ITEMS; ++it)
        if (oidx[it] >= 0) buf[oidx[it]] = res[it];
    __syncthreads();
}

// Copy a plan's radix list into shared memory with compile-time indices, so the
// kernel-parameter struct is never indexed dynamically (which would force a
// local-memory copy of the whole parameter block).  Followed by a barrier in
// the caller before first use.
__device__ __forceinline__ void load_radices(const FftPlanDev& pl, int* s_rad) {
#pragma unroll
    for (int s = 0; s < FFT_MAX_STAGES; ++s)
        if (threadIdx.x == s) s_rad[s] = pl.rad[s];
}

// Full transform of TB interleaved lines of length L in place.  Every thread
// of the block must call this (it contains barriers).
template <typename T, bool INV>
__device__ void fft_lines_ip(cplx_t<T>* buf, const int* s_rad, int nst, int L, int TB, int TBP,
                             const cplx_t<T>* __restrict__ tw, int Ltab) {
    int Ns = 1;
#pragma unroll 1
    for (int s = 0; s < nst; ++s) {
        const int R = s_rad[s];
        const int step = Ltab / (Ns * R);
        switch (R) {
            case 2: stage_ip<T, 2, INV>(buf, L, TB, TBP, Ns, tw, step); break;
            case 3: stage_ip<T, 3, INV>(buf, L, TB, TBP, Ns, tw, step); break;
            case 4: stage_ip<T, 4, INV>(buf, L, TB, TBP, Ns, tw, step); break;
            case 5: stage_ip<T, 5, INV>(buf, L, TB, TBP, Ns, tw, step); break;
            case 7: stage_ip<T, 7, INV>(buf, L, TB, TBP, Ns, tw, step); break;
            case 8: stage_ip<T, 8, INV>(buf, L, TB, TBP, Ns, tw, step); break;
            default: stage_generic_ip<T, INV>(buf, L, TB, TBP, Ns, R, tw, step, Ltab); break;
        }
        Ns *= R;
    }
}

}  // namespace csipm

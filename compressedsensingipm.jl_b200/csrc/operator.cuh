// The masked sampling operator A = P_Omega * sqrt(N) * Re(IDFT(B .)) and its
// adjoint, applied matrix-free through fused real-FFT passes.
//
// Layout in HBM: one half spectrum (M1+1) x N2 x N3 of complex values, dim 1
// fastest, pitch ld1; the mask as one bit per real sample, rows of N1 bits
// padded to 32-bit words.  Pass structure (3D; 2D drops the dim-3 passes; 1D
// rows take one or three launches, long1d.cuh):
//
//   A^T A x :  [gather x -> inverse FFT dim 2] -> [inverse dim 3]
//              -> [row: C2R dim 1, scale, mask, R2C dim 1]
//              -> [forward dim 3] -> [forward dim 2 -> scatter + epilogue]
//
// The beta -> spectrum gather is fused into the first pass and the
// spectrum -> beta scatter (plus any elementwise epilogue, e.g. the CG's
// q = A^T A p + D p and p.q) into the last, so beta-space vectors are touched
// once per product and the real-space samples never reach HBM.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "cplx.cuh"
#include "dft.cuh"
#include "geometry.h"
#include "plan_dev.h"
#include "reduce.cuh"

namespace csipm {

// *_SGATHER / *_SSCATTER: beta-space vectors in solver order (geometry.h)
enum PassIn { IN_SPEC = 0, IN_GATHER = 1, IN_REAL = 2, IN_SGATHER = 3 };
enum PassOut { OUT_SPEC = 0, OUT_SCATTER = 1, OUT_REAL = 2, OUT_SSCATTER = 3 };

constexpr double SQRT2_D = 1.4142135623730951;

template <typename T>
struct PassArgs {
    Geom g;
    FftPlanDev pl;
    const cplx_t<T>* tw;     // Ltab-th roots of unity (global memory)
    int Ltab;
    FftStage fwd[PASS_STAGES], inv[PASS_STAGES];   // the plan's stages, in order and (rows) reversed
    cplx_t<T>* spec;
    // strided passes
    int n_lines;             // number of dim-1 positions (M1+1)
    int n_outer;             // number of lines per dim-1 position (outer index range)
    long long so, sx;        // element strides of the outer index and of the transform index
    int jk_mode;             // 0: (j,k) = (o,x)   1: (j,k) = (x,o)   2: (j,k) = (x,0)
    // tile of the run-time-plan passes (PassCfg)
    TileLay lay;
    int span;                // elements of one tile buffer
    int two;                 // 1: a second tile buffer follows the first
    int primes;              // 1: the plan has prime stages
    // row passes
    int nrows;
    const uint32_t* maskw;
    int wpr;
    double scale;
    const T* real_in;
    T* real_out;
    const int* skip;         // when non-null and *skip != 0 the pass returns at once (converged CG)
};

// ------------------------------------------------------------- dependent launches
// A solve is a chain of some hundred kernels of a few microseconds, each
// reading what the one before wrote.  They are launched with programmatic
// stream serialisation: a kernel's blocks may be placed while the one before
// still drains, and wait in pdl_enter (its first statement, before any memory
// is read) until that one has completed and its writes are visible; then the
// next kernel may be placed in turn.  Every kernel of a chain waits, so the
// order of the stream holds throughout.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
    pdl_wait();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Whether a kernel on N samples is launched that way (dim 0: an element
// kernel).  It hides 1-3 us a launch, and costs when early blocks sit beside a
// pass that fills the shared memory or the HBM queues.  A'A in FP64, plain ->
// early (B200, us): 1D 4096 21.6 -> 18.2, 131072 28.7 -> 25.4, 259200 32.2 ->
// 30.0, 524288 41.0 -> 53.1; 256^2 22.6 -> 17.7, 1024^2 46.6 -> 41.4; 64^3 30.8
// -> 22.8, 160^3 115 -> 105, 256^3 384 -> 398.
// Element kernels take one border in every dimension: with the 1D one for them
// too, 1D recoveries by plain launches lost (FP64, ms, as it is -> with 2^18:
// 524288 3.61 -> 3.90, 777600 4.67 -> 4.87, 2^20 4.82 -> 4.95).
inline bool pdl_pays(int dim, long long N) { return N <= (dim == 1 ? 1LL << 18 : 1LL << 22); }

// Not inside a capture: a graph's kernels already follow one another closely,
// and programmatic edges made its replays slower (1024^2 solve 3.47 -> 3.88 ms,
// 320^3 mixed 42.0 -> 46.4 ms).
template <typename... P, typename... A>
inline cudaError_t launch_pdl(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (early) cudaStreamIsCapturing(st, &cap);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = early && cap == cudaStreamCaptureStatusNone;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

// ------------------------------------------------------------- epilogues
// Two-phase epilogues: pre(l) loads what put(l, v, pre) needs, so a scatter
// loop can issue the loads of several elements before it consumes them.
struct NoPre {};

// pre2 / put2 act on the solver-order pair l (elements 2l, 2l+1) with one
// vector access per operand.
template <typename TO>
struct EpiStore {
    TO* out;
    using Pre = NoPre;
    using Pre2 = NoPre;
    __device__ __forceinline__ NoPre pre(int) const { return {}; }
    __device__ __forceinline__ void put(int l, double v, const NoPre&) { out[l] = (TO)v; }
    __device__ __forceinline__ NoPre pre2(int64_t) const { return {}; }
    __device__ __forceinline__ void put2(int64_t l, double x, double y, const NoPre&) {
        reinterpret_cast<cplx_t<TO>*>(out)[l] = mk((TO)x, (TO)y);
    }
    __device__ __forceinline__ void finish() {}
};

// q = A^T A p + D .* p, accumulating p.q (CG product)
template <typename TV>
struct EpiCG {
    const TV* p;
    const TV* D;
    TV* q;
    RedWorkspace ws;
    double acc;
    struct Pre { double p, d; };
    struct Pre2 { cplx_t<TV> p, d; };
    __device__ __forceinline__ Pre pre(int l) const { return Pre{(double)p[l], (double)D[l]}; }
    __device__ __forceinline__ void put(int l, double v, const Pre& r) {
        const TV qv = (TV)(v + r.d * r.p);
        q[l] = qv;
        acc += r.p * (double)qv;
    }
    __device__ __forceinline__ Pre2 pre2(int64_t l) const {
        return Pre2{reinterpret_cast<const cplx_t<TV>*>(p)[l], reinterpret_cast<const cplx_t<TV>*>(D)[l]};
    }
    __device__ __forceinline__ void put2(int64_t l, TV x, TV y, const Pre2& r) {
        const TV qx = x + r.d.x * r.p.x;
        const TV qy = y + r.d.y * r.p.y;
        reinterpret_cast<cplx_t<TV>*>(q)[l] = mk(qx, qy);
        acc += (double)r.p.x * (double)qx + (double)r.p.y * (double)qy;
    }
    __device__ __forceinline__ void finish() {
        double a[1] = {acc};
        grid_reduce<1>(a, ws, 0u, 0u);
    }
};

// ------------------------------------------------------- gather / scatter
template <typename T, typename TS>
__device__ __forceinline__ cplx_t<T> gather_val(const MapEntry& e, const TS* __restrict__ src) {
    if (e.kind == KIND_VERT) return mk((T)src[e.re], (T)0);
    const T r = (T)0.7071067811865476;   // 1/sqrt(2) (the operator is tolerance-checked, not bitwise)
    const T a = (T)src[e.re], b = (T)src[e.im];
    return e.kind == KIND_PLUS ? mk(a * r, b * r) : mk(a * r, -b * r);
}

template <typename T, class Epi>
__device__ __forceinline__ void scatter_one(const MapEntry& e, cplx_t<T> v, Epi& ep) {
    if (!e.src) return;
    const typename Epi::Pre pr = ep.pre(e.re);
    if (e.kind == KIND_VERT) {
        ep.put(e.re, (double)v.x, pr);
    } else {
        const typename Epi::Pre pi = ep.pre(e.im);
        ep.put(e.re, SQRT2_D * (double)v.x, pr);
        ep.put(e.im, (e.kind == KIND_PLUS ? SQRT2_D : -SQRT2_D) * (double)v.y, pi);
    }
}

__device__ __forceinline__ void jk_of(int mode, int o, int x, int& j, int& k) {
    if (mode == 0) { j = o; k = x; }
    else if (mode == 1) { j = x; k = o; }
    else { j = x; k = 0; }
}

// ------------------------------------------------ sources and destinations of lines
// What a pass along dim 2 or 3 reads its lines from and writes them to; one
// object per thread, which keeps one dim-1 position (ii) for a whole tile.
// load<R>: v[r] = value at x = u + r*m; store<R>: v[r] to x = u + r*Ns;
// one: a single position.

// the half spectrum
template <typename T>
struct SpecLine {
    using C = cplx_t<T>;
    C* p;            // position x = 0 of the line
    long long sx;
    bool live;
    __device__ __forceinline__ C one(int x, int) const { return live ? p[x * sx] : mk((T)0, (T)0); }
    __device__ __forceinline__ void one(int x, int, C v) const {
        if (live) p[x * sx] = v;
    }
    template <int R> __device__ __forceinline__ void load(C* v, int u, int m, int) const {
        if (live) {
            const C* q = p + u * sx;
            const long long d = m * sx;
#pragma unroll
            for (int r = 0; r < R; ++r, q += d) v[r] = *q;
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = mk((T)0, (T)0);
        }
    }
    template <int R> __device__ __forceinline__ void store(const C* v, int u, int Ns, int) const {
        if (!live) return;
        C* q = p + u * sx;
        const long long d = Ns * sx;
#pragma unroll
        for (int r = 0; r < R; ++r, q += d) *q = v[r];
    }
};

// beta along dim 2 (x = j), reference packing (SOL false) or solver order
template <typename T, typename TS, bool SOL>
struct GatherLine {
    using C = cplx_t<T>;
    const TS* src;
    LineMap l;
    int64_t p0;      // solver order, interior line: pair of j = 0
    int ps;          // pairs per step of j
    bool live, pairs;
    __device__ __forceinline__ void set(const Geom& g, const TS* s, int ii, int k, bool on) {
        src = s;
        live = on;
        pairs = SOL && ii >= 1 && ii <= g.m1 - 1;
        if (pairs) {
            p0 = sol_pair(g, ii, 0, k);
            ps = g.m1 - 1;
        } else if (on) {
            l = make_line(g, ii, k, SOL);
        }
    }
    __device__ __forceinline__ C one(int x, int) const {
        if (!live) return mk((T)0, (T)0);
        if (SOL && pairs) {
            const T r = (T)0.7071067811865476;
            const cplx_t<TS> w = reinterpret_cast<const cplx_t<TS>*>(src)[p0 + (int64_t)x * ps];
            return mk((T)w.x * r, (T)w.y * r);
        }
        return gather_val<T>(line_at(l, x), src);
    }
    template <int R> __device__ __forceinline__ void load(C* v, int u, int m, int) const {
        const T rr = (T)0.7071067811865476;
        if (!live) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = mk((T)0, (T)0);
        } else if (SOL && pairs) {
            const cplx_t<TS>* __restrict__ s2 = reinterpret_cast<const cplx_t<TS>*>(src) + p0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const cplx_t<TS> w = s2[(int64_t)(u + r * m) * ps];
                v[r] = mk((T)w.x * rr, (T)w.y * rr);
            }
        } else {
            // two loads per value with no branch between them (a vertex reads
            // its real entry twice)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const MapEntry e = line_at(l, u + r * m);
                const T a = (T)src[e.re], b = (T)src[e.kind == KIND_VERT ? e.re : e.im];
                v[r] = e.kind == KIND_VERT ? mk(a, (T)0) : mk(a * rr, e.kind == KIND_PLUS ? b * rr : -b * rr);
            }
        }
    }
};

// the epilogue along dim 2; U positions' operands are loaded before any is used
template <typename T, class Epi, bool SOL>
struct ScatterLine {
    using C = cplx_t<T>;
    Epi* ep;
    LineMap l;
    int64_t p0;
    int ps;
    bool live, pairs;
    __device__ __forceinline__ void set(const Geom& g, Epi* e, int ii, int k, bool on) {
        ep = e;
        live = on;
        pairs = SOL && ii >= 1 && ii <= g.m1 - 1;
        if (pairs) {
            p0 = sol_pair(g, ii, 0, k);
            ps = g.m1 - 1;
        } else if (on) {
            l = make_line(g, ii, k, SOL);
        }
    }
    __device__ __forceinline__ void pair(int x, C v) const {
        if constexpr (SOL) {
            const int64_t q = p0 + (int64_t)x * ps;
            const typename Epi::Pre2 pr = ep->pre2(q);
            ep->put2(q, (T)SQRT2_D * v.x, (T)SQRT2_D * v.y, pr);
        }
    }
    __device__ __forceinline__ void one(int x, int, C v) const {
        if (!live) return;
        if (SOL && pairs) pair(x, v);
        else scatter_one<T>(line_at(l, x), v, *ep);
    }
    template <int R> __device__ __forceinline__ void store(const C* v, int u, int Ns, int) const {
        if (!live) return;
        if constexpr (SOL) {
            if (pairs) {
                constexpr int U = 4;
#pragma unroll
                for (int r0 = 0; r0 < R; r0 += U) {
                    typename Epi::Pre2 pr[U];
#pragma unroll
                    for (int q = 0; q < U; ++q)
                        if (r0 + q < R) pr[q] = ep->pre2(p0 + (int64_t)(u + (r0 + q) * Ns) * ps);
#pragma unroll
                    for (int q = 0; q < U; ++q)
                        if (r0 + q < R)
                            ep->put2(p0 + (int64_t)(u + (r0 + q) * Ns) * ps, (T)SQRT2_D * v[r0 + q].x,
                                     (T)SQRT2_D * v[r0 + q].y, pr[q]);
                }
                return;
            }
        }
        constexpr int U = sizeof(typename Epi::Pre) > 48 ? 1 : 2;
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += U) {
            MapEntry en[U];
            typename Epi::Pre pr[U], pi[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                if (r0 + q < R) {   // no branch around the loads: a mirrored entry's operands are its pair's
                    en[q] = line_at(l, u + (r0 + q) * Ns);
                    pr[q] = ep->pre(en[q].re);
                    pi[q] = ep->pre(en[q].kind == KIND_VERT ? en[q].re : en[q].im);
                }
            }
#pragma unroll
            for (int q = 0; q < U; ++q) {
                if (r0 + q < R && en[q].src) {
                    const C w = v[r0 + q];
                    if (en[q].kind == KIND_VERT) {
                        ep->put(en[q].re, (double)w.x, pr[q]);
                    } else {
                        ep->put(en[q].re, SQRT2_D * (double)w.x, pr[q]);
                        ep->put(en[q].im, (en[q].kind == KIND_PLUS ? SQRT2_D : -SQRT2_D) * (double)w.y, pi[q]);
                    }
                }
            }
        }
    }
};

// ---------------------------------------------------------------- row pre/post-processing
// Z[k] = (X[k] + conj X[M-k]) + i conj(W^k) (X[k] - conj X[M-k])   (C2R pre-processing)
template <typename C>
__device__ __forceinline__ C c2r_pre(C xa, C xb, C w) {
    C s = cadd(xa, cconj(xb)), d = csub(xa, cconj(xb));
    return cadd(s, cmul_i(cmulc(d, w)));
}
// X[k] = (Z[k] + conj Z[M-k]) - i W^k (Z[k] - conj Z[M-k])            (R2C post-processing)
template <typename C>
__device__ __forceinline__ C r2c_post(C za, C zb, C w) {
    C s = cadd(za, cconj(zb)), d = csub(za, cconj(zb));
    return csub(s, cmul_i(cmul(d, w)));
}

// Opts a kernel into the large dynamic shared-memory carve-out, once per
// (kernel, device).  The attribute is set under the lock and recorded only
// after it succeeded, so a thread that launches the kernel concurrently waits
// for it instead of launching before the opt-in (which fails the launch).
// The opt-in covers dynamic + static shared memory, so the dynamic limit set
// is the device's per-block opt-in maximum minus the kernel's static part.
// Dynamic and static shared memory together may take 48 KB without it; the
// static part of the passes (the reductions' arrays) is below 2 KB.
// `always`: opt in whatever the dynamic part (a kernel with a large static one).
inline cudaError_t smem_optin_fn(const void* fn, size_t smem, bool always = false) {
    if (smem <= 46 * 1024 && !always) return cudaSuccess;
    int dev = 0;
    cudaGetDevice(&dev);
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, size_t> limit;   // dynamic bytes set
    std::lock_guard<std::mutex> lk(mu);
    auto it = limit.find({fn, dev});
    if (it != limit.end()) return smem <= it->second ? cudaSuccess : cudaErrorInvalidValue;
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa{};
    e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return e;
    const int dyn = optin - (int)fa.sharedSizeBytes;
    if (dyn < 0 || (size_t)dyn < smem) return cudaErrorInvalidValue;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
    if (e == cudaSuccess) limit[{fn, dev}] = (size_t)dyn;
    return e;
}

template <typename K>
inline cudaError_t smem_optin(K kernel, size_t smem) {
    return smem_optin_fn((const void*)kernel, smem);
}

// Persistent grid: resident CTAs per SM (occupancy API, cached per kernel,
// device and configuration) times the SM count, capped by the tile count.
inline int persistent_grid(const void* fn, int threads, size_t smem, int tiles) {
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, int, size_t>, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(fn, dev, threads, smem);
    int per_sm = 0, sms = 0;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = cache.find(key);
        if (it != cache.end()) per_sm = it->second;
    }
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (per_sm == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess || per_sm < 1) {
            cudaGetLastError();   // not left for the next launch check to report
            per_sm = 1;
        }
        std::lock_guard<std::mutex> lk(mu);
        cache[key] = per_sm;
    }
    const long long g = (long long)per_sm * (sms > 0 ? sms : 148);
    return (int)std::max<long long>(1, std::min<long long>(g, tiles));
}

}  // namespace csipm

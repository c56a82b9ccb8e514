// What a run-time-plan FFT pass is told about its transform and its tile.
#pragma once

#ifndef CSIPM_HD
#ifdef __CUDACC__
#define CSIPM_HD __host__ __device__ __forceinline__
#else
#define CSIPM_HD inline
#endif
#endif

namespace csipm {

constexpr int FFT_MAX_STAGES = 12;
// Stages of a run-time-plan pass: lengths up to 46874 have at most 6, and a
// line of 25601 values does not fit a tile (lay_pass).
constexpr int PASS_STAGES = 6;

struct FftPlanDev {
    int L;                       // transform length
    int nst;                     // number of stages
    int rad[FFT_MAX_STAGES];     // radices, in order
};

// The radices with a register butterfly in the stage dispatch.  Up to 10: a
// radix-16 FP64 butterfly with its twiddles and addresses does not fit 128
// registers (it spilled kilobytes), and the longer straight-line code cost
// more in instruction fetches than the third stage of a 256-point line.
CSIPM_HD constexpr bool reg_radix(int r) { return r <= 10; }

// One stage of a plan as the kernels read it (fill_stages, plan.cu).  It
// travels in every pass's arguments, which each block reads cold from the
// constant bank before anything else: 12 + 12 stages of 28 bytes -> 6 + 6 of 20
// took an A'A on 4096 samples from 18.3 to 16.7 us, on 777600 from 61.7 to 57.3
// (B200, with the unpadded pair tiles of lay_pass).
struct FftStage {
    unsigned short R, Ns, m;    // radix, product of the earlier radices, L/R (quot: below 2^16)
    unsigned short cs;          // prime stages: where its cosines and sines start (prime_tables)
    int step;                   // Ltab/(Ns*R): table stride of the stage's twiddles
    unsigned mag_ns, mag_m;     // reciprocals of Ns and m (quot)
};

// Shared-memory place of element (x, b) of a tile: x*tbp + b, b fastest, so a
// stage access of 8 FP64 (16 FP32) lines covers whole 128-byte rows.  Narrower
// tiles write with the stride R of a stage and meet 2- or 4-way bank conflicts
// when R is even; padding against them (a slot after every 8 positions) cost
// more in address arithmetic than the conflicts do.
struct TileLay {
    int lg, tbp;   // log2(lines), pitch
    CSIPM_HD int at(int x, int b) const { return x * tbp + b; }
};

}  // namespace csipm

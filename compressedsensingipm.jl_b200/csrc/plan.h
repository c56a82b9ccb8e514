// Host-side FFT planning: radix factorisation.  (Twiddle tables are built on
// the device: launch_twiddles in operator.cuh.)
#pragma once
#include <string>
#include <vector>

#include "plan_dev.h"

namespace csipm {

// Factor L into stages: the fewest register radices (up to 10; plan_dev.h)
// that give its factors 2, 3, 5 and 7, balanced and in descending order, then
// every larger prime as a stage of its own.  Fewer stages mean fewer trips
// through shared memory: 90 = 10*9 takes one, 256 = 8*8*4 and 720 = 10*9*8 two.
bool make_fft_plan(int L, FftPlanDev* out, std::string* err);

// The same for a row pass, which runs the plan reversed and then in order and
// joins the two at the first radix: at least two stages, a register radix first.
bool make_row_plan(int L, FftPlanDev* out, std::string* err);

// The plan's stages in plan order (rev: reversed, as the inverse half of a row
// pass runs it) with twiddles from a table of Ltab-th roots.  Writes pl.nst of
// them: the caller has checked that out holds as many.
void fill_stages(const FftPlanDev& pl, int Ltab, bool rev, FftStage* out);

// Complex values of the plan's prime tables (prime_tables, fft_device.cuh).
int prime_table_size(const FftPlanDev& pl);

// Radices up to 8 for the in-place engine: radix 8 first, then 4/2 for the
// rest of the power of two, then 5, 3, 7; any other prime a direct DFT.
bool make_fft_plan_ip(int L, FftPlanDev* out, std::string* err);

// True when every stage of an in-place plan respects the per-thread register
// budget for `lines` interleaved lines processed by `nthreads` threads.
bool plan_fits(const FftPlanDev& pl, int lines, int nthreads);

}  // namespace csipm

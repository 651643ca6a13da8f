// iir_sweep.h — host side of the state-sweep schedule (iir_sweep.cuh): the compiled kernels, and
// the tables and halo of a filter for one of them.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "iir_host_internal.h"

namespace iirhost {

// Kernels of the recurrence on differences (compiled from this many sections on), beside the
// realizations' own kinds.
constexpr int SWEEP_KIND_PH_DIFF = 100;
constexpr int SWEEP_DIFF_MIN_SECTIONS = 6;

// A compiled sweep kernel: realization, sections, sub-rows of N samples, R per lane, warps per block.
struct SweepKernel {
    int kind, K, N, R, warps;
    const void* fn;
    size_t smem;
    int span() const { return N * R; }
};

// Kernels of a realization and number of sections: the one for large signals, then (if there is
// one) the one for small signals.
std::vector<const SweepKernel*> sweep_kernels(int kind, int K);

// A filter's decay and transition in FP64, from its float32 sections.
struct SweepFilter {
    int K = 0;
    double gain = 1.0;
    std::vector<SectionF32> secs;
    std::vector<double> phi;    // one-sample state transition, 2K x 2K
    std::vector<double> scale;  // each section's output for white noise (the states' own scale)
};
SweepFilter sweep_filter(const SectionF32* secs, int K, double gain);
// Whether a pole alone takes longer than `samples` to fall to 1e-10 (no norm of the transition is below it):
// then the filter does not decay within them, and its tables need not be worked out.
bool sweep_too_slow(const SectionF32* secs, int K, int samples);
// Steps of `unit` samples after which older state is below 1e-10 of the states' own scale, 0 if more
// than `most` are needed.
int sweep_decay(const SweepFilter& f, int unit, int most);
// The tables of one kernel geometry (SweepGeom's layout).
std::vector<float> sweep_tables(const SweepFilter& f, int N, int R);
// What a section's residuals at the end of a sub-row of N samples are held to (sweep_agree).
struct SweepLimits {
    float wd, tol;
};
SweepLimits sweep_limits(const SectionF32& s, int N);
// The schedule's float32 arithmetic on white noise on an offset, with pass B in the direct form or on differences:
// the kernel's steps done on the host over some sub-rows, with its tables. error: against 64 bits (2-norm).
// residual: the largest one, as a fraction of its limit; from about 0.7 on in 40 sub-rows, a tile of 128 is corrected now
// and then on any signal.
struct SweepTrial {
    double error, residual;
};
SweepTrial sweep_trial(const SweepFilter& f, const std::vector<float>& tables, int N, bool diff, int rows, float offset = 0.f);

}  // namespace iirhost

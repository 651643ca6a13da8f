// iir_sweep.h — host side of the state-sweep schedule (iir_sweep.cuh): the compiled kernels, and
// the tables and halo of a filter for one of them.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "iir_host_internal.h"

namespace iirhost {

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
// Steps of `unit` samples after which older state is below 1e-10 of the states' own scale, 0 if more
// than `most` are needed.
int sweep_decay(const SweepFilter& f, int unit, int most);
// The tables of one kernel geometry (SweepGeom's layout).
std::vector<float> sweep_tables(const SweepFilter& f, int N, int R);

}  // namespace iirhost

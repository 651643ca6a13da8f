// iir_batch_sweep.h — what the host and the kernels of the batched state sweep share
// (iir_batch_sweep.cuh), and its host side.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <vector>

#include "iir_sweep.h"

namespace iirgb {

constexpr int BSWEEP_STEPS = 5;  // scan steps: 32 lanes

// States that reach no further than this many lanes have a power of their own for each of them.
constexpr int BSWEEP_NEAR = 8;

// Sections that a cascade of K is filtered with: the compiled numbers are 1, 2, 3, 4, 6 and 8, and 5 and
// 7 get one that passes its input on.
__host__ __device__ constexpr int bsweep_sections(int K) { return K == 5 ? 6 : K == 7 ? 8 : K; }
// Sub-rows of a lane row: four of 32 samples up to 4 sections (independent chains in pass B), two of 64
// above (each join of two sub-rows costs a K x K block product: 2 K^2 multiply-adds); lane rows of 32
// samples are two of 16.
__host__ __device__ constexpr int bsweep_subrow(int K, int span) { return span == 32 ? 16 : K <= 4 ? 32 : 64; }
// How a tile's incoming state gets to its lanes. Up to 4 sections the tile's end state goes out from
// rest, before the incoming one is waited for, and the first lanes add the response to it (near powers).
// Above, the response costs more than waiting: the incoming state enters the scan itself.
__host__ __device__ constexpr bool bsweep_chained(int K) { return K > 4; }

__host__ __device__ constexpr int bsweep_table_floats(int K, int span) {  // BatchSweepGeom::T_LEN
    return 2 * K * bsweep_subrow(K, span) + 8 * K + 4 + ((2 * K + 3) & ~3) +
           4 * (1 + BSWEEP_STEPS + (bsweep_chained(K) ? 0 : BSWEEP_NEAR)) * (K * (K + 1) / 2);
}
// The largest table of up to K sections.
__host__ __device__ constexpr int bsweep_table_capacity(int K, int span) {
    int most = 0;
    for (int k = 1; k <= K; ++k) {
        const int t = bsweep_table_floats(bsweep_sections(k), span);
        most = t > most ? t : most;
    }
    return most;
}

constexpr unsigned BATCH_RUN_NONE = 0xffffffffu;

// Consecutive tiles of one segment. x is on the 16-byte grid; `peel` samples (0..3) lie before it.
struct __align__(16) BatchRun {
    const float* x;
    float* y;
    const float* zi;       // state before the segment (x[-2], x[-1], then every section's y[-2], y[-1]); null: rest
    float* zf;             // state after it, or null
    long long n;           // samples from x on
    unsigned int tile0;    // tiles [tile0, tile0 + count)
    unsigned int count;
    unsigned int table;    // the filter's table, in 16-byte units from the launch's tables
    unsigned char K, rounds, peel;
    unsigned char warm;    // 1: the tile before tile0 leads up to it
    unsigned int withhold; // fault injection: the tile whose end state is not passed on (BATCH_RUN_NONE: none)
    unsigned char pad[4];
};
static_assert(sizeof(BatchRun) == 64, "copied as 16 words");

// Whole tiles move by tensor copies. One map serves every segment: it sees a range of memory from each of
// its 16-byte granules at once, dims {32 samples, granule, 32 lane rows} with strides of 4 bytes, 16 bytes
// and a lane row, so that a tile may start at any granule.
struct IirBatchSweepParams {
    CUtensorMap tmap_x, tmap_y;
    const float* x0;          // granule 0 of the maps
    float* y0;
    const BatchRun* runs;
    const float4* tables;
    IirLaunchState* state;
    long long timeout_ns;
    unsigned int nruns;
    unsigned int unit;  // runs per draw, 1 or 2
    int use_tma;        // the maps are valid
};

}  // namespace iirgb

namespace iirhost {

// A compiled kernel: filters of up to max_k sections, lane rows of `span` samples.
struct BatchSweepKernel {
    int max_k, span;
    int threads;
    const void* fn;
    size_t smem;
    int tile() const { return 32 * span; }
};
void bsweep_kernels2(std::vector<BatchSweepKernel>& v);
void bsweep_kernels4(std::vector<BatchSweepKernel>& v);
void bsweep_kernels8(std::vector<BatchSweepKernel>& v);

// A filter for one kernel geometry: its table and scan steps; fast: it decays within a tile.
struct BatchSweepFilter {
    std::vector<float> table;
    int rounds = 0;
    bool fast = false;
};
BatchSweepFilter bsweep_filter(const SectionF32* secs, int K, double gain, int span);

}  // namespace iirhost

// iir_plr.cu — PLR realization: the whole cascade as ONE direct-form recurrence of order
// K = 2 * sections, solved by the hierarchical merge of Maleki & Burtscher (ASPLOS'18).
//
// Reference: include/plr_kernels.cuh:484-3107 (PLR_2/4/8/16). Per chunk of BT * X samples in
// the strided layout (thread t holds samples v*BT + t, plr_kernels.cuh:520,535):
//   1. FIR t[n] = x[n] + sum_j b_j x[n-1-j] through shared memory (plr_kernels.cuh:539-562);
//   2. intra-warp iterative doubling: at width w the upper half of each w-group adds
//      sum_j fac_j[u] * y_lower[w/2 - K + j], fac_j = n-nacci factors (response at offset u to
//      a unit value in history slot j; plr_kernels.cuh:564-632);
//   3. inter-warp doubling with the same factors through shared memory (plr_kernels.cuh:634-785);
//   4. segment chaining over the X values per thread (plr_kernels.cuh:787-811): here one thread
//      chains the segments' end states with the segment transition (fac_j at the last K offsets)
//      and every segment is then corrected at once, instead of one segment after another with two
//      block barriers each;
//   5. K-dimensional decoupled lookback for the chunk's incoming state and the carry correction
//      val += sum_j fac_j[i] X_j (plr_kernels.cuh:813-899). The lookback is truncated to the m
//      preceding chunks' aggregates when the chunk transition has decayed (||Phi^m|| <= 1e-10),
//      else two-level over groups of 32 chunks.
// Order 2 is a single section, and its direct form is what PH's state sweep runs (iir_sweep.cuh): large
// signals go there when the filter decays within a tile.
// Everything is float32 with plain products and sums, as in the reference, so order 16 keeps
// its direct-form numerical fragility (reported by the accuracy tests, not hidden).
#include "iir_lookk.cuh"
#include "iir_registry.h"

namespace iirgb {

template <int KO, int BT, int X>
struct PlrBlock {
    static constexpr int THREADS = 32 + BT;  // control warp + row threads
    static constexpr int CHUNK = BT * X;
    static constexpr int NWR = BT / 32;
    static_assert(BT % 32 == 0 && KO <= 16 && KO % 2 == 0, "PLR geometry");

    struct Smem {
        float xs[KO + CHUNK];           // input of the chunk with K samples of history
        float sfac[KO][BT];             // fac_j[i] for i < BT
        float wlast[NWR][X][KO];        // last K values of each warp per segment
        float seglast[X][KO];           // last K values of each segment solved from zero state
        float segin[X][KO];             // each segment's true history (last K values of the one before)
        float part[KO];
        float Xc[KO];
        unsigned int chunk, epoch;
        int bail;
    };
    static constexpr size_t SMEM_BYTES = sizeof(Smem);

    __device__ static void run(const IirPlrParams& p, unsigned char* smem_raw) {
        Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        if (tid == 0) {
            uint32_t epoch;
            sm.chunk = take_ticket(p.state, p.nchunks, epoch);
            sm.epoch = epoch;
            sm.bail = 0;
        }
        __syncthreads();
        const uint32_t c = sm.chunk, epoch = sm.epoch;
        const long long cs = static_cast<long long>(c) * CHUNK;
        const bool row = warp > 0;
        const int t = tid - 32;       // row thread index
        const int rw = warp - 1;      // row warp index
        const float gain = p.gain;
        float val[X];
        if (row) {
#pragma unroll
            for (int v = 0; v < X; ++v) {
                const long long gi = cs + v * BT + t;
                const float xv = (gi < p.n) ? __ldg(p.x + gi) * gain : 0.f;
                sm.xs[KO + v * BT + t] = xv;
                val[v] = xv;
            }
            if (t < KO) sm.xs[t] = (c > 0) ? __ldg(p.x + cs - KO + t) * gain : 0.f;
#pragma unroll
            for (int j = 0; j < KO; ++j) sm.sfac[j][t] = __ldg(p.fac + static_cast<size_t>(j) * CHUNK + t);
        }
        __syncthreads();
        if (row) {
            // 1. FIR
#pragma unroll
            for (int v = 0; v < X; ++v) {
                const int i = KO + v * BT + t;
                float acc = val[v];
#pragma unroll
                for (int j = 0; j < KO; ++j) acc = fmaf(p.b[j], sm.xs[i - 1 - j], acc);
                val[v] = acc;
            }
            // 2. intra-warp doubling
#pragma unroll
            for (int half = 1; half < 32; half <<= 1) {
                const int gbase = lane & ~(2 * half - 1);
                const bool upper = (lane & half) != 0;
                const int u = lane & (half - 1);
#pragma unroll
                for (int j = 0; j < KO; ++j) {
                    const int src = half - KO + j;  // position in the group of the lower half's value
                    if (src < 0) continue;
                    const float f = sm.sfac[j][u];
#pragma unroll
                    for (int v = 0; v < X; ++v) {
                        const float y = __shfl_sync(FULL_MASK, val[v], gbase + src);
                        if (upper) val[v] = fmaf(f, y, val[v]);
                    }
                }
            }
            // 3. inter-warp doubling through shared memory (row warps only)
#pragma unroll
            for (int hw = 1; hw < NWR; hw <<= 1) {
                if (lane >= 32 - KO) {
#pragma unroll
                    for (int v = 0; v < X; ++v) sm.wlast[rw][v][lane - (32 - KO)] = val[v];
                }
                named_barrier_rows(NWR);
                if (rw & hw) {
                    const int src = (rw & ~(2 * hw - 1)) + hw - 1;  // last warp of the lower half
                    const int u = (rw & (hw - 1)) * 32 + lane;      // offset in the upper half
#pragma unroll
                    for (int j = 0; j < KO; ++j) {
                        const float f = sm.sfac[j][u];
#pragma unroll
                        for (int v = 0; v < X; ++v) val[v] = fmaf(f, sm.wlast[src][v][j], val[v]);
                    }
                }
                named_barrier_rows(NWR);
            }
            // 4. segment chaining. Segment v (BT samples) was solved from zero history; its true
            // last K values are L_v = local_v + Phi L_(v-1), Phi[i][j] = fac_j[BT - K + i] (the
            // response at the segment's last K offsets to history slot j), L_(-1) = 0 (the chunk's
            // own history enters with the carry, step 5); then segment v adds the response to
            // L_(v-1) at every sample.
            if constexpr (X > 1) {
                if (rw == NWR - 1 && lane >= 32 - KO) {
#pragma unroll
                    for (int v = 0; v < X; ++v) sm.seglast[v][lane - (32 - KO)] = val[v];
                }
                named_barrier_rows(NWR);
                if (t < KO) {  // K threads, one component each, in lockstep within the first warp
                    float L = sm.seglast[0][t];
#pragma unroll
                    for (int v = 1; v < X; ++v) {
                        sm.segin[v][t] = L;
                        __syncwarp(0xffffffffu >> (32 - KO));
                        float nl = sm.seglast[v][t];
#pragma unroll
                        for (int j = 0; j < KO; ++j) nl = fmaf(sm.sfac[j][BT - KO + t], sm.segin[v][j], nl);
                        __syncwarp(0xffffffffu >> (32 - KO));
                        L = nl;
                    }
                    sm.part[t] = L;
                }
                named_barrier_rows(NWR);
#pragma unroll
                for (int v = 1; v < X; ++v) {
#pragma unroll
                    for (int j = 0; j < KO; ++j) val[v] = fmaf(sm.sfac[j][t], sm.segin[v][j], val[v]);
                }
            } else {
                if (rw == NWR - 1 && lane >= 32 - KO) sm.part[lane - (32 - KO)] = val[X - 1];
            }
        }
        __syncthreads();  // (A) chunk aggregate in sm.part
        if (!row) {
            float own[KO], Xc[KO];
#pragma unroll
            for (int j = 0; j < KO; ++j) {
                own[j] = sm.part[j];
                Xc[j] = 0.f;
            }
            const bool withhold = static_cast<long long>(c) == p.withhold_chunk;
            const uint32_t pf = 2u * epoch + 1u, ff = 2u * epoch + 2u;
            unsigned long long* slots = p.carry;
            unsigned long long* gslots = p.carry + static_cast<size_t>(p.carry_cap) * 2 * KO;
            if (lane == 0 && !withhold) publishk<KO>(slots + static_cast<size_t>(c) * 2 * KO, pf, own);
            bool ok = true;
            if (c > 0)
                ok = p.lb_depth > 0 ? lookback_trunc_k<KO>(p, slots, p.pc, c, epoch, p.lb_depth, Xc)
                                    : lookback_hier_k<KO>(p, slots, gslots, p.pc, p.pg, c, epoch, own, withhold, Xc);
            if (lane == 0) {
                if (ok && !withhold) {
                    float f[KO];
                    matvec<KO>(p.pc + KO * KO, Xc, f);  // Phi X
#pragma unroll
                    for (int j = 0; j < KO; ++j) f[j] += own[j];
                    publishk<KO>(slots + static_cast<size_t>(c) * 2 * KO + KO, ff, f);
                    if ((c & 31u) == 31u) publishk<KO>(gslots + static_cast<size_t>(c >> 5) * 2 * KO + KO, ff, f);
                }
#pragma unroll
                for (int j = 0; j < KO; ++j) sm.Xc[j] = Xc[j];
                sm.bail = ok ? 0 : 1;
            }
        }
        __syncthreads();  // (B)
        if (sm.bail || !row) return;
        // 5. carry correction and store
#pragma unroll
        for (int v = 0; v < X; ++v) {
            const int i = v * BT + t;
            float acc = val[v];
#pragma unroll
            for (int j = 0; j < KO; ++j) acc = fmaf(__ldg(p.fac + static_cast<size_t>(j) * CHUNK + i), sm.Xc[j], acc);
            const long long gi = cs + i;
            if (gi < p.n) p.y[gi] = acc;
        }
    }
};

template <int KO, int BT, int X>
__global__ void __launch_bounds__(32 + BT) iir_plr_kernel(const __grid_constant__ IirPlrParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    PlrBlock<KO, BT, X>::run(p, smem);
}

// The same merge with a warp per chunk, for order 4 and segments of BT = 256 samples: lane l holds the 8
// consecutive samples 8 l .. 8 l + 7 of each of the chunk's X segments. The doubling's first three levels
// stay inside a lane, and a wider one takes 4 shuffles per segment for a lane's 8 samples (the last 4 of
// the lower half lie in one lane); a lane's factors of a level are read once for all X segments. Every
// sample sees the same factors in the same order as in PlrBlock, so the outputs are the same to the bit.
// (The direct form's own rounding, 2e-5 of the output at order 4, hangs on that order.)
//
// A block holds one copy of the chunk's factors and W warps, which draw chunks until none is left; no
// barrier after the start. Bound by issue and by the latency of a chunk's phases: 54 instructions per sample
// (37 of them multiply-adds) at half of the issue slots. Measured at order 4 against a block per chunk (GB300,
// graph replays, us): 3e6 samples 33.0 -> 16.1, 2^25 334 -> 95.3, 2^27 1320 -> 347.
template <int X>
struct PlrWarp {
    static constexpr int KO = 4, BT = 256, CHUNK = BT * X;
    static constexpr int W = 12;  // three per scheduler: registers for 64 samples, 32 factors and a segment's shuffles
    static constexpr size_t SMEM_BYTES = KO * CHUNK * sizeof(float);

    // 16-byte unit of a factor row that holds samples 4 g .. 4 g + 3: units of neighbouring lanes (two each)
    // on different banks.
    __device__ __forceinline__ static int unit(int g) { return g ^ ((g >> 3) & 1); }

    __device__ __forceinline__ static void load8(const float* tab, int j, int m, float (&f)[8]) {
        const float4* row = reinterpret_cast<const float4*>(tab) + j * (CHUNK / 4);
        const float4 a = row[unit(2 * m)], b = row[unit(2 * m + 1)];
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
        f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }

    __device__ static void run(const IirPlrParams& p, unsigned char* smem_raw) {
        float* tab = reinterpret_cast<float*>(smem_raw);  // [KO][CHUNK], unit()'s order
        const int lane = threadIdx.x & 31;
        for (int i = threadIdx.x; i < KO * CHUNK / 4; i += W * 32) {
            const int j = i / (CHUNK / 4), g = i % (CHUNK / 4);
            reinterpret_cast<float4*>(tab)[j * (CHUNK / 4) + unit(g)] = __ldg(reinterpret_cast<const float4*>(p.fac) + i);
        }
        __syncthreads();
        const float gain = p.gain;
        const bool xvec = (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0, yvec = (reinterpret_cast<uintptr_t>(p.y) & 15u) == 0;
        uint32_t epoch = 0;
        while (true) {
            unsigned long long ticket = 0;
            if (lane == 0) ticket = atomicAdd(&p.state->ticket, 1ull);
            ticket = __shfl_sync(FULL_MASK, ticket, 0);
            epoch = static_cast<uint32_t>(ticket >> 32);
            const uint32_t c = static_cast<uint32_t>(ticket & 0xffffffffull);
            if (c >= p.nchunks) break;
            const long long cs = static_cast<long long>(c) * CHUNK;
            const bool whole = cs + CHUNK <= p.n;
            float val[X][8];
            if (whole && xvec) {
                const float4* src = reinterpret_cast<const float4*>(p.x + cs) + 2 * lane;
#pragma unroll
                for (int v = 0; v < X; ++v) {
                    const float4 a = __ldg(src + v * (BT / 4)), b = __ldg(src + v * (BT / 4) + 1);
                    val[v][0] = a.x; val[v][1] = a.y; val[v][2] = a.z; val[v][3] = a.w;
                    val[v][4] = b.x; val[v][5] = b.y; val[v][6] = b.z; val[v][7] = b.w;
                }
            } else {
#pragma unroll
                for (int v = 0; v < X; ++v)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long long gi = cs + v * BT + 8 * lane + i;
                        val[v][i] = gi < p.n ? __ldg(p.x + gi) : 0.f;
                    }
            }
            // the chunk that some warp draws next but one round, into L2
            const long long ahead = cs + static_cast<long long>(gridDim.x) * W * CHUNK + 32 * lane;
#pragma unroll
            for (int k = 0; k < CHUNK / 1024; ++k)
                if (ahead + 1024 * k < p.n)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.x + ahead + 1024 * k));
            // the 4 samples before the chunk: lane 31's last ones, as a segment before the first would have
            float last[KO];
#pragma unroll
            for (int k = 0; k < KO; ++k) last[k] = (c > 0 && lane == 31) ? __ldg(p.x + cs - KO + k) * gain : 0.f;
            // 1. FIR, and the doubling's levels inside a lane
            float f0[KO][4];  // fac_j[0..3]
#pragma unroll
            for (int j = 0; j < KO; ++j) {
                const float4 a = reinterpret_cast<const float4*>(tab)[j * (CHUNK / 4)];
                f0[j][0] = a.x; f0[j][1] = a.y; f0[j][2] = a.z; f0[j][3] = a.w;
            }
#pragma unroll
            for (int v = 0; v < X; ++v) {
                float xs[KO + 8];
#pragma unroll
                for (int i = 0; i < 8; ++i) xs[KO + i] = val[v][i] * gain;
#pragma unroll
                for (int k = 0; k < KO; ++k) {
                    // from the lane before; lane 0's from lane 31 of the segment before
                    xs[k] = __shfl_sync(FULL_MASK, lane == 31 ? last[k] : xs[8 + k], (lane + 31) & 31);
                }
#pragma unroll
                for (int k = 0; k < KO; ++k) last[k] = xs[8 + k];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float acc = xs[KO + i];
#pragma unroll
                    for (int j = 0; j < KO; ++j) acc = fmaf(p.b[j], xs[KO + i - 1 - j], acc);
                    val[v][i] = acc;
                }
#pragma unroll
                for (int half = 1; half < 8; half <<= 1)
#pragma unroll
                    for (int j = 0; j < KO; ++j) {
                        const int src = half - KO + j;
                        if (src < 0) continue;
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (i & half)
                                val[v][i] = fmaf(f0[j][i & (half - 1)], val[v][(i & ~(2 * half - 1)) + src], val[v][i]);
                    }
            }
            // 2. levels across lanes (one body for all of them: unrolled, the kernel outgrows the instruction cache)
#pragma unroll 1
            for (int hl = 1; hl < 32; hl <<= 1) {
                const int src = (lane & ~(2 * hl - 1)) + hl - 1;
                const bool upper = (lane & hl) != 0;
#pragma unroll
                for (int j = 0; j < KO; ++j) {
                    float f[8], y[X];
                    load8(tab, j, lane & (hl - 1), f);
#pragma unroll
                    for (int v = 0; v < X; ++v) y[v] = __shfl_sync(FULL_MASK, val[v][8 - KO + j], src);
                    if (upper) {
#pragma unroll
                        for (int v = 0; v < X; ++v)
#pragma unroll
                            for (int i = 0; i < 8; ++i) val[v][i] = fmaf(f[i], y[v], val[v][i]);
                    }
                }
            }
            // 3. segment chaining: every lane runs the chain of end states, and corrects its samples
            float L[KO];
#pragma unroll
            for (int t = 0; t < KO; ++t) L[t] = __shfl_sync(FULL_MASK, val[0][8 - KO + t], 31);
            if constexpr (X > 1) {
                float f[KO][8], fe[KO][KO];  // fac_j at the lane's samples, and at the segment's last 4
#pragma unroll
                for (int j = 0; j < KO; ++j) {
                    load8(tab, j, lane, f[j]);
                    const float4 a = reinterpret_cast<const float4*>(tab)[j * (CHUNK / 4) + unit(BT / 4 - 1)];
                    fe[j][0] = a.x; fe[j][1] = a.y; fe[j][2] = a.z; fe[j][3] = a.w;
                }
#pragma unroll
                for (int v = 1; v < X; ++v) {
                    float nl[KO];
#pragma unroll
                    for (int t = 0; t < KO; ++t) {
                        nl[t] = __shfl_sync(FULL_MASK, val[v][8 - KO + t], 31);
#pragma unroll
                        for (int j = 0; j < KO; ++j) nl[t] = fmaf(fe[j][t], L[j], nl[t]);
                    }
#pragma unroll
                    for (int j = 0; j < KO; ++j)
#pragma unroll
                        for (int i = 0; i < 8; ++i) val[v][i] = fmaf(f[j][i], L[j], val[v][i]);
#pragma unroll
                    for (int t = 0; t < KO; ++t) L[t] = nl[t];
                }
            }
            // 4. lookback
            float Xc[KO] = {0.f, 0.f, 0.f, 0.f};
            const bool withhold = static_cast<long long>(c) == p.withhold_chunk;
            const uint32_t pf = 2u * epoch + 1u, ff = 2u * epoch + 2u;
            unsigned long long* slots = p.carry;
            unsigned long long* gslots = p.carry + static_cast<size_t>(p.carry_cap) * 2 * KO;
            if (lane == 0 && !withhold) publishk<KO>(slots + static_cast<size_t>(c) * 2 * KO, pf, L);
            bool ok = true;
            if (c > 0)
                ok = p.lb_depth > 0 ? lookback_trunc_k<KO>(p, slots, p.pc, c, epoch, p.lb_depth, Xc)
                                    : lookback_hier_k<KO>(p, slots, gslots, p.pc, p.pg, c, epoch, L, withhold, Xc);
            if (!ok) break;
            if (lane == 0 && !withhold && p.lb_depth == 0) {
                float g[KO];
                matvec<KO>(p.pc + KO * KO, Xc, g);  // Phi X
#pragma unroll
                for (int j = 0; j < KO; ++j) g[j] += L[j];
                publishk<KO>(slots + static_cast<size_t>(c) * 2 * KO + KO, ff, g);
                if ((c & 31u) == 31u) publishk<KO>(gslots + static_cast<size_t>(c >> 5) * 2 * KO + KO, ff, g);
            }
            // 5. carry correction and store
#pragma unroll
            for (int v = 0; v < X; ++v) {
#pragma unroll
                for (int j = 0; j < KO; ++j) {
                    float f[8];
                    load8(tab, j, v * 32 + lane, f);
#pragma unroll
                    for (int i = 0; i < 8; ++i) val[v][i] = fmaf(f[i], Xc[j], val[v][i]);
                }
                if (whole && yvec) {
                    float4* dst = reinterpret_cast<float4*>(p.y + cs) + v * (BT / 4) + 2 * lane;
                    dst[0] = make_float4(val[v][0], val[v][1], val[v][2], val[v][3]);
                    dst[1] = make_float4(val[v][4], val[v][5], val[v][6], val[v][7]);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long long gi = cs + v * BT + 8 * lane + i;
                        if (gi < p.n) p.y[gi] = val[v][i];
                    }
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // the last block out starts the next epoch (warps draw past the last chunk)
            __threadfence();
            if (atomicAdd(&p.state->done, 1u) == gridDim.x - 1u) {
                atomicExch(&p.state->done, 0u);
                atomicExch(&p.state->ticket, static_cast<unsigned long long>(epoch + 1u) << 32);
                __threadfence();
            }
        }
    }
};

template <int X>
__global__ void __launch_bounds__(PlrWarp<X>::W * 32, 1) iir_plr_warp_kernel(const __grid_constant__ IirPlrParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    PlrWarp<X>::run(p, smem);
}

template <int X>
static void add_plr_warp(std::vector<KernelEntry>& reg) {
    using R = PlrWarp<X>;
    KernelEntry e{IIR_KIND_PLR, R::BT, X, (const void*)iir_plr_warp_kernel<X>, R::W * 32, R::SMEM_BYTES, R::KO, 0};
    e.pipeline = 1;
    reg.push_back(e);
}

template <int KO, int BT, int X>
static void add_plr(std::vector<KernelEntry>& reg) {
    reg.push_back(KernelEntry{IIR_KIND_PLR, BT, X, (const void*)iir_plr_kernel<KO, BT, X>, 32 + BT,
                              PlrBlock<KO, BT, X>::SMEM_BYTES, KO, 0});
}

// Block sizes per order follow the reference's table (plr_kernels.cuh:57-84): the block
// halves as the order doubles so the per-thread carry footprint fits the register budget.
void register_plr(std::vector<KernelEntry>& reg) {
    add_plr<2, 512, 1>(reg);
    add_plr<2, 512, 4>(reg);
    add_plr<2, 512, 8>(reg);
    add_plr<4, 256, 1>(reg);
    add_plr<4, 256, 4>(reg);
    add_plr<4, 256, 8>(reg);
    add_plr_warp<4>(reg);
    add_plr_warp<8>(reg);
    add_plr<8, 128, 1>(reg);
    add_plr<8, 128, 4>(reg);
    add_plr<8, 128, 8>(reg);
    add_plr<16, 64, 1>(reg);
    add_plr<16, 64, 4>(reg);
    add_plr<16, 64, 8>(reg);
}

}  // namespace iirgb

// iir_batch_sweep.cuh — batched segments on the state sweep (iir_sweep.cuh): many independent signals
// in one launch, each with its own cascade, state in and state out.
//
// A warp filters a tile of 32 lane rows with two sweeps, as there: pass A (states that the sub-rows
// leave behind, 2K dot products), scan, pass B (the whole cascade once from the true states). What a
// batch adds:
//   * the launch's work is a list of runs: consecutive tiles of one segment, after the tile ahead of
//     them (filtered for its end state and not stored). A block's loader
//     warp draws a run, puts its tiles and its filter's table into the block's ring of buffers, and
//     draws the next; the filter warps take the tiles in order. The next run's record is read and the
//     one after it drawn while a run's tiles are waited for.
//   * segments start anywhere: the 0..3 samples before the 16-byte grid of x are filtered one by one
//     by the first tile's warp, so that tiles move by 16-byte copies.
//   * a state before the segment enters with its first tile; the state after it is picked out of pass B
//     at the segment's last sample.
// Filters that take longer than a tile to decay keep the lookback kernel (iir_batch.cu).
#pragma once
#include "iir_batch_sweep.h"
#include "iir_sweep.cuh"

namespace iirgb {

// Table of a cascade of K (compiled) sections for lane rows of SPAN samples; offsets in floats.
template <int K_, int SPAN_>
struct BatchSweepGeom {
    static constexpr int K = K_, SPAN = SPAN_, N = bsweep_subrow(K_, SPAN_), R = SPAN / N, D = 2 * K_;
    static constexpr int TILE = 32 * SPAN;
    static_assert(N % 16 == 0 && R % 2 == 0 && SPAN % 32 == 0, "sub-rows in packed pairs, whole 128-byte lines");
    static constexpr int BLOCKS = K * (K + 1) / 2;
    static constexpr int T_A = 0;                             // [D][N] pass A
    static constexpr int T_H = T_A + D * N;                   // [D][2] response to (x[-2], x[-1])
    static constexpr int T_C = T_H + 2 * D;                   // [K][4] b1, b2, a1, a2, then the input gain
    static constexpr int T_W = T_C + 4 * K + 4;               // [K][2] what residuals are held to (sweep_agree)
    static constexpr int T_PN = T_W + ((2 * K + 3) & ~3);     // [BLOCKS] Phi^N
    static constexpr int T_PS = T_PN + 4 * BLOCKS;            // [BSWEEP_STEPS][BLOCKS] Phi^(SPAN 2^k)
    static constexpr int T_PL = T_PS + 4 * BSWEEP_STEPS * BLOCKS;  // [BSWEEP_NEAR][BLOCKS] Phi^(SPAN l), if not chained
    static constexpr int T_LEN = T_PL + (bsweep_chained(K) ? 0 : 4 * BSWEEP_NEAR * BLOCKS);
    static_assert(T_H % 4 == 0 && T_C % 4 == 0 && T_PN % 4 == 0, "16-byte table rows");
};
// Scan across the lanes (as sweep_scan, with a table of powers of two): S = the state before the lane,
// last = the state after it (lane 31: the tile's end state). CHAINED: X, the state before the tile,
// enters as the end state of a lane before lane 0; else the tile starts from rest.
template <class G, bool CHAINED>
__device__ __forceinline__ void bsweep_scan(const float* tab, int rounds, int lane, const float (&f)[G::D],
                                            const float (&X)[G::D], float (&S)[G::D], float (&last)[G::D]) {
    constexpr int D = G::D;
#pragma unroll
    for (int c = 0; c < D; ++c) last[c] = f[c];
#pragma unroll 1
    for (int k = 0; k < rounds; ++k) {
        const int d = 1 << k;
        float o[D];
#pragma unroll
        for (int c = 0; c < D; ++c) {
            o[c] = __shfl_up_sync(FULL_MASK, last[c], d);
            if (lane < d) o[c] = CHAINED && lane == d - 1 ? X[c] : 0.f;
        }
        tri_mad<G::K>(tab + G::T_PS + 4 * k * G::BLOCKS, o, last, last);
    }
#pragma unroll
    for (int c = 0; c < D; ++c) {
        S[c] = __shfl_up_sync(FULL_MASK, last[c], 1);
        if (lane == 0) S[c] = CHAINED ? X[c] : 0.f;
    }
}

// The response to the state X before the tile, Phi^(SPAN lane) X, added to the lanes' states: every
// lane applies the powers of two of its own number.
template <class G>
__device__ __forceinline__ void bsweep_respond(const float* tab, int rounds, int lane, const float (&X)[G::D],
                                              float (&S)[G::D]) {
    constexpr int D = G::D;
    float d[D], zero[D];
#pragma unroll
    for (int c = 0; c < D; ++c) {
        d[c] = X[c];
        zero[c] = 0.f;
    }
#pragma unroll 1
    for (int k = 0; k < rounds; ++k) {
        float y[D];
        tri_mad<G::K>(tab + G::T_PS + 4 * k * G::BLOCKS, d, zero, y);
#pragma unroll
        for (int c = 0; c < D; ++c) d[c] = (lane >> k) & 1 ? y[c] : d[c];
    }
    if (lane < (1 << rounds)) {
#pragma unroll
        for (int c = 0; c < D; ++c) S[c] += d[c];
    }
}

// Pass B (states as in iir_sweep.cuh, sweep_sign). With CAPTURE, the sections' outputs at sample `at` of this lane's row (-1: not here) and the one before it go to zf[2 s],
// zf[2 s + 1], s < kreal.
template <class G, bool CAPTURE>
__device__ __forceinline__ void bsweep_run(float* buf, const float* tab, int lane, const float (&st)[G::R][G::D],
                                           const float (&xh)[G::R][2], float (&end)[G::R][G::D], int at = -1,
                                           float* zf = nullptr, int kreal = 0) {
    constexpr int K = G::K, N = G::N, R = G::R, P = R / 2;
    float* line = buf + (lane << 5);
    const int l7 = lane & 7;
    f32x2 b1[K], b2[K], a1[K], a2[K];
    float sg[K];
#pragma unroll
    for (int s = 0; s < K; ++s) {
        const float4 c = *reinterpret_cast<const float4*>(tab + G::T_C + 4 * s);
        sg[s] = sweep_sign(c.z);
        b1[s] = pack2(c.x, c.x);
        b2[s] = pack2(c.y, c.y);
        a1[s] = pack2(c.z, c.z);
        a2[s] = pack2(c.w, c.w);
    }
    const float gain = tab[G::T_C + 4 * K];
    const f32x2 g = pack2(gain, gain);
    // h[p][0]: input history; h[p][s + 1]: section s's output history; [..][0] = n - 2, [..][1] = n - 1
    f32x2 h[P][K + 1][2];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            h[p][0][t] = mul2(g, pack2(xh[2 * p][t], xh[2 * p + 1][t]));
#pragma unroll
            for (int s = 0; s < K; ++s) {
                const float* u = st[2 * p] + 2 * s;
                const float* w = st[2 * p + 1] + 2 * s;
                h[p][s + 1][t] = t == 0 ? pack2(sg[s] * (u[1] - u[0]), sg[s] * (w[1] - w[0])) : pack2(u[1], w[1]);
            }
        }
#pragma unroll(K > 4 ? 1 : 2)
    for (int j = 0; j < N / 4; ++j) {
        float4 x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = *reinterpret_cast<const float4*>(line + sub_granule_at<N>(i, j, l7));
        // v[p][s][t]: section s's input (s = K: the output) at samples t - 2, t = 0..5. Four samples go
        // through the sections along the diagonals (sample + section), whose steps do not depend on
        // one another.
        f32x2 v[P][K + 1][6];
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int s = 0; s <= K; ++s) {
                v[p][s][0] = h[p][s][0];
                v[p][s][1] = h[p][s][1];
            }
            v[p][0][2] = mul2(g, pack2(x[2 * p].x, x[2 * p + 1].x));
            v[p][0][3] = mul2(g, pack2(x[2 * p].y, x[2 * p + 1].y));
            v[p][0][4] = mul2(g, pack2(x[2 * p].z, x[2 * p + 1].z));
            v[p][0][5] = mul2(g, pack2(x[2 * p].w, x[2 * p + 1].w));
        }
#pragma unroll
        for (int d = 0; d < K + 3; ++d) {
#pragma unroll
            for (int s = 0; s < K; ++s) {
                const int t = d - s + 2;
                if (t < 2 || t > 5) continue;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const f32x2 w = fma2(b2[s], v[p][s][t - 2], fma2(b1[s], v[p][s][t - 1], v[p][s][t]));
                    v[p][s + 1][t] = fma2(a1[s], v[p][s + 1][t - 1], fma2(a2[s], v[p][s + 1][t - 2], w));
                }
            }
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int s = 0; s <= K; ++s) {
                h[p][s][0] = v[p][s][4];
                h[p][s][1] = v[p][s][5];
            }
            unpack2(v[p][K][2], x[2 * p].x, x[2 * p + 1].x);
            unpack2(v[p][K][3], x[2 * p].y, x[2 * p + 1].y);
            unpack2(v[p][K][4], x[2 * p].z, x[2 * p + 1].z);
            unpack2(v[p][K][5], x[2 * p].w, x[2 * p + 1].w);
        }
#pragma unroll
        for (int i = 0; i < R; ++i) *reinterpret_cast<float4*>(line + sub_granule_at<N>(i, j, l7)) = x[i];
        if constexpr (CAPTURE) {
            if (at >= 0 && (at % N) / 4 == j) {
                const bool odd = ((at / N) & 1) != 0;
                const int pm = at / (2 * N), tm = (at & 3) + 2;
#pragma unroll
                for (int s = 0; s < K; ++s) {
                    f32x2 y2 = 0ull, y1 = 0ull;
#pragma unroll
                    for (int p = 0; p < P; ++p)
#pragma unroll
                        for (int t = 2; t < 6; ++t) {
                            const bool here = p == pm && t == tm;
                            y2 = here ? v[p][s + 1][t - 1] : y2;
                            y1 = here ? v[p][s + 1][t] : y1;
                        }
                    float a0, c0, a1f, c1;
                    unpack2(y2, a0, c0);
                    unpack2(y1, a1f, c1);
                    if (s < kreal) {
                        zf[2 * s] = odd ? c0 : a0;
                        zf[2 * s + 1] = odd ? c1 : a1f;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int s = 0; s < K; ++s) {
            float ya, yb, za, zb;
            unpack2(h[p][s + 1][1], ya, yb);
            unpack2(h[p][s + 1][0], za, zb);
            end[2 * p][2 * s] = fmaf(-sg[s], za, ya);
            end[2 * p + 1][2 * s] = fmaf(-sg[s], zb, yb);
            end[2 * p][2 * s + 1] = ya;
            end[2 * p + 1][2 * s + 1] = yb;
        }
}
// The sections' states after sample m of the tile, to zf[2 s], zf[2 s + 1], s < kreal, ahead of pass B: its
// steps once more from the start of m's sub-row, by every lane alike (bound by their latency: at most N
// samples, about a microsecond per segment). bsweep_run's CAPTURE takes a second copy of pass B in the
// kernel; 1024 segments of 33600 samples, order 8, with states: 99 us with it, 89 with this. The kernel of
// up to 8 sections captures all the same: there these steps cost every tile registers (order 16, mixed
// lengths: 506 us against 476).
template <class G>
__device__ __forceinline__ void bsweep_state(const float* buf, const float* tab, int lane, int m,
                                             const float (&st)[G::R][G::D], const float (&xh)[G::R][2], float* zf,
                                             int kreal) {
    constexpr int K = G::K, N = G::N, R = G::R, D = G::D;
    const int row = m / G::SPAN, sub = (m % G::SPAN) / N;
    float S[D], h2 = 0.f, h1 = 0.f, y2[K], y1[K];
#pragma unroll
    for (int c = 0; c < D; ++c) S[c] = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (i == sub) {
            h2 = xh[i][0];
            h1 = xh[i][1];
#pragma unroll
            for (int c = 0; c < D; ++c) S[c] = st[i][c];
        }
    h2 = __shfl_sync(FULL_MASK, h2, row);
    h1 = __shfl_sync(FULL_MASK, h1, row);
#pragma unroll
    for (int s = 0; s < K; ++s) {
        const float d = __shfl_sync(FULL_MASK, S[2 * s], row), u = __shfl_sync(FULL_MASK, S[2 * s + 1], row);
        y2[s] = sweep_sign(tab[G::T_C + 4 * s + 2]) * (u - d);
        y1[s] = u;
    }
    const float gain = tab[G::T_C + 4 * K];
    h2 *= gain;
    h1 *= gain;
#pragma unroll 1
    for (int n = sub * N; n <= m % G::SPAN; ++n) {
        float w = gain * buf[tile_at(row, n)], g2 = h2, g1 = h1;
        h2 = h1;
        h1 = w;
#pragma unroll
        for (int s = 0; s < K; ++s) {
            const float4 c = *reinterpret_cast<const float4*>(tab + G::T_C + 4 * s);
            w = fmaf(c.y, g2, fmaf(c.x, g1, w));
            g2 = y2[s];
            g1 = y1[s];
            w = fmaf(c.z, g1, fmaf(c.w, g2, w));
            y2[s] = g1;
            y1[s] = w;
        }
    }
#pragma unroll
    for (int s = 0; s < K; ++s)
        if (lane == 0 && s < kreal) {
            zf[2 * s] = y2[s];
            zf[2 * s + 1] = y1[s];
        }
    __syncwarp();  // every lane has read the samples
}

// The same after the states were found to lack g: the response to g at sample m is added to zf, by lane `by`.
template <class G>
__device__ __forceinline__ void bsweep_state_fix(const float* tab, int lane, int m, const float (&g)[G::R][G::D], float* zf,
                                                 int kreal, int by) {
    constexpr int K = G::K, N = G::N, R = G::R, D = G::D;
    const int row = m / G::SPAN, sub = (m % G::SPAN) / N;
    float S[D], y2[K], y1[K];
#pragma unroll
    for (int c = 0; c < D; ++c) {
        S[c] = 0.f;
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (i == sub) S[c] = g[i][c];
        S[c] = __shfl_sync(FULL_MASK, S[c], row);
    }
#pragma unroll
    for (int s = 0; s < K; ++s) {
        y2[s] = sweep_sign(tab[G::T_C + 4 * s + 2]) * (S[2 * s + 1] - S[2 * s]);
        y1[s] = S[2 * s + 1];
    }
#pragma unroll 1
    for (int n = sub * N; n <= m % G::SPAN; ++n) {
        float w = 0.f, g2 = 0.f, g1 = 0.f;
#pragma unroll
        for (int s = 0; s < K; ++s) {
            const float4 c = *reinterpret_cast<const float4*>(tab + G::T_C + 4 * s);
            w = fmaf(c.y, g2, fmaf(c.x, g1, w));
            g2 = y2[s];
            g1 = y1[s];
            w = fmaf(c.z, g1, fmaf(c.w, g2, w));
            y2[s] = g1;
            y1[s] = w;
        }
    }
#pragma unroll
    for (int s = 0; s < K; ++s)
        if (lane == by && s < kreal) {
            zf[2 * s] += y2[s];
            zf[2 * s + 1] += y1[s];
        }
}

// The two steps of a correction (iir_sweep.cuh, sweep_lack and sweep_apply).
template <class G>
__device__ __noinline__ void bsweep_lack(const float* tab, int rounds, int lane, const float (&r)[G::R][G::D],
                                         float (&g)[G::D], float (&last)[G::D]) {
    float f[G::D], none[G::D] = {};
    sweep_join<G>(tab, r, f);
    bsweep_scan<G, false>(tab, rounds, lane, f, none, g, last);
}
// before: what the tile's incoming state lacks, or null; zf: the segment's states, if its last sample m is here, or null.
template <class G>
__device__ __noinline__ void bsweep_apply(float* buf, const float* tab, int rounds, int lane, const float (&r)[G::R][G::D],
                                          const float (&g0)[G::D], const float* before, int m, float* zf, int kreal, int by) {
    float g[G::R][G::D];
#pragma unroll
    for (int c = 0; c < G::D; ++c) g[0][c] = g0[c];
    if (before) {
        float X[G::D];
#pragma unroll
        for (int c = 0; c < G::D; ++c) X[c] = before[c];
        bsweep_respond<G>(tab, rounds, lane, X, g[0]);
    }
#pragma unroll
    for (int j = 1; j < G::R; ++j) tri_mad<G::K>(tab + G::T_PN, g[j - 1], r[j - 1], g[j]);
    sweep_respond<G>(buf, [&](int s) { return *reinterpret_cast<const float4*>(tab + G::T_C + 4 * s); }, lane, g);
    if (zf) bsweep_state_fix<G>(tab, lane, m, g, zf, kreal, by);
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int x, int y, int z, const void* src) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(z), "r"(smem_u32(src))
                 : "memory");
}
// Bytes announced on a barrier without arriving.
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

constexpr unsigned BSWEEP_WARM = 0x80000000u, BSWEEP_FIRST = 0x40000000u;

constexpr int BSWEEP_COPIERS = 3;
constexpr unsigned BSWEEP_SLEEP = 32;  // ns between two looks of a waiting warp

template <int NB>
struct BatchSweepAux {
    // Item and run records are written at most AHEAD items before the copies: with NB items in flight
    // after those, none is overwritten in use.
    static constexpr unsigned RING = 32, RUNS = 32, AHEAD = 12;
    static_assert(NB + AHEAD + BSWEEP_COPIERS < 32, "records of the items in flight");
    BatchRun runs[RUNS];                     // the last runs begun
    unsigned long long full[NB], empty[NB];
    float ends[RING][2 * IIR_MAX_SECTIONS];  // items' end states
    float fix[RING][2 * IIR_MAX_SECTIONS];   // what they lack, where it matters
    unsigned int item_run[RING];             // the item's run ...
    unsigned int item[RING];                 // ... and tile, BSWEEP_WARM (only its end state is wanted), BSWEEP_FIRST
    volatile unsigned int ready[RING];       // i + 1 once item i's end state is in `ends`
    volatile unsigned int checked[RING];     // 2 (i + 1) once it has been checked, plus 1 if `fix` is to be added
    volatile unsigned int issued[NB];        // items put into the buffer so far
    unsigned int tag[NB];                    // the filter whose table the buffer holds (copiers)
    volatile unsigned int copied[BSWEEP_COPIERS];  // 1 + the last item that the copier has issued
    volatile unsigned int recorded;          // items recorded so far
    volatile unsigned int total;             // items of the block, once known
    volatile unsigned int abandon;           // a wait ran out: everybody leaves
    unsigned int next;                       // next item for a free warp
};

// Every wait of a block is bounded; the first to run out sends the whole block home.
template <class Aux, class Cond>
__device__ __forceinline__ bool bsweep_wait(Aux& aux, const IirBatchSweepParams& p, Cond&& cond,
                                            uint32_t code = IIR_DEV_ERR_MBARRIER) {
    if (cond()) return true;
    const uint64_t start = globaltimer_ns();
    uint32_t spins = 0;
    while (!cond()) {
        __nanosleep(BSWEEP_SLEEP);  // leaves the issue slots to the warps that filter
        if ((++spins & 63u) != 0u) continue;
        if (aux.abandon) return false;
        if (globaltimer_ns() - start > static_cast<uint64_t>(p.timeout_ns)) {
            aux.abandon = 1u;
            raise_error(p.state, sweep_epoch(p.state), code);
            return false;
        }
    }
    return true;
}

// This lane's earlier cp.async copies arrive on the barrier when they are done.
__device__ __forceinline__ void cp_async_arrive(unsigned long long* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Dealer warp: draws runs, one or two at a time (one word of a record per lane), and writes down the items
// that they consist of.
template <int NB>
__device__ __forceinline__ void bsweep_dealer(const IirBatchSweepParams& p, BatchSweepAux<NB>& aux) {
    using Aux = BatchSweepAux<NB>;
    const int lane = threadIdx.x & 31;
    const unsigned unit = p.unit;
    auto records = [&](unsigned draw) {
        const unsigned half = lane >> 4, run = unit * draw + half;
        return half < unit && run < p.nruns ? __ldg(reinterpret_cast<const unsigned*>(p.runs + run) + (lane & 15)) : 0u;
    };
    const unsigned ndraws = (p.nruns + unit - 1u) / unit;
    // a block's first two draws are its own, the others come from a counter; the records of the next one
    // are read and the one after it drawn while this one is dealt
    unsigned cur = blockIdx.x, nxt = blockIdx.x + gridDim.x, i = 0, r = 0;
    unsigned words = records(cur);
    while (cur < ndraws) {
        const unsigned mine = words;
        words = records(nxt);
        unsigned ticket = 0;
        if (lane == 0 && nxt < ndraws) ticket = atomicAdd(&p.state->runs, 1u);
        for (unsigned h = 0; h < unit && unit * cur + h < p.nruns; ++h, ++r) {
            // (the record's slot is free: the items of the run 32 runs ago are long done)
            BatchRun& run = aux.runs[r % Aux::RUNS];
            if ((lane >> 4) == static_cast<int>(h)) reinterpret_cast<unsigned*>(&run)[lane & 15] = mine;
            __syncwarp();
            const unsigned tile0 = run.tile0, first = tile0 - run.warm, end = tile0 + run.count;
            for (unsigned t = first; t < end; ++t, ++i) {
                const bool ok = bsweep_wait(aux, p, [&] {
                    bool far = false;
                    for (int c = 0; c < BSWEEP_COPIERS; ++c) far |= aux.copied[c] + Aux::AHEAD < i;
                    return !far;
                });
                if (__any_sync(FULL_MASK, !ok)) return;
                if (lane == 0) {
                    aux.item_run[i % Aux::RING] = r;
                    aux.item[i % Aux::RING] = t | (t < tile0 ? BSWEEP_WARM : 0u) | (t == first ? BSWEEP_FIRST : 0u);
                    __threadfence_block();  // the record before the count
                    aux.recorded = i + 1u;
                }
            }
            __syncwarp();
        }
        cur = nxt;
        nxt = 2u * gridDim.x + __shfl_sync(FULL_MASK, ticket, 0);
    }
    if (lane == 0) {
        __threadfence_block();
        aux.total = i;
    }
}

// Copier warp c: puts the tiles of items c, c + BSWEEP_COPIERS, ... into the ring, whole ones by tensor
// copies of one lane, a segment's last, partial one by 16-byte cp.async copies, with the filter's table where the buffer does not hold it already.
template <int SPAN, int NB>
__device__ __forceinline__ void bsweep_copier(const IirBatchSweepParams& p, BatchSweepAux<NB>& aux, int c, float* bufs,
                                              float* tabs, int tab_stride) {
    constexpr int TILE = 32 * SPAN;
    using Aux = BatchSweepAux<NB>;
    const int lane = threadIdx.x & 31;
    for (unsigned i = c;; i += BSWEEP_COPIERS) {
        const unsigned b = i % NB;
        const bool ok = bsweep_wait(aux, p, [&] { return aux.total <= i || aux.recorded > i; });
        if (__any_sync(FULL_MASK, !ok || aux.total <= i)) break;
        // the buffer's item before, another copier's, has been issued (until then the barrier may be two
        // phases back, and a parity cannot tell those apart) and given back
        if (i >= NB && __any_sync(FULL_MASK, !bsweep_wait(aux, p, [&] {
                return aux.issued[b] == i / NB && mbar_try_wait(aux.empty + b, (i / NB - 1u) & 1u);
            })))
            return;
        __threadfence_block();
        const BatchRun& run = aux.runs[aux.item_run[i % Aux::RING] % Aux::RUNS];
        const unsigned t = aux.item[i % Aux::RING] & ~(BSWEEP_WARM | BSWEEP_FIRST);
        const long long base = static_cast<long long>(t) * TILE, left = run.n - base;
        const int have = left < TILE ? static_cast<int>(left) : TILE;
        const unsigned table = run.table;
        if (aux.tag[b] != table) {
            const int granules = bsweep_table_floats(bsweep_sections(run.K), SPAN) / 4;
            float* dst = tabs + static_cast<size_t>(b) * tab_stride;
            for (int q = lane; q < granules; q += 32) cp_async16(dst + 4 * q, p.tables + table + q);
        }
        float* buf = bufs + static_cast<size_t>(b) * TILE;
        const float* src = run.x + base;
        if (p.use_tma && have == TILE) {
            if (lane == 0) {
                const int g = static_cast<int>((src - p.x0) >> 2);
                mbar_expect_tx(aux.full + b, TILE * 4u);
#pragma unroll
                for (int h = 0; h < SPAN / 32; ++h)
                    tma_load_3d(buf + h * 1024, &p.tmap_x, 0, g + 8 * h, 0, aux.full + b);
            }
        } else {
            constexpr int G = SPAN / 4;  // granules of a lane row
            for (int q = lane; q < have / 4; q += 32) {
                const int row = q / G, k = q % G;
                cp_async16(buf + (row << 5) + ((k >> 3) << 10) + (((k & 7) ^ (row & 7)) << 2), src + 4 * q);
            }
        }
        cp_async_arrive(aux.full + b);
        __syncwarp();
        if (lane == 0) {
            aux.tag[b] = table;
            aux.issued[b] = i / NB + 1u;
            aux.copied[c] = i + 1u;
        }
        __syncwarp();
    }
    if (lane == 0) aux.copied[c] = 0x7fffffffu;  // nothing left for this copier to hold up
}

// One item: the tile in `buf`, whose load has been issued. wait_tile(): it is there; wait_ready(): the item
// before has its end state; wait_checked(): and it has been checked. Returns false when a wait ran out. CAPTURE: how the segment's states are found
// (bsweep_state).
template <class G, int NB, bool CAPTURE, class Tile, class Ready, class Checked>
__device__ __forceinline__ bool bsweep_item(const IirBatchSweepParams& p, BatchSweepAux<NB>& aux, float* buf,
                                            const float* tab, const BatchRun& run, unsigned i, unsigned rec,
                                            Tile&& wait_tile, Ready&& wait_ready, Checked&& wait_checked) {
    constexpr int SPAN = G::SPAN, TILE = G::TILE, R = G::R, K = G::K, D = G::D;
    using Aux = BatchSweepAux<NB>;
    const int lane = threadIdx.x & 31;
    const unsigned t = rec & ~(BSWEEP_WARM | BSWEEP_FIRST);
    const bool warm = (rec & BSWEEP_WARM) != 0u, first = (rec & BSWEEP_FIRST) != 0u;
    const float* x = run.x;
    const long long base = static_cast<long long>(t) * TILE, left = run.n - base;
    const int have = left < TILE ? static_cast<int>(left) : TILE;
    // the two samples before the tile, and the last ones of a segment whose length is not a multiple of
    // four (copies move 16 bytes), on their way while the tile is waited for
    float g2 = 0.f, g1 = 0.f, tail = 0.f, z1 = 0.f;
    if (t > 0) {
        g2 = __ldg(x + base - 2);
        g1 = __ldg(x + base - 1);
    }
    const int q = (have & ~3) + lane;
    if (lane < (have & 3)) tail = __ldg(x + base + q);
    if (!wait_tile()) return false;
    if (lane < (have & 3)) buf[tile_at(q / SPAN, q % SPAN)] = tail;
    float X[D];  // the state before the tile
#pragma unroll
    for (int c = 0; c < D; ++c) X[c] = 0.f;
    if (t == 0) {
        const int kreal = run.K;
        float y2[K], y1[K];
#pragma unroll
        for (int s = 0; s < K; ++s) y2[s] = y1[s] = 0.f;
        if (run.zi) {
            g2 = run.zi[0];
            g1 = z1 = run.zi[1];
#pragma unroll
            for (int s = 0; s < K; ++s)
                if (s < kreal) {
                    y2[s] = run.zi[2 + 2 * s];
                    y1[s] = run.zi[3 + 2 * s];
                }
#pragma unroll
            for (int s = 1; s < K; ++s)
                if (s >= kreal) {  // a section that passes its input on
                    y2[s] = y2[s - 1];
                    y1[s] = y1[s - 1];
                }
        }
        // the samples before the 16-byte grid, one by one
        for (int k = -static_cast<int>(run.peel); k < 0; ++k) {
            const float xv = __ldg(x + k), gain = tab[G::T_C + 4 * K];
            float w = gain * xv, h2 = gain * g2, h1 = gain * g1;
#pragma unroll
            for (int s = 0; s < K; ++s) {
                const float4 c = *reinterpret_cast<const float4*>(tab + G::T_C + 4 * s);
                w = fmaf(c.y, h2, fmaf(c.x, h1, w));
                h2 = y2[s];
                h1 = y1[s];
                w = fmaf(c.z, h1, fmaf(c.w, h2, w));
                y2[s] = h1;
                y1[s] = w;
            }
            g2 = g1;
            g1 = xv;
            if (lane == 0 && !warm) run.y[k] = w;
        }
#pragma unroll
        for (int s = 0; s < K; ++s) {
            X[2 * s] = fmaf(-sweep_sign(tab[G::T_C + 4 * s + 2]), y2[s], y1[s]);
            X[2 * s + 1] = y1[s];
            if (run.zf && have == 0 && lane == 0 && s < kreal) {  // nothing but the peeled samples
                run.zf[2 + 2 * s] = y2[s];
                run.zf[3 + 2 * s] = y1[s];
            }
        }
    }
    __syncwarp();
    float e[R][D], st[R][D], xh[R][2];
    sweep_ends<G>(buf, tab, lane, g2, g1, e, xh);
    {
        float f[D], last[D];
        sweep_join<G>(tab, e, f);
        auto before = [&] {  // X from the item before (a run's first item has it, or starts from rest)
            if (first) return true;
            if (!wait_ready()) return false;
#pragma unroll
            for (int c = 0; c < D; c += 2) {
                const float2 v = *reinterpret_cast<const float2*>(&aux.ends[(i - 1u) % Aux::RING][c]);
                X[c] = v.x;
                X[c + 1] = v.y;
            }
            return true;
        };
        auto publish = [&] {
            if (lane == 31) {
#pragma unroll
                for (int c = 0; c < D; c += 2)
                    *reinterpret_cast<float2*>(&aux.ends[i % Aux::RING][c]) = make_float2(last[c], last[c + 1]);
                __threadfence_block();
                if (t != run.withhold) aux.ready[i % Aux::RING] = i + 1u;
            }
        };
        if constexpr (bsweep_chained(K)) {
            if (!before()) return false;
            bsweep_scan<G, true>(tab, run.rounds, lane, f, X, st[0], last);
            publish();
        } else {
            bsweep_scan<G, false>(tab, run.rounds, lane, f, X, st[0], last);
            publish();
            if (!warm) {
                if (!before()) return false;
                if ((1 << run.rounds) <= BSWEEP_NEAR) {
                    if (lane < (1 << run.rounds)) tri_mad<K>(tab + G::T_PL + 4 * lane * G::BLOCKS, X, st[0], st[0]);
                } else {
                    bsweep_respond<G>(tab, run.rounds, lane, X, st[0]);
                }
            }
        }
    }
#pragma unroll
    for (int j = 1; j < R; ++j) tri_mad<K>(tab + G::T_PN, st[j - 1], e[j - 1], st[j]);
    __syncwarp();  // every lane has read its neighbour's last samples
    const int m = have - 1;  // the segment's last sample, if it is here
    const bool ends = run.zf && left <= TILE;
    float end[R][D];
    if constexpr (CAPTURE) {
        if (ends)
            bsweep_run<G, true>(buf, tab, lane, st, xh, end, m >= 0 && m / SPAN == lane ? m % SPAN : -1, run.zf + 2, run.K);
        else
            bsweep_run<G, false>(buf, tab, lane, st, xh, end);
    } else {
        if (ends && m >= 0) bsweep_state<G>(buf, tab, lane, m, st, xh, run.zf + 2, run.K);
        bsweep_run<G, false>(buf, tab, lane, st, xh, end);
    }
    {
        // the states checked and corrected (iir_sweep.cuh, sweep_agree)
        float r[R][D];
        const bool off = !sweep_agree<G, (K > 4)>([&](int s) { return *reinterpret_cast<const float2*>(tab + G::T_W + 2 * s); }, lane,
                                         have, end, st, aux.ends[i % Aux::RING], r);
        float gs[D];
#pragma unroll
        for (int c = 0; c < D; ++c) gs[c] = 0.f;
        if (off) {
            float rr[R][D], g0[D], last[D];  // (copies: their addresses go to a call, the others stay in registers)
#pragma unroll
            for (int q = 0; q < R; ++q)
#pragma unroll
                for (int c = 0; c < D; ++c) rr[q][c] = r[q][c];
            bsweep_lack<G>(tab, run.rounds, lane, rr, g0, last);
#pragma unroll
            for (int c = 0; c < D; ++c) gs[c] = g0[c];
            if (lane == 31) {
#pragma unroll
                for (int c = 0; c < D; c += 2)
                    *reinterpret_cast<float2*>(&aux.fix[i % Aux::RING][c]) = make_float2(last[c], last[c + 1]);
            }
        }
        if (lane == 31) {
            __threadfence_block();
            aux.checked[i % Aux::RING] = 2u * (i + 1u) + (off ? 1u : 0u);
        }
        if (warm) {
            fence_proxy_async_smem();  // generic accesses of the buffer before the async ones to come
            return true;
        }
        bool before = false;  // the state before the tile lacked something
        if (!first) {
            if (!wait_checked()) return false;
            before = (aux.checked[(i - 1u) % Aux::RING] & 1u) != 0u;
        }
        if (off || before) {
            float rr[R][D], g0[D];
#pragma unroll
            for (int c = 0; c < D; ++c) {
                g0[c] = gs[c];
#pragma unroll
                for (int q = 0; q < R; ++q) rr[q][c] = off ? r[q][c] : 0.f;
            }
            bsweep_apply<G>(buf, tab, run.rounds, lane, rr, g0, before ? aux.fix[(i - 1u) % Aux::RING] : nullptr, m,
                            ends && m >= 0 ? run.zf + 2 : nullptr, run.K, CAPTURE ? m / SPAN : 0);
        }
    }
    if (ends) {
        __syncwarp();
        if (lane == 0) {
            const long long end = run.n;  // raw input history
            run.zf[1] = end + run.peel >= 1 ? __ldg(x + end - 1) : z1;
            run.zf[0] = end + run.peel >= 2 ? __ldg(x + end - 2) : z1;
            // the last section's state is the output as it is written
            if (m >= 0) run.zf[2 * run.K + 1] = buf[tile_at(m / SPAN, m % SPAN)];
            if (m >= 1) run.zf[2 * run.K] = buf[tile_at((m - 1) / SPAN, (m - 1) % SPAN)];
        }
    }
    fence_proxy_async_smem();  // generic accesses of the buffer before the async ones to come
    __syncwarp();
    // the output: a whole tile by tensor copies, a partial one by 16-byte stores where y is on the grid,
    // sample by sample elsewhere
    float* y = run.y + base;
    const bool grid = (reinterpret_cast<uintptr_t>(y) & 15u) == 0;
    if (p.use_tma && grid && have == TILE) {
        if (lane == 0) {
            const int g = static_cast<int>((y - p.y0) >> 2);
#pragma unroll
            for (int h = 0; h < SPAN / 32; ++h) tma_store_3d(&p.tmap_y, 0, g + 8 * h, 0, buf + h * 1024);
            bulk_commit();
        }
    } else if (grid) {
#pragma unroll 4
        for (int g = lane; g < have / 4; g += 32) {
            const int row = g / (SPAN / 4), c = g % (SPAN / 4);
            reinterpret_cast<float4*>(y)[g] =
                *reinterpret_cast<const float4*>(buf + (row << 5) + ((c >> 3) << 10) + (((c & 7) ^ (row & 7)) << 2));
        }
        if (lane < (have & 3)) y[q] = buf[tile_at(q / SPAN, q % SPAN)];
    } else {
#pragma unroll 8
        for (int g = lane; g < have; g += 32) y[g] = buf[tile_at(g / SPAN, g % SPAN)];
    }
    return true;
}

// Blocks of W filter warps, a dealer and three copier warps (one warp issues a tile's 32 copies in about
// a microsecond, which is what an SM's share of a tile takes to filter). Item i lies in buffer i % NB; a warp takes the block's next
// item when it is free.
template <int MAXK, int SPAN, int W, int NB>
__global__ void __launch_bounds__((W + 1 + BSWEEP_COPIERS) * 32) iir_batch_sweep_kernel(const __grid_constant__ IirBatchSweepParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int TILE = 32 * SPAN, TAB = bsweep_table_capacity(MAXK, SPAN);
    using Aux = BatchSweepAux<NB>;
    static_assert(NB >= W, "a buffer per warp");
    float* bufs = reinterpret_cast<float*>(smem);
    float* tabs = bufs + NB * TILE;
    Aux& aux = *reinterpret_cast<Aux*>(tabs + NB * TAB);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == W * 32) {
        for (int b = 0; b < NB; ++b) {
            mbar_init(aux.full + b, 32);
            mbar_init(aux.empty + b, 1);
            aux.issued[b] = 0u;
            aux.tag[b] = 0xffffffffu;
        }
        for (unsigned i = 0; i < Aux::RING; ++i) aux.ready[i] = aux.checked[i] = 0u;
        for (int c = 0; c < BSWEEP_COPIERS; ++c) aux.copied[c] = 0u;
        aux.next = 0u;
        aux.recorded = 0u;
        aux.total = 0xffffffffu;
        aux.abandon = 0u;
        fence_mbar_init();
    }
    __syncthreads();
    if (warp == W) {
        bsweep_dealer<NB>(p, aux);
    } else if (warp > W) {
        bsweep_copier<SPAN, NB>(p, aux, warp - W - 1, bufs, tabs, TAB);
    } else {
        while (true) {
            unsigned i = 0;
            if (lane == 0) i = atomicAdd(&aux.next, 1u);
            i = __shfl_sync(FULL_MASK, i, 0);
            const unsigned b = i % NB;
            // The barrier is looked at only once the item's own load has been issued: until then it may be
            // two phases back, and a parity cannot tell those apart.
            auto issued = [&] { return aux.issued[b] == i / NB + 1u; };
            auto there = [&] { return mbar_try_wait(aux.full + b, (i / NB) & 1u); };
            const bool in = bsweep_wait(aux, p, [&] { return aux.total <= i || issued(); });
            if (__any_sync(FULL_MASK, !in || aux.total <= i)) break;
            __threadfence_block();
            const unsigned rec = aux.item[i % Aux::RING];
            const BatchRun& run = aux.runs[aux.item_run[i % Aux::RING] % Aux::RUNS];
            float* buf = bufs + static_cast<size_t>(b) * TILE;
            const float* tab = tabs + static_cast<size_t>(b) * TAB;
            auto tile = [&] {
                const bool got = bsweep_wait(aux, p, there);
                return !__any_sync(FULL_MASK, !got);
            };
            auto ready = [&] {
                const bool got =
                    bsweep_wait(aux, p, [&] { return aux.ready[(i - 1u) % Aux::RING] == i; }, IIR_DEV_ERR_TIMEOUT);
                __threadfence_block();
                return !__any_sync(FULL_MASK, !got);
            };
            auto checked = [&] {
                const bool got =
                    bsweep_wait(aux, p, [&] { return aux.checked[(i - 1u) % Aux::RING] >> 1 == i; }, IIR_DEV_ERR_TIMEOUT);
                __threadfence_block();
                return !__any_sync(FULL_MASK, !got);
            };
            bool ok = false;
            switch (run.K) {
#define IIR_BSWEEP_CASE(KP)                                                                                  \
    if constexpr (KP <= MAXK)                                                                                 \
        ok = bsweep_item<BatchSweepGeom<KP, SPAN>, NB, (MAXK > 4)>(p, aux, buf, tab, run, i, rec, tile, ready, checked);  \
    break;
                case 1: IIR_BSWEEP_CASE(1)
                case 2: IIR_BSWEEP_CASE(2)
                case 3: IIR_BSWEEP_CASE(3)
                case 4: IIR_BSWEEP_CASE(4)
                case 5:
                case 6: IIR_BSWEEP_CASE(6)
                case 7:
                case 8: IIR_BSWEEP_CASE(8)
#undef IIR_BSWEEP_CASE
                default: break;
            }
            if (!ok) break;
            __syncwarp();
            // The buffer goes back as soon as the store has read it: there are few of them, each with a table
            // (giving it back during the next item costs 12% at order 8).
            if (lane == 0) {
                bulk_wait_read_all();
                mbar_arrive(aux.empty + b);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // loads still in flight (a stopped block) land before the block leaves (iir_sweep.cuh, sweep_tiles)
        if (aux.abandon)
            for (int b = 0; b < NB; ++b)
                if (aux.issued[b] > 0u) (void)wait_mbar_bounded(aux.full + b, (aux.issued[b] - 1u) & 1u, IIR_DRAIN_NS);
        sweep_finish(p.state);
    }
}

template <int MAXK, int SPAN, int NB>
constexpr size_t bsweep_smem() {
    return NB * (size_t(32 * SPAN) + bsweep_table_capacity(MAXK, SPAN)) * 4 + sizeof(BatchSweepAux<NB>);
}

}  // namespace iirgb

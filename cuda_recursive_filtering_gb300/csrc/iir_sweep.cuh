// iir_sweep.cuh — the state-sweep schedule: cascades whose state decays within a tile (a few
// thousand samples), one warp per tile.
//
// A warp owns a tile of 32 lane rows, SPAN = R x N consecutive samples per lane, staged in shared
// memory by TMA. The signal is swept twice:
//   pass A  every lane computes, for each of its R sub-rows of N samples, the state of all K sections
//           that the sub-row leaves behind when it starts from rest: 2K dot products of the N samples
//           with impulse-response tables (2K multiply-adds per sample, no recurrence);
//   scan    the sub-rows' states are joined inside the lane with Phi^N (Phi is the cascade's state
//           transition, block lower triangular), then across the lanes with powers of Phi^SPAN;
//   pass B  every sub-row runs the whole cascade once from its true state, all K sections in
//           registers (4K multiply-adds per sample), and its output replaces the input. Its own end
//           states check the ones that the next sub-rows started from (sweep_agree).
// One pass per section (iir_ph.cuh: zero-state filter, scan, correction folded into the next pass)
// takes 7K operations per sample and a read and a write of shared memory per section; this takes
// 6K, two reads and one write.
//
// The state before a tile is the end state of the tile before it, from rest: the planner takes this
// schedule only if older state is by then below 1e-10 of the states' own scale (FP64). So there is
// no lookback: blocks exchange nothing, the tiles of a block pass their end states through shared
// memory. Filters that decay more slowly keep the lookback schedules.
//
// Arithmetic is packed: fma.rn.f32x2 issues two multiply-adds per lane, which leaves half of the
// issue slots to the shared-memory accesses and shuffles (the FP32 rate is the same: 36 TFMA/s
// measured either way). Pass A packs neighbouring samples (x and the tables come as pairs from
// 16-byte loads), pass B two sub-rows.
//
// Bound by: memory up to 2 sections; above, by dependent steps at 2.2 warps per scheduler (28 instructions
// per sample at 4 sections, 17.5 of them on the FMA pipe, which is 52% busy). Measured on GB300, butter(order,
// 0.1), CUDA graph replays, against the kernels that this replaces (us, before -> after):
//   order        2              4              8              16
//   2^20     (small kernel kept) 8.5 -> 8.4   12.3 -> 9.9    20.6 -> 13.4
//   2^23      14.3 -> 11.7   18.7 -> 14.1   27.0 -> 19.7   52.4 -> 31.5
//   2^25      49.5 -> 45.3   59.9 -> 47.1   84.0 -> 57.5  153.3 -> 97.8
//   2^27     163.7 -> 159.0  192.4 -> 159.5  284 -> 192    565 -> 344
#pragma once
#include "iir_pipe.cuh"

namespace iirgb {

// ------------------------------------------------------------------------------------
// packed float pairs
// ------------------------------------------------------------------------------------
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// ------------------------------------------------------------------------------------
// geometry and tables of one kernel: K sections, R sub-rows of N samples per lane
// ------------------------------------------------------------------------------------
// Most lanes that a state reaches: filters that take longer to decay keep the lookback schedules.
constexpr int SWEEP_LANES = 32;

template <int K_, int N_, int R_>
struct SweepGeom {
    static constexpr int K = K_, N = N_, R = R_, D = 2 * K_;
    static constexpr int SPAN = N * R;
    static constexpr int TILE = 32 * SPAN;
    static constexpr uint32_t TILE_BYTES = TILE * 4u;
    static_assert(N % 32 == 0 && R % 2 == 0, "sub-rows of whole 128-byte lines, in packed pairs");
    static constexpr int BLOCKS = K * (K + 1) / 2;  // 2x2 blocks of a block lower triangular matrix
    // table offsets in floats (iir_sweep.h: the host's copy of this layout)
    static constexpr int T_A = 0;                     // [D][N] pass A
    static constexpr int T_H = T_A + D * N;           // [D][2] response to (x[-2], x[-1])
    static constexpr int T_PN = (T_H + 2 * D + 3) & ~3;  // [BLOCKS] Phi^N, columns (m00, m10, m01, m11)
    // a lane's power, in rows of an odd number of 16-byte units: lanes read their rows side by side
    static constexpr int ROW = BLOCKS | 1;
    static constexpr int T_PL = T_PN + 4 * BLOCKS;       // [SWEEP_LANES][ROW] Phi^(SPAN l)
    static constexpr int T_LEN = T_PL + 4 * SWEEP_LANES * ROW;
    static_assert(T_LEN % 4 == 0 && T_PN % 4 == 0, "16-byte table rows");
};

// Float index of sample n of lane row l in the tile buffer: SPAN / 32 planes of 32-sample columns,
// a 128-byte line per lane, 16-byte units swizzled by the lane (the 128-byte TMA swizzle), so that
// a warp's 16-byte accesses at one column fall on all banks.
__device__ __forceinline__ int tile_at(int l, int n) {
    return ((n >> 5) << 10) + (l << 5) + ((((n >> 2) & 7) ^ (l & 7)) << 2) + (n & 3);
}

// Float offset of granule j (samples 4j .. 4j + 3) of sub-row i (N samples) from the lane's line, l7 =
// lane & 7: one address per j serves every sub-row.
template <int N>
__device__ __forceinline__ int sub_granule_at(int i, int j, int l7) {
    if constexpr (N % 32 == 0) return ((j >> 3) << 10) + (((j & 7) ^ l7) << 2) + i * (N / 32) * 1024;
    else return (((j ^ l7) ^ ((i & 1) << 2)) << 2) + (i >> 1) * 1024;  // N = 16: two sub-rows to a line
}

// o += M v for one 2x2 block in column order: (o0, o1) += (m00, m10) v0 + (m01, m11) v1
__device__ __forceinline__ f32x2 block_mad(const float* m, float v0, float v1, f32x2 o) {
    const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(m);
    return fma2(c.y, pack2(v1, v1), fma2(c.x, pack2(v0, v0), o));
}

// y = M v + e for a block lower triangular matrix (blocks in row order, s = 0..K-1, q = 0..s)
template <int K>
__device__ __forceinline__ void tri_mad(const float* m, const float (&v)[2 * K], const float (&e)[2 * K],
                                        float (&y)[2 * K]) {
    float o[2 * K];
#pragma unroll
    for (int s = 0; s < K; ++s) {
        f32x2 a = pack2(e[2 * s], e[2 * s + 1]);
#pragma unroll
        for (int q = 0; q <= s; ++q) a = block_mad(m + 4 * (s * (s + 1) / 2 + q), v[2 * q], v[2 * q + 1], a);
        unpack2(a, o[2 * s], o[2 * s + 1]);
    }
#pragma unroll
    for (int i = 0; i < 2 * K; ++i) y[i] = o[i];
}

// ------------------------------------------------------------------------------------
// pass A: zero-state end states of the lane's R sub-rows, components [C0, C0 + C) of 2K
// ------------------------------------------------------------------------------------
template <class G, int C0, int C>
__device__ __forceinline__ void sweep_dots(const float* buf, const float* tab, int lane, float (&e)[G::R][G::D]) {
    constexpr int N = G::N, R = G::R;
    f32x2 acc[R][C];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int c = 0; c < C; ++c) acc[i][c] = 0ull;
    const float* row = buf + (lane << 5);
    const float* ta = tab + G::T_A + C0 * N;
    const int l7 = lane & 7;
#pragma unroll 4
    for (int j = 0; j < N / 4; ++j) {
        ulonglong2 x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(row + sub_granule_at<N>(i, j, l7));
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(ta + c * N + 4 * j);
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i][c] = fma2(t.y, x[i].y, fma2(t.x, x[i].x, acc[i][c]));
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float a, b;
            unpack2(acc[i][c], a, b);
            e[i][C0 + c] = a + b;
        }
}

// Pass A of the whole tile: e[i] = zero-state end state of sub-row i, xh[i] = its input history
// (x[-2], x[-1]); lane 0's history before the tile is (g2, g1).
template <class G>
__device__ __forceinline__ void sweep_ends(const float* buf, const float* tab, int lane, float g2, float g1,
                                           float (&e)[G::R][G::D], float (&xh)[G::R][2]) {
    constexpr int N = G::N, R = G::R, D = G::D;
    if constexpr (D <= 8) {
        sweep_dots<G, 0, D>(buf, tab, lane, e);
    } else {
        sweep_dots<G, 0, 8>(buf, tab, lane, e);
        sweep_dots<G, 8, D - 8>(buf, tab, lane, e);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (i > 0 || lane > 0) {
            const int at = i > 0 ? tile_at(lane, i * N - 2) : tile_at(lane - 1, G::SPAN - 2);
            const float2 h = *reinterpret_cast<const float2*>(buf + at);
            xh[i][0] = h.x;
            xh[i][1] = h.y;
        } else {
            xh[i][0] = g2;
            xh[i][1] = g1;
        }
#pragma unroll
        for (int c = 0; c < D; ++c) {
            const float2 t = *reinterpret_cast<const float2*>(tab + G::T_H + 2 * c);
            e[i][c] = fmaf(t.y, xh[i][1], fmaf(t.x, xh[i][0], e[i][c]));
        }
    }
}

// The lane's end state from rest: its sub-rows joined with Phi^N.
template <class G>
__device__ __forceinline__ void sweep_join(const float* tab, const float (&e)[G::R][G::D], float (&f)[G::D]) {
#pragma unroll
    for (int c = 0; c < G::D; ++c) f[c] = e[0][c];
#pragma unroll
    for (int i = 1; i < G::R; ++i) tri_mad<G::K>(tab + G::T_PN, f, e[i], f);
}

// Scan across the lanes from rest before the tile: S = the state before the lane, last = the state
// after it (lane 31: the tile's end state), from the lanes' zero-state end states f. Kogge-Stone with
// the whole state vector per step: a section-by-section scan takes K times as many dependent
// shuffles. `rounds` steps reach 2^rounds lanes back, beyond which nothing is left.
template <class G>
__device__ __forceinline__ void sweep_scan(const float* tab, int rounds, int lane, const float (&f)[G::D],
                                           float (&S)[G::D], float (&last)[G::D]) {
    constexpr int D = G::D;
#pragma unroll
    for (int c = 0; c < D; ++c) last[c] = f[c];
#pragma unroll 1
    for (int k = 0; k < rounds; ++k) {
        float o[D];
#pragma unroll
        for (int c = 0; c < D; ++c) {
            o[c] = __shfl_up_sync(FULL_MASK, last[c], 1u << k);
            if (lane < (1 << k)) o[c] = 0.f;
        }
        tri_mad<G::K>(tab + G::T_PL + 4 * (1 << k) * G::ROW, o, last, last);
    }
#pragma unroll
    for (int c = 0; c < D; ++c) {
        S[c] = __shfl_up_sync(FULL_MASK, last[c], 1);
        if (lane == 0) S[c] = 0.f;
    }
}

// ------------------------------------------------------------------------------------
// pass B, PH form: the cascade's own recurrences, sub-rows in packed pairs
// ------------------------------------------------------------------------------------
// Granules of 4 samples that go through the cascade together. More of them give longer diagonals (steps
// that do not depend on one another) and more code. Measured with 1 / 2 / 4 before the states were checked: order 2
// at 2^23 samples 15.4 / 15.0 / 14.7 us, order 4 16.9 / 16.6 / 16.2; at 2^27 order 8 174.7 / 175.0 / 184.7, order 10
// 237.5 / 234.3 / 230.6, order 12 259 / 267 / 273, order 16 330.7 / 329.8 / 330.7 (on differences 376 / 367
// / 380); and with that, 1 / 2: order 16 at 2^25 96.8 / 100.1, on differences at 2^27 393 / 388.
__host__ __device__ constexpr int sweep_step_granules(int K, bool diff) {
    return K <= 2 || K == 5 ? 4 : K == 8 && diff ? 2 : 1;
}

// A section's state is carried as (y[-1] - sg y[-2], y[-1]), sg = 1 for poles on the right of the circle and -1 on
// the left: two outputs near a slow pole differ by little (near a pole at -1, from the negative), and it is that
// difference that the recurrence amplifies.
__host__ __device__ constexpr float sweep_sign(float a1) { return a1 < 0.f ? -1.f : 1.f; }

struct SweepSection {
    float b1, b2, a1, a2;
    float k;               // a1 + sg (a2 - 1), rounded once: the difference form's coefficient
    float wd, tol;         // sweep_agree: weight of a difference's residual, and the largest ratio to the output
};

// The gain goes on the samples, not on the first section's taps: taps of 1, -2, 1 (a high pass) then cancel an
// offset without rounding it.
//
// DIFF: the recurrence on the outputs' differences,
//     d[n] = w[n] + (a1 + sg (a2 - 1)) y[n-1] - sg a2 d[n-1],   y[n] = sg y[n-1] + d[n],
// one addition more per sample and section. A rounding of y[n] in the direct form enters its recurrence at
// full gain, 1 / A(z), which a low cutoff makes large; here the rounding of y[n] is the only one of y's own
// size, and it meets (1 + sg a2 z^-1) / A(z), smaller by the pole's angle. Error against 64 bits (2-norm,
// butter(16, .)): cutoff 0.05 3.0e-7 (direct form 1.11e-6, precision form 7.4e-7), 0.1 2.6e-7 (5.8e-7,
// 6.5e-7), 0.4 3.0e-7 (2.3e-7, 5.3e-7). Time at 2^27 samples, cutoff 0.1, orders 12 / 16: 305 / 378 us
// against 280 / 343 direct and 446 / 401 in the precision form.
template <class G, bool DIFF>
__device__ __forceinline__ void sweep_run_ph(float* buf, const SweepSection* sec, float gain, int lane,
                                             const float (&st)[G::R][G::D], const float (&xh)[G::R][2],
                                             float (&end)[G::R][G::D]) {
    constexpr int K = G::K, N = G::N, R = G::R, P = R / 2;
    f32x2 b1[K], b2[K], a1[K], a2[K], sg[DIFF ? K : 1];
#pragma unroll
    for (int s = 0; s < K; ++s) {
        const float sign = sweep_sign(sec[s].a1);
        b1[s] = pack2(sec[s].b1, sec[s].b1);
        b2[s] = pack2(sec[s].b2, sec[s].b2);
        a1[s] = DIFF ? pack2(sec[s].k, sec[s].k) : pack2(sec[s].a1, sec[s].a1);
        a2[s] = DIFF ? pack2(-sign * sec[s].a2, -sign * sec[s].a2) : pack2(sec[s].a2, sec[s].a2);
        if constexpr (DIFF) sg[s] = pack2(sign, sign);
    }
    f32x2 dl[P][K];  // DIFF: the sections' last differences
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int s = 0; s < K; ++s) dl[p][s] = pack2(st[2 * p][2 * s], st[2 * p + 1][2 * s]);
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
                const float* v = st[2 * p + 1] + 2 * s;
                const float sign = sweep_sign(sec[s].a1);
                h[p][s + 1][t] = t == 0 ? pack2(sign * (u[1] - u[0]), sign * (v[1] - v[0])) : pack2(u[1], v[1]);
            }
        }
    float* row = buf + (lane << 5);
    const int l7 = lane & 7;
    constexpr int GB = sweep_step_granules(K, DIFF), S = 4 * GB;  // granules and samples per step
#pragma unroll 1
    for (int j = 0; j < N / 4; j += GB) {
        float4 x[GB][R];
        float* at[GB];
#pragma unroll
        for (int b = 0; b < GB; ++b) {
            at[b] = row + ((j >> 3) << 10) + ((((j & 7) + b) ^ l7) << 2);
#pragma unroll
            for (int i = 0; i < R; ++i) x[b][i] = *reinterpret_cast<const float4*>(at[b] + i * (N / 32) * 1024);
        }
        // v[p][s][t]: section s's input (s = K: the output) at samples t - 2. The samples go through the
        // sections along the diagonals (sample + section), whose steps do not depend on one another.
        f32x2 v[P][K + 1][S + 2];
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int s = 0; s <= K; ++s) {
                v[p][s][0] = h[p][s][0];
                v[p][s][1] = h[p][s][1];
            }
#pragma unroll
            for (int b = 0; b < GB; ++b) {
                v[p][0][4 * b + 2] = mul2(g, pack2(x[b][2 * p].x, x[b][2 * p + 1].x));
                v[p][0][4 * b + 3] = mul2(g, pack2(x[b][2 * p].y, x[b][2 * p + 1].y));
                v[p][0][4 * b + 4] = mul2(g, pack2(x[b][2 * p].z, x[b][2 * p + 1].z));
                v[p][0][4 * b + 5] = mul2(g, pack2(x[b][2 * p].w, x[b][2 * p + 1].w));
            }
        }
#pragma unroll
        for (int d = 0; d < K + S - 1; ++d) {
#pragma unroll
            for (int s = 0; s < K; ++s) {
                const int t = d - s + 2;
                if (t < 2 || t > S + 1) continue;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const f32x2 w = fma2(b2[s], v[p][s][t - 2], fma2(b1[s], v[p][s][t - 1], v[p][s][t]));
                    if constexpr (DIFF) {
                        dl[p][s] = fma2(a1[s], v[p][s + 1][t - 1], fma2(a2[s], dl[p][s], w));
                        v[p][s + 1][t] = fma2(sg[s], v[p][s + 1][t - 1], dl[p][s]);
                    } else {
                        v[p][s + 1][t] = fma2(a1[s], v[p][s + 1][t - 1], fma2(a2[s], v[p][s + 1][t - 2], w));
                    }
                }
            }
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int s = 0; s <= K; ++s) {
                h[p][s][0] = v[p][s][S];
                h[p][s][1] = v[p][s][S + 1];
            }
#pragma unroll
            for (int b = 0; b < GB; ++b) {
                unpack2(v[p][K][4 * b + 2], x[b][2 * p].x, x[b][2 * p + 1].x);
                unpack2(v[p][K][4 * b + 3], x[b][2 * p].y, x[b][2 * p + 1].y);
                unpack2(v[p][K][4 * b + 4], x[b][2 * p].z, x[b][2 * p + 1].z);
                unpack2(v[p][K][4 * b + 5], x[b][2 * p].w, x[b][2 * p + 1].w);
            }
        }
#pragma unroll
        for (int b = 0; b < GB; ++b)
#pragma unroll
            for (int i = 0; i < R; ++i) *reinterpret_cast<float4*>(at[b] + i * (N / 32) * 1024) = x[b][i];
    }
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int s = 0; s < K; ++s) {
            float ya, yb;
            unpack2(h[p][s + 1][1], ya, yb);
            end[2 * p][2 * s + 1] = ya;
            end[2 * p + 1][2 * s + 1] = yb;
            if constexpr (DIFF) {
                unpack2(dl[p][s], end[2 * p][2 * s], end[2 * p + 1][2 * s]);
            } else {
                float za, zb;
                unpack2(h[p][s + 1][0], za, zb);
                const float sign = sweep_sign(sec[s].a1);
                end[2 * p][2 * s] = fmaf(-sign, za, ya);
                end[2 * p + 1][2 * s] = fmaf(-sign, zb, yb);
            }
        }
}

// ------------------------------------------------------------------------------------
// the states checked and corrected
// ------------------------------------------------------------------------------------
// Pass A forms a later section's state from the raw samples. Where the cascade takes nearly all of the signal
// away (a tone in the stop band, an offset through a high pass), that sum cancels: its rounding is of the
// samples' size, the state is not. Pass B runs the sections one after another and does not have this, so the
// state that it leaves behind a sub-row tells how far the next one's start was off:
//     r[j+1] = (pass B's end of sub-row j) - (start of sub-row j+1),   error of a start = -g,
//     g[j+1] = Phi^N g[j] + r[j+1].
// Where r stands out of the recurrence's own rounding, g is found by the same join and scan as the states, and
// the response to g is added to the outputs (4K operations per sample). Elsewhere the check is all there is: about
// 4% of a tile's instructions (order 16: 49.9 -> 52.0 per sample) and 4 to 9% of the time from 4 sections on, the two
// ends of tiles being read besides. A signal that has every tile corrected: order 8 97 us at 2^25 samples (57.5
// otherwise; the lookback kernels 84 to 99). Error against 64 bits, cheby1(16, 1, 0.3), noise and a tone 40 dB above it in
// the stop band: 2.0e-3 without, 2.7e-5 with (section by section, iir_ph.cuh: 3.1e-5).

// Residuals r of the lane's sub-rows (r[i]: at its end), from pass B's end states, the states st that it started
// from and the tile's end state `last`. True if they are within the sections' rounding: tol = 4 x 2^-24 x (1 + the
// noise gain of 1 / A over a sub-row) of a section's largest output in the tile, a difference weighed by what it
// grows to. (With 6 for 4, up to twice the lookback's error gets by: a tone in the stop band of cheby1(4, 1, 0.02);
// with 3, white noise is corrected by half as many filters more. Judging a lane by its last sub-row alone is no
// faster, and lets three times the lookback's error by: cheby1(6, 1, 0.04).) limits(s): a section's (wd, tol).
// The first, the middle and the last section speak for all (over 528 designs and signals, the sections in scipy's
// order, reversed, or with zeros and poles paired at random; the last alone lets five times by). PADDED: the last one
// may pass its input on. Sub-rows that end past the tile's first `have` samples hold nothing.
template <class G, bool PADDED = false, class Limits>
__device__ __forceinline__ bool sweep_agree(Limits&& limits, int lane, int have, const float (&end)[G::R][G::D],
                                            const float (&st)[G::R][G::D], const float* last, float (&r)[G::R][G::D]) {
    constexpr int R = G::R, K = G::K, D = G::D;
    const bool whole = have >= G::TILE;
#pragma unroll
    for (int c = 0; c < D; ++c) {
        float next = __shfl_down_sync(FULL_MASK, st[0][c], 1);
        if (lane == 31) next = last[c];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            r[i][c] = end[i][c] - (i + 1 < R ? st[i + 1 < R ? i + 1 : 0][c] : next);
            if (!whole && lane * G::SPAN + (i + 1) * G::N > have) r[i][c] = 0.f;
        }
    }
    bool ok = true;
#pragma unroll
    for (int s = 0; s < K; ++s) {
        if (s != 0 && s != K / 2 && s != K - 1 && !(PADDED && s == K - 2)) continue;
        const float2 lim = limits(s);
        float top = 0.f, off = 0.f, dif = 0.f;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (whole || lane * G::SPAN + (i + 1) * G::N <= have) top = fmaxf(top, fabsf(end[i][2 * s + 1]));
            off = fmaxf(off, fabsf(r[i][2 * s + 1]));
            dif = fmaxf(dif, fabsf(r[i][2 * s]));
        }
        top = __uint_as_float(__reduce_max_sync(FULL_MASK, __float_as_uint(top)));
        ok = ok && fmaxf(off, lim.x * dif) <= lim.y * top;
    }
    return __all_sync(FULL_MASK, ok);
}

// Adds the cascade's response to the states g before the lane's sub-rows to the outputs in the buffer. taps(s): a
// section's (b1, b2, a1, a2).
template <class G, class Taps>
__device__ __forceinline__ void sweep_respond(float* buf, Taps&& taps, int lane, const float (&g)[G::R][G::D]) {
    constexpr int K = G::K, N = G::N, R = G::R, P = R / 2;
    f32x2 b1[K], b2[K], a1[K], a2[K], h[P][K][2];  // h: the sections' last two outputs
#pragma unroll
    for (int s = 0; s < K; ++s) {
        const float4 c = taps(s);
        const float sign = sweep_sign(c.z);
        b1[s] = pack2(c.x, c.x);
        b2[s] = pack2(c.y, c.y);
        a1[s] = pack2(c.z, c.z);
        a2[s] = pack2(c.w, c.w);
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const float *u = g[2 * p] + 2 * s, *v = g[2 * p + 1] + 2 * s;
            h[p][s][0] = pack2(sign * (u[1] - u[0]), sign * (v[1] - v[0]));
            h[p][s][1] = pack2(u[1], v[1]);
        }
    }
    float* row = buf + (lane << 5);
    const int l7 = lane & 7;
#pragma unroll 1
    for (int j = 0; j < N / 4; ++j) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
            float y[2][4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                f32x2 in = 0ull, x2 = 0ull, x1 = 0ull;
#pragma unroll
                for (int s = 0; s < K; ++s) {
                    const f32x2 w = s == 0 ? 0ull : fma2(b2[s], x2, fma2(b1[s], x1, in));
                    x2 = h[p][s][0];
                    x1 = h[p][s][1];
                    in = fma2(a1[s], x1, fma2(a2[s], x2, w));
                    h[p][s][0] = x1;
                    h[p][s][1] = in;
                }
                unpack2(in, y[0][t], y[1][t]);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float4* q = reinterpret_cast<float4*>(row + sub_granule_at<N>(2 * p + i, j, l7));
                const float4 x = *q;
                *q = make_float4(x.x + y[i][0], x.y + y[i][1], x.z + y[i][2], x.w + y[i][3]);
            }
        }
    }
}

// The two steps of a correction, and the staging of tiles off the 16-byte grid, are functions of their own: few tiles
// need them, and the code that every tile goes through then stays in the instruction cache (order 8 at 2^27: 214 us
// with the corrections inline, 204 as calls; and 189 with the lane scan and pass B as loops that are not unrolled).
// g: what the state before each lane lacks, from rest before the tile; last: and the one after the tile.
template <class G>
__device__ __noinline__ void sweep_lack(const float* tab, int rounds, int lane, const float (&r)[G::R][G::D],
                                        float (&g)[G::D], float (&last)[G::D]) {
    float f[G::D];
    sweep_join<G>(tab, r, f);
    sweep_scan<G>(tab, rounds, lane, f, g, last);
}
// Corrects the tile's outputs, g0 before the lane.
template <class G>
__device__ __noinline__ void sweep_apply(float* buf, const float* tab, const SweepSection* sec, int lane,
                                         const float (&r)[G::R][G::D], const float (&g0)[G::D]) {
    float g[G::R][G::D];
#pragma unroll
    for (int c = 0; c < G::D; ++c) g[0][c] = g0[c];
#pragma unroll
    for (int j = 1; j < G::R; ++j) tri_mad<G::K>(tab + G::T_PN, g[j - 1], r[j - 1], g[j]);
    sweep_respond<G>(buf, [&](int s) { return make_float4(sec[s].b1, sec[s].b2, sec[s].a1, sec[s].a2); }, lane, g);
}

// A tile sample by sample, samples past the signal's end zero, and back.
template <class G>
__device__ __noinline__ void sweep_stage(float* buf, const float* x, long long base, long long n, int lane) {
#pragma unroll 8
    for (int j = lane; j < G::TILE; j += 32) {
        const bool have = base + j < n;
        cp_async4(buf + tile_at(j / G::SPAN, j % G::SPAN), have ? x + base + j : x, have ? 4 : 0);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
}
template <class G>
__device__ __noinline__ void sweep_unstage(const float* buf, float* y, long long base, long long n, int lane) {
    __syncwarp();
#pragma unroll 8
    for (int j = lane; j < G::TILE; j += 32)
        if (base + j < n) y[base + j] = buf[tile_at(j / G::SPAN, j % G::SPAN)];
}

// ------------------------------------------------------------------------------------
// launch parameters and the tile loop
// ------------------------------------------------------------------------------------
constexpr unsigned SWEEP_NONE = 0xffffffffu;

struct IirSweepParams {
    CUtensorMap tmap_x;  // x as rows of SPAN samples, box {32, 32}, 128-byte swizzle
    CUtensorMap tmap_y;  // y likewise
    const float* x;
    float* y;
    long long n;
    const float* tables;  // SweepGeom's layout
    IirLaunchState* state;
    long long timeout_ns;
    unsigned int ntiles;
    unsigned int run0, run1;  // tiles of a block's first run, and of the runs drawn after it
    unsigned int withhold;    // fault injection: the tile whose end state is not passed on (SWEEP_NONE: none)
    int lanes, rounds;        // lanes that a state reaches; scan steps that cover them
    int use_tma;              // tensor maps valid (x, y 16-byte aligned, at least one row)
    float gain;
    SweepSection sec[IIR_MAX_SECTIONS];
};

constexpr unsigned SWEEP_RING = 32;  // item records and end states kept of the last items
constexpr unsigned SWEEP_WARM = 0x80000000u;

template <int NB, int D>
struct SweepAux {
    unsigned long long full[NB], empty[NB];
    float ends[SWEEP_RING][D];           // items' end states
    float fix[SWEEP_RING][D];            // what they lack, where it matters
    unsigned int item[SWEEP_RING];       // the item's tile, SWEEP_WARM if only its end state is wanted
    volatile unsigned int ready[SWEEP_RING];  // i + 1 once item i's end state is in `ends`
    volatile unsigned int checked[SWEEP_RING];  // 2 (i + 1) once it has been checked, plus 1 if `fix` is to be added
    volatile unsigned int issued[NB];    // items put into the buffer so far
    volatile unsigned int total;         // items of the block, once known
    volatile unsigned int abandon;       // a wait ran out: everybody leaves
    unsigned int next;                   // next item for a free warp
};

// Blocks of W filter warps and a loader warp. The signal's tiles (32 lane rows each) are dealt out in
// runs of consecutive tiles: block b starts with run b of run0 tiles, then draws runs of run1 tiles
// from a ticket counter until they are gone. SMs differ in the bandwidth they get (a copy kernel
// that splits a signal evenly among blocks reaches 6.2 TB/s, one that draws its tiles 7.0), so the
// last part is drawn. Ahead of a run goes the tile before it, which is filtered for its end state and
// not stored: no block needs anything from another.
//
// Inside a block the items (tiles of its runs, one after another) are taken by the warps in order,
// and item i's end state goes to item i + 1 through shared memory. It is the end state from rest:
// older state has decayed inside the tile, so the items form no chain, and a warp waits for no more
// than the pass A of the item before its own, which another warp began earlier. Its first lanes add
// the response to it, Phi^(SPAN l) for lane l.
//
// Item i lies in buffer i % NB: the loader keeps NB - W items ahead of the warps. A warp gives its
// buffer back when the store of its output has read it. From 3 sections on it waits for that at once,
// so that the loads run further ahead (2^27, before the states were checked: order 8 177.9 -> 175.5 us, order 16
// 345 -> 332.6); at 1 and 2 sections, bound by memory, it looks after it during its next item (after pass A), or
// before it would wait itself (order 4: 158.2 us, 158.7 at once).
template <class G, int W, int NB, class Run>
__device__ __forceinline__ void sweep_tiles(const IirSweepParams& p, unsigned char* smem, Run&& run) {
    constexpr int SPAN = G::SPAN, R = G::R, K = G::K, D = G::D;
    using Aux = SweepAux<NB, D>;
    static_assert(NB >= W && NB + W <= static_cast<int>(SWEEP_RING), "a buffer per warp, a record per item in flight");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* bufs = reinterpret_cast<float*>(smem);
    Aux& aux = *reinterpret_cast<Aux*>(smem + NB * size_t(G::TILE_BYTES));
    float* tab = reinterpret_cast<float*>(smem + NB * size_t(G::TILE_BYTES) + ((sizeof(Aux) + 15) & ~size_t(15)));
    if (threadIdx.x == W * 32) {
        for (int b = 0; b < NB; ++b) {
            mbar_init(aux.full + b, 1);
            mbar_init(aux.empty + b, 1);
            aux.issued[b] = 0u;
        }
        for (unsigned i = 0; i < SWEEP_RING; ++i) aux.ready[i] = aux.checked[i] = 0u;
        aux.next = 0u;
        aux.total = 0xffffffffu;
        aux.abandon = 0u;
        fence_mbar_init();
    }
    // (of Phi^(SPAN l), the powers that the lanes and the scan steps use)
    const int reach = p.lanes > (1 << p.rounds) / 2 + 1 ? p.lanes : (1 << p.rounds) / 2 + 1;
    for (int i = threadIdx.x; i < G::T_PL / 4 + reach * G::ROW; i += (W + 1) * 32)
        reinterpret_cast<float4*>(tab)[i] = __ldg(reinterpret_cast<const float4*>(p.tables) + i);
    __syncthreads();
    // every wait is bounded; the first to run out sends the whole block home
    auto wait_for = [&](auto&& cond, uint32_t code = IIR_DEV_ERR_MBARRIER) {
        if (cond()) return true;
        const uint64_t start = globaltimer_ns();
        uint32_t spins = 0;
        while (!cond()) {
            if ((++spins & 63u) != 0u) continue;
            if (aux.abandon) return false;
            if (globaltimer_ns() - start > static_cast<uint64_t>(p.timeout_ns)) {
                aux.abandon = 1u;
                raise_error(p.state, sweep_epoch(p.state), code);
                return false;
            }
        }
        return true;
    };
    if (warp == W) {
        if (lane == 0) {
            unsigned i = 0;
            unsigned long long first = static_cast<unsigned long long>(blockIdx.x) * p.run0;
            unsigned len = p.run0;
            bool ok = true;
            while (ok && first < p.ntiles) {
                const unsigned a = static_cast<unsigned>(first);
                const unsigned e = p.ntiles - a < len ? p.ntiles : a + len;
                for (unsigned t = a > 0 ? a - 1 : 0; t < e; ++t, ++i) {
                    const unsigned b = i % NB;
                    if (i >= NB) ok = wait_for([&] { return mbar_try_wait(aux.empty + b, (i / NB - 1u) & 1u); });
                    if (!ok) break;
                    aux.item[i % SWEEP_RING] = t < a ? (t | SWEEP_WARM) : t;
                    if (p.use_tma) {
                        float* buf = bufs + static_cast<size_t>(b) * G::TILE;
                        mbar_arrive_expect_tx(aux.full + b, G::TILE_BYTES);
#pragma unroll
                        for (int h = 0; h < SPAN / 32; ++h)
                            tma_load_2d(buf + h * 1024, &p.tmap_x, 32 * h, static_cast<int>(t * 32u), aux.full + b);
                    } else {
                        mbar_arrive(aux.full + b);
                    }
                    aux.issued[b] = i / NB + 1u;
                }
                if (!ok) break;
                len = p.run1;
                first = static_cast<unsigned long long>(gridDim.x) * p.run0 +
                        static_cast<unsigned long long>(atomicAdd(&p.state->runs, 1u)) * p.run1;
            }
            aux.total = i;
        }
    } else {
        const long long rows = p.n / SPAN;  // whole lane rows of the signal
        const int rest = static_cast<int>(p.n - rows * SPAN);
        int back = -1;  // lane 0: the buffer to give back
        auto give_back = [&] {
            bulk_wait_read_all();  // the store has read it
            mbar_arrive(aux.empty + back);
            back = -1;
        };
        while (true) {
            unsigned i = 0;
            if (lane == 0) i = atomicAdd(&aux.next, 1u);
            i = __shfl_sync(FULL_MASK, i, 0);
            const unsigned b = i % NB;
            // Item i is in its buffer. Its barrier is looked at only once the item's own load has been
            // issued: until then the barrier may be two phases back, and a parity cannot tell those apart.
            auto arrived = [&] { return aux.issued[b] == i / NB + 1u && mbar_try_wait(aux.full + b, (i / NB) & 1u); };
            if (back >= 0 && !arrived()) give_back();
            __syncwarp();
            const bool in = wait_for([&] { return aux.total <= i || arrived(); });
            if (__any_sync(FULL_MASK, !in) || aux.total <= i) break;
            const unsigned rec = aux.item[i % SWEEP_RING];
            const bool warm = (rec & SWEEP_WARM) != 0u;
            const unsigned t = rec & ~SWEEP_WARM;
            float* buf = bufs + static_cast<size_t>(b) * G::TILE;
            const long long row0 = static_cast<long long>(t) * 32, base = row0 * SPAN;
            float g2 = 0.f, g1 = 0.f;  // the two samples before the tile
            if (lane == 0 && t > 0) {
                g2 = __ldg(p.x + base - 2);
                g1 = __ldg(p.x + base - 1);
            }
            // the signal's last, partial lane row (the tensor maps hold whole rows), if it is here
            const int part = (rest > 0 && rows >= row0 && rows < row0 + 32) ? static_cast<int>(rows - row0) : -1;
            if (p.use_tma) {
                if (part >= 0) {
                    for (int j = lane; j < rest; j += 32) buf[tile_at(part, j)] = __ldg(p.x + rows * SPAN + j);
                    __syncwarp();
                }
            } else {
                sweep_stage<G>(buf, p.x, base, p.n, lane);
            }
            float e[R][D], st[R][D], xh[R][2];
            sweep_ends<G>(buf, tab, lane, g2, g1, e, xh);
            if (back >= 0) give_back();
            {
                float f[D], last[D];
                sweep_join<G>(tab, e, f);
                sweep_scan<G>(tab, p.rounds, lane, f, st[0], last);
                if (lane == 31) {
#pragma unroll
                    for (int c = 0; c < D; c += 2)
                        *reinterpret_cast<float2*>(&aux.ends[i % SWEEP_RING][c]) = make_float2(last[c], last[c + 1]);
                    __threadfence_block();
                    if (t != p.withhold) aux.ready[i % SWEEP_RING] = i + 1u;
                }
            }
            if (!warm && t > 0) {
                const bool got = wait_for([&] { return aux.ready[(i - 1u) % SWEEP_RING] == i; }, IIR_DEV_ERR_TIMEOUT);
                if (__any_sync(FULL_MASK, !got)) break;
                __threadfence_block();
                if (lane < p.lanes) {
                    float X[D];
#pragma unroll
                    for (int c = 0; c < D; c += 2) {
                        const float2 v = *reinterpret_cast<const float2*>(&aux.ends[(i - 1u) % SWEEP_RING][c]);
                        X[c] = v.x;
                        X[c + 1] = v.y;
                    }
                    tri_mad<K>(tab + G::T_PL + 4 * lane * G::ROW, X, st[0], st[0]);
                }
            }
#pragma unroll
            for (int j = 1; j < R; ++j) tri_mad<K>(tab + G::T_PN, st[j - 1], e[j - 1], st[j]);
            __syncwarp();  // every lane has read its neighbour's last samples
            float end[R][D];
            run(buf, lane, st, xh, end);
            {
                float r[R][D], last[D];
                // (past the signal's end there are zeros)
                const bool off = !sweep_agree<G>([&](int s) { return make_float2(p.sec[s].wd, p.sec[s].tol); }, lane, G::TILE,
                                                 end, st, aux.ends[i % SWEEP_RING], r);
                float gs[D];
#pragma unroll
                for (int c = 0; c < D; ++c) gs[c] = 0.f;
                if (off) {
                    float rr[R][D], g0[D];  // (copies: their addresses go to a call, the others stay in registers)
#pragma unroll
                    for (int q = 0; q < R; ++q)
#pragma unroll
                        for (int c = 0; c < D; ++c) rr[q][c] = r[q][c];
                    sweep_lack<G>(tab, p.rounds, lane, rr, g0, last);
#pragma unroll
                    for (int c = 0; c < D; ++c) gs[c] = g0[c];
                    if (lane == 31) {
#pragma unroll
                        for (int c = 0; c < D; c += 2)
                            *reinterpret_cast<float2*>(&aux.fix[i % SWEEP_RING][c]) = make_float2(last[c], last[c + 1]);
                    }
                }
                if (lane == 31) {
                    __threadfence_block();
                    aux.checked[i % SWEEP_RING] = 2u * (i + 1u) + (off ? 1u : 0u);
                }
                bool before = false;  // the state before the tile lacked something
                if (!warm && t > 0) {
                    const bool got =
                        wait_for([&] { return aux.checked[(i - 1u) % SWEEP_RING] >> 1 == i; }, IIR_DEV_ERR_TIMEOUT);
                    if (__any_sync(FULL_MASK, !got)) break;
                    __threadfence_block();
                    before = (aux.checked[(i - 1u) % SWEEP_RING] & 1u) != 0u;
                }
                if (!warm && (off || before)) {
                    float rr[R][D], g0[D];
#pragma unroll
                    for (int c = 0; c < D; ++c) {
                        g0[c] = gs[c];
#pragma unroll
                        for (int q = 0; q < R; ++q) rr[q][c] = off ? r[q][c] : 0.f;
                    }
                    if (before && lane < p.lanes) {
                        float X[D];
#pragma unroll
                        for (int c = 0; c < D; ++c) X[c] = aux.fix[(i - 1u) % SWEEP_RING][c];
                        tri_mad<K>(tab + G::T_PL + 4 * lane * G::ROW, X, g0, g0);
                    }
                    sweep_apply<G>(buf, tab, p.sec, lane, rr, g0);
                }
            }
            if (p.use_tma) {
                fence_proxy_async_smem();  // generic accesses of the buffer before the async ones to come
                __syncwarp();
                if (lane == 0 && !warm) {
#pragma unroll
                    for (int h = 0; h < SPAN / 32; ++h)
                        tma_store_2d(&p.tmap_y, 32 * h, static_cast<int>(row0), buf + h * 1024);
                    bulk_commit();
                }
                if (!warm && part >= 0)
                    for (int j = lane; j < rest; j += 32) p.y[rows * SPAN + j] = buf[tile_at(part, j)];
            } else if (!warm) {
                sweep_unstage<G>(buf, p.y, base, p.n, lane);
            }
            __syncwarp();
            if (lane == 0) {
                back = static_cast<int>(b);
                if constexpr (K >= 3) give_back();
            }
        }
        if (lane == 0) bulk_wait_read_all();  // shared memory outlives the copies' reads
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // Loads still in flight (a stopped block) land before the block leaves: the last one of each buffer
        // completes its barrier's last phase, and every earlier one had been waited for before it was issued.
        if (aux.abandon)
            for (int b = 0; b < NB; ++b)
                if (aux.issued[b] > 0u) (void)wait_mbar_bounded(aux.full + b, (aux.issued[b] - 1u) & 1u, IIR_DRAIN_NS);
        sweep_finish(p.state);
    }
}

template <int K, int N, int R>
constexpr size_t sweep_smem(int NBv, size_t aux) {
    return NBv * size_t(SweepGeom<K, N, R>::TILE_BYTES) + ((aux + 15) & ~size_t(15)) + SweepGeom<K, N, R>::T_LEN * 4u;
}

}  // namespace iirgb

// iir_sweep.cu — PH kernels on the state-sweep schedule (iir_sweep.cuh) and the host's side of
// that schedule: the tables of a filter, computed in FP64 from its float32 sections.
#include "iir_sweep.cuh"

#include <algorithm>
#include <cmath>

#include "iir_batch_sweep.h"
#include "iir_sweep.h"

namespace iirgb {

template <int K, int N, int R, int W, int NB>
__global__ void __launch_bounds__((W + 1) * 32) iir_ph_sweep_kernel(const __grid_constant__ IirSweepParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    using G = SweepGeom<K, N, R>;
    sweep_tiles<G, W, NB>(p, smem, [&](float* buf, int lane, auto& st, auto& xh, auto& end) {
        sweep_run_ph<G, false>(buf, p.sec, p.gain, lane, st, xh, end);
    });
}

// The recurrence on differences: AUTO's, from 6 sections on, where the direct form rounds too much.
template <int K, int N, int R, int W, int NB>
__global__ void __launch_bounds__((W + 1) * 32) iir_ph_diff_sweep_kernel(const __grid_constant__ IirSweepParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    using G = SweepGeom<K, N, R>;
    sweep_tiles<G, W, NB>(p, smem, [&](float* buf, int lane, auto& st, auto& xh, auto& end) {
        sweep_run_ph<G, true>(buf, p.sec, p.gain, lane, st, xh, end);
    });
}

}  // namespace iirgb

using namespace iirgb;

namespace iirhost {

namespace {

template <int K, int N, int R, int W, int NB>
void add(std::vector<SweepKernel>& v) {
    v.push_back(SweepKernel{IIR_KIND_PH, K, N, R, W, reinterpret_cast<const void*>(iir_ph_sweep_kernel<K, N, R, W, NB>),
                            sweep_smem<K, N, R>(NB, sizeof(SweepAux<NB, 2 * K>))});
    if constexpr (K >= SWEEP_DIFF_MIN_SECTIONS)
        v.push_back(SweepKernel{SWEEP_KIND_PH_DIFF, K, N, R, W,
                                reinterpret_cast<const void*>(iir_ph_diff_sweep_kernel<K, N, R, W, NB>),
                                sweep_smem<K, N, R>(NB, sizeof(SweepAux<NB, 2 * K>))});
}

template <int K>
void add_sections(std::vector<SweepKernel>& v) {
    // Large signals: 16 KB tiles, two warps per scheduler (7, 9 or 10 warps leave the schedulers uneven
    // and 12 leave one buffer to load ahead: 5-10% slower), as many buffers as shared memory holds.
    // Four sub-rows per lane give pass B two independent chains; from 5 sections on the registers and
    // the joins of four sub-rows cost more than that (order 16 at 2^27, before the states were checked: 337 us with two, 395
    // with four).
    if constexpr (K <= 4) add<K, 32, 4, 8, 13>(v);
    else add<K, 64, 2, 8, (K <= 6 ? 13 : 12)>(v);
    // Small signals: short lane rows, so that the signal spreads over more SMs. (Single sections have
    // their 32-row kernel there, which is faster up to 2^20 samples.)
    if constexpr (K > 1) add<K, 32, 2, 4, 6>(v);
}

const std::vector<SweepKernel>& kernels() {
    static const std::vector<SweepKernel> all = [] {
        std::vector<SweepKernel> v;
        add_sections<1>(v);
        add_sections<2>(v);
        add_sections<3>(v);
        add_sections<4>(v);
        add_sections<5>(v);
        add_sections<6>(v);
        add_sections<7>(v);
        add_sections<8>(v);
        return v;
    }();
    return all;
}

using Mat = std::vector<double>;  // D x D, row-major

Mat mat_mul(const Mat& a, const Mat& b, int D) {
    Mat r(static_cast<size_t>(D) * D, 0.0);
    for (int i = 0; i < D; ++i)
        for (int k = 0; k < D; ++k) {
            const double aik = a[static_cast<size_t>(i) * D + k];
            if (aik == 0.0) continue;
            for (int j = 0; j < D; ++j) r[static_cast<size_t>(i) * D + j] += aik * b[static_cast<size_t>(k) * D + j];
        }
    return r;
}

Mat mat_pow(Mat x, int e, int D) {
    Mat r(static_cast<size_t>(D) * D, 0.0);
    for (int i = 0; i < D; ++i) r[static_cast<size_t>(i) * D + i] = 1.0;
    for (; e; e >>= 1) {
        if (e & 1) r = mat_mul(r, x, D);
        if (e > 1) x = mat_mul(x, x, D);
    }
    return r;
}

// 2x2 block (s, q) of a transition of (y[-2], y[-1]) pairs, in the kernels' basis (sweep_sign) and column order.
void put_block(std::vector<float>& t, size_t at, const Mat& m, const std::vector<SectionF32>& secs, int s, int q) {
    const int D = 2 * static_cast<int>(secs.size());
    const double ss = sweep_sign(secs[static_cast<size_t>(s)].a1), sq = sweep_sign(secs[static_cast<size_t>(q)].a1);
    const double* r0 = m.data() + static_cast<size_t>(2 * s) * D + 2 * q;
    const double* r1 = r0 + D;
    // columns: a unit difference is (y[-2], y[-1]) = (-sq, 0), a unit y[-1] is (sq, 1)
    const double d0 = -sq * r0[0], d1 = -sq * r1[0], u0 = sq * r0[0] + r0[1], u1 = sq * r1[0] + r1[1];
    t[at] = static_cast<float>(d1 - ss * d0);
    t[at + 1] = static_cast<float>(d1);
    t[at + 2] = static_cast<float>(u1 - ss * u0);
    t[at + 3] = static_cast<float>(u1);
}

// Response of every section's output to a unit sample entering section 0 after its FIR taps.
std::vector<std::vector<double>> impulse_states(const std::vector<SectionF32>& secs, int len) {
    const size_t K = secs.size();
    std::vector<std::vector<double>> p(K, std::vector<double>(static_cast<size_t>(len), 0.0));
    for (size_t s = 0; s < K; ++s) {
        double y1 = 0.0, y2 = 0.0;
        for (int n = 0; n < len; ++n) {
            double w;
            if (s == 0) {
                w = n == 0 ? 1.0 : 0.0;
            } else {
                const std::vector<double>& x = p[s - 1];
                w = x[n] + (n >= 1 ? secs[s].b1 * x[n - 1] : 0.0) + (n >= 2 ? secs[s].b2 * x[n - 2] : 0.0);
            }
            const double y = w + secs[s].a1 * y1 + secs[s].a2 * y2;
            p[s][static_cast<size_t>(n)] = y;
            y2 = y1;
            y1 = y;
        }
    }
    return p;
}

// Pass A's tables, [2K][N] dot products at 0 and the response to the input history at t_h.
void put_dots(std::vector<float>& t, const SweepFilter& f, int N, size_t t_h) {
    const int K = f.K;
    const std::vector<std::vector<double>> p = impulse_states(f.secs, N);
    auto ps = [&](int s, int n) { return n >= 0 ? p[static_cast<size_t>(s)][static_cast<size_t>(n)] : 0.0; };
    const double b1 = f.secs[0].b1, b2 = f.secs[0].b2, g = f.gain;
    for (int s = 0; s < K; ++s) {
        const double sg = sweep_sign(f.secs[static_cast<size_t>(s)].a1);
        float* t0 = t.data() + static_cast<size_t>(2 * s) * N;  // y[N-1] - sg y[N-2]
        float* t1 = t0 + N;                                      // y[N-1]
        auto h = [&](int m) { return g * (ps(s, m) + b1 * ps(s, m - 1) + b2 * ps(s, m - 2)); };  // impulse response
        for (int n = 0; n < N; ++n) {
            const double y1 = h(N - 1 - n), y2 = h(N - 2 - n);
            t0[n] = static_cast<float>(y1 - sg * y2);
            t1[n] = static_cast<float>(y1);
        }
        // (x[-2], x[-1]) reach the sub-row through section 0's FIR taps
        auto h2 = [&](int m) { return g * b2 * ps(s, m); };
        auto h1 = [&](int m) { return g * (b1 * ps(s, m) + b2 * ps(s, m - 1)); };
        float* th = t.data() + t_h + 4 * s;
        th[0] = static_cast<float>(h2(N - 1) - sg * h2(N - 2));
        th[1] = static_cast<float>(h1(N - 1) - sg * h1(N - 2));
        th[2] = static_cast<float>(h2(N - 1));
        th[3] = static_cast<float>(h1(N - 1));
    }
}

}  // namespace

std::vector<const SweepKernel*> sweep_kernels(int kind, int K) {
    std::vector<const SweepKernel*> r;
    for (const SweepKernel& k : kernels())
        if (k.kind == kind && k.K == K) r.push_back(&k);
    return r;
}

SweepFilter sweep_filter(const SectionF32* secs, int K, double gain) {
    SweepFilter f;
    f.K = K;
    f.gain = gain;
    f.secs.assign(secs, secs + K);
    const int D = 2 * K;
    // state (y_s[n-2], y_s[n-1]) of every section, zero input: section s > 0 sees its predecessor's
    // new output and history through its FIR taps
    f.phi.assign(static_cast<size_t>(D) * D, 0.0);
    std::vector<double> row(static_cast<size_t>(D)), prev(static_cast<size_t>(D), 0.0);
    for (int s = 0; s < K; ++s) {
        std::fill(row.begin(), row.end(), 0.0);
        row[2 * s + 1] += secs[s].a1;
        row[2 * s] += secs[s].a2;
        if (s > 0) {
            for (int j = 0; j < D; ++j) row[j] += prev[j];
            row[2 * (s - 1) + 1] += secs[s].b1;
            row[2 * (s - 1)] += secs[s].b2;
        }
        f.phi[static_cast<size_t>(2 * s) * D + 2 * s + 1] = 1.0;
        for (int j = 0; j < D; ++j) f.phi[static_cast<size_t>(2 * s + 1) * D + j] = row[j];
        prev = row;
    }
    // energy of every section's impulse response, over as many samples as most of it takes
    std::vector<std::vector<double>> p;
    for (const int len : {512, 4096, 65536}) {
        p = impulse_states(f.secs, len);
        double peak = 0.0, tail = 0.0;
        for (int n = 0; n < len; ++n) {
            const double v = std::fabs(p.back()[static_cast<size_t>(n)]);
            (8 * n < 7 * len ? peak : tail) = std::max(8 * n < 7 * len ? peak : tail, v);
        }
        if (!(tail > 1e-3 * peak)) break;
    }
    f.scale.assign(static_cast<size_t>(K), 1.0);
    for (int s = 0; s < K; ++s) {
        double e = 0.0;
        for (double v : p[static_cast<size_t>(s)]) e += v * v;
        f.scale[static_cast<size_t>(s)] = std::sqrt(e);
    }
    return f;
}

bool sweep_too_slow(const SectionF32* secs, int K, int samples) {
    double r = 0.0;
    for (int s = 0; s < K; ++s) {
        const double a1 = secs[s].a1, a2 = secs[s].a2, disc = a1 * a1 + 4.0 * a2;
        r = std::max(r, disc < 0.0 ? std::sqrt(-a2) : 0.5 * (std::fabs(a1) + std::sqrt(disc)));
    }
    return !(samples * std::log(r) <= std::log(1.0000001e-10));
}

int sweep_decay(const SweepFilter& f, int unit, int most) {
    const int D = 2 * f.K;
    for (double s : f.scale)
        if (!std::isfinite(s) || !(s > 0.0)) return 0;
    const Mat step = mat_pow(f.phi, unit, D);
    Mat m = step;
    for (int h = 1; h <= most; ++h) {
        double norm = 0.0;
        for (int i = 0; i < D; ++i) {
            double r = 0.0;
            for (int j = 0; j < D; ++j)
                r += std::fabs(m[static_cast<size_t>(i) * D + j]) * f.scale[j / 2] / f.scale[i / 2];
            norm = std::max(norm, r);
        }
        if (!std::isfinite(norm)) return 0;
        if (norm <= 1e-10) return h;
        m = mat_mul(m, step, D);
    }
    return 0;
}

std::vector<float> sweep_tables(const SweepFilter& f, int N, int R) {
    const int K = f.K, D = 2 * K, span = N * R;
    const int blocks = K * (K + 1) / 2, row = blocks | 1;
    const size_t t_h = static_cast<size_t>(D) * N, t_pn = (t_h + 2 * D + 3) & ~size_t(3),
                 t_pl = t_pn + 4 * static_cast<size_t>(blocks);
    std::vector<float> t(t_pl + 4 * static_cast<size_t>(SWEEP_LANES) * row, 0.f);
    put_dots(t, f, N, t_h);
    auto put = [&](size_t at, const Mat& m) {
        for (int s = 0; s < K; ++s)
            for (int q = 0; q <= s; ++q) put_block(t, at + 4 * static_cast<size_t>(s * (s + 1) / 2 + q), m, f.secs, s, q);
    };
    put(t_pn, mat_pow(f.phi, N, D));
    const Mat step = mat_pow(f.phi, span, D);
    Mat pl = mat_pow(f.phi, 0, D);
    for (int l = 0; l < SWEEP_LANES; ++l) {
        put(t_pl + 4 * static_cast<size_t>(l) * row, pl);
        pl = mat_mul(pl, step, D);
    }
    return t;
}

SweepLimits sweep_limits(const SectionF32& s, int N) {
    const double a1 = s.a1, a2 = s.a2;
    // power gain of 1 / (1 - a1 z^-1 - a2 z^-2) over a sub-row: roundings that enter the recurrence come out by it
    double noise = 0.0, y1 = 0.0, y2 = 0.0;
    for (int n = 0; n < N; ++n) {
        const double y = (n == 0 ? 1.0 : 0.0) + a1 * y1 + a2 * y2;
        noise += y * y;
        y2 = y1;
        y1 = y;
    }
    // an error of the difference grows to about 1 / (the pole's angle from sg) in the output, its square k's size
    const double angle = std::sqrt(std::fabs(a1 + sweep_sign(s.a1) * (a2 - 1.0)));
    return SweepLimits{static_cast<float>(angle < 1.0 ? 1.0 / std::max(angle, 1e-6) : 1.0),
                       static_cast<float>(4.0 * 0x1p-24 * (1.0 + std::sqrt(noise)))};
}

SweepTrial sweep_trial(const SweepFilter& f, const std::vector<float>& t, int N, bool diff, int rows, float offset) {
    const int K = f.K, D = 2 * K;
    std::vector<float> top(static_cast<size_t>(K), 0.f), off(top);  // largest outputs and weighed residuals
    std::vector<SweepLimits> lim;
    for (const SectionF32& s : f.secs) lim.push_back(sweep_limits(s, N));
    const float* th = t.data() + static_cast<size_t>(D) * N;
    const float* pn = t.data() + ((static_cast<size_t>(D) * N + 2 * D + 3) & ~size_t(3));
    std::vector<float> st(static_cast<size_t>(D), 0.f), e(st), next(st);
    std::vector<float> h(static_cast<size_t>(2 * (K + 1)));   // pass B's histories: (n - 2, n - 1) of each stage
    std::vector<double> r(static_cast<size_t>(2 * (K + 1)), 0.0);  // the same in 64 bits
    std::vector<float> x(static_cast<size_t>(N)), dl(static_cast<size_t>(K));
    const float g = static_cast<float>(f.gain);
    float x2 = 0.f, x1 = 0.f;
    double err = 0.0, ref = 0.0;
    unsigned int lcg = 12345u;
    for (int i = 0; i < rows; ++i) {
        for (float& v : x) v = static_cast<float>(static_cast<int>((lcg = 1664525u * lcg + 1013904223u) >> 8)) * 0x1p-23f - 1.f + offset;
        for (int c = 0; c < D; ++c) {
            float a[2] = {0.f, 0.f};
            for (int n = 0; n < N; ++n) a[n & 1] = std::fmaf(t[static_cast<size_t>(c) * N + n], x[n], a[n & 1]);
            e[c] = std::fmaf(th[2 * c + 1], x1, std::fmaf(th[2 * c], x2, a[0] + a[1]));
        }
        h[0] = g * x2;
        h[1] = g * x1;
        for (int s = 0; s < K; ++s) {
            dl[s] = st[2 * s];
            h[2 * s + 2] = sweep_sign(f.secs[static_cast<size_t>(s)].a1) * (st[2 * s + 1] - st[2 * s]);
            h[2 * s + 3] = st[2 * s + 1];
        }
        for (int n = 0; n < N; ++n) {
            float in = g * x[n];
            double rin = f.gain * x[n];
            for (int s = 0; s < K; ++s) {
                const SectionF32& q = f.secs[s];
                const float w = std::fmaf(q.b2, h[2 * s], std::fmaf(q.b1, h[2 * s + 1], in));
                float y;
                if (diff) {
                    const float sg = sweep_sign(q.a1), k = static_cast<float>(q.a1 + sg * (static_cast<double>(q.a2) - 1.0));
                    dl[s] = std::fmaf(k, h[2 * s + 3], std::fmaf(-sg * q.a2, dl[s], w));
                    y = std::fmaf(sg, h[2 * s + 3], dl[s]);
                } else {
                    y = std::fmaf(q.a1, h[2 * s + 3], std::fmaf(q.a2, h[2 * s + 2], w));
                }
                h[2 * s] = h[2 * s + 1];
                h[2 * s + 1] = in;
                in = y;
                const double rw = rin + q.b1 * r[2 * s + 1] + q.b2 * r[2 * s];
                const double ry = rw + q.a1 * r[2 * s + 3] + q.a2 * r[2 * s + 2];
                r[2 * s] = r[2 * s + 1];
                r[2 * s + 1] = rin;
                rin = ry;
            }
            h[2 * K] = h[2 * K + 1];
            h[2 * K + 1] = in;
            r[2 * K] = r[2 * K + 1];
            r[2 * K + 1] = rin;
            err += (in - rin) * (in - rin);
            ref += rin * rin;
        }
        for (int s = 0; s < K; ++s) {
            float a0 = e[2 * s], a1 = e[2 * s + 1];
            for (int q = 0; q <= s; ++q) {
                const float* m = pn + 4 * (s * (s + 1) / 2 + q);
                a0 = std::fmaf(m[2], st[2 * q + 1], std::fmaf(m[0], st[2 * q], a0));
                a1 = std::fmaf(m[3], st[2 * q + 1], std::fmaf(m[1], st[2 * q], a1));
            }
            next[2 * s] = a0;
            next[2 * s + 1] = a1;
            const float y = h[2 * s + 3], sg = sweep_sign(f.secs[static_cast<size_t>(s)].a1);
            top[s] = std::max(top[s], std::fabs(y));
            off[s] = std::max(off[s], std::max(std::fabs(y - a1), lim[s].wd * std::fabs((diff ? dl[s] : y - sg * h[2 * s + 2]) - a0)));
        }
        st = next;
        x2 = x[N - 2];
        x1 = x[N - 1];
    }
    const double e2 = std::sqrt(err / ref);
    double worst = 0.0;
    for (int s = 0; s < K; ++s) worst = std::max(worst, static_cast<double>(off[s]) / (static_cast<double>(lim[s].tol) * top[s]));
    return SweepTrial{std::isfinite(e2) ? e2 : INFINITY, std::isfinite(worst) ? worst : INFINITY};
}

BatchSweepFilter bsweep_filter(const SectionF32* secs, int K, double gain, int span) {
    BatchSweepFilter out;
    if (sweep_too_slow(secs, K, 32 * span)) return out;
    // the compiled number of sections: those past the filter's own pass their input on
    const int KP = bsweep_sections(K);
    std::vector<SectionF32> padded(secs, secs + K);
    padded.resize(static_cast<size_t>(KP), SectionF32{0.f, 0.f, 0.f, 0.f});
    const SweepFilter f = sweep_filter(padded.data(), KP, gain);
    const int D = 2 * KP, N = bsweep_subrow(KP, span), blocks = KP * (KP + 1) / 2;
    auto log2i = [](int v) {
        int l = 0;
        while ((1 << l) < v) ++l;
        return l;
    };
    // squares of the one-sample transition (block lower triangular)
    std::vector<Mat> sq{f.phi};
    auto power = [&](int k) -> const Mat& {  // Phi^(2^k)
        while (static_cast<int>(sq.size()) <= k) {
            const Mat& a = sq.back();
            Mat r(static_cast<size_t>(D) * D, 0.0);
            for (int i = 0; i < D; ++i)
                for (int m = 0; m <= (i | 1); ++m) {
                    const double v = a[static_cast<size_t>(i) * D + m];
                    for (int j = 0; j <= (m | 1); ++j)
                        r[static_cast<size_t>(i) * D + j] += v * a[static_cast<size_t>(m) * D + j];
                }
            sq.push_back(std::move(r));
        }
        return sq[static_cast<size_t>(k)];
    };
    auto decayed = [&](const Mat& m) {
        for (int i = 0; i < D; ++i) {
            double r = 0.0;
            for (int j = 0; j <= (i | 1); ++j)
                r += std::fabs(m[static_cast<size_t>(i) * D + j]) * f.scale[static_cast<size_t>(j / 2)] /
                     f.scale[static_cast<size_t>(i / 2)];
            if (!(r <= 1e-10)) return false;
        }
        return true;
    };
    const int ls = log2i(span);
    int k = 0;
    while (k <= 5 && !decayed(power(ls + k))) ++k;
    if (k > 5) return out;
    out.rounds = k;
    out.fast = true;
    const size_t t_h = static_cast<size_t>(D) * N, t_c = t_h + 2 * D, t_w = t_c + 4 * KP + 4,
                 t_pn = t_w + static_cast<size_t>((2 * KP + 3) & ~3), t_ps = t_pn + 4 * static_cast<size_t>(blocks);
    std::vector<float>& t = out.table;
    t.assign(static_cast<size_t>(bsweep_table_floats(KP, span)), 0.f);
    put_dots(t, f, N, t_h);
    for (int s = 0; s < KP; ++s) {
        float* c = t.data() + t_c + 4 * s;
        c[0] = padded[static_cast<size_t>(s)].b1;
        c[1] = padded[static_cast<size_t>(s)].b2;
        c[2] = padded[static_cast<size_t>(s)].a1;
        c[3] = padded[static_cast<size_t>(s)].a2;
        // (a section that passes its input on is held to nothing of its own)
        const SweepLimits lim = s < K ? sweep_limits(padded[static_cast<size_t>(s)], N) : SweepLimits{0.f, 1.f};
        t[t_w + 2 * static_cast<size_t>(s)] = lim.wd;
        t[t_w + 2 * static_cast<size_t>(s) + 1] = lim.tol;
    }
    t[t_c + 4 * static_cast<size_t>(KP)] = static_cast<float>(gain);
    auto put = [&](size_t at, const Mat& m) {
        for (int s = 0; s < KP; ++s)
            for (int q = 0; q <= s; ++q) put_block(t, at + 4 * static_cast<size_t>(s * (s + 1) / 2 + q), m, f.secs, s, q);
    };
    put(t_pn, power(log2i(N)));
    for (int j = 0; j < BSWEEP_STEPS; ++j) put(t_ps + 4 * static_cast<size_t>(j) * blocks, power(ls + j));
    if (!bsweep_chained(KP)) {
        const size_t t_pl = t_ps + 4 * static_cast<size_t>(BSWEEP_STEPS) * blocks;
        Mat pl = mat_pow(f.phi, 0, D);
        for (int l = 0; l < BSWEEP_NEAR; ++l) {
            put(t_pl + 4 * static_cast<size_t>(l) * blocks, pl);
            if (l + 1 < BSWEEP_NEAR) pl = mat_mul(pl, power(ls), D);
        }
    }
    return out;
}

}  // namespace iirhost

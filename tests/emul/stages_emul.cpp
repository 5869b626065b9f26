// stages_emul.cpp -- CPU emulation, one thread after the other, of the transforms
// whose stages are compiled for their size (the same template code):
//   * the three-stage plans as fft3_ct runs them: 2048 (forward, inverse, and the
//     forward -> transfer -> reversed inverse of a propagation), 4096 and 8192
//     (the rows of the large transforms: forward and inverse);
//   * a column of the large transforms as two passes of short transforms
//     (k_fft_cols_1, k_fft_cols_2).
// Prints "<name> <largest error / largest value>" per check.
#include <array>
#include <cmath>
#include <complex>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "fft_core.cuh"

using namespace atmwfs;
using cd = std::complex<double>;

static uint64_t g_rng = 88172645463325252ull;
static double urand()
{
    g_rng ^= g_rng << 13;
    g_rng ^= g_rng >> 7;
    g_rng ^= g_rng << 17;
    return (double)(g_rng >> 11) * (1.0 / 9007199254740992.0);
}

static std::vector<cd> dft(std::vector<cd> x, int sign)
{
    const size_t n = x.size();
    if (n == 1) return x;
    std::vector<cd> a(n / 2), b(n / 2);
    for (size_t i = 0; i < n / 2; i++) a[i] = x[2 * i], b[i] = x[2 * i + 1];
    a = dft(a, sign), b = dft(b, sign);
    for (size_t k = 0; k < n / 2; k++) {
        const cd w = std::polar(1.0, sign * 2.0 * M_PI * (double)k / (double)n) * b[k];
        x[k] = a[k] + w, x[k + n / 2] = a[k] - w;
    }
    return x;
}

static float2 f2(cd z) { return make_float2((float)z.real(), (float)z.imag()); }
static cd c2(float2 z) { return cd(z.x, z.y); }

static void report(const char* what, int n, const std::vector<cd>& got, const std::vector<cd>& want)
{
    double err = 0, nrm = 0;
    for (size_t k = 0; k < want.size(); k++) {
        err = fmax(err, std::abs(got[k] - want[k]));
        nrm = fmax(nrm, std::abs(want[k]));
    }
    printf("%s_%d %.3e\n", what, n, err / nrm);
}

// fft3_ct of one row: radices RA, RB, RC, twiddles of order `rev`
template <int N, int RA, int RB, int RC>
static void rows3(std::vector<std::array<float2, Plan<N>::E>>& V, std::vector<float2>& buf, const float2* tw, int rev)
{
    constexpr int T = Plan<N>::T, E = Plan<N>::E;
    const float2 *twB = tw + tw_offset<N>(rev, 1), *twC = tw + tw_offset<N>(rev, 2);
    for (int t = 0; t < T; t++) {
        stage_dft<E, RA, -1>(V[t].data());
        stage_store<N, T, E, RA, 1>(V[t].data(), buf.data(), t);
    }
    for (int t = 0; t < T; t++) {
        stage_load<N, T, E, RB>(V[t].data(), buf.data(), t);
        stage_twiddle_rt<N, T, E, RB>(V[t].data(), t, twB, RA);
        stage_dft<E, RB, -1>(V[t].data());
    }
    for (int t = 0; t < T; t++) stage_store<N, T, E, RB, RA>(V[t].data(), buf.data(), t);
    for (int t = 0; t < T; t++) {
        stage_load<N, T, E, RC>(V[t].data(), buf.data(), t);
        stage_twiddle_rt<N, T, E, RC>(V[t].data(), t, twC, RA * RB);
        stage_dft<E, RC, -1>(V[t].data());
    }
}

template <int N>
static void check_rows(bool prop)
{
    constexpr int T = Plan<N>::T, E = Plan<N>::E, RL = last_radix<N>();
    constexpr int R0 = Stages<N>::R0, R1 = Stages<N>::R1, R2 = Stages<N>::R2;
    static_assert(Stages<N>::S == 3, "three stages");
    std::vector<float2> tw(tw_total<N>()), buf(row_stride<N>());
    build_twiddles<N>(tw.data());
    std::vector<cd> x(N), got(N);
    for (auto& v : x) v = c2(f2(cd(urand() - 0.5, urand() - 0.5)));
    std::vector<std::array<float2, E>> V(T);
    auto load = [&](bool conj) {
        for (int t = 0; t < T; t++) {
            for (int e = 0; e < E; e++) V[t][e] = f2(x[t + e * T]);
            if (conj) conj_all<E>(V[t].data());
        }
    };
    for (int sign : {-1, 1}) {
        load(sign > 0);
        rows3<N, R0, R1, R2>(V, buf, tw.data(), 0);
        for (int t = 0; t < T; t++) {
            if (sign > 0) conj_all<E>(V[t].data());
            for (int s = 0; s < E; s++) got[last_index<N, T, RL>(t, s)] = c2(V[t][s]);
        }
        report(sign < 0 ? "fwd" : "inv", N, got, dft(x, sign));
    }
    if (!prop) return;
    std::vector<cd> h(N);
    for (auto& v : h) v = c2(f2(std::polar(1.0 / N, 2.0 * M_PI * urand())));
    load(false);
    rows3<N, R0, R1, R2>(V, buf, tw.data(), 0);
    for (int t = 0; t < T; t++) {  // IFFT(H F) = conj(FFT(conj(H F)))
        for (int s = 0; s < E; s++) V[t][s] = f2(std::conj(c2(V[t][s]) * h[last_index<N, T, RL>(t, s)]));
    }
    rows3<N, R2, R1, R0>(V, buf, tw.data(), 1);
    for (int t = 0; t < T; t++) {
        conj_all<E>(V[t].data());
        for (int e = 0; e < E; e++) got[t + e * T] = c2(V[t][e]);
    }
    std::vector<cd> X = dft(x, -1);
    for (int k = 0; k < N; k++) X[k] *= h[k];
    report("prop", N, got, dft(X, 1));
}

// fft_col of one column: v[t][e] = in(t + e T) -> out(last_index(t, s))
template <int N, typename In, typename Out>
static void column(In in, Out out)
{
    constexpr int T = Plan<N>::T, E = Plan<N>::E, RA = Stages<N>::R0, RB = Stages<N>::R1, RL = last_radix<N>();
    std::vector<float2> tw(tw_total<N>()), buf(N);
    build_twiddles<N>(tw.data());
    std::vector<std::array<float2, E>> V(T);
    for (int t = 0; t < T; t++) {
        for (int e = 0; e < E; e++) V[t][e] = in(t + e * T);
        stage_dft<E, RA, -1>(V[t].data());
        for (int q = 0; q < RA; q++) buf[t * RA + q] = V[t][q];
    }
    for (int t = 0; t < T; t++) {
        for (int w = 0; w < E / RB; w++)
            for (int r = 0; r < RB; r++) V[t][w * RB + r] = buf[t + T * w + r * (N / RB)];
        stage_twiddle_rt<N, T, E, RB>(V[t].data(), t, tw.data() + tw_offset<N>(0, 1), RA);
        stage_dft<E, RB, -1>(V[t].data());
        for (int s = 0; s < E; s++) out(last_index<N, T, RL>(t, s), V[t][s]);
    }
}

template <int N1, int N2>
static void check_columns()
{
    constexpr int M = N1 * N2;
    std::vector<cd> x(M), got(M);
    for (auto& v : x) v = c2(f2(cd(urand() - 0.5, urand() - 0.5)));
    std::vector<float2> wm(M);
    for (int k = 0; k < M; k++) wm[k] = f2(std::polar(1.0, -2.0 * M_PI * k / M));
    for (int sign : {-1, 1}) {
        auto cj = [&](float2 z) { return sign > 0 ? make_float2(z.x, -z.y) : z; };
        std::vector<float2> a(M);
        for (int y = 0; y < M; y++) a[y] = f2(x[y]);
        for (int y2 = 0; y2 < N2; y2++)
            column<N1>([&](int y1) { return cj(a[y1 * N2 + y2]); },
                       [&](int k1, float2 v) { a[k1 * N2 + y2] = cj(cmul(v, wm[y2 * k1])); });
        for (int k1 = 0; k1 < N1; k1++)
            column<N2>([&](int i) { return cj(a[k1 * N2 + i]); },
                       [&](int k2, float2 v) { got[k1 + N1 * k2] = c2(cj(v)); });
        report(sign < 0 ? "colfwd" : "colinv", M, got, dft(x, sign));
    }
}

int main()
{
    check_rows<2048>(true);
    check_rows<4096>(false);
    check_rows<8192>(false);
    check_columns<64, 64>();
    check_columns<64, 128>();
    return 0;
}

// chromat_emul.cpp -- the chromatic zoom's bilinear value (chromat_ff.cuh)
// against the reference's double expressions.  Prints one line per set of
// inputs: "<name> <values> <values that differ> <share left to the doubles>";
// the values left to the doubles are counted, not compared.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>

#include "chromat_ff.cuh"

using namespace atmwfs;

static uint64_t g_rng = 88172645463325252ull;
static double urand()
{
    g_rng ^= g_rng << 13;
    g_rng ^= g_rng >> 7;
    g_rng ^= g_rng << 17;
    return (double)(g_rng >> 11) * (1.0 / 9007199254740992.0);
}

static bool same(float a, float b)
{
    if (std::isnan(a) || std::isnan(b)) return std::isnan(a) && std::isnan(b);
    uint32_t x, y;
    memcpy(&x, &a, 4);
    memcpy(&y, &b, 4);
    return x == y;
}

// f() in (-1, 1) for the fractions (a position between -1 and 0 belongs to pixel
// 0, so that its weights exceed 1 and two taps are subtracted), v() for the values
template <typename Fn, typename Vn>
static void check(const char* name, long n, Fn f, Vn v)
{
    long differ = 0, slow = 0;
    for (long i = 0; i < n; i++) {
        const float u = f(), t = f(), a = v(), b = v(), c = v(), d = v();
        float got;
        if (!chromat_taps(u, t, a, b, c, d, got)) slow++;
        else if (!same(got, chromat_taps_f64(u, t, a, b, c, d))) differ++;
    }
    printf("%s %ld %ld %.9f\n", name, n, differ, (double)slow / (double)n);
}

int main()
{
    auto frac = [] { return (float)urand() < 1.0f ? (float)(urand() * 0.99999994) : 0.5f; };
    auto tiny = [] { return (float)std::exp2(-40.0 * urand() - 1e-3); };               // down to 2^-40
    auto few = [] { return (float)((int)(urand() * 16)) / 16.0f; };                       // 0, 1/16 ..: exact sums, ties
    auto psf = [] { return (float)std::exp(30.0 * urand()); };                            // intensities of a PSF
    auto wide = [] { return (float)std::exp2(-149.0 + 270.0 * urand()); };                // denormals included
    auto faint = [] { return (float)std::exp2(-149.0 + 40.0 * urand()); };
    auto ints = [] { return (float)((int)(urand() * 16777216.0)); };
    auto dark = [] { return urand() < 0.5 ? 0.0f : (float)std::exp(20.0 * urand()); };
    auto odd = [] {
        const double r = urand();
        return r < 0.2 ? std::numeric_limits<float>::infinity() : r < 0.4 ? std::numeric_limits<float>::quiet_NaN()
                                                                : r < 0.6 ? 3.4e38f : r < 0.8 ? 0.0f : (float)urand();
    };
    auto either = [] { return (float)(1.9999999 * urand() - 0.9999999); };
    auto few_either = [] { return (float)((int)(urand() * 31) - 15) / 16.0f; };
    auto close = [] { return (float)(1.0 + 1e-3 * urand()); };                            // the taps nearly cancel
    check("psf", 20000000, frac, psf);
    check("outside", 10000000, either, psf);
    check("outside_few", 5000000, few_either, ints);
    check("outside_close", 5000000, either, close);
    check("outside_wide", 5000000, either, wide);
    check("psf_tiny_fractions", 5000000, tiny, psf);
    check("psf_few_fractions", 5000000, few, psf);
    check("ties", 5000000, few, ints);
    check("dark", 5000000, frac, dark);
    check("dark_few", 5000000, few, dark);
    check("zero", 1000, few, [] { return 0.0f; });
    check("wide", 5000000, frac, wide);
    check("wide_tiny", 5000000, tiny, wide);
    check("faint", 2000000, frac, faint);
    check("nonfinite", 2000000, few, odd);
    return 0;
}

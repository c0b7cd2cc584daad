// Host-side harness for the two-operation quotient and the split boundary mix
// of geopvi_gb300/csrc/fwi2d_exact.h (built by tests/test_step_math.py with
// g++ -ffp-contract=off).
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>

#include "../geopvi_gb300/csrc/fwi2d_exact.h"

using namespace gbfwi;

static bool same(float a, float b) { return std::memcmp(&a, &b, 4) == 0; }

extern "C" {

// div_two and div2_two against IEEE division: every 29th significand of the
// binades klo..khi, both signs, zeros and infinities.
long long harness_div_two(float y, int klo, int khi)
{
    float rh, rl;
    reciprocal_pair(y, &rh, &rl);
    const float least = div2_two_least(y);
    long long bad = 0;
    auto check = [&](float x) {
        if (std::fabs(x) >= kDivLo && !same(div_two(x, rh, rl), x / y)) ++bad;
        if ((x == 0.0f || std::fabs(x) >= least) && !same(div2_two(x, rh, rl), (x / y) / y)) ++bad;
    };
    for (int k = klo; k <= khi; ++k)
        for (uint32_t m = 0; m < (1u << 23); m += 29) {
            const uint32_t bits = ((uint32_t)(127 + k) << 23) | m;
            float x;
            std::memcpy(&x, &bits, 4);
            check(x);
            check(-x);
        }
    for (float x : {0.0f, -0.0f, INFINITY, -INFINITY, 1.0f, 3.4e38f}) check(x);
    return bad;
}

float harness_div2_least(float y) { return div2_two_least(y); }

int harness_two_op_exact(float y) { return two_op_exact(y) ? 1 : 0; }

// The quotients against IEEE division on every significand of the binades where
// their ranges meet: div_two and div2_two from their least dividends on, div2_tiny
// below.  -1: the divisor is refused.
long long harness_quotients_at_their_bounds(float y)
{
    const TwoOpLeast least = two_op_least(y);
    if (std::isinf(least.one)) return -1;
    float rh, rl;
    reciprocal_pair(y, &rh, &rl);
    long long bad = 0;
    auto walk = [&](float from, int binades, auto f) {
        const int k0 = std::ilogb(from);
        for (int k = k0; k < k0 + binades; ++k)
            for (uint32_t m = 0; m < (1u << 23); ++m) {
                const uint32_t bits = ((uint32_t)(127 + k) << 23) | m;
                float x;
                std::memcpy(&x, &bits, 4);
                f(x);
            }
    };
    walk(least.one, 3, [&](float x) { bad += x >= least.one && !same(div_two(x, rh, rl), x / y); });
    walk(least.two, 2, [&](float x) { bad += x >= least.two && !same(div2_two(x, rh, rl), (x / y) / y); });
    walk(0.5f * least.two, 2,
         [&](float x) { bad += x < least.two && !same(div2_tiny(x, y, rh, rl), (x / y) / y); });
    return bad;
}

// div2_tiny against (x / y) / y below kDiv2Lo, down to the subnormals.
long long harness_div2_tiny(float y)
{
    float rh, rl;
    reciprocal_pair(y, &rh, &rl);
    long long bad = 0;
    auto check = [&](float x) {
        if (!same(div2_tiny(x, y, rh, rl), (x / y) / y)) ++bad;
    };
    for (int k = -126; k < -80; ++k)
        for (uint32_t m = 0; m < (1u << 23); m += 61) {
            const uint32_t bits = ((uint32_t)(127 + k) << 23) | m;
            float x;
            std::memcpy(&x, &bits, 4);
            check(x);
            check(-x);
        }
    check(0.0f);
    check(-0.0f);
    for (uint32_t sub = 1; sub < (1u << 23); sub += sub < 100000 ? 1 : 41) {
        float x;
        std::memcpy(&x, &sub, 4);
        check(x);
        check(-x);
    }
    return bad;
}

// The kernels' mix (one FMA, else the split evaluation, else blend_mix)
// against the double formula.  *left counts the trials that reach blend_mix.
long long harness_mix(int pml0, long long trials, unsigned seed, long long *left)
{
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::uniform_int_distribution<int> E(-40, 40), M(-(1 << 20), 1 << 20);
    long long bad = 0, n = 0;
    for (int i = 0; i < pml0; ++i) {
        BlendCoef c;
        blend_coef_init(c, i, pml0);
        for (long long t = 0; t < trials; ++t) {
            float q = (float)(U(rng) * std::ldexp(1.0, E(rng)));
            float ext = q * (float)(1.0 + 0.3 * U(rng));
            switch (t % 16) {
            case 1: ext = (float)(U(rng) * std::ldexp(1.0, E(rng))); break;
            case 2: ext = (float)(-(c.omw * q) / c.w * (1.0 + 1e-6 * U(rng))); break;    // cancellation
            case 3: ext = (float)(-(c.omw * q) / c.w * (1.0 + 1e-3 * U(rng))); break;
            case 4: q = 0.0f; break;
            case 5: q = -0.0f; ext = 0.0f; break;
            case 6: ext = 0.0f; break;
            case 7: q = std::ldexp(q, -95); ext = std::ldexp(ext, -95); break;           // tails
            case 8: q = std::ldexp(q, -118); ext = std::ldexp(ext, -118); break;         // around 2^-126
            case 9: q = 1e-41f * (float)U(rng); ext = 1e-41f * (float)U(rng); break;      // subnormal
            case 10: q = std::ldexp(q, 85); ext = std::ldexp(ext, 85); break;            // near overflow
            case 11: q = std::ldexp((float)(M(rng) | 1), (int)(t / 16 % 40) - 20);         // short significands: ties
                     ext = std::ldexp((float)M(rng), (int)(t / 16 % 40) - 21); break;
            default: break;
            }
            const float a = c.w * ext;
            if (t % 16 >= 14 && c.omw > 0) {  // the sum near a float midpoint
                const float target = (float)(U(rng) * 4.0);
                const double mid = 0.5 * ((double)target + (double)std::nextafter(target, 10.0f));
                q = (float)((mid - (double)a) / c.omw);
            }
            float got;
            if (blend_one_fma(a, q, c.khi2, c.klo2))
                got = std::fma(c.bh, q, a);
            else if (!blend_mix_split(a, q, c.bh, c.bl, &got)) {
                got = blend_mix(a, q, c, 1);
                ++n;
            }
            if (!same(got, (float)((double)a + c.omw * (double)q))) ++bad;
        }
    }
    *left = n;
    return bad;
}

// The adjoint's mix against the double formula (any NaN is a NaN): values of all
// sizes, cancellations, short significands, sums near a float midpoint, infinities.
long long harness_mix_values(int pml0, long long trials, unsigned seed, int fp32_ok)
{
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::uniform_int_distribution<int> E(-148, 127), M(-(1 << 20), 1 << 20);
    long long bad = 0;
    for (int i = 0; i < pml0; ++i) {
        BlendCoef c;
        blend_coef_init(c, i, pml0);
        for (long long t = 0; t < trials; ++t) {
            const int e = E(rng);
            float q = (float)std::ldexp(U(rng), e), a = (float)(q * (1.0 + 0.3 * U(rng)) * c.w);
            switch (t % 8) {
            case 1: a = (float)std::ldexp(U(rng), E(rng)); break;
            case 2: a = (float)(-c.omw * q * (1.0 + std::ldexp(U(rng), -(int)(t / 8 % 30)))); break;
            case 3: q = std::ldexp((float)M(rng), e / 2); a = std::ldexp((float)M(rng), e / 2 - 1); break;
            case 4:
            case 5: {
                const float target = (float)(4.0 * U(rng));
                if (c.omw > 0) q = (float)((0.5 * ((double)target + std::nextafter(target, 9.0f)) - a) / c.omw);
                break;
            }
            case 6: (t & 8 ? a : q) = t & 16 ? INFINITY : -INFINITY; break;
            case 7: if (t & 8) q = t & 16 ? 0.0f : -0.0f; break;
            default: break;
            }
            const float got = blend_mix_values(a, q, c.bh, c.bl, c.khi2, c.klo2, fp32_ok);
            const float want = (float)((double)a + c.omw * (double)q);
            bad += !same(got, want) && !(std::isnan(got) && std::isnan(want));
        }
    }
    return bad;
}

}  // extern "C"

// Host check of fx::sumDouble (csrc/kernels/fixlimb.cuh): six non-negative doubles added left to right on FP32 limbs, the
// last rounding done with the assembly of the double, against the host FPU.
#include <cmath>
#include <cstring>

#include "../dvm-snapshot-r6603-fork_gb300/csrc/kernels/fixlimb.cuh"

static uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// nine binades from exponent field E: zeros, random, sparse, all-ones and few low bits, extremes of the range
static double operand(uint64_t r, uint64_t q, int E) {
    if (q % 12 == 0) return 0.0;
    uint64_t e = (uint64_t)E + (q >> 8) % 9, m = r & sf::MANT;
    if (q % 12 == 1) e = (uint64_t)E + 8;
    switch ((q >> 16) % 5) {
        case 0: m &= ~((1ull << ((q >> 24) % 53)) - 1); break;
        case 1: m |= (1ull << ((q >> 24) % 52)) - 1; break;
        case 2: m &= 7; break;
        case 3: m = sf::MANT; break;
        default: break;
    }
    return sf::from((e << 52) | m);
}

extern "C" long sumlimb_check(long n, uint64_t seed) {
    long bad = 0;
    for (long i = 0; i < n; i++) {
        const uint64_t c = mix(seed ^ (uint64_t)i * 0x9E37ull);
        const int E = c % 3 == 0 ? fx::E_MIN + (int)((c >> 8) % (fx::E_MAX - fx::E_MIN + 1)) : fx::E_DEFAULT;
        fx::Limbs<float> s{};
        volatile double t = 0.0;
        for (int k = 0; k < 6; k++) {
            const double x = operand(mix(c + 2 * k), mix(c + 2 * k + 1), E);
            const uint64_t X = sf::bits(x);
            bool ok = true;
            const fx::Raw r = fx::splitAny(sf::hi32(X), (uint32_t)X, fx::place(sf::hi32(X), E), ok);
            const fx::Limbs<float> v = fx::unbias<float>(fx::ffrom(r.h), fx::ffrom(r.m), fx::ffrom(r.l));
            bad += !ok;
            s = k == 0 ? v : k < 5 ? fx::add(s, v) : fx::plus(s, v);
            t = k == 0 ? x : t + x;
        }
        if (t == 0.0) continue;  // the caller's case
        bad += sf::bits(fx::sumDouble(s, E)) != sf::bits(t);
    }
    return bad;
}

// Host checks of csrc/kernels/fixlimb.cuh: chains of non-negative FP64 additions on FP32 limbs, the division of their
// sum by 6 and by 4, and the splitting of doubles, against the host FPU.
#include "../dvm-snapshot-r6603-fork_gb300/csrc/kernels/fixlimb.cuh"

using Limbs = fx::Limbs<float>;

static uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static bool same(double a, double b) { return sf::bits(a) == sf::bits(b); }

static Limbs limbs(double x, int E, bool &ok) {
    const uint64_t X = sf::bits(x);
    const uint32_t h = sf::hi32(X), l = (uint32_t)X, sh = fx::place(h, E);
    const fx::Raw r = sh <= 8u ? fx::split(h, l, sh) : fx::splitAny(h, l, sh, ok);
    return fx::unbias<float>(fx::ffrom(r.h), fx::ffrom(r.m), fx::ffrom(r.l));
}

// the integer (units 2^(E-1075)) that limbs stand for
static uint64_t whole(const Limbs &s) {
    return ((uint64_t)(s.h * 0x1p-11f) << 40) + ((uint64_t)s.m << 20) + (uint64_t)s.l;
}

// a value of the nine binades from exponent field E: significands with random, sparse, all-ones and few low bits, so
// that ties and carries into the next binade occur; mode: all binades, the upper two, the lower three
static double operand(uint64_t r, uint64_t q, int E, int mode) {
    if (q % 40 == 0) return 0.0;
    const uint64_t e = (uint64_t)E + (mode == 0 ? (q >> 8) % 9 : (mode == 1 ? 7 + (q >> 8) % 2 : (q >> 8) % 3));
    uint64_t m = r & sf::MANT;
    switch ((q >> 16) % 6) {
        case 0: m &= ~((1ull << ((q >> 24) % 53)) - 1); break;
        case 1: m |= (1ull << ((q >> 24) % 52)) - 1; break;
        case 2: m &= 7; break;
        default: break;
    }
    return sf::from((e << 52) | m);
}

extern "C" long fixlimb_check(long n, uint64_t seed) {
    volatile double six = 6.0, four = 4.0;
    long bad = 0;
    for (long i = 0; i < n; i++) {
        const uint64_t c = mix(seed ^ (uint64_t)i * 0x9E37ull);
        const int E = c % 4 == 0 ? fx::E_MIN + (int)((c >> 8) % (fx::E_MAX - fx::E_MIN + 1)) : fx::E_DEFAULT;
        const int mode = (int)((c >> 40) % 3);
        double t = 0;
        Limbs s{};
        for (int k = 0; k < 6; k++) {
            const double x = operand(mix(c + 2 * k), mix(c + 2 * k + 1), E, mode);
            bool ok = true;
            const Limbs v = limbs(x, E, ok);
            bad += !ok || std::ldexp((double)whole(v), E - 1075) != x;
            s = k == 0 ? v : fx::add(s, v);
            t = k == 0 ? x : t + x;
            // the sum, rounded as the FPU rounds it: it has 53 significant bits, so the conversion is exact
            bad += !same(std::ldexp((double)whole(s), E - 1075), t);
            if (k == 3 && fx::magnitude(s) >= 0x1p23f) {
                const fx::Quotient<float> w = fx::whole(s);
                bad += !same(fx::assemble(w.hm, w.mm, w.l, w.b, E, 2), t / four);
                bad += !same(fx::assemble(w.hm, w.mm, w.l, w.b, E), t);
            }
        }
        const float mag = fx::magnitude(s);
        if (mag >= fx::SMALL6) {
            const fx::Quotient<float> q = fx::div6(s);
            const double v = fx::assemble(q.hm, q.mm, q.l, q.b, E);
            bad += !same(v, t / six) || std::ldexp((double)fx::integer(v, E), E - 1075) != v;
        } else {
            bad += mag == 0.0f ? t != 0.0 : t / six >= std::ldexp(1.0, E - 1023);  // below 2^52 units
        }
    }
    return bad;
}

// what the splitting refuses: anything but +0 and the nine binades
extern "C" long fixlimb_check_range(void) {
    long bad = 0;
    const double out[] = {-0.0, -0.5, 1.0, 1.5, 0x1p-10, 0x1.fffffffffffffp-10, 5e-324, 1e300, INFINITY, -INFINITY, NAN};
    for (double x : out) {
        bool ok = true;
        (void)limbs(x, fx::E_DEFAULT, ok);
        bad += ok;
    }
    const double in[] = {0.0, 0x1p-9, 0x1.fffffffffffffp-1, 0.5, 0.1};
    for (double x : in) {
        bool ok = true;
        (void)limbs(x, fx::E_DEFAULT, ok);
        bad += !ok;
    }
    return bad;
}

// round63 against the FPU's rounding: integers of every length, ties and carries among them
extern "C" long fixlimb_check_round63(long n, uint64_t seed) {
    long bad = 0;
    for (long i = 0; i < n; i++) {
        const uint64_t r = mix(seed + 2 * (uint64_t)i), q = mix(seed + 2 * (uint64_t)i + 1);
        uint64_t a = (r | (1ull << 63)) >> (1 + q % 63);
        switch ((q >> 8) % 4) {
            case 0: a &= ~((1ull << ((q >> 16) % 60)) - 1); break;
            case 1: a |= (1ull << ((q >> 16) % 60)) - 1; break;
            case 2: a = (a & ~1023ull) | 512u | (a >> 12 & 1u); break;  // at and beside the tie of a full-length integer
            default: break;
        }
        a &= (1ull << 63) - 1;
        const int64_t v = (q >> 32) & 1 ? -(int64_t)a : (int64_t)a;
        const int E = fx::E_MIN + (int)((q >> 40) % (fx::E_MAX - fx::E_MIN + 1));
        bad += !same(fx::round63(v, E), std::ldexp((double)v, E - 1075));
    }
    return bad + !same(fx::round63(0, fx::E_DEFAULT), 0.0);
}

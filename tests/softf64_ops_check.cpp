// Host check of the grouped integer-pipe product (unpack, prod, in_range), the
// quotient (div), the square
// root (root), the comparison (less), the sum and
// difference (sum_diff, sum), the running
// sum of positive numbers (PosSum) and the FP32 -> FP64 conversion (widen) of dynearthsol-old_gb300/csrc/des_softf64.cuh against the
// host's IEEE arithmetic, bit for bit.
//   softf64_ops_check <pairs per kind>  -> one line per kind; exit 1 on a mismatch
#include "des_softf64.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>

using namespace des::sf;

static uint64_t splitmix(uint64_t &s)
{
    uint64_t z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// significands: any, zero, all ones, few bits at the top, few at the bottom
static double mk(uint64_t &s, uint64_t e)
{
    const uint64_t r = splitmix(s), k = splitmix(s);
    uint64_t f = r & kFrac;
    switch (k % 8) {
    case 0: f = 0; break;
    case 1: f = kFrac; break;
    case 2: f &= ~((1ull << (k >> 8) % 52) - 1); break;
    case 3: f &= (1ull << (k >> 8) % 52) - 1; break;
    }
    return from_bits((r & kSign) | (e << 52) | f);
}

// exponents: 0 near 1; 1 the edges of unpack's range; 2 any; 3 zeros,
// subnormals, infinities, NaN against anything; 4 equal or adjacent operands
static void pair(int kind, uint64_t &s, double &x, double &y)
{
    const uint64_t a = splitmix(s), b = splitmix(s);
    switch (kind) {
    case 0: x = mk(s, 1000 + a % 47); y = mk(s, 1000 + b % 47); break;
    case 1: x = mk(s, (a & 1 ? 510 : 1530) + (a >> 8) % 6); y = mk(s, (b & 1 ? 510 : 1530) + (b >> 8) % 6); break;
    case 2: x = mk(s, a % 2047); y = mk(s, b % 2047); break;
    case 3:
        x = mk(s, a & 1 ? 0 : 2047);
        y = mk(s, b & 1 ? (b >> 8) % 2048 : 1000 + (b >> 8) % 47);
        if (a & 2) x = from_bits(bits(x) & (kSign | kInf));
        if (b & 2) { const double t = x; x = y; y = t; }
        break;
    default: x = mk(s, 1000 + a % 47); y = from_bits(bits(x) + b % 7 - 3); break;
    }
}

static bool same(double a, double b) { return bits(a) == bits(b) || (std::isnan(a) && std::isnan(b)); }

int main(int argc, char **argv)
{
    const long long per = argc > 1 ? atoll(argv[1]) : 1000000;
    long long total = 0;
    for (int kind = 0; kind < 5; ++kind) {
        uint64_t s = 0xd1f0000ull + 1000003ull * kind;
        long long bad = 0, grouped = 0;
        for (long long i = 0; i < per; ++i) {
            double x, y;
            pair(kind, s, x, y);
            volatile double vx = x, vy = y;
            const double m = vx * vy, q = vx / vy;
            uint32_t far = 0;
            const Op a = unpack(x, far), b = unpack(y, far);
            if (in_range(far)) {
                ++grouped;
                bad += bits(m) != bits(prod(a, b));
                // two products of such operands; a pair that falls outside
                // sum_diff's range says so
                double p, d;
                bool rare = false;
                const double other = kind == 4 ? from_bits(bits(m) ^ (i & 1 ? kSign : 0) ^ (uint64_t)(i % 3)) : vx;
                volatile double vo = other, vm = m;
                const double hs = vm + vo, hd = vm - vo;
                sum_diff(m, other, p, d, rare);
                bad += !rare && (bits(hs) != bits(p) || bits(hd) != bits(d));
                rare = false;
                p = sum(m, other, rare);
                bad += !rare && bits(hs) != bits(p);
            }
            bad += !same(q, div(x, y));
            const double sq = std::sqrt(vx);
            bad += !same(sq, root(x));
            bad += less(x, y) != (vx < vy);
        }
        // the range itself: kinds 0 and 4 lie inside it, kind 3's infinities never do
        if ((kind == 0 || kind == 4) && grouped != per) ++bad;
        printf("kind %d: %lld pairs, %lld mismatches\n", kind, per, bad);
        total += bad;
    }
    // sums of 1-30 terms whose exponents spread over 1, 4 or 14 binades; now and
    // then a zero, a negative, an infinite or a subnormal term among them
    const int spread[3] = {1, 4, 14};
    for (int kind = 0; kind < 3; ++kind) {
        uint64_t s = 0x5005000ull + kind;
        long long bad = 0, sums = 0;
        for (long long i = 0; i < per / 4; ++i) {
            const int n = 1 + (int)(splitmix(s) % 30), odd = i % 50 == 0 ? (int)(splitmix(s) % n) : -1;
            const uint64_t base = 200 + splitmix(s) % 1500;
            PosSum p = pos_first(1.0);
            volatile double h = 0;
            for (int j = 0; j < n; ++j) {
                double x = std::fabs(mk(s, base + splitmix(s) % spread[kind]));
                if (j == odd) x = i % 200 == 0 ? 0.0 : i % 200 == 50 ? -x : i % 200 == 100 ? INFINITY : 5e-324;
                h = h + x;
                if (j)
                    pos_add(p, x);
                else
                    p = pos_first(x);
            }
            if (exact(p)) {
                ++sums;
                bad += bits(h) != bits(value(p));
            }
        }
        // terms of one binade always stay within the sum's reach, unless one is odd
        if (kind == 0 && sums < per / 4 * 97 / 100) ++bad;
        printf("sums %d: %lld, %lld mismatches\n", kind, sums, bad);
        total += bad;
    }
    long long bad = 0;
    for (uint64_t i = 0; i < (1ull << 32); i += 257) {
        const float f = float_from_bits((uint32_t)i);
        bad += !same((double)f, widen(f));
    }
    printf("widen: %lld mismatches\n", bad);
    total += bad;
    return total ? 1 : 0;
}

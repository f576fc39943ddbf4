// Host build of the reciprocal-based divisions of the 6x6 solve
// (ornis_gb300/csrc/avbd_rows.cuh) against the IEEE operations: div_by over
// random operands of its range, solve_6x6_div over random systems.  Prints
// one line per check: cases tried, cases the range test sent back, mismatches.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../ornis_gb300/csrc/avbd_rows.cuh"

using namespace avbd;
static uint64_t st = 0x853c49e6748fea9bull;
static uint32_t rnd() {
    st = st * 6364136223846793005ull + 1442695040888963407ull;
    return (uint32_t)(st >> 32);
}
static float u2f(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static uint32_t f2u(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static float uni() { return (float)(rnd() >> 8) * 0x1p-24f; }

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long back = 0, bad = 0;
    for (long i = 0; i < n; i++) {
        // pivots and numerators of any mantissa over (and a little beyond) the stated exponents
        const float b = u2f((uint32_t)(127 - 42 + rnd() % 84) << 23 | (rnd() & 0x7fffffu));
        float a = u2f((rnd() & 0x80000000u) | (uint32_t)(127 - 88 + rnd() % 172) << 23 | (rnd() & 0x7fffffu));
        if (i % 17 == 0) a = (i & 1) ? 0.0f : -0.0f;
        if (i % 5 == 0) a = b * u2f(0x3f800000u | (rnd() & 0x7fffffu));  // quotients near a float
        bool off = false;
        const Recip r = recip_of(b, off);
        const float q = div_by(a, r, off);
        if (off) { back++; continue; }
        if (f2u(q) != f2u(a / b)) {
            if (bad++ < 5) printf("  %a / %a = %a, IEEE %a\n", a, b, q, a / b);
        }
    }
    printf("div_by %ld %ld %ld\n", n, back, bad);
    long sbad = 0, fail = 0;
    for (long i = 0; i < n / 10; i++) {
        Sys s;
        for (float& v : s.h) v = 0.0f;
        const float scale = ldexpf(1.0f, (int)(rnd() % 60) - 25);
        for (int k = 0; k < 6; k++) s.h[tri(k, k)] = scale * (0.5f + uni());
        const int rows = (int)(rnd() % 12);
        for (int j = 0; j < rows; j++) {
            V3 nrm{uni() - 0.5f, uni() - 0.5f, uni() - 0.5f}, r{uni() - 0.5f, uni() - 0.5f, uni() - 0.5f};
            if (j % 3 == 0) nrm = V3{0.0f, 1.0f, 0.0f};  // zero couplings
            stamp_row(s, nrm, ldexpf(1.0f + uni(), (int)(rnd() % 33)), 0.0f, r, (j & 1) ? -1.0f : 1.0f);
        }
        if (i % 50 == 0) s.h[tri(3, 3)] = -1.0f;  // a breakdown
        for (float& v : s.r) v = rnd() % 4 ? scale * (uni() - 0.5f) : 0.0f;
        float x[6] = {0, 0, 0, 0, 0, 0}, y[6] = {0, 0, 0, 0, 0, 0};
        const bool ok = solve_6x6_div(s, x), want = solve_6x6(s, y);
        if (!want) fail++;
        bool same = ok == want;
        for (int k = 0; want && k < 6; k++) same = same && (f2u(x[k]) == f2u(y[k]) || (x[k] != x[k] && y[k] != y[k]));
        if (!same) sbad++;
    }
    printf("solve %ld %ld %ld\n", n / 10, fail, sbad);
    return 0;
}

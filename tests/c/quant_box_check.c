/* quant_box_check.c -- property test of the 8-wide walk's box test (csrc/trace_quant.cuh:
 * quant_axis, quant_advance): for every ray the walk trusts, a quantised box that contains
 * a box which CollideBox (collision.glsl:23-40) accepts is accepted too.
 *
 * The grid (origin o, step 2^e per axis) and the bytes are drawn, the reference's box is
 * the quantised one or lies inside it, its planes pulled towards the ray's origin and to
 * the point at tmax, one ulp either side.
 *
 * Usage: quant_box_check <cases> <seed>; prints counts, exits 1 on a violation.
 * Built with -O2 -ffp-contract=off (the library uses --fmad=false). */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static uint64_t g_s;
static uint64_t rnd(void) {
    g_s ^= g_s << 13; g_s ^= g_s >> 7; g_s ^= g_s << 17;
    return g_s;
}
static double uni(void) { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); }
static float bits(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }

static int collide_box(const float o[3], const float d[3], const float lo[3], const float hi[3], float tmax) {
    float n = 0.0f, f = tmax;
    for (int a = 0; a < 3; ++a) {
        const float t0 = (lo[a] - o[a]) / d[a], t1 = (hi[a] - o[a]) / d[a];
        n = fmaxf(n, fminf(t0, t1));
        f = fminf(f, fmaxf(t0, t1));
    }
    return n < f;
}

static int quant_hit(const float r[3], const float d[3], const float org[3], const int e[3], const int qlo[3], const int qhi[3], float tmax) {
    float n = 0.0f, f = tmax;
    for (int a = 0; a < 3; ++a) {
        const float inv = 1.0f / d[a], B = bits((uint32_t)(e[a] + 127) << 23) * inv, A = (org[a] - r[a]) * inv;
        const float C = fmaf(-32768.0f, B, A), m = fmaf(fabsf(A), 3.814697265625e-06f, fabsf(B) * 0.015625f);
        const int neg = inv < 0.0f;
        const float pn = bits(0x47000000u | (uint32_t)(neg ? qhi[a] : qlo[a]) << 8), pf = bits(0x47000000u | (uint32_t)(neg ? qlo[a] : qhi[a]) << 8);
        n = fmaxf(n, fmaf(pn, B, C - m));
        f = fminf(f, fmaf(pf, B, C + m));
    }
    return n < f;
}

int main(int argc, char** argv) {
    const long cases = argc > 1 ? atol(argv[1]) : 1000000;
    g_s = 88172645463325252ull ^ (argc > 2 ? strtoull(argv[2], 0, 10) * 0x9E3779B97F4A7C15ull : 0);
    long tested = 0, entered = 0, missed = 0, lost = 0;
    for (long c = 0; c < cases; ++c) {
        const double scale = uni() < 0.1 ? exp((uni() - 0.5) * 70.0) : exp((uni() - 0.5) * 16.0);
        float o[3], d[3], org[3], lo[3], hi[3];
        int e[3], qlo[3], qhi[3], ok = 1;
        const float tmax = uni() < 0.2 ? INFINITY : (float)(scale * exp((uni() - 0.5) * 12.0));
        for (int a = 0; a < 3; ++a) {
            o[a] = (float)((uni() * 2.0 - 1.0) * scale * (uni() < 0.05 ? 1e4 : 1.0));
            d[a] = (float)(uni() * 2.0 - 1.0);
            if (uni() < 0.1) d[a] = (float)(d[a] * exp(-uni() * 40.0));
            if (uni() < 0.05) d[a] = (float)(d[a] * exp(uni() * 20.0));
            ok = ok && fabsf(d[a]) >= 3.469446951953614e-18f && fabsf(o[a]) <= 1.152921504606847e18f;
            e[a] = (int)floor(log2(scale)) - (int)(rnd() % 20u);
            const double step = ldexp(1.0, e[a]);
            qlo[a] = (int)(rnd() % 256u);
            qhi[a] = qlo[a] + (int)(rnd() % (uint32_t)(256 - qlo[a]));
            /* the grid's origin such that a plane, or a place between two, meets the ray's origin or its end */
            const double q = uni(), at = uni() < 0.5 ? qlo[a] : qhi[a];
            if (q < 0.4) org[a] = (float)(o[a] - at * step);
            else if (q < 0.7) org[a] = (float)(o[a] + (double)d[a] * (isfinite(tmax) ? tmax : 10.0 * scale) - at * step);
            else org[a] = (float)((uni() * 2.0 - 1.0) * scale);
            if (!(fabsf(org[a]) <= 1.1e18f)) { ok = 0; break; }
            /* the reference's box: floats within the quantised one */
            const double x0 = (double)org[a] + step * qlo[a], x1 = (double)org[a] + step * qhi[a];
            lo[a] = (float)x0;
            if ((double)lo[a] < x0) lo[a] = nextafterf(lo[a], INFINITY);
            hi[a] = (float)x1;
            if ((double)hi[a] > x1) hi[a] = nextafterf(hi[a], -INFINITY);
            if (!(lo[a] <= hi[a])) { ok = 0; break; }
            if (uni() < 0.2) lo[a] = lo[a] + (hi[a] - lo[a]) * (float)uni();
            if (lo[a] > hi[a]) lo[a] = hi[a];
        }
        if (!ok) continue;
        ++tested;
        const int want = collide_box(o, d, lo, hi, tmax), got = quant_hit(o, d, org, e, qlo, qhi, tmax);
        entered += want;
        missed += !got;
        lost += want && !got;
    }
    printf("tested %ld entered %ld missed %ld lost %ld\n", tested, entered, missed, lost);
    return lost ? 1 : 0;
}

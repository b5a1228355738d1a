/* walk_box_check.c -- property test of the box tests of the binary form's two walks.
 *
 * any (csrc/trace_any.cuh: any_init, any_advance): the any-hit rays' test of one box,
 *   planes as fused multiply-adds p * inv + (-o * inv -+ m), m = W |inv|,
 *   W = max(2^-20 (P + |o|), 2^-60), P the largest plane magnitude of the axis, zero
 *   direction components replaced by +-2^-80. Property: for every ray the walk takes,
 *   it accepts each box that CollideBox (collision.glsl:23-40) accepts.
 * pair (csrc/trace_pair.cuh: pair_advance): the closest-hit rays' test of two sibling
 *   boxes. Property: what it decides without divisions (hit or miss of each box, and,
 *   when both are hit, whether child 1 is entered first) is CollideBox's decision.
 *
 * inv is RN(1/d) or either neighbour, as the kernels' 1-ulp reciprocal may give.
 * Cases sit on the boundary: planes through the origin, through the point at tmax and
 * through a sibling's planes, one ulp either side, flat boxes, zero and tiny
 * components, far origins, tmax from 1e-3 to infinity.
 *
 * Usage: walk_box_check <cases> <seed>; prints counts, exits 1 on a violation.
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

static float collide_box(const float o[3], const float d[3], const float lo[3], const float hi[3], float tmax) {
    float s[3], b[3];
    for (int a = 0; a < 3; ++a) {
        const float t0 = (lo[a] - o[a]) / d[a], t1 = (hi[a] - o[a]) / d[a];
        s[a] = fminf(t0, t1);
        b[a] = fmaxf(t0, t1);
    }
    const float tmin = fmaxf(0.0f, fmaxf(s[0], fmaxf(s[1], s[2])));
    const float tm = fminf(tmax, fminf(b[0], fminf(b[1], b[2])));
    return tmin < tm ? tmin : -1.0f;
}

static float rcp(float x) {   /* 1 ulp */
    const float r = 1.0f / x;
    if (!isfinite(r) || r == 0.0f) return r;
    const int k = (int)(rnd() % 3u) - 1;
    return k < 0 ? nextafterf(r, -INFINITY) : (k > 0 ? nextafterf(r, INFINITY) : r);
}
/* max.NaN / min.NaN: NaN when an operand is */
static float maxn(float a, float b) { return isnan(a) || isnan(b) ? NAN : fmaxf(a, b); }
static float minn(float a, float b) { return isnan(a) || isnan(b) ? NAN : fminf(a, b); }

typedef struct { float inv[3], an[3], af[3]; int ok; } AnyRay;

static AnyRay any_init(const float o[3], const float d[3], const float bound[3], float tmax) {
    AnyRay r;
    float m[3], reach[3], tb = tmax;
    int zero = 0;
    r.ok = tmax == tmax;
    for (int a = 0; a < 3; ++a) {
        const int z = d[a] == 0.0f;
        r.inv[a] = rcp(z ? copysignf(8.271806125530277e-25f, d[a]) : d[a]);
        reach[a] = bound[a] + fabsf(o[a]);
        m[a] = fmaxf(reach[a] * 9.5367431640625e-07f, 8.673617379884035e-19f) * fabsf(r.inv[a]);
        const float x = o[a] * r.inv[a];
        r.an[a] = -x - m[a];
        r.af[a] = m[a] - x;
        r.ok = r.ok && fabsf(o[a]) <= 1.099511627776e12f && (z || (fabsf(d[a]) >= 8.673617379884035e-19f && fabsf(d[a]) <= 1.152921504606847e18f));
        if (z) zero = 1;
        else tb = fminf(tb, 1.01f * reach[a] * fabsf(r.inv[a]));
    }
    tb *= 2.0f;
    if (zero)
        for (int a = 0; a < 3; ++a)
            if (d[a] == 0.0f) r.ok = r.ok && m[a] >= tb;
    return r;
}

static int any_hit(const AnyRay* r, const float lo[3], const float hi[3], float tmax) {
    float tn = 0.0f, tf = tmax;
    for (int a = 0; a < 3; ++a) {
        const int neg = r->inv[a] < 0.0f;
        tn = fmaxf(tn, fmaf(neg ? hi[a] : lo[a], r->inv[a], r->an[a]));
        tf = fminf(tf, fmaf(neg ? lo[a] : hi[a], r->inv[a], r->af[a]));
    }
    return tn < tf;
}

/* -1 undecided; else bit 0 child 0 hit, bit 1 child 1 hit, bit 2 child 1 first (both hit) */
static int pair_decide(const float o[3], const float d[3], float lo[2][3], float hi[2][3], float tmax) {
    const float up = 1.0f + 3.814697265625e-06f, down = 1.0f - 3.814697265625e-06f;
    float tiny = 7.888609052210118e-31f, u[2], n[2], T[2], near[2][3];
    for (int a = 0; a < 3; ++a) {
        const float x = fabsf(d[a]);
        if (!(x == 0.0f || (x >= 7.888609052210118e-31f && x <= 1.2676506002282294e30f))) tiny = INFINITY;
    }
    if (!(tmax <= 1.2676506002282294e30f)) tiny = INFINITY;
    float inv[3];
    for (int a = 0; a < 3; ++a) inv[a] = rcp(d[a]);
    for (int k = 0; k < 2; ++k) {
        float far[3];
        for (int a = 0; a < 3; ++a) {
            const int neg = signbit(d[a]) != 0;
            near[k][a] = ((neg ? hi[k][a] : lo[k][a]) - o[a]) * inv[a];
            far[a] = ((neg ? lo[k][a] : hi[k][a]) - o[a]) * inv[a];
        }
        u[k] = maxn(near[k][0], maxn(near[k][1], near[k][2]));
        n[k] = maxn(u[k], 0.0f);
        T[k] = minn(minn(far[0], far[1]), minn(far[2], tmax));
    }
    int h[2], m[2];
    for (int k = 0; k < 2; ++k) {
        h[k] = fmaf(T[k], down, -n[k]) > tiny;
        m[k] = fmaf(T[k], up, -n[k]) < -tiny;
    }
    const int f0 = u[0] < -tiny || fmaf(n[0], up, -n[1]) < -tiny;
    int first1 = fmaf(n[1], up, -n[0]) < -tiny;
    const int order = f0 || first1 || !(h[0] && h[1]);
    if (!((h[0] || m[0]) && (h[1] || m[1]) && order)) {
        const float l = fminf(n[0], n[1]);
        if (!(h[0] && h[1])) return -1;
        for (int a = 0; a < 3; ++a) {
            const int neg = signbit(d[a]) != 0;
            const float p0 = neg ? hi[0][a] : lo[0][a], p1 = neg ? hi[1][a] : lo[1][a];
            if (!(p0 == p1 || fmaf(fmaxf(near[0][a], near[1][a]), up, -l) < -tiny)) return -1;
        }
    }
    return h[0] | h[1] << 1 | (h[0] && h[1] ? first1 << 2 : 0);
}

int main(int argc, char** argv) {
    const long cases = argc > 1 ? atol(argv[1]) : 1000000;
    g_s = 88172645463325252ull ^ (argc > 2 ? strtoull(argv[2], 0, 10) * 0x9E3779B97F4A7C15ull : 0);
    long any_cases = 0, any_accept = 0, any_lost = 0, pair_decided = 0, pair_open = 0, pair_wrong = 0;
    for (long c = 0; c < cases; ++c) {
        const double scale = exp((uni() - 0.5) * 16.0);
        float o[3], d[3], lo[2][3], hi[2][3];
        for (int a = 0; a < 3; ++a) {
            o[a] = (float)((uni() * 2.0 - 1.0) * scale * (uni() < 0.05 ? 1e4 : 1.0));
            d[a] = (float)(uni() * 2.0 - 1.0);
            const double q = uni();
            if (q < 0.08) d[a] = uni() < 0.5 ? 0.0f : -0.0f;
            else if (q < 0.14) d[a] = (float)(d[a] * exp(-uni() * 40.0));
            else if (q < 0.15) d[a] = (float)(d[a] * 1e-39);
        }
        const double w = uni();
        float tmax = w < 0.1 ? INFINITY : (w < 0.2 ? 100.0f : (float)(scale * exp((uni() - 0.5) * 12.0)));
        for (int k = 0; k < 2; ++k)
            for (int a = 0; a < 3; ++a) {
                float p[2];
                for (int e = 0; e < 2; ++e) {
                    const double q = uni();
                    if (q < 0.25) p[e] = o[a];                                        /* through the origin */
                    else if (q < 0.5) p[e] = (float)(o[a] + (double)d[a] * (isfinite(tmax) ? tmax : 10.0 * scale));
                    else if (q < 0.6 && k == 1) p[e] = uni() < 0.5 ? lo[0][a] : hi[0][a];   /* a sibling's plane */
                    else p[e] = (float)((uni() * 2.0 - 1.0) * scale);
                    const int s = (int)(rnd() % 5u);
                    if (s == 0) p[e] = nextafterf(p[e], INFINITY);
                    if (s == 1) p[e] = nextafterf(p[e], -INFINITY);
                }
                if (uni() < 0.05) p[1] = p[0];
                lo[k][a] = fminf(p[0], p[1]);
                hi[k][a] = fmaxf(p[0], p[1]);
            }
        float bound[3];
        for (int a = 0; a < 3; ++a)
            bound[a] = fmaxf(fmaxf(fabsf(lo[0][a]), fabsf(hi[0][a])), fmaxf(fabsf(lo[1][a]), fabsf(hi[1][a])));
        const float d0 = collide_box(o, d, lo[0], hi[0], tmax), d1 = collide_box(o, d, lo[1], hi[1], tmax);
        const AnyRay r = any_init(o, d, bound, tmax);
        if (r.ok) {
            ++any_cases;
            for (int k = 0; k < 2; ++k) {
                const int hit = any_hit(&r, lo[k], hi[k], tmax);
                any_accept += hit;
                if ((k ? d1 : d0) >= 0.0f && !hit) ++any_lost;
            }
        }
        const int q = pair_decide(o, d, lo, hi, tmax);
        if (q < 0) {
            ++pair_open;
        } else {
            ++pair_decided;
            const int want = (d0 >= 0.0f) | (d1 >= 0.0f) << 1 | (d0 >= 0.0f && d1 >= 0.0f ? (d1 < d0) << 2 : 0);
            if (q != want) ++pair_wrong;
        }
    }
    printf("any_cases %ld any_accept %ld any_lost %ld pair_decided %ld pair_open %ld pair_wrong %ld\n", any_cases, any_accept,
           any_lost, pair_decided, pair_open, pair_wrong);
    return any_lost || pair_wrong ? 1 : 0;
}

/* Check of the float forms with exact rounding errors that
 * kittlespt_gb300/csrc/kpt_fsr.cu and kpt_post.cu use in place of the
 * reference's double-precision expressions (upscale.cuh, color.cuh): over
 * every float input where there is one input, over random ones (spread over
 * the exponents the kernels can see, subnormals among them) where there are
 * two or three.  Prints, per expression, the inputs, how many of them give
 * another float than the double form, and on how many the float form does not
 * decide (the kernels then take the double form).  Compiled without
 * contraction; fmaf is the correctly rounded fused multiply-add, as on the
 * GPU. */
#include <math.h>
#include <pthread.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

static float f_of(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static uint32_t u_of(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }

#define NT 16
enum { LOBE, HALF, LUMA, W00, W10, STRETCH, XYY, KINDS };
static const char* names[KINDS] = {"lobe", "half", "luma", "weight00", "weight10", "stretch", "xyy"};
static long long bad[NT][KINDS], unsure[NT][KINDS], total[NT][KINDS];
#define PER_THREAD 4000000

typedef struct { float h, l; } two;
static two two_sum(float a, float b) {
    const float s = a + b, t = s - a;
    two r = {s, (a - (s - t)) + (b - t)};
    return r;
}
static const float C29 = 0.29f, CL29 = (float)(0.29 - (double)0.29f);

/* sure: the candidates agree, so the double form is not asked */
static float rounded(float h, float l, float e, int* sure) {
    const float lo = h + (l - e), hi = h + (l + e);
    *sure = lo == hi;
    return lo;
}
static float lobe(float len, int* sure) {                 /* 0.5 - 0.29 len */
    const float p = C29 * len, pl = fmaf(C29, len, -p);
    const two s = two_sum(0.5f, -p);
    return rounded(s.h, s.l - fmaf(CL29, len, pl), 0x1p-46f, sure);
}
static float weight00(float x, float y, int* sure) {      /* (1 - x) (1 - y) */
    const two u = two_sum(1.0f, -x), v = two_sum(1.0f, -y);
    const float p = u.h * v.h, pl = fmaf(u.h, v.h, -p);
    return rounded(p, fmaf(u.h, v.l, fmaf(u.l, v.h, pl)), p * 0x1p-44f, sure);
}
static float weight10(float x, float y, int* sure) {      /* x (1 - y) */
    const two v = two_sum(1.0f, -y);
    const float p = x * v.h, pl = fmaf(x, v.h, -p);
    return rounded(p, fmaf(x, v.l, pl), p * 0x1p-44f, sure);
}
static float stretched(float s, float len, int* sure) {   /* 1 + (s - 1) len */
    const two a = two_sum(s, -1.0f);
    const float p = a.h * len, pl = fmaf(a.h, len, -p);
    const two r = two_sum(1.0f, p);
    return rounded(r.h, r.l + fmaf(a.l, len, pl), 0x1p-44f, sure);
}
static float luminance_z(float Y, float cx, float cy, int* sure) {   /* Y (1 - cx - cy) / cy */
    const two a = two_sum(1.0f, -cx), b = two_sum(a.h, -cy), m = two_sum(b.h, a.l + b.l);
    const float p = Y * m.h, pl = fmaf(Y, m.l, fmaf(Y, m.h, -p));
    const float rc = 1.0f / cy, q = p * rc;
    return rounded(q, (fmaf(-q, cy, p) + pl) * rc, fabsf(q) * 0x1p-44f, sure);
}

static uint64_t rng(uint64_t* s) { *s ^= *s << 13; *s ^= *s >> 7; *s ^= *s << 17; return *s; }
static float unit(uint64_t* s) { return (float)((rng(s) >> 40) * 0x1p-24); }
/* a positive float with its exponent uniform in [lo, hi] */
static float wide(uint64_t* s, int lo, int hi) {
    const int e = lo + (int)((rng(s) >> 33) % (uint64_t)(hi - lo + 1));
    return (float)ldexp(1.0 + (double)((rng(s) >> 41)) * 0x1p-23, e);
}
static void note(int t, int k, float a, float d, int sure) {
    total[t][k]++;
    if (!sure) unsure[t][k]++;
    else if (u_of(a) != u_of(d)) bad[t][k]++;
}

static void* work(void* arg) {
    const int t = (int)(intptr_t)arg;
    int ok;
    float f;
    for (uint32_t u = (uint32_t)t; u <= u_of(1.0f); u += NT) {
        const float len = f_of(u);
        f = lobe(len, &ok);
        note(t, LOBE, f, (float)(0.5 - 0.29 * (double)len), ok);
    }
    for (uint32_t u = (uint32_t)t; u <= u_of(4.0f); u += NT)
        note(t, HALF, f_of(u) * 0.5f, (float)((double)f_of(u) * 0.5), 1);
    uint64_t s = 0x9e3779b97f4a7c15ull * (uint64_t)(t + 1);
    for (int i = 0; i < PER_THREAD; ++i) {
        const int tiny = i % 4 == 0;
        const float y = tiny ? f_of((uint32_t)(rng(&s) >> 39)) : wide(&s, -60, 27);
        const float z = tiny ? f_of((uint32_t)(rng(&s) >> 38)) : wide(&s, -60, 27);
        note(t, LUMA, 0.5f * (2.0f * y + z), (float)((double)y + 0.5 * (double)z), 1);
        const float px = i % 5 ? unit(&s) : wide(&s, -40, -1), py = i % 3 ? unit(&s) : wide(&s, -40, -1);
        const double dx = px, dy = py;
        f = weight00(px, py, &ok);
        note(t, W00, f, (float)((1.0 - dx) * (1.0 - dy)), ok);
        f = weight10(px, py, &ok);
        note(t, W10, f, (float)(dx * (1.0 - dy)), ok);
        const float st = 1.0f + 0.41421357f * unit(&s), len = i % 2 ? unit(&s) : wide(&s, -40, -1);
        f = stretched(st, len, &ok);
        note(t, STRETCH, f, (float)(1.0 + ((double)st - 1.0) * (double)len), ok);
        /* the luminances and chromaticities the float form takes */
        const float cy = i % 3 ? 0.01f + 0.83f * unit(&s) : wide(&s, -10, -1);
        const float cx = i % 5 ? (0.99f - cy) * unit(&s) : wide(&s, -60, -1), Y = wide(&s, -40, 59);
        f = luminance_z(Y, cx, cy, &ok);
        note(t, XYY, f, (float)((double)Y * (1.0 - (double)cx - (double)cy) / (double)cy), ok);
    }
    return 0;
}

int main(void) {
    pthread_t th[NT];
    for (int t = 0; t < NT; ++t) pthread_create(&th[t], 0, work, (void*)(intptr_t)t);
    for (int t = 0; t < NT; ++t) pthread_join(th[t], 0);
    for (int k = 0; k < KINDS; ++k) {
        long long b = 0, f = 0, n = 0;
        for (int t = 0; t < NT; ++t) { b += bad[t][k]; f += unsure[t][k]; n += total[t][k]; }
        printf("%s %lld %lld %lld\n", names[k], n, b, f);
    }
    return 0;
}

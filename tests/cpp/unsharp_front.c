/*
 * Host check of unsharp_front_f32 (itk-rs_gb300/csrc/unsharp.cuh), restated
 * operation for operation (keep the two in step), against the reference's f64
 * sequence (edges.rs:440-448, `v as f32`): whenever it decides a voxel, its
 * result equals the reference's bit for bit.  f32 amounts only; pairs over the
 * whole exponent range, near-equal and close ones, dyadic grids (where ties
 * are common), thresholds at and beside |o - b|, and the underflow guards.
 * Build: gcc -O2 -ffp-contract=off unsharp_front.c -lm
 */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static float fa(float a, float b) { volatile float r = a + b; return r; }
static float fs(float a, float b) { volatile float r = a - b; return r; }
static float fm(float a, float b) { volatile float r = a * b; return r; }
static void two_sum(float a, float b, float* s, float* t) {
  *s = fa(a, b);
  float a1 = fs(*s, b), b1 = fs(*s, a1);
  *t = fa(fs(a, a1), fs(b, b1));
}

static int front(float o, float b, float ah, float up, float dn, int thr_neg, float* out) {
  float eh, el, sh, s1, p2, p2e, s2, s2e;
  two_sum(o, -b, &eh, &el);
  const float ae = fabsf(eh), ph = fm(ah, eh), t = fmaf(ah, eh, -ph), c = fm(ah, el), ce = fmaf(ah, el, -c);
  two_sum(o, ph, &sh, &s1);
  two_sum(t, c, &p2, &p2e);
  two_sum(s1, p2, &s2, &s2e);
  const int zero = eh == 0.0f, pass = ae > up, stay = ae < dn;
  const int exact = ce == 0.0f && p2e == 0.0f && s2e == 0.0f && (el == 0.0f || fabsf(el) >= fm(ae, 0x1p-29f)) &&
                    (p2 == 0.0f || fabsf(p2) >= fm(fabsf(ph), 0x1p-29f));
  const int sized = ae >= 0x1p-60f && fabsf(ph) >= 0x1p-60f && fabsf(ph) < 0x1p100f;
  *out = pass && !zero ? fa(sh, s2) : o;
  return fmaxf(fabsf(o), fabsf(b)) < 0x1p90f && (zero ? !thr_neg : stay || (pass && exact && sized));
}

static uint64_t rs = 0x9E3779B97F4A7C15ull;
static uint64_t rnd(void) { rs ^= rs << 13; rs ^= rs >> 7; rs ^= rs << 17; return rs; }
static double unif(void) { return (rnd() >> 11) * 0x1p-53; }

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 2000000;
  long undecided = 0, common = 0, common_undecided = 0, bad = 0;
  for (long i = 0; i < n; ++i) {
    const int mode = (int)(i % 6);
    float o, b;
    if (mode == 0) { o = (float)(3 * unif()); b = (float)(o + 0.1 * (unif() - 0.5)); }
    else if (mode == 1) { o = (float)((unif() - 0.5) * 1000); b = (float)((unif() - 0.5) * 1000); }
    else if (mode == 2) { uint32_t u = (uint32_t)rnd(), w = (uint32_t)rnd(); memcpy(&o, &u, 4); memcpy(&b, &w, 4); }
    else if (mode == 3) { o = (float)ldexp(unif() - 0.5, (int)(rnd() % 200) - 120); b = (float)(o * (1 + ldexp(unif() - 0.5, -(int)(rnd() % 24)))); }
    else if (mode == 4) { o = (float)(rnd() % 256) + 0.5f * (float)(rnd() % 2); b = (float)(rnd() % 4096) / 16.0f; }
    else { o = (float)(1 + unif()); b = (float)ldexp(1 + unif(), -(int)(rnd() % 60)); }
    double a;
    switch (rnd() % 5) {
      case 0: a = 0.5; break;
      case 1: a = 1.25; break;
      case 2: a = (double)(float)(unif() * 4 - 2); break;
      case 3: a = (double)(float)ldexp(unif() + 0.5, (int)(rnd() % 58) - 29); break;
      default: a = -0.75;
    }
    const double e = (double)o - (double)b;
    double thr;
    switch (rnd() % 5) {
      case 0: thr = 0; break;
      case 1: thr = fabs(e) * (1 + (unif() - 0.5) * 1e-5); break;
      case 2: thr = -1; break;
      case 3: thr = fabs(e); break;
      default: thr = 0.1 * unif();
    }
    float up = -1, dn = -1;
    if (thr > 0) {
      const double u = thr * (1 + 0x1p-20), d = thr * (1 - 0x1p-20);
      up = (float)u, dn = (float)d;
      if ((double)up < u) up = nextafterf(up, INFINITY);
      if ((double)dn > d) dn = nextafterf(dn, 0);
      if (thr < 0x1p-100) { if (up < 0x1p-100f) up = 0x1p-100f; dn = 0; }
    }
    volatile double p = a * e, v = o + p;
    const float want = (float)(fabs(e) > thr ? v : (double)o);
    float got;
    const int usual = mode == 0 && (a == 0.5 || a == 1.25) && thr <= 0;
    common += usual;
    if (!front(o, b, (float)a, up, dn, thr < 0, &got)) { ++undecided; common_undecided += usual; continue; }
    if (memcmp(&got, &want, 4)) {
      if (bad++ < 5) printf("mismatch o=%a b=%a amount=%a threshold=%a: %a vs %a\n", o, b, a, thr, got, want);
    }
  }
  printf("%ld cases, %ld undecided (%ld of %ld usual ones), %ld mismatches\n", n, undecided, common_undecided, common, bad);
  return bad != 0 || common_undecided * 100 > common;
}

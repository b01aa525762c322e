// Host check of the FP64 in-place transforms (csrc/dev_fft64.cuh): every
// in-register DFT against a long double DFT (both directions, and with the
// upper half of the inputs zero), and whole transforms of many lengths run
// pass by pass on the CPU: forward to the plan's slots, back to n times the
// input, with guard values around the buffer.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "dev_fft64.cuh"

typedef long double ld;
static const ld PI2 = 6.283185307179586476925286766559005768L;
static int bad = 0;

template <int RAD, int SIGN, bool HALF>
static void one_dft() {
  dcx v[RAD], in[RAD];
  for (int r = 0; r < RAD; r++) {
    in[r] = make_double2(drand48() - 0.5, drand48() - 0.5);
    if (HALF && r >= RAD / 2) in[r] = make_double2(0, 0);
    v[r] = in[r];
  }
  if (HALF) dft64_half<RAD, SIGN>(v);
  else dft64<RAD, SIGN>(v);
  for (int q = 0; q < RAD; q++) {
    ld a = 0, b = 0;
    for (int r = 0; r < RAD; r++) {
      const ld t = SIGN * PI2 * ((r * q) % RAD) / RAD, c = cosl(t), s = sinl(t);
      a += in[r].x * c - in[r].y * s;
      b += in[r].x * s + in[r].y * c;
    }
    // RAD additions of values below 1, a few roundings each
    if (fabsl(a - v[q].x) > 4e-16L * RAD || fabsl(b - v[q].y) > 4e-16L * RAD) {
      printf("dft %d sign %d half %d: output %d off by %Lg\n", RAD, SIGN, (int)HALF, q, fabsl(a - v[q].x));
      bad = 1;
    }
  }
}
template <int RAD>
static void dfts() {
  one_dft<RAD, -1, false>();
  one_dft<RAD, 1, false>();
  if constexpr (RAD % 2 == 0) one_dft<RAD, -1, true>();
}

#define CASES(M) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13) M(15) M(16)
static void first(const IpPlan& p, dcx* buf, const dcx* x, bool half) {
  auto ldr = [&](int, int i) { return x[i]; };
  switch (p.r[0]) {
#define K(R)                                                                               \
  case R:                                                                                  \
    if constexpr (R % 2 == 0)                                                              \
      if (half) { ip_first<R, true>(buf, 0, 1, p.tw, p.n, p.S, 0, 1, ldr); break; }        \
    ip_first<R, false>(buf, 0, 1, p.tw, p.n, p.S, 0, 1, ldr);                              \
    break;
    CASES(K)
#undef K
  }
}
static void last(const IpPlan& p, const dcx* buf, dcx* x) {
  auto str = [&](int, int i, dcx v) { x[i] = v; };
  switch (p.r[0]) {
#define K(R) case R: ip_last<R, false>(buf, 0, 1, p.tw, p.n, p.S, 0, 1, str); break;
    CASES(K)
#undef K
  }
}
template <int SIGN>
static bool mid(const IpPlan& p, dcx* buf, int R, int L) {
  switch (R) {
#define K(R) case R: ip_mid<R, SIGN>(buf, 0, 1, p.tw, p.n, p.r[0], p.S, L, 0, 1); return true;
    CASES(K)
#undef K
  }
  return false;
}
// slot of frequency k (digits from the first radix on)
static int slot(const IpPlan& p, int k) {
  int L = p.n / p.r[0], s = (k % p.r[0]) * p.S;
  k /= p.r[0];
  for (int i = 1; i < p.np; i++) {
    L /= p.r[i];
    s += (k % p.r[i]) * L;
    k /= p.r[i];
  }
  return s;
}
static int transform(int n, bool rows, bool half) {
  IpPlan p;
  bool fixed;
  if (!ip_plan(n, rows, half, p, fixed)) return 0;
  int prod = 1;
  for (int i = 0; i < p.np; i++) prod *= p.r[i];
  if (prod != n || p.np < 2 || p.np > IP_MAXP || (half && p.r[0] % 2) || (p.r[p.np - 1] > 6 && !fixed)) {
    printf("n %d: bad plan\n", n);
    bad = 1;
    return 0;
  }
  for (int i = 1; i + 1 < p.np; i++)
    if (p.r[i] > 16) return 0;   // warp passes run on the GPU only
  std::vector<dcx> tw(n), x(n), y(n);
  for (int k = 0; k < n; k++) tw[k] = make_double2(cosl(PI2 * k / n), -sinl(PI2 * k / n));
  p.tw = tw.data();
  for (int k = 0; k < n; k++)
    x[k] = (half && k >= n / 2) ? make_double2(0, 0) : make_double2(drand48() - 0.5, drand48() - 0.5);
  const int G = 64, len = p.r[0] * p.S;
  std::vector<dcx> store(len + 2 * G, make_double2(NAN, NAN));
  dcx* buf = store.data() + G;
  first(p, buf, x.data(), half);
  int L = n / p.r[0];
  for (int i = 1; i < p.np; i++) {
    if (!mid<-1>(p, buf, p.r[i], L)) { printf("n %d: no pass of radix %d\n", n, p.r[i]); bad = 1; return 0; }
    L /= p.r[i];
  }
  const double tol = 3e-16 * n;   // n additions of values below 1, log2(n) roundings deep at most
  for (int k = 0; k < n; k += (n > 600 ? 37 : 1)) {
    ld a = 0, b = 0;
    for (int i = 0; i < n; i++) {
      const ld t = -PI2 * ((long long)i * k % n) / n;
      a += x[i].x * cosl(t) - x[i].y * sinl(t);
      b += x[i].x * sinl(t) + x[i].y * cosl(t);
    }
    const dcx v = buf[slot(p, k)];
    if (!(fabsl(a - v.x) <= tol) || !(fabsl(b - v.y) <= tol)) { printf("n %d: frequency %d off\n", n, k); bad = 1; return 0; }
  }
  for (int i = p.np - 1; i >= 1; i--) {
    L *= p.r[i];
    mid<+1>(p, buf, p.r[i], L);
  }
  last(p, buf, y.data());
  for (int i = 0; i < n; i++)
    if (!(fabs(y[i].x - n * x[i].x) <= tol * 4) || !(fabs(y[i].y - n * x[i].y) <= tol * 4)) {
      printf("n %d: input %d not recovered\n", n, i);
      bad = 1;
      return 0;
    }
  for (int g = 0; g < G; g++)
    if (!isnan(store[g].x) || !isnan(store[G + len + g].x)) { printf("n %d: guard overwritten\n", n); bad = 1; }
  return 1;
}

int main() {
  srand48(7);
#define K(R) dfts<R>();
  CASES(K)
#undef K
  int done = 0;
  for (int n = 1; n <= 400; n++)
    for (int half = 0; half < 2; half++) {
      if (half && n % 2) continue;
      done += transform(n, true, half) + transform(n, false, half);
    }
  for (int n : {450, 512, 750, 800, 1024, 1155, 1440, 1536, 2048, 2310, 3072, 4050, 4096})
    done += transform(n, true, n % 2 == 0) + transform(n, false, n % 2 == 0) + transform(n, false, false);
  printf("%d transforms %s\n", done, bad ? "BAD" : "ok");
  return bad || done < 500;
}

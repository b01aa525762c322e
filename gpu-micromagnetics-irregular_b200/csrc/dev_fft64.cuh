// dev_fft64.cuh — FP64 transform core of the demag chain: in-place mixed-radix
// FFTs in shared memory, decimation in frequency forward and decimation in
// time back, without a reordering pass.
//
// A transform of length n = r0 r1 ... r(p-1) runs one pass per radix.  The
// element with digits (d0, d1, ...) sits at d0 S + d1 n/(r0 r1) + ... (S =
// n/r0, plus one unused element when n/r0 is even), in time order on the way
// in and, after the forward passes, at the slot of frequency
//   k = d0 + r0 d1 + r0 r1 d2 + ...
// The chain multiplies by the tensor in frequency space and transforms back,
// so natural frequency order is never needed: every butterfly reads and
// writes its own slots, a pass needs one barrier, the first forward pass takes
// its inputs from HBM, the last inverse pass hands its outputs to HBM, and the
// last forward and first inverse pass share one trip through registers with
// whatever happens between them.  Against the autosort passes of dev_fft.cuh
// (all reads, barrier, scattered writes, barrier; separate load, multiply and
// store sweeps) the column stage makes 8 shared-memory sweeps instead of 16
// and 4 barriers instead of 16.  Lanes run over d0 first, so a warp's 16-byte
// accesses are S apart (odd): no bank conflicts in any pass.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "dev_fft.cuh"

namespace {

// one transform length: radices (the first is the pass that touches HBM, the
// last the one fused with the multiply or the packing), the twiddle table
// tw[k] = exp(-2 pi i k / n)
constexpr int IP_MAXP = 12;
struct IpPlan {
  int n, np;
  int r[IP_MAXP];
  int S;               // distance of consecutive d0
  const double2* tw;
};

// radices with an in-register DFT here (a prime from 17 to 61: ip_mid_group)
__host__ __device__ constexpr bool ip_radix(int r) {
  return r == 1 || r == 2 || r == 3 || r == 4 || r == 5 || r == 6 || r == 7 || r == 8 || r == 9 || r == 10 ||
         r == 11 || r == 12 || r == 13 || r == 15 || r == 16;
}

using dcx = double2;

// ── in-register DFTs beyond dft_fixed ──
// odd prime length from the real and imaginary parts of the pair sums:
// out[q], out[R-q] = v0 + sum_r cos(2 pi r q / R) (v[r] + v[R-r]) +- i ...
template <int RAD>
struct PrimeCs;
template <>
struct PrimeCs<7> {
  static __host__ __device__ constexpr double c(int m) {
    constexpr double t[4] = {1.0, 0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
    return t[m];
  }
  static __host__ __device__ constexpr double s(int m) {
    constexpr double t[4] = {0.0, 0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
    return t[m];
  }
};
template <>
struct PrimeCs<11> {
  static __host__ __device__ constexpr double c(int m) {
    constexpr double t[6] = {1.0, 0.84125353283118116886, 0.41541501300188642553, -0.14231483827328514044,
                             -0.65486073394528506406, -0.95949297361449738989};
    return t[m];
  }
  static __host__ __device__ constexpr double s(int m) {
    constexpr double t[6] = {0.0, 0.54064081745559758211, 0.90963199535451837141, 0.98982144188093273238,
                             0.75574957435425828377, 0.28173255684142969771};
    return t[m];
  }
};
template <>
struct PrimeCs<13> {
  static __host__ __device__ constexpr double c(int m) {
    constexpr double t[7] = {1.0, 0.88545602565320989590, 0.56806474673115580251, 0.12053668025532305335,
                             -0.35460488704253562597, -0.74851074817110109863, -0.97094181742605202716};
    return t[m];
  }
  static __host__ __device__ constexpr double s(int m) {
    constexpr double t[7] = {0.0, 0.46472317204376854566, 0.82298386589365639458, 0.99270887409805399280,
                             0.93501624268541482344, 0.66312265824079520238, 0.23931566428755776715};
    return t[m];
  }
};
template <int RAD, int SIGN>
FFT_HD void dft_prime(dcx* v) {
  constexpr int H = (RAD - 1) / 2;
  dcx p[H], m[H];
#pragma unroll
  for (int r = 1; r <= H; r++) {
    p[r - 1] = cadd<double>(v[r], v[RAD - r]);
    m[r - 1] = csub<double>(v[r], v[RAD - r]);
  }
  const dcx v0 = v[0];
  dcx s0 = v0;
#pragma unroll
  for (int r = 0; r < H; r++) s0 = cadd<double>(s0, p[r]);
  v[0] = s0;
#pragma unroll
  for (int q = 1; q <= H; q++) {
    dcx a = v0, b = mk<double>(0.0, 0.0);
#pragma unroll
    for (int r = 1; r <= H; r++) {
      const int e = (r * q) % RAD;
      const double c = PrimeCs<RAD>::c(e <= H ? e : RAD - e);
      const double s = (e <= H ? 1.0 : -1.0) * PrimeCs<RAD>::s(e <= H ? e : RAD - e) * (double)SIGN;
      a.x += c * p[r - 1].x;
      a.y += c * p[r - 1].y;
      b.x += s * m[r - 1].x;
      b.y += s * m[r - 1].y;
    }
    v[q] = mk<double>(a.x - b.y, a.y + b.x);
    v[RAD - q] = mk<double>(a.x + b.y, a.y - b.x);
  }
}
// composite odd radices as two stages (index r = B n1 + n2, frequency q = k1 + A k2)
template <int SIGN>
FFT_HD void dft9(dcx* v) {
  const double c1 = 0.76604444311897803520, s1 = 0.64278760968653932632;    // 2 pi / 9
  const double c2 = 0.17364817766693034885, s2 = 0.98480775301220805937;    // 4 pi / 9
  const double c4 = -0.93969262078590838405, s4 = 0.34202014332566873304;   // 8 pi / 9
  dcx a[3][3];
#pragma unroll
  for (int n2 = 0; n2 < 3; n2++) {
#pragma unroll
    for (int n1 = 0; n1 < 3; n1++) a[n2][n1] = v[3 * n1 + n2];
    dft3<double, SIGN>(a[n2]);
  }
  a[1][1] = crot<double, SIGN>(a[1][1], c1, s1);
  a[1][2] = crot<double, SIGN>(a[1][2], c2, s2);
  a[2][1] = crot<double, SIGN>(a[2][1], c2, s2);
  a[2][2] = crot<double, SIGN>(a[2][2], c4, s4);
#pragma unroll
  for (int k1 = 0; k1 < 3; k1++) {
    dcx b[3] = {a[0][k1], a[1][k1], a[2][k1]};
    dft3<double, SIGN>(b);
#pragma unroll
    for (int k2 = 0; k2 < 3; k2++) v[k1 + 3 * k2] = b[k2];
  }
}
// A = 2 or 3 times 5 with coprime factors: the index maps of Good and Thomas
// (r = 5 n1 + A n2, q = 5 k1' + A k2' with the CRT frequencies) need no twiddles
template <int A, int SIGN>
FFT_HD void dft_5x(dcx* v) {
  constexpr int R = 5 * A;
  dcx a[5][A];
#pragma unroll
  for (int n2 = 0; n2 < 5; n2++) {
#pragma unroll
    for (int n1 = 0; n1 < A; n1++) a[n2][n1] = v[(5 * n1 + A * n2) % R];
    dft_fixed<double, A, SIGN>(a[n2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; k1++) {
    dcx b[5];
#pragma unroll
    for (int n2 = 0; n2 < 5; n2++) b[n2] = a[n2][k1];
    dft5<double, SIGN>(b);
    // frequency q with q = k1 mod A and q = k2 mod 5
#pragma unroll
    for (int k2 = 0; k2 < 5; k2++) {
      constexpr int e1 = (A == 2) ? 5 : 10;   // 1 mod A, 0 mod 5; (6 is 0 mod A, 1 mod 5)
      v[(e1 * k1 + 6 * k2) % R] = b[k2];
    }
  }
}

// DFT of RAD values; HALF: the inputs r >= RAD/2 are known to be zero (an
// open boundary's padding) and their additions are left out
template <int SIGN>
FFT_HD void dft4_half(dcx* v) {   // v[2] = v[3] = 0
  const dcx a = v[0], b = v[1], c = rot90<double, SIGN>(v[1]);
  v[0] = cadd<double>(a, b);
  v[2] = csub<double>(a, b);
  v[1] = cadd<double>(a, c);
  v[3] = csub<double>(a, c);
}
template <int RAD, int SIGN>
FFT_HD void dft64(dcx* v) {
  if constexpr (RAD == 1) {
  } else if constexpr (RAD == 7 || RAD == 11 || RAD == 13) {
    dft_prime<RAD, SIGN>(v);
  } else if constexpr (RAD == 9) {
    dft9<SIGN>(v);
  } else if constexpr (RAD == 10) {
    dft_5x<2, SIGN>(v);
  } else if constexpr (RAD == 15) {
    dft_5x<3, SIGN>(v);
  } else {
    dft_fixed<double, RAD, SIGN>(v);
  }
}
template <int RAD, int SIGN>
FFT_HD void dft64_half(dcx* v) {
  if constexpr (RAD == 16) {   // dft16 with its inner 4-point transforms halved
    const double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, h = 0.70710678118654752440;
    dcx a[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
      a[n2][0] = v[n2];
      a[n2][1] = v[4 + n2];
      dft4_half<SIGN>(a[n2]);
    }
    a[1][1] = crot<double, SIGN>(a[1][1], c1, s1);
    a[1][2] = crot<double, SIGN>(a[1][2], h, h);
    a[1][3] = crot<double, SIGN>(a[1][3], s1, c1);
    a[2][1] = crot<double, SIGN>(a[2][1], h, h);
    a[2][2] = rot90<double, SIGN>(a[2][2]);
    a[2][3] = crot<double, SIGN>(a[2][3], -h, h);
    a[3][1] = crot<double, SIGN>(a[3][1], s1, c1);
    a[3][2] = crot<double, SIGN>(a[3][2], -h, h);
    a[3][3] = crot<double, SIGN>(a[3][3], -c1, -s1);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
      dcx b[4] = {a[0][k1], a[1][k1], a[2][k1], a[3][k1]};
      dft4<double, SIGN>(b);
#pragma unroll
      for (int k2 = 0; k2 < 4; k2++) v[k1 + 4 * k2] = b[k2];
    }
  } else if constexpr (RAD == 8) {
    const double h = 0.70710678118654752440;
    dcx e[4] = {v[0], v[2], v[0], v[0]}, o[4] = {v[1], v[3], v[1], v[1]};
    dft4_half<SIGN>(e);
    dft4_half<SIGN>(o);
    const dcx o1 = mk<double>(h * (o[1].x - SIGN * o[1].y), h * (o[1].y + SIGN * o[1].x));
    const dcx o2 = rot90<double, SIGN>(o[2]);
    const dcx o3 = mk<double>(-h * (o[3].x + SIGN * o[3].y), h * (SIGN * o[3].x - o[3].y));
    v[0] = cadd<double>(e[0], o[0]);
    v[4] = csub<double>(e[0], o[0]);
    v[1] = cadd<double>(e[1], o1);
    v[5] = csub<double>(e[1], o1);
    v[2] = cadd<double>(e[2], o2);
    v[6] = csub<double>(e[2], o2);
    v[3] = cadd<double>(e[3], o3);
    v[7] = csub<double>(e[3], o3);
  } else {
#pragma unroll
    for (int r = RAD / 2; r < RAD; r++) v[r] = mk<double>(0.0, 0.0);
    dft64<RAD, SIGN>(v);
  }
}

// v[r] *= w^(r x), w = exp(SIGN 2 pi i / n), r x < n: the powers 1, 2, 4, 8
// from the table, every other one a product of at most three of them
FFT_HD dcx ip_tw(const dcx* tw, int k) {
#ifdef __CUDA_ARCH__
  return __ldg(&tw[k]);
#else
  return tw[k];
#endif
}
template <int RAD, int SIGN>
FFT_HD void ip_twiddle(dcx* v, const dcx* __restrict__ tw, int x) {
  if constexpr (RAD > 1) {
    auto ld = [&](int k) {
      dcx w = ip_tw(tw, k);
      if (SIGN > 0) w.y = -w.y;
      return w;
    };
    dcx w1 = ld(x), w2{}, w4{}, w8{};
    if constexpr (RAD > 2) w2 = ld(2 * x);
    if constexpr (RAD > 4) w4 = ld(4 * x);
    if constexpr (RAD > 8) w8 = ld(8 * x);
    dcx lo[4];   // w^0..w^3 (index 0 unused)
    lo[1] = w1;
    if constexpr (RAD > 2) lo[2] = w2;
    if constexpr (RAD > 3) lo[3] = cmul<double>(w1, w2);
#pragma unroll
    for (int g = 0; g < RAD; g += 4) {
      dcx hi{};
      if (g == 4) hi = w4;
      if (g == 8) hi = w8;
      if (g == 12) hi = cmul<double>(w8, w4);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int r = g + k;
        if (r == 0 || r >= RAD) continue;
        const dcx w = (g == 0) ? lo[k] : (k == 0 ? hi : cmul<double>(hi, lo[k]));
        v[r] = cmul<double>(v[r], w);
      }
    }
  }
}

// ── passes over nb transforms, buf + b * bs each; threads tid, tid + T, ... ──
// first forward pass: inputs ld(b, i) (i the time index), outputs to shared
// memory.  HALF: inputs i >= n/2 are zero.
template <int RAD, bool HALF, typename LD>
FFT_HD void ip_first(dcx* buf, int bs, int nb, const dcx* tw, int n, int S, int tid, int T,
                                         LD&& ld) {
  const int M = n / RAD;
#pragma unroll 1
  for (int q = tid; q < M * nb; q += T) {
    const int b = q / M, j = q - b * M;
    dcx v[RAD];
    constexpr int RL = HALF ? RAD / 2 : RAD;
#pragma unroll
    for (int r = 0; r < RL; r++) v[r] = ld(b, j + r * M);
    if constexpr (HALF) dft64_half<RAD, -1>(v);
    else dft64<RAD, -1>(v);
    ip_twiddle<RAD, -1>(v, tw, j);
    dcx* p = buf + b * bs + j;
#pragma unroll
    for (int r = 0; r < RAD; r++) p[r * S] = v[r];
  }
}
// last inverse pass: outputs st(b, i, value); HALF: only i < n/2 are wanted
template <int RAD, bool HALF, typename ST>
FFT_HD void ip_last(const dcx* buf, int bs, int nb, const dcx* tw, int n, int S, int tid, int T,
                                        ST&& st) {
  const int M = n / RAD;
#pragma unroll 1
  for (int q = tid; q < M * nb; q += T) {
    const int b = q / M, j = q - b * M;
    const dcx* p = buf + b * bs + j;
    dcx v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; r++) v[r] = p[r * S];
    ip_twiddle<RAD, +1>(v, tw, j);
    dft64<RAD, +1>(v);
    constexpr int RL = HALF ? RAD / 2 : RAD;
#pragma unroll
    for (int r = 0; r < RL; r++) st(b, j + r * M, v[r]);
  }
}
// a middle pass, blocks of L (L = n / (radices before it)): forward DFT then
// twiddles, or back twiddles then DFT; in place
template <int RAD, int SIGN>
FFT_HD void ip_mid(dcx* buf, int bs, int nb, const dcx* tw, int n, int r0, int S, int L, int tid,
                                       int T) {
  const int Lr = L / RAD, per = n / RAD, ts = n / L;
#pragma unroll 1
  for (int q = tid; q < per * nb; q += T) {
    const int b = q / per, x = q - b * per;
    const int y = x / r0, d0 = x - y * r0;
    const int blk = y / Lr, j = y - blk * Lr;
    dcx* p = buf + b * bs + d0 * S + blk * L + j;
    dcx v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; r++) v[r] = p[r * Lr];
    if constexpr (SIGN < 0) {
      dft64<RAD, SIGN>(v);
      ip_twiddle<RAD, SIGN>(v, tw, j * ts);
    } else {
      ip_twiddle<RAD, SIGN>(v, tw, j * ts);
      dft64<RAD, SIGN>(v);
    }
#pragma unroll
    for (int r = 0; r < RAD; r++) p[r * Lr] = v[r];
  }
}
// A middle pass of prime radix R, 17..61: a butterfly per group of GL lanes (16
// up to 31, else 32), which fold the values into sums and differences of v[r] and
// v[R-r] in place; lane l then forms the outputs l and R-l from the (R-1)/2 pairs
// (broadcast reads), a quarter of the products of the plain sums.  Only the
// group's own values are touched, so __syncwarp separates reads from writes.
// Against a warp per butterfly and plain sums, which on filled grids ran behind the
// autosort pass of a thread per butterfly: field of 348x512 open (a factor 29) 138
// us autosort, 193 plain, 70 now; 256x361 (19, 19) 135, 172, 64; 1450x1024 915, 1045, 472.
template <int SIGN, int GL>
__device__ __noinline__ void ip_mid_group(dcx* buf, int bs, int nb, const dcx* __restrict__ tw, int n, int r0, int S,
                                          int L, int RAD, int tid, int T) {
  constexpr int G = 32 / GL;   // groups of a warp
  const int Lr = L / RAD, per = n / RAD, ts = n / L, rs = n / RAD, H = (RAD - 1) / 2;
  const int l = tid % GL, total = per * nb;
  for (int q0 = (tid >> 5) * G; q0 < total; q0 += (T >> 5) * G) {   // (the same for all lanes of a warp)
    const int q = q0 + (tid & 31) / GL;
    const bool in = q < total && l <= H;
    const int b = q / per, x = q - b * per;
    const int y = x / r0, d0 = x - y * r0;
    const int blk = y / Lr, j = y - blk * Lr;
    dcx* p = buf + b * bs + d0 * S + blk * L + j;
    auto twiddled = [&](dcx v, int r) {
      dcx w = __ldg(&tw[r * j * ts]);
      if (SIGN > 0) w.y = -w.y;
      return cmul<double>(v, w);
    };
    dcx s = mk<double>(0.0, 0.0), t = s;
    if (in) s = p[0];
    if (in && l > 0) {
      dcx u = p[l * Lr], v = p[(RAD - l) * Lr];
      if constexpr (SIGN > 0) {   // twiddles first
        u = twiddled(u, l);
        v = twiddled(v, RAD - l);
      }
      p[l * Lr] = cadd<double>(u, v);
      p[(RAD - l) * Lr] = csub<double>(u, v);
    }
    __syncwarp();
    if (in) {
      int e = 0;
#pragma unroll 4
      for (int r = 1; r <= H; r++) {
        e += l;
        if (e >= RAD) e -= RAD;   // (r l) mod R
        const dcx u = p[r * Lr], d = p[(RAD - r) * Lr], w = __ldg(&tw[e * rs]);   // cos, -sin
        s.x += w.x * u.x;
        s.y += w.x * u.y;
        t.x += w.y * d.x;
        t.y += w.y * d.y;
      }
    }
    __syncwarp();
    if (in) {
      dcx o = mk<double>(s.x + SIGN * t.y, s.y - SIGN * t.x), m = mk<double>(s.x - SIGN * t.y, s.y + SIGN * t.x);
      if constexpr (SIGN < 0) {
        o = twiddled(o, l);
        m = twiddled(m, RAD - l);
      }
      p[l * Lr] = o;
      if (l > 0) p[(RAD - l) * Lr] = m;
    }
    __syncwarp();
  }
}

// ── plans (host) ──
// Lengths whose kernels are instantiated with constant radices: the 2^k from 32
// to 4096 and the 3 2^k from 48 to 3072, the powers of two that grids are made of
// and one and a half times them.  Every other length reads its radices from the
// plan: the same passes, with integer divisions for the slots and a branch per
// pass, at about half the speed (field, plan read / constant: 32x32 periodic 16.5 /
// 8.3 us, 512x512 31 / 16.5, 2048x2048 330 / 172, 1536x512 open 148 / 76).
//   rows: the radix fused with the packing is the large one (its two groups
//   stay in registers, which saves a sweep); columns: the fused one is 6 at
//   most, since three components' butterflies share the registers there.
#define LLG_ROWS64(M)                                                                            \
  M(32, 8, 1, 1, 4) M(64, 16, 1, 1, 4) M(128, 8, 4, 1, 4) M(256, 8, 8, 1, 4) M(512, 16, 8, 1, 4) \
  M(1024, 16, 16, 1, 4) M(2048, 16, 16, 1, 8) M(4096, 16, 16, 4, 4)                              \
  M(48, 8, 1, 1, 6) M(96, 16, 1, 1, 6) M(192, 16, 1, 1, 12) M(384, 16, 4, 1, 6)                  \
  M(768, 16, 8, 1, 6) M(1536, 16, 16, 1, 6) M(3072, 16, 16, 1, 12)
#define LLG_COLS64(M)                                                                             \
  M(32, 8, 1, 1, 4) M(64, 16, 1, 1, 4) M(128, 8, 4, 1, 4) M(256, 16, 4, 1, 4) M(512, 16, 8, 1, 4) \
  M(1024, 16, 16, 1, 4) M(2048, 16, 8, 4, 4) M(4096, 16, 16, 4, 4)                                \
  M(48, 16, 1, 1, 3) M(96, 16, 1, 1, 6) M(192, 16, 4, 1, 3) M(384, 16, 6, 1, 4)                   \
  M(768, 16, 12, 1, 4) M(1536, 16, 16, 1, 6) M(3072, 16, 16, 3, 4)

// instruction weight per element of one pass of radix r, twiddles included:
// counted from the code above and only used to rank factorisations of the same
// length (a prime's weight never decides, its pass is given)
double pass_cost(int r) {
  switch (r) {
    case 1: return 0;
    case 2: return 5;
    case 3: return 8;
    case 4: return 9;
    case 5: return 12;
    case 6: return 12;
    case 7: return 16;
    case 8: return 13;
    case 9: return 15;
    case 10: return 16;
    case 11: return 26;
    case 12: return 15.5;
    case 13: return 30;
    case 15: return 18;
    case 16: return 16.5;
    default: return 6.0 * r;   // ip_mid_group
  }
}
constexpr double kSweep = 10;   // a pass's shared-memory sweep and barrier, in the same unit (an estimate)

// cheapest middle passes for what is left of the length
void search_mids(int left, int from, std::vector<int>& cur, double cost, double& best, std::vector<int>& out) {
  if (left == 1) {
    if (cost < best) {
      best = cost;
      out = cur;
    }
    return;
  }
  if ((int)cur.size() >= IP_MAXP - 2) return;
  for (int r = from; r >= 2; r--) {
    if (left % r || !(ip_radix(r) || (r > 13 && r < 64 && r % 2 && r % 3 && r % 5 && r % 7))) continue;
    cur.push_back(r);
    search_mids(left / r, r, cur, cost + pass_cost(r) + kSweep, best, out);
    cur.pop_back();
  }
}

bool fixed_list(int n, bool rows, int (&r)[4]) {
#define K(N, A, B, C, D)                     \
  if (n == N) {                              \
    r[0] = A, r[1] = B, r[2] = C, r[3] = D;  \
    return true;                             \
  }
  if (rows) {
    LLG_ROWS64(K)
  } else {
    LLG_COLS64(K)
  }
#undef K
  return false;
}

// radices of length n (half: the first one must be even); false: a prime
// factor above 61
bool ip_plan(int n, bool rows, bool half, IpPlan& p, bool& fixed) {
  int f[4];
  p = IpPlan{};
  p.n = n;
  fixed = fixed_list(n, rows, f);
  if (fixed) {
    for (int k = 0; k < 4; k++)
      if (f[k] > 1) p.r[p.np++] = f[k];
  } else {
    double best = 1e30;
    for (int r0 = 1; r0 <= 16; r0++) {
      if (!ip_radix(r0) || n % r0 || (half && r0 % 2)) continue;
      for (int c = 1; c <= 6; c++) {
        if ((n / r0) % c) continue;
        std::vector<int> cur, mids;
        double b = 1e30;
        search_mids(n / r0 / c, 61, cur, 0.0, b, mids);
        // (8 and more blocks keep a warp's lanes on different banks)
        b += pass_cost(r0) + pass_cost(c) + kSweep * (c > 1 ? 1 : 0.5) + (r0 < 8 ? 6 : 0);
        if (b < best) {
          best = b;
          p.np = 0;
          p.r[p.np++] = r0;
          for (int m : mids) p.r[p.np++] = m;
          p.r[p.np++] = c;
        }
      }
    }
    if (best >= 1e30) return false;
  }
  p.S = n / p.r[0];
  if (p.S % 2 == 0) p.S++;
  return true;
}

}  // namespace

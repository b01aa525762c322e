// k_demag64.cu — the three kernels of the FP64 demag chain on the in-place
// transforms of dev_fft64.cuh (mixed chain: k_demag.cu, k_demag_tc.cu).
//
//   rows_fwd : rows (2p, 2p + 1) of one component packed into one complex
//              transform along x; the last pass's butterflies of the groups g
//              and G - g meet in one thread's registers, are separated into
//              the two rows' half spectra there, and leave as one 32-byte
//              store per frequency (column-major S).
//   cols     : one x-frequency column of the three components: forward along
//              y, 3x3 tensor multiply in the registers of the last pass,
//              inverse along y, kept rows back to S.
//   rows_inv : the mirror image of rows_fwd.
//
// What bounds them: FP64 issue (about 45 FP64 instructions per element and
// transform) and shared-memory sweeps, then the latency of each CTA's load;
// HBM traffic is far below its roof.  The padded half of an open row or column
// is neither loaded nor added, and its half of the last inverse pass is not
// formed.  1536x512 open (3072x1024 transforms), in the stream with the operands
// in L2: rows_fwd 18.9 us, cols 36.6, rows_inv 18.5 (cold caches 27.7, 42.9, 38.4;
// the autosort kernels before them 46.6, 96.3, 35.7 cold).  f of that film through
// the callbacks 205 -> 107 us; 375x225 open (750x450), the field alone, 43 -> 28.6.
// Radix 8 passes at twice the threads ran the same times for rows and 53 us for
// columns; three and four resident CTAs instead of two changed nothing, so the
// radix-16 forms stand.
//
// Tensor spectra: N_xx, N_yy, N_zz are even in the y frequency and, on the open
// grid, N_xy is real and odd in it, so only ky = 0..n/2 is kept, interleaved
// {xx, yy, zz, xy} for one 32-byte load per frequency: 16 B per frequency
// instead of 40.  On the periodic grid (whose d = -P/2 line is its own mirror
// image) N_xy stays a full complex array.
#include <math.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include "dev_fft64.cuh"
#include "launch.h"
#include "llg_internal.h"

namespace {

struct alignas(32) d4 {
  double x, y, z, w;
};
__device__ __forceinline__ d4 ldg4(const d4* p) {   // 32 bytes, read-only data
  d4 v;
  asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
// (past L1: the column kernel before it rewrote S in place, see launch.h)
__device__ __forceinline__ void ld2(const dcx* p, bool vec, bool both, dcx& a, dcx& b) {
  if (vec && both) {
    asm volatile("ld.global.cg.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y)
                 : "l"(p)
                 : "memory");
  } else {
    a = __ldcg(p);
    b = both ? __ldcg(p + 1) : mk<double>(0.0, 0.0);
  }
}
__device__ __forceinline__ void st2(dcx* p, bool vec, bool both, dcx a, dcx b) {
  if (vec && both) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y)
                 : "memory");
  } else {
    p[0] = a;
    if (both) p[1] = b;
  }
}

// ── plans: a length whose radices are constants of its kernels ... ──
template <int N, int R0, int M1, int M2, int C>
struct FixPlan {
  static_assert(N == R0 * M1 * M2 * C, "radices");
  const dcx* tw;
  __device__ __forceinline__ FixPlan(const IpPlan& p) : tw(p.tw) {}
  static constexpr int n() { return N; }
  static constexpr int S() { return N / R0 + ((N / R0) % 2 == 0 ? 1 : 0); }
  static constexpr int bs() { return R0 * S(); }
  static constexpr int last() { return C; }
  template <bool HALF, typename LD>
  __device__ __forceinline__ void first(dcx* buf, int nb, int tid, int T, LD&& ld) const {
    ip_first<R0, HALF>(buf, bs(), nb, tw, N, S(), tid, T, ld);
  }
  template <bool HALF, typename ST>
  __device__ __forceinline__ void final(const dcx* buf, int nb, int tid, int T, ST&& st) const {
    ip_last<R0, HALF>(buf, bs(), nb, tw, N, S(), tid, T, st);
  }
  __device__ __forceinline__ void mids_fwd(dcx* buf, int nb, int tid, int T) const {
    if constexpr (M1 > 1) {
      ip_mid<M1, -1>(buf, bs(), nb, tw, N, R0, S(), N / R0, tid, T);
      __syncthreads();
    }
    if constexpr (M2 > 1) {
      ip_mid<M2, -1>(buf, bs(), nb, tw, N, R0, S(), N / (R0 * M1), tid, T);
      __syncthreads();
    }
  }
  __device__ __forceinline__ void mids_inv(dcx* buf, int nb, int tid, int T) const {
    if constexpr (M2 > 1) {
      ip_mid<M2, +1>(buf, bs(), nb, tw, N, R0, S(), N / (R0 * M1), tid, T);
      __syncthreads();
    }
    if constexpr (M1 > 1) {
      ip_mid<M1, +1>(buf, bs(), nb, tw, N, R0, S(), N / R0, tid, T);
      __syncthreads();
    }
  }
  // slot of last-pass group g (frequencies g + r n/C)
  __device__ __forceinline__ int slot(int g) const {
    const int h = g / R0, d0 = g - h * R0;
    if constexpr (M2 > 1) {
      const int d2 = h / M1, d1 = h - d2 * M1;
      return d0 * S() + (d1 * M2 + d2) * C;
    } else {
      return d0 * S() + h * C;
    }
  }
  template <typename F>
  __device__ __forceinline__ void with_last(F&& f) const {
    f(std::integral_constant<int, C>{});
  }
};

// ... and any other length, its radices read from the plan
struct DynPlan {
  const IpPlan& p;   // (the kernel's parameter)
  __device__ __forceinline__ DynPlan(const IpPlan& q) : p(q) {}
  __device__ __forceinline__ int n() const { return p.n; }
  __device__ __forceinline__ int S() const { return p.S; }
  __device__ __forceinline__ int bs() const { return p.r[0] * p.S; }
#define LLG_IP_CASES(M) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13) M(15) M(16)
  template <bool HALF, typename LD>
  __device__ __forceinline__ void first(dcx* buf, int nb, int tid, int T, LD&& ld) const {
    const int s = bs();
    switch (p.r[0]) {   // (HALF only with an even first radix)
#define K(R)                                                                                      \
  case R:                                                                                         \
    if constexpr (!HALF || R % 2 == 0) ip_first<R, HALF>(buf, s, nb, p.tw, p.n, p.S, tid, T, ld); \
    break;
      LLG_IP_CASES(K)
#undef K
      default:
        if constexpr (!HALF) ip_first<1, false>(buf, s, nb, p.tw, p.n, p.S, tid, T, ld);
    }
  }
  template <bool HALF, typename ST>
  __device__ __forceinline__ void final(const dcx* buf, int nb, int tid, int T, ST&& st) const {
    const int s = bs();
    switch (p.r[0]) {
#define K(R)                                                                                     \
  case R:                                                                                        \
    if constexpr (!HALF || R % 2 == 0) ip_last<R, HALF>(buf, s, nb, p.tw, p.n, p.S, tid, T, st); \
    break;
      LLG_IP_CASES(K)
#undef K
      default:
        if constexpr (!HALF) ip_last<1, false>(buf, s, nb, p.tw, p.n, p.S, tid, T, st);
    }
  }
  template <int SIGN>
  __device__ __forceinline__ void mid(dcx* buf, int nb, int R, int L, int tid, int T) const {
    const int s = bs();
    switch (R) {
#define K(R)                                                                        \
  case R:                                                                           \
    ip_mid<R, SIGN>(buf, s, nb, p.tw, p.n, p.r[0], p.S, L, tid, T);                 \
    break;
      LLG_IP_CASES(K)
#undef K
      default:
        if (R < 32) ip_mid_group<SIGN, 16>(buf, s, nb, p.tw, p.n, p.r[0], p.S, L, R, tid, T);
        else ip_mid_group<SIGN, 32>(buf, s, nb, p.tw, p.n, p.r[0], p.S, L, R, tid, T);
    }
  }
  __device__ __forceinline__ void mids_fwd(dcx* buf, int nb, int tid, int T) const {
    int L = p.n / p.r[0];
#pragma unroll 1
    for (int i = 1; i + 1 < p.np; i++) {
      mid<-1>(buf, nb, p.r[i], L, tid, T);
      __syncthreads();
      L /= p.r[i];
    }
  }
  __device__ __forceinline__ void mids_inv(dcx* buf, int nb, int tid, int T) const {
    int L = p.r[p.np - 1];
#pragma unroll 1
    for (int i = p.np - 2; i >= 1; i--) {
      L *= p.r[i];
      mid<+1>(buf, nb, p.r[i], L, tid, T);
      __syncthreads();
    }
  }
  __device__ __forceinline__ int slot(int g) const {
    int h = g / p.r[0];
    const int d0 = g - h * p.r[0];
    int y = 0;
#pragma unroll 1
    for (int i = 1; i + 1 < p.np; i++) {
      const int q = h / p.r[i];
      y = y * p.r[i] + (h - q * p.r[i]);
      h = q;
    }
    return d0 * p.S + y * p.r[p.np - 1];
  }
  template <typename F>
  __device__ __forceinline__ void with_last(F&& f) const {
    switch (p.r[p.np - 1]) {
      case 2: f(std::integral_constant<int, 2>{}); break;
      case 3: f(std::integral_constant<int, 3>{}); break;
      case 4: f(std::integral_constant<int, 4>{}); break;
      case 5: f(std::integral_constant<int, 5>{}); break;
      case 6: f(std::integral_constant<int, 6>{}); break;
      default: f(std::integral_constant<int, 1>{});
    }
  }
};

// ── columns ──
template <class PL, bool OPEN, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_cols64(const __grid_constant__ IpPlan plan, dcx* __restrict__ S, int ld, int Hx,
                                                       const d4* __restrict__ th, const dcx* __restrict__ txy) {
  extern __shared__ __align__(16) unsigned char smraw[];
  dcx* buf = reinterpret_cast<dcx*>(smraw);
  const PL pl(plan);
  const int n = pl.n(), bs = pl.bs(), kx = blockIdx.x, tid = threadIdx.x, T = blockDim.x;
  const d4* tc = th + (long long)kx * (n / 2 + 1);
  // the column's tensor on its way into L2 while the first passes run (the
  // plan's data: nothing in the stream writes it)
  if (tid == 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(tc), "r"((n / 2 + 1) * (int)sizeof(d4)) : "memory");
  pdl_entry();
  dcx* col = S + (long long)kx * ld;
  const long long cs = (long long)Hx * ld;
  pl.template first<OPEN>(buf, 3, tid, T, [&](int c, int i) { return col[c * cs + i]; });
  __syncthreads();
  pl.mids_fwd(buf, 3, tid, T);
  pl.with_last([&](auto cc) {
    constexpr int C = decltype(cc)::value;
    const int G = n / C;
#pragma unroll 1
    for (int g = tid; g < G; g += T) {
      dcx* p = buf + pl.slot(g);
      dcx X[C], Y[C], Z[C];
      d4 t[C];
#pragma unroll
      for (int r = 0; r < C; r++) {
        const int k = g + r * G, m = n - k;
        t[r] = ldg4(&tc[k <= m ? k : m]);
        if (OPEN && k > m) t[r].w = -t[r].w;
      }
#pragma unroll
      for (int r = 0; r < C; r++) Z[r] = p[2 * bs + r];
      dft64<C, -1>(Z);
#pragma unroll
      for (int r = 0; r < C; r++) Z[r] = mk<double>(t[r].z * Z[r].x, t[r].z * Z[r].y);
      dft64<C, +1>(Z);
#pragma unroll
      for (int r = 0; r < C; r++) p[2 * bs + r] = Z[r];
#pragma unroll
      for (int r = 0; r < C; r++) {
        X[r] = p[r];
        Y[r] = p[bs + r];
      }
      dft64<C, -1>(X);
      dft64<C, -1>(Y);
#pragma unroll
      for (int r = 0; r < C; r++) {
        const dcx x = X[r], y = Y[r];
        if constexpr (OPEN) {
          X[r] = mk<double>(t[r].x * x.x + t[r].w * y.x, t[r].x * x.y + t[r].w * y.y);
          Y[r] = mk<double>(t[r].w * x.x + t[r].y * y.x, t[r].w * x.y + t[r].y * y.y);
        } else {
          const dcx xy = __ldg(&txy[(long long)kx * n + g + r * G]);
          const dcx hx = cmul<double>(xy, y), hy = cmul<double>(xy, x);
          X[r] = mk<double>(t[r].x * x.x + hx.x, t[r].x * x.y + hx.y);
          Y[r] = mk<double>(hy.x + t[r].y * y.x, hy.y + t[r].y * y.y);
        }
      }
      dft64<C, +1>(X);
      dft64<C, +1>(Y);
#pragma unroll
      for (int r = 0; r < C; r++) {
        p[r] = X[r];
        p[bs + r] = Y[r];
      }
    }
  });
  __syncthreads();
  pl.mids_inv(buf, 3, tid, T);
  pl.template final<OPEN>(buf, 3, tid, T, [&](int c, int i, dcx v) { col[c * cs + i] = v; });
}

// ── rows ──
// nb packed transforms per CTA; blockIdx.y = component
template <class PL, bool OPEN, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_rows_fwd64(const __grid_constant__ IpPlan plan, const double* __restrict__ in, long long stride,
                                                           int row_len, int nrows, const double* __restrict__ w,
                                                           dcx* __restrict__ S, int ld, int Hx, int nb, int vec) {
  extern __shared__ __align__(16) unsigned char smraw[];
  dcx* buf = reinterpret_cast<dcx*>(smraw);
  pdl_entry();
  const PL pl(plan);
  const int n = pl.n(), bs = pl.bs(), c = blockIdx.y, tid = threadIdx.x, T = blockDim.x;
  const int y0 = 2 * nb * blockIdx.x;
  const double* src = in + c * stride;
  pl.template first<OPEN>(buf, nb, tid, T, [&](int b, int i) {
    const int ya = y0 + 2 * b;
    const long long qa = (long long)ya * row_len + i, qb = qa + row_len;
    double va = 0.0, vb = 0.0;
    if (ya < nrows) va = src[qa];
    if (ya + 1 < nrows) vb = src[qb];
    if (w) {
      if (ya < nrows) va *= w[qa];
      if (ya + 1 < nrows) vb *= w[qb];
    }
    return mk<double>(va, vb);
  });
  __syncthreads();
  pl.mids_fwd(buf, nb, tid, T);
  pl.with_last([&](auto cc) {
    constexpr int C = decltype(cc)::value;
    const int G = n / C, J = G / 2 + 1;
#pragma unroll 1
    for (int q = tid; q < J * nb; q += T) {
      const int g = q / nb, b = q - g * nb, ya = y0 + 2 * b;   // pairs of one frequency on adjacent lanes
      if (ya >= nrows) continue;
      const bool self = (g == 0 || 2 * g == G);   // the group is its own mirror image
      const dcx* p = buf + b * bs;
      dcx va[C], vb[C];
      const int pa = pl.slot(g), pb = self ? pa : pl.slot(G - g);
#pragma unroll
      for (int r = 0; r < C; r++) {
        va[r] = p[pa + r];
        vb[r] = p[pb + r];
      }
      dft64<C, -1>(va);
      dft64<C, -1>(vb);
#pragma unroll
      for (int r = 0; r < C; r++) {
        const int k = g + r * G;
        // Z[k] and Z[n - k]: entry C - 1 - r of the mirrored group (g = 0: C - r)
        dcx zk = va[r], zm = (g == 0) ? vb[(C - r) % C] : vb[C - 1 - r];
        int kx = k;
        if (2 * k > n) {
          kx = n - k;
          const dcx t = zk;
          zk = zm;
          zm = t;
        }
        st2(&S[((long long)c * Hx + kx) * ld + ya], vec, ya + 1 < nrows,
            mk<double>(0.5 * (zk.x + zm.x), 0.5 * (zk.y - zm.y)), mk<double>(0.5 * (zk.y + zm.y), -0.5 * (zk.x - zm.x)));
      }
    }
  });
}

template <class PL, bool OPEN, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_rows_inv64(const __grid_constant__ IpPlan plan, const dcx* __restrict__ S, int ld, int nrows,
                                                           int Hx, double* __restrict__ h, long long stride, int ng,
                                                           int nb, int vec) {
  extern __shared__ __align__(16) unsigned char smraw[];
  dcx* buf = reinterpret_cast<dcx*>(smraw);
  pdl_entry();
  const PL pl(plan);
  const int n = pl.n(), bs = pl.bs(), c = blockIdx.y, tid = threadIdx.x, T = blockDim.x;
  const int y0 = 2 * nb * blockIdx.x;
  pl.with_last([&](auto cc) {
    constexpr int C = decltype(cc)::value;
    const int G = n / C, J = G / 2 + 1;
#pragma unroll 1
    for (int q = tid; q < J * nb; q += T) {
      const int g = q / nb, b = q - g * nb, ya = y0 + 2 * b;   // pairs of one frequency on adjacent lanes
      if (ya >= nrows) continue;
      const bool self = (g == 0 || 2 * g == G);
      dcx va[C], vb[C];
      dcx A[C], B[C];
#pragma unroll
      for (int r = 0; r < C; r++) {
        const int k = g + r * G, kx = (2 * k > n) ? n - k : k;
        ld2(&S[((long long)c * Hx + kx) * ld + ya], vec, ya + 1 < nrows, A[r], B[r]);
      }
#pragma unroll
      for (int r = 0; r < C; r++) {
        const int k = g + r * G;
        if (k == 0 || 2 * k == n) {
          A[r].y = 0.0;
          B[r].y = 0.0;
        }
        const dcx zk = mk<double>(A[r].x - B[r].y, A[r].y + B[r].x);   // Z[kx]
        const dcx zm = mk<double>(A[r].x + B[r].y, B[r].x - A[r].y);   // Z[n - kx]
        va[r] = (2 * k > n) ? zm : zk;
        vb[C - 1 - r] = (2 * k > n) ? zk : zm;
      }
      dcx* p = buf + b * bs;
      dft64<C, +1>(va);
      const int pa = pl.slot(g);
#pragma unroll
      for (int r = 0; r < C; r++) p[pa + r] = va[r];
      if (!self) {
        dft64<C, +1>(vb);
        const int pb = pl.slot(G - g);
#pragma unroll
        for (int r = 0; r < C; r++) p[pb + r] = vb[r];
      }
    }
  });
  __syncthreads();
  pl.mids_inv(buf, nb, tid, T);
  double* dst = h + c * stride;
  pl.template final<OPEN>(buf, nb, tid, T, [&](int b, int i, dcx v) {
    const int ya = y0 + 2 * b;
    const long long q = (long long)ya * ng + i;
    if (ya < nrows) dst[q] = v.x;
    if (ya + 1 < nrows) dst[q + ng] = v.y;
  });
}

// FP64 tensor spectra (full columns) -> the interleaved lower half
__global__ void k_tensor_half(const double* __restrict__ xx, const double* __restrict__ yy,
                              const double* __restrict__ zz, const dcx* __restrict__ xy, int n, int hx,
                              d4* __restrict__ out) {
  const int nh = n / 2 + 1;
  const long long tot = (long long)hx * nh;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot; e += (long long)gridDim.x * blockDim.x) {
    const long long kx = e / nh, q = kx * n + (e - kx * nh);
    out[e] = d4{xx[q], yy[q], zz[q], xy[q].x};
  }
}

// ── host side ──
using RowsFwd64 = void (*)(IpPlan, const double*, long long, int, int, const double*, dcx*, int, int, int, int);
using RowsInv64 = void (*)(IpPlan, const dcx*, int, int, int, double*, long long, int, int, int);
using Cols64 = void (*)(IpPlan, dcx*, int, int, const d4*, const dcx*);

constexpr int MAXT64 = 256;   // threads of a CTA at most

template <bool OPEN>
RowsFwd64 rows_fwd_fn64(int n, bool fixed) {
#define K(N, A, B, C, D) \
  if (fixed && n == N) return k_rows_fwd64<FixPlan<N, A, B, C, D>, OPEN, MAXT64, 2>;
  LLG_ROWS64(K)
#undef K
  return k_rows_fwd64<DynPlan, OPEN, MAXT64, 2>;
}
template <bool OPEN>
RowsInv64 rows_inv_fn64(int n, bool fixed) {
#define K(N, A, B, C, D) \
  if (fixed && n == N) return k_rows_inv64<FixPlan<N, A, B, C, D>, OPEN, MAXT64, 2>;
  LLG_ROWS64(K)
#undef K
  return k_rows_inv64<DynPlan, OPEN, MAXT64, 2>;
}
template <bool OPEN>
Cols64 cols_fn64(int n, bool fixed) {
#define K(N, A, B, C, D) \
  if (fixed && n == N) return k_cols64<FixPlan<N, A, B, C, D>, OPEN, MAXT64, 2>;
  LLG_COLS64(K)
#undef K
  return k_cols64<DynPlan, OPEN, MAXT64, 2>;
}

struct Cfg64 {   // launch shape (chosen by timing; every shape gives the same bits)
  int nb = 1, tr = 128, tcl = 128;
};
std::mutex g64_mu;
std::map<std::tuple<int, int, int, int>, Cfg64> g64_tuned;   // (px, py, ny, open)

}  // namespace

struct Demag64 {
  int px = 0, py = 0, hx = 0, ng = 0, ny = 0, open = 0;
  bool fixr = false, fixc = false;
  IpPlan pr{}, pc{};
  Cfg64 cfg;
  dcx* S = nullptr;       // the plan's spectrum (not owned)
  d4* th = nullptr;
  dcx* txy = nullptr;     // periodic grid only
};

void demag64_destroy(Demag64* d) {
  if (!d) return;
  cudaFree(d->th);
  cudaFree(d->txy);
  delete d;
}

static size_t rows_smem64(const Demag64* d, int nb) { return sizeof(dcx) * (size_t)nb * d->pr.r[0] * d->pr.S; }
static size_t cols_smem64(const Demag64* d) { return sizeof(dcx) * 3 * (size_t)d->pc.r[0] * d->pc.S; }

int demag64_stage(llg_ctx* c, Demag64* d, int stage, const double* y, const double* w, double* h) {
  const Cfg64& k = d->cfg;
  const int vec = d->ny % 2 == 0;   // 32-byte aligned row pairs of every column
  if (stage == 1) {
    klaunch(d->open ? cols_fn64<true>(d->py, d->fixc) : cols_fn64<false>(d->py, d->fixc), d->hx, k.tcl, cols_smem64(d),
            c->stream, d->pc, d->S, d->ny, d->hx, (const d4*)d->th, (const dcx*)d->txy);
  } else {
    const dim3 g((d->ny + 2 * k.nb - 1) / (2 * k.nb), 3);
    const long long cs = (long long)c->ncell;
    if (stage == 0)
      klaunch(d->open ? rows_fwd_fn64<true>(d->px, d->fixr) : rows_fwd_fn64<false>(d->px, d->fixr), g, k.tr,
              rows_smem64(d, k.nb), c->stream, d->pr, y, cs, d->ng, d->ny, w, d->S, d->ny, d->hx, k.nb, vec);
    else
      klaunch(d->open ? rows_inv_fn64<true>(d->px, d->fixr) : rows_inv_fn64<false>(d->px, d->fixr), g, k.tr,
              rows_smem64(d, k.nb), c->stream, d->pr, (const dcx*)d->S, d->ny, d->ny, d->hx, h, cs, d->ng, k.nb, vec);
  }
  LLG_CUDA_TRY(cudaPeekAtLastError());
  return 0;
}

// Launch shapes: transforms per row CTA and threads per CTA, timed as the
// three-kernel chain under programmatic dependent launch, as the integrator
// issues it; kept per transform size, process-wide.  (in: any field, out:
// scratch)
static int demag64_tune(llg_ctx* c, Demag64* d, const double* in, double* out) {
  const auto key = std::make_tuple(d->px, d->py, d->ny, d->open);
  {
    std::lock_guard<std::mutex> g(g64_mu);
    auto it = g64_tuned.find(key);
    if (it != g64_tuned.end()) {
      d->cfg = it->second;
      return 0;
    }
  }
  cudaEvent_t e0, e1;
  LLG_CUDA_TRY(cudaEventCreate(&e0));
  LLG_CUDA_TRY(cudaEventCreate(&e1));
  Cfg64 best = d->cfg;
  const int maxsm = 227 * 1024;
  // one dimension at a time: column threads, then transforms per row CTA with its threads
  auto time_cfg = [&](const Cfg64& k) -> float {
    d->cfg = k;
    float tmin = 1e30f;
    for (int rep = 0; rep < 3; rep++) {
      cudaEventRecord(e0, c->stream);
      int bad = 0;
      {
        PdlScope pdl(true);
        for (int i = 0; i < 3 && !bad; i++)
          for (int st = 0; st < 3 && !bad; st++) bad = demag64_stage(c, d, st, in, nullptr, out);
      }
      cudaEventRecord(e1, c->stream);
      float ms = 0.f;
      if (bad || cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
        cudaGetLastError();
        return 1e30f;
      }
      if (rep > 0) tmin = std::min(tmin, ms);
    }
    return tmin;
  };
  float tb = time_cfg(best);
  const int ts[] = {32, 64, 96, 128, 160, 192, 256};
  auto useful = [&](int t, int n, int nb) { return t == 32 || t <= nb * n / 4; };
  for (int t : ts) {
    Cfg64 k = best;
    k.tcl = t;
    if (t == best.tcl || !useful(t, d->py, 3)) continue;
    const float ms = time_cfg(k);
    if (ms < tb) tb = ms, best = k;
  }
  for (int nb = 1; nb <= 4; nb *= 2) {
    if ((int)rows_smem64(d, nb) > maxsm || (nb > 1 && 2 * nb > d->ny)) continue;
    for (int t : ts) {
      Cfg64 k = best;
      k.nb = nb;
      k.tr = t;
      if (!useful(t, d->px, nb)) continue;
      const float ms = time_cfg(k);
      if (ms < tb) tb = ms, best = k;
    }
  }
  d->cfg = best;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  pdl_break();
  LLG_CUDA_TRY(cudaGetLastError());
  std::lock_guard<std::mutex> g(g64_mu);
  g64_tuned[key] = best;
  return 0;
}

int demag64_create(llg_ctx* c, int px, int py, int hx, int ng, int ny, int open, const double2* twx, const double2* twy,
                   double2* S, const double* txx, const double* tyy, const double* tzz, const double2* txy,
                   Demag64** out) {
  *out = nullptr;
  Demag64* d = new Demag64();
  d->px = px;
  d->py = py;
  d->hx = hx;
  d->ng = ng;
  d->ny = ny;
  d->open = open;
  d->S = S;
  auto fail = [&](int rc) {
    demag64_destroy(d);
    return rc;
  };
  if (!ip_plan(px, true, open != 0, d->pr, d->fixr) || !ip_plan(py, false, open != 0, d->pc, d->fixc)) {
    llg_set_error("demag: transform length has a prime factor above 61");
    return fail(LLG_ERR_NOTSUP);
  }
  d->pr.tw = twx;
  d->pc.tw = twy;
  const size_t maxsm = 227 * 1024;
  if (cols_smem64(d) > maxsm) d->pc.S = py / d->pc.r[0];   // the longest columns: without the bank padding
  if (cols_smem64(d) > maxsm || rows_smem64(d, 1) > maxsm) {
    llg_set_error("demag grid too large for the shared-memory transform");
    return fail(LLG_ERR_NOTSUP);
  }
  const void* fns[3] = {
      open ? (const void*)rows_fwd_fn64<true>(px, d->fixr) : (const void*)rows_fwd_fn64<false>(px, d->fixr),
      open ? (const void*)rows_inv_fn64<true>(px, d->fixr) : (const void*)rows_inv_fn64<false>(px, d->fixr),
      open ? (const void*)cols_fn64<true>(py, d->fixc) : (const void*)cols_fn64<false>(py, d->fixc)};
  for (const void* f : fns)   // (process-wide per kernel, so the largest a plan can ask for)
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)maxsm) != cudaSuccess) {
      llg_set_error("demag: shared-memory opt-in failed");
      return fail(LLG_ERR_CUDA);
    }
  const long long nh = (long long)hx * (py / 2 + 1), nf = (long long)hx * py;
  if (cudaMalloc(&d->th, sizeof(d4) * nh) != cudaSuccess ||
      (!open && cudaMalloc(&d->txy, sizeof(dcx) * nf) != cudaSuccess)) {
    llg_set_error("demag: tensor spectra allocation failed");
    return fail(LLG_ERR_NOMEM);
  }
  klaunch(k_tensor_half, c->num_sms * 8, 256, 0, c->stream, txx, tyy, tzz, txy, py, hx, d->th);
  if (!open) cudaMemcpyAsync(d->txy, txy, sizeof(dcx) * nf, cudaMemcpyDeviceToDevice, c->stream);
  pdl_break();
  if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) {
    llg_set_error(std::string("demag: tensor spectra: ") + cudaGetErrorString(e));
    return fail(LLG_ERR_CUDA);
  }
  const int rc = demag64_tune(c, d, c->d_hd, c->d_pm);
  if (rc) return fail(rc);
  *out = d;
  return 0;
}

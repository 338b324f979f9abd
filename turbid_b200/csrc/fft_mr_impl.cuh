// Plane transforms of the even lengths up to 512 with prime factors 2, 3, 5 and
// 7 that are not powers of two (reference src/cube_real_cplx.cc:525-555; a
// spectral case's usual lengths 72, 96, 120, 144, 192, ...): the passes of
// fft.cu with radices chosen per length.  Included once per precision
// (fft_mr_f32.cu, fft_mr_f64.cu).
//
// The radices of the general kernels (fours, a two, threes, fives, sevens),
// in their order, are grouped into as few passes of at most 16 values as
// possible (96 = (4 4)(2 3), 120 = (4 2)(3 5), 192 = (4 4)(4 3)), each
// butterfly held in one thread's registers: the operations and their order are
// those of the general kernels, without their passes through memory.  Which
// products are fused into FMAs is left to the code generator (radix 2 apart,
// cmul2), so equal bits are measured, not promised: with nvcc 12.9 every
// compiled length gave the general kernels' values bit for bit, both precisions
// and directions.  The
// first pass takes its values straight from global memory, the last one hands
// them on from its registers, and the passes between work in place on one
// padded shared buffer: a two-pass length crosses shared memory once (twice
// where rows leave as kx columns).  NB transforms share a CTA, one butterfly per thread and pass, the widest pass
// filling about 128 threads.  Everything is compiled per length: one kernel
// with the radices chosen at run time held the widest butterfly's registers
// and every radix's constants (128-255 registers, kilobytes of spills).
//
// Bound by HBM and instruction issue like the power-of-two passes.  Forward /
// backward, 20 M points: 192x192 FP32 265 / 254 us in the general kernels (butterflies in
// dynamically indexed local memory, one pass per radix), 60 / 59 here; 120x96
// FP64 482 / 460 -> 141 / 132 us; 320x320 FP32 90 / 85 us.
#pragma once
#include <utility>

#include "fft_dev.cuh"
#include "fft_mr.cuh"

namespace tg {

namespace {

// The radices of a length, in the order of fft_plan_create: fours, a two,
// threes, fives, sevens.  Runs of them with a product of at most 16 form the
// passes: as few as possible, the smallest product as large as possible.
struct MrPlan {
  int ne = 0, e[10] = {0};             // elementary radices
  int n = 0, at[5] = {0};              // pass p: e[at[p]] .. e[at[p + 1] - 1]
  int r[4] = {1, 1, 1, 1};             // products: values per butterfly of a pass
};
// the best split of the radices from `start` on into n runs: fills f from pass p
// on and returns its smallest product, 0 if there is none
constexpr int mr_group(MrPlan& f, int start, int p, int n) {
  int best = 0;
  MrPlan out = f;
  for (int end = start + 1, r = 1; end <= f.ne; ++end) {
    r *= f.e[end - 1];
    if (r > 16) break;
    if ((n == 1) != (end == f.ne)) continue;
    MrPlan g = f;
    g.at[p] = start;
    g.at[p + 1] = end;
    g.r[p] = r;
    g.n = p + 1;
    int least = n == 1 ? r : mr_group(g, end, p + 1, n - 1);
    least = least < r ? least : r;
    if (least > best) best = least, out = g;
  }
  f = out;
  return best;
}
constexpr MrPlan mr_plan(int L) {
  MrPlan f;
  int n = L;
  while (n % 4 == 0) f.e[f.ne++] = 4, n /= 4;
  for (int q = 2; q <= 7; ++q)
    while (n % q == 0) f.e[f.ne++] = q, n /= q;
  for (int p = 2; p <= 4; ++p)
    if (mr_group(f, 0, 0, p) > 0) break;
  return f;
}

template <int L> struct Mr {
  static constexpr MrPlan F = mr_plan(L);
  static constexpr int n = F.n;
  static_assert(n >= 2, "length without a plan");
  static constexpr int E(int i) { return F.e[i]; }
  static constexpr int R(int p) { return F.r[p]; }
  static constexpr int nb(int p) { return L / F.r[p]; }                            // butterflies of pass p
  static constexpr int Ns(int p) { return p == 0 ? 1 : Ns(p - 1) * F.r[p - 1]; }   // stride of pass p
  static constexpr int widest() {
    int w = 0;
    for (int p = 0; p < n; ++p) w = nb(p) > w ? nb(p) : w;
    return w;
  }
  // transforms per CTA: about 128 butterflies of the widest pass, 256 with three
  // passes (320x320 FP32 90 / 85 us against 92 / 100; 192x192 64 / 61 against 60 / 59)
  static constexpr int NB = (n == 2 ? 128 : 256) / widest() < 1 ? 1 : (n == 2 ? 128 : 256) / widest();
  static constexpr int NT = (NB * widest() + 31) / 32 * 32;
  static constexpr int RS = (L + L / 16 + 1) | 1;                                  // padded row stride
  template <typename T> static constexpr size_t smem() { return (size_t)NB * RS * sizeof(cplx<T>); }
};

// DFT of E values, as the passes of the general kernels compute it
template <int E, int DIR, int L, typename T>
__device__ __forceinline__ void dft_e(cplx<T>* v, const cplx<T>* __restrict__ tw) {
  using C = cplx<T>;
  if constexpr (E == 2) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (E == 4) {
    const C t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]), t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
    const C t3r = (DIR < 0) ? mkc<C>(t3.y, -t3.x) : mkc<C>(-t3.y, t3.x);
    v[0] = cadd(t0, t2);
    v[1] = cadd(t1, t3r);
    v[2] = csub(t0, t2);
    v[3] = csub(t1, t3r);
  } else {
    C w[E], o[E];
#pragma unroll
    for (int k = 1; k < E; ++k) w[k] = tw_get<T, DIR>(tw, k * (L / E));
#pragma unroll
    for (int k = 0; k < E; ++k) {
      o[k] = v[0];
#pragma unroll
      for (int r = 1; r < E; ++r) o[k] = cadd(o[k], k == 0 ? v[r] : cmul(v[r], w[(r * k) % E]));
    }
#pragma unroll
    for (int k = 0; k < E; ++k) v[k] = o[k];
  }
}

// a w, rounded as the general kernels' radix-2 pass rounds it (nvcc 12.9 fuses
// the other product of the imaginary part there)
__device__ __forceinline__ float2 cmul2(float2 a, float2 w) {
  return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, __fmul_rn(a.x, w.y)));
}
__device__ __forceinline__ double2 cmul2(double2 a, double2 w) {
  return make_double2(__fma_rn(a.x, w.x, -__dmul_rn(a.y, w.y)), __fma_rn(a.y, w.x, __dmul_rn(a.x, w.y)));
}

// The elementary radices I .. END-1 of a pass on one butterfly's values in
// registers.  K values per group are already transformed: v[k * T + t], k < K,
// t < T (T = values / K); NS: stride of the pass, jm: the butterfly's twiddle
// index.  The operations and their order are those of one radix after the
// other through memory, whatever the grouping.
template <typename T, int DIR, int L, int I, int END, int NS, int K, int N>
__device__ __forceinline__ void mr_radices(cplx<T>* v, int jm, const cplx<T>* __restrict__ tw) {
  using C = cplx<T>;
  if constexpr (I < END) {
    constexpr int E = Mr<L>::E(I), Tn = N / K, Tm = Tn / E, step = L / (NS * K * E);
    C w[N];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      C f[E];   // twiddles of the digit k
#pragma unroll
      for (int r = 1; r < E; ++r)
        if (NS > 1 || k > 0) f[r] = tw_get<T, DIR>(tw, (NS > 1 ? jm + k * NS : k) * r * step);
#pragma unroll
      for (int t = 0; t < Tm; ++t) {
        C u[E];
#pragma unroll
        for (int r = 0; r < E; ++r) {
          u[r] = v[k * Tn + t + r * Tm];
          if (r > 0 && (NS > 1 || k > 0)) u[r] = E == 2 ? cmul2(u[r], f[r]) : cmul(u[r], f[r]);
        }
        dft_e<E, DIR, L, T>(u, tw);
#pragma unroll
        for (int q = 0; q < E; ++q) w[(k + K * q) * Tm + t] = u[q];
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = w[i];
    mr_radices<T, DIR, L, I + 1, END, NS, K * E, N>(v, jm, tw);
  }
}
template <typename T, int DIR, int L, int PS>
__device__ __forceinline__ void mr_dft(cplx<T>* v, int jm, const cplx<T>* __restrict__ tw) {
  mr_radices<T, DIR, L, Mr<L>::F.at[PS], Mr<L>::F.at[PS + 1], Mr<L>::Ns(PS), 1, Mr<L>::R(PS)>(v, jm, tw);
}

// First pass (stride 1): in(b, x) is value x of transform b; outputs to buf.
// BFAST: consecutive threads take consecutive transforms instead of
// consecutive butterflies (inputs interleaved by transform).
template <typename T, int DIR, int L, bool BFAST, typename In>
__device__ __forceinline__ void mr_first(cplx<T>* buf, const cplx<T>* __restrict__ tw, In&& in) {
  using C = cplx<T>;
  using P = Mr<L>;
  constexpr int R = P::R(0), nb = P::nb(0), idle = P::NT - P::NB * nb;
  const int idx = threadIdx.x;
  if (idle == 0 || idx < P::NB * nb) {
    const int j = BFAST ? idx / P::NB : idx % nb, b = BFAST ? idx % P::NB : idx / nb;
    C v[R];
    in(b, j, v);
    mr_dft<T, DIR, L, 0>(v, 0, tw);
    C* row = buf + b * P::RS;
#pragma unroll
    for (int k = 0; k < R; ++k) row[sp(R * j + k)] = v[k];
  }
  __syncthreads();
}

// loads and butterfly j of pass PS
template <typename T, int DIR, int L, int PS>
__device__ __forceinline__ void mr_butterfly(const cplx<T>* row, int j, const cplx<T>* __restrict__ tw, cplx<T>* v) {
  using P = Mr<L>;
  constexpr int R = P::R(PS), nb = P::nb(PS);
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = row[sp(j + r * nb)];
  mr_dft<T, DIR, L, PS>(v, j % P::Ns(PS), tw);
}

// the passes PS .. END-1, in place
template <typename T, int DIR, int L, int PS, int END>
__device__ __forceinline__ void mr_passes(cplx<T>* buf, const cplx<T>* __restrict__ tw) {
  using C = cplx<T>;
  using P = Mr<L>;
  if constexpr (PS < END) {
    constexpr int R = P::R(PS), nb = P::nb(PS), Ns = P::Ns(PS);
    const int idx = threadIdx.x, j = idx % nb;
    const bool ok = idx < P::NB * nb;
    C* row = buf + (idx / nb) * P::RS;
    C v[R];
    if (ok) mr_butterfly<T, DIR, L, PS>(row, j, tw, v);
    __syncthreads();
    if (ok) {
      const int jm = j % Ns, base = (j - jm) * R + jm;
#pragma unroll
      for (int k = 0; k < R; ++k) row[sp(base + k * Ns)] = v[k];
    }
    __syncthreads();
    mr_passes<T, DIR, L, PS + 1, END>(buf, tw);
  }
}

// The last pass: out(b, x, value) for each output, from registers.
template <typename T, int DIR, int L, bool BFAST, typename Out>
__device__ __forceinline__ void mr_last(const cplx<T>* buf, const cplx<T>* __restrict__ tw, Out&& out) {
  using P = Mr<L>;
  constexpr int PS = P::n - 1, R = P::R(PS), nb = P::nb(PS);
  const int idx = threadIdx.x;
  if (idx >= P::NB * nb) return;
  const int j = BFAST ? idx / P::NB : idx % nb, b = BFAST ? idx % P::NB : idx / nb;
  cplx<T> v[R];
  mr_butterfly<T, DIR, L, PS>(buf + b * P::RS, j, tw, v);
#pragma unroll
  for (int k = 0; k < R; ++k) out(b, j + k * nb, v[k]);
}

// forward x pass: two rows per complex FFT -> work [plane][kx][y]; each field
// formed as a[f] (b[f] + shift) (b[f] null: a[f] as it is), planes z-major
template <typename T, int L>
__global__ void __launch_bounds__(Mr<L>::NT) mr_fx_kernel(int nz, int ny, const cplx<T>* __restrict__ tw,
                                                         cplx<T>* work, PhysProduct prod) {
  pdl_begin();
  using C = cplx<T>;
  using P = Mr<L>;
  constexpr int rows = 2 * P::NB, R = P::R(0), nb = P::nb(0), nxh = L / 3 * 2 / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int y0 = blockIdx.x * rows, z = blockIdx.y / prod.nf, f = blockIdx.y - z * prod.nf;
  const T* src = reinterpret_cast<const T*>(prod.a[f]) + (size_t)z * ny * L;
  const T* srcb = prod.b[f] ? reinterpret_cast<const T*>(prod.b[f]) + (size_t)z * ny * L : nullptr;
  const T shb = (T)prod.sh[f];
  mr_first<T, -1, L, false>(buf, tw, [&](int b, int j, C* v) {
    const int ya = y0 + 2 * b, yb = ya + 1;
    const bool oka = ya < ny, okb = yb < ny;
    const int oa = (oka ? ya : 0) * L + j, ob = (okb ? yb : 0) * L + j;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = mkc<C>(oka ? src[oa + r * nb] : T(0), okb ? src[ob + r * nb] : T(0));
    if (srcb) {
      C w[R];
#pragma unroll
      for (int r = 0; r < R; ++r) w[r] = mkc<C>(oka ? srcb[oa + r * nb] : T(0), okb ? srcb[ob + r * nb] : T(0));
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = mkc<C>(v[r].x * (w[r].x + shb), v[r].y * (w[r].y + shb));
    }
  });
  mr_passes<T, -1, L, 1, P::n>(buf, tw);
  C* dst = work + (size_t)(f * nz + z) * nxh * ny;
  for (int idx = threadIdx.x; idx < rows * nxh; idx += P::NT) {
    const int k = idx / rows, q = idx % rows, y = y0 + q;
    if (y >= ny) continue;
    const C* row = buf + (q >> 1) * P::RS;
    const C Z = row[sp(k)], Zc = cconj(row[sp(k == 0 ? 0 : L - k)]);
    C X;
    if ((q & 1) == 0) {
      X = mkc<C>((Z.x + Zc.x) * T(0.5), (Z.y + Zc.y) * T(0.5));
    } else {
      const C D = csub(Z, Zc);
      X = mkc<C>(D.y * T(0.5), -D.x * T(0.5));
    }
    dst[(size_t)k * ny + y] = X;
  }
}

// forward y pass: kept modes of NB kx columns, FP64, scaled by 1/(Nx*Ny)
template <typename T, int L>
__global__ void __launch_bounds__(Mr<L>::NT) mr_fy_kernel(int nxh, const cplx<T>* __restrict__ tw,
                                                         const cplx<T>* work,
                                                         double2* spec, double scale) {
  pdl_begin();
  using C = cplx<T>;
  using P = Mr<L>;
  constexpr int R = P::R(0), nb = P::nb(0), nyc = L / 3 * 2, h = nyc / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int k0 = blockIdx.x * P::NB;
  const C* src = work + (size_t)blockIdx.y * nxh * L;
  double2* dst = spec + (size_t)blockIdx.y * nxh * nyc;
  mr_first<T, -1, L, false>(buf, tw, [&](int c, int j, C* v) {
    const bool ok = k0 + c < nxh;
    const C* col = src + (ok ? k0 + c : 0) * L + j;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ok ? col[r * nb] : mkc<C>(0, 0);
  });
  mr_passes<T, -1, L, 1, P::n - 1>(buf, tw);
  mr_last<T, -1, L, false>(buf, tw, [&](int c, int y, C z) {
    const bool lo = y < h, hi = y >= L - h;   // kept spectral rows
    if (k0 + c < nxh && (lo || hi))
      dst[(lo ? y : y - (L - nyc)) + nyc * (k0 + c)] = make_double2((double)z.x * scale, (double)z.y * scale);
  });
}

// backward y pass: zero between the kept bands, unscaled; the derivatives of a
// gathered launch formed on load (kx depends on the column, ky on the row
// alone: both tables are constant along the other index)
template <typename T, int L>
__global__ void __launch_bounds__(Mr<L>::NT) mr_by_kernel(int nz, int nxh, const cplx<T>* __restrict__ tw,
                                                         cplx<T>* work, SpecGather gat) {
  pdl_begin();
  using C = cplx<T>;
  using P = Mr<L>;
  constexpr bool RM = bwd_row_major<T>();
  constexpr int R = P::R(0), nb = P::nb(0), nyc = L / 3 * 2, h = nyc / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int k0 = blockIdx.x * P::NB;
  int deriv = 0;
  const double2* src = gather_src(gat, blockIdx.y, nz, nxh * nyc, deriv);
  mr_first<T, +1, L, false>(buf, tw, [&](int c, int j, C* v) {
    const int k = k0 + c;
    const bool okc = k < nxh;
    const double2* col = src + (okc ? k : 0) * nyc;
    double2 w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int y = j + r * nb;
      const bool lo = y < h, hi = y >= L - h;
      w[r] = okc && (lo || hi) ? col[lo ? y : y - (L - nyc)] : make_double2(0.0, 0.0);
    }
    if (deriv != 0) {
      const double kc = okc && deriv == 1 ? gat.kx[k * nyc] : 0.0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int y = j + r * nb;
        const bool lo = y < h, hi = y >= L - h;
        const double kk = deriv == 1 ? kc : lo || hi ? gat.ky[lo ? y : y - (L - nyc)] : 0.0;
        w[r] = make_double2(0.0 * w[r].x - kk * w[r].y, 0.0 * w[r].y + kk * w[r].x);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = mkc<C>((T)w[r].x, (T)w[r].y);
  });
  mr_passes<T, +1, L, 1, P::n - 1>(buf, tw);
  C* dst = work + (size_t)blockIdx.y * nxh * L;
  mr_last<T, +1, L, RM>(buf, tw, [&](int c, int y, C z) {
    const int k = k0 + c;
    if (k < nxh) dst[RM ? y * nxh + k : k * L + y] = z;
  });
}

// packed two-row input of a backward x pass: Z[x] = X1[x] + i X2[x], X[L-k] =
// conj X[k], zero between the kept bands, Im of kx = 0 ignored (c2r)
template <typename T, int L>
__device__ __forceinline__ void mr_bx_first(cplx<T>* buf, const cplx<T>* __restrict__ tw,
                                            const cplx<T>* src, int ny, int y0) {
  using C = cplx<T>;
  using P = Mr<L>;
  constexpr bool RM = bwd_row_major<T>();
  constexpr int R = P::R(0), nb = P::nb(0), nxh = L / 3 * 2 / 2 + 1;
  mr_first<T, +1, L, !RM>(buf, tw, [&](int b, int j, C* v) {
    const int ya = y0 + 2 * b, yb = ya + 1;
    const bool oka = ya < ny, okb = yb < ny;
    const C* r1 = src + (oka ? ya : 0) * (RM ? nxh : 1);
    const C* r2 = src + (okb ? yb : 0) * (RM ? nxh : 1);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int x = j + r * nb;
      const bool lo = x < nxh, in = lo || x > L - nxh;
      const int k = (lo ? x : L - x) * (RM ? 1 : ny);
      C a = oka && in ? r1[k] : mkc<C>(0, 0);
      C c = okb && in ? r2[k] : mkc<C>(0, 0);
      if (x == 0) a.y = c.y = T(0);
      v[r] = lo ? mkc<C>(a.x - c.y, a.y + c.x) : mkc<C>(a.x + c.y, -a.y + c.x);
    }
  });
}

template <typename T, int L>
__global__ void __launch_bounds__(Mr<L>::NT) mr_bx_kernel(int ny, const cplx<T>* __restrict__ tw,
                                                         const cplx<T>* work, T* phys) {
  pdl_begin();
  using C = cplx<T>;
  using P = Mr<L>;
  constexpr int nxh = L / 3 * 2 / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int y0 = blockIdx.x * 2 * P::NB;
  T* dst = phys + (size_t)blockIdx.y * ny * L;
  mr_bx_first<T, L>(buf, tw, work + (size_t)blockIdx.y * nxh * ny, ny, y0);
  mr_passes<T, +1, L, 1, P::n - 1>(buf, tw);
  mr_last<T, +1, L, false>(buf, tw, [&](int b, int x, C z) {
    const int ya = y0 + 2 * b, yb = ya + 1;
    if (ya < ny) dst[ya * L + x] = z.x;
    if (yb < ny) dst[yb * L + x] = z.y;
  });
}

// Backward x pass of ncomp groups of three gradient fields, each reduced to
// the advection term (u + su) d/dx + (v + sv) d/dy + (w + sw) d/dz
// (phase_carrier_flat.cc:786-797, phase_scalar_flat.cc:588-591): a thread's
// last butterfly covers the same points for the three gradients, so the sums
// stay in its registers and the physical gradients are never written.  grid:
// (row blocks x ncomp, nz), component fastest, so that the velocity rows the
// ncomp CTAs share come from DRAM once.  The velocity values of a butterfly
// are loaded side by side, rows beyond the last from the first row (not
// stored): with a branch around each load the kernel waited for one load at a
// time (144x144x145 class 0.380 -> 0.131 ms per step mixed, 0.680 -> 0.271
// FP64).
template <typename T, int L>
__global__ void __launch_bounds__(Mr<L>::NT, sizeof(T) == 4 ? 512 / Mr<L>::NT : 1)
    mr_adv_kernel(int nz, int ny, const cplx<T>* __restrict__ tw, const cplx<T>* work, const T* unl, T* out, int ncomp,
                  double su, double sv, double sw) {
  pdl_begin();
  using C = cplx<T>;
  using P = Mr<L>;
  constexpr int nxh = L / 3 * 2 / 2 + 1, PS = P::n - 1, R = P::R(PS), nb = P::nb(PS);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int z = blockIdx.y, blk = blockIdx.x / ncomp, comp = blockIdx.x - blk * ncomp, y0 = blk * 2 * P::NB;
  const int idx = threadIdx.x, j = idx % nb, b = idx / nb, ya = y0 + 2 * b;
  const bool ok = b < P::NB, oka = ok && ya < ny, okb = ok && ya + 1 < ny;
  const size_t field = (size_t)nz * ny * L, off = ((size_t)z * ny + y0) * L;
  const int oa = (oka ? 2 * b * L : 0) + j, ob = (okb ? (2 * b + 1) * L : 0) + j;
  C acc[R];
#pragma unroll
  for (int k = 0; k < R; ++k) acc[k] = mkc<C>(0, 0);
#pragma unroll 1
  for (int i = 0; i < 3; ++i) {   // d/dy, d/dx, d/dz: u d/dx + v d/dy is one rounded product and one fused one
    const int g = i == 2 ? 2 : 1 - i;
    if (i > 0) __syncthreads();   // buf is refilled
    mr_bx_first<T, L>(buf, tw, work + (size_t)((3 * comp + g) * nz + z) * nxh * ny, ny, y0);
    mr_passes<T, +1, L, 1, PS>(buf, tw);
    if (ok) {
      const T* uj = unl + g * field + off;
      const T sh = (T)(g == 0 ? su : g == 1 ? sv : sw);
      T ua[R], ub[R];
#pragma unroll
      for (int k = 0; k < R; ++k) {
        ua[k] = uj[oa + k * nb];
        ub[k] = uj[ob + k * nb];
      }
      C v[R];
      mr_butterfly<T, +1, L, PS>(buf + b * P::RS, j, tw, v);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        acc[k].x += (ua[k] + sh) * v[k].x;
        acc[k].y += (ub[k] + sh) * v[k].y;
      }
    }
  }
  T* dst = out + comp * field + off;
#pragma unroll
  for (int k = 0; k < R; ++k) {
    if (oka) dst[oa + k * nb] = acc[k].x;
    if (okb) dst[ob + k * nb] = acc[k].y;
  }
}

// ---------------------------------------------------------------------------
// launchers: f(integral_constant<int, L>) for the compiled length L
// ---------------------------------------------------------------------------
template <int L, typename F>
bool mr_at(F& f) {
  if constexpr (mr_length(L)) {
    f(std::integral_constant<int, L>{});
    return true;
  }
  return false;
}
template <typename F, int... I>
bool mr_dispatch(int L, F&& f, std::integer_sequence<int, I...>) {
  return ((L == 2 * I && mr_at<2 * I>(f)) || ...);
}
template <typename F>
bool mr_dispatch(int L, F&& f) {
  return mr_length(L) && mr_dispatch(L, f, std::make_integer_sequence<int, kMrMaxLength / 2 + 1>{});
}
int blocks(int n, int per) { return (n + per - 1) / per; }

}  // namespace

template <typename T>
bool mr_forward_x(const TransformDims& d, const FftPlan& px, const T* phys, void* work, int planes, cudaStream_t s,
                  const PhysProduct* prod) {
  PhysProduct pp{};
  int nz = planes;
  if (prod) {
    pp = *prod;
    nz = d.nz;
  } else {
    pp.a[0] = phys;
    pp.nf = 1;
  }
  return mr_dispatch(d.nx, [&](auto lc) {
    using P = Mr<decltype(lc)::value>;
    launch_pdl(mr_fx_kernel<T, decltype(lc)::value>, dim3(blocks(d.ny, 2 * P::NB), planes), P::NT, P::template smem<T>(), s, nz, d.ny, Tw<T>::get(px), reinterpret_cast<cplx<T>*>(work), pp);
  });
}

template <typename T>
bool mr_forward_y(const TransformDims& d, const FftPlan& py, const void* work, double2* spec, int planes, double scale,
                  cudaStream_t s) {
  return mr_dispatch(d.ny, [&](auto lc) {
    using P = Mr<decltype(lc)::value>;
    launch_pdl(mr_fy_kernel<T, decltype(lc)::value>, dim3(blocks(d.nxh, P::NB), planes), P::NT, P::template smem<T>(), s, d.nxh, Tw<T>::get(py), reinterpret_cast<const cplx<T>*>(work), spec, scale);
  });
}

template <typename T>
bool mr_backward_y(const TransformDims& d, const FftPlan& py, const double2* spec, void* work, int planes,
                   cudaStream_t s, const SpecGather* gather) {
  SpecGather g{};
  int nz = planes;
  if (gather) {
    g = *gather;
    nz = d.nz;
  } else {
    g.src[0] = spec;
    g.nf = 1;
  }
  return mr_dispatch(d.ny, [&](auto lc) {
    using P = Mr<decltype(lc)::value>;
    launch_pdl(mr_by_kernel<T, decltype(lc)::value>, dim3(blocks(d.nxh, P::NB), planes), P::NT, P::template smem<T>(), s, nz, d.nxh, Tw<T>::get(py), reinterpret_cast<cplx<T>*>(work), g);
  });
}

template <typename T>
bool mr_backward_x(const TransformDims& d, const FftPlan& px, const void* work, T* phys, int planes, cudaStream_t s) {
  return mr_dispatch(d.nx, [&](auto lc) {
    using P = Mr<decltype(lc)::value>;
    launch_pdl(mr_bx_kernel<T, decltype(lc)::value>, dim3(blocks(d.ny, 2 * P::NB), planes), P::NT, P::template smem<T>(), s, d.ny, Tw<T>::get(px), reinterpret_cast<const cplx<T>*>(work), phys);
  });
}

template <typename T>
bool mr_backward_adv(const TransformDims& d, const FftPlan& px, const void* work, const T* unl, T* out, int ncomp,
                     double su, double sv, double sw, cudaStream_t s) {
  return mr_dispatch(d.nx, [&](auto lc) {
    using P = Mr<decltype(lc)::value>;
    launch_pdl(mr_adv_kernel<T, decltype(lc)::value>, dim3(blocks(d.ny, 2 * P::NB) * ncomp, d.nz), P::NT, P::template smem<T>(), s, d.nz, d.ny, Tw<T>::get(px), reinterpret_cast<const cplx<T>*>(work), unl, out, ncomp, su, sv, sw);
  });
}

#define TG_MR_INSTANTIATE(T)                                                                                        \
  template bool mr_forward_x<T>(const TransformDims&, const FftPlan&, const T*, void*, int, cudaStream_t,           \
                                const PhysProduct*);                                                                \
  template bool mr_forward_y<T>(const TransformDims&, const FftPlan&, const void*, double2*, int, double,           \
                                cudaStream_t);                                                                      \
  template bool mr_backward_y<T>(const TransformDims&, const FftPlan&, const double2*, void*, int, cudaStream_t,    \
                                 const SpecGather*);                                                                \
  template bool mr_backward_x<T>(const TransformDims&, const FftPlan&, const void*, T*, int, cudaStream_t);         \
  template bool mr_backward_adv<T>(const TransformDims&, const FftPlan&, const void*, const T*, T*, int, double,    \
                                   double, double, cudaStream_t);

}  // namespace tg

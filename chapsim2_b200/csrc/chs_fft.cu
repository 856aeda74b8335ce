// FFTs of the Poisson solvers in at most three stages held in registers.
//
// A length n = 2^a 3^b up to 729 factors into at most three radices of 2, 3, 4, 6, 8, 9 (fft_stages), the largest in
// the middle.  The first Stockham stage takes its inputs from global memory and the last stores its results there, so a
// line passes through shared memory once per stage boundary, twice at most; the middle stage works in place, one
// butterfly per thread between two barriers.  The forward transform of real rows, whose spectra are formed from two
// positions each, passes once more.  Twiddles are read from a copy in shared memory.
//
// z and y lines lie side by side in the tile, as many as 64 KB and 512 threads allow: segments of 256 bytes in every
// row up to 256 points in FP64 (216: 128) and up to 128 in FP32 (108 and above 128: 128, above 256: 64), narrower
// beyond.
// Their accesses are free of bank conflicts from 8 lines (FP64) or 16 (FP32) up.  x rows are padded by one position in
// nine, which keeps the stores of a first radix 2, 4 or 8 apart; 3, 6 and 9 meet in pairs.
//
// The kernels of chs_kernels.cu (radix 4, 2, 3 stages through two shared buffers with twiddles from
// global memory) pass a line through shared memory nst + 1 times; they keep longer lines.  The four transforms of a
// solve, with those and with these: 128x96x128 FP64 54 and 35 us, 384x256x384 FP32 758 and 490, 64^3 (six) 48 and 23.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <initializer_list>
#include <stdexcept>

#include "chs_kernels.cuh"

namespace chs {

namespace {

template <typename C>
struct Sc;
template <>
struct Sc<double2> {
  using S = double;
  static __device__ const double2* tw(const FftPlan& f) { return f.tw; }
};
template <>
struct Sc<float2> {
  using S = float;
  static __device__ const float2* tw(const FftPlan& f) { return f.twf; }
};
template <typename C, typename S>
__device__ __forceinline__ C mk(S x, S y) {
  C c;
  c.x = x;
  c.y = y;
  return c;
}
template <typename C>
__device__ __forceinline__ C add(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <typename C>
__device__ __forceinline__ C sub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
template <typename C>
__device__ __forceinline__ C mul(C a, C b) { return mk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a * (c + i s)
template <typename C, typename S>
__device__ __forceinline__ C rot(C a, S c, S s) { return mk<C>(a.x * c - a.y * s, a.x * s + a.y * c); }
// a * (i sg)
template <typename C, typename S>
__device__ __forceinline__ C rot90(C a, S sg) { return mk<C>(-sg * a.y, sg * a.x); }

// x c for an irrational c = hi + lo.  A constant rounded once errs the same way in every product of every stage,
// forward and back: with hi alone the FP64 solve of a 64^3 box errs by 4.2 units of 2^-53, with both by 3.5
template <typename S>
__device__ __forceinline__ S times(S x, S hi, S lo) { return fma(x, hi, x * lo); }
template <typename S>
struct Root {  // sqrt(3) / 2 and sqrt(1/2)
  static constexpr S h3 = S(0.86602540378443864676), h2 = S(0.70710678118654752440);
  static constexpr S l3 = sizeof(S) == 8 ? S(5.01754211090345140e-17) : S(0.86602540378443864676 - (double)h3);
  static constexpr S l2 = sizeof(S) == 8 ? S(-4.83364665672645673e-17) : S(0.70710678118654752440 - (double)h2);
};

// in place DFT of R values, exponent sign sg
template <typename C, typename S>
__device__ __forceinline__ void dft3(C& a, C& b, C& c, S sg) {
  const C t = add(b, c), d = sub(b, c);
  const C m = mk<C>(a.x - S(0.5) * t.x, a.y - S(0.5) * t.y);
  const C e = mk<C>(-sg * times(d.y, Root<S>::h3, Root<S>::l3), sg * times(d.x, Root<S>::h3, Root<S>::l3));
  a = add(a, t);
  b = add(m, e);
  c = sub(m, e);
}
template <typename C, typename S>
__device__ __forceinline__ void dft4(C& a, C& b, C& c, C& d, S sg) {
  const C p = add(a, c), q = sub(a, c), r = add(b, d), t = rot90(sub(b, d), sg);
  a = add(p, r);
  b = add(q, t);
  c = sub(p, r);
  d = sub(q, t);
}
template <int R, typename C, typename S>
__device__ __forceinline__ void dft(C (&v)[R], S sg) {
  if constexpr (R == 2) {
    const C a = v[0];
    v[0] = add(a, v[1]);
    v[1] = sub(a, v[1]);
  } else if constexpr (R == 3) {
    dft3(v[0], v[1], v[2], sg);
  } else if constexpr (R == 4) {
    dft4(v[0], v[1], v[2], v[3], sg);
  } else if constexpr (R == 6) {
    // prime factors: inputs 3 a + 2 b, outputs 3 a' + 4 b' (mod 6) need no factors between the 3s and the 2s.  The
    // rotations of the common-factor form added 5 % to the error of a transform of 216 and 9 % to that of 36
    dft3(v[0], v[2], v[4], sg);
    dft3(v[3], v[5], v[1], sg);
    const C a0 = v[0], a1 = v[2], a2 = v[4], b0 = v[3], b1 = v[5], b2 = v[1];
    v[0] = add(a0, b0); v[3] = sub(a0, b0);
    v[4] = add(a1, b1); v[1] = sub(a1, b1);
    v[2] = add(a2, b2); v[5] = sub(a2, b2);
  } else if constexpr (R == 8) {
    dft4(v[0], v[2], v[4], v[6], sg);
    dft4(v[1], v[3], v[5], v[7], sg);
    // by 45 and 135 degrees: sqrt(1/2) (1 + i sg) and sqrt(1/2) (-1 + i sg)
    auto diag = [](S x, S y) { return mk<C>(times(x, Root<S>::h2, Root<S>::l2), times(y, Root<S>::h2, Root<S>::l2)); };
    const C p = v[3], q = v[7];
    const C o0 = v[1], o1 = diag(p.x - sg * p.y, sg * p.x + p.y), o2 = rot90(v[5], sg),
            o3 = diag(-q.x - sg * q.y, sg * q.x - q.y);
    const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = add(e0, o0); v[1] = add(e1, o1); v[2] = add(e2, o2); v[3] = add(e3, o3);
    v[4] = sub(e0, o0); v[5] = sub(e1, o1); v[6] = sub(e2, o2); v[7] = sub(e3, o3);
  } else {  // 9
    const S c1 = S(0.76604444311897803520), s1 = sg * S(0.64278760968653932632);   // 40 degrees
    const S c2 = S(0.17364817766693034885), s2 = sg * S(0.98480775301220805937);   // 80
    const S c4 = S(-0.93969262078590838405), s4 = sg * S(0.34202014332566873304);  // 160
    dft3(v[0], v[3], v[6], sg);
    dft3(v[1], v[4], v[7], sg);
    dft3(v[2], v[5], v[8], sg);
    v[4] = rot(v[4], c1, s1);
    v[5] = rot(v[5], c2, s2);
    v[7] = rot(v[7], c2, s2);
    v[8] = rot(v[8], c4, s4);
    // v[m + 3 k1] for residue m: sum over m gives X[k1 + 3 k2]
    dft3(v[0], v[1], v[2], sg);
    dft3(v[3], v[4], v[5], sg);
    dft3(v[6], v[7], v[8], sg);
    C t;
    t = v[1]; v[1] = v[3]; v[3] = t;
    t = v[2]; v[2] = v[6]; v[6] = t;
    t = v[5]; v[5] = v[7]; v[7] = t;
  }
}

// x / d for 0 <= x < 2^23 from a float reciprocal with one correction step
__device__ __forceinline__ int div_small(int x, int d, float inv) {
  int q = __float2int_rz((float)x * inv);
  const int r = x - q * d;
  if (r >= d) ++q;
  else if (r < 0) --q;
  return q;
}

// One Stockham stage of radix R over the thread's butterflies t = tid, tid + T, ...: `split` gives the
// line and column of t, `get(line, p)` the input at position p, `put(line, p, v)` takes the output.  FIRST: no
// twiddles.  SYNC: a barrier between the reads and the writes (in place; at most one butterfly per thread).
template <int R, bool FIRST, bool SYNC, typename C, typename FS, typename FG, typename FP>
__device__ __forceinline__ void stage(int n, int ns, int total, int sign, const C* tw, const FS& split, const FG& get,
                                      const FP& put) {
  using S = typename Sc<C>::S;
  const int nb = n / R, tstep = nb / ns;
  const float ins = 1.0f / (float)ns;
  for (int t0 = threadIdx.x; SYNC ? t0 < (int)blockDim.x : t0 < total; t0 += blockDim.x) {
    const bool on = !SYNC || t0 < total;
    int line, j;
    split(on ? t0 : 0, nb, line, j);
    const int jq = FIRST ? j : div_small(j, ns, ins), k = FIRST ? 0 : j - jq * ns;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = get(line, j + r * nb);
    if (!FIRST) {
#pragma unroll
      for (int r = 1; r < R; ++r) {
        C w = tw[k * r * tstep];
        if (sign > 0) w.y = -w.y;
        v[r] = mul(v[r], w);
      }
    }
    dft<R>(v, S(sign));
    if (SYNC) __syncthreads();
    if (on) {
      const int o = jq * ns * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) put(line, o + r * ns, v[r]);
    }
  }
}
template <bool FIRST, bool SYNC, typename C, typename FS, typename FG, typename FP>
__device__ __forceinline__ void stage_of(int R, int n, int ns, int lines, int sign, const C* tw, const FS& split,
                                         const FG& get, const FP& put) {
  const int total = lines * (n / R);
  if (R == 8) stage<8, FIRST, SYNC, C>(n, ns, total, sign, tw, split, get, put);
  else if (R == 4) stage<4, FIRST, SYNC, C>(n, ns, total, sign, tw, split, get, put);
  else if (R == 6) stage<6, FIRST, SYNC, C>(n, ns, total, sign, tw, split, get, put);
  else if (R == 9) stage<9, FIRST, SYNC, C>(n, ns, total, sign, tw, split, get, put);
  else if (R == 3) stage<3, FIRST, SYNC, C>(n, ns, total, sign, tw, split, get, put);
  else stage<2, FIRST, SYNC, C>(n, ns, total, sign, tw, split, get, put);
}
// the stages of a line: load from `get`, results to `put`, the tile (loc: index of a line's position) between
template <typename C, typename FS, typename FL, typename FG, typename FP>
__device__ __forceinline__ void stages(const FftPlan& fp, int lines, int sign, const C* tw, C* tile, const FS& split,
                                       const FL& loc, const FG& get, const FP& put) {
  const int n = fp.n, m = fp.rst;
  auto sget = [&](int l, int p) { return tile[loc(l, p)]; };
  auto sput = [&](int l, int p, C v) { tile[loc(l, p)] = v; };
  if (m == 1) {
    stage_of<true, false, C>(fp.rrad[0], n, 1, lines, sign, tw, split, get, put);
    return;
  }
  stage_of<true, false, C>(fp.rrad[0], n, 1, lines, sign, tw, split, get, sput);
  __syncthreads();
  int ns = fp.rrad[0];
  if (m == 3) {
    stage_of<false, true, C>(fp.rrad[1], n, ns, lines, sign, tw, split, sget, sput);
    __syncthreads();
    ns *= fp.rrad[1];
  }
  stage_of<false, false, C>(fp.rrad[m - 1], n, ns, lines, sign, tw, split, sget, put);
}

template <typename C>
__device__ __forceinline__ void copy_twiddles(const FftPlan& fp, C* tw) {
  const C* g = Sc<C>::tw(fp);
  for (int t = threadIdx.x; t < fp.n; t += blockDim.x) tw[t] = g[t];
}

// strided lines, 1 << lsh of them per CTA
template <typename C>
__global__ void __launch_bounds__(512, 2) cfft_lines_kernel(const __grid_constant__ FftPlan fp, C* data,
                                                            int na, int nlines, int64_t bstride, int64_t stride,
                                                            int sign, int lsh) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  C* tw = reinterpret_cast<C*>(fft_smem);
  C* tile = tw + fp.n;
  const int lines = 1 << lsh;
  grid_dep_launch();
  copy_twiddles(fp, tw);
  grid_dep_wait();
  // blockDim is a multiple of `lines`: a thread keeps its line
  const int l = threadIdx.x & (lines - 1), g = (blockIdx.x << lsh) + l;
  const bool ok = g < nlines;
  const int b = ok ? g / na : 0, a = ok ? g - b * na : 0;
  C* line = data + (a + b * bstride);
  auto split = [&](int t, int, int& ln, int& j) { ln = l; j = t >> lsh; };
  auto loc = [&](int ln, int p) { return (p << lsh) + ln; };
  auto get = [&](int, int p) { return line[p * stride]; };
  auto put = [&](int, int p, C v) {
    if (ok) line[p * stride] = v;
  };
  stages<C>(fp, lines, sign, tw, tile, split, loc, get, put);
}

// x rows, two real rows per transform, `pairs` transforms per CTA
__device__ __forceinline__ int pad9(int p) { return p + (p >> 3); }

template <typename R, typename C>
__global__ void __launch_bounds__(512, 2) rfft_rows_kernel(const __grid_constant__ FftPlan fp, const R* __restrict__ in,
                                                           C* __restrict__ out, int nrows, int pairs) {
  using S = typename Sc<C>::S;
  extern __shared__ __align__(16) unsigned char fft_smem[];
  C* tw = reinterpret_cast<C*>(fft_smem);
  C* tile = tw + fp.n;
  const int n = fp.n, nh = n / 2 + 1, ls = pad9(n) + 1, pair0 = blockIdx.x * pairs;
  grid_dep_launch();
  copy_twiddles(fp, tw);
  auto split = [&](int t, int nb, int& ln, int& j) {
    ln = div_small(t, nb, 1.0f / (float)nb);
    j = t - ln * nb;
  };
  auto loc = [&](int ln, int p) { return ln * ls + pad9(p); };
  auto get = [&](int ln, int p) {
    const int ra = 2 * (pair0 + ln);
    const R* row = in + (int64_t)ra * n + p;
    return mk<C>(ra < nrows ? (S)row[0] : S(0), ra + 1 < nrows ? (S)row[n] : S(0));
  };
  auto put = [&](int ln, int p, C v) { tile[loc(ln, p)] = v; };
  if (fp.rst == 1) {
    stages<C>(fp, pairs, -1, tw, tile, split, loc, get, put);
  } else {
    // the last stage writes the tile it reads: its results wait in registers behind a barrier, as those of
    // the middle stage do
    const int m = fp.rst;
    auto sget = [&](int l, int p) { return tile[loc(l, p)]; };
    stage_of<true, false, C>(fp.rrad[0], n, 1, pairs, -1, tw, split, get, put);
    __syncthreads();
    int ns = fp.rrad[0];
    for (int s = 1; s < m; ++s) {
      stage_of<false, true, C>(fp.rrad[s], n, ns, pairs, -1, tw, split, sget, put);
      ns *= fp.rrad[s];
      if (s + 1 < m) __syncthreads();
    }
  }
  __syncthreads();
  const float innh = 1.0f / (float)nh;
  for (int t = threadIdx.x; t < pairs * nh; t += blockDim.x) {
    const int l = div_small(t, nh, innh), k = t - l * nh;
    const int ra = 2 * (pair0 + l), rb = ra + 1;
    const C z = tile[loc(l, k)];
    C zc = tile[loc(l, k == 0 ? 0 : n - k)];
    zc.y = -zc.y;
    const C d = sub(z, zc);
    if (ra < nrows) out[(int64_t)ra * nh + k] = mk<C>(S(0.5) * (z.x + zc.x), S(0.5) * (z.y + zc.y));
    if (rb < nrows) out[(int64_t)rb * nh + k] = mk<C>(S(0.5) * d.y, S(-0.5) * d.x);
  }
}

template <typename R, typename C>
__global__ void __launch_bounds__(512, 2) irfft_rows_kernel(const __grid_constant__ FftPlan fp, const C* in,
                                                            R* __restrict__ out, int nrows, double scale, int pairs) {
  using S = typename Sc<C>::S;
  extern __shared__ __align__(16) unsigned char fft_smem[];
  C* tw = reinterpret_cast<C*>(fft_smem);
  C* tile = tw + fp.n;
  const int n = fp.n, nh = n / 2 + 1, ls = pad9(n) + 1, pair0 = blockIdx.x * pairs;
  grid_dep_launch();
  copy_twiddles(fp, tw);
  grid_dep_wait();
  const S sc = (S)scale;
  auto split = [&](int t, int nb, int& ln, int& j) {
    ln = div_small(t, nb, 1.0f / (float)nb);
    j = t - ln * nb;
  };
  auto loc = [&](int ln, int p) { return ln * ls + pad9(p); };
  // xa + i xb from the half spectra of the two rows
  auto get = [&](int ln, int p) {
    const int ra = 2 * (pair0 + ln);
    const bool hi = p > n / 2;
    const int kk = hi ? n - p : p;
    C A = mk<C>(S(0), S(0)), B = A;
    const C* row = in + (int64_t)ra * nh + kk;
    if (ra < nrows) A = row[0];
    if (ra + 1 < nrows) B = row[nh];
    if (kk == 0 || 2 * kk == n) { A.y = S(0); B.y = S(0); }
    if (hi) { A.y = -A.y; B.y = -B.y; }
    return mk<C>(A.x - B.y, A.y + B.x);
  };
  auto put = [&](int ln, int p, C v) {
    const int ra = 2 * (pair0 + ln);
    R* row = out + (int64_t)ra * n + p;
    if (ra < nrows) row[0] = R(v.x * sc);
    if (ra + 1 < nrows) row[n] = R(v.y * sc);
  };
  stages<C>(fp, pairs, +1, tw, tile, split, loc, get, put);
}

// threads for `lines` transforms: one butterfly each in the middle stage, which works in place (and, for rows, in
// the last one)
int fft_threads(const FftPlan& fp, int lines, bool last_in_place) {
  int r = fp.rrad[fp.rst > 1 ? 1 : 0];
  if (fp.rst == 3 && last_in_place) r = std::min(fp.rrad[1], fp.rrad[2]);
  return (lines * (fp.n / r) + 31) / 32 * 32;
}

// transforms of x rows per CTA: about 256 threads, fewer while the grid leaves SMs without two CTAs
int row_pairs(const FftPlan& fp, int npairs) {
  int p = std::max(1, 2048 / fp.n);
  while (p > 1 && fft_threads(fp, p, true) > 512) --p;
  while (p > 1 && (npairs + p - 1) / p < 2 * 148 && fft_threads(fp, p, true) > 64) p = (p + 1) / 2;
  return p;
}

}  // namespace

void fft_stages(FftPlan& fp) {
  // fewest stages, then the smallest sum of radices; the largest in the middle of three, else last
  static const int rad[6] = {2, 3, 4, 6, 8, 9};
  fp.rst = 0;
  int best = 1 << 30;
  auto take = [&](std::initializer_list<int> r) {
    int n = 1, sum = 0, k = 0;
    for (int x : r) { n *= x; sum += x; }
    if (n != fp.n || (fp.rst && ((int)r.size() > fp.rst || ((int)r.size() == fp.rst && sum >= best)))) return;
    fp.rst = (int)r.size();
    best = sum;
    for (int x : r) fp.rrad[k++] = x;
    std::sort(fp.rrad, fp.rrad + k);
    if (k == 3) std::swap(fp.rrad[1], fp.rrad[2]);
  };
  for (int a : rad) {
    take({a});
    for (int b : rad) {
      if (b < a) continue;
      take({a, b});
      for (int c : rad)
        if (c >= b) take({a, b, c});
    }
  }
}

void fft_twiddles(int n, double2* tw) {
  // angles in extended precision: 2 pi k / n formed in FP64 is off by up to several eps.  Error of an FP64 transform
  // of 96 and 216 (rms, relative, in units of 2^-53): 2.4 and 3.0 with such angles, 1.4 and 1.6 with these
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int k = 0; k < n; ++k)
    tw[k] = make_double2((double)std::cos(2 * pi * k / n), -(double)std::sin(2 * pi * k / n));
}

template <typename R, typename C>
void launch_rfft_rows(const FftPlan& fp, const R* in, C* out, int nrows, cudaStream_t st) {
  const int npairs = (nrows + 1) / 2, pairs = row_pairs(fp, npairs), n = fp.n;
  const size_t shm = ((size_t)n + (size_t)pairs * (n + n / 8 + 1)) * sizeof(C);
  allow_smem<rfft_rows_kernel<R, C>>(shm);
  rfft_rows_kernel<R, C><<<(npairs + pairs - 1) / pairs, fft_threads(fp, pairs, true), shm, st>>>(fp, in, out, nrows,
                                                                                                  pairs);
}
template <typename R, typename C>
void launch_irfft_rows(const FftPlan& fp, const C* in, R* out, int nrows, double scale, cudaStream_t st, bool chained) {
  const int npairs = (nrows + 1) / 2, pairs = row_pairs(fp, npairs), n = fp.n;
  const size_t shm = ((size_t)n + (size_t)pairs * (n + n / 8 + 1)) * sizeof(C);
  allow_smem<irfft_rows_kernel<R, C>>(shm);
  launch_chained(irfft_rows_kernel<R, C>, dim3((npairs + pairs - 1) / pairs), dim3(fft_threads(fp, pairs, false)), shm,
                 st, chained, fp, in, out, nrows, scale, pairs);
}
template <typename C>
void launch_cfft_lines(const FftPlan& fp, C* data, int na, int nb, int64_t bstride, int64_t stride, int sign,
                       cudaStream_t st, bool chained) {
  const int64_t nlines = (int64_t)na * nb;
  if (nlines > 0x3fffffff) throw std::runtime_error("FFT: too many lines");
  // 256-byte segments, narrower while the tile exceeds 64 KB or the CTA 512 threads
  int lsh = sizeof(C) == 16 ? 4 : 5;
  while (lsh > 2 && (((size_t)fp.n << lsh) * sizeof(C) > 64 * 1024 || fft_threads(fp, 1 << lsh, false) > 512)) --lsh;
  const size_t shm = ((size_t)fp.n + ((size_t)fp.n << lsh)) * sizeof(C);
  allow_smem<cfft_lines_kernel<C>>(shm);
  launch_chained(cfft_lines_kernel<C>, dim3((unsigned)((nlines + (1 << lsh) - 1) >> lsh)),
                 dim3(fft_threads(fp, 1 << lsh, false)), shm, st, chained, fp, data, na, (int)nlines, bstride, stride,
                 sign, lsh);
}
template void launch_rfft_rows<double, double2>(const FftPlan&, const double*, double2*, int, cudaStream_t);
template void launch_rfft_rows<float, double2>(const FftPlan&, const float*, double2*, int, cudaStream_t);
template void launch_rfft_rows<float, float2>(const FftPlan&, const float*, float2*, int, cudaStream_t);
template void launch_irfft_rows<double, double2>(const FftPlan&, const double2*, double*, int, double, cudaStream_t,
                                                 bool);
template void launch_irfft_rows<float, double2>(const FftPlan&, const double2*, float*, int, double, cudaStream_t,
                                                 bool);
template void launch_irfft_rows<float, float2>(const FftPlan&, const float2*, float*, int, double, cudaStream_t,
                                                 bool);
template void launch_cfft_lines<double2>(const FftPlan&, double2*, int, int, int64_t, int64_t, int, cudaStream_t, bool);
template void launch_cfft_lines<float2>(const FftPlan&, float2*, int, int, int64_t, int64_t, int, cudaStream_t, bool);

}  // namespace chs

// Compact line operators with the line kept in registers (CP4 and CP6).
//
// A CTA owns 32 lines.  Warp w holds rows w*R .. w*R + R-1 of every one of them, lane l those of line l, so a
// thread solves a piece of R rows of one line.  Each direction of the Thomas sweep
//
//   forward   y_i = (r_i - a_i y_{i-1}) D_i       backward   x_i = y_i - C_i x_{i+1}
//
// with D = 1/pivot and C = c/pivot (line_coefs in chs_plan.cpp) needs the value entering the piece.  It follows
// from the ends of the pieces before: end of a piece = its end for a sweep from zero + (product of its -a D, or
// -C) times the value entering it, over at most 16 pieces, which each thread runs for itself from shared memory.
// The end for a sweep from zero is a weighted sum of the piece's rows (host tables): no chain, half the products
// of a sweep.  The last row of a periodic line stands outside the Thomas system (its row of factors passes the
// right-hand side through) and closes it as Solve_TDMA_cyclic does (src/basics_algorithms.f90:60-109).
//
// Sweeping the rows from the value that enters, and not correcting rows swept from zero (y_i += P_i y_in), keeps
// the rounding of the plain sweep: the corrected rows, with r1 dd and a D as one constant each, erred by up to
// 1.34 times as much (CP4 differences at 128 points, 1.74 and 1.28 units of 2^-53; FP32 velocities of a CP6
// channel 4 to 9 % more).
//
// What bounds it: with one thread per line (line_op_kernel) a CTA ran two sweeps of n dependent rows in one warp
// of eight while the others waited, and reached 15 % of the memory rate.  Here every warp sweeps R rows, all R + 3
// input values of a thread are in flight at once, and for y and z lines neither input nor output passes through
// shared memory (32 neighbouring x positions are one 256-byte segment of FP64 at every row); x lines are
// transposed through a shared tile with an odd stride.  Pieces of 8 rows beat 16 (shorter chains, twice the warps):
// FP64 line solves of a substep of the 128x96x128 CP6 channel 479 us (corrected rows 484, of 16 rows 593;
// line_op_kernel 1029), of the Taylor-Green 96^3 box 235 us (239, 322); with FP32 fields 355 and 350 us.
#include <cuda_runtime.h>

#include <stdexcept>

#include "chs_kernels.cuh"
#include "chs_stencil_dev.cuh"

namespace chs {

namespace {

// the factors of one row (line_coefs): d, a | c, x | g, h | m, e
template <typename T>
struct Pair2;
template <>
struct Pair2<double> { using V = double2; };
template <>
struct Pair2<float> { using V = float2; };

template <typename T>
__device__ __forceinline__ typename Pair2<T>::V coef2(const T* __restrict__ tab, int row, int k) {
  return __ldg(reinterpret_cast<const typename Pair2<T>::V*>(tab + (size_t)row * kLineCoefs) + k);
}

template <typename T>
__device__ __forceinline__ T coef1(const T* __restrict__ tab, int row, int k) {
  return __ldg(tab + (size_t)row * kLineCoefs + k);
}

// v[u] = the input expression at the positions at(u), u < N; the modes are switched on once so that the
// loads of all positions are independent
template <typename T, int N, typename FA, typename FS>
__device__ __forceinline__ void load_term(const TermT<T>& t, const FA& at, const FS& set) {
  const T s = T(t.s), c = T(t.c);
  if (t.mode == T_X) {
#pragma unroll
    for (int u = 0; u < N; ++u) set(u, s * t.X[at(u)]);
  } else if (t.mode == T_XY) {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int a = at(u);
      set(u, s * (t.X[a] * t.Y[a]));
    }
  } else if (t.mode == T_XpY) {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int a = at(u);
      set(u, s * (t.X[a] + c * t.Y[a]));
    }
  } else {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int a = at(u);
      set(u, s * (t.X[a] + c * t.Y[a]) * t.Z[a]);
    }
  }
}
template <typename T, int N, typename FA>
__device__ __forceinline__ void load_rows(const LineIOT<T>& io, T (&v)[N], const FA& at) {
  load_term<T, N>(io.t[0], at, [&](int u, T x) { v[u] = x; });
  if (io.t[1].mode != T_NONE) load_term<T, N>(io.t[1], at, [&](int u, T x) { v[u] += x; });
}

// The output mode's store of the values x at the positions at(u) that have(u) holds.  The operands of a
// read-modify-write are loaded before any store; O_FRAC, with three of them, goes four rows at a time.
template <typename T, int R, typename FA, typename FH>
__device__ __forceinline__ void store_rows(const LineIOT<T>& io, const T (&x)[R], const FA& at, const FH& have) {
  const T g = T(io.g);
  if (io.omode == O_STORE && !io.accumulate) {
#pragma unroll
    for (int u = 0; u < R; ++u)
      if (have(u)) io.out[at(u)] = g * x[u];
  } else if (io.omode != O_FRAC) {
    const T* from = io.omode == O_STORE ? io.out : io.onum;
    T o[R];
#pragma unroll
    for (int u = 0; u < R; ++u) o[u] = have(u) ? from[at(u)] : T(0);
#pragma unroll
    for (int u = 0; u < R; ++u)
      if (have(u)) store_out(io, at(u), g, x[u], OutPre<T>{o[u], T(0), T(0)});
  } else {
#pragma unroll
    for (int u0 = 0; u0 < R; u0 += 4) {
      OutPre<T> o[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        o[u] = OutPre<T>{T(0), T(0), T(0)};
        if (have(u0 + u)) o[u] = load_out(io, at(u0 + u));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (have(u0 + u)) store_out(io, at(u0 + u), g, x[u0 + u], o[u]);
    }
  }
}

// CIN: cell input (rows i-2 .. i+1 of M1C2P, D1C2P), else point input (i-1 .. i+2 of M1P2C, D1P2C)
template <typename T, int DIR, bool CIN, int R>
__global__ void __launch_bounds__(kLineWarps * 32, (R == 8 ? 2 : 1))
    line_chunk_kernel(const __grid_constant__ OpPlan P, const __grid_constant__ LineIOT<T> io,
                      const T* __restrict__ tab, int nlines) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5, nt = blockDim.x;
  T* sE = reinterpret_cast<T*>(smem_raw);  // [W][32] ends of the forward pieces
  T* sF = sE + W * 32;                     // [W][32] starts of the backward pieces
  T* sN = sF + W * 32;                     // [2][32] rows n-2 and n-1 of a periodic line
  T* sP = sN + 64;                         // [W] P at the pieces' ends, [W] Q at their starts
  T* sT = sP + 2 * W;                      // x lines: the tile, 32 lines of stride ld
  const int nin = P.nin, nout = P.nout, ld = (nin > nout ? nin : nout) | 1;
  const int L0 = blockIdx.x * 32;
  const bool ok = L0 + lane < nlines;
  const int L = ok ? L0 + lane : nlines - 1;  // lanes past the end repeat the last line and store nothing
  const int i0 = w * R;
  constexpr int kLo = CIN ? -2 : -1, N = R + 3;
  // pieces whose window leaves the line or that hold a boundary row, a row past the end or one of the
  // last two rows of a periodic line
  const bool edge = i0 + kLo < 0 || i0 + kLo + N > nin || i0 < P.b_lo || i0 + R - 1 > P.b_hi || i0 + R > nout - 2;
  if (threadIdx.x < W) {
    sP[threadIdx.x] = coef1(tab, threadIdx.x * R + R - 1, 7);
    sP[W + threadIdx.x] = coef1(tab, threadIdx.x * R, 7);
  }

  int base = 0, obase = 0, ps = 1;  // first value of the line in the input and output, row stride
  if (DIR == 1) {
    const int k = L / io.n1, i = L - k * io.n1;
    base = k * nin * io.n1 + i;
    obase = k * nout * io.n1 + i;
    ps = io.n1;
  } else if (DIR == 2) {
    base = obase = L;
    ps = io.n1 * io.n2;
  }
  // row of window position u: wrapped, or clamped (a clamped value reaches no bulk row)
  auto rowq = [&](int u) {
    int q = i0 + kLo + u;
    if (P.lwrap) {
      q = q < 0 ? q + nin : q;
      q = q >= nin ? q - nin : q;  // rows past the end of a short last piece run further: clamped below
    }
    return q < 0 ? 0 : (q >= nin ? nin - 1 : q);
  };

  // ---- the input rows of the piece
  T v[N];
  if (DIR == 0) {
    // 32 rows are one contiguous run of values, R of them per thread (nin <= W * R)
    const int last = min(32, nlines - L0) * nin - 1, g0 = L0 * nin;
    T x[R];
    load_rows<T, R>(io, x, [&](int u) { return g0 + min((int)threadIdx.x + u * nt, last); });
    const int dl = nt / nin, dp = nt - dl * nin;
    int l = threadIdx.x / nin, p = threadIdx.x - l * nin;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      if (l < 32) sT[l * ld + p] = x[u];
      l += dl;
      p += dp;
      if (p >= nin) { p -= nin; ++l; }
    }
    __syncthreads();
    const T* row = sT + lane * ld;
    if (edge) {
#pragma unroll
      for (int u = 0; u < N; ++u) v[u] = row[rowq(u)];
    } else {
#pragma unroll
      for (int u = 0; u < N; ++u) v[u] = row[i0 + kLo + u];
    }
  } else if (edge) {
    load_rows<T, N>(io, v, [&](int u) { return base + rowq(u) * ps; });
  } else {
    const int b0 = base + (i0 + kLo) * ps;
    load_rows<T, N>(io, v, [&](int u) { return b0 + u * ps; });
  }

  // ---- right-hand side
  T x[R];
  {
    const T r1 = T(P.r1), r2 = T(P.r2), dd = T(P.dd), sg = T(P.sgn);
#pragma unroll
    for (int u = 0; u < R; ++u)  // row i0 + u; v[u] is row i0 + kLo + u
      x[u] = (CIN ? r1 * (v[u + 2] + sg * v[u + 1]) + r2 * (v[u + 3] + sg * v[u])
                  : r1 * (sg * v[u + 1] + v[u + 2]) + r2 * (sg * v[u] + v[u + 3])) * dd;
  }
  if (edge && !P.lwrap) {
    // boundary rows of a line with ends, at most four
    for (int k = 0; k < P.nspec; ++k) {
      const SpecialRow& S = P.sp[k];
      if (S.row < i0 || S.row >= i0 + R || (S.row >= P.b_lo && S.row <= P.b_hi)) continue;
      T s = T(0);
      for (int t = 0; t < S.nt; ++t)
        s += T(S.w[t]) * (DIR == 0 ? sT[lane * ld + S.idx[t]] : eval_expr32(io, base + S.idx[t] * ps));
      for (int u = 0; u < 4; ++u)
        if (S.wb[u] != 0.0) s += T(S.wb[u]) * io.fbc[u * nlines + L];
      s *= T(P.dd);
#pragma unroll
      for (int u = 0; u < R; ++u)
        if (S.row == i0 + u) x[u] = s;
    }
  }
  // ---- end of the forward piece
  {
    // the row that weighs most last, so that the sums before it round finer
    T e[2] = {T(0), T(0)};
#pragma unroll
    for (int u = 0; u < R - 1; ++u) e[u & 1] += coef1(tab, i0 + u, 4) * x[u];
    sE[w * 32 + lane] = coef1(tab, i0 + R - 1, 4) * x[R - 1] + (e[0] + e[1]);
  }
  __syncthreads();
  // ---- forward sweep from the joined value, start of the backward piece
  {
    T y = T(0);
#pragma unroll 4
    for (int m = 0; m < w; ++m) y = sE[m * 32 + lane] + sP[m] * y;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const auto da = coef2(tab, i0 + u, 0);
      y = (x[u] - da.y * y) * da.x;
      x[u] = y;
    }
    if (edge && P.tdma == 2) {
#pragma unroll
      for (int u = 0; u < R; ++u) {
        if (i0 + u == nout - 2) sN[lane] = x[u];
        if (i0 + u == nout - 1) sN[32 + lane] = x[u];
      }
    }
    T f[2] = {T(0), T(0)};
#pragma unroll
    for (int u = R - 1; u > 0; --u) f[u & 1] += coef1(tab, i0 + u, 5) * x[u];
    sF[w * 32 + lane] = x[0] + (f[0] + f[1]);
  }
  __syncthreads();
  // ---- backward sweep from the joined value, cyclic closure, metric and wall slopes
  {
    const T* sQ = sP + W;
    T z = T(0);
#pragma unroll 4
    for (int m = W - 1; m > w; --m) z = sF[m * 32 + lane] + sQ[m] * z;
    T xn = T(0);
    if (P.tdma == 2) {
      T x0 = z;
#pragma unroll 4
      for (int m = w; m >= 0; --m) x0 = sF[m * 32 + lane] + sQ[m] * x0;
      xn = (sN[32 + lane] - T(P.cn) * x0 - T(P.an) * sN[lane]) * T(P.inv_den);
    }
#pragma unroll
    for (int u = R - 1; u >= 0; --u) {
      z = x[u] - coef1(tab, i0 + u, 2) * z;
      x[u] = z;
    }
    if (P.tdma == 2) {
#pragma unroll
      for (int u = 0; u < R; ++u) x[u] += coef1(tab, i0 + u, 3) * xn;
    }
    if (edge && P.tdma == 2) {
#pragma unroll
      for (int u = 0; u < R; ++u)
        if (i0 + u == nout - 1) x[u] = xn;
    }
    if (P.lmap >= 0) {
#pragma unroll
      for (int u = 0; u < R; ++u) x[u] *= coef1(tab, i0 + u, 6);
    }
    if (edge && (P.neu1 || P.neu2)) {
#pragma unroll
      for (int u = 0; u < R; ++u) {
        if (P.neu1 && i0 + u == 0) x[u] = io.fbc[L];
        if (P.neu2 && i0 + u == nout - 1) x[u] = io.fbc[nlines + L];
      }
    }
  }
  // ---- store
  if (DIR == 0) {
    // every warp has read its window: two barriers ago
#pragma unroll
    for (int u = 0; u < R; ++u)
      if (i0 + u < nout) sT[lane * ld + i0 + u] = x[u];
    __syncthreads();
    const int tot = min(32, nlines - L0) * nout, g0 = L0 * nout + threadIdx.x;
    const int dl = nt / nout, dp = nt - dl * nout;
    int l = threadIdx.x / nout, p = threadIdx.x - l * nout;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      x[u] = sT[(l < 32 ? l : 31) * ld + p];
      l += dl;
      p += dp;
      if (p >= nout) { p -= nout; ++l; }
    }
    store_rows<T, R>(io, x, [&](int u) { return g0 + u * nt; },
                     [&](int u) { return (int)threadIdx.x + u * nt < tot; });
  } else if (edge) {
    store_rows<T, R>(io, x, [&](int u) { return obase + (i0 + u) * ps; },
                     [&](int u) { return ok && i0 + u < nout; });
  } else if (ok) {
    const int b0 = obase + i0 * ps;
    store_rows<T, R>(io, x, [&](int u) { return b0 + u * ps; }, [](int) { return true; });
  }
}

template <typename T, int DIR, bool CIN, int R>
void launch_chunk(const OpPlan& P, const LineIOT<T>& io, const T* tab, cudaStream_t st, int nlines) {
  const int nmax = P.nin > P.nout ? P.nin : P.nout;
  const int W = (nmax + R - 1) / R;
  size_t shm = (size_t)(2 * W * 32 + 64 + 2 * W) * sizeof(T);
  if (DIR == 0) shm += (size_t)32 * (nmax | 1) * sizeof(T);
  allow_smem<line_chunk_kernel<T, DIR, CIN, R>>(shm);
  line_chunk_kernel<T, DIR, CIN, R><<<(nlines + 31) / 32, W * 32, shm, st>>>(P, io, tab, nlines);
}

template <typename T, int DIR>
void launch_chunk_dir(const OpPlan& P, const LineIOT<T>& io, const T* tab, cudaStream_t st, int nlines) {
  const bool cin = fam_c_input(P.fam);
#define CHS_R(RR)                                                     \
  case RR:                                                            \
    if (cin) launch_chunk<T, DIR, true, RR>(P, io, tab, st, nlines);  \
    else launch_chunk<T, DIR, false, RR>(P, io, tab, st, nlines);     \
    break;
  switch (P.lrows) {
    CHS_R(8)
    CHS_R(16)
    CHS_R(24)
    default: throw std::runtime_error("line operator: bad piece length");
  }
#undef CHS_R
}

}  // namespace

template <typename T>
void launch_line_chunk(int d, const OpPlan& P, const LineIOT<T>& io, const double* table, cudaStream_t st,
                       int nlines) {
  const T* tab = sizeof(T) == 8 ? reinterpret_cast<const T*>(table + P.lcoef)
                                : reinterpret_cast<const T*>(table + P.lcoef32);
  if (d == 0) launch_chunk_dir<T, 0>(P, io, tab, st, nlines);
  else if (d == 1) launch_chunk_dir<T, 1>(P, io, tab, st, nlines);
  else launch_chunk_dir<T, 2>(P, io, tab, st, nlines);
}
template void launch_line_chunk<double>(int, const OpPlan&, const LineIOT<double>&, const double*, cudaStream_t, int);
template void launch_line_chunk<float>(int, const OpPlan&, const LineIOT<float>&, const double*, cudaStream_t, int);

}  // namespace chs

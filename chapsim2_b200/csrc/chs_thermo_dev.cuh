// Device-side property lookups of the variable-property path (table interpolation of
// src/input_thermo.f90:345-446), shared by the property-update and MLP kernels.
#pragma once
#include "chs_kernels.cuh"

namespace chs {

// Rows of the tables hold the node, the values there and their slopes to the next row, so that a lookup reads one
// row after its search and interpolates without a division (value + slope (x - node)); with single columns a
// cell took 27 gathers and four FP64 divisions, which bound the update:
// all elementwise work of a 384x256x384 mixed substep 941 -> 786 us with the rows.

// a bracket (i, i + 1) of a table with rows of S pairs: the node and first value of row i
struct Bracket {
  int i;
  double x, y;
};
// bisection with the reference's sign test ((col[i1]-x)*(col[im]-x) > MINP moves i1) from the
// state (a, b); at most log2(b - a) iterations
template <int S>
__device__ __forceinline__ Bracket tab_bracket_from(const double2* __restrict__ tab, int a, int b, double x) {
  double2 pa = __ldg(tab + a * S);
  while (b - a > 1) {
    const int m = a + (b - a) / 2;
    const double2 pm = __ldg(tab + m * S);
    if ((pa.x - x) * (pm.x - x) > 1.0e-20) {
      a = m;
      pa = pm;
    } else {
      b = m;
    }
  }
  return Bracket{a, pa.x, pa.y};
}
// the search started from the bracket index of column c (0: rho*h, 1: h) when x lies in the indexed
// range, else from (0, n-1): the same path either way
template <int S>
__device__ __forceinline__ Bracket tab_bracket_ix(const ThermoTab& tb, int c, const double2* __restrict__ tab,
                                                  double x) {
  int a = 0, b = tb.n - 1;
  if (tb.ix[c] && x >= tb.ix_lo[c] && x <= tb.ix_hi[c]) {
    int bi = (int)((x - tb.ix_lo[c]) * tb.ix_iw[c]);
    bi = bi < tb.ix_nb - 1 ? bi : tb.ix_nb - 1;
    const int2 s = __ldg(tb.ix[c] + bi);
    a = s.x;
    b = s.y;
  }
  return tab_bracket_from<S>(tab, a, b, x);
}

// the row of a single column's bracket (the surrogate's row on a table of uneven T)
__device__ __forceinline__ int tab_row(const double* __restrict__ col, int n, double x) {
  int a = 0, b = n - 1;
  while (b - a > 1) {
    const int m = a + (b - a) / 2;
    if ((__ldg(col + a) - x) * (__ldg(col + m) - x) > 1.0e-20) a = m;
    else b = m;
  }
  return a;
}

// Search of a strictly increasing column started near row r: bisection from (r - w, r + w + 1)
// when that range holds x.  Where x lies more than kBracketMargin from both ends of the bracket
// found, every node of the column is that far from x, so each sign test of the full search
// ((col[a]-x)*(col[m]-x) > 1e-20) takes the ordinary bisection branch and the full search ends in
// the same bracket: the result is then exactly the full search's.  false: not verified (the
// caller runs the full search).
constexpr double kBracketMargin = 2.0e-10;
template <int S>
__device__ __forceinline__ bool tab_bracket_near(const double2* __restrict__ tab, int n, int r, int w, double x,
                                                 Bracket& k) {
  int a = r - w, b = r + w + 1;
  if (a < 0) a = 0;
  if (b > n - 1) b = n - 1;
  if (a >= b || !(__ldg(tab + a * S).x < x && x < __ldg(tab + b * S).x)) return false;
  k = tab_bracket_from<S>(tab, a, b, x);
  return (x - k.x) > kBracketMargin && (__ldg(tab + (k.i + 1) * S).x - x) > kBracketMargin;
}

struct CellProps {
  double h, t, k, d, m;
};

// Property lookup from rho*h (ftp_refresh_thermal_properties_from_DH): rho*h -> h0 on the rho*h
// column, h0 -> rho0 on the h column, h = rho*h/rho0, h -> properties on the h column.  hint >= 0:
// a predicted row of the rho*h bracket (e.g. from the surrogate network's T), tried within
// +-win rows; *hit tells whether it was verified
// (the h-column searches start from the bracket index).  Every path returns the full search's
// result.
__device__ __forceinline__ CellProps props_from_dh(const ThermoTab& tb, double rhoh, int hint = -1, int win = 0,
                                                   bool* hit = nullptr) {
  if (rhoh < tb.dhmin) rhoh = tb.dhmin;
  else if (rhoh > tb.dhmax) rhoh = tb.dhmax;
  Bracket k{};
  const bool near = hint >= 0 && tab_bracket_near<2>(tb.rh, tb.n, hint, win, rhoh, k);
  if (hit) *hit = near;
  if (!near) k = tab_bracket_ix<2>(tb, 0, tb.rh, rhoh);
  const double h0 = k.y + __ldg(tb.rh + k.i * 2 + 1).x * (rhoh - k.x);
  k = tab_bracket_ix<5>(tb, 1, tb.hp, h0);
  const double d0 = k.y + __ldg(tb.hp + k.i * 5 + 1).x * (h0 - k.x);
  CellProps p;
  p.h = rhoh / d0;
  k = tab_bracket_ix<5>(tb, 1, tb.hp, p.h);
  const double2* row = tb.hp + k.i * 5;  // (h, rho) (rho', mu) (mu', kappa) (kappa', T) (T', 0)
  const double2 r1 = __ldg(row + 1), r2 = __ldg(row + 2), r3 = __ldg(row + 3);
  const double dx = p.h - k.x;
  p.d = k.y + r1.x * dx;
  p.m = r1.y + r2.x * dx;
  p.k = r2.y + r3.x * dx;
  p.t = r3.y + __ldg(row + 4).x * dx;
  return p;
}


}  // namespace chs

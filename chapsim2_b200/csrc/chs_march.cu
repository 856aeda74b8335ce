// All three momentum components of a CD2 substep in one pass that marches along z (see FzMarch in
// chs_fused.cuh for the equations' form and what the host has checked).
//
// A CTA owns 32 x kTY columns (x, y) and a run of z planes.  Every plane of the inputs it needs (its
// columns, one more to each side, 16-byte aligned) is copied to shared memory by cp.async one plane
// ahead of its use, in a ring of three sets.  Each of the nine stresses -- three at the cell centre, two
// at each of the three edges -- is formed once per cell: the z differences are taken between
// successive planes in registers, the x and y differences through a shared exchange of the six
// stresses that a neighbour needs, for which one extra warp forms the row beyond the tile's y ends and
// another the columns beyond its x ends.
//
// What bounded the pass it replaces (fz_momentum_kernel, a thread per output and component): every
// stress was formed by each output that reads it, 18 evaluations and about 80 loads per cell and
// component through L1 at 64 registers, 22-34 % of the memory rate.  Here a cell's inputs are loaded
// once (1.4x with the halo), and the history and output streams are the only other traffic.  Per substep, the
// three components then and the march now: 128x96x128 heated FP64 150 and 64 us, 384x256x384 heated FP32 2700 and
// 837 us (3.1 TB/s).  FP64 runs 20 warps per SM (96 registers) and waits between the two barriers of a plane: 47 % of the
// issue slots, 56 % of the shared-memory wavefronts, 34 % of the memory rate at 128x96x128.  FP32 runs 30 and fills 66 %
// of the issue slots at the same shared-memory share.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>

#include "chs_fused.cuh"

namespace chs {

namespace {

constexpr int kTY = 8;           // output rows of a CTA, one warp each
constexpr int kRows = kTY + 2;   // rows of a set: j0 - 1 .. j0 + kTY
constexpr int kXS = 36;          // columns of a set: i0 - 2 .. i0 + 33
constexpr int kSets = 3;
constexpr int kThreads = (kTY + 2) * 32;
constexpr int kWall = 2 * 4 * kXS;  // wall planes' rows in a set: below, above of qx, qz, momentum, mu

// two values (16 or 8 bytes) from global to shared memory
template <typename T>
__device__ __forceinline__ void copy_pair(T* dst, const T* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (sizeof(T) == 8) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

enum { QX, QY, QZ, PR, GX, GY, GZ, MU };
enum { WQX, WQZ, WG, WMU };

template <typename T>
struct Exchange {
  T xx[kTY][33];      // normal x stress, columns i0 - 1 .. i0 + 31
  T xy1[kTY][33];     // xy stress of the y component, columns i0 .. i0 + 32
  T xz2[kTY][33];     // xz stress of the z component, columns i0 .. i0 + 32
  T xy0[kTY + 1][32]; // xy stress of the x component, rows j0 .. j0 + kTY
  T yz2[kTY + 1][32]; // yz stress of the z component, rows j0 .. j0 + kTY
  T yy[kTY + 1][32];  // normal y stress, rows j0 - 1 .. j0 + kTY - 1
  double red[kTY];
};

template <typename T, bool TH>
struct MarchSize {
  static constexpr int fields = TH ? 8 : 4;
  static constexpr int pairs = fields * kRows * (kXS / 2);             // pair copies of a set
  static constexpr int copies = (pairs + kThreads - 1) / kThreads;     // per thread
  static constexpr int set = fields * kRows * kXS + kWall;             // values of a set
  static constexpr size_t smem = (size_t)kSets * set * sizeof(T) + (size_t)copies * kThreads * 8 + sizeof(Exchange<T>);
};

template <typename T, bool TH, bool PY>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 8 ? 2 : 3)
    fz_march_kernel(const __grid_constant__ FzMarch<T> f) {
  using Sz = MarchSize<T, TH>;
  constexpr int kSet = Sz::set, kCopies = Sz::copies, kData = Sz::fields * kRows * kXS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  const T** from = reinterpret_cast<const T**>(ring + kSets * kSet);  // [copies][threads]
  Exchange<T>& ex = *reinterpret_cast<Exchange<T>*>(from + kCopies * kThreads);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n0 = f.n0, ny = f.nc1, np1 = f.np1, n2 = f.n2, nl = n0 * n2;
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * kTY;
  const int k0 = blockIdx.z * f.chunk, k1 = min(k0 + f.chunk, n2);
  auto wrapk = [&](int k) { return k < 0 ? k + n2 : (k >= n2 ? k - n2 : k); };

  // ---- this thread's share of a set: copy u is pair threadIdx.x + u * kThreads of the set, from plane 0's
  // address in `from` (its own slots only) and, by the two bits of `kinds`, the plane offset of a
  // cell-centred array (0), of y points (1; ny + 1 rows with walls) or of z points (2; plane k + 1)
  unsigned kinds = 0;
#pragma unroll
  for (int u = 0; u < kCopies; ++u) {
    const int e = threadIdx.x + u * kThreads;
    if (e >= Sz::pairs) continue;
    const int fld = e / (kRows * (kXS / 2)), r = e / (kXS / 2) % kRows, c = e % (kXS / 2) * 2;
    const bool pts = fld == QY || fld == GY;
    int i = i0 - 2 + c, j = j0 - 1 + r;
    i = ((i % n0) + n0) % n0;
    j = PY ? ((j % ny) + ny) % ny : min(max(j, 0), (pts ? np1 : ny) - 1);
    from[u * kThreads + threadIdx.x] = f.a[fld] + (j * n0 + i);
    kinds |= (pts ? 1u : (fld == QZ || fld == GZ) ? 2u : 0u) << (2 * u);
  }
  // wall rows: the pair this thread copies (threads 0 .. 143; null: none)
  const T* wall_from = nullptr;
  if (!PY && threadIdx.x < kWall / 2) {
    const int sd = threadIdx.x / (kWall / 4), q = threadIdx.x / (kXS / 2) % 4, c = threadIdx.x % (kXS / 2) * 2;
    const T* b = q == WQX ? f.bqx : (q == WQZ ? f.bqz : (q == WG ? f.bg : f.bmu));
    const bool has = sd == 0 ? j0 == 0 : j0 + kTY >= ny;
    int i = i0 - 2 + c;
    i = ((i % n0) + n0) % n0;
    if (has && (TH || q < WG)) wall_from = b + sd * nl + i;
  }
  auto load_set = [&](int k, T* set, bool z_only) {
    const int kw = wrapk(k), kz = wrapk(k + 1);
    const int off_c = kw * ny * n0, off_y = kw * np1 * n0, off_z = kz * ny * n0;
#pragma unroll
    for (int u = 0; u < kCopies; ++u) {
      const int e = threadIdx.x + u * kThreads;
      if (e < Sz::pairs) {
        const unsigned kind = kinds >> (2 * u) & 3u;
        if (kind == 2u || !z_only)
          copy_pair(set + 2 * e,
                    from[u * kThreads + threadIdx.x] + (kind == 0u ? off_c : (kind == 1u ? off_y : off_z)));
      }
    }
    if (wall_from && !z_only) copy_pair(set + kData + 2 * threadIdx.x, wall_from + kw * n0);
  };

  const T third = T(1.0 / 3.0), dxi = T(f.dxi), dzi = T(f.dzi), rre = T(f.rre), rre2 = T(2.0 * f.rre);
  const T quarter = T(0.25), rre4 = T(0.25 * f.rre);
  // y weights of row j (cells) and edge j (points)
  auto wcell = [&](int j) { return T(f.wc[PY ? (j + ny) % ny : min(max(j, 0), ny - 1)]); };
  auto wedge = [&](int j) { return T(f.wp[PY ? (j + ny) % ny : min(max(j, 0), np1 - 1)]); };
#define V(S, F, R, C) (S)[((F) * kRows + (R)) * kXS + (C)]

  // ---- the stresses.  A: the set of plane k (qz, gz: k + 1), B: of k - 1 (qz, gz: k); set row r, column c.
  // Interpolated factors enter as sums of two or four values, their halves in one constant.
  // normal stress a of (xx, yy, zz) at the cell centre
  auto normal = [&](const T* A, const T* B, int r, int c, T wc, int a) -> T {
    const T qx0 = V(A, QX, r, c), qx1 = V(A, QX, r, c + 1), qy0 = V(A, QY, r, c), qy1 = V(A, QY, r + 1, c);
    const T qz0 = V(B, QZ, r, c), qz1 = V(A, QZ, r, c);
    const T dx = dxi * (qx1 - qx0), dy = wc * (qy1 - qy0), dz = dzi * (qz1 - qz0);
    const T d = a == 0 ? dx : (a == 1 ? dy : dz);
    T v = rre2 * (d - third * (dx + dy + dz));
    if (TH) v *= V(A, MU, r, c);
    const T q = a == 0 ? qx0 + qx1 : (a == 1 ? qy0 + qy1 : qz0 + qz1);
    T m = q;
    if (TH)
      m = a == 0 ? V(A, GX, r, c) + V(A, GX, r, c + 1)
                 : (a == 1 ? V(A, GY, r, c) + V(A, GY, r + 1, c) : V(B, GZ, r, c) + V(A, GZ, r, c));
    return v - quarter * m * q;
  };
  // rows r and r - 1 of a y-cell array at edge r; beyond a wall (side 1 below, 2 above) the value that
  // puts the wall's (row q of the wall rows of set Wl) in the middle
  auto ypair = [&](const T* S, int fld, int r, int c, const T* Wl, int q, int side, T& hi, T& lo) {
    hi = V(S, fld, r, c);
    lo = V(S, fld, r - 1, c);
    if (!PY && side) {
      const T b = Wl[kData + ((side - 1) * 4 + q) * kXS + c];
      if (side == 1) lo = T(2) * b - hi;
      else hi = T(2) * b - lo;
    }
  };
  // xy edge: the x component's stress e0 and the y component's e1
  auto edge_xy = [&](const T* A, int r, int c, T wp, int side, T& e0, T& e1) {
    T qh, ql;
    ypair(A, QX, r, c, A, WQX, side, qh, ql);
    const T qyr = V(A, QY, r, c), qyl = V(A, QY, r, c - 1), qxs = qh + ql, qys = qyr + qyl;
    T v = wp * (qh - ql) + dxi * (qyr - qyl), m0 = qys, m1 = qxs;
    if (TH) {
      T mh, ml, nh, nlo, gh, gl;
      ypair(A, MU, r, c, A, WMU, side, mh, ml);
      ypair(A, MU, r, c - 1, A, WMU, side, nh, nlo);
      v *= rre4 * ((mh + ml) + (nh + nlo));
      ypair(A, GX, r, c, A, WG, side, gh, gl);
      m0 = V(A, GY, r, c) + V(A, GY, r, c - 1);
      m1 = gh + gl;
    } else {
      v *= rre;
    }
    e0 = v - quarter * m0 * qxs;
    e1 = v - quarter * m1 * qys;
  };
  // xz edge: of the x component (e0) and the z component (e2)
  auto edge_xz = [&](const T* A, const T* B, int r, int c, T& e0, T& e2) {
    const T xa = V(A, QX, r, c), xb = V(B, QX, r, c), zr = V(B, QZ, r, c), zl = V(B, QZ, r, c - 1);
    const T qxs = xa + xb, qzs = zr + zl;
    T v = dzi * (xa - xb) + dxi * (zr - zl), m0 = qzs, m2 = qxs;
    if (TH) {
      v *= rre4 * ((V(A, MU, r, c) + V(A, MU, r, c - 1)) + (V(B, MU, r, c) + V(B, MU, r, c - 1)));
      m0 = V(B, GZ, r, c) + V(B, GZ, r, c - 1);
      m2 = V(A, GX, r, c) + V(B, GX, r, c);
    } else {
      v *= rre;
    }
    e0 = v - quarter * m0 * qxs;
    e2 = v - quarter * m2 * qzs;
  };
  // yz edge: of the y component (e1) and the z component (e2)
  auto edge_yz = [&](const T* A, const T* B, int r, int c, T wp, int side, T& e1, T& e2) {
    T zh, zl;
    ypair(B, QZ, r, c, A, WQZ, side, zh, zl);
    const T ya = V(A, QY, r, c), yb = V(B, QY, r, c), qys = ya + yb, qzs = zh + zl;
    T v = wp * (zh - zl) + dzi * (ya - yb), m1 = qzs, m2 = qys;
    if (TH) {
      T mh, ml, nh, nlo, gh, gl;
      ypair(A, MU, r, c, A, WMU, side, mh, ml);
      ypair(B, MU, r, c, B, WMU, side, nh, nlo);
      v *= rre4 * ((mh + ml) + (nh + nlo));
      ypair(B, GZ, r, c, A, WG, side, gh, gl);
      m1 = gh + gl;
      m2 = V(A, GY, r, c) + V(B, GY, r, c);
    } else {
      v *= rre;
    }
    e1 = v - quarter * m1 * qys;
    e2 = v - quarter * m2 * qzs;
  };
  auto side_of = [&](int j) { return PY ? 0 : (j == 0 ? 1 : (j == ny ? 2 : 0)); };

  // ---- the march: plane k0 - 1 gives the normal z stress below the first plane, plane k1 the x and y
  // components' z edges above the last
  const bool outw = w < kTY;
  const int i = i0 + lane, j = j0 + w, r = w + 1, c = lane + 2;
  const bool valid = outw && i < n0 && j < ny;
  const bool yval = valid && (PY || j > 0);  // wall rows of the y component: fz_wall_rows_kernel
  // the row whose weights the warp's stresses take: its own, the tile's outer rows (normal stress below,
  // edges above), or one row per eight lanes
  const int jh = j0 + (lane & 7);
  const T wc = wcell(outw ? j : (w == kTY ? j0 - 1 : jh)), wp = wedge(outw ? j : (w == kTY ? j0 + kTY : jh));
  const int side = side_of(outw ? j : (w == kTY ? j0 + kTY : jh));
  const T dt = T(f.dt), gam = T(f.gam), zeta = T(f.zeta), alpha = T(f.alpha);
  T zz = T(0), xz0 = T(0), yz1 = T(0);    // of the previous plane
  T fx = T(0), fy = T(0), ax = T(0), ay = T(0), ux = T(0), uy = T(0);  // pending x and y components
  double msum = 0.0;
  const double wy = (valid && f.part) ? f.wy[j] : 0.0;

  load_set(k0 - 2, ring, true);
  load_set(k0 - 1, ring + kSet, false);
  copy_commit();
  int sb = 0, sa = 1;  // sets of planes k - 1 and k
  for (int k = k0 - 1; k <= k1; ++k) {
    copy_wait();
    __syncthreads();  // the set of plane k has arrived; every warp is past plane k - 1
    const int sn = sa == 2 ? 0 : sa + 1;
    if (k < k1) {
      load_set(k + 1, ring + sn * kSet, false);
      copy_commit();
    }
    const T *A = ring + sa * kSet, *B = ring + sb * kSet;
    const bool inner = k >= k0 && k < k1;
    T nzz = T(0), nxz0 = T(0), nyz1 = T(0), xx = T(0), yy = T(0), xy0 = T(0), xy1 = T(0), xz2 = T(0), yz2 = T(0);
    T lx = T(0), ly = T(0), lz = T(0);  // histories of plane k, in flight while the stresses are formed
    const int ac = (k * ny + j) * n0 + i, ap = (k * np1 + j) * n0 + i;
    if (inner && valid) {
      lx = f.m0[0][ac];
      lz = f.m0[2][ac];
      if (yval) ly = f.m0[1][ap];
    }
    if (outw) {
      if (k < k1) nzz = normal(A, B, r, c, wc, 2);
      if (k >= k0) {
        edge_xz(A, B, r, c, nxz0, xz2);
        edge_yz(A, B, r, c, wp, side, nyz1, yz2);
      }
      if (inner) {
        xx = normal(A, B, r, c, wc, 0);
        yy = normal(A, B, r, c, wc, 1);
        edge_xy(A, r, c, wp, side, xy0, xy1);
        ex.xx[w][lane + 1] = xx;
        ex.xy1[w][lane] = xy1;
        ex.xz2[w][lane] = xz2;
        ex.xy0[w][lane] = xy0;
        ex.yz2[w][lane] = yz2;
        ex.yy[w + 1][lane] = yy;
      }
    } else if (inner) {
      T t0, t1;
      if (w == kTY) {
        // the rows beyond the tile
        ex.yy[0][lane] = normal(A, B, 0, c, wc, 1);
        edge_xy(A, kTY + 1, c, wp, side, t0, t1);
        ex.xy0[kTY][lane] = t0;
        edge_yz(A, B, kTY + 1, c, wp, side, t0, t1);
        ex.yz2[kTY][lane] = t1;
      } else {
        // the columns beyond the tile: 8 lanes per stress, one row each
        const int q = lane & 7;
        if (lane < 8) {
          ex.xx[q][0] = normal(A, B, q + 1, 1, wc, 0);
        } else if (lane < 16) {
          edge_xy(A, q + 1, 34, wp, side, t0, t1);
          ex.xy1[q][32] = t1;
        } else if (lane < 24) {
          edge_xz(A, B, q + 1, 34, t0, t1);
          ex.xz2[q][32] = t1;
        }
      }
    }
    if (k > k0 && valid) {
      // x and y components of plane k - 1: their upper z edges are known now
      const int bc = ac - ny * n0, bp = ap - np1 * n0;
      T F = fx + dzi * (nxz0 - xz0);
      T m = dt * (gam * F + ax);
      f.m0[0][bc] = F;
      f.out[0][bc] = f.adv & 1 ? ux + m : m;
      if (f.part) msum += wy * (double)m;
      if (yval) {
        F = fy + dzi * (nyz1 - yz1);
        m = dt * (gam * F + ay);
        f.m0[1][bp] = F;
        f.out[1][bp] = f.adv & 2 ? uy + m : m;
      }
    }
    if (inner) {
      __syncthreads();  // the exchange is complete
      if (valid) {
        const T p0 = V(A, PR, r, c);
        fx = dxi * (xx - ex.xx[w][lane]) + wc * (ex.xy0[w + 1][lane] - xy0);
        fy = dxi * (ex.xy1[w][lane + 1] - xy1) + wp * (yy - ex.yy[w][lane]);
        ax = zeta * lx - alpha * (dxi * (p0 - V(A, PR, r, c - 1)));
        ay = zeta * ly - alpha * (wp * (p0 - V(A, PR, r - 1, c)));
        ux = V(A, TH ? GX : QX, r, c);
        uy = V(A, TH ? GY : QY, r, c);
        const T F = dxi * (ex.xz2[w][lane + 1] - xz2) + wc * (ex.yz2[w + 1][lane] - yz2) + dzi * (nzz - zz);
        const T m = dt * (gam * F + zeta * lz - alpha * (dzi * (p0 - V(B, PR, r, c))));
        f.m0[2][ac] = F;
        f.out[2][ac] = f.adv & 4 ? V(B, TH ? GZ : QZ, r, c) + m : m;
      }
    }
    zz = nzz;
    xz0 = nxz0;
    yz1 = nyz1;
    sb = sa;
    sa = sn;
  }
#undef V

  if (f.part) {
    // the mass-flux mean: per-CTA sums in a fixed order, added up in index order by the CTA that
    // finishes last (the counter is back at zero afterwards)
    for (int o = 16; o > 0; o >>= 1) msum += __shfl_down_sync(0xffffffffu, msum, o);
    if (outw && lane == 0) ex.red[w] = msum;
    __syncthreads();
    __shared__ bool is_last;
    __shared__ double acc[256];
    const int nblk = gridDim.x * gridDim.y * gridDim.z;
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int q = 0; q < kTY; ++q) t += ex.red[q];
      f.part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = t;
      __threadfence();
      is_last = atomicAdd(f.count, 1u) == (unsigned)nblk - 1u;
    }
    __syncthreads();
    if (is_last) {
      __threadfence();
      if (threadIdx.x < 256) {
        double t = 0.0;
        for (int q = threadIdx.x; q < nblk; q += 256) t += __ldcg(f.part + q);
        acc[threadIdx.x] = t;
      }
      __syncthreads();
      for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) acc[threadIdx.x] += acc[threadIdx.x + h];
        __syncthreads();
      }
      if (threadIdx.x == 0) {
        f.bulk[0] = acc[0] / f.vol;
        *f.count = 0u;
      }
    }
  }
}

template <typename T, bool TH, bool PY>
dim3 march_grid(int n0, int ny, int n2, int& chunk) {
  // z runs so that the CTAs fill whole rounds of the SMs: the cost of a split is its rounds times the
  // planes of a run, each run paying two planes more than it owns
  int occ = 1;
  cudaFuncSetAttribute(fz_march_kernel<T, TH, PY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)MarchSize<T, TH>::smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fz_march_kernel<T, TH, PY>, kThreads, MarchSize<T, TH>::smem);
  const int64_t tiles = (int64_t)((n0 + 31) / 32) * ((ny + kTY - 1) / kTY), slots = 148 * (int64_t)std::max(occ, 1);
  double best = 1e300;
  chunk = n2;
  for (int q = 1; q <= n2; ++q) {
    const int runs = (n2 + q - 1) / q;
    const double cost = (double)((tiles * runs + slots - 1) / slots) * (q + 2.0);
    if (cost < best) {
      best = cost;
      chunk = q;
    }
  }
  return dim3((n0 + 31) / 32, (ny + kTY - 1) / kTY, (n2 + chunk - 1) / chunk);
}

template <typename T, bool TH, bool PY>
void launch_march_t(FzMarch<T> f, cudaStream_t st) {
  const dim3 grid = march_grid<T, TH, PY>(f.n0, f.nc1, f.n2, f.chunk);
  fz_march_kernel<T, TH, PY><<<grid, kThreads, MarchSize<T, TH>::smem, st>>>(f);
}

}  // namespace

int fz_march_blocks_max(int n0, int ny, int n2) { return ((n0 + 31) / 32) * ((ny + kTY - 1) / kTY) * n2; }

template <typename T>
void launch_fz_march(const FzMarch<T>& f, bool thermo, bool periodic_y, cudaStream_t st) {
  if (thermo && periodic_y) throw std::invalid_argument("momentum march: variable properties need y walls");
  if (thermo) launch_march_t<T, true, false>(f, st);
  else if (periodic_y) launch_march_t<T, false, true>(f, st);
  else launch_march_t<T, false, false>(f, st);
}
template void launch_fz_march<double>(const FzMarch<double>&, bool, bool, cudaStream_t);
template void launch_fz_march<float>(const FzMarch<float>&, bool, bool, cudaStream_t);

}  // namespace chs

// fcm_packed.cu -- the Stokes solve on a packed half spectrum.
//
// A real line of nz points is transformed along z as H = nz/2 complex points (even
// samples the real, odd ones the imaginary parts) and nothing else is done to it:
// its H values Z(kz) hold the line's nz/2 + 1 modes,
//   X(kz) = (Z(kz) + conj Z(H - kz))/2 + W_nz^kz (Z(kz) - conj Z(H - kz))/(2i),
// kz = 0 the two real modes 0 and H.  The transforms along y and x being linear, the
// separation waits until the projection, where it pairs the modes (kx, ky, kz) and
// (-kx, -ky, H - kz); the projected pair is folded back the same way before the
// inverse transforms.  So
//   - the z passes are complex transforms of half the length with one exchange through
//     shared memory (separating and packing two real lines took a second one: those
//     passes had 85% of the shared-memory and L1 wavefronts, 54% of DRAM throughput);
//   - the Hermitian planes kz = 0 and nz/2 are one column of the same kernels (their
//     modes pair as {k, -k} anyway, see the symmetrisation in fcm_kspace.cu) instead
//     of a launch of their own.
//
// Layout: the x transforms hold all x of a few columns of one row, so a layout with kz
// or y running fastest gives them runs of 32 or 64 bytes at a large stride (their load
// and store steps alone ran at 1.6 and 2.7 TB/s).  Here XB x by TKB columns (XB = 4 and
// 32 bytes of columns, XB = 8 and 16 bytes from 256 points along x on) form a 128-byte tile,
//   C spec[3][2 nkb][nx / XB][ny][XB][TKB],
// of which the x transforms take whole tiles, a y transform of a tile column reads and
// writes one contiguous run of 128 ny bytes, and the z passes write whole tiles, XB x of
// a row per CTA.  The columns 0..H/2 - 1 fill the blocks 0..nkb - 1 in order, H/2 the
// first place of block nkb and H - j (0 < j < H/2) place j from there: the two columns of
// a pair lie nkb blocks apart.  Lengths: those of xfft_factor in all three directions.
//
// Measured per solve against the separate passes on nz/2 + 1 columns with cuFFT's 3D or
// (y, z) plans in FP64 (us, FP64 / FP32): 64^3 29 / 20 (43 / 25), 96^3 60 / 35 (101 / 43),
// 128^3 96 / 59 (138 / 84), 256^3 766 / 393 (922 / 474), 384^3 2650 / 1460 (6010 / 1730),
// 512^3 6490 / 3230 (9420 / 3970).  At 512^3 the z and y passes run at 5.5-6.5 TB/s; the x
// pass (FP32 1.04 ms for 3.2 GB, FP64 2.08) is bound by its five steps between barriers.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "fcm_dft.cuh"
#include "fcm_fluct.cuh"
#include "fcm_internal.cuh"

namespace fcm {

namespace {

// Tiled layout of one precision (see above), XB x per tile.
template <typename C, int XB>
struct Tiles {
  static constexpr int TKB = 128 / XB / (int)sizeof(C);  // columns per tile
  static constexpr int TS = XB * TKB;                    // values per tile
  int H, nkb, nxb, ny;
  long long bs;  // values per column block: nxb ny tiles
  __host__ __device__ __forceinline__ Tiles(int nx, int ny_, int nz)
      : H(nz / 2), nkb((nz / 4 + TKB - 1) / TKB), nxb(nx / XB), ny(ny_), bs((long long)(nx / XB) * ny_ * TS) {}
  // values of one grid's spectrum (three components)
  __host__ __device__ __forceinline__ long long size() const { return 6LL * nkb * bs; }
  // offset of column kz within a component, from the first column of the same (x, y)
  __device__ __forceinline__ long long col(int kz) const {
    const bool second = 2 * kz >= H;
    const int j = second ? (2 * kz == H ? 0 : H - kz) : kz;
    return ((second ? nkb : 0) + j / TKB) * bs + j % TKB;
  }
  // first value of (component or member's component mc, x, y)
  __device__ __forceinline__ long long row(long long mc, int x, int y) const {
    return 2 * mc * nkb * bs + ((long long)(x / XB) * ny + y) * TS + (x % XB) * TKB;
  }
};

// x per tile of a grid of nx points: 8 where the x transforms are long, so that their
// CTAs hold half the columns and twice as many fit on an SM (x pass at 512^3: 1.04 against
// 1.15 ms in FP32, 2.08 against 2.30 in FP64; at 256^3 122 against 125 and 218 against
// 258 us), 4 else (32-byte sectors in the z passes).
__host__ __device__ constexpr int tile_x(int nx) { return nx >= 256 ? 8 : 4; }

// Offsets of the columns k = k0 + S j, j < L (S L = H), of one line: two arithmetic
// sequences where S is a whole number of tile columns (the columns below H/2 upwards, the
// others downwards), so a pass adds a stride per value instead of working out each place.
template <typename C, int XB, int S, int L>
struct ColRun {
  static constexpr int TKB = Tiles<C, XB>::TKB;
  static constexpr bool LINEAR = S % TKB == 0 && L % 2 == 0;
  const Tiles<C, XB>& t;
  int k0;
  long long lo, hi, step;
  __device__ __forceinline__ ColRun(const Tiles<C, XB>& tt, int k) : t(tt), k0(k), lo(0), hi(0), step(0) {
    if constexpr (LINEAR) {
      step = (S / TKB) * t.bs;
      lo = t.col(k0);
      // column k0 + S j = H - (r + S (L - 1 - j)), r = S - k0
      const int r = S - k0;
      hi = (t.nkb + r / TKB) * t.bs + r % TKB + (L - 1) * step;
    }
  }
  __device__ __forceinline__ long long at(int j) const {
    if constexpr (!LINEAR) return t.col(k0 + S * j);
    if (2 * j < L) return lo + j * step;
    if (2 * j == L && k0 == 0) return t.nkb * t.bs;  // column H/2
    return hi - j * step;
  }
};

// ------------------------------------------------------------------ z passes
// H-point complex transforms of lines (n = j Z2 + n2 -> k = k1 + Z1 k2): Z1-point DFTs
// from global memory, twiddles, one exchange, Z2-point DFTs to global memory.  Forward:
// the real grid (seen as complex pairs) into the spectrum; inverse the other way.  A CTA
// takes the lines of a tile's x and Q / XB y; the accesses to the spectrum have the
// columns of a tile in consecutive lanes, then the lines, so that a warp covers whole
// tiles (with the columns first, pieces of many tiles, the inverse took 0.66 ms instead
// of 0.49 at 512^3 in FP32).  Lines are PS values apart in shared memory, which spreads
// those lanes over all banks.
template <typename C, int XB, int Z1, int Z2>
constexpr int z_line_stride() {
  constexpr int E = 128 / (int)sizeof(C), W = Tiles<C, XB>::TKB;  // PS = TKB mod 128 bytes
  return Z1 * (Z2 + 1) + ((W - Z1 * (Z2 + 1)) % E + E) % E;
}
// Item i of Q lines by N values: values of a tile column first, then lines, then the rest.
template <int TKB, int Q, int N>
__device__ __forceinline__ void tile_item(int i, int& p, int& n) {
  constexpr int W = N % TKB == 0 ? TKB : 1;
  p = (i / W) % Q;
  n = i % W + W * (i / (W * Q));
}
template <typename T, typename C, int XB, int Z1, int Z2, int NT, bool INV>
__global__ void __launch_bounds__(NT) k_packed_z(C* __restrict__ real, C* __restrict__ spec, Tiles<C, XB> t,
                                                 const C* __restrict__ tw) {
  chain_begin();
  constexpr int H = Z1 * Z2;
  constexpr int ZM = Z1 > Z2 ? Z1 : Z2;
  constexpr int Q = NT / ZM, YQ = Q / XB;  // lines and rows per CTA
  constexpr int PS = z_line_stride<C, XB, Z1, Z2>(), TKB = Tiles<C, XB>::TKB;
  extern __shared__ __align__(16) unsigned char packed_smem[];
  V2<T>* s = reinterpret_cast<V2<T>*>(packed_smem);
  const int nyb = (t.ny + YQ - 1) / YQ;
  const int yb = blockIdx.x % nyb, xc = blockIdx.x / nyb;  // xc: (member, component, XB x)
  const int xb = xc % t.nxb, mc = xc / t.nxb;
  // line p of the CTA: x = XB xb + p % XB, y = yb YQ + p / XB
  auto line_y = [&](int p) { return yb * YQ + p / XB; };
  auto real_line = [&](int p) {
    return real + (((long long)mc * t.nxb * XB + XB * xb + p % XB) * t.ny + line_y(p)) * H;
  };
  auto spec_line = [&](int p) { return spec + t.row(mc, XB * xb + p % XB, line_y(p)); };
  for (int i = threadIdx.x; i < Q * Z2; i += NT) {
    int p = i / Z2, n2 = i % Z2;
    if (INV) tile_item<TKB, Q, Z2>(i, p, n2);
    if (line_y(p) >= t.ny) continue;
    V2<T> a[Z1];
    if constexpr (INV) {
      const C* src = spec_line(p);
      const ColRun<C, XB, Z2, Z1> col(t, n2);
#pragma unroll
      for (int j = 0; j < Z1; ++j) a[j] = ldt<T>(src[col.at(j)]);
    } else {
      const C* src = real_line(p) + n2;
#pragma unroll
      for (int j = 0; j < Z1; ++j) a[j] = ldt<T>(src[j * Z2]);
    }
    dft<T, Z1, INV>(a);
#pragma unroll
    for (int j = 1; j < Z1; ++j) {
      const V2<T> w = ldt<T>(__ldg(&tw[2 * n2 * j]));  // W_H^(n2 j) = W_nz^(2 n2 j)
      a[j] = INV ? cmulc(a[j], w) : cmul(a[j], w);
    }
#pragma unroll
    for (int j = 0; j < Z1; ++j) s[p * PS + j * (Z2 + 1) + n2] = a[j];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < Q * Z1; i += NT) {
    int p = i / Z1, k1 = i % Z1;
    if (!INV) tile_item<TKB, Q, Z1>(i, p, k1);
    if (line_y(p) >= t.ny) continue;
    V2<T> b[Z2];
#pragma unroll
    for (int j = 0; j < Z2; ++j) b[j] = s[p * PS + k1 * (Z2 + 1) + j];
    dft<T, Z2, INV>(b);
    C* dst = INV ? real_line(p) + k1 : spec_line(p);
    const ColRun<C, XB, Z1, Z2> col(t, k1);
#pragma unroll
    for (int j = 0; j < Z2; ++j) {
      C o;
      o.x = b[j].x;
      o.y = b[j].y;
      dst[INV ? (long long)(Z1 * j) : col.at(j)] = o;
    }
  }
}

// ------------------------------------------------------------------ y pass
// Transforms along y in place: one CTA per tile column, XB x times TKB columns at once in
// a contiguous run of 128 ny bytes, the two steps as above.
template <typename T, typename C, int Y1, int Y2, int NT, bool INV>
__global__ void __launch_bounds__(NT) k_packed_y(C* __restrict__ spec, const C* __restrict__ tw) {
  chain_begin();
  constexpr int TK = 128 / (int)sizeof(C);  // values per tile
  extern __shared__ __align__(16) unsigned char packed_smem[];
  V2<T>* s = reinterpret_cast<V2<T>*>(packed_smem);  // [Y1 Y2][TK]
  C* base = spec + (long long)blockIdx.x * (Y1 * Y2 * TK);
  for (int i = threadIdx.x; i < Y2 * TK; i += NT) {
    const int kzl = i % TK, n2 = i / TK;
    V2<T> a[Y1];
#pragma unroll
    for (int j = 0; j < Y1; ++j) a[j] = ldt<T>(base[(j * Y2 + n2) * TK + kzl]);
    dft<T, Y1, INV>(a);
#pragma unroll
    for (int j = 1; j < Y1; ++j) {
      const V2<T> w = ldt<T>(__ldg(&tw[n2 * j]));
      a[j] = INV ? cmulc(a[j], w) : cmul(a[j], w);
    }
#pragma unroll
    for (int j = 0; j < Y1; ++j) s[(j * Y2 + n2) * TK + kzl] = a[j];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < Y1 * TK; i += NT) {
    const int kzl = i % TK, k1 = i / TK;
    V2<T> b[Y2];
#pragma unroll
    for (int j = 0; j < Y2; ++j) b[j] = s[(k1 * Y2 + j) * TK + kzl];
    dft<T, Y2, INV>(b);
#pragma unroll
    for (int j = 0; j < Y2; ++j) {
      C o;
      o.x = b[j].x;
      o.y = b[j].y;
      base[(k1 + Y1 * j) * TK + kzl] = o;
    }
  }
}

// ------------------------------------------------------------------ (y, z) passes, a CTA per plane
// The z and y transforms of one (component, x) plane of ny == nz = 2 Z1 Z2 = Y1 Y2
// points in one pass each way, the plane's spectrum [ny][H] in shared memory (rows
// padded by one value).  In place: the z steps along the rows, the y steps along the
// columns, the first and last step straight from and to global memory.
template <typename T, typename C, int XB, int Z1, int Z2, int Y1, int Y2, int NT, bool INV>
__global__ void __launch_bounds__(NT) k_packed_plane(C* __restrict__ real, C* __restrict__ spec, Tiles<C, XB> t,
                                                     const C* __restrict__ twy, const C* __restrict__ twz) {
  chain_begin();
  constexpr int H = Z1 * Z2, N = Y1 * Y2, RS = H + 1;
  extern __shared__ __align__(16) unsigned char packed_smem[];
  V2<T>* s = reinterpret_cast<V2<T>*>(packed_smem);
  C* plane = real + (long long)blockIdx.x * N * H;
  const int nx = XB * t.nxb;
  C* sp = spec + t.row(blockIdx.x / nx, blockIdx.x % nx, 0);
  constexpr int TS = Tiles<C, XB>::TS;  // values from one y to the next
  if constexpr (!INV) {
    for (int i = threadIdx.x; i < N * Z2; i += NT) {
      const int y = i / Z2, n2 = i % Z2;
      V2<T> a[Z1];
#pragma unroll
      for (int j = 0; j < Z1; ++j) a[j] = ldt<T>(plane[y * H + j * Z2 + n2]);
      dft<T, Z1, false>(a);
#pragma unroll
      for (int j = 1; j < Z1; ++j) a[j] = cmul(a[j], ldt<T>(__ldg(&twz[2 * n2 * j])));
#pragma unroll
      for (int j = 0; j < Z1; ++j) s[y * RS + j * Z2 + n2] = a[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N * Z1; i += NT) {
      const int k1 = i % Z1, y = i / Z1;
      V2<T> b[Z2];
#pragma unroll
      for (int j = 0; j < Z2; ++j) b[j] = s[y * RS + k1 * Z2 + j];
      dft<T, Z2, false>(b);
#pragma unroll
      for (int j = 0; j < Z2; ++j) s[y * RS + k1 * Z2 + j] = b[j];  // column k1 + Z1 j
    }
    __syncthreads();
    for (int i = threadIdx.x; i < Y2 * H; i += NT) {
      const int c = i % H, n2 = i / H;
      V2<T> a[Y1];
#pragma unroll
      for (int j = 0; j < Y1; ++j) a[j] = s[(j * Y2 + n2) * RS + c];
      dft<T, Y1, false>(a);
#pragma unroll
      for (int j = 1; j < Y1; ++j) a[j] = cmul(a[j], ldt<T>(__ldg(&twy[n2 * j])));
#pragma unroll
      for (int j = 0; j < Y1; ++j) s[(j * Y2 + n2) * RS + c] = a[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < Y1 * H; i += NT) {
      const int kz = i % H, k1 = i / H;
      const int c = (kz % Z1) * Z2 + kz / Z1;
      V2<T> b[Y2];
#pragma unroll
      for (int j = 0; j < Y2; ++j) b[j] = s[(k1 * Y2 + j) * RS + c];
      dft<T, Y2, false>(b);
      C* dst = sp + t.col(kz);
#pragma unroll
      for (int j = 0; j < Y2; ++j) {
        C o;
        o.x = b[j].x;
        o.y = b[j].y;
        dst[(k1 + Y1 * j) * TS] = o;
      }
    }
  } else {
    for (int i = threadIdx.x; i < Y2 * H; i += NT) {
      const int kz = i % H, n2 = i / H;
      const C* src = sp + t.col(kz);
      V2<T> a[Y1];
#pragma unroll
      for (int j = 0; j < Y1; ++j) a[j] = ldt<T>(src[(j * Y2 + n2) * TS]);
      dft<T, Y1, true>(a);
#pragma unroll
      for (int j = 1; j < Y1; ++j) a[j] = cmulc(a[j], ldt<T>(__ldg(&twy[n2 * j])));
#pragma unroll
      for (int j = 0; j < Y1; ++j) s[(j * Y2 + n2) * RS + kz] = a[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < Y1 * H; i += NT) {
      const int c = i % H, k1 = i / H;
      V2<T> b[Y2];
#pragma unroll
      for (int j = 0; j < Y2; ++j) b[j] = s[(k1 * Y2 + j) * RS + c];
      dft<T, Y2, true>(b);
#pragma unroll
      for (int j = 0; j < Y2; ++j) s[(k1 * Y2 + j) * RS + c] = b[j];  // row y = k1 + Y1 j at k1 Y2 + j
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N * Z2; i += NT) {
      const int n2 = i % Z2, r = i / Z2;
      V2<T> a[Z1];
#pragma unroll
      for (int j = 0; j < Z1; ++j) a[j] = s[r * RS + j * Z2 + n2];
      dft<T, Z1, true>(a);
#pragma unroll
      for (int j = 1; j < Z1; ++j) a[j] = cmulc(a[j], ldt<T>(__ldg(&twz[2 * n2 * j])));
#pragma unroll
      for (int j = 0; j < Z1; ++j) s[r * RS + j * Z2 + n2] = a[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N * Z1; i += NT) {
      const int k1 = i % Z1, y = i / Z1;
      const int r = (y % Y1) * Y2 + y / Y1;
      V2<T> b[Z2];
#pragma unroll
      for (int j = 0; j < Z2; ++j) b[j] = s[r * RS + k1 * Z2 + j];
      dft<T, Z2, true>(b);
#pragma unroll
      for (int j = 0; j < Z2; ++j) {
        C o;
        o.x = b[j].x;
        o.y = b[j].y;
        plane[y * H + k1 + Z1 * j] = o;
      }
    }
  }
}

// ------------------------------------------------------------------ x transforms + projection
// One wavenumber component with its square, both rounded from FP64 as project_mode of
// fcm_kspace.cu does.
template <typename T>
struct Wave {
  T q, qq;
};
template <typename T>
__device__ __forceinline__ Wave<T> make_wave(double q) {
  return Wave<T>{(T)q, (T)(q * q)};
}

// u = P(q) f / (eta G), the arithmetic of project_mode in fcm_kspace.cu.
template <typename T>
__device__ __forceinline__ void project_wave(const Wave<T>& w1, const Wave<T>& w2, const Wave<T>& w3,
                                             const V2<T> (&f)[3], V2<T> (&u)[3], T ie) {
  const T norm = (T)1 / ((w2.qq + w1.qq + (T)1e-16) + w3.qq);
  const T kr = (w1.q * f[0].x + w2.q * f[1].x + w3.q * f[2].x) * norm;
  const T ki = (w1.q * f[0].y + w2.q * f[1].y + w3.q * f[2].y) * norm;
  const T sc = norm * ie;
  u[0] = V2<T>{sc * (f[0].x - w1.q * kr), sc * (f[0].y - w1.q * ki)};
  u[1] = V2<T>{sc * (f[1].x - w2.q * kr), sc * (f[1].y - w2.q * ki)};
  u[2] = V2<T>{sc * (f[2].x - w3.q * kr), sc * (f[2].y - w3.q * ki)};
}

// What a CTA's column pair jj of slot y0 holds.  jj >= 1: column jj of row y0 (A) and
// column H - jj of row -y0 (B).  jj = 0 takes the two columns that pair with themselves,
// kz = 0 in the slots y0 < ny/2 and kz = H/2 in the others, rows yy = y0 mod ny/2 (A) and
// -yy (B); the rows 0 and ny/2, which pair with themselves as well, share the slot yy = 0.
struct PairSlot {
  int yA, yB, kA, kz;      // rows, place of A's column (B's nkb blocks on, or the same), kz of A
  bool self, plane;        // rows A and B each pair with themselves; kz = 0 (with nz/2)
};
__device__ __forceinline__ PairSlot pair_slot(int y0, int jj, int ny, int H) {
  PairSlot r;
  if (jj > 0) {
    r.yA = y0;
    r.yB = y0 ? ny - y0 : 0;
    r.kA = r.kz = jj;
    r.self = r.plane = false;
  } else {
    const int h = ny / 2, yy = y0 < h ? y0 : y0 - h;
    r.kz = y0 < h ? 0 : H / 2;
    r.yA = yy;
    r.yB = yy ? ny - yy : h;
    r.kA = 0;
    r.self = yy == 0;
    r.plane = y0 < h;
  }
  return r;
}

// Shared-memory geometry: pencils A and B apart, each [x position][3 TK] (column j * 3 + c),
// position k1 N2 + k2 after the first step, rows of N2 positions padded so that the step
// over n2 (lanes: columns, then k1) meets every bank as often as a contiguous access; the
// pair step's lanes (24 bytes apart in FP32, 48 in FP64) are conflict-free as they are.
template <typename C, int N1, int N2, int TK>
struct XShape {
  static constexpr int N = N1 * N2, C3 = 3 * TK;
  static constexpr int E = 128 / (int)sizeof(C);
  static constexpr int PAD = ((C3 * (1 - N2)) % E + E) % E;
  static constexpr int ROW = N2 * C3 + PAD;  // positions k1 N2 .. k1 N2 + N2 - 1
  static constexpr int SIDE = N1 * ROW;      // pencils A or B
  static constexpr size_t SMEM = (size_t)2 * SIDE * sizeof(C) + (size_t)N * sizeof(C);
  __device__ static __forceinline__ int at(int k1, int k2) { return k1 * ROW + k2 * C3; }
};

// The packed modes a at kx and b (conjugated) at -kx of the pair u, v (the inverse of the
// separation below, doubled as the real transform of 2 H points wants).
template <typename T>
__device__ __forceinline__ void fold_pair(V2<T> (&a)[3], V2<T> (&b)[3], const V2<T> (&u)[3], const V2<T> (&v)[3],
                                          V2<T> p) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const V2<T> e = cadd(u[c], v[c]), d = cmulc(csub(u[c], v[c]), p);
    a[c] = cadd(e, d);
    b[c] = csub(e, d);
  }
}

// The projection of one pair: a, b the packed modes (b conjugated) of A at kx and B at
// -kx; p = -i W_nz^kz.  f = X(kx, yA, kz), g = conj X(-kx, yB, H - kz), both doubled (ie
// carries the 1/2 of the separation).
template <typename T>
__device__ __forceinline__ void project_pair(V2<T> (&a)[3], V2<T> (&b)[3], V2<T> p, const Wave<T>& x, const Wave<T>& xp,
                                             const Wave<T>& y, const Wave<T>& yp, const Wave<T>& z,
                                             const Wave<T>& zp, bool plane, bool zero, T ie) {
  V2<T> f[3], g[3], u[3], v[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const V2<T> e = cadd(a[c], b[c]), d = cmul(csub(a[c], b[c]), p);
    f[c] = cadd(e, d);
    g[c] = csub(e, d);
  }
  project_wave<T>(x, y, z, f, u, ie);
  project_wave<T>(xp, yp, zp, g, v, ie);
  if (plane) {  // kz = 0 and nz/2: the mean over {k, -k}, u(0) = 0
    V2<T> u2[3], v2[3];
    project_wave<T>(xp, yp, z, f, u2, ie);
    project_wave<T>(x, y, zp, g, v2, ie);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      u[c] = V2<T>{(T)0.5 * (u[c].x + u2[c].x), (T)0.5 * (u[c].y + u2[c].y)};
      v[c] = V2<T>{(T)0.5 * (v[c].x + v2[c].x), (T)0.5 * (v[c].y + v2[c].y)};
      if (zero) u[c] = V2<T>{(T)0, (T)0};
    }
  }
  fold_pair<T>(a, b, u, v, p);
}

// The x transforms of TK column pairs of one slot, the projection between.  Five steps:
// N1-point DFTs from global memory, N2-point DFTs in place, the pairs, inverse N2-point
// DFTs in place, inverse N1-point DFTs to global memory.
// NOISE: the pairs are the velocities of the fluctuating stress instead (drawn here, so the
// spectrum is written once), and only the inverse steps run.
struct NoiseArgs {
  uint64_t seed, counter;
  const uint64_t* dargs;  // (seed, counter) in device memory, if given
  double amp_diag, amp_off;
};
template <typename T, typename C, int N1, int N2, int TK, int NT, bool NOISE>
__device__ __forceinline__ void packed_x_cta(C* __restrict__ spec, const KParams& k, const C* __restrict__ twx,
                                             const C* __restrict__ twz, const NoiseArgs& na) {
  using S = XShape<C, N1, N2, TK>;
  constexpr int N = S::N, C3 = S::C3;
  extern __shared__ __align__(16) unsigned char packed_smem[];
  V2<T>* s = reinterpret_cast<V2<T>*>(packed_smem);
  Wave<T>* wx = reinterpret_cast<Wave<T>*>(s + 2 * S::SIDE);
  const int H = k.nz / 2, PC = H / 2;  // column pairs per slot
  const int y0 = blockIdx.y, j0 = (int)blockIdx.x * TK;
  constexpr int XB = tile_x(N);
  const Tiles<C, XB> t(N, k.ny, k.nz);
  for (int i = threadIdx.x; i < N; i += NT) wx[i] = make_wave<T>(wavenumber(i, N, k.fx));
  // value x = 0 of the pencil (side, component, pair j); value x is (x / XB) ny tiles and
  // (x % XB) TKB values on
  auto pencil = [&](int side, int c, int j) -> long long {
    const PairSlot p = pair_slot(y0, j0 + j, k.ny, H);
    const bool second = side && j0 + j > 0 ? true : 2 * p.kz == H;
    return t.row(c, 0, side ? p.yB : p.yA) + ((second ? t.nkb : 0) + p.kA / t.TKB) * t.bs + p.kA % t.TKB;
  };
  const long long xs = (long long)k.ny * t.TS;  // one tile in x
  // value x = q N2 + n2 from that: linear in q where N2 is a multiple of XB
  auto x_at = [&](int q, int n2) -> long long {
    if constexpr (N2 % XB == 0) return (n2 / XB) * xs + (n2 % XB) * t.TKB + q * ((N2 / XB) * xs);
    const int x = q * N2 + n2;
    return (x / XB) * xs + (x % XB) * t.TKB;
  };
  if constexpr (!NOISE) {
    // items (pair j, n2, component, side): consecutive lanes the columns of a tile, then x
    for (int i = threadIdx.x; i < 2 * N2 * C3; i += NT) {
      const int j = i % TK, n2 = (i / TK) % N2, c = (i / (TK * N2)) % 3, side = i / (TK * N2 * 3);
      if (j0 + j >= PC) continue;
      const long long e = pencil(side, c, j);
      V2<T> a[N1];
#pragma unroll
      for (int q = 0; q < N1; ++q) {
        const long long at = e + x_at(q, n2);
        a[q] = FCM_INB(at, t.size(), BS_SPECTRUM) ? ldt<T>(spec[at]) : V2<T>{(T)0, (T)0};
      }
      dft<T, N1, false>(a);
#pragma unroll
      for (int q = 1; q < N1; ++q) a[q] = cmul(a[q], ldt<T>(__ldg(&twx[n2 * q])));
#pragma unroll
      for (int q = 0; q < N1; ++q) s[side * S::SIDE + S::at(q, n2) + 3 * j + c] = a[q];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * N1 * C3; i += NT) {
      const int col = i % C3, k1 = (i / C3) % N1, side = i / (C3 * N1);
      if (j0 + col / 3 >= PC) continue;
      V2<T>* row = s + side * S::SIDE + S::at(k1, 0) + col;
      V2<T> b[N2];
#pragma unroll
      for (int j = 0; j < N2; ++j) b[j] = row[j * C3];
      dft<T, N2, false>(b);
#pragma unroll
      for (int j = 0; j < N2; ++j) row[j * C3] = b[j];
    }
    __syncthreads();
  }
  static_assert(NT % TK == 0, "a thread keeps its column pair");
  const uint64_t seed = NOISE && na.dargs ? na.dargs[0] : na.seed;
  const uint64_t counter = NOISE && na.dargs ? na.dargs[1] : na.counter;
  const T ie = (T)(0.5 * k.inv_etaG);
  const int pj = threadIdx.x % TK;
  const PairSlot p = pair_slot(y0, j0 + pj, k.ny, H);
  const V2<T> w = ldt<T>(__ldg(&twz[p.kz]));
  const V2<T> pw = V2<T>{w.y, -w.x};  // -i W
  const Wave<T> z = make_wave<T>((double)p.kz * k.fz), zp = make_wave<T>((double)(H - p.kz) * k.fz);
  const Wave<T> wyA = make_wave<T>(wavenumber(p.yA, k.ny, k.fy)), wyB = make_wave<T>(wavenumber(p.yB, k.ny, k.fy));
  for (int i = threadIdx.x / TK; i < N && j0 + pj < PC; i += NT / TK) {
    const int k2 = i % N2, k1 = i / N2;
    const int kx = k1 + N1 * k2, kxp = kx ? N - kx : 0;
    const int m1 = kxp % N1, m2 = kxp / N1;
    const int rounds = p.self ? 2 : 1;
    if (p.self && kxp < kx) continue;  // the partner's item takes the pair
    for (int r = 0; r < rounds; ++r) {
      const int yA = r ? p.yB : p.yA;
      const Wave<T> y = r ? wyB : wyA, yp = p.self ? y : wyB;
      V2<T>* sa = s + r * S::SIDE + S::at(k1, k2) + 3 * pj;
      V2<T>* sb = s + (p.self ? r : 1) * S::SIDE + S::at(m1, m2) + 3 * pj;
      V2<T> a[3], b[3];
      if constexpr (NOISE) {
        V2<T> u[3], v[3];
        fluct_velocity<T>(kx, yA, p.kz, k, seed, counter, na.amp_diag, na.amp_off, u);
        fluct_velocity<T>(kxp, p.self ? yA : p.yB, H - p.kz, k, seed, counter, na.amp_diag, na.amp_off, v);
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c].y = -v[c].y;
        fold_pair<T>(a, b, u, v, pw);
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          a[c] = sa[c];
          b[c] = V2<T>{sb[c].x, -sb[c].y};
        }
        project_pair<T>(a, b, pw, wx[kx], wx[kxp], y, yp, z, zp, p.plane, kx == 0 && yA == 0, ie);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sa[c] = a[c];
        sb[c] = V2<T>{b[c].x, -b[c].y};
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * N1 * C3; i += NT) {
    const int col = i % C3, k1 = (i / C3) % N1, side = i / (C3 * N1);
    if (j0 + col / 3 >= PC) continue;
    V2<T>* row = s + side * S::SIDE + S::at(k1, 0) + col;
    V2<T> b[N2];
#pragma unroll
    for (int j = 0; j < N2; ++j) b[j] = row[j * C3];
    dft<T, N2, true>(b);
#pragma unroll
    for (int j = 1; j < N2; ++j) b[j] = cmulc(b[j], ldt<T>(__ldg(&twx[j * k1])));
#pragma unroll
    for (int j = 0; j < N2; ++j) row[j * C3] = b[j];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * N2 * C3; i += NT) {
    const int j = i % TK, n2 = (i / TK) % N2, c = (i / (TK * N2)) % 3, side = i / (TK * N2 * 3);
    if (j0 + j >= PC) continue;
    const long long e = pencil(side, c, j);
    V2<T> a[N1];
#pragma unroll
    for (int q = 0; q < N1; ++q) a[q] = s[side * S::SIDE + S::at(q, n2) + 3 * j + c];
    dft<T, N1, true>(a);
#pragma unroll
    for (int q = 0; q < N1; ++q) {
      const long long at = e + x_at(q, n2);
      C o;
      o.x = a[q].x;
      o.y = a[q].y;
      if (FCM_INB(at, t.size(), BS_SPECTRUM)) spec[at] = o;
    }
  }
}

template <typename T, typename C, int N1, int N2, int TK, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_packed_x(C* __restrict__ spec, KParams k, const C* __restrict__ twx,
                                                       const C* __restrict__ twz) {
  chain_begin();
  packed_x_cta<T, C, N1, N2, TK, NT, false>(spec, k, twx, twz, NoiseArgs{});
}

// The spectrum of a fluctuating velocity field, transformed along x.
template <typename T, typename C, int N1, int N2, int TK, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_packed_noise(C* __restrict__ spec, KParams k, const C* __restrict__ twx,
                                                           const C* __restrict__ twz, NoiseArgs na) {
  chain_begin();
  packed_x_cta<T, C, N1, N2, TK, NT, true>(spec, k, twx, twz, na);
}

// Batched: blockIdx.z = member gidx[blockIdx.z] of a group of equal grids.
template <typename T, typename C, int P, int N1, int N2, int TK, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_b_packed_x(const BMember* __restrict__ mem, const int* __restrict__ gidx,
                                                         int mask, const C* __restrict__ twx,
                                                         const C* __restrict__ twz) {
  chain_begin();
  const BMember& m = mem[gidx[blockIdx.z]];
  if (bskip(m, mask)) return;
  packed_x_cta<T, C, N1, N2, TK, NT, false>((C*)m.spec[P], m.kp, twx, twz, NoiseArgs{});
}

// ------------------------------------------------------------------ launches
// Calls f(integral_constant<N1>, integral_constant<N2>) for a supported length n (or
// half a supported length, for z).
template <typename F>
int with_factors(int n, F&& f) {
  using std::integral_constant;
  switch (n) {
    case 4: return f(integral_constant<int, 2>{}, integral_constant<int, 2>{});
    case 6: return f(integral_constant<int, 2>{}, integral_constant<int, 3>{});
    case 8: return f(integral_constant<int, 2>{}, integral_constant<int, 4>{});
    case 12: return f(integral_constant<int, 3>{}, integral_constant<int, 4>{});
    case 16: return f(integral_constant<int, 4>{}, integral_constant<int, 4>{});
    case 24: return f(integral_constant<int, 4>{}, integral_constant<int, 6>{});
    case 32: return f(integral_constant<int, 4>{}, integral_constant<int, 8>{});
    case 48: return f(integral_constant<int, 6>{}, integral_constant<int, 8>{});
    case 64: return f(integral_constant<int, 8>{}, integral_constant<int, 8>{});
    case 96: return f(integral_constant<int, 8>{}, integral_constant<int, 12>{});
    case 128: return f(integral_constant<int, 8>{}, integral_constant<int, 16>{});
    case 192: return f(integral_constant<int, 12>{}, integral_constant<int, 16>{});
    case 256: return f(integral_constant<int, 16>{}, integral_constant<int, 16>{});
    case 384: return f(integral_constant<int, 16>{}, integral_constant<int, 24>{});
    case 512: return f(integral_constant<int, 16>{}, integral_constant<int, 32>{});
    default: break;
  }
  set_error("packed transforms: unsupported length " + std::to_string(n));
  return FCM_ERR_INVALID;
}

// Dynamic shared memory above the default 48 KB for `kernel`, set once per kernel
// and device (keyed by the kernel's address).
template <typename K>
int smem_attr_once(K kernel, size_t smem) {
  if (smem <= 48 * 1024) return FCM_OK;
  static std::mutex mu;
  static std::vector<std::pair<int, const void*>> done;
  int dev = 0;
  FCM_CUDA(cudaGetDevice(&dev));
  const std::pair<int, const void*> key(dev, reinterpret_cast<const void*>(kernel));
  std::lock_guard<std::mutex> lock(mu);
  if (std::find(done.begin(), done.end(), key) == done.end()) {
    FCM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    done.push_back(key);
  }
  return FCM_OK;
}

template <typename T>
const typename cplx_t<T>::type* xtw(const Ctx& c) {
  return (const typename cplx_t<T>::type*)(sizeof(T) == 4 ? c.d_xtw32 : c.d_xtw64);
}
template <typename T>
const typename cplx_t<T>::type* ytw(const Ctx& c) {
  return (const typename cplx_t<T>::type*)(sizeof(T) == 4 ? c.d_ytw32 : c.d_ytw64);
}
template <typename T>
const typename cplx_t<T>::type* ztw(const Ctx& c) {
  return (const typename cplx_t<T>::type*)(sizeof(T) == 4 ? c.d_ztw32 : c.d_ztw64);
}

// Calls f(integral_constant<XB>) for the tiles of c's grid.
template <typename F>
int with_tiles(const Ctx& c, F&& f) {
  return tile_x(c.g.nx) == 8 ? f(std::integral_constant<int, 8>{}) : f(std::integral_constant<int, 4>{});
}

template <typename T, bool INV>
int packed_z(const Ctx& c, typename cplx_t<T>::type* real, typename cplx_t<T>::type* spec, int members,
             cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  return with_factors(c.g.nz / 2, [&](auto a, auto b) -> int {
    constexpr int Z1 = decltype(a)::value, Z2 = decltype(b)::value, NT = 256;
    if constexpr (Z1 * Z2 > 256) {
      return FCM_ERR_INVALID;  // nz <= 512
    } else {
      return with_tiles(c, [&](auto xb) -> int {
        constexpr int XB = decltype(xb)::value;
        constexpr int Q = NT / (Z1 > Z2 ? Z1 : Z2), YQ = Q / XB;
        constexpr size_t smem = (size_t)Q * z_line_stride<C, XB, Z1, Z2>() * sizeof(C);
        auto kern = k_packed_z<T, C, XB, Z1, Z2, NT, INV>;
        FCM_TRY(smem_attr_once(kern, smem));
        const Tiles<C, XB> t(c.g.nx, c.g.ny, c.g.nz);
        const unsigned ctas = (unsigned)(3LL * members * t.nxb * ((t.ny + YQ - 1) / YQ));
        return launch_chained(kern, dim3(ctas), dim3(NT), smem, s, real, spec, t, ztw<T>(c));
      });
    }
  });
}

template <typename T, bool INV>
int packed_y(const Ctx& c, typename cplx_t<T>::type* spec, int members, cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  return with_factors(c.g.ny, [&](auto a, auto b) -> int {
    constexpr int Y1 = decltype(a)::value, Y2 = decltype(b)::value;
    constexpr int NT = sizeof(T) == 8 ? 128 : 256;
    constexpr size_t smem = (size_t)Y1 * Y2 * 128;
    auto kern = k_packed_y<T, C, Y1, Y2, NT, INV>;
    FCM_TRY(smem_attr_once(kern, smem));
    const long long per = packed_spectrum_size<T>(c) / ((long long)Y1 * Y2 * (128 / (int)sizeof(C)));  // tile columns
    return launch_chained(kern, dim3((unsigned)(per * members)), dim3(NT), smem, s, spec, ytw<T>(c));
  });
}

// Square (y, z) planes of these sizes take the per-plane kernels (39 KB of shared
// memory at 96 points in FP32, 75 KB in FP64).
bool plane_ok(const Ctx& c) {
  switch (c.g.nz) {
    case 16: case 32: case 48: case 64: case 96: return c.g.ny == c.g.nz;
    default: return false;
  }
}

template <typename T, bool INV>
int packed_plane(const Ctx& c, typename cplx_t<T>::type* real, typename cplx_t<T>::type* spec, int members,
                 cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  return with_factors(c.g.nz, [&](auto a, auto b) -> int {
    constexpr int Y1 = decltype(a)::value, Y2 = decltype(b)::value, N = Y1 * Y2;
    return with_factors(N / 2, [&](auto d, auto e) -> int {
      constexpr int Z1 = decltype(d)::value, Z2 = decltype(e)::value, NT = 256;
      if constexpr (2 * Z1 * Z2 != N || N > 96) {
        return FCM_ERR_INVALID;
      } else {
        constexpr size_t smem = (size_t)N * (N / 2 + 1) * sizeof(C);
        return with_tiles(c, [&](auto xb) -> int {
          constexpr int XB = decltype(xb)::value;
          auto kern = k_packed_plane<T, C, XB, Z1, Z2, Y1, Y2, NT, INV>;
          FCM_TRY(smem_attr_once(kern, smem));
          return launch_chained(kern, dim3((unsigned)(3LL * c.g.nx * members)), dim3(NT), smem, s, real, spec,
                                Tiles<C, XB>(c.g.nx, c.g.ny, c.g.nz), ytw<T>(c), ztw<T>(c));
        });
      }
    });
  });
}

// Column pairs per CTA of the x pass (a tile's columns), its threads, and the CTAs per SM
// its registers must allow: small CTAs, since their steps are separated by barriers and
// only other CTAs fill the gaps (49 KB of pencils and four CTAs at 512 points).
template <typename T, int N>
constexpr int px_tk() {
  return 64 / (int)sizeof(T) / tile_x(N);
}
template <typename T, int N>
constexpr int px_threads() {
  return N <= 128 ? 128 : N < 256 ? 192 : N == 256 ? 96 : sizeof(T) == 4 ? 192 : 96;
}
template <typename T, int N>
constexpr int px_min() {
  return N <= 128 ? 4 : N == 256 ? (sizeof(T) == 4 ? 8 : 5) : sizeof(T) == 4 ? 4 : N <= 256 ? 3 : 4;
}

template <typename T>
int packed_x(const Ctx& c, typename cplx_t<T>::type* spec, cudaStream_t s, const BatchGeom* b, const int* gidx, int nm,
             int mask) {
  using C = typename cplx_t<T>::type;
  constexpr int P = sizeof(T) == 8 ? 0 : 1;
  return with_factors(c.g.nx, [&](auto a, auto d) -> int {
    constexpr int N1 = decltype(a)::value, N2 = decltype(d)::value, N = N1 * N2;
    constexpr int TK = px_tk<T, N>(), NT = px_threads<T, N>(), MB = px_min<T, N>();
    constexpr size_t smem = XShape<C, N1, N2, TK>::SMEM;
    const int pairs = c.g.nz / 4;
    const dim3 grid((unsigned)((pairs + TK - 1) / TK), (unsigned)c.g.ny, (unsigned)(b ? nm : 1));
    if (b) {
      auto kern = k_b_packed_x<T, C, P, N1, N2, TK, NT, MB>;
      FCM_TRY(smem_attr_once(kern, smem));
      return launch_chained(kern, grid, dim3(NT), smem, s, b->mem, gidx, mask, xtw<T>(c), ztw<T>(c));
    } else {
      auto kern = k_packed_x<T, C, N1, N2, TK, NT, MB>;
      FCM_TRY(smem_attr_once(kern, smem));
      return launch_chained(kern, grid, dim3(NT), smem, s, spec, make_kparams(c), xtw<T>(c), ztw<T>(c));
    }
  });
}

}  // namespace

int packed_tables_init() { return w96_upload(); }

// The (y, z) transforms of `members` consecutive grids of c's shape: forward from the
// real grid r into the packed spectrum, inverse from the spectrum (overwritten) into r.
template <typename T>
int launch_packed_forward(const Ctx& c, const T* r, typename cplx_t<T>::type* spec, int members, cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  C* real = reinterpret_cast<C*>(const_cast<T*>(r));  // read only in this direction
  if (plane_ok(c)) return packed_plane<T, false>(c, real, spec, members, s);
  FCM_TRY((packed_z<T, false>(c, real, spec, members, s)));
  return packed_y<T, false>(c, spec, members, s);
}

template <typename T>
int launch_packed_inverse(const Ctx& c, typename cplx_t<T>::type* spec, T* r, int members, cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  C* real = reinterpret_cast<C*>(r);
  if (plane_ok(c)) return packed_plane<T, true>(c, real, spec, members, s);
  FCM_TRY((packed_y<T, true>(c, spec, members, s)));
  return packed_z<T, true>(c, real, spec, members, s);
}

template <typename T>
long long packed_spectrum_size(const Ctx& c) {
  using C = typename cplx_t<T>::type;
  return tile_x(c.g.nx) == 8 ? Tiles<C, 8>(c.g.nx, c.g.ny, c.g.nz).size()
                             : Tiles<C, 4>(c.g.nx, c.g.ny, c.g.nz).size();
}

template <typename T>
int launch_packed_project(const Ctx& c, typename cplx_t<T>::type* spec, cudaStream_t s) {
  return packed_x<T>(c, spec, s, nullptr, nullptr, 0, 0);
}

// The fluctuating velocity field of (seed, counter), or d_args[0..1] where given, into r.
int launch_packed_noise(const Ctx& c, cufftDoubleComplex* spec, double* r, uint64_t seed, uint64_t counter,
                        const uint64_t* d_args, cudaStream_t s) {
  using T = double;
  using C = cufftDoubleComplex;
  NoiseArgs na{seed, counter, d_args, 0.0, 0.0};
  stress_amplitudes(c, na.amp_diag, na.amp_off);
  FCM_TRY(with_factors(c.g.nx, [&](auto a, auto d) -> int {
    constexpr int N1 = decltype(a)::value, N2 = decltype(d)::value, N = N1 * N2;
    constexpr int TK = px_tk<T, N>(), NT = px_threads<T, N>(), MB = px_min<T, N>();
    constexpr size_t smem = XShape<C, N1, N2, TK>::SMEM;
    const dim3 grid((unsigned)((c.g.nz / 4 + TK - 1) / TK), (unsigned)c.g.ny);
    auto kern = k_packed_noise<T, C, N1, N2, TK, NT, MB>;
    FCM_TRY(smem_attr_once(kern, smem));
    return launch_chained(kern, grid, dim3(NT), smem, s, spec, make_kparams(c), xtw<T>(c), ztw<T>(c), na);
  }));
  return launch_packed_inverse<T>(c, spec, r, 1, s);
}

template <typename T>
int b_packed_project(const BatchGeom& b, const Ctx& c0, const int* gidx, int nm, int mask, cudaStream_t s) {
  return packed_x<T>(c0, nullptr, s, &b, gidx, nm, mask);
}

template long long packed_spectrum_size<double>(const Ctx&);
template long long packed_spectrum_size<float>(const Ctx&);
template int launch_packed_forward<double>(const Ctx&, const double*, cufftDoubleComplex*, int, cudaStream_t);
template int launch_packed_forward<float>(const Ctx&, const float*, cufftComplex*, int, cudaStream_t);
template int launch_packed_inverse<double>(const Ctx&, cufftDoubleComplex*, double*, int, cudaStream_t);
template int launch_packed_inverse<float>(const Ctx&, cufftComplex*, float*, int, cudaStream_t);
template int launch_packed_project<double>(const Ctx&, cufftDoubleComplex*, cudaStream_t);
template int launch_packed_project<float>(const Ctx&, cufftComplex*, cudaStream_t);
template int b_packed_project<double>(const BatchGeom&, const Ctx&, const int*, int, int, cudaStream_t);
template int b_packed_project<float>(const BatchGeom&, const Ctx&, const int*, int, int, cudaStream_t);

FCM_BOUNDS_READER(bounds_read_packed)

}  // namespace fcm

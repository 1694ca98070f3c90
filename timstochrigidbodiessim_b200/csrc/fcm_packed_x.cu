// fcm_packed_x.cu -- x passes of the Stokes solve on a packed half spectrum: forward
// transform, projection and inverse transform, and the draw of the fluctuating field, for
// one precision and class of lengths per object (build.py), a batch's kernels in objects of
// their own.
#include "fcm_fluct.cuh"
#include "fcm_packed.cuh"

#ifndef FCM_PACKED_T
#define FCM_PACKED_T double
#define FCM_PACKED_CLASS 0
#endif
#ifndef FCM_PACKED_BATCH
#define FCM_PACKED_BATCH 0
#endif

namespace fcm {

namespace {

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
// kz = 0 in the slots y0 < ny/2 and kz = H/2 (H even) in the others, rows yy = y0 mod ny/2 (A) and
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
  const int H = k.nz / 2, PC = (H + 1) / 2;  // column pairs per slot
  const int y0 = blockIdx.y, j0 = (int)blockIdx.x * TK;
  // no pair: past the last one, or the place of column H/2 where there is none
  auto no_pair = [&](int j) { return j0 + j >= PC || (j0 + j == 0 && H % 2 && 2 * y0 >= k.ny); };
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
      if (no_pair(j)) continue;
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
      if (no_pair(col / 3)) continue;
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
  for (int i = threadIdx.x / TK; i < N && !no_pair(pj); i += NT / TK) {
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
    if (no_pair(col / 3)) continue;
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
    if (no_pair(j)) continue;
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

// Column pairs per CTA of the x pass (a tile's columns), its threads, and the CTAs per SM
// its registers must allow: small CTAs, since their steps are separated by barriers and
// only other CTAs fill the gaps (49 KB of pencils and four CTAs at 512 points).  In FP64
// 192 threads leave 96 registers, which spill: 128 threads up to 216 points (solve at 200
// points 426 -> 402 us, 160 195 -> 186), above which five of their CTAs no longer fit (240
// points 671 -> 708 us).  From 256 points on, where a CTA has half the columns: us of a solve
// with 256 x 256 points along y and z, by 96 threads (FP64 five CTAs, FP32 eight), 128 (four,
// six) and beyond that 96 in FP64 (four CTAs) and 192 in FP32 (four):
//   FP64  256 758 763 771   280 873 865 877   288 905 889 902   320 1041 969 987   384 1200 1173 1142
//   FP32  256 380 381 377   280 454 444 454   288 462 449 460   320 507 492 508    384 595 585 577
// (400, 480 and 512 as 384), so the first below 280 points, the second to 320.
template <typename T, int N>
constexpr int px_tk() {
  return 64 / (int)sizeof(T) / tile_x(N);
}
template <typename T, int N>
constexpr int px_threads() {
  if (N <= 128 || (sizeof(T) == 8 && N <= 216)) return 128;
  if (N < 256) return 192;
  if (N < 280) return 96;
  if (N <= 320) return 128;
  return sizeof(T) == 4 ? 192 : 96;
}
template <typename T, int N>
constexpr int px_min() {
  if (N <= 128 || (sizeof(T) == 8 && N <= 216)) return 4;
  if (N < 256) return sizeof(T) == 4 ? 4 : 3;
  if (N < 280) return sizeof(T) == 4 ? 8 : 5;
  if (N <= 320) return sizeof(T) == 4 ? 6 : 4;
  return 4;
}

using Real = FCM_PACKED_T;
using Cplx = cplx_t<Real>::type;
constexpr int CLASS = FCM_PACKED_CLASS;

// Calls f(kernel of this length's sizes, threads, shared memory, grid of nm members).
template <typename F>
int with_x_length(const Ctx& c, int nm, F&& f) {
  return with_length<CLASS>(c.g.nx, [&](auto l) -> int {
    constexpr PackedLength L = PACKED_LENGTHS[decltype(l)::value];
    if constexpr (x_length(L.n)) {
      constexpr int TK = px_tk<Real, L.n>();
      const int pairs = (c.g.nz / 2 + 1) / 2;
      return f(l, XShape<Cplx, L.n1, L.n2, TK>::SMEM,
               dim3((unsigned)((pairs + TK - 1) / TK), (unsigned)c.g.ny, (unsigned)nm));
    } else {
      set_error("packed transforms: unsupported length along x");
      return FCM_ERR_INVALID;
    }
  });
}

}  // namespace

#if FCM_PACKED_BATCH

template <>
int b_packed_x_init<Real, CLASS>() {
  return roots_upload();
}
template <>
int b_packed_x_pass<Real, CLASS>(const BatchGeom& b, const Ctx& c0, const int* gidx, int nm, int mask,
                                 cudaStream_t s) {
  return with_x_length(c0, nm, [&](auto l, size_t smem, dim3 grid) -> int {
    constexpr PackedLength L = PACKED_LENGTHS[decltype(l)::value];
    constexpr int NT = px_threads<Real, L.n>();
    auto kern = k_b_packed_x<Real, Cplx, sizeof(Real) == 8 ? 0 : 1, L.n1, L.n2, px_tk<Real, L.n>(), NT,
                             px_min<Real, L.n>()>;
    FCM_TRY(smem_attr_once(kern, smem));
    return launch_chained(kern, grid, dim3(NT), smem, s, b.mem, gidx, mask, xtw<Real>(c0), ztw<Real>(c0));
  });
}

template <>
FCM_BOUNDS_READER(bounds_read_b_packed_x<2 * CLASS + (sizeof(Real) == 4)>)

#else

template <>
int packed_x_init<Real, CLASS>() {
  return roots_upload();
}
template <>
int packed_x_pass<Real, CLASS>(const Ctx& c, Cplx* spec, cudaStream_t s) {
  return with_x_length(c, 1, [&](auto l, size_t smem, dim3 grid) -> int {
    constexpr PackedLength L = PACKED_LENGTHS[decltype(l)::value];
    constexpr int NT = px_threads<Real, L.n>();
    auto kern = k_packed_x<Real, Cplx, L.n1, L.n2, px_tk<Real, L.n>(), NT, px_min<Real, L.n>()>;
    FCM_TRY(smem_attr_once(kern, smem));
    return launch_chained(kern, grid, dim3(NT), smem, s, spec, make_kparams(c), xtw<Real>(c), ztw<Real>(c));
  });
}

// FP64 only: the spectrum of the fluctuating velocity field.
template <int CL>
int packed_noise_pass(const Ctx& c, cufftDoubleComplex* spec, uint64_t seed, uint64_t counter, const uint64_t* d_args,
                      cudaStream_t s) {
  NoiseArgs na{seed, counter, d_args, 0.0, 0.0};
  stress_amplitudes(c, na.amp_diag, na.amp_off);
  return with_x_length(c, 1, [&](auto l, size_t smem, dim3 grid) -> int {
    constexpr PackedLength L = PACKED_LENGTHS[decltype(l)::value];
    // the draws need more threads than the transforms (field at 256 x 128 x 128 153 -> 145 us, 512
    // 366 -> 352)
    constexpr bool LONG = L.n >= 256;
    constexpr int NT = LONG ? 128 : px_threads<double, L.n>();
    auto kern = k_packed_noise<double, cufftDoubleComplex, L.n1, L.n2, px_tk<double, L.n>(), NT,
                               LONG ? 4 : px_min<double, L.n>()>;
    FCM_TRY(smem_attr_once(kern, smem));
    return launch_chained(kern, grid, dim3(NT), smem, s, spec, make_kparams(c), xtw<double>(c), ztw<double>(c), na);
  });
}
#ifdef FCM_PACKED_NOISE
template int packed_noise_pass<CLASS>(const Ctx&, cufftDoubleComplex*, uint64_t, uint64_t, const uint64_t*,
                                      cudaStream_t);
#endif

template <>
FCM_BOUNDS_READER(bounds_read_packed_x<2 * CLASS + (sizeof(Real) == 4)>)

#endif

}  // namespace fcm

// fcm_packed_zy.cu -- z and y passes of the Stokes solve on a packed half spectrum, for one
// precision and class of lengths per object (build.py).
#include "fcm_packed.cuh"

#ifndef FCM_PACKED_T
#define FCM_PACKED_T double
#define FCM_PACKED_CLASS 0
#endif

namespace fcm {

namespace {

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
  constexpr int YQ = NT / ZM / XB, Q = YQ * XB;  // rows and lines per CTA
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
  [[maybe_unused]] const long long comps = gridDim.x / ((unsigned)nyb * t.nxb);  // components of all members
  [[maybe_unused]] const long long nreal = comps * t.nxb * XB * t.ny * H, nspec = comps / 3 * t.size();
  for (int i = threadIdx.x; i < Q * Z2; i += NT) {
    int p = i / Z2, n2 = i % Z2;
    if (INV) tile_item<TKB, Q, Z2>(i, p, n2);
    if (line_y(p) >= t.ny) continue;
    V2<T> a[Z1];
    if constexpr (INV) {
      const C* src = spec_line(p);
      const ColRun<C, XB, Z2, Z1> col(t, n2);
#pragma unroll
      for (int j = 0; j < Z1; ++j)
        a[j] = FCM_INB(src + col.at(j) - spec, nspec, BS_SPECTRUM) ? ldt<T>(src[col.at(j)]) : V2<T>{(T)0, (T)0};
    } else {
      const C* src = real_line(p) + n2;
#pragma unroll
      for (int j = 0; j < Z1; ++j)
        a[j] = FCM_INB(src + j * Z2 - real, nreal, BS_GRID) ? ldt<T>(src[j * Z2]) : V2<T>{(T)0, (T)0};
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
      const long long at = INV ? (long long)(Z1 * j) : col.at(j);
      if (INV ? FCM_INB(dst + at - real, nreal, BS_GRID) : FCM_INB(dst + at - spec, nspec, BS_SPECTRUM)) dst[at] = o;
    }
  }
}

// ------------------------------------------------------------------ y pass
// Transforms along y in place: one CTA per tile column, XB x times TKB columns at once in
// a contiguous run of 128 ny bytes, the two steps as above.
template <typename T, typename C, int Y1, int Y2, int NT, bool INV>
__global__ void __launch_bounds__(NT) k_packed_y(C* __restrict__ spec, const C* __restrict__ tw,
                                                 [[maybe_unused]] long long nspec) {
  chain_begin();
  constexpr int TK = 128 / (int)sizeof(C);  // values per tile
  extern __shared__ __align__(16) unsigned char packed_smem[];
  V2<T>* s = reinterpret_cast<V2<T>*>(packed_smem);  // [Y1 Y2][TK]
  C* base = spec + (long long)blockIdx.x * (Y1 * Y2 * TK);
  auto in = [&](int i) { return FCM_INB(base + i - spec, nspec, BS_SPECTRUM); };
  for (int i = threadIdx.x; i < Y2 * TK; i += NT) {
    const int kzl = i % TK, n2 = i / TK;
    V2<T> a[Y1];
#pragma unroll
    for (int j = 0; j < Y1; ++j) {
      const int at = (j * Y2 + n2) * TK + kzl;
      a[j] = in(at) ? ldt<T>(base[at]) : V2<T>{(T)0, (T)0};
    }
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
      if (in((k1 + Y1 * j) * TK + kzl)) base[(k1 + Y1 * j) * TK + kzl] = o;
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
  [[maybe_unused]] const long long nreal = (long long)gridDim.x * N * H, nspec = gridDim.x / (3u * nx) * t.size();
  if constexpr (!INV) {
    for (int i = threadIdx.x; i < N * Z2; i += NT) {
      const int y = i / Z2, n2 = i % Z2;
      V2<T> a[Z1];
#pragma unroll
      for (int j = 0; j < Z1; ++j) {
        const int at = y * H + j * Z2 + n2;
        a[j] = FCM_INB(plane + at - real, nreal, BS_GRID) ? ldt<T>(plane[at]) : V2<T>{(T)0, (T)0};
      }
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
        if (FCM_INB(dst + (k1 + Y1 * j) * TS - spec, nspec, BS_SPECTRUM)) dst[(k1 + Y1 * j) * TS] = o;
      }
    }
  } else {
    for (int i = threadIdx.x; i < Y2 * H; i += NT) {
      const int kz = i % H, n2 = i / H;
      const C* src = sp + t.col(kz);
      V2<T> a[Y1];
#pragma unroll
      for (int j = 0; j < Y1; ++j) {
        const int at = (j * Y2 + n2) * TS;
        a[j] = FCM_INB(src + at - spec, nspec, BS_SPECTRUM) ? ldt<T>(src[at]) : V2<T>{(T)0, (T)0};
      }
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
        if (FCM_INB(plane + y * H + k1 + Z1 * j - real, nreal, BS_GRID)) plane[y * H + k1 + Z1 * j] = o;
      }
    }
  }
}

// Calls f(integral_constant<XB>) for the tiles of c's grid.
template <typename F>
int with_tiles(const Ctx& c, F&& f) {
  return tile_x(c.g.nx) == 8 ? f(std::integral_constant<int, 8>{}) : f(std::integral_constant<int, 4>{});
}

template <typename T, int CL, bool INV>
int packed_z(const Ctx& c, typename cplx_t<T>::type* real, typename cplx_t<T>::type* spec, int members,
             cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  return with_length<CL>(c.g.nz, [&](auto l) -> int {
    constexpr PackedLength L = PACKED_LENGTHS[decltype(l)::value];
    constexpr int Z1 = L.h1, Z2 = L.h2, NT = 256;
    return with_tiles(c, [&](auto xb) -> int {
      constexpr int XB = decltype(xb)::value;
      constexpr int YQ = NT / (Z1 > Z2 ? Z1 : Z2) / XB, Q = YQ * XB;
      constexpr size_t smem = (size_t)Q * z_line_stride<C, XB, Z1, Z2>() * sizeof(C);
      auto kern = k_packed_z<T, C, XB, Z1, Z2, NT, INV>;
      FCM_TRY(smem_attr_once(kern, smem));
      const Tiles<C, XB> t(c.g.nx, c.g.ny, c.g.nz);
      const unsigned ctas = (unsigned)(3LL * members * t.nxb * ((t.ny + YQ - 1) / YQ));
      return launch_chained(kern, dim3(ctas), dim3(NT), smem, s, real, spec, t, ztw<T>(c));
    });
  });
}

template <typename T, int CL, bool INV>
int packed_y(const Ctx& c, typename cplx_t<T>::type* spec, int members, cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  return with_length<CL>(c.g.ny, [&](auto l) -> int {
    constexpr PackedLength L = PACKED_LENGTHS[decltype(l)::value];
    constexpr int NT = sizeof(T) == 8 ? 128 : 256;
    constexpr size_t smem = (size_t)L.n * 128;
    auto kern = k_packed_y<T, C, L.n1, L.n2, NT, INV>;
    FCM_TRY(smem_attr_once(kern, smem));
    const long long size = packed_spectrum_size<T>(c), per = size / ((long long)L.n * (128 / (int)sizeof(C)));
    return launch_chained(kern, dim3((unsigned)(per * members)), dim3(NT), smem, s, spec, ytw<T>(c),
                          (long long)members * size);  // a CTA per tile column
  });
}

template <typename T, bool INV>
int packed_plane(const Ctx& c, typename cplx_t<T>::type* real, typename cplx_t<T>::type* spec, int members,
                 cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  return with_length<0>(c.g.nz, [&](auto l) -> int {
    constexpr PackedLength L = PACKED_LENGTHS[decltype(l)::value];
    constexpr int NT = 256;
    constexpr size_t smem = (size_t)L.n * (L.n / 2 + 1) * sizeof(C);
    return with_tiles(c, [&](auto xb) -> int {
      constexpr int XB = decltype(xb)::value;
      auto kern = k_packed_plane<T, C, XB, L.h1, L.h2, L.n1, L.n2, NT, INV>;
      FCM_TRY(smem_attr_once(kern, smem));
      return launch_chained(kern, dim3((unsigned)(3LL * c.g.nx * members)), dim3(NT), smem, s, real, spec,
                            Tiles<C, XB>(c.g.nx, c.g.ny, c.g.nz), ytw<T>(c), ztw<T>(c));
    });
  });
}

using Real = FCM_PACKED_T;
using Cplx = cplx_t<Real>::type;
constexpr int CLASS = FCM_PACKED_CLASS;

}  // namespace

template <>
int packed_zy_init<Real, CLASS>() {
  return roots_upload();
}
template <>
int packed_z_pass<Real, CLASS>(const Ctx& c, Cplx* real, Cplx* spec, int members, bool inverse, cudaStream_t s) {
  return inverse ? packed_z<Real, CLASS, true>(c, real, spec, members, s)
                 : packed_z<Real, CLASS, false>(c, real, spec, members, s);
}
template <>
int packed_y_pass<Real, CLASS>(const Ctx& c, Cplx* spec, int members, bool inverse, cudaStream_t s) {
  return inverse ? packed_y<Real, CLASS, true>(c, spec, members, s)
                 : packed_y<Real, CLASS, false>(c, spec, members, s);
}
#if FCM_PACKED_CLASS == 0
template <>
int packed_plane_pass<Real>(const Ctx& c, Cplx* real, Cplx* spec, int members, bool inverse, cudaStream_t s) {
  return inverse ? packed_plane<Real, true>(c, real, spec, members, s)
                 : packed_plane<Real, false>(c, real, spec, members, s);
}
#endif

template <>
FCM_BOUNDS_READER(bounds_read_packed_zy<2 * CLASS + (sizeof(Real) == 4)>)

}  // namespace fcm

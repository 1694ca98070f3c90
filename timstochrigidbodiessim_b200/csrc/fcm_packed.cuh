// fcm_packed.cuh -- layout, lengths and launch helpers of the Stokes solve on a packed half
// spectrum (fcm_packed.cu: z and y passes, fcm_packed_x.cu: x passes).
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
// a row per CTA.  The columns j < H/2 fill the blocks 0..nkb - 1 in order, H/2 (where it is a
// whole number) the first place of block nkb and H - j (0 < j < H/2) place j from there: the
// two columns of a pair lie nkb blocks apart.  Lengths: those of with_length.
//
// Measured per solve against the separate passes on nz/2 + 1 columns with cuFFT's 3D or
// (y, z) plans in FP64 (us, FP64 / FP32): 64^3 29 / 20 (43 / 25), 96^3 60 / 35 (101 / 43),
// 128^3 96 / 59 (138 / 84), 256^3 766 / 393 (922 / 474), 384^3 2650 / 1460 (6010 / 1730),
// 512^3 6490 / 3230 (9420 / 3970).  At 512^3 the z and y passes run at 5.5-6.5 TB/s; the x
// pass (FP32 1.04 ms for 3.2 GB, FP64 2.08) is bound by its five steps between barriers.
#pragma once
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "fcm_dft.cuh"
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
      : H(nz / 2), nkb(((nz / 2 + 1) / 2 + TKB - 1) / TKB), nxb(nx / XB), ny(ny_), bs((long long)(nx / XB) * ny_ * TS) {}
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

// Calls f(integral_constant<N1>, integral_constant<N2>) with the two register DFT sizes of
// length n along y: the even numbers with factors 2, 3, 5 and 7 from 32 to 320 whose
// register sizes stay within 20 points, and a few smaller and longer ones.
template <typename F>
int with_length(int n, F&& f) {
  using std::integral_constant;
  switch (n) {
    case 8: return f(integral_constant<int, 2>{}, integral_constant<int, 4>{});
    case 12: return f(integral_constant<int, 3>{}, integral_constant<int, 4>{});
    case 16: return f(integral_constant<int, 4>{}, integral_constant<int, 4>{});
    case 24: return f(integral_constant<int, 4>{}, integral_constant<int, 6>{});
    case 32: return f(integral_constant<int, 4>{}, integral_constant<int, 8>{});
    case 36: return f(integral_constant<int, 6>{}, integral_constant<int, 6>{});
    case 40: return f(integral_constant<int, 5>{}, integral_constant<int, 8>{});
    case 42: return f(integral_constant<int, 6>{}, integral_constant<int, 7>{});
    case 48: return f(integral_constant<int, 6>{}, integral_constant<int, 8>{});
    case 50: return f(integral_constant<int, 5>{}, integral_constant<int, 10>{});
    case 54: return f(integral_constant<int, 6>{}, integral_constant<int, 9>{});
    case 56: return f(integral_constant<int, 7>{}, integral_constant<int, 8>{});
    case 60: return f(integral_constant<int, 6>{}, integral_constant<int, 10>{});
    case 64: return f(integral_constant<int, 8>{}, integral_constant<int, 8>{});
    case 70: return f(integral_constant<int, 7>{}, integral_constant<int, 10>{});
    case 72: return f(integral_constant<int, 8>{}, integral_constant<int, 9>{});
    case 80: return f(integral_constant<int, 8>{}, integral_constant<int, 10>{});
    case 84: return f(integral_constant<int, 7>{}, integral_constant<int, 12>{});
    case 90: return f(integral_constant<int, 9>{}, integral_constant<int, 10>{});
    case 96: return f(integral_constant<int, 8>{}, integral_constant<int, 12>{});
    case 98: return f(integral_constant<int, 7>{}, integral_constant<int, 14>{});
    case 100: return f(integral_constant<int, 10>{}, integral_constant<int, 10>{});
    case 108: return f(integral_constant<int, 9>{}, integral_constant<int, 12>{});
    case 112: return f(integral_constant<int, 8>{}, integral_constant<int, 14>{});
    case 120: return f(integral_constant<int, 10>{}, integral_constant<int, 12>{});
    case 126: return f(integral_constant<int, 9>{}, integral_constant<int, 14>{});
    case 128: return f(integral_constant<int, 8>{}, integral_constant<int, 16>{});
    case 140: return f(integral_constant<int, 10>{}, integral_constant<int, 14>{});
    case 144: return f(integral_constant<int, 12>{}, integral_constant<int, 12>{});
    case 150: return f(integral_constant<int, 10>{}, integral_constant<int, 15>{});
    case 160: return f(integral_constant<int, 10>{}, integral_constant<int, 16>{});
    case 162: return f(integral_constant<int, 9>{}, integral_constant<int, 18>{});
    case 168: return f(integral_constant<int, 12>{}, integral_constant<int, 14>{});
    case 180: return f(integral_constant<int, 12>{}, integral_constant<int, 15>{});
    case 192: return f(integral_constant<int, 12>{}, integral_constant<int, 16>{});
    case 196: return f(integral_constant<int, 14>{}, integral_constant<int, 14>{});
    case 200: return f(integral_constant<int, 10>{}, integral_constant<int, 20>{});
    case 210: return f(integral_constant<int, 14>{}, integral_constant<int, 15>{});
    case 216: return f(integral_constant<int, 12>{}, integral_constant<int, 18>{});
    case 224: return f(integral_constant<int, 14>{}, integral_constant<int, 16>{});
    case 240: return f(integral_constant<int, 15>{}, integral_constant<int, 16>{});
    case 252: return f(integral_constant<int, 14>{}, integral_constant<int, 18>{});
    case 256: return f(integral_constant<int, 16>{}, integral_constant<int, 16>{});
    case 270: return f(integral_constant<int, 15>{}, integral_constant<int, 18>{});
    case 280: return f(integral_constant<int, 14>{}, integral_constant<int, 20>{});
    case 288: return f(integral_constant<int, 16>{}, integral_constant<int, 18>{});
    case 300: return f(integral_constant<int, 15>{}, integral_constant<int, 20>{});
    case 320: return f(integral_constant<int, 16>{}, integral_constant<int, 20>{});
    case 384: return f(integral_constant<int, 16>{}, integral_constant<int, 24>{});
    case 400: return f(integral_constant<int, 20>{}, integral_constant<int, 20>{});
    case 480: return f(integral_constant<int, 20>{}, integral_constant<int, 24>{});
    case 512: return f(integral_constant<int, 16>{}, integral_constant<int, 32>{});
    default: break;
  }
  set_error("packed transforms: unsupported length " + std::to_string(n));
  return FCM_ERR_INVALID;
}
// The same along x: whole tiles.
constexpr bool x_length(int n) { return n % tile_x(n) == 0; }
template <typename F>
int with_length_x(int n, F&& f) {
  return with_length(n, [&](auto a, auto b) -> int {
    if constexpr (x_length(decltype(a)::value * decltype(b)::value)) {
      return f(a, b);
    } else {
      set_error("packed transforms: unsupported length along x");
      return FCM_ERR_INVALID;
    }
  });
}
// The same for half a length (the z transforms).
template <typename F>
int with_half_length(int h, F&& f) {
  using std::integral_constant;
  switch (h) {
    case 4: return f(integral_constant<int, 2>{}, integral_constant<int, 2>{});
    case 6: return f(integral_constant<int, 2>{}, integral_constant<int, 3>{});
    case 8: return f(integral_constant<int, 2>{}, integral_constant<int, 4>{});
    case 12: return f(integral_constant<int, 3>{}, integral_constant<int, 4>{});
    case 16: return f(integral_constant<int, 4>{}, integral_constant<int, 4>{});
    case 18: return f(integral_constant<int, 3>{}, integral_constant<int, 6>{});
    case 20: return f(integral_constant<int, 4>{}, integral_constant<int, 5>{});
    case 21: return f(integral_constant<int, 3>{}, integral_constant<int, 7>{});
    case 24: return f(integral_constant<int, 4>{}, integral_constant<int, 6>{});
    case 25: return f(integral_constant<int, 5>{}, integral_constant<int, 5>{});
    case 27: return f(integral_constant<int, 3>{}, integral_constant<int, 9>{});
    case 28: return f(integral_constant<int, 4>{}, integral_constant<int, 7>{});
    case 30: return f(integral_constant<int, 5>{}, integral_constant<int, 6>{});
    case 32: return f(integral_constant<int, 4>{}, integral_constant<int, 8>{});
    case 35: return f(integral_constant<int, 5>{}, integral_constant<int, 7>{});
    case 36: return f(integral_constant<int, 6>{}, integral_constant<int, 6>{});
    case 40: return f(integral_constant<int, 5>{}, integral_constant<int, 8>{});
    case 42: return f(integral_constant<int, 6>{}, integral_constant<int, 7>{});
    case 45: return f(integral_constant<int, 5>{}, integral_constant<int, 9>{});
    case 48: return f(integral_constant<int, 6>{}, integral_constant<int, 8>{});
    case 49: return f(integral_constant<int, 7>{}, integral_constant<int, 7>{});
    case 50: return f(integral_constant<int, 5>{}, integral_constant<int, 10>{});
    case 54: return f(integral_constant<int, 6>{}, integral_constant<int, 9>{});
    case 56: return f(integral_constant<int, 7>{}, integral_constant<int, 8>{});
    case 60: return f(integral_constant<int, 6>{}, integral_constant<int, 10>{});
    case 63: return f(integral_constant<int, 7>{}, integral_constant<int, 9>{});
    case 64: return f(integral_constant<int, 8>{}, integral_constant<int, 8>{});
    case 70: return f(integral_constant<int, 7>{}, integral_constant<int, 10>{});
    case 72: return f(integral_constant<int, 8>{}, integral_constant<int, 9>{});
    case 75: return f(integral_constant<int, 5>{}, integral_constant<int, 15>{});
    case 80: return f(integral_constant<int, 8>{}, integral_constant<int, 10>{});
    case 81: return f(integral_constant<int, 9>{}, integral_constant<int, 9>{});
    case 84: return f(integral_constant<int, 7>{}, integral_constant<int, 12>{});
    case 90: return f(integral_constant<int, 9>{}, integral_constant<int, 10>{});
    case 96: return f(integral_constant<int, 8>{}, integral_constant<int, 12>{});
    case 98: return f(integral_constant<int, 7>{}, integral_constant<int, 14>{});
    case 100: return f(integral_constant<int, 10>{}, integral_constant<int, 10>{});
    case 105: return f(integral_constant<int, 7>{}, integral_constant<int, 15>{});
    case 108: return f(integral_constant<int, 9>{}, integral_constant<int, 12>{});
    case 112: return f(integral_constant<int, 8>{}, integral_constant<int, 14>{});
    case 120: return f(integral_constant<int, 10>{}, integral_constant<int, 12>{});
    case 126: return f(integral_constant<int, 9>{}, integral_constant<int, 14>{});
    case 128: return f(integral_constant<int, 8>{}, integral_constant<int, 16>{});
    case 135: return f(integral_constant<int, 9>{}, integral_constant<int, 15>{});
    case 140: return f(integral_constant<int, 10>{}, integral_constant<int, 14>{});
    case 144: return f(integral_constant<int, 12>{}, integral_constant<int, 12>{});
    case 150: return f(integral_constant<int, 10>{}, integral_constant<int, 15>{});
    case 160: return f(integral_constant<int, 10>{}, integral_constant<int, 16>{});
    case 192: return f(integral_constant<int, 12>{}, integral_constant<int, 16>{});
    case 200: return f(integral_constant<int, 10>{}, integral_constant<int, 20>{});
    case 240: return f(integral_constant<int, 15>{}, integral_constant<int, 16>{});
    case 256: return f(integral_constant<int, 16>{}, integral_constant<int, 16>{});
    default: break;
  }
  set_error("packed transforms: unsupported half length " + std::to_string(h));
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

}  // namespace

}  // namespace fcm

// fcm_packed.cuh -- layout, lengths and launch helpers of the Stokes solve on a packed half
// spectrum (fcm_packed_zy.cu: z and y passes, fcm_packed_x.cu: x passes, fcm_packed.cu: the
// choice among them).
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
// two columns of a pair lie nkb blocks apart.  Lengths: PACKED_LENGTHS.
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

// The sources of the passes are compiled once per precision and class of lengths (build.py):
// each object is a module of its own, which the driver loads when a context first needs it.
// As one module per source the first context of a process took 100 ms at 64^3 in FP64 and
// 110 ms at 256^3 in mixed precision instead of 15 and 40, and the library 79 s to build
// instead of 54.
constexpr int PACKED_CLASSES = 3;
constexpr int length_class(int n) { return n <= 96 ? 0 : n <= 216 ? 1 : 2; }

template <typename T, int CL>
int packed_zy_init();  // the tables of the module, before its first launch
template <typename T, int CL>
int packed_z_pass(const Ctx& c, typename cplx_t<T>::type* real, typename cplx_t<T>::type* spec, int members,
                  bool inverse, cudaStream_t s);
template <typename T, int CL>
int packed_y_pass(const Ctx& c, typename cplx_t<T>::type* spec, int members, bool inverse, cudaStream_t s);
template <typename T>
int packed_plane_pass(const Ctx& c, typename cplx_t<T>::type* real, typename cplx_t<T>::type* spec, int members,
                      bool inverse, cudaStream_t s);  // class 0
template <typename T, int CL>
int packed_x_init();
template <typename T, int CL>
int packed_x_pass(const Ctx& c, typename cplx_t<T>::type* spec, cudaStream_t s);
template <int CL>
int packed_noise_pass(const Ctx& c, cufftDoubleComplex* spec, uint64_t seed, uint64_t counter, const uint64_t* d_args,
                      cudaStream_t s);
template <typename T, int CL>
int b_packed_x_init();
template <typename T, int CL>
int b_packed_x_pass(const BatchGeom& b, const Ctx& c0, const int* gidx, int nm, int mask, cudaStream_t s);

// The bounds records of the modules, by 2 * class + (1 in FP32).
template <int ID>
int bounds_read_packed_zy(BoundsRecord* out, int reset);
template <int ID>
int bounds_read_packed_x(BoundsRecord* out, int reset);
template <int ID>
int bounds_read_b_packed_x(BoundsRecord* out, int reset);

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

// The lengths: the even numbers with factors 2, 3, 5 and 7 from 32 to 320 whose register DFT
// sizes stay within 20 points, and a few smaller and longer ones.  n1 n2 = n along x (whole
// tiles only) and y, h1 h2 = n / 2 along z.
struct PackedLength {
  int n, n1, n2, h1, h2;
};
constexpr PackedLength PACKED_LENGTHS[] = {
    {8, 2, 4, 2, 2}, {12, 3, 4, 2, 3}, {16, 4, 4, 2, 4}, {24, 4, 6, 3, 4}, {32, 4, 8, 4, 4}, {36, 6, 6, 3, 6},
    {40, 5, 8, 4, 5}, {42, 6, 7, 3, 7}, {48, 6, 8, 4, 6}, {50, 5, 10, 5, 5}, {54, 6, 9, 3, 9}, {56, 7, 8, 4, 7},
    {60, 6, 10, 5, 6}, {64, 8, 8, 4, 8}, {70, 7, 10, 5, 7}, {72, 8, 9, 6, 6}, {80, 8, 10, 5, 8}, {84, 7, 12, 6, 7},
    {90, 9, 10, 5, 9}, {96, 8, 12, 6, 8}, {98, 7, 14, 7, 7}, {100, 10, 10, 5, 10}, {108, 9, 12, 6, 9},
    {112, 8, 14, 7, 8}, {120, 10, 12, 6, 10}, {126, 9, 14, 7, 9}, {128, 8, 16, 8, 8}, {140, 10, 14, 7, 10},
    {144, 12, 12, 8, 9}, {150, 10, 15, 5, 15}, {160, 10, 16, 8, 10}, {162, 9, 18, 9, 9}, {168, 12, 14, 7, 12},
    {180, 12, 15, 9, 10}, {192, 12, 16, 8, 12}, {196, 14, 14, 7, 14}, {200, 10, 20, 10, 10}, {210, 14, 15, 7, 15},
    {216, 12, 18, 9, 12}, {224, 14, 16, 8, 14}, {240, 15, 16, 10, 12}, {252, 14, 18, 9, 14}, {256, 16, 16, 8, 16},
    {270, 15, 18, 9, 15}, {280, 14, 20, 10, 14}, {288, 16, 18, 12, 12}, {300, 15, 20, 10, 15},
    {320, 16, 20, 10, 16}, {384, 16, 24, 12, 16}, {400, 20, 20, 10, 20}, {480, 20, 24, 15, 16},
    {512, 16, 32, 16, 16}};
constexpr int NUM_PACKED_LENGTHS = sizeof(PACKED_LENGTHS) / sizeof(PACKED_LENGTHS[0]);

// Whether a length is taken along x: whole tiles.
constexpr bool x_length(int n) { return n % tile_x(n) == 0; }

// Calls f(integral_constant<I>) for the entry I of length n among those of class CL.
template <int CL, int I = 0, typename F>
int with_length(int n, F&& f) {
  if constexpr (I == NUM_PACKED_LENGTHS) {
    set_error("packed transforms: unsupported length " + std::to_string(n));
    return FCM_ERR_INVALID;
  } else {
    if constexpr (length_class(PACKED_LENGTHS[I].n) == CL)
      if (n == PACKED_LENGTHS[I].n) return f(std::integral_constant<int, I>{});
    return with_length<CL, I + 1>(n, f);
  }
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

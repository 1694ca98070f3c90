// fcm_dft.cuh -- complex pairs, wavenumbers and the in-register DFTs of the transform
// kernels (fcm_kspace.cu, fcm_packed_zy.cu, fcm_packed_x.cu).
#pragma once
#include <cmath>
#include <mutex>
#include <vector>

#include "fcm_internal.cuh"

namespace fcm {
namespace {

template <typename T>
struct alignas(2 * sizeof(T)) V2 {
  T x, y;
};

template <typename C>
__device__ __forceinline__ V2<double> ld(const C& v) {
  return V2<double>{(double)v.x, (double)v.y};
}

// Wavenumber of index i on an n-point grid (fcm_fluid_solver.cpp:77-91).
__device__ __forceinline__ double wavenumber(int i, int n, double fac) {
  return (i <= n / 2) ? (double)i * fac : (double)(i - n) * fac;
}

template <typename T, typename C>
__device__ __forceinline__ V2<T> ldt(const C& v) {
  return V2<T>{(T)v.x, (T)v.y};
}

// exp(-2 pi i k / n) for n = 96, 90 and 140 one after the other: every register DFT size
// divides one of them.
constexpr int W_SIZES[3] = {96, 90, 140};
constexpr int W_ALL = 96 + 90 + 140;
__constant__ static double2 c_wd[W_ALL];
__constant__ static float2 c_wf[W_ALL];

template <typename T>
__device__ __forceinline__ V2<T> w_at(int k);
template <>
__device__ __forceinline__ V2<double> w_at<double>(int k) {
  const double2 w = c_wd[k];
  return V2<double>{w.x, w.y};
}
template <>
__device__ __forceinline__ V2<float> w_at<float>(int k) {
  const float2 w = c_wf[k];
  return V2<float>{w.x, w.y};
}
// exp(-2 pi i k / R)
template <typename T, int R>
__device__ __forceinline__ V2<T> w_root(int k) {
  static_assert(96 % R == 0 || 90 % R == 0 || 140 % R == 0, "register DFT sizes divide 96, 90 or 140");
  if constexpr (96 % R == 0) return w_at<T>(k * (96 / R));
  if constexpr (90 % R == 0) return w_at<T>(96 + k * (90 / R));
  return w_at<T>(186 + k * (140 / R));
}

template <typename T>
__device__ __forceinline__ V2<T> cadd(V2<T> a, V2<T> b) { return V2<T>{a.x + b.x, a.y + b.y}; }
template <typename T>
__device__ __forceinline__ V2<T> csub(V2<T> a, V2<T> b) { return V2<T>{a.x - b.x, a.y - b.y}; }
template <typename T>
__device__ __forceinline__ V2<T> cmul(V2<T> a, V2<T> b) { return V2<T>{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
template <typename T>
__device__ __forceinline__ V2<T> cmulc(V2<T> a, V2<T> b) { return V2<T>{a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y}; }
// -i z (forward) or +i z (inverse)
template <typename T, bool INV>
__device__ __forceinline__ V2<T> rot(V2<T> z) { return INV ? V2<T>{-z.y, z.x} : V2<T>{z.y, -z.x}; }

// DFT of an odd prime R from its definition, the terms j and R - j taken together:
// X_k = a_0 + sum_j (a_j + a_(R-j)) cos(2 pi j k / R) -+ i (a_j - a_(R-j)) sin(2 pi j k / R).
template <typename T, int R, bool INV>
__device__ __forceinline__ void dft_prime(V2<T> (&a)[R], const T (&co)[R / 2], const T (&si)[R / 2]) {
  constexpr int H = R / 2;
  V2<T> t[H], d[H];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    t[j] = cadd(a[j + 1], a[R - 1 - j]);
    d[j] = rot<T, INV>(csub(a[j + 1], a[R - 1 - j]));
  }
  const V2<T> a0 = a[0];
#pragma unroll
  for (int j = 0; j < H; ++j) a[0] = cadd(a[0], t[j]);
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    V2<T> e = a0, o{(T)0, (T)0};
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      const int m = (j * k) % R;  // cos(2 pi m / R) = co[min(m, R - m) - 1], the sine odd
      const int q = m <= H ? m : R - m;
      const T c = co[q - 1], s = m <= H ? si[q - 1] : -si[q - 1];
      e.x += c * t[j - 1].x;
      e.y += c * t[j - 1].y;
      o.x += s * d[j - 1].x;
      o.y += s * d[j - 1].y;
    }
    a[k] = cadd(e, o);
    a[R - k] = csub(e, o);
  }
}

// In-register DFT of R points, R with factors 2, 3, 5 and 7: forward exp(-2 pi i n k / R),
// inverse exp(+2 pi i n k / R), unnormalised.  Decimation in time, R = P * Q.
template <typename T, int R, bool INV>
__device__ __forceinline__ void dft(V2<T> (&a)[R]) {
  if constexpr (R == 1) {
    return;
  } else if constexpr (R == 2) {
    const V2<T> t = a[1];
    a[1] = csub(a[0], t);
    a[0] = cadd(a[0], t);
  } else if constexpr (R == 5) {
    const T co[2] = {(T)0.30901699437494742410, (T)-0.80901699437494742410};
    const T si[2] = {(T)0.95105651629515357212, (T)0.58778525229247312917};
    dft_prime<T, 5, INV>(a, co, si);
  } else if constexpr (R == 7) {
    const T co[3] = {(T)0.62348980185873353053, (T)-0.22252093395631440429, (T)-0.90096886790241912624};
    const T si[3] = {(T)0.78183148246802980871, (T)0.97492791218182360702, (T)0.43388373911755812048};
    dft_prime<T, 7, INV>(a, co, si);
  } else if constexpr (R == 3) {
    // W_3 = -1/2 -+ i sqrt(3)/2
    const T h = (T)0.86602540378443864676;
    const V2<T> t1 = cadd(a[1], a[2]);
    const V2<T> t2 = V2<T>{a[0].x - (T)0.5 * t1.x, a[0].y - (T)0.5 * t1.y};
    const V2<T> d = rot<T, INV>(csub(a[1], a[2]));
    a[0] = cadd(a[0], t1);
    a[1] = V2<T>{t2.x + h * d.x, t2.y + h * d.y};
    a[2] = V2<T>{t2.x - h * d.x, t2.y - h * d.y};
  } else if constexpr (R == 4) {
    const V2<T> s0 = cadd(a[0], a[2]), s1 = csub(a[0], a[2]);
    const V2<T> s2 = cadd(a[1], a[3]), s3 = rot<T, INV>(csub(a[1], a[3]));
    a[0] = cadd(s0, s2);
    a[2] = csub(s0, s2);
    a[1] = cadd(s1, s3);
    a[3] = csub(s1, s3);
  } else {
    constexpr int P = (R % 4 == 0) ? 4 : ((R % 2 == 0) ? 2 : ((R % 3 == 0) ? 3 : 5));
    constexpr int Q = R / P;
    V2<T> b[P][Q];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int m = 0; m < Q; ++m) b[p][m] = a[P * m + p];
#pragma unroll
    for (int p = 0; p < P; ++p) dft<T, Q, INV>(b[p]);
#pragma unroll
    for (int p = 1; p < P; ++p)
#pragma unroll
      for (int m = 1; m < Q; ++m) {
        const int k = (p * m) % R;
        if (4 * k == R) {  // -i forward, +i inverse
          b[p][m] = rot<T, INV>(b[p][m]);
        } else {
          const V2<T> w = w_root<T, R>(k);
          b[p][m] = INV ? cmulc(b[p][m], w) : cmul(b[p][m], w);
        }
      }
#pragma unroll
    for (int m = 0; m < Q; ++m) {
      V2<T> c[P];
#pragma unroll
      for (int p = 0; p < P; ++p) c[p] = b[p][m];
      dft<T, P, INV>(c);
#pragma unroll
      for (int j = 0; j < P; ++j) a[m + Q * j] = c[j];
    }
  }
}

// The roots of unity into this translation unit's constant tables of the current device
// (once per device).
inline int roots_upload() {
  static std::mutex mu;
  static std::vector<bool> done;
  int dev = 0;
  FCM_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if ((int)done.size() <= dev) done.resize(dev + 1, false);
  if (done[dev]) return FCM_OK;
  const double PI = 3.14159265358979323846264338327950288;
  double2 wd[W_ALL];
  float2 wf[W_ALL];
  int at = 0;
  for (int n : W_SIZES)
    for (int j = 0; j < n; ++j, ++at) {
      wd[at] = make_double2(std::cos(2.0 * PI * j / n), -std::sin(2.0 * PI * j / n));
      wf[at] = make_float2((float)wd[at].x, (float)wd[at].y);
    }
  FCM_CUDA(cudaMemcpyToSymbol(c_wd, wd, sizeof(wd)));
  FCM_CUDA(cudaMemcpyToSymbol(c_wf, wf, sizeof(wf)));
  done[dev] = true;
  return FCM_OK;
}
}  // namespace
}  // namespace fcm

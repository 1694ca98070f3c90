// fcm_dft.cuh -- complex pairs, wavenumbers and the in-register DFTs of the transform
// kernels (fcm_kspace.cu, fcm_packed.cu).
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

__constant__ static double2 c_w96d[96];  // exp(-2 pi i k / 96)
__constant__ static float2 c_w96f[96];

template <typename T>
__device__ __forceinline__ V2<T> w96(int k);
template <>
__device__ __forceinline__ V2<double> w96<double>(int k) {
  const double2 w = c_w96d[k];
  return V2<double>{w.x, w.y};
}
template <>
__device__ __forceinline__ V2<float> w96<float>(int k) {
  const float2 w = c_w96f[k];
  return V2<float>{w.x, w.y};
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

// In-register DFT of R points, R a divisor of 96: forward exp(-2 pi i n k / R),
// inverse exp(+2 pi i n k / R), unnormalised.  Decimation in time, R = P * Q.
template <typename T, int R, bool INV>
__device__ __forceinline__ void dft(V2<T> (&a)[R]) {
  if constexpr (R == 1) {
    return;
  } else if constexpr (R == 2) {
    const V2<T> t = a[1];
    a[1] = csub(a[0], t);
    a[0] = cadd(a[0], t);
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
    constexpr int P = (R % 4 == 0) ? 4 : ((R % 2 == 0) ? 2 : 3);
    constexpr int Q = R / P;
    static_assert(96 % R == 0, "register DFT sizes divide 96");
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
        constexpr int S = 96 / R;
        const int k = ((p * m) % R) * S;
        if (k == 24) {  // W_4: -i forward, +i inverse
          b[p][m] = rot<T, INV>(b[p][m]);
        } else {
          const V2<T> w = w96<T>(k);
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

// exp(-2 pi i k / 96) into this translation unit's constant tables of the current
// device (once per device).
inline int w96_upload() {
  static std::mutex mu;
  static std::vector<bool> done;
  int dev = 0;
  FCM_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if ((int)done.size() <= dev) done.resize(dev + 1, false);
  if (done[dev]) return FCM_OK;
  const double PI = 3.14159265358979323846264338327950288;
  double2 wd[96];
  float2 wf[96];
  for (int j = 0; j < 96; ++j) {
    wd[j] = make_double2(std::cos(2.0 * PI * j / 96.0), -std::sin(2.0 * PI * j / 96.0));
    wf[j] = make_float2((float)wd[j].x, (float)wd[j].y);
  }
  FCM_CUDA(cudaMemcpyToSymbol(c_w96d, wd, sizeof(wd)));
  FCM_CUDA(cudaMemcpyToSymbol(c_w96f, wf, sizeof(wf)));
  done[dev] = true;
  return FCM_OK;
}

}  // namespace
}  // namespace fcm

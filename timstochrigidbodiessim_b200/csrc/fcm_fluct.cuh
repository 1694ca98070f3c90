// fcm_fluct.cuh -- the fluctuating stress drawn in Fourier space and its velocity, one mode
// at a time (fcm_kspace.cu, fcm_packed_x.cu).
#pragma once
#include "fcm_dft.cuh"
#include "fcm_internal.cuh"

namespace fcm {
namespace {

// Projection of one complex mode (re and im share the real factors).  The
// reference divides every component by eta*G; here one reciprocal of the
// mode's |q|^2 and a precomputed 1/(eta*G) are used instead (a last-bit change).
template <typename T>
__device__ __forceinline__ void project_mode(double q1, double q2, double q3, const V2<T> f[3], V2<T> u[3],
                                             T inv_etaG) {
  const T t1 = (T)q1, t2 = (T)q2, t3 = (T)q3;
  const T qq = (T)(q2 * q2) + (T)(q1 * q1) + (T)1e-16;
  const T norm = (T)1 / (qq + (T)(q3 * q3));
  const T kr = (t1 * f[0].x + t2 * f[1].x + t3 * f[2].x) * norm;
  const T ki = (t1 * f[0].y + t2 * f[1].y + t3 * f[2].y) * norm;
  const T sc = norm * inv_etaG;
  const T qv[3] = {t1, t2, t3};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    u[c].x = sc * (f[c].x - qv[c] * kr);
    u[c].y = sc * (f[c].y - qv[c] * ki);
  }
}

// f = i (q~ . sigma) for one mode; sigma order xx, yy, zz, xy, xz, yz.
template <typename T>
__device__ __forceinline__ void stress_divergence(double q1, double q2, double q3, const V2<T> s[6], V2<T> f[3]) {
  const T a = (T)q1, b = (T)q2, c = (T)q3;
  // (q.sigma)_x = q1 sxx + q2 sxy + q3 sxz, etc.; i*(r + i m) = -m + i r
  const T rx = a * s[0].x + b * s[3].x + c * s[4].x, mx = a * s[0].y + b * s[3].y + c * s[4].y;
  const T ry = a * s[3].x + b * s[1].x + c * s[5].x, my = a * s[3].y + b * s[1].y + c * s[5].y;
  const T rz = a * s[4].x + b * s[5].x + c * s[2].x, mz = a * s[4].y + b * s[5].y + c * s[2].y;
  f[0].x = -mx; f[0].y = rx;
  f[1].x = -my; f[1].y = ry;
  f[2].x = -mz; f[2].y = rz;
}

// Nyquist-zeroed wavenumbers of the stress divergence (fcm_fluid_solver.cpp:245-278).
__device__ __forceinline__ void divergence_q(int x, int y, int kz, const KParams& k, double& q1, double& q2,
                                             double& q3) {
  q1 = (x == k.nx / 2) ? 0.0 : wavenumber(x, k.nx, k.fx);
  q2 = (y == k.ny / 2) ? 0.0 : wavenumber(y, k.ny, k.fy);
  q3 = (kz == k.nzh - 1) ? 0.0 : (double)kz * k.fz;
}

// Two standard normals from two 32-bit words (Box-Muller, single precision).
__device__ __forceinline__ void box_muller(unsigned int a, unsigned int b, float& n1, float& n2) {
  const float u1 = ((float)a + 0.5f) * 2.3283064365386963e-10f;
  const float u2 = ((float)b + 0.5f) * 2.3283064365386963e-10f;
  const float r = sqrtf(-2.0f * logf(u1));
  float sn, cs;
  sincospif(2.0f * u2, &sn, &cs);
  n1 = r * cs;
  n2 = r * sn;
}

// Twelve normals for mode index m: three Philox blocks with counter
// (m, block, counter_lo, counter_hi), key (seed_lo, seed_hi).
__device__ __forceinline__ void mode_normals(unsigned long long m, uint64_t seed, uint64_t counter, float nrm[12]) {
  const uint2 key = make_uint2((unsigned int)seed, (unsigned int)(seed >> 32));
#pragma unroll
  for (int blk = 0; blk < 3; ++blk) {
    const uint4 r = philox4x32_10(make_uint4((unsigned int)m, (unsigned int)blk, (unsigned int)counter,
                                             (unsigned int)(counter >> 32)), key);
    box_muller(r.x, r.y, nrm[4 * blk], nrm[4 * blk + 1]);
    box_muller(r.z, r.w, nrm[4 * blk + 2], nrm[4 * blk + 3]);
  }
}

// Velocity of the fluctuating stress at mode (x, y, kz), 0 <= kz <= nz/2, as the inverse
// transform takes it: in the Hermitian planes the mean over {k, -k} (see fcm_kspace.cu).
// For white real-space noise of variance v^2 per point, the unnormalised DFT has
// E|s(k)|^2 = G v^2, independent real and imaginary parts of variance G v^2/2 for
// k != -k, a real value of variance G v^2 for self-conjugate k, and s(-k) = conj(s(k));
// the Fourier-space draw reproduces exactly that law.  Of a pair {k, -k} the mode with the
// smaller index is drawn, the other is its conjugate.
template <typename T>
__device__ __forceinline__ void fluct_velocity(int x, int y, int kz, const KParams& k, uint64_t seed, uint64_t counter,
                                               double amp_diag, double amp_off, V2<T> (&u)[3]) {
  const bool plane = kz == 0 || 2 * kz == k.nz;
  int xp = x, yp = y;
  bool conj_of = false;
  if (plane) {
    xp = x ? k.nx - x : 0;
    yp = y ? k.ny - y : 0;
    if ((long long)xp * k.ny + yp < (long long)x * k.ny + y) {
      const int tx = x, ty = y;
      x = xp;
      y = yp;
      xp = tx;
      yp = ty;
      conj_of = true;
    }
  }
  if (x == 0 && y == 0 && kz == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = V2<T>{(T)0, (T)0};
    return;
  }
  const bool self = plane && xp == x && yp == y;
  V2<T> s[6];
  if (k.slip) {
    // Image-symmetric stress of a slip channel (fcm_fluid_solver.cpp:186-217): xx, yy,
    // zz, xz even in y, xy and yz odd, the even ones with twice the variance on the
    // wall rows 0 and ny/2 and the odd ones zero there.  Its DFT along y is real
    // and even (odd: imaginary and odd) with independent rows ky = 0..ny/2, those of
    // the even components of variance ny v^2 (2 ny v^2 on ky = 0, ny/2), those of
    // the odd ones ny v^2 (0 on ky = 0, ny/2).  So row y takes the draw of row
    // yr = min(y, ny - y): even components a white (x, z) spectrum of variance
    // G v^2 (doubled on the wall rows), odd ones -i times one (zero on the wall
    // rows), negated for y > ny/2.  In the kz = 0 and nz/2 planes (x, yr) pairs
    // with (-x, yr) as the 2D spectrum of a real field.
    const int h = k.ny / 2;
    const int yr = y <= h ? y : k.ny - y;
    const bool wall = yr == 0 || yr == h;
    const int xm = (k.nx - x) % k.nx;
    const int xr = (plane && xm < x) ? xm : x;
    const bool cj = xr != x, xself = plane && xm == x;
    float nrm[12];
    mode_normals((unsigned long long)(((long long)xr * k.ny + yr) * k.nzh + kz), seed, counter, nrm);
    for (int c = 0; c < 6; ++c) {
      const double amp = (c < 3) ? amp_diag : amp_off;  // order xx, yy, zz, xy, xz, yz
      double re, im;
      if (xself) {
        re = amp * 1.4142135623730951 * (double)nrm[2 * c];
        im = 0.0;
      } else {
        re = amp * (double)nrm[2 * c];
        im = amp * (double)nrm[2 * c + 1];
      }
      if (cj) im = -im;
      if (c == 3 || c == 5) {  // odd: -i (re + i im), zero on the walls, negated above ny/2
        const double sg = wall ? 0.0 : (y > h ? -1.0 : 1.0);
        const double r2 = sg * im, i2 = -sg * re;
        re = r2;
        im = i2;
      } else if (wall) {
        re *= 1.4142135623730951;
        im *= 1.4142135623730951;
      }
      s[c].x = (T)re;
      s[c].y = (T)im;
    }
  } else {
    float nrm[12];
    mode_normals((unsigned long long)(((long long)x * k.ny + y) * k.nzh + kz), seed, counter, nrm);
    for (int c = 0; c < 6; ++c) {
      const double amp = (c < 3) ? amp_diag : amp_off;
      if (self) {
        s[c].x = (T)(amp * 1.4142135623730951 * (double)nrm[2 * c]);
        s[c].y = 0;
      } else {
        s[c].x = (T)(amp * (double)nrm[2 * c]);
        s[c].y = (T)(amp * (double)nrm[2 * c + 1]);
      }
    }
  }
  const T ie = (T)k.inv_etaG;
  double q1, q2, q3;
  divergence_q(x, y, kz, k, q1, q2, q3);
  V2<T> f[3];
  stress_divergence<T>(q1, q2, q3, s, f);
  const double r3 = (double)kz * k.fz;
  project_mode<T>(wavenumber(x, k.nx, k.fx), wavenumber(y, k.ny, k.fy), r3, f, u, ie);
  if (!plane) return;
  if (self) {
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c].y = 0;
    return;
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) s[c].y = -s[c].y;
  divergence_q(xp, yp, kz, k, q1, q2, q3);
  stress_divergence<T>(q1, q2, q3, s, f);
  V2<T> up[3];
  project_mode<T>(wavenumber(xp, k.nx, k.fx), wavenumber(yp, k.ny, k.fy), r3, f, up, ie);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    u[c].x = (T)0.5 * (u[c].x + up[c].x);
    u[c].y = (T)0.5 * (u[c].y - up[c].y);
    if (conj_of) u[c].y = -u[c].y;
  }
}

}  // namespace
}  // namespace fcm

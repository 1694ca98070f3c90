// fcm_rigid.cuh -- rotations and the rigid-body operators K and K^T of one blob or
// body, shared by the rigid-body kernels (fcm_bodies.cu) and the fused end of the
// saddle-point product (fcm_grid.cu).
#pragma once
#include "fcm_internal.cuh"

namespace fcm {
namespace {

// quaternion.cpp:61-103 with round-to-nearest intrinsics, so the product order
// (and therefore every bit) matches a non-contracting CPU build.
__device__ __forceinline__ void quat_matrix(const double* q, double R[3][3]) {
  const double s = q[0], v0 = q[1], v1 = q[2], v2 = q[3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) R[i][j] = (i == j) ? 1.0 : 0.0;
  double t = __dmul_rn(__dmul_rn(2.0, v0), v0);
  R[1][1] = __dsub_rn(R[1][1], t); R[2][2] = __dsub_rn(R[2][2], t);
  t = __dmul_rn(__dmul_rn(2.0, v1), v1);
  R[0][0] = __dsub_rn(R[0][0], t); R[2][2] = __dsub_rn(R[2][2], t);
  t = __dmul_rn(__dmul_rn(2.0, v2), v2);
  R[0][0] = __dsub_rn(R[0][0], t); R[1][1] = __dsub_rn(R[1][1], t);
  t = __dmul_rn(__dmul_rn(2.0, v0), v1);
  R[1][0] = __dadd_rn(R[1][0], t); R[0][1] = __dadd_rn(R[0][1], t);
  t = __dmul_rn(__dmul_rn(2.0, v0), v2);
  R[2][0] = __dadd_rn(R[2][0], t); R[0][2] = __dadd_rn(R[0][2], t);
  t = __dmul_rn(__dmul_rn(2.0, v1), v2);
  R[1][2] = __dadd_rn(R[1][2], t); R[2][1] = __dadd_rn(R[2][1], t);
  t = __dmul_rn(__dmul_rn(2.0, s), v2);
  R[1][0] = __dadd_rn(R[1][0], t); R[0][1] = __dsub_rn(R[0][1], t);
  t = __dmul_rn(__dmul_rn(2.0, s), v1);
  R[2][0] = __dsub_rn(R[2][0], t); R[0][2] = __dadd_rn(R[0][2], t);
  t = __dmul_rn(__dmul_rn(2.0, s), v0);
  R[2][1] = __dadd_rn(R[2][1], t); R[1][2] = __dsub_rn(R[1][2], t);
}

__device__ __forceinline__ void rot(const double R[3][3], const double* v, double* o) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
    o[i] = __dadd_rn(__dadd_rn(__dmul_rn(R[i][0], v[0]), __dmul_rn(R[i][1], v[1])), __dmul_rn(R[i][2], v[2]));
}
__device__ __forceinline__ void rotT(const double R[3][3], const double* v, double* o) {
#pragma unroll
  for (int i = 0; i < 3; ++i) o[i] = R[0][i] * v[0] + R[1][i] * v[1] + R[2][i] * v[2];
}
__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

// U + Omega x (R r_m) of blob i (collection_of_rigid_bodies.cpp:707-731).
__device__ __forceinline__ void blob_K_velocity(const double* __restrict__ q, const double* __restrict__ ref, int rs,
                                                const double* __restrict__ in, int i, int nb, double v[3]) {
  const int n = i / nb, m = i - n * nb;
  double R[3][3];
  quat_matrix(q + 4 * n, R);
  double r[3], c[3];
  rot(R, ref + (size_t)n * rs + 3 * m, r);
  cross3(in + 6 * n + 3, r, c);
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] = in[6 * n + d] + c[d];
}

// collection_of_rigid_bodies.cpp:707-731: out_m (+)= U + Omega x (R r_m).
__device__ __forceinline__ void multiply_K_one(const double* __restrict__ q, const double* __restrict__ ref, int rs,
                                               const double* __restrict__ in, double* __restrict__ out, int i,
                                               int nb, int subtract) {
  double v[3];
  blob_K_velocity(q, ref, rs, in, i, nb, v);
#pragma unroll
  for (int d = 0; d < 3; ++d) out[3 * i + d] = subtract ? out[3 * i + d] - v[d] : v[d];
}

// collection_of_rigid_bodies.cpp:733-757: F = sum lambda_m, T = sum (R r_m) x lambda_m;
// out = scale * K^T in + add_scale * add.
__device__ __forceinline__ void multiply_KT_one(const double* __restrict__ q, const double* __restrict__ ref, int rs,
                                                const double* __restrict__ in, double* __restrict__ out, int n,
                                                int nb, double scale, const double* __restrict__ add,
                                                double add_scale) {
  double R[3][3];
  quat_matrix(q + 4 * n, R);
  ref += (size_t)n * rs;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int m = 0; m < nb; ++m) {
    const double* l = in + 3 * (n * nb + m);
    double r[3], c[3];
    rot(R, ref + 3 * m, r);
    cross3(r, l, c);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      acc[d] += l[d];
      acc[3 + d] += c[d];
    }
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) out[6 * n + d] = scale * acc[d] + (add ? add_scale * add[6 * n + d] : 0.0);
}

}  // namespace
}  // namespace fcm

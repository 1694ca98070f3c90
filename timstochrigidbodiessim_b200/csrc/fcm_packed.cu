// fcm_packed.cu -- the Stokes solve on a packed half spectrum: the grids that have it and the
// passes of each (fcm_packed_zy.cu, fcm_packed_x.cu) by the classes of its lengths.
#include "fcm_packed.cuh"

namespace fcm {

namespace {

// Calls f(integral_constant<CL>) for the class of length n.
template <typename F>
int with_class(int n, F&& f) {
  static_assert(PACKED_CLASSES == 3, "a case per class");
  switch (length_class(n)) {
    case 0: return f(std::integral_constant<int, 0>{});
    case 1: return f(std::integral_constant<int, 1>{});
    default: return f(std::integral_constant<int, 2>{});
  }
}

template <typename T>
int z_pass(const Ctx& c, typename cplx_t<T>::type* real, typename cplx_t<T>::type* spec, int members, bool inverse,
           cudaStream_t s) {
  return with_class(c.g.nz, [&](auto cl) {
    return packed_z_pass<T, decltype(cl)::value>(c, real, spec, members, inverse, s);
  });
}
template <typename T>
int y_pass(const Ctx& c, typename cplx_t<T>::type* spec, int members, bool inverse, cudaStream_t s) {
  return with_class(c.g.ny,
                    [&](auto cl) { return packed_y_pass<T, decltype(cl)::value>(c, spec, members, inverse, s); });
}

template <typename T>
int tables_init(const Ctx& c) {
  for (int n : {c.g.ny, c.g.nz})
    FCM_TRY(with_class(n, [](auto cl) { return packed_zy_init<T, decltype(cl)::value>(); }));
  return with_class(c.g.nx, [](auto cl) { return packed_x_init<T, decltype(cl)::value>(); });
}

// Square (y, z) planes up to 96 points take the per-plane kernels (39 KB of shared memory
// at 96 points in FP32, 75 KB in FP64).
bool plane_ok(const Ctx& c) { return c.g.ny == c.g.nz && c.g.nz >= 16 && c.g.nz <= 96; }

}  // namespace

bool packed_lengths(int nx, int ny, int nz) {
  if (!x_length(nx)) return false;
  auto listed = [](int n) {
    for (const PackedLength& l : PACKED_LENGTHS)
      if (l.n == n) return true;
    return false;
  };
  return listed(nx) && listed(ny) && listed(nz);
}

// Whether the FP64 fluctuating field is drawn in the x pass of the packed spectrum.  From 140
// points along x on, a CTA's draws take 25-45 us however few CTAs there are (a tile's
// columns of one row each), so slender boxes of less than one and a half CTAs per SM draw the
// whole half spectrum and take cuFFT's transform (us of a field, cuFFT / packed: 512 x 8 x 8 23
// / 43, 400 x 24 x 24 29 / 42, 200 x 24 x 24 24 / 30; 240 x 32 x 32 (128 CTAs) 30 / 32, 320 x 32 x 32 (256)
// 35 / 31, 160 x 42 x 42 (252) 30 / 29, 256 x 40 x 40 (400) 38 / 26).
bool packed_noise(const Ctx& c) {
  if (!c.packed_cap) return false;
  const int tk = 8 / tile_x(c.g.nx), pairs = (c.g.nz / 2 + 1) / 2;
  const long long ctas = (long long)((pairs + tk - 1) / tk) * c.g.ny;
  return c.g.nx < 140 || 2 * ctas >= 3 * 148;
}

int packed_tables_init(const Ctx& c) {
  FCM_TRY(tables_init<double>(c));
  return c.p.precision == 1 ? tables_init<float>(c) : (int)FCM_OK;
}

// The (y, z) transforms of `members` consecutive grids of c's shape: forward from the
// real grid r into the packed spectrum, inverse from the spectrum (overwritten) into r.
template <typename T>
int launch_packed_forward(const Ctx& c, const T* r, typename cplx_t<T>::type* spec, int members, cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  C* real = reinterpret_cast<C*>(const_cast<T*>(r));  // read only in this direction
  if (plane_ok(c)) return packed_plane_pass<T>(c, real, spec, members, false, s);
  FCM_TRY(z_pass<T>(c, real, spec, members, false, s));
  return y_pass<T>(c, spec, members, false, s);
}

template <typename T>
int launch_packed_inverse(const Ctx& c, typename cplx_t<T>::type* spec, T* r, int members, cudaStream_t s) {
  using C = typename cplx_t<T>::type;
  C* real = reinterpret_cast<C*>(r);
  if (plane_ok(c)) return packed_plane_pass<T>(c, real, spec, members, true, s);
  FCM_TRY(y_pass<T>(c, spec, members, true, s));
  return z_pass<T>(c, real, spec, members, true, s);
}

template <typename T>
int launch_packed_project(const Ctx& c, typename cplx_t<T>::type* spec, cudaStream_t s) {
  return with_class(c.g.nx, [&](auto cl) { return packed_x_pass<T, decltype(cl)::value>(c, spec, s); });
}

// The fluctuating velocity field of (seed, counter), or d_args[0..1] where given, into r.
int launch_packed_noise(const Ctx& c, cufftDoubleComplex* spec, double* r, uint64_t seed, uint64_t counter,
                        const uint64_t* d_args, cudaStream_t s) {
  FCM_TRY(with_class(
      c.g.nx, [&](auto cl) { return packed_noise_pass<decltype(cl)::value>(c, spec, seed, counter, d_args, s); }));
  return launch_packed_inverse<double>(c, spec, r, 1, s);
}

template <typename T>
int b_packed_init(const Ctx& c0) {
  return with_class(c0.g.nx, [](auto cl) { return b_packed_x_init<T, decltype(cl)::value>(); });
}

template <typename T>
int b_packed_project(const BatchGeom& b, const Ctx& c0, const int* gidx, int nm, int mask, cudaStream_t s) {
  return with_class(c0.g.nx,
                    [&](auto cl) { return b_packed_x_pass<T, decltype(cl)::value>(b, c0, gidx, nm, mask, s); });
}

template <typename T>
long long packed_spectrum_size(const Ctx& c) {
  using C = typename cplx_t<T>::type;
  return tile_x(c.g.nx) == 8 ? Tiles<C, 8>(c.g.nx, c.g.ny, c.g.nz).size()
                             : Tiles<C, 4>(c.g.nx, c.g.ny, c.g.nz).size();
}

int bounds_read_packed(BoundsRecord* out, int reset) {
  int (*const readers[])(BoundsRecord*, int) = {
      bounds_read_packed_zy<0>,  bounds_read_packed_zy<1>,  bounds_read_packed_zy<2>,  bounds_read_packed_zy<3>,
      bounds_read_packed_zy<4>,  bounds_read_packed_zy<5>,  bounds_read_packed_x<0>,   bounds_read_packed_x<1>,
      bounds_read_packed_x<2>,   bounds_read_packed_x<3>,   bounds_read_packed_x<4>,   bounds_read_packed_x<5>,
      bounds_read_b_packed_x<0>, bounds_read_b_packed_x<1>, bounds_read_b_packed_x<2>, bounds_read_b_packed_x<3>,
      bounds_read_b_packed_x<4>, bounds_read_b_packed_x<5>};
  *out = BoundsRecord{};
  for (auto rd : readers) {
    BoundsRecord r{};
    FCM_TRY(rd(&r, reset));
    if (!out->count) *out = r;
    else out->count += r.count;
  }
  return FCM_OK;
}

template long long packed_spectrum_size<double>(const Ctx&);
template long long packed_spectrum_size<float>(const Ctx&);
template int launch_packed_forward<double>(const Ctx&, const double*, cufftDoubleComplex*, int, cudaStream_t);
template int launch_packed_forward<float>(const Ctx&, const float*, cufftComplex*, int, cudaStream_t);
template int launch_packed_inverse<double>(const Ctx&, cufftDoubleComplex*, double*, int, cudaStream_t);
template int launch_packed_inverse<float>(const Ctx&, cufftComplex*, float*, int, cudaStream_t);
template int launch_packed_project<double>(const Ctx&, cufftDoubleComplex*, cudaStream_t);
template int launch_packed_project<float>(const Ctx&, cufftComplex*, cudaStream_t);
template int b_packed_init<double>(const Ctx&);
template int b_packed_init<float>(const Ctx&);
template int b_packed_project<double>(const BatchGeom&, const Ctx&, const int*, int, int, cudaStream_t);
template int b_packed_project<float>(const BatchGeom&, const Ctx&, const int*, int, int, cudaStream_t);

}  // namespace fcm

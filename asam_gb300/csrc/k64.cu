// FP64 kernels, compiled with -fmad=false: every product and sum is rounded
// separately, as in the reference Fortran built without FMA contraction.
#include "launchers_impl.cuh"

ASAM_DEFINE_LAUNCHERS(double, double)

namespace {
__global__ void k_cvt_d2f(size_t len, const double* __restrict__ x, float* __restrict__ y) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < len; q += (size_t)gridDim.x * blockDim.x)
    y[q] = (float)x[q];
}
__global__ void k_cvt_f2d(size_t len, const float* __restrict__ x, double* __restrict__ y) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < len; q += (size_t)gridDim.x * blockDim.x)
    y[q] = (double)x[q];
}
// y += s * x widened to FP64 (the refinement's correction, one pass).  The
// conversion and the product run on the integer units; on the FP64 unit they took
// twice the time of the memory traffic (256x256x128, 10 components: 506 us, set 503).
__global__ void k_add_f2d(size_t len, const float* __restrict__ x, double s, double* __restrict__ y) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < len; q += (size_t)gridDim.x * blockDim.x)
    y[q] = y[q] + fpi::mul_rn(s, fpi::widen(x[q]));
}
// (float)(s * x): the residual handed to the FP32 inner solver, scaled to
// unit norm so that neither tiny nor huge residuals leave the FP32 range; into
// the inner solver's residual, shadow residual and search direction
__global__ void k_cvt_d2f_scaled3(size_t len, const double* __restrict__ x, double s, float* __restrict__ y0,
                                  float* __restrict__ y1, float* __restrict__ y2) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < len; q += (size_t)gridDim.x * blockDim.x) {
    const float v = fpi::narrow(fpi::mul_rn(s, x[q]));
    y0[q] = v;
    y1[q] = v;
    y2[q] = v;
  }
}
// y = 0 + s * x: k_add_f2d on a zero y
__global__ void k_set_f2d(size_t len, const float* __restrict__ x, double s, double* __restrict__ y) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < len; q += (size_t)gridDim.x * blockDim.x) {
    const double v = fpi::mul_rn(s, fpi::widen(x[q]));
    y[q] = (__double_as_longlong(v) << 1) == 0 ? 0.0 : v;  // 0 + -0
  }
}
// out = s*base (base itself unless kScale), then out = a_j x_j + out for every
// term: a stage's right-hand side or state in one pass over its arrays instead
// of a copy or a scaling and a pass per term, with the same roundings.  Bound by
// HBM: the number of terms is a template parameter so that a thread has the
// loads of all terms and of two elements in flight.
struct LinTerms {
  int n;
  double a[4];
  const double* x[4];
};
template <int kN, bool kScale>
__global__ void k_lincomb(size_t len, LinTerms t, const double* base, double s, double* out) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < len; q += 2 * stride) {
    const size_t p = q + stride;
    const bool two = p < len;
    double v = base[q], w = two ? base[p] : 0.0, xv[kN + 1], xw[kN + 1];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      xv[j] = t.x[j][q];
      xw[j] = two ? t.x[j][p] : 0.0;
    }
    if (kScale) v = s * v, w = s * w;
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      v = t.a[j] * xv[j] + v;
      w = t.a[j] * xw[j] + w;
    }
    out[q] = v;
    if (two) out[p] = w;
  }
}
template <bool kScale>
void run_lincomb(const asam::Launch& L, size_t len, const LinTerms& t, const double* base, double s, double* out) {
  const int g = gs_grid(L, (len + 1) / 2);
  switch (t.n) {
    case 0: k_lincomb<0, kScale><<<g, kBlock, 0, L.stream>>>(len, t, base, s, out); break;
    case 1: k_lincomb<1, kScale><<<g, kBlock, 0, L.stream>>>(len, t, base, s, out); break;
    case 2: k_lincomb<2, kScale><<<g, kBlock, 0, L.stream>>>(len, t, base, s, out); break;
    case 3: k_lincomb<3, kScale><<<g, kBlock, 0, L.stream>>>(len, t, base, s, out); break;
    default: k_lincomb<4, kScale><<<g, kBlock, 0, L.stream>>>(len, t, base, s, out);
  }
}
// slots 7 and 8 of the DIA storage: 1/diagonal (correctly rounded) and its
// 64-bit reciprocal
__global__ void k_recip_diag(size_t n, double* __restrict__ val) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
  {
    const double dg = val[3 * n + q];
    const unsigned long long R = fpi::recip(dg);
    val[7 * n + q] = fpi::quot_rn(1.0, dg, R);
    val[8 * n + q] = __longlong_as_double((long long)R);
  }
}
}  // namespace

namespace asam {
void launch_beta(const Launch& L, KrylovScalars* sc) {
  k_beta<<<1, 1, 0, L.stream>>>(sc);
  count_launches(1);
}
void launch_mass(const Launch& L, const Dims& d, const double* c, const double* volc, double* partial, double* out) {
  k_mass_partial<<<RED_GRID, RED_BLOCK, 0, L.stream>>>(d, c, volc, partial);
  k_dot_final<<<1, RED_BLOCK, 0, L.stream>>>(partial, RED_GRID, nullptr, -1, out);
  count_launches(2);
}
void launch_recip_diag(const Launch& L, size_t npad, double* val) {
  k_recip_diag<<<gs_grid(L, npad), kBlock, 0, L.stream>>>(npad, val);
  count_launches(1);
}
void launch_convert_f64_to_f32(const Launch& L, size_t len, const double* x, float* y) {
  k_cvt_d2f<<<gs_grid(L, len), kBlock, 0, L.stream>>>(len, x, y);
  count_launches(1);
}
void launch_add_f32_to_f64(const Launch& L, size_t len, const float* x, double s, double* y) {
  k_add_f2d<<<gs_grid(L, len), kBlock, 0, L.stream>>>(len, x, s, y);
  count_launches(1);
}
void launch_convert_f64_to_f32_scaled3(const Launch& L, size_t len, const double* x, double s, float* y0, float* y1,
                                       float* y2) {
  k_cvt_d2f_scaled3<<<gs_grid(L, len), kBlock, 0, L.stream>>>(len, x, s, y0, y1, y2);
  count_launches(1);
}
void launch_set_f32_to_f64(const Launch& L, size_t len, const float* x, double s, double* y) {
  k_set_f2d<<<gs_grid(L, len), kBlock, 0, L.stream>>>(len, x, s, y);
  count_launches(1);
}
void launch_lincomb(const Launch& L, size_t len, const double* base, const double* scale, int nterm, const double* a,
                    const double* x, double* out) {
  LinTerms t{};
  for (int j = 0; j < nterm; ++j)
    if (a[j] != 0.0) {
      t.a[t.n] = a[j];
      t.x[t.n++] = x + (size_t)j * len;
    }
  if (scale)
    run_lincomb<true>(L, len, t, base, *scale, out);
  else
    run_lincomb<false>(L, len, t, base, 1.0, out);
  count_launches(1);
}
void launch_resid_dot(const Launch& L, const Dims& d, int ncomp, const double* val, const double* x, const double* b,
                      double* r, double* partial, KrylovScalars* sc, int op, double* out) {
  k_resid_dot<double><<<RED_GRID, RED_BLOCK, 0, L.stream>>>(d, ncomp, val, x, b, r, partial);
  k_dot_final<<<1, RED_BLOCK, 0, L.stream>>>(partial, RED_GRID, sc, op, out);
  count_launches(2);
}
void launch_convert_f32_to_f64(const Launch& L, size_t len, const float* x, double* y) {
  k_cvt_f2d<<<gs_grid(L, len), kBlock, 0, L.stream>>>(len, x, y);
  count_launches(1);
}
}  // namespace asam

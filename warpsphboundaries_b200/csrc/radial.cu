// Solid half-spaces and solid spheres in 3-D: the nine axial invariants of the kernel integrals over the part of a
// query's support that lies inside the solid, and their rotation into Cartesian channels (the 28 baseline requests
// |alpha| + |derivative| <= 2, or any subset).
//
// Reference: src/warpSPHBoundaries/fluxbridge/radial.py:20-71 (functions: element + select + batch) and the native
// element of src/warpSPHBoundaries/fluxbridge/_radial_code.py:43-148.  The invariants are the shell integrals of
// fluxbridge/radial_reference.py:17-56: at radius r the support sphere meets the solid in a spherical cap mu >= cap
// along the inward axis (cap = -d/r for a half-space, (R^2 - D^2 - r^2) / (2 D r) with D = R + d for a sphere of
// radius R whose surface is at signed distance d), and integrating the monomials over the cap gives
//   a0 = 2 pi (1 + cap), a1 = pi (cap^2 - 1), at = pi (cap - cap^3/3 + 2/3), an = 2 pi (cap^3 + 1) / 3.
// The reference integrates products of linear factors in Bernstein form; here each radial sub-interval (per kernel
// piece: the full-ball region [0, min(1, -d)] and the cap region [|d|, min(1, 2R + d)]) is integrated by the
// Gauss-Legendre rule that is exact for its polynomial integrands (w2 7 nodes in the cap region, w4 8, w6 10; 12 nodes
// leave < 1e-17 relative on cubic's outer Laurent piece, r >= 1/2; float32 takes 12 throughout).  Cancellation is avoided
// by factoring the angular terms, with the factor r kept inside so that no node divides:
//   ru = r (1 + cap) = (r - d)(2R + d - r) / (2 D),  rv = r (1 - cap) = (r + d)(r + d + 2R) / (2 D)   (sphere)
//   ru = r - d,                                      rv = r + d                                       (half-space)
//   r a0 = 2 ru, r^2 a1 = -ru rv, r^3 at = ru^2 (r + rv) / 3, r^3 an = 2/3 ru (rc^2 - r rc + r^2), rc = r cap
//   (times pi; pi cancels against W)
// and the kernel profiles W, W'/r and (W'/r)' are evaluated as r^p (hi - r)^k g(r) with exact factors.
#include "common.cuh"


namespace wsb {
namespace {

struct RadialRequests {            // up to 28 requests: degree, i, j, order (reference metadata, radial.py:124-128)
  int n;
  signed char meta[28][4];
};

template <typename T>
struct Inv9 {
  T v[9];
};

// nodes of a region: those that are exact for it in float64; in float32 always 12, over which the roundings of the profile's
// values average out (with 7 to 10 the error of w4 and w6 is 1.1 to 1.2 times as large)
template <typename T>
constexpr int radial_nodes(int exact) {
  return sizeof(T) == 4 ? 12 : exact;
}

// one piece's contribution: the full-ball region [lo, hi] (cap = 1) and the cap region [clo, chi]
template <class KR, int P, typename T>
__device__ __forceinline__ void radial_piece(T d, T R, T inv2D, bool sphere, T full_end, T cap_end, Inv9<T>& acc) {
  const T plo = T(KR::kLo[P]), phi = T(KR::kHi[P]);
  {
    constexpr int N = radial_nodes<T>(KR::kBall[P]);
    const T lo = plo, hi = fmin(phi, full_end);
    if (hi > lo) {
      const T c = T(0.5) * (hi + lo), hw = T(0.5) * (hi - lo);
      T s0 = 0, s2 = 0, s5 = 0, s7 = 0;
#pragma unroll
      for (int g = 0; g < N; ++g) {
        const T r = fma_t(hw, T(radial_gx<N>(g)), c), wg = T(radial_gw<N>(g));
        T w, l, dl;
        KR::template eval<P, T>(r, w, l, dl);
        const T r2 = wg * r * r, r3 = r2 * r, r4 = r3 * r;
        s0 = fma_t(r2, w, s0);
        s2 = fma_t(r4, w, s2);
        s5 = fma_t(r4, l, s5);
        s7 = fma_t(T(4) * r2, l, fma_t(T(4.0 / 3.0) * r3, dl, s7));
      }
      acc.v[0] += hw * T(4) * s0;
      acc.v[2] += hw * T(4.0 / 3.0) * s2;
      acc.v[3] += hw * T(4.0 / 3.0) * s2;
      acc.v[5] -= hw * T(4.0 / 3.0) * s5;
      acc.v[6] -= hw * T(4.0 / 3.0) * s5;
      acc.v[7] += hw * s7;
      acc.v[8] += hw * s7;
    }
  }
  {
    constexpr int N = radial_nodes<T>(KR::kCap[P]);
    const T lo = fmax(plo, fabs(d)), hi = fmin(phi, cap_end);
    if (hi > lo) {
      const T c = T(0.5) * (hi + lo), hw = T(0.5) * (hi - lo);
      T s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int g = 0; g < N; ++g) {
        const T r = fma_t(hw, T(radial_gx<N>(g)), c), wg = T(radial_gw<N>(g));
        T w, l, dl;
        KR::template eval<P, T>(r, w, l, dl);
        T ru = r - d, rv = r + d;
        if (sphere) {
          ru *= ((R - r) + (R + d)) * inv2D;
          rv *= (rv + T(2) * R) * inv2D;
        }
        const T rc = T(0.5) * (ru - rv), a1 = ru * rv, at = ru * ru * (r + rv), an = ru * fma_t(rc, rc - r, r * r);
        const T wr = wg * r, ww = wr * w, wl = wr * l, lu = wl * ru, wd = wg * T(1.0 / 6.0) * dl;
        s[0] = fma_t(ww, ru, s[0]);
        s[1] = fma_t(ww, a1, s[1]);
        s[2] = fma_t(ww, at, s[2]);
        s[3] = fma_t(ww, an, s[3]);
        s[4] = fma_t(wl, a1, s[4]);
        s[5] = fma_t(wl, at, s[5]);
        s[6] = fma_t(wl, an, s[6]);
        // (the Hessian's two terms cancel: they are combined at the node, not in sums of their own)
        s[7] += fma_t(wd, at, lu);
        s[8] += fma_t(T(2) * wd, an, lu);
      }
      const T h3 = hw * T(1.0 / 3.0);
      acc.v[0] += T(2) * hw * s[0];
      acc.v[1] -= hw * s[1];
      acc.v[2] += h3 * s[2];
      acc.v[3] += T(2) * h3 * s[3];
      acc.v[4] += hw * s[4];
      acc.v[5] -= h3 * s[5];
      acc.v[6] -= T(2) * h3 * s[6];
      acc.v[7] += T(2) * hw * s[7];
      acc.v[8] += T(2) * hw * s[8];
    }
  }
}

// the nine invariants at unit support: (lam, m1_axial, m2_tangent, m2_axial, G_axial, g1_tangent, g1_axial,
// H_tangent, H_axial); d = signed outward distance / h, R = radius / h (ignored for a half-space)
template <class KR, typename T>
__device__ __forceinline__ void radial_invariants(T d, T R, bool sphere, Inv9<T>& acc) {
#pragma unroll
  for (int j = 0; j < 9; ++j) acc.v[j] = T(0);
  const T cap_end = sphere ? fmin(T(1), T(2) * R + d) : T(1);
  if (d <= T(-1)) {
    // the whole support lies in the solid (for a sphere |x - c| + h <= R): exact constants
    KR::template full<T>(acc.v);
    return;
  }
  if (d >= T(1)) return;                       // the support does not reach the solid
  const T full_end = fmin(T(1), fmax(T(0), -d));
  const T inv2D = sphere ? T(1) / (T(2) * (R + d)) : T(0);
  radial_piece<KR, 0, T>(d, R, inv2D, sphere, full_end, cap_end, acc);
  if constexpr (KR::kPieces > 1) radial_piece<KR, 1, T>(d, R, inv2D, sphere, full_end, cap_end, acc);
  static_assert(KR::kPieces <= 2, "radial kernels have at most two pieces");
}

constexpr int kRadialThreads = 128;

__device__ __forceinline__ double pick3(int i, double x, double y, double z) { return i == 0 ? x : (i == 1 ? y : z); }

// the 28 baseline requests of a row in their order, from its invariants and normal
__device__ __forceinline__ void baseline_row(const double inv[9], const double n[3], double* o) {
  o[0] = inv[0];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[1 + i] = inv[1] * n[i];
    o[10 + i] = inv[4] * n[i];
  }
  const double dm = inv[3] - inv[2], dg = inv[6] - inv[5], dh = inv[8] - inv[7];
  int k = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j, ++k) {
      o[4 + k] = dm * n[i] * n[j] + (i == j ? inv[2] : 0.0);
      o[22 + k] = dh * n[i] * n[j] + (i == j ? inv[7] : 0.0);
    }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) o[13 + 3 * i + j] = dg * n[i] * n[j] + (i == j ? inv[5] : 0.0);
}

// One thread per row; the block's rows are contiguous, so their outputs [row0 .. row0 + 128) x n_requests (and their
// invariants, x 9) are one contiguous range each: every thread puts its row into shared memory (odd strides against bank
// conflicts), then the block stores the range coalesced.  FULL: the 28 baseline requests in their order -- written
// straight from the invariants; other sets look up each request's row of the table (half of the instructions of a full
// row before).  2^21 sphere rows (w4) on B200: 0.131 ms with 8 + 7 nodes a row and no division in a node (float32, 12 + 12
// nodes: 0.132); 0.47 ms with 12 + 12 nodes, a division each, and the table for every set.
template <class KR, typename T, bool FULL>
__global__ void __launch_bounds__(kRadialThreads, 6) k_radial(const double* __restrict__ dist,
                                                              const double* __restrict__ radii,
                                                              const double* __restrict__ normals,
                                                              const double* __restrict__ supports, int64_t n,
                                                              int sphere, RadialRequests req,
                                                              double* __restrict__ out, double* __restrict__ inv_out,
                                                              int32_t* __restrict__ status) {
  __shared__ double stage[kRadialThreads * 29];
  const int64_t row0 = (int64_t)blockIdx.x * kRadialThreads;
  const int64_t row = row0 + threadIdx.x;
  const int nreq = FULL ? 28 : req.n, stride = nreq | 1;
  const int rows_here = (int)(n - row0 < kRadialThreads ? n - row0 : kRadialThreads);
  double inv[9];
  if (row < n) {
    const double h = supports[row], dd = dist[row];
    const double Rr = sphere ? radii[row] : 0.0;
    const double nrm[3] = {normals[3 * row], normals[3 * row + 1], normals[3 * row + 2]};
    const bool ok = h > 0.0 && isfinite(h) && isfinite(dd) && isfinite(nrm[0]) && isfinite(nrm[1]) && isfinite(nrm[2]) &&
                    (!sphere || (Rr > 0.0 && isfinite(Rr) && dd >= -Rr));
    Inv9<T> acc;
    if (ok) {
      radial_invariants<KR, T>(T(dd / h), T(Rr / h), sphere != 0, acc);
      const double ih = 1.0 / h;
      const double scale[9] = {1.0, h, h * h, h * h, ih, 1.0, 1.0, ih * ih, ih * ih};
#pragma unroll
      for (int j = 0; j < 9; ++j) inv[j] = (double)acc.v[j] * scale[j];
    } else {
#pragma unroll
      for (int j = 0; j < 9; ++j) inv[j] = __longlong_as_double(0x7ff8000000000000LL);
    }
    if (status) status[row] = ok ? 0 : 1;
    double* const mine = stage + threadIdx.x * stride;
    if constexpr (FULL) {
      double o[28];
      baseline_row(inv, nrm, o);
#pragma unroll
      for (int c = 0; c < 28; ++c) mine[c] = o[c];
    } else {
#pragma unroll 4
      for (int c = 0; c < nreq; ++c) {
        const int degree = req.meta[c][0], i = req.meta[c][1], j = req.meta[c][2], order = req.meta[c][3];
        const double ni = pick3(i, nrm[0], nrm[1], nrm[2]), nj = pick3(j, nrm[0], nrm[1], nrm[2]);
        double v;
        if (degree == 0 && order == 0) {
          v = inv[0];
        } else if (degree == 1 && order == 0) {
          v = inv[1] * ni;
        } else if (degree == 0 && order == 1) {
          v = inv[4] * ni;
        } else {
          // tangent / axial pair of the second-order entry: m2 (2, 3), g1 (5, 6), Hessian (7, 8)
          const double tan = order == 0 ? inv[2] : (order == 1 ? inv[5] : inv[7]);
          const double axi = order == 0 ? inv[3] : (order == 1 ? inv[6] : inv[8]);
          v = (axi - tan) * ni * nj + (i == j ? tan : 0.0);
        }
        mine[c] = v;
      }
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < rows_here * nreq; k += kRadialThreads)
    out[row0 * nreq + k] = stage[k / nreq * stride + k % nreq];
  if (inv_out) {
    __syncthreads();
    if (row < n) {
#pragma unroll
      for (int j = 0; j < 9; ++j) stage[threadIdx.x * 9 + j] = inv[j];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < rows_here * 9; k += kRadialThreads) inv_out[row0 * 9 + k] = stage[k];
  }
}

// whether the requests are the 28 baseline requests in their order: value moments of degree 0, 1, 2, first-derivative
// moments of degree 0 and 1 per axis, the Hessian's upper triangle
bool is_baseline(const RadialRequests& req) {
  if (req.n != 28) return false;
  int c = 0;
  bool same = true;
  auto row = [&](int degree, int i, int j, int order) {
    const signed char* m = req.meta[c++];
    same = same && m[0] == degree && m[1] == i && m[2] == j && m[3] == order;
  };
  row(0, 0, 0, 0);
  for (int i = 0; i < 3; ++i) row(1, i, 0, 0);
  for (int i = 0; i < 3; ++i)
    for (int j = i; j < 3; ++j) row(2, i, j, 0);
  for (int j = 0; j < 3; ++j) row(0, j, 0, 1);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) row(1, i, j, 1);
  for (int i = 0; i < 3; ++i)
    for (int j = i; j < 3; ++j) row(0, i, j, 2);
  return same;
}

template <typename T>
int launch_radial(int kernel, const double* d, const double* r, const double* nrm, const double* h, int64_t n,
                  int sphere, const RadialRequests& req, double* out, double* inv, int32_t* status,
                  cudaStream_t st) {
  const unsigned grid = (unsigned)((n + kRadialThreads - 1) / kRadialThreads);
  constexpr int B = kRadialThreads;
  auto launch = [&](auto kr) {
    using KR = decltype(kr);
    if (is_baseline(req))
      k_radial<KR, T, true><<<grid, B, 0, st>>>(d, r, nrm, h, n, sphere, req, out, inv, status);
    else
      k_radial<KR, T, false><<<grid, B, 0, st>>>(d, r, nrm, h, n, sphere, req, out, inv, status);
  };
  switch (kernel) {
    case WSB_KERNEL_CUBIC: launch(Rad_cubic{}); break;
    case WSB_KERNEL_W2: launch(Rad_w2{}); break;
    case WSB_KERNEL_W4: launch(Rad_w4{}); break;
    case WSB_KERNEL_W6: launch(Rad_w6{}); break;
    default: return fail(WSB_ERR_UNSUPPORTED, "wsb_radial_channels: the radial family serves cubic, w2, w4, w6");
  }
  WSB_CUDA(cudaGetLastError());
  return WSB_OK;
}

}  // namespace
}  // namespace wsb

using namespace wsb;

extern "C" int wsb_radial_channels(int kind, int kernel, int precision, const double* distances, const double* radii,
                                   const double* normals, const double* supports, int64_t n, const int32_t* requests,
                                   int n_requests, double* out, double* invariants, int32_t* status, void* stream) {
  if (kind != WSB_RADIAL_PLANE && kind != WSB_RADIAL_SPHERE)
    return fail(WSB_ERR_ARG, "wsb_radial_channels: kind must be WSB_RADIAL_PLANE or WSB_RADIAL_SPHERE");
  if (n < 0) return fail(WSB_ERR_ARG, "wsb_radial_channels: negative size");
  if (n_requests < 0 || n_requests > 28) return fail(WSB_ERR_ARG, "wsb_radial_channels: 0..28 requests");
  if (precision != WSB_PREC_FP64 && precision != WSB_PREC_FP32)
    return fail(WSB_ERR_UNSUPPORTED, "wsb_radial_channels: precision must be WSB_PREC_FP64 or WSB_PREC_FP32");
  if (kernel < 0 || kernel > WSB_KERNEL_W6)
    return fail(WSB_ERR_UNSUPPORTED, "wsb_radial_channels: the radial family serves cubic, w2, w4, w6");
  RadialRequests req{};
  req.n = n_requests;
  for (int c = 0; c < n_requests; ++c) {
    const int32_t* m = requests + 4 * c;
    const int degree = m[0], i = m[1], j = m[2], order = m[3];
    if (degree < 0 || order < 0 || degree + order > 2 || i < 0 || i > 2 || j < 0 || j > 2)
      return fail(WSB_ERR_ARG, "wsb_radial_channels: request rows are (degree, i, j, order) with degree + order <= 2");
    for (int q = 0; q < 4; ++q) req.meta[c][q] = (signed char)m[q];
  }
  if (n == 0) return WSB_OK;
  if (!distances || !normals || !supports || (n_requests && !out) || (kind == WSB_RADIAL_SPHERE && !radii))
    return fail(WSB_ERR_ARG, "wsb_radial_channels: NULL array");
  cudaStream_t st = (cudaStream_t)stream;
  return precision == WSB_PREC_FP64
             ? launch_radial<double>(kernel, distances, radii, normals, supports, n, kind, req, out, invariants, status, st)
             : launch_radial<float>(kernel, distances, radii, normals, supports, n, kind, req, out, invariants, status, st);
}

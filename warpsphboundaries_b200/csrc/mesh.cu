// Closed triangle surfaces in 3-D: the 28 baseline kernel integrals over the part of each query's support inside the
// solid (value moments |alpha| <= 2, kernel-gradient moments |alpha| <= 1, the kernel Hessian).
//
// Reference: the closed-surface element of src/warpSPHBoundaries/fluxbridge/wp_func.py:119-333 (face -> edge
// reductions, solid-angle term summed over every face), its exact mpmath counterpart
// src/warpSPHBoundaries/mesh3d/reference.py:221-311 (ClosedSurface), the whole-element search of
// fluxbridge/geometry.py:86-170 / device_search.py:158-212 and the per-query reduction of
// fluxbridge/evaluate.py:177-187.
//
// Reduction (unit support: y = (vertex - query) / h, W~ = pi W):
//  * volume -> faces.  For |alpha| = k, y y^alpha G_k(r) with (r^(3+k) G_k)' = r^(2+k) W~ has divergence y^alpha W~;
//    splitting off the homogeneous field y y^alpha Q_k(1) / r^(3+k), whose flux through the closed surface is
//    ind * int_{S^2} yhat^alpha (ind = 1 inside the solid), leaves the compact profile
//    K_k = (Q_k(r) - Q_k(1)) / r^(3+k):   M_alpha = sum_faces z_f int_f y^alpha K_k dS + ind Q_k(1) int yhat^alpha.
//    Kernel-gradient moments are -sum_f N_j int_f y^alpha W~ dS (+ alpha_j M_(alpha - e_j)); the Hessian is
//    sum_f N_i int_f y_j W~'/r dS.  Only faces within the support contribute: no solid-angle sum over all faces.
//  * face -> edges.  With y = z N + u (u in the face plane, r^2 = z^2 + |u|^2) and the compact potential
//    A_F(r) = -int_r^1 t F(t) dt of a profile F:   int_f F = sum_e w_e int_e (A_F(r) - A_F(|z|)) / (r^2 - z^2) ds,
//    int_f u F = sum_e mu_e int_e A_F ds,  int_f u u^T F = sum_e mu_e (x) int_e u A_F ds - P int_f A_F
//    (w_e: signed distance of the foot point to the edge line, mu_e: in-plane outward edge normal, P = I - N N^T).
//  * edges.  Beyond the block's radius the first integrand is -A_F(|z|) / rho^2: an angle.  Inside, every integrand has
//    a closed form in r = sqrt(c^2 + s^2), c^2 = z^2 + w^2, a = |z|.  A_F is taken in powers of t = r - R/2 (and its one
//    negative power of r); with P_n = int t^n ds, Q_n = int t^n / r ds, p = R/2 (`rho` in the code):
//      (n + 1) P_n = [s t^n] - n p P_(n-1) + n c^2 Q_(n-1),   Q_n = P_(n-1) - p Q_(n-1),   P_0 = D,  Q_0 = L,
//    errors shrink by p a step, and the line integrals of A_F are dot products with the P_n.  In the divided difference
//    (A(r) - A(a)) / (r - a) is a polynomial in t (synthetic division at a - p), so a face needs its edges' w-weighted
//    sums alone: V_k = sum_e w_e int t^k / (r + a) ds, V_k = sum_e w_e P_(k-1) - (a + p) V_(k-1), V_0 = Lambda.  With
//    Y = (s1 r0 - s0 r1) / c^2 (formed without cancellation), U = c^2 Y + c D, B = (r1 + c)(r0 + c), kappa = w / (c + a):
//      L = int ds / r = 2 atanh(D / (r0 + r1)),   int c ds / r^2 = 2 atan(U / (B + s0 s1)) = Theta,
//      int ds / r^3 = Y / (r0 r1),                int w ds / (r (r + a)) = 2 atan(kappa U / (B + kappa^2 s0 s1)) = Omega,
//      Lambda = sum_e (w L - a Omega),
//      [s t^n] = D/2 (t1^n + t0^n + S^2 / (r0 + r1) T_n),  T_n = (t1^n - t0^n) / (t1 - t0)      (D = s1 - s0, S = s1 + s0).
//    Why about R/2: in powers of r itself the terms of A cancel to one part in 445 (w4) or 3718 (w6), about R/2 to one in 3
//    or 4 (in V_k, which meets t = -a - p, to one in 19 or 54 at a = 0.3), so the rounding of a channel was four to twelve
//    times that of 32 quadrature nodes an edge and is now the same (rms over 1200 rows near a surface, units of the support:
//    w2 8e-15 -> 4e-15, w4 1.2e-13 -> 4e-14, w6 1.5e-12 -> 3.5e-13; the quadrature 4e-15, 4.5e-14, 4e-13), for 4 % of the
//    time (2^21 queries, 2.6 M pairs of a row and a face: 729 -> 757 us).
//    Powers z^p multiply the profiles whose potentials hold r^-m (m <= p) so that every face term stays bounded as
//    the query approaches the face plane.
//  * kernels of several pieces are sums of truncated blocks P(r) 1[r <= R] (the decomposition of the 2-D tables); every
//    channel is the sum of its blocks' channels, so no integral crosses a knot.
// The exact rational potentials are generated by warpsphboundaries_b200/kernels.py (mesh_blocks, emit_mesh).
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"

namespace wsb {

struct Mesh {
  int device = 0;
  int64_t n_verts = 0, n_faces = 0;
  double support_max = 0;
  double lo[3] = {0, 0, 0};
  double cell = 1;
  int32_t nx = 1, ny = 1, nz = 1;
  int64_t n_items = 0, n_col_items = 0;
  double* fdata = nullptr;     // [n_faces * kFaceDoubles]
  int32_t words = 1;           // 64-bit words of a row's hit mask (at most kMaxWords)
  int32_t eval_rows = 32;      // rows a warp of the evaluation takes at most (fewer where their faces would pass 2^31)
  int64_t* nstart = nullptr;   // [nx*ny*nz + 1]
  int32_t* nitems = nullptr;   // per cell the faces a query of the cell may reach (each once)
  double col = 1;              // size of an (x, y) column: half a cell (a cell where that would list too many faces)
  int32_t ncx = 1, ncy = 1;
  int32_t* colstart = nullptr; // [ncx*ncy + 1] faces per column
  int32_t* colitems = nullptr;
  uint8_t* cflag = nullptr;    // [nx*ny*nz] kCellEmpty | kCellInside | kCellNear
};

// per-cell flags: no face box meets the cell (so the surface does not cross it and every point of it has the inside
// status of its centre); that status; the cell's face list is not empty (a query in the cell may have candidate faces)
enum : uint8_t { kCellEmpty = 1, kCellInside = 2, kCellNear = 4 };

// per face, one 256-byte record: v0 v1 v2 (9), unit normal N (3), edge tangents t0 t1 t2 (9), edge lengths (3), box lo
// (3), box hi (3), the edges that run from the lower to the higher vertex id (bits 0-2, as a number), 1 unused
constexpr int kFaceDoubles = 32;
enum { kFV = 0, kFN = 9, kFT = 12, kFLEN = 21, kFLO = 24, kFHI = 27, kFORD = 30 };

struct MeshView {
  const double* fdata;
  const int64_t* nstart;
  const int32_t* nitems;
  const int32_t* colstart;
  const int32_t* colitems;
  const uint8_t* cflag;
  double lo0, lo1, lo2, cell, col;
  int32_t nx, ny, nz, ncx, ncy;
};

namespace {

MeshView view_of(const Mesh* m) {
  return MeshView{m->fdata, m->nstart, m->nitems, m->colstart, m->colitems, m->cflag,
                  m->lo[0], m->lo[1], m->lo[2], m->cell, m->col, m->nx, m->ny, m->nz, m->ncx, m->ncy};
}

__device__ __forceinline__ int cell_coord(double x, double lo, double cell, int n) {
  const double f = floor((x - lo) / cell);
  return f < -1.0 ? -2 : (f > (double)n ? n + 1 : (int)f);
}

// ------------------------------------------------------------------------------------------ inside indicator
// Parity of the crossings of the vertical ray {(x, y, t): t > z} with the surface.  A face's projection owns the
// point when every edge function is positive, or zero on an edge that the ownership rule gives to this side: edge
// functions are evaluated with the edge's vertices in id order (so the two faces of an edge see exactly opposite
// values) and an edge with zero value belongs to the face for which its counter-clockwise direction d has
// d.y > 0 or (d.y == 0 and d.x < 0) -- exactly one of the two faces of a shared edge.
// rounded products and differences (never contracted into an fma): a query on a vertex gives exactly 0, and the
// two faces of an edge compute bit-identical values
__device__ __forceinline__ double edge_fn(double ax, double ay, double bx, double by, double qx, double qy) {
  return __dsub_rn(__dmul_rn(__dsub_rn(bx, ax), __dsub_rn(qy, ay)), __dmul_rn(__dsub_rn(by, ay), __dsub_rn(qx, ax)));
}

// whether the vertical ray {(x, y, t): t > z} crosses face f of the column (its projection owns (x, y) and the face
// lies above z)
__device__ __forceinline__ bool column_cross(const MeshView& M, int f, double x, double y, double z) {
  const double* F = M.fdata + (int64_t)f * kFaceDoubles;
  double V[12];                                     // the vertices and the normal, loaded together
#pragma unroll
  for (int k = 0; k < 3; ++k) ld4_nc(F + 4 * k, V[4 * k], V[4 * k + 1], V[4 * k + 2], V[4 * k + 3]);
  const int ord = (int)F[kFORD];
  const double nzf = V[kFN + 2];
  if (nzf == 0.0) return false;                     // vertical face: its projection has no interior
  const double sgn = nzf > 0.0 ? 1.0 : -1.0;        // counter-clockwise projection for N.z > 0
  bool owns = true;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const double ax = V[3 * e], ay = V[3 * e + 1], bx = V[3 * ((e + 1) % 3)], by = V[3 * ((e + 1) % 3) + 1];
    const bool fwd = (ord >> e) & 1;
    double E = fwd ? edge_fn(ax, ay, bx, by, x, y) : -edge_fn(bx, by, ax, ay, x, y);
    E *= sgn;
    if (E < 0.0) owns = false;
    if (E == 0.0) {
      const double dx = (bx - ax) * sgn, dy = (by - ay) * sgn;
      if (!(dy > 0.0 || (dy == 0.0 && dx < 0.0))) owns = false;
    }
  }
  const double zt = V[2] - (V[kFN] * (x - V[0]) + V[kFN + 1] * (y - V[1])) / nzf;
  return owns && zt > z;
}

// the column of (x, y), -1 outside the grid (no face above or below)
__device__ __forceinline__ int column_of(const MeshView& M, double x, double y) {
  const int ix = cell_coord(x, M.lo0, M.col, M.ncx), iy = cell_coord(y, M.lo1, M.col, M.ncy);
  return ix < 0 || iy < 0 || ix >= M.ncx || iy >= M.ncy ? -1 : iy * M.ncx + ix;
}

__device__ int mesh_inside(const MeshView& M, double x, double y, double z) {
  const int col = column_of(M, x, y);
  if (col < 0) return 0;
  int parity = 0;
  for (int k = M.colstart[col]; k < M.colstart[col + 1]; ++k)
    if (column_cross(M, M.colitems[k], x, y, z)) parity ^= 1;
  return parity;
}

// squared distance from the origin to the triangle P (unit coordinates relative to the query)
__device__ __forceinline__ double tri_dist2(const double P[3][3]) {
  // closest point by the Voronoi-region tests on the barycentric parameters (vertex, edge or interior region)
  const double* A = P[0];
  const double ab[3] = {P[1][0] - A[0], P[1][1] - A[1], P[1][2] - A[2]};
  const double ac[3] = {P[2][0] - A[0], P[2][1] - A[1], P[2][2] - A[2]};
  const double ap[3] = {-A[0], -A[1], -A[2]};
  auto dot = [](const double* x, const double* y) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; };
  const double d1 = dot(ab, ap), d2 = dot(ac, ap);
  double cp[3];
  auto setp = [&](double v, double w) {
    for (int k = 0; k < 3; ++k) cp[k] = A[k] + v * ab[k] + w * ac[k];
  };
  if (d1 <= 0.0 && d2 <= 0.0) {
    setp(0.0, 0.0);
  } else {
    const double bp[3] = {-P[1][0], -P[1][1], -P[1][2]};
    const double e3 = dot(ab, bp), e4 = dot(ac, bp);
    if (e3 >= 0.0 && e4 <= e3) {
      setp(1.0, 0.0);
    } else {
      const double vc = d1 * e4 - e3 * d2;
      if (vc <= 0.0 && d1 >= 0.0 && e3 <= 0.0) {
        setp(d1 / (d1 - e3), 0.0);
      } else {
        const double cpn[3] = {-P[2][0], -P[2][1], -P[2][2]};
        const double e5 = dot(ab, cpn), e6 = dot(ac, cpn);
        if (e6 >= 0.0 && e5 <= e6) {
          setp(0.0, 1.0);
        } else {
          const double vb = e5 * d2 - d1 * e6;
          if (vb <= 0.0 && d2 >= 0.0 && e6 <= 0.0) {
            setp(0.0, d2 / (d2 - e6));
          } else {
            const double va = e3 * e6 - e5 * e4;
            if (va <= 0.0 && (e4 - e3) >= 0.0 && (e5 - e6) >= 0.0) {
              const double t = (e4 - e3) / ((e4 - e3) + (e5 - e6));
              setp(1.0 - t, t);
            } else {
              const double den = 1.0 / (va + vb + vc);
              setp(vb * den, vc * den);
            }
          }
        }
      }
    }
  }
  return cp[0] * cp[0] + cp[1] * cp[1] + cp[2] * cp[2];
}

// ------------------------------------------------------------------------------------------ candidate faces
// the faces by cell as the host counts them: every cell lists the faces whose box overlaps it
struct BoxLists {
  const int32_t* start;   // [nx*ny*nz + 1]
  const int32_t* items;
  const int32_t* fcell;   // [n_faces * 3] lowest cell of the face's box
};

// The candidate list of one cell, once per mesh, by a warp: the faces listed in the 27 cells around it whose box comes
// within a cell's size (>= every support) of the cell's box -- each face once (a face listed in several of the 27 cells
// is taken in the lowest of them inside the block), in cell order and item order within a cell.  The margin of 1e-6
// is far above the rounding of the cell boxes: a face is only left out when clearly beyond reach.  Writes the list to
// `dst` when it is given; returns its length.
__device__ __forceinline__ int cell_faces(const MeshView& M, const BoxLists& L, int64_t c, int lane, int32_t* dst) {
  const int cx = (int)(c % M.nx), cy = (int)((c / M.nx) % M.ny), cz = (int)(c / ((int64_t)M.nx * M.ny));
  const double b[3] = {fma((double)cx, M.cell, M.lo0), fma((double)cy, M.cell, M.lo1), fma((double)cz, M.cell, M.lo2)};
  const double reach2 = M.cell * M.cell * (1.0 + 1e-6);
  int len = 0;
  for (int k = max(cz - 1, 0); k <= min(cz + 1, M.nz - 1); ++k)
    for (int j = max(cy - 1, 0); j <= min(cy + 1, M.ny - 1); ++j) {
      const int64_t r0 = ((int64_t)k * M.ny + j) * M.nx;
      for (int i = max(cx - 1, 0); i <= min(cx + 1, M.nx - 1); ++i) {
        const int e = L.start[r0 + i + 1];
        for (int base = L.start[r0 + i]; base < e; base += 32) {
          bool take = false;
          int f = 0;
          if (base + lane < e) {
            f = L.items[base + lane];
            const int32_t* fc = L.fcell + 3 * (int64_t)f;
            if (max(fc[0], cx - 1) == i && max(fc[1], cy - 1) == j && max(fc[2], cz - 1) == k) {
              const double* F = M.fdata + (int64_t)f * kFaceDoubles;
              double d2 = 0.0;
#pragma unroll
              for (int a = 0; a < 3; ++a) {
                const double d = fmax(0.0, fmax(F[kFLO + a] - (b[a] + M.cell), b[a] - F[kFHI + a]));
                d2 = fma(d, d, d2);
              }
              take = d2 < reach2;
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, take);
          if (dst && take) dst[len + __popc(m & ((1u << lane) - 1))] = f;
          len += __popc(m);
        }
      }
    }
  return len;
}

// whether face f comes within h of the query (unit coordinates relative to the query, the operations of the face
// integral's)
__device__ __forceinline__ bool face_within(const MeshView& M, int f, const double q[3], double ih) {
  const double* F = M.fdata + (int64_t)f * kFaceDoubles;
  double v[12];
#pragma unroll
  for (int k = 0; k < 3; ++k) ld4_nc(F + kFV + 4 * k, v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
  double P[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int a = 0; a < 3; ++a) P[k][a] = (v[3 * k + a] - q[a]) * ih;
  return tri_dist2(P) < 1.0;
}

// The items that a warp's batch of rows brings, flattened over the lanes: lane r < kRows holds the length of its row's
// items and the exclusive prefix of the lengths before it (lanes past the batch: the total).  Unsigned: a round may
// start past the last item.
template <int kRows>
struct Flat {
  unsigned len, pref, total;
  __device__ __forceinline__ void set(unsigned length, int lane) {
    len = length;
    unsigned inc = length;
#pragma unroll
    for (int o = 1; o < kRows; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    total = __shfl_sync(0xffffffffu, inc, kRows - 1);
    pref = lane < kRows ? inc - len : total;
  }
  // the batch row of item t (the last lane whose prefix is <= t) and the item's place in it; every lane takes part
  __device__ __forceinline__ int row_of(unsigned t, unsigned& place) const {
    int r = 0;
#pragma unroll
    for (int step = kRows / 2; step > 0; step >>= 1)
      if (__shfl_sync(0xffffffffu, pref, r + step) <= t) r += step;
    place = t - __shfl_sync(0xffffffffu, pref, r);
    return r;
  }
  // of the round that starts at item `base`: the first of lane r's items in it, the lane that holds it, how many
  __device__ __forceinline__ int part(unsigned base, unsigned& place, int& lane0) const {
    const int64_t a = max((int64_t)pref - base, (int64_t)0), b = min((int64_t)pref + len - base, (int64_t)32);
    lane0 = (int)a;
    place = (unsigned)(base + a - pref);
    return (int)(b - a);
  }
};

// a row with faces, as the integration reads it: the query, its support, its list and the hits among the list's first
// 64 x words faces (a word of the mask each 64); faces beyond are tested when they are integrated
constexpr int kMaxWords = 8;
struct __align__(32) MeshRow {
  double q[3], h;
  int64_t first;        // first item of the list
  int32_t len, tag;     // its length; row | inside << 30
  int32_t at, pad[3];   // the row's place in the masks
};
static_assert(sizeof(MeshRow) == 64, "row record layout");
constexpr int kRowMask = (1 << 30) - 1;

// ------------------------------------------------------------------------------------------ face integrals
template <int I, int N, class Fn>
__device__ __forceinline__ void static_for(Fn&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}
template <int K>
__device__ __forceinline__ double zpow(double z) {
  if constexpr (K == 0) return 1.0;
  else if constexpr (K == 1) return z;
  else if constexpr (K == 2) return z * z;
  else return z * z * z;
}

// coefficient of (r - R/2)^n of potential f of block B, and the coefficient of its negative power of r
template <class B, int f, int n>
struct MeshC {
  static constexpr double v = B::kC[f][n];
};
template <class B, int f>
struct MeshNu {
  static constexpr double v = B::kNu[f];
};

// the highest power of potential f of block B
template <class B, int f, int n = B::kTop>
constexpr int mesh_degree() {
  if constexpr (n == 0 || MeshC<B, f, n>::v != 0.0) return n;
  else return mesh_degree<B, f, n - 1>();
}

// the power z^p that multiplies each potential (rows of the block tables) and its one negative power r^-m
constexpr int kZPow[6] = {1, 2, 3, 0, 0, 1};
constexpr int kNeg[6] = {1, 2, 3, 0, 0, 1};

// the face's sums over its edges that carry the edges' vectors: sum mu LK1, sum mu LK2, sum (mu mu w LK2b + sym(mu t)
// TK2), sum mu LW, sum mu LL / 2 (LK1 = z int A_K1, LK2b = z int A_K2, LK2 = z LK2b, TK2 = z int s A_K2, LW = int A_W,
// LL = int A_L); and J_F = sum_e w_e int z^p DD_F ds
struct FaceSums {
  double k1[3], k2[3], kk[6], lw[3], ll[3], J[6];
};

// one block's contribution to the sums of the face F (query q, 1 / support ih; z = signed distance of the query to the
// face plane in supports, N its normal)
template <class B>
__device__ __forceinline__ void face_block(const double* __restrict__ F, const double q[3], double ih,
                                           const double N[3], double z, FaceSums& A) {
  constexpr double R = B::kR, rho = B::kRho;
  const double a = fabs(z), sg = z > 0.0 ? 1.0 : (z < 0.0 ? -1.0 : 0.0);
  if (!(a < R)) return;                 // no point of the plane within R: no chord, and the potentials vanish at |z|
  double M[B::kLine + 1];               // sum_e w_e P_n
#pragma unroll
  for (int n = 0; n <= B::kLine; ++n) M[n] = 0.0;
  double lam = 0.0, om = 0.0, th = 0.0, s3 = 0.0, ox = 1.0, oy = 0.0;
  float turn = 0.0f;
  bool beyond = false;                  // some edge has a part beyond R
  const double zz = z * z;
#pragma unroll 1
  for (int e = 0; e < 3; ++e) {
    const double P[3] = {(F[kFV + 3 * e] - q[0]) * ih, (F[kFV + 3 * e + 1] - q[1]) * ih,
                         (F[kFV + 3 * e + 2] - q[2]) * ih};
    const double t[3] = {F[kFT + 3 * e], F[kFT + 3 * e + 1], F[kFT + 3 * e + 2]};
    const double mu[3] = {t[1] * N[2] - t[2] * N[1], t[2] * N[0] - t[0] * N[2], t[0] * N[1] - t[1] * N[0]};
    const double w = mu[0] * P[0] + mu[1] * P[1] + mu[2] * P[2];
    const double lo = t[0] * P[0] + t[1] * P[1] + t[2] * P[2], hi = lo + F[kFLEN + e] * ih;
    const double c2 = fma(w, w, zz) + 1e-200, c = sqrt(c2);
    double s0 = 0.0, s1 = 0.0;
    if (c < R) {
      const double L = sqrt((R - c) * (R + c));
      s0 = fmax(lo, -L);
      s1 = fmin(hi, L);
    }
    const bool in = s1 > s0;
    // the angle under which the foot of the query sees the part of the edge beyond R: the parts' rotations multiplied
    // (their sum lies in (-pi, pi), with the sign of w), and those of the three edges: one atan2 a face; the float sum
    // of the edges' angles only tells the full turns (it may cancel to 0 where the angle is 1e-7)
    if (w != 0.0 && (!in || lo < s0 || s1 < hi)) {
      const double ww = w * w;
      double x, y;
      if (!in) {
        x = fma(lo, hi, ww);
        y = w * (hi - lo);
      } else {
        const bool l = lo < s0, r = s1 < hi;
        const double xl = l ? fma(lo, s0, ww) : 1.0, yl = l ? w * (s0 - lo) : 0.0;
        const double xr = r ? fma(s1, hi, ww) : 1.0, yr = r ? w * (hi - s1) : 0.0;
        x = xl * xr - yl * yr;
        y = xl * yr + yl * xr;
      }
      const double m = 1.0 / (fabs(x) + fabs(y));
      x *= m;
      y *= m;
      beyond = true;
      turn += atan2f((float)y, (float)x);
      const double t0 = ox * x - oy * y;
      oy = ox * y + oy * x;
      ox = t0;
    }
    if (!in) continue;
    const double r0 = lo < s0 ? R : sqrt(fma(s0, s0, c2)), r1 = s1 < hi ? R : sqrt(fma(s1, s1, c2));
    const double D = s1 - s0, S = s1 + s0;
    const bool same = s0 > 0.0 || s1 < 0.0;                       // the chord on one side of the foot
    const double Y = (same ? D * S : s1 * r0 - s0 * r1) / (same ? s1 * r0 + s0 * r1 : c2);
    const double U = fma(Y, c2, c * D), Bc = (r1 + c) * (r0 + c), s01 = s0 * s1, ca = c + a;
    const double ica = 1.0 / (c * ca), ic = ica * ca, kap = w * (ica * c);
    const double rr = r0 * r1, rs = r0 + r1, irs = 1.0 / (rr * rs), ir = irs * rs, Y3 = Y * ir;
    // int ds / r = 2 atanh(D / rs) = log1p(2 D / (rs - D)); towards D = rs in the form that does not cancel
    const bool mid = D < 0.75 * rs;
    const double as = log1p(2.0 * (mid ? D : U) / (mid ? rs - D : (r1 - s1 + c) * (r0 + s0 + c)));
    const double Om = 2.0 * atan(kap * U / fmax(fma(kap * kap, s01, Bc), 1e-300));
    const double Th = 2.0 * atan(U / fmax(Bc + s01, 1e-300));
    om += Om;
    lam += w * as - a * Om;
    th += w * ic * Th;
    s3 += a * w * Y3;
    const double sr = S * (irs * rr), qs = S * sr, eh = 0.5 * D, t1 = r1 - rho, t0 = r0 - rho;
    double pb = 1.0, pa = 1.0, T = 0.0, nc2 = 0.0;                // t1^n, t0^n, T_n, n c^2
    double Pm = D, Qm = as;                                       // P_(n-1), Q_(n-1)
    M[0] = fma(w, D, M[0]);
    // the four line integrals of the potentials and (A2_K2(r1) - A2_K2(r0)) / (r1 - r0)
    double k1 = fma(MeshC<B, 1, 0>::v, D, MeshNu<B, 1>::v * Th * ic), k2 = fma(MeshC<B, 2, 0>::v, D, MeshNu<B, 2>::v * Y3);
    double lw = MeshC<B, 3, 0>::v * D, ll = MeshC<B, 4, 0>::v * D, t2 = -MeshNu<B, 5>::v * ir;
    static_for<1, B::kTop + 1>([&](auto nn) {
      constexpr int n = decltype(nn)::value;
      T = fma(t1, T, pa);
      t2 = fma(MeshC<B, 5, n>::v, T, t2);
      pa *= t0;
      if constexpr (n <= B::kLine) {
        pb *= t1;
        nc2 += c2;
        const double Pn = fma(nc2, Qm, fma(-n * rho, Pm, eh * fma(qs, T, pb + pa))) * (1.0 / (n + 1));
        Qm = fma(-rho, Qm, Pm);
        Pm = Pn;
        M[n] = fma(w, Pn, M[n]);
        k1 = fma(MeshC<B, 1, n>::v, Pn, k1);
        k2 = fma(MeshC<B, 2, n>::v, Pn, k2);
        lw = fma(MeshC<B, 3, n>::v, Pn, lw);
        if constexpr (MeshC<B, 4, n>::v != 0.0) ll = fma(MeshC<B, 4, n>::v, Pn, ll);
      }
    });
    const double lk1 = z * k1, lk2b = z * k2, lk2 = z * lk2b, hk = 0.5 * z * (D * sr * t2), wk = w * lk2b, hl = 0.5 * ll;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      A.k1[i] = fma(mu[i], lk1, A.k1[i]);
      A.k2[i] = fma(mu[i], lk2, A.k2[i]);
      A.lw[i] = fma(mu[i], lw, A.lw[i]);
      A.ll[i] = fma(mu[i], hl, A.ll[i]);
    }
    int k = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j, ++k)
        A.kk[k] += mu[i] * (mu[j] * wk + t[j] * hk) + t[i] * (mu[j] * hk);
  }
  double out = 0.0;
  if (beyond) {
    out = atan2(oy, ox);
    out += kTwoPi * rint((turn - out) * (1.0 / kTwoPi));
  }
  // V_k = sum_e w_e int (r - rho)^k / (r + a) ds, in the place of the M_k
  double vk = lam;
  static_for<0, B::kLine + 1>([&](auto kk) {
    constexpr int k = decltype(kk)::value;
    const double next = fma(-(a + rho), vk, M[k]);
    M[k] = vk;
    vk = next;
  });
  const double ta = a - rho;
  static_for<0, 6>([&](auto ff) {
    constexpr int f = decltype(ff)::value, p = kZPow[f], m = kNeg[f];
    constexpr int top = mesh_degree<B, f>();
    static_assert(top <= B::kLine + 2, "powers of the quotient");
    // (A(r) - A(a)) / (r - a) in powers of r - rho by synthetic division, the remainder A(a)
    double J = 0.0, g = MeshC<B, f, top>::v;
    static_for<0, top>([&](auto kk) {
      constexpr int k = top - 1 - decltype(kk)::value;
      J = fma(g, k > B::kLine ? vk : M[k > B::kLine ? 0 : k], J);
      g = fma(ta, g, MeshC<B, f, k>::v);
    });
    J *= zpow<p>(z);
    double Aa = g * zpow<p>(z);                                  // z^p A_F(|z|)
    if constexpr (m > 0) {
      constexpr double nu = MeshNu<B, f>::v;
      const double zr = zpow<p - m>(z);
      if constexpr (m == 1) J -= nu * sg * zr * om;
      if constexpr (m == 2) J -= nu * sg * sg * zr * th;            // (a query in the face's plane: no r^-m term)
      if constexpr (m == 3) J -= nu * sg * zr * (s3 + om);
      Aa += nu * zr * zpow<m>(sg);
    }
    A.J[f] += J - Aa * out;
  });
}

template <class M, int B = 0>
__device__ __forceinline__ void face_blocks(const double* __restrict__ F, const double q[3], double ih,
                                            const double N[3], double z, FaceSums& A) {
  if constexpr (B < M::kBlocks) {
    face_block<typename M::template Block<B>>(F, q, ih, N, z, A);
    face_blocks<M, B + 1>(F, q, ih, N, z, A);
  }
}

// The 28 accumulators of a row (W~ units, unit support): M0, M1[3], M2[6] (00 01 02 11 12 22), G0[3], G1[9] (i-major),
// H[6]; face f adds  M0 += J0;  M1_i += N_i J1 + k1_i;
// M2_ij += N_i N_j (J2 + J5) + N_i k2_j + k2_i N_j + kk_ij - d_ij J5;
// G0_i -= N_i J3;  G1_ij -= z N_i N_j J3 + lw_i N_j;  H_ij += z N_i N_j J4 + N_i ll_j + ll_i N_j.
template <class M>
__device__ __forceinline__ void face_channels(const double* __restrict__ F, const double q[3], double ih, double* o) {
  const double N[3] = {F[kFN], F[kFN + 1], F[kFN + 2]};
  const double z = N[0] * ((F[kFV] - q[0]) * ih) + N[1] * ((F[kFV + 1] - q[1]) * ih) + N[2] * ((F[kFV + 2] - q[2]) * ih);
  FaceSums A;
#pragma unroll
  for (int i = 0; i < 3; ++i) A.k1[i] = A.k2[i] = A.lw[i] = A.ll[i] = 0.0;
#pragma unroll
  for (int i = 0; i < 6; ++i) A.kk[i] = A.J[i] = 0.0;
  face_blocks<M>(F, q, ih, N, z, A);
  o[0] = A.J[0];
  const double j25 = A.J[2] + A.J[5], z3 = z * A.J[3], z4 = z * A.J[4];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[1 + i] = fma(N[i], A.J[1], A.k1[i]);
    o[10 + i] = -N[i] * A.J[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) o[13 + 3 * i + j] = -N[j] * fma(z3, N[i], A.lw[i]);
  }
  int k = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j, ++k) {
      const double NN = N[i] * N[j];
      o[4 + k] = fma(NN, j25, N[i] * A.k2[j] + A.k2[i] * N[j]) + (i == j ? A.kk[k] - A.J[5] : A.kk[k]);
      o[22 + k] = fma(NN, z4, N[i] * A.ll[j] + A.ll[i] * N[j]);
    }
}

// what the accumulator k of a row becomes: its power of the support, and whether the indicator's constants enter (M0;
// the diagonal of M2; the diagonal of G1, which takes the row's M0)
struct Channel {
  int hpow;
  bool m0, m2, g1;
};
__device__ __forceinline__ Channel channel_of(int k) {
  return {k == 0 ? 0 : (k < 4 ? 1 : (k < 10 ? 2 : (k < 13 ? -1 : (k < 22 ? 0 : -2)))), k == 0,
          k == 4 || k == 7 || k == 9, k == 13 || k == 17 || k == 21};
}
template <class M>
__device__ __forceinline__ double channel_value(const Channel& c, double acc, double acc0, double ind, double h,
                                                double ih) {
  const double ip = kInvPi, m0 = acc0 * ip + ind * 4.0 * M::kQ0;
  double v = c.m0 ? m0 : acc * ip + (c.g1 ? m0 : 0.0) + (c.m2 ? ind * (4.0 / 3.0) * M::kQ2 : 0.0);
  if (c.hpow == 1) v *= h;
  if (c.hpow == 2) v *= h * h;
  if (c.hpow == -1) v *= ih;
  if (c.hpow == -2) v *= ih * ih;
  return v;
}

// ------------------------------------------------------------------------------------------ kernels
constexpr int kMeshThreads = 128;

// the length of every cell's candidate list (fill == 0), then the lists (fill == 1): a warp per cell, once per mesh
__global__ void __launch_bounds__(kMeshThreads) k_mesh_lists(MeshView M, BoxLists L, int fill, int32_t* __restrict__ len,
                                                            int32_t* __restrict__ items) {
  const int lane = threadIdx.x & 31;
  const int64_t n = (int64_t)M.nx * M.ny * M.nz, warps = (int64_t)gridDim.x * (kMeshThreads / 32);
  for (int64_t c = (int64_t)blockIdx.x * (kMeshThreads / 32) + threadIdx.x / 32; c < n; c += warps) {
    if (fill) {
      if (M.nstart[c + 1] > M.nstart[c]) cell_faces(M, L, c, lane, items + M.nstart[c]);
    } else {
      const int m = cell_faces(M, L, c, lane, nullptr);
      if (lane == 0) {
        len[c] = m;
        if (m) atomicMax(&len[n], m);                  // the longest list, after the lengths
      }
    }
  }
}

// exclusive prefix sums of the list lengths (64-bit: the lists of a mesh far finer than its supports may pass 2^31
// faces), one block, 1024 lengths at a time
constexpr int kPrefixThreads = 1024;
__global__ void __launch_bounds__(kPrefixThreads) k_mesh_prefix(const int32_t* __restrict__ len, int64_t n,
                                                               int64_t* __restrict__ start) {
  __shared__ int64_t s_warp[kPrefixThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t carry = 0;
  for (int64_t base = 0; base < n; base += kPrefixThreads) {
    const int64_t k = base + threadIdx.x;
    const int64_t v = k < n ? len[k] : 0;
    int64_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    int64_t before = 0, total = 0;
    for (int w = 0; w < kPrefixThreads / 32; ++w) {
      if (w < wid) before += s_warp[w];
      total += s_warp[w];
    }
    if (k < n) start[k] = carry + before + x - v;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) start[n] = carry;
}

// the per-cell flags, once per mesh: emptiness, the inside status of an empty cell's centre (the column parity test),
// whether the cell's candidate list holds a face
__global__ void k_mesh_cellflags(MeshView M, BoxLists L, const int32_t* __restrict__ len, uint8_t* __restrict__ flags) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nxy = (int64_t)M.nx * M.ny;
  if (c >= nxy * M.nz) return;
  const int i = (int)(c % M.nx), j = (int)((c / M.nx) % M.ny), k = (int)(c / nxy);
  uint8_t f = len[c] > 0 ? kCellNear : 0;
  if (L.start[c] == L.start[c + 1]) {
    f |= kCellEmpty;
    const double x = M.lo0 + (i + 0.5) * M.cell, y = M.lo1 + (j + 0.5) * M.cell, z = M.lo2 + (k + 0.5) * M.cell;
    if (mesh_inside(M, x, y, z)) f |= kCellInside;
  }
  flags[c] = f;
}

__device__ __forceinline__ int64_t cell_of_query(const MeshView& M, const double q[3]) {
  const int cx = cell_coord(q[0], M.lo0, M.cell, M.nx), cy = cell_coord(q[1], M.lo1, M.cell, M.ny),
            cz = cell_coord(q[2], M.lo2, M.cell, M.nz);
  if (cx < 0 || cy < 0 || cz < 0 || cx >= M.nx || cy >= M.ny || cz >= M.nz) return -1;
  return ((int64_t)cz * M.ny + cy) * M.nx + cx;
}

// First pass, one thread per query: the cell's flags settle the rows away from the surface (outside the grid, which
// reaches a cell past the surface's box: outside the solid, no face within the support; an empty candidate list: the
// cell is empty and its centre's status holds); the others are appended to `near` for the second pass.  Invalid rows (a
// support above the grid cell would reach faces beyond the lists, non-finite input) are marked -1 and come back as NaN.
// Every row's constants -- whole-support values inside, zeros outside, NaN -- are built in shared memory (stride 29
// doubles against bank conflicts) and the block writes its contiguous slab of 128 x 28 outputs coalesced (the second
// pass overwrites its rows).  One global atomic a block for the list: one a warp took 54 us for 2^21 rows, the row
// constants in a kernel of their own another 75.
constexpr int kRowStride = 29;

template <class M>
__global__ void __launch_bounds__(kMeshThreads) k_mesh_rowinfo(MeshView Mv, const double* __restrict__ pos,
                                                              const double* __restrict__ sup, int64_t n,
                                                              int32_t* __restrict__ ind, int32_t* __restrict__ near,
                                                              int32_t* __restrict__ nnear, double* __restrict__ out) {
  __shared__ double s_rows[kMeshThreads * kRowStride];
  __shared__ int32_t s_count[kMeshThreads / 32 + 1];
  const int64_t row0 = (int64_t)blockIdx.x * kMeshThreads;
  const int64_t row = row0 + threadIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  bool listed = false;
  if (row < n) {
    const double q[3] = {pos[3 * row], pos[3 * row + 1], pos[3 * row + 2]};
    const double h = sup[row];
    const bool ok = h > 0.0 && h <= Mv.cell && isfinite(q[0]) && isfinite(q[1]) && isfinite(q[2]);
    int in = ok ? 0 : -1;
    if (ok) {
      const int64_t c = cell_of_query(Mv, q);
      const uint8_t f = c >= 0 ? Mv.cflag[c] : (uint8_t)0;
      listed = f & kCellNear;
      in = !listed && (f & kCellInside) ? 1 : 0;
    }
    if (!listed) ind[row] = in;
    double* const mine = s_rows + threadIdx.x * kRowStride;
    const double id = in < 0 ? __longlong_as_double(0x7ff8000000000000LL) : (double)in, ih = 1.0 / h;
    for (int k = 0; k < 28; ++k)
      mine[k] = in < 0 ? id : channel_value<M>(channel_of(k), 0.0, 0.0, id, h, ih);
  }
  const unsigned mask = __ballot_sync(0xffffffffu, listed);
  if (lane == 0) s_count[wid] = __popc(mask);
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
    for (int w = 0; w < kMeshThreads / 32; ++w) {
      const int v = s_count[w];
      s_count[w] = total;
      total += v;
    }
    s_count[kMeshThreads / 32] = total ? atomicAdd(nnear, total) : 0;
  }
  const int rows = (int)min((int64_t)kMeshThreads, n - row0);
  for (int k = threadIdx.x; k < rows * 28; k += kMeshThreads)
    out[row0 * 28 + k] = s_rows[(k / 28) * kRowStride + k % 28];
  __syncthreads();
  if (listed) near[s_count[kMeshThreads / 32] + s_count[wid] + __popc(mask & ((1u << lane) - 1))] = (int32_t)row;
}

// Second pass, the listed rows.  A warp takes up to eight rows at a time: lane r loads row r and its list, then the
// inside tests (the cell's flag where the cell is empty, the column parity otherwise) and the face search run over the
// eight rows' items flattened on the lanes, so the chain of loads from a row to its faces is paid once for eight rows
// and the rounds are full although a list holds some 40 faces.  A row's hits are kept as a mask over its list; rows with
// hits are appended to `rows`, the others get their constants.
// (2^21 particles, 20480 faces: 0.21 ms on B200; a warp per row over the 27 cells' box lists, in which a face of the
// cell's size is met six times, and the inside test a warp per row: 1.3 ms, half of it a second search in the
// integration.  A kernel of its own, 8 CTAs per SM, because it waits for loads: inside the integration's kernel, at 3
// CTAs per SM, the search of 20011 near rows took 109 us of 169, here 49.)
constexpr int kBatch = 8;
constexpr int kSearchBlocks = 8;

// rows per batch: as many as the warps' even share allows (a share of 12 rows in two batches of 6, not 8 and 4)
__device__ __forceinline__ int batch_rows(int n, int warps, int most) {
  const int share = (n + warps - 1) / warps, nb = (share + most - 1) / most;
  return nb ? (share + nb - 1) / nb : 1;
}

template <class M>
__global__ void __launch_bounds__(kMeshThreads, kSearchBlocks)
    k_mesh_search(MeshView Mv, const double* __restrict__ pos, const double* __restrict__ sup,
                  const int32_t* __restrict__ near, int32_t* __restrict__ counts, int words, int32_t* __restrict__ ind,
                  MeshRow* __restrict__ rows, uint64_t* __restrict__ mask, double* __restrict__ out) {
  __shared__ double s_row[kMeshThreads / 32][kBatch][4];      // the batch's queries and 1 / support
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const Channel ch = channel_of(lane);
  const int n = counts[0], warps = gridDim.x * (kMeshThreads / 32), per = batch_rows(n, warps, kBatch);
  for (int it = (blockIdx.x * (kMeshThreads / 32) + wib) * per; it < n; it += warps * per) {
    const bool mine = lane < per && it + lane < n;
    MeshRow row{};
    int cbeg = 0, clen = 0, inside = 0;
    __syncwarp();
    if (mine) {
      const int64_t i = near[it + lane];
      row.q[0] = pos[3 * i];
      row.q[1] = pos[3 * i + 1];
      row.q[2] = pos[3 * i + 2];
      row.h = sup[i];
      const int64_t c = cell_of_query(Mv, row.q);      // listed: inside the grid
      const uint8_t fl = Mv.cflag[c];
      row.first = Mv.nstart[c];
      row.len = (int)(Mv.nstart[c + 1] - row.first);
      row.tag = (int)i;
      if (fl & kCellEmpty) {
        inside = (fl & kCellInside) ? 1 : 0;
      } else {
        const int col = column_of(Mv, row.q[0], row.q[1]);
        if (col >= 0) {
          cbeg = Mv.colstart[col];
          clen = Mv.colstart[col + 1] - cbeg;
        }
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) s_row[wib][lane][a] = row.q[a];
      s_row[wib][lane][3] = 1.0 / row.h;
    }
    __syncwarp();
    Flat<kBatch> flat;
    unsigned place;
    int r, lane0;
    flat.set(clen, lane);
    for (unsigned base = 0; base < flat.total; base += 32) {
      r = flat.row_of(base + lane, place);
      const int beg = __shfl_sync(0xffffffffu, cbeg, r);
      const double* q = s_row[wib][r];
      const bool cross = base + lane < flat.total && column_cross(Mv, Mv.colitems[beg + place], q[0], q[1], q[2]);
      const unsigned m = __ballot_sync(0xffffffffu, cross);
      const int cnt = flat.part(base, place, lane0);
      if (cnt > 0) inside ^= __popc((m >> lane0) & (0xffffffffu >> (32 - cnt))) & 1;
    }
    if (mine) {
      ind[row.tag] = inside;
      row.tag |= inside << 30;
    }
    flat.set(row.len, lane);
    // the mask is built in the listed row's place (it + lane): the place among the rows with faces is not known yet
    row.at = it + lane;
    uint64_t* const words_r = mask + (int64_t)row.at * words;
    uint64_t word = 0;
    bool any = false;
    for (unsigned base = 0; base < flat.total; base += 32) {
      r = flat.row_of(base + lane, place);
      const int64_t beg = __shfl_sync(0xffffffffu, row.first, r);
      const double* q = s_row[wib][r];
      const bool hit = base + lane < flat.total && face_within(Mv, Mv.nitems[beg + place], q, q[3]);
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      const int cnt = flat.part(base, place, lane0);
      if (cnt > 0) {
        const uint64_t bits = (m >> lane0) & (0xffffffffu >> (32 - cnt));
        const int at = (int)(place & 63u), w = (int)(place >> 6);
        any = any || bits;
        word |= bits << at;
        if (at + cnt >= 64 || place + cnt == flat.len) {       // the word is full, or the list ends
          if (w < words) words_r[w] = word;
          word = at + cnt > 64 ? bits >> (64 - at) : 0;
          if (at + cnt > 64 && place + cnt == flat.len && w + 1 < words) words_r[w + 1] = word;
        }
      }
    }
    // rows with faces: their records; the others: the constants
    const unsigned with = __ballot_sync(0xffffffffu, mine && any);
    int slot = 0;
    if (lane == 0 && with) slot = atomicAdd(&counts[1], __popc(with));
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (mine && any) rows[slot + __popc(with & ((1u << lane) - 1))] = row;
    for (unsigned none = __ballot_sync(0xffffffffu, mine && !any); none; none &= none - 1) {
      const int b = __ffs(none) - 1, tag = __shfl_sync(0xffffffffu, row.tag, b);
      const double h = __shfl_sync(0xffffffffu, row.h, b);
      if (lane < 28)
        out[(int64_t)(tag & kRowMask) * 28 + lane] = channel_value<M>(ch, 0.0, 0.0, (double)(tag >> 30), h, 1.0 / h);
    }
  }
}

// the place of the k-th set bit (k = 0, 1, ...) of m, which has more than k
__device__ __forceinline__ int select_bit(uint64_t m, int k) {
  unsigned x = (unsigned)m;
  int c = __popc(x), at = 0;
  if (k >= c) {
    k -= c;
    x = (unsigned)(m >> 32);
    at = 32;
  }
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    c = __popc(x & ((1u << w) - 1));
    if (k >= c) {
      k -= c;
      x >>= w;
      at += w;
    }
  }
  return at;
}

// Third pass, the rows with faces: the (row, face) pairs of up to 32 rows flattened on a warp's lanes, every lane one
// pair, whatever row it belongs to, so the lanes stay full although a row has some 20 faces.  The 28 terms of each pair
// go through shared memory to the lanes k < 28, which add accumulator k of the row pair after pair in the list's order
// and finish the row when the next row's first pair comes: the result does not depend on the other rows.
// On the 2^21-particle scene of 20480 faces (w4, 106 825 rows with faces, 2.6 M pairs): 0.46 ms on B200, 20011 near queries
// (w2) 0.105 ms; 12 warps per SM, bound by the latency of the float64 chains (38 % of the pipe, issue 44 %; 4 CTAs at 128
// registers: no gain).  Before, a warp took one row and spread the quadrature nodes of one edge after the other over its
// lanes (7.0 ms with the search).
constexpr int kEvalBlocks = 3;        // resident CTAs per SM (168 registers)
constexpr int kEvalRows = 32;
static_assert((INT32_MAX / 8) * (int64_t)kBatch < ((int64_t)1 << 31) && ((int64_t)1 << 26) * kEvalRows <= ((int64_t)1 << 31),
              "the flattened lists of a batch fit 32 bits: at most INT32_MAX / 8 faces a list");
constexpr int kPairStride = 29;       // doubles per pair in shared memory (28 and one against bank conflicts)

template <class M>
__global__ void __launch_bounds__(kMeshThreads, kEvalBlocks)
    k_mesh_eval(MeshView Mv, const MeshRow* __restrict__ rows, const uint64_t* __restrict__ mask, int words, int most,
                const int32_t* __restrict__ nrows, double* __restrict__ out) {
  __shared__ double s_val[kMeshThreads / 32][32 * kPairStride];
  __shared__ double s_h[kMeshThreads / 32][32];               // the round's supports and tags
  __shared__ int32_t s_tag[kMeshThreads / 32][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  double* const val = s_val[wib];
  const Channel ch = channel_of(lane);
  const int n = *nrows, warps = gridDim.x * (kMeshThreads / 32), per = batch_rows(n, warps, most);
  for (int it = (blockIdx.x * (kMeshThreads / 32) + wib) * per; it < n; it += warps * per) {
    unsigned pairs = 0;
    if (lane < per && it + lane < n) {
      const MeshRow& row = rows[it + lane];
      const uint64_t* m = mask + (int64_t)row.at * words;
      const int full = min(words, (row.len + 63) / 64);
      for (int w = 0; w < full; ++w) pairs += __popcll(m[w]);
      pairs += max(row.len - 64 * words, 0);
    }
    Flat<kEvalRows> flat;
    flat.set(pairs, lane);
    int f = -1, r = 0;
    // this lane's pair of the round at `base`: its row and its face (~face: beyond the mask, still to be tested)
    auto fetch = [&](unsigned base) {
      unsigned k;
      r = flat.row_of(base + lane, k);
      if (base + lane >= flat.total) return;
      const MeshRow& row = rows[it + r];
      const uint64_t* m = mask + (int64_t)row.at * words;
      const int full = min(words, (row.len + 63) / 64);
      for (int w = 0; w < full; ++w) {
        const uint64_t bits = m[w];
        const unsigned c = __popcll(bits);
        if (k < c) {
          f = Mv.nitems[row.first + 64 * w + select_bit(bits, (int)k)];
          return;
        }
        k -= c;
      }
      f = ~Mv.nitems[row.first + 64 * words + k];
    };
    fetch(0);
    int cur = -1;
    double acc = 0.0, h = 1.0;                                // accumulator `lane` of the row `cur`, its support
    auto finish = [&]() {
      const double a0 = __shfl_sync(0xffffffffu, acc, 0);
      if (cur >= 0 && lane < 28)
        out[(int64_t)(cur & kRowMask) * 28 + lane] = channel_value<M>(ch, acc, a0, (double)(cur >> 30), h, 1.0 / h);
    };
    for (unsigned base = 0; base < flat.total; base += 32) {
      const int f0 = f, r0 = r;
      if (base + 32 < flat.total) fetch(base + 32);           // (the next round's loads run ahead of the integration)
      if (base + lane < flat.total) {
        const MeshRow& row = rows[it + r0];
        double q[3], hr;
        ld4_nc(row.q, q[0], q[1], q[2], hr);
        const double ih = 1.0 / hr;
        s_tag[wib][lane] = row.tag;
        s_h[wib][lane] = hr;
        double o[28];
        if (f0 >= 0 || face_within(Mv, ~f0, q, ih)) {
          face_channels<M>(Mv.fdata + (int64_t)(f0 < 0 ? ~f0 : f0) * kFaceDoubles, q, ih, o);
        } else {
#pragma unroll
          for (int k = 0; k < 28; ++k) o[k] = 0.0;
        }
#pragma unroll
        for (int k = 0; k < 28; ++k) val[lane * kPairStride + k] = o[k];
      }
      __syncwarp();
      const int cnt = (int)min(flat.total - base, 32u);
      for (int k = 0; k < cnt; ++k) {
        const int tag = s_tag[wib][k];
        if (tag != cur) {
          finish();
          cur = tag;
          h = s_h[wib][k];
          acc = 0.0;
        }
        if (lane < 28) acc += val[k * kPairStride + lane];
      }
      __syncwarp();
    }
    finish();
  }
}

__global__ void k_mesh_inside_only(MeshView M, const double* __restrict__ pos, int64_t n, int32_t* __restrict__ ind) {
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n) return;
  ind[row] = mesh_inside(M, pos[3 * row], pos[3 * row + 1], pos[3 * row + 2]);
}

template <typename T>
int upload_vec(T** dst, const std::vector<T>& src) {
  const size_t bytes = std::max<size_t>(src.size(), 1) * sizeof(T);
  WSB_CUDA(cudaMalloc((void**)dst, bytes));
  if (!src.empty()) WSB_CUDA(cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
  return WSB_OK;
}

void free_mesh(Mesh* m) {
  void* ptrs[] = {m->fdata, m->nstart, m->nitems, m->colstart, m->colitems, m->cflag};
  for (void* p : ptrs)
    if (p) cudaFree(p);
}

inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// the candidate lists and flags of every cell: lengths, their prefix sums, the lists, the flags
int mesh_lists(Mesh* m, const BoxLists& L, int64_t ncells, int32_t** len) {
  WSB_CUDA(cudaMalloc((void**)len, sizeof(int32_t) * (size_t)(ncells + 1)));
  WSB_CUDA(cudaMemset(*len + ncells, 0, sizeof(int32_t)));
  WSB_CUDA(cudaMalloc((void**)&m->nstart, sizeof(int64_t) * (size_t)(ncells + 1)));
  WSB_CUDA(cudaMalloc((void**)&m->cflag, (size_t)ncells));
  constexpr int W = kMeshThreads / 32;
  const unsigned grid = (unsigned)std::min<int64_t>((ncells + W - 1) / W, 148 * 64);
  k_mesh_lists<<<grid, kMeshThreads>>>(view_of(m), L, 0, *len, nullptr);
  k_mesh_prefix<<<1, kPrefixThreads>>>(*len, ncells, m->nstart);
  int64_t total = 0;
  int32_t longest = 0;
  WSB_CUDA(cudaMemcpy(&longest, *len + ncells, sizeof(longest), cudaMemcpyDeviceToHost));
  m->eval_rows = longest > (1 << 26) ? kBatch : kEvalRows;   // the lists of a batch are flattened in 32 bits
  m->words = std::min(kMaxWords, std::max(1, (longest + 63) / 64));
  WSB_CUDA(cudaMemcpy(&total, m->nstart + ncells, sizeof(total), cudaMemcpyDeviceToHost));
  WSB_CUDA(cudaMalloc((void**)&m->nitems, sizeof(int32_t) * (size_t)std::max<int64_t>(total, 1)));
  k_mesh_lists<<<grid, kMeshThreads>>>(view_of(m), L, 1, *len, m->nitems);
  k_mesh_cellflags<<<(unsigned)((ncells + 255) / 256), 256>>>(view_of(m), L, *len, m->cflag);
  WSB_CUDA(cudaGetLastError());
  WSB_CUDA(cudaDeviceSynchronize());
  return WSB_OK;
}

// Queries are taken kMeshSlice at a time, so the workspace stops growing there (80 bytes a query and 8 per mask word past
// the first: 0.34 to 0.57 GB; 21 GB for 2^28 queries at once).  A slice of that size takes some milliseconds, its three
// launches a few microseconds.
constexpr int64_t kMeshSlice = 1 << 22;

// the workspace of n queries (of one slice): the listed rows, their number and that of the rows with faces, the indicator
// (where the caller wants none), the rows with faces and their masks
struct MeshWork {
  int32_t *near, *counts, *ind;
  MeshRow* rows;
  uint64_t* mask;
  size_t total;
};
MeshWork carve_mesh(const Mesh* m, int64_t n, void* base) {
  MeshWork w{};
  const uintptr_t p = ((uintptr_t)base + 255) & ~(uintptr_t)255;
  const size_t k = (size_t)std::min<int64_t>(std::max<int64_t>(n, 1), kMeshSlice);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += al256(bytes);
    return (void*)(p + o);
  };
  w.counts = (int32_t*)take(2 * sizeof(int32_t));
  w.near = (int32_t*)take(k * sizeof(int32_t));
  w.ind = (int32_t*)take(k * sizeof(int32_t));
  w.rows = (MeshRow*)take(k * sizeof(MeshRow));
  w.mask = (uint64_t*)take(k * m->words * sizeof(uint64_t));
  w.total = off + 256;
  return w;
}

template <class M>
int launch_mesh(const Mesh* m, const double* pos_all, const double* sup_all, int64_t n_all, double* out_all, int32_t* inside,
                const MeshWork& w, cudaStream_t st) {
  const MeshView v = view_of(m);
  const int warps = kMeshThreads / 32;
  for (int64_t at = 0; at < n_all; at += kMeshSlice) {
    const int64_t n = std::min(kMeshSlice, n_all - at);
    const double *pos = pos_all + 3 * at, *sup = sup_all + at;
    double* out = out_all + 28 * at;
    int32_t* ind = inside ? inside + at : w.ind;
    const unsigned grid = (unsigned)((n + kMeshThreads - 1) / kMeshThreads);
    const auto grid_of = [&](int blocks) {         // the resident warps, striding over the rows; no more warps than rows
      return (unsigned)std::min<int64_t>((n + warps - 1) / warps, (int64_t)148 * blocks);
    };
    WSB_CUDA(cudaMemsetAsync(w.counts, 0, 2 * sizeof(int32_t), st));
    k_mesh_rowinfo<M><<<grid, kMeshThreads, 0, st>>>(v, pos, sup, n, ind, w.near, w.counts, out);
    WSB_CUDA(cudaGetLastError());
    k_mesh_search<M><<<grid_of(kSearchBlocks), kMeshThreads, 0, st>>>(v, pos, sup, w.near, w.counts, m->words, ind, w.rows,
                                                                      w.mask, out);
    WSB_CUDA(cudaGetLastError());
    k_mesh_eval<M><<<grid_of(kEvalBlocks), kMeshThreads, 0, st>>>(v, w.rows, w.mask, m->words, m->eval_rows, w.counts + 1,
                                                                  out);
    WSB_CUDA(cudaGetLastError());
  }
  return WSB_OK;
}

}  // namespace
}  // namespace wsb

using namespace wsb;

struct wsb_mesh : public Mesh {};

extern "C" int wsb_mesh_create(const double* verts, int64_t n_verts, const int32_t* faces, int64_t n_faces,
                               double support_max, int device, wsb_mesh** out) {
  if (!out) return fail(WSB_ERR_ARG, "wsb_mesh_create: NULL handle pointer");
  *out = nullptr;
  if (!verts || !faces || n_verts < 3 || n_faces < 4)
    return fail(WSB_ERR_ARG, "wsb_mesh_create: a closed surface needs >= 3 vertices and >= 4 faces");
  if (n_faces > (int64_t)(INT32_MAX / 8)) return fail(WSB_ERR_SIZE, "wsb_mesh_create: too many faces");
  if (!(support_max > 0.0) || !std::isfinite(support_max))
    return fail(WSB_ERR_ARG, "wsb_mesh_create: support_max must be positive and finite");
  for (int64_t i = 0; i < 3 * n_verts; ++i)
    if (!std::isfinite(verts[i])) return fail(WSB_ERR_ARG, "wsb_mesh_create: non-finite vertex");
  // watertight, consistently oriented 2-manifold: every undirected edge twice, once in each direction (an open-addressing
  // table of the undirected edges, at most half full: 3 n_faces / 2 edges of a closed surface, 3 n_faces of any other)
  {
    size_t cap = 16;
    while (cap < (size_t)n_faces * 6) cap *= 2;
    std::vector<uint64_t> keys(cap, ~0ull);
    std::vector<uint8_t> dir(cap, 0);
    for (int64_t f = 0; f < n_faces; ++f) {
      const int32_t* v = faces + 3 * f;
      for (int k = 0; k < 3; ++k)
        if (v[k] < 0 || v[k] >= n_verts) return fail(WSB_ERR_ARG, "wsb_mesh_create: face index out of range");
      if (v[0] == v[1] || v[1] == v[2] || v[0] == v[2]) return fail(WSB_ERR_ARG, "wsb_mesh_create: repeated vertex");
      for (int k = 0; k < 3; ++k) {
        const int32_t a = v[k], b = v[(k + 1) % 3];
        const uint64_t key = ((uint64_t)(uint32_t)std::min(a, b) << 32) | (uint32_t)std::max(a, b);
        size_t h = (size_t)((key * 0x9E3779B97F4A7C15ull) >> 20) & (cap - 1);
        while (keys[h] != key && keys[h] != ~0ull) h = (h + 1) & (cap - 1);
        keys[h] = key;
        const uint8_t bit = a < b ? 1 : 2;
        if (dir[h] & bit)
          return fail(WSB_ERR_ARG, "wsb_mesh_create: surface must be watertight and consistently oriented");
        dir[h] |= bit;
      }
    }
    for (size_t h = 0; h < cap; ++h)
      if (keys[h] != ~0ull && dir[h] != 3)
        return fail(WSB_ERR_ARG, "wsb_mesh_create: surface must be watertight and consistently oriented");
  }
  // face records, box, signed volume (relative to the first vertex: outward normals give a positive volume)
  double vol6 = 0.0;
  const double* o = verts;
  std::vector<double> hf((size_t)n_faces * kFaceDoubles);
  double blo[3] = {INFINITY, INFINITY, INFINITY}, bhi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t f = 0; f < n_faces; ++f) {
    const int32_t* v = faces + 3 * f;
    double P[3][3];
    for (int i = 0; i < 3; ++i)
      for (int k = 0; k < 3; ++k) P[i][k] = verts[3 * v[i] + k];
    const double a[3] = {P[0][0] - o[0], P[0][1] - o[1], P[0][2] - o[2]};
    const double b[3] = {P[1][0] - o[0], P[1][1] - o[1], P[1][2] - o[2]};
    const double c[3] = {P[2][0] - o[0], P[2][1] - o[1], P[2][2] - o[2]};
    vol6 += a[0] * (b[1] * c[2] - b[2] * c[1]) - a[1] * (b[0] * c[2] - b[2] * c[0]) + a[2] * (b[0] * c[1] - b[1] * c[0]);
    double* F = hf.data() + f * kFaceDoubles;
    for (int i = 0; i < 3; ++i)
      for (int k = 0; k < 3; ++k) F[kFV + 3 * i + k] = P[i][k];
    const double e1[3] = {P[1][0] - P[0][0], P[1][1] - P[0][1], P[1][2] - P[0][2]};
    const double e2[3] = {P[2][0] - P[0][0], P[2][1] - P[0][1], P[2][2] - P[0][2]};
    const double N[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    const double nl = std::sqrt(N[0] * N[0] + N[1] * N[1] + N[2] * N[2]);
    if (!(nl > 0.0)) return fail(WSB_ERR_ARG, "wsb_mesh_create: degenerate (zero-area) face");
    for (int k = 0; k < 3; ++k) F[kFN + k] = N[k] / nl;
    for (int e = 0; e < 3; ++e) {
      const double* A = P[e];
      const double* B = P[(e + 1) % 3];
      double t[3] = {B[0] - A[0], B[1] - A[1], B[2] - A[2]};
      const double len = std::sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
      for (int k = 0; k < 3; ++k) t[k] /= len;
      for (int k = 0; k < 3; ++k) F[kFT + 3 * e + k] = t[k];
      if (v[e] < v[(e + 1) % 3]) F[kFORD] += (double)(1 << e);
      F[kFLEN + e] = len;
    }
    for (int k = 0; k < 3; ++k) {
      F[kFLO + k] = std::min(P[0][k], std::min(P[1][k], P[2][k]));
      F[kFHI + k] = std::max(P[0][k], std::max(P[1][k], P[2][k]));
      blo[k] = std::min(blo[k], F[kFLO + k]);
      bhi[k] = std::max(bhi[k], F[kFHI + k]);
    }
  }
  if (!(vol6 > 0.0)) return fail(WSB_ERR_ARG, "wsb_mesh_create: surface must have positive signed volume");
  // cell grid over the box grown by one cell; the cell is support_max, enlarged if the grid would pass 2^26 cells
  double cell = support_max;
  int64_t nx = 0, ny = 0, nz = 0;
  double lo[3] = {0, 0, 0};
  for (int tries = 0; tries < 64; ++tries) {
    for (int k = 0; k < 3; ++k) lo[k] = blo[k] - cell;
    nx = (int64_t)std::floor((bhi[0] + cell - lo[0]) / cell) + 1;
    ny = (int64_t)std::floor((bhi[1] + cell - lo[1]) / cell) + 1;
    nz = (int64_t)std::floor((bhi[2] + cell - lo[2]) / cell) + 1;
    if (nx * ny * nz <= ((int64_t)1 << 26)) break;
    cell *= 1.5;
  }
  const int64_t n3[3] = {nx, ny, nz};
  auto cidx = [&](double x, int k) {
    const int64_t i = (int64_t)std::floor((x - lo[k]) / cell);
    return std::min<int64_t>(std::max<int64_t>(i, 0), n3[k] - 1);
  };
  const int64_t ncell = nx * ny * nz;
  std::vector<int64_t> cnt(ncell + 1, 0), ccnt;
  std::vector<int32_t> fcell((size_t)n_faces * 3);
  std::vector<int64_t> range((size_t)n_faces * 6);
  for (int64_t f = 0; f < n_faces; ++f) {
    const double* F = hf.data() + f * kFaceDoubles;
    for (int k = 0; k < 3; ++k) {
      range[6 * f + 2 * k] = cidx(F[kFLO + k], k);
      range[6 * f + 2 * k + 1] = cidx(F[kFHI + k], k);
      fcell[3 * f + k] = (int32_t)range[6 * f + 2 * k];
    }
    for (int64_t kz = range[6 * f + 4]; kz <= range[6 * f + 5]; ++kz)
      for (int64_t jy = range[6 * f + 2]; jy <= range[6 * f + 3]; ++jy)
        for (int64_t ix = range[6 * f]; ix <= range[6 * f + 1]; ++ix) ++cnt[(kz * ny + jy) * nx + ix + 1];
  }
  // (x, y) columns of half a cell: the inside test meets 24 faces a column on the 20480-face scene instead of 46 with
  // whole cells; whole cells where faces far larger than a cell would list more than 2^28 items
  double col = 0.0;
  int64_t ncx = 0, ncy = 0;
  auto crange = [&](int64_t f, int64_t r[4]) {
    const double* F = hf.data() + f * kFaceDoubles;
    for (int k = 0; k < 2; ++k) {
      const int64_t top = (k == 0 ? ncx : ncy) - 1;
      r[2 * k] = std::min<int64_t>(std::max<int64_t>((int64_t)std::floor((F[kFLO + k] - lo[k]) / col), 0), top);
      r[2 * k + 1] = std::min<int64_t>(std::max<int64_t>((int64_t)std::floor((F[kFHI + k] - lo[k]) / col), 0), top);
    }
  };
  for (int split = 2; split >= 1; --split) {
    col = cell / split;
    ncx = nx * split;
    ncy = ny * split;
    ccnt.assign((size_t)(ncx * ncy) + 1, 0);
    int64_t total = 0;
    for (int64_t f = 0; f < n_faces; ++f) {
      int64_t r[4];
      crange(f, r);
      total += (r[1] - r[0] + 1) * (r[3] - r[2] + 1);
      if (split > 1 && total > ((int64_t)1 << 28)) break;
      for (int64_t jy = r[2]; jy <= r[3]; ++jy)
        for (int64_t ix = r[0]; ix <= r[1]; ++ix) ++ccnt[jy * ncx + ix + 1];
    }
    if (split == 1 || total <= ((int64_t)1 << 28)) break;
  }
  const int64_t ncol = ncx * ncy;
  for (int64_t c = 0; c < ncell; ++c) cnt[c + 1] += cnt[c];
  for (int64_t c = 0; c < ncol; ++c) ccnt[c + 1] += ccnt[c];
  if (cnt[ncell] > INT32_MAX || ccnt[ncol] > INT32_MAX)
    return fail(WSB_ERR_SIZE, "wsb_mesh_create: cell lists exceed 2^31 items");
  std::vector<int32_t> items((size_t)cnt[ncell]), citems((size_t)ccnt[ncol]);
  std::vector<int32_t> start(cnt.begin(), cnt.end()), cstart(ccnt.begin(), ccnt.end());
  {
    std::vector<int64_t>&cur = cnt, &ccur = ccnt;      // (the starts are copied: the counts serve as fill cursors)
    for (int64_t f = 0; f < n_faces; ++f) {
      for (int64_t kz = range[6 * f + 4]; kz <= range[6 * f + 5]; ++kz)
        for (int64_t jy = range[6 * f + 2]; jy <= range[6 * f + 3]; ++jy)
          for (int64_t ix = range[6 * f]; ix <= range[6 * f + 1]; ++ix)
            items[cur[(kz * ny + jy) * nx + ix]++] = (int32_t)f;
      int64_t r[4];
      crange(f, r);
      for (int64_t jy = r[2]; jy <= r[3]; ++jy)
        for (int64_t ix = r[0]; ix <= r[1]; ++ix) citems[ccur[jy * ncx + ix]++] = (int32_t)f;
    }
  }
  WSB_CUDA(cudaSetDevice(device));
  Mesh* m = new wsb_mesh();
  m->device = device;
  m->n_verts = n_verts;
  m->n_faces = n_faces;
  m->support_max = support_max;
  for (int k = 0; k < 3; ++k) m->lo[k] = lo[k];
  m->cell = cell;
  m->nx = (int32_t)nx;
  m->ny = (int32_t)ny;
  m->nz = (int32_t)nz;
  m->col = col;
  m->ncx = (int32_t)ncx;
  m->ncy = (int32_t)ncy;
  m->n_items = (int64_t)items.size();
  m->n_col_items = (int64_t)citems.size();
  // the cells' candidate lists and flags, from the box lists (device copies for the length of this call)
  const int64_t ncells = (int64_t)m->nx * m->ny * m->nz;
  int32_t *d_start = nullptr, *d_items = nullptr, *d_fcell = nullptr, *d_len = nullptr;
  int rc;
  if ((rc = upload_vec(&m->fdata, hf)) || (rc = upload_vec(&m->colstart, cstart)) ||
      (rc = upload_vec(&m->colitems, citems)) || (rc = upload_vec(&d_start, start)) ||
      (rc = upload_vec(&d_items, items)) || (rc = upload_vec(&d_fcell, fcell))) {
  } else {
    rc = mesh_lists(m, BoxLists{d_start, d_items, d_fcell}, ncells, &d_len);
  }
  for (void* p : {(void*)d_start, (void*)d_items, (void*)d_fcell, (void*)d_len})
    if (p) cudaFree(p);
  if (rc) {
    free_mesh(m);
    delete m;
    return rc;
  }
  *out = static_cast<wsb_mesh*>(m);
  return WSB_OK;
}

extern "C" int wsb_mesh_destroy(wsb_mesh* m) {
  if (!m) return WSB_OK;
  cudaSetDevice(m->device);
  free_mesh(m);
  delete m;
  return WSB_OK;
}

extern "C" size_t wsb_mesh_workspace_size(const wsb_mesh* m, int64_t n) {
  if (!m || n < 0) return 0;
  return carve_mesh(m, n, nullptr).total;
}

extern "C" int wsb_mesh_inside(const wsb_mesh* m, const double* pos, int64_t n, int32_t* inside, void* stream) {
  if (!m) return fail(WSB_ERR_ARG, "wsb_mesh_inside: NULL mesh");
  if (n < 0) return fail(WSB_ERR_ARG, "wsb_mesh_inside: negative size");
  if (n == 0) return WSB_OK;
  if (!pos || !inside) return fail(WSB_ERR_ARG, "wsb_mesh_inside: NULL array");
  WSB_CUDA(cudaSetDevice(m->device));
  k_mesh_inside_only<<<(unsigned)((n + kMeshThreads - 1) / kMeshThreads), kMeshThreads, 0, (cudaStream_t)stream>>>(
      view_of(m), pos, n, inside);
  WSB_CUDA(cudaGetLastError());
  return WSB_OK;
}

extern "C" int wsb_mesh_channels(const wsb_mesh* m, int kernel, const double* pos, const double* sup, int64_t n,
                                 double* out, int32_t* inside, void* workspace, size_t workspace_bytes, void* stream) {
  if (!m) return fail(WSB_ERR_ARG, "wsb_mesh_channels: NULL mesh");
  if (n < 0) return fail(WSB_ERR_ARG, "wsb_mesh_channels: negative size");
  if (kernel < 0 || kernel > WSB_KERNEL_W6)
    return fail(WSB_ERR_UNSUPPORTED, "wsb_mesh_channels: closed surfaces serve cubic, w2, w4, w6");
  if (n == 0) return WSB_OK;
  if (!pos || !sup || !out || !workspace) return fail(WSB_ERR_ARG, "wsb_mesh_channels: NULL array");
  if (n > (int64_t)INT32_MAX / 8) return fail(WSB_ERR_SIZE, "wsb_mesh_channels: more than 2^28 queries");
  if (workspace_bytes < wsb_mesh_workspace_size(m, n))
    return fail(WSB_ERR_SIZE, "wsb_mesh_channels: workspace smaller than wsb_mesh_workspace_size");
  WSB_CUDA(cudaSetDevice(m->device));
  const MeshWork w = carve_mesh(m, n, workspace);
  cudaStream_t st = (cudaStream_t)stream;
  switch (kernel) {
    case WSB_KERNEL_CUBIC: return launch_mesh<Mesh_cubic>(m, pos, sup, n, out, inside, w, st);
    case WSB_KERNEL_W2: return launch_mesh<Mesh_w2>(m, pos, sup, n, out, inside, w, st);
    case WSB_KERNEL_W4: return launch_mesh<Mesh_w4>(m, pos, sup, n, out, inside, w, st);
    default: return launch_mesh<Mesh_w6>(m, pos, sup, n, out, inside, w, st);
  }
}

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
//    a closed form in r = sqrt(c^2 + s^2), c^2 = z^2 + w^2, a = |z|: the line integrals of A_F are moments
//    I_n = int r^n ds (n >= -1, -2, -3), and in the divided difference
//      (r^(2m) - a^(2m)) / (r^2 - a^2)   = sum_(i<m) r^(2i) a^(2(m-1-i)),
//      (r^(2m+1) - a^(2m+1)) / (r^2 - a^2) = sum_(i<m) r^(2i+1) a^(2(m-1-i)) + a^(2m) / (r + a),
//    so a face needs its edges' w-weighted moments sum_e w_e I_n and Lambda = sum_e w_e int ds / (r + a) only, each
//    potential one dot product with them (synthetic division by r^2 - a^2, once per face).  With
//    Y = (s1 r0 - s0 r1) / c^2 (formed without cancellation), U = c^2 Y + c D, B = (r1 + c)(r0 + c), kappa = w / (c + a):
//      int ds / r = asinh Y,                      int c ds / r^2 = 2 atan(U / (B + s0 s1)) = Theta,
//      int ds / r^3 = Y / (r0 r1),                int w ds / (r (r + a)) = 2 atan(kappa U / (B + kappa^2 s0 s1)) = Omega,
//      w int ds / (r + a) = w asinh Y - a Omega,  I_n = (E_n + n c^2 I_(n-2)) / (n + 1),  E_n = [s r^n],
//      E_n = D/2 (r1^n + r0^n + S^2 / (r0 + r1) T_n),  T_n = (r1^n - r0^n) / (r1 - r0)      (D = s1 - s0, S = s1 + s0):
//    sums of terms of one sign throughout, so a short edge keeps its relative accuracy.  The rounding of a channel is
//    that of the potentials' monomial form (sum |c_n| / max |A|).
//    Powers z^p multiply the profiles whose potentials hold r^-m (m <= p) so that every face term stays bounded as
//    the query approaches the face plane.
//  * kernels of several pieces are sums of truncated blocks P(r) 1[r <= R] (the decomposition of the 2-D tables); every
//    channel is the sum of its blocks' channels, so no integral crosses a knot.
// The exact rational potentials are generated by warpsphboundaries_b200/kernels.py (mesh_blocks, emit_mesh).
#include <algorithm>
#include <cmath>
#include <map>
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
  int32_t* fcell = nullptr;    // [n_faces * 3] lowest cell of the face's box
  int32_t* fvid = nullptr;     // [n_faces * 3] vertex ids
  int32_t* cstart = nullptr;   // [nx*ny*nz + 1]
  int32_t* citems = nullptr;   // faces per cell
  int32_t* colstart = nullptr; // [nx*ny + 1] faces per (x, y) column
  int32_t* colitems = nullptr;
  uint8_t* cflag = nullptr;    // [nx*ny*nz] kCellEmpty | kCellInside | kCellNear
};

// per-cell flags: no face box meets the cell (so the surface does not cross it and every point of it has the inside
// status of its centre); that status; a face box meets one of the 27 cells around it (a query in the cell may have
// candidate faces)
enum : uint8_t { kCellEmpty = 1, kCellInside = 2, kCellNear = 4 };

// per face, one 256-byte record: v0 v1 v2 (9), unit normal N (3), edge tangents t0 t1 t2 (9), edge lengths (3), box lo
// (3), box hi (3), 2 unused; read by 32-byte loads
constexpr int kFaceDoubles = 32;
enum { kFV = 0, kFN = 9, kFT = 12, kFLEN = 21, kFLO = 24, kFHI = 27 };

struct MeshView {
  const double* fdata;
  const int32_t* fcell;
  const int32_t* fvid;
  const int32_t* cstart;
  const int32_t* citems;
  const int32_t* colstart;
  const int32_t* colitems;
  const uint8_t* cflag;
  double lo0, lo1, lo2, cell;
  int32_t nx, ny, nz;
};

namespace {

MeshView view_of(const Mesh* m) {
  return MeshView{m->fdata, m->fcell, m->fvid, m->cstart, m->citems, m->colstart, m->colitems, m->cflag,
                  m->lo[0], m->lo[1], m->lo[2], m->cell, m->nx, m->ny, m->nz};
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
  const double nzf = F[kFN + 2];
  if (nzf == 0.0) return false;                     // vertical face: its projection has no interior
  const int* vid = M.fvid + 3 * f;
  const double sgn = nzf > 0.0 ? 1.0 : -1.0;        // counter-clockwise projection for N.z > 0
  for (int e = 0; e < 3; ++e) {
    const int a = e, b = (e + 1) % 3;
    const bool fwd = vid[a] < vid[b];
    const double* A = F + kFV + 3 * (fwd ? a : b);
    const double* B = F + kFV + 3 * (fwd ? b : a);
    double E = edge_fn(A[0], A[1], B[0], B[1], x, y);
    if (!fwd) E = -E;
    E *= sgn;
    if (E < 0.0) return false;
    if (E == 0.0) {
      const double* P0 = F + kFV + 3 * a;
      const double* P1 = F + kFV + 3 * b;
      const double dx = (P1[0] - P0[0]) * sgn, dy = (P1[1] - P0[1]) * sgn;
      if (!(dy > 0.0 || (dy == 0.0 && dx < 0.0))) return false;
    }
  }
  const double zt = F[kFV + 2] - (F[kFN] * (x - F[kFV]) + F[kFN + 1] * (y - F[kFV + 1])) / nzf;
  return zt > z;
}

__device__ int mesh_inside(const MeshView& M, double x, double y, double z) {
  const int ix = cell_coord(x, M.lo0, M.cell, M.nx), iy = cell_coord(y, M.lo1, M.cell, M.ny);
  if (ix < 0 || iy < 0 || ix >= M.nx || iy >= M.ny) return 0;
  const int col = iy * M.nx + ix;
  int parity = 0;
  for (int k = M.colstart[col]; k < M.colstart[col + 1]; ++k)
    if (column_cross(M, M.colitems[k], x, y, z)) parity ^= 1;
  return parity;
}

// mesh_inside for a whole warp (every lane calls it with the same point): the lanes test the column's faces 32 at a
// time; the parity of the crossings (an integer count) is the same as the serial walk's
__device__ __forceinline__ int mesh_inside_warp(const MeshView& M, double x, double y, double z, int lane) {
  const int ix = cell_coord(x, M.lo0, M.cell, M.nx), iy = cell_coord(y, M.lo1, M.cell, M.ny);
  if (ix < 0 || iy < 0 || ix >= M.nx || iy >= M.ny) return 0;
  const int col = iy * M.nx + ix;
  const int e = M.colstart[col + 1];
  int crossings = 0;
  for (int base = M.colstart[col]; base < e; base += 32) {
    const int k = base + lane;
    crossings += __popc(__ballot_sync(0xffffffffu, k < e && column_cross(M, M.colitems[k], x, y, z)));
  }
  return crossings & 1;
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
// The cells of the block x0..x1, y0..y1, z0..z1 (at most 27) for a warp: lane l < number of cells takes cell ordinal
// l (z outermost, then y, then x -- the order of nested loops) and returns its first item (beg) and the exclusive
// prefix of the items of the cells before it (pref; a cell `keep` rejects has none).  Returns the block's total.
template <class Keep>
__device__ __forceinline__ int block_cells(const MeshView& M, int x0, int x1, int y0, int y1, int z0, int z1, int lane,
                                           Keep&& keep, int& beg, int& pref) {
  const int nxr = x1 - x0 + 1, nyr = y1 - y0 + 1, nc = nxr * nyr * (z1 - z0 + 1);
  int cnt = 0;
  beg = 0;
  if (lane < nc) {
    const int i = x0 + lane % nxr, j = y0 + (lane / nxr) % nyr, k = z0 + lane / (nxr * nyr);
    if (keep(i, j, k)) {
      const int c = (k * M.ny + j) * M.nx + i;
      beg = M.cstart[c];
      cnt = M.cstart[c + 1] - beg;
    }
  }
  int inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  pref = inc - cnt;
  return __shfl_sync(0xffffffffu, inc, 31);
}

// the cell ordinal of flattened item t (< total): the last lane whose prefix is <= t (prefixes do not decrease with
// the lane; an empty cell shares the next cell's prefix, lanes past the cells hold the total), by a binary search over
// the lanes; every lane of the warp takes part
__device__ __forceinline__ int cell_ordinal(int pref, int t) {
  int lo = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    const int pv = __shfl_sync(0xffffffffu, pref, lo + step);
    if (pv <= t) lo += step;
  }
  return lo;
}

// The faces of the 27 cells around the query's cell that come within h of the query (box first, then the exact
// triangle distance, both tested by the lanes in parallel); a face listed in several of those cells is taken in one of
// them only (the lowest corner of its box inside the 27-cell block).  Held by a whole warp for one query: the (cell,
// item) pairs of the block are flattened over the lanes, next() tests 32 of them (whatever cell they belong to) and
// returns the mask of the lanes whose face f is within h -- in cell order and item order within a cell, a fixed order,
// so the sums over the faces do not depend on the launch.
struct FaceSearch {
  double q[3], h;
  int cx, cy, cz, x0, y0, z0, nxr, nyr, beg, pref, base, total;

  __device__ __forceinline__ void start(const MeshView& M, const double* __restrict__ pos, double sup, int lane) {
#pragma unroll
    for (int a = 0; a < 3; ++a) q[a] = pos[a];
    h = sup;
    cx = cell_coord(q[0], M.lo0, M.cell, M.nx);
    cy = cell_coord(q[1], M.lo1, M.cell, M.ny);
    cz = cell_coord(q[2], M.lo2, M.cell, M.nz);
    x0 = max(cx - 1, 0);
    y0 = max(cy - 1, 0);
    z0 = max(cz - 1, 0);
    const int x1 = min(cx + 1, M.nx - 1), y1 = min(cy + 1, M.ny - 1), z1 = min(cz + 1, M.nz - 1);
    nxr = x1 - x0 + 1;
    nyr = y1 - y0 + 1;
    base = total = 0;
    if (x0 > x1 || y0 > y1 || z0 > z1) return;
    total = block_cells(M, x0, x1, y0, y1, z0, z1, lane, [](int, int, int) { return true; }, beg, pref);
  }

  __device__ __forceinline__ unsigned next(const MeshView& M, int lane, int& f) {
    const int t = base + lane;
    base += 32;
    const int o = cell_ordinal(pref, t);
    const int b = __shfl_sync(0xffffffffu, beg, o), p = __shfl_sync(0xffffffffu, pref, o);
    f = -1;
    bool hit = false;
    if (t < total) {
      const int i = x0 + o % nxr, j = y0 + (o / nxr) % nyr, k = z0 + o / (nxr * nyr);
      f = M.citems[b + (t - p)];
      const int* fc = M.fcell + 3 * f;
      if (max(fc[0], cx - 1) == i && max(fc[1], cy - 1) == j && max(fc[2], cz - 1) == k) {
        const double* F = M.fdata + (int64_t)f * kFaceDoubles;
        double d2 = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double d = fmax(0.0, fmax(F[kFLO + a] - q[a], q[a] - F[kFHI + a]));
          d2 = fma(d, d, d2);
        }
        if (d2 < h * h) {
          // the exact triangle distance (unit coordinates relative to the query, the operations of the face integral's)
          const double ih = 1.0 / h;
          double P[3][3];
#pragma unroll
          for (int v = 0; v < 3; ++v)
#pragma unroll
            for (int a = 0; a < 3; ++a) P[v][a] = (F[kFV + 3 * v + a] - q[a]) * ih;
          hit = tri_dist2(P) < 1.0;
        }
      }
    }
    return __ballot_sync(0xffffffffu, hit);
  }
};

// whether any face box comes within h of the query (the cells of FaceSearch, stopping at the first hit),
// for a whole warp (every lane calls it with the same query): the (cell, item) pairs are flattened over the lanes.
// A cell whose own box is h or more from the query is skipped: a face box within h of the query has its point nearest
// to the query in a cell within h, and every cell its box overlaps lists the face (a relative margin far above the
// rounding of the cell boxes: a cell is only skipped when clearly out of reach).
__device__ __forceinline__ bool has_candidate_warp(const MeshView& M, const double q[3], double h, int lane) {
  const int cx = cell_coord(q[0], M.lo0, M.cell, M.nx), cy = cell_coord(q[1], M.lo1, M.cell, M.ny),
            cz = cell_coord(q[2], M.lo2, M.cell, M.nz);
  const int x0 = max(cx - 1, 0), x1 = min(cx + 1, M.nx - 1), y0 = max(cy - 1, 0), y1 = min(cy + 1, M.ny - 1),
            z0 = max(cz - 1, 0), z1 = min(cz + 1, M.nz - 1);
  if (x0 > x1 || y0 > y1 || z0 > z1) return false;
  const double h2 = h * h;
  auto gap2 = [&](double x, double lo, int i) {
    const double a = fma((double)i, M.cell, lo), d = fmax(0.0, fmax(a - x, x - (a + M.cell)));
    return d * d;
  };
  auto reach = [&](int i, int j, int k) {
    return gap2(q[0], M.lo0, i) + gap2(q[1], M.lo1, j) + gap2(q[2], M.lo2, k) < h2 * (1.0 + 1e-9);
  };
  int beg, pref;
  const int total = block_cells(M, x0, x1, y0, y1, z0, z1, lane, reach, beg, pref);
  for (int base = 0; base < total; base += 32) {
    const int t = base + lane;
    const int o = cell_ordinal(pref, t);
    const int b = __shfl_sync(0xffffffffu, beg, o), p = __shfl_sync(0xffffffffu, pref, o);
    bool hit = false;
    if (t < total) {
      const double* F = M.fdata + (int64_t)M.citems[b + (t - p)] * kFaceDoubles;
      double d2 = 0.0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double d = fmax(0.0, fmax(F[kFLO + a] - q[a], q[a] - F[kFHI + a]));
        d2 = fma(d, d, d2);
      }
      hit = d2 < h2;
    }
    if (__any_sync(0xffffffffu, hit)) return true;
  }
  return false;
}

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

// coefficient n of potential f of block B, and the coefficient of its negative power
template <class B, int f, int n>
struct MeshC {
  static constexpr double v = B::kC[f][n];
};
template <class B, int f>
struct MeshNu {
  static constexpr double v = B::kNu[f];
};

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
  constexpr double R = B::kR;
  const double a = fabs(z), sg = z > 0.0 ? 1.0 : (z < 0.0 ? -1.0 : 0.0);
  if (!(a < R)) return;                 // no point of the plane within R: no chord, and the potentials vanish at |z|
  double M[B::kLine + 1];               // sum_e w_e I_n
#pragma unroll
  for (int n = 0; n <= B::kLine; ++n) M[n] = 0.0;
  double lam = 0.0, om = 0.0, th = 0.0, s3 = 0.0, out = 0.0;
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
    // the angle under which the foot of the query sees the part of the edge beyond R: the parts' unit rotations
    // multiplied (their sum lies in (-pi, pi), with the sign of w)
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
      out += atan2(y, x);
    }
    if (!in) continue;
    const double r0 = lo < s0 ? R : sqrt(fma(s0, s0, c2)), r1 = s1 < hi ? R : sqrt(fma(s1, s1, c2));
    const double D = s1 - s0, S = s1 + s0;
    const bool same = s0 > 0.0 || s1 < 0.0;                       // the chord on one side of the foot
    const double Y = (same ? D * S : s1 * r0 - s0 * r1) / (same ? s1 * r0 + s0 * r1 : c2);
    const double as = asinh(Y), U = fma(Y, c2, c * D), Bc = (r1 + c) * (r0 + c), s01 = s0 * s1, ic = 1.0 / c;
    const double kap = w / (c + a);
    const double Om = 2.0 * atan(kap * U / fmax(fma(kap * kap, s01, Bc), 1e-300));
    const double Th = 2.0 * atan(U / fmax(Bc + s01, 1e-300));
    const double ir = 1.0 / (r0 * r1), Y3 = Y * ir;
    om += Om;
    lam += w * as - a * Om;
    th += w * ic * Th;
    s3 += a * w * Y3;
    const double sr = S / (r0 + r1), qs = S * sr, eh = 0.5 * D;
    double pb = r1, pa = r0, T = 1.0, nc2 = c2;
    double Im = D;                                                // I_(n-1), I_n
    double I = 0.5 * fma(eh, (r1 + r0) + qs, c2 * as);
    M[0] = fma(w, D, M[0]);
    M[1] = fma(w, I, M[1]);
    // the four line integrals of the potentials and (A2_K2(r1) - A2_K2(r0)) / (r1 - r0)
    double k1 = fma(MeshC<B, 1, 0>::v, D, MeshNu<B, 1>::v * Th * ic), k2 = fma(MeshC<B, 2, 0>::v, D, MeshNu<B, 2>::v * Y3);
    double lw = MeshC<B, 3, 0>::v * D, ll = MeshC<B, 4, 0>::v * D, t2 = MeshC<B, 5, 1>::v - MeshNu<B, 5>::v * ir;
    if constexpr (MeshC<B, 1, 1>::v != 0.0) k1 = fma(MeshC<B, 1, 1>::v, I, k1);
    if constexpr (MeshC<B, 2, 1>::v != 0.0) k2 = fma(MeshC<B, 2, 1>::v, I, k2);
    if constexpr (MeshC<B, 3, 1>::v != 0.0) lw = fma(MeshC<B, 3, 1>::v, I, lw);
    if constexpr (MeshC<B, 4, 1>::v != 0.0) ll = fma(MeshC<B, 4, 1>::v, I, ll);
    static_for<2, B::kTop + 1>([&](auto nn) {
      constexpr int n = decltype(nn)::value;
      T = fma(r1, T, pa);
      if constexpr (MeshC<B, 5, n>::v != 0.0) t2 = fma(MeshC<B, 5, n>::v, T, t2);
      pa *= r0;
      if constexpr (n <= B::kLine) {
        pb *= r1;
        nc2 += c2;
        const double In = fma(nc2, Im, eh * fma(qs, T, pb + pa)) * (1.0 / (n + 1));
        M[n] = fma(w, In, M[n]);
        if constexpr (MeshC<B, 1, n>::v != 0.0) k1 = fma(MeshC<B, 1, n>::v, In, k1);
        if constexpr (MeshC<B, 2, n>::v != 0.0) k2 = fma(MeshC<B, 2, n>::v, In, k2);
        if constexpr (MeshC<B, 3, n>::v != 0.0) lw = fma(MeshC<B, 3, n>::v, In, lw);
        if constexpr (MeshC<B, 4, n>::v != 0.0) ll = fma(MeshC<B, 4, n>::v, In, ll);
        Im = I;
        I = In;
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
  static_for<0, 6>([&](auto ff) {
    constexpr int f = decltype(ff)::value, p = kZPow[f], m = kNeg[f];
    constexpr int top = f == 5 ? B::kTop : B::kLine;
    double J = 0.0, Aa = 0.0, b = 0.0;
    // even powers, then odd ones: synthetic division in r^2 by r^2 - z^2
    static_for<0, top / 2>([&](auto kk) {
      constexpr int i = top / 2 - decltype(kk)::value;
      b = fma(zz, b, MeshC<B, f, 2 * i>::v);
      J = fma(b, M[2 * i - 2], J);
    });
    Aa = fma(zz, b, MeshC<B, f, 0>::v);
    b = 0.0;
    static_for<0, (top + 1) / 2 - 1>([&](auto kk) {
      constexpr int i = (top + 1) / 2 - 1 - decltype(kk)::value;
      b = fma(zz, b, MeshC<B, f, 2 * i + 1>::v);
      J = fma(b, M[2 * i - 1], J);
    });
    b = fma(zz, b, MeshC<B, f, 1>::v);
    J = fma(b, lam, J) * zpow<p>(z);
    Aa = fma(a, b, Aa) * zpow<p>(z);                             // z^p A_F(|z|)
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

// the per-cell flags, once per mesh: emptiness, the inside status of an empty cell's centre (the column parity test),
// whether any of the 27 cells around holds a face
__global__ void k_mesh_cellflags(MeshView M, uint8_t* __restrict__ flags) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nxy = (int64_t)M.nx * M.ny;
  if (c >= nxy * M.nz) return;
  const int i = (int)(c % M.nx), j = (int)((c / M.nx) % M.ny), k = (int)(c / nxy);
  uint8_t f = 0;
  if (M.cstart[c] == M.cstart[c + 1]) {
    f |= kCellEmpty;
    const double x = M.lo0 + (i + 0.5) * M.cell, y = M.lo1 + (j + 0.5) * M.cell, z = M.lo2 + (k + 0.5) * M.cell;
    if (mesh_inside(M, x, y, z)) f |= kCellInside;
  }
  for (int dk = -1; dk <= 1; ++dk)
    for (int dj = -1; dj <= 1; ++dj)
      for (int di = -1; di <= 1; ++di) {
        const int a = i + di, b = j + dj, e = k + dk;
        if (a < 0 || b < 0 || e < 0 || a >= M.nx || b >= M.ny || e >= M.nz) continue;
        const int64_t n = ((int64_t)e * M.ny + b) * M.nx + a;
        if (M.cstart[n] != M.cstart[n + 1]) f |= kCellNear;
      }
  flags[c] = f;
}

// Per query, first pass: the cell's flags settle the rows away from the surface (inside status of an empty cell, no
// faces within the support when no face box meets the 27 cells around); the others are appended to `near`, so the
// second pass runs the parity walk and the face search on full warps of such rows.  Invalid rows (a support above the
// grid cell would reach faces outside the 27-cell block, non-finite input) are marked -1 and come back as NaN.
__global__ void __launch_bounds__(kMeshThreads) k_mesh_rowinfo(MeshView M, const double* __restrict__ pos,
                                                              const double* __restrict__ sup, int64_t n,
                                                              int32_t* __restrict__ ind, int32_t* __restrict__ near,
                                                              int32_t* __restrict__ nnear) {
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool listed = false;
  if (row < n) {
    const double q[3] = {pos[3 * row], pos[3 * row + 1], pos[3 * row + 2]};
    const double h = sup[row];
    const bool ok = h > 0.0 && h <= M.cell && isfinite(q[0]) && isfinite(q[1]) && isfinite(q[2]);
    if (!ok) {
      ind[row] = -1;
    } else {
      const int cx = cell_coord(q[0], M.lo0, M.cell, M.nx), cy = cell_coord(q[1], M.lo1, M.cell, M.ny),
                cz = cell_coord(q[2], M.lo2, M.cell, M.nz);
      const bool in_grid = cx >= 0 && cy >= 0 && cz >= 0 && cx < M.nx && cy < M.ny && cz < M.nz;
      // more than a cell outside the grid along some axis (cell_coord gives -2 or n + 1): the grid reaches a cell
      // (>= the support) past the surface's box, so no face is within the support and the query is outside the solid
      const bool far = cx == -2 || cy == -2 || cz == -2 || cx == M.nx + 1 || cy == M.ny + 1 || cz == M.nz + 1;
      const uint8_t f = in_grid ? M.cflag[((int64_t)cz * M.ny + cy) * M.nx + cx] : (uint8_t)(far ? 0 : kCellNear);
      if (!(f & kCellNear)) {
        ind[row] = (f & kCellInside) ? 1 : 0;     // no face box in the 27 cells: the cell is empty as well
      } else {
        listed = true;
      }
    }
  }
  const unsigned mask = __ballot_sync(0xffffffffu, listed);
  if (mask) {
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(nnear, __popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (listed) near[base + __popc(mask & ((1u << lane) - 1))] = (int32_t)row;
  }
}

// Second pass over the listed rows: the inside test (the cell's flag where the cell is empty, the parity walk
// otherwise) and whether any face is within the support; rows with faces are appended to `work`
__global__ void __launch_bounds__(kMeshThreads) k_mesh_rownear(MeshView M, const double* __restrict__ pos,
                                                              const double* __restrict__ sup,
                                                              const int32_t* __restrict__ near,
                                                              const int32_t* __restrict__ nnear,
                                                              int32_t* __restrict__ ind, int32_t* __restrict__ work,
                                                              int32_t* __restrict__ nwork) {
  // one warp per listed row (the warps of the grid stride over them): the column's faces and the candidate cells'
  // items are tested 32 at a time
  const int lane = threadIdx.x & 31;
  const int64_t m = *nnear;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t t = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; t < m; t += warps) {
    const int32_t row = near[t];
    const double q[3] = {pos[3 * row], pos[3 * row + 1], pos[3 * row + 2]};
    const double h = sup[row];
    const int cx = cell_coord(q[0], M.lo0, M.cell, M.nx), cy = cell_coord(q[1], M.lo1, M.cell, M.ny),
              cz = cell_coord(q[2], M.lo2, M.cell, M.nz);
    const bool in_grid = cx >= 0 && cy >= 0 && cz >= 0 && cx < M.nx && cy < M.ny && cz < M.nz;
    const uint8_t f = in_grid ? M.cflag[((int64_t)cz * M.ny + cy) * M.nx + cx] : (uint8_t)0;
    const int inside = (f & kCellEmpty) ? ((f & kCellInside) ? 1 : 0) : mesh_inside_warp(M, q[0], q[1], q[2], lane);
    const bool has = has_candidate_warp(M, q, h, lane);
    if (lane == 0) {
      ind[row] = inside;
      if (has) work[atomicAdd(nwork, 1)] = row;     // (the order is irrelevant: each row is computed alone)
    }
  }
}

// rows without faces in their support: whole-support constants inside, zeros outside, NaN for invalid rows.  Each
// thread builds its row in shared memory (stride 29 doubles against bank conflicts) and the block writes its
// contiguous slab of 128 x 28 outputs coalesced.
constexpr int kRowStride = 29;

template <class M>
__global__ void __launch_bounds__(kMeshThreads) k_mesh_rows(const double* __restrict__ sup, int64_t n,
                                                           const int32_t* __restrict__ ind, double* __restrict__ out) {
  __shared__ double s_rows[kMeshThreads * kRowStride];
  const int64_t row0 = (int64_t)blockIdx.x * kMeshThreads;
  const int64_t row = row0 + threadIdx.x;
  double* const mine = s_rows + threadIdx.x * kRowStride;
  if (row < n) {
    if (ind[row] < 0) {
      for (int k = 0; k < 28; ++k) mine[k] = __longlong_as_double(0x7ff8000000000000LL);
    } else {
      const double id = (double)ind[row], h = sup[row];
      for (int k = 0; k < 28; ++k) mine[k] = channel_value<M>(channel_of(k), 0.0, 0.0, id, h, 1.0 / h);
    }
  }
  __syncthreads();
  const int rows = (int)min((int64_t)kMeshThreads, n - row0);
  for (int k = threadIdx.x; k < rows * 28; k += kMeshThreads)
    out[row0 * 28 + k] = s_rows[(k / 28) * kRowStride + k % 28];
}

// The rows with faces.  A warp takes rows in turn, its lanes search a row's faces together (FaceSearch), and
// the (row, face) pairs wait in the warp's queue until there are 32: then every lane integrates one pair, whatever row
// it belongs to, so the lanes stay full although a row has some 20 faces.  The 28 terms of each pair go through shared
// memory to the lanes k < 28, which add accumulator k of the row pair after pair in queue order -- the row's face order
// -- and finish the row at its last pair: the result does not depend on the other rows of the queue.
// On the 2^21-particle scene of 20480 faces (w4, 129 562 rows, 2.6 M pairs) this takes 1.33 ms on B200 against 7.0 ms with
// a warp per row, the quadrature nodes of one edge after the other over its lanes: 0.45 Kflop an edge instead of some
// 15 Kflop, and no reduction over the lanes.
constexpr int kEvalWarps = kMeshThreads / 32;
constexpr int kEvalBlocks = 3;        // resident CTAs per SM (168 registers)
constexpr int kPairStride = 29;       // doubles per pair in shared memory (28 and one against bank conflicts)

template <class M>
__global__ void __launch_bounds__(kMeshThreads, kEvalBlocks) k_mesh_eval(MeshView Mv, const double* __restrict__ pos,
                                                                        const double* __restrict__ sup,
                                                                        const int32_t* __restrict__ ind,
                                                                        const int32_t* __restrict__ work,
                                                                        const int32_t* __restrict__ nwork,
                                                                        double* __restrict__ out) {
  __shared__ double s_val[kEvalWarps][32 * kPairStride];
  __shared__ int2 s_queue[kEvalWarps][64];             // (row, face), the row's last pair marked by ~face
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  double* const val = s_val[wib];
  int2* const queue = s_queue[wib];
  const Channel ch = channel_of(lane);
  const int nw = *nwork;
  int qn = 0;
  double acc = 0.0;                                    // accumulator `lane` of the queue's first row
  // integrates the first m pairs of the queue and finishes the rows that end among them
  auto flush = [&](int m) {
    __syncwarp();
    if (lane < m) {
      const int2 p = queue[lane];
      const int64_t row = p.x;
      const double qp[3] = {pos[3 * row], pos[3 * row + 1], pos[3 * row + 2]};
      double o[28];
      face_channels<M>(Mv.fdata + (int64_t)(p.y < 0 ? ~p.y : p.y) * kFaceDoubles, qp, 1.0 / sup[row], o);
#pragma unroll
      for (int k = 0; k < 28; ++k) val[lane * kPairStride + k] = o[k];
    }
    __syncwarp();
    for (int k = 0; k < m; ++k) {
      if (lane < 28) acc += val[k * kPairStride + lane];
      const int2 p = queue[k];
      if (p.y < 0) {
        const double acc0 = __shfl_sync(0xffffffffu, acc, 0), h = sup[p.x];
        if (lane < 28) out[(int64_t)p.x * 28 + lane] = channel_value<M>(ch, acc, acc0, (double)ind[p.x], h, 1.0 / h);
        acc = 0.0;
      }
    }
    // the pairs that stay move to the front
    const int2 p = lane + m < 64 ? queue[lane + m] : make_int2(0, 0);
    __syncwarp();
    queue[lane] = p;
    __syncwarp();
    qn -= m;
  };
  const int warps = gridDim.x * kEvalWarps;
  int it = blockIdx.x * kEvalWarps + wib - warps, row = 0;
  bool any = false;                                    // the searched row has pairs
  FaceSearch fs;
  fs.base = fs.total = 0;
  for (;;) {
    // fill the queue past 32 pairs: the first 32 then never hold the last pair of a row whose search goes on, which may
    // still have to be marked
    while (qn <= 32 && it < nw) {
      if (fs.base < fs.total) {
        int f;
        const unsigned mask = fs.next(Mv, lane, f);
        if ((mask >> lane) & 1u) queue[qn + __popc(mask & ((1u << lane) - 1))] = make_int2(row, f);
        qn += __popc(mask);
        any = any || mask;
        continue;
      }
      if (any) {
        __syncwarp();
        if (lane == 0) queue[qn - 1].y = ~queue[qn - 1].y;
        any = false;
      }
      it += warps;
      if (it >= nw) break;
      row = work[it];
      fs.start(Mv, pos + 3 * (int64_t)row, sup[row], lane);
    }
    if (qn == 0) break;
    flush(min(qn, 32));
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
  void* ptrs[] = {m->fdata, m->fcell, m->fvid, m->cstart, m->citems, m->colstart, m->colitems, m->cflag};
  for (void* p : ptrs)
    if (p) cudaFree(p);
}

inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

template <class M>
int launch_mesh(const Mesh* m, const double* pos, const double* sup, int64_t n, double* out, int32_t* ind,
                int32_t* work, int32_t* nwork, int32_t* near, cudaStream_t st) {
  const MeshView v = view_of(m);
  const unsigned grid = (unsigned)((n + kMeshThreads - 1) / kMeshThreads);
  WSB_CUDA(cudaMemsetAsync(nwork, 0, 3 * sizeof(int32_t), st));      // work rows, (unused), listed rows
  k_mesh_rowinfo<<<grid, kMeshThreads, 0, st>>>(v, pos, sup, n, ind, near, nwork + 2);
  WSB_CUDA(cudaGetLastError());
  const unsigned grid_near = (unsigned)std::min<int64_t>((n + kMeshThreads / 32 - 1) / (kMeshThreads / 32), 8192);
  k_mesh_rownear<<<grid_near, kMeshThreads, 0, st>>>(v, pos, sup, near, nwork + 2, ind, work, nwork);
  WSB_CUDA(cudaGetLastError());
  k_mesh_rows<M><<<grid, kMeshThreads, 0, st>>>(sup, n, ind, out);
  WSB_CUDA(cudaGetLastError());
  // the resident warps, striding over the work rows (no more warps than rows)
  const unsigned egrid =
      (unsigned)std::min<int64_t>((n + kEvalWarps - 1) / kEvalWarps, (int64_t)148 * kEvalBlocks);
  k_mesh_eval<M><<<egrid, kMeshThreads, 0, st>>>(v, pos, sup, ind, work, nwork, out);
  WSB_CUDA(cudaGetLastError());
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
  // watertight, consistently oriented 2-manifold: every undirected edge twice, once in each direction
  std::map<std::pair<int32_t, int32_t>, int> dir;
  for (int64_t f = 0; f < n_faces; ++f) {
    const int32_t* v = faces + 3 * f;
    for (int k = 0; k < 3; ++k)
      if (v[k] < 0 || v[k] >= n_verts) return fail(WSB_ERR_ARG, "wsb_mesh_create: face index out of range");
    if (v[0] == v[1] || v[1] == v[2] || v[0] == v[2]) return fail(WSB_ERR_ARG, "wsb_mesh_create: repeated vertex");
    for (int k = 0; k < 3; ++k) {
      const int32_t a = v[k], b = v[(k + 1) % 3];
      const auto key = std::make_pair(std::min(a, b), std::max(a, b));
      const int bit = a < b ? 1 : 2;
      int& d = dir[key];
      if (d & bit) return fail(WSB_ERR_ARG, "wsb_mesh_create: surface must be watertight and consistently oriented");
      d |= bit;
    }
  }
  for (const auto& kv : dir)
    if (kv.second != 3) return fail(WSB_ERR_ARG, "wsb_mesh_create: surface must be watertight and consistently oriented");
  // face records, box, signed volume (relative to the first vertex: outward normals give a positive volume)
  double vol6 = 0.0;
  const double* o = verts;
  std::vector<double> hf((size_t)n_faces * kFaceDoubles);
  std::vector<int32_t> hvid((size_t)n_faces * 3);
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
      F[kFLEN + e] = len;
    }
    for (int k = 0; k < 3; ++k) {
      F[kFLO + k] = std::min(P[0][k], std::min(P[1][k], P[2][k]));
      F[kFHI + k] = std::max(P[0][k], std::max(P[1][k], P[2][k]));
      blo[k] = std::min(blo[k], F[kFLO + k]);
      bhi[k] = std::max(bhi[k], F[kFHI + k]);
      hvid[3 * f + k] = v[k];
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
  const int64_t ncell = nx * ny * nz, ncol = nx * ny;
  std::vector<int64_t> cnt(ncell + 1, 0), ccnt(ncol + 1, 0);
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
    for (int64_t jy = range[6 * f + 2]; jy <= range[6 * f + 3]; ++jy)
      for (int64_t ix = range[6 * f]; ix <= range[6 * f + 1]; ++ix) ++ccnt[jy * nx + ix + 1];
  }
  for (int64_t c = 0; c < ncell; ++c) cnt[c + 1] += cnt[c];
  for (int64_t c = 0; c < ncol; ++c) ccnt[c + 1] += ccnt[c];
  if (cnt[ncell] > INT32_MAX || ccnt[ncol] > INT32_MAX)
    return fail(WSB_ERR_SIZE, "wsb_mesh_create: cell lists exceed 2^31 items");
  std::vector<int32_t> items((size_t)cnt[ncell]), citems((size_t)ccnt[ncol]);
  std::vector<int32_t> start(cnt.begin(), cnt.end()), cstart(ccnt.begin(), ccnt.end());
  {
    std::vector<int64_t> cur(cnt.begin(), cnt.end() - 1), ccur(ccnt.begin(), ccnt.end() - 1);
    for (int64_t f = 0; f < n_faces; ++f) {
      for (int64_t kz = range[6 * f + 4]; kz <= range[6 * f + 5]; ++kz)
        for (int64_t jy = range[6 * f + 2]; jy <= range[6 * f + 3]; ++jy)
          for (int64_t ix = range[6 * f]; ix <= range[6 * f + 1]; ++ix)
            items[cur[(kz * ny + jy) * nx + ix]++] = (int32_t)f;
      for (int64_t jy = range[6 * f + 2]; jy <= range[6 * f + 3]; ++jy)
        for (int64_t ix = range[6 * f]; ix <= range[6 * f + 1]; ++ix) citems[ccur[jy * nx + ix]++] = (int32_t)f;
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
  m->n_items = (int64_t)items.size();
  m->n_col_items = (int64_t)citems.size();
  int rc;
  if ((rc = upload_vec(&m->fdata, hf)) || (rc = upload_vec(&m->fcell, fcell)) || (rc = upload_vec(&m->fvid, hvid)) ||
      (rc = upload_vec(&m->cstart, start)) || (rc = upload_vec(&m->citems, items)) ||
      (rc = upload_vec(&m->colstart, cstart)) || (rc = upload_vec(&m->colitems, citems)) ||
      (rc = upload_vec(&m->cflag, std::vector<uint8_t>((size_t)m->nx * m->ny * m->nz, 0)))) {
    free_mesh(m);
    delete m;
    return rc;
  }
  const int64_t ncells = (int64_t)m->nx * m->ny * m->nz;
  k_mesh_cellflags<<<(unsigned)((ncells + 255) / 256), 256>>>(view_of(m), m->cflag);
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    free_mesh(m);
    delete m;
    return cuda_fail(e, "wsb_mesh_create: cell flags");
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
  return al256(sizeof(int32_t) * (size_t)std::max<int64_t>(n, 1)) * 3 + 256;
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
  char* base = (char*)workspace;
  const size_t s = al256(sizeof(int32_t) * (size_t)n);
  int32_t* work = (int32_t*)base;
  int32_t* ind = inside ? inside : (int32_t*)(base + s);
  int32_t* nwork = (int32_t*)(base + 2 * s);     // [3]: work rows, (unused), listed rows
  int32_t* near = (int32_t*)(base + 2 * s + 256);
  cudaStream_t st = (cudaStream_t)stream;
  switch (kernel) {
    case WSB_KERNEL_CUBIC: return launch_mesh<Mesh_cubic>(m, pos, sup, n, out, ind, work, nwork, near, st);
    case WSB_KERNEL_W2: return launch_mesh<Mesh_w2>(m, pos, sup, n, out, ind, work, nwork, near, st);
    case WSB_KERNEL_W4: return launch_mesh<Mesh_w4>(m, pos, sup, n, out, ind, work, nwork, near, st);
    default: return launch_mesh<Mesh_w6>(m, pos, sup, n, out, ind, work, nwork, near, st);
  }
}

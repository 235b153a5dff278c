// Signed distance of points to a surface: the nearest edge by a bounding-box tree over the edges, the sign by the
// winding indicator (src/warpSPHBoundaries/scene/scene.py:1312-1372).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <vector>

#include "common.cuh"

namespace wsb {
namespace {

constexpr int kDistThreads = 128;
constexpr int kGroup = 8;            // lanes per point, children per node, edges per leaf
constexpr int kTreeLevels = 11;      // 8^10 leaves of 8 edges cover 2^31 edges

// The tree: edges in Morton order of their midpoints, leaves of 8 consecutive edges, node i of a level over the nodes
// 8i .. 8i+7 of the level below; boxes of a level's nodes stored one after the other (off[level]), leaves first.
struct TreeView {
  const double4* box;       // (lo x, lo y, hi x, hi y) of every node, by level
  const double4* rec;       // edge records (a, b) in tree order
  const int32_t* id;        // their edge ids
  int32_t n_edges;
  int32_t levels;           // the root's level (its only node)
  int32_t off[kTreeLevels], cnt[kTreeLevels];
};

// the segment distance of a point to edge record r with the rounding of the reference's brute force; the nearest
// edge wins, the lower edge id on an exact tie (the order of a scan over all edges)
__device__ __forceinline__ void nearest_edge(double px, double py, const double4& r, int32_t e, double& best, double& bx,
                                             double& by, int32_t& be) {
  const double ex = __dsub_rn(r.z, r.x), ey = __dsub_rn(r.w, r.y);
  double t = __ddiv_rn(__dadd_rn(__dmul_rn(__dsub_rn(px, r.x), ex), __dmul_rn(__dsub_rn(py, r.y), ey)),
                       __dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)));
  t = fmin(fmax(t, 0.0), 1.0);
  const double cx = __dadd_rn(r.x, __dmul_rn(t, ex)), cy = __dadd_rn(r.y, __dmul_rn(t, ey));
  const double ddx = __dsub_rn(px, cx), ddy = __dsub_rn(py, cy);
  const double dist = __dsqrt_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)));
  if (dist < best || (dist == best && e < be)) {
    best = dist;
    bx = cx;
    by = cy;
    be = e;
  }
}

// squared distance of a point to a box
__device__ __forceinline__ double box_d2(double px, double py, const double4& b) {
  const double dx = fmax(0.0, fmax(b.x - px, px - b.z)), dy = fmax(0.0, fmax(b.y - py, py - b.w));
  return fma(dx, dx, dy * dy);
}

// minimum over the eight lanes of a group
__device__ __forceinline__ uint32_t group_min(uint32_t v, unsigned mask) {
#pragma unroll
  for (int o = kGroup / 2; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(mask, v, o, kGroup));
  return v;
}

// The nearest edge of a point, for a group of eight lanes (lane k of them: sub): lane k tests child k of a node and edge
// k of a leaf.  Nodes are visited nearest first and skipped when their box is farther than the best distance (a margin
// of 1e-12 over the rounding of the box distance, so an edge at the same distance is met and the lower id wins): same
// distance, closest point and edge as a scan over all edges, from some dozen boxes and leaves.  `keys` (this lane's
// column of shared memory, a row per level): the child's squared distance as a float rounded down, its lowest three bits
// replaced by the lane; ~0 for no child or one already visited.
// (Measured on B200, 200 003 random points among 17 400 edges: square rings of support-sized cells 12.3 ms -- and all
// edges for points outside the grid -- , a thread per point over a 4-ary tree 0.72 ms at 5 of 32 lanes active, this
// 0.42 ms; still far from the 0.01 ms of its memory: some 1350 instructions a point in visits to nodes and leaves.)
__device__ __forceinline__ void nearest_in_tree(const TreeView& T, double px, double py, int sub, unsigned mask,
                                                uint32_t* keys, double& best, double& bx, double& by, int32_t& be) {
  auto child_key = [&](int level, int32_t node) {      // of child `sub` of a node of `level` >= 1
    const int32_t c = kGroup * node + sub;
    if (c >= T.cnt[level - 1]) return 0xffffffffu;
    return (__float_as_uint(__double2float_rd(box_d2(px, py, T.box[T.off[level - 1] + c]))) & ~7u) | (uint32_t)sub;
  };
  auto scan_leaf = [&](int32_t leaf) {
    const int32_t i = kGroup * leaf + sub;
    if (i < T.n_edges) nearest_edge(px, py, T.rec[i], T.id[i], best, bx, by, be);
    return group_min(__float_as_uint(__double2float_ru(best * best * (1.0 + 1e-12))), mask);
  };
  uint32_t lim = 0x7f800000u;        // the best squared distance, rounded up (the bits of a float >= 0 order as it does)
  int level = T.levels;
  int32_t node = 0;
  uint32_t key = 0xffffffffu;
  if (level == 0)
    scan_leaf(0);
  else
    key = child_key(level, 0);
  for (;;) {
    const uint32_t m = group_min(key, mask);
    if (m == 0xffffffffu || (m & ~7u) > lim) {         // no child left within reach: back to the parent
      if (level == T.levels) break;
      ++level;
      node /= kGroup;
      key = keys[level * kDistThreads];
      continue;
    }
    const int c = (int)(m & 7u);
    if (sub == c) key = 0xffffffffu;
    if (level == 1) {
      lim = scan_leaf(kGroup * node + c);
    } else {
      keys[level * kDistThreads] = key;
      --level;
      node = kGroup * node + c;
      key = child_key(level, node);
    }
  }
  // the group's nearest, the lower id on a tie, in every lane
#pragma unroll
  for (int o = kGroup / 2; o > 0; o >>= 1) {
    const double d = __shfl_xor_sync(mask, best, o, kGroup), x = __shfl_xor_sync(mask, bx, o, kGroup),
                 y = __shfl_xor_sync(mask, by, o, kGroup);
    const int32_t e = __shfl_xor_sync(mask, be, o, kGroup);
    if (e >= 0 && (be < 0 || d < best || (d == best && e < be))) {
      best = d;
      bx = x;
      by = y;
      be = e;
    }
  }
}

// The winding indicator of a point, for its group of lanes: in a cell with edges the cell centre's exact winding and the
// signed crossings of the segment from the centre to the point over the cell's candidates (as the row pass of the
// aggregate; some 10 edges instead of the 110 of a y bin), the ray cast where an orientation is uncertain or the centre's
// winding is.
__device__ __forceinline__ double indicator_near(const SurfView& S, double px, double py, double h, bool in_grid,
                                                 int32_t cid, int sub, unsigned mask) {
  if (in_grid && S.cempty[cid] == 0 && S.cok[cid] != 0) {
    const int32_t cx = cid / S.ny, cy = cid % S.ny;
    const double rx = __dadd_rn(S.lo_x, __dmul_rn(__dadd_rn((double)cx, 0.5), S.cell));
    const double ry = __dadd_rn(S.lo_y, __dmul_rn(__dadd_rn((double)cy, 0.5), S.cell));
    bool degenerate = false;
    int cross = 0;
    const int32_t k1 = S.cstart[cid + 1];
    for (int32_t k = S.cstart[cid] + sub; k < k1; k += kGroup)
      cross += segment_crossing(rx, ry, px, py, S.crec[k], &degenerate);
    int v = cross + (degenerate ? 1 << 24 : 0);        // (a lane's crossings stay far below 2^20)
#pragma unroll
    for (int o = kGroup / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, kGroup);
    if (v < (1 << 23)) return S.cind[cid] + (double)v;
  }
  return indicator_at(S, px, py, h, in_grid, cid);
}

struct Nearest {
  double d, cx, cy, n0, n1;      // signed distance, closest point, outward normal
  int32_t edge;
};

__device__ __forceinline__ Nearest signed_nearest(const SurfView& S, const TreeView& T, const double4* __restrict__ erec,
                                                  double px, double py, double norm_support, int sub, unsigned mask,
                                                  uint32_t* keys) {
  Nearest o{INFINITY, 0.0, 0.0, 0.0, 0.0, -1};
  double best = INFINITY;
  int32_t be = -1;
  nearest_in_tree(T, px, py, sub, mask, keys, best, o.cx, o.cy, be);
  int32_t cid;
  const bool in_grid = cell_of(S, px, py, cid);
  const double ind = indicator_near(S, px, py, norm_support > 0.0 ? norm_support : 1.0, in_grid, cid,
                                    sub, mask);
  const bool ins = ind > 0.5;
  o.d = ins ? -best : best;
  o.edge = be;
  if (be >= 0) {
    const double4 r = erec[be];
    const double ex = r.z - r.x, ey = r.w - r.y;
    const double el = sqrt(ex * ex + ey * ey);
    o.n0 = ey / el;
    o.n1 = -ex / el;
  }
  const double vx = px - o.cx, vy = py - o.cy;
  const double dn = sqrt(vx * vx + vy * vy);
  if (dn > 1e-12 && !ins) {
    o.n0 = vx / fmax(dn, 1e-300);
    o.n1 = vy / fmax(dn, 1e-300);
  }
  return o;
}

// the point of a group of eight lanes, the lane's place in it, the group's lanes of the warp and the lane's column of keys
struct Group {
  int64_t i;
  int sub;
  unsigned mask;
};
__device__ __forceinline__ Group group_of() {
  const int lane = threadIdx.x & 31;
  return {(blockIdx.x * (int64_t)kDistThreads + threadIdx.x) / kGroup, lane % kGroup,
          0xffu << (lane / kGroup * kGroup)};
}

__global__ void __launch_bounds__(kDistThreads, 16) k_signed_distance(SurfView S, const TreeView T,
                                                                 const double* __restrict__ lpos, int64_t m,
                                                                 double norm_support, double* d, double* cp, double* nl,
                                                                 int32_t* edge) {
  __shared__ uint32_t s_keys[kTreeLevels * kDistThreads];
  const Group g = group_of();
  const int64_t i = g.i;
  if (i >= m) return;
  const Nearest o = signed_nearest(S, T, S.erec, lpos[2 * i], lpos[2 * i + 1], norm_support, g.sub, g.mask,
                                   s_keys + threadIdx.x);
  if (g.sub != 0) return;
  d[i] = o.d;
  cp[2 * i] = o.cx;
  cp[2 * i + 1] = o.cy;
  edge[i] = o.edge;
  nl[2 * i] = o.n0;
  nl[2 * i + 1] = o.n1;
}

// One surface of a body in one pass over world points: into the body frame, the signed distance, the normal back to the
// world frame, and the nearest body so far kept (d < best; `first`: nothing before).  The frame changes are the rounded
// operations of Pose.toLocal / vecToWorld (scene.py:75-90).
__global__ void __launch_bounds__(kDistThreads, 16) k_body_distance(SurfView S, const TreeView T,
                                                               const double* __restrict__ pos, int64_t m,
                                                               const double* __restrict__ pose, double norm_support,
                                                               int first, int64_t body, double* best, double* normal,
                                                               int64_t* bidx) {
  __shared__ uint32_t s_keys[kTreeLevels * kDistThreads];
  const Group g = group_of();
  const int64_t i = g.i;
  if (i >= m) return;
  const double c = pose[2], s = pose[3];
  double lx, ly;
  to_local_rn(pos[2 * i], pos[2 * i + 1], pose[0], pose[1], c, s, lx, ly);
  const Nearest o = signed_nearest(S, T, S.erec, lx, ly, norm_support, g.sub, g.mask, s_keys + threadIdx.x);
  if (g.sub != 0) return;
  const bool better = o.d < (first ? INFINITY : best[i]);
  if (!better && !first) return;
  best[i] = better ? o.d : INFINITY;
  normal[2 * i] = better ? __dsub_rn(__dmul_rn(o.n0, c), __dmul_rn(o.n1, s)) : 0.0;
  normal[2 * i + 1] = better ? __dadd_rn(__dmul_rn(o.n0, s), __dmul_rn(o.n1, c)) : 0.0;
  if (bidx) bidx[i] = better ? body : -1;
}

TreeView view_of_tree(const Surface* s) {
  TreeView T{};
  T.box = s->tbox;
  T.rec = s->trec;
  T.id = s->tid;
  T.n_edges = (int32_t)s->n_edges;
  int64_t n = (s->n_edges + kGroup - 1) / kGroup, off = 0;
  for (int l = 0; l < kTreeLevels; ++l) {
    T.off[l] = (int32_t)off;
    T.cnt[l] = (int32_t)n;
    T.levels = l;
    if (n == 1) break;
    off += n;
    n = (n + kGroup - 1) / kGroup;
  }
  return T;
}

// the tree's host arrays: boxes by level, edge ids in Morton order (11 bits an axis over the midpoints'
// box, finer than the leaves need)
void edge_tree(const std::vector<double4>& erec, std::vector<double4>& box, std::vector<int32_t>& id) {
  const int64_t n = (int64_t)erec.size();
  const double4* rec = erec.data();
  double lx = INFINITY, ly = INFINITY, hx = -INFINITY, hy = -INFINITY;
  for (int64_t e = 0; e < n; ++e) {
    const double mx = 0.5 * rec[e].x + 0.5 * rec[e].z, my = 0.5 * rec[e].y + 0.5 * rec[e].w;
    lx = std::min(lx, mx);
    ly = std::min(ly, my);
    hx = std::max(hx, mx);
    hy = std::max(hy, my);
  }
  auto spread = [](uint32_t v) {
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    return (v | (v << 1)) & 0x55555555u;
  };
  const double sx = hx > lx ? 2047.0 / (hx - lx) : 0.0, sy = hy > ly ? 2047.0 / (hy - ly) : 0.0;
  std::vector<uint64_t> key((size_t)n), tmp((size_t)n);
  uint64_t* kp = key.data();
  for (int64_t e = 0; e < n; ++e) {
    const double mx = 0.5 * rec[e].x + 0.5 * rec[e].z, my = 0.5 * rec[e].y + 0.5 * rec[e].w;
    const uint32_t qx = (uint32_t)(int32_t)std::min(2047.0, std::max(0.0, (mx - lx) * sx));
    const uint32_t qy = (uint32_t)(int32_t)std::min(2047.0, std::max(0.0, (my - ly) * sy));
    kp[e] = ((uint64_t)(spread(qx) | (spread(qy) << 1)) << 32) | (uint64_t)e;
  }
  std::vector<uint32_t> count(2 * 2048, 0);
  uint32_t* c0 = count.data();
  for (int64_t e = 0; e < n; ++e) {
    ++c0[(kp[e] >> 32) & 2047];
    ++c0[2048 + (kp[e] >> 43)];
  }
  uint64_t *a = kp, *b = tmp.data();
  for (int pass = 0; pass < 2; ++pass) {               // radix sort of the 22-bit codes
    uint32_t* c = c0 + 2048 * pass;
    uint32_t sum = 0;
    for (int k = 0; k < 2048; ++k) {
      const uint32_t v = c[k];
      c[k] = sum;
      sum += v;
    }
    for (int64_t e = 0; e < n; ++e) b[c[(a[e] >> (32 + 11 * pass)) & 2047]++] = a[e];
    std::swap(a, b);
  }
  id.resize((size_t)n);
  int32_t* ip = id.data();
  for (int64_t i = 0; i < n; ++i) ip[i] = (int32_t)(uint32_t)a[i];
  size_t n_box = 0;
  for (int64_t m = n; m > 1 || n_box == 0;) {
    m = (m + kGroup - 1) / kGroup;
    n_box += (size_t)m;
  }
  box.resize(n_box);
  double4* bp = box.data();
  size_t end = 0;
  for (int64_t i = 0; i < n; i += kGroup) {
    double x0 = INFINITY, y0 = INFINITY, x1 = -INFINITY, y1 = -INFINITY;
    const int64_t last = std::min<int64_t>(i + kGroup, n);
    for (int64_t k = i; k < last; ++k) {
      const double4& r = rec[ip[k]];
      x0 = std::min(x0, std::min(r.x, r.z));
      y0 = std::min(y0, std::min(r.y, r.w));
      x1 = std::max(x1, std::max(r.x, r.z));
      y1 = std::max(y1, std::max(r.y, r.w));
    }
    bp[end++] = make_double4(x0, y0, x1, y1);
  }
  for (size_t start = 0, stop = end; stop - start > 1; start = stop, stop = end) {
    for (size_t i = start; i < stop; i += kGroup) {
      double4 v = bp[i];
      for (size_t k = i + 1; k < std::min(i + kGroup, stop); ++k)
        v = make_double4(std::min(v.x, bp[k].x), std::min(v.y, bp[k].y), std::max(v.z, bp[k].z), std::max(v.w, bp[k].w));
      bp[end++] = v;
    }
  }
}

// The tree of a surface, built by the first signed distance asked of it: 0.26 ms on the host for 17 400 edges, which the
// surfaces of callers that ask for none (aggregates, adjoints, a geometry rebuilt each step) do not pay.  Safe from any
// thread; a stream that is being captured is not touched (a stream of its own, host-synchronised before the tree is
// published), and allocations during another stream's capture are permitted for the length of the call.
int edge_tree_of(const Surface* s, TreeView* out) try {
  std::lock_guard<std::mutex> lock(s->tree_mu);
  if (!s->tbox) {
    std::vector<double4> box;
    std::vector<int32_t> id;
    edge_tree(s->herec, box, id);
    const size_t nb = box.size(), n = (size_t)s->n_edges;
    std::vector<double4> all(nb + n + (n * sizeof(int32_t) + sizeof(double4) - 1) / sizeof(double4));
    std::copy(box.begin(), box.end(), all.begin());
    for (size_t i = 0; i < n; ++i) all[nb + i] = s->herec[(size_t)id[i]];
    std::memcpy(all.data() + nb + n, id.data(), n * sizeof(int32_t));
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    WSB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    double4* dev = nullptr;
    cudaStream_t st = nullptr;
    cudaError_t e = cudaMalloc((void**)&dev, all.size() * sizeof(double4));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dev, all.data(), all.size() * sizeof(double4), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (st) cudaStreamDestroy(st);
    if (e != cudaSuccess && dev) cudaFree(dev);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {
      cudaGetLastError();                              // (an allocation that failed is not the next launch's error)
      return cuda_fail(e, "signed distance: edge tree");
    }
    s->trec = dev + nb;
    s->tid = reinterpret_cast<const int32_t*>(dev + nb + n);
    s->tbox = dev;
    std::vector<double4>().swap(s->herec);
  }
  *out = view_of_tree(s);
  return WSB_OK;
} catch (const std::bad_alloc&) {
  return fail(WSB_ERR_DEVICE, "signed distance: no host memory for the edge tree");
}

}  // namespace
}  // namespace wsb

using namespace wsb;

extern "C" int wsb_signed_distance(const wsb_surface* s_, const double* lpos, int64_t m, double norm_support,
                                   double* d, double* cp, double* n_loc, int32_t* edge, void* stream) {
  const Surface* s = reinterpret_cast<const Surface*>(s_);
  if (!s) return fail(WSB_ERR_ARG, "wsb_signed_distance: NULL surface");
  if (m < 0) return fail(WSB_ERR_ARG, "wsb_signed_distance: negative point count");
  if (m == 0) return WSB_OK;
  if (!lpos || !d || !cp || !n_loc || !edge) return fail(WSB_ERR_ARG, "wsb_signed_distance: NULL array");
  WSB_CUDA(cudaSetDevice(s->device));
  TreeView tree;
  if (const int rc = edge_tree_of(s, &tree)) return rc;
  k_signed_distance<<<(unsigned)((m * kGroup + kDistThreads - 1) / kDistThreads), kDistThreads, 0, (cudaStream_t)stream>>>(
      view_of(s), tree, lpos, m, norm_support, d, cp, n_loc, edge);
  WSB_CUDA(cudaGetLastError());
  return WSB_OK;
}

extern "C" int wsb_body_distance(const wsb_surface* s_, const double* pos, int64_t m, const double* pose,
                                 double norm_support, int first, int64_t body, double* best, double* normal,
                                 int64_t* body_index, void* stream) {
  const Surface* s = reinterpret_cast<const Surface*>(s_);
  if (!s) return fail(WSB_ERR_ARG, "wsb_body_distance: NULL surface");
  if (m < 0) return fail(WSB_ERR_ARG, "wsb_body_distance: negative point count");
  if (m == 0) return WSB_OK;
  if (!pos || !pose || !best || !normal) return fail(WSB_ERR_ARG, "wsb_body_distance: NULL array");
  WSB_CUDA(cudaSetDevice(s->device));
  TreeView tree;
  if (const int rc = edge_tree_of(s, &tree)) return rc;
  k_body_distance<<<(unsigned)((m * kGroup + kDistThreads - 1) / kDistThreads), kDistThreads, 0, (cudaStream_t)stream>>>(
      view_of(s), tree, pos, m, pose, norm_support, first, body, best, normal, body_index);
  WSB_CUDA(cudaGetLastError());
  return WSB_OK;
}

// LBVH build on the device: triangle records, Morton codes sorted (m2s_sort.cu),
// Karras (2012) binary radix tree emission, a bottom-up refit and pillboxes.
//
// The tree replaces the bvh 0.10 / rstar 0.12 trees of the Rust crate
// (generate/generic/bvh.rs:230-254, rtree.rs:279-304, rtree_bvh.rs:100-141,
// generate/grid.rs:95-114).  Those trees only pre-filter candidates; every
// result is decided by the exact f32 tests of m2s_geo.cuh, so any tree over
// the same padded boxes (geo.rs:4-22) yields the same answers.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "m2s_internal.cuh"

namespace m2s {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ uint32_t load_index(const void* idx, int bits, uint64_t k) {
  if (bits == 16) return ((const uint16_t*)idx)[k];
  if (bits == 32) return ((const uint32_t*)idx)[k];
  return (uint32_t)k;
}

// Topology::get_triangles (lib.rs:193-215): a list takes indices 3t..3t+2, a
// strip the window t..t+2 with no winding flip.  Indices >= n_vertices raise
// M2S_ERR_INDEX_RANGE (the crate panics through slice indexing).
__global__ void k_setup(MeshInput in, TriRec* __restrict__ tris, float4* __restrict__ boxes, uint32_t* status) {
  uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= in.n_tris) return;
  uint64_t base = in.topology == 0 ? 3 * t : t;
  uint64_t i0 = in.index_bits ? load_index(in.d_indices, in.index_bits, base) : base;
  uint64_t i1 = in.index_bits ? load_index(in.d_indices, in.index_bits, base + 1) : base + 1;
  uint64_t i2 = in.index_bits ? load_index(in.d_indices, in.index_bits, base + 2) : base + 2;
  if (i0 >= in.n_vertices || i1 >= in.n_vertices || i2 >= in.n_vertices) {
    atomicOr(status, bit(M2S_ERR_INDEX_RANGE));
    i0 = i1 = i2 = 0;
    if (in.n_vertices == 0) return;
  }
  const float* v = in.d_vertices;
  P3 a = {v[3 * i0], v[3 * i0 + 1], v[3 * i0 + 2]};
  P3 b = {v[3 * i1], v[3 * i1 + 1], v[3 * i1 + 2]};
  P3 c = {v[3 * i2], v[3 * i2 + 1], v[3 * i2 + 2]};
  int kind = degenerate_kind(a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z);
  TriRec r;
  r.a = make_float4(a.x, a.y, a.z, __int_as_float(kind));
  r.b = make_float4(b.x, b.y, b.z, __uint_as_float((uint32_t)t));
  r.c = make_float4(c.x, c.y, c.z, 0.0f);
  tris[t] = r;
  P3 lo, hi;
  padded_box(a, b, c, &lo, &hi);
  boxes[2 * t] = make_float4(lo.x, lo.y, lo.z, 0.0f);
  boxes[2 * t + 1] = make_float4(hi.x, hi.y, hi.z, 0.0f);
}

// Order-preserving float <-> uint maps for atomic min / max.
__device__ __forceinline__ uint32_t f2o(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

__global__ void k_bounds_init(uint32_t* b) {
  if (threadIdx.x < 3) b[threadIdx.x] = 0xFFFFFFFFu;
  else if (threadIdx.x < 6) b[threadIdx.x] = 0u;
}

// Bounds of the box centroids (the Morton quantisation domain).
__global__ void k_bounds(const float4* __restrict__ boxes, uint64_t n, uint32_t* b) {
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x) {
    float4 lo = boxes[2 * t], hi = boxes[2 * t + 1];
    float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
    for (int d = 0; d < 3; ++d) {
      mn[d] = fminf(mn[d], c[d]);
      mx[d] = fmaxf(mx[d], c[d]);
    }
  }
  for (int d = 0; d < 3; ++d)
    for (int o = 16; o; o >>= 1) {
      mn[d] = fminf(mn[d], __shfl_xor_sync(0xFFFFFFFFu, mn[d], o));
      mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xFFFFFFFFu, mx[d], o));
    }
  if ((threadIdx.x & 31) == 0)
    for (int d = 0; d < 3; ++d) {
      atomicMin(&b[d], f2o(mn[d]));
      atomicMax(&b[3 + d], f2o(mx[d]));
    }
}

// 10-bit spread: bit i of x moves to bit 3i.
__device__ __forceinline__ uint32_t spread10(uint32_t x) {
  x &= 0x3FFu;
  x = (x | (x << 16)) & 0x030000FFu;
  x = (x | (x << 8)) & 0x0300F00Fu;
  x = (x | (x << 4)) & 0x030C30C3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

__global__ void k_morton(const float4* __restrict__ boxes, uint64_t n, const uint32_t* b, uint32_t* keys,
                         uint32_t* vals) {
  uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  float4 lo = boxes[2 * t], hi = boxes[2 * t + 1];
  float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
  uint32_t q[3];
  for (int d = 0; d < 3; ++d) {
    float mn = o2f(b[d]), mx = o2f(b[3 + d]);
    float ext = mx - mn;
    float u = ext > 0.0f ? (c[d] - mn) / ext : 0.0f;
    u = fminf(fmaxf(u * 1024.0f, 0.0f), 1023.0f);
    q[d] = (uint32_t)u;
  }
  keys[t] = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
  vals[t] = (uint32_t)t;
}

// ---- Karras hierarchy --------------------------------------------------------
__device__ __forceinline__ int kdelta(const uint32_t* __restrict__ k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  uint32_t a = k[i], b = k[j];
  if (a == b) return 32 + __clz((uint32_t)(i ^ j));
  return __clz(a ^ b);
}

__global__ void k_karras(const uint32_t* __restrict__ keys, int n, BvhNode* nodes, uint32_t* node_parent,
                         uint32_t* leaf_parent, uint2* range) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = kdelta(keys, n, i, i - d);
  long lmax = 2;
  while (kdelta(keys, n, i, (int)(i + lmax * d)) > dmin) lmax *= 2;
  long l = 0;
  for (long t = lmax / 2; t >= 1; t /= 2)
    if (kdelta(keys, n, i, (int)(i + (l + t) * d)) > dmin) l += t;
  int j = (int)(i + l * d);
  int dnode = kdelta(keys, n, i, j);
  long s = 0, t = l;
  do {
    t = (t + 1) >> 1;
    if (kdelta(keys, n, i, (int)(i + (s + t) * d)) > dnode) s += t;
  } while (t > 1);
  int gamma = (int)(i + s * d + min(d, 0));
  range[i] = make_uint2((uint32_t)min(i, j), (uint32_t)max(i, j));  // the node's leaves
  uint32_t left = (min(i, j) == gamma) ? (LEAF_BIT | (uint32_t)gamma) : (uint32_t)gamma;
  uint32_t right = (max(i, j) == gamma + 1) ? (LEAF_BIT | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
  nodes[i].l_lo.w = __uint_as_float(left);
  nodes[i].l_hi.w = __uint_as_float(right);
  if (left & LEAF_BIT) leaf_parent[gamma] = i;
  else node_parent[gamma] = i;
  if (right & LEAF_BIT) leaf_parent[gamma + 1] = i;
  else node_parent[gamma + 1] = i;
  if (i == 0) node_parent[0] = 0xFFFFFFFFu;
  nodes[i].r_lo.w = nodes[i].r_hi.w = 0.0f;  // no pillboxes (k_pills)
}

__global__ void k_no_pills(BvhNode* nodes, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) nodes[i].r_lo.w = nodes[i].r_hi.w = 0.0f;
}

__global__ void k_gather_leaves(const TriRec* __restrict__ tris, const uint32_t* __restrict__ perm, int n,
                                TriRec* stris) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) stris[k] = tris[perm[k]];
}

__device__ __forceinline__ void store_child_box(BvhNode* node, bool left, float4 lo, float4 hi) {
  float* f = reinterpret_cast<float*>(node);
  int o = left ? 0 : 8;
  __stcg(f + o + 0, lo.x);
  __stcg(f + o + 1, lo.y);
  __stcg(f + o + 2, lo.z);
  __stcg(f + o + 4, hi.x);
  __stcg(f + o + 5, hi.y);
  __stcg(f + o + 6, hi.z);
}

__global__ void k_refit(const float4* __restrict__ boxes, const uint32_t* __restrict__ perm, int n, BvhNode* nodes,
                        const uint32_t* __restrict__ node_parent, const uint32_t* __restrict__ leaf_parent,
                        uint32_t* counters) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  uint32_t tri = perm[k];
  float4 lo = boxes[2 * tri], hi = boxes[2 * tri + 1];
  uint32_t child = LEAF_BIT | (uint32_t)k;
  uint32_t p = leaf_parent[k];
  // At most n - 1 levels; the bound keeps a malformed tree from looping.
  for (int guard = 0; guard < n; ++guard) {
    BvhNode* node = &nodes[p];
    bool left = __float_as_uint(__ldcg(&node->l_lo.w)) == child;
    store_child_box(node, left, lo, hi);
    __threadfence();
    if (atomicAdd(&counters[p], 1u) == 0) return;
    __threadfence();
    float4 a = __ldcg(&node->l_lo), b = __ldcg(&node->l_hi), c = __ldcg(&node->r_lo), d = __ldcg(&node->r_hi);
    lo = make_float4(fminf(a.x, c.x), fminf(a.y, c.y), fminf(a.z, c.z), 0.0f);
    hi = make_float4(fmaxf(b.x, d.x), fmaxf(b.y, d.y), fmaxf(b.z, d.z), 0.0f);
    uint32_t up = node_parent[p];
    if (up == 0xFFFFFFFFu) return;
    child = p;
    p = up;
  }
}

// ---- pillboxes ---------------------------------------------------------------
// Leaves first .. last of the tree under one pillbox, by `lanes` lanes of a
// warp (1 or 32; lane k takes leaves first + k, first + k + lanes, ...).  The
// axis is the sum of the triangles' area vectors, turned to the side of the
// first (a strip's windows alternate); the extents are those of the vertices
// about the stored centre and axis.
template <int LANES>
__device__ __forceinline__ Pill make_pill(const TriRec* __restrict__ stris, uint32_t first, uint32_t last, uint32_t lane) {
  auto sum = [&](float v) {
    if (LANES > 1)
      for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
  };
  auto most = [&](float v) {
    if (LANES > 1)
      for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
  };
  auto area = [](const TriRec& t) {
    const float ux = t.b.x - t.a.x, uy = t.b.y - t.a.y, uz = t.b.z - t.a.z;
    const float vx = t.c.x - t.a.x, vy = t.c.y - t.a.y, vz = t.c.z - t.a.z;
    return P3{uy * vz - uz * vy, uz * vx - ux * vz, ux * vy - uy * vx};
  };
  const P3 ref = area(stris[first]);
  float nx = 0.f, ny = 0.f, nz = 0.f, limit = INFINITY;  // limit: the least reach
  float lox = INFINITY, loy = INFINITY, loz = INFINITY, hix = -INFINITY, hiy = -INFINITY, hiz = -INFINITY;
  for (uint32_t k = first + lane; k <= last; k += LANES) {
    const TriRec t = stris[k];
    const P3 w = area(t);
    const float s = w.x * ref.x + w.y * ref.y + w.z * ref.z < 0.f ? -1.f : 1.f;
    nx += s * w.x;
    ny += s * w.y;
    nz += s * w.z;
    lox = fminf(lox, fminf(t.a.x, fminf(t.b.x, t.c.x)));
    loy = fminf(loy, fminf(t.a.y, fminf(t.b.y, t.c.y)));
    loz = fminf(loz, fminf(t.a.z, fminf(t.b.z, t.c.z)));
    hix = fmaxf(hix, fmaxf(t.a.x, fmaxf(t.b.x, t.c.x)));
    hiy = fmaxf(hiy, fmaxf(t.a.y, fmaxf(t.b.y, t.c.y)));
    hiz = fmaxf(hiz, fmaxf(t.a.z, fmaxf(t.b.z, t.c.z)));
    if (__float_as_int(t.a.w) == TRI_PROPER) limit = fminf(limit, tri_reach(&t.a.x, &t.b.x, &t.c.x));
  }
  nx = sum(nx);
  ny = sum(ny);
  nz = sum(nz);
  limit = -most(-limit);
  lox = -most(-lox);
  loy = -most(-loy);
  loz = -most(-loz);
  hix = most(hix);
  hiy = most(hiy);
  hiz = most(hiz);
  const float nn = nx * nx + ny * ny + nz * nz;
  if (nn > 0.f && nn < INFINITY) {
    const float inv = 1.0f / sqrtf(nn);
    nx *= inv;
    ny *= inv;
    nz *= inv;
  }
  const float one = nx * nx + ny * ny + nz * nz;
  if (!(one > 0.99999f && one < 1.00001f)) nx = 0.f, ny = 0.f, nz = 1.f;  // no area: any axis is right
  float cx = 0.5f * (lox + hix), cy = 0.5f * (loy + hiy), cz = 0.5f * (loz + hiz);
  float omin = INFINITY, omax = -INFINITY;
  auto along = [&](float4 v) { return (v.x - cx) * nx + (v.y - cy) * ny + (v.z - cz) * nz; };
  for (uint32_t k = first + lane; k <= last; k += LANES) {
    const TriRec t = stris[k];
    const float a = along(t.a), b = along(t.b), c = along(t.c);
    omin = fminf(omin, fminf(a, fminf(b, c)));
    omax = fmaxf(omax, fmaxf(a, fmaxf(b, c)));
  }
  omin = -most(-omin);
  omax = most(omax);
  const float mid = 0.5f * (omin + omax);
  cx += mid * nx;
  cy += mid * ny;
  cz += mid * nz;
  float h = 0.f, r2 = 0.f;
  for (uint32_t k = first + lane; k <= last; k += LANES) {
    const TriRec t = stris[k];
    for (const float4& v : {t.a, t.b, t.c}) {
      const float o = along(v), x = v.x - cx, y = v.y - cy, z = v.z - cz, qq = x * x + y * y + z * z;
      h = fmaxf(h, fabsf(o));
      r2 = fmaxf(r2, qq * (1.0f + 0x1p-20f) - o * o);
    }
  }
  h = most(h);
  r2 = most(r2);
  const float scale = fmaxf(fmaxf(fmaxf(fabsf(lox), fabsf(hix)), fmaxf(fabsf(loy), fabsf(hiy))),
                            fmaxf(fabsf(loz), fabsf(hiz)));
  const float slack = kPillSlack * scale;
  auto up16 = [](float v) { return (__float_as_uint(v) + 0xFFFFu) >> 16; };  // v >= 0
  const float hs = h + slack, rs = sqrtf(r2) * 1.00001f + slack;
  const float bx = hix - lox + 2e-4f, by = hiy - loy + 2e-4f, bz = hiz - loz + 2e-4f;  // the padded box
  const float limit2 = fminf(limit * limit, 0x1p126f);
  // NaN, infinite or huge vertices, and boxes of many reaches: never prune.
  const bool fine = hs < 0x1p60f && rs < 0x1p60f && scale < kReachScale &&
                    bx * bx + by * by + bz * bz <= kReachSpan * kReachSpan * limit2;
  // Where the pillbox is not much flatter than the box is along its axis, the
  // box alone prunes about as well: a search then skips it (limit 0).
  const float flat = 0.5f * ((hix - lox) * fabsf(nx) + (hiy - loy) * fabsf(ny) + (hiz - loz) * fabsf(nz));
  Pill p;
  p.a = make_float4(cx, cy, cz, __uint_as_float(fine ? (up16(hs) << 16) | up16(rs) : 0u));
  p.b = make_float4(nx, ny, nz, fine && h < kPillFlat * flat ? limit2 : 0.0f);
  return p;
}

constexpr uint32_t kPillThread = 8;  // children of at most this many leaves take one lane, others a warp
__global__ void k_pills(const TriRec* __restrict__ stris, BvhNode* __restrict__ nodes,
                        const uint2* __restrict__ range, uint32_t children, Pill* __restrict__ pills) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
  uint32_t first = 0, last = 0;
  bool wide = false;
  auto store = [&](const Pill& p) {
    pills[i] = p;
    (i & 1u ? nodes[i >> 1].r_hi : nodes[i >> 1].r_lo).w = p.b.w;
  };
  if (i < children) {
    const BvhNode& nd = nodes[i >> 1];
    const uint32_t gamma = __float_as_uint(nd.l_lo.w) & ~LEAF_BIT;  // the left child's last leaf
    const uint2 rg = range[i >> 1];
    first = i & 1u ? gamma + 1u : rg.x;
    last = i & 1u ? rg.y : gamma;
    const uint32_t m = last - first + 1u;
    if (m <= kPillThread) store(make_pill<1>(stris, first, last, 0u));
    else if (m <= kPillLeaves) wide = true;
    else store(Pill{make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 1.f, 0.f)});
  }
  uint32_t todo = __ballot_sync(0xFFFFFFFFu, wide);
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1u;
    const Pill p = make_pill<32>(stris, __shfl_sync(0xFFFFFFFFu, first, src), __shfl_sync(0xFFFFFFFFu, last, src), lane);
    if (lane == (uint32_t)src) store(p);
  }
}

inline unsigned grid_for(uint64_t n, int threads = kThreads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

int drop_pills(DeviceMesh* m, cudaStream_t s) {
  if (!m->pills.p) return M2S_OK;
  k_no_pills<<<grid_for(m->nodes.n), kThreads, 0, s>>>(m->nodes.p, (uint32_t)m->nodes.n);
  M2S_CUDA(cudaGetLastError());
  M2S_CUDA(cudaStreamSynchronize(s));
  m->pills.release();
  return M2S_OK;
}

int build_device_mesh(const MeshInput& in, DeviceMesh* out, uint32_t* d_status, cudaStream_t s, bool with_tree,
                      bool with_pills) {
  if (in.n_tris > 0x7FFFFFFFull) return M2S_ERR_INVALID_ARGUMENT;
  const uint32_t T = (uint32_t)in.n_tris;
  out->n_tris = T;
  out->root = T == 1 ? LEAF_BIT : 0;
  int st;
  if ((st = out->tris.alloc(T, s))) return st;
  if (T == 0) return M2S_OK;
  DevBuf<float4> boxes;
  DevBuf<uint32_t> keys, perm, bounds;
  if ((st = boxes.alloc(2ull * T, s)) || (st = keys.alloc(T, s)) || (st = perm.alloc(T, s)) ||
      (st = bounds.alloc(6, s)))
    return st;
  k_setup<<<grid_for(T), kThreads, 0, s>>>(in, out->tris.p, boxes.p, d_status);
  M2S_CUDA(cudaGetLastError());
  if (!with_tree) return M2S_OK;
  k_bounds_init<<<1, 32, 0, s>>>(bounds.p);
  k_bounds<<<std::min(grid_for(T), 1184u), kThreads, 0, s>>>(boxes.p, T, bounds.p);
  k_morton<<<grid_for(T), kThreads, 0, s>>>(boxes.p, T, bounds.p, keys.p, perm.p);
  M2S_CUDA(cudaGetLastError());
  if ((st = radix_sort_pairs(keys.p, perm.p, T, 30, s))) return st;
  if ((st = out->stris.alloc(T, s))) return st;
  k_gather_leaves<<<grid_for(T), kThreads, 0, s>>>(out->tris.p, perm.p, (int)T, out->stris.p);
  M2S_CUDA(cudaGetLastError());
  if (T < 2) return M2S_OK;
  DevBuf<uint32_t> node_parent, leaf_parent, counters;
  DevBuf<uint2> range;
  if ((st = out->nodes.alloc(T - 1, s)) || (st = node_parent.alloc(T - 1, s)) || (st = leaf_parent.alloc(T, s)) ||
      (st = counters.alloc(T - 1, s)) || (st = range.alloc(T - 1, s)))
    return st;
  // (pillboxes only make searches faster: a mesh whose tree just fits goes without)
  if (with_pills && out->pills.alloc(2ull * (T - 1), s)) cudaGetLastError();
  M2S_CUDA(cudaMemsetAsync(counters.p, 0, (T - 1) * sizeof(uint32_t), s));
  k_karras<<<grid_for(T - 1), kThreads, 0, s>>>(keys.p, (int)T, out->nodes.p, node_parent.p, leaf_parent.p,
                                          range.p);
  M2S_CUDA(cudaGetLastError());
  k_refit<<<grid_for(T), kThreads, 0, s>>>(boxes.p, perm.p, (int)T, out->nodes.p, node_parent.p, leaf_parent.p,
                                           counters.p);
  if (out->pills.p)
    k_pills<<<grid_for(2ull * (T - 1), 128), 128, 0, s>>>(out->stris.p, out->nodes.p, range.p, 2u * (T - 1), out->pills.p);
  M2S_CUDA(cudaGetLastError());
  return M2S_OK;
}

}  // namespace m2s

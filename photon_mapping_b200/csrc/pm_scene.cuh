// Device scene: triangles, materials, area lights and the BVH that
// replaces the reference's Embree scene (scene.h:275-348).
//
// Layout in HBM (n faces, the reference's per-face unshared vertices):
//   tri    float4[3n]  p0, p1, p2 per face (face order)
//   nrm    float4[3n]  vertex normals n0, n1, n2 per face
//   geo    float4[n]   geometric normal (triangle.h:30) and area (:33)
//   mat    Material[n] per-face BxDF and emission (scene.h:21-51)
//   lights int[m]      faces with emission > 0, in face order
//   mt     float4[3n]  leaf order: {p0, face id}, {p1 - p0}, {p2 - p0}
//   nodes  float4[8(n-1)] one record per inner node i of the binary tree, of its
//                      up to 4 grandchildren (a child that is a leaf counts
//                      itself): lo.x, lo.y, lo.z, hi.x, hi.y, hi.z of the four,
//                      their ids (>= 0: inner node, < 0: leaf ~id, kNoChild:
//                      none), and {entries of the left child (1: a leaf, or 2),
//                      left child, right child, -} of the binary node. A walk
//                      from node 0 takes two levels of the binary tree per step.
#pragma once

#include "pm_math.cuh"

namespace pm {

constexpr int kBvhStack = 64;

struct SceneDev {
  const float4* __restrict__ tri;
  const float4* __restrict__ nrm;
  const float4* __restrict__ geo;
  const Material* __restrict__ mat;
  const int* __restrict__ lights;
  const float4* __restrict__ mt;
  const float4* __restrict__ nodes;
  int n_faces;
  int n_lights;
  int* err;  // device error word (bit 0: traversal stack overflow)
};

struct Hit {
  float t, u, v;
  int prim;  // face id, -1 when nothing was hit
};

__device__ __forceinline__ V3 f4v3(float4 a) { return v3(a.x, a.y, a.z); }

// Moller-Trumbore ray/triangle test (Moller & Trumbore 1997), two-sided.
// The hit is valid when tmin <= t <= tmax, Embree's convention for
// [tnear, tfar]; (u, v) weight p1 and p2 like Embree's barycentrics.
__device__ __forceinline__ bool ray_triangle(V3 o, V3 d, V3 p0, V3 e1, V3 e2,
                                             float& t, float& u, float& v) {
  const V3 pvec = cross(d, e2);
  const float det = dot(e1, pvec);
  if (!(det != 0.f)) return false;
  const float inv = 1.0f / det;
  const V3 tvec = o - p0;
  u = dot(tvec, pvec) * inv;
  if (!(u >= 0.f && u <= 1.f)) return false;
  const V3 qvec = cross(tvec, e1);
  v = dot(d, qvec) * inv;
  if (!(v >= 0.f && u + v <= 1.f)) return false;
  t = dot(e2, qvec) * inv;
  return t == t;
}

constexpr int kNoChild = (int)0x80000000;

// Entries of the stack of a walk for which STACK was chosen. A step pushes up to 3
// where two levels of the binary tree push 2. With 32 and 64 that holds any tree a
// mesh gives (17 full levels need 2^34 faces); a ray that needs more sets error bit 0.
// 16 can be too few, and no ratio of the two walks' needs holds for every tree, so a
// ray that finds the smaller stack full is answered by the binary walk
// (intersect_binary) and 16 accepts whatever that does with 16 entries. (One entry
// less than 3 per 2: full trees of one level more, the first that the binary walk
// refuses, fill 24.) Walks for 32 and 64 leave the binary walk out: with the call in
// it the path tracer took 3.97 ms instead of 3.65 (512 x 512 x 4, 563k faces).
template <int STACK>
__host__ __device__ constexpr bool stack_refers() {
  return STACK <= 16;
}
template <int STACK>
__host__ __device__ constexpr int stack_entries() {
  return STACK + STACK / 2 - (stack_refers<STACK>() ? 1 : 0);
}
constexpr int kStackFull = -2;  // the "next node" of a ray for the binary walk

// One step of a walk: the boxes of node `node` against the ray (o, inv) in
// [tmin, tmax]. Returns the inner child entered first (-1: none) and pushes the
// other inner children hit, the nearest on top; when they do not fit, the walk is
// over with kStackFull (REFERS), or they are lost and error bit 0 is set. `leaves`
// gets a bit per leaf child hit, its id in ids.
//
// Slab test; NaN products (0 * inf) impose no constraint. The exit distance is
// widened by 1 + 2*gamma(3) (Ize 2013) and the boxes themselves are padded at
// build time, so a box is never culled when a triangle inside it is hit. Two
// boxes at a time in packed arithmetic.
struct RayPacked {
  F2 ox, oy, oz, ix, iy, iz;  // minus the origin, and 1 / direction, twice each
  __device__ __forceinline__ void set(V3 o, V3 d) {
    ox = f2(-o.x, -o.x), oy = f2(-o.y, -o.y), oz = f2(-o.z, -o.z);
    const V3 inv = v3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    ix = f2(inv.x, inv.x), iy = f2(inv.y, inv.y), iz = f2(inv.z, inv.z);
  }
};

// Largest / smallest of three (NaN ignored), one instruction.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

template <bool REFERS, int N>
__device__ __forceinline__ int walk_step(const float4* __restrict__ nodes, int node,
                                         const RayPacked& r, float tmin, float tmax,
                                         int (&stack)[N], int& sp, int* err, unsigned& leaves,
                                         int4& ids) {
  const ulonglong2* n = reinterpret_cast<const ulonglong2*>(nodes + 8 * (size_t)node);
  const ulonglong2 lx = __ldg(n), ly = __ldg(n + 1), lz = __ldg(n + 2);
  const ulonglong2 hx = __ldg(n + 3), hy = __ldg(n + 4), hz = __ldg(n + 5);
  ids = __ldg(reinterpret_cast<const int4*>(n + 6));
  uint32_t key[4];  // entry distance of inner children hit, index in the low bits
  leaves = 0;
  const int id[4] = {ids.x, ids.y, ids.z, ids.w};
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const float2 x0 = f2_split(f2_mul(f2_add(p ? lx.y : lx.x, r.ox), r.ix));
    const float2 x1 = f2_split(f2_mul(f2_add(p ? hx.y : hx.x, r.ox), r.ix));
    const float2 y0 = f2_split(f2_mul(f2_add(p ? ly.y : ly.x, r.oy), r.iy));
    const float2 y1 = f2_split(f2_mul(f2_add(p ? hy.y : hy.x, r.oy), r.iy));
    const float2 z0 = f2_split(f2_mul(f2_add(p ? lz.y : lz.x, r.oz), r.iz));
    const float2 z1 = f2_split(f2_mul(f2_add(p ? hz.y : hz.x, r.oz), r.iz));
    const float na = fmaxf(max3(fminf(x0.x, x1.x), fminf(y0.x, y1.x), fminf(z0.x, z1.x)), tmin);
    const float nb = fmaxf(max3(fminf(x0.y, x1.y), fminf(y0.y, y1.y), fminf(z0.y, z1.y)), tmin);
    const float fa = fminf(min3(fmaxf(x0.x, x1.x), fmaxf(y0.x, y1.x), fmaxf(z0.x, z1.x)), tmax);
    const float fb = fminf(min3(fmaxf(x0.y, x1.y), fmaxf(y0.y, y1.y), fmaxf(z0.y, z1.y)), tmax);
    const bool ha = na <= fa * 1.00000072f, hb = nb <= fb * 1.00000072f;
    const int i = 2 * p;
    key[i] = ha && id[i] >= 0 ? (__float_as_uint(na) & ~3u) | (unsigned)i : 0xffffffffu;
    key[i + 1] = hb && id[i + 1] >= 0 ? (__float_as_uint(nb) & ~3u) | (unsigned)(i + 1) : 0xffffffffu;
    if (ha && id[i] < 0) leaves |= 1u << i;
    if (hb && id[i + 1] < 0) leaves |= 2u << i;
  }
  // nearest first (a network of 5 exchanges)
  auto order = [](uint32_t& a, uint32_t& b) {
    const uint32_t l = min(a, b);
    b = max(a, b);
    a = l;
  };
  order(key[0], key[1]);
  order(key[2], key[3]);
  order(key[0], key[2]);
  order(key[1], key[3]);
  order(key[1], key[2]);
  auto child = [&](uint32_t k) {
    const int lo = k & 1u ? ids.y : ids.x, hi = k & 1u ? ids.w : ids.z;
    return k & 2u ? hi : lo;
  };
  // the others, the farthest first
  const int more = (key[1] != 0xffffffffu) + (key[2] != 0xffffffffu) + (key[3] != 0xffffffffu);
  if (sp + more <= N) {
    if (more > 0) stack[sp + more - 1] = child(key[1]);
    if (more > 1) stack[sp + more - 2] = child(key[2]);
    if (more > 2) stack[sp] = child(key[3]);
    sp += more;
  } else {
    if (REFERS) return kStackFull;
    atomicOr(err, 1);  // their subtrees are lost
  }
  if (key[0] != 0xffffffffu) return child(key[0]);
  return sp > 0 ? stack[--sp] : -1;
}

__device__ __forceinline__ void test_leaf(const SceneDev& sc, int leaf, V3 o,
                                          V3 d, float tmin, Hit& h) {
  const float4 a = __ldg(sc.mt + 3 * leaf);
  const float4 b = __ldg(sc.mt + 3 * leaf + 1);
  const float4 c = __ldg(sc.mt + 3 * leaf + 2);
  float t, u, v;
  if (ray_triangle(o, d, f4v3(a), f4v3(b), f4v3(c), t, u, v)) {
    const int prim = __float_as_int(a.w);
    if (t >= tmin && t <= h.t &&
        (t < h.t || h.prim < 0 || prim < h.prim)) {
      h.t = t;
      h.u = u;
      h.v = v;
      h.prim = prim;
    }
  }
}

// intersect_t by the binary tree, from the same records: a binary child's box is that
// of its own children. For the few rays that need more stack than a walk has;
// one that needs more than STACK entries here sets error bit 0 and loses the
// subtree.
template <int STACK>
__device__ __noinline__ Hit intersect_binary(const float4* __restrict__ nodes,
                                             const float4* __restrict__ mt, int* err, V3 o, V3 d,
                                             float tmin, float tmax) {
  SceneDev sc{};
  sc.mt = mt;
  Hit h{tmax, 0.f, 0.f, -1};
  const V3 inv = v3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
  // entry distance into the box of entries [a, b) of node n, if it is met (the
  // arithmetic of walk_step)
  auto enter = [&](const float* n, int a, int b, float& tn) {
    float lo[3], hi[3];
    for (int x = 0; x < 3; ++x) {
      lo[x] = n[4 * x + a];
      hi[x] = n[12 + 4 * x + a];
      for (int e = a + 1; e < b; ++e) {
        lo[x] = fminf(lo[x], n[4 * x + e]);
        hi[x] = fmaxf(hi[x], n[12 + 4 * x + e]);
      }
    }
    const float x0 = (lo[0] - o.x) * inv.x, x1 = (hi[0] - o.x) * inv.x;
    const float y0 = (lo[1] - o.y) * inv.y, y1 = (hi[1] - o.y) * inv.y;
    const float z0 = (lo[2] - o.z) * inv.z, z1 = (hi[2] - o.z) * inv.z;
    tn = fmaxf(fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fminf(z0, z1)), tmin);
    const float tf = fminf(fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1)), h.t);
    return tn <= tf * 1.00000072f;
  };
  int stack[STACK];
  int sp = 0;
  int node = 0;
  while (true) {
    const float* n = reinterpret_cast<const float*>(nodes + 8 * (size_t)node);
    const int nl = __float_as_int(n[28]);
    const int left = __float_as_int(n[29]), right = __float_as_int(n[30]);
    float tl, tr;
    const bool hl = enter(n, 0, nl, tl);
    const bool hr = enter(n, nl, nl + (right < 0 ? 1 : 2), tr);
    if (hl && left < 0) test_leaf(sc, ~left, o, d, tmin, h);
    if (hr && right < 0) test_leaf(sc, ~right, o, d, tmin, h);
    int next = hl && left >= 0 ? left : -1;
    if (hr && right >= 0) {
      int other = next;
      if (next < 0 || tr < tl) next = right;
      else other = right;
      if (other >= 0) {
        if (sp < STACK) stack[sp++] = other;
        else atomicOr(err, 1);
      }
    }
    if (next < 0) {
      if (sp == 0) return h;
      next = stack[--sp];
    }
    node = next;
  }
}

// Closest hit with tmin <= t <= tmax; ties in t go to the smaller face id,
// so the result does not depend on the traversal order. STACK: entries of
// traversal stack (stack_entries).
template <int STACK>
__device__ __forceinline__ bool intersect_t(const SceneDev& sc, V3 o, V3 d,
                                            float tmin, float tmax, Hit& h) {
  h.t = tmax;
  h.prim = -1;
  h.u = h.v = 0.f;
  if (sc.n_faces <= 0) return false;
  if (sc.n_faces == 1) {
    test_leaf(sc, 0, o, d, tmin, h);
    return h.prim >= 0;
  }
  RayPacked r;
  r.set(o, d);
  int stack[stack_entries<STACK>()];
  int sp = 0;
  int node = 0;
  while (node >= 0) {
    unsigned leaves;
    int4 ids;
    node = walk_step<stack_refers<STACK>()>(sc.nodes, node, r, tmin, h.t, stack, sp, sc.err,
                                            leaves, ids);
    while (leaves) {
      const int i = __ffs(leaves) - 1;
      leaves &= leaves - 1;
      const int lo = i & 1 ? ids.y : ids.x, hi = i & 1 ? ids.w : ids.z;
      const int id = i & 2 ? hi : lo;
      if (id != kNoChild) test_leaf(sc, ~id, o, d, tmin, h);
    }
  }
  if constexpr (stack_refers<STACK>()) {
    if (node == kStackFull)
      h = intersect_binary<STACK>(sc.nodes, sc.mt, sc.err, o, d, tmin, tmax);
  }
  return h.prim >= 0;
}

__device__ __forceinline__ bool intersect(const SceneDev& sc, V3 o, V3 d,
                                          float tmin, float tmax, Hit& h) {
  return intersect_t<kBvhStack>(sc, o, d, tmin, tmax, h);
}

// A closest-hit query in progress, for kernels that let the lanes of a warp
// work on rays of different lengths (pm_trace.cu). The result is that of
// intersect_t: the same boxes and triangles are tested with the same arithmetic,
// in an order that does not matter. The stack (kept beside it: an array indexed
// at run time would take the whole struct out of registers) holds the same
// entries. Leaves met wait in a queue of kLeafQueue in shared memory, entry e of
// a thread at queue[e * BLOCK], so that a lane goes on through the tree while
// its warp is not testing triangles.
constexpr int kLeafQueue = 8;  // 6 and 12: the same within 2 %

struct Walk {
  const float4* nodes;
  const float4* mt;
  RayPacked r;
  float tmin;
  Hit h;
  int node;  // inner node to visit next, -1: none, kStackFull: h is not to be had here
  int sp;
  int waiting;  // leaves in the queue

  __device__ __forceinline__ bool can_visit() const {
    return node >= 0 && waiting <= kLeafQueue - 4;
  }
  __device__ __forceinline__ bool over() const { return node < 0 && waiting == 0; }

  __device__ __forceinline__ void start(const SceneDev& sc, V3 ro, V3 rd, float t0, float t1,
                                        int* queue) {
    nodes = sc.nodes;
    mt = sc.mt;
    r.set(ro, rd);
    tmin = t0;
    h.t = t1;
    h.prim = -1;
    h.u = h.v = 0.f;
    sp = 0;
    node = sc.n_faces > 1 ? 0 : -1;
    waiting = sc.n_faces == 1 ? 1 : 0;
    queue[0] = 0;  // the only leaf
  }

  // Visits `node`; can_visit() holds.
  template <int BLOCK, bool REFERS, int N>
  __device__ __forceinline__ void visit(int (&stack)[N], int* queue, int* err) {
    unsigned leaves;
    int4 ids;
    node = walk_step<REFERS>(nodes, node, r, tmin, h.t, stack, sp, err, leaves, ids);
    const int id[4] = {ids.x, ids.y, ids.z, ids.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if ((leaves & (1u << i)) && id[i] != kNoChild) queue[waiting++ * BLOCK] = ~id[i];
  }

  // Tests the last leaf of the queue against the ray (o, d) given to start().
  template <int BLOCK>
  __device__ __forceinline__ void test(V3 o, V3 d, const int* queue) {
    const float4* leaf = mt + 3 * (size_t)queue[--waiting * BLOCK];
    const float4 a = __ldg(leaf), b = __ldg(leaf + 1), c = __ldg(leaf + 2);
    float t, u, v;
    if (ray_triangle(o, d, f4v3(a), f4v3(b), f4v3(c), t, u, v)) {
      const int prim = __float_as_int(a.w);
      if (t >= tmin && t <= h.t && (t < h.t || h.prim < 0 || prim < h.prim)) {
        h.t = t;
        h.u = u;
        h.v = v;
        h.prim = prim;
      }
    }
  }
};

// Surface frame at a hit (scene.h:324-337): position = ray(t), shading
// normal interpolated and not re-normalised (triangle.h:64-71), tangent
// frame from orthonormalBasis.
struct Surf {
  V3 pos, ng, ns, dpdu, dpdv;
};

__device__ __forceinline__ V3 shading_normal(const SceneDev& sc, int f,
                                             float b0, float b1) {
  const V3 n1 = f4v3(__ldg(sc.nrm + 3 * f));
  const V3 n2 = f4v3(__ldg(sc.nrm + 3 * f + 1));
  const V3 n3 = f4v3(__ldg(sc.nrm + 3 * f + 2));
  return n1 * (1.0f - b0 - b1) + n2 * b0 + n3 * b1;
}

__device__ __forceinline__ Surf surface_at(const SceneDev& sc, V3 o, V3 d,
                                           const Hit& h) {
  Surf s;
  s.pos = o + h.t * d;
  s.ng = f4v3(__ldg(sc.geo + h.prim));
  s.ns = shading_normal(sc, h.prim, h.u, h.v);
  orthonormal_basis(s.ns, s.dpdu, s.dpdv);
  return s;
}

// Triangle::samplePoint (triangle.h:84-114): uniform point, pdf = 1/area.
// Draws one getNext2D.
__device__ __forceinline__ void sample_triangle_point(const SceneDev& sc, int f, Rng& rng, V3& pos,
                                                      V3& ns, float& pdf) {
  float u0, u1;
  rng.next2d(u0, u1);
  const float su0 = sqrtf(u0);
  const float b0 = 1.0f - su0, b1 = u1 * su0;
  const V3 p1 = f4v3(__ldg(sc.tri + 3 * f));
  const V3 p2 = f4v3(__ldg(sc.tri + 3 * f + 1));
  const V3 p3 = f4v3(__ldg(sc.tri + 3 * f + 2));
  pos = (1.0f - b0 - b1) * p1 + b0 * p2 + b1 * p3;
  ns = shading_normal(sc, f, b0, b1);
  pdf = 1.0f / __ldg(sc.geo + f).w;
}

// Scene::sampleLight (scene.h:350-355): uniform over the light faces by
// count; getNext1D can return 1.0, clamped to the last light.
__device__ __forceinline__ int sample_light(const SceneDev& sc, Rng& rng,
                                            float& pdf) {
  unsigned idx = (unsigned)((float)sc.n_lights * rng.next1d());
  if (idx == (unsigned)sc.n_lights) idx--;
  pdf = 1.0f / (float)sc.n_lights;
  return __ldg(sc.lights + idx);
}

}  // namespace pm

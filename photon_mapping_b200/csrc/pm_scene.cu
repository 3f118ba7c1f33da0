// Scene upload and BVH build on the device (replaces the Embree BVH of
// scene.h:275-304): per-face constants, Morton codes of the triangle
// centroids, radix sort, then the tree built by parallel locally-ordered
// clustering over the sorted leaves (PLOC, below).
#include "pm_scene.cuh"
#include "pm_scene_build.cuh"
#include "pm_sort.cuh"

#include <cooperative_groups.h>
#include <float.h>

#include <algorithm>
#include <cstring>

namespace pm {

// Per-face constants (triangle.h:25-34) and the leaf records.
__global__ void face_setup_kernel(const float* __restrict__ verts, int n,
                                  float4* __restrict__ tri,
                                  float4* __restrict__ geo) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n) return;
  const float* v = verts + 9 * (size_t)f;
  const V3 p1 = v3(v[0], v[1], v[2]);
  const V3 p2 = v3(v[3], v[4], v[5]);
  const V3 p3 = v3(v[6], v[7], v[8]);
  tri[3 * f] = make_float4(p1.x, p1.y, p1.z, 0.f);
  tri[3 * f + 1] = make_float4(p2.x, p2.y, p2.z, 0.f);
  tri[3 * f + 2] = make_float4(p3.x, p3.y, p3.z, 0.f);
  const V3 c = cross(p2 - p1, p3 - p1);
  const V3 g = normalize(c);
  geo[f] = make_float4(g.x, g.y, g.z, 0.5f * length(c));
}

// Vertex normals, 3 per face.
__global__ void normals_kernel(const float* __restrict__ nrms, int n3, float4* __restrict__ nrm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n3) return;
  const float* v = nrms + 3 * (size_t)i;
  nrm[i] = make_float4(v[0], v[1], v[2], 0.f);
}

void scene_normals_launch(const float* nrms, int n, float4* nrm, cudaStream_t st) {
  if (n > 0) normals_kernel<<<(3 * n + 255) / 256, 256, 0, st>>>(nrms, 3 * n, nrm);
}

__global__ void scene_bbox_kernel(const float4* __restrict__ tri, int n,
                                  uint32_t* __restrict__ bb) {
  float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
  float hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < n;
       f += gridDim.x * blockDim.x) {
    for (int k = 0; k < 3; ++k) {
      const float4 p = tri[3 * f + k];
      lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
      hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
    }
  }
  for (int a = 0; a < 3; ++a) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(kFull, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(kFull, hi[a], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    for (int a = 0; a < 3; ++a) {
      atomicMin(&bb[a], ordered_bits(lo[a]));
      atomicMax(&bb[3 + a], ordered_bits(hi[a]));
    }
  }
}

__global__ void tri_morton_kernel(const float4* __restrict__ tri, int n,
                                  const uint32_t* __restrict__ bb,
                                  uint32_t* __restrict__ keys,
                                  uint32_t* __restrict__ vals) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n) return;
  float lo[3], ext[3];
  for (int a = 0; a < 3; ++a) {
    lo[a] = from_ordered(bb[a]);
    ext[a] = from_ordered(bb[3 + a]) - lo[a];
  }
  const float4 a = tri[3 * f], b = tri[3 * f + 1], c = tri[3 * f + 2];
  const float cx = (a.x + b.x + c.x) * (1.0f / 3.0f);
  const float cy = (a.y + b.y + c.y) * (1.0f / 3.0f);
  const float cz = (a.z + b.z + c.z) * (1.0f / 3.0f);
  keys[f] = (spread10(cell10(cx, lo[0], ext[0])) << 2) |
            (spread10(cell10(cy, lo[1], ext[1])) << 1) |
            spread10(cell10(cz, lo[2], ext[2]));
  vals[f] = (uint32_t)f;
}

// Leaf records in sorted order: {p0, face id}, {p1 - p0}, {p2 - p0}.
__global__ void leaf_setup_kernel(const float4* __restrict__ tri, int n,
                                  const uint32_t* __restrict__ order,
                                  float4* __restrict__ mt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int f = (int)order[i];
  const V3 p0 = f4v3(tri[3 * f]), p1 = f4v3(tri[3 * f + 1]),
           p2 = f4v3(tri[3 * f + 2]);
  const V3 e1 = p1 - p0, e2 = p2 - p0;
  mt[3 * i] = make_float4(p0.x, p0.y, p0.z, __int_as_float(f));
  mt[3 * i + 1] = make_float4(e1.x, e1.y, e1.z, 0.f);
  mt[3 * i + 2] = make_float4(e2.x, e2.y, e2.z, 0.f);
}

// ------------------------------------------------------------ BVH (PLOC)
//
// Parallel locally-ordered clustering (Meister & Bittner, IEEE TVCG 2018):
// the clusters start as the leaves in Morton order; each pass finds every
// cluster's nearest neighbour among the kPlocRadius clusters on either side
// (the distance is the surface area of the two boxes' union), merges every
// mutual pair into a new internal node and compacts the clusters in order.
// Pairs are ordered by (union area, index distance, parity of the smaller
// index, smaller index): a total order on pairs, so the globally first pair
// is mutual and every pass merges at least one pair, and clusters with
// equal boxes pair up as (2k, 2k + 1), a balanced tree, instead of all
// choosing one neighbour (a chain one merge per pass). Internal nodes are
// numbered from the top down in creation order (the last merge, the root,
// is node 0). Leaf boxes are padded by `pad`, so ray/box rounding never
// culls a hit triangle; a parent's box is the union of its children's.

constexpr int kPlocRadius = 16;
constexpr int kPlocBlock = 256;
constexpr int kPlocMaxBlocks = 4096;

__device__ __forceinline__ float union_area(float4 alo, float4 ahi, float4 blo, float4 bhi) {
  const float dx = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x);
  const float dy = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y);
  const float dz = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
  const float a = dx * dy + dy * dz + dz * dx;
  return a <= FLT_MAX ? a : FLT_MAX;  // NaN and infinity order last
}

// Leaf clusters: id ~leaf, box of the leaf triangle padded by 4e-5 of the
// scene's size (largest extent or coordinate).
__global__ void ploc_leaf_kernel(const float4* __restrict__ mt, int n,
                                 const uint32_t* __restrict__ bb, int* __restrict__ cid,
                                 float4* __restrict__ blo, float4* __restrict__ bhi) {
  const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
  if (leaf >= n) return;
  float size = 0.f;
  for (int a = 0; a < 3; ++a) {
    const float lo = from_ordered(bb[a]), hi = from_ordered(bb[3 + a]);
    size = fmaxf(size, fmaxf(hi - lo, fmaxf(fabsf(lo), fabsf(hi))));
  }
  const float pad = 4e-5f * size + 1e-30f;
  const V3 p0 = f4v3(mt[3 * leaf]);
  const V3 p1 = p0 + f4v3(mt[3 * leaf + 1]);
  const V3 p2 = p0 + f4v3(mt[3 * leaf + 2]);
  blo[leaf] = make_float4(fminf(fminf(p0.x, p1.x), p2.x) - pad,
                          fminf(fminf(p0.y, p1.y), p2.y) - pad,
                          fminf(fminf(p0.z, p1.z), p2.z) - pad, 0.f);
  bhi[leaf] = make_float4(fmaxf(fmaxf(p0.x, p1.x), p2.x) + pad,
                          fmaxf(fmaxf(p0.y, p1.y), p2.y) + pad,
                          fmaxf(fmaxf(p0.z, p1.z), p2.z) + pad, 0.f);
  cid[leaf] = ~leaf;
}

// All passes in one cooperative launch. Launched pass by pass (9 launches and a
// read-back each), the 55 passes of 249k triangles took 2.1 ms of kernels and
// most of the 7.7 ms of an upload with the gaps between them; the clusters left
// decide the next pass, so the launch waits for itself at grid barriers instead,
// and once the clusters left fit one block, that block goes on alone: 0.64 ms,
// 4.8 ms the upload (1.8 ms with the other copies beside it, upload_scene).
//
// A pass: block b owns the clusters [b * per, (b + 1) * per).
//   1. nn[i] = the cluster j != i, |i - j| <= kPlocRadius, whose pair with i
//      comes first in the pair order;
//   2. the block counts its merges (mutual pairs i < nn[i], owned by i) and the
//      clusters it keeps (all but the absorbed ones);
//   3. the counts of the blocks before it give each owner's node (top - 1 - its
//      rank among the owners) and each kept cluster's new place.

// Boxes of a tile of clusters and kPlocRadius more on either side.
struct PlocTile {
  float4 lo[kPlocBlock + 2 * kPlocRadius];
  float4 hi[kPlocBlock + 2 * kPlocRadius];
};

__device__ __forceinline__ void ploc_neighbours(PlocTile& t, const float4* blo, const float4* bhi,
                                                int m, int first, int last, int* nn) {
  for (int c0 = first; c0 < last; c0 += kPlocBlock) {
    const int base = c0 - kPlocRadius;
    __syncthreads();
    for (int q = threadIdx.x; q < kPlocBlock + 2 * kPlocRadius; q += kPlocBlock) {
      const int k = base + q;
      if (k >= 0 && k < m) {
        t.lo[q] = blo[k];
        t.hi[q] = bhi[k];
      }
    }
    __syncthreads();
    const int i = c0 + threadIdx.x;
    if (i >= last) continue;
    const float4 lo = t.lo[threadIdx.x + kPlocRadius], hi = t.hi[threadIdx.x + kPlocRadius];
    float best = INFINITY;
    int bj = -1, bkey = 0;
    for (int o = -kPlocRadius; o <= kPlocRadius; ++o) {
      const int j = i + o;
      if (o == 0 || j < 0 || j >= m) continue;
      const int q = threadIdx.x + kPlocRadius + o;
      const float c = union_area(lo, hi, t.lo[q], t.hi[q]);
      // ties: nearer first, then an even smaller index, then the smaller one
      const int mn = min(i, j);
      const int key = (abs(o) << 2) | ((mn & 1) << 1) | (o > 0 ? 1 : 0);
      if (c < best || (c == best && key < bkey)) {
        best = c;
        bj = j;
        bkey = key;
      }
    }
    nn[i] = bj;
  }
}

// {merges owned, clusters kept} of cluster i as two 16-bit counts (a block of
// at most 256 x 255 clusters per scan).
__device__ __forceinline__ uint32_t ploc_flags(const int* nn, int i) {
  const int j = nn[i];
  const bool mutual = nn[j] == i;
  return (mutual && i < j ? 1u : 0u) | (mutual && j < i ? 0u : 0x10000u);
}

// Merges and compacts the clusters [first, last); `merged` owners and `kept`
// clusters lie before them.
__device__ __forceinline__ void ploc_merge(const int* cid, const float4* blo, const float4* bhi,
                                           const int* nn, int first, int last, int merged, int kept,
                                           int top, int* cid2, float4* blo2, float4* bhi2,
                                           float4* nodes, uint32_t* ws) {
  for (int c0 = first; c0 < last; c0 += kPlocBlock) {
    const int i = c0 + threadIdx.x;
    const uint32_t f = i < last ? ploc_flags(nn, i) : 0u;
    uint32_t total;
    const uint32_t before = block_exclusive_scan(f, ws, &total);
    if (f >> 16) {
      const float4 alo = blo[i], ahi = bhi[i];
      const int o = kept + (int)(before >> 16);
      if (!(f & 1u)) {
        cid2[o] = cid[i];
        blo2[o] = alo;
        bhi2[o] = ahi;
      } else {
        const int j = nn[i];
        const float4 clo = blo[j], chi = bhi[j];
        const int idx = top - 1 - (merged + (int)(before & 0xffffu));
        float4* nd = nodes + 4 * (size_t)idx;
        nd[0] = make_float4(alo.x, alo.y, alo.z, __int_as_float(cid[i]));
        nd[1] = make_float4(ahi.x, ahi.y, ahi.z, __int_as_float(cid[j]));
        nd[2] = make_float4(clo.x, clo.y, clo.z, 0.f);
        nd[3] = make_float4(chi.x, chi.y, chi.z, 0.f);
        cid2[o] = idx;
        blo2[o] = make_float4(fminf(alo.x, clo.x), fminf(alo.y, clo.y), fminf(alo.z, clo.z), 0.f);
        bhi2[o] = make_float4(fmaxf(ahi.x, chi.x), fmaxf(ahi.y, chi.y), fmaxf(ahi.z, chi.z), 0.f);
      }
    }
    merged += (int)(total & 0xffffu);
    kept += (int)(total >> 16);
  }
}

// Clusters left that one block takes alone (16 rounds of its threads).
constexpr int kPlocAlone = 16 * kPlocBlock;

__global__ void __launch_bounds__(kPlocBlock)
    ploc_kernel(int* cid_a, float4* blo_a, float4* bhi_a, int* cid_b, float4* blo_b, float4* bhi_b,
                int* nn, int n, float4* nodes, int2* counts, int* left) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  __shared__ PlocTile tile;
  __shared__ uint32_t ws[kPlocBlock / 32];
  __shared__ int2 sum;
  int m = n, top = n - 1;
  // every pass merges at least one pair: at most n - 1 passes
  for (int pass = 0; m > 1 && pass < n; ++pass) {
    const bool alone = m <= kPlocAlone;
    if (alone && blockIdx.x != 0) return;
    const int per = alone ? m : (m + (int)gridDim.x - 1) / (int)gridDim.x;
    const int first = min((int)blockIdx.x * per, m), last = min(first + per, m);
    ploc_neighbours(tile, blo_a, bhi_a, m, first, last, nn);
    if (alone) __syncthreads();
    else grid.sync();
    int2 mine = make_int2(0, 0);
    for (int i = first + threadIdx.x; i < last; i += kPlocBlock) {
      const uint32_t f = ploc_flags(nn, i);
      mine.x += (int)(f & 1u);
      mine.y += (int)(f >> 16);
    }
    if (threadIdx.x == 0) sum = make_int2(0, 0);
    __syncthreads();
    mine.x = __reduce_add_sync(kFull, mine.x);
    mine.y = __reduce_add_sync(kFull, mine.y);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&sum.x, mine.x);
      atomicAdd(&sum.y, mine.y);
    }
    __syncthreads();
    int2 before = make_int2(0, 0), all = sum;
    if (!alone) {
      if (threadIdx.x == 0) counts[blockIdx.x] = sum;
      grid.sync();
      // every block adds up all blocks' counts
      int2 b = make_int2(0, 0), t = make_int2(0, 0);
      for (int q = threadIdx.x; q < (int)gridDim.x; q += kPlocBlock) {
        const int2 c = counts[q];
        t.x += c.x;
        t.y += c.y;
        if (q < (int)blockIdx.x) {
          b.x += c.x;
          b.y += c.y;
        }
      }
      __shared__ int tot[4];
      if (threadIdx.x < 4) tot[threadIdx.x] = 0;
      __syncthreads();
      b.x = __reduce_add_sync(kFull, b.x);
      b.y = __reduce_add_sync(kFull, b.y);
      t.x = __reduce_add_sync(kFull, t.x);
      t.y = __reduce_add_sync(kFull, t.y);
      if ((threadIdx.x & 31) == 0) {
        atomicAdd(&tot[0], b.x);
        atomicAdd(&tot[1], b.y);
        atomicAdd(&tot[2], t.x);
        atomicAdd(&tot[3], t.y);
      }
      __syncthreads();
      before = make_int2(tot[0], tot[1]);
      all = make_int2(tot[2], tot[3]);
    }
    // every block sees the same counts, so all end together
    if (all.x < 1 || all.x > top || all.y != m - all.x) break;  // cannot happen with the tie rule
    ploc_merge(cid_a, blo_a, bhi_a, nn, first, last, before.x, before.y, top, cid_b, blo_b, bhi_b,
               nodes, ws);
    if (alone) __syncthreads();
    else grid.sync();
    m = all.y;
    top -= all.x;
    int* ci = cid_a;
    cid_a = cid_b;
    cid_b = ci;
    float4* f = blo_a;
    blo_a = blo_b;
    blo_b = f;
    f = bhi_a;
    bhi_a = bhi_b;
    bhi_b = f;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    left[0] = m;
    left[1] = top;
  }
}

// Record i of the tree that walks use (pm_scene.cuh) from the binary nodes
// {left lo, left child}, {left hi, right child}, {right lo}, {right hi}: the
// grandchildren of node i, and its children that are leaves.
__global__ void widen_kernel(const float4* __restrict__ binary, int n, float4* __restrict__ wide) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 lo[4], hi[4];
  int id[4];
  int m = 0;
  auto add = [&](const float4& l, const float4& u, int child) {
    // m is known at compile time in none of the calls: write every slot that
    // matches
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j == m) {
        lo[j] = l;
        hi[j] = u;
        id[j] = child;
      }
    ++m;
  };
  const float4* b = binary + 4 * (size_t)i;
  const float4 b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int child = __float_as_int(c ? b1.w : b0.w);
    if (child < 0) {
      add(c ? b2 : b0, c ? b3 : b1, child);
    } else {
      const float4* g = binary + 4 * (size_t)child;
      const float4 g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3];
      add(g0, g1, __float_as_int(g0.w));
      add(g2, g3, __float_as_int(g1.w));
    }
  }
  // absent children: a point far outside (should a ray meet it all the same,
  // the id says that there is nothing)
  const float4 far = make_float4(1e38f, -1e38f, 2e38f, 0.f);
  while (m < 4) add(far, far, kNoChild);
  float4* w = wide + 8 * (size_t)i;
  w[0] = make_float4(lo[0].x, lo[1].x, lo[2].x, lo[3].x);
  w[1] = make_float4(lo[0].y, lo[1].y, lo[2].y, lo[3].y);
  w[2] = make_float4(lo[0].z, lo[1].z, lo[2].z, lo[3].z);
  w[3] = make_float4(hi[0].x, hi[1].x, hi[2].x, hi[3].x);
  w[4] = make_float4(hi[0].y, hi[1].y, hi[2].y, hi[3].y);
  w[5] = make_float4(hi[0].z, hi[1].z, hi[2].z, hi[3].z);
  w[6] = make_float4(__int_as_float(id[0]), __int_as_float(id[1]), __int_as_float(id[2]),
                     __int_as_float(id[3]));
  const int left = __float_as_int(b0.w);
  w[7] = make_float4(__int_as_float(left < 0 ? 1 : 2), b0.w, b1.w, 0.f);
}

static float host_from_ordered(uint32_t u) {
  u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
  float f;
  memcpy(&f, &u, 4);
  return f;
}

size_t scene_build_scratch_bytes(int n) {
  const size_t nn = (size_t)(n > 1 ? n : 2);
  // cluster boxes a/b (4n float4), the binary nodes (4n float4), sort keys /
  // values a/b (4n), histogram, scene box, cluster ids a/b and neighbours (3n),
  // clusters left, and the counts of up to kPlocMaxBlocks blocks
  return 4 * nn * 16 + 4 * nn * 16 + 4 * nn * 4 + sort_hist_words(nn) * 4 + 64 + 3 * nn * 4 + 32 +
         kPlocMaxBlocks * sizeof(int2) + 64;
}

cudaError_t scene_build_launch(const float* verts, int n, float4* tri, float4* geo, float4* mt,
                               float4* wide, void* scratch, SceneBuildResult* result,
                               cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  float4* blo_a = (float4*)scratch;
  float4* bhi_a = blo_a + n;
  float4* blo_b = bhi_a + n;
  float4* bhi_b = blo_b + n;
  float4* nodes = bhi_b + n;
  uint32_t* ka = (uint32_t*)(nodes + 4 * (size_t)n);
  uint32_t* kb = ka + n;
  uint32_t* va = kb + n;
  uint32_t* vb = va + n;
  uint32_t* hist = vb + n;
  uint32_t* bb = hist + sort_hist_words(n);
  int* cid_a = (int*)(bb + 16);
  int* cid_b = cid_a + n;
  int* nn = cid_b + n;
  int* out = (int*)bb + 8;
  int2* counts = (int2*)(((uintptr_t)(nn + n) + 15) & ~(uintptr_t)15);
  const int tb = 256;
  const int gb = (n + tb - 1) / tb;
  *result = SceneBuildResult{bb};
  face_setup_kernel<<<gb, tb, 0, st>>>(verts, n, tri, geo);
  cudaMemsetAsync(bb, 0xff, 3 * sizeof(uint32_t), st);
  cudaMemsetAsync(bb + 3, 0x00, 13 * sizeof(uint32_t), st);
  scene_bbox_kernel<<<min(gb, 1184), tb, 0, st>>>(tri, n, bb);
  tri_morton_kernel<<<gb, tb, 0, st>>>(tri, n, bb, ka, va);
  const bool in_b = radix_sort_pairs<uint32_t>(ka, va, kb, vb, n, 30, hist, st);
  const uint32_t* order = in_b ? vb : va;
  leaf_setup_kernel<<<gb, tb, 0, st>>>(tri, n, order, mt);
  if (n == 1) return cudaGetLastError();
  ploc_leaf_kernel<<<gb, tb, 0, st>>>(mt, n, bb, cid_a, blo_a, bhi_a);
  int dev = 0, sms = 148, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ploc_kernel, kPlocBlock, 0);
  if (e != cudaSuccess) return e;
  int blocks = std::min((n + kPlocBlock - 1) / kPlocBlock, sms * std::max(1, std::min(per_sm, 4)));
  blocks = std::min(blocks, kPlocMaxBlocks);
  if (n <= kPlocAlone) blocks = 1;
  void* args[] = {&cid_a, &blo_a, &bhi_a, &cid_b, &blo_b, &bhi_b, &nn, &n, &nodes, &counts, &out};
  if ((e = cudaLaunchCooperativeKernel((const void*)ploc_kernel, blocks, kPlocBlock, args, 0, st)))
    return e;
  widen_kernel<<<(n - 1 + tb - 1) / tb, tb, 0, st>>>(nodes, n - 1, wide);
  return cudaGetLastError();
}

bool SceneBuildResult::read(const uint32_t host[16], int n, float lo[3], float hi[3]) {
  for (int a = 0; a < 3; ++a) {
    lo[a] = host_from_ordered(host[a]);
    hi[a] = host_from_ordered(host[3 + a]);
  }
  return n == 1 || (host[8] == 1u && host[9] == 0u);
}

// Batched closest-hit queries (Scene::intersect, scene.h:307-348).
// rays: 8 floats each {origin, tmin, direction, tmax}.
__global__ void intersect_kernel(SceneDev sc, const float4* __restrict__ rays,
                                 int64_t n, float4* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = rays[2 * i], b = rays[2 * i + 1];
  Hit h;
  const bool hit = intersect(sc, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), a.w,
                             b.w, h);
  out[i] = hit ? make_float4(h.t, h.u, h.v, __int_as_float(h.prim))
               : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
}

void intersect_launch(const SceneDev& sc, const float4* rays, int64_t n,
                      float4* out, cudaStream_t st) {
  if (n <= 0) return;
  const int tb = 128;
  intersect_kernel<<<(unsigned)((n + tb - 1) / tb), tb, 0, st>>>(sc, rays, n,
                                                                 out);
}

}  // namespace pm

// Radiance estimates of spatially sorted queries (computeRadianceWithPhotonMap,
// integrator.h:133-152): a warp answers 32 neighbouring queries from one walk
// of the photon map's box tree.
//
// The warp-per-query search (pm_photonmap.cu) spends about 3,100 warp
// instructions per query, most of them on the tree walk, the ballots of the
// candidate appends and the selection, each executed by 32 lanes for one query.
// Neighbouring queries need nearly the same photons, so here
//   1. one walk lists the 8-photon groups within a radius of the box of the
//      queries, apart by residue of the group index mod 4;
//   2. per sub-tile of 8 queries the lists are filtered against their box. Row
//      t of the sub-tile is entry t of the four lists: 32 photons, one per lane,
//      and lane l only ever holds photons i with i & 31 == l;
//   3. every row's photons are binned for all 8 queries: byte = bin of the
//      squared distance among 126 equal bins of [0, tau), kept in shared memory.
//      A photon is loaded once per 8 queries, by the one lane that needs it: a
//      first version with 4 lanes per query read each group by broadcast and was
//      bound by the 128 B per cycle that the L1 returns to registers;
//   4. four lanes per query count its bytes against thresholds until few photons
//      are left around the k-th, rank those exactly by (dist2, index) and mark
//      the kept ones (byte 0);
//   5. a second pass over the rows sums the kept photons: lane l sums class l
//      in the walk's order, then the 32 classes are added by a fixed tree. The
//      warp-per-query kernel sums the same way (kept_sum), so a query's result
//      does not depend on the kernel, the tile or the radius that answered it.
// A query that cannot be answered here (a list that stays too long, more than
// 16 photons in the k-th bin, fewer than k photons) goes to a list that the
// warp-per-query kernel answers afterwards.
#include "pm_batch.cuh"
#include "pm_knn_tile.cuh"

#include <float.h>

#include <algorithm>

namespace pm {

namespace {

constexpr int kTileQ = 32;      // queries per work item
constexpr int kSubQ = 8;        // queries of a sub-tile
constexpr int kLanesQ = kWarp / kSubQ;  // lanes per query in step 4
// Queries summed at a time in step 5: 4 skip more rows than 8 (1.195 against 1.50
// ms, which also spills) and load less often than 2 (1.25 ms).
constexpr int kPassQ = 4;
constexpr int kBins = 126;      // bins of [0, tau): bytes 1 .. 126; 127: outside, 0: kept
constexpr int kListCap = 96;    // groups per residue of a walk's list
constexpr int kCrit = 16;       // photons around the k-th that are ranked here
constexpr int kFewEnough = 8;   // ... that end the search for the k-th
// Radii (squared, as factors): the walk's over the sub-tile's, so that a
// sub-tile rarely needs another walk; the next sub-tile's over the largest
// k-th distance of the last one.
constexpr float kWalkSlack = 1.6f;
constexpr float kNextSlack = 1.15f;
// Largest distance (squared, over the search radius squared) from the first
// query of a walk, or of a sub-tile, to its others. Frames and 65k to 900k unordered
// queries: a walk's 9 is the same within 1 %, 100 up to 2.5 % slower; a sub-tile's 1 is
// 2 to 12 % slower, 16 up to 4 %.
constexpr float kWalkReach = 25.f;
constexpr float kSubReach = 4.f;
constexpr int kTries = 24;
// When a warp stops trying. Where photons crowd the tree's sort cells, groups overlap
// so much that a list fills at any radius, or the radius that a query needs meets too
// many: with 24 tries for every item, 150k estimates on 500k clustered photons (k =
// 50) took 10.1 ms, and on photons with a few far outside three times as long as
// by the warp-per-query kernel; 2.8 ms and its time this way.
// Walks of one query that may find too many groups, each at a quarter of the
// radius, before the queries are left; and in a warp whose last item was left so.
constexpr int kFullWalks = 4;
constexpr int kFullWalksWary = 1;
// Queries are left once a radius with too few photons is this part of one with too
// many groups: in between, one or the other would come again. After many tries, or in
// a warp whose last item was left, a wider gap is enough (at once, it costs 3 % of
// estimates that would succeed: 916k of 1M photons in a cube, k = 100, 1.22 against
// 1.19 ms).
constexpr float kNoRoom = 0.8f, kNoRoomLate = 0.25f;
constexpr int kLate = 12;

struct TileWarp {
  uint32_t list[4][kListCap];
  float nx[kSubQ], ny[kSubQ], nz[kSubQ];     // minus the queries' positions
  float sx[kSubQ], sy[kSubQ], sz[kSubQ];     // their shading normals
  uint32_t below[kSubQ];                     // byte + this < 0x80: kept
  uint32_t ql[kSubQ];                        // their lanes
  uint32_t ccnt[kSubQ], kth[kSubQ];
  uint32_t key[kSubQ][kCrit], oid[kSubQ][kCrit];  // photons around the k-th
  uint16_t at[kSubQ][kCrit];                      // and their bytes' places
  // Of the first query left: the largest squared radius known to hold fewer than k
  // photons, the smallest known to meet too many groups, and the walks that did.
  // Every lane writes and reads the same value (registers are short).
  float few, many;
  int full;
  // The warp's last item was left without an answer, as the next will be where groups
  // overlap too much for lists: a query by itself finds out.
  int wary;
};

// Words of one query's bytes ([row / 4][lane], 4 rows per word); 4 more keep the
// queries' words in different banks.
__host__ __device__ constexpr int tile_query_words(int rows) { return rows * 8 + 4; }

__host__ __device__ constexpr size_t tile_bytes(int rows) {
  return sizeof(TileWarp) + 4 * (size_t)(4 * rows + kSubQ * tile_query_words(rows));
}
static_assert(sizeof(TileWarp) % 16 == 0, "16-byte words behind");

__device__ __forceinline__ float redux_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float redux_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

struct Box3 {
  float3 lo, hi;
};

// Box of the positions of the lanes with `in`.
__device__ __forceinline__ Box3 warp_box(float x, float y, float z, bool in) {
  Box3 b;
  b.lo.x = redux_min(in ? x : FLT_MAX);
  b.lo.y = redux_min(in ? y : FLT_MAX);
  b.lo.z = redux_min(in ? z : FLT_MAX);
  b.hi.x = redux_max(in ? x : -FLT_MAX);
  b.hi.y = redux_max(in ? y : -FLT_MAX);
  b.hi.z = redux_max(in ? z : -FLT_MAX);
  return b;
}

// Lower bound of dist2_ref(q, p) over q in b and p in [lo, hi] (box_dist2's
// argument: the same subtractions, and rounding is monotone).
__device__ __forceinline__ float boxes_dist2(const Box3& b, const float4& lo, const float4& hi) {
  const float dx = fmaxf(fmaxf(lo.x - b.hi.x, b.lo.x - hi.x), 0.f);
  const float dy = fmaxf(fmaxf(lo.y - b.hi.y, b.lo.y - hi.y), 0.f);
  const float dz = fmaxf(fmaxf(lo.z - b.hi.z, b.lo.z - hi.z), 0.f);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// Lists the groups within squared distance tau of b, depth first in the
// order of the warp-per-query walk. Lane l holds child l of a node, so group
// g comes from a lane with l & 3 == g & 3: each residue class has its own
// list. Returns the length of the lane's class's list; -1 in every lane when
// a list is full.
__device__ __forceinline__ int tile_walk(const MapDev& m, const TileLevels& L, TileWarp& s,
                                         uint32_t* stack, const Box3& b, float tau, int lane) {
  const unsigned cls = 0x11111111u << (lane & 3);
  int mine = 0;
  if (lane == 0) stack[0] = (uint32_t)(m.nlevels - 1) << 28;
  int sp = 1;
  __syncwarp();
  while (sp > 0) {
    // two nodes per step when both are parents of groups: their loads overlap
    const uint32_t e = stack[sp - 1], e2 = stack[max(sp - 2, 0)];
    const int cl = (int)(e >> 28) - 1;  // level of the children
    const bool two = cl == 0 && sp > 1 && (e2 >> 28) == 1u;
    const int2 oc = L.oc[cl];
    const int c = (int)(e & 0x0fffffffu) * 32 + lane;
    const int c2 = (int)(e2 & 0x0fffffffu) * 32 + lane;
    const bool in = c < oc.y, in2 = two && c2 < oc.y;
    const int jb = oc.x + (in ? c : 0), jb2 = oc.x + (in2 ? c2 : 0);
    const float4 lo = __ldg(m.boxes + 2 * jb), hi = __ldg(m.boxes + 2 * jb + 1);
    const float4 lo2 = __ldg(m.boxes + 2 * jb2), hi2 = __ldg(m.boxes + 2 * jb2 + 1);
    const bool pass = in && boxes_dist2(b, lo, hi) <= tau;
    const bool pass2 = in2 && boxes_dist2(b, lo2, hi2) <= tau;
    const unsigned bal = __ballot_sync(kFull, pass);
    const unsigned bal2 = __ballot_sync(kFull, pass2);
    sp -= two ? 2 : 1;
    if (cl == 0) {
      const unsigned own = bal & cls, own2 = bal2 & cls;
      const int next = mine + __popc(own);
      if (__any_sync(kFull, next + __popc(own2) > kListCap)) return -1;
      if (pass) s.list[lane & 3][mine + __popc(own & lt_mask(lane))] = (uint32_t)c;
      if (pass2) s.list[lane & 3][next + __popc(own2 & lt_mask(lane))] = (uint32_t)c2;
      mine = next + __popc(own2);
    } else {
      if (pass) stack[sp + __popc(bal & lt_mask(lane))] = ((uint32_t)cl << 28) | c;
      sp += __popc(bal);
    }
    __syncwarp();
  }
  return mine;
}

// Copies the listed groups within squared distance tau of b to sub (residue x
// from sub[x * rows] on), each residue filled up with the group `none` without
// photons to the same number of rows, a multiple of 4. Returns it; more than
// `rows` when they do not fit.
__device__ __forceinline__ int tile_filter(const MapDev& m, int none, const TileWarp& s,
                                           uint32_t* sub, int rows, int mine, const Box3& b,
                                           float tau, int lane) {
  // lane l takes entries l / 4, l / 4 + 8, ... of residue l & 3 (whose length it
  // knows), one round of loads ahead
  const int x = lane & 3;
  const unsigned cls = 0x11111111u << x;
  const int most = (int)__reduce_max_sync(kFull, (unsigned)mine);
  int n = 0, e = lane >> 2;
  uint32_t g = e < mine ? s.list[x][e] : 0u;
  float4 lo = __ldg(m.boxes + 2 * g), hi = __ldg(m.boxes + 2 * g + 1);
#pragma unroll 1
  for (int r = 0; r < most; r += 8) {
    const uint32_t gc = g;
    const bool pass = e < mine && boxes_dist2(b, lo, hi) <= tau;
    e += 8;
    g = e < mine ? s.list[x][e] : 0u;
    lo = __ldg(m.boxes + 2 * g);
    hi = __ldg(m.boxes + 2 * g + 1);
    const unsigned own = __ballot_sync(kFull, pass) & cls;
    const int o = n + __popc(own & lt_mask(lane));
    if (pass && o < rows) sub[x * rows + o] = gc;
    n += __popc(own);
  }
  const int used = ((int)__reduce_max_sync(kFull, (unsigned)n) + 3) & ~3;
  if (used <= rows)
    for (int t = n + (lane >> 2); t < used; t += 8) sub[x * rows + t] = (uint32_t)none;
  __syncwarp();
  return used;
}

// The first queries of `from` (a lane each) up to `most` lanes on, cut before
// the first one farther than sqrt(reach2) from the first: the sorted order
// jumps where the space-filling curve does.
__device__ __forceinline__ unsigned near_run(unsigned from, int most, float reach2, float x, float y,
                                             float z, int lane) {
  const int a = __ffs(from) - 1;
  const float d2 = dist2_ref(x, y, z, __shfl_sync(kFull, x, a), __shfl_sync(kFull, y, a),
                             __shfl_sync(kFull, z, a));
  unsigned far = __ballot_sync(kFull, ((from >> lane) & 1u) && !(d2 <= reach2));
  far &= ~(1u << a);
  if (a + most < 32) far |= 1u << (a + most);
  return far ? from & ((1u << (__ffs(far) - 1)) - 1u) : from;
}

// c + 128 x the bytes of v with the high bit set.
__device__ __forceinline__ uint32_t above_add(uint32_t v, uint32_t c) {
  return __dp4a(v & 0x80808080u, 0x01010101u, c);
}

// Bytes of 4 rows (a lane's photons p[0..3]) for the queries 2 qp and 2 qp + 1.
// byte = min(floor(dist2 sc) + 1, 127) in the low mantissa bits of a float in
// [2^23, 2^24); NaN (padding, absent queries) gives 127. p - q instead of
// q - p: the squares are the same.
__device__ __forceinline__ void tile_bins(const F2 px[4], const F2 py[4], const F2 pz[4], F2 nx, F2 ny,
                                          F2 nz, F2 sc, uint32_t& w0, uint32_t& w1) {
  const F2 one = f2(8388609.f, 8388609.f);
  const float top = 8388608.f + (float)(kBins + 1);
  uint32_t a[4], b[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const F2 dx = f2_add(px[i], nx), dy = f2_add(py[i], ny), dz = f2_add(pz[i], nz);
    const F2 d2 = f2_add(f2_add(f2_mul(dx, dx), f2_mul(dy, dy)), f2_mul(dz, dz));
    const float2 t = f2_split(f2_fma_rz(d2, sc, one));
    a[i] = __float_as_uint(fminf(t.x, top));
    b[i] = __float_as_uint(fminf(t.y, top));
  }
  w0 = __byte_perm(__byte_perm(a[0], a[1], 0x0040), __byte_perm(a[2], a[3], 0x0040), 0x5410);
  w1 = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}

// Adds the adjoints of the kept photons: for query q of the sub-tile and each
// photon it keeps whose direction its normal (s.sx ..) sees, (s.nx, s.ny, s.nz)[q].
__device__ __forceinline__ void tile_scatter(const MapDev& m, const TileWarp& s, const uint32_t* sub,
                                             const uint32_t* words, int rows, int used, int ns,
                                             int lane, float4* __restrict__ photon_adj) {
  const int qw = tile_query_words(rows);
  const uint32_t* mysub = sub + (lane >> 3) * rows;
#pragma unroll 1
  for (int t = 0; t < used; t += 4) {
    uint32_t some = 0;
    const uint32_t* w = words + 8 * t + lane;
    for (int q = 0; q < ns; ++q) some |= ~(w[q * qw] + s.below[q]);
    some &= 0x80808080u;
    if (!__any_sync(kFull, some != 0u)) continue;
    const uint4 g = *reinterpret_cast<const uint4*>(mysub + t);
    const uint32_t gs[4] = {g.x, g.y, g.z, g.w};
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      if (!(some & (0x80u << (8 * i)))) continue;
      const uint32_t id = (i < 2 ? (i == 0 ? gs[0] : gs[1]) : (i == 2 ? gs[2] : gs[3])) * kGroup + (lane & 7);
      const float wx = __ldg(m.thr4 + id).w;
      const float2 wi = __ldg(m.wi2 + id);
      const uint32_t to = __float_as_uint(__ldg(m.pos4 + id).w);
      float3 sum = make_float3(0.f, 0.f, 0.f);
      bool add = false;
      for (int q = 0; q < ns; ++q) {
        const uint32_t keep = ~(w[q * qw] + s.below[q]);
        // Lambert::evaluate returns 0 when either cosine is < 0
        if ((keep & (0x80u << (8 * i))) &&
            !(dot_ref(wx, wi.x, wi.y, s.sx[q], s.sy[q], s.sz[q]) < 0.f)) {
          sum.x += s.nx[q];
          sum.y += s.ny[q];
          sum.z += s.nz[q];
          add = true;
        }
      }
      if (add) atomicAdd(photon_adj + to, make_float4(sum.x, sum.y, sum.z, 0.f));
    }
  }
}

__device__ __forceinline__ bool no_room(const TileWarp& s, int tries) {
  return s.few >= (tries > kLate || s.wary ? kNoRoomLate : kNoRoom) * s.many;
}

// Leaves a query to the warp-per-query kernel, with a radius to try.
__device__ __forceinline__ void leave(const TileDefer& defer, uint32_t query, float tau) {
  const uint32_t o = atomicAdd(defer.count, 1u);
  defer.list[o] = query;
  defer.tau[o] = tau;
}

// Queries [q0, q0 + nq) (nq <= 32) in the order of `order`. tau: the squared
// search radius to try first (in/out). A: the adjoint of the estimates, adj_in
// scattered onto the kept photons in photon_adj, instead of the estimates.
template <bool A>
__device__ __forceinline__ void tile_item(const MapDev& m, const TileLevels& L, TileWarp& s, int rows,
                                          int lane, const float4* __restrict__ queries,
                                          const uint32_t* __restrict__ order, int stride4,
                                          int64_t q0, int nq, int k, float n_emitted,
                                          float* __restrict__ rgb, const TileDefer& defer,
                                          float& tau, const float* __restrict__ adj_in = nullptr,
                                          float4* __restrict__ photon_adj = nullptr) {
  uint32_t* const sub = reinterpret_cast<uint32_t*>(&s + 1);
  uint32_t* const words = sub + 4 * rows;  // [query][row / 4][lane]
  uint32_t* const stack = words;           // free during a walk
  const int qw = tile_query_words(rows);
  const int none = L.oc[0].y;  // the group without photons
  const int h = lane & (kLanesQ - 1), qs = lane / kLanesQ;  // kLanesQ lanes per query in step 4
  const uint32_t rec = lane < nq ? __ldg(order + q0 + lane) : 0u;
  float px = 0.f, py = 0.f, pz = 0.f;
  if (lane < nq) {
    const float4 r0 = __ldg(queries + (size_t)stride4 * rec);
    px = r0.x;
    py = r0.y;
    pz = r0.z;
  }
  const bool bad = isnan(px) || isnan(py) || isnan(pz);
  if (!A && lane < nq && bad) rgb[3 * (size_t)rec] = rgb[3 * (size_t)rec + 1] = rgb[3 * (size_t)rec + 2] = 0.f;
  unsigned todo = __ballot_sync(kFull, lane < nq && !bad);
  float good = tau;      // from the last queries answered
  int span = s.wary ? 1 : kTileQ, sq = kSubQ, tries = 0;
  s.few = 0.f;
  s.many = FLT_MAX;
  s.full = 0;
  while (todo) {
    const float tw = tau * kWalkSlack;
    const bool hopeless = no_room(s, tries) ||
                          s.full > (s.wary ? kFullWalksWary : kFullWalks);
    if (__any_sync(kFull, ++tries > kTries || !(tw > 1e-30f && tw < 1e30f) || hopeless)) {
      const float hint = s.few > 0.f ? 2.f * s.few : s.full > 0 ? 0.f : tau;
      if ((todo >> lane) & 1u) leave(defer, defer.positions ? (uint32_t)(q0 + lane) : rec, hint);
      s.wary = 1;
      break;
    }
    unsigned wm = near_run(todo, span, kWalkReach * tau, px, py, pz, lane);
    const int mine =
        tile_walk(m, L, s, stack, warp_box(px, py, pz, (wm >> lane) & 1u), tw, lane);
    if (mine < 0) {
      // too many groups: the queries lie apart, or the radius is too large
      if (__popc(wm) > 1) {
        span = max(1, __popc(wm) >> 1);
      } else {
        const int full = s.full;
        __syncwarp();
        s.full = full + 1;
        s.many = fminf(s.many, tau);
        tau *= 0.25f;
        __syncwarp();
      }
      continue;
    }
    float tf = tau;
    while (wm) {
      const unsigned sm = near_run(wm, sq, kSubReach * tf, px, py, pz, lane);
      const int ns = __popc(sm);
      const bool in = (sm >> lane) & 1u;
      const int used =
          tile_filter(m, none, s, sub, rows, mine, warp_box(px, py, pz, in), tf, lane);
      if (used > rows) {
        if (ns > 1) {
          sq = 1 << (31 - __clz(ns - 1));  // the next smaller power of 2
        } else {
          s.many = fminf(s.many, tf);
          tf *= 0.5f;
        }
        if (++tries > kTries || no_room(s, tries)) break;
        continue;
      }
      // the sub-tile's queries in order; absent ones are NaN
      if (lane < kSubQ) s.nx[lane] = s.ny[lane] = s.nz[lane] = __int_as_float(0x7fc00000);
      __syncwarp();
      if (in) {
        const int o = __popc(sm & lt_mask(lane));
        s.nx[o] = -px;
        s.ny[o] = -py;
        s.nz[o] = -pz;
        s.ql[o] = (uint32_t)lane;
      }
      __syncwarp();
      // ---- step 3: the bytes
      {
        const float sc = __fmul_rn(__fdiv_rn((float)kBins, tf), 1.000001f);
        const F2 sc2 = f2(sc, sc);
        const uint32_t* mysub = sub + (lane >> 3) * rows;
        const float4* mypos = m.pos4 + (lane & 7);
#pragma unroll 1
        for (int t = 0; t < used; t += 4) {
          const uint4 g = *reinterpret_cast<const uint4*>(mysub + t);
          const float4 p0 = __ldg(mypos + (size_t)g.x * kGroup), p1 = __ldg(mypos + (size_t)g.y * kGroup);
          const float4 p2 = __ldg(mypos + (size_t)g.z * kGroup), p3 = __ldg(mypos + (size_t)g.w * kGroup);
          const F2 x[4] = {f2(p0.x, p0.x), f2(p1.x, p1.x), f2(p2.x, p2.x), f2(p3.x, p3.x)};
          const F2 y[4] = {f2(p0.y, p0.y), f2(p1.y, p1.y), f2(p2.y, p2.y), f2(p3.y, p3.y)};
          const F2 z[4] = {f2(p0.z, p0.z), f2(p1.z, p1.z), f2(p2.z, p2.z), f2(p3.z, p3.z)};
          uint32_t* w = words + 8 * t + lane;
          // a loop, not four copies: the kernel's instructions have to stay in
          // the instruction cache
#pragma unroll 1
          for (int q = 0; q < ns; q += 2, w += 2 * qw) {
            uint32_t w0, w1;
            tile_bins(x, y, z, *reinterpret_cast<const F2*>(s.nx + q),
                      *reinterpret_cast<const F2*>(s.ny + q),
                      *reinterpret_cast<const F2*>(s.nz + q), sc2, w0, w1);
            w[0] = w0;
            w[qw] = w1;
          }
        }
      }
      __syncwarp();
      // ---- step 4: four lanes per query; lane h of them has words 8h .. 8h + 7
      // of every 4 rows
      const bool act = qs < ns;
      const uint32_t* myw = words + qs * qw + kSubQ * h;
      const int all = 32 * used;
      // bytes <= lo: clo < k photons; bytes <= hi: chi photons, >= k unless the
      // radius was too small. The counts grow about linearly (photons on
      // surfaces), so the thresholds tried are interpolated for a few more and a
      // few fewer than k photons in turn
      int lo = 0, clo = 0, hi = kBins, chi = 0;
      bool fail = false;
#pragma unroll 1
      for (int step = 0;; ++step) {
        const bool more = step == 0 || (act && chi - clo > kFewEnough && hi - lo > 1);
        if (!__any_sync(kFull, more)) break;
        int b = hi;
        if (step > 0 && more) {
          if (step < 7) {
            const float want = (float)(k - clo) + ((step & 1) ? 3.f : -3.5f);
            b = lo + (int)rintf(__fdividef(want * (float)(hi - lo), (float)(chi - clo)));
            b = min(max(b, lo + 1), hi - 1);
          } else {
            b = (lo + hi) >> 1;
          }
        }
        const uint32_t add = (0x7fu - (uint32_t)b) * 0x01010101u;
        uint32_t c128 = 0;  // 128 x bytes above b
#pragma unroll 1
        for (int t = 0; t < used; t += 4) {
#pragma unroll
          for (int j = 0; j < kSubQ / 4; ++j) {
            const uint4 u = *reinterpret_cast<const uint4*>(myw + 8 * t + 4 * j);
            c128 = above_add(u.x + add, c128);
            c128 = above_add(u.y + add, c128);
            c128 = above_add(u.z + add, c128);
            c128 = above_add(u.w + add, c128);
          }
        }
#pragma unroll
        for (int o = 1; o < kLanesQ; o <<= 1) c128 += __shfl_xor_sync(kFull, c128, o);
        const int c = all - (int)(c128 >> 7);
        if (step == 0) {
          chi = c;
          fail = act && chi < k;
          if (__any_sync(kFull, fail)) break;
        } else if (more) {
          if (c >= k) {
            hi = b;
            chi = c;
          } else {
            lo = b;
            clo = c;
          }
        }
      }
      if (__any_sync(kFull, fail)) {
        // the count grows about as the squared radius on surfaces; a radius without
        // any photon says nothing but that it is far too small (at a fixed 1.2 k
        // times, k = 1 crept up: 1M estimates from 3M photons took 20.9 ms, 1.99 so)
        float need = 0.f;
        if (fail) need = tf * (chi > 0 ? fminf(1.2f * (float)k / (float)chi, 4.f) : 4.f);
        need = fmaxf(redux_max(need), 1.1f * tf);
        if (ns == 1) s.few = fmaxf(s.few, tf);
        if (++tries > kTries || no_room(s, tries)) break;
        tau = need;
        tf = need;
        if (need > tw) break;  // walk again
        continue;
      }
      const int ne = act ? chi - clo : 0;
      if (__any_sync(kFull, ne > kCrit)) {
        // far too large a radius for these queries: bins too coarse
        const int top = (int)__reduce_max_sync(kFull, act ? (unsigned)hi : 0u);
        if (top <= kBins / 2 && tries < kTries) {
          ++tries;
          tf *= 1.05f * (float)top / (float)kBins;
          continue;
        }
      }
      const bool fit = act && ne <= kCrit;
      if (lane < kSubQ) s.ccnt[lane] = 0;
      __syncwarp();
      {
        // photons with byte in (lo, hi]
        const uint32_t alo = (0x7fu - (uint32_t)lo) * 0x01010101u;
        const uint32_t ahi = (0x7fu - (uint32_t)hi) * 0x01010101u;
        const float qx = -s.nx[qs], qy = -s.ny[qs], qz = -s.nz[qs];
#pragma unroll 1
        for (int t = 0; t < used; t += 4) {
          uint32_t hit = 0;  // 4 bits per word: rows t .. t + 3 of kSubQ lanes
#pragma unroll
          for (int j = 0; j < kSubQ / 4; ++j) {
            const uint4 u = *reinterpret_cast<const uint4*>(myw + 8 * t + 4 * j);
            const uint32_t z0 = (u.x + alo) & ~(u.x + ahi) & 0x80808080u;
            const uint32_t z1 = (u.y + alo) & ~(u.y + ahi) & 0x80808080u;
            const uint32_t z2 = (u.z + alo) & ~(u.z + ahi) & 0x80808080u;
            const uint32_t z3 = (u.w + alo) & ~(u.w + ahi) & 0x80808080u;
            // the high bits' weights gather them: 8 bits per two words, x 128
            const uint32_t a = __dp4a(z0, 0x08040201u, __dp4a(z1, 0x80402010u, 0u));
            const uint32_t c = __dp4a(z2, 0x08040201u, __dp4a(z3, 0x80402010u, 0u));
            hit |= ((a >> 7) | (c << 1)) << (16 * j);
          }
          if (!fit) hit = 0;
          while (__any_sync(kFull, hit != 0u)) {
            if (hit != 0u) {
              const int bit = __ffs(hit) - 1;
              hit &= hit - 1;
              const int src = kSubQ * h + (bit >> 2);      // lane of the photon
              const int row = t + (bit & 3);
              const uint32_t i = sub[(src >> 3) * rows + row] * kGroup + (src & 7);
              const float4 p = __ldg(m.pos4 + i);
              const uint32_t o = atomicAdd(&s.ccnt[qs], 1u);
              if (o < kCrit) {
                s.key[qs][o] = __float_as_uint(dist2_ref(qx, qy, qz, p.x, p.y, p.z));
                s.oid[qs][o] = __float_as_uint(p.w);
                s.at[qs][o] = (uint16_t)((8 * t + src) * 4 + (row & 3));
              }
            }
          }
        }
      }
      __syncwarp();
      {
        const int n = fit ? ne : 0, kk = k - clo;
        const int most = (int)__reduce_max_sync(kFull, (unsigned)n);
        for (int e = h; e < most + h; e += kLanesQ) {
          uint32_t ke = 0xffffffffu, oe = 0xffffffffu;
          int rank = 0;
          if (e < n) {
            ke = s.key[qs][e];
            oe = s.oid[qs][e];
          }
          for (int f = 0; f < n; ++f) {
            const uint32_t kf = s.key[qs][f], of = s.oid[qs][f];
            rank += kf < ke || (kf == ke && of < oe);
          }
          if (e < n && rank < kk) {
            reinterpret_cast<unsigned char*>(words + qs * qw)[s.at[qs][e]] = 0;
            if (rank == kk - 1) s.kth[qs] = ke;
          }
        }
      }
      // byte + below < 0x80: kept (bytes 0 .. lo; none when not answered here:
      // then even byte 0, of which there is none, would fail)
      if (h == 0) s.below[qs] = (fit ? 0x7fu - (uint32_t)lo : 0x80u) * 0x01010101u;
      // ---- step 5
      const uint32_t rq = __shfl_sync(kFull, rec, act ? (int)s.ql[qs] : 0);
      float rho = 0.f, cos_o = 0.f;
      if (act) {
        const float4* q4 = queries + (size_t)stride4 * rq;
        const float4 r0 = __ldg(q4), r1 = __ldg(q4 + 1), r2 = __ldg(q4 + 2);
        rho = h == 0 ? r0.w : h == 1 ? r1.w : r2.w;  // lane h writes channel h
        cos_o = dot_ref(r1.x, r1.y, r1.z, r2.x, r2.y, r2.z);
        if (h == 0) {
          s.sx[qs] = r2.x;
          s.sy[qs] = r2.y;
          s.sz[qs] = r2.z;
        }
      } else if (h == 0) {
        s.sx[qs] = s.sy[qs] = s.sz[qs] = 0.f;
      }
      uint32_t kth;
      if constexpr (A) {
        kth = fit ? s.kth[qs] : 0u;
        // d estimate / d throughput_i = f(wo, wi_i) / (n_emitted pi maxd2) for
        // the kept photons (integrator.h:141-150), the warp-per-query kernel's
        // expression. Lane l adds the queries' parts for its photon of each row,
        // then adds them to the photon's adjoint at once: a query at a time, the
        // 50 additions per query to memory bound the pass.
        float v = fit && h < 3 ? adj_in[3 * (size_t)rq + h] : 0.f;
        const bool any = (__ballot_sync(kFull, v != 0.f) >> (lane & ~(kLanesQ - 1))) & 0xfu;
        v = __fdiv_rn(__fmul_rn(v, __fdiv_rn(rho, kPI)),
                      __fmul_rn(__fmul_rn(n_emitted, kPI), __uint_as_float(kth)));
        if (!any || cos_o < 0.f) {
          v = 0.f;
          if (h == 0) s.below[qs] = 0x80808080u;
        }
        // the positions' places
        if (h < 3) (h == 0 ? s.nx : h == 1 ? s.ny : s.nz)[qs] = v;
        __syncwarp();
        tile_scatter(m, s, sub, words, rows, used, ns, lane, photon_adj);
      } else {
      __syncwarp();
#pragma unroll 1
      for (int qb = 0; qb < ns; qb += kPassQ) {
        float acc[kPassQ][3];
#pragma unroll
        for (int q = 0; q < kPassQ; ++q) acc[q][0] = acc[q][1] = acc[q][2] = 0.f;
        F2 nx[kPassQ / 2], ny[kPassQ / 2], nz[kPassQ / 2];
#pragma unroll
        for (int p = 0; p < kPassQ / 2; ++p) {
          nx[p] = reinterpret_cast<const F2*>(s.sx + qb)[p];
          ny[p] = reinterpret_cast<const F2*>(s.sy + qb)[p];
          nz[p] = reinterpret_cast<const F2*>(s.sz + qb)[p];
        }
        const uint32_t* mysub = sub + (lane >> 3) * rows;
        const float4* mythr = m.thr4 + (lane & 7);
        const float2* mywi = m.wi2 + (lane & 7);
        const uint32_t* myword = words + qb * qw + lane;
#pragma unroll 1
        for (int t = 0; t < used; t += 4) {
          uint32_t keep[kPassQ], some = 0;
#pragma unroll
          for (int q = 0; q < kPassQ; ++q) {
            keep[q] = ~(myword[q * qw + 8 * t] + s.below[qb + q]);
            some |= keep[q];
          }
          // rows in which no lane keeps a photon for these queries are left out
          some = __reduce_or_sync(kFull, some & 0x80808080u);
          if (some == 0u) continue;
          const uint4 g = *reinterpret_cast<const uint4*>(mysub + t);
          const uint32_t gs[4] = {g.x, g.y, g.z, g.w};
          float4 th[4];
          float2 wi[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (some & (0x80u << (8 * i))) {
              th[i] = __ldg(mythr + (size_t)gs[i] * kGroup);
              wi[i] = __ldg(mywi + (size_t)gs[i] * kGroup);
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (some & (0x80u << (8 * i))) {
              const F2 wx = f2(th[i].w, th[i].w), wy = f2(wi[i].x, wi[i].x),
                       wz = f2(wi[i].y, wi[i].y);
#pragma unroll
              for (int p = 0; p < kPassQ / 2; ++p) {
                const float2 c = f2_split(
                    f2_add(f2_add(f2_mul(wx, nx[p]), f2_mul(wy, ny[p])), f2_mul(wz, nz[p])));
                // Lambert::evaluate returns 0 when either cosine is < 0
                if ((keep[2 * p] & (0x80u << (8 * i))) && !(c.x < 0.f)) {
                  acc[2 * p][0] = __fadd_rn(acc[2 * p][0], th[i].x);
                  acc[2 * p][1] = __fadd_rn(acc[2 * p][1], th[i].y);
                  acc[2 * p][2] = __fadd_rn(acc[2 * p][2], th[i].z);
                }
                if ((keep[2 * p + 1] & (0x80u << (8 * i))) && !(c.y < 0.f)) {
                  acc[2 * p + 1][0] = __fadd_rn(acc[2 * p + 1][0], th[i].x);
                  acc[2 * p + 1][1] = __fadd_rn(acc[2 * p + 1][1], th[i].y);
                  acc[2 * p + 1][2] = __fadd_rn(acc[2 * p + 1][2], th[i].z);
                }
              }
            }
          }
        }
        // the tree of kept_sum: groups (lanes 8, 16 apart), then photons (1, 2,
        // 4). The sums go through shared memory, where lane (query, channel) adds
        // its 32 parts
        __syncwarp();
        float* mine_part = reinterpret_cast<float*>(words + qb * qw) + lane;
#pragma unroll
        for (int q = 0; q < kPassQ; ++q) {
#pragma unroll
          for (int c = 0; c < 3; ++c) mine_part[(3 * q + c) * 36] = acc[q][c];
        }
      }
      __syncwarp();
      float v;  // channel h of query qs
      {
        const float4* part = reinterpret_cast<const float4*>(
            words + qs / kPassQ * kPassQ * qw + (3 * (qs % kPassQ) + min(h, 2)) * 36);
        float4 a = part[0], b = part[2];
        const float4 a1 = part[4], b1 = part[6];
        a.x = __fadd_rn(__fadd_rn(a.x, b.x), __fadd_rn(a1.x, b1.x));
        a.y = __fadd_rn(__fadd_rn(a.y, b.y), __fadd_rn(a1.y, b1.y));
        a.z = __fadd_rn(__fadd_rn(a.z, b.z), __fadd_rn(a1.z, b1.z));
        a.w = __fadd_rn(__fadd_rn(a.w, b.w), __fadd_rn(a1.w, b1.w));
        v = __fadd_rn(__fadd_rn(a.x, a.y), __fadd_rn(a.z, a.w));
        a = part[1], b = part[3];
        const float4 a2 = part[5], b2 = part[7];
        a.x = __fadd_rn(__fadd_rn(a.x, b.x), __fadd_rn(a2.x, b2.x));
        a.y = __fadd_rn(__fadd_rn(a.y, b.y), __fadd_rn(a2.y, b2.y));
        a.z = __fadd_rn(__fadd_rn(a.z, b.z), __fadd_rn(a2.z, b2.z));
        a.w = __fadd_rn(__fadd_rn(a.w, b.w), __fadd_rn(a2.w, b2.w));
        v = __fadd_rn(v, __fadd_rn(__fadd_rn(a.x, a.y), __fadd_rn(a.z, a.w)));
      }
      kth = fit ? s.kth[qs] : 0u;
      if (fit && h < 3)
        rgb[3 * (size_t)rq + h] = radiance_from_sum(v, rho, cos_o, n_emitted, __uint_as_float(kth));
      }
      if (act && !fit && h == 0)  // the radius up to byte hi holds k photons
        leave(defer, defer.positions ? (uint32_t)(q0 + s.ql[qs]) : rq,
              tf * (float)hi * (1.01f / (float)kBins));
      todo &= ~sm;
      wm &= ~sm;
      const uint32_t far = __reduce_max_sync(kFull, kth);
      if (far != 0u) good = tau = kNextSlack * __uint_as_float(far);
      tf = fminf(tau, tw);
      tries = 0;
      s.few = 0.f;
      s.many = FLT_MAX;
      s.full = s.wary = 0;
      sq = min(2 * sq, kSubQ);
      __syncwarp();
    }
    if (span < kTileQ && !wm) span <<= 1;
  }
  tau = good;
}

// 8 bits per axis separate the queries of a frame as finely as tiles of 32 need.
__global__ void __launch_bounds__(256)
    query_keys_kernel(const float4* __restrict__ boxes, const float4* __restrict__ queries,
                      int64_t nq, int stride4, uint32_t* __restrict__ keys,
                      uint32_t* __restrict__ vals) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const float4 lo = __ldg(boxes), hi = __ldg(boxes + 1);
  const float4 q = __ldg(queries + stride4 * i);
  const uint32_t mc = (spread10(cell10(q.x, lo.x, hi.x - lo.x)) << 2) |
                      (spread10(cell10(q.y, lo.y, hi.y - lo.y)) << 1) |
                      spread10(cell10(q.z, lo.z, hi.z - lo.z));
  keys[i] = mc >> (30 - kQueryKeyBits);
  vals[i] = (uint32_t)i;
}

constexpr int kTileWarps = 4;  // per block

// Measured on 891k primary-hit queries over 3.26M traced photons, k = 100, with
// the sort of the queries and the launch for those left over: 1.195 ms against
// 3.13 ms by the warp-per-query kernel. 5 blocks (20 warps) per SM, which the
// shared memory allows for k = 100, take 96 registers without spills; 4 blocks
// of 126 registers: 1.250 ms, 6 of 80: spills, 1.40 ms.
template <bool A>
__global__ void __launch_bounds__(32 * kTileWarps, 5)
    knn_tile_kernel(MapDev m, const float4* __restrict__ queries,
                    const uint32_t* __restrict__ order, int64_t nq, int stride4, int k,
                    float n_emitted, float* __restrict__ rgb, int rows, int item, TileDefer defer,
                    unsigned long long* __restrict__ counter, const float* __restrict__ adj_in,
                    float4* __restrict__ photon_adj) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TileLevels L;
  const int lane = threadIdx.x & 31;
  TileWarp& s = *reinterpret_cast<TileWarp*>(smem_raw + (threadIdx.x >> 5) * tile_bytes(rows));
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kMaxLevels; ++i) L.oc[i] = make_int2(m.lvl_off[i], m.lvl_cnt[i]);
  }
  __syncthreads();
  float tau = even_tau(m, L.oc[m.nlevels - 1].x, k);
  s.wary = 0;
  while (true) {
    unsigned long long c0 = 0;
    if (lane == 0) c0 = atomicAdd(counter, 1ull);
    c0 = __shfl_sync(kFull, c0, 0);
    const int64_t q0 = (int64_t)c0 * item;
    if (q0 >= nq) break;
    tile_item<A>(m, L, s, rows, lane, queries, order, stride4, q0,
                 (int)min((int64_t)item, nq - q0), k, n_emitted, rgb, defer, tau, adj_in,
                 photon_adj);
    __syncwarp();
  }
}

// The same for every scene of a batch: a work item is up to `item` consecutive
// sorted queries of one scene. A warp switches its copy of the map when the
// scene changes. Scenes whose map is too small leave their items whole, so that
// the warp-per-query kernel goes from neighbour to neighbour there (24 scenes of
// 3,600 photons, 1.4M queries, k = 50: 2.55 ms; 3.41 before there were tiles, 4.69
// with every query left by itself). Measured on
// 8 random scenes (50k to 1M photons emitted, k = 50 and 100): 2.63 ms for the
// estimates of a step, 7.97 ms by the warp-per-query kernel.
__global__ void __launch_bounds__(32 * kTileWarps, 5)
    knn_tile_batch_kernel(BatchTables t, const float4* __restrict__ slots,
                          const uint32_t* __restrict__ order, const int64_t* __restrict__ qoff,
                          const int64_t* __restrict__ item_off, int item, float* __restrict__ rgb,
                          int rows, TileDefer defer, unsigned long long* __restrict__ counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int64_t ioff[kMaxBatchScenes + 1];
  __shared__ MapDev wmap[kTileWarps];
  __shared__ TileLevels wlev[kTileWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  TileWarp& s = *reinterpret_cast<TileWarp*>(smem_raw + warp * tile_bytes(rows));
  batch_load_offsets(ioff, item_off, t.n_scenes);
  __syncthreads();
  const int64_t total = ioff[t.n_scenes];
  int cur = -1, k = 0;
  float tau = 0.f, n_emitted = 0.f;
  s.wary = 0;
  while (true) {
    unsigned long long c0 = 0;
    if (lane == 0) c0 = atomicAdd(counter, 1ull);
    c0 = __shfl_sync(kFull, c0, 0);
    if ((int64_t)c0 >= total) break;
    const int sc = batch_find(ioff, t.n_scenes, (int64_t)c0);
    if (sc != cur) {
      __syncwarp();
      const BatchScene& bs = t.scenes[sc];
      if (lane == 0) wmap[warp] = bs.map;
      if (lane < kMaxLevels) wlev[warp].oc[lane] = make_int2(bs.map.lvl_off[lane], bs.map.lvl_cnt[lane]);
      __syncwarp();
      cur = sc;
      s.wary = 0;
      k = bs.k;
      n_emitted = bs.n_emitted;
      if (wmap[warp].n >= kTileMinPhotons)
        tau = even_tau(wmap[warp], wmap[warp].lvl_off[wmap[warp].nlevels - 1], k);
    }
    const int64_t q0 = qoff[sc] + ((int64_t)c0 - ioff[sc]) * item;
    const int nq = (int)min((int64_t)item, qoff[sc + 1] - q0);
    if (wmap[warp].n < kTileMinPhotons) {
      if (lane == 0) {  // the whole item, to one warp
        const uint32_t o = atomicAdd(defer.count, 1u);
        defer.list[o] = (uint32_t)q0;
        defer.tau[o] = -(float)nq;
      }
      continue;
    }
    tile_item<false>(wmap[warp], wlev[warp], s, rows, lane, slots, order, 4, q0, nq, k,
                     n_emitted, rgb, defer, tau);
    __syncwarp();
  }
}

}  // namespace

// Rows of 32 photons that a sub-tile may take: about 8 photons per kept one
// for small k (the queries' spheres side by side), fewer for large k.
// At least 16: a pass's sums fit the place of its queries' bytes.
int tile_rows(int k) {
  const int r = (12 + k * 9 / 64 + 3) & ~3;
  return r < 16 ? 16 : r;
}
static_assert(tile_query_words(16) >= 3 * 36, "place of the sums");

// Lets a tile kernel use the shared memory of the largest k, whatever k it is
// launched for: the limit belongs to the function, so one set for a single k
// would be another context's or batch's limit too, which may launch for a
// larger k in between.
template <class F>
static cudaError_t allow_tile_smem(F kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(kTileWarps * tile_bytes(tile_rows(kTileMaxK))));
}

void query_keys_launch(const MapDev& m, const void* queries, int64_t nq, int stride4,
                       uint32_t* keys, uint32_t* vals, cudaStream_t st) {
  if (nq <= 0) return;
  query_keys_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(
      m.boxes + 2 * m.lvl_off[m.nlevels - 1], (const float4*)queries, nq, stride4, keys, vals);
}

cudaError_t knn_tile_launch(const MapDev& m, const void* queries, int64_t nq, int k,
                            float n_emitted, float* rgb, const TileDefer& defer,
                            unsigned long long* counter, int num_sms, cudaStream_t st,
                            const uint32_t* order, int stride4, const float* adj_in,
                            float4* photon_adj) {
  const auto kern = photon_adj ? knn_tile_kernel<true> : knn_tile_kernel<false>;
  const int rows = tile_rows(k);
  const size_t smem = kTileWarps * tile_bytes(rows);
  cudaError_t e = allow_tile_smem(kern);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kTileWarps, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  int64_t blocks = (int64_t)num_sms * per_sm;
  // a walk serves up to 32 queries; with few queries items are shorter, down to
  // a sub-tile, so that every resident warp gets some (65,536 unordered queries
  // of 1M photons at k = 50: 300 us with items of 32, 263 us with this rule; 1 to 8
  // items per warp are within 5 %)
  int item = kTileQ;
  while (item > kSubQ && nq < 4 * item * blocks * kTileWarps) item >>= 1;
  const int64_t items = (nq + item - 1) / item;
  const int64_t need = (items + kTileWarps - 1) / kTileWarps;
  if (blocks > need) blocks = need;
  if ((e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st)) != cudaSuccess ||
      (e = cudaMemsetAsync(defer.count, 0, sizeof(uint32_t), st)) != cudaSuccess)
    return e;
  kern<<<(unsigned)blocks, 32 * kTileWarps, smem, st>>>(
      m, (const float4*)queries, order, nq, stride4, k, n_emitted, rgb, rows, item, defer, counter,
      adj_in, photon_adj);
  return cudaGetLastError();
}

int batch_tile_item(int64_t nq, int num_sms) {
  int item = kTileQ;
  while (item > kSubQ && nq < 4 * (int64_t)item * num_sms * 5 * kTileWarps) item >>= 1;
  return item;
}

cudaError_t batch_tile_prepare(int max_k, int* blocks_per_sm) {
  const size_t smem = kTileWarps * tile_bytes(tile_rows(max_k));
  cudaError_t e = allow_tile_smem(knn_tile_batch_kernel);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, knn_tile_batch_kernel,
                                                    32 * kTileWarps, smem);
  *blocks_per_sm = per_sm < 1 ? 1 : per_sm;
  return e;
}

cudaError_t batch_tile_launch(const BatchTables& t, const float4* slots, const uint32_t* order,
                              const int64_t* qoff, const int64_t* item_off, int64_t max_items,
                              int item, int max_k, float* res, uint32_t* left, float* left_tau, uint32_t* left_n,
                              int blocks_per_sm, unsigned long long* counter, int num_sms,
                              cudaStream_t st) {
  const int rows = tile_rows(max_k);
  const int64_t need = (max_items + kTileWarps - 1) / kTileWarps;
  const int64_t blocks =
      std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)num_sms * blocks_per_sm));
  cudaError_t e;
  if ((e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st)) != cudaSuccess ||
      (e = cudaMemsetAsync(left_n, 0, sizeof(uint32_t), st)) != cudaSuccess)
    return e;
  knn_tile_batch_kernel<<<(unsigned)blocks, 32 * kTileWarps, kTileWarps * tile_bytes(rows), st>>>(
      t, slots, order, qoff, item_off, item, res, rows, TileDefer{left, left_tau, left_n, true}, counter);
  return cudaGetLastError();
}

}  // namespace pm

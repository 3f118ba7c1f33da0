// Radiance estimates of sorted queries, 32 neighbouring queries per warp
// (pm_knn_tile.cu), and the arithmetic it shares with the warp-per-query
// kernel (pm_photonmap.cu).
#pragma once

#include "pm_photonmap.cuh"

namespace pm {

struct TileLevels {
  int2 oc[kMaxLevels];  // {offset of the level's boxes, boxes in the level}
};

// Queries left to the warp-per-query kernel: records (or, with `positions`,
// places in the sorted order), and how many.
struct TileDefer {
  uint32_t* list;
  float* tau;  // a squared radius to try for each of them (0: none known), or minus
               // the number of consecutive places that the entry stands for
  uint32_t* count;
  bool positions;
};

// The radiance estimate of one channel from the kept photons' summed
// throughput: (rho / pi) sum / (n_emitted pi maxd2), integrator.h:141-150 with
// the Lambert BRDF (zero when the cosine of wo is negative); maxd2 is the k-th
// squared distance. One rounding instead of the five of the same expression in
// float, which makes room for the error of the classes' sums.
__device__ __forceinline__ float radiance_from_sum(float sum, float rho, float cos_o,
                                                   float n_emitted, float maxd2) {
  constexpr double pi = 3.14159265359;  // core.h:7
  const double l = cos_o < 0.f ? 0.0 : (double)rho * (double)sum;
  return (float)(l / ((double)n_emitted * (pi * pi) * (double)maxd2));
}

// Sort keys of nq radiance records (stride4 float4 each): the Morton code of
// the position in the map's box, kQueryKeyBits bits; vals[i] = i.
constexpr int kQueryKeyBits = 24;
void query_keys_launch(const MapDev& m, const void* queries, int64_t nq, int stride4,
                       uint32_t* keys, uint32_t* vals, cudaStream_t st);

// No crossing: tiles are faster from 1,000 photons on (1M queries, k = 50: 0.59 against
// 1.57 ms; 100k: 0.15 against 0.19). The size from which the tests cover them.
constexpr int kTileMinPhotons = 4096;
constexpr int kTileMaxK = 448;
// With photon_adj, the adjoint instead (KnnOut::adj_in, photon_adj; rgb unused).
cudaError_t knn_tile_launch(const MapDev& m, const void* queries, int64_t nq, int k,
                            float n_emitted, float* rgb, const TileDefer& defer,
                            unsigned long long* counter, int num_sms, cudaStream_t st,
                            const uint32_t* order, int stride4, const float* adj_in = nullptr,
                            float4* photon_adj = nullptr);

}  // namespace pm

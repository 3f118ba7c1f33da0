// Host-side launchers of the scene build and of the batched intersection.
#pragma once

#include "pm_scene.cuh"

namespace pm {

// Scratch bytes scene_build_launch needs for n faces.
size_t scene_build_scratch_bytes(int n);

// What a build leaves in its scratch: 16 words to be read back once the stream
// has reached them.
struct SceneBuildResult {
  const uint32_t* words;
  // The vertices' bounds; false when the tree was not completed.
  static bool read(const uint32_t host[16], int n, float lo[3], float hi[3]);
};

// verts: device, 9 floats per face. Fills tri, geo (face order), mt (leaf
// order) and nodes (n - 1 records of 8 float4). Does not synchronise.
cudaError_t scene_build_launch(const float* verts, int n, float4* tri, float4* geo, float4* mt,
                               float4* nodes, void* scratch, SceneBuildResult* result,
                               cudaStream_t st);

// nrms: device, 9 floats per face; nrm: 3 float4 per face.
void scene_normals_launch(const float* nrms, int n, float4* nrm, cudaStream_t st);

// rays: 2 float4 per ray {origin, tmin}, {direction, tmax}; out: one float4
// per ray {t, u, v, face id bits (-1: miss)}.
void intersect_launch(const SceneDev& sc, const float4* rays, int64_t n,
                      float4* out, cudaStream_t st);

}  // namespace pm

// weftk_scene.cuh — a file's decode between its layout and the decoder walk (weftk_entropy.cu), shared with
// the host entry point (weftk_api.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "../../include/weftk_entropy.h"

namespace weftk {

struct ScenePlan {
    bool ok;      // false: a form the general decoder handles (or refuses)
    bool layered;  // many layers to evaluate (WEFTK_WALK_LAYERED)
    int scaled, n_items, cap_prims, cap_cp48;
    int64_t raw_len;
    double sx, sy;
    std::vector<WeftRansChunk> chunks;
};

struct SceneBuffers {  // device memory
    const uint8_t* blob;
    const WeftRansChunk* chunks;
    uint8_t* raw;
    WeftTileDecodeDesc* descs;
    WeftPrim* prims;
    float *cp48, *grids;
    int2* items;
    int* ctl;  // status, number of items
};

int scene_plan(const WeftSceneFile& f, ScenePlan& plan);
int scene_launch(const WeftSceneFile& f, const ScenePlan& plan, const SceneBuffers& b, cudaStream_t s);

}  // namespace weftk

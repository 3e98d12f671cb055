// Read-only view of a scene's device state for entry points outside renderer.cu.
#pragma once
#include <cuda_runtime.h>

#include "../../include/raymond.h"
#include "device/traverse.cuh"
#include "device/wavefront.cuh"

namespace rmdhost {

// Pinned counters (two) and events of rmd_render_noalloc's loop, which may not
// allocate them.  A context has its own: they come with it, nothing replaces
// them under a call, and a context made after a device reset has new ones.
struct LoopHost {
    rmd::Counters *counters = nullptr;
    cudaEvent_t events[2] = {};
    cudaError_t create() {
        cudaError_t e = cudaMallocHost((void **)&counters, 2 * sizeof(rmd::Counters));
        for (cudaEvent_t &ev : events)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        return e;
    }
    ~LoopHost() {
        for (cudaEvent_t ev : events)
            if (ev) cudaEventDestroy(ev);
        if (counters) cudaFreeHost(counters);
    }
};

struct SceneView {
    rmd::Context ctx;              // device view of geometry, lights, materials, camera
    const rmd::WideNode *nodes;     // nullptr for a scene without triangles
    const float4 *tris;
    cudaKernel_t shade;            // shading megakernel of the scene's material module
    int shadeBlocks;
    cudaStream_t stream;
    LoopHost *loop;                // of the scene's context
    int device;
    int smCount;
};

// false for a null scene
bool sceneView(const rmd_scene *scene, SceneView &out);
// records `msg` as the calling thread's rmd_last_error and returns `status`
rmd_status setLastError(rmd_status status, const char *msg);
// looks up the device address of rmd_render_noalloc's scratch array on `device` (current)
rmd_status noallocSetup(int device);

}  // namespace rmdhost

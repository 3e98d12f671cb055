// The host-driven loop of wavefront iterations.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <tuple>

#include "device/wavefront.cuh"

namespace rmdhost {

// Waits for a stream when a call returns early: an object's end does not wait,
// so a call that fails leaves no work behind.  done(): the call has waited.
struct WaitOnReturn {
    cudaStream_t stream;
    bool waits = true;
    explicit WaitOnReturn(cudaStream_t s) : stream(s) {}
    ~WaitOnReturn() {
        if (waits) cudaStreamSynchronize(stream);
    }
    void done() { waits = false; }
};

// Enqueues iterations until `check` ends the loop.  iterate(cur, paths)
// enqueues one iteration of parity cur with at most `paths` active paths (what
// its grids need to cover); check(counters, iterations) returns whether the
// render is over (done, or failed).
//
// The counters are read after every sixteenth iteration until every path has
// been handed out and could have ended, and then after every second, each read
// looked at once the iterations up to the next are enqueued: the device never
// waits for the host, for at most four empty iterations at the end, and a
// device error ends a render of any length within 32 iterations.  (Reading them
// after every fourth iteration and waiting left a gap of 10-20 us each time; a
// read breaks the overlap of two launches, 3-7 us: one more in the 10 iterations
// of a 640 x 360 render cost 0.6 % of it.)  `slots`: two Counters in pinned
// memory; `events`: two events.  On return the last iterations may still run.
template <class Iterate, class Check>
cudaError_t driveWavefront(const rmd::Counters *cnt, uint64_t numPaths, uint32_t capacity, rmd::Counters *slots,
                           cudaEvent_t *events, cudaStream_t st, Iterate iterate, Check check) {
    uint64_t it = 0, paths = std::min<uint64_t>(numPaths, capacity);
    const uint64_t handedOut = ((numPaths + capacity - 1) / capacity + 3) & ~uint64_t(1);
    uint64_t next = std::min<uint64_t>(handedOut, 16);
    for (uint32_t k = 0;; k++, next = next < handedOut ? std::min(handedOut, next + 16) : next + 2) {
        cudaError_t e;
        for (; it < next; it++)
            if ((e = iterate((uint32_t)(it & 1u), paths)) != cudaSuccess) return e;
        if ((e = cudaMemcpyAsync(&slots[k & 1u], cnt, sizeof(rmd::Counters), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
            (e = cudaEventRecord(events[k & 1u], st)) != cudaSuccess)
            return e;
        if (k == 0) continue;
        if ((e = cudaEventSynchronize(events[(k - 1u) & 1u])) != cudaSuccess) return e;
        const rmd::Counters &h = slots[(k - 1u) & 1u];
        if (check(h, it)) return cudaSuccess;
        if (h.handOut[0] >= h.endPath) paths = std::min<uint64_t>(paths, std::max(h.nQ[0], 1u));
    }
}

// Launches a kernel that begins with waitForPreviousKernel so that its set-up
// overlaps the end of the kernel before it on the stream.
inline cudaError_t launchOverlapped(const void *kernel, int blocks, int threads, void **args, cudaStream_t st) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelExC(&cfg, kernel, args);
    if (e != cudaSuccess) cudaGetLastError();  // the caller's to report, not the next launch check's
    return e;
}
template <class... Params, class... Args>
cudaError_t launchOverlapped(void (*kernel)(Params...), int blocks, int threads, cudaStream_t st, Args... values) {
    std::tuple<Params...> params(values...);
    return std::apply(
        [&](Params &...p) {
            void *args[] = {(void *)&p...};
            return launchOverlapped((const void *)kernel, blocks, threads, args, st);
        },
        params);
}

// blocks of `threads` threads that give `paths` paths a thread each, at most `most`
inline int gridFor(uint64_t paths, int threads, int most) {
    return (int)std::max<uint64_t>(1, std::min<uint64_t>((paths + threads - 1) / threads, (uint64_t)most));
}

// Trace grid: the resident one, or as many blocks as give every closest-hit
// and shadow ray of `paths` paths its 8 lanes.
inline int traceGridFor(uint64_t paths, int most) { return gridFor(2 * paths + 8, 16, most); }

}  // namespace rmdhost

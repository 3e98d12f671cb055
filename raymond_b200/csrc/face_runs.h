// The faces of a scene's shapes in runs that the cores check in parallel.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace rmdhost {

constexpr uint32_t kFaceRun = 1u << 16;  // faces of a run at most
struct FaceRun {
    int shape;
    uint32_t begin, end;
};
// the runs of a shape's faces; a shape without faces has an empty one (its vertices go with the first)
inline void appendFaceRuns(std::vector<FaceRun> &runs, int shape, uint32_t faces) {
    for (uint64_t f = 0; f == 0 || f < faces; f += kFaceRun)  // 64 bits: the last step may pass 2^32
        runs.push_back({shape, (uint32_t)f, (uint32_t)std::min<uint64_t>(faces, f + kFaceRun)});
}

}  // namespace rmdhost

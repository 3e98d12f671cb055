// Byte offsets of the render loop's counters, for tests that play the device's part.
#include <cstddef>

#include "device/wavefront.cuh"

extern "C" size_t fake_counters_layout(int field) {
    const size_t at[] = {sizeof(rmd::Counters), offsetof(rmd::Counters, errors), offsetof(rmd::Counters, numPaths),
                         offsetof(rmd::Counters, pathsDone), offsetof(rmd::Counters, numSamples)};
    return at[field];
}

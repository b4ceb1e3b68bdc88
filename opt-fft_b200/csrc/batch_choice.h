// batch_choice.h -- which batches may share the result of a race between the launch
// strategies (host only; batch.cu keeps the results, hostcheck.cpp tests the key).
#pragma once

#include <stdint.h>

#include <array>
#include <vector>

#include "../../include/fft3d_b200.h"

namespace fft3d {

using BatchChoiceKey = std::vector<std::array<long long, 7>>;

// Everything that the race's times depend on: the same segments in the same order,
// their counts exactly (whether widths are timed at all depends on their bytes, and
// which strategy wins on how far each fills the GPU), and whether their buffers lie
// on 16 bytes (complex float off that boundary is copied by elements).
inline BatchChoiceKey batch_choice_key(int device, int cls, bool use_graph, const fft3d_b200_segment *segs,
                                       size_t nseg)
{
    BatchChoiceKey key;
    key.push_back({device, cls, use_graph ? 1 : 0, 0, 0, 0, 0});
    for (size_t i = 0; i < nseg; ++i) {
        const fft3d_b200_segment &s = segs[i];
        const long long off = ((uintptr_t)s.in % 16 ? 1 : 0) + ((uintptr_t)s.out % 16 ? 2 : 0);
        key.push_back({s.n0, s.n1, s.n2, s.precision, s.direction, s.batch, off});
    }
    return key;
}

// A timing that failed.
constexpr float RACE_FAILED_MS = 1e30f;

// Whether a race's times may be kept for other batches: both were measured.
inline bool race_measured(float t_seg, float t_persist)
{
    return t_seg > 0.f && t_seg < RACE_FAILED_MS && t_persist > 0.f && t_persist < RACE_FAILED_MS;
}

}  // namespace fft3d

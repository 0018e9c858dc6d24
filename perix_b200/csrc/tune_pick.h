// The autotuner's decision where schedules are timed twice.
#pragma once

#include <cstddef>
#include <vector>

namespace pxb {

// The schedule whose loop is fastest among those whose single steps (step_ms, a large value: not to be had) are within a
// tenth of the fastest, `flushed`.  loop(v, &t) times schedule v in a loop: 1 timed, 0 not to be had, -1 the loop could not
// be run to its end.  Then the choice is `flushed` whatever the others took: half of the evidence decides nothing.
// The first `exact` schedules are the more accurate ones: the fastest of them is chosen where its loop is within a
// thirtieth of the fastest of all.
template <typename Loop>
int pick_by_loop(const std::vector<float> &step_ms, int flushed, int exact, Loop loop) {
    int best = flushed, first = -1;
    float best_t = 1e30f, first_t = 1e30f;
    for (size_t v = 0; v < step_ms.size(); ++v) {
        if (step_ms[v] > 1.1f * step_ms[(size_t)flushed]) continue;
        float t = 0.f;
        const int r = loop((int)v, &t);
        if (r < 0) return flushed;
        if (r > 0 && t < best_t) {
            best_t = t;
            best = (int)v;
        }
        if (r > 0 && (int)v < exact && t < first_t) {
            first_t = t;
            first = (int)v;
        }
    }
    return first >= 0 && first_t * 30.f <= best_t * 31.f ? first : best;
}

}  // namespace pxb

// Which buffers the jobs of a batch share (plain C++, used by the batch runner and its CPU test).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace mach_b200 {

struct JobRange {
    uintptr_t begin, end;
    uint32_t job;
};

inline void add_range(std::vector<JobRange>& to, const void* p, uint64_t bytes, uint32_t job) {
    if (p && bytes) to.push_back({reinterpret_cast<uintptr_t>(p), reinterpret_cast<uintptr_t>(p) + bytes, job});
}

// Whether a job writes what another job writes or reads (one written range per job; sorts `written`).
inline bool jobs_share_outputs(std::vector<JobRange>& written, const std::vector<JobRange>& read) {
    std::sort(written.begin(), written.end(), [](const JobRange& a, const JobRange& b) { return a.begin < b.begin; });
    for (size_t i = 1; i < written.size(); ++i) {
        if (written[i].begin < written[i - 1].end) return true;
    }
    // (the written ranges are disjoint from here on)
    for (const JobRange& r : read) {
        auto w = std::lower_bound(written.begin(), written.end(), r.end,
                                  [](const JobRange& a, uintptr_t end) { return a.begin < end; });
        while (w != written.begin() && (--w)->end > r.begin) {
            if (w->job != r.job) return true;
        }
    }
    return false;
}

}  // namespace mach_b200

// tune.h -- the autotuner's cache of launch choices (tile widths), keyed on
// the problem (points per axis, quadrature count, batch) and the device.
// Choices live in the process and, when a cache file is set
// (dage_set_tune_cache or the DAGE_TUNE_CACHE environment variable), are
// read from and appended to that file, so later processes skip the timing.
#pragma once

#include <string>
#include <vector>

namespace dage {

// Revision of the tuned kernels, part of every key: raised when a change to
// them can move which choice is fastest, so that a persistent cache's entries
// for earlier kernels are timed anew instead of deciding the launch.  (2: FP64
// stages with K ranges per 32 columns and two blocks per SM, bulk-copied
// split-precision stages, paired t-points of the near field; keys without a
// revision are older.)
constexpr int kTuneRevision = 2;

// Key prefix naming the current device (name and SM count) and the kernels'
// revision: a file shared by different GPUs keeps their choices apart.
std::string tune_device_key();
bool tune_lookup(const std::string &key, std::vector<int> &val);
void tune_store(const std::string &key, const std::vector<int> &val);

}  // namespace dage

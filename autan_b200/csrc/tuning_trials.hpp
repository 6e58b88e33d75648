// The autotuner's trials (included by euler_device.cu; host code only).
//
// Every trial steps the handle, and a step of a partitioned mesh exchanges with the other ranks: all
// ranks have to make the same trials. What a trial depends on besides the scheme and the precision (the
// cells of a rank, whether its blocks of cells fit) is therefore agreed between the ranks first, and a
// trial is made where every rank can make it.
#pragma once

#include <vector>

namespace autan_b200 {

constexpr int kSplitTrials[2] = {32, 64};      // cells a block of the split gradients
constexpr int kFaceTrials[3] = {32, 64, 128};  // cells a block of the face blocks

struct TrialScope {
  bool split[2] = {false, false};
  bool small = false;  // the forms that only small meshes win with
  bool faces[3] = {false, false, false};
};

// `face_cells`: the most cells whose face blocks can win (beyond, their copy of the face records is not
// made to be tried). `any` (bool -> bool): whether any rank has the flag set; every rank calls it together. `split_fits`,
// `face_fits` (cells a block -> bool): whether this rank's blocks of that many cells fit.
template <class Any, class SplitFits, class FaceFits>
TrialScope trial_scope(bool second, long long cells, long long face_cells, Any&& any, SplitFits&& split_fits,
                       FaceFits&& face_fits) {
  auto all = [&](bool mine) { return !any(!mine); };
  TrialScope s;
  // the split form where every mesh is small enough for it to win
  if (second && all(cells <= 148 * 2048))
    for (int i = 0; i < 2; ++i) s.split[i] = all(split_fits(kSplitTrials[i]));
  s.small = all(cells <= 148 * 512);
  const bool blocks = all(cells <= face_cells);
  for (int i = 0; i < 3; ++i)
    if (s.small || (blocks && kFaceTrials[i] == 128)) s.faces[i] = all(face_fits(kFaceTrials[i]));
  return s;
}

struct GradTrial {
  int mode, chunk, block, minb;
};
// (the pipelined, ring and widening forms were never the fastest on any measured case: they stay open
// to set_tuning and are not tried)
inline std::vector<GradTrial> grad_trials(const TrialScope& s, bool fp32_limited) {
  std::vector<GradTrial> t;
  for (int block : {64, 128}) {
    for (int chunk : {1, 2, 4}) t.push_back({0, chunk, block, 7});
    for (int chunk : {4, 8}) t.push_back({1, chunk, block, 7});
  }
  if (fp32_limited)
    for (int minb : {7, 6, 5}) t.push_back({4, minb == 5 ? 4 : 2, 128, minb});
  for (int i = 0; i < 2; ++i)
    if (s.split[i]) t.push_back({6, 2, kSplitTrials[i], 7});
  return t;
}

struct FaceTrial {
  int mode, block, threads;
};
inline std::vector<FaceTrial> face_trials(const TrialScope& s, bool batched) {
  std::vector<FaceTrial> t;
  if (s.small) t.push_back({0, 64, 256});
  for (int mode : {1, 2})
    for (int block : {64, 128})
      for (int gather : {128, 256})
        if (mode == 1 || !batched) t.push_back({mode, block, gather});  // mode 2 with cases: as mode 1
  for (int i = 0; i < 3; ++i)
    for (int k : {1, 2, 4, 8})
      if (s.faces[i] && k * kFaceTrials[i] <= 256) t.push_back({3, kFaceTrials[i], k * kFaceTrials[i]});
  return t;
}

}  // namespace autan_b200

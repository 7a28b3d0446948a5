// batch_width.hpp -- threads per CTA of the batched kernel by the LPs of a call. Host code without
// CUDA headers, so that the rule can be checked without a GPU.
#pragma once

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

namespace sov {

constexpr int kBatchMaxRows = 128;  // IPM rows of an LP the batched kernel takes

// row bound of an LP's size bucket
inline int bucket_of(int m) { return std::max(32, ((m + 31) / 32) * 32); }

// The LPs of one call that the batched kernel solves. Every part of a call that is cut into parts goes by
// the whole call's numbers: the parts are on the GPU together, and an LP's bits depend on its width.
struct BatchCall {
  int lps = 0, max_cols = 0;  // model columns, without slacks
  double cols = 0.0;
  bool tuned = true;  // autotuned choices apply
  void add(int rows, int columns) {
    if (rows > kBatchMaxRows || columns <= 0) return;  // another path's
    ++lps;
    cols += columns;
    max_cols = std::max(max_cols, columns);
  }
};

// Width of the CTAs of the bucket with row bound mmax, where no pin and no autotuned choice says otherwise.
// An SM holds one CTA of 512 threads, two of 256, or four of 128 (three above 96 rows, by shared
// memory). Device times in ms, LPs x columns, at 128 / 256 / 512 threads:
//  - an SM for every LP: the widest (its column and row passes scale, the factor's pivot chain does not):
//    148 x 2500 1.84 / 1.37 / 1.18, 148 x 324 0.44 / 0.41 / 0.39.
//  - LPs of about one size: as narrow as it takes to have all on the GPU at once, a second wave costs
//    more than the width gives: 200 x 1225 1.08 / 0.83 / 1.38, 350 x 324 0.45 / 0.73 / 0.98, 592 x 576 0.70 / 1.05 /
//    1.82, 350 x 1600 1.38 / 2.03 / 2.32. Above 96 rows three LPs an SM is all there is at 128, and between three and
//    four LPs an SM two waves of 256 beat two of 128 (592 x 1100 2.74 / 2.28). With more LPs than that, those of more than
//    64 rows with long column passes want the wider CTA (1500 x 2500 at 100 rows 11.1 / 10.0), the others the more resident
//    LPs (1000 x 900 1.93 / 2.61, 3000 x 576 3.64 / 5.09, 2000 x 300 at 120 rows 7.28 / 7.88); with few rows the line lies where
//    the passes are nearly everything (2000 x 2000 at 20 rows 9.07 / 8.22; no size between 1024 and 2000
//    columns was measured there).
//  - sizes mixed: the call waits for its largest LPs, which are started first, so the width that is best for
//    them (transportation LPs with 10 to 60 sources and sinks, 1225 columns on average: 350 LPs 2.70 / 1.78, 592
//    3.19 / 1.93, 1000 5.02 / 3.47, 4096 16.9 / 13.3; up to 30 by 30, 290 columns on average: 350 0.69 / 0.61, but 1000 1.07 /
//    1.20, 2000 1.73 / 2.34), and up to two LPs an SM that of a single LP (200 LPs 1.64 at 256, 1.36 with the larger ones at 512).
inline int width_for(int sms, const BatchCall& call, int mmax) {
  if (call.lps <= sms) return 512;
  const double mean = call.cols / call.lps;
  if (call.max_cols >= 1.25 * mean) {
    if (call.lps <= 2 * sms) return mean >= 1000.0 ? 512 : 256;
    return mean >= (call.lps <= 4 * sms ? 250.0 : 600.0) ? 256 : 128;
  }
  if (call.lps <= 2 * sms) return 256;
  const bool wide = mean >= (mmax > 64 ? 600.0 : 1200.0);
  if (mmax > 64 || !wide) {
    if (call.lps <= 3 * sms) return 128;
    if (call.lps <= 4 * sms) return mmax > 96 ? 256 : 128;
  }
  return wide ? 256 : 128;
}

// LPs per SM of a call: 1 .. 4, 5 for more. The lines of width_for lie between these.
inline int lps_per_sm(int sms, int lps) { return std::min(5, std::max(1, (lps + sms - 1) / sms)); }

// The autotuner's choices. A choice holds for the size bucket and the LPs per SM it was timed at: the width
// that is fastest for 4096 LPs costs a batch of 24 or a single LP up to twice its time.
class TunedWidths {
 public:
  struct Choice {
    int threads = 0;  // 0: none
    int per_sm = 0;   // resident CTAs per SM (0: all that fit)
  };
  Choice find(int mmax, int load) {
    std::lock_guard<std::mutex> g(mu_);
    const auto it = choices_.find({mmax, load});
    return it != choices_.end() ? it->second : Choice{};
  }
  void set(int mmax, int load, Choice c) {
    std::lock_guard<std::mutex> g(mu_);
    choices_[{mmax, load}] = c;
  }

 private:
  std::mutex mu_;
  std::map<std::pair<int, int>, Choice> choices_;
};

}  // namespace sov

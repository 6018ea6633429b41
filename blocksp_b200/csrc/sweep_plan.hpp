// sweep_plan.hpp — lays the two triangular sweeps of a preconditioner out.
#pragma once
#include <functional>
#include <future>
#include "sweep_cost.h"
#include "sweep_stream.hpp"
#include "sweep_wave.hpp"

namespace bsp {

// f and g, on a thread each when `beside` (a thread that cannot be had: one
// after the other).
std::future<void> run_beside(bool beside, std::function<void()> f);
template <class F, class G> void both(bool beside, F f, G g) {
  std::future<void> other = run_beside(beside, f);
  g();
  other.get();
}
// Rows above which the two sweeps are planned on a thread each: 300 x 257 rows of
// 4 x 4 blocks are analysed in 17.5 ms so and in 23 one after another, but at 64 x
// 64 (2.3 ms) starting the threads costs as much as they save.
constexpr int kThreadRows = 8000;

// The forward and the backward sweep of a factor, or of SOR on A's own blocks.
// start() hands the host work (estimates, then the layout of the kernel that
// takes them) to threads of its own while the caller goes on with the rest of
// the analysis; finish() waits for it and uploads.  At most one of the layouts
// is made: none means that the level-ordered kernels run the sweeps (sizes that
// no other kernel takes, patterns where they are faster, a layout that is too
// long or does not fit memory).
class SweepPlanner {
 public:
  SweepEntries lo, up;  // what the rows of each sweep read
  bool lo_d = false, up_d = false, up_trans = false, up_trans_d = false;
  bool in_place = false;  // SOR: both sweeps read and write rows in natural order

  // true: finish() has layouts to upload
  bool start(int n, int bs);
  int finish(std::shared_ptr<WaveSym>& wv_lo, std::shared_ptr<WaveSym>& wv_up, std::shared_ptr<StreamSym>& ss_lo,
             std::shared_ptr<StreamSym>& ss_up);
  ~SweepPlanner();

 private:
  void plan();
  int n_ = 0, bs_ = 0;
  bool wave_ = false, stream_ = false;
  WavePlan w_lo_, w_up_;
  StreamPlan s_lo_, s_up_;
  std::future<void> job_;
};

}  // namespace bsp

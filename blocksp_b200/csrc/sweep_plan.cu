// sweep_plan.cu — see sweep_plan.hpp.
#include <new>
#include <system_error>
#include "sweep_plan.hpp"

namespace bsp {

std::future<void> run_beside(bool beside, std::function<void()> f) {
  if (beside) {
    try {
      return std::async(std::launch::async, f);
    } catch (const std::system_error&) {  // no thread to be had: when it is waited for
    }
  }
  return std::async(std::launch::deferred, f);
}

void SweepPlanner::plan() {
  const bool beside = n_ >= kThreadRows, streamed = !in_place && stream_supported(bs_);
  const SweepKernel other = streamed ? SweepKernel::kStreamed : SweepKernel::kPolled;
  try {
    if (wave_supported(bs_)) {
      double cost[2];
      both(beside, [&] { cost[0] = sweep_cost_us(other, bs_, n_, true, lo); },
           [&] { cost[1] = sweep_cost_us(other, bs_, n_, false, up); });
      const double limit = kWaveShare * (cost[0] + cost[1]);
      const WaveShape S = wave_shape(bs_, 1);
      bool ok[2];
      both(beside, [&] { ok[0] = wave_plan(n_, true, S, lo_d, lo, {}, w_lo_, limit); },
           [&] { ok[1] = wave_plan(n_, false, S, up_d, up, {}, w_up_, limit); });
      wave_ = ok[0] && ok[1] && w_lo_.est_us + w_up_.est_us <= limit;
    }
    if (wave_) return;
    w_lo_ = WavePlan{};
    w_up_ = WavePlan{};
    if (streamed) {
      int st[2];
      both(beside, [&] { st[0] = stream_plan(n_, true, stream_warps(bs_), lo, s_lo_); },
           [&] { st[1] = stream_plan(n_, false, stream_warps(bs_), up, s_up_); });
      stream_ = st[0] == BSP_OK && st[1] == BSP_OK;
    }
  } catch (const std::bad_alloc&) {
    wave_ = stream_ = false;
    w_lo_ = WavePlan{};
    w_up_ = WavePlan{};
  }
}

bool SweepPlanner::start(int n, int bs) {
  n_ = n;
  bs_ = bs;
  if (!wave_supported(bs) && (in_place || !stream_supported(bs))) return false;
  job_ = run_beside(n >= kThreadRows, [this] { plan(); });
  return true;
}

SweepPlanner::~SweepPlanner() {
  if (job_.valid()) job_.wait();
}

int SweepPlanner::finish(std::shared_ptr<WaveSym>& wv_lo, std::shared_ptr<WaveSym>& wv_up,
                         std::shared_ptr<StreamSym>& ss_lo, std::shared_ptr<StreamSym>& ss_up) {
  wv_lo = wv_up = nullptr;
  ss_lo = ss_up = nullptr;
  if (!job_.valid()) return BSP_OK;
  job_.get();
  auto upload = [&]() -> int {
    if (wave_) {
      auto a = std::make_shared<WaveSym>(), b = std::make_shared<WaveSym>();
      std::vector<int> up_item;  // per row: the item of the backward sweep that reads it
      BSP_TRY(wave_upload(std::move(w_up_), bs_, up_trans, up_d, up_trans_d, nullptr, &up_item, *b));
      BSP_TRY(wave_upload(std::move(w_lo_), bs_, false, lo_d, false, in_place ? nullptr : &up_item, nullptr, *a));
      wv_lo = a;
      wv_up = b;
    } else if (stream_) {
      auto a = std::make_shared<StreamSym>(), b = std::make_shared<StreamSym>();
      BSP_TRY(stream_upload(s_up_, up_trans, up_d, up_trans_d, *b));
      BSP_TRY(stream_upload(s_lo_, false, lo_d, false, *a));
      ss_lo = a;
      ss_up = b;
    }
    return BSP_OK;
  };
  const int st = upload();
  if (st != BSP_OUT_OF_MEMORY) return st;
  record_error("");  // the level-ordered kernels need no layout
  return BSP_OK;
}

}  // namespace bsp

// What an operator makes on first use (host code, no CUDA).
#pragma once

#include <atomic>
#include <mutex>

#include "../../include/hedge_b200.h"

namespace hb {

// Up to 16 variants, each made on its first use by whichever thread comes
// first.  One that is refused as unsupported stays refused; any other failure
// (memory that is short now) is tried again by the next use.
class Prepared {
 public:
  bool has(int variant) const { return state_.load(std::memory_order_acquire) >> variant & 1u; }

  // Whether `variant` is ready, made by prepare() -> hb_status if need be;
  // failed() clears what a failing prepare left behind.
  template <typename PREPARE, typename FAILED>
  bool ready(int variant, PREPARE prepare, FAILED failed) {
    const unsigned made = 1u << variant, refused = 0x10000u << variant;
    const unsigned now = state_.load(std::memory_order_acquire);
    if (now & (made | refused)) return now & made;
    try {
      std::lock_guard<std::mutex> lock(mutex_);
      const unsigned then = state_.load(std::memory_order_acquire);
      if (then & (made | refused)) return then & made;
      const hb_status st = prepare();
      if (st == HB_OK || st == HB_ERR_UNSUPPORTED)
        state_.fetch_or(st == HB_OK ? made : refused, std::memory_order_acq_rel);
      if (st == HB_OK) return true;
    } catch (...) {   // host memory; nothing may leave through the C interface
    }
    failed();
    return false;
  }

 private:
  std::mutex mutex_;
  std::atomic<unsigned> state_{0};
};

}  // namespace hb

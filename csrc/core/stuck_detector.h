// What the watchdog of a communicator concludes from its readings of the operator counters: an operator is stuck when started and
// finished counts differ and neither moves for a whole budget (reference: per-communicator head/tail counters compared by a host
// watchdog, stuck_detect_counter_helper.h).  A reading that does not come back counts as no progress, too: the copy may wait
// behind the very operator that is stuck.
#pragma once
#include <cstdint>

namespace hccl {

class StuckDetector {
public:
    explicit StuckDetector(double budgetS) : budgetS_(budgetS) {}
    // A reading at `nowS`; `answered` == false: it has not come back.  True: report it (again after another budget).
    bool Observe(bool answered, uint64_t started, uint64_t finished, double nowS)
    {
        const bool moved = answered && (started != started_ || finished != finished_ || started == finished);
        if (answered) { started_ = started; finished_ = finished; }
        if (moved || sinceS_ < 0) { sinceS_ = nowS; return false; }
        idleS_ = nowS - sinceS_;
        if (idleS_ <= budgetS_) return false;
        sinceS_ = nowS;
        return true;
    }
    uint64_t started() const { return started_; }       // of the last reading that came back
    uint64_t finished() const { return finished_; }
    double idleS() const { return idleS_; }             // without progress when it last reported

private:
    double budgetS_, sinceS_ = -1, idleS_ = 0;
    uint64_t started_ = 0, finished_ = 0;
};

}  // namespace hccl

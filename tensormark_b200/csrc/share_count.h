// share_count.h — the counter behind a vector that the CTAs of a launch stage together, and the host's idea of it.
//
// Every launch adds a number of parts to the device counter and waits for the sum of all launches since it was zeroed. The
// host therefore counts a launch when it was made, not before: one that failed adds nothing on the device, and a sum ahead
// of the counter would be waited for in vain by every later launch.
#pragma once

namespace tmc {

struct ShareCount {
    unsigned* parts = nullptr;               // device: parts staged since it was zeroed
    unsigned total = 0;                      // what the launches since then add up to
    bool level = false;                      // both say the same: false until zeroed, and after a call whose kernel may not have run
    // go(want) launches a kernel that adds n parts and waits for `want`.
    template <typename Launch> bool launch(unsigned n, Launch go) {
        const unsigned want = total + n;     // wraps as the counter does
        if (!go(want)) return false;
        total = want;
        return true;
    }
};

}  // namespace tmc

// How many SMs a launch plans with when other launches share the GPU.
//
// The forms with several lanes to an item (verify_w.cu, g1.cuh, h2c.cuh, g2.cuh) buy a
// small batch latency with SM time: a block of the 32-item kernel fills an SM, and 32
// items on four lanes each hold 4 SMs for 2.49 ms where a lane each holds one for 3.42,
// 2.9 times as much.  That is right while the SMs would stand idle, and wrong when other
// launches would have run on them: three launches of 1,184 items are 37 blocks each and
// run side by side with a lane an item, but fill the chip three times over with four
// (together 3.48 and 7.48 ms; 8 x 300 items 3.50 and 7.44).
// So every call that launches such a kernel is counted on its device from where it
// starts to where its work has run, with the SMs that its verify launch holds, and a
// launch plans with the SMs the others leave.  Only the time depends on it: every
// number of lanes gives the same values.
//
// No CUDA in this file: what is counted are host calls.
#pragma once
#include <algorithm>
#include <mutex>

namespace bls {

constexpr int kBlockItems = 32;   // items of a k_verify_w block with a lane to each

// Lanes to an item for the items of n that fill no whole wave of `sms` blocks, of which
// the launch plans to use `share`: as many as still give each item a place at once.
inline int verify_item_lanes(int n, int sms, int share) {
    const int rest = n % (kBlockItems * sms);
    return rest == 0 ? 1 : rest <= 8 * share ? 4 : rest <= 16 * share ? 2 : 1;
}
// SMs that those launches hold at the most
inline int verify_sms_held(int n, int sms, int lanes) {
    if (n > kBlockItems * sms) return sms;
    return (int)std::min<long long>(sms, ((long long)n * lanes + kBlockItems - 1) / kBlockItems);
}

// One call at work on a device (or a server's slot, or its ring kernel).  begin() and
// end() from one thread at a time; a use that outlives its call (end_when) is ended by
// whichever call next looks at the device and finds its work done.
class ChipUse {
  public:
    ChipUse() = default;
    ChipUse(const ChipUse&) = delete;
    ChipUse& operator=(const ChipUse&) = delete;
    ~ChipUse() { end(); }

    // caller: a call of a context; false for a server's launches, which come from a queue
    // that the server sees, and tell nothing about how many callers there will be
    void begin(int device, int sms, bool caller = true) {
        end();
        Chip& c = chip(device);
        std::lock_guard<std::mutex> lk(c.mu);
        reap(c);
        chip_ = &c;
        sms_ = sms;
        on_ = waiting_ = true;
        next_ = c.uses;
        c.uses = this;
        caller_ = caller;
        ++c.users;
        if (caller) c.peak = std::max(c.peak, ++c.callers);
    }
    void end() {
        if (!chip_) return;
        std::lock_guard<std::mutex> lk(chip_->mu);
        if (on_) leave(*chip_);
    }
    // Ends once done(what) says so; called under the device's lock, from any thread.
    void end_when(bool (*done)(const void*), const void* what) {
        std::lock_guard<std::mutex> lk(chip_->mu);
        if (!on_) return;
        waiting_ = false;
        done_ = done;
        what_ = what;
    }

    // SMs a launch that needs at least `need` of them plans with: of those that no
    // other use holds an equal part, the uses that have not launched yet having theirs to
    // come.  expect: as many callers are expected as met the last time there were any
    // (calls that return before their work is done show up one after another; a server
    // knows its own queue).  Where the part is too small the launch has to wait for others
    // in any case, and plans with an equal part of the whole chip, of which the uses that
    // hold less keep what they hold.
    int share(int need, bool expect = true) {
        std::lock_guard<std::mutex> lk(chip_->mu);
        reap(*chip_);
        return share_locked(need, expect);
    }
    // Lanes to an item for a verify launch of n items, whose SMs this use holds from now on.
    int plan_verify(int n, bool expect = true) {
        std::lock_guard<std::mutex> lk(chip_->mu);
        reap(*chip_);
        // a remainder after whole waves runs when what the others hold now is long done
        const int need = n > kBlockItems * sms_ ? sms_ + 1 : verify_sms_held(n, sms_, 1);
        const int lanes = verify_item_lanes(n, sms_, share_locked(need, expect));
        hold_locked(verify_sms_held(n, sms_, lanes));
        return lanes;
    }
    // SMs held by a launch that was planned elsewhere
    void hold(int sms) {
        std::lock_guard<std::mutex> lk(chip_->mu);
        hold_locked(sms);
    }

  private:
    struct Chip {
        std::mutex mu;
        ChipUse* uses = nullptr;       // begun and not ended, linked by next_
        int users = 0, callers = 0;    // how many, and of those, calls of contexts
        int peak = 0, last_peak = 0;   // most callers at once: since there was none, and before
    };
    static constexpr int kChips = 64;
    static Chip& chip(int device) {
        static Chip chips[kChips];
        return chips[(unsigned)device % kChips];
    }

    int share_locked(int need, bool expect) const {
        const Chip& c = *chip_;
        const int missing = expect ? std::max(0, c.last_peak - c.callers) : 0;
        int held = 0, waiting = 0;
        for (const ChipUse* u = c.uses; u; u = u->next_) {
            if (u == this) continue;
            held += u->held_;
            waiting += u->waiting_;
        }
        const int part = std::max(0, sms_ - held) / (1 + std::max(waiting, missing));
        if (need <= part) return part;
        for (int level = sms_ / (c.users + missing);;) {
            int rest = sms_, equal = 1 + missing;   // SMs and uses but for those that hold less
            for (const ChipUse* u = c.uses; u; u = u->next_) {
                if (u == this) continue;
                if (!u->waiting_ && u->held_ < level) rest -= u->held_;
                else ++equal;
            }
            if (rest / equal <= level) return std::max(1, level);
            level = rest / equal;
        }
    }
    void hold_locked(int sms) {
        if (!on_) return;
        waiting_ = false;
        held_ = sms;
    }
    void leave(Chip& c) {
        ChipUse** at = &c.uses;
        while (*at != this) at = &(*at)->next_;
        *at = next_;
        --c.users;
        if (caller_ && --c.callers == 0) {
            c.last_peak = c.peak;
            c.peak = 0;
        }
        on_ = waiting_ = false;
        held_ = 0;
        done_ = nullptr;
    }
    static void reap(Chip& c) {
        for (ChipUse *u = c.uses, *next; u; u = next) {
            next = u->next_;
            if (u->done_ && u->done_(u->what_)) u->leave(c);
        }
    }

    Chip* chip_ = nullptr;
    int sms_ = 0, held_ = 0;
    bool on_ = false, waiting_ = false, caller_ = false;
    bool (*done_)(const void*) = nullptr;
    const void* what_ = nullptr;
    ChipUse* next_ = nullptr;
};

}  // namespace bls

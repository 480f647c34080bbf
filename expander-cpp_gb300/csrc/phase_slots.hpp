// Which persistent sumcheck phases may be on a device together.  Host code only.
#pragma once
#include <stdint.h>

#include <atomic>

namespace gkrgpu {

// The CTAs of a persistent phase wait for their host thread, which waits for all of them, so a
// phase's CTAs end only once all have started.  Two rules hold for the CTAs of all phases of the
// process on a device (every context and lane); a phase that they keep out is launched round by
// round.
// - At most what the device holds (two an SM, `per_sm`), so that none is queued behind others'
//   whole phases.
// - Those not yet known to be on the device: at most one an SM.  Phases that are wholly on it end
//   by themselves, whatever the others do, so only the rest could keep each other out for good;
//   of those, as long as a CTA has no place some SM has none of their CTAs, and takes it.  It is
//   not enough that the device holds them all: a launch sets the split of an SM's memory, and CTAs
//   of 97 KB do not start beside one of 26 KB, nor ones of 50 KB beside one of 97, before that
//   one has ended.  (Asking all launches for the largest shared-memory part instead leaves the M31
//   phases less L1: layers of 2^10 rows and 16 copies 1.01 -> 1.03 ms a proof, 16 mixed proofs in
//   as many lanes 26.2 -> 26.9 ms.  One CTA an SM in all, placed or not, takes 40 copies of 2^10
//   BN254 rows in 8 lanes from 243 to 303 us a proof, 512 copies of 2^10 M31 rows from 459 to 509.)
// A phase of more CTAs than SMs comes in when no other is on its way, and its launch has to ask
// for the largest part.  Other kernels only delay a phase: they end by themselves.
class PhaseSlots {
   public:
    // `state` is the device's, shared by all its phases: CTAs admitted, and in the high word those
    // not yet placed.
    PhaseSlots(std::atomic<uint64_t>& state, int sms, int per_sm)
        : state_(state), sms_((uint32_t)sms), cap_((uint32_t)(sms * per_sm)) {}
    PhaseSlots(const PhaseSlots&) = delete;
    ~PhaseSlots() { state_ -= (uint64_t)waiting_ << 32 | held_; }
    uint32_t capacity() const { return cap_; }
    // n more CTAs; beyond a lane's own share of the device only while half of it stays free.
    bool acquire(uint32_t n, bool own_share) {
        uint64_t s = state_.load();
        do {
            const uint32_t held = (uint32_t)s, waiting = (uint32_t)(s >> 32);
            if (held + n > (own_share ? cap_ : cap_ / 2)) return false;
            if (waiting && waiting + n > sms_) return false;
        } while (!state_.compare_exchange_weak(s, s + ((uint64_t)n << 32 | n)));
        held_ += n;
        waiting_ += n;
        return true;
    }
    // All of this phase's CTAs are on the device (its first round has been published).
    void placed() {
        state_ -= (uint64_t)waiting_ << 32;
        waiting_ = 0;
    }

   private:
    std::atomic<uint64_t>& state_;
    uint32_t sms_, cap_, held_ = 0, waiting_ = 0;
};

}  // namespace gkrgpu

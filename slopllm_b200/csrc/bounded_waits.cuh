// Waits of one thread on barriers of its block that end also where the barrier's phase never comes: once a wait has run out, in this thread or
// in another of the block, none waits any more.  `Dev` is what the waits need of the machine (mbarriers and clocks on the device):
//
//   Bar, try_wait(bar, parity)   waits a moment at most; test(bar, parity) does not wait
//   now_ns()                     a clock
//   any(flag)                    true where the flag is true in any thread that waits along
//   report(err, code)            writes the error word
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SL_WAITS_FN __device__ __forceinline__
#else
#define SL_WAITS_FN inline
#endif

template <typename Dev>
struct BoundedWaits {
    static constexpr uint64_t LIMIT_NS = 2000000000ull;
    static constexpr uint32_t POLLS = 1u << 22;      // of `either`, some 0.2 s

    volatile int* failed;                            // the block's
    int* err;
    int code;
    bool alive = true;

    SL_WAITS_FN bool operator()(typename Dev::Bar* bar, uint32_t parity) {
        if (!alive) return false;
        if (Dev::try_wait(bar, parity)) return true;
        uint64_t t0 = 0;
        for (uint32_t i = 1;; ++i) {
            if (Dev::try_wait(bar, parity)) return true;
            if ((i & 255u) == 0u) {
                const uint64_t now = Dev::now_ns();
                if (t0 == 0) t0 = now;
                if (*failed != 0 || now - t0 > LIMIT_NS) break;
            }
        }
        *failed = 1;
        Dev::report(err, code);
        alive = false;
        return false;
    }

    // Polls until the phase of `a` or that of `b` has passed.  True: that of `b` has, and `a`'s had not when it was looked at.  False also where
    // a wait has run out or the polls have: the caller waits for `a` next, which is bounded.  For threads that have `alive` in common.
    SL_WAITS_FN bool second_of(typename Dev::Bar* a, uint32_t parity_a, typename Dev::Bar* b, uint32_t parity_b) const {
        for (uint32_t i = 1; alive && i <= POLLS; ++i) {
            if (Dev::any(Dev::test(a, parity_a))) return false;
            if (Dev::any(Dev::test(b, parity_b))) return true;
            if ((i & 255u) == 0u && Dev::any(*failed != 0)) return false;
        }
        return false;
    }
};

// The policy of a kernel's bounded waits, apart from the barrier and the clock
// they look at.
#pragma once
#include <stdint.h>

namespace sg {
namespace tc {

constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;

// Look until `ready` holds (true), the CTA's abort word is set, or limit_ns of
// `now` have passed (false). The word is read before the first look and the
// clock once in 64, so that a wait behind another's timeout costs nothing.
template <class Ready, class Now>
__device__ bool bounded_wait(Ready ready, Now now, const volatile uint32_t* abort, uint64_t limit_ns) {
    const uint64_t t0 = now();
    do {
        if (*abort) return false;
        for (int i = 0; i < 64; ++i)
            if (ready()) return true;
    } while (now() - t0 < limit_ns);
    return false;
}

}  // namespace tc
}  // namespace sg

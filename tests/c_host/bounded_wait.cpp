// Host-side check of the kernels' bounded waits (csrc/wait.cuh), compiled with
// g++: a clock that advances with every reading and a barrier that completes
// at a given look, or never.
#include <stdio.h>

#define __device__
#include "../../lambda_vm_b200/csrc/wait.cuh"

static uint64_t g_now, g_step;
static unsigned g_looks, g_ready_at;   // 0: never
static volatile uint32_t g_abort;
static unsigned g_abort_at;            // look at which another thread gives up, 0: never

static uint64_t now() { return g_now += g_step; }
static bool ready() {
    ++g_looks;
    if (g_looks == g_abort_at) g_abort = 1;
    return g_looks == g_ready_at;
}
static bool wait(uint64_t step, unsigned ready_at, unsigned abort_at, uint32_t abort) {
    g_now = 0, g_step = step, g_looks = 0, g_ready_at = ready_at, g_abort_at = abort_at, g_abort = abort;
    return sg::tc::bounded_wait(ready, now, &g_abort, sg::tc::WAIT_LIMIT_NS);
}

#define EXPECT(cond)                                       \
    do {                                                   \
        if (!(cond)) {                                     \
            printf("FAIL line %d: %s\n", __LINE__, #cond); \
            return 1;                                      \
        }                                                  \
    } while (0)

int main() {
    const uint64_t ms = 1000000;
    EXPECT(wait(6 * ms, 1, 0, 0) && g_looks == 1);
    EXPECT(wait(6 * ms, 1000, 0, 0) && g_looks == 1000);
    // never complete: it gives up, and within the limit plus one round of looks
    EXPECT(!wait(6 * ms, 0, 0, 0) && g_now >= sg::tc::WAIT_LIMIT_NS && g_now <= sg::tc::WAIT_LIMIT_NS + 12 * ms);
    EXPECT(!wait(sg::tc::WAIT_LIMIT_NS, 0, 0, 0) && g_looks == 64);
    // another thread gave up before: not one look; during: no further round
    EXPECT(!wait(6 * ms, 5, 0, 1) && g_looks == 0);
    EXPECT(!wait(6 * ms, 0, 70, 0) && g_looks == 128);
    EXPECT(wait(6 * ms, 100, 70, 0) && g_looks == 100);
    printf("ok\n");
    return 0;
}

// The waits of the tensor-core base conversion (tc_poll, bconv_tc_plan.h) against barriers that end after a number of polls, or
// never. Prints "ok" or the first rule that is broken.
#include <cstdio>

#include "bconv_tc_plan.h"

struct Barrier {
    uint64_t ends_after, polls = 0;
    bool operator()() { return ++polls > ends_after; }
};
static const uint64_t NEVER = ~0ull;

static bool wait(Barrier &b, volatile uint32_t *gave_up, bool drain) { return b2::tc_poll([&] { return b(); }, gave_up, drain); }

int main() {
    volatile uint32_t flag;
    for (uint64_t n : {0ull, 1ull, 5000ull, (unsigned long long)b2::TC_WAIT_LIMIT - 1}) {
        for (int drain = 0; drain < 2; drain++) {
            Barrier b{n};
            flag = 0;
            if (!wait(b, &flag, drain) || flag || b.polls != n + 1) return printf("a wait of %llu polls\n", (unsigned long long)n), 1;
        }
        // another wait of the CTA has run out: what is in flight is waited for all the same, everything else is left at once
        Barrier copy{n}, other{n};
        flag = 1;
        if (!wait(copy, &flag, true) || copy.polls != n + 1) return printf("a copy in flight is left after %llu polls\n", (unsigned long long)copy.polls), 1;
        if (wait(other, &flag, false) != (n == 0) || other.polls != 1) return printf("a wait goes on after another gave up\n"), 1;
    }
    for (int drain = 0; drain < 2; drain++) {
        Barrier b{NEVER};
        flag = 0;
        if (wait(b, &flag, drain) || !flag || b.polls != b2::TC_WAIT_LIMIT) return printf("a wait without an end\n"), 1;
    }
    Barrier b{NEVER};
    flag = 1;
    if (wait(b, &flag, true) || b.polls != b2::TC_WAIT_LIMIT) return printf("a drain without an end\n"), 1;
    printf("ok\n");
    return 0;
}

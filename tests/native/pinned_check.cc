// Check of the range test that lets a request's pinned buffer be copied by a
// kernel.  Prints "ok".
#include <cstdio>

#include "../../multians_gb300/csrc/mans_pinned.h"

static int fails = 0;
static void check(bool got, bool want, const char* what) {
    if (got != want) {
        std::printf("%s: %d, want %d\n", what, got, want);
        ++fails;
    }
}

int main() {
    using mans::range_covers;
    const uint64_t s = 0x7f0000010000ull, z = 65536;
    check(range_covers(s, z, s, z), true, "all of it");
    check(range_covers(s, z, s + 1, z - 1), true, "to its end");
    check(range_covers(s, z, s + 1, z), false, "one byte past its end");
    check(range_covers(s, z, s - 1, 10), false, "one byte before it");
    check(range_covers(s, z, s + z, 1), false, "behind it");
    check(range_covers(s, z, s + z - 1, 1), true, "its last byte");
    // two registrations with a hole between: the first one ends before the buffer does
    check(range_covers(s, z, s + 100, 3 * z - 200), false, "over a hole");
    check(range_covers(0, 0, 0, 0), false, "no range");
    check(range_covers(s, 0, s, 0), false, "range of no size");
    check(range_covers(~0ull - 9, 10, ~0ull - 9, 10), true, "at the top");
    check(range_covers(~0ull - 9, 10, ~0ull - 4, 10), false, "past the top");
    if (!fails) std::printf("ok\n");
    return fails != 0;
}

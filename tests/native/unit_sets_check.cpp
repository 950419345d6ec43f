// Checks the split of a batch into sets of situations for every batch size up to 3000 and every first
// size: all situations covered, no more sets than counter slots, and each retry smaller, down to the
// smallest set.  Prints "ok" or the first failure.
#include <cstdio>

#include "batch_rules.h"

using namespace gral;

static bool good(int nb, int units) {
    return units >= 1 && units <= nb && (nb + units - 1) / units <= kCounterSlots;
}

int main() {
    for (int nb = 1; nb <= 3000; ++nb)
        for (int fit = 0; fit <= nb + 1; fit += 1 + fit / 8) {
            int units = set_units(nb, (size_t)fit), last = 0;
            if (!good(nb, units) || (fit >= min_units(nb) && units > fit)) {
                std::printf("set_units(%d, %d) = %d\n", nb, fit, units);
                return 1;
            }
            for (int tries = 0; units; ++tries) {
                last = units;
                units = fewer_units(nb, units);
                if (units && (!good(nb, units) || units >= last || tries > 40)) {
                    std::printf("fewer_units(%d, %d) = %d\n", nb, last, units);
                    return 1;
                }
            }
            if (last != min_units(nb)) {
                std::printf("retries of %d end at %d\n", nb, last);
                return 1;
            }
        }
    std::puts("ok");
    return 0;
}

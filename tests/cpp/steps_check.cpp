// Exercises tgbm::each_step.  Prints "<name> <positions met by all lanes> <sum of their distances from the begin> <largest distance>".
#include <climits>
#include <cstdio>

#include "../../thundergbm_b200/csrc/tgbm_steps.h"

static void scenario(const char *name, int begin, int end, unsigned lanes) {
    unsigned long long met = 0, sum = 0, most = 0;
    for (unsigned lane = 0; lane < lanes; ++lane)
        tgbm::each_step(begin, end, lane, lanes, [&](unsigned j) {
            const unsigned long long d = (unsigned long long)j - (unsigned)begin;
            ++met; sum += d;
            if (d > most) most = d;
        });
    printf("%s %llu %llu %llu\n", name, met, sum, most);
}

int main() {
    scenario("few", 5, 12, 32);
    scenario("none", 12, 12, 32);
    scenario("many", 0, 100000, 32);
    scenario("last_warp", INT_MAX - 70, INT_MAX, 32);
    scenario("last_value", INT_MAX - 1, INT_MAX, 64);
    scenario("last_grid", INT_MAX - 1000, INT_MAX, 1184 * 256);
    return 0;
}

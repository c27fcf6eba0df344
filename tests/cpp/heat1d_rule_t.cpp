// Prints memory_limit (csrc/heat1d_schedule.hpp) for the books on stdin: "<groups> <sms>", then one line
// "n rows lanes steps" per group.  With the argument "shape": "W R" for every "rows least most".
#include "heat1d_schedule.hpp"

#include <cstdio>

int main(int argc, char **)
{
    if (argc > 1) {
        int rows, least, most, W, R;
        while (std::scanf("%d %d %d", &rows, &least, &most) == 3) {
            lss_gb300::heat1d::register_shape(rows, least, most, W, R);
            std::printf("%d %d\n", W, R);
        }
        return 0;
    }
    int count, sms;
    while (std::scanf("%d %d", &count, &sms) == 2) {
        std::vector<lss_gb300::heat1d::group_cost> g(count);
        for (auto &c : g)
            if (std::scanf("%d %d %d %d", &c.n, &c.rows, &c.lanes, &c.steps) != 4) return 1;
        std::printf("%d\n", lss_gb300::heat1d::memory_limit(g, sms, 16));
    }
    return 0;
}

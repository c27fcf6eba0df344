// Prints table_at<slots> (csrc/adi_index.hpp) of every "t slot q pitch slots" line on stdin.
#include <cstdio>

#include "adi_index.hpp"

int main()
{
    int t, slot, q, pitch, slots;
    while (std::scanf("%d %d %d %d %d", &t, &slot, &q, &pitch, &slots) == 5)
        std::printf("%lld\n", slots == 18 ? lss_gb300::table_at<18>(t, slot, q, pitch)
                              : slots == 10 ? lss_gb300::table_at<10>(t, slot, q, pitch)
                              : slots == 5 ? lss_gb300::table_at<5>(t, slot, q, pitch)
                                           : lss_gb300::table_at<3>(t, slot, q, pitch));
    return 0;
}

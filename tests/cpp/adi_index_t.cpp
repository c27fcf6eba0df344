// Prints the element offset (csrc/adi_index.hpp) of every "t slot q pitch slots" line on stdin (slots 180: the
// 18 slots of rows up to NEAR_PITCH) and that limit.
#include <cstdio>

#include "adi_index.hpp"

template <int SLOTS, bool FAR = true> static long long offset(int t, int slot, int q, int pitch)
{
    const lss_gb300::table_index<SLOTS, FAR> i(pitch);
    return i.base() + i.at(t, slot, q);
}

int main()
{
    int t, slot, q, pitch, slots;
    while (std::scanf("%d %d %d %d %d", &t, &slot, &q, &pitch, &slots) == 5)
        std::printf("%lld\n", slots == 18 ? offset<18>(t, slot, q, pitch)
                              : slots == 180 ? offset<18, false>(t, slot, q, pitch)
                              : slots == 50 ? offset<5, false>(t, slot, q, pitch)
                              : slots == 10 ? offset<10>(t, slot, q, pitch)
                              : slots == 5 ? offset<5>(t, slot, q, pitch)
                                           : offset<3>(t, slot, q, pitch));
    std::printf("%d\n", lss_gb300::NEAR_PITCH);
    return 0;
}

// adi_index.hpp -- element offset in the line tables of the batched kernels: row t holds all its SLOTS tables of
// `pitch` (at most 2^28) elements one after the other.  Plain C++, shared with the host tests.
#pragma once

#ifdef __CUDACC__
#define LSS_HD __host__ __device__
#else
#define LSS_HD
#endif

namespace lss_gb300 {

// A row of the S tables alone passes 2^31 elements on a grid of 4 x 2^28 points.  FP64 (ten slots): half a
// row fits an int, counted from the row's middle slot.  FP32 (18 slots): 64 bits; its v tables (five)
// unsigned numbers.  The choice is the kernels': with 64-bit or unsigned rows the FP64 ones lose 3 to 5 %
// (20000 Craig-Sneyd calls of 64 x 16 126.5 against 119.9 ms), with signed v rows FP32 Douglas-Rachford
// 40 % (768 uneven calls 72 against 52 ms).  Against rows counted in ints, which the longest do not fit, the
// FP32 kernels take 1 to 3 % longer (604 Craig-Sneyd calls 50.2 and 49.2 ms).
template <int SLOTS> struct table_index {
    static constexpr bool half = SLOTS == 10, wide = SLOTS == 18, plain = SLOTS == 3;
    static_assert(half || wide || plain || SLOTS == 5, "elements of a row");
    int pitch;
    int part; // elements of a row, or of half a row
    LSS_HD explicit table_index(int p = 0) : pitch(p), part(plain ? SLOTS * p : half ? SLOTS / 2 * p : 0) {}
    // added once to the tables' address
    LSS_HD long long base() const { return half ? part : 0; }
    // element q of slot `slot` in row t, from there
    LSS_HD long long at(int t, int slot, int q) const
    {
        if (half) return static_cast<long long>(2 * t) * part + ((slot - SLOTS / 2) * pitch + q);
        if (plain) return static_cast<long long>(t) * part + (slot * pitch + q);
        if (wide) return t * (static_cast<long long>(pitch) * SLOTS) + static_cast<long long>(slot) * pitch + q;
        const unsigned p = static_cast<unsigned>(pitch);
        return static_cast<long long>(static_cast<unsigned long long>(t) * (p * SLOTS) + (static_cast<unsigned>(slot) * p + static_cast<unsigned>(q)));
    }
};

} // namespace lss_gb300

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
// row fits an int, counted from the row's middle slot.  FP32 (18 slots): rows counted in ints up to
// NEAR_PITCH, in 64 bits beyond, by kernels of their own (FAR); its v tables (five) in 64 bits.  The choice
// is the kernels': with 64-bit or unsigned rows the FP64 ones lose 3 to 5 % (20000 Craig-Sneyd calls of
// 64 x 16 126.5 against 119.9 ms), the FP32 ones 2 to 3 % (768 uneven Douglas-Rachford calls 52.6 against
// 50.8 ms) and with other mixtures up to 40 % (v rows counted in ints 70 ms).
constexpr int NEAR_PITCH = 2147483647 / 18;
template <int SLOTS, bool FAR = true> struct table_index {
    static constexpr bool half = SLOTS == 10, wide = (SLOTS == 18 && FAR) || SLOTS == 5;
    static_assert(half || SLOTS == 18 || SLOTS == 3 || SLOTS == 5, "elements of a row");
    int pitch;
    int part; // elements of a row, or of half a row
    LSS_HD explicit table_index(int p = 0) : pitch(p), part(wide ? 0 : half ? SLOTS / 2 * p : SLOTS * p) {}
    // added once to the tables' address
    LSS_HD long long base() const { return half ? part : 0; }
    // element q of slot `slot` in row t, from there
    LSS_HD long long at(int t, int slot, int q) const
    {
        if (half) return static_cast<long long>(2 * t) * part + ((slot - SLOTS / 2) * pitch + q);
        if (wide) return t * (static_cast<long long>(pitch) * SLOTS) + static_cast<long long>(slot) * pitch + q;
        return static_cast<long long>(t) * part + (slot * pitch + q);
    }
};

} // namespace lss_gb300

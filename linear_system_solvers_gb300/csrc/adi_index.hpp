// adi_index.hpp -- element offset in the line tables of the batched kernels: row t holds all its SLOTS tables of
// `pitch` (at most 2^28) elements one after the other.  Plain C++, shared with the host tests.
#pragma once

#ifdef __CUDACC__
#define LSS_HD __host__ __device__
#else
#define LSS_HD
#endif

namespace lss_gb300 {

// A row alone passes 2^31 elements on a grid of 4 x 2^28 points.  Ten slots (FP64) stay below 2^32, so
// their row is a 32-bit unsigned number; 18 slots (FP32) need 64 bits in every product.  (64 bits for
// both cost the FP64 kernels 3 %: 1024 uneven calls 194.8 against 188.2 ms; FP32 is unchanged.)
template <int SLOTS> LSS_HD inline long long table_at(int t, int slot, int q, int pitch)
{
    if (SLOTS <= 15) {
        const unsigned p = static_cast<unsigned>(pitch);
        return static_cast<long long>(static_cast<unsigned long long>(t) * (p * SLOTS) + (static_cast<unsigned>(slot) * p + static_cast<unsigned>(q)));
    }
    return t * (static_cast<long long>(pitch) * SLOTS) + static_cast<long long>(slot) * pitch + q;
}

} // namespace lss_gb300

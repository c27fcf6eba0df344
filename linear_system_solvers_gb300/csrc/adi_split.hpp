// adi_split.hpp -- partition of the line solves of one instance over the whole GPU: plain C++, shared by
// the kernels (adi_wide.cuh), their host side (adi_wide.cu) and the host tests.
#pragma once

#ifdef __CUDACC__
#define LSS_HD __host__ __device__
#else
#define LSS_HD
#endif

namespace lss_gb300 {
namespace wide {

constexpr int MAX_CTA = 512; // threads per CTA (128 registers each)

// One direction's partition.
struct split {
    int L = 8, PC = 1; // lines per CTA, chunks per line
    int R = 4;         // rows per chunk (compiled: 5, 8, 16 for S lines, 4, 8, 16 for v lines)
    int gs = 1;        // chunks per group of the composition
    int tiles = 1;
    LSS_HD int groups() const { return (PC + gs - 1) / gs; }
};

// Partition of a line's `rows` rows, of which a direction has `lines`; chunks > 0 forces the chunk count.
// Short chunks as long as they fit one CTA: the time of a small instance is the chain of one chunk and
// the composition, and few lines per CTA spread the FP64 work over more SMs (one 32-byte sector of
// doubles per row of an S stage, at 4 lines).  Measured per step (S and v stages of one split, others
// alike): 1000 x 500 HV 64 us with v (8 lines, 63 chunks of 8), 75 us with (8, 32 of 16), 107 us with
// S (4, 63 of 16) instead of (4, 125 of 8).  At least five rows per S chunk (four per v chunk, boundary
// rows included).
//
// Longer lines take tiles of 16 rows per chunk, one after the other.  S lines that fill the SMs at 8
// lines per CTA take 32 chunks (4096 x 2048 HV 0.84 ms a step with S (8, 32 of 16) or v (4, 64 of 16),
// 0.88 ms with 8 rows per chunk).  Fewer lines take the 128 chunks that a count may have, 4 lines per CTA,
// or 2 (FP64) where 2 do not fill the SMs either: three HV steps of 4096 x 1000 1.64 ms (8, 32 of 16: 2.30),
// of 6000 x 200 2.0 ms (5.4), of 20000 x 64 3.9 ms (11.1).  Half a sector per row is the least: with
// two lines FP32 takes 1.3 ms instead of 0.88 on 6000 x 200.
inline split choose_split(int rows, int lines, bool vec, int chunks, int sms, int word)
{
    split s;
    const int sizes_s[] = {5, 8, 16}, sizes_v[] = {4, 8, 16};
    const int *sizes = vec ? sizes_v : sizes_s;
    const int most = chunks > 0 ? chunks : vec ? 64 : 128;
    s.R = 16;
    for (int k = 2; k >= 0; --k)
        if ((rows + sizes[k] - 1) / sizes[k] <= most) s.R = sizes[k];
    s.PC = chunks > 0 ? chunks : (rows + s.R - 1) / s.R;
    s.L = vec ? 8 : 4;
    if (chunks <= 0 && s.PC > most) { // longer lines: tiles
        const int few = (lines + 7) / 8 <= sms;
        s.PC = vec ? 64 : few ? 128 : 32;
        s.L = vec ? 4 : !few ? 8 : (lines + 1) / 2 <= sms && word == 8 ? 2 : 4;
    }
    while (s.L > 1 && s.L * s.PC > MAX_CTA) s.L /= 2;
    s.tiles = (rows + s.R * s.PC - 1) / (s.R * s.PC);
    s.gs = 1;
    while (s.gs * s.gs < s.PC) ++s.gs;
    return s;
}

// Shared-memory values of one sweep's composition: end values and products of the chunks and of the groups.
LSS_HD inline int carry_words(const split &s) { return 2 * s.L * (s.PC + s.groups()); }

// Values of one sweep's table of products (a product and a prefix per chunk, a product per group), for
// `stride` lines.  The stride is the number of lines of that direction alone: with the longer of
// the two, the tables of a grid of 400000 x 8 points would take 350 GB instead of 10 MB.
inline long long carry_table(const split &s, long long stride)
{
    return static_cast<long long>(s.tiles) * (2 * s.PC + s.groups()) * stride;
}

} // namespace wide
} // namespace lss_gb300

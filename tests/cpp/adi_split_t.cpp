// Prints the partition that csrc/adi_split.hpp gives: one line "vec rows lines chunks sms word stride" per query on stdin,
// one line "L PC R gs tiles groups carry_words carry_table" per answer.
#include <cstdio>

#include "adi_split.hpp"

int main()
{
    int vec, rows, lines, chunks, sms, word;
    long long stride;
    while (std::scanf("%d %d %d %d %d %d %lld", &vec, &rows, &lines, &chunks, &sms, &word, &stride) == 7) {
        const lss_gb300::wide::split s = lss_gb300::wide::choose_split(rows, lines, vec != 0, chunks, sms, word);
        std::printf("%d %d %d %d %d %d %d %lld\n", s.L, s.PC, s.R, s.gs, s.tiles, s.groups(), lss_gb300::wide::carry_words(s),
                    lss_gb300::wide::carry_table(s, stride));
    }
    return 0;
}

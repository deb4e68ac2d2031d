// Arrivals at one counter word (csrc/hp_dt_count.h): two calls whose blocks
// interleave in a random order leave the word in some state; the calls that
// follow one after another must each find exactly one last block, the one
// that arrives last.  Prints the number of later calls that did not.
#include <cstdio>
#include <random>

#include "../multiphase-code_b200/csrc/hp_dt_count.h"

int main() {
    std::mt19937 rng(7);
    int wrong = 0, mixed = 0;
    const unsigned sizes[] = {1, 2, 3, 20, 188, 65536};
    for (int trial = 0; trial < 2000; trial++) {
        unsigned long long word = trial % 3 ? 0 : 5, call = 1;
        const unsigned n[2] = {sizes[rng() % 5], sizes[rng() % 5]};
        unsigned left[2] = {n[0], n[1]};
        const unsigned long long id[2] = {call, call + 1};
        call += 2;
        int lasts = 0;
        while (left[0] + left[1]) {   // the overlap
            const int k = left[0] && (!left[1] || (rng() & 1)) ? 0 : 1;
            hp::dt_count_open(&word, id[k]);
            lasts += hp::dt_count_arrive(&word, id[k], n[k]);
            left[k]--;
        }
        mixed += lasts != 2;
        for (int c = 0; c < 3; c++, call += 1 + rng() % 2000) {
            const unsigned b = sizes[rng() % (c == 0 && trial % 50 == 0 ? 6 : 5)];
            int n_last = 0;
            bool at_end = false;
            for (unsigned k = 0; k < b; k++) hp::dt_count_open(&word, call);   // blocks open early,
            for (unsigned k = 0; k < b; k++) {
                if (k % 3 == 0) hp::dt_count_open(&word, call);                // or while others arrive
                at_end = hp::dt_count_arrive(&word, call, b);
                n_last += at_end;
            }
            wrong += n_last != 1 || !at_end;
        }
    }
    std::printf("overlaps that mixed %d, later calls wrong %d\n", mixed, wrong);
    return wrong != 0;
}

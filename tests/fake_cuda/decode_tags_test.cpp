/* The rule of decode_tags.h over several turns of the round counter: launches of one to 32 layers
 * and one to eight tokens, the many of them rare, and in every layer no word but those that it
 * writes itself may carry its tag.  Without the clearing the same launches do find such words. */
#include <cstdio>
#include <cstdint>

#include "decode_tags.h"

static uint64_t state = 1;
static unsigned draw(unsigned n) {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return (unsigned)((state >> 33) % n);
}

static long stale(bool clears, unsigned start, int turns) {
    const int ROWS = 8, PLACES = 6;     /* a row's code word, and places of its list of chains */
    unsigned words[ROWS][PLACES] = {};
    unsigned counter = start;
    long wrong = 0;
    for (int wraps = 0; wraps < turns;) {
        const unsigned kind = draw(1u << 24), before = counter;
        /* one layer and one token nearly always, as a long generation has it (tags of every
         * round), or stacks; more tokens and chains a few times in a turn */
        const int n = kind < (1u << 18) ? 1 + (int)draw(apus::DS_LAYERS) : 1,
                  T = kind < 8 ? 1 + (int)draw(ROWS) : 1;
        unsigned target = counter + apus::DF_ROUND;
        if (clears && apus::stack_clears(target)) {
            for (auto &row : words)
                for (unsigned &w : row) w = 0;
            target += apus::DF_ROUND;
        }
        for (int l = 0; l < n; l++, target += apus::DF_ROUND) {
            if (l) target += apus::DF_ROUND;
            const unsigned tag = clears ? apus::stack_tag(target) : target;
            const int open = kind < 8 ? (int)draw(PLACES) : 0;
            for (int t = 0; t < ROWS; t++)
                for (int p = 0; p < PLACES; p++) wrong += words[t][p] == tag;
            for (int t = 0; t < T; t++)
                for (int p = 0; p <= open; p++) words[t][p] = tag;
        }
        counter = target - apus::DF_ROUND;
        wraps += counter < before;
    }
    return wrong;
}

int main() {
    long with = 0, without = 0;
    const unsigned starts[] = {0u, 0u - 1000u * apus::DF_ROUND, 0u - 512u * apus::DF_ROUND,
                               0u - 3u * apus::DF_ROUND};
    for (unsigned s : starts) with += stale(true, s, 2);
    without = stale(false, 0, 2);
    printf("%ld stale words with the clearing, %ld without\n", with, without);
    return with != 0 || without == 0;
}

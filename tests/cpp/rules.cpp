// Reads questions from stdin, one per line, and prints what rf_rules.h answers.
//   pairs W H S    whether a single pair's level takes two pixels per thread
#include <cstdio>
#include <cstring>

#include "rf_rules.h"

int main() {
    char what[16];
    while (std::scanf("%15s", what) == 1) {
        int w, h, s;
        if (std::strcmp(what, "pairs") == 0 && std::scanf("%d %d %d", &w, &h, &s) == 3)
            std::printf("%d\n", rf::use_pairs(w, h, s));
        else
            return 2;
    }
    return 0;
}

// Reads questions from stdin, one per line, and prints what rf_rules.h answers.
//   pairs W H S    whether a single pair's level takes two pixels per thread
//   tile W H SMS   a level's k_recon_tile (1 .. 4, 0: none) and its blocks
//   conv NPOS SMEM SMS   whether a convolution takes 256 positions per block
#include <cstdio>
#include <cstring>

#include "rf_rules.h"

int main() {
    char what[16];
    while (std::scanf("%15s", what) == 1) {
        int w, h, s;
        long long n;
        unsigned long long m;
        if (std::strcmp(what, "pairs") == 0 && std::scanf("%d %d %d", &w, &h, &s) == 3)
            std::printf("%d\n", rf::use_pairs(w, h, s));
        else if (std::strcmp(what, "tile") == 0 && std::scanf("%d %d %d", &w, &h, &s) == 3) {
            const int rows[5] = {0, 10, 12, 20, 20}, k[5] = {0, 2, 2, 3, 2};
            const int kind = rf::recon_tile_kind(w, h, s);
            std::printf("%d %lld\n", kind,
                        kind ? rf::recon_tile_blocks(w, h, rows[kind], k[kind]) : 0ll);
        } else if (std::strcmp(what, "conv") == 0 && std::scanf("%lld %llu %d", &n, &m, &s) == 3)
            std::printf("%d\n", rf::conv_wide_tile(n, m, s));
        else
            return 2;
    }
    return 0;
}

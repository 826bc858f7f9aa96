// loose_blocks_touched (csrc/fused.cuh) on the host against the same count in 64 bits, over the sizes a call may have.
// Prints the number of mismatches; exit status 0 when there are none.
#include "fused.cuh"

int main() {
    const int sizes[] = {72, 80, 1000, 4096, 32768, 100000, 1 << 20, (1 << 30) - 8, 1 << 30}, lengths[] = {1, 7, 8, 64, 72, 29055, 29056, 32768};
    long long bad = 0;
    for (int qbs : sizes)
        for (int n : lengths)
            for (int lrem0 : {0, 8, qbs / 16 * 8, qbs - 16, qbs - 8})
                bad += mab::loose_blocks_touched(lrem0, n, qbs) != ((int64_t)lrem0 + n + qbs - 1) / qbs;
    printf("block count mismatches %lld\n", bad);
    return bad == 0 ? 0 : 1;
}

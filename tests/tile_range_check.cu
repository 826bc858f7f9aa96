// tiles_of_cta (csrc/fused.cuh) on the host: the ranges follow each other and cover all tiles, and the SMs, each with the CTAs b,
// b + 148 and b + 296, differ by one tile at most.  Prints the number of violations; exit status 0 when there are none.
#include "fused.cuh"

int main() {
    long long bad = 0;
    const int sms = 148;
    for (int total : {1, 2, 147, 148, 149, 444, 445, 500, 600, 700, 1000, 1500, 2368, 3300, 7500, 276000, 1 << 30}) {
        const int ctas = std::min(total, 3 * sms);
        int load[sms] = {}, at = 0;
        for (int b = 0; b < ctas; ++b) {
            const mab::TileRange r = mab::tiles_of_cta(total, ctas, b);
            bad += r.first != at || r.end <= r.first;
            at = r.end;
            load[b % sms] += r.end - r.first;
        }
        bad += at != total;
        bad += *std::max_element(load, load + std::min(ctas, sms)) - *std::min_element(load, load + std::min(ctas, sms)) > 1;
    }
    printf("tile range violations %lld\n", bad);
    return bad == 0 ? 0 : 1;
}

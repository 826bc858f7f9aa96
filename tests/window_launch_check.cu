// plan_tile_launch (csrc/window_launch.cuh) on the host, over windows, tiles and GPUs with 148 SMs and fewer.  Prints the number of violations; exit
// status 0 when there are none.
#include "window_launch.cuh"

int main() {
    const int optin = 227 * 1024;
    long long plans = 0, bad_early = 0, bad_ahead = 0, bad_fit = 0;
    int early_at_148 = 0;
    for (int sms : {16, 37, 74, 132, 148, 160})
        for (int rows : {1, 2, 3, 5, 10, 20, 32, 128})
            for (int max_k = 1; max_k <= 16384 / rows; max_k += max_k < 400 ? 1 : 37)
                for (int tiles : {1, 2, 15, 16, 17, 37, 38, 74, 75, 111, 132, 133, 147, 148, 149, 296, 297, 444, 445, 5000})
                    for (int form = 0; form < 7; ++form) {   // the update with alpha 0, in (0, 1) and -2, fp32 and bf16; the operator
                        const int alpha = form < 6 ? form % 3 : 0;
                        const mab::TileLaunch L = mab::plan_tile_launch(form == 6 ? 1 + (rows & 1) : 0, alpha, form >= 3, rows, max_k, tiles, form != 6, sms, optin);
                        if (L.smem == 0) continue;
                        ++plans;
                        // no more CTAs than an SM holds (228 KB, 1 KB for each of them), which a second, nearly empty wave would follow, and 384
                        // threads only where two CTAs have room
                        const int held = (228 * 1024) / (L.smem + mab::WT_STATIC_BYTES + 1024);
                        bad_fit += L.grid > (int64_t)sms * held || held < 1 || (alpha && L.threads == 384 && L.grid < std::min(tiles, 2 * sms));
                        // the form that starts before kernel A ends stages one tile's rows: a CTA must not get a second one
                        bad_early += L.early && (tiles > L.grid || L.ahead);
                        // rows staged ahead: bf16 alpha forms only, and not without a next tile unless the row loop is the one with two entries
                        bad_ahead += L.ahead && (form < 4 || form > 5 || (tiles <= L.grid && (L.threads != 256 || max_k <= 256 || max_k > 512 || rows < 4)));
                        early_at_148 += L.early && sms == 148 && rows == 10 && max_k == 291 && tiles == 148;
                    }
    for (int sms : {16, 37, 74, 132, 148})                   // the resident form, two CTAs per SM
        for (int tiles = 1; tiles <= 400; ++tiles) {
            const int grid = std::min(tiles, 2 * sms);
            bad_early += mab::early_form(tiles, grid, sms) && tiles > grid;
        }
    // what kernel A may let start early with up to a CTA per SM: tile and resident forms with a tile per CTA, neither the wide form (20 rows of 5 %) nor
    // one CTA of 1024 threads per SM
    const int dbs = 29056;
    bool form_ok = true;
    for (int sms : {74, 132, 148})
        for (int tiles : {sms / 2, sms, sms + 1}) {
            const bool one = tiles <= sms;
            form_ok = form_ok && mab::update_is_early(tiles, 10, 291, dbs, true, 0, sms, optin) == one;
            form_ok = form_ok && mab::update_is_early(tiles, 10, 291, dbs, false, 0, sms, optin) == one;
            form_ok = form_ok && mab::update_is_early(tiles, 10, 291, dbs, true, 1, sms, optin) == one;
            for (bool bf16 : {false, true}) {
                form_ok = form_ok && !mab::update_is_early(tiles, 20, 1453, dbs, bf16, 0, sms, optin) && !mab::update_is_early(tiles, 5, 14528, dbs, bf16, 1, sms, optin);
                form_ok = form_ok && !mab::update_is_early(tiles, 10, 1453, dbs, bf16, 0, sms, optin);
            }
        }
    printf("plans %lld, early forms with more tiles than CTAs %lld, rows ahead of nothing %lld, CTAs without room %lld, what may start early %s\n", plans, bad_early, bad_ahead, bad_fit, form_ok ? "right" : "wrong");
    return form_ok && bad_ahead == 0 && bad_fit == 0 && plans > 100000 && early_at_148 == 6 && bad_early == 0 ? 0 : 1;
}

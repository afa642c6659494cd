/* sor_box_host.cu -- TEST INFRASTRUCTURE: the linear box solver's enumeration
 * of a colour's nodes (csrc/sor_box.h) compiled as host code, against plain
 * 64-bit division.  Built by tests/test_sor_box_host.py with nvcc into a
 * temporary folder. */
#include "sor_box.h"

using namespace espic;

extern "C" int sor_host_short(int ni, int nj, int nk) { return sor_short_indices(Geo{ni, nj, nk}); }

/* entries first, first + step, ... of both colours that the solver's route
 * places elsewhere than plain division does */
extern "C" int64_t sor_host_misplaced(int ni, int nj, int nk, int64_t first, int64_t step) {
    const Geo g{ni, nj, nk};
    const bool brief = sor_short_indices(g);
    const int64_t hx = (ni - 1) / 2, count = hx * (nj - 2) * (nk - 2);
    int64_t bad = 0;
    for (int64_t t = first; t < count; t += step)
        for (int c = 0; c < 2; c++) {
            const int64_t k = 1 + t / hx / (nj - 2), j = 1 + t / hx % (nj - 2);
            const int64_t i = 1 + 2 * (t % hx) + ((1 + j + k + c) & 1);
            const int64_t want = i <= ni - 2 ? (k * nj + j) * ni + i : -1;
            int64_t got = -1;
            if (brief) {
                int32_t u;
                if (sor_entry(g, (uint32_t)hx, (uint32_t)t, c, u)) got = u;
            } else {
                sor_entry(g, (uint64_t)hx, (uint64_t)t, c, got);
            }
            bad += got != want;
        }
    return bad;
}

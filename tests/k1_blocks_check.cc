// CPU check of K1's cut of a case's radii into blocks (lmie_b200/csrc/k1_blocks.h):
// every radius is in exactly one block, in order; a block has at most `most`
// radii; and their shared-memory rows never add up to more than the block is
// laid out for, for radii that descend, ascend, rise and fall, or are in no
// order.  Radii from the largest down get the blocks that the first one's rows
// give.  Prints "ok" or the failed check.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "k1_blocks.h"

namespace {

// the truncation and its shared-memory rows (mie_radius.cuh, MIE_B = 4)
int rows_of(double x) { return ((int) (x + 4.05 * std::pow(x, 1. / 3.) + 8) + 8) & ~3; }

int check(const std::vector<int> &need, int rows, int most, bool falling) {
    int at = 0, bad = 0;
    const int nb = k1_cut((int) need.size(), rows, most, [&](int i) { return need[i]; }, [&](int i, int n) {
        long long sum = 0;
        for (int k = i; k < i + n && k < (int) need.size(); ++k) sum += need[k];
        if (i != at || n < 1 || n > most || i + n > (int) need.size()) bad |= 1;
        if (sum > rows) bad |= 2;
        if (falling && n != std::min(std::min(most, (int) need.size() - i), std::max(1, rows / need[i]))) bad |= 4;
        at = i + n;
    });
    if (at != (int) need.size() || nb < (int) (need.size() + most - 1) / most) bad |= 8;
    return bad;
}

}  // namespace

int main() {
    std::mt19937 gen(7);
    for (int nr : {1, 2, 31, 300, 800})
        for (double top : {3., 20., 60., 400., 900.})
            for (int most : {1, 4, 7, 32}) {
                std::vector<int> up(nr);
                for (int i = 0; i < nr; ++i) up[i] = rows_of(.01 + top * (i + 1.) / nr);
                const int rows = std::max(up.back(), 1500);
                std::vector<int> down(up.rbegin(), up.rend()), wave(up), mixed(up);
                // (largest in the middle, smallest in the middle, no order)
                for (int i = 0; i < nr; ++i) wave[i] = i < nr / 2 ? up[2 * i] : down[std::min(nr - 1, 2 * (i - nr / 2))];
                std::vector<int> valley(wave.rbegin() + nr / 2, wave.rend());
                valley.insert(valley.end(), wave.begin(), wave.begin() + nr / 2);
                std::shuffle(mixed.begin(), mixed.end(), gen);
                const std::vector<int> *all[] = {&down, &up, &wave, &valley, &mixed};
                for (int q = 0; q < 5; ++q) {
                    const int bad = check(*all[q], rows, most, q == 0);
                    if (bad) {
                        printf("order %d: %d radii to x = %g, %d a block: failure %d\n", q, nr, top, most, bad);
                        return 1;
                    }
                }
            }
    printf("ok\n");
    return 0;
}

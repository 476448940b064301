// k1_blocks.h -- how K1's blocks of several radii (mie_radius.cuh) take the
// radii of one case: a block's shared memory is laid out for a fixed number of
// rows, so its radii's rows must not add up to more.  The host layer refuses
// radii of more orders than r2 has, so the orders of the radii it accepts ascend;
// the cut does not lean on that.  Host code without CUDA, so that the rule can be
// checked by itself.
#pragma once

// Cuts radii 0 .. nr - 1 of a case, radius i needing rows_of(i) <= rows rows,
// into blocks of at most `most` neighbours: put(i, n) per block, radii i ..
// i + n - 1.  A block's radii number at most rows over the rows of its longest
// one, which for radii from the largest down is known from the first.  Returns
// the number of blocks.
template <class Rows, class Put>
inline int k1_cut(int nr, int rows, int most, Rows &&rows_of, Put &&put) {
    int nb = 0;
    for (int i = 0; i < nr; ++nb) {
        int longest = rows_of(i), fit = rows / longest, n = 1;
        if (fit > most) fit = most;
        if (fit > nr - i) fit = nr - i;
        for (; n < fit; ++n) {
            const int next = rows_of(i + n);
            if (next > longest) {
                longest = next;
                if (fit > rows / longest) fit = rows / longest;
                if (n >= fit) break;
            }
        }
        put(i, n);
        i += n;
    }
    return nb;
}

// tm_generic_forms.h -- which form of the run-time-length column pass a height takes
// (host code without CUDA; the kernels are in tm_generic.cuh).
#pragma once
#include <stddef.h>

namespace tmk {

constexpr size_t kBlockSharedLimit = 232448;   // bytes of shared memory a block can have, static and dynamic

// Shared memory of k_pass_b_gen2 with `pairs` pairs of columns (16 bytes per element of a pair):
// two buffers | the twiddle table (tab) | the next orientation's rows of A (staged).
constexpr size_t gen_pass_b_smem(int pairs, int T, int Y, bool tab, bool staged) {
    return (size_t)32 * pairs * Y + (tab ? 8 * (size_t)(Y + Y % 2) : 0) + (staged ? (size_t)16 * pairs * T : 0);
}

struct GenColForm {
    int pairs;           // pairs of columns per block; 0: one column (k_pass_b_gen)
    bool tab, staged;
    size_t smem;
    int columns() const { return pairs ? 2 * pairs : 1; }
};

// As many columns as fit, with the table and the staged rows where they fit too: few warps wait for the
// loads that these hide.  Only where nothing else lets a pair of columns in are the rows of A read when they
// are needed (a 256 template: heights from 7137 to 7264; 256 x 7200, 32 orientations of 2700 columns: 5.9 ms,
// 11.3 with one column per block and 12.1 with two that are not pairs).
inline GenColForm gen_col_form(int T, int Y) {
    for (int pairs = 2; pairs >= 1; pairs--)
        for (int tab = 1; tab >= 0; tab--) {
            const size_t smem = gen_pass_b_smem(pairs, T, Y, tab, true);
            if (smem <= kBlockSharedLimit) return {pairs, tab != 0, true, smem};
        }
    const size_t smem = gen_pass_b_smem(1, T, Y, false, false);
    if (smem <= kBlockSharedLimit) return {1, false, false, smem};
    return {0, false, false, (size_t)16 * Y};
}

}  // namespace tmk

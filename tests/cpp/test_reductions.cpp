// Sizes of the FP64 hop's grid reductions (hila_b200/csrc/hop_shapes.h): the partial sums of
// every launch shape fit the buffer reserved for it, at every lattice size.  No GPU involved.
#include <cstdio>

#include "hop_shapes.h"

using namespace hw;

int main() {
    int failures = 0;
    // sites per parity: the smallest, around the rule for small lattices, 48^3 x 96, 64^4, 96^4
    const long sizes[] = {8, 31, 32, 33, 9240, kHopSplitSites, kHopSplitSites + 1, 48L * 48 * 48 * 96 / 2,
                          64L * 64 * 64 * 64 / 2, 96L * 96 * 96 * 96 / 2};
    for (long Vh : sizes)
        for (int v = 0; v < kHopVariants; v++) {
            const long nb = hop_blocks(v, Vh);
            const bool covers = nb * hop_sites(v) >= Vh && (nb - 1) * hop_sites(v) < Vh;
            // the explicit residual sums two values per block of the hop, the start of a solve two
            // per 256 sites
            const size_t most = 2 * (size_t)nb, init = 2 * (size_t)((Vh + 255) / 256);
            if (!covers || most > red_doubles(nb) || init > red_doubles(nb)) {
                std::printf("FAILED: shape %d at %ld sites per parity\n", v, Vh);
                failures++;
            }
        }
    // the capacity of blocks of 128 sites does not hold shape 3's sums at 48^3 x 96
    const long big = 48L * 48 * 48 * 96 / 2;
    if (!(2 * (size_t)hop_blocks(3, big) == 331776 && red_doubles(hop_blocks(3, big)) >= 331776)) failures++;
    if (failures == 0) std::printf("reduction sizes passed\n");
    return failures;
}

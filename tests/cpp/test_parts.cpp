// How the engine divides its tiles' slots over blocks (hila_b200/csrc/engine_parts.h): every slot
// in exactly one part, no part empty, nothing divided where it cannot help.  No GPU involved.
#include <cstdio>
#include <initializer_list>

#include "engine_parts.h"

using namespace hw;

static int failures = 0;
#define CHECK(c)                                                       \
    do {                                                               \
        if (!(c)) {                                                    \
            std::printf("FAILED line %d: %s\n", __LINE__, #c);         \
            failures++;                                                \
        }                                                              \
    } while (0)

int main() {
    const int max_parts = 16;
    for (int unit : {1, 2})
        for (int n = 1; n <= 16; n++)
            for (int parts = 1; parts <= max_parts; parts++) {
                const int count = part_count(n, parts, unit), per = part_slots(n, parts, unit);
                CHECK(count >= 1 && count <= parts && per % unit == 0);
                CHECK((count - 1) * per < n && count * per >= n);  // the parts with slots cover them
                // fewer active slots than the lattice holds stay within the same parts
                for (int na = 1; na < n; na++) CHECK(parts * part_slots(na, parts, unit) >= na);
            }
    CHECK(part_count(0, 16, 1) == 0 && part_slots(0, 16, 1) == 0);
    const PartsShape low{888, 1, 1, kPartsOverheadF32}, pk{444, 2, 1, kPartsOverheadPair},
        stag{444, 2, 2, kPartsOverheadPair};
    for (const PartsShape &S : {low, pk, stag})
        for (int nt : {1, 16, 81, 256, 512, 625, 887, 888, 945, 1296, 4096}) {
            // slots that fill one unit are never divided, nor is any lattice from two tiles per block on
            for (int n = 0; n <= S.unit; n++) {
                const PartsLattice one{nt, n};
                CHECK(choose_parts(&one, 1, S, max_parts) == 1);
            }
            for (int n = 1; n <= 16; n++) {
                const PartsLattice one{nt, n};
                const int parts = choose_parts(&one, 1, S, max_parts);
                CHECK(parts >= 1 && part_count(n, parts, S.unit) == parts);
                if (nt >= 2 * S.blocks) CHECK(parts == 1);
                CHECK(parts_time(&one, 1, S, parts) <= parts_time(&one, 1, S, 1));
            }
        }
    // few tiles: a part per unit; a ragged second wave: divided; one that is not helped: whole tiles
    const PartsLattice small{16, 12}, ragged{945, 6}, whole{625, 3};
    CHECK(choose_parts(&small, 1, low, max_parts) == 12 && choose_parts(&small, 1, pk, max_parts) == 6);
    CHECK(choose_parts(&ragged, 1, low, max_parts) > 1 && choose_parts(&whole, 1, low, max_parts) == 1);
    // a lattice with one slot beside one with twelve, and one without any
    const PartsLattice mixed[] = {{256, 12}, {16, 1}, {64, 0}};
    CHECK(choose_parts(mixed, 3, low, max_parts) == 8);
    const PartsLattice light[] = {{256, 2}, {16, 1}};  // no more parts than the fullest has units
    CHECK(choose_parts(light, 2, low, max_parts) == 2 && choose_parts(light, 2, pk, max_parts) == 1);
    CHECK(choose_parts(mixed, 0, low, max_parts) == 1);
    if (failures == 0) std::printf("parts passed\n");
    return failures;
}

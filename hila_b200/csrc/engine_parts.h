// How a hop phase of the engine divides its tiles' slots over blocks (no CUDA types: a CPU test
// drives it).
//
// A work item is a tile of a lattice and a part of the lattice's slots.  With whole tiles as
// items a launch of few tiles leaves blocks idle, or has a ragged second wave, while each block
// goes through all slots of its tile; with more parts the links and neighbours of a site are
// fetched by several blocks.  choose_parts() tries the numbers of parts that the slots fill on the
// launch's own lattices, and keeps the one whose items the blocks finish first, each block taking
// the next item when it is free.
//
// Microseconds per iteration, undivided -> divided so (12-real FP64 links, one lattice): FP32 with
// 3 and 6 sources, 16^4 131 -> 107, 230 -> 162, 20x12x28x36 (945 tiles for 888 blocks) 312 -> 272,
// 570 -> 472; FP16 with 12, 8^4 379 -> 128, 16^4 361 -> 286; staggered FP16 with 12, 8^4 170 -> 112.
// A division into powers of two that did not look at the slots was slower wherever they did not
// fill its parts: 20^4 FP16 with 1 source 103-159 against 89, FP32 with 1 104 against 77 and with
// 3 199 against 184, staggered FP16 12^4 with 1 74 against 52 and 18^4 with 8 225 against 162.
#pragma once

namespace hw {

// what an item costs, in quarters of the time that one unit of slots takes; its links, neighbours
// and barriers (FP16 links are staged in shared memory): of 1, 2, 3, 4 and 6 quarters the ones
// with the fewest slower cases over 8^4 to 24^4 and 1 to 12 sources
constexpr int kPartsUnitCost = 4;
constexpr int kPartsOverheadF32 = 1, kPartsOverheadF16 = 3, kPartsOverheadPair = 4;
constexpr int kPartsEmptyCost = 1;  // an item without slots
constexpr int kPartsGroups = 16;    // in which a lattice's uneven parts alternate (parts_time)

struct PartsLattice {
    int ntiles;
    int nslots;  // 0: the phase has nothing to do on it
};

// how the launch's blocks work through an item
struct PartsShape {
    int blocks;
    int unit;      // slots that a thread serves together
    int teams;     // units that a block serves at a time
    int overhead;  // of an item (kPartsOverhead*)
};

// slots of a part (the last part may have fewer)
constexpr int part_slots(int nslots, int parts, int unit) {
    return ((nslots + parts - 1) / parts + unit - 1) / unit * unit;
}
// parts that hold slots
constexpr int part_count(int nslots, int parts, int unit) {
    return nslots <= 0 ? 0 : (nslots + part_slots(nslots, parts, unit) - 1) / part_slots(nslots, parts, unit);
}

// whether every part of every lattice holds as many slots
inline bool parts_even(const PartsLattice *lat, int nlat, const PartsShape &S, int parts) {
    for (int l = 0; l < nlat; l++) {
        const int n = (lat[l].nslots + S.unit - 1) / S.unit * S.unit;
        if (n != parts * part_slots(lat[l].nslots, parts, S.unit)) return false;
    }
    return true;
}

// When the launch ends: the mean of two reckonings, as the truth lies between them.  One takes the
// items in turn by the next free block, each at its full cost (whole waves); the other lets the
// last, partly filled wave run faster (the work spread over all blocks and half an item).  A launch
// of one wave ends with its longest item.  Times are below kPartsTimes for up to two tiles per
// block of up to 16 slots (a tile costs up to 16 x (kPartsUnitCost + overhead)).  Takes some
// microseconds on the host.
constexpr int kPartsTimes = 512;
inline double parts_time(const PartsLattice *lat, int nlat, const PartsShape &S, int parts) {
    long free_at[kPartsTimes] = {S.blocks};  // blocks that become free then
    long now = 0, end = 0, items = 0, work = 0, longest = 0;
    auto run = [&](long n, int slots) {
        const int units = (slots + S.unit - 1) / S.unit;
        const long cost = slots ? (long)(units + S.teams - 1) / S.teams * kPartsUnitCost + S.overhead : kPartsEmptyCost;
        items += n;
        work += n * cost;
        if (n > 0 && cost > longest) longest = cost;
        while (n > 0) {
            while (now < kPartsTimes && free_at[now] == 0) now++;
            if (now + cost >= kPartsTimes) {
                end = kPartsTimes;
                return;
            }
            const long k = free_at[now] < n ? free_at[now] : n;
            free_at[now] -= k;
            free_at[now + cost] += k;
            if (now + cost > end) end = now + cost;
            n -= k;
        }
    };
    for (int l = 0; l < nlat; l++) {
        const int n = lat[l].nslots, count = part_count(n, parts, S.unit);
        const int per = n > 0 ? part_slots(n, parts, S.unit) : 0;
        // a tile's parts follow one another: uneven ones alternate, here in groups of tiles
        const int groups = count * per == n && count == parts ? 1 : kPartsGroups;
        for (int g = 0; g < groups; g++) {
            const long nt = (long)lat[l].ntiles * (g + 1) / groups - (long)lat[l].ntiles * g / groups;
            if (count > 1) run(nt * (count - 1), per);
            if (count > 0) run(nt, n - (count - 1) * per);
            run(nt * (parts - count), 0);
        }
    }
    return items <= S.blocks ? (double)end : 0.5 * (end + (double)work / S.blocks + 0.5 * longest);
}

// The number of parts for a launch: the fewest that end it first, but within one wave the most
// (they reach more SMs).  From two tiles per block on, tiles are not divided (32^4, 12 sources:
// as fast or faster).  Where lattices differ in their slots, light items fill the gaps that heavy
// ones leave, and the reckoning is off: there the parts double until the launch has two items per
// block or the fullest lattice has no more units (a stream of four lattices with 4 to 13 sources,
// 928 tiles: 53.1 ms undivided, 46.8 so, 47.1 to 48.2 by the reckoning).
inline int choose_parts(const PartsLattice *lat, int nlat, const PartsShape &S, int max_parts) {
    long ntiles = 0;
    int most = 0;
    bool alike = true;
    for (int l = 0; l < nlat; l++) {
        ntiles += lat[l].ntiles;
        if (lat[l].nslots == 0) continue;
        if (most > 0 && lat[l].nslots != most) alike = false;
        if (lat[l].nslots > most) most = lat[l].nslots;
    }
    if (ntiles >= 2L * S.blocks) return 1;
    int best = 1;
    if (!alike) {
        while (ntiles * best < 2L * S.blocks && best * S.unit < most && 2 * best <= max_parts) best *= 2;
        return best;
    }
    double best_time = parts_time(lat, nlat, S, 1);
    for (int parts = 2; parts <= max_parts; parts++) {
        if (part_count(most, parts, S.unit) != parts) continue;
        const double t = parts_time(lat, nlat, S, parts);
        if (t < best_time || (t == best_time && ntiles * parts <= S.blocks)) best = parts, best_time = t;
    }
    return best;
}

}  // namespace hw

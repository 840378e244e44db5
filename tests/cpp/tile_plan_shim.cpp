// A host build of the large chunks' sizes and choice of render (tile_plan.h)
// for tests/test_tile_plan_cpu.py: the functions the library itself uses.
#include "tile_plan.h"

using namespace dmann;

extern "C" {
long long pairs_bound(long long n, int nside) { return (long long)tile_pairs_bound(n, nside); }
long long capacity(long long n, int nside) { return (long long)tile_capacity(n, nside); }
long long slots(long long n, int nside, long long list) { return (long long)tile_slots(n, nside, list); }
int always_fits(long long n, int nside) { return tile_always_fits(n, nside, tile_capacity(n, nside)); }
// bit 0 tiles, 1 segments, 2 the pair count
int plan(int have_tile, int fits, int have_seg) {
    const LargePlan p = plan_large(have_tile, fits, have_seg);
    return p.tile | p.seg << 1 | p.count << 2;
}
int mode(long long est, long long min_est, long long blocks, long long pairs, long long pair_cap, long long items,
         long long item_cap) {
    return large_mode(est, min_est, blocks, pairs, pair_cap, items, item_cap);
}
int cls(int oct, int omax, int omin) { return tile_class(oct, omax, omin); }
int unit_len(long long pairs) { return tile_unit_len(pairs); }
long long units_of(long long pairs, long long nt) { return tile_units_of(pairs, nt); }
long long unit_capacity(long long slots, int nside) { return (long long)tile_unit_capacity(slots, nside); }
int unit_max() { return kUnitMax; }
}

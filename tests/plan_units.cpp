// Host side of the work-unit tables: prints what the library's scheduling functions
// give, for test_plan_units.py.  No GPU.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../chime-x_b200/csrc/chimex_internal.h"

using namespace chx;

// costs TILE E T: the cost and the number of x tiles of every unit of one channel.
static int costs(int tile, int E, int T) {
    std::vector<Unit> u;
    tc_append_tile_units(tile, u, 0, E, 0, T, 1, 0);
    for (const Unit &x : u) printf("%d %d\n", x.cost, (x.tyx >> 20) & 3);
    return 0;
}

int main(int argc, char **argv) {
    auto arg = [&](int i) { return i < argc ? atoi(argv[i]) : 0; };
    if (argc > 1 && !strcmp(argv[1], "costs")) return costs(arg(2), arg(3), arg(4));
    return 2;
}

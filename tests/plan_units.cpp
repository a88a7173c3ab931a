// Host side of the work-unit tables: prints what the library's scheduling functions
// give, for test_plan_units.py.  No GPU.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <chrono>

#include "../chime-x_b200/csrc/chimex_internal.h"

using namespace chx;

// costs TILE E T: the cost and the number of x tiles of every unit of one channel.
static int costs(int tile, int E, int T) {
    std::vector<Unit> u;
    tc_append_tile_units(tile, u, 0, E, 0, T, 1, 0);
    for (const Unit &x : u) printf("%d %d\n", x.cost, (x.tyx >> 20) & 3);
    return 0;
}

// inverse: budgets at which unit_stages is not the inverse of unit_cost.
static int inverse() {
    for (int tile = 1; tile <= kTileSmall; tile++)
        for (int nx = 1; nx <= 2; nx++)
            for (int budget = 0, n = 0; budget < 200000; budget++) {
                while (unit_cost(tile, 0, (n + 1) * kUnitStageSamples, nx) <= budget) n++;
                if (unit_stages(tile, budget, nx) != n) printf("%d %d %d\n", tile, nx, budget);
            }
    return 0;
}

// The units of a plan whose options are unset, storing (add = 0) or adding.
static bool plan_table(int E, int F, int T, int add, std::vector<Unit> &u, std::vector<int> &off) {
    const int sms = 148, tile = tc_launch_tile(tc_default_tile(E), E);
    const int slots = tc_tile_slots(tile, sms);
    const long long zeroing = add ? 0 : tc_zeroing_cost(F * num_blocks_of(E) * 8192);
    const TcShape s = tc_choose_shape(
        tile, 0, sms, zeroing,
        [&](TcShape k, std::vector<int> &costs) { tc_append_costs(k, E, T, F, costs); });
    if (s.span > 0) {
        for (int f = 0; f < F; f++) tc_append_tile_units(tile, u, f, E, 0, T, 1, 0);
        if (tc_balance(s, tile, zeroing, u, slots, off)) return true;
        u.clear();
    }
    for (int f = 0; f < F; f++) tc_append_tile_units(s.tile, u, f, E, 0, T, s.split, 0);
    tc_schedule(u, (int)std::min(u.size(), (size_t)slots), off);
    return false;
}

// table E F T ADD: whether it is balanced; then every unit's channel, tyx, range, split
// flag and CTA.
static int table(int E, int F, int T, int add) {
    std::vector<Unit> u;
    std::vector<int> off;
    printf("%d\n", plan_table(E, F, T, add, u, off) ? 1 : 0);
    for (size_t b = 0; b + 1 < off.size(); b++)
        for (int i = off[b]; i < off[b + 1]; i++)
            printf("%d %d %d %d %d %zu\n", u[i].chan, u[i].tyx, u[i].t0, u[i].t1, u[i].split, b);
    return 0;
}

// times E F T: us for both tables of a plan, and for scheduling its units with each of
// one to eight equal ranges.
static int times(int E, int F, int T) {
    const int tile = tc_launch_tile(tc_default_tile(E), E), slots = tc_tile_slots(tile, 148);
    auto shortest = [](auto work) {
        double best = 1e30;
        for (int i = 0; i < 200; i++) {
            const auto t = std::chrono::steady_clock::now();
            work();
            best = std::min(best, std::chrono::duration<double, std::micro>(
                                      std::chrono::steady_clock::now() - t).count());
        }
        return best;
    };
    const double both = shortest([&] {
        for (int add = 0; add < 2; add++) {
            std::vector<Unit> u;
            std::vector<int> off;
            plan_table(E, F, T, add, u, off);
        }
    });
    const double equal = shortest([&] {
        for (int k = 1; k <= 8; k++) {
            std::vector<Unit> u;
            std::vector<int> off;
            for (int f = 0; f < F; f++) tc_append_tile_units(tile, u, f, E, 0, T, k, 0);
            tc_schedule(u, (int)std::min(u.size(), (size_t)slots), off);
        }
    });
    printf("%f %f\n", both, equal);
    return 0;
}

// sums VBLOCKS NGROUPS SMS: warps and CTAs of the offset sums.
static int sums(int vblocks, int ngroups, int sms) {
    const OffsetSplit s = offset_split(vblocks, ngroups, sms);
    printf("%d %lld\n", s.warps, (long long)s.ctas);
    return 0;
}

// rows T: operand rows of a small launch whose longest unit has T samples.
static int rows(int T) {
    printf("%d\n", small_two_rows(T) ? 2 : 3);
    return 0;
}

int main(int argc, char **argv) {
    auto arg = [&](int i) { return i < argc ? atoi(argv[i]) : 0; };
    if (argc > 1 && !strcmp(argv[1], "costs")) return costs(arg(2), arg(3), arg(4));
    if (argc > 1 && !strcmp(argv[1], "inverse")) return inverse();
    if (argc > 1 && !strcmp(argv[1], "table")) return table(arg(2), arg(3), arg(4), arg(5));
    if (argc > 1 && !strcmp(argv[1], "times")) return times(arg(2), arg(3), arg(4));
    if (argc > 1 && !strcmp(argv[1], "sums")) return sums(arg(2), arg(3), arg(4));
    if (argc > 1 && !strcmp(argv[1], "rows")) return rows(arg(2));
    return 2;
}

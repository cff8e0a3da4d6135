// Host check of the triangle-dimer schedule (csrc/rt_tdschedule.h): moves in
// random order, made with every refresh of the reference's phase program and
// made with TdSchedule's, must leave the same eight arrays, whatever the
// start.  Both run on the integer rule (csrc/rt_tridimer.cuh).
//
//   tdschedule_check M ROUNDS MOVES   (random states and moves; the flushes
//       fall after random moves, as launches that continue a walk cut it)
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

namespace rtb {
// Host stand-ins for the walk kernel's argument block and phase-descriptor
// accessors, which the rule's walk-kernel glue names.
struct WalkArgs {
    int n, wpad;
};
inline uint32_t ph_op(uint32_t d) { return d & 0xffu; }
inline uint32_t ph_a(uint32_t d) { return (d >> 8) & 0xffu; }
inline uint32_t ph_b(uint32_t d) { return (d >> 16) & 0xffu; }
}  // namespace rtb

#include "rt_tdplane.cuh"
#include "rt_tdschedule.h"
#include "rt_tridimer.cuh"

using namespace rtb;

namespace {

uint64_t mix(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t x = a * 0x9E3779B97F4A7C15ull ^ (b + 0x632BE59BD9B4E019ull) * 0xBF58476D1CE4E5B9ull ^ c * 0x94D049BB133111EBull;
    x ^= x >> 31;
    x *= 0xD6E8FEB86659FD93ull;
    return x ^ (x >> 32);
}

struct State {
    int m;
    std::vector<int32_t> a;
    uint64_t draw = 0;  // number of the drawing move
    long phases = 0;
    void run(uint32_t op, uint32_t p, uint32_t q, bool draws) {
        TriDimerRule::Ctx x;
        x.base = a.data();
        x.plane = m * m;
        x.w = m;
        x.m = m;
        x.row0 = 0;
        x.op = op;
        x.a = p;
        x.b = q;
        // as the kernels do: every site from the state before the phase (a phase
        // reads no site it writes)
        for (int i = 0; i < m; ++i)
            for (int j = 0; j < m; ++j)
                TriDimerRule::site_on(x, i, j, draws ? (uint32_t)(mix(7, draw, (uint64_t)(i * m + j)) >> 9) & 0x7fffffu : 0u);
        ++phases;
    }
};

}  // namespace

int main(int argc, char** argv) {
    if (argc != 4) return 2;
    const int m = atoi(argv[1]), rounds = atoi(argv[2]), moves = atoi(argv[3]);
    long full_phases = 0, lazy_phases = 0, flips = 0;
    for (int r = 0; r < rounds; ++r) {
        State full{m, std::vector<int32_t>((size_t)8 * m * m)};
        for (int arr = 0; arr < 8; ++arr)
            for (int e = 0; e < m * m; ++e) {
                // random bits, with the states that flip mixed in
                const uint64_t h = mix(r + 1, arr, e);
                int32_t v = (int32_t)(h >> 20) & ((1 << tdp::cover_bits_of(arr)) - 1);
                if (h & 3) v = arr < 3 ? (h & 4 ? 5 : 10) : arr < 5 ? (h & 4 ? 45 : 54) : (h & 4 ? 85 : 170);
                full.a[(size_t)arr * m * m + e] = v;
            }
        State lazy = full;
        TdSchedule td;
        auto emit = [&](uint32_t op, uint32_t a, uint32_t b, bool draws) { lazy.run(op, a, b, draws); };
        for (int s = 0; s < moves; ++s) {
            const uint64_t h = mix(1000 + r, s, 5);
            const uint32_t kind = h % 3, r1 = (h >> 8) % 3, r2 = (h >> 16) & 1, p1 = (h >> 24) % 3, p2 = (h >> 32) & 1;
            full.draw = lazy.draw = (uint64_t)r * moves + s;
            const std::vector<int32_t> before = full.a;
            if (kind == 0) {
                full.run(TD_ROT_LOZ, r1, r2, true);
                full.run(TD_LOZ_FLIPPED, r1, r2, false);
                full.run(TD_LOZ_OTHER, r1, 0, false);
                full.run(TD_UP_FROM_LOZ, 0, 0, false);
                full.run(TD_TRI_OTHER, 0, 7, false);
                td.lozenges(r1, r2, emit);
            } else if (kind == 1) {
                full.run(TD_ROT_TRI, r2, r1, true);
                full.run(TD_TRI_FLIPPED, r2, r1, false);
                full.run(TD_TRI_OTHER, r2, 0, false);
                full.run(TD_LOZ_FROM_TRI, 0, 0, false);
                full.run(TD_BFLY_FROM_LOZ, 0, 7, false);
                td.triangles(r2, r1, emit);
            } else {
                full.run(TD_ROT_BFLY, r1, p1 | (p2 << 2), true);
                full.run(TD_BFLY_SAME, r1, p1 | (p2 << 2), false);
                full.run(TD_BFLY_21, r1, p1, false);
                full.run(TD_BFLY_22, r1, p1, false);
                full.run(TD_BFLY_23_LOZ, r1, p1, false);
                full.run(TD_BFLY_FROM_LOZ, 1, 7u & ~(1u << r1), false);
                full.run(TD_TRI_OTHER, 0, 0, false);
                td.butterflies(r1, p1, p2, emit);
            }
            for (size_t e = 0; e < before.size(); ++e) flips += before[e] != full.a[e];
            if ((h >> 40) % 5 == 0 || s + 1 == moves) {
                td.flush(emit);
                for (size_t e = 0; e < full.a.size(); ++e)
                    if (full.a[e] != lazy.a[e]) {
                        printf("MISMATCH round %d move %d array %zu site %zu: %d, schedule %d\n", r, s,
                               e / ((size_t)m * m), e % ((size_t)m * m), full.a[e], lazy.a[e]);
                        return 1;
                    }
            }
        }
        full_phases += full.phases;
        lazy_phases += lazy.phases;
    }
    // the fast mode's sweep
    TdSchedule td;
    int sweep = 0;
    auto count = [&](uint32_t, uint32_t, uint32_t, bool) { ++sweep; };
    for (uint32_t mv = 0; mv < 30; ++mv) td_fast_move(td, mv, count);
    sweep = 0;
    for (uint32_t mv = 0; mv < 30; ++mv) td_fast_move(td, mv, count);
    printf("ok %ld phases, schedule %ld, values changed %ld, sweep %d\n", full_phases, lazy_phases, flips, sweep);
    return 0;
}

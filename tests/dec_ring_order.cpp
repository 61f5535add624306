// Plays the decode attention's ring of stages (csrc/dec_ring.h) through without a GPU: the warps of a block, each with its list of steps
// as attn_dec4_kernel takes them, run in a random order, copies land at random times, and barriers are modelled by their phases. Counts what goes
// wrong: a stage read before it is there or after another took its place, a slot armed twice or over a stage that is still wanted,
// a copy into the merge's slots, warps that wait for ever. `look` = 0 leaves out the look at a slot's number.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "dec_ring.h"

struct Op { enum { LOOK, WAIT, ARM, BAR, COPY, READ, MERGE } what; int slot, number, x; };  // x: parity, barrier's threads, on / off
struct Slot { int done = 0, landed = 0, holds = -1, unread = 0, asked = 0; bool armed = false, full = false; };
struct Bar { int here = 0, round = 0; };

template <int QUADS, int NSTG, int OFF>
int play(std::mt19937& rng, bool look) {
    using Ring = qb::DecRing<QUADS, NSTG, OFF>;
    constexpr int WARPS = 4 * QUADS;
    std::vector<int> lens(OFF ? 1 + rng() % 6 : 1);
    for (int& n : lens) n = 1 + rng() % 22;
    std::vector<std::vector<Op>> ops(WARPS);
    std::vector<bool> fresh(lens.size());
    for (size_t i = 0; i < lens.size(); i++) fresh[i] = i == 0 || rng() % 2;
    for (int w = 0; w < WARPS; w++) {
        auto& o = ops[w];
        Ring r;
        const int quad = w >> 2, lane4 = w & 3;
        auto arm = [&](int j) { o.push_back({Op::ARM, Ring::slot(j), r.number(j), 0}); };
        auto copy = [&](int j) { o.push_back({Op::COPY, Ring::slot(j), r.number(j), 0}); };
        auto bar = [&](int id, int n) { o.push_back({Op::BAR, id, 0, n}); };
        const int begin = lens[0] < NSTG ? lens[0] : NSTG;
        if (w < begin) arm(w);
        bar(1, WARPS);
        for (int x = w; x < 4 * begin; x += WARPS) copy(x >> 2);
        for (size_t s = 0; s < lens.size(); s++) {
            const int n = lens[s];
            if (fresh[s]) { bar(1, WARPS); bar(1, WARPS); }
            for (int j = quad; j < n; j += QUADS) {
                if (look && Ring::looks(j)) o.push_back({Op::LOOK, Ring::slot(j), r.number(j), 0});
                o.push_back({Op::WAIT, Ring::slot(j), 0, (int)r.parity(j)});
                const int refill = Ring::in_the_middle(j, n), behind = Ring::at_the_end(j, n);
                if (refill >= 0 && lane4 == 0) arm(refill);
                bar(2 + quad, 4);
                if (refill >= 0) copy(refill);
                bar(2 + quad, 4);
                o.push_back({Op::READ, Ring::slot(j), r.number(j), 0});
                if (behind >= 0) {
                    if (lane4 == 0) arm(behind);
                    bar(2 + quad, 4);
                    copy(behind);
                }
            }
            bar(1, WARPS);
            o.push_back({Op::MERGE, 0, 0, 1});
            Ring next = r;
            next.next_split(n);
            const int more = s + 1 < lens.size() ? (lens[s + 1] < NSTG ? lens[s + 1] : NSTG) : 0;
            auto begin_with = [&](int a, int b) {
                const int j = a + lane4;
                if (j >= (b < more ? b : more)) return;
                o.push_back({Op::ARM, Ring::slot(j), next.number(j), 0});
                for (int part = 0; part < 4; part++) o.push_back({Op::COPY, Ring::slot(j), next.number(j), 0});
            };
            for (int round = 1; round < QUADS; round <<= 1) {
                bar(1, WARPS);
                if (round == 1 && quad == 1) begin_with(0, NSTG - OFF);
                if (round * 2 >= QUADS) o.push_back({Op::MERGE, 0, 0, 0});
                bar(1, WARPS);
            }
            if (quad == 1) begin_with(NSTG - OFF, NSTG);
            r = next;
        }
    }
    Slot slots[NSTG];
    Bar bars[16];
    std::vector<size_t> at(WARPS, 0);
    std::vector<int> waits(WARPS, -1);  // the barrier round that the warp waits for the end of
    std::vector<std::pair<int, int>> flying;
    int wrong = 0, merging = 0;
    const int slow = rng() % (NSTG + 1), rarely = 100 + rng() % 400;  // copies to this slot (or to none) take long
    for (int idle = 0; idle < 20000;) {
        idle++;
        const size_t i = flying.empty() ? 0 : rng() % flying.size();
        if (!flying.empty() && rng() % (flying[i].first == slow ? rarely : 3) == 0) {  // a copy lands
            Slot& s = slots[flying[i].first];
            if (!s.armed || s.holds != flying[i].second) wrong++;
            if (++s.landed == 4) { s.landed = 0; s.armed = false; s.full = true; s.done++; }
            flying[i] = flying.back();
            flying.pop_back();
            idle = 0;
            continue;
        }
        const int w = rng() % WARPS;
        if (at[w] == ops[w].size()) continue;
        const Op& op = ops[w][at[w]];
        Slot& s = slots[op.slot % NSTG];
        bool goes_on = true;
        switch (op.what) {
            case Op::LOOK: goes_on = s.asked == op.number; break;
            case Op::WAIT: goes_on = (s.done & 1) != op.x; break;
            case Op::ARM:
                if (s.armed) wrong++;
                s.armed = true; s.asked = op.number;
                break;
            case Op::COPY:
                if (!s.armed || s.asked != op.number || (op.slot < OFF && merging)) wrong++;
                if (s.holds != op.number) {  // the first of its four pieces: the stage before is no longer wanted
                    if (s.unread) wrong++;
                    s.holds = op.number; s.unread = 4; s.full = false;
                }
                flying.push_back({op.slot, op.number});
                break;
            case Op::READ:
                if (s.holds != op.number || !s.full) wrong++;
                s.unread--;
                break;
            case Op::MERGE: merging += op.x ? 1 : -1; break;
            case Op::BAR: {
                Bar& b = bars[op.slot];
                if (waits[w] < 0) {
                    waits[w] = b.round;
                    if (++b.here == op.x) { b.here = 0; b.round++; }
                }
                goes_on = b.round > waits[w];
                if (goes_on) waits[w] = -1;
                break;
            }
        }
        if (goes_on) { at[w]++; idle = 0; }
        if (wrong) return wrong;
    }
    for (int w = 0; w < WARPS; w++) wrong += at[w] != ops[w].size();  // stuck
    return wrong;
}

int main(int argc, char** argv) {
    const bool look = argc > 1 && atoi(argv[1]);
    std::mt19937 rng(7);
    int bad[5] = {0, 0, 0, 0, 0};
    for (int i = 0; i < 3000; i++) {
        bad[0] += play<2, 5, 0>(rng, look) > 0;
        bad[1] += play<4, 6, 0>(rng, look) > 0;
        bad[2] += play<2, 5, 3>(rng, look) > 0;  // the splits dealt out: two row tiles,
        bad[3] += play<2, 5, 4>(rng, look) > 0;  // three,
        bad[4] += play<4, 6, 2>(rng, look) > 0;  // one
    }
    printf("%d %d %d %d %d\n", bad[0], bad[1], bad[2], bad[3], bad[4]);
    return 0;
}

// Host side of the chains (qf_w4a16_linear_batched): which linears one launch takes, in which steps, and what each gets of the things
// that several of them share. Plain C++, no GPU.
#include <algorithm>

#include "qf_stream.cuh"

namespace qf {

namespace {
struct Range {
    uintptr_t lo, hi;
    bool meets(const Range &o) const { return lo < o.hi && o.lo < hi; }
};
Range range_of(const void *p, int64_t bytes) { return Range{(uintptr_t)p, (uintptr_t)p + (p ? (uintptr_t)bytes : 0u)}; }
struct Touched {
    Range x, r, w, y;
    // Whether this linear has to come behind an earlier one: reads what that writes, writes what that reads or writes. (Weights are
    // read ahead of all waits: where an earlier result becomes weights, stream_chain_length ends the chain.)
    bool after(const Touched &o) const {
        return o.y.meets(x) || o.y.meets(r) || o.y.meets(y) || y.meets(o.x) || y.meets(o.r) || y.meets(o.w);
    }
};
Touched touched(const StreamLinear &l) {
    const qf_linear_desc &d = *l.d;
    const int64_t cols = d.epilogue == QF_EPI_SILU_MUL ? d.N / 2 : d.N, size = d.out_dtype == QF_F32 ? 4 : 2;
    return Touched{range_of(l.X, d.M * d.K * 2), range_of(d.epilogue == QF_EPI_RESIDUAL_ADD ? l.residual : nullptr, d.M * cols * size),
                   range_of(l.blob, d.N / 64 * (d.K / 128) * QF_SLAB_UNIT_BYTES), range_of(l.Y, d.M * cols * size)};
}
}  // namespace

void chain_phases(const StreamLinear *l, int count, const int64_t *room, int64_t room_step, int64_t room_two, std::vector<int> *order,
                  std::vector<ChainPhase> *phases) {
    std::vector<Touched> all;
    std::vector<int> step_of;
    int steps = 0;
    int64_t used = 0;
    for (int i = 0; i < count; ++i) {
        all.push_back(touched(l[i]));
        bool fresh = steps == 0 || used + room[i] > room_step;
        for (int o = i; !fresh && o-- > 0 && step_of[o] == steps - 1;) fresh = all[i].after(all[o]);
        if (fresh) {
            ++steps;
            used = 0;
        }
        used += room[i];
        step_of.push_back(steps - 1);
    }
    int last = -1, last_two = -1, late_before = -1, late = -1;  // phases: of the step before and of two steps back; late ones likewise
    for (int q = 0, i0 = 0, i1, i2; q < steps; ++q, i0 = i1) {
        for (i1 = i0; i1 < count && step_of[i1] == q;) ++i1;
        for (i2 = i1; i2 < count && step_of[i2] == q + 1;) ++i2;
        int64_t here = 0, there = 0;
        for (int i = i0; i < i1; ++i) here += room[i];
        for (int i = i1; i < i2; ++i) there += room[i];
        std::vector<char> waits(i1 - i0, i1 == i2 || here + there > room_two);
        bool any = false;
        for (int i = i0; i < i1; ++i) {
            for (int o = i1; o < i2; ++o) waits[i - i0] = waits[i - i0] || all[o].after(all[i]);
            any = any || waits[i - i0];
        }
        if (!any) waits.assign(i1 - i0, 1);
        const int wait0 = last, wait1 = late_before;
        const int slots_wait = last_two;
        last_two = last;
        late_before = late;
        late = -1;
        for (int part = 0; part < 2; ++part) {
            ChainPhase c{(int)order->size(), 0, {wait0, wait1}, slots_wait, q, part == 1, here, i1, i2, 0, 0, 0};
            for (int i = i0; i < i1; ++i)
                if ((waits[i - i0] != 0) == (part == 0)) order->push_back(i), ++c.count;
            if (c.count == 0) continue;
            (part == 0 ? last : late) = (int)phases->size();
            phases->push_back(c);
        }
    }
}

void plan_stream_chain(const StreamLinear *l, int count, int streams, int room, ChainPlan *plan) {
    std::vector<int64_t> slots(count);
    *plan = ChainPlan{};
    plan->linears.resize(count);
    for (int i = 0; i < count; ++i) {
        slots[i] = l[i].split > 1 ? row_blocks(*l[i].d) * l[i].split : 0;
        plan->linears[i].slots = (int)slots[i];
    }
    chain_phases(l, count, slots.data(), room, room, &plan->order, &plan->phases);
    // Where activations come from. The last linear before this one that writes any of them has made them, if they are its results whole.
    int64_t flags = 0;
    for (int i = 0; i < count; ++i) {
        ChainLinear &x = plan->linears[i];
        x.maker = kChainThere;
        x.flags = -1;
        const Touched t = touched(l[i]);
        int from = i;
        while (from-- > 0 && !touched(l[from]).y.meets(t.x)) {
        }
        if (from < 0) continue;
        const qf_linear_desc &d = *l[from].d;
        const int64_t cols = d.epilogue == QF_EPI_SILU_MUL ? d.N / 2 : d.N;
        x.maker = kChainMixed;
        if (l[from].Y != l[i].X || cols != l[i].d->K || d.out_dtype == QF_F32) continue;
        ChainLinear &m = plan->linears[from];
        if (m.flags < 0) {
            if (flags + row_blocks(d) > kStreamFlagWords) continue;
            m.flags = (int)flags;
            flags += row_blocks(d);
        }
        x.maker = from;
    }
    auto pieces_of = [&](int i) { return row_blocks(*l[i].d) * l[i].split; };
    struct Slots {
        int lo = 0, hi = 0;
        bool meets(int a, int b) const { return a < hi && lo < b; }
    };
    std::vector<Slots> of_main, of_late;  // by step
    int used = 0;                         // of the step so far
    for (ChainPhase &c : plan->phases) {
        // slots: from the lower end and the upper one in turn, so that a late phase and the next step have their own, and what is not late
        // at the very end, where it meets the step before least
        int own = 0;
        for (int k = c.first; k < c.first + c.count; ++k) own += (int)slots[plan->order[k]];
        if (!c.late) {
            used = 0;
            of_main.emplace_back();
            of_late.emplace_back();
        }
        int slot = c.step & 1 ? room - used - own : used;
        (c.late ? of_late : of_main).back() = Slots{slot, slot + own};
        // What two steps back is complete does not speak for: the step before, and what was late three steps back (for which the step
        // before does).
        const int q = c.step;
        if ((q >= 1 && of_main[q - 1].meets(slot, slot + own)) || (q >= 3 && of_late[q - 3].meets(slot, slot + own))) c.slots_wait = c.wait[0];
        used += own;
        for (int k = c.first; k < c.first + c.count; ++k) {
            plan->linears[plan->order[k]].slot = slot;
            slot += (int)slots[plan->order[k]];
        }
        c.streams = streams;
        if (c.late) {
            // to the streams that have nothing in the next step, if they can do it in that time; else to all, those first
            // that had nothing in this one
            int64_t pieces = 0, longest = 0, work = 0;
            for (int i = c.next0; i < c.next1; ++i) {
                pieces += pieces_of(i);
                longest = std::max<int64_t>(longest, l[i].per);
            }
            for (int k = c.first; k < c.first + c.count; ++k) work += pieces_of(plan->order[k]) * l[plan->order[k]].per;
            if (pieces < streams && work <= longest * (streams - pieces)) {
                c.home = (int)pieces;
                c.streams = streams - (int)pieces;
            } else {
                c.flip = 1;
            }
        }
    }
}

bool plan_slab_chain(const StreamLinear *l, int count, int sms, ChainPlan *plan) {
    const int blocks = kSlabChainPlaces * sms;
    std::vector<int64_t> per_sm(count);
    *plan = ChainPlan{};
    plan->linears.resize(count);
    for (int i = 0; i < count; ++i) {
        int depth;
        ChainLinear &x = plan->linears[i];
        slab_geometry(l[i].d->M, l[i].d->N, l[i].d->K, kSmCount, 0, &x.grid, &depth);
        if (x.grid > blocks) return false;
        x.slots = x.grid;
        per_sm[i] = x.per_sm = (x.grid + sms - 1) / sms;
    }
    chain_phases(l, count, per_sm.data(), kSlabChainPlaces, 2 * kSlabChainPlaces, &plan->order, &plan->phases);
    int home = 0, first_sm = 0, used = 0;  // places of the step
    for (const ChainPhase &c : plan->phases) {
        if (!c.late) used = 0;
        for (int k = c.first; k < c.first + c.count; ++k) {
            ChainLinear &x = plan->linears[plan->order[k]];
            x.home = home;
            x.first_sm = first_sm;
            x.slot = (c.step & 1) * blocks + used * sms;
            // the next linear begins where this one ends: what small ones leave idle is spread, and reads ahead
            home = (home + x.per_sm) % kSlabChainPlaces;
            first_sm = (first_sm + (x.grid + x.per_sm - 1) / x.per_sm) % sms;
            used += x.per_sm;
        }
    }
    return true;
}

int stream_chain_length(const StreamLinear *l, int count) {
    const void *x_of[kStreamMaxX];
    int64_t x_k[kStreamMaxX];
    std::vector<Range> written;
    int maps = 0, n = 0;
    for (; n < count && n < kStreamMaxLinears; ++n) {
        const qf_linear_desc &d = *l[n].d;
        if (d.M != l[0].d->M || d.act_dtype != l[0].d->act_dtype || row_blocks(d) * l[n].split > (1 << 24)) break;
        int m = 0;
        while (m < maps && !(x_of[m] == l[n].X && x_k[m] == d.K)) ++m;
        if (m == kStreamMaxX) break;
        // weights are read ahead of the phases: they must not be an earlier linear's result
        const Touched t = touched(l[n]);
        bool meets = false;
        for (const Range &y : written) meets = meets || y.meets(t.w);
        if (meets) break;
        if (m == maps) {
            x_of[maps] = l[n].X;
            x_k[maps++] = d.K;
        }
        bool known = false;
        for (const Range &o : written) known = known || (o.lo <= t.y.lo && t.y.hi <= o.hi);
        if (!known) written.push_back(t.y);
    }
    return n;
}

// Estimated times in us of linears of more than kSlabGemvRows rows, one by one and as a chain; the chain is taken where it is the shorter.
// One by one a linear costs `base` (it starts beside its predecessor), `member` for each further thread block with a share of a row
// block, whose partial sums the last one adds one after the other, and `unit` for each unit of 64 x 128 codes of an SM: the streaming
// GEMV kernel's costs, also where the tcgen05 kernel serves a linear alone (such batches are chains). A chain costs its launch, and for
// each step `step` from the last product to the next one's first, kChunk for each 128 codes of its longest piece, at least four of them,
// `split` where partial sums are exchanged, and `round` for each further round of pieces.
// Fitted to 64 batches at 9 to 32 rows on weights not in L2, graph replays, of former chains: activations awaited phase by phase, every phase
// counted, sums fetched by eights. Of those its standard deviation was 10 % and a wrong pick cost 7 %, 10 % on 19 other batches. Present
// chains are up to 25 % shorter than it says, so small batches go one by one that would be faster as chains, by 22 % at most below. It
// stands because the way that is taken decides about the order of the sums. (It plans with the fewest slots: the way does not depend on the
// workspace either.) Measured, one by one -> chain, at 9 / 16 / 24 / 32 rows; * marks what the estimate picks otherwise (N x K):
//   one reads the other, 2 linears:  512 x 512       8.3 -> 12.5 / 8.8 -> 12.2 / 12.2 -> 13.6 / 12.7 -> 15.5
//                                    1024 x 2816     12.8 -> 14.8 / 13.6 -> 16.6 / 18.8 -> 18.4* / 21.3 -> 20.6*
//                                    2048 x 5632     16.7 -> 16.5* / 18.3 -> 16.9* / 29.5 -> 19.4 / 31.5 -> 20.2
//                                    4096 x 4096     17.1 -> 17.5* / 19.7 -> 18.1 / 29.8 -> 20.7 / 32.4 -> 21.7
//                                    256 x 18944     33.0 -> 18.2 / 33.6 -> 18.8 / 58.9 -> 20.6 / 59.5 -> 21.4
//                       16 linears:  1024 x 1024     121 -> 93.9* / 124 -> 112* / 183 -> 129 / 187 -> 155
//                                    1024 x 2816     99.8 -> 96.0* / 106 -> 109 / 169 -> 124 / 163 -> 141
//   side by side, 2 linears:         256 x 256       6.0 -> 6.4 / 6.5 -> 6.8 / 8.6 -> 7.6* / 9.2 -> 7.9*
//                                    14336 x 1024    12.8 -> 14.5 / 14.4 -> 16.4 / 21.0 -> 19.5 / 23.5 -> 22.1
//                                    4096 x 4096     17.3 -> 14.0 / 19.7 -> 14.4 / 29.8 -> 16.3 / 32.4 -> 17.7
//                 4 linears:         512 x 512       16.6 -> 7.3 / 17.3 -> 7.6 / 24.1 -> 8.4 / 25.3 -> 8.7
//   one layer of seven:              512 / 1024      32.2 -> 22.7 / 33.8 -> 24.3 / 46.8 -> 27.7 / 48.1 -> 28.4
//                                    4096 / 14336    77.8 -> 47.4 / 84.4 -> 50.0 / 112 -> 56.7 / 120 -> 61.9
//   28 layers of four, epilogues:    256 / 256       405 -> 336* / 445 -> 432* / 592 -> 466 / 654 -> 595
bool stream_chain_pays(const StreamLinear *l, int count) {
    struct Costs {
        double base, member, unit, step, split, round;
    };
    const Costs c = l[0].d->M <= 16 ? Costs{3.2, 0.43, 0.23, 3.2, 1.2, 2.9} : Costs{4.0, 0.81, 0.37, 4.7, 1.5, 4.0};
    constexpr double kChunk = 0.48, kLaunch = 4.0;
    constexpr int64_t kStreams = 2 * kSmCount;
    double codes = 0, alone = 0;
    for (int i = 0; i < count; ++i) codes += 0.5 * (double)l[i].d->N * (double)l[i].d->K;
    if (count >= 4 && codes >= 5e6 * count) return true;  // 1.1 times as fast and more wherever measured
    for (int i = 0; i < count; ++i) {
        const qf_linear_desc &d = *l[i].d;
        const int64_t chunks = d.K / 128, units = d.N / 64 * chunks;
        int blocks, depth;
        slab_geometry(d.M, d.N, d.K, kSmCount, 0, &blocks, &depth);
        const int64_t share = units / blocks;  // where it is even, row blocks may begin with shares
        const bool even = units % blocks == 0 && (share % chunks == 0 || chunks % share == 0);
        const int64_t members = even ? std::max<int64_t>(1, chunks / share) : (chunks - 1) * blocks / units + 2;
        const int64_t per_sm = (units + blocks - 1) / blocks * ((blocks + kSmCount - 1) / kSmCount);
        alone += c.base + c.member * (double)(members - 1) + c.unit * (double)per_sm;
    }
    ChainPlan plan;
    plan_stream_chain(l, count, (int)kStreams, kStreamSlots, &plan);
    double chain = kLaunch;
    for (size_t q = 0, end; q < plan.phases.size(); q = end) {
        int64_t pieces = 0, longest = 4;
        bool split = false;
        for (end = q; end < plan.phases.size() && plan.phases[end].step == plan.phases[q].step; ++end)
            for (int k = plan.phases[end].first; k < plan.phases[end].first + plan.phases[end].count; ++k) {
                const StreamLinear &x = l[plan.order[k]];
                pieces += row_blocks(*x.d) * x.split;
                longest = std::max<int64_t>(longest, x.per);
                split = split || x.split > 1;
            }
        const double rounds = (double)((pieces + kStreams - 1) / kStreams);
        chain += c.step + kChunk * (double)longest * rounds + (split ? c.split : 0) + c.round * (rounds - 1);
    }
    return alone > chain;
}

}  // namespace qf

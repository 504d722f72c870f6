// How the chain kernels number their work: plain arithmetic, the same for the device and for a C++ compiler on the host, where it is
// tested.
#pragma once

#ifdef __CUDACC__
#define QF_HD __host__ __device__ __forceinline__
#else
#define QF_HD inline
#endif

namespace qf {

// ------------------------------ streaming tcgen05 kernel (qf_stream.cu) ------------------------------
struct StreamPhase {
    int first;       // entry
    int pieces;      // 0: ranges of units; else how many pieces the phase has
    int q, r;        // ranges: units of the phase = q * G + r, streams 0..r-1 have q + 1
    int streams;     // ranges: G; pieces: the streams from `home` on that they are dealt to, forwards and backwards in turn
    int home, flip;  // flip: backwards first
    int active;      // streams that have work
    int wait[2];     // phases that are complete before this one writes a result (or -1)
    int slots_wait;  // the phase that, with wait[1], is complete before this one writes partial sums (or -1)
    int awaited;     // whether a later phase waits for this one
};
// Units of stream `id` in a phase: how many, and *u0 the first.
QF_HD int stream_range(const StreamPhase &ph, int id, int *u0) {
    *u0 = id * ph.q + (id < ph.r ? id : ph.r);
    return ph.q + (id < ph.r ? 1 : 0);
}
// The piece that stream `id` gets in a round of dealing (none: a number from ph.pieces on).
QF_HD int stream_piece(const StreamPhase &ph, int id, int round) {
    const int k = id - ph.home;
    if ((unsigned)k >= (unsigned)ph.streams) return ph.pieces;
    return round * ph.streams + ((round ^ ph.flip) & 1 ? ph.streams - 1 - k : k);
}
// The stream that has unit u.
QF_HD int stream_of(const StreamPhase &ph, int u) {
    const int head = ph.r * (ph.q + 1);
    return u < head ? u / (ph.q + 1) : ph.r + (u - head) / ph.q;
}

// ------------------------------ chains of up to 8 rows (qf_slab_chain.cu) ------------------------------
constexpr int kSlabChainPlaces = 4;  // thread blocks per SM

// The place of a thread block: 4 * SM + its place on the SM. An entry takes `per_sm` places of SMs from `first_sm` on, around, those from
// `home` on, around, and numbers its blocks SM by SM: shares of the work differ by a unit, and in this order every SM gets the same
// sum (numbered across the SMs, the larger shares of a linear whose rows repeat after 148 blocks pile up on a few: 772 us a step of
// 16 layers of 4096 / 14336 at one row against 691).
QF_HD unsigned sc_number(unsigned n_sm, int home, int per_sm, int first_sm, unsigned place) {
    const unsigned i = (place - (unsigned)home) % kSlabChainPlaces;
    unsigned sm = place / kSlabChainPlaces + n_sm - (unsigned)first_sm;
    if (sm >= n_sm) sm -= n_sm;
    return i < (unsigned)per_sm ? sm * (unsigned)per_sm + i : 0xffffffffu;
}

// The place that a thread block takes on SM `sm` of `sms` numbers. started(): how many blocks the SM had before; given(i): how many SMs'
// i-th places had been given out before.
template <typename Started, typename Given>
QF_HD unsigned sc_place(unsigned n_sm, unsigned sm, unsigned sms, Started started, Given given) {
    unsigned i = started();
    if (i > kSlabChainPlaces - 1u) i = kSlabChainPlaces - 1u;
    if (sms == n_sm) return sm * kSlabChainPlaces + i;  // every SM has as many blocks as it can hold
    // numbers of SMs with gaps: the first blocks of the SMs take the first places, and so on; where those are used up (on an uneven
    // placement) others are left
    for (int k = 0; k < kSlabChainPlaces; ++k) {
        const unsigned n = given(i);
        if (n < n_sm) return n * kSlabChainPlaces + i;
        i = (i + 1u) % kSlabChainPlaces;
    }
    return 0u;  // never: as many places as blocks
}

}  // namespace qf

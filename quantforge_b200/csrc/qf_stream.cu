// K4: W4A16 linears of up to 32 rows on QF_LAYOUT_GEMV_SLAB weights, converted into tensor memory; one linear, or a chain of them in
// one launch.
//
// Y[M,N] = X[M,K] . W^T as Y^T = W . X^T: the dequantised weights are the A operand of tcgen05 MMAs (128 weight rows x 16 codes an
// instruction) and live in TMEM only, the activations are B from shared memory. What the streaming GEMV kernel (mma.sync) spends
// on fragments of X and on the MMAs themselves, which take issue slots and packed-half time from the conversion and grow with the
// rows, is here one thread's work. Without memory, converters and MMAs alone take 283 cycles per 128 x 128 codes and SM; HBM delivers
// those in 377; the kernel takes about 450, bound by the issue slots that the conversion and its hand-overs share. In a chain there are 5 to
// 6 us from the last MMA of a step to the first of the next (the median stream's; eight layers of 4096 / 14336, each linear behind the one
// before, 9 and 16 rows; 6.5 to 8 at 32 rows): partial sums, results, a release (1 us and more behind stores), counters, a copy of
// activations.
//
// Work split. Units of 128 rows x 128 codes. Of a single linear they are numbered row block major, K chunk minor, and stream i of G
// owns a contiguous range of them (the first r streams one more than the others): every stream moves the same number of bytes
// whatever the shape is. A chain is a list of phases, each of linears that do not depend on each other, and each with the phases that
// it waits for. What the next step of the chain does not touch (q, k and v beside o) is a phase of its own that holds nothing up: it
// goes to streams that have nothing to do in that step, or fills the time in which the others hand over (the linears of 32 layers at
// 16 rows 1459 -> 1355 us). Only results wait for whole phases. Activations that are another linear's results are read row block by row
// block as these are finished (a counter each), and partial sums are exchanged as soon as their slots are free (linears of 32 layers,
// 4096 / 14336, with the code of the results made smaller, sums fetched by fours and phases that nobody waits for not counted: 16 rows
// 1372 -> 1280 us, 9 rows 1338 -> 1207; eight layers of seven linears 437 -> 371 at 16 rows, 495 -> 421 at 24). In a chain K is cut
// into pieces exactly as the tcgen05 kernel (qf_gemm_tcgen05.cu) cuts it for the same sizes on other layouts, so that each sum is made
// of the same partial sums in the same order: a deep stack of 16-bit layers turns any other order into another rounding of everything
// behind it (32 layers: hidden states 0.9 % apart, where the same bits are the least surprise). The pieces of a phase are dealt to the
// streams forwards and backwards in turn. Weights are requested as far ahead as the ring of stages allows, across linears and phases;
// only activations and results wait.
//
// A thread block has its SM to itself and runs two streams side by side (one stream's waits are the other's time to convert), each
// with half of its threads, shared memory and TMEM. (One block per SM because a cooperative launch admits no more of a kernel that
// allocates TMEM.) Of a stream's sixteen warps:
//   warps 0-7    two converter groups, alternating units: thread t owns weight row t of the unit, reads its 64 bytes of codes and
//                its constants from the swizzled stage, converts and writes them to TMEM lane t (tcgen05.st).
//   one warp     copies of weights: one TMA box per unit, a chunk of two row blocks of the blob as 64-byte lines.
//   one warp     copies of activations (MMA B tiles, K-major, 128-byte swizzle); those that are another linear's results as soon as
//                their row block is finished.
//   one warp     one thread issues the MMAs of a unit once its weights and activations are there.
//   one warp     waits for the phases that results may not overtake, and tells warps 12-15.
//   warps 12-15  results: a row block's accumulators go from TMEM to Y, or to the workspace where others have chunks of it too.
//
// Row blocks whose K range is shared by several streams (its members): a member leaves its partial sums in a slot of the workspace
// as 8-byte (value, token) words - no fence, no atomic. The members finish the pairs of batch rows in turn (one member
// reading ten others' sums of 16 rows would be a dozen trips to L2 in a row): whoever finishes a pair polls all members' words
// (bounded), adds in their order (deterministic), writes Y and clears the words for the next user of the slots. As streams wait for one
// another, the launch is cooperative, and without programmatic dependent launch: it would find no room beside another kernel's blocks.
//
// Shared memory takes all but a few KB of the SM's first-level cache, so a spilled register is a trip to L2: the registers are split
// between the roles such that none is (see setmaxnreg below).
#include <algorithm>
#include <vector>

#include "qf_stream.cuh"
#include "qf_tcgen05.cuh"

namespace qf {

constexpr int ST_THREADS = 1024;                             // two streams of sixteen warps
constexpr int ST_LINES = QF_SLAB_UNIT_BYTES / 64;            // 64-byte lines of a unit of 64 rows
constexpr int ST_UNIT_BYTES = 2 * QF_SLAB_UNIT_BYTES;        // two row blocks, one chunk
constexpr int ST_NA = 3;                                     // A operand buffers in TMEM, 64 columns each
constexpr int ST_TMEM_COLS = 256;                            // of a stream: half an SM's

// NB: the MMA's N, batch rows padded to 16 or 32.
template <int NB>
struct StreamCfg {
    static constexpr int W_STAGES = 8;
    static constexpr int X_STAGES = NB == 16 ? 8 : 4;
    static constexpr int X_BOX_BYTES = NB * 128;             // 64 codes
    static constexpr int X_BYTES = 2 * X_BOX_BYTES;
    static constexpr int W_OFF = X_STAGES * X_BYTES;
    static constexpr int BAR_OFF = W_OFF + W_STAGES * ST_UNIT_BYTES;
    static constexpr int BARS = 2 * W_STAGES + 2 * X_STAGES + 2 * ST_NA + 2 * 2;
    static constexpr int STREAM_BYTES = (BAR_OFF + BARS * 8 + 1023) / 1024 * 1024;
    static_assert(2 * NB + ST_NA * 64 <= ST_TMEM_COLS, "two accumulators and the A operands");
};

struct StreamEntry {  // one linear
    void *Y;
    const void *residual;
    int N, chunks;   // chunks of 128 codes along K
    int begin, end;  // its units (or pieces) within the phase
    int split, per;  // pieces: K is cut into `split` of them, `per` chunks each (the last may be shorter)
    int slot;        // of its first piece, where there are several to a row block
    int x_map;
    // Where the activations come from: kXThere, kXGate, or the first counter of the row blocks of the linear that makes them, its
    // results. A counter is complete at x_want; x_two: two row blocks to a chunk (SiLU * mul).
    int x_from;
    int flags;       // this linear's first counter (or -1: nobody looks)
    int16_t x_want, x_two;
    int16_t out_dtype, epilogue;
};
constexpr int kXThere = -1;  // no linear of the launch writes them
constexpr int kXGate = -2;   // they are there when the phase may write its results

struct StreamArgs {
    unsigned long long *slots;  // [kStreamSlots or kChainSlots][slot_words] (value | token << 32), zero between launches
    // [phases] streams that have finished the phase, [kStreamMaxLinears] result warps that have finished everything, from kStreamFlags
    // on result warps that have finished a row block; `words` of them, zero between launches
    unsigned *done;
    int *status;
    int slot_words;
    int M, x_rows;              // x_rows: rows of an X box (M rounded up to 8)
    int phases, linears, words;
};
constexpr int kStreamFlags = (kStreamMaxLinears + 4) / 4 * 4;
template <int CAP>
struct StreamParams {
    static constexpr int XCAP = CAP == 1 ? 1 : kStreamMaxX;
    CUtensorMap w[CAP];
    CUtensorMap x[XCAP];
    StreamEntry e[CAP];
    StreamPhase ph[CAP];
    StreamArgs a;
};
static_assert(sizeof(StreamParams<kStreamMaxLinears>) <= 32764, "kernel parameters");
static_assert(kStreamFlags > kStreamMaxLinears && kStreamFlags * sizeof(unsigned) <= kCounterBytes, "the counter region of the workspace");
// The lists of linears and phases, in shared memory: every role reads the next phase's when it gets there, and from the parameter
// space that was a miss of the constant cache each time.
template <int CAP>
struct StreamTables {
    StreamEntry e[CAP];
    StreamPhase ph[CAP];
};
template <int NB, int CAP>
constexpr int stream_smem_bytes() {
    return 2 * StreamCfg<NB>::STREAM_BYTES + 1024 /*alignment*/ + (int)sizeof(StreamTables<CAP>);
}
static_assert(stream_smem_bytes<16, kStreamMaxLinears>() <= 227 << 10 && stream_smem_bytes<32, kStreamMaxLinears>() <= 227 << 10,
              "shared memory of a block");

// Consecutive chunks of one row block, and who else has chunks of it: `members` of which this one is number `self`. A member's sums go
// to slot `base` + its number, the first member's to `slot0`.
struct Segment {
    int e, b, c, len;
    int members, self, slot0, base;
};
template <int CAP>
__device__ __forceinline__ bool stream_works(const StreamPhase &ph, int id) {
    int u;
    return CAP > 1 ? stream_piece(ph, id, 0) < ph.pieces : stream_range(ph, id, &u) > 0;
}
// Walks a stream's work segment by segment; f returns whether to go on.
template <int CAP, typename F>
__device__ __forceinline__ void for_segments(const StreamTables<CAP> &t, int phase, int id, F f) {
    const StreamPhase ph = t.ph[phase];
    int e = ph.first;
    Segment g;
    if (CAP > 1) {
        for (int round = 0;; ++round) {
            const int j = stream_piece(ph, id, round);
            if (j >= ph.pieces) return;
            while (j >= t.e[e].end) ++e;
            const int split = t.e[e].split, local = j - t.e[e].begin;
            g.e = e;
            g.b = local / split;
            g.self = local - g.b * split;
            g.c = g.self * t.e[e].per;
            g.len = min(t.e[e].per, t.e[e].chunks - g.c);
            g.members = split;
            g.base = g.slot0 = t.e[e].slot + g.b * split;
            if (!f(g)) return;
        }
    }
    int u;
    const int n = stream_range(ph, id, &u);
    if (n == 0) return;
    const int end = u + n, chunks = t.e[e].chunks;
    g.e = e;
    g.b = u / chunks;
    g.c = u - g.b * chunks;
    while (true) {
        g.len = min(chunks - g.c, end - u);
        const int first = g.c + g.len == chunks && g.c == 0 ? id : stream_of(ph, u - g.c);
        g.members = (g.len == chunks ? id : stream_of(ph, u - g.c + chunks - 1)) - first + 1;
        g.self = id - first;
        g.base = first;
        g.slot0 = ph.streams + first;  // a stream's last segment may begin a row block, while its first one ends another
        if (!f(g)) return;
        u += g.len;
        if (u == end) return;
        ++g.b;
        g.c = 0;
    }
}

__device__ __forceinline__ void st_words2(unsigned long long *ptr, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(ptr), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_words2(const unsigned long long *ptr, unsigned long long &a, unsigned long long &b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(ptr) : "memory");
}
__device__ __forceinline__ unsigned long long word_of(uint32_t v) { return (unsigned long long)v | (1ull << 32); }
__device__ __forceinline__ unsigned ld_acquire(const unsigned *ptr) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
    return v;
}
// Between ordinary accesses to global memory and accesses of the copy engine.
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Finished sums leave as pairs of neighbouring outputs of a batch row, a pair to a lane: of two neighbouring lanes, which hold two batch
// rows of neighbouring weight rows, the even one takes the first batch row and the odd one the second. Code that runs once a phase
// costs what its instructions take to arrive, so there are few of them: 16-bit types differ in one selection, and a pair of outputs
// is one store. (One output per store with a branch per type and store, 74 KB of code instead of 58: 32 layers of 4096 / 14336 at 16 rows
// 1362 us instead of 1283.)
struct StreamOut {
    int64_t o;  // element of the first of the two outputs, of the first pair of batch rows
    int step;   // elements from one pair of batch rows to the next
    int m;      // this lane's batch row of the first pair
};
__device__ __forceinline__ StreamOut stream_out(const StreamEntry &e, int n, int m0) {
    const int m = m0 + (n & 1);
    return StreamOut{(int64_t)m * e.N + (n & ~1), 2 * e.N, m};
}
// What the residual epilogue adds to PAIRS pairs of batch rows, as it lies in memory.
template <int PAIRS>
__device__ __forceinline__ void stream_residual(const StreamEntry &e, int M, const StreamOut &at, uint2 (&r)[PAIRS]) {
    const bool f32 = e.out_dtype == QF_F32;
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
        r[i] = make_uint2(0u, 0u);
        const int64_t o = at.o + (int64_t)i * at.step;
        if (at.m + 2 * i < M) {
            if (f32) r[i] = *reinterpret_cast<const uint2 *>(reinterpret_cast<const float *>(e.residual) + o);
            else r[i].x = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const uint16_t *>(e.residual) + o);
        }
    }
}
__device__ __forceinline__ void stream_put(const StreamEntry &e, int64_t o, float lo, float hi) {
    if (e.out_dtype == QF_F32) {
        *reinterpret_cast<float2 *>(reinterpret_cast<float *>(e.Y) + o) = make_float2(lo, hi);
        return;
    }
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    const __half2 h = __floats2half2_rn(lo, hi);
    *reinterpret_cast<uint32_t *>(reinterpret_cast<uint16_t *>(e.Y) + o) =
        e.out_dtype == QF_BF16 ? *reinterpret_cast<const uint32_t *>(&b) : *reinterpret_cast<const uint32_t *>(&h);
}
// Writes finished sums: PAIRS pairs of batch rows from row m0 on (as far as M goes) of weight row n; `r`: stream_residual's. All 32
// lanes of a warp, which hold 32 consecutive weight rows. The steps of all pairs go side by side: these warps run a chain of dependent
// instructions otherwise, 450 cycles a pair.
template <int PAIRS>
__device__ __forceinline__ void stream_emit(const StreamEntry &e, int M, int n, int m0, const float (&v)[2 * PAIRS], const StreamOut &at,
                                            const uint2 (&r)[PAIRS]) {
    const bool odd = n & 1;
    if (e.epilogue == QF_EPI_SILU_MUL) {
        // rows 0..7 of sixteen are gate rows, 8..15 the matching up rows: of a pair the gate lane does the first batch row, the up lane
        // the second
        const bool up_lane = n & 8;
        const int cols = e.N >> 1, col = (n >> 4) * 8 + (n & 7);
        float gate[PAIRS], up[PAIRS];
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, up_lane ? v[2 * i] : v[2 * i + 1], 8);
            gate[i] = up_lane ? other : v[2 * i];
            up[i] = up_lane ? v[2 * i + 1] : other;
        }
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) up[i] = gate[i] / (1.f + expf(-gate[i])) * up[i];
        const int m = m0 + (up_lane ? 1 : 0);
#pragma unroll
        for (int i = 0; i < PAIRS; ++i)
            if (m + 2 * i < M) store_out(e.Y, e.out_dtype, (int64_t)(m + 2 * i) * cols + col, up[i]);
        return;
    }
    const bool add = e.epilogue == QF_EPI_RESIDUAL_ADD;
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * i] : v[2 * i + 1], 1);
        float lo = odd ? other : v[2 * i], hi = odd ? v[2 * i + 1] : other;
        if (add) {
            float a = __uint_as_float(r[i].x), b = __uint_as_float(r[i].y);
            if (e.out_dtype == QF_BF16) b = __uint_as_float(r[i].x & 0xffff0000u), a = __uint_as_float(r[i].x << 16);
            if (e.out_dtype == QF_F16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&r[i].x));
                a = f.x, b = f.y;
            }
            lo += a;
            hi += b;
        }
        if (at.m + 2 * i < M) stream_put(e, at.o + (int64_t)i * at.step, lo, hi);
    }
}

// Word of a member's slot (32 bits: 888 slots of at most 4096 words).
__device__ __forceinline__ unsigned slot_of(const StreamArgs &a, const Segment &g, int member) {
    return (unsigned)((member == 0 ? g.slot0 : g.base + member) * a.slot_words);
}
// Adds the members' shares of a pair of batch rows, in their order, and clears their words; the words of WORDS members are requested at
// a time (missing ones are the last member's again, so a linear of wide N, with two to four members a row block, takes four: together
// with plain stores of SiLU * mul and eight rows at a time, 32 rows: 5120 x 27648 38.9 -> 35.3 us, 8192 x 57344 73.8 -> 69.9, SiLU *
// mul of 4096 x 28672 32.6 -> 30.8; four for everybody: 8192 x 8192 22.1 -> 22.6). A chain always takes four, which is less code: the
// linears of 32 layers of 4096 / 14336 at 16 rows 1297 -> 1280 us, eight layers of seven 391 -> 371, at 32 rows 494 -> 465 (with both
// in the code, by members, 1297 and 484). Warp-uniform; false when a wait ran out. (Two pairs at a time: the linears of 32 layers at 9
// to 16 rows 1417 to 1461 us, then 1500 to 1528.)
template <int WORDS>
__device__ __forceinline__ bool stream_sum(const StreamArgs &a, const Segment &g, int pair, int row, float (&v)[2],
                                           volatile int *abort_flag) {
    v[0] = v[1] = 0.f;
    const unsigned at = (unsigned)(pair * 128 + row) * 2u;
#pragma unroll 1
    for (int m0 = 0; m0 < g.members; m0 += WORDS) {
        // (where there are fewer, the last member's words take the place of the missing ones; what is added for them is +0, and a sum that
        // begins with +0 is never -0)
        unsigned src[WORDS];
        unsigned long long w[WORDS][2];
#pragma unroll
        for (int j = 0; j < WORDS; ++j) src[j] = slot_of(a, g, min(m0 + j, g.members - 1)) + at;
        const long long t0 = clock64();
        while (true) {
            unsigned miss = 0u;
#pragma unroll
            for (int j = 0; j < WORDS; ++j) ld_words2(a.slots + src[j], w[j][0], w[j][1]);
#pragma unroll
            for (int j = 0; j < WORDS; ++j) miss |= ((unsigned)(w[j][0] >> 32) ^ 1u) | ((unsigned)(w[j][1] >> 32) ^ 1u);
            if (!__any_sync(0xffffffffu, miss != 0u)) break;
            if (__any_sync(0xffffffffu, clock64() - t0 > kWaitCycles || *abort_flag != 0)) return false;
        }
#pragma unroll
        for (int j = 0; j < WORDS; ++j) {
            const bool real = m0 + j < g.members;
            v[0] += real ? __uint_as_float((uint32_t)w[j][0]) : 0.f;
            v[1] += real ? __uint_as_float((uint32_t)w[j][1]) : 0.f;
            st_words2(a.slots + src[j], 0ull, 0ull);
        }
    }
    return true;
}

// Bounded wait. The thread asks to be suspended for up to 20 us at a time: a warp that waits takes no issue slots, which the
// converters need.
__device__ __forceinline__ bool stream_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool stream_wait_on(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    const long long t0 = clock64();
    while (true) {
        if (stream_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abort_flag = 1;
            return false;
        }
    }
}

__device__ __forceinline__ bool stream_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return stream_try_wait(bar, parity) || stream_wait_on(bar, parity, abort_flag);
}

// Warp-uniform: waits until the phases behind `gate` are complete; false when another role gave up.
__device__ __forceinline__ bool stream_gate(volatile int *gates, int gate, volatile int *abort_flag) {
    bool ok = true;
    const long long t0 = clock64();
    while (ok && *gates < gate) {
        __nanosleep(40);
        if (*abort_flag) ok = false;
        else if (clock64() - t0 > kWaitCycles) *abort_flag = 1;
    }
    ok = __all_sync(0xffffffffu, ok);
    __threadfence_block();
    return ok;
}
// Waits until phase w (or -1) is complete; one thread.
__device__ __forceinline__ bool stream_phase_done(const StreamArgs &a, int w, unsigned want, volatile int *abort_flag) {
    const long long t0 = clock64();
    while (ld_acquire(a.done + w) < want) {
        __nanosleep(40);
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abort_flag = 1;
            return false;
        }
    }
    return true;
}
// Waits for the row blocks that chunk c of an entry's activations comes from, and looks at those of the n - 1 chunks behind it: how many
// chunks are there (at least one), or 0 when it gave up. All 32 lanes, each a chunk's counters.
__device__ __forceinline__ int stream_arrived(const StreamArgs &a, const StreamEntry &e, int c, int n, int lane, volatile int *abort_flag) {
    const unsigned want = (unsigned)e.x_want;
    const unsigned *count = a.done + e.x_from + (e.x_two ? 2 * (c + lane) : c + lane);
    bool there = lane >= n;
    const long long t0 = clock64();
    while (true) {
        if (!there) there = ld_acquire(count) >= want && (!e.x_two || ld_acquire(count + 1) >= want);
        const unsigned yet = ~__ballot_sync(0xffffffffu, there);
        if (!(yet & 1u)) {
            __syncwarp();
            // the results were stored through the generic proxy and are read by the copy engine
            fence_proxy_async_all();
            return min(n, yet ? __ffs(yet) - 1 : 32);
        }
        if (clock64() - t0 > kWaitCycles) *abort_flag = 1;
        if (__any_sync(0xffffffffu, *abort_flag != 0)) return 0;
        __nanosleep(20);
    }
}
// Whether this is the last of a stream's four result warps to get here; it then speaks for the stores of all four.
__device__ __forceinline__ bool stream_last_warp(unsigned *count) {
    unsigned before;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(smem_u32(count)) : "memory");
    return (before & 3u) == 3u;
}

template <bool BF16, int NB, int CAP>
__global__ void __launch_bounds__(ST_THREADS, 1) stream_kernel(const __grid_constant__ StreamParams<CAP> p) {
    using C = StreamCfg<NB>;
    extern __shared__ uint8_t stream_smem[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    // Of a stream: of the phases that it has work in, two steps each: partial sums may be written, results may be.
    __shared__ int s_gates[2];
    __shared__ unsigned s_finished[2][4];  // result warps that have finished a phase, by its number modulo 4

    const int tid = threadIdx.x & 511;
    const int half = threadIdx.x >> 9;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    // The single threads of the two streams sit on different schedulers (a warp's is its number mod 4): weights 8 and 10,
    // activations 9 and 11, MMAs 10 and 8.
    // roles: 0 converts, 1 weights, 2 activations, 3 MMAs, 4 results, 5 waits for phases
    const int role = warp < 8 ? 0 : warp >= 12 ? 4 : (half == 0 ? 0x5321 : 0x2153) >> (4 * (warp - 8)) & 7;
    const int id = half * (int)gridDim.x + (int)blockIdx.x;  // of the stream: two streams of a block differ by at most a unit
    const uint32_t base = ((smem_u32(stream_smem) + 1023u) & ~1023u) + (uint32_t)half * C::STREAM_BYTES;
    const uint32_t bars = base + C::BAR_OFF;
    auto x_stage = [&](int s) { return base + (uint32_t)s * C::X_BYTES; };
    auto w_stage = [&](int s) { return base + C::W_OFF + (uint32_t)s * ST_UNIT_BYTES; };
    auto wfull = [&](int s) { return bars + 8u * s; };
    auto wempty = [&](int s) { return bars + 8u * (C::W_STAGES + s); };
    auto xfull = [&](int s) { return bars + 8u * (2 * C::W_STAGES + s); };
    auto xempty = [&](int s) { return bars + 8u * (2 * C::W_STAGES + C::X_STAGES + s); };
    constexpr int AB = 2 * C::W_STAGES + 2 * C::X_STAGES;
    auto afull = [&](int a) { return bars + 8u * (AB + a); };
    auto aempty = [&](int a) { return bars + 8u * (AB + ST_NA + a); };
    auto dfull = [&](int d) { return bars + 8u * (AB + 2 * ST_NA + d); };
    auto dempty = [&](int d) { return bars + 8u * (AB + 2 * ST_NA + 2 + d); };
    volatile int *gates = &s_gates[half];

    const StreamArgs &a = p.a;
    StreamTables<CAP> &t = *reinterpret_cast<StreamTables<CAP> *>(
        stream_smem + ((1024u - (smem_u32(stream_smem) & 1023u)) & 1023u) + 2 * C::STREAM_BYTES);
    const int phases = CAP == 1 ? 1 : a.phases;
    volatile int *abort_flag = &s_abort;

    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < C::W_STAGES; ++s) {
            mbar_init(wfull(s), 1);
            mbar_init(wempty(s), 4);  // the warps of the group that converts the unit
        }
        for (int s = 0; s < C::X_STAGES; ++s) {
            mbar_init(xfull(s), 1);
            mbar_init(xempty(s), 1);
        }
        for (int i = 0; i < ST_NA; ++i) {
            mbar_init(afull(i), 4);
            mbar_init(aempty(i), 1);
        }
        for (int d = 0; d < 2; ++d) {
            mbar_init(dfull(d), 1);
            mbar_init(dempty(d), 4);
        }
        s_gates[half] = 0;
        for (int i = 0; i < 4; ++i) s_finished[half][i] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 10 && half == 0) tmem_alloc<false>(smem_u32(&s_tmem_base), 2 * ST_TMEM_COLS);
    if (a.x_rows < NB) {
        // the rows of the B tiles that no copy writes
        for (uint32_t o = tid * 16u; o < (uint32_t)C::W_OFF; o += 512u * 16u)
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(base + o), "r"(0u) : "memory");
        fence_proxy_async_shared();
    }
    for (int i = threadIdx.x; i < a.linears * (int)(sizeof(StreamEntry) / 4); i += ST_THREADS)
        reinterpret_cast<uint32_t *>(t.e)[i] = reinterpret_cast<const uint32_t *>(p.e)[i];
    for (int i = threadIdx.x; i < phases * (int)(sizeof(StreamPhase) / 4); i += ST_THREADS)
        reinterpret_cast<uint32_t *>(t.ph)[i] = reinterpret_cast<const uint32_t *>(p.ph)[i];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem_base + (uint32_t)half * ST_TMEM_COLS;  // two accumulators of NB columns, then the A operands

    // Registers: 64 a thread at launch; a stream's four warpgroups share them as 2 x 48, 56 and 104. With 64 for all, the result warps
    // spilled addresses and sums in flight: a first form of the chain took 1971 us for 32 layers at 16 rows, with 64, 40 and 88 1557,
    // with this 1495.
    if (role == 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    else if (role == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    int issued = 0;  // copies of this thread (elected lanes of roles 1 and 2)
    if (role == 1) {
        // ------------------------------ weights ------------------------------
        const bool leader = elect_one();
        if (leader) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int phase = 0; phase < phases && ok; ++phase)
                for_segments(t, phase, id, [&](const Segment &g) {
                    if (g.e + 1 < a.linears) tma_prefetch_desc(&p.w[g.e + 1]);
                    for (int i = 0; i < g.len; ++i) {
                        if (!stream_wait(wempty(s), ph ^ 1u, abort_flag)) return ok = false;
                        mbar_arrive_expect_tx(wfull(s), ST_UNIT_BYTES);
                        tma_load_4d(w_stage(s), &p.w[g.e], wfull(s), 0, 0, g.c + i, 2 * g.b);
                        ++issued;
                        if (++s == C::W_STAGES) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                    return true;
                });
        }
        __syncwarp();
    } else if (role == 2) {
        // ------------------------------ activations ------------------------------
        const bool leader = elect_one();
        int s = 0, nth = 0;
        uint32_t ph = 0;
        bool ok = true;
        const uint32_t tx = 2u * (uint32_t)a.x_rows * 128u;
        for (int phase = 0; phase < phases && ok; ++phase) {
            if (!stream_works<CAP>(t.ph[phase], id)) continue;
            ++nth;
            bool open = false;
            for_segments(t, phase, id, [&](const Segment &g) {
                const StreamEntry &en = t.e[g.e];
                const CUtensorMap *map = &p.x[en.x_map];
                if (leader) tma_prefetch_desc(map);
                int there = CAP > 1 && en.x_from >= 0 ? 0 : g.len;  // chunks that can be read
                if (CAP > 1 && en.x_from == kXGate && !open) {
                    ok = stream_gate(gates, 2 * nth, abort_flag);
                    if (!ok) return false;
                    fence_proxy_async_all();
                    open = true;
                }
                for (int i = 0; i < g.len; ++i) {
                    if (CAP > 1 && i == there) {
                        const int n = stream_arrived(a, en, g.c + i, g.len - i, lane, abort_flag);
                        ok = n > 0;
                        if (!ok) return false;
                        there += n;
                    }
                    ok = __all_sync(0xffffffffu, !leader || stream_wait(xempty(s), ph ^ 1u, abort_flag));
                    if (!ok) return false;
                    if (leader) {
                        mbar_arrive_expect_tx(xfull(s), tx);
                        tma_load_2d(x_stage(s), map, xfull(s), (g.c + i) * 128, 0);
                        tma_load_2d(x_stage(s) + C::X_BOX_BYTES, map, xfull(s), (g.c + i) * 128 + 64, 0);
                    }
                    ++issued;
                    if (++s == C::X_STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                return true;
            });
        }
        __syncwarp();
    } else if (role == 5) {
        // ------------------------------ waits for phases ------------------------------
        // The results of a phase come behind the phases that it waits for; its activations may be there before (stream_arrived), and its
        // partial sums may be exchanged as soon as the last phase with the same slots is complete.
        if (CAP > 1 && elect_one()) {
            int passed[3] = {-1, -1, -1}, opened = 0;
            bool ok = true;
            for (int phase = 0; phase < phases && ok; ++phase) {
                if (!stream_works<CAP>(t.ph[phase], id)) continue;
                const int waits[3] = {t.ph[phase].slots_wait, t.ph[phase].wait[1], t.ph[phase].wait[0]};
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int w = waits[i];
                    if (ok && w >= 0 && w != passed[i]) ok = stream_phase_done(a, w, (unsigned)t.ph[w].active, abort_flag);
                    passed[i] = w;
                    if (ok && i > 0) {
                        __threadfence_block();
                        *gates = ++opened;
                    }
                }
            }
        }
        __syncwarp();
    } else if (role == 3) {
        // ------------------------------ MMAs ------------------------------
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10) | ((uint32_t)(NB >> 3) << 17) |
                                   ((uint32_t)(128 >> 4) << 24);
            const uint64_t desc0 = make_b_desc(x_stage(0));
            int i = 0, s = 0, seg = 0;
            uint32_t aph = 0, xph = 0;
            bool ok = true;
            for (int phase = 0; phase < phases && ok; ++phase)
                for_segments(t, phase, id, [&](const Segment &g) {
                    const int d = seg & 1;
                    if (!stream_wait(dempty(d), ((uint32_t)(seg >> 1) & 1u) ^ 1u, abort_flag)) return ok = false;
                    const uint32_t d_tmem = tmem + d * NB;
                    for (int k = 0; k < g.len; ++k) {
                        if (!stream_wait(afull(i), aph, abort_flag) || !stream_wait(xfull(s), xph, abort_flag)) return ok = false;
                        tc_fence_after();
                        const uint32_t a_tmem = tmem + 2 * NB + i * 64;
                        const uint64_t desc = desc0 + (uint32_t)s * (uint32_t)(C::X_BYTES >> 4);
                        umma_ts<false>(d_tmem, a_tmem, desc, idesc, k > 0 ? 1u : 0u);
#pragma unroll
                        for (int kk = 1; kk < 8; ++kk)
                            umma_ts<false>(d_tmem, a_tmem + kk * 8, desc + (uint32_t)(((kk >> 2) * C::X_BOX_BYTES + (kk & 3) * 32) >> 4),
                                           idesc, 1u);
                        umma_commit<false>(aempty(i));
                        umma_commit<false>(xempty(s));
                        if (++i == ST_NA) {
                            i = 0;
                            aph ^= 1u;
                        }
                        if (++s == C::X_STAGES) {
                            s = 0;
                            xph ^= 1u;
                        }
                    }
                    umma_commit<false>(dfull(d));
                    ++seg;
                    return true;
                });
        }
        __syncwarp();
    } else if (role == 0) {
        // ------------------------------ converters ------------------------------
        int total = 0;
        for (int q = CAP == 1 ? 0 : lane; q < phases; q += 32) for_segments(t, q, id, [&](const Segment &g) { return total += g.len, true; });
        if (CAP > 1) total = __reduce_add_sync(0xffffffffu, total);
        const int row = tid & 127;
        const uint32_t lane_tmem = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 2 * NB;
        // A tile of the blob is 17 lines of 64 bytes, sixteen rows and their constants; line l of a stage holds its 16-byte piece i
        // at i ^ (l / 2 % 4).
        const int tile = (row >> 6) * ST_LINES + ((row & 63) >> 4) * 17;
        const int line = tile + (row & 15), cline = tile + 16;
        const uint32_t w_off = (uint32_t)line * 64u + (((uint32_t)(line >> 1) & 3u) << 4);  // its piece 0
        const uint32_t c_off = (uint32_t)cline * 64u + ((((uint32_t)(row & 15) >> 2) ^ ((uint32_t)(cline >> 1) & 3u)) << 4) +
                               ((uint32_t)row & 3u) * 4u;
        int s = warp >> 2, i = warp >> 2;  // stage and A operand buffer of the unit
        uint32_t wph = 0u, aph = 1u;
        for (int it = warp >> 2; it < total; it += 2) {
            bool ready = stream_wait(wfull(s), wph, abort_flag);
            ready = ready && stream_wait(aempty(i), aph, abort_flag);
            if (!__all_sync(0xffffffffu, ready)) break;  // the tcgen05.st below is warp-collective
            tc_fence_after();
            const uint32_t stage = w_stage(s);
            ShortConvert<BF16> conv;
            conv.set_slab(lds32(stage + c_off));
            // Piece j holds words j, j + 4, j + 8, j + 12 of the row's sixteen; the next piece is on its way while one is converted.
            // (All four pieces first and stores of 16 columns: 59.6 us on 57344 x 8192, this form 56.6.)
            const uint32_t piece = stage + w_off;
            uint32_t col = lane_tmem + i * 64;
            uint4 v = lds128(piece);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint4 next = j < 3 ? lds128(piece ^ ((uint32_t)(j + 1) << 4)) : v;
                uint32_t q[4];
                conv(v.x, q);
                tmem_st4(col, q);
                conv(v.y, q);
                tmem_st4(col + 16, q);
                conv(v.z, q);
                tmem_st4(col + 32, q);
                conv(v.w, q);
                tmem_st4(col + 48, q);
                v = next;
                col += 4;
            }
            if (BF16 && conv.wide) {
                // once more in the form for scales of 2^126 and more (see ShortConvert). It reads everything again: values kept
                // for it would cost the ordinary path registers (59 -> 63 us on 57344 x 8192)
                tmem_wait_st();
                ShortConvert<BF16> again;
                again.set_slab(lds32(stage + c_off));
#pragma unroll 1
                for (int j = 0; j < 16; ++j) {
                    uint32_t q[4];
                    dequant8<BF16>(lds32((piece ^ (((uint32_t)j & 3u) << 4)) + ((uint32_t)j & 12u)), again.zs, q);
                    tmem_st4(lane_tmem + i * 64 + j * 4, q);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            fence_proxy_async_shared();  // this thread's reads of the stage, before the copy engine refills it
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(afull(i));
                mbar_arrive(wempty(s));
            }
            if ((s += 2) >= C::W_STAGES) {
                s -= C::W_STAGES;
                wph ^= 1u;
            }
            if ((i += 2) >= ST_NA) {
                i -= ST_NA;
                aph ^= 1u;
            }
        }
    } else if (role == 4) {
        // ------------------------------ results ------------------------------
        const int quad = warp & 3;  // TMEM lanes 32 * quad ..
        const int row = quad * 32 + lane;
        const uint32_t lane_tmem = tmem + ((uint32_t)(quad * 32) << 16);
        int seg = 0, nth = 0;
        bool ok = true;
        // (behind the stores of a row block: whoever waits for it may read it)
        auto finished = [&](const StreamEntry &en, int b) {
            if (CAP == 1 || en.flags < 0) return;
            __syncwarp();
            if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.done + en.flags + b) : "memory");
        };
        for (int phase = 0; phase < phases; ++phase) {
            if (!stream_works<CAP>(t.ph[phase], id)) continue;
            ++nth;
            bool open = CAP == 1;  // results may be written
            if (CAP > 1) ok = ok && stream_gate(gates, 2 * nth - 1, abort_flag);
            auto opens = [&]() {
                if (!open) ok = stream_gate(gates, 2 * nth, abort_flag);
                open = true;
                return ok;
            };
            for_segments(t, phase, id, [&](const Segment &g) {
                const int d = seg & 1;
                const StreamEntry &en = t.e[g.e];
                const int n = g.b * 128 + row;
                const bool in = g.b * 128 + quad * 32 < en.N;  // N is a multiple of 64: the last row block may be half
                unsigned long long *slot = a.slots + slot_of(a, g, g.self) + row * 2;
                ok = __all_sync(0xffffffffu, ok && stream_wait(dfull(d), (uint32_t)(seg >> 1) & 1u, abort_flag));
                if (!ok) return false;
                ++seg;
                if (g.members == 1 && !opens()) return false;
                tc_fence_after();
                if (g.members == 1) {
                    // (eight rows at a time are no faster in a chain, and more code)
                    constexpr int ROWS = CAP == 1 ? 8 : 4;
#pragma unroll 1
                    for (int m0 = 0; m0 < a.M; m0 += ROWS) {
                        uint32_t r[ROWS];
                        if constexpr (ROWS == 8) tmem_ld8(lane_tmem + d * NB + m0, r);
                        else tmem_ld4(lane_tmem + d * NB + m0, r);
                        tmem_wait_ld();
                        if (!in) continue;
                        float v[ROWS];
#pragma unroll
                        for (int j = 0; j < ROWS; ++j) v[j] = __uint_as_float(r[j]);
                        uint2 add[ROWS / 2];
                        const StreamOut at = stream_out(en, n, m0);
                        if (en.epilogue == QF_EPI_RESIDUAL_ADD) stream_residual<ROWS / 2>(en, a.M, at, add);
                        stream_emit<ROWS / 2>(en, a.M, n, m0, v, at, add);
                    }
                } else {
#pragma unroll 1
                    for (int m0 = 0; m0 < a.M; m0 += 16, slot += 16 * 128) {
                        uint32_t r[16];
                        tmem_ld16(lane_tmem + d * NB + m0, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; j += 2)
                            if (in && m0 + j < a.M) st_words2(slot + j * 128, word_of(r[j]), word_of(r[j + 1]));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(dempty(d));
                if (g.members == 1) finished(en, g.b);
                return true;
            });
            // The members of a shared row block finish its pairs of batch rows in turn.
            for_segments(t, phase, id, [&](const Segment &g) {
                const StreamEntry &en = t.e[g.e];
                const int pairs = (a.M + 1) >> 1, first = g.members - 1 - g.self;
                if (!ok || g.members == 1 || first >= pairs) return ok;
                if (g.b * 128 + quad * 32 < en.N) {
#pragma unroll 1
                    for (int pair = first; pair < pairs; pair += g.members) {
                        float v[2];
                        uint2 add[1];
                        const StreamOut at = stream_out(en, g.b * 128 + row, 2 * pair);
                        const bool adds = en.epilogue == QF_EPI_RESIDUAL_ADD;
                        // what is added is on its way while the sums are awaited, where it is known to be there
                        if (!open && __all_sync(0xffffffffu, *gates >= 2 * nth) && !opens()) return false;
                        const bool early = open;
                        if (early && adds) stream_residual<1>(en, a.M, at, add);
                        ok = CAP > 1 || g.members <= 4 ? stream_sum<4>(a, g, pair, row, v, abort_flag) : stream_sum<8>(a, g, pair, row, v, abort_flag);
                        if (!ok) {
                            *abort_flag = 1;
                            return false;
                        }
                        if (!early) {
                            if (!opens()) return false;
                            if (adds) stream_residual<1>(en, a.M, at, add);
                        }
                        stream_emit<1>(en, a.M, g.b * 128 + row, 2 * pair, v, at, add);
                    }
                }
                finished(en, g.b);
                return true;
            });
            if (CAP > 1) {
                // a phase that is complete says that those are that it waits for, also where this stream had no result to write
                if (ok) opens();
                __syncwarp();
                if (t.ph[phase].awaited && lane == 0 && ok && stream_last_warp(&s_finished[half][nth & 3]))
                    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.done + phase) : "memory");
            }
        }
        if (CAP > 1 && a.words > 0) {
            // The last result warp of the launch leaves the counters as they were: behind everybody's last count and wait. (Where
            // nothing waits for a phase it is not counted, and a launch without counts ends without this: a release behind stores takes
            // 1 us. Two of 4096 x 4096 side by side at 9 rows 14.9 -> 13.8 us, four of 512 x 512 8.7 -> 7.3.)
            unsigned before = 0;
            if (lane == 0 && ok)
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(a.done + kStreamMaxLinears) : "memory");
            if (__shfl_sync(0xffffffffu, before + 1u, 0) == 8u * gridDim.x && __all_sync(0xffffffffu, ok)) {
                __syncwarp();
                for (int q = lane * 4; q < a.words; q += 128) *reinterpret_cast<uint4 *>(a.done + q) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    }

    // ------------------------------ teardown ------------------------------
    tc_fence_before();
    __syncthreads();
    if (s_abort) {
        // this block's own copies, before its shared memory goes away
        int dummy = 0;
        volatile int *no_abort = &dummy;
        if (role == 1)
            for (int it = max(0, issued - C::W_STAGES); it < issued; ++it)
                stream_wait(wfull(it % C::W_STAGES), (uint32_t)(it / C::W_STAGES) & 1u, no_abort);
        if (role == 2)
            for (int it = max(0, issued - C::X_STAGES); it < issued; ++it)
                stream_wait(xfull(it % C::X_STAGES), (uint32_t)(it / C::X_STAGES) & 1u, no_abort);
        if (threadIdx.x == 0) atomicExch(a.status, QF_ERR_TIMEOUT);
        __syncthreads();
    }
    if (warp == 10 && half == 0) {
        tc_fence_after();
        tmem_dealloc<false>(tmem, 2 * ST_TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
template <bool BF16, int NB, int CAP>
static cudaError_t stream_set_attr() {
    cudaError_t e = cudaFuncSetAttribute(stream_kernel<BF16, NB, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (stream_smem_bytes<NB, CAP>()));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(stream_kernel<BF16, NB, CAP>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    return e;
}

int stream_init(qf_ctx *ctx) {
    QF_CUDA_TRY(ctx, (stream_set_attr<false, 16, 1>()));
    QF_CUDA_TRY(ctx, (stream_set_attr<false, 32, 1>()));
    QF_CUDA_TRY(ctx, (stream_set_attr<true, 16, 1>()));
    QF_CUDA_TRY(ctx, (stream_set_attr<true, 32, 1>()));
    QF_CUDA_TRY(ctx, (stream_set_attr<false, 16, kStreamMaxLinears>()));
    QF_CUDA_TRY(ctx, (stream_set_attr<false, 32, kStreamMaxLinears>()));
    QF_CUDA_TRY(ctx, (stream_set_attr<true, 16, kStreamMaxLinears>()));
    QF_CUDA_TRY(ctx, (stream_set_attr<true, 32, kStreamMaxLinears>()));
    return QF_OK;
}

static size_t slot_words(int64_t M) { return (size_t)((M + 1) / 2) * 2 * 128; }

size_t stream_workspace_bytes(int64_t M, int slots) { return (size_t)slots * slot_words(M) * sizeof(unsigned long long); }

template <bool BF16, int NB, int CAP>
static cudaError_t stream_go(const StreamParams<CAP> &p, int grid, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(ST_THREADS);
    cfg.dynamicSmemBytes = (stream_smem_bytes<NB, CAP>());
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.numAttrs = 1;
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, stream_kernel<BF16, NB, CAP>, p);
}

template <int CAP>
static cudaError_t stream_dispatch(const StreamParams<CAP> &p, bool bf16, int grid, cudaStream_t s) {
    if (p.a.M <= 16) return bf16 ? stream_go<true, 16, CAP>(p, grid, s) : stream_go<false, 16, CAP>(p, grid, s);
    return bf16 ? stream_go<true, 32, CAP>(p, grid, s) : stream_go<false, 32, CAP>(p, grid, s);
}

template <int CAP>
static int stream_launch(qf_ctx *ctx, const StreamLinear *l, int count, void *ws, size_t counter_bytes, int slots, cudaStream_t s) {
    StreamParams<CAP> p;
    const qf_linear_desc &d0 = *l[0].d;
    p.a.slots = (unsigned long long *)((char *)ws + counter_bytes);
    p.a.done = (unsigned *)ws;
    p.a.status = ctx->dev_status;
    p.a.slot_words = (int)slot_words(d0.M);
    p.a.M = (int)d0.M;
    p.a.x_rows = (int)((d0.M + 7) / 8) * 8;
    p.a.words = 0;
    const void *x_of[StreamParams<CAP>::XCAP];
    int64_t x_k[StreamParams<CAP>::XCAP];
    int maps = 0, phases = 0, next = 0;
    // The linear at `i` becomes the next entry, of the phase at hand.
    auto enter = [&](int i) {
        const qf_linear_desc &d = *l[i].d;
        StreamPhase &ph = p.ph[phases - 1];
        StreamEntry &e = p.e[next];
        e.Y = l[i].Y;
        e.residual = l[i].residual;
        e.N = (int)d.N;
        e.chunks = (int)(d.K / 128);
        e.split = l[i].split;
        e.per = l[i].per;
        e.slot = 0;
        e.begin = ph.pieces;
        e.end = ph.pieces += (int)row_blocks(d) * (CAP == 1 ? e.chunks : e.split);
        e.out_dtype = (int16_t)d.out_dtype;
        e.epilogue = (int16_t)d.epilogue;
        int st = get_slab_map(ctx, &p.w[next++], l[i].blob, (uint64_t)(d.N / 64), (uint64_t)e.chunks);
        if (st != QF_OK) return st;
        e.x_from = kXThere;
        e.flags = -1;
        e.x_want = e.x_two = 0;
        e.x_map = 0;
        while (e.x_map < maps && !(x_of[e.x_map] == l[i].X && x_k[e.x_map] == d.K)) ++e.x_map;
        if (e.x_map == maps) {
            x_of[maps] = l[i].X;
            x_k[maps] = d.K;
            st = get_tensor_map(ctx, &p.x[maps++], l[i].X, 1, (uint64_t)d.K, (uint64_t)d.M, 64, (uint32_t)p.a.x_rows,
                                CU_TENSOR_MAP_SWIZZLE_128B);
        }
        return st;
    };
    const int sms = std::min(ctx->sm_count, kSmCount);
    int grid = 1;
    if (CAP == 1) {
        p.ph[phases++] = StreamPhase{0, 0, 0, 0, 0, 0, 0, 0, {-1, -1}, -1, 0};
        const int st = enter(0);
        if (st != QF_OK) return st;
        StreamPhase &ph = p.ph[0];
        grid = std::min(sms, (ph.pieces + 1) / 2);
        ph.streams = 2 * grid;
        ph.q = ph.pieces / ph.streams;
        ph.r = ph.pieces % ph.streams;
        ph.pieces = 0;
    } else {
        grid = sms;
        ChainPlan plan;
        plan_stream_chain(l, count, 2 * grid, slots, &plan);
        std::vector<int> entry_of(count);
        for (const ChainPhase &c : plan.phases) {
            StreamPhase &ph = p.ph[phases++];
            ph = StreamPhase{next, 0, 0, 0, c.streams, c.home, c.flip, 0, {c.wait[0], c.wait[1]}, c.slots_wait, 0};
            for (int w : {c.wait[0], c.wait[1], c.slots_wait})
                if (w >= 0) p.ph[w].awaited = 1, p.a.words = std::max(p.a.words, kStreamFlags);
            for (int k = c.first; k < c.first + c.count; ++k) {
                const int st = enter(plan.order[k]);
                if (st != QF_OK) return st;
                p.e[next - 1].slot = plan.linears[plan.order[k]].slot;
                entry_of[plan.order[k]] = next - 1;
            }
            ph.active = std::min(ph.pieces, ph.streams);
        }
        for (int i = 0; i < count; ++i) {
            const ChainLinear &at = plan.linears[i];
            StreamEntry &e = p.e[entry_of[i]];
            e.x_from = at.maker == kChainThere ? kXThere : kXGate;
            if (at.maker < 0 || plan.linears[at.maker].flags < 0) continue;
            const StreamLinear &from = l[at.maker];
            e.x_from = kStreamFlags + plan.linears[at.maker].flags;
            e.x_two = from.d->epilogue == QF_EPI_SILU_MUL;
            // the warps of the members that finish a pair of batch rows
            e.x_want = (int16_t)(4 * std::min<int64_t>(from.split, (d0.M + 1) / 2));
        }
        for (int i = 0; i < count; ++i)
            if (plan.linears[i].flags >= 0) {
                p.e[entry_of[i]].flags = kStreamFlags + plan.linears[i].flags;
                p.a.words = std::max(p.a.words, kStreamFlags + plan.linears[i].flags + (int)row_blocks(*l[i].d));
            }
    }
    p.a.phases = phases;
    p.a.linears = count;
    const cudaError_t e = stream_dispatch<CAP>(p, d0.act_dtype == QF_BF16, grid, s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return kStreamNoRoom;
    }
    return launched(ctx, e, "streaming linear");
}

int launch_stream(qf_ctx *ctx, const StreamLinear &l, void *ws, size_t counter_bytes, cudaStream_t s) {
    return stream_launch<1>(ctx, &l, 1, ws, counter_bytes, kStreamSlots, s);
}

int launch_stream_chain(qf_ctx *ctx, const StreamLinear *l, int count, void *ws, size_t counter_bytes, int slots, cudaStream_t s) {
    return stream_launch<kStreamMaxLinears>(ctx, l, count, ws, counter_bytes, slots, s);
}

}  // namespace qf

// Host interface of the streaming tcgen05 kernel on QF_LAYOUT_GEMV_SLAB weights (qf_stream.cu), of the chains of up to 8 rows
// (qf_slab_chain.cu) and of the planner of both (qf_chain_plan.cu).
#pragma once

#include <vector>

#include "qf_chain_index.cuh"
#include "qf_common.cuh"

namespace qf {

constexpr int kStreamMaxLinears = 112;  // of one launch: the tensor maps travel as kernel parameters (32 764 bytes)
constexpr int kStreamMaxX = 16;         // different activations of one launch, likewise
// Slots of partial sums: two for each of the two streams of an SM. A chain gets more where the workspace has room for them, so that those of
// neighbouring steps fit side by side: a step exchanges its sums before the one before is complete, and late linears may be late (32
// layers of seven linears, 4096 / 14336, 16 rows: 1564 us instead of 1675).
constexpr int kStreamSlots = 4 * kSmCount, kChainSlots = 6 * kSmCount;

// A checked linear on slab weights. In a chain K is cut into `split` pieces of `per` chunks of 128 codes.
struct StreamLinear {
    const qf_linear_desc *d;
    const void *X, *blob, *residual;
    void *Y;
    int split, per;
};

// Steps of a chain: linears that do not touch each other's results, each step behind the one before. Of a step only what the next
// one touches holds that up; the rest ("late") is a phase of its own, which the step after the next waits for.
struct ChainPhase {
    int first, count;  // of the order
    int wait[2];       // phases that are complete before this one writes its results (or -1)
    int slots_wait;    // the phase that, with wait[1], is complete before this one writes partial sums (or -1)
    int step;
    bool late;
    int64_t room;      // of the whole step
    int next0, next1;  // the linears of the next step
    int home, streams, flip;  // more than kSlabGemvRows rows: the streams from `home` on that its pieces are dealt to, backwards first
};
// room[i]: what linear i needs of something that a step has room_step of, and a step with late linears and the next one together
// room_two.
void chain_phases(const StreamLinear *l, int count, const int64_t *room, int64_t room_step, int64_t room_two, std::vector<int> *order,
                  std::vector<ChainPhase> *phases);

// What a linear of a chain gets.
struct ChainLinear {
    int slot, slots;  // of partial sums
    // more than kSlabGemvRows rows: the linear whose results are this one's activations, row block for chunk, or kChainThere (no linear
    // of the launch writes them) or kChainMixed; and the first of this linear's row block counters (-1: nobody looks at them)
    int maker, flags;
    // up to kSlabGemvRows rows: thread blocks, those of an SM, and where they are (see sc_number)
    int grid, per_sm, home, first_sm;
};
constexpr int kChainThere = -1, kChainMixed = -2;
constexpr int kStreamFlagWords = 16384 - 128;  // counters of row blocks of one launch
struct ChainPlan {
    std::vector<int> order;  // the linears, phase by phase
    std::vector<ChainPhase> phases;
    std::vector<ChainLinear> linears;
};
inline int64_t row_blocks(const qf_linear_desc &d) { return (d.N + 127) / 128; }
void plan_stream_chain(const StreamLinear *l, int count, int streams, int slots, ChainPlan *plan);
// false: more thread blocks than the SMs have places for.
bool plan_slab_chain(const StreamLinear *l, int count, int sms, ChainPlan *plan);

// Returned by the launches where the current context has fewer SMs than the device (a partition of it), so that the blocks of a
// cooperative launch do not fit: nothing was launched, and the other kernels serve.
constexpr int kStreamNoRoom = 1;

int stream_init(qf_ctx *ctx);
// Bytes behind the counter region of the workspace, for linears of M rows.
size_t stream_workspace_bytes(int64_t M, int slots = kStreamSlots);
int launch_stream(qf_ctx *ctx, const StreamLinear &l, void *ws, size_t counter_bytes, cudaStream_t s);
// How many of the linears from the first on one launch can take: the same rows and activation type, weights that no earlier one
// writes.
int stream_chain_length(const StreamLinear *l, int count);
// Whether one launch is the faster way.
bool stream_chain_pays(const StreamLinear *l, int count);
// Linears of one launch, each seeing the results of the earlier ones.
int launch_stream_chain(qf_ctx *ctx, const StreamLinear *l, int count, void *ws, size_t counter_bytes, int slots, cudaStream_t s);

// The same for linears of up to kSlabGemvRows rows, with the arithmetic of the streaming GEMV kernel (qf_slab_chain.cu).
int slab_chain_init(qf_ctx *ctx);
bool slab_chain_takes(const qf_linear_desc *d);
// Whether one launch is the faster way.
bool slab_chain_pays(const StreamLinear *l, int count);
size_t slab_chain_workspace_bytes();
int launch_slab_chain(qf_ctx *ctx, const StreamLinear *l, int count, void *ws, size_t counter_bytes, cudaStream_t s);

}  // namespace qf

// K2c: chains of linears of up to 8 rows on QF_LAYOUT_GEMV_SLAB weights in one launch, with the arithmetic of the streaming GEMV kernel
// (qf_gemv_slab.cu) and its division of work: the same units to the same numbers of thread blocks, the same partial sums added in the
// same order, so the results are the bits of the linears launched one by one.
//
// What one launch saves. Behind one another the linears of a layer stack each pay for a kernel boundary, the fetch of the activations
// and the start of the weight stream, 3 to 5 us a linear that their bytes do not explain. Here the thread blocks stay: a block goes from
// its share of one linear to its share of the next, its ring of weight copies runs ahead across linears, and only the activations
// wait for the linears that they depend on (chain_phases): a counter per phase, which each thread block raises behind its stores
// (release) and the producers poll before they request activations (acquire). One addition per block: with one per warp the 2368
// additions to a word and the polls on it cost 1.7 us a phase (1593 us a step of 32 layers of 4096 / 14336 against 1380).
//
// What bounds it. The converters, 560 cycles for 128 x 128 weights and SM as in the streaming GEMV kernel, 27 us of the 42 of a layer of
// 4096 / 14336, and for each phase the way from the last product to the next one's first, about 4 us: partial sums to their owner,
// results, counter, activations. Linears of a step share that way, which is why layers of seven linears gain the most (x1.1 to x1.45)
// and those of four 1.06 to 1.2: a token of 32 layers of 4096 / 14336 from and to the host 1426 us -> 1339.
//
// A linear that the streaming GEMV kernel runs with G thread blocks takes G of this launch's blocks (four per SM, all resident: the
// launch is cooperative); linears of one step take different ones. Roles inside a block, the ring of pairs of units, the sharing of
// row blocks and the epilogues are those of the streaming GEMV kernel; a block's slot of partial sums belongs to one of two banks,
// used by the steps of the chain in turn.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "qf_slab.cuh"
#include "qf_stream.cuh"

namespace qf {

constexpr int SC_BLOCKS_PER_SM = kSlabChainPlaces;
constexpr int kSlabChainMax = 112;  // linears of a launch
// Words of the counter region, all zero between launches: thread blocks that have finished a phase, and everything; thread blocks
// that an SM has started; places given out among the first, second, ... of the SMs.
constexpr int SC_END = kSlabChainMax, SC_SM = 256, SC_SMS = 256, SC_PLACE = SC_SM + SC_SMS;
static_assert((SC_PLACE + SC_BLOCKS_PER_SM) * sizeof(unsigned) <= kCounterBytes, "counter region");

struct SlabChainEntry {  // one linear
    const uint8_t *blob;
    const uint16_t *X;
    void *Y;
    const void *residual;
    int64_t M, N, K;
    unsigned units, grid;  // (N / 64) * (K / 128); thread blocks it is divided among
    int chunks;            // K / 128
    unsigned slot;         // its first slot of partial sums
    int home, per_sm, first_sm;  // its thread blocks: see sc_number
    int out_dtype, epilogue;
};
struct SlabChainPhase {
    int first, count;  // entries
    int blocks;        // thread blocks that work in it
    int bank;          // of the slots
    int wait[2];       // phases that are complete before activations are read (or -1)
};
struct SlabChainParams {
    SlabChainEntry e[kSlabChainMax];
    SlabChainPhase ph[kSlabChainMax];
    unsigned long long *pairs;  // [2][blocks of the launch][4 warps][32 lanes][4] (value | token << 32), zero between launches
    unsigned *done;             // the counter region
    int *status;
    int phases, depth, m_pad;
    int64_t M;
};
static_assert(sizeof(SlabChainParams) <= 32764, "kernel parameters");

__device__ __forceinline__ unsigned sc_acquire(const unsigned *ptr) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
    return v;
}

// Whether this is the last of the block's four consumer warps to get here; it then speaks for the stores of all four.
__device__ __forceinline__ bool sc_last_warp(unsigned *done) {
    unsigned before;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(smem_u32(done)) : "memory");
    return (before & 3u) == 3u;
}

// Takes a place. The hardware hands consecutive blocks to a few SMs first, so the block's index says nothing.
__device__ __forceinline__ unsigned sc_claim(unsigned *words) {
    unsigned sm, sms;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    asm volatile("mov.u32 %0, %%nsmid;" : "=r"(sms));
    return sc_place(
        gridDim.x / SC_BLOCKS_PER_SM, sm, sms, [&] { return atomicAdd(words + SC_SM + sm % SC_SMS, 1u); },
        [&](unsigned i) { return atomicAdd(words + SC_PLACE + i, 1u); });
}

// This block's entry of a phase and its number among the entry's blocks, or -1.
__device__ __forceinline__ int sc_entry(const SlabChainParams &p, int phase, unsigned place, unsigned *v) {
    const int first = p.ph[phase].first, n = p.ph[phase].count;
    for (int e = first; e < first + n; ++e) {
        *v = sc_number(gridDim.x / SC_BLOCKS_PER_SM, p.e[e].home, p.e[e].per_sm, p.e[e].first_sm, place);
        if (*v < p.e[e].grid) return e;
    }
    return -1;
}

template <bool BF16>
__global__ void __launch_bounds__(SLAB_THREADS, SC_BLOCKS_PER_SM) slab_chain_kernel(const __grid_constant__ SlabChainParams p) {
    extern __shared__ __align__(128) uint8_t slab_smem[];
    __shared__ int s_abort;
    __shared__ unsigned s_place;  // see sc_claim
    __shared__ unsigned s_done[3];  // consumer warps that have finished a phase of either bank; everything

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const uint32_t stage_bytes = 2u * SLAB_UNIT_BYTES + (uint32_t)p.m_pad * SLAB_X_PITCH;
    const uint32_t ring = (smem_u32(slab_smem) + 127u) & ~127u;
    const uint32_t bar_base = ring + (uint32_t)p.depth * stage_bytes;
    auto full_bar = [&](int s) { return bar_base + 16u * (uint32_t)s; };
    auto empty_bar = [&](int s) { return bar_base + 16u * (uint32_t)s + 8u; };
    volatile int *abort_flag = &s_abort;

    if (tid == 0) {
        s_abort = 0;
        s_place = sc_claim(p.done);
        s_done[0] = s_done[1] = s_done[2] = 0;
        for (int s = 0; s < p.depth; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == 4) {
        // ------------------------------ producer ------------------------------
        const int M = (int)p.M;
        int s = 0, issued = 0, passed[2] = {-1, -1};
        uint32_t ph = 1u;  // parity of the consumers' previous pass over stage s (the first pass finds every stage free)
        bool ok = true;
        for (int phase = 0; phase < p.phases && ok; ++phase) {
            unsigned v;
            const int e = sc_entry(p, phase, s_place, &v);
            if (e < 0) continue;
            const unsigned units = p.e[e].units, grid = p.e[e].grid;
            const int chunks = p.e[e].chunks;
            const unsigned u0 = v * units / grid;
            const int n_units = (int)((v + 1) * units / grid - u0), n_pairs = (n_units + 1) >> 1;
            const uint8_t *src = p.e[e].blob + (size_t)u0 * SLAB_UNIT_BYTES;
            const uint16_t *row = p.e[e].X + (size_t)lane * p.e[e].K;
            auto issue_w = [&](int ip) {  // stage s, lane 0
                const uint32_t nu = (uint32_t)min(2, n_units - 2 * ip);
                bulk_load(ring + (uint32_t)s * stage_bytes, src + (size_t)ip * (2 * SLAB_UNIT_BYTES), nu * (uint32_t)SLAB_UNIT_BYTES,
                          full_bar(s));
            };
            int c = (int)(u0 % (unsigned)chunks);  // K chunk of the next pair's first unit
            // The stage's arrival comes here, behind the wait of the phase: what the consumers do behind the barrier is ordered after it.
            auto issue_x = [&](int ip, int st) {   // lanes < M
                if (lane == 0) {
                    const uint32_t nu = (uint32_t)min(2, n_units - 2 * ip);
                    mbar_arrive_expect_tx(full_bar(st), nu * ((uint32_t)SLAB_UNIT_BYTES + (uint32_t)M * 256u));
                }
                __syncwarp();
                const uint32_t dst = ring + (uint32_t)st * stage_bytes + 2u * SLAB_UNIT_BYTES + (uint32_t)lane * SLAB_X_PITCH;
                const int nu = min(2, n_units - 2 * ip);
                if (lane < M) {
                    if (nu == 2 && c + 1 < chunks) {
                        bulk_load(dst, row + (size_t)c * 128, 512u, full_bar(st));
                    } else {
                        bulk_load(dst, row + (size_t)c * 128, 256u, full_bar(st));
                        if (nu == 2) bulk_load(dst + 256u, row, 256u, full_bar(st));  // first chunk of the next row block
                    }
                }
                c += 2;
                while (c >= chunks) c -= chunks;
            };
            auto next_stage = [&]() {
                if (++s == p.depth) {
                    s = 0;
                    ph ^= 1u;
                }
            };
            // weights as far ahead as the ring goes, then the activations once they exist
            const int ahead = min(p.depth, n_pairs), s0 = s;
            int got = 0;
            for (; got < ahead; ++got) {
                if (!__all_sync(0xffffffffu, mbar_wait(empty_bar(s), ph, abort_flag))) break;
                if (lane == 0) issue_w(got);
                next_stage();
            }
            ok = got == ahead;
            if (p.ph[phase].wait[0] >= 0 || p.ph[phase].wait[1] >= 0) {
                for (int i = 0; i < 2 && ok; ++i) {
                    const int w = p.ph[phase].wait[i];
                    if (w < 0 || w == passed[i]) continue;
                    const unsigned want = (unsigned)p.ph[w].blocks;
                    const long long t0 = clock64();
                    while (!__all_sync(0xffffffffu, lane != 0 || sc_acquire(p.done + w) >= want)) {
                        __nanosleep(100);  // leaves issue slots and the counter's word to the others (0.5 to 1 % of a step)
                        if (clock64() - t0 > kWaitCycles) *abort_flag = 1;
                        if (__any_sync(0xffffffffu, *abort_flag != 0)) {
                            ok = false;
                            break;
                        }
                    }
                    passed[i] = w;
                }
                // Lane 0 has acquired the counters, and all lanes issue copies: a vote orders no memory, the barrier does. Then the
                // results, which were stored through the generic proxy, are read by the copy engine.
                __syncwarp();
                asm volatile("fence.proxy.async;" ::: "memory");
            }
            // (behind a wait that ran out as well: the stages are complete then, and can be waited for)
            __syncwarp();
            for (int i = 0, st = s0; i < got; ++i) {
                issue_x(i, st);
                if (++st == p.depth) st = 0;
            }
            issued += got;
            for (int ip = ahead; ip < n_pairs && ok; ++ip) {
                if (!__all_sync(0xffffffffu, mbar_wait(empty_bar(s), ph, abort_flag))) {
                    ok = false;
                    break;
                }
                if (lane == 0) issue_w(ip);
                __syncwarp();
                issue_x(ip, s);
                ++issued;
                next_stage();
            }
        }
        if (*abort_flag) {
            // drain this block's own copies before its shared memory goes away (the consumers stopped waiting)
            int dummy = 0;
            volatile int *no_abort = &dummy;
            for (int ip = max(0, issued - p.depth); ip < issued; ++ip)
                mbar_wait(full_bar(ip % p.depth), (uint32_t)(ip / p.depth) & 1u, no_abort);
            if (lane == 0) atomicExch(p.status, QF_ERR_TIMEOUT);
        }
        return;
    }

    // ------------------------------ consumers ------------------------------
    const int g = lane >> 2;
    const int t = lane & 3;
    int s = 0;
    uint32_t ph = 0;
    uint32_t fbar = full_bar(0);
    uint32_t wptr = ring + (uint32_t)warp * SLAB_TILE_BYTES + (uint32_t)lane * 16u;      // this lane's codes
    const uint32_t cst_off = 1024u + (uint32_t)g * 4u - (uint32_t)lane * 16u;            // -> its row's constants
    const uint32_t x_off = 2u * SLAB_UNIT_BYTES - (uint32_t)warp * SLAB_TILE_BYTES - (uint32_t)lane * 16u + (uint32_t)t * 16u +
                           (uint32_t)(g & (p.m_pad - 1)) * SLAB_X_PITCH;                 // -> its activation row
    const uint32_t ring_bytes = (uint32_t)p.depth * stage_bytes;
    const uint32_t bars_bytes = 16u * (uint32_t)p.depth;
    bool aborted = false;

#pragma unroll 1
    for (int phase = 0; phase < p.phases && !aborted; ++phase) {
        unsigned vb;
        const int e = sc_entry(p, phase, s_place, &vb);
        if (e < 0) continue;
        const int chunks = p.e[e].chunks;
        const unsigned u0 = vb * p.e[e].units / p.e[e].grid;
        const int n_units = (int)((vb + 1) * p.e[e].units / p.e[e].grid - u0);
        auto slot = [&](unsigned v) {
            return p.pairs + (size_t)(p.e[e].slot + v) * 512 + warp * 128 + lane * 4;
        };
        float acc[2][4] = {};
        float held[1][4] = {};
        bool have_held = false;
        int held_b = 0;
        int b = (int)(u0 / (unsigned)chunks), c = (int)(u0 % (unsigned)chunks), c_lo = c;
        int units_left = n_units, seg_left = min(chunks - c, n_units), seg_len = seg_left;
        auto unit = [&](auto ub) {
            constexpr int WO = decltype(ub)::value * SLAB_UNIT_BYTES;
            constexpr int XO = decltype(ub)::value * 256;
            const uint4 va = lds128_at<WO>(wptr);
            const uint4 vb4 = lds128_at<WO + 512>(wptr);
            const uint32_t cptr = wptr + cst_off;
            const ZeroScale<BF16> za = slab_consts<BF16>(lds32_at<WO>(cptr));
            const ZeroScale<BF16> zb = slab_consts<BF16>(lds32_at<WO + 32>(cptr));
            const uint32_t wa[4] = {va.x, va.y, va.z, va.w};
            const uint32_t wb[4] = {vb4.x, vb4.y, vb4.z, vb4.w};
            const uint32_t xptr = wptr + x_off;
            auto step = [&](auto jc) {
                constexpr int j = decltype(jc)::value;
                uint32_t pa[4], pb[4];
                dequant8<BF16>(wa[j], za, pa);
                dequant8<BF16>(wb[j], zb, pb);
                const uint4 xb = lds128_at<XO + j * 64>(xptr);
                mma_16816<BF16>(acc[0], pa[0], pb[0], pa[1], pb[1], xb.x, xb.y);
                mma_16816<BF16>(acc[1], pa[2], pb[2], pa[3], pb[3], xb.z, xb.w);
            };
            step(std::integral_constant<int, 0>{});
            step(std::integral_constant<int, 1>{});
            step(std::integral_constant<int, 2>{});
            step(std::integral_constant<int, 3>{});
        };
        auto end_segment = [&]() {
            c += seg_len;
            units_left -= seg_len;
            float v[1][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[0][i] = acc[0][i] + acc[1][i];
                acc[0][i] = 0.f;
                acc[1][i] = 0.f;
            }
            if (c_lo == 0 && c == chunks) {
                slab_store<1>(p.e[e], (int64_t)b * 64 + warp * 16, g, t, v);
            } else if (c == chunks) {
                // this block owns row block b (it holds the end of its K range): finished at the end of its share
#pragma unroll
                for (int i = 0; i < 4; ++i) held[0][i] = v[0][i];
                have_held = true;
                held_b = b;
            } else {
                unsigned long long *mine = slot(vb);
                st_pairs2(mine, pair_of(v[0][0]), pair_of(v[0][1]));
                st_pairs2(mine + 2, pair_of(v[0][2]), pair_of(v[0][3]));
            }
            if (c == chunks) {
                c = 0;
                ++b;
            }
            c_lo = c;
            seg_len = min(chunks - c, units_left);
            seg_left = seg_len;
        };
#pragma unroll 1
        while (units_left > 0) {
            if (!__all_sync(0xffffffffu, mbar_try_wait(fbar, ph) != 0)) {
                if (!__all_sync(0xffffffffu, mbar_wait(fbar, ph, abort_flag))) {
                    aborted = true;
                    break;
                }
            }
            unit(std::integral_constant<int, 0>{});
            if (--seg_left == 0) end_segment();
            if (units_left > 0) {  // (the last unit ends a segment; the last pair may hold one only)
                unit(std::integral_constant<int, 1>{});
                if (--seg_left == 0) end_segment();
            }
            fence_proxy_async_shared();  // the reads above, before the copy engine refills the stage
            __syncwarp();
            if (lane == 0) mbar_arrive_at<8>(fbar);
            wptr += stage_bytes;
            fbar += 16u;
            if (++s == p.depth) {
                s = 0;
                ph ^= 1u;
                wptr -= ring_bytes;
                fbar -= bars_bytes;
            }
        }
        if (aborted) break;
        if (have_held) {
            // contributors of row block held_b: the blocks from the one that holds its first unit up to this one, added in that order
            const unsigned first = (((unsigned)held_b * (unsigned)chunks + 1u) * p.e[e].grid - 1u) / p.e[e].units;
            constexpr int BATCH = 4;  // contributors whose words are in flight together
            const long long t0 = clock64();
#pragma unroll 1
            for (unsigned j0 = first; j0 < vb && !aborted; j0 += BATCH) {
                unsigned long long w[BATCH][4];
                bool need[BATCH];
#pragma unroll
                for (int q = 0; q < BATCH; ++q) need[q] = j0 + q < vb;
                while (true) {
                    bool miss = false;
#pragma unroll
                    for (int q = 0; q < BATCH; ++q)
                        if (need[q]) {
                            const unsigned long long *src = slot(j0 + q);
                            ld_pairs2(src, w[q][0], w[q][1]);
                            ld_pairs2(src + 2, w[q][2], w[q][3]);
                        }
#pragma unroll
                    for (int q = 0; q < BATCH; ++q)
                        if (need[q]) {
                            bool all = true;
#pragma unroll
                            for (int i = 0; i < 4; ++i) all = all && (uint32_t)(w[q][i] >> 32) == 1u;
                            if (all) need[q] = false;
                            else miss = true;
                        }
                    if (!__any_sync(0xffffffffu, miss)) break;
                    if (__any_sync(0xffffffffu, clock64() - t0 > kWaitCycles || *abort_flag != 0)) {
                        aborted = true;
                        break;
                    }
                }
                if (aborted) break;
#pragma unroll
                for (int q = 0; q < BATCH; ++q)
                    if (j0 + q < vb) {
                        unsigned long long *src = slot(j0 + q);
#pragma unroll
                        for (int i = 0; i < 4; ++i) held[0][i] += __uint_as_float((uint32_t)w[q][i]);
                        st_pairs2(src, 0ull, 0ull);
                        st_pairs2(src + 2, 0ull, 0ull);
                    }
            }
            if (aborted) break;
            slab_store<1>(p.e[e], (int64_t)held_b * 64 + warp * 16, g, t, held);
        }
        __syncwarp();
        // (a warp cannot be two steps ahead of another one, so phases of a bank do not mix)
        if (lane == 0 && sc_last_warp(s_done + p.ph[phase].bank))
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.done + phase) : "memory");
    }
    if (aborted) {
        if (lane == 0) {
            *abort_flag = 1;
            atomicExch(p.status, QF_ERR_TIMEOUT);
        }
        return;
    }
    if (lane == 0) {
        // the last thread block of the launch leaves the counters as they were: behind everybody's last count and wait
        if (sc_last_warp(s_done + 2)) {
            unsigned before;
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(p.done + SC_END) : "memory");
            if (before + 1u == gridDim.x) {
                for (int q = 0; q < p.phases; ++q) p.done[q] = 0u;
                p.done[SC_END] = 0u;
                for (int q = 0; q < SC_SMS + SC_BLOCKS_PER_SM; ++q) p.done[SC_SM + q] = 0u;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
static size_t sc_stage_bytes(int m_pad) { return 2 * SLAB_UNIT_BYTES + (size_t)m_pad * SLAB_X_PITCH; }
// Shared memory of a block: a quarter of the SM's.
constexpr size_t kSlabChainSmem = (228u << 10) / SC_BLOCKS_PER_SM - 1024 - 128;

int slab_chain_init(qf_ctx *ctx) {
    for (auto *fn : {slab_chain_kernel<false>, slab_chain_kernel<true>}) {
        QF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSlabChainSmem));
        QF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
    }
    return QF_OK;
}

size_t slab_chain_workspace_bytes() { return (size_t)2 * SC_BLOCKS_PER_SM * kSmCount * 512 * sizeof(unsigned long long); }

int launch_slab_chain(qf_ctx *ctx, const StreamLinear *l, int count, void *ws, size_t counter_bytes, cudaStream_t s) {
    SlabChainParams p;
    const qf_linear_desc &d0 = *l[0].d;
    const int sms = std::min(ctx->sm_count, kSmCount), blocks = SC_BLOCKS_PER_SM * sms;
    ChainPlan plan;
    if (!plan_slab_chain(l, count, sms, &plan)) return kStreamNoRoom;
    p.phases = (int)plan.phases.size();
    int next = 0;
    for (int q = 0; q < p.phases; ++q) {
        const ChainPhase &c = plan.phases[q];
        SlabChainPhase &ph = p.ph[q];
        ph = SlabChainPhase{next, c.count, 0, c.step & 1, {c.wait[0], c.wait[1]}};
        for (int k = c.first; k < c.first + c.count; ++k) {
            const StreamLinear &x = l[plan.order[k]];
            const ChainLinear &at = plan.linears[plan.order[k]];
            SlabChainEntry &e = p.e[next++];
            e.blob = (const uint8_t *)x.blob;
            e.X = (const uint16_t *)x.X;
            e.Y = x.Y;
            e.residual = x.residual;
            e.M = x.d->M;
            e.N = x.d->N;
            e.K = x.d->K;
            e.chunks = (int)(x.d->K / 128);
            e.units = (unsigned)(x.d->N / 64 * e.chunks);
            e.grid = (unsigned)at.grid;
            e.home = at.home;
            e.out_dtype = x.d->out_dtype;
            e.epilogue = x.d->epilogue;
            e.per_sm = at.per_sm;
            e.first_sm = at.first_sm;
            e.slot = (unsigned)at.slot;
            ph.blocks += at.grid;
        }
    }
    p.pairs = (unsigned long long *)((char *)ws + counter_bytes);
    p.done = (unsigned *)ws;
    p.status = ctx->dev_status;
    p.M = d0.M;
    p.m_pad = slab_m_pad(d0.M);
    // (as deep as the streaming GEMV kernel's: 4 and 6 measured equal or up to 2 % slower)
    p.depth = (int)std::min<size_t>(3, (kSlabChainSmem - 128) / (sc_stage_bytes(p.m_pad) + 16));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(SLAB_THREADS);
    cfg.dynamicSmemBytes = kSlabChainSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = d0.act_dtype == QF_BF16 ? cudaLaunchKernelEx(&cfg, slab_chain_kernel<true>, p)
                                                  : cudaLaunchKernelEx(&cfg, slab_chain_kernel<false>, p);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return kStreamNoRoom;
    }
    return launched(ctx, e, "chain of slab GEMVs");
}

// Measured, us a step of the linears of a decoder stack (16 layers where not said, one row, linear by linear -> chain; hidden / ffn):
//   7 linears a layer, in 4 steps (q k v, o, gate up, down); MB of codes a linear
//     0.8 (1024 / 2816) 459 -> 340   3.2 (2048 / 5632) 605 -> 418   7.0 (3072 / 8192) 728 -> 559   15.6 (4096 / 14336) 898 -> 822
//     14.5 (4096 / 11008) 882 -> 795   28 (4864 / 23296) 1158 -> 1105   25 (7168 / 11264, 10 layers) 725 -> 748   25 (8192 / 8192, 8) 573 -> 586
//   4 linears one behind the other (qkv, o, gate+up, down)
//     none above 16 MB, some small enough for one block per SM: 1024 / 2816 284 -> 267, 2048 / 5632 415 -> 338; none that small:
//     2816 / 3840 351 -> 342, 4096 / 2048 360 -> 362, 5120 / 2048 400 -> 406 (two blocks per SM leave room for the next kernel's)
//     one in four above 16 MB: 3072 / 8192 492 -> 431, 1024 / 28672 476 -> 466
//     two: 4096 / 14336 704 -> 663, 1792 / 23040 580 -> 553, 5120 / 13824 (12 layers) 595 -> 569; but 6656 / 2304 (qkv and o) 562 -> 586
//     more: 5888 / 6400 646 -> 674; above 80 MB: 4096 / 24576 (12 layers) 683 -> 683, 8192 / 28672 (6) 675 -> 738
// (In these o stands beside qkv, which it does not read here: 4 linears in 3 steps.) Linears of which each waits for the one before it
// gain nothing: a step of a chain takes longer than a launch that may begin beside its predecessor. 16 in a row, one / eight rows:
//   1024 x 2816 69 -> 88 / 75 -> 94, 2048 x 5632 87 -> 104 / 94 -> 112, 4096 x 14336 187 -> 197 / 204 -> 204; 8 layers of 4 with o behind
//   qkv: 1024 / 2816 143 -> 167 / 154 -> 179, 2048 / 5632 205 -> 203 / 220 -> 217, 4096 / 14336 350 -> 372 / 387 -> 390
// At 8 rows the chain gains 2 to 7 points more. One or two layers pay for the start of the launch (4 us): 1024 / 2816, 4 linears 21 -> 23,
// 4096 / 14336 46 -> 49; 8 linears 36 -> 39, 90 -> 90; 7 linears of 7.0 MB 47 -> 40, of 15.6 MB 59 -> 59. The line is drawn between these.
bool slab_chain_pays(const StreamLinear *l, int count) {
    const std::vector<int64_t> any(count, 0);
    std::vector<int> order;
    std::vector<ChainPhase> chain;
    chain_phases(l, count, any.data(), 1, 1, &order, &chain);
    const int steps = chain.back().step + 1;
    if (steps == count) return false;
    double sum = 0, most = 0;
    int large = 0;
    for (int i = 0; i < count; ++i) {
        const double bytes = 0.5 * (double)l[i].d->N * (double)l[i].d->K;
        sum += bytes;
        most = std::max(most, bytes);
        large += bytes * QF_SLAB_UNIT_BYTES / 4096 > (double)kSlabSmallBytes;
    }
    const double mean = sum / count;
    const bool wide = 2 * count >= 3 * steps && mean <= 18e6;
    if (wide ? count < 7 || (count < 14 && mean > 8e6) : count < 8 || (count < 16 && (mean < 4e6 || mean > 16e6))) return false;
    if (!wide && large > 0 && (2 * large > count || most > 80e6 || (4 * large > count && most < 1.7 * mean))) return false;
    // (thread blocks are looked at last: a linear's number of them takes longer to find than all of the above)
    ChainPlan plan;
    if (!plan_slab_chain(l, count, kSmCount, &plan) || plan.phases.back().step + 1 == count) return false;
    bool small = wide || large > 0 || mean <= 7e6;
    for (const ChainLinear &x : plan.linears) small = small || x.grid <= kSmCount;
    return small;
}

bool slab_chain_takes(const qf_linear_desc *d) {
    // From 160 MiB on a linear goes by itself, so that its size does not speak for those around it (slab_chain_pays). That also keeps
    // units times blocks within 32 bits.
    static_assert((160ull << 20) / QF_SLAB_UNIT_BYTES * (SC_BLOCKS_PER_SM * kSmCount + 1) <= UINT32_MAX, "share arithmetic");
    return d->M <= kSlabGemvRows && (d->N / 64) * (d->K / 128) <= (160 << 20) / QF_SLAB_UNIT_BYTES;
}

}  // namespace qf

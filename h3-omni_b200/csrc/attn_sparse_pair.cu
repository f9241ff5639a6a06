// Block-sparse attention forward for video sparse attention (tcgen05 + TMEM + TMA), bf16, head
// dim 128: the fine stage behind h3_vsa_hopper (replaces fwd_attend_ker<128>,
// cuda/vendor/vsa_hopper_forward.cuh:68-270 of the reference).
//
// One item of work is a pair of adjacent 64-row query tiles: 128 query rows on the M axis of every
// MMA. It walks the sorted union of the two lists, one 64-key tile per step,
//      S[128 x 64] = Q . K^T      (A = Q from TMEM, B = K tile from shared memory)
//      O[128 x 128] += P . V      (A = P from TMEM, B = V tile from shared memory, MN-major)
// and a half that did not select a tile contributes zero weights without taking an exponential.
//
// What bounds it, per step: 512 cycles of tensor pipe (eight N = 64 and four N = 128 MMAs), 64 KB
// through the SM's shared-memory port (32 KB of fills, 32 KB of operand reads) = 512 cycles, and 32 KB
// from L2. Q in TMEM is what keeps the first two at that: with Q in shared memory the eight N = 64 MMAs
// take 431 cycles instead of 305, and the kernels that did so (one per pair of tiles with Q in shared
// memory; one with the keys on the M axis that walked each tile's own list) took 990 cycles per union
// tile and 692 per list entry.
//
// Four score tiles are in flight, so neither the softmax nor the tensor pipe waits for the other's
// round trip (S ready -> P -> PV done -> next S takes about 2000 cycles). TMEM, 512 columns: O 128,
// S/P four times 64, Q twice 64 (the next item's Q is put there while this one runs).
//
// One warp issues all MMAs, step after step and across items: PV(g), then QK(g + 4) into the score tile
// that PV(g) has just read. In that order nothing but P(g) has to be waited for: the loads come as units of
// {K of step g + 4, V of step g}, and a watcher warp adds its arrival to P(g)'s barrier when unit g has
// landed. A step takes 890 to 1010 cycles: the issuing warp's own time (205 for the four PV MMAs, 470 for the eight
// QK MMAs beside busy softmax warps, 100 for the probe, 170 around them) is the bound now. With a warp for QK and
// one for PV a step took 976 to 1060.
// 287 tiles x 56 heads, neighbouring lists that join to 67 % of their entries: 1.62 ms; a whole call 2354 us, with the
// single kernel 2626.
//
// Softmax: two groups of four warps take alternate steps, one thread per query row. Online maxima would
// tie the groups together, so a row keeps ONE exponent reference: its largest score in the item's first
// tile. Any reference gives the exact softmax as long as nothing over- or underflows: a row whose sum
// leaves [2^-60, 2^100) (or is not finite) puts its query tile on the `redo` list, and the launcher recomputes
// listed tiles with the running-maximum kernel of attn_tc5.cu. The sums add the bf16-rounded weights the
// PV product uses, so numerator and denominator agree; the logsumexp is of the weights as they were.
//
// Persistent kernel, one CTA per SM, 16 warps:
//   warps 0-3 / 4-7 : softmax groups; group g takes the steps whose running number is g mod 2
//   warp 8          : TMA issue
//   warp 9          : MMA issue
//   warp 10         : scheduler: takes a ticket, merges the pair's two lists into the walk
//   warp 11         : watcher of the loads
//   warps 12-15     : Q of the next item into TMEM; O / l -> bf16 rows in global memory
// A walk has at least four steps (shorter ones are padded with steps that nobody selected): the loads and
// the QK products then reach at most one item ahead of the PV products, and an item's buffers are
// published once the item two before it is over.
// Tickets go to the long lists first (prefix tiles attend everything: one such walk is as long as
// several others, and started last it would run alone), then head by head.
// Every wait is bounded and ends in the device status word.
#include <cuda.h>

#include "softmax_tc5.cuh"
#include "sparse_choice.cuh"

namespace h3b {
namespace {

constexpr int SP_THREADS = 512;
constexpr int SP_SOFTMAX_REGS = 144, SP_ISSUE_REGS = 80, SP_EPILOGUE_REGS = 144;
static_assert(SP_SOFTMAX_REGS * 256 + SP_ISSUE_REGS * 128 + SP_EPILOGUE_REGS * 128 <= 65536, "register file");
constexpr int SP_TILE = 64 * 128 * 2;      // one K or V tile: two 64-dim halves of [64 rows][128 B]
constexpr int SP_HALF = 64 * 128;
constexpr int SP_AHEAD = 4;                // score tiles; steps that QK runs ahead of PV
constexpr int SP_SLOTS = 6;                // units of a K and a V tile
constexpr int SP_MAX_TILES = 4096;
constexpr int SP_OFF_WALK = SP_SLOTS * 2 * SP_TILE;                 // [2][SP_MAX_TILES] 16-bit steps
constexpr int SP_OFF_VALID = SP_OFF_WALK + 2 * SP_MAX_TILES * 2;    // [2][SP_MAX_TILES] their valid keys
constexpr int SP_SMEM = SP_OFF_VALID + 2 * SP_MAX_TILES + 1024;
constexpr int SP_O_COL = 0, SP_S_COL = 128, SP_Q_COL = 384;

// A step of a walk: tile number, and which halves selected the tile.
__device__ __forceinline__ uint16_t walk_word(int tile, uint32_t halves) { return (uint16_t)(tile | halves << 12); }
__device__ __forceinline__ int walk_tile(uint16_t w) { return w & 0xfff; }

struct SparsePairParams {
    const int *indices, *counts, *sizes;
    const uint4 *q;
    __nv_bfloat16 *out;
    float *lse;
    SparseWork work;
    int *status;
    int tiles, heads, force_redo;
    float scale_log2;
};

struct Item {
    int head, pair, n, empty;      // n = steps (at least four), n < 0: no more work; empty: bit per half with an empty list
};

// Sums for the choice between the kernels (sparse_choice.cuh), and the list of long pairs: those whose lists
// together hold more than half of what they could. A warp per pair, eight pairs of a head per block; both lists ascending.
__global__ void __launch_bounds__(256)
sparse_sums_kernel(const int *indices, const int *counts, const SparseWork work, int tiles) {
    wait_for_previous_kernel();
    allow_next_kernel();
    __shared__ uint32_t bits[8][SP_MAX_TILES / 32];
    __shared__ unsigned sums[2][8];   // entries and entries left, of each warp's pair
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pairs = (tiles + 1) / 2;
    const int pair = blockIdx.x * 8 + warp, head = blockIdx.y;
    int entries = 0, joined = 0;
    if (pair < pairs) {
        const int qa = 2 * pair, qb = qa + 1;
        const size_t row = (size_t)head * tiles + qa;
        const int na = max(0, min(counts[row], tiles)), nb = qb < tiles ? max(0, min(counts[row + 1], tiles)) : 0;
        for (int w = lane; w < SP_MAX_TILES / 32; w += 32) bits[warp][w] = 0u;
        __syncwarp();
        for (int i = lane; i < na; i += 32) {
            const int kt = indices[row * tiles + i];
            if (kt >= 0 && kt < tiles) atomicOr(&bits[warp][kt >> 5], 1u << (kt & 31));
        }
        __syncwarp();
        int common = 0;
        for (int i = lane; i < nb; i += 32) {
            const int kt = indices[(row + 1) * tiles + i];
            if (kt >= 0 && kt < tiles) common += (bits[warp][kt >> 5] >> (kt & 31)) & 1u;
        }
        entries = na + nb;
        joined = entries - __reduce_add_sync(0xffffffffu, common);
        if (lane == 0 && entries > tiles)
            work.long_pairs[atomicAdd(work.counters + SparseWork::LONG, 1u)] = (unsigned)(head * pairs + pair);
    }
    if (lane == 0) {
        sums[0][warp] = (unsigned)entries;
        sums[1][warp] = (unsigned)joined;
    }
    __syncthreads();
    if (warp == 0) {   // the block's eight pairs lie in one word of the head's set
        const unsigned e = lane < 8 ? sums[0][lane] : 0u, u = lane < 8 ? sums[1][lane] : 0u;
        const bool joins = pair_joins(e, u);
        const unsigned joining = __ballot_sync(0xffffffffu, joins);
        const unsigned all_e = __reduce_add_sync(0xffffffffu, e), all_u = __reduce_add_sync(0xffffffffu, u);
        const unsigned own_e = __reduce_add_sync(0xffffffffu, joins ? e : 0u), own_u = __reduce_add_sync(0xffffffffu, joins ? u : 0u);
        SparseWork::HeadSums *total = work.head_sums + head;
        if (lane == 0) atomicAdd(&total->entries, all_e);
        if (lane == 1) atomicAdd(&total->joined, all_u);
        if (lane == 2) atomicAdd(&total->entries_joining, own_e);
        if (lane == 3) atomicAdd(&total->joined_joining, own_u);
        if (lane == 4) atomicAdd(&total->joining, (unsigned)__popc(joining));
        if (lane == 5)
            atomicOr(work.pair_sets + (size_t)head * SparseWork::words(tiles) + (blockIdx.x >> 2), joining << (blockIdx.x % 4 * 8));
    }
}

// LSE: the logsumexp is wanted as well (2 % of a call for the sums it is of).
template <bool LSE>
__global__ void __launch_bounds__(SP_THREADS, 1)
attn_sparse_pair_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const SparsePairParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bars[11 + 2 * SP_AHEAD + 2 * SP_SLOTS];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    __shared__ Item desc[2];
    __shared__ float mref[2][128], lpart[2][2][128], lexact[2][2][LSE ? 128 : 1];
    __shared__ uint32_t bits[2][SP_MAX_TILES / 32];   // scheduler: the two lists as sets

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *const base_ptr = smem_raw + (base - smem_u32(smem_raw));
    uint16_t *const walk = reinterpret_cast<uint16_t *>(base_ptr + SP_OFF_WALK);
    uint8_t *const valid_keys = base_ptr + SP_OFF_VALID;

    const uint32_t bar0 = smem_u32(bars);
    auto bar_item_ready = [&](int b) { return bar0 + 8u * (0 + b); };
    auto bar_item_free = [&](int b) { return bar0 + 8u * (2 + b); };
    auto bar_item_done = [&](int b) { return bar0 + 8u * (4 + b); };
    auto bar_q_full = [&](int b) { return bar0 + 8u * (6 + b); };
    auto bar_mref = [&](int b) { return bar0 + 8u * (8 + b); };
    const uint32_t bar_watching = bar0 + 8u * 10;   // once: the watcher has seen the units that P does not gate
    auto bar_s_full = [&](int s) { return bar0 + 8u * (11 + s); };
    auto bar_p_full = [&](int s) { return bar0 + 8u * (11 + SP_AHEAD + s); };
    auto bar_full = [&](int s) { return bar0 + 8u * (11 + 2 * SP_AHEAD + s); };
    auto bar_empty = [&](int s) { return bar0 + 8u * (11 + 2 * SP_AHEAD + SP_SLOTS + s); };

    if (tid == 0) {
        for (int b = 0; b < 2; b++) {
            mbar_init(bar_item_ready(b), 1);
            mbar_init(bar_item_free(b), 4);     // the four epilogue warps
            // the last PV and the eight softmax warps. (The other readers of an item's descriptor and walk
            // are done before: the loads and the watcher precede its last PV.)
            mbar_init(bar_item_done(b), 9);
            mbar_init(bar_q_full(b), 128);
            mbar_init(bar_mref(b), 128);
        }
        mbar_init(bar_watching, 1);
        for (int s = 0; s < SP_AHEAD; s++) {
            mbar_init(bar_s_full(s), 1);
            mbar_init(bar_p_full(s), 128 + 1);   // the softmax threads and the watcher
        }
        for (int s = 0; s < SP_SLOTS; s++) {
            mbar_init(bar_full(s), 1);
            mbar_init(bar_empty(s), 1);
        }
        mbar_fence_init();
        abort_word = 0;
    }
    if (warp == 9) {
        tmem_alloc(smem_u32(&tmem_slot), 512);
        tmem_relinquish();
    }
    wait_for_previous_kernel();
    tc5_fence_before();
    __syncthreads();
    tc5_fence_after();
    const uint32_t tmem = tmem_slot;
    if (tid == 0) allow_next_kernel();
    const int pairs = (p.tiles + 1) / 2;

    // Item `i`'s descriptor, for a whole warp: lane 0 polls (fewer probes of shared memory, which the
    // tensor core is reading its operands from).
    auto fetch_warp = [&](int i, Item &it) -> bool {
        if (!mbar_wait_uniform(bar_item_ready(i & 1), (i >> 1) & 1, &abort_word)) return false;
        it = desc[i & 1];
        return true;
    };

    if (warp >= 8 && warp < 12) {
        warpgroup_reg_dec<SP_ISSUE_REGS>();
        if (warp == 10) {
            // ------------------------------ scheduler ------------------------------
            const unsigned long_count = min(p.work.counters[SparseWork::LONG], (unsigned)(pairs * p.heads));
            unsigned head_nth = 0xffffffffu;
            int natural_head = -1;
            bool natural_split = false;
            const int words = (p.tiles + 31) / 32;
            for (int i = 0;; i++) {
                const int b = i & 1;
                if (i >= 2 && !mbar_wait_warp(bar_item_free(b), ((i >> 1) - 1) & 1, &abort_word)) break;
                int head = -1, pair = 0;
                size_t row = 0;
                bool second = false;
                for (;;) {   // the next of this kernel's pairs: the long ones, then the others in order
                    unsigned ticket = 0;
                    if (lane == 0) ticket = atomicAdd(p.work.counters + SparseWork::TICKET_PAIR, 1u);
                    ticket = __shfl_sync(0xffffffffu, ticket, 0);
                    bool split;
                    if (ticket < long_count) {
                        const unsigned id = p.work.long_pairs[ticket];
                        head = (int)(id / (unsigned)pairs);
                        pair = (int)(id % (unsigned)pairs);
                        const HeadShare share = head_share(p.work, head);
                        if (share == HeadShare::SINGLE) continue;
                        split = share == HeadShare::SPLIT;
                    } else {
                        const unsigned nth = (ticket - long_count) / (unsigned)pairs;
                        if (nth != head_nth) {
                            head_nth = nth;
                            natural_head = nth_head(p.work, p.heads, HeadShare::PAIR, nth, natural_split);
                        }
                        head = natural_head;
                        split = natural_split;
                        pair = (int)((ticket - long_count) % (unsigned)pairs);
                    }
                    if (head < 0) break;
                    if (split && !in_pair_set(p.work, p.tiles, head, pair)) continue;
                    row = (size_t)head * p.tiles + 2 * pair;
                    second = 2 * pair + 1 < p.tiles;
                    const int na = max(0, min(p.counts[row], p.tiles));
                    const int nb = second ? max(0, min(p.counts[row + 1], p.tiles)) : 0;
                    if (ticket < long_count || na + nb <= p.tiles) break;
                }
                if (head < 0) {
                    if (lane == 0) {
                        desc[b] = Item{0, 0, -1, 0};
                        mbar_arrive(bar_item_ready(b));
                    }
                    break;
                }
                const int raw_a = p.counts[row], raw_b = second ? p.counts[row + 1] : 0;
                bool bad = raw_a < 0 || raw_a > p.tiles || raw_b < 0 || raw_b > p.tiles;
                const int na = max(0, min(raw_a, p.tiles)), nb = max(0, min(raw_b, p.tiles));
                for (int w = lane; w < words; w += 32) bits[0][w] = bits[1][w] = 0u;
                __syncwarp();
                const int *list = p.indices + row * p.tiles;
                for (int half = 0; half < 2; half++) {
                    const int n = half ? nb : na;
                    for (int e = lane; e < n; e += 32) {
                        const int kt = list[(size_t)half * p.tiles + e];
                        if (kt < 0 || kt >= p.tiles) bad = true;   // refused, never dereferenced
                        else atomicOr(&bits[half][kt >> 5], 1u << (kt & 31));
                    }
                }
                __syncwarp();
                int n = 0;
                for (int w = 0; w < words; w++) {
                    const uint32_t a = bits[0][w], c = bits[1][w], both = a | c;
                    if (both >> lane & 1u) {
                        const int kt = w * 32 + lane, at = b * SP_MAX_TILES + n + __popc(both & ((1u << lane) - 1u));
                        walk[at] = walk_word(kt, (a >> lane & 1u) | (c >> lane & 1u) << 1);
                        valid_keys[at] = (uint8_t)max(0, min(p.sizes[kt], 64));
                    }
                    n += __popc(both);
                }
                for (; n < SP_AHEAD; n++) {   // padding: tile 0, selected by nobody
                    walk[b * SP_MAX_TILES + n] = walk_word(0, 0);
                    valid_keys[b * SP_MAX_TILES + n] = 0;
                }
                if (__any_sync(0xffffffffu, bad) && lane == 0) atomicCAS(p.status, STATUS_OK, STATUS_BAD_ARGUMENT);
                __syncwarp();
                if (lane == 0) {
                    desc[b] = Item{head, pair, n, (na == 0 ? 1 : 0) | (nb == 0 ? 2 : 0)};
                    mbar_arrive(bar_item_ready(b));
                }
            }
        } else if (warp == 8) {
            // ------------------------------ TMA issue ------------------------------
            // Unit u: K of running step u and V of running step u - 4, as far as they exist.
            if (lane == 0) {
                tma_prefetch_desc(&map_k);
                tma_prefetch_desc(&map_v);
                struct Cursor {
                    Item it;
                    int item, j;
                } kc{Item{0, 0, 0, 0}, -1, 0}, vc = kc;
                auto advance = [&](Cursor &c) -> bool {   // to the next step; false: waited in vain
                    if (c.it.n < 0 || ++c.j < c.it.n) return true;
                    c.item++;
                    c.j = 0;
                    if (!mbar_wait_parked(bar_item_ready(c.item & 1), (c.item >> 1) & 1, &abort_word)) return false;
                    c.it = desc[c.item & 1];
                    return true;
                };
                auto load = [&](const Cursor &c, const void *map, uint32_t dst, uint32_t bar) {
                    const int row = walk_tile(walk[(c.item & 1) * SP_MAX_TILES + c.j]) * 64;
                    tma_load_4d(dst, map, bar, 0, row, c.it.head, 0);
                    tma_load_4d(dst + SP_HALF, map, bar, 64, row, c.it.head, 0);
                };
                int slot = 0;
                uint32_t phase = 1u;   // parity the slot's "empty" barrier has to show; 1 passes on a fresh one
                for (int u = 0;; u++) {
                    if (!advance(kc) || (u >= SP_AHEAD && !advance(vc))) break;
                    const bool has_k = kc.it.n >= 0, has_v = u >= SP_AHEAD && vc.it.n >= 0;
                    if (!has_k && !has_v) break;   // all loaded
                    // Slots 0-3 are first freed by QK products that need nothing of the watcher: their second phase
                    // must not be over before it has seen the first (it would wait for a third, and P for it).
                    if (u == SP_SLOTS && !mbar_wait_parked(bar_watching, 0, &abort_word)) break;
                    if (!mbar_wait_parked(bar_empty(slot), phase, &abort_word)) break;
                    const uint32_t dst = base + slot * 2 * SP_TILE, bar = bar_full(slot);
                    mbar_arrive_expect_tx(bar, (has_k ? SP_TILE : 0) + (has_v ? SP_TILE : 0));
                    if (has_k) load(kc, &map_k, dst, bar);
                    if (has_v) load(vc, &map_v, dst + SP_TILE, bar);
                    if (++slot == SP_SLOTS) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
            }
        } else if (warp == 9) {
            // ------------------------------ MMA issue ------------------------------
            // The whole warp walks the loop and one elected lane issues: inside a one-lane branch
            // every descriptor word would be per-thread data that has to be moved to a uniform
            // register in front of each MMA.
            const bool leader = elect_one();
            constexpr uint32_t idesc_qk = mma_idesc(128, 64, 1, 0), idesc_pv = mma_idesc(128, 128, 1, 1);
            const uint64_t k_proto = smem_desc_sw128(base, 16, 1024), v_proto = smem_desc_sw128(base + SP_TILE, SP_HALF, 1024);
            const uint32_t k_lo0 = (uint32_t)k_proto, k_hi = (uint32_t)(k_proto >> 32);
            const uint32_t v_lo0 = (uint32_t)v_proto, v_hi = (uint32_t)(v_proto >> 32);
            // the step the next QK product belongs to; q_item < 0 or q_left < 0: none any more
            int q_item = -1, q_left = 0;
            auto issue_qk = [&](int s, int slot) -> bool {
                if (q_left == 0) {   // on to the next item
                    Item it;
                    if (!fetch_warp(++q_item, it)) return false;
                    q_left = it.n;
                    if (q_left >= 0 && !mbar_wait_converged(bar_q_full(q_item & 1), (q_item >> 1) & 1, &abort_word)) return false;
                    tc5_fence_after();
                }
                if (q_left > 0) {
                    q_left--;
                    const uint32_t k_lo = k_lo0 + slot * (2 * SP_TILE >> 4), d_tmem = tmem + SP_S_COL + s * 64;
                    const uint32_t q_tmem = tmem + SP_Q_COL + (q_item & 1) * 64;
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < 8; kk++)
                            mma_ts_words(d_tmem, q_tmem + kk * 8, k_lo + (kk / 4) * (SP_HALF >> 4) + (kk % 4) * 2, k_hi,
                                         idesc_qk, kk > 0);
                        mma_commit(bar_s_full(s));
                    }
                }
                if (leader) mma_commit(bar_empty(slot));
                __syncwarp();
                return true;
            };
            // (A CTA without an item leaves the ring alone, here and in the two other roles: a slot freed before the
            // load that expects it fresh would keep that load waiting.)
            int slot = 0;
            Item first;
            bool alive = fetch_warp(0, first) && first.n >= 0;
            for (int g = 0; alive && g < SP_AHEAD; g++) {   // units 0-3 hold no V; a walk has as many steps
                alive = mbar_wait_converged(bar_full(slot), 0, &abort_word);
                tc5_fence_after();
                alive = alive && issue_qk(g, slot++);
            }
            int g = 0;
            for (int i = 0; alive; i++) {
                Item it;
                const int b = i & 1;
                if (!fetch_warp(i, it) || it.n < 0) break;
                // the epilogue has taken the previous item's accumulator out of TMEM
                if (i >= 1 && !mbar_wait_converged(bar_item_free(b ^ 1), ((i - 1) >> 1) & 1, &abort_word)) break;
                for (int j = 0; j < it.n; j++, g++) {
                    const int s = g % SP_AHEAD;
                    // P of this step, and (through the watcher) its V and the K of step g + 4
                    alive = mbar_wait_converged(bar_p_full(s), (g / SP_AHEAD) & 1, &abort_word);
                    if (!alive) break;
                    tc5_fence_after();
                    const uint32_t v_lo = v_lo0 + slot * (2 * SP_TILE >> 4), p_tmem = tmem + SP_S_COL + s * 64;
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < 4; kk++)
                            mma_ts_words(tmem + SP_O_COL, p_tmem + kk * 8, v_lo + kk * (2048 >> 4), v_hi, idesc_pv,
                                         j > 0 || kk > 0);
                        if (j + 1 == it.n) mma_commit(bar_item_done(b));
                    }
                    __syncwarp();
                    alive = issue_qk(s, slot);
                    if (!alive) break;
                    if (++slot == SP_SLOTS) slot = 0;
                }
            }
        } else if (warp == 11) {
            // ------------------------------ watcher ------------------------------
            // Unit u has landed: step u - 4 may go on as far as the loads are concerned.
            if (lane == 0) {
                // (The first units, which the issuer waits for itself, are waited for here too: loads complete in
                // any order, and the wait for a slot's second phase passes while its first is still open.)
                int u = 0;
                bool ok = mbar_wait_parked(bar_item_ready(0), 0, &abort_word) && desc[0].n >= 0;
                for (; ok && u < SP_AHEAD; u++) ok = mbar_wait_parked(bar_full(u), 0, &abort_word);
                if (ok) mbar_arrive(bar_watching);
                for (int i = 0; ok; i++) {
                    if (!mbar_wait_parked(bar_item_ready(i & 1), (i >> 1) & 1, &abort_word)) break;
                    const int n = desc[i & 1].n;
                    if (n < 0) break;
                    for (int j = 0; ok && j < n; j++, u++) {
                        const int g = u - SP_AHEAD, s = g % SP_AHEAD;
                        ok = mbar_wait_parked(bar_full(u % SP_SLOTS), (u / SP_SLOTS) & 1, &abort_word);
                        // one arrival per phase: the score tile's previous step has to be over
                        if (ok && g >= SP_AHEAD) ok = mbar_wait_parked(bar_p_full(s), (g / SP_AHEAD - 1) & 1, &abort_word);
                        if (ok) mbar_arrive(bar_p_full(s));
                    }
                }
            }
        }
    } else if (warp >= 12) {
        warpgroup_reg_inc<SP_EPILOGUE_REGS>();
        // ------------------------------ Q in, O out ------------------------------
        const int r = tid - 384;   // query row of the pair == TMEM lane
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        auto load_q = [&](int i, const Item &it) {
            const int padded = it.pair * 128 + r;
            const bool real = padded < p.tiles * 64;
            const uint4 *src = p.q + ((size_t)it.head * p.tiles * 64 + (real ? padded : 0)) * 16;
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint32_t v[32];
#pragma unroll
                for (int x = 0; x < 8; x++) {
                    const uint4 w = real ? src[c * 8 + x] : make_uint4(0u, 0u, 0u, 0u);
                    v[4 * x] = w.x;
                    v[4 * x + 1] = w.y;
                    v[4 * x + 2] = w.z;
                    v[4 * x + 3] = w.w;
                }
                tmem_st32(tmem + lane_base + SP_Q_COL + (i & 1) * 64 + c * 32, v);
            }
            tmem_wait_st();
            tc5_fence_before();
            mbar_arrive(bar_q_full(i & 1));
        };
        Item it, next;
        bool alive = fetch_warp(0, it);
        if (alive && it.n >= 0) load_q(0, it);
        for (int i = 0; alive && it.n >= 0; i++, it = next) {
            const int b = i & 1;
            alive = fetch_warp(i + 1, next);
            if (!alive) break;
            // the buffer's previous Q was used up by item i - 1, which is over
            if (next.n >= 0) load_q(i + 1, next);
            alive = __all_sync(0xffffffffu, mbar_wait_parked(bar_item_done(b), (i >> 1) & 1, &abort_word));
            if (!alive) break;
            tc5_fence_after();
            const int half = r >> 6, qt = 2 * it.pair + half;
            const bool has_keys = !(it.empty >> half & 1);   // else zero rows
            const float l = lpart[b][0][r] + lpart[b][1][r], m = mref[b][r];
            const float l_exact = LSE ? lexact[b][0][LSE ? r : 0] + lexact[b][1][LSE ? r : 0] : 0.0f;
            const float inv = has_keys && l > 0.0f ? 1.0f / l : 0.0f;
            uint32_t row[4][16];
            float finite = 0.0f;   // stays zero while every value is finite
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t v[32];
                tmem_ld32(tmem + lane_base + SP_O_COL + c * 32, v);
                tmem_wait_ld();
#pragma unroll
                for (int x = 0; x < 16; x++) {
                    const float lo = __uint_as_float(v[2 * x]), hi = __uint_as_float(v[2 * x + 1]);
                    finite = fmaf(lo, 0.0f, fmaf(hi, 0.0f, finite));
                    row[c][x] = has_keys ? pack_bf16(lo * inv, hi * inv) : 0u;
                }
            }
            tc5_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_item_free(b));   // accumulator, sums and descriptor are in registers
            if (qt < p.tiles) {
                const size_t out_row = ((size_t)it.head * p.tiles + qt) * 64 + (r & 63);
                // NaN, infinity, overflow and underflow of a real query row all fail this test (and so does
                // a value that is not finite: the other half's tiles are multiplied by zero weights here,
                // which an infinite or NaN value of V turns into NaN)
                const bool bad = has_keys && (r & 63) < max(0, min(p.sizes[qt], 64)) &&
                                 !(l >= 0x1p-60f && l < 0x1p100f && finite == 0.0f);
                if (__any_sync(0xffffffffu, bad || p.force_redo) && lane == 0) {
                    const unsigned id = (unsigned)it.head * p.tiles + qt, bit = 1u << (id & 31);
                    if (!(atomicOr(p.work.marks + (id >> 5), bit) & bit))
                        p.work.redo[atomicAdd(p.work.counters + SparseWork::REDO, 1u)] = id;
                }
                if (LSE)
                    p.lse[out_row] = has_keys ? (__logf(l_exact) + (m == -INFINITY ? 0.0f : m) * p.scale_log2 * 0.69314718056f) *
                                                    -11.313708499f
                                              : INFINITY;
                uint4 *dst = reinterpret_cast<uint4 *>(p.out + out_row * 128);
#pragma unroll
                for (int x = 0; x < 16; x++)
                    dst[x] = make_uint4(row[x / 4][x % 4 * 4], row[x / 4][x % 4 * 4 + 1], row[x / 4][x % 4 * 4 + 2],
                                        row[x / 4][x % 4 * 4 + 3]);
            }
            __syncwarp();
        }
    } else {
        warpgroup_reg_inc<SP_SOFTMAX_REGS>();
        // ------------------------------ softmax ------------------------------
        const int k = warp >> 2;             // this group takes running steps g with g % 2 == k
        const int r = tid & 127;             // query row of the pair == TMEM lane
        const int half = r >> 6;             // the same for all rows of a warp
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        int G = 0;                           // running number of the current item's first step
        bool alive = true;
        for (int i = 0; alive; i++) {
            const int b = i & 1;
            Item it;
            if (!fetch_warp(i, it) || it.n < 0) break;
            float l = 0.0f, l_exact = 0.0f, neg = 0.0f;
            bool have_ref = false;
            for (int j = (G & 1) ^ k; j < it.n; j += 2) {
                const int g = G + j, s = g % SP_AHEAD;
                const int valid = valid_keys[b * SP_MAX_TILES + j];
                const bool mine = walk[b * SP_MAX_TILES + j] >> (12 + half) & 1;
                const uint32_t s_addr = tmem + lane_base + SP_S_COL + s * 64;
                alive = __all_sync(0xffffffffu, mbar_wait(bar_s_full(s), (g / SP_AHEAD) & 1, &abort_word));
                if (!alive) break;
                tc5_fence_after();
                uint32_t s0[32], s1[32];
                if (mine || j == 0) {
                    tmem_ld32(s_addr, s0);
                    tmem_ld32(s_addr + 32, s1);
                    tmem_wait_ld();
                    if (valid < 64) {
                        mask_chunk(s0, valid);
                        mask_chunk(s1, valid - 32);
                    }
                }
                if (j == 0) {
                    // the row's exponent reference
                    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                    max_chunk4(s0, mx);
                    max_chunk4(s1, mx);
                    const float m = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                    mref[b][r] = m;
                    mbar_arrive(bar_mref(b));
                    neg = m == -INFINITY ? 0.0f : -m * p.scale_log2;
                    have_ref = true;
                } else if (!have_ref) {
                    alive = __all_sync(0xffffffffu, mbar_wait(bar_mref(b), (i >> 1) & 1, &abort_word));
                    if (!alive) break;
                    const float m = mref[b][r];
                    neg = m == -INFINITY ? 0.0f : -m * p.scale_log2;
                    have_ref = true;
                }
                uint32_t packed[16];
                if (mine) {
                    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), neg2 = make_float2(neg, neg);
                    float2 sum0 = make_float2(0.f, 0.f), sum1 = make_float2(0.f, 0.f), exact = make_float2(0.f, 0.f);
                    exp_chunk<true, LSE>(s0, packed, scale2, neg2, sum0, sum1, exact);   // masked scores are -inf: weight zero
                    tmem_st16(s_addr, packed);
                    exp_chunk<true, LSE>(s1, packed, scale2, neg2, sum0, sum1, exact);
                    tmem_st16(s_addr + 16, packed);
                    l += (sum0.x + sum0.y) + (sum1.x + sum1.y);
                    l_exact += exact.x + exact.y;
                } else {
                    store_zero_p<64>(s_addr);   // this half did not select the tile
                }
                tmem_wait_st();
                tc5_fence_before();
                mbar_arrive(bar_p_full(s));
            }
            if (!alive) break;
            // Filed by the parity of the item's OWN step numbers, not by the group's: which group gets an
            // item's first step depends on what the CTA computed before, and the result's last bit must not.
            lpart[b][k ^ (G & 1)][r] = l;
            if (LSE) lexact[b][k ^ (G & 1)][LSE ? r : 0] = l_exact;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_item_done(b));
            G += it.n;
        }
    }

    // ---------------------------------- teardown ----------------------------------
    tc5_fence_before();
    __syncthreads();
    if (abort_word) {
        if (tid == 0) atomicCAS(p.status, STATUS_OK, STATUS_WAIT_TIMEOUT);
        if (warp == 8) __nanosleep(1000000);   // let copies in flight land before smem is reused
        __syncthreads();
    }
    if (warp == 9) {
        tc5_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace

cudaError_t attn_sparse_assign(const int *indices, const int *counts, unsigned tiles, unsigned heads,
                               const SparseWork &work, cudaStream_t stream) {
    const cudaError_t e = cudaMemsetAsync(work.counters, 0, SparseWork::zeroed(tiles, heads), stream);
    if (e != cudaSuccess || work.assign == 0) return e;
    return launch_overlapped(sparse_sums_kernel, dim3(((tiles + 1) / 2 + 7) / 8, heads), 256, 0, stream, indices, counts, work,
                             (int)tiles);
}

namespace {
template <bool LSE>
cudaError_t launch_sparse_pair(const CUtensorMap &mk, const CUtensorMap &mv, const SparsePairParams &p, cudaStream_t stream) {
    static thread_local int configured_device = -1, sms = 0;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (configured_device != device) {
        // setmaxnreg moves registers inside what the CTA was given at launch; a build that was given
        // fewer would wait for them for ever, so it is refused here
        cudaFuncAttributes attributes{};
        if ((e = cudaFuncGetAttributes(&attributes, attn_sparse_pair_kernel<LSE>)) != cudaSuccess) return e;
        if (attributes.numRegs * SP_THREADS <
            SP_SOFTMAX_REGS * 256 + SP_ISSUE_REGS * 128 + SP_EPILOGUE_REGS * 128)
            return cudaErrorInvalidConfiguration;
        e = cudaFuncSetAttribute(attn_sparse_pair_kernel<LSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SP_SMEM);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (e != cudaSuccess) return e;
        configured_device = device;
    }
    const unsigned items = (unsigned)(p.tiles + 1) / 2 * (unsigned)p.heads;
    const unsigned grid = items < (unsigned)sms ? items : (unsigned)sms;   // one persistent CTA per SM
    return launch_overlapped(attn_sparse_pair_kernel<LSE>, dim3(grid), SP_THREADS, SP_SMEM, stream, mk, mv, p);
}
}  // namespace

cudaError_t attn_sparse_pair_launch(const CUtensorMap_st *mk, const CUtensorMap_st *mv, const void *q, void *out,
                                    float *lse, const int *indices, const int *counts, const int *sizes, unsigned tiles,
                                    unsigned heads, const SparseWork &work, bool force_redo, int *status,
                                    cudaStream_t stream) {
    SparsePairParams p{};
    p.indices = indices;
    p.counts = counts;
    p.sizes = sizes;
    p.q = static_cast<const uint4 *>(q);
    p.out = static_cast<__nv_bfloat16 *>(out);
    p.lse = lse;
    p.work = work;
    p.status = status;
    p.tiles = (int)tiles;
    p.heads = (int)heads;
    p.force_redo = force_redo ? 1 : 0;
    p.scale_log2 = 0.08838834764831845f * 1.4426950408889634f;   // 1/sqrt(128), fixed by the reference kernel
    return lse ? launch_sparse_pair<true>(*mk, *mv, p, stream) : launch_sparse_pair<false>(*mk, *mv, p, stream);
}

}  // namespace h3b

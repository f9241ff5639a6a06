// Dense attention forward, two query tiles per CTA (tcgen05 + TMEM + TMA): bf16 with head dim 128,
// non-causal or causal, and fp16 with head dim 64.
//
// The single-tile kernel in attn_tc5.cu relies on two co-resident CTAs to overlap softmax
// with MMAs, but nothing keeps the two CTAs out of phase, and each loads K/V for itself.
// Here one CTA owns 256 query rows as two 128-row tiles A and B that share every K/V tile,
// and the MMA warp enforces the interleaving
//      PV_A(j)  QK_A(j+1)  PV_B(j)  QK_B(j+1)  ...
// so that while softmax warpgroup A works on S_A(j+1) the tensor pipe runs B's MMAs and vice
// versa. One CTA per SM: all 512 TMEM columns (S_A, S_B, O_A, O_B, 128 each), 64 KB of Q and a
// five-slot K/V ring in shared memory.
//   warps 0-3 / 4-7 : softmax warpgroups A / B (one thread per query row, the row's 128
//                     scores held in registers: one TMEM read pass)
//   warp 8          : TMA producer
//   warp 9          : MMA issuer      (warps 8-11 give most of their registers to the
//                                      softmax warpgroups with setmaxnreg)
//   warp 10         : watches the K/V ring for the issuer (see below)
// Whatever the issuing thread does between two batches of MMAs leaves the tensor pipe idle (its
// queue is short), and a probe of an mbarrier costs that thread 80-100 cycles even when the
// barrier is long complete. So the issuer waits on exactly two barriers per step, P_A and P_B:
// a thread of warp 10 waits for V_j and K_j+1 to land and adds its arrival to P_A's barrier; and
// the softmax threads need no "PV done" signal inside the loop because the commit that announces
// S(j) also covers PV(j-1), issued before it by the same thread. The ring has five slots: a tile
// takes 2000-3000 cycles from the request to shared memory when every SM asks at once, and with
// four slots (two steps of K/V) the request for step j+2 cannot leave before step j is over.
// P goes to the issuer in three pieces (keys 0-63, 64-95, 96-127), so six of a tile's eight PV
// MMAs run while the rest of its exponentials is still being taken; waits that are expected to be long park
// in hardware (mbar_wait_parked) - at the board's power limit a spinning warp costs clock.
// A fixed fraction of the exponentials is evaluated by a polynomial on the FMA pipe (see
// softmax_tc5.cuh) so the exponential unit is not the critical resource.
// Serves h3_flash3_bf16 / h3_flash3_cross_bf16 / non-causal h3_flash_bf16 whenever the call
// has more than one query tile (replacing the reference's cuda/flash3_attention.cu:18-94).
#include <cuda.h>

#include <type_traits>

#include "attn_kernels.h"
#include "softmax_tc5.cuh"

namespace h3b {
namespace {

constexpr int PBM = 128, PBN = 128, PHD = 128;
constexpr int PAIR_THREADS = 384;                  // three warpgroups: softmax A, softmax B, {TMA, MMA}
constexpr int PAIR_SOFTMAX_REGS = 208, PAIR_OTHER_REGS = 88;   // what setmaxnreg leaves the warpgroups with
constexpr int PAIR_HALF_BYTES = PBN * 128;          // one 64-column half of a tile
constexpr int PAIR_O_COL = 256;
constexpr int PAIR_POLY = 0x55;                     // which groups of four columns take a pair of exponentials on the FMA pipe (25 %)

// What depends on the head dimension. HD = 128: 64 KB of Q and five slots of 32 KB. HD = 64: half
// of each, so the ring gets eight slots.
template <int HD>
struct PairConfig {
    static constexpr int STAGES = HD == 128 ? 5 : 8;      // K0 V0 K1 V1 ... ring of tiles
    static constexpr int HALVES = HD / 64;
    static constexpr int TILE_BYTES = PBN * HD * 2;
    static constexpr int Q_TILE_BYTES = PBM * HD * 2;
    static constexpr int SMEM_BYTES = 2 * Q_TILE_BYTES + STAGES * TILE_BYTES + 1024;
};

constexpr int PAIR_MAX_SEGMENTS = 6;
// K/V may be given as up to six separate row ranges (live mode: text, sink, two recent chunks,
// current chunk ...) that are attended as if concatenated; every range has its own tensor maps
// and may end in a partial tile.
struct PairKvMaps {
    CUtensorMap k[PAIR_MAX_SEGMENTS], v[PAIR_MAX_SEGMENTS];
};

struct PairParams {
    int segments, seg_rows[PAIR_MAX_SEGMENTS];
    int lq, lk, heads, kv_heads;
    // Split-KV for short query blocks: when split_tiles > 0, blockIdx.z is not a batch but a
    // slice of split_tiles key tiles; the CTA writes its partial output and logsumexp as if
    // they were batch element blockIdx.z, and merge_splits_kernel combines the slices.
    int split_tiles;
    float scale, scale_log2;
    uint16_t *out;   // bf16, or fp16 in the fp16 kernel
    float *lse;
    int *status;
    // sequence-gather fused into the epilogue (see PeerOutput); rows_per_rank == 0: off
    uint16_t *peer_out[16];
    unsigned rows_per_rank, rank, total_heads;
};

// CAUSAL: key k is attended by query rows >= k (lq == lk); every query tile walks its own number of
// key tiles. Work is handed out longest walk first: blockIdx.x is the head, blockIdx.y counts the
// pairs of query tiles from the end.
template <int HD, bool F16, bool CAUSAL>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
attn_tc5_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ PairKvMaps kv,
                     const PairParams p) {
    using Cfg = PairConfig<HD>;
    constexpr int ST = Cfg::STAGES;
    // How far a row's maximum may run ahead of its reference before O is rescaled. The long bf16 walks of the
    // non-causal kernel leave it at 2^8. The causal and the fp16 kernel follow the maximum, so that a row's largest
    // weight rounds to exactly 1 (2 to 4 % more error with 2^8: a short row has few weights, and fp16 ones are
    // otherwise as exact as the result), and take every exponential on the exponential unit.
    constexpr bool FOLLOW = CAUSAL || F16;
    constexpr float RESCALE_LOG2 = FOLLOW ? 0.0f : 8.0f;
    // What is left to the mma.sync kernel then is that it follows the maximum of 64 keys and has such a weight more
    // often: 0.2 to 0.4 % (causal) and 0.1 to 1 % (fp16) less error. An eighth of the weights goes in with twice the
    // bits, as a second operand of what their rounding took: error against 64 bits, mma.sync / without / so, causal
    // 128 rows 1.911 / 1.914 / 1.733e-3, 4096 rows 2.061 / 2.068 / 1.947e-3, fp16 256 rows 2.699 / 2.725 / 2.650e-4,
    // 8192 rows 2.866 / 2.868 / 2.781e-4.
    constexpr int REST_KEYS = FOLLOW ? 16 : 0, REST_COL = 64;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bars[1 + 2 * ST + 9];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    __shared__ int skip_launch;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t q_smem = smem_base;
    const uint32_t ring = q_smem + 2 * Cfg::Q_TILE_BYTES;

    const uint32_t bar0 = smem_u32(bars);
    const uint32_t bar_q_full = bar0;
    // tile number 2j is K_j, 2j+1 is V_j; tile i lives in slot i % ST and is that slot's use i / ST
    auto bar_full = [&](int s) { return bar0 + 8u * (1 + s); };
    auto bar_empty = [&](int s) { return bar0 + 8u * (1 + ST + s); };
    auto bar_s_full = [&](int t) { return bar0 + 8u * (1 + 2 * ST + t); };
    // P is handed over in three pieces (keys 0-63, 64-95, 96-127) so that PV MMAs run while the
    // later exponentials are still being taken
    auto bar_p_full = [&](int t, int piece) { return bar0 + 8u * (1 + 2 * ST + 2 + 3 * t + piece); };
    const uint32_t bar_pv_done = bar0 + 8u * (1 + 2 * ST + 8);   // the last PV of both tiles

    const int head = CAUSAL ? blockIdx.x : blockIdx.y, batch = p.split_tiles ? 0 : blockIdx.z, out_batch = blockIdx.z;
    const int kv_head = head / (p.heads / p.kv_heads);
    const int q_row0 = (CAUSAL ? gridDim.y - 1 - blockIdx.y : blockIdx.x) * 2 * PBM;
    const int tile0 = p.split_tiles * (int)blockIdx.z;   // first key tile of this CTA's slice (0 without split)
    // key rows of range s as this CTA sees it (a split call has one range and takes a slice of it)
    const int slice_rows = p.split_tiles ? min(p.seg_rows[0] - tile0 * PBN, p.split_tiles * PBN) : 0;
    auto seg_rows = [&](int s) { return p.split_tiles ? slice_rows : p.seg_rows[s]; };
    int n_tiles = 0;   // key tiles over all segments
    for (int s = 0; s < p.segments; s++) n_tiles += (seg_rows(s) + PBN - 1) / PBN;
    // Steps of query tiles A and B. The last CTA of a sequence may have no tile B; a causal tile ends
    // at its own diagonal. n_tiles: steps of the CTA.
    const bool has_b = q_row0 + PBM < p.lq;
    const int steps_a = CAUSAL ? min(n_tiles, q_row0 / PBN + 1) : n_tiles;
    const int steps_b = !has_b ? 0 : CAUSAL ? min(n_tiles, q_row0 / PBN + 2) : n_tiles;
    if (CAUSAL) n_tiles = max(steps_a, steps_b);

    // The thread that issues the loads sets the barriers up and requests Q and the first K before the CTA is complete:
    // their latency (2000 cycles and more) then covers the allocation of tensor memory and the barrier below. fp16 4096 x 8
    // 59.7 -> 58.8 us; causal and longer calls within what two runs differ by.
    if (tid == 256) {
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&kv.k[0]);
        mbar_init(bar_q_full, 1);
        for (int s = 0; s < ST; s++) {
            mbar_init(bar_full(s), 1);
            mbar_init(bar_empty(s), 1);
        }
        for (int t = 0; t < 2; t++) mbar_init(bar_s_full(t), 1);
        mbar_init(bar_p_full(0, 0), 128 + 1);   // the softmax threads of tile A and the ring watcher
        mbar_init(bar_p_full(0, 1), 128);
        mbar_init(bar_p_full(0, 2), 128);
        mbar_init(bar_p_full(1, 0), 128);
        mbar_init(bar_p_full(1, 1), 128);
        mbar_init(bar_p_full(1, 2), 128);
        mbar_init(bar_pv_done, 1);
        mbar_fence_init();
        abort_word = 0;
        wait_for_previous_kernel();
        // A launch whose stream has already recorded a failure does nothing: when a protocol
        // error makes every CTA run into its wait limit, the CTAs that start later leave at once.
        const int failed = *reinterpret_cast<volatile int *>(p.status);
        mbar_arrive_expect_tx(bar_q_full, (has_b ? 2 : 1) * Cfg::Q_TILE_BYTES);
        for (int t = 0; t < (has_b ? 2 : 1); t++)
            for (int h = 0; h < Cfg::HALVES; h++)
                tma_load_4d(q_smem + t * Cfg::Q_TILE_BYTES + h * PAIR_HALF_BYTES, &map_q, bar_q_full, 64 * h, head,
                            q_row0 + t * PBM, batch);
        mbar_arrive_expect_tx(bar_full(0), Cfg::TILE_BYTES);
        for (int h = 0; h < Cfg::HALVES; h++)
            tma_load_4d(ring + h * PAIR_HALF_BYTES, &kv.k[0], bar_full(0), 64 * h, kv_head, tile0 * PBN, batch);
        skip_launch = failed != STATUS_OK;
    }
    __syncwarp();
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

    if (skip_launch) {
        // straight to the teardown, once what has been requested is there
        if (tid == 256 && mbar_wait_parked(bar_q_full, 0, &abort_word)) mbar_wait_parked(bar_full(0), 0, &abort_word);
    } else if (warp >= 8) {
    warpgroup_reg_dec<PAIR_OTHER_REGS>();
    if (warp == 8) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            int idx = 0;   // tile number: even = K, odd = V
            bool ok = true;
            for (int seg = 0; ok && seg < p.segments; seg++) {
                const int tiles = CAUSAL ? n_tiles : (seg_rows(seg) + PBN - 1) / PBN;
                for (int tile = 0; ok && tile < tiles; tile++) {
                    for (int which = 0; which < 2; which++, idx++) {
                        if (idx == 0) continue;   // requested above
                        const int s = idx % ST, use = idx / ST;
                        if (use > 0 && !mbar_wait_parked(bar_empty(s), (use - 1) & 1, &abort_word)) {
                            ok = false;
                            break;
                        }
                        const uint32_t dst = ring + s * Cfg::TILE_BYTES;
                        const void *map = which ? (const void *)&kv.v[seg] : (const void *)&kv.k[seg];
                        mbar_arrive_expect_tx(bar_full(s), Cfg::TILE_BYTES);
                        for (int h = 0; h < Cfg::HALVES; h++)
                            tma_load_4d(dst + h * PAIR_HALF_BYTES, map, bar_full(s), 64 * h, kv_head,
                                        (tile0 + tile) * PBN, batch);
                    }
                }
            }
        }
    } else if (warp == 9) {
        // ------------------------------- MMA issuer -------------------------------
        // The whole warp walks the loop and one elected lane issues: with the loop inside a
        // one-lane branch every descriptor word is per-thread data that has to be moved to a
        // uniform register in front of each MMA.
        {
            const bool leader = elect_one();
            constexpr uint32_t idesc_qk = mma_idesc(PBM, PBN, F16 ? 0 : 1, 0);
            constexpr uint32_t idesc_pv = mma_idesc(PBM, HD, F16 ? 0 : 1, 1);
            // Descriptors are built once (Q) or once per stage (K, V); a K-step only adds to
            // the low word: +2 per 32 bytes inside a 64-column half, +1024 for the second half
            // (16 KB), +128 per 16 V rows (2 KB).
            uint32_t q_lo[2], q_hi[2];
            for (int t = 0; t < 2; t++) {
                const uint64_t d = smem_desc_sw128(q_smem + t * Cfg::Q_TILE_BYTES, 16, 1024);
                q_lo[t] = (uint32_t)d;
                q_hi[t] = (uint32_t)(d >> 32);
            }
            const uint64_t k_proto = smem_desc_sw128(ring, 16, 1024);
            const uint64_t v_proto = smem_desc_sw128(ring, PAIR_HALF_BYTES, 1024);
            const uint32_t k_hi = (uint32_t)(k_proto >> 32), v_hi = (uint32_t)(v_proto >> 32);
            const uint32_t k_ring_lo = (uint32_t)k_proto, v_ring_lo = (uint32_t)v_proto;  // LBO lives in the low word
            auto issue_qk = [&](int j, int t) {   // S_t = Q_t . K_j^T
                const uint32_t k_lo = k_ring_lo + ((2 * j) % ST) * (Cfg::TILE_BYTES >> 4);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < HD / 16; kk++) {
                        const uint32_t off = (kk / 4) * (PAIR_HALF_BYTES >> 4) + (kk % 4) * 2;
                        mma_ss_words(tmem + t * PBN, q_lo[t] + off, q_hi[t], k_lo + off, k_hi, idesc_qk,
                                     kk > 0);
                    }
                    mma_commit(bar_s_full(t));   // also tells the softmax threads that PV_t(j-1) is complete
                }
                __syncwarp();
            };
            auto issue_pv = [&](int j, int t, int piece) {   // O_t += P_t . V_j over keys 0-63, 64-95 or 96-127
                const uint32_t v_lo = v_ring_lo + ((2 * j + 1) % ST) * (Cfg::TILE_BYTES >> 4);
                const int first = piece == 0 ? 0 : piece == 1 ? 4 : 6, last = piece == 0 ? 4 : piece == 1 ? 6 : 8;
                // On the diagonal rows 0-63 are left out of the products of keys 64-127: a zero weight does not keep an
                // infinite or NaN value of a later key away from them.
                const uint32_t spare = CAUSAL && j + 1 == (t ? steps_b : steps_a) ? 0xffffffffu : 0u;
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < 8; kk++) {
                        if (kk < first || kk >= last) continue;
                        const uint32_t o_tmem = tmem + PAIR_O_COL + t * HD, p_tmem = tmem + t * PBN + kk * 8;
                        if (CAUSAL && kk >= 4)
                            mma_ts_words_sparing(o_tmem, p_tmem, v_lo + kk * (2048 >> 4), v_hi, idesc_pv, 1, spare);
                        else
                            mma_ts_words(o_tmem, p_tmem, v_lo + kk * (2048 >> 4), v_hi, idesc_pv, (j > 0) || (kk > 0));
                    }
                    if (FOLLOW && piece == 0)
                        mma_ts_words(tmem + PAIR_O_COL + t * HD, tmem + t * PBN + REST_COL, v_lo, v_hi, idesc_pv, 1);
                }
                __syncwarp();
            };
            auto release = [&](int tile) {   // the slot may be refilled once the MMAs issued so far are done
                if (leader) mma_commit(bar_empty(tile % ST));
            };
            bool alive = mbar_wait_converged(bar_q_full, 0, &abort_word) &&
                         mbar_wait_converged(bar_full(0), 0, &abort_word);
            if (alive) {
                tc5_fence_after();
                issue_qk(0, 0);
                if (steps_b > 0) issue_qk(0, 1);
                release(0);
            }
            // EVEN: both tiles take every step (the hot case, straight-line: a branch in this warp's loop
            // leaves the tensor pipe idle, 1.7 % of a long call). Otherwise each tile has its own number.
            auto walk = [&](auto even) {
            constexpr bool EVEN = decltype(even)::value;
            for (int j = 0; alive && j < n_tiles; j++) {
                const bool more = j + 1 < n_tiles;
                if (EVEN || j < steps_a) {
                    // P of tile A, and (through the ring watcher) V of this step and K of the next
                    if (!mbar_wait_converged(bar_p_full(0, 0), j & 1, &abort_word)) break;
                    tc5_fence_after();
                    issue_pv(j, 0, 0);
                    if (!mbar_wait_converged(bar_p_full(0, 1), j & 1, &abort_word)) break;
                    tc5_fence_after();
                    issue_pv(j, 0, 1);
                    if (!mbar_wait_converged(bar_p_full(0, 2), j & 1, &abort_word)) break;
                    tc5_fence_after();
                    issue_pv(j, 0, 2);
                    if (EVEN ? more : j + 1 < steps_a) issue_qk(j + 1, 0);
                } else {
                    // tile A has passed its diagonal (its watcher is done): V of this step directly
                    const int v = 2 * j + 1;
                    if (!mbar_wait_converged(bar_full(v % ST), (v / ST) & 1, &abort_word)) break;
                    tc5_fence_after();
                }
                if (EVEN || j < steps_b) {
                    if (!mbar_wait_converged(bar_p_full(1, 0), j & 1, &abort_word)) break;
                    tc5_fence_after();
                    issue_pv(j, 1, 0);
                    if (!mbar_wait_converged(bar_p_full(1, 1), j & 1, &abort_word)) break;
                    tc5_fence_after();
                    issue_pv(j, 1, 1);
                    if (!mbar_wait_converged(bar_p_full(1, 2), j & 1, &abort_word)) break;
                    tc5_fence_after();
                    issue_pv(j, 1, 2);
                }
                release(2 * j + 1);
                if (more) {
                    if (EVEN || j + 1 < steps_b) issue_qk(j + 1, 1);
                    release(2 * j + 2);
                } else if (leader) {
                    mma_commit(bar_pv_done);      // both accumulators are final
                }
                __syncwarp();
            }
            };
            if (!CAUSAL && has_b) walk(std::true_type{});
            else walk(std::false_type{});
        }
    } else if (warp == 10) {
        // ------------------------------- ring watcher -------------------------------
        if (lane == 0) {
            // One arrival per phase of P_A's barrier: the next tiles are often there before the
            // softmax threads are done, so wait for the phase to end before arriving again.
            for (int g = 0; g < steps_a; g++) {
                const int v = 2 * g + 1, k = 2 * g + 2;
                if (!mbar_wait_parked(bar_full(v % ST), (v / ST) & 1, &abort_word)) break;
                if (g + 1 < n_tiles && !mbar_wait_parked(bar_full(k % ST), (k / ST) & 1, &abort_word)) break;
                mbar_arrive(bar_p_full(0, 0));
                if (!mbar_wait_parked(bar_p_full(0, 0), g & 1, &abort_word)) break;
            }
        }
    }
    } else {
        warpgroup_reg_inc<PAIR_SOFTMAX_REGS>();
        // ------------------------------ online softmax ------------------------------
        const int t = warp >> 2;                // which query tile
        const int r = tid & 127;                // row inside the tile == TMEM lane
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t s_addr = tmem + lane_base + t * PBN;
        const uint32_t o_addr = tmem + lane_base + PAIR_O_COL + t * HD;
        const int steps = t ? steps_b : steps_a;
        float m_ref = -INFINITY, l = 0.0f;
        bool alive = true;
        // One step of this thread's row: scores from TMEM (the whole row in registers, one read pass),
        // P back over them in three pieces. MASKED: only the first nvalid scores count.
        auto softmax_step = [&](auto masked, int j, int nvalid) {
            constexpr bool MASKED = decltype(masked)::value;
            constexpr int POLY = MASKED || FOLLOW ? 0 : PAIR_POLY;   // a masked score is -inf: exactly zero weight
            uint32_t s0[32], s1[32], s2[32], s3[32];
            tmem_ld32(s_addr, s0);
            tmem_ld32(s_addr + 32, s1);
            tmem_ld32(s_addr + 64, s2);
            tmem_ld32(s_addr + 96, s3);
            tmem_wait_ld();
            if (MASKED) {
                mask_chunk(s0, nvalid);
                mask_chunk(s1, nvalid - 32);
                mask_chunk(s2, nvalid - 64);
                mask_chunk(s3, nvalid - 96);
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            max_chunk4<true>(s0, mx);
            max_chunk4<true>(s1, mx);
            max_chunk4<true>(s2, mx);
            max_chunk4<true>(s3, mx);
            // A NaN score makes the maximum NaN, and that the row: not every column's exponential keeps it.
            const float m_new = max3<true>(max3<true>(m_ref, mx[0], mx[1]), mx[2], mx[3]);
            const bool grow = !((m_new - m_ref) * p.scale_log2 <= RESCALE_LOG2);
            if (__any_sync(0xffffffffu, grow)) {
                // A score of +inf leaves the row no defined weights: NaN, in every column and from here on. Only scores
                // of -inf so far: nothing to weigh, and (FOLLOW) nothing to rescale.
                const bool none = FOLLOW && m_new == -INFINITY;
                const float alpha = grow && !none ? fast_exp2((m_ref - m_new) * p.scale_log2) : 1.0f;
                if (grow) m_ref = m_new == INFINITY ? NAN : m_new;
                l *= alpha;
                if (j > 0) {   // PV(j-1) is complete: S(j)'s commit covered it
#pragma unroll
                    for (int c = 0; c < HD / 32; c++) {
                        uint32_t v[32];
                        tmem_ld32(o_addr + c * 32, v);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i++)
                            v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
                        tmem_st32(o_addr + c * 32, v);
                    }
                    tmem_wait_st();
                }
            }
            const float neg = FOLLOW && m_ref == -INFINITY ? 0.0f : -m_ref * p.scale_log2;
            const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
            const float2 neg2 = make_float2(neg, neg);
            float2 sum0 = make_float2(0.f, 0.f), sum1 = make_float2(0.f, 0.f);
            uint32_t packed[16];
            uint32_t rest[8];
            exp_chunk_mixed<POLY, F16, REST_KEYS>(s0, packed, scale2, neg2, sum0, sum1, rest);
            tmem_st16(s_addr, packed);
            if (FOLLOW) tmem_st8(s_addr + REST_COL, rest);   // over scores that are in registers
            exp_chunk_mixed<POLY, F16>(s1, packed, scale2, neg2, sum0, sum1);
            tmem_st16(s_addr + 16, packed);
            tmem_wait_st();
            tc5_fence_before();
            mbar_arrive(bar_p_full(t, 0));
            exp_chunk_mixed<POLY, F16>(s2, packed, scale2, neg2, sum0, sum1);
            tmem_st16(s_addr + 32, packed);
            tmem_wait_st();
            tc5_fence_before();
            mbar_arrive(bar_p_full(t, 1));
            exp_chunk_mixed<POLY, F16>(s3, packed, scale2, neg2, sum0, sum1);
            tmem_st16(s_addr + 48, packed);
            l += (sum0.x + sum0.y) + (sum1.x + sum1.y);
            tmem_wait_st();
            tc5_fence_before();
            mbar_arrive(bar_p_full(t, 2));
        };
        int seg = 0, seg_tile = 0;   // which segment, which tile of it, step j is
        for (int j = 0; j < steps; j++) {
            while (seg_tile * PBN >= seg_rows(seg)) {
                seg++;
                seg_tile = 0;
            }
            const int in_range = min(PBN, seg_rows(seg) - seg_tile * PBN);
            seg_tile++;
            alive = __all_sync(0xffffffffu, mbar_wait_parked(bar_s_full(t), j & 1, &abort_word));
            if (!alive) break;
            tc5_fence_after();
            // keys up to the row's own, counted from the tile's first key: of the warp's first row
            const int causal_first = q_row0 + t * PBM + (warp & 3) * 32 + 1 - j * PBN;
            if (min(in_range, CAUSAL ? causal_first : PBN) >= PBN)
                softmax_step(std::false_type{}, j, PBN);
            else
                softmax_step(std::true_type{}, j, CAUSAL ? min(in_range, causal_first + lane) : in_range);
        }

        // -------- epilogue: O / l -> 16 bits, through shared memory to global --------
        alive = alive && steps > 0;
        if (alive) alive = __all_sync(0xffffffffu, mbar_wait(bar_pv_done, 0, &abort_word));
        if (alive) {
            tc5_fence_after();
            const float inv = 1.0f / l;
            const int row = q_row0 + t * PBM + r;
            if (row < p.lq && p.lse)
                p.lse[((size_t)out_batch * p.heads + head) * p.lq + row] = m_ref * p.scale + (FOLLOW ? logf(l) : __logf(l));
            // Rows go through shared memory (the tile's Q, which no MMA reads any more), so that the lanes of a warp store whole
            // rows; a lane storing its own row writes 16 bytes in each of 32 places. Causal 1000 x 32 / 8 heads 23.8 -> 22.8 us,
            // 13,088 x 52,301 x 24 7241 -> 7147 us, 15,400 x 56 heads 5828 -> 5775 us; fp16 4096 x 8 59.0 -> 58.8 us.
            constexpr int CHUNKS = HD / 8, ROWS = 32 / CHUNKS;   // 16-byte pieces of a row; rows stored at a time
            uint4 *const stage = reinterpret_cast<uint4 *>(smem_raw + (q_smem - smem_u32(smem_raw)) + t * Cfg::Q_TILE_BYTES) +
                                 (warp & 3) * 32 * CHUNKS;
#pragma unroll
            for (int c = 0; c < HD / 32; c++) {
                uint32_t v[32];
                tmem_ld32(o_addr + c * 32, v);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    uint4 w;
                    w.x = pack_p<F16>(__uint_as_float(v[i * 8 + 0]) * inv, __uint_as_float(v[i * 8 + 1]) * inv);
                    w.y = pack_p<F16>(__uint_as_float(v[i * 8 + 2]) * inv, __uint_as_float(v[i * 8 + 3]) * inv);
                    w.z = pack_p<F16>(__uint_as_float(v[i * 8 + 4]) * inv, __uint_as_float(v[i * 8 + 5]) * inv);
                    w.w = pack_p<F16>(__uint_as_float(v[i * 8 + 6]) * inv, __uint_as_float(v[i * 8 + 7]) * inv);
                    stage[lane * CHUNKS + ((4 * c + i) ^ (lane & 7))] = w;
                }
            }
            __syncwarp();
            const int chunk = lane % CHUNKS;
#pragma unroll 4
            for (int i = 0; i < 32; i += ROWS) {
                const int local = i + lane / CHUNKS, mine = q_row0 + t * PBM + (warp & 3) * 32 + local;
                if (mine >= p.lq) break;
                uint16_t *dst;
                if (p.rows_per_rank) {
                    // this row belongs to another rank's row shard: store it there, in place
                    const unsigned owner = (unsigned)mine / p.rows_per_rank, there = (unsigned)mine % p.rows_per_rank;
                    dst = p.peer_out[owner] + ((size_t)there * p.total_heads + (size_t)p.rank * p.heads + head) * HD;
                } else {
                    dst = p.out + (((size_t)out_batch * p.lq + mine) * p.heads + head) * HD;
                }
                reinterpret_cast<uint4 *>(dst)[chunk] = stage[local * CHUNKS + (chunk ^ (local & 7))];
            }
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

// Combines the slices of a split-KV call: out[r][h][:] = sum_s w_s O_s[r][h][:] / sum_s w_s with
// w_s = exp(lse_s - max_s lse_s). One thread per (row, head, eight dims).
__global__ void __launch_bounds__(256)
merge_splits_kernel(__nv_bfloat16 *out, float *lse_out, const uint4 *partial, const float *lse, int splits, int lq,
                    int heads) {
    wait_for_previous_kernel();
    allow_next_kernel();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)lq * heads * (PHD / 8);
    if (i >= total) return;
    const int v = (int)(i % (PHD / 8)), head = (int)((i / (PHD / 8)) % heads), row = (int)(i / ((size_t)(PHD / 8) * heads));
    float top = -INFINITY;
    for (int s = 0; s < splits; s++) top = fmaxf(top, lse[((size_t)s * heads + head) * lq + row]);
    float acc[8] = {}, weight = 0.0f;
    for (int s = 0; s < splits; s++) {
        const float w = __expf(lse[((size_t)s * heads + head) * lq + row] - top);
        const uint4 x = partial[(((size_t)s * lq + row) * heads + head) * (PHD / 8) + v];
        const uint32_t words[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            acc[2 * k] = fmaf(w, __uint_as_float(words[k] << 16), acc[2 * k]);
            acc[2 * k + 1] = fmaf(w, __uint_as_float(words[k] & 0xffff0000u), acc[2 * k + 1]);
        }
        weight += w;
    }
    const float inv = 1.0f / weight;
    uint4 y;
    y.x = pack_bf16(acc[0] * inv, acc[1] * inv);
    y.y = pack_bf16(acc[2] * inv, acc[3] * inv);
    y.z = pack_bf16(acc[4] * inv, acc[5] * inv);
    y.w = pack_bf16(acc[6] * inv, acc[7] * inv);
    reinterpret_cast<uint4 *>(out)[i] = y;
    if (lse_out && v == 0) lse_out[(size_t)head * lq + row] = top + __logf(weight);
}

}  // namespace

cudaError_t attn_merge_splits(void *out, float *lse_out, const void *partial, const float *lse, unsigned splits,
                              unsigned lq, unsigned heads, cudaStream_t stream) {
    const size_t total = (size_t)lq * heads * (PHD / 8);
    return launch_overlapped(merge_splits_kernel, dim3((unsigned)((total + 255) / 256)), 256, 0, stream,
                             static_cast<__nv_bfloat16 *>(out), lse_out, static_cast<const uint4 *>(partial), lse, (int)splits,
                             (int)lq, (int)heads);
}

namespace {

template <int HD, bool F16, bool CAUSAL>
cudaError_t launch_pair(const CUtensorMap &mq, const PairKvMaps &kv, const PairParams &p, unsigned slices,
                        cudaStream_t stream) {
    auto kernel = attn_tc5_pair_kernel<HD, F16, CAUSAL>;
    static thread_local int configured_device = -1;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (configured_device != device) {
        // setmaxnreg moves registers inside what the CTA was given at launch; a build that was given
        // fewer would wait for them for ever, so it is refused here
        cudaFuncAttributes attributes{};
        if ((e = cudaFuncGetAttributes(&attributes, kernel)) != cudaSuccess) return e;
        if (attributes.numRegs * PAIR_THREADS < PAIR_SOFTMAX_REGS * 256 + PAIR_OTHER_REGS * 128)
            return cudaErrorInvalidConfiguration;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PairConfig<HD>::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        configured_device = device;
    }
    const unsigned pairs = ((unsigned)p.lq + 2 * PBM - 1) / (2 * PBM), heads = (unsigned)p.heads;
    if (CAUSAL && pairs > 65535u) return cudaErrorInvalidValue;
    const dim3 grid = CAUSAL ? dim3(heads, pairs, slices) : dim3(pairs, heads, slices);
    return launch_overlapped(kernel, grid, PAIR_THREADS, PairConfig<HD>::SMEM_BYTES, stream, mq, kv, p);
}

}  // namespace

cudaError_t attn_dense_tc5_pair(const CUtensorMap_st *mq, const CUtensorMap_st *mk,
                                const CUtensorMap_st *mv, void *out, float *lse, unsigned batch,
                                unsigned lq, unsigned lk, unsigned heads, unsigned kv_heads,
                                float scale, int *status, cudaStream_t stream, const PeerOutput *peer,
                                unsigned segments, const unsigned *segment_rows, unsigned split_tiles,
                                PairKind kind) {
    // mk / mv point to `segments` maps each; without a segment list: one range of lk rows
    if (segments > (unsigned)PAIR_MAX_SEGMENTS || (segments > 1 && batch != 1)) return cudaErrorInvalidValue;
    if (kind != PairKind::BF16_D128 && (segments || split_tiles || peer)) return cudaErrorInvalidValue;
    if (kind == PairKind::BF16_D128_CAUSAL && lq != lk) return cudaErrorInvalidValue;
    // split-KV: one key range, batch 1, no peer output; the slices ride on grid.z
    unsigned splits = 1;
    if (split_tiles) {
        if (segments > 1 || batch != 1 || peer || !lse) return cudaErrorInvalidValue;
        splits = ((lk + PBN - 1) / PBN + split_tiles - 1) / split_tiles;
    }
    PairKvMaps kv{};
    PairParams p{};
    p.segments = segments ? (int)segments : 1;
    for (int i = 0; i < p.segments; i++) {
        kv.k[i] = mk[i];
        kv.v[i] = mv[i];
        p.seg_rows[i] = segments ? (int)segment_rows[i] : (int)lk;
        if (p.seg_rows[i] <= 0) return cudaErrorInvalidValue;
    }
    p.lq = (int)lq;
    p.lk = (int)lk;
    p.heads = (int)heads;
    p.kv_heads = (int)kv_heads;
    p.scale = scale;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.out = static_cast<uint16_t *>(out);
    p.lse = lse;
    p.status = status;
    p.split_tiles = (int)split_tiles;
    if (peer) {
        if (batch != 1 || !peer->rows_per_rank) return cudaErrorInvalidValue;
        for (int i = 0; i < 16; i++) p.peer_out[i] = static_cast<uint16_t *>(peer->base[i]);
        p.rows_per_rank = peer->rows_per_rank;
        p.rank = peer->rank;
        p.total_heads = peer->total_heads;
    }
    const unsigned slices = split_tiles ? splits : batch;
    switch (kind) {
        case PairKind::BF16_D128_CAUSAL: return launch_pair<128, false, true>(*mq, kv, p, slices, stream);
        case PairKind::F16_D64: return launch_pair<64, true, false>(*mq, kv, p, slices, stream);
        default: return launch_pair<128, false, false>(*mq, kv, p, slices, stream);
    }
}

}  // namespace h3b

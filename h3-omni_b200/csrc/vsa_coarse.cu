// Video sparse attention, coarse stage and merge: token-cube pooling, pooled scores with
// warp-level top-k tile selection, the pooled-softmax compression branch, and the gated
// merge back to token-major rows. These are HBM-bound passes; they replace tile_pool,
// the two cuBLAS SGEMMs, select_blocks, pooled_softmax and untile_merge of the reference's
// cuda/vsa.cuh:18-181,263-300 with three launches (pool x3 fused, score+select+compress,
// merge) and never materialise the [heads][tiles][tiles] score matrix unless asked to.
#include <cuda_bf16.h>
#include <math_constants.h>

#include <cstdio>

#include "attn_kernels.h"
#include "sm100_ptx.cuh"

namespace h3b {
namespace {

constexpr int VD = 128, VT = 64;

__device__ __forceinline__ float bf16_bits_to_f32(uint32_t x) { return __uint_as_float(x << 16); }
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float x) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x));
}
__device__ __forceinline__ float bf16_round(float x) { return bf16_bits_to_f32(f32_to_bf16_bits(x)); }

// ---- pooling ---------------------------------------------------------------------
// One CTA = one tile x 8 heads x one of {Q, K, V}; thread = (head, four dims = 8 bytes), so
// every token row contributes one contiguous 2 KB read per CTA. Bound by HBM: a thread requests 32 rows before it
// stores the first of them (a load does not move up across a store that may be to the same place). The loop over
// the two halves stays rolled, or all 64 row numbers are held at once and one CTA fits an SM instead of two.
// 287 tiles x 56 heads: 266 us with all loads through the read-only path, 243 so; 905 x 24 362 -> 328; 144 x 14
// 37.2 -> 33.9; 50 x 7 6.9 -> 7.6. (One lane at a time, three CTAs per SM: 247, 334, 34.1 and 9.3.)
// The per-dimension summation order is the reference's
// (cuda/vsa.cuh:22-42): 4 lanes x 4 slot accumulators, element i = lane + 4*slot + 16*round,
// ((a0+a1)+a2)+a3 per lane, (l0+l2)+(l1+l3), then / size.
struct PoolArgs {
    const uint2 *src[3];
    uint2 *tiled[3];
    float *pooled[3];
};

template <bool TILED>
__global__ void __launch_bounds__(256, 2)
tile_pool_kernel(PoolArgs a, const int *map, const int *sizes, int tiles, int heads) {
    wait_for_previous_kernel();
    allow_next_kernel();
    __shared__ int rows[VT];
    const int tile = blockIdx.x, which = blockIdx.z;
    const int head = blockIdx.y * 8 + (threadIdx.x >> 5), dq = threadIdx.x & 31;
    if (threadIdx.x < VT) rows[threadIdx.x] = map[tile * VT + threadIdx.x];
    __syncthreads();
    if (head >= heads) return;
    const uint2 *src = which == 0 ? a.src[0] : which == 1 ? a.src[1] : a.src[2];
    uint2 *tiled = which == 0 ? a.tiled[0] : which == 1 ? a.tiled[1] : a.tiled[2];
    float *pooled = which == 0 ? a.pooled[0] : which == 1 ? a.pooled[1] : a.pooled[2];
    float even[4], sum[4];   // lanes 0 and 2; the two lanes of this turn
#pragma unroll 1
    for (int first = 0; first < 2; first++) {
        uint2 held[2][16];   // [lane / 2][slot + 4 * round]
#pragma unroll
        for (int n = 0; n < 32; n++) {
            const int row = rows[first + 2 * (n / 16) + 4 * (n % 16)];
            held[n / 16][n % 16] = make_uint2(0u, 0u);
            if (row >= 0) held[n / 16][n % 16] = src[((size_t)row * heads + head) * (VD / 4) + dq];
        }
#pragma unroll
        for (int which_lane = 0; which_lane < 2; which_lane++) {
            const int lane = first + 2 * which_lane;
            float acc[4][4];   // [slot][dim]
#pragma unroll
            for (int slot = 0; slot < 4; slot++)
#pragma unroll
                for (int d = 0; d < 4; d++) acc[slot][d] = 0.0f;
#pragma unroll
            for (int n = 0; n < 16; n++) {
                const uint2 x = held[which_lane][n];
                if (TILED) tiled[((size_t)head * tiles * VT + tile * VT + lane + 4 * n) * (VD / 4) + dq] = x;
                acc[n % 4][0] += bf16_bits_to_f32(x.x & 0xffffu);
                acc[n % 4][1] += bf16_bits_to_f32(x.x >> 16);
                acc[n % 4][2] += bf16_bits_to_f32(x.y & 0xffffu);
                acc[n % 4][3] += bf16_bits_to_f32(x.y >> 16);
            }
#pragma unroll
            for (int d = 0; d < 4; d++) {
                const float own = ((acc[0][d] + acc[1][d]) + acc[2][d]) + acc[3][d];
                sum[d] = which_lane ? sum[d] + own : own;
            }
        }
        if (first == 0)
#pragma unroll
            for (int d = 0; d < 4; d++) even[d] = sum[d];
    }
    const float size = (float)sizes[tile];
    float4 mean;
    mean.x = (even[0] + sum[0]) / size;
    mean.y = (even[1] + sum[1]) / size;
    mean.z = (even[2] + sum[2]) / size;
    mean.w = (even[3] + sum[3]) / size;
    reinterpret_cast<float4 *>(pooled)[((size_t)head * tiles + tile) * (VD / 4) + dq] = mean;
}

// ---- scores + top-k selection + compression -----------------------------------------
constexpr int KCHUNK = 256, KPART = 32;   // pooled K staged per step: 256 rows x 32 dims
constexpr int QPAD = VD + 4;              // rows 4 banks apart
constexpr int VCHUNK = 64;                // pooled V rows staged per step
static_assert(VCHUNK * VD <= KCHUNK * KPART, "V stage fits the K stage");
// Where dims d .. d + 3 of row r are staged: the eight 16-byte pieces of a row change places with the row's number, so
// that 8 rows x 16 bytes hit 32 distinct banks without padding.
__device__ __forceinline__ int staged(int r, int d) { return r * KPART + (d ^ (r & 7) * 4); }
// Floats between two score rows: float4-aligned and 4 banks apart like the rows above.
__host__ __device__ constexpr int score_stride(int tiles) { return (tiles + 31) / 32 * 32 + 4; }
constexpr size_t score_select_smem(int tiles, int qt) {
    return sizeof(float) * ((size_t)qt * score_stride(tiles) + KCHUNK * KPART + (size_t)qt * QPAD);
}
// Two CTAs of 16 query tiles share an SM's 228 KB (1 KB of which each CTA's launch takes) up to 1152 tiles, two of 8 up to 2432.
// Where one has it to itself a call takes a third longer: 24 heads of 1120 tiles 1235 us with one, 905 with two; of 1152 940
// and of 1160 1290; 8 heads of 2390 tiles 2774 and 2031.
static_assert(2 * (score_select_smem(1152, 16) + 1024) <= 228 * 1024 && 2 * (score_select_smem(2432, 8) + 1024) <= 228 * 1024,
              "two CTAs per SM");

// Order-preserving key of a float, the one cub's radix sort uses: larger float -> larger key.
__device__ __forceinline__ uint32_t sort_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ uint32_t tile_key(float f) { return max(sort_key(f), 1u); }   // 0 stands for "no tile"
__device__ __forceinline__ float key_value(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? k ^ 0x80000000u : ~k);
}

// One CTA = 8 * QPW query tiles of one head, 8 warps. Pooled K (then V) rows stream through shared
// memory, the next chunk's global loads in flight while the current one is used, so each pooled row is
// read from L2 once per 8 * QPW query tiles.
//   scores row = scale * fmaf-chain over d = 0..127 (ascending), one fixed order.
//   Selection (cuda/vsa.cuh:47-76): prefix query tiles keep all tiles; video query tiles keep
//   all prefix tiles plus the `keep` best video tiles (ties: lower index first), ascending.
//   Compression (cuda/vsa.cuh:80-166,291-294): softmax over the whole row in the ATen lane
//   order, then sum_k p[k] * poolv[k][:] as one fmaf chain over k ascending.
// Both products are bound by shared-memory reads unless a read feeds several FMAs: a warp covers 8 rows
// (or 8 x 4 dims) by 4 query tiles, so that the lanes of a vector read share addresses, and a thread takes 4 keys x 2 QPW
// query tiles of the scores (4 + 2 QPW reads per 32 * QPW FMAs) and 4 dims x QPW query tiles of the compression (4 + QPW
// per 4 keys and 16 * QPW FMAs).
// 905 tiles x 24 heads: 754 us with a key row (or four dims) per lane and a bit-by-bit search, 704 with four keys x QPW
// query tiles per thread, 644 with the interval search below, 582 with 2 QPW query tiles per thread (256 keys x 32 dims
// staged instead of 128 x 64), 560 with ordinary loads and the dims of a part unrolled. 450 x 14: 172, 146, 142 us in the last three steps,
// 287 x 56 189, 177, 170, 50 x 3 12.1, 11.7, 11.4.
template <int QPW>
__global__ void __launch_bounds__(256, 2)
score_select_kernel(const float *poolq, const float *poolk, const float *poolv, float *scores_out, int *indices,
                    int *counts, float *compression, int tiles, int prefix, int keep, float scale) {
    wait_for_previous_kernel();
    allow_next_kernel();
    constexpr int QT = 8 * QPW;
    extern __shared__ __align__(16) float sm[];
    const int stride = score_stride(tiles);
    float *row_scores = sm;                                // [QT][stride]
    float *stage = row_scores + (size_t)QT * stride;       // [KCHUNK][KPART] (see staged()), later [VCHUNK][VD]
    float *qrows = stage + KCHUNK * KPART;                 // [QT][QPAD]

    const int head = blockIdx.y, qt0 = blockIdx.x * QT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nq = min(QT, tiles - qt0);
    const int in8 = lane & 7, in4 = lane >> 3;

    for (int i = tid; i < QT * VD; i += 256) {
        const int qi = i / VD, d = i % VD;
        qrows[qi * QPAD + d] = qi < nq ? poolq[((size_t)head * tiles + qt0 + qi) * VD + d] : 0.0f;
    }
    // ---- scores: warp = 32 keys (of 256) x all query tiles ----
    {
        const float *pk = poolk + (size_t)head * tiles * VD;
        const bool wide = reinterpret_cast<uintptr_t>(poolk) % 16 == 0;   // a caller's own array need not be
        constexpr int PER_THREAD = KCHUNK * KPART / 4 / 256, NQ = 2 * QPW;
        float4 next[PER_THREAD];   // this thread's part of the stage being fetched
        auto fetch = [&](int k0, int part) {
#pragma unroll
            for (int u = 0; u < PER_THREAD; u++) {
                const int i = tid + u * 256, r = i / (KPART / 4), c = i % (KPART / 4);
                const float *at = pk + (size_t)(k0 + r) * VD + part * KPART + c * 4;
                next[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k0 + r < tiles)
                    next[u] = wide ? *reinterpret_cast<const float4 *>(at) : make_float4(at[0], at[1], at[2], at[3]);
            }
        };
        fetch(0, 0);
        const int key0 = warp * 32 + in8, q0 = in4;
        for (int k0 = 0; k0 < tiles; k0 += KCHUNK) {
            const bool busy = k0 + warp * 32 < tiles;   // the last chunk may have no keys for a warp
            float dot[4][NQ];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int u = 0; u < NQ; u++) dot[i][u] = 0.0f;
#pragma unroll 1
            for (int part = 0; part < VD / KPART; part++) {
                __syncthreads();   // the stage is used up
#pragma unroll
                for (int u = 0; u < PER_THREAD; u++) {
                    const int i = tid + u * 256;
                    *reinterpret_cast<float4 *>(stage + staged(i / (KPART / 4), i % (KPART / 4) * 4)) = next[u];
                }
                __syncthreads();
                if (part + 1 < VD / KPART) fetch(k0, part + 1);
                else if (k0 + KCHUNK < tiles) fetch(k0 + KCHUNK, 0);
                if (!busy) continue;
#pragma unroll
                for (int d = 0; d < KPART; d += 4) {
                    float4 kv[4], qv[NQ];
#pragma unroll
                    for (int i = 0; i < 4; i++) kv[i] = *reinterpret_cast<const float4 *>(stage + staged(key0, d) + 8 * i * KPART);
#pragma unroll
                    for (int u = 0; u < NQ; u++)
                        qv[u] = *reinterpret_cast<const float4 *>(qrows + (q0 + 4 * u) * QPAD + part * KPART + d);
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int u = 0; u < NQ; u++) {
                            dot[i][u] = fmaf(qv[u].x, kv[i].x, dot[i][u]);
                            dot[i][u] = fmaf(qv[u].y, kv[i].y, dot[i][u]);
                            dot[i][u] = fmaf(qv[u].z, kv[i].z, dot[i][u]);
                            dot[i][u] = fmaf(qv[u].w, kv[i].w, dot[i][u]);
                        }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int u = 0; u < NQ; u++)
                    if (k0 + key0 + 8 * i < tiles && q0 + 4 * u < nq)
                        row_scores[(size_t)(q0 + 4 * u) * stride + k0 + key0 + 8 * i] = scale * dot[i][u];
        }
    }
    __syncthreads();

    // ---- selection and pooled softmax: warp `warp` owns query tiles qt0 + warp + 8 g ----
#pragma unroll 1
    for (int g = 0; g < QPW; g++) {
        const int qi = warp + 8 * g;
        if (qi >= nq) break;
        const int qt = qt0 + qi;
        float *mine = row_scores + (size_t)qi * stride;
        const size_t row = (size_t)head * tiles + qt;
        if (scores_out)
            for (int j = lane; j < tiles; j += 32) scores_out[row * tiles + j] = mine[j];
        int *dst = indices + row * tiles;
        if (qt < prefix) {
            for (int j = lane; j < tiles; j += 32) dst[j] = j;
            if (lane == 0) counts[row] = tiles;
        } else {
            // The keep-th largest key among the video tiles lies in [low, high): at least `keep` keys are
            // >= low, fewer are >= high. The interval is halved first by value, then (ties, infinities)
            // by key, until exactly `keep` keys are >= low - about a dozen counts, where a bit-by-bit search
            // takes 32 - or one key is left. Counting is a compare per key and one warp reduction: no
            // shared-memory histogram, no atomics.
            uint32_t key[32];   // up to 1024 video tiles: this lane's keys stay in registers
            const bool in_registers = tiles - prefix <= 32 * 32;
            const int groups = (tiles - prefix + 255) / 256;   // of eight keys per lane
            if (in_registers) {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    const int j = prefix + lane + 32 * i;
                    if (i / 8 < groups) key[i] = j < tiles ? tile_key(mine[j]) : 0u;   // 0 is below every real key
                }
            }
            auto each_key = [&](auto visit) {
                if (in_registers) {
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (i / 8 < groups) visit(key[i]);
                } else {
                    for (int j = prefix + lane; j < tiles; j += 32) visit(tile_key(mine[j]));
                }
            };
            auto how_many = [&](uint32_t least) {
                int count = 0;
                each_key([&](uint32_t k) { count += k >= least; });
                return __reduce_add_sync(0xffffffffu, count);
            };
            uint32_t low = 0xffffffffu, high = 0u;
            each_key([&](uint32_t k) {
                if (k) low = min(low, k);
                high = max(high, k);
            });
            low = __reduce_min_sync(0xffffffffu, low);
            high = __reduce_max_sync(0xffffffffu, high);
            bool exact = false;   // exactly `keep` keys are >= low
            if (high != 0xffffffffu) high++;
            else if (how_many(high) >= keep) low = high;   // NaN scores
            for (int round = 0; high - low > 1u; round++) {
                uint32_t middle = low + (high - low) / 2;
                if (round < 16) {
                    const uint32_t by_value = tile_key(0.5f * key_value(low) + 0.5f * key_value(high));
                    if (by_value > low && by_value < high) middle = by_value;
                }
                const int count = how_many(middle);
                if (count >= keep) low = middle;
                else high = middle;
                exact = count == keep;
                if (exact) break;
            }
            const uint32_t want = exact ? low - 1u : low;
            const int greater = exact ? keep : high > low ? how_many(high) : 0;
            const int remaining = keep - greater;   // how many keys equal to `want` to take
            // Take every larger key and the first `remaining` equal keys in index order;
            // emit ascending.
            int written = 0, equal_seen = 0;
#pragma unroll 4
            for (int base = 0; base < tiles; base += 32) {
                const int j = base + lane;
                bool take = false, equal = false;
                if (j < tiles) {
                    if (j < prefix) {
                        take = true;
                    } else {
                        const uint32_t key = tile_key(mine[j]);
                        take = key > want;
                        equal = key == want;
                    }
                }
                const unsigned eq_mask = __ballot_sync(0xffffffffu, equal);
                if (equal && equal_seen + __popc(eq_mask & ((1u << lane) - 1u)) < remaining)
                    take = true;
                equal_seen += __popc(eq_mask);
                const unsigned take_mask = __ballot_sync(0xffffffffu, take);
                if (take) dst[written + __popc(take_mask & ((1u << lane) - 1u))] = j;
                written += __popc(take_mask);
            }
            if (lane == 0) counts[row] = written;
        }
        if (!compression) continue;

        // pooled softmax, in place, ATen reduction order
        float largest = -CUDART_INF_F, total = 0.0f;
        for (int j = lane; j < tiles; j += 32) largest = fmaxf(largest, mine[j]);
#pragma unroll
        for (int o = 16; o; o >>= 1)
            largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, o));
        if (tiles <= 2048) {
            for (int j = lane; j < tiles; j += 32) {
                const float e = expf(mine[j] - largest);
                mine[j] = e;
                total += e;
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        } else {
            // 1024-thread two-level shuffle-down order of the reference's block variant:
            // virtual thread t = w*32 + lane sums columns t, t+1024, ...
            float warp_sums = 0.0f;  // lane w keeps virtual warp w's sum
            for (int w = 0; w < 32; w++) {
                float part = 0.0f;
                for (int i = 0; i < 4; i++) {
                    const int col = w * 32 + lane + i * 1024;
                    if (col < tiles) part += expf(mine[col] - largest);
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
                part = __shfl_sync(0xffffffffu, part, 0);
                if (lane == w) warp_sums = part;
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) warp_sums += __shfl_down_sync(0xffffffffu, warp_sums, o);
            total = __shfl_sync(0xffffffffu, warp_sums, 0);
            for (int j = lane; j < tiles; j += 32) mine[j] = expf(mine[j] - largest);
        }
        __syncwarp();
        for (int j = lane; j < tiles; j += 32) mine[j] = mine[j] / total;
    }
    if (!compression) return;

    // ---- compression: warp = 32 dims x 4 * QPW query tiles, thread = 4 dims x QPW query tiles ----
    const float4 *pv = reinterpret_cast<const float4 *>(poolv + (size_t)head * tiles * VD);
    const int dim4 = (warp & 3) * 8 + in8, q0 = (warp >> 2) * 4 * QPW + in4;
    float4 acc[QPW];
#pragma unroll
    for (int u = 0; u < QPW; u++) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [](float4 &a, float w, const float4 &v) {
        a.x = fmaf(w, v.x, a.x);
        a.y = fmaf(w, v.y, a.y);
        a.z = fmaf(w, v.z, a.z);
        a.w = fmaf(w, v.w, a.w);
    };
    float4 *stage4 = reinterpret_cast<float4 *>(stage);  // [VCHUNK][VD/4]
    constexpr int PER_THREAD4 = VCHUNK * (VD / 4) / 256;
    float4 next4[PER_THREAD4];
    auto fetch4 = [&](int k0) {
#pragma unroll
        for (int u = 0; u < PER_THREAD4; u++) {
            const int i = tid + u * 256, r = i / (VD / 4);
            next4[u] = k0 + r < tiles ? pv[(size_t)(k0 + r) * (VD / 4) + i % (VD / 4)] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch4(0);
    for (int k0 = 0; k0 < tiles; k0 += VCHUNK) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < PER_THREAD4; u++) stage4[tid + u * 256] = next4[u];
        __syncthreads();
        if (k0 + VCHUNK < tiles) fetch4(k0 + VCHUNK);
        const int n = min(VCHUNK, tiles - k0), whole = n & ~3;
#pragma unroll 2
        for (int r = 0; r < whole; r += 4) {
            float4 w[QPW];
#pragma unroll
            for (int u = 0; u < QPW; u++)
                w[u] = *reinterpret_cast<const float4 *>(row_scores + (size_t)(q0 + 4 * u) * stride + k0 + r);
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const float4 v = stage4[(r + x) * (VD / 4) + dim4];
#pragma unroll
                for (int u = 0; u < QPW; u++) add(acc[u], x == 0 ? w[u].x : x == 1 ? w[u].y : x == 2 ? w[u].z : w[u].w, v);
            }
        }
        for (int r = whole; r < n; r++)
#pragma unroll
            for (int u = 0; u < QPW; u++)
                add(acc[u], row_scores[(size_t)(q0 + 4 * u) * stride + k0 + r], stage4[r * (VD / 4) + dim4]);
    }
#pragma unroll
    for (int u = 0; u < QPW; u++)
        if (q0 + 4 * u < nq)
            reinterpret_cast<float4 *>(compression + ((size_t)head * tiles + qt0 + q0 + 4 * u) * VD)[dim4] = acc[u];
}

// ---- merge ---------------------------------------------------------------------------
// out[row][h][:] = bf16(fmaf(bf16_round(compression[h][tile][:]), gate[row][h][:], sparse))
// for every non-padded tiled row (cuda/vsa.cuh:168-181); one 16-byte vector per thread.
__global__ void __launch_bounds__(256)
untile_merge_kernel(uint4 *output, const uint4 *tiled, const uint4 *gate, const float *compression, const int *map,
                    int tiles, int heads) {
    wait_for_previous_kernel();
    allow_next_kernel();
    const size_t total = (size_t)tiles * VT * heads * (VD / 8);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int v = (int)(i % (VD / 8));
    const int head = (int)((i / (VD / 8)) % heads);
    const int padded = (int)(i / ((size_t)(VD / 8) * heads));
    const int row = map[padded];
    if (row < 0) return;
    const uint4 x = tiled[((size_t)head * tiles * VT + padded) * (VD / 8) + v];
    const size_t dst = ((size_t)row * heads + head) * (VD / 8) + v;
    const uint4 gt = gate[dst];
    const float4 *cp = reinterpret_cast<const float4 *>(
        compression + ((size_t)head * tiles + padded / VT) * VD + v * 8);
    const float4 c0 = cp[0], c1 = cp[1];
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, gs[4] = {gt.x, gt.y, gt.z, gt.w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float lo = fmaf(bf16_round(c[2 * k]), bf16_bits_to_f32(gs[k] & 0xffffu),
                              bf16_bits_to_f32(xs[k] & 0xffffu));
        const float hi = fmaf(bf16_round(c[2 * k + 1]), bf16_bits_to_f32(gs[k] >> 16),
                              bf16_bits_to_f32(xs[k] >> 16));
        o[k] = f32_to_bf16_bits(lo) | (f32_to_bf16_bits(hi) << 16);
    }
    output[dst] = make_uint4(o[0], o[1], o[2], o[3]);
}

}  // namespace

cudaError_t vsa_tile_pool3(const void *const src[3], void *const tiled[3], float *const pooled[3],
                           const int *map, const int *sizes, int tiles, int heads, int count,
                           cudaStream_t stream) {
    PoolArgs a{};
    for (int i = 0; i < count; i++) {
        a.src[i] = static_cast<const uint2 *>(src[i]);
        a.tiled[i] = static_cast<uint2 *>(tiled[i]);
        a.pooled[i] = pooled[i];
    }
    dim3 grid(tiles, (heads + 7) / 8, count);
    return launch_overlapped(a.tiled[0] ? tile_pool_kernel<true> : tile_pool_kernel<false>, grid, 256, 0, stream, a, map, sizes,
                             tiles, heads);
}

template <int QPW>
static cudaError_t launch_score_select(const float *poolq, const float *poolk, const float *poolv,
                                       float *scores, int *indices, int *counts, float *compression,
                                       int tiles, int prefix, int keep, int heads, float scale,
                                       cudaStream_t stream) {
    constexpr int QT = 8 * QPW;
    static thread_local int configured_device = -1;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (configured_device != device) {
        e = cudaFuncSetAttribute(score_select_kernel<QPW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)score_select_smem(QPW == 1 ? 4096 : 2048, QT));
        if (e != cudaSuccess) return e;
        configured_device = device;
    }
    dim3 grid((tiles + QT - 1) / QT, heads);
    return launch_overlapped(score_select_kernel<QPW>, grid, 256, score_select_smem(tiles, QT), stream, poolq, poolk, poolv,
                             scores, indices, counts, compression, tiles, prefix, keep, scale);
}

cudaError_t vsa_score_select_compress(const float *poolq, const float *poolk, const float *poolv,
                                      float *scores, int *indices, int *counts,
                                      float *compression, int tiles, int prefix, int keep,
                                      int heads, float scale, cudaStream_t stream) {
    if (tiles < 1 || tiles > 4096 || keep < 1 || prefix < 0 || prefix > tiles)
        return cudaErrorInvalidValue;
    // 16 query tiles per CTA up to 1400 tiles (two such CTAs share an SM up to 1152 tiles,
    // one beyond), 8 per CTA beyond that: the score rows of a CTA must fit its shared memory.
    // A CTA's time is its own chain of chunks (products bound by shared-memory wavefronts, a dozen counts per query
    // tile for the threshold), so a call takes about one CTA's time as long as every CTA is resident: with few
    // heads (a rank's share under sequence parallelism) 8 tiles per CTA halve that time and still fill the GPU.
    static thread_local int sms_device = -1, sms = 0;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess && device != sms_device) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (e == cudaSuccess) sms_device = device;
    }
    if (e != cudaSuccess) return e;
    if (tiles <= 1400 && (size_t)((tiles + 15) / 16) * heads >= (size_t)4 * sms)
        return launch_score_select<2>(poolq, poolk, poolv, scores, indices, counts, compression, tiles,
                                      prefix, keep, heads, scale, stream);
    return launch_score_select<1>(poolq, poolk, poolv, scores, indices, counts, compression, tiles,
                                  prefix, keep, heads, scale, stream);
}

cudaError_t vsa_untile_merge(void *output, const void *tiled, const void *gate,
                             const float *compression, const int *map, int tiles, int heads,
                             cudaStream_t stream) {
    const size_t total = (size_t)tiles * VT * heads * (VD / 8);
    const size_t blocks = (total + 255) / 256;
    if (blocks > 0x7fffffffu) return cudaErrorInvalidValue;
    return launch_overlapped(untile_merge_kernel, dim3((unsigned)blocks), 256, 0, stream, static_cast<uint4 *>(output),
                             static_cast<const uint4 *>(tiled), static_cast<const uint4 *>(gate), compression, map, tiles,
                             heads);
}

}  // namespace h3b

// ---- top-k tile selection without any allocation -----------------------------------
// For callers that may not allocate device memory at the point of the call: code running
// inside someone else's memory plan (a fixed arena handed out once at start-up), under a
// memory-capped container where a late allocation can fail, or on a real-time path where
// the driver's allocator lock is not acceptable. The pooled means of Q and K - the only
// intermediate the selection needs - live in one file-scope device array instead of buffers
// owned by an h3_gpu_vsa object.
namespace h3b {
namespace {
constexpr unsigned STATIC_TOPK_MAX_ROWS = 8192;  // heads * tiles
// [2][heads * tiles][128] f32 = 8 MiB, resident on every GPU that loads the library.
static __device__ __align__(256) float g_topk_pool[2 * (size_t)STATIC_TOPK_MAX_ROWS * VD];
thread_local char g_topk_error[160] = "";
}  // namespace
}  // namespace h3b

extern "C" const char *h3b_vsa_topk_static_error(void) { return h3b::g_topk_error; }

extern "C" cudaError_t h3b_vsa_topk_static(const void *query, const void *key, const int *map,
                                           const int *sizes, int *indices, int *counts,
                                           unsigned tiles, unsigned prefix, unsigned keep,
                                           unsigned heads, cudaStream_t stream) {
    using namespace h3b;
    g_topk_error[0] = 0;
    if (!query || !key || !map || !sizes || !indices || !counts) {
        snprintf(g_topk_error, sizeof g_topk_error, "h3b_vsa_topk_static: null pointer argument");
        return cudaErrorInvalidValue;
    }
    if (!tiles || !heads || tiles > 4096u || prefix > tiles || !keep || keep > tiles - prefix) {
        snprintf(g_topk_error, sizeof g_topk_error,
                 "h3b_vsa_topk_static: bad geometry (tiles %u, prefix %u, keep %u, heads %u)", tiles,
                 prefix, keep, heads);
        return cudaErrorInvalidValue;
    }
    if ((size_t)heads * tiles > STATIC_TOPK_MAX_ROWS) {
        snprintf(g_topk_error, sizeof g_topk_error,
                 "h3b_vsa_topk_static: heads * tiles = %zu exceeds the static scratch limit of %u",
                 (size_t)heads * tiles, STATIC_TOPK_MAX_ROWS);
        return cudaErrorInvalidValue;
    }
    // Device address of the scratch array, resolved once per device with that device current.
    // (In host code the array's name is only a handle for the runtime, not an address.)
    static float *pool_of_device[64] = {};
    // every failing return leaves its reason in the thread's error text
    auto failed = [](cudaError_t code, const char *where) {
        snprintf(g_topk_error, sizeof g_topk_error, "h3b_vsa_topk_static: %s: %s", where, cudaGetErrorString(code));
        return code;
    };
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return failed(e, "current device");
    if (device < 0 || device >= 64) return failed(cudaErrorInvalidDevice, "device ordinal above 63");
    float *pool = __atomic_load_n(&pool_of_device[device], __ATOMIC_ACQUIRE);
    if (!pool) {
        e = cudaGetSymbolAddress(reinterpret_cast<void **>(&pool), g_topk_pool);
        if (e != cudaSuccess) return failed(e, "address of the static scratch");
        __atomic_store_n(&pool_of_device[device], pool, __ATOMIC_RELEASE);
    }
    float *poolq = pool, *poolk = pool + (size_t)STATIC_TOPK_MAX_ROWS * VD;
    const void *src[3] = {query, key, nullptr};
    void *no_tiled[3] = {nullptr, nullptr, nullptr};
    float *pooled[3] = {poolq, poolk, nullptr};
    e = vsa_tile_pool3(src, no_tiled, pooled, map, sizes, (int)tiles, (int)heads, 2, stream);
    if (e != cudaSuccess) return failed(e, "pooling launch");
    e = vsa_score_select_compress(poolq, poolk, nullptr, nullptr, indices, counts, nullptr, (int)tiles,
                                  (int)prefix, (int)keep, (int)heads, 1.0f / sqrtf(128.0f), stream);
    return e == cudaSuccess ? e : failed(e, "selection launch");
}

// Decode attention whose keys and values come by TMA: heads of 64 or 128 values, at most eight query heads to a kv head, pages of 16
// positions and more.
//
// The kernels of attention_decode_staged.cuh let the 128 threads of a block gather every tile themselves (look-ups, address
// arithmetic, cp.async, a barrier of the block per tile): 550 instructions a warp and tile of 64 keys, and with two warps a
// scheduler the step waited for them, not for the memory. Here a fifth warp does nothing but look pages up and ask for
// tiles (one TMA box per page, half of a head and plane, straight from the cache seen as a matrix of rows, into the 128-byte swizzle) in
// a ring of three, as far ahead as the ring allows and across the stretches of a block; the four consuming warps wait for a tile
// (mbarrier), take their 16 keys of it and give it back, without meeting one another before the end of a stretch. The tensor cores'
// rows 8 to 15 are always zero with at most eight heads, so their half of the softmax is left out. What is left is the stream of
// the cache: 8 rows of 4,095 keys, 32 heads over 8, 26.3 us (32.8 before, 19.9 at the memory's rate); 64 rows of 1,800 keys 77 (91
// before, 68); 32 rows of 4,096 keys, 40 heads 80 (105 before, 78); one row of 777 keys 7.2 (8.5 before: launch, look-ups and the
// meeting of its parts).
// Work, partials, counters and the combining are those of the staged kernels. Every mbarrier wait is bounded and raises the error
// word of the tcgen05 attention kernels (51: producer, 52: consumers).
#pragma once
#include "attention_decode_staged.cuh"
#include "tcgen05_common.cuh"

int* jllm_attention_tc_error_word_ptr();   // attention_prefill_tc.cu

namespace ring {

using staged::Extras;
using staged::Fresh;
using staged::TILE;

constexpr int STAGES = 3, CONSUMERS = 128, THREADS = 160, HEADS = 8;

template <int HD>
struct Layout {
    static constexpr int TILE_BYTES = TILE * HD * 2, STAGE_BYTES = 2 * TILE_BYTES, HALVES = HD / 64;
    static constexpr int Q = STAGES * STAGE_BYTES;                 // [HEADS][HD] queries
    static constexpr int AREA = Q + HEADS * HD * 2;                // [2][HEADS][HD] float: the warps' sums meet here
    static constexpr int ML = AREA + 2 * HEADS * HD * 4;           // [4][HEADS][2] float: maximum, weight
    static constexpr int FRESH = ML + 4 * HEADS * 2 * 4;           // [2][HD]: the row's newest key and value
    static constexpr int BARS = FRESH + 2 * HD * 2;                // full [STAGES], empty [STAGES], abort flag
    static constexpr size_t BYTES = BARS + 8 * 2 * STAGES + 16;
};

// the four consuming warps meet
__device__ __forceinline__ void meet() { asm volatile("barrier.cta.sync 1, 128;" ::: "memory"); }

// one stretch of a block's work: tiles [tile_lo, tile_lo + n_tiles) of one (row, kv head)
struct Stretch {
    int r, kvh, P, first, tile_lo, n_tiles;
    const int* table;
};

struct Args {
    const __nv_bfloat16* q;
    int q_stride;
    __nv_bfloat16* out;
    int out_stride;
    const int *row_seg, *row_pos, *block_tables;
    int table_stride, rows, heads, kv_heads, page_size, page_shift, num_pages, window;
    float scale_log2;
    int splits;
    float *part_o, *part_ml;
    int* counters;
    Fresh fresh;
    VecRef sink;
    int has_sink;
    ScoreCap cap;
    int* error_word;
};

// byte offset of 16-byte chunk c of row r in a tile of 64 rows: halves of 64 columns, 128-byte swizzle
__device__ __forceinline__ uint32_t off(int r, int c) { return (uint32_t)((c >> 3) * (TILE * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)); }

// The producing warp: the tiles of a stretch, as numbers seq, seq + 1, ... of the ring. `from`, `to`: which of them now.
template <int HD>
__device__ __forceinline__ bool produce(uint32_t base, const Args& a, const CUtensorMap* map_k, const CUtensorMap* map_v, const Stretch& s,
                                        uint32_t seq, int from, int to, volatile int* abort_flag) {
    using L = Layout<HD>;
    const int lane = threadIdx.x & 31;
    const int per_page = 2 * L::HALVES, pages = max(1, TILE >> a.page_shift), rows_box = min(a.page_size, TILE);
    const int p = lane / per_page, which = lane % per_page / L::HALVES, half = lane % L::HALVES;
    for (int i = from; i < to; ++i) {
        const uint32_t n = seq + i, stage = n % STAGES;
        const int key0 = s.first + (s.tile_lo + i) * TILE, key = key0 + p * rows_box;       // (a tile starts at a page's or a box's edge)
        const bool mine = p < pages && key <= s.P;                                           // a page without a live key is left out
        int y = 0;
        if (mine) {
            // checked build: a bad entry gives -1 and a box of negative rows, which TMA fills with zeros
            const long long page = jllm_page_of(s.table, key >> a.page_shift, a.table_stride, a.num_pages);
            y = (int)((page * a.kv_heads + s.kvh) * a.page_size) + (key & (a.page_size - 1));
        }
        if (n >= STAGES) {
            bool ok = true;
            if (lane == 0) ok = tc::mbar_wait(base + L::BARS + 8 * (STAGES + stage), (n / STAGES - 1) & 1u, abort_flag);
            if (!__shfl_sync(0xffffffffu, ok, 0)) return false;
        }
        const int live = min(pages, (s.P - key0) / rows_box + 1);
        const uint32_t full = base + L::BARS + 8 * stage;
        if (lane == 0) tc::mbar_expect_tx(full, live * rows_box * HD * 4);
        __syncwarp();
        if (mine)
            tc::tma_load_2d(base + stage * L::STAGE_BYTES + which * L::TILE_BYTES + half * (TILE * 128) + p * rows_box * 128,
                            which ? map_v : map_k, half * 64, y, full);
    }
    return true;
}

// The consuming warps: one stretch. The result goes to `out` if these are all the row's keys (`whole`), else as a partial (sums, maximum,
// weight) for head j of the group to part_o + j * o_stride and part_ml + j * ml_stride.
template <int HD>
__device__ __forceinline__ bool consume(uint8_t* smem, uint32_t base, const Args& a, const Stretch& s, uint32_t seq, bool whole,
                                        float* part_o, size_t o_stride, float* part_ml, size_t ml_stride, bool ok, volatile int* abort_flag) {
    using L = Layout<HD>;
    constexpr int CHUNKS = HD / 8, V = HD / 64;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int G = a.heads / a.kv_heads;
    uint8_t* s_q = smem + L::Q;
    __nv_bfloat16* s_fresh = reinterpret_cast<__nv_bfloat16*>(smem + L::FRESH);
    const bool fused = a.fresh.qkv != nullptr;
    const int fresh_tile = (s.P - s.first) / TILE - s.tile_lo;      // of this stretch's tiles, the one with position P (if any)
    if (fused) {
        // the queries: a warp per head, norm and rotation in registers; the newest key (warp 0) and value (warp 1) where they are ours
        const bool makes_kv = fresh_tile >= 0 && fresh_tile < s.n_tiles;
        const __nv_bfloat16* mine = a.fresh.qkv + (size_t)s.r * a.fresh.stride;
        const float *cos_row = a.fresh.cos_t + (size_t)s.P * (HD / 2), *sin_row = a.fresh.sin_t + (size_t)s.P * (HD / 2);
        float ka[V], kb[V];
        uint4 vv = make_uint4(0, 0, 0, 0);
        if (makes_kv && warp == 0) staged::head_load<V>(mine + (size_t)(a.heads + s.kvh) * HD, lane, ka, kb);
        if (makes_kv && warp == 1 && lane < CHUNKS)
            vv = *reinterpret_cast<const uint4*>(mine + (size_t)(a.heads + a.kv_heads + s.kvh) * HD + lane * 8);
        for (int row = warp; row < HEADS; row += 4) {
            if (row < G) {
                float qa[V], qb[V];
                staged::head_load<V>(mine + (size_t)(s.kvh * G + row) * HD, lane, qa, qb);
                head_norm_rope<V>(qa, qb, lane, a.fresh.use_norm, a.fresh.eps, a.fresh.q_gain, cos_row, sin_row);
                staged::head_store<HD>(s_q, row, lane, qa, qb);
            } else if (lane < CHUNKS) {
                *reinterpret_cast<uint4*>(s_q + staged::off<HD>(row, lane)) = make_uint4(0, 0, 0, 0);
            }
        }
        if (makes_kv && warp < 2) {
            const long long page = jllm_page_of(s.table, s.P >> a.page_shift, a.table_stride, a.num_pages);   // -1: checked build, bad entry
            const bool writes = !kCheckBounds || page >= 0;
            const size_t at = writes ? (((size_t)page * a.kv_heads + s.kvh) * a.page_size + (s.P & (a.page_size - 1))) * HD : 0;
            if (warp == 0) {
                head_norm_rope<V>(ka, kb, lane, a.fresh.use_norm, a.fresh.eps, a.fresh.k_gain, cos_row, sin_row);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const int e0 = lane * V + i, e1 = HD / 2 + e0;
                    const __nv_bfloat16 v0 = __float2bfloat16_rn(ka[i]), v1 = __float2bfloat16_rn(kb[i]);
                    s_fresh[e0] = v0, s_fresh[e1] = v1;
                    if (writes) a.fresh.k_out[at + e0] = v0, a.fresh.k_out[at + e1] = v1;
                }
            } else if (lane < CHUNKS) {
                reinterpret_cast<uint4*>(s_fresh + HD)[lane] = vv;
                if (writes) *reinterpret_cast<uint4*>(a.fresh.v_out + at + lane * 8) = vv;
            }
        }
    } else if (tid < HEADS * CHUNKS) {
        const int row = tid / CHUNKS, c = tid % CHUNKS;
        *reinterpret_cast<uint4*>(s_q + staged::off<HD>(row, c)) =
            row < G ? *reinterpret_cast<const uint4*>(a.q + (size_t)s.r * a.q_stride + (size_t)(s.kvh * G + row) * HD + c * 8)
                    : make_uint4(0, 0, 0, 0);
    }
    meet();
    // the queries' fragments of rows 0 to 7 (a0 and a2 of two k steps at a time); a1 and a3, rows 8 to 15, are zero
    uint32_t qf[HD / 16][2];
#pragma unroll
    for (int ks = 0; ks < HD / 16; ks += 2) {
        uint32_t x[4];
        staged::ldsm4(x, base + L::Q + staged::off<HD>(lane & 7, ks * 2 + (lane >> 3)));
        qf[ks][0] = x[0], qf[ks][1] = x[1], qf[ks + 1][0] = x[2], qf[ks + 1][1] = x[3];
    }
    float o[HD / 8][4];
#pragma unroll
    for (int j = 0; j < HD / 8; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[j][i] = 0.f;
    float m = -INFINITY, l = 0.f;
    // where this lane's rows of a tile begin: keys for K (non-transposed) and V (transposed) fragments
    const int krow = warp * 16 + (lane & 7) + ((lane >> 4) << 3), vrow = warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
    for (int i = 0; i < s.n_tiles; ++i) {
        const uint32_t n = seq + i, stage = n % STAGES;
        ok = ok && tc::mbar_wait(base + L::BARS + 8 * stage, (n / STAGES) & 1u, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        const int key0 = s.first + (s.tile_lo + i) * TILE + warp * 16;
        if (ok && key0 <= s.P) {                        // (else the warp's keys of the last tile are all past the end)
            const uint32_t sk = base + stage * L::STAGE_BYTES, sv = sk + L::TILE_BYTES;
            if (key0 + 15 >= s.P) {                     // the warp with position P: a warp reads its own 16 rows only
                uint8_t* tile = smem + stage * L::STAGE_BYTES;
                const int last = s.P - key0;            // values past the end may be anything: zero them (scores are masked)
                for (int e = lane; e < (15 - last) * CHUNKS; e += 32)
                    *reinterpret_cast<uint4*>(tile + L::TILE_BYTES + off(warp * 16 + last + 1 + e / CHUNKS, e % CHUNKS)) = make_uint4(0, 0, 0, 0);
                if (fused && lane < 2 * CHUNKS)         // the copy brought whatever the cache held there
                    *reinterpret_cast<uint4*>(tile + lane / CHUNKS * L::TILE_BYTES + off(warp * 16 + last, lane % CHUNKS)) =
                        reinterpret_cast<const uint4*>(s_fresh)[lane];
                tc::fence_async_proxy();                // (the next copy into this stage comes behind these stores)
                __syncwarp();
            }
            float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
                uint32_t kf[4];
                staged::ldsm4(kf, sk + off(krow, ks * 2 + ((lane >> 3) & 1)));
                const uint32_t qa[4] = {qf[ks][0], 0u, qf[ks][1], 0u};
                staged::mma(sc[0], qa, kf[0], kf[1]);
                staged::mma(sc[1], qa, kf[2], kf[3]);
            }
            float mx = -INFINITY;
#pragma unroll
            for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int key = key0 + tile * 8 + 2 * t + e;
                    sc[tile][e] = key <= s.P ? (a.cap ? a.cap(sc[tile][e]) : sc[tile][e] * a.scale_log2) : -INFINITY;
                    mx = fmaxf(mx, sc[tile][e]);
                }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m, mx);           // finite: key0 <= P, so the warp sees at least one key
            const float corr = staged::ex2(m - m_new);
            m = m_new;
            uint32_t pf[4] = {0u, 0u, 0u, 0u};
            l *= corr;
#pragma unroll
            for (int tile = 0; tile < 2; ++tile) {
                const float p0 = staged::ex2(sc[tile][0] - m), p1 = staged::ex2(sc[tile][1] - m);
                l += p0 + p1;
                __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
                pf[tile * 2] = *reinterpret_cast<uint32_t*>(&b);
            }
            if (!__all_sync(0xffffffffu, corr == 1.f)) {       // a row's maximum moved
#pragma unroll
                for (int j = 0; j < HD / 8; ++j) o[j][0] *= corr, o[j][1] *= corr;
            }
#pragma unroll
            for (int jp = 0; jp < HD / 16; ++jp) {
                uint32_t vf[4];
                staged::ldsm4t(vf, sv + off(vrow, jp * 2 + (lane >> 4)));
                staged::mma(o[2 * jp], pf, vf[0], vf[1]);
                staged::mma(o[2 * jp + 1], pf, vf[2], vf[3]);
            }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(base + L::BARS + 8 * (STAGES + stage));
    }
    // ---- the four warps' sums: warps 2 and 3 lay theirs down, 0 and 1 add their own, then the two halves are added ----
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    float* area = reinterpret_cast<float*>(smem + L::AREA);
    float* sml = reinterpret_cast<float*>(smem + L::ML);
    if (t == 0) {
        sml[(warp * HEADS + g) * 2] = m;
        sml[(warp * HEADS + g) * 2 + 1] = l;
    }
    meet();
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) top = fmaxf(top, sml[(w * HEADS + g) * 2]);
    const float scale_w = m == -INFINITY ? 0.f : exp2f(m - top);
    float2* mine = reinterpret_cast<float2*>(area + (size_t)((warp & 1) * HEADS + g) * HD + 2 * t);
    if (warp >= 2 && g < G) {
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) mine[j * 4] = make_float2(o[j][0] * scale_w, o[j][1] * scale_w);
    }
    meet();
    if (warp < 2 && g < G) {
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) {
            const float2 x = mine[j * 4];
            mine[j * 4] = make_float2(o[j][0] * scale_w + x.x, o[j][1] * scale_w + x.y);
        }
    }
    meet();
    for (int e = tid; e < G * HD; e += CONSUMERS) {
        const int row = e / HD, d = e % HD;
        float acc = area[row * HD + d] + area[(HEADS + row) * HD + d], mm = -INFINITY, ll = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) mm = fmaxf(mm, sml[(w * HEADS + row) * 2]);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float mw = sml[(w * HEADS + row) * 2];
            ll += mw == -INFINITY ? 0.f : sml[(w * HEADS + row) * 2 + 1] * exp2f(mw - mm);
        }
        if (whole) {
            if (a.has_sink) {         // (2^(sink - max) may overflow where every score lies far below the sink: the result is 0)
                const float sl = a.sink[s.kvh * G + row] * LOG2E, above = fmaxf(mm, sl);
                acc *= exp2f(mm - above);
                ll = ll * exp2f(mm - above) + exp2f(sl - above);
            }
            a.out[(size_t)s.r * a.out_stride + (size_t)(s.kvh * G + row) * HD + d] = __float2bfloat16_rn(acc / ll);
        } else {
            part_o[(size_t)row * o_stride + d] = acc;
            if (d == 0) {
                part_ml[(size_t)row * ml_stride] = mm;
                part_ml[(size_t)row * ml_stride + 1] = ll;
            }
        }
    }
    return ok;
}

// true in all consuming threads of the one block that is the `expected`-th of a pair to arrive (see staged::last_of_pair)
__device__ __forceinline__ bool last_of_pair(int* counter, int expected, volatile int* s_last) {
    __threadfence();
    meet();
    if (threadIdx.x == 0) {
        const int seen = atomicAdd(counter, 1);
        *s_last = seen == expected - 1;
        if (seen == expected - 1) *counter = 0;
    }
    meet();
    const bool last = *s_last != 0;
    if (last) __threadfence();
    return last;
}

// FLAT: the key tiles of all (row, kv head) pairs dealt out evenly over the blocks (staged::attention_decode_flat_kernel); else one
// block per (row, kv head, split).
template <int HD, bool FLAT>
__global__ void __launch_bounds__(THREADS, 2)
attention_decode_ring_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ Args a) {
    using L = Layout<HD>;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ int s_cum[FLAT ? staged::FLAT_MAX_ROWS + 1 : 1];
    __shared__ int s_last;
    const uint32_t base = tc::smem_u32(smem);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::BARS + 8 * 2 * STAGES);
    const int warp = threadIdx.x >> 5, G = a.heads / a.kv_heads;
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            tc::mbar_init(base + L::BARS + 8 * i, 1);
            tc::mbar_init(base + L::BARS + 8 * (STAGES + i), 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (FLAT) {
        pdl_wait();
        pdl_trigger();
        if (threadIdx.x < 32) staged::flat_prefix(a.row_pos, a.rows, a.window, s_cum);
        __syncthreads();
        const long long all = (long long)a.kv_heads * s_cum[a.rows];
        const long long end = all * (blockIdx.x + 1) / gridDim.x;
        long long at = all * blockIdx.x / gridDim.x;
        int lo = 0, hi = a.rows - 1;                     // the row whose tiles hold position `at`
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if ((long long)a.kv_heads * s_cum[mid + 1] <= at) lo = mid + 1; else hi = mid;
        }
        int r = lo;
        uint32_t seq = 0;
        bool ok = true;
        while (at < end) {
            while ((long long)a.kv_heads * s_cum[r + 1] <= at) ++r;
            const int tiles_r = s_cum[r + 1] - s_cum[r];
            const long long in_row = at - (long long)a.kv_heads * s_cum[r];
            const int P = a.row_pos[r];
            const Stretch s{r, (int)(in_row / tiles_r), P, jllm_first_key(P, a.window), (int)(in_row % tiles_r),
                            (int)min((long long)(tiles_r - in_row % tiles_r), end - at), a.block_tables + (size_t)a.row_seg[r] * a.table_stride};
            if (warp == 4) {
                ok = produce<HD>(base, a, &map_k, &map_v, s, seq, 0, s.n_tiles, abort_flag);
                if (!ok) break;
            } else {
                const size_t slot = (size_t)r * a.kv_heads + s.kvh + blockIdx.x;
                // the blocks whose runs meet this pair follow one another (the host sees to it that no run is empty)
                const long long start = at - s.tile_lo;
                auto block_of = [&](long long tile) { return (int)(((tile + 1) * gridDim.x + all - 1) / all - 1); };
                const int b_first = block_of(start), parts = block_of(start + tiles_r - 1) - b_first + 1;
                const bool alone = a.counters != nullptr && parts == 1;       // this block has all of the pair: no partial
                ok = consume<HD>(smem, base, a, s, seq, alone, a.part_o + slot * G * HD, (size_t)HD, a.part_ml + slot * G * 2, (size_t)2, ok,
                                 abort_flag);
                if (a.counters != nullptr && !alone && last_of_pair(a.counters + (size_t)r * a.kv_heads + s.kvh, parts, &s_last)) {
                    const size_t slot0 = (size_t)r * a.kv_heads + s.kvh + b_first;      // the slots of the pair's parts follow one another
                    staged::combine_pair<HD>(a.part_o + slot0 * G * HD, (size_t)G * HD, (size_t)HD, a.part_ml + slot0 * G * 2, (size_t)G * 2,
                                             (size_t)2, parts, G, a.out + (size_t)r * a.out_stride + (size_t)s.kvh * G * HD);
                }
            }
            at += s.n_tiles;
            seq += s.n_tiles;
        }
        if (!ok && (threadIdx.x & 31) == 0) { *abort_flag = 1; atomicExch(a.error_word, warp == 4 ? 51 : 52); }
    } else {
        const int r = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
        const int P = a.row_pos[r], first = jllm_first_key(P, a.window);
        const int tiles_total = (P + 1 - first + TILE - 1) / TILE, per_split = (tiles_total + a.splits - 1) / a.splits;
        const int tile_lo = split * per_split, n_tiles = max(0, min(tiles_total, tile_lo + per_split) - tile_lo);
        const Stretch s{r, kvh, P, first, tile_lo, n_tiles, a.block_tables + (size_t)a.row_seg[r] * a.table_stride};
        __syncthreads();
        bool ok = true;
        if (warp == 4) {
            // Tiles that end before position P were written by earlier steps, and positions and tables came from the host: the first
            // of them are asked for while the kernel in front still runs.
            const int before = max(0, min(min(n_tiles, STAGES), (P - first) / TILE - tile_lo));
            ok = produce<HD>(base, a, &map_k, &map_v, s, 0, 0, before, abort_flag);
            pdl_wait();
            pdl_trigger();
            ok = ok && produce<HD>(base, a, &map_k, &map_v, s, 0, before, n_tiles, abort_flag);
        } else {
            pdl_wait();
            pdl_trigger();
            // partials: (row, head, split) -> head_dim sums in part_o, (maximum, weight) in part_ml
            const size_t slot = ((size_t)r * a.heads + kvh * G) * a.splits + split;
            ok = consume<HD>(smem, base, a, s, 0, a.splits == 1, a.part_o + slot * HD, (size_t)a.splits * HD, a.part_ml + slot * 2,
                             (size_t)a.splits * 2, true, abort_flag);
            // (without counters a combine kernel follows)
            if (a.splits > 1 && a.counters != nullptr && last_of_pair(a.counters + (size_t)r * a.kv_heads + kvh, a.splits, &s_last)) {
                const size_t slot0 = ((size_t)r * a.heads + kvh * G) * a.splits;
                Extras ex;
                ex.sink = a.sink;
                ex.has_sink = a.has_sink;
                staged::combine_pair<HD>(a.part_o + slot0 * HD, (size_t)HD, (size_t)a.splits * HD, a.part_ml + slot0 * 2, (size_t)2,
                                         (size_t)a.splits * 2, a.splits, G, a.out + (size_t)r * a.out_stride + (size_t)kvh * G * HD, ex, kvh * G);
            }
        }
        if (!ok && (threadIdx.x & 31) == 0) { *abort_flag = 1; atomicExch(a.error_word, warp == 4 ? 51 : 52); }
    }
}

// Whether these kernels take a step: what the boxes and the eight rows need. Every row's first visible key has to lie at a page's start: all
// keys, or chunks of whole pages.
inline bool fits(int heads, int kv_heads, int head_dim, int page_size, int window, int keep_first) {
    return (head_dim == 64 || head_dim == 128) && heads / kv_heads <= HEADS && page_size >= 16 && (page_size & (page_size - 1)) == 0 &&
           keep_first == 0 && (window == 0 || (window < 0 && -window % page_size == 0));
}

template <int HD, bool FLAT>
int launch(Args a, const void* k_cache, const void* v_cache, dim3 grid, cudaStream_t stream) {
    using L = Layout<HD>;
    a.page_shift = 0;
    while ((1 << a.page_shift) < a.page_size) ++a.page_shift;
    a.num_pages = jllm_pool_pages();
    a.error_word = jllm_attention_tc_error_word_ptr();
    if (!a.error_word) return jllm_fail(JLLM_CUDA_ERROR, "attention_decode: no error word");
    // (the cache's length is not known here; the tables name the pages, as for the kernels without a map)
    CUtensorMap map_k, map_v;
    const int box = a.page_size < TILE ? a.page_size : TILE;
    int rc = tc::tensor_map_for(k_cache, 0x7fffffffll, HD, HD, box, &map_k);
    if (rc == JLLM_OK) rc = tc::tensor_map_for(v_cache, 0x7fffffffll, HD, HD, box, &map_v);
    if (rc != JLLM_OK) return rc;
    auto kern = attention_decode_ring_kernel<HD, FLAT>;
    if (jllm_allow_smem((const void*)kern, L::BYTES) != cudaSuccess)
        return jllm_fail(JLLM_CUDA_ERROR, "attention_decode: %zu bytes of shared memory refused", L::BYTES);
    jllm_launch(kern, grid, dim3(THREADS), L::BYTES, stream, LAUNCH_DEPENDENT, map_k, map_v, a);
    return JLLM_OK;
}

}  // namespace ring

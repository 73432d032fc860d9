// Paged causal flash attention for prompt portions on tcgen05 where ONE cached row of 256 values is key and value at once
// (attention over a cached latent).
//
// One block per (128 query rows of a segment, head). A key tile (128 rows x 256) is loaded once and serves both products:
//     S = Q K^T      A = Q tile [128 x 256], B = key tile (K-major), D = S in tensor memory (two buffers of 128 columns);
//     O += P K       A = P from tensor memory (packed bfloat16 over its own S), B = the same bytes as an MN-major operand,
//                    D = O in tensor memory (256 columns, or the first `value_quarters` x 64 of them: a caller that reads
//                    fewer of a head's columns is not charged for the others).
// A tile travels in four pieces of 64 columns through a ring of ten 16 KB slots. Both products walk it piece by piece, so a
// piece is given back as soon as its part of O is done (a piece with no part in O after its part of S), and with 64 KB for Q the
// ring still holds two and a half tiles. S of tile j + 1 is issued in front of O += P_j K_j, so the softmax of one tile runs
// beside the products of its neighbours. Two softmax warpgroups share a tile's columns (64 each, the row's maximum exchanged
// through shared memory): one warp a scheduler alone is bound by the latency of its own chain of 128 exponentials.
// The MMAs of one thread complete in order, so S_(j+2) may overwrite P_j once O += P_j K_j has been issued.
// What bounds it is a block's chain, not a unit: a key tile's products are 2,048 clocks on the tensor cores and as many of
// shared-memory reads, its exponentials 1,024, and a tile takes 2.7 us (5,200 clocks; 16 heads of 128 rows over 8,000 keys, 16
// blocks, 179 us; over none 8.8): scores, their maxima, the exponentials and the next product wait for one another with one
// block to an SM, and only neighbouring tiles overlap. A causal prompt of 2,048 rows x 16 heads: 274 us on mma.sync
// (attention_prefill.cu, which fetches every row twice and keeps 64-key tiles), 62 us here, 54 where 192 of the 256 columns are
// read: 2,176 key tiles over 148 SMs are 40 of them, the rest is the blocks' starts and ends and the uneven last ones.
// Every mbarrier wait is bounded; the softmax threads agree at the exchange of the maxima whether to go on.
//
// Requirements: bfloat16, rows of 256 values, page_size a power of two <= 128, 16-byte aligned q rows.
#include "tcgen05_common.cuh"

namespace {

using namespace tc;

constexpr int BQ = 128, BKV = 128, W = 256, QUARTERS = W / 64, THREADS = 320;
constexpr int PIECE_BYTES = 128 * 64 * 2;          // 128 rows x 64 columns
constexpr int SLOTS = 10;
constexpr float LOG2E = 1.4426950408889634f;
constexpr int BARS = 1 + 2 * SLOTS + 6;
constexpr size_t TAIL_BYTES = 2 * 2 * BQ * sizeof(float) + 8 * BARS + 16;
constexpr size_t SMEM_BYTES = (QUARTERS + SLOTS) * PIECE_BYTES + TAIL_BYTES;      // (no room to round the base up: it is declared aligned)
static_assert(SMEM_BYTES <= 227 * 1024, "does not fit an SM");
constexpr int TMEM_COLS = 512;                      // S0 0, S1 128, O 256
// M = 128, N = 64, A K-major (from tensor memory), B MN-major
constexpr uint32_t IDESC_128x64_KMN = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24) | (1u << 16);

__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The 256 softmax threads meet; true if `ok` holds for all of them.
__device__ __forceinline__ bool softmax_meet(bool ok) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, 256, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all) : "r"((uint32_t)ok) : "memory");
    return all != 0;
}

template <bool CAP>
__global__ void __launch_bounds__(THREADS, 1)
attention_prefill_latent_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                const __nv_bfloat16* __restrict__ cache, __nv_bfloat16* __restrict__ out, int out_stride,
                                const int* __restrict__ seg_start, const int* __restrict__ seg_len,
                                const int* __restrict__ seg_kv_len, const int* __restrict__ block_tables, int table_stride,
                                int num_segs, int heads, int kv_heads, int page_size, int page_shift, int num_pages, int window,
                                int value_quarters, float scale_log2, int* __restrict__ error_word, ScoreCap cap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t base = smem_u32(smem);
    auto s_q = [&](int c) { return base + c * PIECE_BYTES; };
    auto s_k = [&](int slot) { return base + (QUARTERS + slot) * PIECE_BYTES; };
    float* row_max = reinterpret_cast<float*>(smem + (QUARTERS + SLOTS) * PIECE_BYTES);      // [2 tiles][2 halves][128]
    const uint32_t bars = smem_u32(row_max + 4 * BQ);
    enum { Q_FULL = 0, FULL = 1, EMPTY = FULL + SLOTS, S_FULL = EMPTY + SLOTS, P_READY = S_FULL + 2, PV_DONE = P_READY + 2 };
    auto bar = [&](int i) { return bars + 8u * i; };
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(row_max + 4 * BQ) + 2 * BARS;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);

    // ---- which tile of which segment: the tiles with the most keys before them start first ----
    int seg = 0, tile = gridDim.y - 1 - blockIdx.y;
    for (; seg < num_segs; ++seg) {
        const int nt = (seg_len[seg] + BQ - 1) / BQ;
        if (tile < nt) break;
        tile -= nt;
    }
    if (seg >= num_segs) return;                       // whole block: before any barrier or allocation
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int head = blockIdx.x, kvh = head / (heads / kv_heads);
    const int n_rows = seg_len[seg], q0 = tile * BQ;
    const int rows_here = min(BQ, n_rows - q0);
    const int row0 = seg_start[seg] + q0;
    const int pos0 = seg_kv_len[seg] - n_rows + q0, pos_last = pos0 + rows_here - 1;
    const int first_key = jllm_first_key(pos0, window);     // (the tile's first row sees the earliest key)
    const int kt_lo = first_key / BKV;
    const int n_tiles = pos_last / BKV - kt_lo + 1;
    const int* table = block_tables + (size_t)seg * table_stride;

    if (threadIdx.x == 0) {
        mbar_init(bar(Q_FULL), 1);
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(bar(FULL + s), 1);
            mbar_init(bar(EMPTY + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar(S_FULL + b), 1);
            mbar_init(bar(P_READY + b), 256);
            mbar_init(bar(PV_DONE + b), 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        // ---------------- loader ----------------
        bool ok = true;
        if (lane == 0) {
            mbar_expect_tx(bar(Q_FULL), QUARTERS * PIECE_BYTES);
            for (int c = 0; c < QUARTERS; ++c) tma_load_2d(s_q(c), &map_q, head * W + c * 64, row0, bar(Q_FULL));
        }
        const int pages = BKV >> page_shift;                   // pages of a tile
        auto is_whole = [&](int j) {                           // every row of tile j is a live, written key
            const int key0 = (kt_lo + j) * BKV;
            return key0 >= first_key && key0 + BKV - 1 <= pos_last;
        };
        auto row_of = [&](int j, int p) {                      // the cache row at which page p of tile j starts
            // checked build: a bad entry gives -1 and a box of negative rows, which TMA fills with zeros
            const long long pg = jllm_page_of(table, (((kt_lo + j) * BKV) >> page_shift) + p, table_stride, num_pages);
            return (int)((pg * kv_heads + kvh) * page_size);
        };
        // a lane's page of the next tile is looked up a tile ahead: the look-up is a trip to L2. (A page without a live key has no
        // entry to look up.)
        auto look_up = [&](int j) {
            const int key0 = (kt_lo + j) * BKV + (lane << page_shift);
            return lane < pages && key0 <= pos_last && key0 + page_size > first_key ? row_of(j, lane) : 0;
        };
        int y_next = look_up(0);
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int y_mine = y_next;
            const bool whole = is_whole(j);
            if (j + 1 < n_tiles) y_next = look_up(j + 1);
            const __nv_bfloat16* edge[4];                      // an edge tile's rows lane, lane + 32, ...: where they lie, and if they live
            int bytes[4];
            if (!whole) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int r = lane + 32 * k, key = (kt_lo + j) * BKV + r, p = r >> page_shift;
                    const bool live = key >= first_key && key <= pos_last;
                    int y = __shfl_sync(0xffffffffu, y_mine, p & 31);
                    if (p >= 32) y = live ? row_of(j, p) : 0;
                    bytes[k] = live && y >= 0 ? 16 : 0;        // (y < 0: the checked build's bad entry)
                    edge[k] = cache + (bytes[k] ? (size_t)(y + (r & (page_size - 1))) * W : 0);
                }
            }
            for (int c = 0; c < QUARTERS; ++c) {
                const int n = j * QUARTERS + c, slot = n % SLOTS;
                if (n >= SLOTS) {
                    if (lane == 0) ok = mbar_wait(bar(EMPTY + slot), (uint32_t)(n / SLOTS - 1) & 1u, abort_flag);
                    ok = __shfl_sync(0xffffffffu, ok, 0);
                    if (!ok) break;
                }
                if (whole) {
                    if (lane == 0) mbar_expect_tx(bar(FULL + slot), PIECE_BYTES);
                    __syncwarp();
                    for (int p = lane; p < pages; p += 32)
                        tma_load_2d(s_k(slot) + ((p << page_shift) << 7), &map_k, c * 64, p < 32 ? y_mine : row_of(j, p), bar(FULL + slot));
                } else {
                    // edge tile: a lane's four rows piece by piece, zeros where no live key is (the barrier's arrival follows behind
                    // the four pieces; one warp does this, so what counts is its instructions)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int ch = 0; ch < 8; ++ch)
                            cp_async_16(s_k(slot) + (lane + 32 * k) * 128 + ((ch ^ (lane & 7)) << 4), edge[k] + c * 64 + ch * 8, bytes[k]);
                }
            }
            if (ok && !whole) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                fence_async_proxy();
                __syncwarp();
                if (lane < QUARTERS) mbar_arrive(bar(FULL + (j * QUARTERS + lane) % SLOTS));
            }
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(error_word, 41); }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // (the whole warp walks the tiles, one elected lane issues: see tcgen05_common.cuh)
        {
            bool ok = warp_wait(bar(Q_FULL), 0, abort_flag);
            auto issue_s = [&](int j) {       // S[j & 1] = Q K_j^T, piece by piece
                const uint32_t d = tmem_base + (j & 1) * 128;
#pragma unroll 1
                for (int c = 0; c < QUARTERS; ++c) {
                    const int n = j * QUARTERS + c, slot = n % SLOTS;
                    if (!warp_wait(bar(FULL + slot), (uint32_t)(n / SLOTS) & 1u, abort_flag)) return false;
                    tcgen05_fence_after();
                    if (elect_one()) {
                        const uint64_t q = smem_desc_sw128(s_q(c)), key = smem_desc_sw128(s_k(slot));
#pragma unroll
                        for (int k = 0; k < 4; ++k) tcgen05_mma_bf16(d, q + 2 * k, key + 2 * k, IDESC_128x128_KK, (c > 0 || k > 0) ? 1u : 0u);
                        if (c >= value_quarters) tcgen05_commit(bar(EMPTY + slot));
                        if (c == QUARTERS - 1) tcgen05_commit(bar(S_FULL + (j & 1)));
                    }
                    __syncwarp();
                }
                return true;
            };
            if (ok) ok = issue_s(0);
            for (int j = 0; j < n_tiles && ok; ++j) {
                if (j + 1 < n_tiles) ok = issue_s(j + 1);
                if (!ok || !warp_wait(bar(P_READY + (j & 1)), (uint32_t)(j >> 1) & 1u, abort_flag)) {
                    ok = false;
                    break;
                }
                tcgen05_fence_after();
#pragma unroll 1
                for (int c = 0; c < value_quarters; ++c) {
                    const int slot = (j * QUARTERS + c) % SLOTS;
                    if (elect_one()) {
                        const uint32_t d = tmem_base + 256 + c * 64, a = tmem_base + (j & 1) * 128;
                        const uint64_t value = smem_desc_mn_sw128(s_k(slot), PIECE_BYTES);
#pragma unroll
                        for (int k = 0; k < BKV / 16; ++k)
                            mma_bf16_ts(d, a + k * 8, value + k * (2048 >> 4), IDESC_128x64_KMN, (j > 0 || k > 0) ? 1u : 0u);
                        tcgen05_commit(bar(EMPTY + slot));
                        if (c == value_quarters - 1) tcgen05_commit(bar(PV_DONE + (j & 1)));
                    }
                    __syncwarp();
                }
            }
            if (!ok && lane == 0) { *abort_flag = 1; atomicExch(error_word, 42); }
        }
    } else {
        // ---------------- softmax: two threads to a query row (= TMEM lane), 64 of a tile's keys each ----------------
        const int x = warp >= 6 ? 1 : 0, quad = warp & 3, r = quad * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
        const int P = pos0 + min(r, rows_here - 1);            // rows past the end copy the last row, and are not stored
        const int lo = jllm_first_key(P, window);              // the first key this row sees (window or chunk)
        const int lo_last = jllm_first_key(pos_last, window);
        const float to_log2 = CAP ? 1.f : scale_log2;          // (a capped score is in base 2 already)
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        for (int j = 0; j < n_tiles; ++j) {
            const int key0 = (kt_lo + j) * BKV + x * 64;
            const uint32_t s_addr = lane_addr + (j & 1) * 128;
            float* mine = row_max + (j & 1) * 2 * BQ;
            uint32_t v[2][32];
            ok = ok && mbar_wait(bar(S_FULL + (j & 1)), (uint32_t)(j >> 1) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                tcgen05_fence_after();
#pragma unroll
                for (int c = 0; c < 2; ++c) tmem_ld_32x32b_x32(s_addr + x * 64 + c * 32, v[c]);
                tmem_ld_wait();
                if constexpr (CAP) cap.tile(v);
                if (key0 + 63 > pos0 || key0 < lo_last) {
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int key = key0 + c * 32 + i;
                            if (!(key <= P && key >= lo)) v[c][i] = __float_as_uint(-INFINITY);
                        }
                }
                // (four chains, then their maximum: one chain of dependent comparisons is pure latency)
                float mxs[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) mxs[i & 3] = fmaxf(mxs[i & 3], __uint_as_float(v[c][i]));
                mine[x * BQ + r] = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3]));
            }
            // Both halves of every row have left tensor memory (P may overwrite them) and both maxima are known. The buffer of
            // maxima is written again two tiles on, behind the next meeting.
            tcgen05_fence_before();
            if (!softmax_meet(ok)) { ok = false; break; }
            tcgen05_fence_after();
            const float mx = fmaxf(mine[r], mine[BQ + r]);
            // The reference point of the exponentials only moves when the maximum grew by more than 2^8: until
            // then p stays below 256, which bfloat16 and the float32 sum hold as well, and O needs no rescaling.
            const float m_cand = fmaxf(m, mx * to_log2);
            const float m_new = (m_cand - m > 8.f) ? m_cand : m;
            const float m_use = m_new == -INFINITY ? 0.f : m_new;
            const float corr = fast_exp2(m - m_use);
            float sums[2] = {0.f, 0.f};
            uint32_t pk[32];
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float p0 = fast_exp2(fmaf(__uint_as_float(v[c][i]), to_log2, -m_use));
                    const float p1 = fast_exp2(fmaf(__uint_as_float(v[c][i + 1]), to_log2, -m_use));
                    sums[(i >> 1) & 1] += p0 + p1;
                    __nv_bfloat162 b2 = __floats2bfloat162_rn(p0, p1);
                    pk[(c * 32 + i) >> 1] = *reinterpret_cast<uint32_t*>(&b2);
                }
            tmem_st_32x32b_x32(s_addr + x * 32, pk);           // P over the first 64 columns of S
            m = m_new;
            l = l * corr + (sums[0] + sums[1]);
            if (j > 0 && __any_sync(0xffffffffu, corr != 1.f)) {  // the reference moved for a row of this warp
                // O holds what the tiles before added once O += P K of tile j - 1 has completed (S_j ran in front of it). Its
                // barrier cannot be a phase behind or ahead: S_(j-1), which this thread has seen, ran behind the product of tile
                // j - 3, and that of tile j + 1 needs this thread's P.
                ok = mbar_wait(bar(PV_DONE + ((j - 1) & 1)), (uint32_t)((j - 1) >> 1) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (ok) {
                    tcgen05_fence_after();
#pragma unroll 1
                    for (int c = 0; c < value_quarters; ++c) {    // 32 columns of every 64 are this thread's
                        const uint32_t at = lane_addr + 256 + c * 64 + x * 32;
                        uint32_t o[32];
                        tmem_ld_32x32b_x32(at, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                        tmem_st_32x32b_x32(at, o);
                    }
                }
            }
            tmem_st_wait();
            tcgen05_fence_before();
            if (ok) mbar_arrive(bar(P_READY + (j & 1)));
        }
        // ---- O / l -> out ----
        ok = ok && mbar_wait(bar(PV_DONE + ((n_tiles - 1) & 1)), (uint32_t)((n_tiles - 1) >> 1) & 1u, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        float* sums = row_max + (n_tiles & 1) * 2 * BQ;        // (the buffer that the last tile did not use)
        sums[x * BQ + r] = l;
        if (softmax_meet(ok)) {
            tcgen05_fence_after();
            const float inv = 1.f / (sums[r] + sums[BQ + r]);
            __nv_bfloat16* dst = out + (size_t)(row0 + r) * out_stride + (size_t)head * W;
#pragma unroll 1
            for (int c = 0; c < value_quarters; ++c) {
                const int c0 = c * 64 + x * 32;
                uint32_t v[32];
                tmem_ld_32x32b_x32(lane_addr + 256 + c0, v);
                tmem_ld_wait();
                if (r < rows_here) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(v[8 * i + 2 * e]) * inv,
                                                                      __uint_as_float(v[8 * i + 2 * e + 1]) * inv);
                            w[e] = *reinterpret_cast<uint32_t*>(&b2);
                        }
                        *reinterpret_cast<uint4*>(dst + c0 + 8 * i) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        } else if (lane == 0) { *abort_flag = 1; atomicExch(error_word, 43); }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 2) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace

int* jllm_attention_tc_error_word_ptr();   // attention_prefill_tc.cu: one error word for the tcgen05 attention kernels

JLLM_BOUNDS_READER(attention_prefill_latent)

// cache [pages, kv_heads, page_size, 256]: keys and values at once. Of a head's 256 result columns the first `value_cols`
// (rounded up to 64) are written.
JLLM_EXPORT int jllm_attention_prefill_latent(const void* q, int q_stride, const void* cache, long long cache_pages, void* out,
                                              int out_stride, const int* seg_start, const int* seg_len, const int* seg_kv_len,
                                              const int* block_tables, int table_stride, int num_segs, int rows, int heads,
                                              int kv_heads, int head_dim, int value_cols, int page_size, int window, float scale,
                                              float softcap, cudaStream_t stream) {
    JLLM_REQUIRE(rows >= 0 && num_segs >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && cache_pages > 0,
                 "attention_prefill_latent: rows=%d segments=%d heads=%d kv_heads=%d pages=%lld", rows, num_segs, heads,
                 kv_heads, cache_pages);
    JLLM_REQUIRE(head_dim == W && value_cols > 0 && value_cols <= W && page_size >= 1 && page_size <= 128 &&
                     (page_size & (page_size - 1)) == 0 && q_stride % 8 == 0 && out_stride % 8 == 0,
                 "attention_prefill_latent: needs rows of 256 values, a power-of-two page size <= 128 and 16-byte aligned rows "
                 "(head_dim=%d value_cols=%d page_size=%d q_stride=%d out_stride=%d)", head_dim, value_cols, page_size, q_stride,
                 out_stride);
    JLLM_REQUIRE(((uintptr_t)q % 16) == 0 && ((uintptr_t)cache % 16) == 0 && ((uintptr_t)out % 16) == 0,
                 "attention_prefill_latent: q, cache and out must be 16-byte aligned");
    JLLM_REQUIRE(rows / BQ + num_segs < 65535, "attention_prefill_latent: %d rows in %d segments are too many blocks", rows, num_segs);
    if (rows == 0 || num_segs == 0) return JLLM_OK;
    CUtensorMap map_q, map_k;
    int rc = tensor_map_for(q, rows, (long long)heads * W, q_stride, BQ, &map_q);
    if (rc != JLLM_OK) return rc;
    rc = tensor_map_for(cache, cache_pages * kv_heads * page_size, W, W, page_size, &map_k);
    if (rc != JLLM_OK) return rc;
    int* error_word = jllm_attention_tc_error_word_ptr();
    if (!error_word) return jllm_fail(JLLM_CUDA_ERROR, "attention_prefill_latent: no error word");
    int page_shift = 0;
    while ((1 << page_shift) < page_size) ++page_shift;
    auto kern = softcap > 0.f ? attention_prefill_latent_kernel<true> : attention_prefill_latent_kernel<false>;
    if (jllm_allow_smem((const void*)kern, SMEM_BYTES) != cudaSuccess)
        return jllm_fail(JLLM_CUDA_ERROR, "attention_prefill_latent: %zu bytes of shared memory refused", SMEM_BYTES);
    const dim3 grid(heads, (rows + BQ - 1) / BQ + num_segs);
    jllm_launch(kern, grid, dim3(THREADS), SMEM_BYTES, stream, true, map_q, map_k, (const __nv_bfloat16*)cache,
                (__nv_bfloat16*)out, out_stride, seg_start, seg_len, seg_kv_len, block_tables, table_stride, num_segs, heads,
                kv_heads, page_size, page_shift, (int)cache_pages, window, (value_cols + 63) / 64, scale * LOG2E, error_word,
                score_cap(softcap, scale));
    return jllm_check_launch("attention_prefill_latent");
}

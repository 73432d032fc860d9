// out[m, n] (+)= sum_k a[m, k] * w[n, k] (+ bias[n]) on the 5th-generation tensor cores, two SMs to a tile (tcgen05 cta_group::2),
// bfloat16, with the WEIGHT rows as the M side: 256 weight rows by any multiple of 16 tokens up to 256. The product of some hundreds of
// rows up to a prompt's.
//
// What bounds a product's main loop here is shared memory: a k block's bytes are written once by TMA and read once by the MMA, 128 bytes a
// clock together. A one-SM tile of 128 tokens x 192 weight rows moves 80 KB a k block for 384 clocks of multiply-adds; a pair's tile of
// 256 weight rows x T tokens moves 32 KB + 128 T bytes per SM for 2 T clocks. gemm_pair.cu has the same balance with the tokens as its M
// side, in steps of 256: 613 tokens are 768 there (640 in 128-row tiles). Here a tile's tokens are cut to what is there (613 = 3 x 208),
// or to what fills the pairs: T is chosen so that the rounds of tiles, times T + 256 clocks a k block, come out least.
//
//   * warp 0 of BOTH blocks is a producer (the warp walks, one elected lane issues: tcgen05_common.cuh): its 128 rows of W (one packed tile: a tiled copy without swizzle of its 16 KB) and
//     half of the tile's tokens (tiled copy, 128-byte swizzle), all completing on the FIRST block's barrier of the stage. The first
//     stages' weights are asked for before the wait for the kernel in front;
//   * warp 1 of the first block, again by one elected lane, issues 4 x tcgen05.mma.cta_group::2 (M 256, N T, K 16) per k block and commits to both blocks;
//   * warps 2-9 of both blocks are the epilogue of their block's 128 weight rows: a thread has one weight row and 16 tokens at a time, so
//     that a warp's store of one token is 32 neighbouring outputs. Gate and up rows lie 8 lanes apart and meet by shuffles.
// Tensor memory holds two accumulators of at most 256 columns, so a tile's epilogue lies under the next tile's main loop. Tiles are walked
// with the tokens fastest: the pairs that run together share W in L2. Edges: TMA fills tokens beyond M with zeros; a block whose half of the
// W rows lies beyond the padded matrix brings none, and its rows are never stored.
//
// 8B layer shapes, us, the kernels whose place it takes and this one: QKV of 200, 300, 613, 1,024 rows 17.8 and 14.8, 18.5 and 16.5, 28.9 and
// 24.7, 42.5 and 38.1; O 15.5 and 15.0, 17.2 and 14.3, 22.5 and 18.5 (1,024: not taken); gate_up 47.4 and 43.7, 62.8 and 52.4, 101 and 88
// (1,390 TFLOP/s, what the power limit leaves); down of 300, 512, 613 rows 47.3 and 35.5, 51.0 and 42.9, 59.6 and 50.7. A round of tiles of
// 64 k blocks takes 14.3 us with 80 tokens, 18.5 with 160, 22.2 with 208, 27 with 256, start and end included.
//
// Every wait is bounded (codes 34 to 36): the kernel raises the error word, tells its partner, all roles leave their loops, both blocks
// meet at the cluster's barrier and tensor memory is freed.
#include "common.cuh"
#include "tcgen05_pair.cuh"

namespace {

using namespace tc;

constexpr int WM = 128, BK = 64;
constexpr int W_BYTES = WM * BK * 2;
constexpr int EPILOGUE_WARPS = 8, THREADS = 64 + 32 * EPILOGUE_WARPS;
constexpr int TMEM_COLS = 512, MAX_TOKENS = 256, MAX_STAGES = 12;
constexpr size_t SMEM_BYTES = 226 * 1024;

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// 16 tokens (rows m0 .. m0 + 15 of the output, those below m_end) of this thread's weight row n. A warp's lanes are 32 neighbouring n.
template <typename Tout>
__device__ __forceinline__ void store16(uint32_t (&v)[16], Tout* __restrict__ out, int ldo, int accumulate, VecRef bias, int has_bias,
                                        const GluArgs& swiglu, int m0, int m_end, int n, int N, bool pairs_fit) {
    const int lane = threadIdx.x & 31;
    if (swiglu) {
        // Rows come in blocks of 16: 8 gate rows, then the 8 up rows of the same hidden units. A gate lane takes the first eight tokens
        // of its unit, the lane with the unit's up row the other eight.
        const bool gate_lane = (lane & 8) == 0;
        const int unit = (n >> 4) * 8 + (n & 7), m = m0 + (gate_lane ? 0 : 8);
        float gate[8], up[8], h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float got = __uint_as_float(__shfl_xor_sync(0xffffffffu, gate_lane ? v[8 + j] : v[j], 8));
            gate[j] = gate_lane ? __uint_as_float(v[j]) : got;
            up[j] = gate_lane ? got : __uint_as_float(v[8 + j]);
        }
        glu_units<8>(swiglu.word_of(unit), [&](int j) { return gate[j]; }, [&](int j) { return up[j]; }, 1.f, h);
        const bool live = (gate_lane ? n + 8 : n) < N;
        if (swiglu.weights != nullptr) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (live && m + j < m_end) h[j] = __fmul_rn(h[j], swiglu.weight(m + j, unit));
        }
        if (sizeof(Tout) == 2 && pairs_fit) {
            // two neighbouring units to a store: the even lane takes four tokens of both, the odd lane the other four
            const bool even = (lane & 1) == 0;
            const int mm = m + (even ? 0 : 4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float got = __shfl_xor_sync(0xffffffffu, even ? h[4 + j] : h[j], 1);
                const __nv_bfloat162 two = even ? __floats2bfloat162_rn(h[j], got) : __floats2bfloat162_rn(got, h[4 + j]);
                if (live && mm + j < m_end) *reinterpret_cast<__nv_bfloat162*>(out + (size_t)(mm + j) * ldo + (unit & ~1)) = two;
            }
        } else if (live) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (m + j < m_end) out[(size_t)(m + j) * ldo + unit] = from_float<Tout>(h[j]);
        }
        return;
    }
    const float b = has_bias && n < N ? bias[n] : 0.f;
    if constexpr (sizeof(Tout) == 2) {
        float x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = epilogue_act(has_bias ? __uint_as_float(v[j]) + b : __uint_as_float(v[j]), accumulate);
        if (pairs_fit && accumulate != EPI_ADD) {
            const bool even = (lane & 1) == 0;
            const int m = m0 + (even ? 0 : 8), n2 = n & ~1;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float got = __shfl_xor_sync(0xffffffffu, even ? x[8 + j] : x[j], 1);
                const __nv_bfloat162 two = even ? __floats2bfloat162_rn(x[j], got) : __floats2bfloat162_rn(got, x[8 + j]);
                if (n2 < N && m + j < m_end) *reinterpret_cast<__nv_bfloat162*>(out + (size_t)(m + j) * ldo + n2) = two;
            }
        } else if (n < N) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                Tout* dst = out + (size_t)(m0 + j) * ldo + n;
                if (m0 + j < m_end) *dst = from_float<Tout>(accumulate == EPI_ADD ? x[j] + to_float(*dst) : x[j]);
            }
        }
    } else if (n < N) {
        Tout* dst = out + (size_t)m0 * ldo + n;
        if (accumulate == EPI_ADD) {
            // added where the data lies (in L2): the SM neither loads the old values nor waits for them; nobody else adds here
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (m0 + j < m_end)
                    asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(dst + (size_t)j * ldo), "f"(__uint_as_float(v[j]) + b) : "memory");
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (m0 + j < m_end) dst[(size_t)j * ldo] = epilogue_act(__uint_as_float(v[j]) + b, accumulate);
        }
    }
}

template <typename Tout>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_pair_swap_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, VecRef bias, int has_bias,
                      Tout* __restrict__ out, int ldo, int accumulate, int M, int N, int K, GluArgs swiglu, int tokens, int tiles_m,
                      int stages, int* __restrict__ error_word) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_words[2 * MAX_STAGES + 4];
    __shared__ uint32_t tmem_base_word;
    __shared__ int abort_word;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // swizzled tiles want 1024-byte alignment
    const uint32_t bars = smem_u32(bar_words);
    // barriers: full[stages] (the first block's are used), empty[stages] (each block its own), acc_full[2] (each its own), acc_empty[2]
    // (the first block's)
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (MAX_STAGES + s); };
    auto acc_full_bar = [&](int b) { return bars + 8u * (2 * MAX_STAGES + b); };
    auto acc_empty_bar = [&](int b) { return bars + 8u * (2 * MAX_STAGES + 2 + b); };
    volatile int* abort_flag = &abort_word;

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();             // 0: the pair's first block, which issues the MMAs
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int tiles = tiles_m * ((N + 2 * WM - 1) / (2 * WM));
    const int k_blocks = (K + BK - 1) / BK;
    const int packed_tiles = (N + WM - 1) / WM;
    const uint32_t half_bytes = (uint32_t)tokens * 64u, stage_bytes = W_BYTES + half_bytes;      // (a block's half of the tokens)

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full_bar(b), 1);
            mbar_init(acc_empty_bar(b), 2 * EPILOGUE_WARPS);
        }
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {   // the same warp of both blocks allocates all 512 columns in both (one block per SM)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_word)), "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();      // the partner's barriers are set up and its tensor memory is there before anything reaches them
    tcgen05_fence_after();
    const uint32_t tmem_base = tmem_base_word;

    auto give_up = [&](int code) {
        *abort_flag = 1;
        store_cluster(in_block(smem_u32(&abort_word), rank ^ 1u), 1);
        atomicExch(error_word, code);
    };

    if (warp == 0) {
        // ---------------- producer (both blocks) ----------------
        const uint32_t first_full = in_block(full_bar(0), 0);
        int s = 0, early = 0;
        long long asked = 0;
        uint32_t parity = 1, dst = base;
        bool ok = true, first = true;
        for (int tile = pair; ok && tile < tiles; tile += pairs) {
            const int m0 = (tile % tiles_m) * tokens + (int)rank * (tokens >> 1), tn = (tile / tiles_m) * 2;
            const bool mine = tn + (int)rank < packed_tiles;           // this block's half of the W rows exists
            const uint32_t tx = 2 * half_bytes + (tn + 1 < packed_tiles ? 2 : 1) * W_BYTES;     // both blocks' bytes
            int wy = (tn + (int)rank) * k_blocks * 128;                // row of the packed weight
            if (first) {
                // nobody writes weights: the first stages' are asked for before the wait for the kernel in front
                first = false;
                early = min(stages, k_blocks);
                if (elect_one())
                    for (int i = 0; i < early; ++i) {
                        if (rank == 0) mbar_expect_tx(full_bar(i), tx);
                        if (mine) tma_load_2d_pair(base + (uint32_t)i * stage_bytes, &map_w, 0, wy + i * 128, first_full + 8u * i);
                    }
                __syncwarp();
                pdl_wait();
                pdl_trigger();
            }
            for (int kb = 0; kb < k_blocks; ++kb, wy += 128) {
                const bool w_asked = early > 0;
                if (w_asked) --early;
                else if (!warp_wait(empty_bar(s), parity, abort_flag)) { ok = false; break; }
                if (elect_one()) {
                    const uint32_t full0 = first_full + 8u * s;
                    if (!w_asked) {
                        if (rank == 0) mbar_expect_tx(full_bar(s), tx);
                        if (mine) tma_load_2d_pair(dst, &map_w, 0, wy, full0);
                    }
                    tma_load_2d_pair(dst + W_BYTES, &map_a, kb * BK, m0, full0);
                }
                __syncwarp();
                ++asked;
                dst += stage_bytes;
                if (++s == stages) { s = 0; parity ^= 1u; dst = base; }
            }
        }
        if (!ok) {
            if (lane == 0) give_up(34);
            // neither block ends with copies on their way (they all complete in the first block): the last one of every stage
            for (long long n = asked > stages ? asked - stages : 0; rank == 0 && n < asked; ++n)
                for (uint32_t i = 0; i < SPIN_LIMIT && !mbar_try_wait(full_bar((int)(n % stages)), (uint32_t)(n / stages) & 1u); ++i) {}
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer (the first block) ----------------
        if (rank == 0) {
            // kind::f16: float32 accumulate, A and B bfloat16, both K-major, N >> 3 at [17,23), M >> 4 at [24,29): M is the pair's 256
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(tokens >> 3) << 17) | ((256u >> 4) << 24);
            const uint64_t desc_w0 = smem_desc_sw128(base), desc_b0 = smem_desc_sw128(base + W_BYTES);
            uint64_t desc_w = desc_w0, desc_b = desc_b0;          // (a stage further is an addition to the address field)
            uint32_t local_tile = 0, parity = 0;
            int s = 0;
            bool ok = true;
            for (int tile = pair; ok && tile < tiles; tile += pairs, ++local_tile) {
                const uint32_t buf = local_tile & 1u;
                if (!warp_wait(acc_empty_bar(buf), ((local_tile >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                tcgen05_fence_after();
                const uint32_t tmem_d = tmem_base + buf * MAX_TOKENS;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!warp_wait(full_bar(s), parity, abort_flag)) { ok = false; break; }
                    tcgen05_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) mma_pair(tmem_d, desc_w + 2 * k, desc_b + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        commit_pair(empty_bar(s));          // both blocks' stage is free when these MMAs have read it
                    }
                    __syncwarp();
                    desc_w += stage_bytes >> 4;
                    desc_b += stage_bytes >> 4;
                    if (++s == stages) { s = 0; parity ^= 1u; desc_w = desc_w0; desc_b = desc_b0; }
                }
                if (ok && elect_one()) commit_pair(acc_full_bar(buf));
                __syncwarp();
            }
            if (!ok && lane == 0) give_up(35);
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: warps 2..9 of both blocks, TMEM lanes 32 * (warp % 4), every second 16 columns ----------------
        pdl_wait();          // the residual stream it may add into was written by the kernels before
        pdl_trigger();
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const bool pairs_fit = sizeof(Tout) == 2 && ((uintptr_t)out & 3u) == 0 && (ldo & 1) == 0 && (swiglu || (N & 1) == 0);
        uint32_t local_tile = 0;
        bool ok = true;
        for (int tile = pair; tile < tiles; tile += pairs, ++local_tile) {
            const int m0 = (tile % tiles_m) * tokens, m_end = min(M, m0 + tokens);
            const int n_warp = ((tile / tiles_m) * 2 + (int)rank) * WM + quad * 32;
            const uint32_t buf = local_tile & 1u;
            ok = mbar_wait(acc_full_bar(buf), (local_tile >> 1) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + buf * MAX_TOKENS + ((uint32_t)(quad * 32) << 16);
            if (n_warp < N) {
#pragma unroll 1
                for (int c = half * 16; c < tokens && m0 + c < m_end; c += 32) {
                    uint32_t v[16];
                    tmem_ld_32x32b_x16(taddr + c, v);
                    tmem_ld_wait();
                    store16(v, out, ldo, accumulate, bias, has_bias, swiglu, m0 + c, m_end, n_warp + lane, N, pairs_fit);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(in_block(acc_empty_bar(buf), 0));
        }
        if (!ok && lane == 0) give_up(36);
        __syncwarp();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();      // neither block leaves, or frees tensor memory, while the other may still reach into it
    if (warp == 2) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace

int* jllm_gemm_error_word();

// w: ops.pack_weight of the [N, K] weight (k_blocks_packed = ceil(K / 64) its k blocks). `tokens`: the tokens of a tile, a multiple of 16
// up to 256; `pairs`: at most so many pairs of blocks.
JLLM_EXPORT int jllm_gemm_pair_swap(const void* a, int lda, const void* w, int k_blocks_packed, const void* bias, int bias_dtype, void* out,
                                    int out_dtype, int ldo, int accumulate, int M, int N, int K, int tokens, int pairs, int swiglu_word,
                                    const void* glu_more, cudaStream_t stream) {
    const GluArgs swiglu = glu_args(swiglu_word, glu_more);
    JLLM_REQUIRE(swiglu.in_eights(), "gemm_pair_swap: units of %d in front of %d do not come in eights", swiglu.ff, swiglu.split);
    JLLM_REQUIRE(M >= 1 && N >= 1 && K >= 8 && K % 8 == 0 && lda % 8 == 0 && ((uintptr_t)a % 16) == 0 && ((uintptr_t)w % 16) == 0,
                 "gemm_pair_swap: needs K %% 8 == 0 and 16-byte aligned rows (M=%d N=%d K=%d lda=%d)", M, N, K, lda);
    JLLM_REQUIRE(k_blocks_packed == (K + BK - 1) / BK, "gemm_pair_swap: the packed weight has %d k blocks, K=%d needs %d", k_blocks_packed, K,
                 (K + BK - 1) / BK);
    JLLM_REQUIRE(ldo >= (swiglu ? N / 2 : N), "gemm_pair_swap: ldo=%d < N=%d", ldo, N);
    JLLM_REQUIRE(!swiglu || (N % 16 == 0 && !bias && !accumulate),
                 "gemm_pair_swap: the SwiGLU epilogue needs N %% 16 == 0, no bias and no accumulation (N=%d)", N);
    JLLM_REQUIRE(tokens >= 16 && tokens <= MAX_TOKENS && tokens % 16 == 0, "gemm_pair_swap: tiles of %d tokens", tokens);
    JLLM_REQUIRE(pairs >= 1, "gemm_pair_swap: on %d pairs", pairs);
    const long long packed_rows = (long long)((N + 127) / 128) * k_blocks_packed * 128;
    JLLM_REQUIRE(packed_rows < (1LL << 31), "gemm_pair_swap: a packed weight of %lld rows of 128 bytes is too long", packed_rows);
    CUtensorMap map_a, map_w;
    int rc = tensor_map_for(a, M, K, lda, tokens / 2, &map_a);
    if (rc != JLLM_OK) return rc;
    rc = packed_map_for(w, packed_rows, &map_w);
    if (rc != JLLM_OK) return rc;
    int* error_word = jllm_gemm_error_word();
    if (!error_word) return jllm_fail(JLLM_CUDA_ERROR, "gemm_pair_swap: no error word");
    const int tiles_m = (M + tokens - 1) / tokens;
    const long long tiles = (long long)tiles_m * ((N + 2 * WM - 1) / (2 * WM));
    JLLM_REQUIRE(tiles < (1LL << 30), "gemm_pair_swap: %lld tiles are too many", tiles);
    if (pairs > tiles) pairs = (int)tiles;
    int stages = (int)((SMEM_BYTES - 2048) / (W_BYTES + (size_t)tokens * 64));
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    const size_t smem = (size_t)stages * (W_BYTES + (size_t)tokens * 64) + 1024;
    const VecRef b{bias, bias_dtype};
#define JLLM_GO(T)                                                                                                                  \
    do {                                                                                                                            \
        auto kern = gemm_pair_swap_kernel<T>;                                                                                       \
        if (jllm_allow_smem((const void*)kern, smem) != cudaSuccess) return jllm_check_launch("gemm_pair_swap");                    \
        jllm_launch(kern, dim3(2 * pairs), dim3(THREADS), smem, stream, LAUNCH_DEPENDENT, map_a, map_w, b, (int)(bias != nullptr),  \
                    (T*)out, ldo, accumulate, M, N, K, swiglu, tokens, tiles_m, stages, error_word);                                \
    } while (0)
    if (out_dtype == JLLM_F32) JLLM_GO(float); else JLLM_GO(__nv_bfloat16);
#undef JLLM_GO
    return jllm_check_launch("gemm_pair_swap");
}

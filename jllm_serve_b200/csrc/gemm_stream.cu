// out[m, n] (+)= sum_k a[m, k] * w[n, k] (+ bias[n]) for FEW rows m (a decode step, at most 256): a stream of the
// weights through the 5th-generation tensor cores with the operands swapped.
//
// With few rows the product is nothing but reading W once, so everything is shaped for that read:
//   * W is kept PACKED (ops.pack_weight, once at load): tiles of 128 weight rows x 64 k, each tile the 16 KB image
//     that the tensor cores read from shared memory (rows of 128 bytes, 128-byte swizzle), tile (t, kb) at
//     (t * k_blocks + kb) * 16 KB. One tile is ONE contiguous bulk copy (cp.async.bulk, no multicast) completing on
//     a stage's mbarrier: no thread's registers hold weights, and the memory system sees 16 KB bursts;
//   * the weight rows are the M side of tcgen05.mma (128 rows a tile), the token rows the N side (padded to a
//     multiple of 16), so no tensor-core work is spent on padding 8 tokens to 128; the accumulator [128 weight rows
//     x tokens] lives in tensor memory, two of them so that an epilogue overlaps the next tile's stream;
//   * the k blocks of ALL tiles, in tile order, are dealt out in equal runs over one block per SM, so every SM
//     streams the same number of bytes whatever the matrix's height; a tile whose k blocks fall to several blocks
//     is finished by those blocks together: each parks its part, and when all have, those that end their run in the
//     tile each add up a share of the token columns over the parts in k order (the result does not depend on who
//     came when);
//   * the activations' tile of a k block (tokens x 64) comes by TMA from the [rows, K] matrix (L2 resident);
//   * the producer requests its first weights BEFORE it waits for the kernel in front of it (programmatic dependent
//     launch): weights do not depend on it.
// Roles: warp 0 producer, warp 1 MMA issuer (both walk as a warp, one elected lane issues: tcgen05_common.cuh), warps 2-5 epilogue (bias / float32 residual add /
// SwiGLU over interleaved gate and up rows / store). Every wait is bounded and raises the error word of
// gemm_tcgen05 (codes 11-13; the clusters' kernel 14-16).
#include <mutex>
#include <unordered_map>

#include "tcgen05_common.cuh"

namespace {

using namespace tc;

constexpr int WM = 128, BK = 64;
constexpr int W_TILE_BYTES = WM * BK * 2;       // 16 KB
constexpr int THREADS = 192;
constexpr int MAX_TOKENS = 256;                  // the N side of one tcgen05.mma; two accumulators of 256 columns are all of tensor memory
constexpr int MAX_TILES = 65536;                 // counter words at the head of the workspace

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// What J tokens from m0 on of weight row n are added to (all the old values are requested before the first store: a load behind a
// store through the same pointer would wait for it).
template <typename Tout, int J>
__device__ __forceinline__ void residual(float (&old)[J], const Tout* out, int ldo, int accumulate, int m0, int M, int n, int N) {
#pragma unroll
    for (int j = 0; j < J; ++j)
        old[j] = accumulate == EPI_ADD && n < N && m0 + j < M ? to_float(out[(size_t)(m0 + j) * ldo + n]) : 0.f;
}
// The values of those tokens: bias / residual / SwiGLU and the store. The lanes of a warp hold neighbouring weight rows.
template <typename Tout, int J>
__device__ __forceinline__ void finish(const float (&v)[J], const float (&old)[J], Tout* out, int ldo, int accumulate, const VecRef& bias,
                                       int has_bias, const GluArgs& swiglu, int m0, int M, int n, int N) {
    if (swiglu) {
        // rows come in blocks of 16: 8 gate rows, then the 8 up rows of the same hidden units
        const int unit = (n >> 4) * 8 + (n & 7);
        float other[J], units[J];
#pragma unroll
        for (int j = 0; j < J; ++j) other[j] = __shfl_xor_sync(0xffffffffu, v[j], 8);
        if ((threadIdx.x & 8) == 0 && n + 8 < N) {
            glu_units<J>(swiglu.word_of(unit), [&](int j) { return v[j]; }, [&](int j) { return other[j]; }, 1.f, units);
#pragma unroll
            for (int j = 0; j < J; ++j) {
                if (m0 + j >= M) continue;
                if (swiglu.weights != nullptr) units[j] = __fmul_rn(units[j], swiglu.weight(m0 + j, unit));
                out[(size_t)(m0 + j) * ldo + unit] = from_float<Tout>(units[j]);
            }
        }
    } else if (n < N) {
        const float b = has_bias ? bias[n] : 0.f;
        Tout* dst = out + (size_t)m0 * ldo + n;
#pragma unroll
        for (int j = 0; j < J; ++j)
            if (m0 + j < M) dst[(size_t)j * ldo] = from_float<Tout>(epilogue_act(v[j] + b, accumulate) + old[j]);
    }
}

template <typename Tout>
__global__ void __launch_bounds__(THREADS, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_a, const __nv_bfloat16* __restrict__ w_packed, VecRef bias,
                   int has_bias, Tout* __restrict__ out, int ldo, int accumulate, int M, int N, int k_blocks, GluArgs swiglu,
                   int ntok, int stages, uint32_t tmem_cols, float* __restrict__ partials,
                   int* __restrict__ counters, int* __restrict__ error_word) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t b_bytes = (uint32_t)ntok * 128u, stage_bytes = W_TILE_BYTES + b_bytes;
    const uint32_t bars = base + (uint32_t)stages * stage_bytes;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (stages + s); };
    auto acc_full_bar = [&](int b) { return bars + 8u * (2 * stages + b); };
    auto acc_empty_bar = [&](int b) { return bars + 8u * (2 * stages + 2 + b); };
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(aligned + (size_t)stages * stage_bytes + 8 * (2 * stages + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
    volatile int* last_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 2);

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int tiles = (N + WM - 1) / WM;
    // the work: (tile, k block) pairs in tile order, one equal run per block
    const long long total = (long long)tiles * k_blocks;
    const long long run_lo = total * blockIdx.x / gridDim.x, run_hi = total * (blockIdx.x + 1) / gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full_bar(b), 1);
            mbar_init(acc_empty_bar(b), 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    const uint32_t acc_cols = tmem_cols >> 1;       // columns of one accumulator

    if (warp == 0) {
        // ---------------- producer: weights by bulk copy, activations by TMA ----------------
        bool ok = true;
        const int n = (int)(run_hi - run_lo), early = min(stages, n);
        const __nv_bfloat16* src = w_packed + (size_t)run_lo * (WM * BK);
        // the first weights are requested before the kernel in front of this one has finished
        if (elect_one())
            for (int i = 0; i < early; ++i) {
                mbar_expect_tx(full_bar(i), stage_bytes);
                bulk_copy(base + (uint32_t)i * stage_bytes, src + (size_t)i * (WM * BK), W_TILE_BYTES, full_bar(i));
            }
        __syncwarp();
        pdl_wait();
        pdl_trigger();
        int kb = (int)(run_lo % k_blocks);
        for (int i = 0; i < early; ++i) {
            if (elect_one()) tma_load_2d(base + (uint32_t)i * stage_bytes + W_TILE_BYTES, &map_a, kb * BK, 0, full_bar(i));
            __syncwarp();
            if (++kb == k_blocks) kb = 0;
        }
        src += (size_t)early * (WM * BK);
        int s = early == stages ? 0 : early;
        uint32_t parity = early == stages ? 0u : 1u;      // the ring's second lap waits for the first lap's release
        for (int i = early; i < n; ++i, src += WM * BK) {
            if (!warp_wait(empty_bar(s), parity, abort_flag)) { ok = false; break; }
            if (elect_one()) {
                const uint32_t dst = base + (uint32_t)s * stage_bytes;
                mbar_expect_tx(full_bar(s), stage_bytes);
                bulk_copy(dst, src, W_TILE_BYTES, full_bar(s));
                tma_load_2d(dst + W_TILE_BYTES, &map_a, kb * BK, 0, full_bar(s));
            }
            __syncwarp();
            if (++kb == k_blocks) kb = 0;
            if (++s == stages) { s = 0; parity ^= 1u; }
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(error_word, 11); }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        {
            // kind::f16: float32 accumulate, A and B bfloat16, both K-major, N = tokens, M = 128 weight rows
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ntok >> 3) << 17) | ((uint32_t)(WM >> 4) << 24);
            const uint64_t desc_w0 = smem_desc_sw128(base), desc_b0 = smem_desc_sw128(base + W_TILE_BYTES);
            uint64_t desc_w = desc_w0, desc_b = desc_b0;          // (a stage further is an addition to the address field)
            bool ok = true;
            int s = 0;
            uint32_t parity = 0, segment = 0;
            long long g = run_lo;
            while (ok && g < run_hi) {
                const int kb0 = (int)(g % k_blocks);
                const long long seg_end = min(run_hi, g + (k_blocks - kb0));      // the tile's k blocks that are this block's
                const uint32_t buf = segment & 1u;
                if (!warp_wait(acc_empty_bar(buf), ((segment >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                tcgen05_fence_after();
                const uint32_t tmem_d = tmem_base + buf * acc_cols;
                for (bool first = true; g < seg_end; ++g, first = false) {
                    if (!warp_wait(full_bar(s), parity, abort_flag)) { ok = false; break; }
                    tcgen05_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            tcgen05_mma_bf16(tmem_d, desc_w + 2 * k, desc_b + 2 * k, idesc, (!first || k > 0) ? 1u : 0u);
                        tcgen05_commit(empty_bar(s));
                    }
                    __syncwarp();
                    desc_w += stage_bytes >> 4;
                    desc_b += stage_bytes >> 4;
                    if (++s == stages) { s = 0; parity ^= 1u; desc_w = desc_w0; desc_b = desc_b0; }
                }
                if (ok && elect_one()) tcgen05_commit(acc_full_bar(buf));
                __syncwarp();
                ++segment;
            }
            if (!ok && lane == 0) { *abort_flag = 1; atomicExch(error_word, 12); }
        }
    } else {
        // ---------------- epilogue: warps 2..5, TMEM lanes 32 * (warp % 4) = weight rows of the tile ----------------
        pdl_wait();          // the residual stream it may add into was written by the kernels before
        pdl_trigger();
        const int quad = warp & 3;
        bool ok = true;
        uint32_t segment = 0;
        long long g = run_lo;
        const int G = gridDim.x;
        auto run_start = [&](long long c) { return total * c / G; };
        auto block_of = [&](long long index) { return (int)(((index + 1) * G + total - 1) / total - 1); };
        while (ok && g < run_hi) {
            const int tile = (int)(g / k_blocks), kb0 = (int)(g % k_blocks);
            const long long seg_end = min(run_hi, g + (k_blocks - kb0));
            const int kb1 = kb0 + (int)(seg_end - g);
            const uint32_t buf = segment & 1u;
            if (!mbar_wait(acc_full_bar(buf), (segment >> 1) & 1u, abort_flag)) { ok = false; break; }
            tcgen05_fence_after();
            const int row_in_tile = quad * 32 + lane;
            const int n = tile * WM + row_in_tile;                 // this thread's weight row = output column
            const uint32_t taddr = tmem_base + buf * acc_cols + ((uint32_t)(quad * 32) << 16);
            // value of (token m, weight row n): bias / residual / SwiGLU and the store
            auto finalize16 = [&](const float (&v)[16], int m0) {
                if (swiglu) {
                    // rows come in blocks of 16: 8 gate rows, then the 8 up rows of the same hidden units
                    const int unit = (n >> 4) * 8 + (n & 7);
                    float other[16], units[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) other[j] = __shfl_xor_sync(0xffffffffu, v[j], 8);
                    if ((lane & 8) == 0 && n + 8 < N) {
                        glu_units<16>(swiglu.word_of(unit), [&](int j) { return v[j]; }, [&](int j) { return other[j]; }, 1.f, units);
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            if (m0 + j >= M) continue;
                            if (swiglu.weights != nullptr) units[j] = __fmul_rn(units[j], swiglu.weight(m0 + j, unit));
                            out[(size_t)(m0 + j) * ldo + unit] = from_float<Tout>(units[j]);
                        }
                    }
                } else if (n < N) {
                    const float b = has_bias ? bias[n] : 0.f;
                    Tout* dst = out + (size_t)m0 * ldo + n;
                    float old[16];
                    // all the old values are requested before the first store (a load behind a store through the
                    // same pointer would wait for it: 16 round trips instead of one)
#pragma unroll
                    for (int j = 0; j < 16; ++j) old[j] = (accumulate == EPI_ADD && m0 + j < M) ? to_float(dst[(size_t)j * ldo]) : 0.f;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (m0 + j < M) dst[(size_t)j * ldo] = from_float<Tout>(epilogue_act(v[j] + b, accumulate) + old[j]);
                }
            };
            if (kb0 == 0 && kb1 == k_blocks) {                      // the whole tile is this block's
#pragma unroll 1
                for (int c0 = 0; c0 < ntok; c0 += 16) {
                    uint32_t raw[16];
                    tmem_ld_32x32b_x16(taddr + c0, raw);
                    tmem_ld_wait();
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(raw[j]);
                    finalize16(v, c0);
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty_bar(buf));
            } else {
                // ---- this block holds some of the tile's k blocks: park the part ([block][first or later part of the
                // block][token][128 rows]); the blocks that hold parts of one tile are consecutive ----
                const long long tile_g0 = (long long)tile * k_blocks;
                const int c_first = block_of(tile_g0), parts = block_of(tile_g0 + k_blocks - 1) - c_first + 1;
                auto part_of = [&](int c) {
                    const int slot = run_start(c) >= tile_g0 ? 0 : 1;
                    return partials + (size_t)(2 * c + slot) * MAX_TOKENS * WM + row_in_tile;
                };
                float* mine = part_of(blockIdx.x);
#pragma unroll 1
                for (int c0 = 0; c0 < ntok; c0 += 16) {
                    uint32_t raw[16];
                    tmem_ld_32x32b_x16(taddr + c0, raw);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) __stcg(mine + (size_t)(c0 + j) * WM, __uint_as_float(raw[j]));
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty_bar(buf));
                asm volatile("bar.sync 1, 128;" ::: "memory");       // the four epilogue warps have written
                // The parts of a tile are added up by the blocks that hold one and END their run in it: number p of them takes
                // the 16-token chunks p, p + np, ... (a block may have none), so that each has one batch of loads to wait
                // for instead of one block having them all. They finish their runs at about the same time, so waiting for
                // one another costs little, and nothing is behind that wait in their runs. The block that only BEGINS its
                // run in this tile (the tile's last holder, if its run goes on into other tiles) parks its part long
                // before and waits for nobody: a wait there would hold up its later tiles, and through them the blocks
                // that wait for those. Every holder counts itself in; the wait is a bounded one on that counter (all
                // blocks of the grid are resident, one per SM).
                const int p_me = (int)blockIdx.x - c_first, chunks = ntok >> 4;
                const bool tail_goes_on = run_start(c_first + parts) > tile_g0 + k_blocks;
                const int np = parts - (tail_goes_on ? 1 : 0);              // holders that take part in the adding
                const bool takes_part = seg_end == run_hi;                   // (p_me < np says the same)
                const bool has_share = takes_part && p_me < chunks;
                if (warp == 2 && lane == 0) {
                    __threadfence();
                    atomicAdd(&counters[tile], 1);
                    int seen = has_share ? 0 : parts;
                    for (uint32_t spin = 0; seen < parts && spin < SPIN_LIMIT; ++spin) {
                        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(counters + tile) : "memory");
                        if (seen < parts) {
                            if ((spin & 255u) == 255u && *abort_flag) break;
                            __nanosleep(32);
                        }
                    }
                    *last_flag = seen >= parts;
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (!*last_flag) { ok = false; break; }
                if (has_share) {
#pragma unroll 1
                    for (int c0 = p_me * 16; c0 < ntok; c0 += np * 16) {
                        float acc[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[j] = 0.f;
                        for (int p0 = 0; p0 < parts; p0 += 4) {     // four parts' loads in flight, added in k order
                            float x[4][16];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const float* src = part_of(c_first + min(p0 + q, parts - 1)) + (size_t)c0 * WM;
#pragma unroll
                                for (int j = 0; j < 16; ++j) x[q][j] = __ldcg(src + (size_t)j * WM);
                            }
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                if (p0 + q < parts) {
#pragma unroll
                                    for (int j = 0; j < 16; ++j) acc[j] += x[q][j];
                                }
                        }
                        finalize16(acc, c0);
                    }
                }
                // of those that take part, the one that is done last puts the tile's two counters back to zero for the next
                // product (all have read the first counter by then, and the early holder never reads it)
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (takes_part && warp == 2 && lane == 0) {
                    if (atomicAdd(&counters[MAX_TILES + tile], 1) == np - 1) {
                        counters[tile] = 0;
                        counters[MAX_TILES + tile] = 0;
                        __threadfence();
                    }
                }
            }
            g = seg_end;
            ++segment;
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(error_word, 13); }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 2) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}


// ---- a cluster of blocks to a tile --------------------------------------------------------------------------------------
// What the equal runs above pay for is the meeting: a tile's parts go to a workspace and back, a fence and a counter between
// (5 to 7 us of a product whose bytes take 5 to 15). Where the tiles come out even, a cluster of `gridDim.x / tiles` blocks has
// one tile instead, each block a part of its k blocks, and the parts never leave the SMs: every block finishes a share of the
// tokens, the others write their parts of it straight into its shared memory (st.shared::cluster), and after the cluster's
// barrier it adds them up in k order. Launched back to back, equal runs and clusters: 64 rows against O (4,096 x 4,096) 14.0 and
// 11.5 us, against down (4,096 x 12,288) 24.5 and 21.7, 24 rows against them 13.8 and 10.5, 23.4 and 20.3; 64 rows against 2,048 x
// 8,192 16.5 and 12.7. (These with one lane in the issuing loops, 0.33 us a k block with 32 tokens; with whole warps, see tcgen05_common.cuh,
// clusters take 9.3 us for 64 rows of O, 23.0 of down, 13.4 of QKV.) What bounds it is what an SM takes in on the SMs that have a block,
// and about 5 us from launch to first bytes and for the meeting.
// `overlay`: the parts lie over the ring (many tokens leave no room beside it); the cluster then meets once more, when every block
// is done with its ring, before anything is written.
constexpr int CLUSTER_MAX = 8;
constexpr double MEETING_K_BLOCKS = 16;         // k blocks an SM streams in the time of a meeting in the workspace (5 to 6 us)

__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

template <typename Tout>
__global__ void __launch_bounds__(THREADS, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap map_a, const __nv_bfloat16* __restrict__ w_packed, VecRef bias,
                    int has_bias, Tout* __restrict__ out, int ldo, int accumulate, int M, int N, int k_blocks, GluArgs swiglu,
                    int ntok, int stages, uint32_t tmem_cols, int blocks, int share, int overlay, int* __restrict__ error_word) {
    // `share`: tokens (a multiple of 8) that a block of the cluster finishes: block p those from p * share on
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t stage_bytes = W_TILE_BYTES + (uint32_t)ntok * 128u, ring = (uint32_t)stages * stage_bytes;
    const uint32_t part_bytes = (uint32_t)share * WM * 4;          // one block's part of a share, [share / 4][128 rows][4 tokens]
    const uint32_t parts_at = overlay ? 0u : ring;
    const uint32_t bars_at = overlay ? max(ring, (blocks - 1) * part_bytes) : ring + (blocks - 1) * part_bytes;
    const uint32_t bars = base + bars_at;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (stages + s); };
    const uint32_t acc_bar = bars + 16u * stages;
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(aligned + bars_at + 8 * (2 * stages + 1));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int tile = (int)blockIdx.x / blocks, rank = (int)blockIdx.x % blocks;      // (clusters lie along x: this is the rank)
    const int kb_lo = k_blocks * rank / blocks, kb_hi = k_blocks * (rank + 1) / blocks, n_kb = kb_hi - kb_lo;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(acc_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    // The first meeting says that every block runs (without overlay: from here on its shared memory may be written), or
    // that every block is done with its ring (overlay: the epilogue warps arrive then).
    if (!overlay || warp < 2) cluster_arrive();

    if (warp == 0) {
        // ---------------- producer: weights by bulk copy, activations by TMA ----------------
        bool ok = true;
        const __nv_bfloat16* w = w_packed + ((size_t)tile * k_blocks + kb_lo) * (WM * BK);
        const int early = min(stages, n_kb);
        // the first weights are requested before the kernel in front of this one has finished
        if (elect_one())
            for (int i = 0; i < early; ++i) {
                mbar_expect_tx(full_bar(i), stage_bytes);
                bulk_copy(base + (uint32_t)i * stage_bytes, w + (size_t)i * (WM * BK), W_TILE_BYTES, full_bar(i));
            }
        __syncwarp();
        pdl_wait();
        pdl_trigger();
        if (elect_one())
            for (int i = 0; i < early; ++i)
                tma_load_2d(base + (uint32_t)i * stage_bytes + W_TILE_BYTES, &map_a, (kb_lo + i) * BK, 0, full_bar(i));
        __syncwarp();
        int s = 0;
        uint32_t parity = 0;                                   // the ring's second lap waits for the first lap's release
        for (int i = stages; i < n_kb; ++i) {
            if (!warp_wait(empty_bar(s), parity, abort_flag)) { ok = false; break; }
            if (elect_one()) {
                const uint32_t dst = base + (uint32_t)s * stage_bytes;
                mbar_expect_tx(full_bar(s), stage_bytes);
                bulk_copy(dst, w + (size_t)i * (WM * BK), W_TILE_BYTES, full_bar(s));
                tma_load_2d(dst + W_TILE_BYTES, &map_a, (kb_lo + i) * BK, 0, full_bar(s));
            }
            __syncwarp();
            if (++s == stages) { s = 0; parity ^= 1u; }
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(error_word, 14); }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ntok >> 3) << 17) | ((uint32_t)(WM >> 4) << 24);
        const uint64_t desc_w0 = smem_desc_sw128(base), desc_b0 = smem_desc_sw128(base + W_TILE_BYTES);
        uint64_t desc_w = desc_w0, desc_b = desc_b0;          // (a stage further is an addition to the address field)
        bool ok = true;
        int s = 0;
        uint32_t parity = 0;
        for (int i = 0; i < n_kb; ++i) {
            if (!warp_wait(full_bar(s), parity, abort_flag)) { ok = false; break; }
            tcgen05_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    tcgen05_mma_bf16(tmem_base, desc_w + 2 * k, desc_b + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                tcgen05_commit(empty_bar(s));
            }
            __syncwarp();
            desc_w += stage_bytes >> 4;
            desc_b += stage_bytes >> 4;
            if (++s == stages) { s = 0; parity ^= 1u; desc_w = desc_w0; desc_b = desc_b0; }
        }
        if (ok) {
            if (elect_one()) tcgen05_commit(acc_bar);
        } else if (lane == 0) { *abort_flag = 1; atomicExch(error_word, 15); }
        __syncwarp();
    } else {
        pdl_wait();          // the residual stream it may add into was written by the kernels before
        pdl_trigger();
    }
    if (warp < 2) {
        cluster_wait();
        cluster_arrive();
        cluster_wait();
    } else {
        // ---------------- epilogue: warps 2..5, TMEM lanes 32 * (warp % 4) = weight rows of the tile ----------------
        const int quad = warp & 3, row = quad * 32 + lane, n = tile * WM + row, mine = rank * share;
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
        float old[8];
        residual(old, out, ldo, accumulate, mine, min(M, ntok), n, N);      // asked for while the weights still come
        bool ok = mbar_wait(acc_bar, 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        tcgen05_fence_after();
        if (overlay) cluster_arrive();
        cluster_wait();
        if (ok)
            for (int d = 1; d < blocks; ++d) {          // (every block begins with its neighbour: nobody is written by all at once)
                const int p = (rank + d) % blocks, t0 = p * share;
                // of block p's blocks - 1 parts this block's is number `rank`, or rank - 1 if p is below it
                const uint32_t at = base + parts_at + (uint32_t)(rank - (rank > p ? 1 : 0)) * part_bytes + (uint32_t)row * 16;
                uint32_t dst;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(at), "r"(p));
                for (int t = t0; t < min(t0 + share, ntok); t += 8) {
                    uint32_t v[8];
                    tmem_ld_32x32b_x8(taddr + t, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(dst + (uint32_t)((t - t0) / 4 + q) * (WM * 16)), "r"(v[4 * q]), "r"(v[4 * q + 1]),
                                     "r"(v[4 * q + 2]), "r"(v[4 * q + 3])
                                     : "memory");
                }
            }
        cluster_arrive();
        cluster_wait();
        if (ok) {
            const uint8_t* parts = aligned + parts_at + (size_t)row * 16;
            for (int t = mine; t < min(mine + share, ntok); t += 8) {
                uint32_t own[8];
                tmem_ld_32x32b_x8(taddr + t, own);
                tmem_ld_wait();
                float v[8] = {};
                for (int p = 0; p < blocks; ++p) {      // in k order
                    if (p == rank) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] += __uint_as_float(own[j]);
                    } else {
                        const uint8_t* src = parts + (size_t)(p - (p > rank ? 1 : 0)) * part_bytes + (size_t)((t - mine) / 4) * (WM * 16);
                        const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + WM * 16);
                        v[0] += x.x, v[1] += x.y, v[2] += x.z, v[3] += x.w, v[4] += y.x, v[5] += y.y, v[6] += y.z, v[7] += y.w;
                    }
                }
                if (t > mine) residual(old, out, ldo, accumulate, t, M, n, N);
                finish(v, old, out, ldo, accumulate, bias, has_bias, swiglu, t, M, n, N);
            }
        } else if (lane == 0) { *abort_flag = 1; atomicExch(error_word, 16); }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 2) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// How a cluster product of `ntok` tokens lies in shared memory
struct ClusterCut {
    int blocks, share, overlay, stages;
    size_t smem;
};
ClusterCut cluster_cut(int blocks, int ntok) {
    ClusterCut c{blocks, ((ntok + 7) / 8 + blocks - 1) / blocks * 8, 0, 0, 0};
    const size_t stage = W_TILE_BYTES + (size_t)ntok * 128, parts = (size_t)(blocks - 1) * c.share * WM * 4, room = 224 * 1024;
    c.stages = (int)((room - parts) / stage);
    if (c.stages < 6) c.overlay = 1, c.stages = (int)(room / stage);
    if (c.stages > 12) c.stages = 12;
    const size_t ring = c.stages * stage;
    c.smem = (c.overlay ? (ring > parts ? ring : parts) : ring + parts) + 1024 + 8 * (2 * c.stages + 1) + 16;
    return c;
}

template <typename Tout>
cudaLaunchConfig_t cluster_config(const ClusterCut& c, int tiles, cudaLaunchAttribute* attr, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * c.blocks);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = c.smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c.blocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// clusters of that many blocks the device runs at a time with that much shared memory
template <typename Tout>
int resident_clusters(const ClusterCut& c) {
    int n = 0;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = cluster_config<Tout>(c, 1, attr, nullptr);
    if (jllm_allow_smem((const void*)gemm_cluster_kernel<Tout>, c.smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_cluster_kernel<Tout>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

// The cluster of `n` blocks to a tile for a product, or one of no blocks where it does not fit: fewer k blocks than blocks, no room for
// two stages, or more tiles than clusters are resident at once
ClusterCut cluster_of(int n, int ntok, int tiles, int k_blocks, int out_dtype) {
    if (n < 1 || n > CLUSTER_MAX || n > k_blocks) return ClusterCut{};
    const ClusterCut one = cluster_cut(n, ntok);
    if (one.stages < 2) return ClusterCut{};
    const int resident = out_dtype == JLLM_F32 ? resident_clusters<float>(one) : resident_clusters<__nv_bfloat16>(one);
    return tiles <= resident ? one : ClusterCut{};
}

// A cluster to a tile where the clusters of all tiles are resident at once and a block's k blocks take no longer than an equal run and
// the meeting it saves; of the sizes that fit, the one with the fewest k blocks a block (a larger cluster meets for longer). The meeting
// counts what it costs in a step, more than back to back, where the next product's start hides it: QKV (6,144 x 4,096, two blocks to a
// cluster) at 64 rows takes 16.4 us in equal runs and 16.8 in clusters launched back to back, and a decode step of 64 requests,
// eight layers, 1,621 us with it in equal runs and 1,587 in clusters (a prompt of 47 rows 1,092 and 1,067). Back to back, equal runs and
// clusters: 2,048 x 8,192 (six), 64 rows 15.0 and 12.6 us; 7,168 x 5,120 (two), 128 rows 27.1 and 25.3; 12,288 x 2,048 (one), 32 rows
// 15.4 and 15.9, 128 rows 28.2 and 26.7; 6,144 x 4,096, 128 rows 20.0 and 21.3; 2,048 x 12,288 (six), 64 rows 16.4 and 15.8, 128 17.8 and 19.0.
// (The driver is asked once per shape and device: the choice is kept.)
ClusterCut choose_cluster(int ntok, int tiles, int k_blocks, int out_dtype, int sms) {
    static std::mutex mu;
    static std::unordered_map<unsigned long long, ClusterCut> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return ClusterCut{};
    const unsigned long long key =
        ((((unsigned long long)k_blocks << 24 | (unsigned)tiles) << 5 | (unsigned)(ntok / 16)) << 2 | (unsigned)out_dtype) << 6 | (unsigned)dev;
    std::lock_guard<std::mutex> lock(mu);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    ClusterCut c{};
    double best = (double)tiles * k_blocks / sms + MEETING_K_BLOCKS;
    for (int n = 1; n <= CLUSTER_MAX && n <= k_blocks; ++n) {
        const double cost = (k_blocks + n - 1) / n + 0.5 * n;
        if (cost >= best) continue;
        const ClusterCut one = cluster_of(n, ntok, tiles, k_blocks, out_dtype);
        if (one.blocks > 0) best = cost, c = one;
    }
    if (known.size() >= 4096) known.clear();
    return known[key] = c;
}

}  // namespace

// The error word is gemm_tcgen05's (one word for the tcgen05 products).
int* jllm_gemm_error_word();

JLLM_EXPORT long long jllm_gemm_stream_workspace_floats() { return 2LL * MAX_TILES + 2LL * 160 * MAX_TOKENS * WM; }

// The blocks of the clusters that a product of M rows against an [N, K] weight runs in (0: equal runs)
JLLM_EXPORT int jllm_gemm_stream_cluster(int M, int N, int K, int out_dtype) {
    if (M < 1 || M > MAX_TOKENS || N < 1 || K < 1) return 0;
    const int sms = jllm_device_sm_count() > 0 ? jllm_device_sm_count() : 1;
    return choose_cluster((M + 15) / 16 * 16, (N + WM - 1) / WM, (K + BK - 1) / BK, out_dtype, sms).blocks;
}

// a [M, K] bfloat16 (row stride lda), w_packed: ops.pack_weight of the [N, K] weight (k padded to k_blocks * 64, rows
// to a multiple of 128, zeros), out [M, N] (or [M, N / 2] with swiglu) float32 or bfloat16. `workspace`: zeroed floats
// (counters, then parked parts), at least jllm_gemm_stream_workspace_floats(). `cluster` (tests): the blocks of a cluster, 0 as the
// shape has it, -1 equal runs.
JLLM_EXPORT int jllm_gemm_stream(const void* a, int lda, const void* w_packed, int k_blocks, const void* bias,
                                 int bias_dtype, void* out, int out_dtype, int ldo, int accumulate, int M, int N, int K,
                                 int swiglu_word, const void* glu_more, float* workspace, long long workspace_floats, int max_blocks,
                                 int cluster, cudaStream_t stream) {
    const GluArgs swiglu = glu_args(swiglu_word, glu_more);
    JLLM_REQUIRE(swiglu.in_eights(), "gemm_stream: units of %d in front of %d do not come in eights", swiglu.ff, swiglu.split);
    JLLM_REQUIRE(M >= 1 && M <= MAX_TOKENS && N >= 1 && K >= 8 && K % 8 == 0 && lda % 8 == 0 && ((uintptr_t)a % 16) == 0 &&
                     ((uintptr_t)w_packed % 16) == 0,
                 "gemm_stream: needs 1 <= rows <= %d, K %% 8 == 0 and 16-byte aligned rows and weights "
                 "(M=%d N=%d K=%d lda=%d)", MAX_TOKENS, M, N, K, lda);
    JLLM_REQUIRE(k_blocks == (K + BK - 1) / BK, "gemm_stream: the packed weight has %d k blocks, K=%d needs %d", k_blocks, K,
                 (K + BK - 1) / BK);
    JLLM_REQUIRE(ldo >= (swiglu ? N / 2 : N), "gemm_stream: ldo=%d < N=%d", ldo, N);
    JLLM_REQUIRE(!swiglu || (N % 16 == 0 && !bias && !accumulate),
                 "gemm_stream: the SwiGLU epilogue needs N %% 16 == 0, no bias and no accumulation (N=%d)", N);
    const int tiles = (N + WM - 1) / WM;
    JLLM_REQUIRE(tiles <= MAX_TILES && workspace != nullptr && workspace_floats >= jllm_gemm_stream_workspace_floats(),
                 "gemm_stream: %d tiles (at most %d) and a workspace of %lld floats (got %lld)", tiles, MAX_TILES,
                 jllm_gemm_stream_workspace_floats(), workspace_floats);
    const int sms = jllm_device_sm_count() > 0 ? jllm_device_sm_count() : 1;
    const int ntok = (M + 15) / 16 * 16;
    uint32_t acc_cols = 32;
    while ((int)acc_cols < ntok) acc_cols <<= 1;
    const uint32_t tmem_cols = 2 * acc_cols;
    const size_t stage_bytes = W_TILE_BYTES + (size_t)ntok * 128;
    const size_t budget = 200 * 1024;
    int stages = (int)(budget / stage_bytes);
    if (stages > 12) stages = 12;
    const size_t smem = (size_t)stages * stage_bytes + 1024 + 8 * (2 * stages + 4) + 64;
    CUtensorMap map_a;
    int rc = tc::tensor_map_for(a, M, K, lda, ntok, &map_a);
    if (rc != JLLM_OK) return rc;
    int* error_word = jllm_gemm_error_word();
    if (!error_word) return jllm_fail(JLLM_CUDA_ERROR, "gemm_stream: no error word");
    const VecRef b{bias, bias_dtype};
    if (max_blocks <= 0 && cluster >= 0) {
        const ClusterCut c = cluster > 0 ? cluster_of(cluster, ntok, tiles, k_blocks, out_dtype)
                                         : choose_cluster(ntok, tiles, k_blocks, out_dtype, sms);
        JLLM_REQUIRE(cluster == 0 || c.blocks == cluster, "gemm_stream: clusters of %d blocks do not take %d tiles of %d k blocks, %d rows",
                     cluster, tiles, k_blocks, M);
        if (c.blocks > 0) {
#define JLLM_CLUSTER_GO(T)                                                                                          \
    do {                                                                                                            \
        auto kern = gemm_cluster_kernel<T>;                                                                         \
        if (jllm_allow_smem((const void*)kern, c.smem) != cudaSuccess)                                              \
            return jllm_fail(JLLM_CUDA_ERROR, "gemm_stream: %zu bytes of shared memory refused", c.smem);           \
        cudaLaunchAttribute attr[2];                                                                                \
        cudaLaunchConfig_t cfg = cluster_config<T>(c, tiles, attr, stream);                                         \
        if (jllm_launch_overlaps(c.smem, LAUNCH_DEPENDENT)) {                                                       \
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;                                        \
            attr[1].val.programmaticStreamSerializationAllowed = 1;                                                 \
            cfg.numAttrs = 2;                                                                                       \
        }                                                                                                           \
        cudaLaunchKernelEx(&cfg, kern, map_a, (const __nv_bfloat16*)w_packed, b, (int)(bias != nullptr), (T*)out, ldo, accumulate, \
                           M, N, k_blocks, swiglu, ntok, c.stages, acc_cols, c.blocks, c.share, c.overlay, error_word); \
    } while (0)
            if (out_dtype == JLLM_F32) JLLM_CLUSTER_GO(float); else JLLM_CLUSTER_GO(__nv_bfloat16);
#undef JLLM_CLUSTER_GO
            return jllm_check_launch("gemm_cluster");
        }
    }
    const long long total = (long long)tiles * k_blocks;
    int grid = total < sms ? (int)total : sms;
    if (grid > 160) grid = 160;
    if (max_blocks > 0 && grid > max_blocks) grid = max_blocks;
    int* counters = reinterpret_cast<int*>(workspace);
    float* partials = workspace + 2 * MAX_TILES;      // two counters per tile (counted in, done), then the parked parts
#define JLLM_STREAM_GO(T)                                                                                           \
    do {                                                                                                            \
        auto kern = gemm_stream_kernel<T>;                                                                          \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                         \
        jllm_launch(kern, dim3(grid), dim3(THREADS), smem, stream, LAUNCH_DEPENDENT, map_a,                          \
                    (const __nv_bfloat16*)w_packed, b, (int)(bias != nullptr), (T*)out, ldo, accumulate, M, N, k_blocks, \
                    swiglu, ntok, stages, tmem_cols, partials, counters, error_word);                               \
    } while (0)
    if (out_dtype == JLLM_F32) JLLM_STREAM_GO(float); else JLLM_STREAM_GO(__nv_bfloat16);
#undef JLLM_STREAM_GO
    return jllm_check_launch("gemm_stream");
}

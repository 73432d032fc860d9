// out[m, n] (+)= sum_k a[m, k] * w[n, k] (+ bias[n]) on the CUDA cores, true 32-bit products and sums.
//
// This is the matrix product of the float32 path (no tensor cores, no reduced-precision mode) and the fallback of the
// bfloat16 path for shapes the tensor-core kernels refuse.
//
// The order of an element's sum is fixed by K alone: k is cut into four groups of neighbouring values, a group is summed
// over its even and its odd k in two chains of fused multiply-adds in ascending k, and the result is
// ((g0 + g1) + g2) + g3, g = even + odd. It does not depend on the tile an element falls in, on M, on the other rows of the
// batch or on how the operands are loaded, so a row has the same bits however its prompt was cut. (A value that lies
// outside the operands counts as an exact zero product.)
//
// What the split is for: a cluster of four blocks works on one tile, a group of k each, and adds the groups up through
// distributed shared memory; a product of few rows, whose only work is to stream the weights, has blocks for every SM even
// where the matrix has few rows (4096 x 4096: 256 blocks), with no workspace and no second pass. The two chains are the two
// halves of a packed multiply-add (fma.rn.f32x2): both operands are register pairs just as 16-byte loads along k deliver
// them, one instruction does two products, and the issue slots it leaves free take the loads from shared memory.
//
// Tiles of 4, 16, 32 or 64 rows by 64 or 128 weight rows by 32 k, brought by 16-byte cp.async into a ring of stages whose
// rows are 128 bytes with their 16-byte pieces exchanged by the row's number (no bank is hit twice by the eight weight rows
// that a quarter of a warp reads). A warp is 4 rows x 8 weight rows of threads, a thread holds up to 8 x 8 elements. What
// bounds it: from 32 rows on the multiply-adds, below that the weights' bytes. 300 rows of the 8B layer products: 43 TFLOP/s
// (5 before: 4 x 4 elements a thread, scalar loads, no loads ahead); one row: 5.3 TB/s of weights (a prompt of 300 rows and
// four rows behind it, two layers and the head: 44.3 ms of products before, 9.8 now). Operands whose rows are no multiples of 16
// bytes are loaded value by value into the same ring. So are bfloat16 ones, or four at a time where rows and pieces allow; theirs wait
// in registers while the step in hand is worked on.
#include <cooperative_groups.h>

#include "common.cuh"

namespace {

constexpr int BK = 32, GROUPS = 4, THREADS = 128;

__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// four bfloat16 values as they lie in memory
struct Four {
    uint2 v;
    __device__ __forceinline__ float4 floats() const {
        return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                           __uint_as_float(v.y & 0xffff0000u));
    }
};
// the values k .. k + 3 of a row in front of `end`, zeros behind it; `whole`: the four lie inside or outside together, aligned
__device__ __forceinline__ Four fetch4(const __nv_bfloat16* p, int k, int end, int whole) {
    Four x = {make_uint2(0u, 0u)};
    if (whole) {
        if (k < end) x.v = *reinterpret_cast<const uint2*>(p + k);
    } else {
        const uint16_t* u = reinterpret_cast<const uint16_t*>(p);
        if (k + 0 < end) x.v.x = u[k];
        if (k + 1 < end) x.v.x |= (uint32_t)u[k + 1] << 16;
        if (k + 2 < end) x.v.y = u[k + 2];
        if (k + 3 < end) x.v.y |= (uint32_t)u[k + 3] << 16;
    }
    return x;
}

__device__ __forceinline__ void copy16(uint32_t smem, const void* p, bool inside) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(p), "r"(inside ? 16 : 0) : "memory");
}

// k values of a group: a quarter of K, rounded up so that no piece of four lies in two groups
__host__ __device__ __forceinline__ int group_size(int K) { return ((K + GROUPS - 1) / GROUPS + 3) / 4 * 4; }

// TI x TJ elements a thread, WM x WN warps; blocks of a cluster are the groups of k of one tile, tiles of the same weight
// rows follow one another (they meet in L2)
template <int TI, int TJ, int WM, int WN, int STAGES, typename Tin, typename Tout, bool WIDE>
__global__ void __cluster_dims__(GROUPS, 1, 1) __launch_bounds__(THREADS)
gemm_plain_kernel(const Tin* __restrict__ a, int lda, const Tin* __restrict__ w, int ldw, VecRef bias, int has_bias,
                  Tout* __restrict__ out, int ldo, int accumulate, int M, int N, int K, int row_tiles, int whole) {
    constexpr int BM = 4 * TI * WM, BN = 8 * TJ * WN, ROWS = BM + BN, STAGE = ROWS * BK;
    constexpr int PIECES = (ROWS * 8 + THREADS - 1) / THREADS;
    constexpr bool HELD = sizeof(Tin) == 2;
    constexpr int AHEAD = HELD ? 1 : STAGES - 1;         // steps between a load and the step in hand
    static_assert(32 * WM * WN == THREADS, "four warps");
    extern __shared__ __align__(128) float smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = blockIdx.x & (GROUPS - 1), tile = blockIdx.x / GROUPS;
    const int m0 = (tile % row_tiles) * BM, n0 = (tile / row_tiles) * BN;
    const int per = group_size(K), k_lo = min(K, group * per), k_hi = min(K, k_lo + per);
    const int steps = (k_hi - k_lo + BK - 1) / BK;

    // stage `s` takes the k values from k_lo + step * BK on: rows [0, BM) are a's, the rest w's (HELD: they are fetched here and `put` there)
    Four held[HELD ? PIECES : 1];
    auto load = [&](int step, int s) {
        const int kb = k_lo + step * BK;
        float* to = smem + s * STAGE;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const int u = tid + i * THREADS, r = u >> 3, c = u & 7;
            if (ROWS * 8 % THREADS != 0 && u >= ROWS * 8) break;
            const int k = kb + c * 4, row = r < BM ? m0 + r : n0 + r - BM;
            const bool there = r < BM ? row < M : row < N;
            const Tin* p = r < BM ? a + (size_t)(there ? row : 0) * lda : w + (size_t)(there ? row : 0) * ldw;
            float* dst = to + r * BK + ((c ^ (r & 7)) << 2);
            if constexpr (WIDE) {
                const bool inside = there && k < k_hi;
                copy16((uint32_t)__cvta_generic_to_shared(dst), inside ? p + k : p, inside);
            } else if constexpr (HELD) {
                held[i] = fetch4(p, k, there ? k_hi : 0, whole);
            } else {
                float4 v;
                v.x = there && k + 0 < k_hi ? to_float(p[k + 0]) : 0.f;
                v.y = there && k + 1 < k_hi ? to_float(p[k + 1]) : 0.f;
                v.z = there && k + 2 < k_hi ? to_float(p[k + 2]) : 0.f;
                v.w = there && k + 3 < k_hi ? to_float(p[k + 3]) : 0.f;
                *reinterpret_cast<float4*>(dst) = v;
            }
        }
    };
    auto put = [&](int s) {
        if constexpr (HELD) {
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const int u = tid + i * THREADS, r = u >> 3, c = u & 7;
                if (ROWS * 8 % THREADS != 0 && u >= ROWS * 8) break;
                *reinterpret_cast<float4*>(smem + s * STAGE + r * BK + ((c ^ (r & 7)) << 2)) = held[i].floats();
            }
        }
    };

    if constexpr (WIDE) {       // the first weights are asked for while the predecessor still runs
        for (int u = tid; u < BN * (STAGES - 1); u += THREADS) {
            const int n = n0 + u % BN, k = k_lo + u / BN * BK;
            if (n < N && k < k_hi) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (size_t)n * ldw + k));
        }
    }
    pdl_wait();
    pdl_trigger();

    uint64_t acc[TI][TJ];
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) acc[i][j] = 0;

#pragma unroll
    for (int s = 0; s < AHEAD; ++s) {
        if (s < steps) {
            load(s, s);
            put(s);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int ar = (warp / WN) * 4 * TI + (lane >> 3), wr = BM + (warp % WN) * 8 * TJ + (lane & 7);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory");
        __syncthreads();
        if (step + AHEAD < steps) load(step + AHEAD, (step + AHEAD) % STAGES);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* s = smem + (step % STAGES) * STAGE;
#pragma unroll
        for (int c = 0; c < BK / 4; ++c) {
            ulonglong2 wv[TJ];
#pragma unroll
            for (int j = 0; j < TJ; ++j)       // (BM is a multiple of 4 only: a row's number decides, not the lane's)
                wv[j] = *reinterpret_cast<const ulonglong2*>(s + (wr + 8 * j) * BK + ((c ^ ((wr + 8 * j) & 7)) << 2));
#pragma unroll
            for (int i = 0; i < TI; ++i) {
                const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(s + (ar + 4 * i) * BK + ((c ^ ((ar + 4 * i) & 7)) << 2));
#pragma unroll
                for (int j = 0; j < TJ; ++j) fma2(acc[i][j], av.x, wv[j].x);
#pragma unroll
                for (int j = 0; j < TJ; ++j) fma2(acc[i][j], av.y, wv[j].y);
            }
        }
        if (HELD && step + AHEAD < steps) put((step + AHEAD) % STAGES);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // the group's sums of the tile, then every block of the cluster adds a quarter of the columns up over the four groups
    constexpr int PITCH = BN + 4;
    static_assert(BM * PITCH <= STAGES * STAGE, "the tile's sums fit the ring");
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) {
            float even, odd;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(acc[i][j]));
            smem[(ar + 4 * i) * PITCH + wr - BM + 8 * j] = __fadd_rn(even, odd);
        }
    const auto cluster = cooperative_groups::this_cluster();
    cluster.sync();
    const float* part[GROUPS];
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) part[g] = cluster.map_shared_rank(smem, g);
    constexpr int COLS = BN / GROUPS;
    for (int u = tid; u < BM * COLS; u += THREADS) {
        const int r = u / COLS, col = group * COLS + u % COLS, m = m0 + r, n = n0 + col;
        if (m >= M || n >= N) continue;
        float v = part[0][r * PITCH + col];
#pragma unroll
        for (int g = 1; g < GROUPS; ++g) v = __fadd_rn(v, part[g][r * PITCH + col]);
        if (has_bias) v = __fadd_rn(v, bias[n]);
        Tout* dst = out + (size_t)m * ldo + n;
        v = epilogue_act(v, accumulate);
        if (accumulate == EPI_ADD) v = __fadd_rn(v, to_float(*dst));
        *dst = from_float<Tout>(v);
    }
    cluster.sync();        // nobody leaves while its sums are being read
}

template <int TI, int TJ, int WM, int WN, int STAGES, typename Tin, typename Tout, bool WIDE>
int launch_tile(const void* a, int lda, const void* w, int ldw, VecRef bias, int has_bias, void* out, int ldo, int accumulate,
                int M, int N, int K, cudaStream_t stream) {
    constexpr int BM = 4 * TI * WM, BN = 8 * TJ * WN;
    constexpr size_t smem = (size_t)STAGES * (BM + BN) * BK * sizeof(float);
    auto kernel = gemm_plain_kernel<TI, TJ, WM, WN, STAGES, Tin, Tout, WIDE>;
    if (jllm_allow_smem((const void*)kernel, smem) != cudaSuccess) return jllm_check_launch("gemm_plain");
    const long long row_tiles = (M + BM - 1) / BM, tiles = row_tiles * ((N + BN - 1) / BN);
    JLLM_REQUIRE(tiles <= 0x7fffffffll / GROUPS, "gemm: M=%d N=%d are too many tiles", M, N);
    const size_t piece = 4 * sizeof(Tin);
    const int whole = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)a % piece == 0 && (uintptr_t)w % piece == 0;
    if (jllm_launch(kernel, dim3((unsigned)(tiles * GROUPS)), dim3(THREADS), smem, stream, LAUNCH_DEPENDENT, (const Tin*)a, lda,
                    (const Tin*)w, ldw, bias, has_bias, (Tout*)out, ldo, accumulate, M, N, K, (int)row_tiles, whole) != cudaSuccess)
        return jllm_check_launch("gemm_plain");
    return jllm_check_launch("gemm_plain");
}

// The tile for M rows. A tile of 64 rows reads least from shared memory per multiply-add; the smaller ones are for products
// that would leave most of it empty: up to 4 and 16 rows the weights' stream is the bound (more, smaller tiles keep more
// bytes on their way), up to 32 rows, and where 32-row tiles leave a fifth fewer rows empty, the multiply-adds. Where even the blocks
// of 16-row tiles are on the SMs at once, a larger tile only makes the few blocks longer (64 rows, 48 x 32: 7.9 us in one tile, 3.9
// in four); of a short k two such blocks share an SM and wait together (300 rows, 300 x 64, bfloat16: 10.3 us in 64-row tiles).
template <typename Tin, typename Tout, bool WIDE>
int launch(const void* a, int lda, const void* w, int ldw, VecRef bias, int has_bias, void* out, int ldo, int accumulate, int M,
           int N, int K, cudaStream_t stream) {
    if (M <= 4) return launch_tile<1, 2, 1, 4, 6, Tin, Tout, WIDE>(a, lda, w, ldw, bias, has_bias, out, ldo, accumulate, M, N, K, stream);
    const int sms = jllm_device_sm_count();
    if (M <= 16 || (M + 15ll) / 16 * ((N + 127ll) / 128) * GROUPS <= (K <= 128 ? 2 : 1) * sms)
        return launch_tile<4, 4, 1, 4, 4, Tin, Tout, WIDE>(a, lda, w, ldw, bias, has_bias, out, ldo, accumulate, M, N, K, stream);
    const long long in32 = (M + 31) / 32 * 32ll, in64 = (M + 63) / 64 * 64ll;
    if (in32 * 6 > in64 * 5)
        return launch_tile<8, 8, 2, 2, 3, Tin, Tout, WIDE>(a, lda, w, ldw, bias, has_bias, out, ldo, accumulate, M, N, K, stream);
    return launch_tile<8, 4, 1, 4, 3, Tin, Tout, WIDE>(a, lda, w, ldw, bias, has_bias, out, ldo, accumulate, M, N, K, stream);
}

bool wide_rows(const void* p, int stride) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && stride % 4 == 0; }

}  // namespace

JLLM_EXPORT int jllm_gemm_plain(const void* a, int in_dtype, int lda, const void* w, int ldw, const void* bias,
                                int bias_dtype, void* out, int out_dtype, int ldo, int accumulate, int M, int N, int K,
                                cudaStream_t stream) {
    JLLM_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm: M=%d N=%d K=%d", M, N, K);
    JLLM_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm: strides lda=%d ldw=%d ldo=%d for K=%d N=%d", lda, ldw, ldo, K, N);
    JLLM_REQUIRE((M + 63) / 64 <= 65535, "gemm: M=%d is above %d rows", M, 65535 * 64);
    if (M == 0) return JLLM_OK;
    const VecRef b{bias, bias_dtype};
    const int hb = bias != nullptr;
    if (in_dtype == JLLM_F32 && out_dtype == JLLM_F32) {
        if (K % 4 == 0 && wide_rows(a, lda) && wide_rows(w, ldw))
            return launch<float, float, true>(a, lda, w, ldw, b, hb, out, ldo, accumulate, M, N, K, stream);
        return launch<float, float, false>(a, lda, w, ldw, b, hb, out, ldo, accumulate, M, N, K, stream);
    }
    if (in_dtype == JLLM_BF16 && out_dtype == JLLM_F32)
        return launch<__nv_bfloat16, float, false>(a, lda, w, ldw, b, hb, out, ldo, accumulate, M, N, K, stream);
    if (in_dtype == JLLM_BF16 && out_dtype == JLLM_BF16)
        return launch<__nv_bfloat16, __nv_bfloat16, false>(a, lda, w, ldw, b, hb, out, ldo, accumulate, M, N, K, stream);
    return jllm_fail(JLLM_UNSUPPORTED, "gemm: float32 inputs with a bfloat16 result are not built");
}

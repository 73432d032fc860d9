// Causal grouped-query attention over the paged cache, one thread block per (row, up to four query heads of a kv head).
//
// The kernel of the float32 path, and the one the bfloat16 path falls back to for head sizes its
// tensor-core kernels refuse (a head size they do not take, keys and values of different widths). A row at
// position P of request `seg` sees the keys [first, P] of that request, first = jllm_first_key(P, window): 0,
// max(0, P + 1 - window) under a window, the start of P's own chunk of -window positions under chunks.
//
// The visible keys are walked in ascending order, CHUNK at a time. A chunk stands for itself: its largest score, the
// exponentials of its scores less that, their sum and the weighted sum of its values; then it is merged into what the chunks
// before it gave. Which keys form a chunk depends on the row's own keys only, and so does every sum's order: a row's result
// does not depend on how the prompt was cut, on the other rows of the batch, on the pages, or on how many blocks share its
// chunks.
//
// What bounds it is latency (a row has a few hundred keys): a warp takes four keys at a time, a key's row is read once, by
// the lanes side by side, for all heads of the block, and the lanes' parts of 4 keys x 4 heads are added up by exchanging halves
// (16 shuffles for 16 sums). Steps of few rows, which would give few blocks, put a cluster of eight on a row: block z takes
// chunk z of every eight, the first one merges them through distributed shared memory. 300 causal rows of 32 heads over 8: 0.10 ms
// with the wait for its predecessor, one row behind them 20 us (1.9 and 0.17 ms with a thread to a key and a block to a head).
//
// Two things a mixer may add. `keep_first` > 0 (with a window): the request's first keep_first keys stay visible to every
// later row, so a row sees [0, keep_first) and [first, P]; the keys in between are passed over. `sink` (one number per query
// head, else null): the softmax's denominator also holds exp(sink[h]), a key without a value that is not multiplied by the
// scale; the running maximum starts from it, so nothing overflows whichever is larger. And a cap on the scores (`softcap` > 0):
// s = softcap * tanh(scale (q . k) / softcap).
//
// Layouts: q [rows, q_stride] with head h at h * head_dim; cache K and V
// [pages, kv_heads, page_size, cache_dim], a key in the first head_dim values of its row and a value in the first
// value_dim; out [rows, out_stride] with head h at h * value_dim; block_tables [segments, table_stride]
// (page id of position p of a segment: table[p / page_size]).
#include <cooperative_groups.h>

#include "common.cuh"

namespace {

constexpr int THREADS = 128, WARPS = 4, CHUNK = 64, SHARERS = 8;
constexpr int MAX_DIMS_PER_THREAD = 8;  // value_dim <= 1024

__device__ __forceinline__ float4 four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)),
                 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
template <typename T> __device__ __forceinline__ float4 four_of(const T* p, int n) {     // the first n values, zeros behind them
    return make_float4(n > 0 ? to_float(p[0]) : 0.f, n > 1 ? to_float(p[1]) : 0.f, n > 2 ? to_float(p[2]) : 0.f,
                       n > 3 ? to_float(p[3]) : 0.f);
}

// HG query heads of one kv head a block, NC value dims a thread; SHARED: the blocks of a cluster along z share the chunks
template <typename T, int HG, int NC, bool SHARED>
__global__ void __launch_bounds__(THREADS)
attention_plain_kernel(const T* __restrict__ q, int q_stride, const T* __restrict__ k_cache,
                       const T* __restrict__ v_cache, T* __restrict__ out, int out_stride,
                       const int* __restrict__ row_seg, const int* __restrict__ row_pos,
                       const int* __restrict__ block_tables, int table_stride, int heads, int kv_heads, int head_dim,
                       int value_dim, int cache_dim, int page_size, int num_pages, int window, float scale, int keep_first,
                       VecRef sink, int has_sink, float softcap, int wide) {
    constexpr int KEYS = 4, VALUES = KEYS * HG;         // keys a warp takes at a time
    extern __shared__ __align__(16) float smem[];
    const int padded = (head_dim + 127) / 128 * 128;
    float* qs = smem;                                   // [HG][padded], zeros behind head_dim
    float* es = qs + HG * padded;                       // [CHUNK][HG] scores, then exponentials
    float* tops = es + CHUNK * HG;                      // [HG] the chunk's largest scores
    float* sums = tops + HG;                            // [HG] its sums
    long long* rows_at = reinterpret_cast<long long*>(sums + HG + (HG & 1 ? 2 : 0));     // [CHUNK] the keys' rows in the cache, -1: none
    float* parts = reinterpret_cast<float*>(rows_at + CHUNK);      // SHARED: [HG][NC * THREADS] the chunk's weighted values
    const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = heads / kv_heads, sets = (per + HG - 1) / HG;
    const int kvh = blockIdx.y / sets, h0 = kvh * per + blockIdx.y % sets * HG, live = min(HG, per - blockIdx.y % sets * HG);
    pdl_wait();
    pdl_trigger();
    const int P = row_pos[r];
    const int first = jllm_first_key(P, window);
    const int kept = window > 0 ? min(keep_first, first) : 0;      // keys [0, kept) in front of the window
    const int* table = block_tables + (size_t)row_seg[r] * table_stride;
    for (int i = tid; i < HG * padded; i += THREADS) {
        const int h = i / padded, d = i % padded;
        qs[i] = h < live && d < head_dim ? to_float(q[(size_t)r * q_stride + (size_t)(h0 + h) * head_dim + d]) : 0.f;
    }
    // the visible keys in ascending order: index u < kept is key u, index u >= kept is key first + (u - kept)
    const int visible = kept + (P + 1 - first), chunks = (visible + CHUNK - 1) / CHUNK;
    const int sharers = SHARED ? SHARERS : 1, mine = SHARED ? blockIdx.z : 0;

    // what the chunks so far gave (SHARED: in the cluster's first block)
    float top[HG], sum[HG], acc[HG][NC];
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        top[h] = has_sink && h < live ? sink[h0 + h] : -INFINITY;
        sum[h] = has_sink ? 1.f : 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[h][c] = 0.f;
    }
    // (Nothing is skipped: a chunk without a finite score has weights of 0, or of NaN where a score was NaN, and either goes on
    // into the sums. Its maximum is -inf, from which no difference is taken.)
    auto merge = [&](int h, float t, float s, const float (&v)[NC]) {
        const float m = fmaxf(top[h], t), from = m == -INFINITY ? 0.f : m, old = expf(top[h] - from), add = expf(t - from);
        top[h] = m;
        sum[h] = __fmaf_rn(s, add, __fmul_rn(sum[h], old));
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[h][c] = __fmaf_rn(v[c], add, __fmul_rn(acc[h][c], old));
    };

    for (int base = 0; base < chunks; base += sharers) {
        const int u0 = (base + mine) * CHUNK, n = min(CHUNK, visible - u0);     // SHARED: n <= 0 in the blocks without a chunk
        __syncthreads();
        for (int j = tid; j < n; j += THREADS) {
            const int u = u0 + j, s = u < kept ? u : first + (u - kept);
            const long long page = jllm_page_of(table, s / page_size, table_stride, num_pages);
            rows_at[j] = kCheckBounds && page < 0 ? -1 : (page * kv_heads + kvh) * page_size + s % page_size;
        }
        __syncthreads();
        for (int j0 = warp * KEYS; j0 < n; j0 += WARPS * KEYS) {
            float v[VALUES];
#pragma unroll
            for (int i = 0; i < VALUES; ++i) v[i] = 0.f;
            long long at[KEYS];
#pragma unroll
            for (int k = 0; k < KEYS; ++k) at[k] = j0 + k < n ? rows_at[j0 + k] : -1;
            for (int d0 = 0; d0 < head_dim; d0 += 128) {
                const int d = d0 + lane * 4, have = head_dim - d;
                float4 kv[KEYS];
#pragma unroll
                for (int k = 0; k < KEYS; ++k) {
                    const T* p = k_cache + (at[k] < 0 ? 0 : at[k]) * cache_dim + d;
                    kv[k] = at[k] < 0 || have <= 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : wide ? four(p) : four_of(p, have);
                }
#pragma unroll
                for (int h = 0; h < HG; ++h) {
                    const float4 x = four(qs + h * padded + d);
#pragma unroll
                    for (int k = 0; k < KEYS; ++k)
                        v[k * HG + h] = fmaf(x.w, kv[k].w, fmaf(x.z, kv[k].z, fmaf(x.y, kv[k].y, fmaf(x.x, kv[k].x, v[k * HG + h]))));
                }
            }
            // lane l ends with the sum of value l / (32 / VALUES): halves are exchanged until one value is left, then added up
            int width = 16;
#pragma unroll
            for (int half = VALUES / 2; half > 0; half /= 2, width /= 2)
#pragma unroll
                for (int i = 0; i < half; ++i) {
                    const bool upper = lane & width;
                    const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
                    v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, width));
                }
#pragma unroll
            for (int o = 32 / VALUES / 2; o > 0; o /= 2) v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
            if (lane % (32 / VALUES) == 0) {
                const int value = lane / (32 / VALUES), k = value / HG, h = value % HG;
                const float scaled = __fmul_rn(v[0], scale);
                float s = softcap > 0.f ? __fmul_rn(softcap, tanhf(scaled / softcap)) : scaled;
                if (j0 + k < n) es[(j0 + k) * HG + h] = kCheckBounds && rows_at[j0 + k] < 0 ? -INFINITY : s;
            }
        }
        __syncthreads();
        for (int h = warp; h < HG; h += WARPS) {
            float t = -INFINITY, s = 0.f;
            for (int j = lane; j < n; j += 32) t = fmaxf(t, es[j * HG + h]);
            t = warp_max(t);                            // (-inf: no score is above it, but some may be NaN)
            const float from = t == -INFINITY ? 0.f : t;
            for (int j = lane; j < n; j += 32) {
                const float e = expf(es[j * HG + h] - from);
                es[j * HG + h] = e;
                s += e;
            }
            s = warp_sum(s);
            if (lane == 0) tops[h] = t, sums[h] = s;
        }
        __syncthreads();
        float add[HG][NC];
#pragma unroll
        for (int h = 0; h < HG; ++h)
#pragma unroll
            for (int c = 0; c < NC; ++c) add[h][c] = 0.f;
#pragma unroll 8
        for (int j = 0; j < n; ++j) {
            const long long at = rows_at[j];
            if (kCheckBounds && at < 0) continue;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int d = tid + c * THREADS;
                const float x = d < value_dim ? to_float(v_cache[at * cache_dim + d]) : 0.f;
#pragma unroll
                for (int h = 0; h < HG; ++h) add[h][c] = fmaf(es[j * HG + h], x, add[h][c]);
            }
        }
        if constexpr (SHARED) {
            const auto cluster = cooperative_groups::this_cluster();
#pragma unroll
            for (int h = 0; h < HG; ++h)
#pragma unroll
                for (int c = 0; c < NC; ++c) parts[h * NC * THREADS + c * THREADS + tid] = add[h][c];
            cluster.sync();
            if (mine == 0) {
                for (int z = 0; z < sharers && base + z < chunks; ++z) {
                    const float *t = cluster.map_shared_rank(tops, z), *s = cluster.map_shared_rank(sums, z),
                                *p = cluster.map_shared_rank(parts, z);
#pragma unroll
                    for (int h = 0; h < HG; ++h) {
                        float v[NC];
#pragma unroll
                        for (int c = 0; c < NC; ++c) v[c] = p[h * NC * THREADS + c * THREADS + tid];
                        merge(h, t[h], s[h], v);
                    }
                }
            }
            cluster.sync();        // the parts are read before they are written again, and before a block leaves
        } else {
#pragma unroll
            for (int h = 0; h < HG; ++h) merge(h, tops[h], sums[h], add[h]);
        }
    }
    if (mine != 0) return;
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        if (h >= live) break;
        const float inv = 1.f / sum[h];
        T* orow = out + (size_t)r * out_stride + (size_t)(h0 + h) * value_dim;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = tid + c * THREADS;
            if (d < value_dim) orow[d] = from_float<T>(__fmul_rn(acc[h][c], inv));
        }
    }
}

struct PlainArgs {
    const void *q, *k, *v;
    void* out;
    int q_stride, out_stride;
    const int *row_seg, *row_pos, *tables;
    int table_stride, rows, heads, kv_heads, head_dim, value_dim, cache_dim, page_size, window;
    float scale;
    int keep_first;
    VecRef sink;
    int has_sink;
    float softcap;
    int wide;
};

template <typename T, int HG, int NC, bool SHARED>
int launch_plain(const PlainArgs& a, cudaStream_t stream) {
    const size_t padded = (a.head_dim + 127) / 128 * 128;
    const size_t smem = (HG * padded + CHUNK * HG + 2 * HG + (HG & 1 ? 2 : 0) + (SHARED ? HG * NC * THREADS : 0)) * sizeof(float) +
                        CHUNK * sizeof(long long);
    auto kernel = attention_plain_kernel<T, HG, NC, SHARED>;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return jllm_check_launch("attention_plain");
    const int per = a.heads / a.kv_heads;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.rows, a.kv_heads * ((per + HG - 1) / HG), SHARED ? SHARERS : 1);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (SHARED) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1, attr[n].val.clusterDim.y = 1, attr[n++].val.clusterDim.z = SHARERS;
    }
    if (jllm_launch_overlaps(smem, LAUNCH_DEPENDENT)) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, kernel, (const T*)a.q, a.q_stride, (const T*)a.k, (const T*)a.v, (T*)a.out, a.out_stride, a.row_seg,
                       a.row_pos, a.tables, a.table_stride, a.heads, a.kv_heads, a.head_dim, a.value_dim, a.cache_dim, a.page_size,
                       jllm_pool_pages(), a.window, a.scale, a.keep_first, a.sink, a.has_sink, a.softcap, a.wide);
    return jllm_check_launch("attention_plain");
}

// A cluster shares a row's chunks where the blocks of all rows would leave SMs idle (one row of 32 heads over 8: 8 blocks). Eight rows in
// clusters and sixteen without, float32, 32 heads of 128 over 8: 1,000 keys 39 and 152 us, 300 keys 18 and 30, 100 keys 14 and 13, 20 keys
// 8.5 and 6.0 (a cluster's start is 2 us, which rows of a chunk or two do not win back; their length is not known here).
template <typename T, int HG, int NC>
int launch_shared(const PlainArgs& a, cudaStream_t stream) {
    const long long blocks = (long long)a.rows * a.kv_heads * ((a.heads / a.kv_heads + HG - 1) / HG);
    const int sms = jllm_device_sm_count();
    if (sms > 0 && blocks * 2 <= sms) return launch_plain<T, HG, NC, true>(a, stream);
    return launch_plain<T, HG, NC, false>(a, stream);
}

template <typename T, int HG>
int launch_dims(const PlainArgs& a, cudaStream_t stream) {
    if (a.value_dim <= THREADS) return launch_shared<T, HG, 1>(a, stream);
    if (a.value_dim <= 2 * THREADS) return launch_shared<T, HG, 2>(a, stream);
    return launch_shared<T, HG, MAX_DIMS_PER_THREAD>(a, stream);
}

template <typename T>
int launch_heads(const PlainArgs& a, cudaStream_t stream) {
    const int per = a.heads / a.kv_heads;
    if (per == 1 || a.head_dim > 2048) return launch_dims<T, 1>(a, stream);      // (four queries of 2,048 values: 32 KB)
    if (per == 2) return launch_dims<T, 2>(a, stream);
    return launch_dims<T, 4>(a, stream);
}

}  // namespace

JLLM_BOUNDS_READER(attention_plain)

JLLM_EXPORT int jllm_attention_plain(const void* q, int q_stride, const void* k_cache, const void* v_cache, void* out,
                                     int out_stride, const int* row_seg, const int* row_pos, const int* block_tables,
                                     int table_stride, int rows, int heads, int kv_heads, int head_dim, int value_dim,
                                     int cache_dim, int page_size, int window, float scale, int dtype, int keep_first,
                                     const void* sink, int sink_dtype, float softcap, cudaStream_t stream) {
    JLLM_REQUIRE(rows >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && head_dim > 0 && page_size > 0,
                 "attention: rows=%d heads=%d kv_heads=%d head_dim=%d page_size=%d", rows, heads, kv_heads, head_dim,
                 page_size);
    JLLM_REQUIRE(value_dim > 0 && value_dim <= THREADS * MAX_DIMS_PER_THREAD && head_dim <= 8192,
                 "attention: head_dim=%d is above 8192 or value_dim=%d above %d", head_dim, value_dim, THREADS * MAX_DIMS_PER_THREAD);
    JLLM_REQUIRE(cache_dim >= head_dim && cache_dim >= value_dim, "attention: cache rows of %d values hold no key of %d or value of %d",
                 cache_dim, head_dim, value_dim);
    JLLM_REQUIRE(heads <= 65535, "attention: heads=%d", heads);
    JLLM_REQUIRE(keep_first >= 0 && (keep_first == 0 || window > 0), "attention: keep_first=%d needs a window (window=%d)",
                 keep_first, window);
    if (rows == 0) return JLLM_OK;
    // (keys of whole pieces of four values, every cache row on a piece's boundary)
    const size_t piece = 4 * (dtype == JLLM_F32 ? sizeof(float) : sizeof(__nv_bfloat16));
    const int wide = head_dim % 4 == 0 && cache_dim % 4 == 0 && reinterpret_cast<uintptr_t>(k_cache) % piece == 0;
    const PlainArgs a{q, k_cache, v_cache, out, q_stride, out_stride, row_seg, row_pos, block_tables, table_stride, rows, heads,
                      kv_heads, head_dim, value_dim, cache_dim, page_size, window, scale, keep_first, VecRef{sink, sink_dtype},
                      sink != nullptr, softcap, wide};
    return dtype == JLLM_F32 ? launch_heads<float>(a, stream) : launch_heads<__nv_bfloat16>(a, stream);
}

// Gated linear attention: the recurrence over a request's tokens, and the per-head norm and gate of its output.
//
// Per head, with dk key channels and dv value channels, a request carries a state S [dk, dv] in 32-bit floats:
//     S_t = diag(d_t) S_(t-1) + k_t v_t^T,    o_t = S_t^T (scale * q_t),    d_t = sigmoid(z_t)^(1 / tau)
// d_t is formed as exp(log_sigmoid(z_t) / tau) in float32 by a kernel in front. The columns of S do not depend on one
// another, so a block owns CB columns (32, or 16 where that gives more SMs a block) of one (segment, head). A thread holds R
// rows of one column in registers (row group g, column c); every token's k, d, q and v are staged through shared
// memory eight tokens at a time, the next eight being fetched into registers while these are worked on, and the G
// partial sums of o_t are added in the order of g. A token's arithmetic is the same sequence of operations wherever its
// portion begins, whatever else the batch holds and however the columns are dealt out, so the result has the same
// bits for every cut.
//
// A segment is a run of consecutive rows of one request (a prompt portion, or one decoded token); its state lies in
// `state[slot]` ([slots, heads, dk, dv]), is read at the segment's first token and written back after its last. The
// same kernel serves a prompt and a decode step; the float32 and the bfloat16 path differ in the type of q, k, v only.
#include <cstdlib>

#include "common.cuh"

namespace {

constexpr int TOKENS = 8;       // tokens staged at a time

// d = sigmoid(z)^(1 / tau), in place over [rows, heads x dk] float32: log(sigmoid(z)) = min(z, 0) - log1p(exp(-|z|)),
// times 1 / tau, exponentiated. Done once per step and element, in front of the recurrence (whose blocks would
// otherwise each redo it for the columns they own).
__global__ void gla_decay_kernel(float* __restrict__ z, float inv_tau, size_t total, int as_log) {
    pdl_wait();
    pdl_trigger();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const float v = z[i];
        const float l = __fmul_rn(fminf(v, 0.f) - log1pf(expf(-fabsf(v))), inv_tau);
        z[i] = as_log ? l : expf(l);        // (the chunked kernels want the logarithm: they add it up over a chunk)
    }
}

// Linear attention with ONE fixed decay per head (no decay projection; "lightning" attention) runs through the same
// kernels: this pass fills the decay table with decay[h] for every key channel of head h (its logarithm for the chunked
// form; a decay of 0 becomes a logarithm of -1e30, whose differences are 0 or below -1e30 and never NaN), and applies
// the activation of such a mixer to its projections in place: q, k, v <- silu (activation 1). A block per row.
__device__ __forceinline__ float2 load_two(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load_two(const __nv_bfloat16* p) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}
__device__ __forceinline__ void store_two(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void store_two(__nv_bfloat16* p, float a, float b) {
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}

template <typename T>
__global__ void __launch_bounds__(256)
fixed_decay_prepare_kernel(T* __restrict__ proj, int ld, int q_off, int k_off, int v_off, float* __restrict__ z,
                           const float* __restrict__ decay, int heads, int dk, int dv, int as_log, int activation) {
    pdl_wait();
    pdl_trigger();
    const size_t r = blockIdx.x;
    float* zr = z + r * heads * dk;
    if (z == nullptr) {
        // (the tensor-core form of the chunks takes the decays themselves: no table)
    } else if ((dk & 3) == 0) {        // (the table's rows are whole float4s then: heads * dk is a multiple of 4, z is an allocation's start)
        for (int i = threadIdx.x; i < heads * dk / 4; i += blockDim.x) {
            const float d = decay[(4 * i) / dk], e = as_log ? fmaxf(logf(d), -1e30f) : d;
            reinterpret_cast<float4*>(zr)[i] = make_float4(e, e, e, e);
        }
    } else {
        for (int i = threadIdx.x; i < heads * dk; i += blockDim.x) {
            const float d = decay[i / dk];
            zr[i] = as_log ? fmaxf(logf(d), -1e30f) : d;
        }
    }
    if (!activation) return;
    T* row = proj + r * ld;
    auto silu = [](float x) { return x / (1.f + expf(-x)); };
    auto run = [&](int off, int n) {
        T* p = row + off;
        if ((n & 1) == 0 && (((uintptr_t)p) & (2 * sizeof(T) - 1)) == 0) {
            for (int i = threadIdx.x; i < n / 2; i += blockDim.x) {
                const float2 v = load_two(p + 2 * i);
                store_two(p + 2 * i, silu(v.x), silu(v.y));
            }
        } else {
            for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = from_float<T>(silu(to_float(p[i])));
        }
    };
    run(q_off, heads * dk);
    run(k_off, heads * dk);
    run(v_off, heads * dv);
}

template <typename T>
int launch_fixed_decay(void* proj, int ld, int q_off, int k_off, int v_off, float* z, const float* decay, int rows, int heads,
                       int dk, int dv, int as_log, int activation, cudaStream_t stream) {
    jllm_launch(fixed_decay_prepare_kernel<T>, dim3(rows), dim3(256), 0, stream, LAUNCH_DEPENDENT, (T*)proj, ld, q_off, k_off,
                v_off, z, decay, heads, dk, dv, as_log, activation);
    return jllm_check_launch("fixed_decay_prepare");
}

template <typename T, int R, int CB, bool V4>
__global__ void __launch_bounds__(1024)
gla_recurrent_kernel(const T* __restrict__ proj, int ld, int q_off, int k_off, int v_off, const float* __restrict__ decay,
                     float* __restrict__ state, const int* __restrict__ seg_start, const int* __restrict__ seg_len,
                     const int* __restrict__ state_slots, float* __restrict__ o, int heads, int dk, int dv, float q_scale,
                     int num_slots, const float* __restrict__ head_decay, int activation) {
    // `head_decay` (else null): one fixed decay per head instead of the table; `activation` 1: q, k and v are taken through
    // silu as they are fetched (and rounded to the projections' type, as a pass that stored them would have left them)
    constexpr int EPT = TOKENS * R / CB;            // staged values of k (and of q, of d) a thread fetches per round
    extern __shared__ __align__(16) float smem[];
    const int threads = blockDim.x, G = threads / CB;
    const int stage = TOKENS * (3 * dk + CB);       // floats of one staging buffer: k, d, q [TOKENS][dk], v [TOKENS][CB]
    float* part = smem + 2 * stage;                 // [TOKENS][G][CB]
    pdl_wait();
    pdl_trigger();
    const int seg = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * CB;
    const int tid = threadIdx.x, c = tid % CB, g = tid / CB, j = c0 + c;
    const int first = seg_start[seg], n = seg_len[seg], slot = state_slots[seg];
    if (!jllm_in_bounds(slot, num_slots, BOUNDS_SLOT)) return;
    float* S = state + (((size_t)slot * heads + h) * dk) * dv;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = g * R + r;
        s[r] = (i < dk && j < dv) ? S[(size_t)i * dv + j] : 0.f;
    }
    // which staged values this thread fetches: the same places of every round, worked out once
    int st[EPT], sp[EPT], sd[EPT];                  // token within the round (TOKENS: none), offsets into proj and decay
#pragma unroll
    for (int u = 0; u < EPT; ++u) {
        const int e = tid + u * threads;
        st[u] = e < TOKENS * dk ? e / dk : TOKENS;
        const int i = e - st[u] * dk;
        sp[u] = st[u] * ld + h * dk + i;
        sd[u] = st[u] * heads * dk + h * dk + i;
    }
    const int vt = tid / CB, vc = tid - vt * CB;    // the one value of v this thread fetches (threads >= TOKENS x CB / 1)
    const int vpt = (TOKENS * CB + threads - 1) / threads;
    float fk[EPT], fq[EPT], fd[EPT], fv[TOKENS];
    const float fixed = head_decay ? head_decay[h] : 1.f;
    auto act = [&](float x) { return activation ? to_float(from_float<T>(x / (1.f + expf(-x)))) : x; };

    auto fetch = [&](int t0) {      // the round that starts at token t0: from global memory into registers
        const int nt = min(TOKENS, n - t0);
        const size_t base = (size_t)(first + t0);
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            fk[u] = fq[u] = 0.f;
            fd[u] = 1.f;
            if (st[u] < nt) {
                const T* p = proj + base * ld + sp[u];
                fk[u] = act(to_float(p[k_off]));
                fq[u] = act(to_float(p[q_off]));
                fd[u] = head_decay ? fixed : decay[base * ((size_t)heads * dk) + sd[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < TOKENS; ++u) {
            fv[u] = 0.f;
            if (u < vpt) {
                const int t = vt + u * (threads / CB);
                if (t < nt && c0 + vc < dv) fv[u] = act(to_float(proj[(base + t) * ld + v_off + (size_t)h * dv + c0 + vc]));
            }
        }
    };
    auto park = [&](int b) {        // ... and from the registers into staging buffer b
        float* ks = smem + b * stage;
        float* ds = ks + TOKENS * dk;
        float* qs = ds + TOKENS * dk;
        float* vs = qs + TOKENS * dk;
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            const int e = tid + u * threads;
            if (e < TOKENS * dk) {
                ks[e] = fk[u];
                ds[e] = fd[u];
                qs[e] = __fmul_rn(fq[u], q_scale);
            }
        }
#pragma unroll
        for (int u = 0; u < TOKENS; ++u) {
            const int t = vt + u * (threads / CB);
            if (u < vpt && t < TOKENS) vs[t * CB + vc] = fv[u];
        }
    };

    if (n > 0) {
        fetch(0);
        park(0);
    }
    __syncthreads();
    const bool rows_in = g * R < dk;
    for (int t0 = 0, b = 0; t0 < n; t0 += TOKENS, b ^= 1) {
        const int nt = min(TOKENS, n - t0);
        const bool more = t0 + TOKENS < n;
        if (more) fetch(t0 + TOKENS);               // on their way while this round's tokens are worked on
        const float* ks = smem + b * stage + g * R;
        const float* ds = ks + TOKENS * dk;
        const float* qs = ds + TOKENS * dk;
        const float* vs = smem + b * stage + 3 * TOKENS * dk;
        for (int t = 0; t < nt; ++t) {
            const float v = vs[t * CB + c];
            float acc0 = 0.f, acc1 = 0.f;
            if constexpr (V4) {     // dk a multiple of 4: four rows' k, d and q in one load each
                if (rows_in) {
#pragma unroll
                    for (int r = 0; r < R; r += 4) {
                        if (g * R + r < dk) {
                            const float4 kk = *reinterpret_cast<const float4*>(ks + t * dk + r);
                            const float4 dd = *reinterpret_cast<const float4*>(ds + t * dk + r);
                            const float4 qq = *reinterpret_cast<const float4*>(qs + t * dk + r);
                            s[r] = fmaf(dd.x, s[r], __fmul_rn(kk.x, v));
                            s[r + 1] = fmaf(dd.y, s[r + 1], __fmul_rn(kk.y, v));
                            s[r + 2] = fmaf(dd.z, s[r + 2], __fmul_rn(kk.z, v));
                            s[r + 3] = fmaf(dd.w, s[r + 3], __fmul_rn(kk.w, v));
                            acc0 = fmaf(s[r], qq.x, acc0);
                            acc1 = fmaf(s[r + 1], qq.y, acc1);
                            acc0 = fmaf(s[r + 2], qq.z, acc0);
                            acc1 = fmaf(s[r + 3], qq.w, acc1);
                        }
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; r += 2) {
                    if (g * R + r < dk) {
                        s[r] = fmaf(ds[t * dk + r], s[r], __fmul_rn(ks[t * dk + r], v));
                        acc0 = fmaf(s[r], qs[t * dk + r], acc0);
                    }
                    if (g * R + r + 1 < dk) {
                        s[r + 1] = fmaf(ds[t * dk + r + 1], s[r + 1], __fmul_rn(ks[t * dk + r + 1], v));
                        acc1 = fmaf(s[r + 1], qs[t * dk + r + 1], acc1);
                    }
                }
            }
            part[(t * G + g) * CB + c] = acc0 + acc1;
        }
        if (more) park(b ^ 1);                      // (the other buffer: its last readers passed the barrier below)
        __syncthreads();
        for (int e = tid; e < nt * CB; e += threads) {
            const int t = e / CB, cc = e - t * CB;
            if (c0 + cc >= dv) continue;
            float acc = 0.f;
            for (int gg = 0; gg < G; ++gg) acc += part[(t * G + gg) * CB + cc];
            o[(size_t)(first + t0 + t) * ((size_t)heads * dv) + (size_t)h * dv + c0 + cc] = acc;
        }
        __syncthreads();                            // `part` and buffer b may be written again
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = g * R + r;
        if (i < dk && j < dv) S[(size_t)i * dv + j] = s[r];
    }
}

template <typename T, int R, int CB, bool V4>
int launch_recurrent(const void* proj, int ld, int q_off, int k_off, int v_off, const float* decay, float* state,
                     const int* seg_start, const int* seg_len, const int* state_slots, float* o, int segments, int heads,
                     int dk, int dv, float q_scale, int num_slots, const float* head_decay, int activation,
                     cudaStream_t stream) {
    const int per_warp = 32 / CB;
    const int G = ((dk + R - 1) / R + per_warp - 1) / per_warp * per_warp;       // row groups: whole warps
    const size_t smem = (size_t)(2 * TOKENS * (3 * dk + CB) + TOKENS * G * CB) * sizeof(float);
    auto kernel = gla_recurrent_kernel<T, R, CB, V4>;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return jllm_fail(JLLM_CUDA_ERROR, "gla_recurrent: %zu bytes of shared memory refused", smem);
    jllm_launch(kernel, dim3(segments, heads, (dv + CB - 1) / CB), dim3(G * CB), smem, stream, LAUNCH_DEPENDENT,
                (const T*)proj, ld, q_off, k_off, v_off, decay, state, seg_start, seg_len, state_slots, o, heads, dk, dv,
                q_scale, num_slots, head_decay, activation);
    return jllm_check_launch("gla_recurrent");
}

// Columns per block: 32 (a warp is one row group), or 16 where 32 columns per block leave SMs without one. The choice
// changes which thread holds which value, not what is computed.
template <typename T, int R>
int launch_recurrent_cols(const void* proj, int ld, int q_off, int k_off, int v_off, const float* decay, float* state,
                          const int* seg_start, const int* seg_len, const int* state_slots, float* o, int segments,
                          int heads, int dk, int dv, float q_scale, int num_slots, const float* head_decay, int activation,
                          cudaStream_t stream) {
    const long long sms = max(1, jllm_device_sm_count());
    const long long units = (long long)segments * heads;
    const bool wide = units * ((dv + 31) / 32) >= sms || dv <= 16;
#define JLLM_GLA_COLS(CB, V4)                                                                                                  \
    return launch_recurrent<T, R, CB, V4>(proj, ld, q_off, k_off, v_off, decay, state, seg_start, seg_len, state_slots, o, \
                                          segments, heads, dk, dv, q_scale, num_slots, head_decay, activation, stream)
    if (dk % 4 == 0) {
        if (wide) JLLM_GLA_COLS(32, true);
        JLLM_GLA_COLS(16, true);
    }
    if (wide) JLLM_GLA_COLS(32, false);
    JLLM_GLA_COLS(16, false);
#undef JLLM_GLA_COLS
}

// ---- a prompt portion in chunks of 16 tokens ---------------------------------------------------------------------------
// Within a chunk that starts with the state S0, with L_t the sum of the log-decays of the chunk's tokens up to t (per key
// channel, <= 0) and L the sum over the whole chunk:
//     o_t = (q_t * exp(L_t))^T S0  +  sum over s <= t of a_ts v_s,     a_ts = sum_i q_t[i] k_s[i] exp(L_t[i] - L_s[i])
//     S   = diag(exp(L)) S0 + sum_s (k_s * exp(L - L_s)) v_s^T
// Every exponent is a difference that is <= 0: nothing overflows however strong a decay is. The same multiply-adds as
// token by token (plus the a_ts, a sixteenth more), but as small matrix products whose rows do not wait for one another:
// `prepare` makes q * exp(L_t), k * exp(L - L_s), exp(L) and the a_ts for all chunks of all segments at once (nothing
// there depends on the state), and `chunk` walks a segment's chunks in order, a block per (segment, head, 32 columns of
// S) as in the kernel above. All of it float32; against the token-by-token kernel only the grouping of sums differs.
constexpr int CHUNK = 16;

template <typename T>
__global__ void __launch_bounds__(128)
gla_chunk_prepare_kernel(const T* __restrict__ proj, int ld, int q_off, int k_off, float* __restrict__ logd,
                         const int* __restrict__ seg_start, const int* __restrict__ seg_len, float* __restrict__ qb,
                         float* __restrict__ ke, float* __restrict__ scores, int heads, int dk, float q_scale) {
    extern __shared__ __align__(16) float smem[];
    const int dkp = dk + 1;                 // rows one float apart in the banks: threads of a warp read one column of many rows
    float* L = smem;                        // [CHUNK][dkp]
    float* Q = L + CHUNK * dkp;
    float* K = Q + CHUNK * dkp;
    pdl_wait();
    pdl_trigger();
    const int seg = blockIdx.x, t0 = blockIdx.y * CHUNK, h = blockIdx.z, n = seg_len[seg];
    if (t0 >= n) return;
    const int nt = min(CHUNK, n - t0);
    const size_t row0 = (size_t)seg_start[seg] + t0, hd = (size_t)heads * dk;
    for (int i = threadIdx.x; i < dk; i += blockDim.x) {
        float run = 0.f;
        for (int t = 0; t < nt; ++t) {
            run += logd[(row0 + t) * hd + (size_t)h * dk + i];
            L[t * dkp + i] = run;
            const T* p = proj + (row0 + t) * ld + (size_t)h * dk + i;
            Q[t * dkp + i] = __fmul_rn(to_float(p[q_off]), q_scale);
            K[t * dkp + i] = to_float(p[k_off]);
        }
        for (int t = 0; t < nt; ++t) {
            qb[(row0 + t) * hd + (size_t)h * dk + i] = __fmul_rn(Q[t * dkp + i], expf(L[t * dkp + i]));
            ke[(row0 + t) * hd + (size_t)h * dk + i] = __fmul_rn(K[t * dkp + i], expf(run - L[t * dkp + i]));
        }
        logd[row0 * hd + (size_t)h * dk + i] = expf(run);      // the chunk's whole decay, at its first row
    }
    __syncthreads();
    for (int p = threadIdx.x; p < CHUNK * CHUNK; p += blockDim.x) {
        const int t = p / CHUNK, sx = p - t * CHUNK;
        if (t >= nt) continue;
        float acc = 0.f;
        if (sx <= t)
            for (int i = 0; i < dk; ++i)
                acc = fmaf(__fmul_rn(Q[t * dkp + i], K[sx * dkp + i]), expf(L[t * dkp + i] - L[sx * dkp + i]), acc);
        scores[((row0 + t) * heads + h) * CHUNK + sx] = acc;
    }
}

template <typename T, int R, bool V4>
__global__ void __launch_bounds__(512)
gla_chunk_kernel(const T* __restrict__ proj, int ld, int v_off, const float* __restrict__ chunk_decay,
                 const float* __restrict__ qb, const float* __restrict__ ke, const float* __restrict__ scores,
                 float* __restrict__ state, const int* __restrict__ seg_start, const int* __restrict__ seg_len,
                 const int* __restrict__ state_slots, float* __restrict__ o, int heads, int dk, int dv, int num_slots) {
    extern __shared__ __align__(16) float smem[];
    const int threads = blockDim.x, G = threads >> 5;
    const int stage = 2 * CHUNK * dk + CHUNK * 32 + CHUNK * CHUNK + dk;     // qb, ke [CHUNK][dk], v [CHUNK][32], a, decay [dk]
    float* part = smem + 2 * stage;                                         // [CHUNK][G][32]
    pdl_wait();
    pdl_trigger();
    const int seg = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * 32;
    const int tid = threadIdx.x, c = tid & 31, g = tid >> 5, j = c0 + c;
    const int first = seg_start[seg], n = seg_len[seg], slot = state_slots[seg];
    if (!jllm_in_bounds(slot, num_slots, BOUNDS_SLOT)) return;
    float* S = state + (((size_t)slot * heads + h) * dk) * dv;
    const size_t hd = (size_t)heads * dk;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = g * R + r;
        s[r] = (i < dk && j < dv) ? S[(size_t)i * dv + j] : 0.f;
    }
    constexpr int EPT = CHUNK * R / 32;         // values of qb (and of ke) a thread fetches per chunk: CHUNK x dk / threads
    float fq[EPT], fk[EPT], fv, fa, fd;
    const int vt = tid >> 5, vpt_ok = tid < CHUNK * 32;      // (threads >= 32 x ... : v has CHUNK x 32 values)
    auto fetch = [&](int t0) {
        const int nt = min(CHUNK, n - t0);
        const size_t base = (size_t)(first + t0);
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            const int e = tid + u * threads, t = e / dk, i = e - t * dk;
            fq[u] = fk[u] = 0.f;
            if (e < CHUNK * dk && t < nt) {
                fq[u] = qb[(base + t) * hd + (size_t)h * dk + i];
                fk[u] = ke[(base + t) * hd + (size_t)h * dk + i];
            }
        }
        fv = fa = 0.f;
        fd = 1.f;
        // v: one value a thread where the block has CHUNK x 32 threads or more, else several rounds (below)
        if (vpt_ok && vt < nt && j < dv && threads >= CHUNK * 32)
            fv = to_float(proj[(base + vt) * ld + v_off + (size_t)h * dv + j]);
        if (tid < CHUNK * CHUNK && threads >= CHUNK * CHUNK) {
            const int t = tid / CHUNK;
            if (t < nt) fa = scores[((base + t) * heads + h) * CHUNK + (tid - t * CHUNK)];
        }
        if (tid < dk) fd = chunk_decay[base * hd + (size_t)h * dk + tid];
    };
    auto park = [&](int b, int t0) {
        float* qs = smem + b * stage;
        float* ks = qs + CHUNK * dk;
        float* vs = ks + CHUNK * dk;
        float* as = vs + CHUNK * 32;
        float* dsm = as + CHUNK * CHUNK;
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
            const int e = tid + u * threads;
            if (e < CHUNK * dk) {
                qs[e] = fq[u];
                ks[e] = fk[u];
            }
        }
        if (threads >= CHUNK * 32) {
            if (vpt_ok) vs[tid] = fv;
        } else {        // a small block: it reads its values of v here, late (they are few)
            const int nt = min(CHUNK, n - t0);
            for (int e = tid; e < CHUNK * 32; e += threads) {
                const int t = e >> 5, cc = e & 31;
                vs[e] = (t < nt && c0 + cc < dv) ? to_float(proj[(size_t)(first + t0 + t) * ld + v_off + (size_t)h * dv + c0 + cc]) : 0.f;
            }
        }
        if (threads >= CHUNK * CHUNK) {
            if (tid < CHUNK * CHUNK) as[tid] = fa;
        } else {
            const int nt = min(CHUNK, n - t0);
            for (int e = tid; e < CHUNK * CHUNK; e += threads) {
                const int t = e / CHUNK;
                as[e] = t < nt ? scores[(((size_t)(first + t0 + t)) * heads + h) * CHUNK + (e - t * CHUNK)] : 0.f;
            }
        }
        for (int i = tid; i < dk; i += threads)
            dsm[i] = i == tid ? fd : chunk_decay[(size_t)(first + t0) * hd + (size_t)h * dk + i];
    };
    if (n > 0) {
        fetch(0);
        park(0, 0);
    }
    __syncthreads();
    for (int t0 = 0, b = 0; t0 < n; t0 += CHUNK, b ^= 1) {
        const int nt = min(CHUNK, n - t0);
        const bool more = t0 + CHUNK < n;
        if (more) fetch(t0 + CHUNK);
        const float* qs = smem + b * stage;
        const float* ks = qs + CHUNK * dk;
        const float* vs = ks + CHUNK * dk;
        const float* as = vs + CHUNK * 32;
        const float* dsm = as + CHUNK * CHUNK;
        // what the state at the chunk's start gives every token, and the state at its end
        float acc[CHUNK];
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) acc[t] = 0.f;
        float vreg[CHUNK];
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) vreg[t] = vs[t * 32 + c];
        if constexpr (V4) {     // dk a multiple of 4: four rows' values in one load (shared-memory instructions are what
                                // bounds this loop: an SM issues one a clock)
#pragma unroll
            for (int r = 0; r < R; r += 4) {
                const int i = g * R + r;
                if (i < dk) {
                    const float4 d4 = *reinterpret_cast<const float4*>(dsm + i);
                    const float a0 = s[r], a1 = s[r + 1], a2 = s[r + 2], a3 = s[r + 3];
                    float n0 = __fmul_rn(d4.x, a0), n1 = __fmul_rn(d4.y, a1), n2 = __fmul_rn(d4.z, a2), n3 = __fmul_rn(d4.w, a3);
#pragma unroll
                    for (int t = 0; t < CHUNK; ++t) {
                        const float4 q4 = *reinterpret_cast<const float4*>(qs + t * dk + i);
                        const float4 k4 = *reinterpret_cast<const float4*>(ks + t * dk + i);
                        acc[t] = fmaf(q4.x, a0, acc[t]);
                        acc[t] = fmaf(q4.y, a1, acc[t]);
                        acc[t] = fmaf(q4.z, a2, acc[t]);
                        acc[t] = fmaf(q4.w, a3, acc[t]);
                        n0 = fmaf(k4.x, vreg[t], n0);
                        n1 = fmaf(k4.y, vreg[t], n1);
                        n2 = fmaf(k4.z, vreg[t], n2);
                        n3 = fmaf(k4.w, vreg[t], n3);
                    }
                    s[r] = n0;
                    s[r + 1] = n1;
                    s[r + 2] = n2;
                    s[r + 3] = n3;
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = g * R + r;
                if (i < dk) {
                    const float s0 = s[r];
                    float sn = __fmul_rn(dsm[i], s0);
#pragma unroll
                    for (int t = 0; t < CHUNK; ++t) {
                        acc[t] = fmaf(qs[t * dk + i], s0, acc[t]);
                        sn = fmaf(ks[t * dk + i], vreg[t], sn);
                    }
                    s[r] = sn;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) part[(t * G + g) * 32 + c] = acc[t];
        if (more) park(b ^ 1, t0 + CHUNK);
        __syncthreads();
        for (int e = tid; e < nt * 32; e += threads) {
            const int t = e >> 5, cc = e & 31;
            if (c0 + cc >= dv) continue;
            // four running sums each way: one chain of dependent additions would be all latency (the order is fixed)
            float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
            int gg = 0;
            for (; gg + 4 <= G; gg += 4) {
                p0 += part[(t * G + gg) * 32 + cc];
                p1 += part[(t * G + gg + 1) * 32 + cc];
                p2 += part[(t * G + gg + 2) * 32 + cc];
                p3 += part[(t * G + gg + 3) * 32 + cc];
            }
            for (; gg < G; ++gg) p0 += part[(t * G + gg) * 32 + cc];
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
            int sx = 0;
            for (; sx + 4 <= t + 1; sx += 4) {
                a0 = fmaf(as[t * CHUNK + sx], vs[sx * 32 + cc], a0);
                a1 = fmaf(as[t * CHUNK + sx + 1], vs[(sx + 1) * 32 + cc], a1);
                a2 = fmaf(as[t * CHUNK + sx + 2], vs[(sx + 2) * 32 + cc], a2);
                a3 = fmaf(as[t * CHUNK + sx + 3], vs[(sx + 3) * 32 + cc], a3);
            }
            for (; sx <= t; ++sx) a0 = fmaf(as[t * CHUNK + sx], vs[sx * 32 + cc], a0);
            o[(size_t)(first + t0 + t) * ((size_t)heads * dv) + (size_t)h * dv + c0 + cc] =
                ((p0 + p1) + (p2 + p3)) + ((a0 + a1) + (a2 + a3));
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = g * R + r;
        if (i < dk && j < dv) S[(size_t)i * dv + j] = s[r];
    }
}

template <typename T, int R, bool V4>
int launch_chunked(const void* proj, int ld, int v_off, const float* chunk_decay, const float* qb, const float* ke,
                   const float* scores, float* state, const int* seg_start, const int* seg_len, const int* state_slots,
                   float* o, int segments, int heads, int dk, int dv, int num_slots, cudaStream_t stream) {
    const int G = (dk + R - 1) / R;
    const size_t smem = (size_t)(2 * (2 * CHUNK * dk + CHUNK * 32 + CHUNK * CHUNK + dk) + CHUNK * G * 32) * sizeof(float);
    auto kernel = gla_chunk_kernel<T, R, V4>;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return jllm_fail(JLLM_CUDA_ERROR, "gla_chunk: %zu bytes of shared memory refused", smem);
    jllm_launch(kernel, dim3(segments, heads, (dv + 31) / 32), dim3(G * 32), smem, stream, LAUNCH_DEPENDENT, (const T*)proj, ld,
                v_off, chunk_decay, qb, ke, scores, state, seg_start, seg_len, state_slots, o, heads, dk, dv, num_slots);
    return jllm_check_launch("gla_chunk");
}

// y[r, h, :] = o[r, h, :] / sqrt(mean(o[r, h, :]^2) + eps) * gain * act(gate[r, h, :]) * scale, act = silu or (gate_kind bit 0)
// sigmoid; one warp per (row, head). A norm over all heads together is the case heads = 1. Bit 1 of gate_kind: the gate
// comes first, y = rms(o * act(gate)) * gain * scale (the statistics are those of the gated values). Bit 2: the gain has a
// value per column of the whole row (heads x dv) and not one per column of a head.
template <typename T, typename TG = T>
__global__ void __launch_bounds__(256)
gated_head_norm_kernel(const float* __restrict__ o, const TG* __restrict__ gate, int ld_gate, VecRef gain, T* __restrict__ y,
                       int rows, int heads, int dv, float eps, float scale, int gate_kind) {
    pdl_wait();
    pdl_trigger();
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= rows * heads) return;
    const int r = w / heads, h = w - r * heads;
    const float* src = o + ((size_t)r * heads + h) * dv;
    const TG* gp = gate + (size_t)r * ld_gate + (size_t)h * dv;
    const bool logistic = gate_kind & 1, gate_first = gate_kind & 2;
    const int g0 = (gate_kind & 4) ? h * dv : 0;
    auto gate_of = [&](int i) {
        const float gv = to_float(gp[i]);
        return (logistic ? 1.f : gv) / (1.f + expf(-gv));                          // silu, or (bit 0) the logistic function
    };
    float ss = 0.f;
    for (int i = lane; i < dv; i += 32) {
        const float v = gate_first ? __fmul_rn(src[i], gate_of(i)) : src[i];
        ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    const float inv = 1.f / sqrtf(ss / (float)dv + eps);
    T* dst = y + ((size_t)r * heads + h) * dv;
    for (int i = lane; i < dv; i += 32) {
        const float gated = gate_of(i);
        if (gate_first)
            dst[i] = from_float<T>(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(src[i], gated), inv), gain[g0 + i]), scale));
        else
            dst[i] = from_float<T>(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(src[i], inv), gain[g0 + i]), gated), scale));
    }
}

// The same for many rows of 128, 256, 512 ... values: W warps to a (row, head), a thread's values read once, four at a time, and kept
// in registers. The kernels above and below read everything twice, value by value, and take the gate's exponential twice: launched
// back to back, 1,536 rows x 8 heads of 512 values with a float32 gate 17.1 us there, 11.6 here (63 MB: 9.6 at the memory's
// rate); 2,048 rows of 2,048 with a bfloat16 gate 14.9 and 8.9 (34 MB: 5.1).
__device__ __forceinline__ float4 four_values(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four_values(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store_four(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store_four(__nv_bfloat16* p, const float (&v)[4]) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}

template <typename T, typename TG, int W, int NV>
__global__ void __launch_bounds__(256)
gated_norm_vec_kernel(const float* __restrict__ o, const TG* __restrict__ gate, int ld_gate, VecRef gain, T* __restrict__ y,
                      long long total, int heads, float eps, float scale, int gate_kind) {
    constexpr int DV = W * NV * 128;
    __shared__ float sums[8];
    pdl_wait();
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = warp % W;
    const long long at = (long long)blockIdx.x * (8 / W) + warp / W;           // (row, head)
    const bool live = at < total;
    int r = 0, h = 0;
    if (live) split_item(at, heads, r, h);
    const bool logistic = gate_kind & 1, gate_first = gate_kind & 2;
    const int g0 = (gate_kind & 4) ? h * DV : 0;
    const float* src = o + ((size_t)r * heads + h) * DV;
    const TG* gp = gate + (size_t)r * ld_gate + (size_t)h * DV;
    float v[NV][4], gt[NV][4], ss = 0.f;
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        const int i = ((c * W + sub) * 32 + lane) * 4;
        const float4 x = four_values(src + i), z = four_values(gp + i);
        v[c][0] = x.x, v[c][1] = x.y, v[c][2] = x.z, v[c][3] = x.w;
        gt[c][0] = z.x, gt[c][1] = z.y, gt[c][2] = z.z, gt[c][3] = z.w;
    }
#pragma unroll
    for (int c = 0; c < NV; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            gt[c][e] = (logistic ? 1.f : gt[c][e]) / (1.f + expf(-gt[c][e]));
            if (gate_first) v[c][e] = __fmul_rn(v[c][e], gt[c][e]);
            ss = fmaf(v[c][e], v[c][e], ss);
        }
    ss = warp_sum(ss);
    if constexpr (W > 1) {
        if (lane == 0) sums[warp] = ss;
        __syncthreads();
        ss = 0.f;
#pragma unroll
        for (int w = 0; w < W; ++w) ss += sums[warp / W * W + w];
    }
    if (!live) return;
    const float inv = 1.f / sqrtf(ss / (float)DV + eps);
    T* dst = y + ((size_t)r * heads + h) * DV;
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        const int i = ((c * W + sub) * 32 + lane) * 4;
        float out[4];
        const float4 g4 = gain.four(g0 + i);
        const float gn[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float n = __fmul_rn(__fmul_rn(v[c][e], inv), gn[e]);
            out[e] = __fmul_rn(gate_first ? n : __fmul_rn(n, gt[c][e]), scale);
        }
        store_four(dst + i, out);
    }
}

// launches it where it takes the shape: 1,024 rows x heads and more (fewer leave SMs idle: the kernel below gives a block to each), whole
// pieces of four values. At 1,024 rows x heads, float32 gate, launched back to back, the general kernels and this one: 128 values 2.8 and
// 2.0 us, 256 3.4 and 2.5, 512 4.2 and 3.5, 1,024 5.9 and 4.1, 2,048 9.3 and 5.2, 4,096 15.9 and 8.2, 8,192 37.6 and 20.4; at 4,096
// 512 values 6.9 and 4.9, 2,048 30.2 and 14.6, 8,192 167 and 72.
template <typename T, typename TG>
bool launch_gated_norm_vec(const float* o, const TG* gate, int ld_gate, VecRef gain, T* y, long long total, int heads, int dv, float eps,
                           float scale, int gate_kind, cudaStream_t stream) {
    const size_t gate_piece = 4 * sizeof(TG), out_piece = 4 * sizeof(T);
    if (total < 1024 || ld_gate % 4 != 0 || (uintptr_t)o % 16 || (uintptr_t)gate % gate_piece || (uintptr_t)y % out_piece) return false;
#define JLLM_NORM_VEC(W, NV)                                                                                                  \
    do {                                                                                                                      \
        jllm_launch(gated_norm_vec_kernel<T, TG, W, NV>, dim3((unsigned)((total + 8 / W - 1) / (8 / W))), dim3(256), 0, stream, \
                    LAUNCH_DEPENDENT, o, gate, ld_gate, gain, y, total, heads, eps, scale, gate_kind);                        \
        return true;                                                                                                          \
    } while (0)
    switch (dv) {
        case 128: JLLM_NORM_VEC(1, 1);
        case 256: JLLM_NORM_VEC(1, 2);
        case 512: JLLM_NORM_VEC(1, 4);
        case 1024: JLLM_NORM_VEC(2, 4);
        case 2048: JLLM_NORM_VEC(4, 4);
        case 4096: JLLM_NORM_VEC(8, 4);
        case 8192: JLLM_NORM_VEC(8, 8);
        default: return false;
    }
#undef JLLM_NORM_VEC
}

// The same with a block per (row, head), for norms over many values (all heads of a row together: thousands): a warp
// alone would walk them one after the other.
template <typename T, typename TG = T>
__global__ void __launch_bounds__(256)
gated_row_norm_kernel(const float* __restrict__ o, const TG* __restrict__ gate, int ld_gate, VecRef gain, T* __restrict__ y,
                      int heads, int dv, float eps, float scale, int gate_kind) {
    __shared__ float scratch[33];
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.x / heads, h = blockIdx.x - r * heads;
    const float* src = o + ((size_t)r * heads + h) * dv;
    const TG* gp = gate + (size_t)r * ld_gate + (size_t)h * dv;
    const bool logistic = gate_kind & 1, gate_first = gate_kind & 2;
    const int g0 = (gate_kind & 4) ? h * dv : 0;
    auto gate_of = [&](int i) {
        const float gv = to_float(gp[i]);
        return (logistic ? 1.f : gv) / (1.f + expf(-gv));
    };
    float ss = 0.f;
    for (int i = threadIdx.x; i < dv; i += blockDim.x) {
        const float v = gate_first ? __fmul_rn(src[i], gate_of(i)) : src[i];
        ss = fmaf(v, v, ss);
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.f / sqrtf(ss / (float)dv + eps);
    T* dst = y + ((size_t)r * heads + h) * dv;
    for (int i = threadIdx.x; i < dv; i += blockDim.x) {
        const float gated = gate_of(i);
        if (gate_first)
            dst[i] = from_float<T>(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(src[i], gated), inv), gain[g0 + i]), scale));
        else
            dst[i] = from_float<T>(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(src[i], inv), gain[g0 + i]), gated), scale));
    }
}


// whether the tensor-core form takes this shape (JLLM_B200_LIGHTNING_TC=0 keeps every shape on the float32 kernels)
inline bool chunks_fit(int dtype, int ld, int q_off, int k_off, int v_off, int dk, int dv, const void* proj) {
    static const bool on = [] {
        const char* e = getenv("JLLM_B200_LIGHTNING_TC");
        return !(e && e[0] == '0');
    }();
    return on && dtype == JLLM_BF16 && (dk == 64 || dk == 128) && dv % 8 == 0 && ld % 8 == 0 && q_off % 8 == 0 &&
           k_off % 8 == 0 && v_off % 8 == 0 && ((uintptr_t)proj % 16) == 0;
}

}  // namespace

JLLM_BOUNDS_READER(linear_attention)

// chunk_scan.cu
int jllm_fixed_decay_chunks(const __nv_bfloat16* proj, int ld, int q_off, int k_off, int v_off, const float* head_decay, float* state,
                            int num_slots, const int* seg_start, const int* seg_len, const int* state_slots, float* o, int rows,
                            int segments, int longest, int heads, int dk, int dv, float q_scale, float* workspace,
                            long long workspace_floats, cudaStream_t stream);

// proj [rows, ld]: q at column q_off (heads x dk), k at k_off, v at v_off (heads x dv); z [rows, heads x dk] float32:
// the decay logits, which this call turns into the decays in place; state [num_slots, heads, dk, dv] float32; o [rows,
// heads x dv] float32. Two launches.
JLLM_EXPORT int jllm_gla_recurrent(const void* proj, int dtype, int ld, int q_off, int k_off, int v_off, float* z, int rows,
                                   float* state, int num_slots, const int* seg_start, const int* seg_len,
                                   const int* state_slots, float* o, int segments, int heads, int dk, int dv, float q_scale,
                                   float tau, const float* head_decay, int activation, cudaStream_t stream) {
    JLLM_REQUIRE(segments >= 0 && rows >= 0 && heads > 0 && dk > 0 && dv > 0 && tau > 0.f,
                 "gla_recurrent: segments=%d heads=%d dk=%d dv=%d", segments, heads, dk, dv);
    JLLM_REQUIRE(dk <= 512 && heads <= 65535 && (dv + 7) / 8 <= 65535, "gla_recurrent: dk=%d is above 512", dk);
    if (segments == 0 || rows == 0) return JLLM_OK;
    const float inv_tau = 1.f / tau;
    if (head_decay) {
        // one fixed decay per head: the recurrence takes the decays themselves and activates q, k, v as it fetches them (no
        // table, no pass in front; `proj` is left as it is)
    } else {       // the decay logits become decays, in place
        const size_t total = (size_t)rows * heads * dk;
        const int blocks = (int)min((size_t)65535, (total + 255) / 256);
        jllm_launch(gla_decay_kernel, dim3(blocks), dim3(256), 0, stream, LAUNCH_DEPENDENT, z, inv_tau, total, 0);
        const int code = jllm_check_launch("gla_decay");
        if (code) return code;
    }
#define JLLM_GLA(T, R)                                                                                                       \
    return launch_recurrent_cols<T, R>(proj, ld, q_off, k_off, v_off, z, state, seg_start, seg_len, state_slots, o, segments, \
                                       heads, dk, dv, q_scale, num_slots, head_decay, head_decay ? activation : 0, stream)
    // A step of single tokens is a chain of a few round trips to memory per block, whatever the block's size: many rows a
    // thread make blocks small enough for several to share an SM. A prompt portion waits more than it computes: few rows
    // a thread, so that more threads hide more of the waiting (at most 32 row groups of 32 columns: 1,024 threads).
    // (Only the grouping of the partial sums of o differs between the two.)
    const bool single = rows == segments;
    if (dtype == JLLM_F32) {
        if (single) JLLM_GLA(float, 16);
        if (dk <= 128) JLLM_GLA(float, 4);
        if (dk <= 256) JLLM_GLA(float, 8);
        JLLM_GLA(float, 16);
    }
    if (single) JLLM_GLA(__nv_bfloat16, 16);
    if (dk <= 128) JLLM_GLA(__nv_bfloat16, 4);
    if (dk <= 256) JLLM_GLA(__nv_bfloat16, 8);
    JLLM_GLA(__nv_bfloat16, 16);
#undef JLLM_GLA
}

// Whether a step with prompt portions goes through the tensor-core chunks (jllm_gla_chunked then wants their workspace)
JLLM_EXPORT int jllm_gla_chunks_fit(const void* proj, int dtype, int ld, int q_off, int k_off, int v_off, int dk, int dv) {
    return chunks_fit(dtype, ld, q_off, k_off, v_off, dk, dv, proj);
}

// The same recurrence for steps with prompt portions, in chunks of 16 tokens (three launches: the log-decays in place
// of z, the chunks' operands, the walk through the chunks). qb, ke [rows, heads x dk] and scores [rows, heads x 16] are
// float32 scratch; `max_len`: the longest segment's rows.
JLLM_EXPORT int jllm_gla_chunked(const void* proj, int dtype, int ld, int q_off, int k_off, int v_off, float* z, int rows,
                                 float* qb, float* ke, float* scores, float* state, int num_slots, const int* seg_start,
                                 const int* seg_len, const int* state_slots, float* o, int segments, int max_len, int heads,
                                 int dk, int dv, float q_scale, float tau, const float* head_decay, int activation,
                                 float* workspace, long long workspace_floats, cudaStream_t stream) {
    JLLM_REQUIRE(segments >= 0 && rows >= 0 && heads > 0 && dk > 0 && dv > 0 && tau > 0.f && max_len >= 0,
                 "gla_chunked: segments=%d heads=%d dk=%d dv=%d", segments, heads, dk, dv);
    JLLM_REQUIRE(dk <= 512 && heads <= 65535 && (dv + 31) / 32 <= 65535 && (max_len + CHUNK - 1) / CHUNK <= 65535,
                 "gla_chunked: dk=%d is above 512, or a segment of %d rows is too long", dk, max_len);
    if (segments == 0 || rows == 0 || max_len == 0) return JLLM_OK;
    if (head_decay && chunks_fit(dtype, ld, q_off, k_off, v_off, dk, dv, proj)) {
        // one decay per head, bfloat16 projections, key heads of 64 or 128: all chunks of 64 tokens at once on the tensor cores
        if (activation) {
            const int code = launch_fixed_decay<__nv_bfloat16>((void*)proj, ld, q_off, k_off, v_off, nullptr, head_decay, rows,
                                                               heads, dk, dv, 1, activation, stream);
            if (code) return code;
        }
        return jllm_fixed_decay_chunks((const __nv_bfloat16*)proj, ld, q_off, k_off, v_off, head_decay, state, num_slots, seg_start,
                                       seg_len, state_slots, o, rows, segments, max_len, heads, dk, dv, q_scale, workspace,
                                       workspace_floats, stream);
    }
    if (head_decay) {
        const int code = dtype == JLLM_F32
            ? launch_fixed_decay<float>((void*)proj, ld, q_off, k_off, v_off, z, head_decay, rows, heads, dk, dv, 1, activation, stream)
            : launch_fixed_decay<__nv_bfloat16>((void*)proj, ld, q_off, k_off, v_off, z, head_decay, rows, heads, dk, dv, 1, activation, stream);
        if (code) return code;
    } else {
        const size_t total = (size_t)rows * heads * dk;
        const int blocks = (int)min((size_t)65535, (total + 255) / 256);
        jllm_launch(gla_decay_kernel, dim3(blocks), dim3(256), 0, stream, LAUNCH_DEPENDENT, z, 1.f / tau, total, 1);
        const int code = jllm_check_launch("gla_decay");
        if (code) return code;
    }
    {
        const size_t smem = (size_t)3 * CHUNK * (dk + 1) * sizeof(float);
        const dim3 grid(segments, (max_len + CHUNK - 1) / CHUNK, heads);
        if (dtype == JLLM_F32) {
            if (smem > 48 * 1024) cudaFuncSetAttribute(gla_chunk_prepare_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            jllm_launch(gla_chunk_prepare_kernel<float>, grid, dim3(128), smem, stream, LAUNCH_DEPENDENT, (const float*)proj, ld,
                        q_off, k_off, z, seg_start, seg_len, qb, ke, scores, heads, dk, q_scale);
        } else {
            if (smem > 48 * 1024) cudaFuncSetAttribute(gla_chunk_prepare_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            jllm_launch(gla_chunk_prepare_kernel<__nv_bfloat16>, grid, dim3(128), smem, stream, LAUNCH_DEPENDENT,
                        (const __nv_bfloat16*)proj, ld, q_off, k_off, z, seg_start, seg_len, qb, ke, scores, heads, dk, q_scale);
        }
        const int code = jllm_check_launch("gla_chunk_prepare");
        if (code) return code;
    }
#define JLLM_GLA_CHUNK(T, R)                                                                                                  \
    return dk % 4 == 0 ? launch_chunked<T, R, true>(proj, ld, v_off, z, qb, ke, scores, state, seg_start, seg_len, state_slots, \
                                                    o, segments, heads, dk, dv, num_slots, stream)                           \
                       : launch_chunked<T, R, false>(proj, ld, v_off, z, qb, ke, scores, state, seg_start, seg_len,            \
                                                     state_slots, o, segments, heads, dk, dv, num_slots, stream)
    if (dtype == JLLM_F32) {
        if (dk <= 32) JLLM_GLA_CHUNK(float, 4);
        if (dk <= 128) JLLM_GLA_CHUNK(float, 8);
        if (dk <= 256) JLLM_GLA_CHUNK(float, 16);
        JLLM_GLA_CHUNK(float, 32);
    }
    if (dk <= 32) JLLM_GLA_CHUNK(__nv_bfloat16, 4);
    if (dk <= 128) JLLM_GLA_CHUNK(__nv_bfloat16, 8);
    if (dk <= 256) JLLM_GLA_CHUNK(__nv_bfloat16, 16);
    JLLM_GLA_CHUNK(__nv_bfloat16, 32);
#undef JLLM_GLA_CHUNK
}

JLLM_EXPORT int jllm_gated_head_norm(const float* o, const void* gate, int dtype, int ld_gate, const void* gain,
                                     int gain_dtype, void* y, int rows, int heads, int dv, float eps, float scale,
                                     int gate_kind, int gate_dtype, cudaStream_t stream) {
    // `dtype`: the type of y; `gate_dtype`: the gate's (the same, or float32 beside a bfloat16 y: a gate that a product left
    // in float32)
    JLLM_REQUIRE(rows >= 0 && heads > 0 && dv > 0, "gated_head_norm: rows=%d heads=%d dv=%d", rows, heads, dv);
    JLLM_REQUIRE(gate_dtype == dtype || gate_dtype == JLLM_F32, "gated_head_norm: a gate of type %d beside a result of type %d",
                 gate_dtype, dtype);
    if (rows == 0) return JLLM_OK;
    const VecRef g{gain, gain_dtype};
    const long long warps = (long long)rows * heads;
    const bool wide_gate = gate_dtype != dtype;
    if (warps <= 2147483647ll &&
        (dtype == JLLM_F32 ? launch_gated_norm_vec(o, (const float*)gate, ld_gate, g, (float*)y, warps, heads, dv, eps, scale, gate_kind, stream)
         : wide_gate ? launch_gated_norm_vec(o, (const float*)gate, ld_gate, g, (__nv_bfloat16*)y, warps, heads, dv, eps, scale, gate_kind, stream)
                     : launch_gated_norm_vec(o, (const __nv_bfloat16*)gate, ld_gate, g, (__nv_bfloat16*)y, warps, heads, dv, eps, scale,
                                             gate_kind, stream)))
        return jllm_check_launch("gated_head_norm");
    // long norms: a block each; also norms of 256 values and more where a step has so few of them that a warp each would
    // leave the device idle (a step of single rows)
    if ((dv > 512 || (dv >= 256 && warps <= 2048)) && warps <= 2147483647ll) {
        if (dtype == JLLM_F32)
            jllm_launch(gated_row_norm_kernel<float>, dim3((unsigned)warps), dim3(256), 0, stream, LAUNCH_DEPENDENT, o,
                        (const float*)gate, ld_gate, g, (float*)y, heads, dv, eps, scale, gate_kind);
        else if (wide_gate)
            jllm_launch(gated_row_norm_kernel<__nv_bfloat16, float>, dim3((unsigned)warps), dim3(256), 0, stream, LAUNCH_DEPENDENT, o,
                        (const float*)gate, ld_gate, g, (__nv_bfloat16*)y, heads, dv, eps, scale, gate_kind);
        else
            jllm_launch(gated_row_norm_kernel<__nv_bfloat16>, dim3((unsigned)warps), dim3(256), 0, stream, LAUNCH_DEPENDENT, o,
                        (const __nv_bfloat16*)gate, ld_gate, g, (__nv_bfloat16*)y, heads, dv, eps, scale, gate_kind);
        return jllm_check_launch("gated_head_norm");
    }
    const dim3 grid((unsigned)((warps + 7) / 8));
    if (dtype == JLLM_F32)
        jllm_launch(gated_head_norm_kernel<float>, grid, dim3(256), 0, stream, LAUNCH_DEPENDENT, o, (const float*)gate,
                    ld_gate, g, (float*)y, rows, heads, dv, eps, scale, gate_kind);
    else if (wide_gate)
        jllm_launch(gated_head_norm_kernel<__nv_bfloat16, float>, grid, dim3(256), 0, stream, LAUNCH_DEPENDENT, o,
                    (const float*)gate, ld_gate, g, (__nv_bfloat16*)y, rows, heads, dv, eps, scale, gate_kind);
    else
        jllm_launch(gated_head_norm_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, LAUNCH_DEPENDENT, o,
                    (const __nv_bfloat16*)gate, ld_gate, g, (__nv_bfloat16*)y, rows, heads, dv, eps, scale, gate_kind);
    return jllm_check_launch("gated_head_norm");
}

// Linear recurrences of prompt portions in chunks of 64 tokens, all chunks at once, on the tensor cores.
//
// The recurrence S_t = a_t S_(t-1) + (b_t k_t) v_t^T, o_t = S_t^T (s q_t) [+ D v_t] has one decay a and one input scale b per
// token and head (a selective state space, a matrix memory) or one decay per head (FIXED: "lightning" attention, b = 1). With cl_t
// the sum of log a over a chunk's tokens up to t, a chunk is
//     P[t, s] = (q_t . k_s) s exp(cl_t - cl_s) b_s  for s <= t       o_t = sum_s P[t, s] v_s + exp(cl_t) s (q_t^T S0) [+ D v_t]
//     S       = exp(cl_n) S0 + sum_s k_s (b_s exp(cl_n - cl_s) v_s)^T
// Every exponent is a difference that is <= 0. Only the state walks from chunk to chunk, so three launches do the work:
//     chunk_states   every chunk's own sum_s k_s (w_s v_s)^T                      (a block per chunk and some heads)
//     chunk_scan     the states in front of every chunk, element by element       (a thread per four state values)
//     chunk_out      every chunk's o from its q, k, v and the state in front      (a block per chunk and some heads)
// Short segments have no chunks to run beside one another: a fourth kernel, chunk_walk, takes theirs one after the other.
// An item is a head and a slab of 32 or 64 of its value columns. Heads whose q and k are the same (a group) share the chunk's q, k
// and their product q k^T, which a warp keeps in registers. q, k and v are projections and enter as bfloat16 operands (float32 sources are rounded on their way
// into shared memory); the float32 factors meet float32 values (the scores behind their product, the values in front of theirs,
// the state as it was summed) and what has to become an operand then becomes two, the bfloat16 value and the bfloat16 of what that
// rounding left: 16 bits of mantissa, summed in float32.
// The states travel in the layout of the tensor cores' fragments: the accumulators of the transposed product (value columns down,
// key channels across) hold exactly what a thread of chunk_out needs of S0 as a B operand, so chunk_states stores float4, chunk_scan
// turns each into two pairs of operands in place, and chunk_out loads 16 bytes a thread and tile straight into mma.sync.
//
// What bounds it: the states' way through L2 (written, read, written, read: 16 bytes per state value and chunk) and, per chunk and
// head, mma.sync with its fragments. It took the place of kernels that gave a block to (request, head, value columns) and walked
// its chunks one after the other (state in registers, weighted keys transposed by two-byte stores, a 32-byte piece of another row per
// lane). 1,536 tokens of 2 requests, 64 heads with states of 128 x 64 in groups of 8: 230 us there, 94 here (33 + 19 + 52 by
// themselves); 8 heads of 128 x 264: 112 and 60; 2,048 tokens, 16 heads of 128 x 128, one decay per head: 148 and 53.
// It is mma.sync, not tcgen05: the products are 64 tokens high, the scores and the states are float32 values that become
// operands by an elementwise step, and registers are where that step happens.
#include <climits>

#include "common.cuh"

namespace {

constexpr int C = 64;            // tokens of a chunk

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Four 8 x 8 matrices of bfloat16 from shared memory into a warp's fragments: lane l names row l & 7 of matrix l >> 3
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
// A fragment: rows row0.. of a row-major operand, contraction values k0..
__device__ __forceinline__ void load_a(uint32_t (&a)[4], const __nv_bfloat16* m, int ld, int row0, int k0, int lane) {
    ldmatrix4(a, m + (row0 + (lane & 7) + ((lane >> 3) & 1) * 8) * ld + k0 + (lane >> 4) * 8);
}
// A fragment of the transpose of an operand stored [contraction][rows]
__device__ __forceinline__ void load_a_trans(uint32_t (&a)[4], const __nv_bfloat16* m, int ld, int row0, int k0, int lane) {
    ldmatrix4_trans(a, m + (k0 + (lane & 7) + (lane >> 4) * 8) * ld + row0 + ((lane >> 3) & 1) * 8);
}
// B fragments of two neighbouring 8-wide tiles of an operand stored [columns][contraction]
__device__ __forceinline__ void load_b2(uint32_t (&b)[4], const __nv_bfloat16* m, int ld, int n0, int k0, int lane) {
    ldmatrix4(b, m + (n0 + (lane & 7) + (lane >> 4) * 8) * ld + k0 + ((lane >> 3) & 1) * 8);
}
// ... of one stored [contraction][columns]
__device__ __forceinline__ void load_b2_trans(uint32_t (&b)[4], const __nv_bfloat16* m, int ld, int n0, int k0, int lane) {
    ldmatrix4_trans(b, m + (k0 + (lane & 7) + ((lane >> 3) & 1) * 8) * ld + n0 + (lane >> 4) * 8);
}

__device__ __forceinline__ uint32_t pack(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
// (a, b) as two operands: their bfloat16 values, and the bfloat16 of what that rounding left
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    hi = pack(a, b);
    const float2 h = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi));
    lo = pack(a - h.x, b - h.y);
}
// eight values as bfloat16
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ uint4 load8(const float* p) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    return make_uint4(pack(a.x, a.y), pack(a.z, a.w), pack(b.x, b.y), pack(b.z, b.w));
}
__device__ __forceinline__ void cp_async_16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

struct ChunkArgs {
    const void *q, *k, *v;
    int ld_q, q_off, ld_k, k_off, ld_v, v_off;
    int groups, per_group;              // heads of a group (per_group) share q and k; head h reads q at q_off + (h / q_share) DK
    int q_share, k_share;
    const float *la, *b, *decay;        // per token and head, or (FIXED) per head
    VecRef skip;
    int has_skip;
    float* state;
    const int *seg_start, *seg_len, *state_slots;
    float* o;
    int segments, heads, dv, num_slots;
    float q_scale;
    float4* ws;                         // the chunks' states: [chunk][head of the pass][slab][DK / 16][SLAB / 8][32]
    float* ends;                        // [chunk][head of the pass]: exp(cl_n)
    int chunks;                         // room for so many chunks
    int walked;                         // segments of so many chunks and fewer are left to chunk_walk (0: none)
    int group0, pass_heads;             // this pass covers the heads from group0 * per_group on
    int slabs, items;                   // slabs of a head; items a block takes
};

// the chunks of a segment; those that the three launches take care of
__device__ __forceinline__ int all_chunks(const ChunkArgs& a, int seg) { return (a.seg_len[seg] + C - 1) / C; }
__device__ __forceinline__ int scanned_chunks(const ChunkArgs& a, int seg) {
    const int n = all_chunks(a, seg);
    return n <= a.walked ? 0 : n;
}
// which chunk of which segment a block has; false past the last
__device__ __forceinline__ bool find_chunk(const ChunkArgs& a, int chunk, int& seg, int& t0) {
    for (seg = 0; seg < a.segments; ++seg) {
        const int n = scanned_chunks(a, seg);
        if (chunk < n) { t0 = chunk * C; return true; }
        chunk -= n;
    }
    return false;
}

// `rows` (64) rows of DK values into shared memory, zeros from row nt on
template <typename TS, int DK>
__device__ __forceinline__ void load_rows(__nv_bfloat16* dst, const TS* src, int ld, int nt, int rows = C) {
#pragma unroll 4
    for (int e = threadIdx.x; e < rows * (DK / 8); e += 256) {
        const int row = e / (DK / 8), piece = e % (DK / 8);
        *reinterpret_cast<uint4*>(dst + row * (DK + 8) + piece * 8) =
            row < nt ? load8(src + (size_t)row * ld + piece * 8) : make_uint4(0, 0, 0, 0);
    }
}

// The same by way of registers: fetched while the rows before are still read
template <typename TS, int DK>
struct Rows {
    static constexpr int N = C * (DK / 8) / 256;
    uint4 piece[N];
    __device__ __forceinline__ void fetch(const TS* src, int ld, int nt) {
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int e = threadIdx.x + u * 256, row = e / (DK / 8);
            piece[u] = row < nt ? load8(src + (size_t)row * ld + e % (DK / 8) * 8) : make_uint4(0, 0, 0, 0);
        }
    }
    __device__ __forceinline__ void put(__nv_bfloat16* dst) const {
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int e = threadIdx.x + u * 256;
            *reinterpret_cast<uint4*>(dst + e / (DK / 8) * (DK + 8) + e % (DK / 8) * 8) = piece[u];
        }
    }
};

// An item's gates: cl [C] and bs [C] (not FIXED; zeros of bs past the chunk's end), or pw [C + 1] = d^0 .. d^C (FIXED, in the same
// place). They are fetched an item ahead (`fetch`: the first warp, a lane two neighbouring tokens) and put in place by that warp.
template <bool FIXED>
struct Gates {
    float l0, l1, b0, b1;
    __device__ __forceinline__ void fetch(const ChunkArgs& a, int row0, int nt, int h) {
        if (threadIdx.x >= 32) return;
        if constexpr (FIXED) {
            l0 = a.decay[h];
        } else {
            const int t = 2 * threadIdx.x;
            const size_t at = (size_t)(row0 + t) * a.heads + h;
            l0 = t < nt ? a.la[at] : 0.f, b0 = t < nt ? a.b[at] : 0.f;
            l1 = t + 1 < nt ? a.la[at + a.heads] : 0.f, b1 = t + 1 < nt ? a.b[at + a.heads] : 0.f;
        }
    }
    __device__ __forceinline__ void put(float* cl, float* bs) const {
        if (threadIdx.x >= 32) return;
        const int lane = threadIdx.x;
        if constexpr (FIXED) {
            const float l = fmaxf(logf(l0), -1e30f);                    // (a decay of 0: d^0 = 1, every other power 0)
            for (int i = lane; i <= C; i += 32) cl[i] = expf((float)i * l);
        } else {
            float v = l0 + l1;                                          // the pairs' sums, added up over the lanes
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d) v += up;
            }
            float before = __shfl_up_sync(0xffffffffu, v, 1);
            if (lane == 0) before = 0.f;
            cl[2 * lane] = before + l0, cl[2 * lane + 1] = v;
            bs[2 * lane] = b0, bs[2 * lane + 1] = b1;
        }
    }
};
// A thread's pieces of an item's values [C][SLAB], as bfloat16 (zeros past the chunk's end and the head's columns)
template <typename TS, int SLAB>
struct Values {
    static constexpr int N = C * (SLAB / 8) / 256;
    uint4 piece[N];
    __device__ __forceinline__ static int row(int u) { return (threadIdx.x + u * 256) / (SLAB / 8); }
    __device__ __forceinline__ static int col(int u) { return (threadIdx.x + u * 256) % (SLAB / 8) * 8; }
    __device__ __forceinline__ void fetch(const ChunkArgs& a, int row0, int nt, int h, int c0) {
#pragma unroll
        for (int u = 0; u < N; ++u)
            piece[u] = row(u) < nt && c0 + col(u) < a.dv
                           ? load8(static_cast<const TS*>(a.v) + (size_t)(row0 + row(u)) * a.ld_v + a.v_off + (size_t)h * a.dv + c0 + col(u))
                           : make_uint4(0, 0, 0, 0);
    }
};

// item i of a block: the head (counted from the pass's first) and its slab
struct Item { int head, slab; };
__device__ __forceinline__ Item item_of(const ChunkArgs& a, int group, int i) {
    return {group * a.per_group + i / a.slabs, i % a.slabs};
}

constexpr int GATES = 2 * C + 8;        // floats of an item's gates

// An item's values times their weights towards the chunk's end, as two operands [C][LDV]
template <typename TS, int SLAB, bool FIXED>
__device__ __forceinline__ void weigh(const Values<TS, SLAB>& v, __nv_bfloat16* Vh, __nv_bfloat16* Vl, const float* cl, const float* bs,
                                      int nt) {
    constexpr int LDV = SLAB + 8;
#pragma unroll
    for (int u = 0; u < v.N; ++u) {
        const int row = v.row(u);
        const float w = row >= nt ? 0.f : FIXED ? cl[nt - 1 - row] : __fmul_rn(bs[row], expf(cl[nt - 1] - cl[row]));
        const uint32_t in[4] = {v.piece[u].x, v.piece[u].y, v.piece[u].z, v.piece[u].w};
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&in[x]));
            split2(f.x * w, f.y * w, hi[x], lo[x]);
        }
        *reinterpret_cast<uint4*>(Vh + row * LDV + v.col(u)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(Vl + row * LDV + v.col(u)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}
// ... and U^T [value columns x key channels] = (w v)^T k over the chunk's first `rows` tokens: 16 value columns from mt * 16 on, NT
// tiles of channels from tile part * NT on
template <int DK, int SLAB, int NT>
__device__ __forceinline__ void own_state(float (&acc)[NT][4], const __nv_bfloat16* Vh, const __nv_bfloat16* Vl, const __nv_bfloat16* Ks,
                                          int mt, int part, int lane, int rows = C) {
    constexpr int LDK = DK + 8, LDV = SLAB + 8;
#pragma unroll
    for (int k0 = 0; k0 < C; k0 += 16)
        if (k0 < rows) {
            uint32_t ah[4], al[4];
            load_a_trans(ah, Vh, LDV, mt * 16, k0, lane);
            load_a_trans(al, Vl, LDV, mt * 16, k0, lane);
#pragma unroll
            for (int j = 0; j < NT; j += 2) {
                uint32_t b[4];
                load_b2_trans(b, Ks, LDK, (part * NT + j) * 8, k0, lane);
                mma_bf16(acc[j], ah, b[0], b[1]);
                mma_bf16(acc[j + 1], ah, b[2], b[3]);
                mma_bf16(acc[j], al, b[0], b[1]);
                mma_bf16(acc[j + 1], al, b[2], b[3]);
            }
        }
}

// q k^T of 16 tokens (from mt * 16 on) and the keys up to the last of them
template <int DK>
__device__ __forceinline__ void own_scores(float (&qk)[8][4], const __nv_bfloat16* Qs, const __nv_bfloat16* Ks, int mt, int lane) {
    constexpr int LDK = DK + 8;
#pragma unroll 1
    for (int k0 = 0; k0 < DK; k0 += 16) {
        uint32_t q[4];
        load_a(q, Qs, LDK, mt * 16, k0, lane);
#pragma unroll
        for (int j = 0; j < 8; j += 2)
            if (j <= 2 * mt) {
                uint32_t b[4];
                load_b2(b, Ks, LDK, j * 8, k0, lane);
                mma_bf16(qk[j], q, b[0], b[1]);
                mma_bf16(qk[j + 1], q, b[2], b[3]);
            }
    }
}
// acc = q^T S0 of those tokens and the first `live` of NT tiles of value columns; `s0`: the lane's operands of the first
template <int DK, int NT>
__device__ __forceinline__ void from_state(float (&acc)[NT][4], const __nv_bfloat16* Qs, const uint4* s0, int live, int mt, int lane) {
    constexpr int LDK = DK + 8;
#pragma unroll 2
    for (int kt = 0; kt < DK / 16; ++kt) {
        uint32_t q[4];
        load_a(q, Qs, LDK, mt * 16, kt * 16, lane);
#pragma unroll
        for (int j = 0; j < NT; ++j)
            if (j < live) {
                const uint4 x = s0[(kt * 2 * NT + j) * 32];
                mma_bf16(acc[j], q, x.x, x.y);
                mma_bf16(acc[j], q, x.z, x.w);
            }
    }
}
// o = exp(cl_t) s acc + P v [+ D v]; `c0`: the first of the warp's value columns, `at`: its place in the slab, dst0: o of row 0
template <int SLAB, bool FIXED, int NT>
__device__ __forceinline__ void finish(const ChunkArgs& a, float (&acc)[NT][4], const float (&qk)[8][4], const __nv_bfloat16* Vs,
                                       const float* cl, const float* bs, int h, int c0, int at, int live, int row0, int nt, int mt, int lane) {
    constexpr int LDV = SLAB + 8;
    const int g = lane >> 2, t = lane & 3, tok0 = mt * 16 + g;
    const size_t row_o = (size_t)a.heads * a.dv;
    const float f0 = __fmul_rn(FIXED ? cl[tok0 + 1] : expf(cl[tok0]), a.q_scale);
    const float f1 = __fmul_rn(FIXED ? cl[tok0 + 9] : expf(cl[tok0 + 8]), a.q_scale);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        acc[j][0] = __fmul_rn(acc[j][0], f0), acc[j][1] = __fmul_rn(acc[j][1], f0);
        acc[j][2] = __fmul_rn(acc[j][2], f1), acc[j][3] = __fmul_rn(acc[j][3], f1);
    }
    // the accumulators of q k^T, weighted, are the A operand as they lie
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
        if (kk <= mt) {
            uint32_t ph[4], pl[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {                     // rows g, g + 8; keys 2t and 2t + 8 of the sixteen
                const int j = 2 * kk + (x >> 1), tok = tok0 + (x & 1) * 8, key = j * 8 + 2 * t;
                float w0, w1;
                if constexpr (FIXED) {
                    w0 = cl[max(tok - key, 0)], w1 = cl[max(tok - key - 1, 0)];
                } else {
                    const float ct = cl[tok];
                    w0 = __fmul_rn(expf(ct - cl[key]), bs[key]), w1 = __fmul_rn(expf(ct - cl[key + 1]), bs[key + 1]);
                }
                const float p0 = key <= tok ? __fmul_rn(__fmul_rn(qk[j][2 * (x & 1)], a.q_scale), w0) : 0.f;
                const float p1 = key + 1 <= tok ? __fmul_rn(__fmul_rn(qk[j][2 * (x & 1) + 1], a.q_scale), w1) : 0.f;
                split2(p0, p1, ph[x], pl[x]);
            }
#pragma unroll
            for (int j = 0; j < NT; j += 2) {
                uint32_t b[4];
                load_b2_trans(b, Vs, LDV, at + j * 8, kk * 16, lane);
                mma_bf16(acc[j], ph, b[0], b[1]);
                mma_bf16(acc[j + 1], ph, b[2], b[3]);
                mma_bf16(acc[j], pl, b[0], b[1]);
                mma_bf16(acc[j + 1], pl, b[2], b[3]);
            }
        }
    const float d_skip = a.has_skip ? a.skip[h] : 0.f;
#pragma unroll
    for (int below = 0; below < 2; ++below) {
        const int tok = tok0 + below * 8;
        if (tok < nt) {
            float* dst = a.o + (size_t)(row0 + tok) * row_o + (size_t)h * a.dv + c0 + 2 * t;
#pragma unroll
            for (int j = 0; j < NT; ++j)
                if (j < live) {
                    float2 r = make_float2(acc[j][2 * below], acc[j][2 * below + 1]);
                    if (a.has_skip) {
                        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Vs + tok * LDV + at + j * 8 + 2 * t));
                        r.x = fmaf(d_skip, x.x, r.x), r.y = fmaf(d_skip, x.y, r.y);
                    }
                    *reinterpret_cast<float2*>(dst + j * 8) = r;
                }
        }
    }
}

// ---- every chunk's own part of the state: U^T [value columns x key channels] = (w v)^T k ----
template <typename TS, int DK, int SLAB, bool FIXED>
__global__ void __launch_bounds__(256, 2) chunk_states_kernel(const __grid_constant__ ChunkArgs a) {
    constexpr int LDK = DK + 8, LDV = SLAB + 8;
    constexpr int MT = SLAB / 16, PARTS = 8 / MT, NT = DK / 8 / PARTS;      // 16-column tiles; warps that share one; their channel tiles
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(chunk_smem);       // [C][LDK]
    __nv_bfloat16* Vh = Ks + C * LDK;                                       // [C][LDV]: w v
    __nv_bfloat16* Vl = Vh + C * LDV;                                       //           ... and what its rounding left
    float* cl = reinterpret_cast<float*>(Vl + C * LDV);
    float* bs = cl + C;
    pdl_wait();
    pdl_trigger();
    int seg, t0;
    if (!find_chunk(a, blockIdx.x, seg, t0)) return;
    if (!jllm_in_bounds(a.state_slots[seg], a.num_slots, BOUNDS_SLOT)) return;
    const int blocks_per_group = (a.per_group * a.slabs + a.items - 1) / a.items;
    const int group = blockIdx.y / blocks_per_group, i0 = blockIdx.y % blocks_per_group * a.items;
    const int i_end = min(i0 + a.items, a.per_group * a.slabs);
    const int row0 = a.seg_start[seg] + t0, nt = min(C, a.seg_len[seg] - t0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h0 = a.group0 * a.per_group;
    Values<TS, SLAB> v;
    Gates<FIXED> gates;
    auto fetch = [&](int i) {
        const Item it = item_of(a, group, i);
        v.fetch(a, row0, nt, h0 + it.head, it.slab * SLAB);
        gates.fetch(a, row0, nt, h0 + it.head);
    };
    fetch(i0);
    load_rows<TS, DK>(Ks, static_cast<const TS*>(a.k) + (size_t)row0 * a.ld_k + a.k_off +
                              (size_t)((h0 + group * a.per_group) / a.k_share) * DK, a.ld_k, nt);
    const int mt = warp % MT, part = warp / MT;
    for (int i = i0; i < i_end; ++i) {
        const Item it = item_of(a, group, i);
        const int c0 = it.slab * SLAB;
        gates.put(cl, bs);
        __syncthreads();
        weigh<TS, SLAB, FIXED>(v, Vh, Vl, cl, bs, nt);
        const size_t place = (size_t)blockIdx.x * a.pass_heads + it.head;
        if (it.slab == 0 && threadIdx.x == 0) a.ends[place] = FIXED ? cl[nt] : expf(cl[nt - 1]);
        if (i + 1 < i_end) fetch(i + 1);
        __syncthreads();
        if (c0 + mt * 16 < a.dv) {
            float acc[NT][4] = {};
            own_state<DK, SLAB, NT>(acc, Vh, Vl, Ks, mt, part, lane);
            float4* dst = a.ws + ((place * a.slabs + it.slab) * (DK / 16) + part * (NT / 2)) * (SLAB / 8) * 32 + mt * 64 + lane;
#pragma unroll
            for (int j = 0; j < NT; j += 2) {
                float4* d = dst + (j / 2) * (SLAB / 8) * 32;
                d[0] = make_float4(acc[j][0], acc[j][1], acc[j + 1][0], acc[j + 1][1]);
                d[32] = make_float4(acc[j][2], acc[j][3], acc[j + 1][2], acc[j + 1][3]);
            }
        }
    }
}

// ---- the state in front of every chunk, as operands, in place of the chunk's own part ----
template <int DK, int SLAB>
__global__ void __launch_bounds__(256) chunk_scan_kernel(const __grid_constant__ ChunkArgs a) {
    constexpr int AHEAD = 4;
    pdl_wait();
    pdl_trigger();
    const int seg = blockIdx.y, per_head = a.slabs * (DK / 16) * (SLAB / 8) * 32;
    const int n = scanned_chunks(a, seg), slot = a.state_slots[seg];
    if (n == 0 || !jllm_in_bounds(slot, a.num_slots, BOUNDS_SLOT)) return;
    const long long e = (long long)blockIdx.x * 256 + threadIdx.x;
    if (e >= (long long)a.pass_heads * per_head) return;
    const int head = (int)(e / per_head), lane = (int)(e & 31), tile = (int)(e % per_head) / 32;
    const int nt = tile % (SLAB / 8), kt = tile / (SLAB / 8) % (DK / 16), slab = tile / (SLAB / 8) / (DK / 16);
    const int col = slab * SLAB + nt * 8 + (lane >> 2), ch = kt * 16 + 2 * (lane & 3);
    if (slab * SLAB + nt * 8 >= a.dv) return;
    int first = 0;
    for (int s = 0; s < seg; ++s) first += scanned_chunks(a, s);
    float* S = a.state + (((size_t)slot * a.heads + a.group0 * a.per_group + head) * DK + ch) * a.dv + col;
    float s[4] = {S[0], S[a.dv], S[8 * (size_t)a.dv], S[9 * (size_t)a.dv]};
    float4* u = a.ws + (size_t)first * a.pass_heads * per_head + e;
    const float* end = a.ends + (size_t)first * a.pass_heads + head;
    const size_t step = (size_t)a.pass_heads * per_head;
    for (int c0 = 0; c0 < n; c0 += AHEAD) {
        float4 x[AHEAD];
        float d[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n) {
                x[i] = u[i * step];
                d[i] = end[(size_t)(c0 + i) * a.pass_heads];
            }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < n) {
                uint4 p;
                split2(s[0], s[1], p.x, p.z);
                split2(s[2], s[3], p.y, p.w);
                *reinterpret_cast<uint4*>(u + i * step) = p;
                s[0] = __fadd_rn(__fmul_rn(s[0], d[i]), x[i].x);
                s[1] = __fadd_rn(__fmul_rn(s[1], d[i]), x[i].y);
                s[2] = __fadd_rn(__fmul_rn(s[2], d[i]), x[i].z);
                s[3] = __fadd_rn(__fmul_rn(s[3], d[i]), x[i].w);
            }
        u += AHEAD * step;
    }
    S[0] = s[0];
    S[a.dv] = s[1];
    S[8 * (size_t)a.dv] = s[2];
    S[9 * (size_t)a.dv] = s[3];
}

// ---- o of every chunk: a warp has 16 of its tokens and half of the slab's columns ----
template <typename TS, int DK, int SLAB, bool FIXED>
__global__ void __launch_bounds__(256, 2) chunk_out_kernel(const __grid_constant__ ChunkArgs a) {
    constexpr int LDK = DK + 8, LDV = SLAB + 8, NT = SLAB / 16, STATE = DK * SLAB / 4;      // 8-wide tiles of a warp; float4 of an item's state
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    uint4* S0 = reinterpret_cast<uint4*>(chunk_smem);                       // two items' states, the next one's on its way
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(S0 + 2 * STATE);   // [C][LDK]
    __nv_bfloat16* Ks = Qs + C * LDK;                                       // [C][LDK]
    __nv_bfloat16* Vs = Ks + C * LDK;                                       // [C][LDV]
    float* cl = reinterpret_cast<float*>(Vs + C * LDV);
    float* bs = cl + C;
    int seg, t0;
    if (!find_chunk(a, blockIdx.x, seg, t0)) return;
    if (!jllm_in_bounds(a.state_slots[seg], a.num_slots, BOUNDS_SLOT)) return;
    const int blocks_per_group = (a.per_group * a.slabs + a.items - 1) / a.items;
    const int group = blockIdx.y / blocks_per_group, i0 = blockIdx.y % blocks_per_group * a.items;
    const int i_end = min(i0 + a.items, a.per_group * a.slabs);
    const int row0 = a.seg_start[seg] + t0, nt = min(C, a.seg_len[seg] - t0);
    const int tid = threadIdx.x, side = tid >> 7, mt = (tid >> 5) & 3, lane = tid & 31;
    const int h0 = a.group0 * a.per_group, hg = h0 + group * a.per_group;
    Values<TS, SLAB> v;
    Gates<FIXED> gates;
    auto fetch_state = [&](int i) {
        const Item it = item_of(a, group, i);
        const float4* src = a.ws + (((size_t)blockIdx.x * a.pass_heads + it.head) * a.slabs + it.slab) * STATE;
        uint4* dst = S0 + ((i - i0) & 1) * STATE;
#pragma unroll
        for (int e = 0; e < STATE / 256; ++e) cp_async_16(dst + e * 256 + tid, src + e * 256 + tid);
    };
    auto fetch_values = [&](int i) {
        const Item it = item_of(a, group, i);
        v.fetch(a, row0, nt, h0 + it.head, it.slab * SLAB);
        gates.fetch(a, row0, nt, h0 + it.head);
    };
    // q, k, v and the gates were there before chunk_states began, whose end chunk_scan's blocks have waited for before they let this
    // kernel in: only the states are waited for, and the rest overlaps chunk_scan.
    fetch_values(i0);
    load_rows<TS, DK>(Qs, static_cast<const TS*>(a.q) + (size_t)row0 * a.ld_q + a.q_off + (size_t)(hg / a.q_share) * DK, a.ld_q, nt);
    load_rows<TS, DK>(Ks, static_cast<const TS*>(a.k) + (size_t)row0 * a.ld_k + a.k_off + (size_t)(hg / a.k_share) * DK, a.ld_k, nt);
    __syncthreads();
    float qk[8][4] = {};
    own_scores<DK>(qk, Qs, Ks, mt, lane);
    pdl_wait();
    pdl_trigger();
    fetch_state(i0);
    for (int i = i0; i < i_end; ++i) {
        const Item it = item_of(a, group, i);
        const int h = h0 + it.head, c0 = it.slab * SLAB + side * NT * 8, live = min(NT, (a.dv - c0 + 7) / 8);     // (live <= 0: no column)
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();       // the item's state has arrived; nobody reads the values, gates and state of the item before
#pragma unroll
        for (int u = 0; u < v.N; ++u) *reinterpret_cast<uint4*>(Vs + v.row(u) * LDV + v.col(u)) = v.piece[u];
        gates.put(cl, bs);
        if (i + 1 < i_end) {
            fetch_state(i + 1);
            fetch_values(i + 1);
        }
        float acc[NT][4] = {};
        from_state<DK, NT>(acc, Qs, S0 + ((i - i0) & 1) * STATE + side * NT * 32 + lane, live, mt, lane);
        __syncthreads();       // values and gates are in place
        finish<SLAB, FIXED, NT>(a, acc, qk, Vs, cl, bs, h, c0, side * NT * 8, live, row0, nt, mt, lane);
    }
}

// ---- short segments: a block walks the chunks of one (segment, head, slab), the state in its registers ----
// A segment of a chunk or two has no chunks to run beside one another, and the way of its states through the workspace and two more
// launches are what it would wait for. The pieces and their order are those of the three kernels: the results have the same bits.
template <typename TS, int DK, int SLAB, bool FIXED>
__global__ void __launch_bounds__(256, 2) chunk_walk_kernel(const __grid_constant__ ChunkArgs a) {
    constexpr int LDK = DK + 8, LDV = SLAB + 8, STATE = DK * SLAB / 4;
    constexpr int MT = SLAB / 16, PARTS = 8 / MT, NS = DK / 8 / PARTS, NT = SLAB / 16;
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    uint4* S0 = reinterpret_cast<uint4*>(chunk_smem);
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(S0 + STATE);
    __nv_bfloat16 *Ks = Qs + C * LDK, *Vs = Ks + C * LDK, *Vh = Vs + C * LDV, *Vl = Vh + C * LDV;
    float *cl = reinterpret_cast<float*>(Vl + C * LDV), *bs = cl + C;
    const int seg = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * SLAB, chunks = all_chunks(a, seg), slot = a.state_slots[seg];
    pdl_wait();
    pdl_trigger();
    if (chunks == 0 || chunks > a.walked) return;
    if (!jllm_in_bounds(slot, a.num_slots, BOUNDS_SLOT)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int first = a.seg_start[seg], n = a.seg_len[seg];
    const int smt = warp % MT, part = warp / MT;                // the state: 16 value columns, NS tiles of channels
    const int side = warp >> 2, mt = warp & 3;                  // the results: half of the columns, 16 tokens
    const int col0 = c0 + side * NT * 8, live = min(NT, (a.dv - col0 + 7) / 8);
    Values<TS, SLAB> v;
    Gates<FIXED> gates;
    v.fetch(a, first, min(C, n), h, c0);
    gates.fetch(a, first, min(C, n), h);
    // (channels of 64: the next chunk's q and k wait in registers; of 128 they do not fit, and other blocks hide the way)
    constexpr bool AHEAD = DK == 64;
    auto q_from = [&](int row) { return static_cast<const TS*>(a.q) + (size_t)row * a.ld_q + a.q_off + (size_t)(h / a.q_share) * DK; };
    auto k_from = [&](int row) { return static_cast<const TS*>(a.k) + (size_t)row * a.ld_k + a.k_off + (size_t)(h / a.k_share) * DK; };
    Rows<TS, DK> qr, kr;
    if constexpr (AHEAD) {
        qr.fetch(q_from(first), a.ld_q, min(C, n));
        kr.fetch(k_from(first), a.ld_k, min(C, n));
    }
    float* S = a.state + (((size_t)slot * a.heads + h) * DK + part * (NS * 8) + 2 * t) * a.dv + c0 + smt * 16 + g;
    float s[NS][4];
#pragma unroll
    for (int j = 0; j < NS; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            s[j][e] = c0 + smt * 16 + (e >> 1) * 8 < a.dv ? S[(size_t)(j * 8 + (e & 1)) * a.dv + (e >> 1) * 8] : 0.f;
    for (int t0 = 0; t0 < n; t0 += C) {
        const int row0 = first + t0, nt = min(C, n - t0), rows = (nt + 15) / 16 * 16;
        if (t0 > 0) __syncthreads();       // nobody reads the chunk before any more
        if constexpr (AHEAD) {
            qr.put(Qs);
            kr.put(Ks);
        } else {
            load_rows<TS, DK>(Qs, q_from(row0), a.ld_q, nt, rows);
            load_rows<TS, DK>(Ks, k_from(row0), a.ld_k, nt, rows);
        }
        gates.put(cl, bs);
#pragma unroll
        for (int u = 0; u < v.N; ++u) *reinterpret_cast<uint4*>(Vs + v.row(u) * LDV + v.col(u)) = v.piece[u];
#pragma unroll
        for (int j = 0; j < NS; j += 2)
#pragma unroll
            for (int below = 0; below < 2; ++below) {
                uint4 p;
                split2(s[j][2 * below], s[j][2 * below + 1], p.x, p.z);
                split2(s[j + 1][2 * below], s[j + 1][2 * below + 1], p.y, p.w);
                S0[((part * (NS / 2) + j / 2) * (SLAB / 8) + smt * 2 + below) * 32 + lane] = p;
            }
        __syncthreads();
        weigh<TS, SLAB, FIXED>(v, Vh, Vl, cl, bs, nt);
        if (t0 + C < n) {
            v.fetch(a, row0 + C, min(C, n - t0 - C), h, c0);
            gates.fetch(a, row0 + C, min(C, n - t0 - C), h);
            if constexpr (AHEAD) {
                qr.fetch(q_from(row0 + C), a.ld_q, min(C, n - t0 - C));
                kr.fetch(k_from(row0 + C), a.ld_k, min(C, n - t0 - C));
            }
        }
        if (mt * 16 < nt) {
            float qk[8][4] = {}, acc[NT][4] = {};
            own_scores<DK>(qk, Qs, Ks, mt, lane);
            from_state<DK, NT>(acc, Qs, S0 + side * NT * 32 + lane, live, mt, lane);
            finish<SLAB, FIXED, NT>(a, acc, qk, Vs, cl, bs, h, col0, side * NT * 8, live, row0, nt, mt, lane);
        }
        __syncthreads();                   // the weighted values are in place
        float own[NS][4] = {};
        own_state<DK, SLAB, NS>(own, Vh, Vl, Ks, smt, part, lane, rows);
        const float d = FIXED ? cl[nt] : expf(cl[nt - 1]);
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[j][e] = __fadd_rn(__fmul_rn(s[j][e], d), own[j][e]);
    }
#pragma unroll
    for (int j = 0; j < NS; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (c0 + smt * 16 + (e >> 1) * 8 < a.dv) S[(size_t)(j * 8 + (e & 1)) * a.dv + (e >> 1) * 8] = s[j][e];
}

// A test's switch: the value columns of an item (32 or 64; 0: chosen from the shape).
int g_slab = 0;

// How the work is cut. Slabs of 64 value columns, or of 32 where a head has no more or 64 would leave SMs with fewer than four items
// (an item of 32 columns splits P as often for half the columns: a state space of 1,536 tokens x 64 heads 122 us with 32, 94 with 64).
// Items a block takes, of the heads that share q and k: two blocks run on an SM at a time, and a block's start (its q and k, their
// product) costs about 0.7 of an item; the number of rounds times their length is least. Where all heads' states do not fit the
// workspace, a pass takes as many groups as do.
struct Cut {
    int walked, walk_slab;       // segments of so many chunks and fewer are walked, in slabs of so many columns
    int slab, slabs, chunks, items, pass_groups;
    long long floats;            // 0: every segment is walked
    int launches;
};
constexpr long long WORKSPACE_FLOATS = 64ll << 20;      // 256 MB: 2,048 tokens of 64 heads with states of 128 x 64 take a quarter

// All segments are walked where that takes no longer than the three launches: a walked chunk takes as long as its block's chain (3.5 to
// 5 us), once more for every block beyond the first on an SM; the three launches take about two such chunks and 0.0095 for a chunk of
// one head and 64 value columns. Launched back to back, 64 heads with states of 128 x 64: one segment of 64 tokens 7 us walked and 16 in
// three launches, of 256 tokens 23 and 28, of 512 43 and 35; eight of 512 160 and 206. 16 fixed-decay heads of 128 x 128: one of 64
// tokens 6 and 12, of 192 14 and 13, of 512 35 and 20; eight of 512 71 and 101. Where the longer segments take the three launches, those
// of up to two chunks are walked all the same: their states would go the long way (32 single tokens beside a portion of 512, 64
// heads of 128 x 64: 179 us in three launches, 115 with the single ones walked).
constexpr int WALKED = 2, WALKED_MOST = 12;      // (no more chunks than measured)
bool walks_all(int rows, int segments, int longest, int heads, int dv, int sms) {
    const long long pairs = (long long)segments * heads, wide = pairs * ((dv + 63) / 64);
    const bool narrow = wide < sms;
    const double rounds = (double)(((narrow ? pairs * ((dv + 31) / 32) : wide) + sms - 1) / sms) * (narrow ? 0.9 : 1.);
    const double chunks = (double)((rows + 32ll * segments) / C);          // (a segment's last chunk is half full)
    return longest <= WALKED_MOST * C && (longest + C - 1) / C * (rounds > 1. ? rounds : 1.) < 2. + 0.0095 * chunks * heads * (dv / 64.);
}

// `longest`: the rows of the longest segment
Cut cut_of(int rows, int segments, int longest, int heads, int groups, int dk, int dv) {
    const int sms = jllm_device_sm_count() > 0 ? jllm_device_sm_count() : 148;
    Cut c{};
    longest = longest > rows ? rows : longest;
    const bool scans = longest > WALKED * C && !walks_all(rows, segments, longest, heads, dv, sms);
    if (!scans || segments > 1) {
        c.walked = scans ? WALKED : INT_MAX;
        c.walk_slab = g_slab ? g_slab : (dv <= 32 || (long long)segments * heads * ((dv + 63) / 64) < sms ? 32 : 64);
        c.launches = 1;
    }
    if (!scans) return c;
    const int longs = rows / (c.walked * C + 1);                 // no more segments than that are longer
    c.chunks = rows / C + (longs < segments ? longs : segments);
    const int per_group = heads / groups;
    c.slab = g_slab ? g_slab : (dv <= 32 || (long long)c.chunks * heads * ((dv + 63) / 64) < 4ll * sms ? 32 : 64);
    c.slabs = (dv + c.slab - 1) / c.slab;
    const int items = per_group * c.slabs;
    float best = 0.f;
    for (int n = 1; n <= items; ++n) {
        const long long blocks = (long long)c.chunks * groups * ((items + n - 1) / n);
        const float cost = (float)((blocks + 2 * sms - 1) / (2 * sms)) * (n + 0.7f);
        if (n == 1 || cost < best) best = cost, c.items = n;
    }
    const long long group_floats = (long long)c.chunks * per_group * (c.slabs * c.slab * dk + 1);
    c.pass_groups = (int)(WORKSPACE_FLOATS / group_floats);
    c.pass_groups = c.pass_groups < 1 ? 1 : c.pass_groups > groups ? groups : c.pass_groups;
    c.floats = group_floats * c.pass_groups;
    c.launches += 3 * ((groups + c.pass_groups - 1) / c.pass_groups);
    return c;
}

template <typename TS, int DK, int SLAB, bool FIXED>
int run_walk(const ChunkArgs& a, cudaStream_t stream) {
    constexpr size_t smem = (size_t)DK * SLAB * 4 + 2 * (size_t)C * (DK + 8) * 2 + 3 * (size_t)C * (SLAB + 8) * 2 + GATES * sizeof(float);
    if (jllm_allow_smem((const void*)chunk_walk_kernel<TS, DK, SLAB, FIXED>, smem) != cudaSuccess)
        return jllm_fail(JLLM_CUDA_ERROR, "chunk_walk: %zu bytes of shared memory refused", smem);
    jllm_launch(chunk_walk_kernel<TS, DK, SLAB, FIXED>, dim3(a.segments, a.heads, (a.dv + SLAB - 1) / SLAB), dim3(256), smem, stream,
                LAUNCH_DEPENDENT, a);
    return jllm_check_launch("chunk_walk");
}

template <typename TS, int DK, int SLAB, bool FIXED>
int run_passes(ChunkArgs a, const Cut& c, float* workspace, cudaStream_t stream) {
    const size_t tail = GATES * sizeof(float), values = (size_t)C * (SLAB + 8) * 2, rows = (size_t)C * (DK + 8) * 2;
    const size_t smem_s = rows + 2 * values + tail, smem_o = 2 * (size_t)DK * SLAB * 4 + 2 * rows + values + tail;
    if (jllm_allow_smem((const void*)chunk_states_kernel<TS, DK, SLAB, FIXED>, smem_s) != cudaSuccess ||
        jllm_allow_smem((const void*)chunk_out_kernel<TS, DK, SLAB, FIXED>, smem_o) != cudaSuccess)
        return jllm_fail(JLLM_CUDA_ERROR, "chunk_scan: %zu bytes of shared memory refused", smem_s > smem_o ? smem_s : smem_o);
    const int per_head = c.slabs * (DK / 16) * (SLAB / 8) * 32;
    for (int g0 = 0; g0 < a.groups; g0 += c.pass_groups) {
        const int pass = a.groups - g0 < c.pass_groups ? a.groups - g0 : c.pass_groups;
        a.group0 = g0;
        a.pass_heads = pass * a.per_group;
        a.ws = reinterpret_cast<float4*>(workspace);
        a.ends = workspace + (size_t)c.chunks * a.pass_heads * per_head * 4;
        const dim3 grid(c.chunks, pass * ((a.per_group * c.slabs + c.items - 1) / c.items));
        jllm_launch(chunk_states_kernel<TS, DK, SLAB, FIXED>, grid, dim3(256), smem_s, stream, LAUNCH_DEPENDENT, a);
        int code = jllm_check_launch("chunk_states");
        if (code) return code;
        const long long elements = (long long)a.pass_heads * per_head;
        jllm_launch(chunk_scan_kernel<DK, SLAB>, dim3((unsigned)((elements + 255) / 256), a.segments), dim3(256), 0, stream, LAUNCH_DEPENDENT, a);
        code = jllm_check_launch("chunk_scan");
        if (code) return code;
        jllm_launch(chunk_out_kernel<TS, DK, SLAB, FIXED>, grid, dim3(256), smem_o, stream, LAUNCH_DEPENDENT, a);
        code = jllm_check_launch("chunk_out");
        if (code) return code;
    }
    return JLLM_OK;
}

template <typename TS, bool FIXED>
int run_chunks(ChunkArgs a, int rows, int longest, int dk, float* workspace, long long workspace_floats, cudaStream_t stream) {
    const Cut c = cut_of(rows, a.segments, longest, a.heads, a.groups, dk, a.dv);
    JLLM_REQUIRE(c.floats == 0 || (workspace != nullptr && workspace_floats >= c.floats && ((uintptr_t)workspace % 16) == 0),
                 "chunk_scan: a workspace of %lld floats where %lld are needed (16-byte aligned)", workspace_floats, c.floats);
    JLLM_REQUIRE(c.floats == 0 || ((long long)a.groups * ((a.per_group * c.slabs + c.items - 1) / c.items) <= 65535 && a.segments <= 65535),
                 "chunk_scan: %d heads in %d segments are too many blocks", a.heads, a.segments);
    a.chunks = c.chunks, a.walked = c.walked, a.slabs = c.slabs, a.items = c.items;
    if (c.walked) {
        const bool wide = c.walk_slab == 64;
        const int code = dk == 64 ? (wide ? run_walk<TS, 64, 64, FIXED>(a, stream) : run_walk<TS, 64, 32, FIXED>(a, stream))
                                  : (wide ? run_walk<TS, 128, 64, FIXED>(a, stream) : run_walk<TS, 128, 32, FIXED>(a, stream));
        if (code || c.floats == 0) return code;
    }
    if (dk == 64) return c.slab == 64 ? run_passes<TS, 64, 64, FIXED>(a, c, workspace, stream) : run_passes<TS, 64, 32, FIXED>(a, c, workspace, stream);
    return c.slab == 64 ? run_passes<TS, 128, 64, FIXED>(a, c, workspace, stream) : run_passes<TS, 128, 32, FIXED>(a, c, workspace, stream);
}

}  // namespace

JLLM_BOUNDS_READER(chunk_scan)

JLLM_EXPORT int jllm_lightning_block_width(int width) {
    JLLM_REQUIRE(width == 0 || width == 32 || width == 64, "lightning_block_width: %d is not 0, 32 or 64", width);
    g_slab = width;
    return JLLM_OK;
}

// What a step's chunks take: the launches; `floats`: the workspace (0: none). Heads in `groups` that share q and k, the longest segment
// of `longest` rows.
JLLM_EXPORT int jllm_chunk_plan(int rows, int segments, int longest, int heads, int groups, int dk, int dv, long long* floats) {
    *floats = 0;
    if (rows <= 0 || segments <= 0 || heads <= 0 || groups <= 0 || heads % groups || dk <= 0 || dv <= 0) return 0;
    const Cut c = cut_of(rows, segments, longest, heads, groups, dk, dv);
    *floats = c.floats;
    return c.launches;
}

// ... and the passes over the heads that segments of any length make in it
JLLM_EXPORT int jllm_chunk_passes(int rows, int segments, int heads, int groups, int dk, int dv) {
    if (rows <= 0 || segments <= 0 || heads <= 0 || groups <= 0 || heads % groups || dk <= 0 || dv <= 0) return 0;
    const int at_once = cut_of(rows, segments, rows, heads, groups, dk, dv).pass_groups;
    return at_once ? (groups + at_once - 1) / at_once : 0;
}

// one fixed decay per head, q, k, v pieces of one bfloat16 matrix (called by jllm_gla_chunked)
int jllm_fixed_decay_chunks(const __nv_bfloat16* proj, int ld, int q_off, int k_off, int v_off, const float* head_decay, float* state,
                            int num_slots, const int* seg_start, const int* seg_len, const int* state_slots, float* o, int rows,
                            int segments, int longest, int heads, int dk, int dv, float q_scale, float* workspace,
                            long long workspace_floats, cudaStream_t stream) {
    ChunkArgs a{};
    a.q = a.k = a.v = proj;
    a.ld_q = a.ld_k = a.ld_v = ld;
    a.q_off = q_off, a.k_off = k_off, a.v_off = v_off;
    a.groups = heads, a.per_group = a.q_share = a.k_share = 1;
    a.decay = head_decay;
    a.skip = VecRef{nullptr, JLLM_F32};
    a.state = state, a.num_slots = num_slots;
    a.seg_start = seg_start, a.seg_len = seg_len, a.state_slots = state_slots;
    a.o = o, a.segments = segments, a.heads = heads, a.dv = dv, a.q_scale = q_scale;
    return run_chunks<__nv_bfloat16, true>(a, rows, longest, dk, workspace, workspace_floats, stream);
}

// Whether jllm_scalar_gated_chunked takes a shape: key heads of 64 or 128 channels, 16-byte aligned rows and pieces.
JLLM_EXPORT int jllm_scalar_gated_chunks_fit(const void* q, int ld_q, int q_off, int q_groups, const void* k, int ld_k, int k_off,
                                             int k_groups, const void* v, int ld_v, int v_off, int dtype, int heads, int dk, int dv) {
    const int per = dtype == JLLM_F32 ? 4 : 8;          // values of a 16-byte piece
    const bool aligned = ld_q % per == 0 && ld_k % per == 0 && ld_v % per == 0 && q_off % per == 0 && k_off % per == 0 &&
                         v_off % per == 0 && dv % 8 == 0 && ((uintptr_t)q % 16) == 0 && ((uintptr_t)k % 16) == 0 &&
                         ((uintptr_t)v % 16) == 0;
    return (dk == 64 || dk == 128) && aligned && q_groups > 0 && k_groups > 0 && heads % q_groups == 0 && heads % k_groups == 0 &&
           heads <= 65535;
}

// The recurrence with a decay and an input scale per token and head (`jllm_scalar_gated_recurrent`, which this stands in for
// where a step holds prompt portions), without a normalizer. q, k, v: views of type `dtype` (float32 or bfloat16). Returns
// JLLM_UNSUPPORTED without launching where jllm_scalar_gated_chunks_fit says no (the caller then runs token by token). `longest`: the
// rows of the longest segment; `workspace`: what jllm_chunk_plan says for the heads in q_groups groups if that equals k_groups, else
// a group per head.
JLLM_EXPORT int jllm_scalar_gated_chunked(const void* q, int ld_q, int q_off, int q_groups, const void* k, int ld_k, int k_off,
                                          int k_groups, const void* v, int ld_v, int v_off, int dtype, const float* la,
                                          const float* b, const void* skip, int skip_dtype, float* state, int num_slots,
                                          const int* seg_start, const int* seg_len, const int* state_slots, float* o,
                                          int rows, int segments, int longest, int heads, int dk, int dv, float q_scale,
                                          float* workspace, long long workspace_floats, cudaStream_t stream) {
    if (!jllm_scalar_gated_chunks_fit(q, ld_q, q_off, q_groups, k, ld_k, k_off, k_groups, v, ld_v, v_off, dtype, heads, dk, dv))
        return JLLM_UNSUPPORTED;
    if (segments == 0 || rows == 0) return JLLM_OK;
    ChunkArgs a{};
    a.q = q, a.k = k, a.v = v;
    a.ld_q = ld_q, a.ld_k = ld_k, a.ld_v = ld_v;
    a.q_off = q_off, a.k_off = k_off, a.v_off = v_off;
    a.groups = q_groups == k_groups ? q_groups : heads;
    a.per_group = heads / a.groups;
    a.q_share = heads / q_groups, a.k_share = heads / k_groups;
    a.la = la, a.b = b;
    a.skip = VecRef{skip, skip_dtype}, a.has_skip = skip != nullptr;
    a.state = state, a.num_slots = num_slots;
    a.seg_start = seg_start, a.seg_len = seg_len, a.state_slots = state_slots;
    a.o = o, a.segments = segments, a.heads = heads, a.dv = dv, a.q_scale = q_scale;
    return dtype == JLLM_F32 ? run_chunks<float, false>(a, rows, longest, dk, workspace, workspace_floats, stream)
                             : run_chunks<__nv_bfloat16, false>(a, rows, longest, dk, workspace, workspace_floats, stream);
}

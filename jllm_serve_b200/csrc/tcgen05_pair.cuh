// Pieces shared by the products that two SMs make together (tcgen05 cta_group::2): where a block is in its pair, what reaches into the
// partner's shared memory, the pair's MMA and commit, and the tensor map of a packed weight.
#pragma once

#include "tcgen05_common.cuh"

namespace tc {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the address, in the cluster's shared window, of `addr` (an address in this block's shared memory) in block `rank`
__device__ __forceinline__ uint32_t in_block(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void store_cluster(uint32_t cluster_addr, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// a tiled copy into THIS block's shared memory that completes on a barrier that may be the partner's
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(cluster_bar)
        : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives, when the MMAs issued so far are done, on the barrier at this offset in both blocks of the pair
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}

// The packed weight ([tiles of 128 rows][k blocks][128 rows][64 values], each 16 KB tile the swizzled shared-memory
// image) as a matrix of 128-byte rows, copied in boxes of one tile without any further swizzle.
struct PackedKey {
    const void* ptr;
    long long rows;
    bool operator==(const PackedKey& o) const { return ptr == o.ptr && rows == o.rows; }
};
struct PackedKeyHash {
    size_t operator()(const PackedKey& k) const { return std::hash<const void*>()(k.ptr) * 1000003u ^ std::hash<long long>()(k.rows); }
};
inline int packed_map_for(const void* ptr, long long rows, CUtensorMap* out) {
    static std::unordered_map<PackedKey, CUtensorMap, PackedKeyHash> cache;
    static std::mutex mu;
    const PackedKey key{ptr, rows};
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return JLLM_OK;
    }
    EncodeTiledFn fn = encode_fn();
    if (!fn) return jllm_fail(JLLM_CUDA_ERROR, "gemm: the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {64, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {128};
    const cuuint32_t box[2] = {64, 128};
    const cuuint32_t elem[2] = {1, 1};
    CUtensorMap map;
    const CUresult r = fn(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return jllm_fail(JLLM_CUDA_ERROR, "gemm: cuTensorMapEncodeTiled failed (%d) for a packed weight of %lld rows",
                         (int)r, rows);
    if (cache.size() > 4096) cache.clear();
    cache.emplace(key, map);
    *out = map;
    return JLLM_OK;
}

}  // namespace tc

// KV-cache data movement over the block-major pool [num_blocks][block_size][kv_heads][D]:
// scatter-append, block reset and block gather.
//
// Stands in for kv_append_kernel / kv_reset_kernel / kv_gather_kernel
// (src/kv_cache/kv_cache_kernels.cu:17-86), which move one byte per thread (reset, gather) or one
// whole row per thread in a byte loop (append). Here every thread moves 16 bytes, consecutive
// threads touch consecutive 16-byte chunks of the same row (fully coalesced 128-byte lines), and K
// and V are handled in the same pass. Addressing follows src/kv_cache/kv_cache_layout.cuh:32-38.
// Rows whose byte length or base addresses are not 16-byte multiples fall back to single bytes so
// the result is bit-exact for any geometry.
//
// Algorithmic traffic: append = 2 * tokens * kv_heads * D * elem bytes read + the same written;
// reset = 2 * blocks * block_bytes written; gather = blocks * block_bytes read + written.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace sca_b200 {
namespace {

constexpr int kKvThreads = 256;

// A list of rows of `width` pieces of type V, cut into runs of kPieces * kKvThreads consecutive pieces, one run per CTA at a
// time. A thread takes kPieces of a run, kKvThreads apart, and has all of their loads in flight before its first store. I is
// 32 bits wide where the pieces can be counted in it: a 64-bit division per piece costs more than moving 16 bytes. Bound by
// HBM: 668 MB (50 thousand tokens appended, 3000 blocks of 32 KB copied out, 1000 cleared, four launches) 126.4 us with one
// piece and 64-bit counters, 115.4 now (5.8 TB/s); pieces of 32 bytes two at a time 115.2, four at a time 117.7.
constexpr int kPieces = 4;

template <typename V, typename I>
__global__ void __launch_bounds__(kKvThreads)
kv_append_kernel(V* layer_k, V* layer_v, const V* k_new, const V* v_new, const int32_t* slots, const I total,
                 const ScaKvCacheShape shape, const I token_vecs) {
    // token_vecs = kv_heads * D * elem_bytes / sizeof(V): one token's K (or V) payload is contiguous
    // both in the source [token][head][D] and in the pool [slot][head][D].
    BeginAfterPredecessor();
    constexpr int N = kPieces;
    const int64_t pool_tokens = shape.num_blocks * shape.block_size;
    for (I run = static_cast<I>(blockIdx.x) * (N * kKvThreads); run < total; run += static_cast<I>(gridDim.x) * (N * kKvThreads)) {
        V k[N], v[N];
        int64_t dst[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const I idx = run + i * kKvThreads + threadIdx.x;
            dst[i] = -1;
            if (idx >= total) continue;
            const int32_t slot = slots[idx / token_vecs];
            if (slot < 0) continue;                    // "do not store" sentinel
            if (slot >= pool_tokens) continue;         // never write out of range
            dst[i] = static_cast<int64_t>(slot) * token_vecs + idx % token_vecs;
            k[i] = k_new[idx];
            v[i] = v_new[idx];
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (dst[i] < 0) continue;
            layer_k[dst[i]] = k[i];
            layer_v[dst[i]] = v[i];
        }
    }
}

// Same scatter with the slot computed on the device from the page table: one new token per
// sequence at position seq_lens[s] - 1.
template <typename V>
__global__ void __launch_bounds__(kKvThreads)
kv_append_batched_kernel(V* layer_k, V* layer_v, const V* k_new, const V* v_new, const int32_t* page_table, const int32_t* seq_lens,
                         const int64_t num_seqs, const int64_t max_blocks_per_seq, const ScaKvCacheShape shape,
                         const int64_t token_vecs) {
    BeginAfterPredecessor();
    const int64_t total = num_seqs * token_vecs;
    for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
         idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t seq = idx / token_vecs;
        const int64_t within = idx % token_vecs;
        const V k = k_new[idx], v = v_new[idx];  // on their way while the length and the table entry are looked up
        const int64_t pos = static_cast<int64_t>(seq_lens[seq]) - 1;
        if (pos < 0) continue;
        const int64_t logical = pos / shape.block_size;
        if (logical >= max_blocks_per_seq) continue;
        const int32_t phys = page_table[seq * max_blocks_per_seq + logical];
        if (phys < 0 || phys >= shape.num_blocks) continue;
        const int64_t slot = static_cast<int64_t>(phys) * shape.block_size + pos % shape.block_size;
        const int64_t dst = slot * token_vecs + within;
        layer_k[dst] = k;
        layer_v[dst] = v;
    }
}

template <typename V, typename I>
__global__ void __launch_bounds__(kKvThreads)
kv_reset_kernel(V* layer_k, V* layer_v, const int32_t* ids, const I total, const int64_t num_blocks, const I block_vecs) {
    BeginAfterPredecessor();
    constexpr int N = kPieces;
    V zero;
    memset(&zero, 0, sizeof(V));
    for (I run = static_cast<I>(blockIdx.x) * (N * kKvThreads); run < total; run += static_cast<I>(gridDim.x) * (N * kKvThreads)) {
        int64_t dst[N];  // all of a run's ids are read ahead of its first store
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const I idx = run + i * kKvThreads + threadIdx.x;
            dst[i] = -1;
            if (idx >= total) continue;
            const int32_t phys = ids[idx / block_vecs];
            if (phys < 0 || phys >= num_blocks) continue;
            dst[i] = static_cast<int64_t>(phys) * block_vecs + idx % block_vecs;
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (dst[i] < 0) continue;
            layer_k[dst[i]] = zero;
            layer_v[dst[i]] = zero;
        }
    }
}

template <typename V, typename I>
__global__ void __launch_bounds__(kKvThreads)
kv_gather_kernel(const V* layer, const int32_t* ids, const I total, V* out, const int64_t num_blocks, const I block_vecs) {
    BeginAfterPredecessor();
    constexpr int N = kPieces;
    for (I run = static_cast<I>(blockIdx.x) * (N * kKvThreads); run < total; run += static_cast<I>(gridDim.x) * (N * kKvThreads)) {
        V v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const I idx = run + i * kKvThreads + threadIdx.x;
            if (idx >= total) continue;
            const int32_t phys = ids[idx / block_vecs];
            if (phys < 0 || phys >= num_blocks) memset(&v[i], 0, sizeof(V));
            else v[i] = layer[static_cast<int64_t>(phys) * block_vecs + idx % block_vecs];
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const I idx = run + i * kKvThreads + threadIdx.x;
            if (idx < total) out[idx] = v[i];
        }
    }
}

unsigned GridFor(int64_t items) {
    // enough CTAs to cover the work once, capped at a few waves of the machine: the loops are
    // grid-stride, and HBM is saturated long before more CTAs would help
    const int64_t want = (items + kKvThreads - 1) / kKvThreads;
    const int64_t cap = static_cast<int64_t>(SmCount()) * 32;
    return static_cast<unsigned>(std::max<int64_t>(1, std::min(want, cap)));
}

// Calls f(piece, total, width) with a null pointer to the piece type and counters of the index type the call allows: `rows`
// rows of `row_bytes` bytes; `aligned`: all pointers lie on 16-byte boundaries. What a run may step past `total` fits too.
template <typename F>
void ForPieces(int64_t rows, int64_t row_bytes, bool aligned, const F& f) {
    auto counted = [&](auto* piece) {
        const int64_t width = row_bytes / static_cast<int64_t>(sizeof(*piece)), total = rows * width;
        if (total < (1ll << 31)) f(piece, static_cast<uint32_t>(total), static_cast<uint32_t>(width));
        else f(piece, total, width);
    };
    if (row_bytes % 16 == 0 && aligned) counted(static_cast<uint4*>(nullptr));
    else counted(static_cast<unsigned char*>(nullptr));
}

int CheckShape(const ScaKvCacheShape* shape, int64_t elem_bytes, const char* what) {
    if (shape == nullptr) return Fail(SCA_INVALID_ARGUMENT, std::string(what) + ": null shape");
    if (shape->num_blocks <= 0 || shape->block_size <= 0 || shape->num_kv_heads <= 0 ||
        shape->head_dim <= 0 || elem_bytes <= 0) {
        return Fail(SCA_INVALID_ARGUMENT, std::string(what) + ": non-positive geometry");
    }
    return SCA_OK;
}

// Block-id lists are documented as device memory, but the reference's own PagedKVCache::ResetSeq hands
// KVCache::Reset the ids straight out of a std::vector (src/kv_cache/paged_kv_cache.cpp:150-156), which only
// works where the GPU can read pageable host memory. A list that lives in host memory is therefore copied into
// a stream-ordered temporary first (the copy out of pageable memory completes before the call returns, so the
// caller may drop its vector right away); device and managed pointers are used as they are.
class StagedIds {
public:
    StagedIds() = default;
    StagedIds(const StagedIds&) = delete;
    StagedIds& operator=(const StagedIds&) = delete;
    ~StagedIds() {
        if (staged_ != nullptr && cudaFreeAsync(staged_, stream_) != cudaSuccess) cudaGetLastError();
    }
    int Stage(const int32_t* ids, int64_t count, cudaStream_t stream, const char* what) {
        ids_ = ids;
        cudaPointerAttributes attr{};
        if (cudaPointerGetAttributes(&attr, ids) != cudaSuccess) {
            cudaGetLastError();
            return SCA_OK;  // no usable device: the launch below reports it
        }
        if (attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged) return SCA_OK;
        if (attr.type == cudaMemoryTypeHost && attr.devicePointer != nullptr) {
            ids_ = static_cast<const int32_t*>(attr.devicePointer);  // pinned and mapped: readable in place
            return SCA_OK;
        }
        const size_t bytes = static_cast<size_t>(count) * sizeof(int32_t);
        stream_ = stream;
        if (cudaError_t err = cudaMallocAsync(reinterpret_cast<void**>(&staged_), bytes, stream); err != cudaSuccess) {
            staged_ = nullptr;
            cudaGetLastError();
            return FailCuda(err, what);
        }
        if (int rc = SendToDevice(staged_, ids, bytes, stream, what)) return rc;
        ids_ = staged_;
        return SCA_OK;
    }
    const int32_t* get() const { return ids_; }

private:
    const int32_t* ids_{nullptr};
    int32_t* staged_{nullptr};
    cudaStream_t stream_{nullptr};
};

}  // namespace
}  // namespace sca_b200

using namespace sca_b200;

extern "C" int sca_launch_kv_append(void* layer_k, void* layer_v, const void* k_new, const void* v_new,
                                    const int32_t* slot_mapping, int64_t num_tokens,
                                    const ScaKvCacheShape* shape, int64_t elem_bytes, void* stream) {
    ClearError();
    if (layer_k == nullptr || layer_v == nullptr || k_new == nullptr || v_new == nullptr ||
        slot_mapping == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "kv append: null pointer");
    }
    if (num_tokens <= 0) return Fail(SCA_INVALID_ARGUMENT, "kv append: num_tokens <= 0");
    if (int rc = CheckShape(shape, elem_bytes, "kv append")) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t token_bytes = shape->num_kv_heads * shape->head_dim * elem_bytes;
    const bool aligned = Aligned16(layer_k) && Aligned16(layer_v) && Aligned16(k_new) && Aligned16(v_new);
    ForPieces(num_tokens, token_bytes, aligned, [&](auto* piece, auto total, auto width) {
        using V = std::remove_pointer_t<decltype(piece)>;
        LaunchDependent(kv_append_kernel<V, decltype(total)>, GridFor((total + kPieces - 1) / kPieces), kKvThreads, 0, s, 1,
            static_cast<V*>(layer_k), static_cast<V*>(layer_v), static_cast<const V*>(k_new), static_cast<const V*>(v_new), slot_mapping,
            total, *shape, width);
    });
    return CheckLaunch("kv_append_kernel", s);
}

extern "C" int sca_launch_kv_append_batched(void* layer_k, void* layer_v, const void* k_new,
                                            const void* v_new, const int32_t* page_table,
                                            const int32_t* seq_lens, int64_t num_seqs,
                                            int64_t max_blocks_per_seq, const ScaKvCacheShape* shape,
                                            int64_t elem_bytes, void* stream) {
    ClearError();
    if (layer_k == nullptr || layer_v == nullptr || k_new == nullptr || v_new == nullptr ||
        page_table == nullptr || seq_lens == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "kv append (batched): null pointer");
    }
    if (num_seqs <= 0 || max_blocks_per_seq <= 0) {
        return Fail(SCA_INVALID_ARGUMENT, "kv append (batched): num_seqs/max_blocks_per_seq <= 0");
    }
    if (int rc = CheckShape(shape, elem_bytes, "kv append (batched)")) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t token_bytes = shape->num_kv_heads * shape->head_dim * elem_bytes;
    const bool vec = token_bytes % 16 == 0 && Aligned16(layer_k) && Aligned16(layer_v) &&
                     Aligned16(k_new) && Aligned16(v_new);
    if (vec) {
        const int64_t tv = token_bytes / 16;
        LaunchDependent(kv_append_batched_kernel<uint4>, GridFor(num_seqs * tv), kKvThreads, 0, s, 1,
            static_cast<uint4*>(layer_k), static_cast<uint4*>(layer_v), static_cast<const uint4*>(k_new),
            static_cast<const uint4*>(v_new), page_table, seq_lens, num_seqs, max_blocks_per_seq, *shape, tv);
    } else {
        LaunchDependent(kv_append_batched_kernel<unsigned char>, GridFor(num_seqs * token_bytes), kKvThreads, 0, s, 1,
            static_cast<unsigned char*>(layer_k), static_cast<unsigned char*>(layer_v),
            static_cast<const unsigned char*>(k_new), static_cast<const unsigned char*>(v_new), page_table,
            seq_lens, num_seqs, max_blocks_per_seq, *shape, token_bytes);
    }
    return CheckLaunch("kv_append_batched_kernel", s);
}

extern "C" int sca_launch_kv_reset_block(void* layer_k, void* layer_v, const int32_t* block_ids,
                                         int64_t num_blocks, const ScaKvCacheShape* shape,
                                         int64_t elem_bytes, void* stream) {
    ClearError();
    if (layer_k == nullptr || layer_v == nullptr || block_ids == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "kv reset: null pointer");
    }
    if (num_blocks <= 0) return SCA_OK;
    if (int rc = CheckShape(shape, elem_bytes, "kv reset")) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    StagedIds ids;
    if (int rc = ids.Stage(block_ids, num_blocks, s, "kv reset: staging host block ids")) return rc;
    block_ids = ids.get();
    const int64_t block_bytes = shape->block_size * shape->num_kv_heads * shape->head_dim * elem_bytes;
    ForPieces(num_blocks, block_bytes, Aligned16(layer_k) && Aligned16(layer_v), [&](auto* piece, auto total, auto width) {
        using V = std::remove_pointer_t<decltype(piece)>;
        LaunchDependent(kv_reset_kernel<V, decltype(total)>, GridFor((total + kPieces - 1) / kPieces), kKvThreads, 0, s, 1,
            static_cast<V*>(layer_k), static_cast<V*>(layer_v), block_ids, total, shape->num_blocks, width);
    });
    return CheckLaunch("kv_reset_kernel", s);
}

extern "C" int sca_launch_kv_gather(const void* layer, const int32_t* block_ids, int64_t num_blocks,
                                    void* out, const ScaKvCacheShape* shape, int64_t elem_bytes,
                                    void* stream) {
    ClearError();
    if (layer == nullptr || block_ids == nullptr || out == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "kv gather: null pointer");
    }
    if (num_blocks <= 0) return SCA_OK;
    if (int rc = CheckShape(shape, elem_bytes, "kv gather")) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    StagedIds ids;
    if (int rc = ids.Stage(block_ids, num_blocks, s, "kv gather: staging host block ids")) return rc;
    block_ids = ids.get();
    const int64_t block_bytes = shape->block_size * shape->num_kv_heads * shape->head_dim * elem_bytes;
    ForPieces(num_blocks, block_bytes, Aligned16(layer) && Aligned16(out), [&](auto* piece, auto total, auto width) {
        using V = std::remove_pointer_t<decltype(piece)>;
        LaunchDependent(kv_gather_kernel<V, decltype(total)>, GridFor((total + kPieces - 1) / kPieces), kKvThreads, 0, s, 1,
            static_cast<const V*>(layer), block_ids, total, static_cast<V*>(out), shape->num_blocks, width);
    });
    return CheckLaunch("kv_gather_kernel", s);
}

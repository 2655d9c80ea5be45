// Host side of the prefill: tensor maps, work lists of ragged batches, the choice of the launch. The kernel is in
// flash_kernel.cuh.
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "flash_kernel.cuh"

namespace sca_b200 {
namespace {

using namespace flash;

constexpr int kMaxStatusDevices = 64;

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn GetEncodeTiled() {
    static EncodeTiledFn fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            sym = nullptr;
        }
        return reinterpret_cast<EncodeTiledFn>(sym);
    }();
    return fn;
}

// [batch][heads][seq][D] through element strides (sb, sh, ss); box = 64 elements x box_rows rows, 128B swizzle,
// out-of-range elements read as zero.
int MakeMap(CUtensorMap* map, const void* base, int dtype_id, int64_t d, int64_t seq, int64_t heads, int64_t batch,
            int64_t ss, int64_t sh, int64_t sb, int box_rows, const char* what, int box_heads = 1) {
    EncodeTiledFn encode = GetEncodeTiled();
    if (encode == nullptr) return Fail(SCA_CUDA_ERROR, "flash attention: cuTensorMapEncodeTiled is unavailable");
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(d), static_cast<cuuint64_t>(seq),
                                static_cast<cuuint64_t>(heads), static_cast<cuuint64_t>(batch)};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(ss) * 2, static_cast<cuuint64_t>(sh) * 2,
                                   static_cast<cuuint64_t>(sb) * 2};
    const cuuint32_t box[4] = {64, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(box_heads), 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    const CUtensorMapDataType type =
        dtype_id == SCA_DTYPE_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const CUresult rc = encode(map, type, 4, const_cast<void*>(base), dims, strides, box, elem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) {
        return Fail(SCA_INVALID_ARGUMENT, std::string("flash attention: tensor map for ") + what +
                                              " rejected (CUresult " + std::to_string(static_cast<int>(rc)) +
                                              "); base must be 16-byte aligned and strides multiples of 8 elements");
    }
    return SCA_OK;
}

// One host-visible word per device that a kernel sets when one of its bounded waits expires (1 + the warp that
// gave up). The words live in one pinned, mapped, portable allocation; sca_flash_status reads and clears them.

int* ErrorWords(int** host_view) {
    static int* host = nullptr;
    static int* dev = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        if (cudaHostAlloc(reinterpret_cast<void**>(&host), kMaxStatusDevices * sizeof(int),
                          cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            host = nullptr;
            return;
        }
        for (int i = 0; i < kMaxStatusDevices; ++i) host[i] = 0;
        if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev), host, 0) != cudaSuccess) {
            cudaGetLastError();
            dev = nullptr;
        }
    });
    if (host_view != nullptr) *host_view = host;
    return dev;
}

// Device-side address of the current device's word (nullptr when the mapping could not be made).
int* ErrorWordForCurrentDevice() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    int* dev = ErrorWords(nullptr);
    return (dev != nullptr && device >= 0 && device < kMaxStatusDevices) ? dev + device : nullptr;
}

// A packed variable-length batch: host offsets and a device scratch area for the work list.
struct VarlenWork {
    const int32_t* cu_q;
    const int32_t* cu_kv;
    int64_t num_seqs;
    void* workspace;
    int64_t workspace_bytes;
};

// log2 of the query heads that share a tile: the largest power of two that divides the GQA group, at most 1 << kMaxPackShift.
constexpr int kMaxPackShift = 2;
int PackShift(int64_t group) {
    int shift = 0;
    while (shift < kMaxPackShift && group % (2ll << shift) == 0) ++shift;
    return shift;
}

// Whether query heads should share tiles (us in a lasting load, heads alone / four to a tile, 32 / 8 heads).
// They fill the rows that a ragged end leaves empty, and they let both tiles of a causal item need the same KV tiles: D=128,
// S=3000 with B=1 94.5 / 92.5, B=4 350 / 342; D=64, B=8, S=1024 84 / 80; without a mask that is worth nothing. But the four
// heads of a kv head no longer stand side by side in the work list, each of them at the same key: with many kv heads or
// much K/V in flight that costs energy and bandwidth: D=128, B=4, S=4096 595 / 607 (no mask 1090 / 1134), B=8, S=4096 1209 /
// 1276, B=16, S=2048 698 / 767, B=32, S=256 60 / 66.5; D=256, B=8, S=1024 without a mask 348 / 377.
bool PackingPays(const ScaFlashFwdParams& f, int shift) {
    const int64_t tokens = kBlockM >> shift;
    const int64_t alone = (f.seq_q + kBlockM - 1) / kBlockM * kBlockM, packed = (f.seq_q + tokens - 1) / tokens * tokens;
    if (alone * 100 > packed * 107) return true;  // B=8, S=700 without a mask 106 / 97
    const int64_t pairs = f.batch * f.num_kv_heads;
    return f.causal && pairs <= 64 && pairs * f.seq_kv * f.head_dim * 4 <= 55000000;
}
// The same for a packed batch, whose ends are ragged and whose entries are in the order of their weight in any case:
// D=128, 10 sequences of 64 to 4096 594 / 580, 64 of 100 to 900 378 / 361. Long causal ones with much K/V lose: 16 of 4096
// 2467 / 2656, 32 of 2000 1394 / 1494; not without a mask (24 of 3000 to 4000 5055 / 4989) nor at D=64 (2156 / 2108).
bool PackingPays(const VarlenWork& vw, const ScaFlashFwdParams& f, int shift) {
    const int64_t kv_bytes = f.seq_kv * f.num_kv_heads * f.head_dim * 4;
    if (!f.causal || f.head_dim <= 64 || kv_bytes <= 150000000) return true;
    const int64_t tokens = kBlockM >> shift;
    int64_t alone = 0, packed = 0;
    for (int64_t s = 0; s < vw.num_seqs; ++s) {
        const int64_t rows = std::max<int64_t>(0, static_cast<int64_t>(vw.cu_q[s + 1]) - vw.cu_q[s]);
        alone += (rows + kBlockM - 1) / kBlockM * kBlockM;
        packed += (rows + tokens - 1) / tokens * tokens;
    }
    return alone * 100 > packed * 106;
}

int64_t VarlenWorkspaceBytes(int64_t num_seqs, int64_t total_q) {
    // one int4 per sequence + one int2 per (sequence, query block); a block covers at least kBlockM >> kMaxPackShift tokens
    return num_seqs * 16 + (total_q / (kBlockM >> kMaxPackShift) + num_seqs) * 8 + 64;
}

// Entries of the work list when one entry covers `tokens` query tokens, and the bytes the list takes.
int64_t VarlenEntries(const VarlenWork& vw, int64_t tokens) {
    int64_t n = 0;
    for (int64_t s = 0; s < vw.num_seqs; ++s) n += std::max<int64_t>(0, (static_cast<int64_t>(vw.cu_q[s + 1]) - vw.cu_q[s] + tokens - 1) / tokens);
    return n;
}
int64_t VarlenListBytes(const VarlenWork& vw, int64_t tokens) {
    return vw.num_seqs * static_cast<int64_t>(sizeof(int4)) + VarlenEntries(vw, tokens) * static_cast<int64_t>(sizeof(int2));
}

// Every sequence has tokens on both sides. Nothing may be sized by the offsets before this holds: offsets that go up and down
// between the right ends describe any number of entries.
int CheckSequences(const VarlenWork& vw, bool causal) {
    for (int64_t s = 0; s < vw.num_seqs; ++s) {
        const int64_t sq = static_cast<int64_t>(vw.cu_q[s + 1]) - vw.cu_q[s];
        const int64_t skv = static_cast<int64_t>(vw.cu_kv[s + 1]) - vw.cu_kv[s];
        if (sq <= 0 || skv <= 0 || (causal && skv < sq)) {
            return Fail(SCA_INVALID_ARGUMENT, "flash varlen: sequence " + std::to_string(s) + " has S_q=" + std::to_string(sq) +
                                                  ", S_kv=" + std::to_string(skv) + (causal ? " (causal needs 0 < S_q <= S_kv)" : " (both must be > 0)"));
        }
    }
    return SCA_OK;
}

// Builds {first q token, first kv token, S_q, S_kv} per sequence and the (sequence, query block) list, heaviest
// block first, and copies both into the workspace (stream-ordered; the host vector may die on return).
int UploadVarlenWork(const VarlenWork& vw, int tokens_per_entry, int block_n, bool causal, cudaStream_t stream,
                     const int4** seqs_out, const int2** entries_out, int* num_entries_out) {
    const size_t seq_bytes = static_cast<size_t>(vw.num_seqs) * sizeof(int4);
    struct Weighted {
        int2 entry;
        int64_t tiles;
    };
    std::vector<int4> image(static_cast<size_t>(vw.num_seqs));  // the sequences, then the entries
    std::vector<Weighted> list;
    list.reserve(static_cast<size_t>(VarlenEntries(vw, tokens_per_entry)));
    for (int64_t s = 0; s < vw.num_seqs; ++s) {
        const int64_t sq = static_cast<int64_t>(vw.cu_q[s + 1]) - vw.cu_q[s];
        const int64_t skv = static_cast<int64_t>(vw.cu_kv[s + 1]) - vw.cu_kv[s];
        image[static_cast<size_t>(s)] = make_int4(vw.cu_q[s], vw.cu_kv[s], static_cast<int>(sq), static_cast<int>(skv));
        for (int64_t mb = 0; mb * tokens_per_entry < sq; ++mb) {
            int64_t limit = skv;
            if (causal) limit = std::min<int64_t>(limit, std::min<int64_t>(sq, (mb + 1) * tokens_per_entry) + (skv - sq));
            list.push_back({make_int2(static_cast<int>(s), static_cast<int>(mb)), (limit + block_n - 1) / block_n});
        }
    }
    std::stable_sort(list.begin(), list.end(), [](const Weighted& a, const Weighted& b) { return a.tiles > b.tiles; });
    const size_t bytes = seq_bytes + list.size() * sizeof(int2);
    if (vw.workspace == nullptr || static_cast<int64_t>(bytes) > vw.workspace_bytes) {
        return Fail(SCA_INVALID_ARGUMENT, "flash varlen: workspace of " + std::to_string(vw.workspace_bytes) + " bytes is too small (" +
                                              std::to_string(bytes) + " needed)");
    }
    image.resize((bytes + sizeof(int4) - 1) / sizeof(int4));
    int2* entries = reinterpret_cast<int2*>(reinterpret_cast<unsigned char*>(image.data()) + seq_bytes);
    for (size_t i = 0; i < list.size(); ++i) entries[i] = list[i].entry;
    unsigned char* base = static_cast<unsigned char*>(vw.workspace);
    if (int rc = SendToDevice(base, image.data(), bytes, stream, "cudaMemcpyAsync(varlen work list)")) return rc;
    *seqs_out = reinterpret_cast<const int4*>(base);
    *entries_out = reinterpret_cast<const int2*>(base + seq_bytes);
    *num_entries_out = static_cast<int>(list.size());
    return SCA_OK;
}

// A paged KV pool behind a packed batch: f.k / f.v point at one layer's pool [num_blocks, block_size, H_kv, D].
struct PagedWork {
    const int32_t* page_table;
    int64_t num_blocks, block_size, max_blocks_per_seq;
};

int CheckFlash(cudaStream_t stream) {
    if (int rc = CheckLaunch("flash_fwd_sm100_kernel", stream)) return rc;
    // With SCI_ATTENTION_DEBUG_SYNC=1 CheckLaunch has waited for the kernel: a wait that ran out is known now.
    if (DebugSyncEnabled()) {
        int device = 0, code = 0;
        if (cudaGetDevice(&device) == cudaSuccess && sca_flash_status(device, &code) == SCA_OK && code != 0) {
            return Fail(SCA_CUDA_ERROR, "flash attention: the launch gave up waiting on a barrier (role " +
                                            std::to_string(code) + "); its output is invalid");
        }
    }
    return SCA_OK;
}

// How many CTAs share the KV tiles of one item (a power of two; 1: no split). `items` tiles on their own leave SMs idle, and
// each of them is a chain of `tiles` steps of 1.2 / 1.7 / 1.45 us (D=64 / 128 / 256). The exchange costs 4 to 5 / 4 to 5.5 / 6 to
// 8 us: every CTA fetches its rows of all parts, 64 KB at D=128, from the shared memory of the others. So a split has to save
// 4 / 3 / 6 steps; one fewer loses (graph-timed, whole / split: D=128, 8 heads, 100 tokens against 384 9.2 / 9.2, 32 / 8 heads 9.4 /
// 10.8; D=64 against 512 8.7 / 9.7; D=256 11.4 / 13.2). What it gives: D=128, 40 tokens against 3000 44.8 / 18.5, 300 against 1024
// 18.3 / 12.5, 1000 against 1000 (8 heads) 18.2 / 15.6; D=64, 100 against 5000 52 / 19; D=256, 64 against 6000 59.6 / 20.7; chunks of
// 4 sequences of up to 6000 97 / 57.
template <typename T, int DP, int QT, int BN>
int SplitCluster(int64_t items, int64_t tiles) {
    int best = 1;
    int64_t best_steps = tiles - (DP == 64 ? 3 : DP == 128 ? 2 : 5);
    for (int c = 2; c <= kMaxSplit; c *= 2) {
        const int64_t steps = (tiles + c - 1) / c;
        if (items * c > SmCount() || steps >= best_steps) continue;
        if (items > ResidentClusters<T, DP, QT, BN>(c)) continue;
        best = c;
        best_steps = steps;
    }
    return best;
}

template <typename T, int DP, int QT, int BN>
int LaunchFlash(const ScaFlashFwdParams& f, cudaStream_t stream, const VarlenWork* varlen = nullptr,
                const PagedWork* paged = nullptr) {
    using G = FlashGeom<DP, QT, BN>;
    CUtensorMap map_q, map_k, map_v;
    // rows of a query tile: P heads x 128 / P tokens
    int pack_shift = PackShift(f.num_heads / f.num_kv_heads);
    int tiles_per_item = QT;
    if (pack_shift > 0 && !(varlen == nullptr ? PackingPays(f, pack_shift)
                                              : paged != nullptr || PackingPays(*varlen, f, pack_shift))) {
        pack_shift = 0;
    }
    if (varlen != nullptr) {
        while (pack_shift > 0 && VarlenListBytes(*varlen, (QT * kBlockM) >> pack_shift) > varlen->workspace_bytes) --pack_shift;
    }
    if (QT > 1) {
        // fewer tiles than SMs: one tile per CTA (a step of one tile alone takes 0.9 of a step of two)
        const int64_t tokens = kBlockM >> pack_shift;
        const int64_t tiles = (varlen != nullptr ? VarlenEntries(*varlen, tokens) : (f.seq_q + tokens - 1) / tokens * f.batch) *
                              (f.num_heads >> pack_shift);
        if (tiles <= SmCount() && (varlen == nullptr || VarlenListBytes(*varlen, tokens) <= varlen->workspace_bytes)) tiles_per_item = 1;
    }
    if (int rc = MakeMap(&map_q, f.q, f.dtype_id, f.head_dim, f.num_heads, f.seq_q, f.batch, f.q_sh, f.q_ss, f.q_sb, 1 << pack_shift,
                         "q", kBlockM >> pack_shift)) return rc;
    if (paged != nullptr) {
        // the pool as [rows = blocks * block_size, H_kv, D]; one box = one page of one kv head and column block
        const int64_t rows = paged->num_blocks * paged->block_size;
        const int64_t row_elems = f.num_kv_heads * f.head_dim;
        if (int rc = MakeMap(&map_k, f.k, f.dtype_id, f.head_dim, rows, f.num_kv_heads, 1, row_elems, f.head_dim, rows * row_elems,
                             static_cast<int>(paged->block_size), "k pool")) return rc;
        if (int rc = MakeMap(&map_v, f.v, f.dtype_id, f.head_dim, rows, f.num_kv_heads, 1, row_elems, f.head_dim, rows * row_elems,
                             static_cast<int>(paged->block_size), "v pool")) return rc;
    } else
    if (int rc = MakeMap(&map_k, f.k, f.dtype_id, f.head_dim, f.seq_kv, f.num_kv_heads, f.batch, f.k_ss, f.k_sh, f.k_sb, BN, "k")) return rc;
    if (paged == nullptr) {
        if (PvFormat<T>::kConvertV && (!Aligned16(f.v) || f.v_sb % 8 != 0 || f.v_sh % 8 != 0 || f.v_ss % 8 != 0)) {
            return Fail(SCA_INVALID_ARGUMENT, "flash attention: v must be 16-byte aligned with strides that are multiples of 8 elements");
        }
        if (int rc = MakeMap(&map_v, f.v, f.dtype_id, f.head_dim, f.seq_kv, f.num_kv_heads, f.batch, f.v_ss, f.v_sh, f.v_sb, G::kVKeys, "v")) return rc;
    }

    FlashKernelParams p{};
    p.out = f.out;
    p.lse = f.return_lse ? f.lse : nullptr;
    p.error_word = ErrorWordForCurrentDevice();
    p.seq_q = static_cast<int>(f.seq_q);
    p.seq_kv = static_cast<int>(f.seq_kv);
    p.heads = static_cast<int>(f.num_heads);
    p.kv_heads = static_cast<int>(f.num_kv_heads);
    p.head_dim = static_cast<int>(f.head_dim);
    p.batch = static_cast<int>(f.batch);
    p.o_sb = f.o_sb;
    p.o_sh = f.o_sh;
    p.o_ss = f.o_ss;
    p.wide_stores = (reinterpret_cast<uintptr_t>(f.out) & 31u) == 0 && f.o_sb % 16 == 0 && f.o_sh % 16 == 0 && f.o_ss % 16 == 0;
    p.scale_log2 = f.scale * kLog2e;
    p.causal = f.causal ? 1 : 0;
    p.diagonal = static_cast<int>(f.causal ? f.diagonal : 0);
    p.pack_shift = pack_shift;
    p.tiles_per_item = tiles_per_item;
    const int item_tokens = (tiles_per_item * kBlockM) >> pack_shift;
    p.m_blocks = static_cast<int>((f.seq_q + item_tokens - 1) / item_tokens);
    int64_t most_keys = f.seq_kv;  // of a sequence
    if (varlen != nullptr) {
        most_keys = 0;
        for (int64_t i = 0; i < varlen->num_seqs; ++i) most_keys = std::max<int64_t>(most_keys, static_cast<int64_t>(varlen->cu_kv[i + 1]) - varlen->cu_kv[i]);
        if (int rc = UploadVarlenWork(*varlen, item_tokens, BN, f.causal != 0, stream, &p.seqs, &p.entries, &p.num_entries)) return rc;
    }
    const int64_t ctas = (varlen != nullptr ? static_cast<int64_t>(p.num_entries) : static_cast<int64_t>(p.m_blocks) * p.batch) *
                         (p.heads >> pack_shift);
    if (ctas <= 0 || ctas > 0x7fffffffLL) {
        return Fail(SCA_INVALID_ARGUMENT, "flash attention: grid of " + std::to_string(ctas) + " blocks is out of range");
    }
    p.cluster = tiles_per_item == 1 ? SplitCluster<T, DP, QT, BN>(ctas, (most_keys + BN - 1) / BN) : 1;
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(ctas, SmCount()));  // one persistent CTA per SM
    constexpr unsigned threads = FlashThreads<T, DP, QT>();
    if (paged != nullptr) {
        p.page_table = paged->page_table;
        p.max_blocks_per_seq = static_cast<int>(paged->max_blocks_per_seq);
        p.num_kv_blocks = static_cast<int>(paged->num_blocks);
        p.block_size = static_cast<int>(paged->block_size);
        p.block_shift = 0;
        while ((1 << p.block_shift) < p.block_size) ++p.block_shift;
        if (p.cluster > 1) {
            if (int rc = LaunchSplit<T, DP, QT, BN, true, true>(ctas, stream, map_q, map_k, map_v, p)) return rc;
            return CheckFlash(stream);
        }
        const void* fn = reinterpret_cast<const void*>(&flash_fwd_sm100_kernel<T, DP, QT, BN, true, true>);
        if (int rc = EnsureDynamicSmem(fn, G::kSmemBytes, "flash_fwd_sm100_kernel")) return rc;
        LaunchDependent(flash_fwd_sm100_kernel<T, DP, QT, BN, true, true>, grid, threads, G::kSmemBytes, stream, 1, map_q, map_k, map_v, p);
    } else if (varlen != nullptr) {
        if (p.cluster > 1) {
            if (int rc = LaunchSplit<T, DP, QT, BN, true, false>(ctas, stream, map_q, map_k, map_v, p)) return rc;
            return CheckFlash(stream);
        }
        const void* fn = reinterpret_cast<const void*>(&flash_fwd_sm100_kernel<T, DP, QT, BN, true>);
        if (int rc = EnsureDynamicSmem(fn, G::kSmemBytes, "flash_fwd_sm100_kernel")) return rc;
        LaunchDependent(flash_fwd_sm100_kernel<T, DP, QT, BN, true>, grid, threads, G::kSmemBytes, stream, 1, map_q, map_k, map_v, p);
    } else {
        if (p.cluster > 1) {
            if (int rc = LaunchSplit<T, DP, QT, BN, false, false>(ctas, stream, map_q, map_k, map_v, p)) return rc;
            return CheckFlash(stream);
        }
        const void* fn = reinterpret_cast<const void*>(&flash_fwd_sm100_kernel<T, DP, QT, BN, false>);
        if (int rc = EnsureDynamicSmem(fn, G::kSmemBytes, "flash_fwd_sm100_kernel")) return rc;
        LaunchDependent(flash_fwd_sm100_kernel<T, DP, QT, BN, false>, grid, threads, G::kSmemBytes, stream, 1, map_q, map_k, map_v, p);
    }
    return CheckFlash(stream);
}

int ValidateFlash(const ScaFlashFwdParams* params) {
    if (params == nullptr || params->q == nullptr || params->k == nullptr || params->v == nullptr ||
        params->out == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "flash attention: null tensor pointer");
    }
    const ScaFlashFwdParams& f = *params;
    if (f.dtype_id != SCA_DTYPE_F16 && f.dtype_id != SCA_DTYPE_BF16) {
        return Fail(SCA_INVALID_ARGUMENT, "flash attention: only fp16/bf16 are instantiated (dtype_id=" +
                                              std::to_string(f.dtype_id) + "); use the naive or tiled backend for FP32");
    }
    if (f.batch < 1 || f.num_heads < 1 || f.num_kv_heads < 1 || f.seq_q < 1 || f.seq_kv < 1 ||
        f.num_heads % f.num_kv_heads != 0) {
        return Fail(SCA_INVALID_ARGUMENT, "flash attention: invalid geometry");
    }
    if (f.seq_q > 0x7fffff00LL || f.seq_kv > 0x7fffff00LL) {
        return Fail(SCA_INVALID_ARGUMENT, "flash attention: sequence length exceeds the 32-bit tile index range");
    }
    if (!(f.scale > 0.0f)) return Fail(SCA_INVALID_ARGUMENT, "flash attention: scale must be > 0");
    if (f.return_lse && f.lse == nullptr) return Fail(SCA_INVALID_ARGUMENT, "flash attention: return_lse without a buffer");
    if (!Aligned16(f.out) || f.o_sb % 8 != 0 || f.o_sh % 8 != 0 || f.o_ss % 8 != 0) {
        return Fail(SCA_INVALID_ARGUMENT, "flash attention: out must be 16-byte aligned with strides that are multiples of 8 elements");
    }
    return SCA_OK;
}

template <typename T>
int LaunchFlashTyped(const ScaFlashFwdParams& f, cudaStream_t stream, const VarlenWork* varlen = nullptr,
                     const PagedWork* paged = nullptr) {
    // head dims that are not a multiple of 64 run on the next padded geometry: the TMA unit
    // zero-fills the missing columns of Q, K and V, which leaves S and the real columns of O unchanged
    switch (f.head_dim) {
        case 32:
        case 64: return LaunchFlash<T, 64, 2, 128>(f, stream, varlen, paged);
        case 96:
        case 128: return LaunchFlash<T, 128, 2, 128>(f, stream, varlen, paged);
        case 160:
        case 192:
        case 256: return LaunchFlash<T, 256, 1, 128>(f, stream, varlen, paged);
        default: break;
    }
    return Fail(SCA_INVALID_ARGUMENT, "flash attention: head_dim=" + std::to_string(f.head_dim) + " is not instantiated");
}

}  // namespace
}  // namespace sca_b200

using namespace sca_b200;

extern "C" int sca_flash_status(int device_id, int32_t* status_out) {
    if (status_out == nullptr) return Fail(SCA_INVALID_ARGUMENT, "flash status: null output");
    if (device_id < 0 || device_id >= kMaxStatusDevices) {
        return Fail(SCA_INVALID_ARGUMENT, "flash status: device index " + std::to_string(device_id) + " is out of range");
    }
    int* host = nullptr;
    ErrorWords(&host);
    // the kernel writes the word over the bus with a plain store; the host takes it with one atomic exchange
    *status_out = host != nullptr ? __atomic_exchange_n(host + device_id, 0, __ATOMIC_ACQ_REL) : 0;
    return SCA_OK;
}

extern "C" long long sca_flash_smem_bytes_for(int head_dim, long long elem_bytes, int block_m, int block_n,
                                              int stages) {
    if (head_dim <= 0 || elem_bytes <= 0 || block_m <= 0 || block_n <= 0 || stages <= 0) return -1;
    const long long q = static_cast<long long>(block_m) * head_dim * elem_bytes;
    const long long kv = static_cast<long long>(block_n) * head_dim * elem_bytes * stages;
    return q + 2 * kv + 1024;
}

extern "C" int sca_launch_flash_fwd(const ScaFlashFwdParams* params, void* stream) {
    ClearError();
    if (int rc = ValidateFlash(params)) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return params->dtype_id == SCA_DTYPE_F16 ? LaunchFlashTyped<__half>(*params, s)
                                             : LaunchFlashTyped<__nv_bfloat16>(*params, s);
}

extern "C" long long sca_flash_varlen_workspace_bytes(int64_t num_seqs, int64_t total_q) {
    if (num_seqs < 1 || total_q < 1) return -1;
    return VarlenWorkspaceBytes(num_seqs, total_q);
}

// Packed variable-length prefill in ONE launch (the reference loops over the sequences on the host,
// src/backends/flash/flash_backend.cpp:312-363): the persistent kernel's work list simply spans all sequences.
extern "C" int sca_launch_flash_varlen(const ScaFlashVarlenParams* params, void* stream) try {
    ClearError();
    if (params == nullptr || params->cu_seqlens_q == nullptr || params->cu_seqlens_kv == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "flash varlen: null parameter block or host offsets");
    }
    const ScaFlashVarlenParams& x = *params;
    if (x.num_seqs < 1 || x.total_q < 1 || x.total_kv < 1) return Fail(SCA_INVALID_ARGUMENT, "flash varlen: empty batch");
    if (x.cu_seqlens_q[0] != 0 || x.cu_seqlens_kv[0] != 0 || x.cu_seqlens_q[x.num_seqs] != x.total_q ||
        x.cu_seqlens_kv[x.num_seqs] != x.total_kv) {
        return Fail(SCA_INVALID_ARGUMENT, "flash varlen: offsets must start at 0 and end at the token totals");
    }
    ScaFlashFwdParams f{};
    f.q = x.q;
    f.k = x.k;
    f.v = x.v;
    f.out = x.out;
    f.batch = 1;
    f.num_heads = x.num_heads;
    f.num_kv_heads = x.num_kv_heads;
    f.seq_q = x.total_q;
    f.seq_kv = x.total_kv;
    f.head_dim = x.head_dim;
    f.q_ss = x.num_heads * x.head_dim;
    f.q_sh = x.head_dim;
    f.q_sb = x.total_q * f.q_ss;
    f.k_ss = x.num_kv_heads * x.head_dim;
    f.k_sh = x.head_dim;
    f.k_sb = x.total_kv * f.k_ss;
    f.v_ss = f.k_ss;
    f.v_sh = f.k_sh;
    f.v_sb = f.k_sb;
    f.o_ss = f.q_ss;
    f.o_sh = f.q_sh;
    f.o_sb = f.q_sb;
    f.scale = x.scale;
    f.causal = x.causal;
    f.dtype_id = x.dtype_id;
    if (int rc = ValidateFlash(&f)) return rc;
    VarlenWork vw{x.cu_seqlens_q, x.cu_seqlens_kv, x.num_seqs, x.workspace, x.workspace_bytes};
    if (int rc = CheckSequences(vw, f.causal != 0)) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return f.dtype_id == SCA_DTYPE_F16 ? LaunchFlashTyped<__half>(f, s, &vw)
                                       : LaunchFlashTyped<__nv_bfloat16>(f, s, &vw);
} catch (const std::exception& e) {  // host memory for the work list
    return Fail(SCA_CUDA_ERROR, std::string("flash varlen: on the host: ") + e.what());
}

extern "C" int sca_launch_flash_paged(const ScaFlashPagedParams* params, void* stream) try {
    ClearError();
    if (params == nullptr || params->cu_seqlens_q == nullptr || params->seq_lens_kv == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "flash paged: null parameter block or host lengths");
    }
    const ScaFlashPagedParams& x = *params;
    if (x.q == nullptr || x.out == nullptr || x.k_pool == nullptr || x.v_pool == nullptr || x.page_table == nullptr) {
        return Fail(SCA_INVALID_ARGUMENT, "flash paged: null tensor pointer");
    }
    if (x.num_seqs < 1 || x.total_q < 1) return Fail(SCA_INVALID_ARGUMENT, "flash paged: empty batch");
    if (x.cu_seqlens_q[0] != 0 || x.cu_seqlens_q[x.num_seqs] != x.total_q) {
        return Fail(SCA_INVALID_ARGUMENT, "flash paged: query offsets must start at 0 and end at total_q");
    }
    if (x.block_size != 8 && x.block_size != 16 && x.block_size != 32 && x.block_size != 64) {
        return Fail(SCA_INVALID_ARGUMENT, "flash paged: block_size=" + std::to_string(x.block_size) +
                                              " (pages are loaded as boxes of 8, 16, 32 or 64 tokens)");
    }
    if (x.num_blocks < 1 || x.max_blocks_per_seq < 1 || x.num_blocks * x.block_size > 0x7fffff00LL) {
        return Fail(SCA_INVALID_ARGUMENT, "flash paged: invalid pool geometry");
    }
    // kv offsets for the shared work-list builder: only the lengths are used on the device
    std::vector<int32_t> cu_kv(static_cast<size_t>(x.num_seqs) + 1, 0);
    for (int64_t s = 0; s < x.num_seqs; ++s) {
        const int64_t have = x.seq_lens_kv[s];
        if (have < 1 || have > x.max_blocks_per_seq * x.block_size) {
            return Fail(SCA_INVALID_ARGUMENT, "flash paged: sequence " + std::to_string(s) + " has " + std::to_string(have) +
                                                  " tokens in the cache (the page-table row holds " +
                                                  std::to_string(x.max_blocks_per_seq * x.block_size) + ")");
        }
        const int64_t next = static_cast<int64_t>(cu_kv[static_cast<size_t>(s)]) + have;
        if (next > 0x7fffffffLL) return Fail(SCA_INVALID_ARGUMENT, "flash paged: more than 2^31 cached tokens in one call");
        cu_kv[static_cast<size_t>(s) + 1] = static_cast<int32_t>(next);
    }
    ScaFlashFwdParams f{};
    f.q = x.q;
    f.k = x.k_pool;
    f.v = x.v_pool;
    f.out = x.out;
    f.batch = 1;
    f.num_heads = x.num_heads;
    f.num_kv_heads = x.num_kv_heads;
    f.seq_q = x.total_q;
    f.seq_kv = cu_kv.back();
    f.head_dim = x.head_dim;
    f.q_ss = x.num_heads * x.head_dim;
    f.q_sh = x.head_dim;
    f.q_sb = x.total_q * f.q_ss;
    f.o_ss = f.q_ss;
    f.o_sh = f.q_sh;
    f.o_sb = f.q_sb;
    f.scale = x.scale;
    f.causal = x.causal;
    f.dtype_id = x.dtype_id;
    if (int rc = ValidateFlash(&f)) return rc;
    VarlenWork vw{x.cu_seqlens_q, cu_kv.data(), x.num_seqs, x.workspace, x.workspace_bytes};
    if (int rc = CheckSequences(vw, f.causal != 0)) return rc;
    PagedWork pw{x.page_table, x.num_blocks, x.block_size, x.max_blocks_per_seq};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (f.dtype_id) {
        case SCA_DTYPE_F16: return LaunchFlashTyped<__half>(f, s, &vw, &pw);
        case SCA_DTYPE_BF16: return LaunchFlashTyped<__nv_bfloat16>(f, s, &vw, &pw);
        default: break;
    }
    return Fail(SCA_INVALID_ARGUMENT, "flash paged: unsupported dtype id");
} catch (const std::exception& e) {  // host memory for the work list
    return Fail(SCA_CUDA_ERROR, std::string("flash paged: on the host: ") + e.what());
}

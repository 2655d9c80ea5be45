// Flash prefill for sm_100a: O = softmax(scale * Q K^T + mask) V with the score matrix kept on chip.
//
// Stands in for the reference's flash_fwd_kernel (src/backends/flash/flash_fwd_impl.cuh:45-279, an
// sm_80 mma.sync + ldmatrix + cp.async design with 64x64 tiles and one CTA-wide barrier pair per
// tile). Same arithmetic contract - fp16/bf16 inputs, fp32 accumulation, online softmax through
// exp2, bottom-right aligned causal mask, GQA, optional log-sum-exp - on a Blackwell execution plan:
//
//   * one persistent CTA per SM walks a list of work items; an item is 256 query rows of one batch element and kv
//     head - one query head, or up to four that share the kv head, interleaved token by token - as two 128-row tiles that
//     ping-pong, so the tensor core works on one tile while the other tile's softmax runs;
//   * warp 0 is the TMA producer: Q tiles once, then K_j, V_j, K_j+1, ... into a ring of 128-byte
//     swizzled shared-memory slots, each guarded by a full/empty mbarrier pair. Loads are plain
//     per-CTA tensor loads (one CTA, one destination); K/V reuse between the CTAs of a kv head comes
//     from L2. Rows past the end of a sequence are zero-filled by the TMA unit;
//   * warp 1 issues every tcgen05.mma from one thread: S_t = Q_t K_j^T (both operands in shared
//     memory, K-major) into tensor memory, and O_t += P_t V_j with P_t read from tensor memory and
//     V_j as an MN-major shared-memory operand (no transposition of V anywhere);
//   * four warps per query tile are its softmax group, one thread per query row: they read their S row from tensor
//     memory once, exponentiate against the reference point the row already has, keep the running sum in registers
//     and write P to tensor memory as packed 16-bit values, handed over in two pieces so that P V starts under the last
//     exponentials. The reference point moves (and O and the sum are rescaled) only when a row exceeds it by more
//     than 2^8; the final division by the row sum absorbs the stale reference point exactly;
//   * bf16: two to four more warps rewrite each V tile in shared memory as fp16 (see PvFormat);
//   * tensor memory, 512 columns: at D=128 S_0 | S_1 | O_0 | O_1 take them all and P_t lies over S_t, so that the next
//     scores follow P V. Up to D=64, and above 128 with its one query tile, P_t has columns of its own (see FlashGeom).
//
// Packed variable-length batches run on the same kernel: the work list then holds (sequence, query block)
// entries and every item carries its sequence's lengths and token offsets (see sca_launch_flash_varlen).
//
// Every wait on an mbarrier is bounded (sm100.cuh): on expiry the role raises a CTA-wide abort flag,
// the kernel records a code in a host-visible word, frees its tensor memory and returns.
//
// FLOPs per (query, key) pair that is visible: 4 * D. Algorithmic HBM bytes: Q + K + V + O once.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "kv_ring.cuh"
#include "sm100.cuh"

namespace sca_b200 {
namespace flash {

using namespace sm100;

constexpr int kBlockM = 128;

__device__ __forceinline__ float2 UnpackBf16(uint32_t v) {
    return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
// bf16 inputs: the probabilities are handed to the P V product as fp16, not bf16. They lie in [0, 2^8], where fp16
// resolves 2^-11 relative against 2^-8 - with bf16 the rounding of P alone costs about 1e-3 of relative L2 error in
// the output. The tensor core wants both operands of one product in the same 16-bit format (a descriptor that mixes
// them raises "illegal instruction" on sm_100a), so for bf16 inputs V is rewritten as fp16 in shared memory, tile by
// tile, by warps that do nothing else (values beyond the fp16 range saturate). A copy of V made by a kernel of its own
// ahead of the launch is no faster at the largest sizes (B=4, S=4096, D=128: 15 us of copying and a 5 us gap in 537 us,
// against 523 us) and costs a short prompt a second launch and an allocation (S=203: 35 against 27 us).
template <typename T>
struct PvFormat {
    using type = __half;
    static constexpr bool kConvertV = std::is_same<T, __nv_bfloat16>::value;
};
constexpr int kTmemColumns = 512;
constexpr float kRescaleThreshold = 8.0f;  // log2 domain: P stays <= 2^8
constexpr int kMaxSplit = 8;               // CTAs that share an item at most (the portable cluster size)

// DP: padded head dim (64 / 128 / 256); QT: query tiles per CTA; BN: keys per KV tile.
// 64 and 128 run two query tiles; 256 needs 256 TMEM columns for O, so it runs one.
template <int DP, int QT, int BN>
struct FlashGeom {
    static constexpr int kKBlocks = DP / 64;               // 64-element (128-byte) column blocks per row
    static constexpr int kQBlockBytes = kBlockM * 128;      // one column block of a query tile
    static constexpr int kQTileBytes = kKBlocks * kQBlockBytes;
    // K/V ring. A tile of D=256 takes two slots: K in halves of its columns, V in halves of its keys, each freed when its
    // half of the products is done.
    static constexpr int kParts = RingOf(DP).parts;
    static constexpr int kKBlockBytes = BN * 128;           // one column block of K in a slot
    static constexpr int kVKeys = BN / kParts;              // keys of V in a slot
    static constexpr int kVBlockBytes = kVKeys * 128;       // one column block of V in a slot
    static constexpr int kSlotBytes = BN * DP * 2 / kParts;
    static constexpr int kSlots = RingOf(DP).slots;
    static constexpr int kBarrierBytes = 512;
    static constexpr int kSmemBytes = 1024 + QT * kQTileBytes + kSlots * kSlotBytes + kBarrierBytes;
    static constexpr int kSCol = 0;                         // S_t at kSCol + t * BN
    static constexpr int kOCol = 256;                       // O_t at kOCol + t * DP
    // P_t has columns of its own wherever O leaves room for them: S_t(j+1) then goes out as soon as S_t(j) is in registers
    // and is there when the softmax group comes back for it, instead of following P_t(j) V_j. At D=128 there is no room.
    // us in a lasting load, P over S / apart: D=64 B=3 S=2900 without a mask 310 / 297, four prompts of 4096 412 / 390, 10
    // ragged ones 415 / 371, B=1 S=800 18.5 / 16.5. D=256 went from 64-key tiles with two score buffers (where the score
    // products run at 3/4 of their rate) to 128 keys: B=1 S=3000 168 / 149, B=2 without a mask 655 / 545. A step takes 2960
    // clocks then, 2420 for fp16, 2048 of them products; 448 KB go through shared memory (Q and K for the scores, V, the loads,
    // V rewritten), 320 KB where V is not rewritten.
    static constexpr bool kOwnP = RingOf(DP).scores_ahead;
    static constexpr int kPCol = !kOwnP ? kSCol : DP == 64 ? 384 : 128;  // P_t at kPCol + t * kPStride
    static constexpr int kPStride = kOwnP ? BN / 2 : BN;
    static_assert(BN == 128 && (DP == 256 ? QT == 1 : QT == 2), "geometry");
    static_assert(kOCol + QT * DP <= kTmemColumns && kPCol + QT * kPStride <= kTmemColumns, "tensor memory budget");
    static_assert(kSmemBytes <= 232448, "exceeds the 227 KiB per-CTA limit");
};

struct FlashKernelParams {
    void* out;
    float* lse;
    int* error_word; // host-visible; non-zero after a wait expired
    int seq_q, seq_kv, heads, kv_heads, head_dim, batch;
    int64_t o_sb, o_sh, o_ss;
    bool wide_stores;  // every row of `out` starts on a 32-byte boundary
    float scale_log2;
    int causal;
    int diagonal;
    int m_blocks;
    int pack_shift;      // log2 of the query heads that share a tile (see "Packed heads")
    int tiles_per_item;  // query tiles a work item fills (at most QT)
    // packed variable-length batches (null for dense [B, H, S, D] problems): seqs[s] = {first query token,
    // first key token, S_q, S_kv}; entries[e] = {sequence, query block}, heaviest first
    const int4* seqs;
    const int2* entries;
    int num_entries;
    // paged K/V (kPaged kernels): the K/V tensor maps cover one layer's pool viewed as [blocks * block_size, H_kv, D]
    // with a box of block_size rows; a KV tile is assembled page by page through the sequence's page-table row
    const int32_t* page_table;   // device [num_seqs, max_blocks_per_seq], -1 = unmapped
    int max_blocks_per_seq, num_kv_blocks;
    int block_size, block_shift;  // block_size = 1 << block_shift
    int cluster;  // kSplit kernels: CTAs that share an item
};

// 16 elements of an output row: one 32-byte store where every row starts on a 32-byte boundary, else two of 16 bytes. A
// thread writes a row of its own, so each store of a warp touches 32 separate rows and takes the load/store unit 32 turns
// whatever its width; writing O with 16-byte stores took 3500 clocks per tile at D=128, as long as one KV step. Lasting load,
// 16 / 32 bytes: B=2, S=1500 57.5 / 51.2 us, 40 prompts of 16 to 400 77.2 / 66.5, four of 4096 575 / 569, D=256 S=3000 159 / 149.
template <typename T>
__device__ __forceinline__ void StoreRow16(T* dst, const uint32_t (&v)[8], bool wide) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                     "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    } else {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}

// KV tiles a query tile of `tokens` tokens starting at token m0 of its sequence has to visit.
template <int BN>
__device__ __forceinline__ int TilesFor(int m0, int tokens, int seq_q, int seq_kv, int causal, int diagonal) {
    if (m0 >= seq_q) return 0;
    int64_t limit = seq_kv;
    if (causal) limit = min(limit, static_cast<int64_t>(min(m0 + tokens, seq_q)) + diagonal);
    if (limit <= 0) return 0;
    return static_cast<int>((limit + BN - 1) / BN);
}

// Warps that rewrite V as fp16. At D=256 a step has twice the bytes and its slots are the scarce thing: two warps 173 us,
// three 172, four 146 (B=1, S=3000, lasting load). One warp is too few at D=128 (four prompts of 4096: 632 against 595).
template <typename T, int DP>
constexpr int ConverterWarps() {
    return PvFormat<T>::kConvertV ? RingOf(DP).converters : 0;
}
// Warps of a CTA: 0 TMA and tensor-memory owner, 1 MMA, 2 and 3 V converters (idle for fp16), then four per query tile for
// the softmax, then what converters are left.
constexpr int kFirstSoftmax = 4;
template <typename T, int DP, int QT>
constexpr int FlashThreads() {
    return 32 * (kFirstSoftmax + 4 * QT + (ConverterWarps<T, DP>() > 2 ? ConverterWarps<T, DP>() - 2 : 0));
}

// kVarlen: the work list comes from the (sequence, query block) table of a packed ragged batch; otherwise it is
// computed from the dense [B, H, S, D] geometry and every per-sequence quantity is a launch constant.
// kPaged (only with kVarlen): K and V of a sequence are scattered over the pages of a KV pool.
// kSplit: the CTAs of a cluster share one item of one query tile. Each takes a part of its KV tiles, and the parts are merged
// through distributed shared memory at the end (SplitCluster says when).
template <typename T, int DP, int QT, int BN, bool kVarlen, bool kPaged = false, bool kSplit = false>
__global__ void __launch_bounds__(FlashThreads<T, DP, QT>(), 1)
flash_fwd_sm100_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const FlashKernelParams p) {
    using G = FlashGeom<DP, QT, BN>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem_base = (SmemAddr(smem_raw) + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (smem_base - SmemAddr(smem_raw));

    const uint32_t q_smem = smem_base;
    const uint32_t ring_smem = smem_base + QT * G::kQTileBytes;
    const uint32_t bar_base = ring_smem + G::kSlots * G::kSlotBytes;
    auto bar = [&](int i) { return bar_base + 8u * i; };
    // Barriers. A wait names a phase by its parity, so it is sound where the role knows that the phase before is over and
    // that the one after cannot be. For all but o_done the role waits for every phase in turn, and the next one takes an
    // arrival that this role (or one that waits for it) makes later. Where P lies over S, o_done is waited for where O moves
    // and at the end of an item only. The phase before it: its product went out ahead of scores the softmax has waited for
    // since. The phase after: its product wants a P that this group has yet to write.
    constexpr int kTiles = QT;
    constexpr int kQFull = 0;                       // [kTiles]
    constexpr int kKvFull = kQFull + kTiles;        // [2 * kSlots], see RingFullBarrier
    constexpr int kKvEmpty = kKvFull + 2 * G::kSlots;   // [kSlots]
    constexpr int kSFull = kKvEmpty + G::kSlots;    // [kTiles]
    constexpr int kPFull = kSFull + kTiles;         // [kTiles]
    constexpr int kODone = kPFull + kTiles;         // [kTiles]
    constexpr int kQEmpty = kODone + kTiles;        // [kTiles]
    constexpr int kOFree = kQEmpty + kTiles;        // [kTiles]
    constexpr int kPLast = kOFree + kTiles;         // [kTiles]
    constexpr int kVReady = kPLast + kTiles;        // [kSlots] bf16: V tile rewritten as fp16 in place
    constexpr int kSRead = kVReady + G::kSlots;     // [kTiles] kOwnP: scores in registers
    constexpr int kNumBars = kSRead + kTiles;
    auto full_bar = [&](bool is_v, uint32_t slot) { return bar(kKvFull + RingFullBarrier(is_v, static_cast<int>(slot), G::kSlots)); };
    using PT = typename PvFormat<T>::type;
    constexpr bool kCvtInKernel = PvFormat<T>::kConvertV;
    constexpr int kConverters = ConverterWarps<T, DP>();
    // P is handed over in two pieces: the first kPEarly keys let P V start while the rest is still in the softmax
    constexpr int kPEarly = DP == 256 ? 64 : 96;
    static_assert(!kPaged || kVarlen, "paged K/V runs on the packed work list");
    static_assert(kNumBars * 8 + 16 <= G::kBarrierBytes, "barrier area too small");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + (bar_base - smem_base) + kNumBars * 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    // paged K/V: which pages of a KV tile are mapped (bit i = i-th page of the tile), written by the producer when
    // it loads the K tile and read by the softmax groups; indexed by the CTA's running KV-tile count
    constexpr int kValidRing = 16;
    volatile uint32_t* valid_ring = reinterpret_cast<volatile uint32_t*>(tmem_slot + 2);
    static_assert(kNumBars * 8 + 8 + kValidRing * 4 <= G::kBarrierBytes, "barrier area too small");

    constexpr bool kOwnP = G::kOwnP;
    constexpr int kParts = G::kParts;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    constexpr int kEndSoftmax = kFirstSoftmax + 4 * QT;
    const int converter = warp < kFirstSoftmax ? warp - 2 : warp >= kEndSoftmax ? warp - kEndSoftmax + 2 : -1;

    // ---- Packed heads: P = 1 << pack_shift query heads of one kv head share a query tile (row r = token m0 + r / P, head
    // h + r % P). They read the same K/V tiles, so the rows of a short or ragged chunk fill up with other heads instead
    // of padding, and the two tiles of a causal item lie 128 / P tokens apart instead of 128, so that both need the same
    // number of KV tiles in all but one item of P (a tile left alone for a step has nothing to overlap with). ----
    // ---- work items: (query block, batch * packed head), heaviest causal blocks first. The list is dealt to the
    // CTAs in rounds of gridDim.x items, every other round in reverse CTA order, so that the CTA that got
    // the heaviest item of one round gets the lightest of the next (the static schedule then ends within
    // about one KV tile of each other on all SMs). Every role of a CTA walks the same sequence. ----------
    const int tile_tokens = kBlockM >> p.pack_shift;
    const int packed_heads = p.heads >> p.pack_shift;
    const int bh_count = p.batch * packed_heads;
    const int total_items = kVarlen ? p.num_entries * packed_heads : p.m_blocks * bh_count;
    struct Item {
        int b, h, h_kv;               // h: first of the item's query heads
        int seq;                      // index of the sequence (row of the page table); 0 for dense problems
        int q_tok0, kv_tok0;          // first row of the sequence in the packed tensors (0 for dense problems)
        int seq_q, seq_kv, diagonal;  // of this item's sequence
        int m0[kTiles];               // first token of each tile, relative to the sequence
        int ntiles[kTiles];
        int n_max;
        int first_tile;               // kSplit: this CTA's first KV tile; 0 otherwise
    };
    auto decode_item = [&](int idx) {
        Item w;
        int mb;
        if constexpr (kVarlen) {
            const int2 entry = p.entries[idx / packed_heads];
            const int4 seq = p.seqs[entry.x];
            mb = entry.y;
            w.seq = entry.x;
            w.b = 0;
            w.h = (idx % packed_heads) << p.pack_shift;
            w.q_tok0 = seq.x;
            w.kv_tok0 = seq.y;
            w.seq_q = seq.z;
            w.seq_kv = seq.w;
            w.diagonal = p.causal ? seq.w - seq.z : 0;  // bottom-right aligned mask
        } else {
            mb = p.m_blocks - 1 - idx / bh_count;
            w.seq = 0;
            const int bh = idx % bh_count;
            w.b = bh / packed_heads;
            w.h = (bh % packed_heads) << p.pack_shift;
            w.q_tok0 = 0;
            w.kv_tok0 = 0;
            w.seq_q = p.seq_q;
            w.seq_kv = p.seq_kv;
            w.diagonal = p.diagonal;
        }
        w.h_kv = w.h / (p.heads / p.kv_heads);
        w.n_max = 0;
#pragma unroll
        for (int t = 0; t < kTiles; ++t) {
            w.m0[t] = (mb * p.tiles_per_item + t) * tile_tokens;
            w.ntiles[t] = t < p.tiles_per_item ? TilesFor<BN>(w.m0[t], tile_tokens, w.seq_q, w.seq_kv, p.causal, w.diagonal) : 0;
            w.n_max = max(w.n_max, w.ntiles[t]);
        }
        w.first_tile = 0;
        if constexpr (kSplit) {
            const int share = (w.n_max + p.cluster - 1) / p.cluster;
            w.first_tile = min(static_cast<int>(ClusterRank()) * share, w.n_max);
            w.n_max = w.ntiles[0] = min(share, w.n_max - w.first_tile);
        }
        return w;
    };
    const int rounds = kSplit ? 1 : (total_items + gridDim.x - 1) / gridDim.x;
    auto item_of_round = [&](int r) {  // -1: this CTA has no item in round r (only in the last, partial round)
        if constexpr (kSplit) return static_cast<int>(blockIdx.x) / p.cluster;
        const int pos = (r & 1) ? static_cast<int>(gridDim.x - 1 - blockIdx.x) : static_cast<int>(blockIdx.x);
        const int idx = r * static_cast<int>(gridDim.x) + pos;
        return idx < total_items ? idx : -1;
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < kTiles; ++i) {
            MbarInit<1>(bar(kQFull + i));
            MbarInit<1>(bar(kQEmpty + i));
            MbarInit<1>(bar(kSFull + i));
            MbarInit<4>(bar(kPFull + i));
            MbarInit<4>(bar(kPLast + i));
            MbarInit<1>(bar(kODone + i));
            MbarInit<4>(bar(kOFree + i));
            MbarInit<4>(bar(kSRead + i));
        }
        for (int i = 0; i < 2 * G::kSlots; ++i) MbarInit<1>(bar(kKvFull + i));
        for (int i = 0; i < G::kSlots; ++i) {
            MbarInit<1>(bar(kKvEmpty + i));
            if constexpr (kCvtInKernel) MbarInit<32 * kConverters>(bar(kVReady + i));
        }
        *abort_flag = 0;
        FenceBarrierInit();
    }
    if (warp == 0) {
        __syncwarp();  // lane 0 comes from the initialisation; the instruction wants the whole warp
        TmemAlloc(SmemAddr(tmem_slot), kTmemColumns);
        TmemRelinquish();
    }
    TcFenceBefore();
    __syncthreads();
    TcFenceAfter();
    const uint32_t tmem_base = *tmem_slot;
    BeginAfterPredecessor();

    bool failed = false;
    // kSplit: a row of a CTA's part is {O[DP], m, l}, padded so that neighbouring rows lie on different banks
    constexpr int kPartLd = DP + 4;
    static_assert(!kSplit || kBlockM * kPartLd * 4 <= G::kSlots * G::kSlotBytes, "a part has to fit the ring");

    if (warp == 0 && kPaged) {
        // ================================ TMA producer, paged K/V ===================================
        // The whole warp walks the work list: the lanes fetch the page ids of a tile together (one coalesced read
        // of the table row), lane 0 waits for the ring slot and one lane issues a box load per page and column block. The
        // loads decide at D=256, so what can be known at compile time about them is: with run-time block counts a box took
        // 170 clocks to issue instead of 90 (20 chunks, D=256: 1790 us, 1032 now, 1094 with 64-key tiles). A
        // page that is unmapped (entry < 0 or >= num_kv_blocks) is loaded from beyond the pool, i.e. zero-filled,
        // and its columns are masked in the softmax through valid_ring.
        if (lane == 0) {
            PrefetchTensorMap(&map_q);
            PrefetchTensorMap(&map_k);
            PrefetchTensorMap(&map_v);
        }
        uint32_t q_uses[kTiles] = {};
        uint32_t kv_loads = 0;
        uint32_t tiles_before = 0;  // KV tiles of the items this CTA has finished
        const int pages_per_tile = BN >> p.block_shift;
        const int page_bytes = p.block_size * 128;  // one page inside one 64-element column block
        const int pages_per_v = G::kVKeys >> p.block_shift;  // in one slot
        bool ok = true;
        for (int r = 0; r < rounds && ok; ++r) {
            const int idx = item_of_round(r);
            if (idx < 0) continue;
            const Item w = decode_item(idx);
            if (lane == 0) {
                for (int t = 0; t < QT && ok; ++t) {
                    if (w.ntiles[t] == 0) continue;
                    if (q_uses[t] > 0) ok = MbarWait(bar(kQEmpty + t), (q_uses[t] - 1) & 1u, abort_flag);
                    if (!ok) break;
                    MbarExpectTx(bar(kQFull + t), G::kQTileBytes);
                    for (int kb = 0; kb < G::kKBlocks; ++kb) {
                        TmaLoad4D(q_smem + t * G::kQTileBytes + kb * G::kQBlockBytes, &map_q, bar(kQFull + t), kb * 64,
                                  w.h, w.q_tok0 + w.m0[t], w.b);
                    }
                    ++q_uses[t];
                }
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            const int32_t* row = p.page_table + static_cast<int64_t>(w.seq) * p.max_blocks_per_seq;
            // Page ids of a KV tile, one per lane; looked up a tile ahead, so that the ring does not wait for the table. At D=128 a
            // look-up per load is short against the step, and what looking ahead adds to the loop costs more than it saves (20
            // chunks against 512 to 6000 keys, lasting load, ahead / per load: D=128 429 / 400 us, D=64 299 / 324, D=256 1032 / 1125).
            constexpr bool kLookAhead = kOwnP;
            auto page_ids = [&](int tile) {
                const int logical = ((kSplit ? w.first_tile : 0) + tile) * pages_per_tile + lane;
                const bool in = lane < pages_per_tile && logical < p.max_blocks_per_seq && (static_cast<int64_t>(logical) << p.block_shift) < w.seq_kv;
                return in ? row[logical] : -1;
            };
            int32_t ids_before = -1, ids = -1, ids_next = kLookAhead ? page_ids(0) : -1;  // of the tiles before, of and behind the last K loaded
            for (int it = 0; it < 2 * w.n_max * kParts && ok; ++it, ++kv_loads) {
                const RingLoad load = RingOrder(it / kParts, w.n_max, kOwnP);
                const bool is_v = load.is_v;
                const int tile = load.tile;
                int32_t phys;
                if constexpr (kLookAhead) {
                    if (!is_v && it % kParts == 0) {
                        ids_before = ids;
                        ids = ids_next;
                        if (tile + 1 < w.n_max) ids_next = page_ids(tile + 1);
                    }
                    phys = is_v && tile + 1 < w.n_max ? ids_before : ids;
                } else {
                    phys = page_ids(tile);
                }
                const bool mapped = phys >= 0 && phys < p.num_kv_blocks;
                const uint32_t valid = __ballot_sync(0xffffffffu, mapped);
                const uint32_t slot = kv_loads % G::kSlots;
                const uint32_t phase = (kv_loads / G::kSlots) & 1u;
                if (lane == 0) {
                    ok = MbarWait(bar(kKvEmpty + slot), phase ^ 1u, abort_flag);
                    if (ok) {
                        if (!is_v) valid_ring[(tiles_before + tile) % kValidRing] = valid;
                        MbarExpectTx(full_bar(is_v, slot), G::kSlotBytes);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (!ok) break;
                const int part = it % kParts;
                // `blocks` column blocks of every page of the slot; an unmapped page reads from the first row behind the pool
                auto load_pages = [&](const CUtensorMap* map, int first_page, int pages, int first_block, auto blocks, uint32_t block_bytes) {
                    const uint32_t full = full_bar(is_v, slot);
                    uint32_t dst = ring_smem + slot * G::kSlotBytes;
                    for (int pg = 0; pg < pages; ++pg, dst += page_bytes) {
                        const int32_t id = __shfl_sync(0xffffffffu, phys, first_page + pg);
                        const int first_row = ((valid >> (first_page + pg)) & 1u) ? (id << p.block_shift) : (p.num_kv_blocks << p.block_shift);
                        if (ElectOne()) {
#pragma unroll
                            for (int kb = 0; kb < blocks.value; ++kb) {
                                TmaLoad4D(dst + kb * block_bytes, map, full, (first_block + kb) * 64, first_row, w.h_kv, 0);
                            }
                        }
                    }
                };
                if (is_v) {
                    load_pages(&map_v, part * pages_per_v, pages_per_v, 0, std::integral_constant<int, G::kKBlocks>{}, G::kVBlockBytes);
                } else {
                    load_pages(&map_k, 0, pages_per_tile, part * (G::kKBlocks / kParts), std::integral_constant<int, G::kKBlocks / kParts>{},
                               G::kKBlockBytes);
                }
            }
            tiles_before += static_cast<uint32_t>(w.n_max);
        }
        failed = !ok;
    } else if (warp == 0) {
        // ================================ TMA producer =============================================
        if (ElectOne()) {
            PrefetchTensorMap(&map_q);
            PrefetchTensorMap(&map_k);
            PrefetchTensorMap(&map_v);
            uint32_t q_uses[kTiles] = {};   // how often each query buffer has been filled so far
            uint32_t kv_loads = 0;         // K/V tiles loaded so far (ring position)
            bool ok = true;
            for (int r = 0; r < rounds && ok; ++r) {
                const int idx = item_of_round(r);
                if (idx < 0) continue;
                const Item w = decode_item(idx);
                for (int t = 0; t < QT && ok; ++t) {
                    if (w.ntiles[t] == 0) continue;
                    // the previous item's last S = Q K^T must have read the buffer
                    if (q_uses[t] > 0) ok = MbarWait(bar(kQEmpty + t), (q_uses[t] - 1) & 1u, abort_flag);
                    if (!ok) break;
                    MbarExpectTx(bar(kQFull + t), G::kQTileBytes);
                    for (int kb = 0; kb < G::kKBlocks; ++kb) {
                        TmaLoad4D(q_smem + t * G::kQTileBytes + kb * G::kQBlockBytes, &map_q, bar(kQFull + t), kb * 64,
                                  w.h, w.q_tok0 + w.m0[t], w.b);
                    }
                    ++q_uses[t];
                }
                for (int it = 0; it < 2 * w.n_max * kParts && ok; ++it, ++kv_loads) {
                    const RingLoad load = RingOrder(it / kParts, w.n_max, kOwnP);
                    const uint32_t slot = kv_loads % G::kSlots;
                    const uint32_t phase = (kv_loads / G::kSlots) & 1u;
                    ok = MbarWait(bar(kKvEmpty + slot), phase ^ 1u, abort_flag);
                    if (!ok) break;
                    const uint32_t full = full_bar(load.is_v, slot);
                    MbarExpectTx(full, G::kSlotBytes);
                    const int part = it % kParts;
                    const uint32_t dst = ring_smem + slot * G::kSlotBytes;
                    const int first_key = w.kv_tok0 + ((kSplit ? w.first_tile : 0) + load.tile) * BN;
                    if (load.is_v) {
                        for (int kb = 0; kb < G::kKBlocks; ++kb) {
                            TmaLoad4D(dst + kb * G::kVBlockBytes, &map_v, full, kb * 64, first_key + part * G::kVKeys, w.h_kv, w.b);
                        }
                    } else {
                        for (int kb = 0; kb < G::kKBlocks / kParts; ++kb) {
                            TmaLoad4D(dst + kb * G::kKBlockBytes, &map_k, full, (part * (G::kKBlocks / kParts) + kb) * 64, first_key,
                                      w.h_kv, w.b);
                        }
                    }
                }
            }
            failed = !ok;
        }
    } else if (warp == 1) {
        // ================================ MMA issuer ================================================
        if (ElectOne()) {
            constexpr uint32_t fmt = std::is_same<T, __half>::value ? kFmtF16 : kFmtBf16;
            constexpr uint32_t idesc_s = MakeInstrDesc(fmt, fmt, 0, 0, kBlockM, BN);  // Q K^T: both K-major
            // P V: V is MN-major; both operands in the P V format (fp16 also for bf16 inputs, see PvFormat)
            constexpr uint32_t fmt_pv = PvFormat<T>::kConvertV ? kFmtF16 : fmt;
            constexpr uint32_t idesc_o = MakeInstrDesc(fmt_pv, fmt_pv, 0, 1, kBlockM, DP);
            // Descriptors are built once and advanced by compile-time constants, so that issuing one
            // tcgen05.mma costs a handful of instructions (this thread alone has to keep the tensor pipe fed).
            const uint64_t kmajor_hi = MakeSmemDesc(0, 16, 1024);                 // K-major operands (Q and K)
            const uint64_t vmajor_hi = MakeSmemDesc(0, G::kVBlockBytes, 1024);    // MN-major operand (V)
            // A descriptor holds 18 bits of an address. The rest says which CTA of a cluster the memory belongs to, and would
            // run into the offset of the next column block.
            const uint32_t q_at = (q_smem & 0x3FFFFu) >> 4, ring_at = (ring_smem & 0x3FFFFu) >> 4;
            auto q_desc = [&](int t) { return kmajor_hi | (q_at + t * (G::kQTileBytes >> 4)); };
            auto s_tmem = [&](int t) { return tmem_base + G::kSCol + t * BN; };
            auto p_tmem = [&](int t) { return tmem_base + G::kPCol + t * G::kPStride; };
            auto o_tmem = [&](int t) { return tmem_base + G::kOCol + t * DP; };
            // the columns of S that the K of this slot contributes to: all of Q K^T, or one half of its products
            auto issue_s = [&](int t, uint32_t slot, int part) {
                const uint64_t a0 = q_desc(t) + ((part * (G::kKBlocks / kParts) * G::kQBlockBytes) >> 4);
                const uint64_t b0 = kmajor_hi | (ring_at + slot * (G::kSlotBytes >> 4));
#pragma unroll
                for (int ks = 0; ks < DP / kParts / 16; ++ks) {
                    constexpr int kStep = 32 >> 4;  // 16 elements = 32 bytes inside a 128-byte swizzle row
                    const uint32_t qa = ((ks >> 2) * G::kQBlockBytes >> 4) + (ks & 3) * kStep;
                    const uint32_t kb = ((ks >> 2) * G::kKBlockBytes >> 4) + (ks & 3) * kStep;
                    if (ks == 0 && part == 0) MmaSS<false>(s_tmem(t), a0 + qa, b0 + kb, idesc_s);
                    else MmaSS<true>(s_tmem(t), a0 + qa, b0 + kb, idesc_s);
                }
            };
            // P V over the keys of V in this slot; waits for the second piece of P (parity `parity`) where it begins
            auto issue_pv = [&](int t, uint32_t slot, int part, bool first, uint32_t parity) {
                const uint64_t b0 = vmajor_hi | (ring_at + slot * (G::kSlotBytes >> 4));
#pragma unroll
                for (int i = 0; i < G::kVKeys / 16; ++i) {
                    // 16 keys further: 8 packed P columns in tensor memory, 16 rows (2048 bytes) of V
                    const int ks = part * (G::kVKeys / 16) + i;
                    if (ks == kPEarly / 16) {
                        if (!MbarWait(bar(kPLast + t), parity, abort_flag)) return false;
                        TcFenceAfter();
                    }
                    if (ks == 0) MmaTSFlag(o_tmem(t), p_tmem(t), b0, idesc_o, first ? 0u : 1u);
                    else MmaTS<true>(o_tmem(t), p_tmem(t) + ks * 8, b0 + i * (2048 >> 4), idesc_o);
                }
                return true;
            };
            uint32_t q_uses[kTiles] = {};    // items finished per query buffer
            uint32_t steps[kTiles] = {};     // KV tiles processed per query tile (phase of s_full / p_full / o_done)
            uint32_t kv_base = 0;           // ring position of this item's K_0
            RingPhases k_phases, v_phases;  // of the K barriers and of v_ready (no converter: the V barriers)
            bool ok = true;
            auto k_landed = [&](uint32_t slot) { return MbarWait(full_bar(false, slot), k_phases.Take(slot), abort_flag); };
            auto v_ready = [&](uint32_t slot) {
                return MbarWait(kCvtInKernel ? bar(kVReady + slot) : full_bar(true, slot), v_phases.Take(slot), abort_flag);
            };
            if constexpr (kOwnP) {
                // S_t(j+1) goes out as soon as S_t(j) is in registers, P_t(j) V_j when P_t(j) has been written
                uint32_t scores[kTiles] = {};  // score tiles issued per query tile (phase of s_read)
                auto next_slots = [&](uint32_t (&slots)[kParts]) {
                    for (int part = 0; part < kParts; ++part) slots[part] = kv_base++ % G::kSlots;
                };
                // K and V are waited for with the first query tile, also where it has no use for them, and freed with the last
                auto score_step = [&](int t, const uint32_t (&k)[kParts], bool active, bool wait_k, bool last) {
                    if (active && scores[t] > 0 && !MbarWait(bar(kSRead + t), (scores[t] - 1) & 1u, abort_flag)) return false;
#pragma unroll
                    for (int part = 0; part < kParts; ++part) {
                        if (wait_k && !k_landed(k[part])) return false;
                        TcFenceAfter();
                        if (active) issue_s(t, k[part], part);
                        if (t == QT - 1) MmaCommit(bar(kKvEmpty + k[part]));
                    }
                    if (active) {
                        MmaCommit(bar(kSFull + t));
                        if (last) MmaCommit(bar(kQEmpty + t));
                        ++scores[t];
                    }
                    return true;
                };
                for (int r = 0; r < rounds && ok; ++r) {
                    const int idx = item_of_round(r);
                    if (idx < 0) continue;
                    const Item w = decode_item(idx);
                    const int n = w.n_max;
                    if (n == 0) continue;
                    uint32_t k[kParts], v[kParts];
                    next_slots(k);
#pragma unroll
                    for (int t = 0; t < QT; ++t) {
                        if (!ok) break;
                        if (w.ntiles[t] > 0) ok = MbarWait(bar(kQFull + t), q_uses[t] & 1u, abort_flag);
                        ok = ok && score_step(t, k, w.ntiles[t] > 0, t == 0, w.ntiles[t] == 1);
                    }
                    for (int j = 0; j < n && ok; ++j) {
                        if (j + 1 < n) next_slots(k);
                        next_slots(v);
#pragma unroll
                        for (int t = 0; t < QT; ++t) {
                            if (!ok) break;
                            if (j + 1 < n) ok = score_step(t, k, j + 1 < w.ntiles[t], t == 0, j + 2 == w.ntiles[t]);
                            const bool active = j < w.ntiles[t];
                            if (ok && active) ok = MbarWait(bar(kPFull + t), steps[t] & 1u, abort_flag);
                            // the first P V of an item overwrites O: the previous item's O must have been read out
                            if (ok && active && j == 0 && q_uses[t] > 0) ok = MbarWait(bar(kOFree + t), (q_uses[t] - 1) & 1u, abort_flag);
                            if (!ok) break;
#pragma unroll
                            for (int part = 0; part < kParts; ++part) {
                                if (t == 0) ok = v_ready(v[part]);
                                if (!ok) break;
                                TcFenceAfter();
                                if (active) ok = issue_pv(t, v[part], part, j == 0, steps[t] & 1u);
                                if (!ok) break;
                                if (t == QT - 1) MmaCommit(bar(kKvEmpty + v[part]));
                            }
                            if (ok && active) {
                                MmaCommit(bar(kODone + t));
                                ++steps[t];
                            }
                        }
                    }
#pragma unroll
                    for (int t = 0; t < QT; ++t) {
                        if (w.ntiles[t] > 0) ++q_uses[t];
                    }
                }
            }
            // P over S: P_t(j) V_j, then S_t(j+1), tile by tile
            for (int r = 0; r < rounds && ok && !kOwnP; ++r) {
                const int idx = item_of_round(r);
                if (idx < 0) continue;
                const Item w = decode_item(idx);
                auto slot_of = [&](int it) { return (kv_base + it) % G::kSlots; };
                for (int t = 0; t < QT && ok; ++t) {
                    if (w.ntiles[t] > 0) ok = MbarWait(bar(kQFull + t), q_uses[t] & 1u, abort_flag);
                }
                if (ok && w.n_max > 0) {
                    ok = k_landed(slot_of(0));
                    if (ok) {
                        TcFenceAfter();
                        for (int t = 0; t < QT; ++t) {
                            if (w.ntiles[t] == 0) continue;
                            issue_s(t, slot_of(0), 0);
                            MmaCommit(bar(kSFull + t));
                            if (w.ntiles[t] == 1) MmaCommit(bar(kQEmpty + t));  // last read of this query tile
                        }
                        MmaCommit(bar(kKvEmpty + slot_of(0)));
                    }
                }
                for (int j = 0; j < w.n_max && ok; ++j) {
                    const int it_v = 2 * j + 1;
                    const int it_k = 2 * j + 2;
                    ok = v_ready(slot_of(it_v));
                    if (ok && j + 1 < w.n_max) ok = k_landed(slot_of(it_k));
                    if (!ok) break;
                    for (int t = 0; t < QT; ++t) {
                        if (j >= w.ntiles[t]) continue;
                        ok = MbarWait(bar(kPFull + t), steps[t] & 1u, abort_flag);
                        // the first P V of an item overwrites O: the previous item's O must have been read out
                        if (ok && j == 0 && q_uses[t] > 0) ok = MbarWait(bar(kOFree + t), (q_uses[t] - 1) & 1u, abort_flag);
                        if (!ok) break;
                        TcFenceAfter();
                        ok = issue_pv(t, slot_of(it_v), 0, j == 0, steps[t] & 1u);
                        if (!ok) break;
                        MmaCommit(bar(kODone + t));
                        ++steps[t];
                        if (j + 1 < w.ntiles[t]) {
                            issue_s(t, slot_of(it_k), 0);
                            MmaCommit(bar(kSFull + t));
                            if (j + 2 == w.ntiles[t]) MmaCommit(bar(kQEmpty + t));
                        }
                    }
                    if (!ok) break;
                    MmaCommit(bar(kKvEmpty + slot_of(it_v)));
                    if (j + 1 < w.n_max) MmaCommit(bar(kKvEmpty + slot_of(it_k)));
                }
                for (int t = 0; t < QT; ++t) {
                    if (w.ntiles[t] > 0) ++q_uses[t];
                }
                kv_base += 2 * w.n_max;
            }
            failed = !ok;
        }
    } else if (converter >= 0 && converter < kConverters) {
        // ================================ V converter (bf16) ========================================
        // Walks the ring in the producer's order; every V tile is rewritten in place from bf16 to fp16 once its
        // bytes have landed, then handed to the MMA thread through v_ready. K tiles are not touched.
        uint32_t kv_loads = 0;
        RingPhases v_phases;
        bool ok = true;
        for (int r = 0; r < rounds && ok; ++r) {
            const int idx = item_of_round(r);
            if (idx < 0) continue;
            const Item w = decode_item(idx);
            for (int it = 0; it < 2 * w.n_max * kParts && ok; ++it, ++kv_loads) {
                if (!RingOrder(it / kParts, w.n_max, kOwnP).is_v) continue;
                const uint32_t slot = kv_loads % G::kSlots;
                ok = __all_sync(0xffffffffu, MbarWait(full_bar(true, slot), v_phases.Take(slot), abort_flag));
                if (!ok) break;
                uint4* tile = reinterpret_cast<uint4*>(smem + (ring_smem - smem_base) + slot * G::kSlotBytes);
#pragma unroll 8
                for (int c = converter * 32 + lane; c < G::kSlotBytes / 16; c += 32 * kConverters) {
                    uint4 x = tile[c];
                    uint32_t* word = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = UnpackBf16(word[e]);
                        // one instruction for both lanes; values beyond the fp16 range saturate instead of becoming inf
                        asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(word[e]) : "f"(f.y), "f"(f.x));
                    }
                    tile[c] = x;
                }
                FenceProxyAsync();  // generic-proxy writes -> visible to the tensor core's reads
                MbarArrive(bar(kVReady + slot));
            }
        }
        failed = !ok;
    } else if (warp >= kFirstSoftmax && warp < kEndSoftmax) {
        // ================================ softmax groups ============================================
        const int t = (warp - kFirstSoftmax) >> 2;
        const int quad = warp & 3;
        const int row_in_tile = quad * 32 + lane;
        const uint32_t lane_bits = static_cast<uint32_t>(quad * 32) << 16;
        const uint32_t s_addr = tmem_base + lane_bits + G::kSCol + t * BN;
        const uint32_t p_addr = tmem_base + lane_bits + G::kPCol + t * G::kPStride;
        const uint32_t o_addr = tmem_base + lane_bits + G::kOCol + t * DP;
        uint32_t steps = 0;  // KV tiles this group has processed (phase of s_full / p_full / o_done)
        uint32_t tiles_before = 0;  // paged K/V: KV tiles of the items this CTA has finished (index into valid_ring)
        float* part_row = reinterpret_cast<float*>(smem + (ring_smem - smem_base)) + row_in_tile * kPartLd;  // kSplit
        const uint32_t all_pages = kPaged ? ((BN >> p.block_shift) >= 32 ? 0xffffffffu : (1u << (BN >> p.block_shift)) - 1u) : 0u;
        bool ok = true;

        for (int r = 0; r < rounds && ok; ++r) {
            const int idx = item_of_round(r);
            if (idx < 0) continue;
            const Item w = decode_item(idx);
            int n_t = 0, m_t = 0;
#pragma unroll
            for (int i = 0; i < kTiles; ++i) {
                if (i == t) n_t = w.ntiles[i], m_t = w.m0[i];
            }
            const uint32_t tiles_base = tiles_before;
            tiles_before += static_cast<uint32_t>(w.n_max);
            if (n_t == 0) {
                if (kSplit && t == 0) *reinterpret_cast<float2*>(part_row + DP) = make_float2(-CUDART_INF_F, 0.0f);
                continue;
            }
            const int row = m_t + (row_in_tile >> p.pack_shift);                 // token of the sequence
            const int head = w.h + (row_in_tile & ((1 << p.pack_shift) - 1));
            float m_ref = -CUDART_INF_F;  // reference point of the exponentials (log2 domain)
            float l_sum = 0.0f;

            for (int j = 0; j < n_t; ++j, ++steps) {
                ok = __all_sync(0xffffffffu, MbarWait(bar(kSFull + t), steps & 1u, abort_flag));
                if (!ok) break;
                TcFenceAfter();
                // The row goes to registers whole. The exponentials use the reference point the row already has; the
                // row's maximum is only checked against it. If it exceeds the reference by more than the threshold
                // (always in the first step of an item), the reference moves and O and the row sum are rescaled.
                // P (16-bit pairs) goes to columns of its own or to the first BN / 2 columns of S_t, which has been read by
                // then; its first kPEarly keys are handed over early, so that P V starts under the last exponentials.
                const int col0 = ((kSplit ? w.first_tile : 0) + j) * BN;
                const int kv_limit = w.seq_kv - col0;                                   // columns >= kv_limit do not exist
                const int causal_limit = p.causal ? (row + w.diagonal - col0 + 1) : BN;  // columns >= limit are masked
                const int limit = min(kv_limit, causal_limit);
                const uint32_t pages = kPaged ? valid_ring[(tiles_base + j) % kValidRing] : 0u;
                const bool holes = kPaged && pages != all_pages;   // some page of this tile is unmapped
                const bool ragged = limit < BN || holes;
                uint32_t sc[BN / 32][32];
#pragma unroll
                for (int c = 0; c < BN / 32; ++c) TmemLd32(s_addr + c * 32, sc[c]);
                TmemWaitLd();
                if constexpr (kOwnP) {
                    TcFenceBefore();
                    __syncwarp();
                    if (lane == 0) MbarArrive(bar(kSRead + t));
                }
                bool pv_done = j == 0;  // P(j-1) V_j-1: O and the columns of P may be written
                auto wait_pv = [&] {
                    if (!pv_done) {
                        ok = __all_sync(0xffffffffu, MbarWait(bar(kODone + t), (steps - 1) & 1u, abort_flag));
                        TcFenceAfter();
                        pv_done = true;
                    }
                };
                if (ragged) {
#pragma unroll
                    for (int c = 0; c < BN / 32; ++c) {
                        // bit i: column 32 * c + i is visible
                        const int seen = limit - 32 * c;
                        uint32_t visible = seen >= 32 ? 0xffffffffu : seen <= 0 ? 0u : (1u << seen) - 1u;
                        if (kPaged && holes) {
#pragma unroll
                            for (int g = 0; g < 4; ++g) {  // a page has 8 keys at least
                                if (!((pages >> ((32 * c + 8 * g) >> p.block_shift)) & 1u)) visible &= ~(0xffu << (8 * g));
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            if (!(visible & (1u << i))) sc[c][i] = 0xff800000u;  // -inf
                        }
                    }
                }
                {
                    float mx4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) mx4[e] = fmaxf(__uint_as_float(sc[0][e]), __uint_as_float(sc[0][4 + e]));
#pragma unroll
                    for (int i = 8; i < BN; i += 8) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            mx4[e] = Max3(mx4[e], __uint_as_float(sc[i / 32][i % 32 + e]), __uint_as_float(sc[i / 32][i % 32 + 4 + e]));
                        }
                    }
                    const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;  // scale > 0
                    const bool move = mx > m_ref + kRescaleThreshold;  // false for a fully masked row (-inf)
                    if (__any_sync(0xffffffffu, move)) {
                        const float alpha = move ? Exp2(m_ref - mx) : 1.0f;  // m_ref = -inf -> 0
                        if (j > 0) {
                            wait_pv();
                            if (!ok) break;
#pragma unroll 1
                            for (int cblk = 0; cblk < DP / 16; ++cblk) {
                                uint32_t r[16];
                                TmemLd16(o_addr + cblk * 16, r);
                                TmemWaitLd();
#pragma unroll
                                for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
                                TmemSt16(o_addr + cblk * 16, r);
                            }
                        }
                        l_sum *= alpha;
                        if (move) m_ref = mx;
                    }
                }
                // Exponentials of columns [32 * first, 32 * end): P to tensor memory, their sum onto sum[]. With kBehind the
                // additions and conversions of a batch of 8 come behind the exponentials of the next one: a warp alone on
                // its scheduler takes 1190 clocks for 128 exponentials that way and 1331 when it waits for each batch
                // (1030 is the rate of the special-function unit), two warps 2070 and 2110. D=128, where the groups meet
                // the products half of the time, gains 2 % (528 against 535 us at B=4, S=4096); D=64, where they mostly
                // run side by side, loses 10 % (359 against 322 us at B=3, S=2900).
                constexpr bool kBehind = DP != 64;
                const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
                float2 sum[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[e] = make_float2(0.0f, 0.0f);
                auto fold_sum = [&] {
                    l_sum += ((sum[0].x + sum[0].y) + (sum[1].x + sum[1].y)) + ((sum[2].x + sum[2].y) + (sum[3].x + sum[3].y));
                };
                auto exponentials = [&](int first, int end) {
                    const float neg_m = (m_ref == -CUDART_INF_F) ? 0.0f : -m_ref;
                    const float2 shift2 = make_float2(neg_m, neg_m);
                    float2 x[2][4];
                    uint32_t pk[16];
                    constexpr int kLag = kBehind ? 1 : 0;
#pragma unroll
                    for (int b = 0; b < BN / 8 + kLag; ++b) {
                        if (b < 4 * first || b >= 4 * end + kLag) continue;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if (b < 4 * end) {
                                x[b & 1][e] = Fma2(make_float2(__uint_as_float(sc[b / 4][(b % 4) * 8 + 2 * e]), __uint_as_float(sc[b / 4][(b % 4) * 8 + 2 * e + 1])), scale2, shift2);
                                x[b & 1][e] = make_float2(Exp2(x[b & 1][e].x), Exp2(x[b & 1][e].y));
                            }
                            const int d = b - kLag;
                            if (d >= 4 * first) {
                                sum[kBehind ? e : e & 1] = Add2(sum[kBehind ? e : e & 1], x[d & 1][e]);
                                pk[(d % 4) * 4 + e] = Pack2<PT>(x[d & 1][e].x, x[d & 1][e].y);
                            }
                        }
                        if (b - kLag >= 4 * first && (b - kLag) % 4 == 3) {
                            if (kOwnP && b - kLag == 3) wait_pv();
                            TmemSt16(p_addr + (b - kLag) / 4 * 16, pk);
                        }
                    }
                };
                auto hand_over = [&](uint32_t barrier) {
                    TmemWaitSt();
                    TcFenceBefore();
                    __syncwarp();
                    if (lane == 0) MbarArrive(barrier);
                };
                exponentials(0, kPEarly / 32);
                if (!ok) break;
                hand_over(bar(kPFull + t));
                if (kBehind && kPEarly < BN) {  // eight registers less across the second piece
                    fold_sum();
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[e] = make_float2(0.0f, 0.0f);
                }
                if constexpr (kPEarly < BN) {
                    exponentials(kPEarly / 32, BN / 32);
                    hand_over(bar(kPLast + t));
                }
                fold_sum();
            }
            if (!ok) break;

            // ---- epilogue: O / l -> global, optional LSE; O is handed back as soon as it is in registers ----
            ok = __all_sync(0xffffffffu, MbarWait(bar(kODone + t), (steps - 1) & 1u, abort_flag));
            if (!ok) break;
            TcFenceAfter();
            if constexpr (kSplit) {
                // all K/V of the item has been consumed: the ring holds this CTA's part
#pragma unroll
                for (int cblk = 0; cblk < DP / 32; ++cblk) {
                    uint32_t r[32];
                    TmemLd32(o_addr + cblk * 32, r);
                    TmemWaitLd();
#pragma unroll
                    for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(part_row + cblk * 32 + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
                }
                *reinterpret_cast<float2*>(part_row + DP) = make_float2(m_ref, l_sum);
                continue;
            }
            const float inv = l_sum > 0.0f ? 1.0f / l_sum : 0.0f;
            T* o_row = reinterpret_cast<T*>(p.out) + w.b * p.o_sb + head * p.o_sh + static_cast<int64_t>(w.q_tok0 + row) * p.o_ss;
#pragma unroll
            for (int cblk = 0; cblk < DP / 32; ++cblk) {
                uint32_t r[32];
                TmemLd32(o_addr + cblk * 32, r);
                TmemWaitLd();
                if (cblk == DP / 32 - 1) {
                    TcFenceBefore();
                    __syncwarp();
                    if (lane == 0) MbarArrive(bar(kOFree + t));
                }
                if (row < w.seq_q) {
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t pk[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            pk[i] = Pack2<T>(__uint_as_float(r[half * 16 + 2 * i]) * inv, __uint_as_float(r[half * 16 + 2 * i + 1]) * inv);
                        }
                        const int d0 = cblk * 32 + half * 16;
                        if (d0 < p.head_dim) StoreRow16(o_row + d0, pk, p.wide_stores);
                    }
                }
            }
            if (p.lse != nullptr && row < w.seq_q) {
                p.lse[(static_cast<int64_t>(w.b) * p.heads + head) * p.seq_q + row] =
                    l_sum > 0.0f ? (m_ref + log2f(l_sum)) * kLn2 : -CUDART_INF_F;
            }
        }
        failed = !ok;
    }

    if (failed && p.error_word != nullptr) *p.error_word = 1 + warp;

    // ---- teardown ------------------------------------------------------------------------------------
    // One lane of warps 0 and 1 comes from its loop long after the others; the tensor-memory instructions are for whole
    // warps, and neither the end of a branch nor __syncthreads promises that the lanes have met.
    __syncwarp();
    TcFenceBefore();
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        TcFenceAfter();
        TmemDealloc(tmem_base, kTmemColumns);
    }
    if constexpr (kSplit) {
        __syncwarp();
        ClusterBarrier();
        // Every CTA merges its share of the rows: first a thread per row for the weights of the parts, then all threads for the
        // columns, four at a time, so that many loads from the other CTAs are under way at once.
        const int rank = static_cast<int>(ClusterRank());
        const Item w = decode_item(static_cast<int>(blockIdx.x) / p.cluster);
        const int rows = kBlockM / p.cluster, row0 = rank * rows;
        float* weights = reinterpret_cast<float*>(smem + (q_smem - smem_base));  // [rows][kMaxSplit], where Q was
        auto out_row = [&](int r, int* token, int* head) {
            *token = w.m0[0] + (r >> p.pack_shift);
            *head = w.h + (r & ((1 << p.pack_shift) - 1));
            return *token < w.seq_q;
        };
        if (threadIdx.x < rows) {
            const int i = threadIdx.x;
            float2 ml[kMaxSplit];
            float m_all = -CUDART_INF_F, l_all = 0.0f;
#pragma unroll
            for (int c = 0; c < kMaxSplit; ++c) {
                ml[c] = c < p.cluster ? LoadFromRank2(ring_smem + ((row0 + i) * kPartLd + DP) * 4, c) : make_float2(-CUDART_INF_F, 0.0f);
                m_all = fmaxf(m_all, ml[c].x);
            }
#pragma unroll
            for (int c = 0; c < kMaxSplit; ++c) {
                // a part without a key for the row; a row of NaN has no maximum either, but a sum that is NaN
                if (ml[c].x == -CUDART_INF_F && ml[c].y == 0.0f) continue;
                l_all += ml[c].y * Exp2(ml[c].x - m_all);
            }
            const float inv = l_all > 0.0f ? 1.0f / l_all : 0.0f;
            // -1: no key of that part is visible to the row, and the CTA may hold no O
#pragma unroll
            for (int c = 0; c < kMaxSplit; ++c) {
                weights[i * kMaxSplit + c] = ml[c].x == -CUDART_INF_F && ml[c].y == 0.0f ? -1.0f : Exp2(ml[c].x - m_all) * inv;
            }
            int token, head;
            if (p.lse != nullptr && out_row(row0 + i, &token, &head)) {
                p.lse[(static_cast<int64_t>(w.b) * p.heads + head) * p.seq_q + token] = l_all > 0.0f ? (m_all + log2f(l_all)) * kLn2 : -CUDART_INF_F;
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int item = threadIdx.x; item < rows * (DP / 4); item += FlashThreads<T, DP, QT>()) {
            const int i = item / (DP / 4), d = item % (DP / 4) * 4;
            int token, head;
            if (!out_row(row0 + i, &token, &head) || d >= p.head_dim) continue;
            float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int c = 0; c < kMaxSplit; ++c) {
                const float weight = c < p.cluster ? weights[i * kMaxSplit + c] : -1.0f;
                if (weight < 0.0f) continue;
                const float4 x = LoadFromRank4(ring_smem + ((row0 + i) * kPartLd + d) * 4, c);
                acc.x += x.x * weight, acc.y += x.y * weight, acc.z += x.z * weight, acc.w += x.w * weight;
            }
            T* o_row = reinterpret_cast<T*>(p.out) + w.b * p.o_sb + head * p.o_sh + static_cast<int64_t>(w.q_tok0 + token) * p.o_ss;
            *reinterpret_cast<uint2*>(o_row + d) = make_uint2(Pack2<T>(acc.x, acc.y), Pack2<T>(acc.z, acc.w));
        }
        __syncwarp();
        ClusterBarrier();  // nobody leaves while its shared memory is being read
    }
}

// The kSplit kernels are compiled in flash_split.cu.
template <typename T, int DP, int QT, int BN, bool kVarlen, bool kPaged>
int LaunchSplit(int64_t items, cudaStream_t stream, const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v,
                const FlashKernelParams& p);
// Clusters of `cluster` CTAs that run at the same time (0 when the device cannot say).
template <typename T, int DP, int QT, int BN>
int ResidentClusters(int cluster);

}  // namespace flash
}  // namespace sca_b200

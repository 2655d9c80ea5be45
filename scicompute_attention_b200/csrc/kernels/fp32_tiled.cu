// Attention for fp32 inputs with fp32 arithmetic throughout, tiled through shared memory.
//
// Bound by the FMA pipe: 4 * D FLOPs per visible (query, key) pair against 128 FMA per clock and SM. The one-warp-per-
// row kernel of simt.cu spends its time elsewhere: it fetches every K and V row from L2 once per query row and reduces
// every score with five shuffles (B=1, H=8, S=1024, D=128: 1404 us = 3 TFLOP/s; here 112 us = 38 TFLOP/s, and 650 to
// 95 us for a single query row against 1024 keys). Here a CTA keeps BM query rows and streams K/V tiles, and every thread owns an RT x CT block of scores and an RT x D/8 block of the output, so that one
// 16-byte shared-memory load feeds 8 to 16 FMAs (packed two to an instruction).
//
//   * two groups of 4 warps share the BM query rows and take alternate key tiles; each keeps its own running softmax
//     (m, l, O), merged through shared memory at the end. Two warps per scheduler hide the load latency that one
//     leaves, and one group's loads and softmax overlap the other's products without a second buffer;
//   * a warp's 32 lanes are 4 row groups x 8 column groups; a row of scores lives in 8 lanes of one warp, so the row
//     maxima and sums take three shuffles and P never leaves the warp that reads it back for P V;
//   * rows in shared memory are padded by 16 bytes: the operand loads are free of bank conflicts;
//   * K_j+1 is fetched (16-byte cp.async, zero-filled past the end) as soon as S_j is complete, V_j+1 after P_j V_j.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace sca_b200 {
namespace {

constexpr int kGroups = 2;          // key-tile groups per CTA
constexpr int kGroupThreads = 128;  // 4 warps
constexpr int kF32Threads = kGroups * kGroupThreads;

template <int D, int RT>
struct F32Geom {
    static constexpr int kBM = 16 * RT;             // 4 warps x 4 row groups x RT rows
    static constexpr int kBN = D <= 128 ? 64 : 32;  // keys per tile and group
    static constexpr int kCT = kBN / 8;             // score columns per thread
    static constexpr int kLd = D + 4;               // padded row of Q and K
    static constexpr int kPLd = kBN + 4;            // padded row of P
    static constexpr int kQFloats = kBM * kLd;
    static constexpr int kKFloats = kBN * kLd;
    static constexpr int kVFloats = kBN * D;
    static constexpr int kPFloats = kBM * kPLd;
    static constexpr int kGroupFloats = kKFloats + kVFloats + kPFloats;
    static constexpr int kSmemBytes = 4 * (kQFloats + kGroups * kGroupFloats);
    static_assert(D % 32 == 0 && D <= 256, "head_dim");
    static_assert(kSmemBytes <= 232448, "exceeds the 227 KiB per-CTA limit");
    static_assert(kGroupFloats >= kBM * (D + 4), "the second group hands its O over in its own tile buffers");
};

struct F32Params {
    const float* q;
    const float* k;
    const float* v;
    float* out;
    float* lse;
    int heads, kv_heads, seq_q, seq_kv, bh_count, m_blocks;
    int64_t q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss, o_sb, o_sh, o_ss;
    float scale_log2;
    int causal;
    int64_t diagonal;
};

__device__ __forceinline__ float4 LdsF4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void GroupBarrier(int group) {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kGroupThreads) : "memory");
}

// O += P V for one key tile. kMasked: keys at or beyond a row's limit are left out of the sum altogether (their V may
// hold anything, infinities included).
template <int D, int RT, bool kMasked>
__device__ __forceinline__ void AccumulatePv(const float* p_rows, const float* v_tile, int cg, const int (&limit)[RT],
                                             float2 (&o)[RT][D / 16]) {
    using G = F32Geom<D, RT>;
#pragma unroll 2
    for (int key = 0; key < G::kBN; key += 4) {
        float4 pr[RT];
#pragma unroll
        for (int i = 0; i < RT; ++i) pr[i] = LdsF4(p_rows + 4 * i * G::kPLd + key);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            float4 vr[D / 32];
#pragma unroll
            for (int c = 0; c < D / 32; ++c) vr[c] = LdsF4(v_tile + (key + kk) * D + 32 * c + 4 * cg);
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                if (kMasked && key + kk >= limit[i]) continue;
                const float w = kk == 0 ? pr[i].x : kk == 1 ? pr[i].y : kk == 2 ? pr[i].z : pr[i].w;
                const float2 ww = make_float2(w, w);
#pragma unroll
                for (int c = 0; c < D / 32; ++c) {
                    o[i][2 * c] = Fma2(ww, make_float2(vr[c].x, vr[c].y), o[i][2 * c]);
                    o[i][2 * c + 1] = Fma2(ww, make_float2(vr[c].z, vr[c].w), o[i][2 * c + 1]);
                }
            }
        }
    }
}

template <int D, int RT>
__global__ void __launch_bounds__(kF32Threads, 1) fp32_tiled_attention_kernel(const F32Params p) {
    using G = F32Geom<D, RT>;
    extern __shared__ __align__(128) float f32_smem[];
    BeginAfterPredecessor();
    const int lane = threadIdx.x & 31;
    const int group = threadIdx.x / kGroupThreads;
    const int tid = threadIdx.x % kGroupThreads;
    const int rg = lane >> 3;  // row group
    const int cg = lane & 7;   // column group
    float* q_tile = f32_smem;
    float* k_tile = f32_smem + G::kQFloats + group * G::kGroupFloats;
    float* v_tile = k_tile + G::kKFloats;
    float* p_tile = v_tile + G::kVFloats;
    const int row0 = (tid >> 5) * (4 * RT) + rg;  // this thread's rows in the tile: row0 + 4 * i

    // causal problems: the blocks that see the most keys first
    const int mb = p.m_blocks - 1 - static_cast<int>(blockIdx.x / p.bh_count);
    const int bh = static_cast<int>(blockIdx.x % p.bh_count);
    const int b = bh / p.heads, h = bh % p.heads, h_kv = h / (p.heads / p.kv_heads);
    const int m0 = mb * G::kBM;
    const float* q_base = p.q + b * p.q_sb + h * p.q_sh;
    const float* k_base = p.k + b * p.k_sb + h_kv * p.k_sh;
    const float* v_base = p.v + b * p.v_sb + h_kv * p.v_sh;

    // keys any row of this block sees
    int64_t visible = p.seq_kv;
    if (p.causal) visible = min(visible, min(static_cast<int64_t>(m0) + G::kBM, static_cast<int64_t>(p.seq_q)) + p.diagonal);
    const int tiles = visible > 0 ? static_cast<int>((visible + G::kBN - 1) / G::kBN) : 0;

    constexpr int kChunks = D / 4;  // 16-byte pieces of a row
    auto load_rows = [&](float* tile, int ld, const float* base, int64_t stride, int first, int count, int rows, int thread,
                         int threads) {
        for (int item = thread; item < count * kChunks; item += threads) {
            const int r = item / kChunks, c = item % kChunks;
            const bool in = first + r < rows;
            CpAsync16(SmemAddr(tile + r * ld + 4 * c), base + (in ? (first + r) * stride : 0) + 4 * c, in ? 16 : 0);
        }
    };
    load_rows(q_tile, G::kLd, q_base, p.q_ss, m0, G::kBM, p.seq_q, threadIdx.x, kF32Threads);
    CpAsyncCommit();
    if (group < tiles) load_rows(k_tile, G::kLd, k_base, p.k_ss, group * G::kBN, G::kBN, p.seq_kv, tid, kGroupThreads);
    CpAsyncCommit();
    if (group < tiles) load_rows(v_tile, D, v_base, p.v_ss, group * G::kBN, G::kBN, p.seq_kv, tid, kGroupThreads);
    CpAsyncCommit();
    CpAsyncWait<2>();
    __syncthreads();

    float m[RT], l[RT];
    float2 o[RT][D / 16];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        m[i] = -CUDART_INF_F;
        l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < D / 16; ++c) o[i][c] = make_float2(0.0f, 0.0f);
    }

    for (int t = group; t < tiles; t += kGroups) {
        const int col0 = t * G::kBN;
        CpAsyncWait<1>();  // K_t
        GroupBarrier(group);
        // S = Q K^T; even and odd elements of the head dimension accumulate separately
        float2 s2[RT][G::kCT];
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < G::kCT; ++j) s2[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll 2
        for (int d = 0; d < D; d += 4) {
            float4 a[RT];
#pragma unroll
            for (int i = 0; i < RT; ++i) a[i] = LdsF4(q_tile + (row0 + 4 * i) * G::kLd + d);
#pragma unroll
            for (int j = 0; j < G::kCT; ++j) {
                const float4 kr = LdsF4(k_tile + (cg + 8 * j) * G::kLd + d);
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    s2[i][j] = Fma2(make_float2(a[i].x, a[i].y), make_float2(kr.x, kr.y), s2[i][j]);
                    s2[i][j] = Fma2(make_float2(a[i].z, a[i].w), make_float2(kr.z, kr.w), s2[i][j]);
                }
            }
        }
        GroupBarrier(group);  // everybody has read K_t
        if (t + kGroups < tiles) {
            load_rows(k_tile, G::kLd, k_base, p.k_ss, col0 + kGroups * G::kBN, G::kBN, p.seq_kv, tid, kGroupThreads);
        }
        CpAsyncCommit();

        // columns at or beyond limit[i] are not visible to row i
        int limit[RT];
        bool masked = false;
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            int64_t lim = p.seq_kv;
            if (p.causal) lim = min(lim, static_cast<int64_t>(m0) + row0 + 4 * i + p.diagonal + 1);
            limit[i] = static_cast<int>(max(static_cast<int64_t>(0), min(lim - col0, static_cast<int64_t>(G::kBN))));
            masked |= limit[i] < G::kBN;
        }
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            float s[G::kCT];
            float mx = -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < G::kCT; ++j) {
                s[j] = (s2[i][j].x + s2[i][j].y) * p.scale_log2;
                if (cg + 8 * j < limit[i]) mx = fmaxf(mx, s[j]);
            }
#pragma unroll
            for (int off = 4; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float m_new = fmaxf(m[i], mx);
            const float alpha = m_new == m[i] ? 1.0f : Exp2(m[i] - m_new);  // m = -inf -> 0
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < G::kCT; ++j) {
                const float w = cg + 8 * j < limit[i] ? Exp2(s[j] - m_new) : 0.0f;
                sum += w;
                p_tile[(row0 + 4 * i) * G::kPLd + cg + 8 * j] = w;
            }
            l[i] = l[i] * alpha + sum;  // this lane's columns; the lanes of a row are added up at the end
            m[i] = m_new;
            const float2 alpha2 = make_float2(alpha, alpha);
#pragma unroll
            for (int c = 0; c < D / 16; ++c) o[i][c] = Fma2(o[i][c], alpha2, make_float2(0.0f, 0.0f));
        }
        CpAsyncWait<1>();  // V_t
        GroupBarrier(group);
        if (__any_sync(0xffffffffu, masked)) AccumulatePv<D, RT, true>(p_tile + row0 * G::kPLd, v_tile, cg, limit, o);
        else AccumulatePv<D, RT, false>(p_tile + row0 * G::kPLd, v_tile, cg, limit, o);
        GroupBarrier(group);  // everybody has read V_t
        if (t + kGroups < tiles) {
            load_rows(v_tile, D, v_base, p.v_ss, col0 + kGroups * G::kBN, G::kBN, p.seq_kv, tid, kGroupThreads);
        }
        CpAsyncCommit();
    }
    CpAsyncWait<0>();

#pragma unroll
    for (int i = 0; i < RT; ++i) {
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], off);
    }

    // ---- the second group hands (O, m, l) to the first through its own (now idle) tile buffers ----------------
    GroupBarrier(group);
    float* hand = f32_smem + G::kQFloats + G::kGroupFloats;  // [BM][D + 4]: O, then m and l
    if (group == 1) {
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            float* row = hand + (row0 + 4 * i) * (D + 4);
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                *reinterpret_cast<float4*>(row + 32 * c + 4 * cg) =
                    make_float4(o[i][2 * c].x, o[i][2 * c].y, o[i][2 * c + 1].x, o[i][2 * c + 1].y);
            }
            if (cg == 0) {
                row[D] = m[i];
                row[D + 1] = l[i];
            }
        }
    }
    __syncthreads();
    if (group == 1) return;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int row = m0 + row0 + 4 * i;
        if (row >= p.seq_q) continue;
        const float* other = hand + (row0 + 4 * i) * (D + 4);
        const float m_other = other[D], l_other = other[D + 1];
        const float m_all = fmaxf(m[i], m_other);
        const float w0 = m[i] == m_all ? 1.0f : Exp2(m[i] - m_all);
        const float w1 = m_other == m_all ? 1.0f : Exp2(m_other - m_all);
        const float l_all = l[i] * w0 + l_other * w1;
        const float inv = l_all > 0.0f ? 1.0f / l_all : 0.0f;
        float* o_row = p.out + b * p.o_sb + h * p.o_sh + row * p.o_ss;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
            const float4 x = LdsF4(other + 32 * c + 4 * cg);
            float4 r;
            r.x = (o[i][2 * c].x * w0 + x.x * w1) * inv;
            r.y = (o[i][2 * c].y * w0 + x.y * w1) * inv;
            r.z = (o[i][2 * c + 1].x * w0 + x.z * w1) * inv;
            r.w = (o[i][2 * c + 1].y * w0 + x.w * w1) * inv;
            *reinterpret_cast<float4*>(o_row + 32 * c + 4 * cg) = r;
        }
        if (p.lse != nullptr && cg == 0) {
            p.lse[static_cast<int64_t>(bh) * p.seq_q + row] = l_all > 0.0f ? m_all * kLn2 + logf(l_all) : -CUDART_INF_F;
        }
    }
}

template <int D, int RT>
int LaunchF32(F32Params p, int64_t bh, cudaStream_t stream) {
    using G = F32Geom<D, RT>;
    p.m_blocks = (p.seq_q + G::kBM - 1) / G::kBM;
    const int64_t grid = bh * p.m_blocks;
    if (grid > 0x7fffffffLL) {
        return Fail(SCA_INVALID_ARGUMENT, "fp32 attention: grid of " + std::to_string(grid) + " blocks is out of range");
    }
    const void* fn = reinterpret_cast<const void*>(&fp32_tiled_attention_kernel<D, RT>);
    if (int rc = EnsureDynamicSmem(fn, G::kSmemBytes, "fp32_tiled_attention_kernel")) return rc;
    LaunchDependent(fp32_tiled_attention_kernel<D, RT>, grid, kF32Threads, G::kSmemBytes, stream, 1, p);
    return CheckLaunch("fp32_tiled_attention_kernel", stream);
}

// One CTA per SM at a time. A wave of 32-row tiles takes 0.83 of the time of a wave of 64-row tiles (93 against 112
// us at H=8, S=1024, D=128: the shared operand loads are spread over half the products), so the flat tile pays
// where it saves waves or where one wave holds either (H=8, S=256: 29.9 us flat, 35.1 tall).
struct F32Tiling {
    bool flat;
    int64_t waves;
};
F32Tiling TilingFor(int64_t bh, int64_t seq_q) {
    const int64_t sms = SmCount();
    const int64_t tall = (bh * ((seq_q + 63) / 64) + sms - 1) / sms;
    const int64_t flat = (bh * ((seq_q + 31) / 32) + sms - 1) / sms;
    return flat * 5 < tall * 6 ? F32Tiling{true, flat} : F32Tiling{false, tall};
}

// Whether one warp per query row is faster: a few rows or keys under very many heads, whose tiles are mostly padding. Both
// times in us, fitted to 490 calls (D=32 to 256; 1, 8, 32 and 512 heads in all; 1x1 to 300x300, 1x1000 and 130x1000 query
// rows and keys; warp per row / tiled): 512 heads, D=128 1x1 18 / 34, 17x17 29 / 36, 33x33 85 / 47, 1x64 39 / 35; D=256 1x64
// 39 / 59, 4x200 115 / 180, 33x33 89 / 71, 1x1000 1064 / 738; up to 148 tiles the tiled kernel wins at every size.
bool WarpPerRowIsFaster(const ScaFlashFwdParams& f) {
    const int64_t bh = f.batch * f.num_heads;
    const F32Tiling tiling = TilingFor(bh, f.seq_q);
    if (tiling.waves <= 1 || f.head_dim <= 32) return false;
    const double d = static_cast<double>(f.head_dim), keys = static_cast<double>(f.seq_kv), rows = static_cast<double>(f.seq_q);
    const double tiles = std::ceil(keys / (f.head_dim <= 128 ? 64.0 : 32.0));
    const double tiled = static_cast<double>(tiling.waves) * (3.5 + (f.head_dim <= 128 ? 0.042 : 0.0235) * d * tiles) * (tiling.flat ? 1.0 : 1.2);
    // a warp walks its keys one by one, more slowly where K and V do not fit into L2; many rows share the issue slots
    const double kv_bytes = static_cast<double>(f.batch * f.num_kv_heads) * keys * d * 8.0;
    const double chain = 6.0 + keys * (f.head_dim <= 96 ? 0.35 : 0.5) * (kv_bytes > 130e6 ? 2.1 : 1.0);
    const double pairs = static_cast<double>(bh) * rows * (keys - (f.causal ? (rows - 1.0) / 2.0 : 0.0)) * 1e-3;
    const double warp_per_row = std::max({chain, 18.0 + 0.07 * pairs, pairs * (f.head_dim <= 64 ? 0.13 : 0.15)});
    return tiled > 1.05 * warp_per_row;
}

template <int D>
int LaunchF32ForDim(const F32Params& p, int64_t bh, cudaStream_t stream) {
    return TilingFor(bh, p.seq_q).flat ? LaunchF32<D, 2>(p, bh, stream) : LaunchF32<D, 4>(p, bh, stream);
}

}  // namespace

// The calls the tiled kernel takes: 16-byte accesses to every row, 32-bit row indices, tiles that are not mostly padding.
// The others and the 16-bit types stay with the one-warp-per-row kernel.
bool Fp32TiledTakes(const ScaFlashFwdParams& f) {
    const int64_t strides[] = {f.q_sb, f.q_sh, f.q_ss, f.k_sb, f.k_sh, f.k_ss, f.v_sb, f.v_sh, f.v_ss, f.o_sb, f.o_sh, f.o_ss};
    for (const int64_t s : strides) {
        if (s % 4 != 0) return false;
    }
    return f.dtype_id == SCA_DTYPE_F32 && Aligned16(f.q) && Aligned16(f.k) && Aligned16(f.v) && Aligned16(f.out) &&
           f.seq_q < 0x7fffff00LL && f.seq_kv < 0x7fffff00LL && f.batch * f.num_heads < 0x7fffffffLL && !WarpPerRowIsFaster(f);
}

int LaunchFp32Tiled(const ScaFlashFwdParams& f, cudaStream_t stream) {
    F32Params p{};
    p.q = static_cast<const float*>(f.q);
    p.k = static_cast<const float*>(f.k);
    p.v = static_cast<const float*>(f.v);
    p.out = static_cast<float*>(f.out);
    p.lse = f.return_lse ? f.lse : nullptr;
    p.heads = static_cast<int>(f.num_heads);
    p.kv_heads = static_cast<int>(f.num_kv_heads);
    p.seq_q = static_cast<int>(f.seq_q);
    p.seq_kv = static_cast<int>(f.seq_kv);
    const int64_t bh = f.batch * f.num_heads;
    p.bh_count = static_cast<int>(bh);
    p.q_sb = f.q_sb; p.q_sh = f.q_sh; p.q_ss = f.q_ss;
    p.k_sb = f.k_sb; p.k_sh = f.k_sh; p.k_ss = f.k_ss;
    p.v_sb = f.v_sb; p.v_sh = f.v_sh; p.v_ss = f.v_ss;
    p.o_sb = f.o_sb; p.o_sh = f.o_sh; p.o_ss = f.o_ss;
    p.scale_log2 = f.scale * kLog2e;
    p.causal = f.causal;
    p.diagonal = f.diagonal;
    switch (f.head_dim) {
        case 32: return LaunchF32ForDim<32>(p, bh, stream);
        case 64: return LaunchF32ForDim<64>(p, bh, stream);
        case 96: return LaunchF32ForDim<96>(p, bh, stream);
        case 128: return LaunchF32ForDim<128>(p, bh, stream);
        case 160: return LaunchF32ForDim<160>(p, bh, stream);
        case 192: return LaunchF32ForDim<192>(p, bh, stream);
        case 224: return LaunchF32ForDim<224>(p, bh, stream);
        case 256: return LaunchF32ForDim<256>(p, bh, stream);
        default: break;
    }
    return Fail(SCA_INVALID_ARGUMENT, "attention: head_dim=" + std::to_string(f.head_dim) + " is not instantiated");
}

}  // namespace sca_b200

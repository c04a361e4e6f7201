// The large-product GEMM: CTA pairs (tcgen05 cta_group::2) on 256 x 512 output tiles.
//
// Two CTAs of a cluster share a tile. CTA r stages rows [128 r, 128 r + 128) of the A tile and of each of the tile's two
// 256-column B blocks; the even CTA issues, per 16-wide step, two M = 256, N = 256 MMAs that read both CTAs' shared memory
// and the same A rows, and each CTA finds its own 128 rows x 512 columns in its tensor memory - all of it.
//
// Why this tile: a 256 x 256 pair tile moves 32 KB per CTA from L2 to shared memory and reads 32 KB back for every 512
// cycles of MMA, which is the shared-memory port's whole 128 bytes a cycle; its tensor pipe was active 82 % of the cycles
// (ncu, 8192 x 8192 x 4096). Sharing A between two column blocks brings that to 48 + 64 KB per 1,024 cycles and takes a
// quarter of the L2 traffic away. Measured under the power cap (0.5 s loops, bf16, TFLOP/s; before = the better of 128 x 256
// single-CTA and 256 x 256 pair tiles / now):
//   8192 x 24576 x 4096 (y = x W^T)      1142 / 1302     24576 x 4096 x 8192 (dy^T x)    1176 / 1380
//   8192 x 4096 x 12288 (y = x W^T)      1177 / 1378     4096 x 12288 x 8192 (dy^T x)    1134 / 1332
//   8192 x 4096 x 24576 (dy W)           1200 / 1400     4096 x 151936 x 2048 (logits)   1079 / 1277
//   8192 x 12288 x 4096 (dy W)           1163 / 1337     4096 x 2048 x 151936 (dlogits W) 1153 / 1384
//   151936 x 2048 x 4096, fp32 +=        1005 / 1268     SwiGLU 8192 x 24576 x 4096      1096 / 1287
//
// Tensor memory holds no second tile, so the epilogue is kept off the critical path differently. The two column blocks are
// two accumulators with barriers of their own: all eight epilogue warps take block 0 into registers first, and the next
// tile's MMAs start on it - up to kWideAhead stages ahead - while block 1 is being taken; only then is anything stored.
//
// Tiles that do not fill the last wave of pairs are cut into their two column blocks where that lets the wave end sooner.
// No TMA load uses cluster multicast. Every wait is bounded (see sm100_common.cuh).
#pragma once

#include "gemm_sm100.cuh"

namespace halo {

constexpr int kWideStages = 4;
constexpr int kWideAhead = 3;                                   // stages block 0 may run ahead of block 1
constexpr int kWideStageBytes = 3 * kATileBytes;                // A 128 x 64, B 2 x 128 x 64 per CTA
constexpr int kWideEpiWarps = 8;
constexpr int kWideThreads = 64 + 32 * kWideEpiWarps;
constexpr int kWideStoreBytes = 4096;                           // per epilogue warp: 32 rows x 128 bytes
constexpr int kWideSmemBytes = kWideStages * kWideStageBytes + 1024 + kWideEpiWarps * kWideStoreBytes;

// tile load whose completion is counted on the even CTA's barrier (no multicast: one destination)
__device__ __forceinline__ void wide_tma(uint32_t dst, const CUtensorMap* m, uint32_t bar_cluster_addr, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
        "{%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void wide_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void wide_commit(uint32_t bar) {     // on the barrier at this offset in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}

// A work item of this kernel: GemmWork with b_mn / b_mn2 the origins of the two 256-column blocks (128 columns of each per
// CTA), pad0 the number of blocks (1 or 2), m_valid up to 256 and n_valid up to 512 (SwiGLU: up to 256, block 0 gate and
// block 1 up).
__device__ __forceinline__ bool wide_fetch(const GemmParams& p, int idx, int total, GemmWork& w) {
    if (idx >= total) return false;
    if (p.list) {
        w = p.list[idx];
        return true;
    }
    // whole tiles first; `pad_full` of them, then column halves (see launch_wide)
    int t = idx, half = -1;
    if (idx >= p.wide_full) {
        t = p.wide_full + ((idx - p.wide_full) >> 1);
        half = (idx - p.wide_full) & 1;
    }
    const int tiles_m = (p.M + 255) / 256;
    const int group_m = 8;                      // tile-rows that run together share B blocks through L2
    const int per_group = group_m * p.tiles_n;
    const int g = t / per_group;
    const int first_m = g * group_m;
    const int gsz = min(tiles_m - first_m, group_m);
    const int in_g = t - g * per_group;
    const int tm = first_m + in_g % gsz, tn = in_g / gsz;
    w.a_mn = tm * 256;
    w.a_k = w.b_k = 0;
    w.k_iters = (p.K + kBlockK - 1) / kBlockK;
    w.c_row = tm * 256;
    w.m_valid = min(256, p.M - tm * 256);
    w.pad1 = 0;
    if (p.epi == kEpiSwiglu) {
        w.b_mn = tn * 256;
        w.b_mn2 = p.swiglu_f + tn * 256;
        w.c_col = tn * 256;
        w.n_valid = min(256, p.swiglu_f - tn * 256);
        w.pad0 = 2;
    } else {
        w.c_col = tn * 512 + (half > 0 ? 256 : 0);
        w.b_mn = w.c_col;
        w.b_mn2 = w.c_col + 256;
        w.n_valid = max(0, min(half < 0 ? 512 : 256, p.N - w.c_col));
        w.pad0 = w.n_valid > 256 ? 2 : 1;
        if (w.n_valid == 0) w.k_iters = 0, w.m_valid = 0;       // the empty half of a ragged tile
    }
    return true;
}

// 128 bytes of each of a warp's 32 rows (the lane's row, eight 16-byte units in `v`) go through shared memory, so that eight
// lanes write one row's 128 bytes. `f` is called once per 16-byte unit with (row, unit, value).
template <typename F>
__device__ __forceinline__ void through_smem(uint32_t stage, int lane, const uint32_t (&v)[32], F&& f) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + lane * 128 + ((u ^ (lane & 7)) << 4)), "r"(v[4 * u]),
                     "r"(v[4 * u + 1]), "r"(v[4 * u + 2]), "r"(v[4 * u + 3])
                     : "memory");
    __syncwarp();
    const int u = lane & 7;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 4 * i + (lane >> 3);
        uint4 x;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(stage + r * 128 + ((u ^ (r & 7)) << 4)));
        f(r, u, x);
    }
    __syncwarp();
}

// A warp's share of an accumulator block - 32 rows, 128 columns - leaves tensor memory before it is stored, as packed bf16
// pairs all at once (32 * N32 columns), or as fp32 values in two halves, so that the next tile can have the block.
template <int N32>
__device__ __forceinline__ void wide_take_bf16(uint32_t t_addr, float alpha, bool zero, uint32_t (&pk)[16 * N32]) {
#pragma unroll
    for (int c = 0; c < N32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(t_addr + 32 * c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j)
            pk[16 * c + j] = zero ? 0u : pack_bf16(__uint_as_float(r[2 * j]) * alpha, __uint_as_float(r[2 * j + 1]) * alpha);
    }
}
// Where a warp's rows go: by TMA (`map`, with the warp's first row and the tile's column 0 in C) where a whole 32-row block of
// 128 bytes exists, else by the lanes. Ordinary stores from the transposition buffer - four 128-byte pieces an instruction -
// take longer than the products they follow once the reduction is short: weight gradients of experts with 190 rows, 805 MB of
// them, took 332 us that way, 198 us without the stores and 305 us by TMA.
struct WideOut {
    const CUtensorMap* map;     // null: the lanes store
    void* base;                 // the warp's first row, column 0 of the tile
    long long ld;
    int row, col;               // coordinates of `base` in the map
    int rows, n_valid;          // rows of this warp that exist, columns of the tile
    uint32_t stage;
    int lane;
};

// 128 bytes of the warp's 32 rows to columns col .. of the tile (`col` counted in elements of BYTES bytes)
template <int BYTES, bool ADD>
__device__ __forceinline__ void wide_put_row_block(const WideOut& o, const uint32_t (&v)[32], int col) {
    constexpr int kUnit = 16 / BYTES, kCols = 128 / BYTES;
    if (o.map && o.rows == 32 && col + kCols <= o.n_valid) {        // uniform over the warp
        if (o.lane == 0) tma_store_wait_read<0>();                  // the buffer's previous block has been read
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 8; ++u)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o.stage + o.lane * 128 + ((u ^ (o.lane & 7)) << 4)),
                         "r"(v[4 * u]), "r"(v[4 * u + 1]), "r"(v[4 * u + 2]), "r"(v[4 * u + 3])
                         : "memory");
        fence_proxy_async_smem();
        __syncwarp();
        if (o.lane == 0) {
            if (ADD) tma_reduce_add_2d(o.map, o.stage, o.col + col, o.row);
            else tma_store_2d(o.map, o.stage, o.col + col, o.row);
            tma_store_commit();
        }
        return;
    }
    if (o.map) {                                                    // the lanes take over a buffer that TMA may still read
        if (o.lane == 0) tma_store_wait_read<0>();
        __syncwarp();
    }
    through_smem(o.stage, o.lane, v, [&](int rr, int u, uint4 x) {
        const int c = col + u * kUnit;
        if (rr >= o.rows || c + kUnit > o.n_valid) return;
        uint8_t* d = reinterpret_cast<uint8_t*>(o.base) + ((long long)rr * o.ld + c) * BYTES;
        if (ADD) {
            const float4 c0 = *reinterpret_cast<const float4*>(d);
            *reinterpret_cast<float4*>(d) = make_float4(c0.x + __uint_as_float(x.x), c0.y + __uint_as_float(x.y),
                                                        c0.z + __uint_as_float(x.z), c0.w + __uint_as_float(x.w));
        } else {
            *reinterpret_cast<uint4*>(d) = x;
        }
    });
}

template <int N64>
__device__ __forceinline__ void wide_put_bf16(const WideOut& o, const uint32_t (&pk)[32 * N64], int col0) {
#pragma unroll
    for (int h = 0; h < N64; ++h) {
        if (col0 + 64 * h >= o.n_valid) break;                     // uniform over the warp
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = pk[32 * h + j];
        wide_put_row_block<2, false>(o, v, col0 + 64 * h);
    }
}
__device__ __forceinline__ void wide_take_f32(uint32_t t_addr, float alpha, bool zero, uint32_t (&v)[2][32]) {
#pragma unroll
    for (int c = 0; c < 2; ++c) tmem_ld_32x32(t_addr + 32 * c, v[c]);
    tmem_ld_wait();
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < 32; ++j) v[c][j] = zero ? 0u : __float_as_uint(__uint_as_float(v[c][j]) * alpha);
}
// fp32 output; accumulation of whole blocks is a TMA reduction in L2: every element receives exactly one addition per launch,
// so the result is that of a load, an addition and a store, without the wait for the load. Subnormal sums survive it, which
// they do not in `red.global.add.f32`.
template <bool ADD>
__device__ __forceinline__ void wide_put_f32(const WideOut& o, const uint32_t (&v)[2][32], int col0) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        if (col0 + 32 * c >= o.n_valid) break;
        wide_put_row_block<4, ADD>(o, v[c], col0 + 32 * c);
    }
}
// bf16 output += tile: the sum is formed in fp32 and rounded once
__device__ __forceinline__ void wide_add_bf16(__nv_bfloat16* dst, long long ld, const uint32_t (&v)[2][32], int col0, int n_valid, int rows,
                                              int lane) {
    if (lane >= rows) return;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            const int col = col0 + 32 * c + j;
            if (col + 8 > n_valid) continue;
            uint4* d = reinterpret_cast<uint4*>(dst + (long long)lane * ld + col);
            const uint4 old = *d;
            const uint32_t o[4] = {old.x, old.y, old.z, old.w};
            uint32_t n[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o[q]));
                n[q] = pack_bf16(f.x + __uint_as_float(v[c][j + 2 * q]), f.y + __uint_as_float(v[c][j + 2 * q + 1]));
            }
            *d = make_uint4(n[0], n[1], n[2], n[3]);
        }
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kWideThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmAux,
                 const __grid_constant__ GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[kWideStages], bar_empty[kWideStages], bar_tfull[2], bar_tempty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    const bool leader = rank == 0;
    const uint32_t tiles_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const bool poisoned = status_poisoned(p.status);

    if (threadIdx.x == 0) {
        abort_flag = poisoned ? 1 : 0;
        for (int s = 0; s < kWideStages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);    // the even CTA's: its producer's arrive + both CTAs' bytes
            mbar_init(smem_u32(&bar_empty[s]), 1);   // one multicast commit
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&bar_tfull[a]), 1);                       // one multicast commit
            mbar_init(smem_u32(&bar_tempty[a]), 2 * kWideEpiWarps);      // the even CTA's: the epilogue warps of both CTAs
        }
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();         // the peer's barriers exist before anything is signalled across the pair
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    // Every role reads its next item before it works on this one: a listed item comes from L2 or HBM, and the wait for it would
    // otherwise drain the tensor pipe between tiles.
    const int total = p.list ? *p.list_count : p.wide_items;
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (warp == 0) {
        // ---------------- TMA producer (both CTAs, each for its halves) ----------------
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            GemmWork w, next;
            bool more = wide_fetch(p, first, total, next);
            for (int idx = first + step; more && !abort_flag; idx += step) {
                w = next;
                more = wide_fetch(p, idx, total, next);
                const int a_mn = w.a_mn + int(rank) * 128;
                for (int kb = 0; kb < w.k_iters; ++kb) {
                    if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, &abort_flag, p.status)) break;
                    if (leader) mbar_expect_tx(smem_u32(&bar_full[stage]), 2 * (1 + w.pad0) * kATileBytes);
                    const uint32_t full = map_to_cta(smem_u32(&bar_full[stage]), 0);
                    const uint32_t sa = tiles_base + stage * kWideStageBytes;
                    if (A_MN) {
                        wide_tma(sa, &tmA, full, a_mn, w.a_k + kb * kBlockK);
                        wide_tma(sa + 8192, &tmA, full, a_mn + 64, w.a_k + kb * kBlockK);
                    } else {
                        wide_tma(sa, &tmA, full, w.a_k + kb * kBlockK, a_mn);
                    }
                    for (int j = 0; j < w.pad0; ++j) {
                        const uint32_t sb = sa + (1 + j) * kATileBytes;
                        const int b_mn = (j ? w.b_mn2 : w.b_mn) + int(rank) * 128;
                        if (B_MN) {
                            wide_tma(sb, &tmB, full, b_mn, w.b_k + kb * kBlockK);
                            wide_tma(sb + 8192, &tmB, full, b_mn + 64, w.b_k + kb * kBlockK);
                        } else {
                            wide_tma(sb, &tmB, full, w.b_k + kb * kBlockK, b_mn);
                        }
                    }
                    if (++stage == kWideStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (even CTA only) ----------------
        if (lane == 0 && leader) {
            constexpr uint32_t idesc = make_idesc_bf16(256, kBlockN, A_MN ? 1 : 0, B_MN ? 1 : 0);
            int stage = 0;
            uint32_t phase = 0, used[2] = {0, 0};       // tiles each accumulator block has served
            GemmWork w, next;
            auto issue = [&](int s, int block, bool accumulate) {
                const uint32_t sa = tiles_base + s * kWideStageBytes, sb = sa + (1 + block) * kATileBytes;
#pragma unroll
                for (int k = 0; k < kBlockK / 16; ++k) {
                    const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, 8192, 1024) : make_smem_desc(sa + k * 32, 16, 1024);
                    const uint64_t db = B_MN ? make_smem_desc(sb + k * 2048, 8192, 1024) : make_smem_desc(sb + k * 32, 16, 1024);
                    wide_mma(tmem_base + block * kBlockN, da, db, idesc, (accumulate || k) ? 1u : 0u);
                }
            };
            bool more = wide_fetch(p, first, total, next);
            for (int idx = first + step; more && !abort_flag; idx += step) {
                w = next;
                more = wide_fetch(p, idx, total, next);
                if (!mbar_wait(smem_u32(&bar_tempty[0]), (used[0] & 1u) ^ 1u, &abort_flag, p.status)) break;
                tc_fence_after();
                ++used[0];
                bool ok = true;
                if (w.pad0 == 1) {
                    for (int kb = 0; kb < w.k_iters; ++kb) {
                        if (!mbar_wait(smem_u32(&bar_full[stage]), phase, &abort_flag, p.status)) { ok = false; break; }
                        tc_fence_after();
                        issue(stage, 0, kb != 0);
                        wide_commit(smem_u32(&bar_empty[stage]));
                        if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
                    }
                    if (!ok) break;
                    wide_commit(smem_u32(&bar_tfull[0]));
                    continue;
                }
                // block 0 of the first stages, then - once the previous tile's block 1 is drained - block 1 of the same
                const int ahead = min(w.k_iters, kWideAhead);
                int s0 = stage;
                uint32_t ph0 = phase;
                for (int kb = 0; kb < ahead; ++kb) {
                    if (!mbar_wait(smem_u32(&bar_full[s0]), ph0, &abort_flag, p.status)) { ok = false; break; }
                    tc_fence_after();
                    issue(s0, 0, kb != 0);
                    if (++s0 == kWideStages) { s0 = 0; ph0 ^= 1u; }
                }
                // a short reduction: block 0 is complete, and its epilogue need not wait for the other block's turn
                if (ok && w.k_iters <= ahead) wide_commit(smem_u32(&bar_tfull[0]));
                if (!ok || !mbar_wait(smem_u32(&bar_tempty[1]), (used[1] & 1u) ^ 1u, &abort_flag, p.status)) break;
                tc_fence_after();
                ++used[1];
                for (int kb = 0; kb < ahead; ++kb) {
                    issue(stage, 1, kb != 0);
                    wide_commit(smem_u32(&bar_empty[stage]));    // both CTAs' producers may refill the stage
                    if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
                }
                for (int kb = ahead; kb < w.k_iters; ++kb) {
                    if (!mbar_wait(smem_u32(&bar_full[stage]), phase, &abort_flag, p.status)) { ok = false; break; }
                    tc_fence_after();
                    issue(stage, 0, true);
                    if (kb + 1 == w.k_iters) wide_commit(smem_u32(&bar_tfull[0]));
                    issue(stage, 1, true);
                    wide_commit(smem_u32(&bar_empty[stage]));
                    if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
                }
                if (!ok) break;
                wide_commit(smem_u32(&bar_tfull[1]));
            }
        }
    } else {
        // ---------------- epilogue (both CTAs, each its own 128 rows) ----------------
        const int quarter = warp & 3;                    // tensor-memory lanes this warp may read
        const int row0 = quarter * 32;
        const int half = (warp - 2) >> 2;                // which 128 of a block's 256 columns
        const uint32_t stage = tiles_base + kWideStages * kWideStageBytes + (warp - 2) * kWideStoreBytes;
        const uint32_t t_row = tmem_base + (uint32_t(row0) << 16) + half * 128;
        const bool f32 = p.epi == kEpiStoreF32 || p.epi == kEpiAccumF32;
        const bool wide_values = f32 || p.epi == kEpiAccumBf16;
        uint32_t used[2] = {0, 0};
        GemmWork w, next;
        auto ready = [&](int block) -> bool {            // the block's products are complete
            if (!mbar_wait_warp(smem_u32(&bar_tfull[block]), used[block]++ & 1u, &abort_flag, p.status)) return false;
            tc_fence_after();
            return true;
        };
        auto release = [&](int block) {                  // the block may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&bar_tempty[block]), 0));
        };
        bool more = wide_fetch(p, first, total, next);
        for (int idx = first + step; more && !warp_aborted(&abort_flag); idx += step) {
            w = next;
            more = wide_fetch(p, idx, total, next);
            const int rows = max(0, min(32, w.m_valid - int(rank) * 128 - row0));       // rows of this warp that exist
            const long long c_row = (long long)w.c_row + int(rank) * 128 + row0;
            const bool zero = w.k_iters == 0;
            WideOut out{p.tma_c ? &tmC : nullptr, nullptr, p.ldc, (int)c_row, w.c_col, rows, w.n_valid, stage, lane};
            out.base = reinterpret_cast<uint8_t*>(p.C) + (c_row * p.ldc + w.c_col) * (f32 ? 4 : 2);
            if (wide_values) {
                bool ok = true;
                for (int block = 0; block < w.pad0; ++block) {
                    if (!(ok = ready(block))) break;
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        uint32_t v[2][32];
                        wide_take_f32(t_row + block * kBlockN + 64 * h, p.alpha, zero, v);
                        if (h == 1) release(block);
                        const int col0 = block * 256 + half * 128 + 64 * h;
                        if (p.epi == kEpiAccumF32) wide_put_f32<true>(out, v, col0);
                        else if (f32) wide_put_f32<false>(out, v, col0);
                        else wide_add_bf16(reinterpret_cast<__nv_bfloat16*>(out.base), p.ldc, v, col0, w.n_valid, rows, lane);
                    }
                }
                if (!ok) break;
                continue;
            }
            if (p.epi == kEpiSwiglu) {
                // block 0 is the gate, block 1 the up half; both rounded to bf16 first, so that a recomputation from the saved
                // pre-activations sees the same values
                if (!ready(0) || !ready(1)) break;
                WideOut gate = out, up = out;
                gate.map = up.map = p.tma_aux ? &tmAux : nullptr;
                gate.ld = up.ld = p.ld_aux;
                gate.base = reinterpret_cast<__nv_bfloat16*>(p.aux) + c_row * p.ld_aux + w.c_col;
                up.base = reinterpret_cast<__nv_bfloat16*>(gate.base) + p.swiglu_f;
                up.col = w.c_col + p.swiglu_f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t g[32], u[32];
                    wide_take_bf16<2>(t_row + 64 * h, p.alpha, zero, g);
                    wide_take_bf16<2>(t_row + kBlockN + 64 * h, p.alpha, zero, u);
                    if (h == 1) {
                        release(0);
                        release(1);
                    }
                    const int col0 = half * 128 + 64 * h;
                    if (p.aux) {
                        wide_put_bf16<1>(gate, g, col0);
                        wide_put_bf16<1>(up, u, col0);
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g[j]));
                        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[j]));
                        g[j] = pack_bf16(x.x * sigmoid_fast(x.x) * y.x, x.y * sigmoid_fast(x.y) * y.y);
                    }
                    wide_put_bf16<1>(out, g, col0);
                }
                continue;
            }
            bool ok = true;
#pragma unroll 1
            for (int block = 0; block < w.pad0; ++block) {
                uint32_t v[64];
                if (!(ok = ready(block))) break;
                wide_take_bf16<4>(t_row + block * kBlockN, p.alpha, zero, v);
                release(block);
                wide_put_bf16<2>(out, v, block * 256 + half * 128);
            }
            if (!ok) break;
        }
        if (lane == 0) tma_store_wait<0>();              // every block handed to TMA has been written
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (abort_flag && !poisoned) {
        uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) { }
        __syncthreads();
    }
    cluster_sync_all();         // nothing of the pair is in flight towards the other CTA's memory any more
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
    }
}

}  // namespace halo

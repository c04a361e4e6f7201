// Products with few rows (the tokens of a sampling step): C[m, n] = alpha * sum_k X[m, k] W[n, k], M <= 256, both operands
// K-major, with a plain bf16 / fp32 store or the SwiGLU epilogue.
//
// What bounds them: the weight is read once and M is far below the machine's balance, so HBM bandwidth is the floor. The
// large-tile kernels give such a product N / 256 tiles - 16 for a 4096-wide projection, on 148 SMs - and spend the rest of
// their 128 or 256 tile rows on padding. Here the WEIGHT rows are the 128 rows of the tensor-core tile and the tokens are
// its columns (16 .. 256, padded to a power of two), and a cluster of up to 8 CTAs cuts the reduction, so that every SM
// streams weights. Each CTA keeps a ring of 16 KB weight tiles in flight (two CTAs fit an SM, so one CTA's prologue and
// epilogue run under the other's stream); the partial sums stay fp32, meet in distributed shared memory in a fixed order,
// and every CTA of the cluster finishes its share of the tokens. No workspace, one launch. The cuts and the choice of kernel follow
// the number of tokens (few_rows_wins), so a token's result may differ in its last bit between calls of different sizes; calls
// of one size repeat exactly.
//
// Measured (B200, weights cycled so that L2 does not hold them; the large-tile kernels as they were / this one, us; floor =
// weight bytes at the measured copy rate; short reductions: see few_rows_wins):
//   N x K             floor    M = 1          16             64             128            256
//   4096 x 12288      15.4     69.7 / 22.8    69.9 / 23.8    69.9 / 24.8    71.0 / 28.2    71.4 / 39.7
//   6144 x 4096        7.7     28.1 / 14.8    28.1 / 15.2    28.6 / 17.2    30.5 / 20.5    30.6 / 40.9
//   4096 x 4096        5.1     27.8 / 11.9    27.7 / 12.2    27.7 / 13.9    28.9 / 16.3    29.1 / 23.7
//   5120 x 2048        3.2     17.3 /  9.8    17.4 / 10.3    18.1 / 12.2    20.7 / 15.2    20.7 / 33.2
//   128 x 2048         0.1     15.3 /  6.1    15.3 /  6.4    15.4 /  7.9    16.0 / 10.1    16.1 / 14.5
//   151936 x 4096    190.3    215.8 / 197.5  208.1 / 205.7  212.8 / 241.7  220.4 / 286.1  293.2 / 511.5
//   SwiGLU 24576 x 4096 30.8   53.4 / 40.5    44.3 / 41.7    45.1 / 48.9    45.0 / 57.5    63.7 / 121.2
//   SwiGLU 12288 x 2048  7.7   21.5 / 14.5    21.1 / 15.6    20.7 / 20.1    20.7 / 26.6    20.7 / 46.3
// Tiles of fewer weight rows, so that the grid fills all 296 block slots, measured slower (4096 x 12288: 34 against 23 us):
// clusters of eight then no longer find room in one wave.
#pragma once

#include "gemm_sm100.cuh"

namespace halo {

constexpr int kFewThreads = 192;
constexpr int kFewMaxStages = 6;
constexpr int kFewWBytes = 128 * kBlockK * 2;      // weight tile of one stage: 128 rows x 64

// The ring for tiles of m_pad columns: two CTAs an SM up to 128 columns, one above. Once all products are done it holds the
// [m_pad][128] fp32 partial sums.
__host__ __device__ constexpr int few_stage_bytes(int m_pad) { return kFewWBytes + m_pad * kBlockK * 2; }
__host__ __device__ constexpr int few_stages(int m_pad) {
    const int n = (m_pad <= 128 ? 110 : 220) * 1024 / few_stage_bytes(m_pad);
    return n < kFewMaxStages ? n : kFewMaxStages;
}
__host__ __device__ constexpr int few_smem_bytes(int m_pad) { return few_stages(m_pad) * few_stage_bytes(m_pad) + 1024; }     // + alignment
__host__ __device__ constexpr bool few_sums_fit(int m_pad) { return m_pad * 128 * 4 <= few_stages(m_pad) * few_stage_bytes(m_pad); }
static_assert(few_sums_fit(16) && few_sums_fit(32) && few_sums_fit(64) && few_sums_fit(128) && few_sums_fit(256),
              "the partial sums fit over the ring");
constexpr int kFewMaxSmemBytes = few_smem_bytes(256);
static_assert(few_smem_bytes(16) <= kFewMaxSmemBytes && few_smem_bytes(32) <= kFewMaxSmemBytes &&
              few_smem_bytes(64) <= kFewMaxSmemBytes && few_smem_bytes(128) <= kFewMaxSmemBytes, "the widest tile needs the most");

struct FewParams {
    void* C;
    void* aux;           // SwiGLU: optional [M, 2F] pre-activations
    long long ldc, ld_aux;
    int epi;             // kEpiStoreBf16, kEpiStoreF32 or kEpiSwiglu
    float alpha;
    int M, N, K;         // N: rows of W (2F for SwiGLU)
    int m_pad;           // tile columns: 16, 32, 64, 128 or 256
    int stages;
    int parts;           // CTAs of a cluster = cuts of the reduction
    int swiglu_f;        // F for SwiGLU, else 0
    int* status;
};

__device__ __forceinline__ float2 ld_cluster_f2(uint32_t local_addr, uint32_t rank) {
    float2 v;
    const uint32_t a = map_to_cta(local_addr, rank);
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}

__global__ void __launch_bounds__(kFewThreads)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                     const __grid_constant__ FewParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[kFewMaxStages], bar_empty[kFewMaxStages], bar_done;
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t rank = cluster_cta_rank();
    const int tile = blockIdx.x / p.parts;
    const int stage_bytes = few_stage_bytes(p.m_pad);
    const int tmem_cols = p.m_pad < 32 ? 32 : p.m_pad;

    if (threadIdx.x == 0) {
        // the CTAs of a cluster may see the status word at different times: nobody leaves early, the barriers below are met
        abort_flag = status_poisoned(p.status) ? 1 : 0;
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_done), 1);
        mbar_fence_init();
        tma_prefetch_desc(&tmW);
        tma_prefetch_desc(&tmX);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_slot;

    // this CTA's share of the reduction, in 64-wide blocks
    const int kb_total = (p.K + kBlockK - 1) / kBlockK;
    const int kb_share = (kb_total + p.parts - 1) / p.parts;
    const int kb_lo = min(kb_total, (int)rank * kb_share), kb_n = min(kb_total, kb_lo + kb_share) - kb_lo;

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < kb_n && !abort_flag; ++i) {
                const int s = i % p.stages;
                if (!mbar_wait(smem_u32(&bar_empty[s]), ((i / p.stages) & 1) ^ 1u, &abort_flag, p.status)) break;
                const uint32_t full = smem_u32(&bar_full[s]), sw = base + s * stage_bytes, sx = sw + kFewWBytes;
                const int k0 = (kb_lo + i) * kBlockK;
                mbar_expect_tx(full, stage_bytes);
                if (p.swiglu_f) {
                    tma_load_2d(sw, &tmW, full, k0, tile * 64);            // 64 gate rows, then their 64 up rows
                    tma_load_2d(sw + kFewWBytes / 2, &tmW, full, k0, p.swiglu_f + tile * 64);
                } else {
                    tma_load_2d(sw, &tmW, full, k0, tile * 128);
                }
                tma_load_2d(sx, &tmX, full, k0, 0);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = make_idesc_bf16(128, p.m_pad, 0, 0);
            bool ok = true;
            for (int i = 0; i < kb_n && !abort_flag; ++i) {
                const int s = i % p.stages;
                if (!mbar_wait(smem_u32(&bar_full[s]), (i / p.stages) & 1, &abort_flag, p.status)) { ok = false; break; }
                tc_fence_after();
                const uint32_t sw = base + s * stage_bytes, sx = sw + kFewWBytes;
#pragma unroll
                for (int k = 0; k < kBlockK / 16; ++k)
                    tc_mma_f16(tmem, make_smem_desc(sw + k * 32, 16, 1024), make_smem_desc(sx + k * 32, 16, 1024), idesc,
                               (i | k) != 0 ? 1u : 0u);
                tc_commit(smem_u32(&bar_empty[s]));
            }
            if (ok) tc_commit(smem_u32(&bar_done));
        }
    } else {
        // partial sums to shared memory, token-major: [m_pad][128] fp32 over the ring, which is dead once all MMAs are done
        const int quarter = warp & 3;
        float* part = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw)));
        if (mbar_wait_warp(smem_u32(&bar_done), 0, &abort_flag, p.status)) {
            tc_fence_after();
            const uint32_t t_row = tmem + (uint32_t(quarter * 32) << 16);
#pragma unroll 1
            for (int c = 0; c < p.m_pad; c += 16) {
                uint32_t r[16];
                if (kb_n > 0) {
                    tmem_ld_32x16(t_row + c, r);
                    tmem_ld_wait();
                }
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    part[(c + j) * 128 + quarter * 32 + lane] = kb_n > 0 ? __uint_as_float(r[j]) * p.alpha : 0.f;
            }
            tc_fence_before();
        }
    }
    __syncthreads();
    if (p.parts > 1) cluster_sync_all();            // every CTA's partial sums are in place

    if (warp >= 2 && !abort_flag) {
        // thread t of the four warps owns two neighbouring columns of every second token of this CTA's share
        const int t = threadIdx.x - 64;
        const int pair = t & 63, half = t >> 6;
        for (int m = 2 * (int)rank + half; m < p.M; m += 2 * p.parts) {
            if (!p.swiglu_f) {
                const int n = tile * 128 + 2 * pair;
                if (n >= p.N) continue;
                const uint32_t a = base + 4u * (uint32_t)(m * 128 + 2 * pair);
                float2 v = make_float2(0.f, 0.f);
                for (int c = 0; c < p.parts; ++c) {
                    const float2 u = ld_cluster_f2(a, c);
                    v.x += u.x;
                    v.y += u.y;
                }
                if (p.epi == kEpiStoreF32)
                    *reinterpret_cast<float2*>(reinterpret_cast<float*>(p.C) + (long long)m * p.ldc + n) = v;
                else
                    *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)m * p.ldc + n) = pack_bf16(v.x, v.y);
            } else if (pair < 32) {
                const int n = tile * 64 + 2 * pair;
                if (n >= p.swiglu_f) continue;
                const uint32_t a = base + 4u * (uint32_t)(m * 128 + 2 * pair);
                float2 g = make_float2(0.f, 0.f), u = make_float2(0.f, 0.f);
                for (int c = 0; c < p.parts; ++c) {
                    const float2 x = ld_cluster_f2(a, c), y = ld_cluster_f2(a + 256, c);
                    g.x += x.x; g.y += x.y;
                    u.x += y.x; u.y += y.y;
                }
                // rounded to bf16 before the activation, as the large-tile epilogue does (see gemm_sm100.cuh)
                const uint32_t gp = pack_bf16(g.x, g.y), up = pack_bf16(u.x, u.y);
                const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gp));
                const float2 uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&up));
                *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)m * p.ldc + n) =
                    pack_bf16(gf.x * sigmoid_fast(gf.x) * uf.x, gf.y * sigmoid_fast(gf.y) * uf.y);
                if (p.aux) {
                    __nv_bfloat16* pre = reinterpret_cast<__nv_bfloat16*>(p.aux) + (long long)m * p.ld_aux + n;
                    *reinterpret_cast<uint32_t*>(pre) = gp;
                    *reinterpret_cast<uint32_t*>(pre + p.swiglu_f) = up;
                }
            }
        }
    }
    // teardown
    __syncthreads();
    if (abort_flag) {
        // copies that may still be in flight land before the CTA's memory is reused
        uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) { }
        __syncthreads();
    }
    if (p.parts > 1) cluster_sync_all();            // nobody leaves while its partial sums are still being read
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, tmem_cols);
    }
}

}  // namespace halo

// bf16 GEMM for sm_100a on the 5th-generation tensor cores.
//
//   D[m, n] (+)= alpha * sum_k A(m, k) * B(n, k)
//
// One persistent CTA per SM walks a list of 128 x 256 output tiles. Operand tiles are brought
// into 128-byte-swizzled shared memory by TMA (each CTA fetches its own tiles), a single thread
// issues tcgen05.mma into one of two 256-column TMEM accumulators, and four epilogue warps drain
// the other accumulator with tcgen05.ld while the next tile is being multiplied.
//
// Either operand may be "K-major" (the reduction index is the contiguous one, the layout of
// y = x W^T) or "MN-major" (the reduction index walks rows, the layout of dx = dy W and of
// dW = dy^T x), so forward, data-gradient and weight-gradient products all read the tensors in
// place. The tile list is either derived from (M, N, K) or read from device memory, which is how
// the grouped (per-expert) products of an MoE layer run without a host round trip.
//
// Replaces what the reference obtains from cuBLAS (F.linear) and from torch's grouped_mm
// (halo/kernels/grouped_mm.py:30-51, halo/kernels/expert_gemm.py:14-35).
#include "gemm_few_rows.cuh"
#include "gemm_sm100.cuh"
#include "gemm_wide_sm100.cuh"

#include <stdio.h>

namespace halo {

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ GemmParams p) {
    if (status_poisoned(p.status)) return;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[kStages], bar_empty[kStages], bar_tfull[2], bar_tempty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t tiles_base = (smem_u32(smem_raw) + 1023u) & ~1023u;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&bar_tfull[a]), 1);
            mbar_init(smem_u32(&bar_tempty[a]), 4);
        }
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    const int total = p.list ? *p.list_count : p.tiles_m * p.tiles_n;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            GemmWork w;
            for (int idx = blockIdx.x; fetch_work(p, idx, total, w) && !abort_flag;
                 idx += gridDim.x) {
                for (int kb = 0; kb < w.k_iters; ++kb) {
                    if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, &abort_flag, p.status))
                        break;
                    const uint32_t full = smem_u32(&bar_full[stage]);
                    const uint32_t sa = tiles_base + stage * kStageBytes;
                    const uint32_t sb = sa + kATileBytes;
                    mbar_expect_tx(full, kStageBytes);
                    if (A_MN) {
                        tma_load_2d(sa, &tmA, full, w.a_mn, w.a_k + kb * kBlockK);
                        tma_load_2d(sa + 8192, &tmA, full, w.a_mn + 64, w.a_k + kb * kBlockK);
                    } else {
                        tma_load_2d(sa, &tmA, full, w.a_k + kb * kBlockK, w.a_mn);
                    }
                    if (B_MN) {
                        tma_load_2d(sb, &tmB, full, w.b_mn, w.b_k + kb * kBlockK);
                        tma_load_2d(sb + 8192, &tmB, full, w.b_mn + 64, w.b_k + kb * kBlockK);
                        tma_load_2d(sb + 16384, &tmB, full, w.b_mn2, w.b_k + kb * kBlockK);
                        tma_load_2d(sb + 24576, &tmB, full, w.b_mn2 + 64, w.b_k + kb * kBlockK);
                    } else {
                        tma_load_2d(sb, &tmB, full, w.b_k + kb * kBlockK, w.b_mn);
                        tma_load_2d(sb + 16384, &tmB, full, w.b_k + kb * kBlockK, w.b_mn2);
                    }
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            constexpr uint32_t idesc = make_idesc_bf16(kBlockM, kBlockN, A_MN ? 1 : 0, B_MN ? 1 : 0);
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            GemmWork w;
            for (int idx = blockIdx.x; fetch_work(p, idx, total, w) && !abort_flag;
                 idx += gridDim.x) {
                if (!mbar_wait(smem_u32(&bar_tempty[acc]), acc_phase ^ 1u, &abort_flag, p.status))
                    break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * kBlockN;
                bool ok = true;
                for (int kb = 0; kb < w.k_iters; ++kb) {
                    if (!mbar_wait(smem_u32(&bar_full[stage]), phase, &abort_flag, p.status)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = tiles_base + stage * kStageBytes;
                    const uint32_t sb = sa + kATileBytes;
#pragma unroll
                    for (int k = 0; k < kBlockK / 16; ++k) {
                        const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, 8192, 1024)
                                                 : make_smem_desc(sa + k * 32, 16, 1024);
                        const uint64_t db = B_MN ? make_smem_desc(sb + k * 2048, 8192, 1024)
                                                 : make_smem_desc(sb + k * 32, 16, 1024);
                        tc_mma_f16(d_tmem, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
                    }
                    tc_commit(smem_u32(&bar_empty[stage]));  // stage reusable once these MMAs retire
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                tc_commit(smem_u32(&bar_tfull[acc]));  // accumulator complete
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1u;
                }
            }
        }
    } else {
        // ---------------- epilogue: TMEM -> registers -> global ----------------
        const int quarter = warp & 3;  // TMEM lanes this warp may read: [32*quarter, 32*quarter+32)
        const int row_in_tile = quarter * 32 + lane;
        const uint32_t epi_stage = tiles_base + kStages * kStageBytes + quarter * kEpiStageBytesPerWarp;
        int acc = 0;
        uint32_t acc_phase = 0;
        GemmWork w;
        for (int idx = blockIdx.x; fetch_work(p, idx, total, w) && !warp_aborted(&abort_flag); idx += gridDim.x) {
            if (!mbar_wait_warp(smem_u32(&bar_tfull[acc]), acc_phase, &abort_flag, p.status)) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + acc * kBlockN + (uint32_t(quarter * 32) << 16);
            epilogue_tile(p, w, t_row, row_in_tile, epi_stage);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[acc]));
            if (++acc == 2) {
                acc = 0;
                acc_phase ^= 1u;
            }
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (abort_flag) {
        // give copies that may still be in flight time to land before the CTA's memory is reused
        uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 2000000ull) { }
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}


// ---------------------------------------------------------------------------------------------
// Tile lists for grouped (per-expert) products, built on the device from the expert segments.
// Segment e occupies rows [seg_start[e], seg_start[e] + seg_rows[e]) of the grouped operand;
// seg_start is a multiple of 128 and the rows between segments are zero.
// ---------------------------------------------------------------------------------------------

// Rows grouped along M:  C[rows of e] = A[rows of e] * op(B_e).
//   b_mn_stride / b_k_stride: how far expert e's weights sit along B's N / reduction coordinate.
// One block per expert: it adds up the items of the experts before it and writes its own. (One block walking the experts took
// 20 us for 128 experts of a handful of rows and 156 us for 65,536 tokens; now about 5 us.)
__global__ void __launch_bounds__(256)
plan_grouped_m_kernel(const int* __restrict__ seg_start, const int* __restrict__ seg_rows, int num_experts, int n_cols, int k_dim,
                      int b_mn_stride, int b_k_stride, int swiglu_f, GemmWork* __restrict__ list, int* __restrict__ count,
                      int max_items, int tile_m) {
    // tile_m: 128 (one CTA per tile) or 256 (a CTA pair per 256 x 512 tile, see gemm_wide_sm100.cuh; the second half of a
    // segment's last tile may reach past the segment's padded rows, in which case only 128 rows of it are stored)
    __shared__ int s_before, s_all;
    const bool wide = tile_m == 256;
    const int tile_n = (swiglu_f ? 128 : kBlockN) * (wide ? 2 : 1);
    const int width = swiglu_f ? swiglu_f : n_cols;
    const int tiles_n = (width + tile_n - 1) / tile_n;
    const int e = blockIdx.x;
    if (threadIdx.x == 0) s_before = s_all = 0;
    __syncthreads();
    int before = 0, all = 0;
    for (int j = threadIdx.x; j < num_experts; j += blockDim.x) {
        const int n = (seg_rows[j] + tile_m - 1) / tile_m * tiles_n;
        all += n;
        if (j < e) before += n;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        before += __shfl_xor_sync(0xffffffffu, before, o);
        all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_before, before);
        atomicAdd(&s_all, all);
    }
    __syncthreads();
    const int base = s_before;
    if (e == 0 && threadIdx.x == 0) *count = min(s_all, max_items);
    const int rows = seg_rows[e], start = seg_start[e];
    const int tiles_m = (rows + tile_m - 1) / tile_m, n_items = tiles_m * tiles_n;
    const int padded = (rows + kBlockM - 1) / kBlockM * kBlockM;
    for (int i = threadIdx.x; i < n_items && base + i < max_items; i += blockDim.x) {
        // wide tiles go column by column, so that a ragged last column of narrower tiles is spread over the pairs
        const int tm = wide ? i % tiles_m : i / tiles_n, tn = wide ? i / tiles_m : i % tiles_n;
        GemmWork w;
        w.a_mn = start + tm * tile_m;
        w.a_k = 0;
        w.b_k = e * b_k_stride;
        w.k_iters = (k_dim + kBlockK - 1) / kBlockK;
        w.c_row = w.a_mn;
        // whole 128-row blocks are written: the pad rows of a segment are zero on input, so they come out as zeros and later
        // reductions over padded row ranges stay finite
        w.m_valid = min(tile_m, padded - tm * tile_m);
        w.b_mn = e * b_mn_stride + tn * tile_n;
        w.b_mn2 = swiglu_f ? e * b_mn_stride + swiglu_f + tn * tile_n : w.b_mn + (wide ? 256 : 128);
        w.c_col = tn * tile_n;
        w.n_valid = min(tile_n, width - tn * tile_n);
        w.pad0 = !wide ? 0 : (swiglu_f || w.n_valid > 256) ? 2 : 1;
        w.pad1 = 0;
        list[base + i] = w;
    }
}

// Rows grouped along the reduction:  C_e[m, n] = sum_{r in rows of e} A[r, m] * B[r, n]
// (the per-expert weight gradient dW_e = dY_e^T X_e). C is viewed as [E * m_dim, n_dim].
//
// The items of a list are dealt to the `slots` CTAs (or pairs) in turn, and here their lengths differ: an expert's rows are
// the reduction. So the experts are listed longest first and every other round of `slots` items runs backwards, which evens
// out what one CTA gets. (65,536 tokens of the 30B-A3B shapes, loads of 45 to 21,570 rows an
// expert: 4,400 + 1,922 us in expert order on the single-CTA kernel, 2,817 + 1,583 us now; 2,754 + 1,661 us with even loads.) An expert's
// tiles stay together - they share its rows through L2 -, column by column, a ragged last column of narrower tiles at the end.
constexpr int kSortExperts = 1024;

__global__ void __launch_bounds__(256)
plan_grouped_k_kernel(const int* __restrict__ seg_start, const int* __restrict__ seg_rows, int num_experts, int m_dim, int n_dim,
                      GemmWork* __restrict__ list, int* __restrict__ count, int max_items, int tile_m, int slots) {
    __shared__ int s_rows[kSortExperts];
    const bool wide = tile_m == 256;
    const int tile_n = wide ? 2 * kBlockN : kBlockN;
    const int tiles_m = (m_dim + tile_m - 1) / tile_m, tiles_n = (n_dim + tile_n - 1) / tile_n;
    const int per_e = tiles_m * tiles_n;
    const int total = min(per_e * num_experts, max_items);
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = total;
    const bool sorted = num_experts <= kSortExperts;
    if (sorted) {
        for (int e = threadIdx.x; e < num_experts; e += blockDim.x) s_rows[e] = seg_rows[e];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    for (int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); e < num_experts; e += gridDim.x * (blockDim.x >> 5)) {
        const int rows = seg_rows[e], start = seg_start[e];
        int rank = 0;                                  // experts listed before this one
        if (sorted) {
            for (int j = lane; j < num_experts; j += 32) rank += s_rows[j] > rows || (s_rows[j] == rows && j < e);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
        } else {
            rank = e;
        }
        for (int i = lane; i < per_e; i += 32) {
            const int pos = rank * per_e + i;
            if (pos >= total) continue;
            const int round = pos / slots, at = pos - round * slots;
            const int slot = (sorted && (round & 1) && (round + 1) * slots <= total) ? round * slots + slots - 1 - at : pos;
            const int tm = i % tiles_m, tn = i / tiles_m;
            GemmWork w;
            w.a_mn = tm * tile_m;
            w.b_mn = tn * tile_n;
            w.b_mn2 = w.b_mn + tile_n / 2;
            w.a_k = start;
            w.b_k = start;
            w.k_iters = (rows + kBlockK - 1) / kBlockK;
            w.c_row = e * m_dim + tm * tile_m;
            w.c_col = tn * tile_n;
            w.m_valid = min(tile_m, m_dim - tm * tile_m);
            w.n_valid = min(tile_n, n_dim - tn * tile_n);
            w.pad0 = !wide ? 0 : w.n_valid > kBlockN ? 2 : 1;
            w.pad1 = 0;
            list[slot] = w;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// 2-D bf16 tensor [rows, cols] with `ld` elements between rows; box = 64 columns x box_rows.
int make_tmap_bf16(CUtensorMap* m, const void* base, long long rows, long long cols, long long ld,
                   int box_rows) {
    // The encoder is a driver call: make sure this thread has the device's context current
    // (a fresh autograd worker thread may not have made any runtime call yet).
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) return -4;
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -1;
    if ((reinterpret_cast<uintptr_t>(base) & 15u) || (ld % 8) != 0) return -2;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1u, 1u};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        fprintf(stderr, "halo: cuTensorMapEncodeTiled failed (%d): base=%p rows=%lld cols=%lld ld=%lld box_rows=%d\n",
                (int)r, base, rows, cols, ld, box_rows);
        return -3;
    }
    return 0;
}

// Output map of the wide kernel: 32 rows x 128 bytes, rows `ld` elements apart, as many as a launch can name.
static int make_tmap_out(CUtensorMap* m, void* base, long long ld, bool f32) {
    EncodeTiledFn fn = get_encode_fn();
    const int bytes = f32 ? 4 : 2;
    if (!fn || (reinterpret_cast<uintptr_t>(base) & 15u) || (ld * bytes) % 16 || ld <= 0) return -2;
    cuuint64_t dims[2] = {(cuuint64_t)ld, (cuuint64_t)1 << 30};
    cuuint64_t strides[1] = {(cuuint64_t)ld * bytes};
    cuuint32_t box[2] = {128u / bytes, 32u};
    cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = fn(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -3;
}

static int g_num_sms = 0;
static int num_sms() {
    if (!g_num_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_num_sms <= 0) g_num_sms = 148;
    }
    return g_num_sms;
}

constexpr int kGemmSmemBytes = kStages * kStageBytes + 1024 + 4 * kEpiStageBytesPerWarp;

template <bool A_MN, bool B_MN>
static int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int grid,
                       cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(gemm_bf16_kernel<A_MN, B_MN>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kGemmSmemBytes) != cudaSuccess)
            return -10;
        configured = true;
    }
    gemm_bf16_kernel<A_MN, B_MN><<<grid, kGemmThreads, kGemmSmemBytes, stream>>>(ta, tb, p);
    return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

static int dispatch_gemm(int a_mn, int b_mn, const CUtensorMap& ta, const CUtensorMap& tb,
                         const GemmParams& p, int grid, cudaStream_t s) {
    if (!a_mn && !b_mn) return launch_gemm<false, false>(ta, tb, p, grid, s);
    if (!a_mn && b_mn) return launch_gemm<false, true>(ta, tb, p, grid, s);
    if (a_mn && b_mn) return launch_gemm<true, true>(ta, tb, p, grid, s);
    return launch_gemm<true, false>(ta, tb, p, grid, s);
}

// Whether gemm_few_rows_kernel takes a product (both operands K-major, plain store or SwiGLU). Three things set the lines
// (few-row kernel / the better large-tile kernel, us, weights cycled past L2):
//  * It hands out the tokens one after the other when the products are done, which a short reduction does not cover. Up to 16
//    rows it wins all the same, except by a microsecond for outputs of one tile; above that from K = 1024 on, above 64 rows from
//    2048 (4096 columns: 17 rows K = 512 / 1024  7.5 / 8.3 against 7.8 / 11.7; 64 rows 11.4 / 10.1 against 7.9 / 11.6;
//    128 rows K = 512 / 1024 / 2048  17.0 / 12.8 / 14.4 against 8.8 / 12.5 / 18.5).
//  * The tokens' own tiles, which every CTA re-reads from L2, grow with M while the large tiles gain CTAs with N (`tiles_n`), so
//    wide outputs stay there: 12,288 columns are for up to 64 rows and K >= 2048 (K = 1024 / 2048: 1.18 / 1.00 of their time).
//  * Above 128 rows only one CTA fits an SM, which pays where the large tiles leave three quarters of the SMs idle.
static bool few_rows_wins(int M, int N, int K, int tiles_n, bool glu) {
    if (M <= 16) return glu || M <= 8 || K >= 1024 || N > 128;
    if (M <= 64) return K >= 1024 && (tiles_n <= 32 || (tiles_n <= 48 && K >= 2048));
    if (M <= 128) return K >= 2048 && tiles_n <= 32;
    return M <= 256 && !glu && K >= 4096 && (N + 127) / 128 * 4 <= num_sms();
}

static int launch_few_rows(const void* X, const void* W, long long ldx, long long ldw, FewParams p, cudaStream_t stream) {
    p.m_pad = 16;
    while (p.m_pad < p.M) p.m_pad *= 2;
    const int n_tiles = p.swiglu_f ? (p.swiglu_f + 63) / 64 : (p.N + 127) / 128;
    const int kb = (p.K + kBlockK - 1) / kBlockK;
    // cut the reduction while the clusters still fit the SMs at once and a part keeps at least 4 blocks of it
    const int slots = (p.m_pad <= 128 ? 2 : 1) * num_sms(), most = p.m_pad <= 128 ? 8 : 4;
    p.parts = 1;
    while (p.parts < most && n_tiles * p.parts * 2 <= slots && kb >= 8 * p.parts) p.parts *= 2;
    CUtensorMap tw, tx;
    int rc = make_tmap_bf16(&tx, X, p.M, p.K, ldx, p.m_pad);
    if (rc) return rc;
    rc = make_tmap_bf16(&tw, W, p.N, p.K, ldw, p.swiglu_f ? 64 : 128);
    if (rc) return rc * 10;
    p.stages = few_stages(p.m_pad);
    const int smem = few_smem_bytes(p.m_pad);
    // Set for the current device at every launch, and always to what the widest tile needs: the attribute belongs to the function,
    // and another thread's call for another tile may come between this one's attribute and its launch.
    if (cudaFuncSetAttribute(gemm_few_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewMaxSmemBytes) != cudaSuccess) return -10;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_tiles * p.parts), 1, 1);
    cfg.blockDim = dim3(kFewThreads, 1, 1);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.parts;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, gemm_few_rows_kernel, tw, tx, p) == cudaSuccess) return 0;
    cudaGetLastError();                 // reported here, not at a later launch's check
    return -11;
}

template <bool A_MN, bool B_MN>
static int launch_wide_t(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tx,
                         const GemmParams& p, int n_pairs, cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(gemm_wide_kernel<A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmemBytes) != cudaSuccess)
            return -10;
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * n_pairs, 1, 1);
    cfg.blockDim = dim3(kWideThreads, 1, 1);
    cfg.dynamicSmemBytes = kWideSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, gemm_wide_kernel<A_MN, B_MN>, ta, tb, tc, tx, p) == cudaSuccess) return 0;
    cudaGetLastError();                 // reported here, not at a later launch's check
    return -11;
}

static int launch_wide(int a_mn, int b_mn, const CUtensorMap& ta, const CUtensorMap& tb, GemmParams p, int n_pairs, cudaStream_t s) {
    // Only whole 32-row blocks of 128 bytes go through these maps, so their extents need not be the tensors' (a list names rows
    // of a bank whose height is not passed); a base or stride that cannot be encoded leaves the stores to the lanes.
    CUtensorMap tc{}, tx{};
    const bool f32 = p.epi == kEpiStoreF32 || p.epi == kEpiAccumF32;
    if (p.epi != kEpiAccumBf16) p.tma_c = make_tmap_out(&tc, p.C, p.ldc, f32) == 0;
    if (p.epi == kEpiSwiglu && p.aux) p.tma_aux = make_tmap_out(&tx, p.aux, p.ld_aux, false) == 0;
    if (!a_mn && !b_mn) return launch_wide_t<false, false>(ta, tb, tc, tx, p, n_pairs, s);
    if (!a_mn && b_mn) return launch_wide_t<false, true>(ta, tb, tc, tx, p, n_pairs, s);
    if (a_mn && b_mn) return launch_wide_t<true, true>(ta, tb, tc, tx, p, n_pairs, s);
    return launch_wide_t<true, false>(ta, tb, tc, tx, p, n_pairs, s);
}

// Work items of a dense product: whole 256 x 512 tiles for the full waves of pairs; a last wave that would leave more than
// half of the pairs idle is cut into column halves, which take half the time.
static int plan_wide(GemmParams& p, int pairs) {
    const int tiles_m = (p.M + 255) / 256;
    p.tiles_n = p.swiglu_f ? (p.swiglu_f + 255) / 256 : (p.N + 511) / 512;
    const long long tiles = (long long)tiles_m * p.tiles_n;
    const int rest = (int)(tiles % pairs);
    const bool cut = !p.swiglu_f && rest > 0 && 2 * rest <= pairs;
    p.wide_full = (int)(cut ? tiles - rest : tiles);
    p.wide_items = (int)(cut ? tiles + rest : tiles);
    return p.wide_items < pairs ? p.wide_items : pairs;
}

// HALO_GEMM_PAIR: 1 (default) = the CTA-pair kernel (256 x 512 tiles) where its waves are cheaper, 0 = never, 2 = everywhere
static int g_use_pair = -1;
static bool use_pair() {
    if (g_use_pair < 0) {
        const char* e = getenv("HALO_GEMM_PAIR");
        g_use_pair = e ? atoi(e) : 1;
    }
    return g_use_pair != 0;
}

}  // namespace halo

using namespace halo;

extern "C" {

// Dense product. A is [a_rows, a_cols] with leading dimension lda, likewise B.
//   a_mn_major = 0: A is [M, K] (K contiguous);  1: A is [K, M] (M contiguous)
//   b_mn_major = 0: B is [N, K] (K contiguous);  1: B is [K, N] (N contiguous)
// epi selects the epilogue (store / accumulate, bf16 / fp32, SwiGLU). For SwiGLU, B is the
// stacked [2F, K] weight (gate rows then up rows), N must be 2F and C is [M, F].
int halo_gemm_bf16(const void* A, const void* B, void* C, void* aux, int M, int N, int K,
                   long long lda, long long ldb, long long ldc, long long ld_aux, int a_mn_major,
                   int b_mn_major, int epi, float alpha, int* status, void* stream) {
    if (M <= 0 || N <= 0 || K < 0) return 0;
    CUtensorMap ta, tb;
    int rc;
    const bool glu = epi == kEpiSwiglu;
    if (glu && N % 2) return -20;
    use_pair();                       // reads HALO_GEMM_PAIR: 2 sends every product to the pair kernel
    // The large tiles store 16 bytes at a time, the few-row kernel a pair of elements: outputs off the 16-byte boundary go to it as
    // far as it reaches and are refused beyond.
    const uintptr_t outs = reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(aux);
    const bool aligned = (outs & 15u) == 0, pairs_aligned = (outs & (epi == kEpiStoreF32 ? 7u : 3u)) == 0;
    const bool few_ok = K > 0 && !a_mn_major && !b_mn_major && (epi == kEpiStoreBf16 || epi == kEpiStoreF32 || glu);
    if (!aligned && !(few_ok && M <= 256 && pairs_aligned)) return -23;
    if (few_ok && (!aligned || (g_use_pair != 2 && few_rows_wins(M, N, K, glu ? (N / 2 + 127) / 128 : (N + kBlockN - 1) / kBlockN, glu)))) {
        FewParams f{};
        f.C = C; f.aux = aux; f.ldc = ldc; f.ld_aux = ld_aux; f.epi = epi; f.alpha = alpha;
        f.M = M; f.N = N; f.K = K; f.swiglu_f = glu ? N / 2 : 0; f.status = status;
        return launch_few_rows(A, B, lda, ldb, f, (cudaStream_t)stream);
    }
    if (a_mn_major) rc = make_tmap_bf16(&ta, A, K, M, lda, 64);
    else rc = make_tmap_bf16(&ta, A, M, K, lda, 128);
    if (rc) return rc;
    if (b_mn_major) rc = make_tmap_bf16(&tb, B, K, N, ldb, 64);
    else rc = make_tmap_bf16(&tb, B, N, K, ldb, 128);
    if (rc) return rc * 10;
    GemmParams p{};
    p.C = C; p.aux = aux; p.ldc = ldc; p.ld_aux = ld_aux; p.epi = epi; p.alpha = alpha;
    p.M = M; p.N = N; p.K = K;
    p.tiles_m = (M + kBlockM - 1) / kBlockM;
    if (epi_is_glu(epi)) {
        if (N % 2) return -20;
        p.swiglu_f = N / 2;
        p.tiles_n = (p.swiglu_f + 127) / 128;
    } else {
        p.swiglu_f = 0;
        p.tiles_n = (N + kBlockN - 1) / kBlockN;
    }
    p.list = nullptr; p.list_count = nullptr; p.status = status;
    // Which kernel. First the one whose waves of tiles take fewer cycles per 64-wide block of the reduction: a 256 x 512 tile keeps a
    // pair of SMs 1,024 cycles at the rate the wide kernel reaches (0.92 of the tensor pipe, measured), a 128 x 256 tile one SM
    // 512 cycles at 0.78. That says nothing about what surrounds the products; where it decides (wide / single, us):
    //  * One wave of single tiles is latency, and the pair's launch and epilogue are longer: bf16 4096 x 64 x 64  8 / 6, 600 x 2048 x
    //    512  10 / 9. The wide kernel is quicker at fp32 (4096 x 768 x 256  10 / 15) unless half the tile is padding (4096 x 128 x
    //    512  10 / 9).
    //  * SwiGLU without the pre-activations: little is stored, and the single kernel's second accumulator hides it, which pays for
    //    reductions from 512 to 2048 (8192 x 2 x 6144, K = 256 / 512 / 2048 / 4096  86 / 117 / 325 / 595 against 94 / 104 / 295 / 639).
    //  * bf16 +=: the lanes read and write C themselves, and the wide kernel has no second tile to do it under
    //    (16384 x 12288 x 4096  1,746 / 1,312; 4096 x 24576 x 8192  1,168 / 1,354).
    // Over 4,860 shapes timed on both sides (all stores but fp32 +=, which the wide kernel is hardly ever slower at) the chosen kernel is
    // within 0.7 % of the better one on average; by the waves alone 3.3 %.
    const long long single_tiles = (long long)p.tiles_m * p.tiles_n;
    const bool stores = epi == kEpiStoreBf16 || epi == kEpiStoreF32;
    const bool stay = (stores && single_tiles <= num_sms() && (epi == kEpiStoreBf16 || N <= 128)) ||
                      (glu && !aux && K > 256 && K <= 2048) || (epi == kEpiAccumBf16 && K <= 4096);
    if (g_use_pair && K > 0 && epi != kEpiClampedGlu && (g_use_pair == 2 || !stay)) {
        GemmParams wide = p;
        const int pairs = num_sms() / 2, n_pairs = plan_wide(wide, pairs);
        const long long whole = (wide.wide_full + pairs - 1) / pairs, halves = wide.wide_items > wide.wide_full ? 1 : 0;
        const double wide_cost = (1024.0 * whole + 512.0 * halves) / 0.92;
        const double single_cost = 512.0 * ((single_tiles + num_sms() - 1) / num_sms()) / 0.78;
        if (g_use_pair == 2 || wide_cost <= single_cost)
            return launch_wide(a_mn_major, b_mn_major, ta, tb, wide, n_pairs, (cudaStream_t)stream);
    }
    int grid = (int)(single_tiles < num_sms() ? single_tiles : num_sms());
    return dispatch_gemm(a_mn_major, b_mn_major, ta, tb, p, grid, (cudaStream_t)stream);
}

// Row-parallel product fused with the reduce-scatter's transfer: C_partial = A B^T is never stored locally; every
// tile goes into slot `rank` of its owner's staging area (see GemmParams). `stage_ptrs`: HOST array of n_ranks
// device pointers (rank d's [n_ranks][rows_per_rank][N] bf16 staging area as mapped into this process). After the
// kernel and a barrier over the ranks, each rank sums its n_ranks slots.
int halo_gemm_bf16_reduce_scatter(const void* A, const void* B, void* const* stage_ptrs, int n_ranks, int rank,
                                  int M, int N, int K, long long lda, long long ldb, int b_mn_major, int* status,
                                  void* stream) {
    if (n_ranks < 2 || n_ranks > 8 || M % n_ranks) return -21;
    const int rows = M / n_ranks;
    if (rows % kBlockM || N % 8) return -22;
    CUtensorMap ta, tb;
    int rc = make_tmap_bf16(&ta, A, M, K, lda, 128);
    if (rc) return rc;
    if (b_mn_major) rc = make_tmap_bf16(&tb, B, K, N, ldb, 64);
    else rc = make_tmap_bf16(&tb, B, N, K, ldb, 128);
    if (rc) return rc * 10;
    GemmParams p{};
    p.C = nullptr; p.aux = nullptr; p.ldc = N; p.ld_aux = 0; p.epi = kEpiStoreBf16; p.alpha = 1.f;
    p.M = M; p.N = N; p.K = K;
    p.tiles_m = M / kBlockM;
    p.tiles_n = (N + kBlockN - 1) / kBlockN;
    p.swiglu_f = 0;
    p.list = nullptr; p.list_count = nullptr; p.status = status;
    for (int i = 0; i < n_ranks; ++i) p.c_peers[i] = stage_ptrs[i];
    p.rs_ranks = n_ranks; p.rs_rank = rank; p.rs_rows = rows;
    long long tiles = (long long)p.tiles_m * p.tiles_n;
    int grid = (int)(tiles < num_sms() ? tiles : num_sms());
    return dispatch_gemm(0, b_mn_major, ta, tb, p, grid, (cudaStream_t)stream);
}

// Product over a device-resident tile list (see plan_grouped_*). The operands are described as
// plain 2-D tensors; the list carries every coordinate.
int halo_gemm_bf16_list(const void* A, long long a_rows, long long a_cols, long long lda,
                        const void* B, long long b_rows, long long b_cols, long long ldb, void* C,
                        void* aux, long long ldc, long long ld_aux, int a_mn_major, int b_mn_major,
                        int epi, float alpha, int swiglu_f, const void* list, const int* list_count,
                        int* status, void* stream, int pair) {
    CUtensorMap ta, tb;
    int rc = make_tmap_bf16(&ta, A, a_rows, a_cols, lda, a_mn_major ? 64 : 128);
    if (rc) return rc;
    rc = make_tmap_bf16(&tb, B, b_rows, b_cols, ldb, b_mn_major ? 64 : 128);
    if (rc) return rc * 10;
    GemmParams p{};
    p.C = C; p.aux = aux; p.ldc = ldc; p.ld_aux = ld_aux; p.epi = epi; p.alpha = alpha;
    p.swiglu_f = swiglu_f;
    p.list = reinterpret_cast<const GemmWork*>(list);
    p.list_count = list_count;
    p.status = status;
    // `pair`: the list holds 256 x 512 tiles planned for the CTA-pair kernel (see halo_plan_grouped_*)
    if (pair) return launch_wide(a_mn_major, b_mn_major, ta, tb, p, num_sms() / 2, (cudaStream_t)stream);
    return dispatch_gemm(a_mn_major, b_mn_major, ta, tb, p, num_sms(), (cudaStream_t)stream);
}

// As halo_gemm_bf16_list with the clamped-GLU epilogue: `bias` is the expert bias bank [E, 2F] in bf16, read through
// the tile's B coordinates (the list must have been planned with swiglu_f = F and b_mn_stride = 2F, so that a tile's
// gate / up column origins are also its origins in the bias bank).
int halo_gemm_bf16_list_glu(const void* A, long long a_rows, long long a_cols, long long lda,
                            const void* B, long long b_rows, long long b_cols, long long ldb, void* C,
                            void* aux, long long ldc, long long ld_aux, int swiglu_f, const void* bias, float limit,
                            float glu_alpha, const void* list, const int* list_count, int* status, void* stream) {
    if (!bias || swiglu_f <= 0 || swiglu_f % 8) return -1;
    CUtensorMap ta, tb;
    int rc = make_tmap_bf16(&ta, A, a_rows, a_cols, lda, 128);
    if (rc) return rc;
    rc = make_tmap_bf16(&tb, B, b_rows, b_cols, ldb, 128);
    if (rc) return rc * 10;
    GemmParams p{};
    p.C = C; p.aux = aux; p.ldc = ldc; p.ld_aux = ld_aux; p.epi = kEpiClampedGlu; p.alpha = 1.f;
    p.swiglu_f = swiglu_f;
    p.list = reinterpret_cast<const GemmWork*>(list);
    p.list_count = list_count;
    p.status = status;
    p.glu_bias = bias; p.glu_limit = limit; p.glu_alpha = glu_alpha;
    return dispatch_gemm(0, 0, ta, tb, p, num_sms(), (cudaStream_t)stream);
}

int halo_plan_grouped_m(const int* seg_start, const int* seg_rows, int num_experts, int n_cols,
                        int k_dim, int b_mn_stride, int b_k_stride, int swiglu_f, void* list,
                        int* count, int max_items, void* stream, int pair) {
    if (num_experts > 1024) return -1;
    if (num_experts < 1) return cudaMemsetAsync(count, 0, sizeof(int), (cudaStream_t)stream) == cudaSuccess ? 0 : -11;
    plan_grouped_m_kernel<<<num_experts, 256, 0, (cudaStream_t)stream>>>(
        seg_start, seg_rows, num_experts, n_cols, k_dim, b_mn_stride, b_k_stride, swiglu_f,
        reinterpret_cast<GemmWork*>(list), count, max_items, pair ? 256 : kBlockM);
    return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int halo_plan_grouped_k(const int* seg_start, const int* seg_rows, int num_experts, int m_dim,
                        int n_dim, void* list, int* count, int max_items, void* stream, int pair) {
    plan_grouped_k_kernel<<<32, 256, 0, (cudaStream_t)stream>>>(
        seg_start, seg_rows, num_experts, m_dim, n_dim, reinterpret_cast<GemmWork*>(list), count,
        max_items, pair ? 256 : kBlockM, pair ? num_sms() / 2 : num_sms());
    return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int halo_gemm_work_bytes() { return (int)sizeof(GemmWork); }

// 1 unless HALO_GEMM_PAIR=0: callers of the list entry points may plan 256-row tiles for the CTA-pair kernel
int halo_gemm_pair_enabled() { return use_pair() ? g_use_pair : 0; }

}  // extern "C"

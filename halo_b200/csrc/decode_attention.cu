// Decode-step attention against a padded key/value cache: one query token per sequence, all query heads of a
// key/value head handled together so every cached key and value is read from HBM exactly once.
//
//   cache layout  k, v: [batch, max_len, kv_heads, head_dim] bf16 (one layer's slice)
//   q:                  [batch, heads * head_dim] bf16        cols[b]: index of the newest key of sequence b
//   out[b, h, :] = softmax_j<=cols[b](scale * <q[b, h], k[b, j, h / G]>) @ v[b, j, h / G]
//
// What bounds it: the cache is streamed once, nothing is written but the output row, so HBM bandwidth is the floor. Three
// things decide how close a kernel comes. (1) Enough blocks: a (sequence, key/value head) pair is cut over a CLUSTER of
// blocks, each of which takes an equal, 16-key aligned part of that sequence's keys; the parts' softmax states are merged
// through distributed shared memory, so there is no workspace and no second launch. (2) Bytes in flight: every warp runs
// its own cp.async ring of 16-key tiles and never meets a block barrier inside the loop. (3) Arithmetic off the critical
// path: the group's G query heads against 16 keys are a 16 x 16 x head_dim product, done with mma.sync (a memory-bound
// kernel needs 2 % of the tensor rate; tcgen05's 128-row tiles would be mostly padding).
//
// Precision: queries, keys and values are bf16 already, sums and softmax are fp32. The probabilities that meet the values are
// fp32 split into two bf16 terms (p = hi + lo, off by at most 2^-16 p) that go through the same product. With G <= 8 the split is
// free: the product has 16 rows, the heads use rows 0-7 and the low terms ride in rows 8-15.
//
// Measured (B200, 64 sequences of 2,000-8,000 keys, 32 / 4 heads of 128: 655 MB of cache): 3,662 us before (one block of
// four warps per pair, shuffles and scalar products), 109 us now = 6.0 TB/s of cache (0.92 of the measured copy rate).
// Against 64 bits the error of the bf16 output is the former kernel's in seven digits (14 shapes, flat and sharp softmax).
//
// Sequence lengths are read on the device - the host never synchronises on them.
// Stands where the reference's rollout engines run their paged decode kernels; here the cache is the sampler's own
// (halo_b200/inference/generate.py).
#include "sm100_common.cuh"

#include <math.h>

namespace halo {
namespace decode {

constexpr unsigned kMaxGridZ = 65535;
constexpr int kMaxGroup = 16;      // query heads per key/value head
constexpr int kTileKeys = 16;      // keys per warp and step
constexpr int kStages = 3;         // ring depth per warp: 2 blocks of 96 KB per SM keep 128 KB of loads in flight

// 16 bytes of the cache; in four pieces where its rows do not start on 16-byte boundaries (A16 false)
template <bool A16>
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool live) {
    if (A16) {
        const int bytes = live ? 16 : 0;    // 0: the 16 bytes are filled with zeros, nothing is read
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    } else {
        const int bytes = live ? 4 : 0;
#pragma unroll
        for (int i = 0; i < 16; i += 4)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + i),
                         "l"(reinterpret_cast<const uint8_t*>(src) + i), "r"(bytes) : "memory");
    }
}
__device__ __forceinline__ void ldmatrix4(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
// c += a (16 x 16) * b (16 x 8)
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ld_cluster(uint32_t local_addr, uint32_t rank) {
    float v;
    const uint32_t a = map_to_cta(local_addr, rank);
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

template <int D, int WARPS>
__host__ __device__ constexpr int ring_bytes() { return WARPS * kStages * kTileKeys * D * 2 * 2; }
// per-warp partial states, laid over the ring once the loop is over: m, l [kMaxGroup] and acc [kMaxGroup][D] fp32
template <int D>
__host__ __device__ constexpr int state_floats() { return 2 * kMaxGroup + kMaxGroup * D; }

// SPLIT2: groups of more than 8 heads use all 16 rows of the product, so the low terms need a product of their own.
// WARPS: 4, or 1 for caches of few keys (see the entry point).
template <int D, bool SPLIT2, int WARPS, bool A16>
__global__ void __launch_bounds__(WARPS * 32, 8 / WARPS)
decode_attention_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ kc,
                        const __nv_bfloat16* __restrict__ vc, const long long* __restrict__ cols,
                        __nv_bfloat16* __restrict__ out, int n_heads, int n_kv_heads, long long max_len, float scale,
                        int parts, int batch) {
    static_assert(WARPS * state_floats<D>() * 4 <= ring_bytes<D, WARPS>(), "the partial states fit over the ring");
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t base = smem_u32(smem);
    constexpr int kRow = D * 2;                     // bytes of a key
    constexpr int kTile = kTileKeys * kRow;         // bytes of a warp's key (or value) tile
    constexpr int kChunks = D / 8;                  // 16-byte chunks per row
    const int hk = blockIdx.y;
    const long long b = blockIdx.z + (long long)(blockIdx.x / parts) * gridDim.z;       // x holds several only above 65,535 sequences
    if (b >= batch) return;                         // the whole cluster
    const uint32_t part = cluster_cta_rank();
    const int G = n_heads / n_kv_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;          // fragment row and column pair of this lane
    long long n_keys = cols[b] + 1;
    if (n_keys > max_len) n_keys = max_len;         // never read past the cache, whatever the host passed
    if (n_keys < 1) n_keys = 1;
    // this block's keys: an equal share in whole tiles
    const long long tiles = (n_keys + kTileKeys - 1) / kTileKeys;
    const long long share = (tiles + parts - 1) / parts;
    const long long tile_lo = min(tiles, share * part), tile_hi = min(tiles, tile_lo + share);
    const int mine = (int)max(0ll, (tile_hi - tile_lo - warp + WARPS - 1) / WARPS);   // tiles tile_lo + warp + 4 i

    const long long key_stride = (long long)n_kv_heads * D;
    const __nv_bfloat16* kb = kc + b * max_len * key_stride + (long long)hk * D;
    const __nv_bfloat16* vb = vc + b * max_len * key_stride + (long long)hk * D;
    const uint32_t ring = base + warp * (kStages * 2 * kTile);

    auto load_tile = [&](int i) {
        if (i < mine) {
            const long long k0 = (tile_lo + warp + (long long)i * WARPS) * kTileKeys;
            const uint32_t dst = ring + (i % kStages) * 2 * kTile;
#pragma unroll
            for (int c = 0; c < kTileKeys * kChunks / 32; ++c) {
                const int u = c * 32 + lane, r = u / kChunks, ch = u % kChunks;
                const bool live = k0 + r < n_keys;
                const long long off = (live ? k0 + r : 0) * key_stride + ch * 8;
                const uint32_t d = dst + r * kRow + ((ch ^ (r & 7)) << 4);     // chunks swizzled by row
                cp_async16<A16>(d, kb + off, live);
                cp_async16<A16>(d + kTile, vb + off, live);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");                   // empty groups keep the count uniform
    };
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) load_tile(i);

    // query fragments: row g is head g (and g + 8: the head again, so that its low terms find their scores in place)
    uint32_t qa[D / 16][4];
    {
        const __nv_bfloat16* qb = q + (b * n_heads + (long long)hk * G) * D;
        const int r0 = g, r1 = SPLIT2 ? g + 8 : g;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            const int c = ks * 16 + t * 2;
            qa[ks][0] = r0 < G ? *reinterpret_cast<const uint32_t*>(qb + (long long)r0 * D + c) : 0u;
            qa[ks][1] = r1 < G ? *reinterpret_cast<const uint32_t*>(qb + (long long)r1 * D + c) : 0u;
            qa[ks][2] = r0 < G ? *reinterpret_cast<const uint32_t*>(qb + (long long)r0 * D + c + 8) : 0u;
            qa[ks][3] = r1 < G ? *reinterpret_cast<const uint32_t*>(qb + (long long)r1 * D + c + 8) : 0u;
        }
    }
    float o[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;      // rows g and g + 8
    const float c_log2 = scale * 1.4426950408889634f;

    for (int i = 0; i < mine; ++i) {
        load_tile(i + kStages - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
        __syncwarp();
        const uint32_t sk = ring + (i % kStages) * 2 * kTile, sv = sk + kTile;
        const long long k0 = (tile_lo + warp + (long long)i * WARPS) * kTileKeys;
        float s[2][4];                              // scores: keys 0-7 and 8-15 of the tile
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
        {
            // matrices of one ldmatrix: (keys 0-7, d 0-7), (keys 0-7, d 8-15), (keys 8-15, d 0-7), (keys 8-15, d 8-15)
            const int r = (lane & 7) + ((lane >> 4) << 3), hi = (lane >> 3) & 1;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                uint32_t kf[4];
                ldmatrix4(sk + r * kRow + (((2 * ks + hi) ^ (r & 7)) << 4), kf);
                mma16816(s[0], qa[ks], kf[0], kf[1]);
                mma16816(s[1], qa[ks], kf[2], kf[3]);
            }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] *= c_log2;      // base-2 logits
        if (k0 + kTileKeys > n_keys) {
            const int lim = (int)(n_keys - k0);
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n * 8 + t * 2 + (e & 1) >= lim) s[n][e] = -INFINITY;
        }
        float x0 = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
        float x1 = fmaxf(fmaxf(s[0][2], s[0][3]), fmaxf(s[1][2], s[1][3]));
#pragma unroll
        for (int sh = 1; sh < 4; sh <<= 1) {
            x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, sh));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, sh));
        }
        // every tile holds at least one visible key, so the new maxima are finite
        const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
        if (__any_sync(0xffffffffu, n0 > m0 || n1 > m1)) {
            const float a0 = exp2f(m0 - n0), a1 = exp2f(m1 - n1);
            l0 *= a0;
            l1 *= a1;
#pragma unroll
            for (int n = 0; n < D / 8; ++n) {
                o[n][0] *= a0; o[n][1] *= a0;
                o[n][2] *= a1; o[n][3] *= a1;
            }
            m0 = n0;
            m1 = n1;
        }
        float p[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            p[n][0] = exp2f(s[n][0] - m0); p[n][1] = exp2f(s[n][1] - m0);
            p[n][2] = exp2f(s[n][2] - m1); p[n][3] = exp2f(s[n][3] - m1);
        }
        l0 += (p[0][0] + p[0][1]) + (p[1][0] + p[1][1]);
        l1 += (p[0][2] + p[0][3]) + (p[1][2] + p[1][3]);
        // the probabilities as the A operand: hi terms, and what rounding left over as lo terms
        uint32_t pa[4], pl[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
#pragma unroll
            for (int hrow = 0; hrow < 2; ++hrow) {
                const float u = p[n][2 * hrow], v = p[n][2 * hrow + 1];
                // hi: the upper half of the word (truncated, so that lo >= 0); lo is kept above zero so that an infinite
                // value stays infinite instead of meeting a zero
                const uint32_t ub = __float_as_uint(u), vbits = __float_as_uint(v);
                const uint32_t hi = __byte_perm(ub, vbits, 0x7632);
                const uint32_t lo = pack_bf16(fmaxf(u - __uint_as_float(ub & 0xFFFF0000u), 1.17549435e-38f),
                                              fmaxf(v - __uint_as_float(vbits & 0xFFFF0000u), 1.17549435e-38f));
                if (SPLIT2) {
                    pa[2 * n + hrow] = hi;
                    pl[2 * n + hrow] = lo;
                } else {
                    pa[2 * n + hrow] = hrow ? lo : hi;     // rows 8-15 repeat the heads: they carry the low terms
                }
            }
        }
        {
            // value fragments (transposed load): (keys 0-7, d 0-7), (keys 8-15, d 0-7), (keys 0-7, d 8-15), (keys 8-15, d 8-15)
            const int r = (lane & 7) + (((lane >> 3) & 1) << 3), hi = lane >> 4;
#pragma unroll
            for (int n = 0; n < D / 16; ++n) {
                uint32_t vf[4];
                ldmatrix4_trans(sv + r * kRow + (((2 * n + hi) ^ (r & 7)) << 4), vf);
                mma16816(o[2 * n], pa, vf[0], vf[1]);
                mma16816(o[2 * n + 1], pa, vf[2], vf[3]);
                if (SPLIT2) {
                    mma16816(o[2 * n], pl, vf[0], vf[1]);
                    mma16816(o[2 * n + 1], pl, vf[2], vf[3]);
                }
            }
        }
        __syncwarp();                               // every lane is done with the tile before its slot is refilled
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int sh = 1; sh < 4; sh <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, sh);
        l1 += __shfl_xor_sync(0xffffffffu, l1, sh);
    }
    __syncthreads();                                // the ring is dead: partial states take its place
    float* st = reinterpret_cast<float*>(smem);
    {
        float* w = st + warp * state_floats<D>();
        if (t == 0) {
            w[g] = m0;
            w[kMaxGroup + g] = l0;
            if (SPLIT2) {
                w[g + 8] = m1;
                w[kMaxGroup + g + 8] = l1;
            }
        }
#pragma unroll
        for (int n = 0; n < D / 8; ++n) {
            float* row = w + 2 * kMaxGroup + g * D + n * 8 + t * 2;
            if (SPLIT2) {
                *reinterpret_cast<float2*>(row) = make_float2(o[n][0], o[n][1]);
                *reinterpret_cast<float2*>(row + 8 * D) = make_float2(o[n][2], o[n][3]);
            } else {
                *reinterpret_cast<float2*>(row) = make_float2(o[n][0] + o[n][2], o[n][1] + o[n][3]);
            }
        }
    }
    __syncthreads();
    __nv_bfloat16* out_rows = out + (b * n_heads + (long long)hk * G) * D;
    if (parts == 1) {                                   // the block's warps are all there is to merge
        for (int e = 2 * threadIdx.x; e < G * D; e += 2 * WARPS * 32) {
            const int h = e / D;
            float big = -INFINITY;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) big = fmaxf(big, st[w * state_floats<D>() + h]);
            float den = 0.f, na = 0.f, nb = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                const float* sw = st + w * state_floats<D>();
                const float f = sw[h] == -INFINITY ? 0.f : exp2f(sw[h] - big);     // a warp that saw no key: weight 0
                den += sw[kMaxGroup + h] * f;
                na += sw[2 * kMaxGroup + e] * f;
                nb += sw[2 * kMaxGroup + e + 1] * f;
            }
            const float inv = 1.f / den;
            *reinterpret_cast<uint32_t*>(out_rows + e) = pack_bf16(na * inv, nb * inv);
        }
        return;
    }
    // fold the block's warps into warp 0's slot: element (head, d) belongs to one thread, the statistics are read first
    for (int e = threadIdx.x; e < G * D; e += WARPS * 32) {
        const int h = e / D;
        float big = -INFINITY;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) big = fmaxf(big, st[w * state_floats<D>() + h]);
        float num = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float mw = st[w * state_floats<D>() + h];
            const float f = mw == -INFINITY ? 0.f : exp2f(mw - big);   // a warp that saw no key: weight 0
            num += st[w * state_floats<D>() + 2 * kMaxGroup + e] * f;
        }
        st[2 * kMaxGroup + e] = num;
    }
    __syncthreads();
    if ((int)threadIdx.x < G) {
        const int h = threadIdx.x;
        float big = -INFINITY, den = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) big = fmaxf(big, st[w * state_floats<D>() + h]);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float mw = st[w * state_floats<D>() + h];
            den += mw == -INFINITY ? 0.f : st[w * state_floats<D>() + kMaxGroup + h] * exp2f(mw - big);
        }
        st[h] = big;
        st[kMaxGroup + h] = den;
    }
    __syncthreads();
    cluster_sync_all();                                 // every part's state is in its block's shared memory
    for (int e = 2 * (part * (WARPS * 32) + threadIdx.x); e < G * D; e += 2 * parts * (WARPS * 32)) {
        const int h = e / D;
        float big = -INFINITY;
        for (int c = 0; c < parts; ++c) big = fmaxf(big, ld_cluster(base + 4 * h, c));
        float den = 0.f, na = 0.f, nb = 0.f;
        for (int c = 0; c < parts; ++c) {
            const float mc = ld_cluster(base + 4 * h, c);
            const float f = mc == -INFINITY ? 0.f : exp2f(mc - big);
            den += ld_cluster(base + 4 * (kMaxGroup + h), c) * f;
            na += ld_cluster(base + 4 * (2 * kMaxGroup + e), c) * f;
            nb += ld_cluster(base + 4 * (2 * kMaxGroup + e + 1), c) * f;
        }
        const float inv = 1.f / den;
        *reinterpret_cast<uint32_t*>(out_rows + e) = pack_bf16(na * inv, nb * inv);
    }
    cluster_sync_all();                                 // nobody leaves while its state is still being read
}

static int num_sms() {                  // asked once: every GPU of a machine has as many
    static const int n = [] {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) v = 0;
        return v > 0 ? v : 148;
    }();
    return n;
}

template <int D, bool SPLIT2, int WARPS, bool A16>
static int launch(const void* q, const void* kc, const void* vc, const long long* cols, void* out, int batch, int n_heads,
                  int n_kv_heads, long long max_len, float scale, int parts, cudaStream_t s) {
    auto kernel = decode_attention_kernel<D, SPLIT2, WARPS, A16>;
    constexpr int kSmem = ring_bytes<D, WARPS>();
    // set for the current device at every launch: the call costs well under a microsecond and keeps no state here
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return -10;
    cudaLaunchConfig_t cfg = {};
    const unsigned z = batch < kMaxGridZ ? batch : kMaxGridZ;
    cfg.gridDim = dim3(parts * ((batch + z - 1) / z), (unsigned)n_kv_heads, z);
    cfg.blockDim = dim3(WARPS * 32, 1, 1);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)parts;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, (const __nv_bfloat16*)q, (const __nv_bfloat16*)kc,
                                             (const __nv_bfloat16*)vc, cols, (__nv_bfloat16*)out, n_heads, n_kv_heads, max_len,
                                             scale, parts, batch);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return -11;
    }
    return 0;
}

template <int D, bool SPLIT2, typename... Args>
static int launch_form(int warps, bool a16, Args... args) {
    if (!a16) return launch<D, SPLIT2, 4, false>(args...);
    return warps == 1 ? launch<D, SPLIT2, 1, true>(args...) : launch<D, SPLIT2, 4, true>(args...);
}

}  // namespace decode
}  // namespace halo

extern "C" {

// q, out: [batch, n_heads * head_dim] bf16 contiguous. kc, vc: one layer of the cache, [batch, max_len, n_kv_heads,
// head_dim] bf16 contiguous, on 4-byte boundaries. cols: [batch] int64 on the device.
int halo_decode_attention(const void* q, const void* kc, const void* vc, const long long* cols, void* out, int batch,
                          int n_heads, int n_kv_heads, int head_dim, long long max_len, float scale, void* stream) {
    using namespace halo::decode;
    if (batch < 0 || n_kv_heads < 1 || n_heads % n_kv_heads || n_heads / n_kv_heads > kMaxGroup || max_len < 1) return -1;
    if (head_dim != 128 && head_dim != 64) return -1;
    if (batch == 0) return 0;
    if (n_kv_heads > 65535) return -1;
    if ((reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 3u) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    // Parts per (sequence, key/value head) and warps per block. `wave` blocks of four warps run at once, and every further part
    // costs a cluster, its barriers and a merge, whatever the sequences hold (64 sequences of 4 such heads, 1 / 2 / 4 parts, us:
    // 30 keys each 6 / 14 / 25; caches of 1,024, ragged, 20 / 28 / 37; of 4,000 62 / 66 / 66; of 8,000 117 / 120 / 110).
    //  * Caches below 400 keys are not cut.
    //  * Longer ones are cut to fill one wave, and from 3,000 keys on beyond it, for then the longest of a ragged batch decides.
    //  * Eight parts wait for eight free blocks in one GPC at a time and lose, except where even then no SM gets a second block
    //    (2 sequences of 8,000 keys: 4 / 8 parts 23 / 16 us).
    //  * More pairs than one and a half waves over caches of at most 500 keys: one-warp blocks, of which nine fit an SM and which
    //    have no merge at all (1,000 sequences of 4 heads, 4 / 1 warps: 1 key each 47 / 20, 300 keys 110 / 104).
    const int sms = num_sms();
    const long long pairs = (long long)batch * n_kv_heads, wave = 2ll * sms;
    const int most = pairs * 8 <= sms ? 8 : 4;
    int parts = 1;
    if (max_len >= 400)
        while (parts < most && pairs * parts < 2 * wave && max_len > 128ll * parts && (pairs * parts * 2 <= wave || max_len >= 3000)) parts *= 2;
    const int warps = parts == 1 && 2 * pairs > 3 * wave && max_len <= 500 ? 1 : 4;
    const bool split2 = n_heads / n_kv_heads > 8;
    const bool a16 = ((reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15u) == 0;
    if (head_dim == 128)
        return split2 ? launch_form<128, true>(warps, a16, q, kc, vc, cols, out, batch, n_heads, n_kv_heads, max_len, scale, parts, s)
                      : launch_form<128, false>(warps, a16, q, kc, vc, cols, out, batch, n_heads, n_kv_heads, max_len, scale, parts, s);
    return split2 ? launch_form<64, true>(warps, a16, q, kc, vc, cols, out, batch, n_heads, n_kv_heads, max_len, scale, parts, s)
                  : launch_form<64, false>(warps, a16, q, kc, vc, cols, out, batch, n_heads, n_kv_heads, max_len, scale, parts, s);
}

}  // extern "C"

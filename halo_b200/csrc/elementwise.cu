// Memory-bound kernels of the decoder layer: RMSNorm (with the residual add folded in), the
// per-head q/k RMSNorm + rotary embedding of Qwen3 attention, SwiGLU, and the row-wise
// cross-entropy that turns a logits chunk into its gradient in place. All math is fp32 on bf16
// storage with 16-byte accesses; each kernel touches every byte once.
//
// They stand where the reference swaps in Liger's Triton RMSNorm / RoPE / SwiGLU / cross-entropy
// or ATen's rms_norm (halo/model_loading/liger/dispatch.py:416, family_specs.py:34-36) and its
// own GLU kernel (halo/kernels/fused_glu.py:118-205).
#include "sm100_common.cuh"

#include <stdio.h>

#include "halo_noalloc.h"

namespace halo {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float bf16_round(float v) {
    return __bfloat162float(__float2bfloat16_rn(v));
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 t = __bfloat1622float2(h[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                      pack_bf16(f[6], f[7]));
}

// ---------------------------------------------------------------------------------------------
// RMSNorm forward. L threads share a row (L = 32, 128 or 256), each owning VPT 8-element vectors:
// H = 8 * L * VPT. Optional residual: h = x + res (written to h_out), y = norm(h).
//   y = w * bf16(h * rstd)   (the rounding order of the Hugging Face Qwen3 module)
// ---------------------------------------------------------------------------------------------
template <int L>
__device__ __forceinline__ float row_sum(float v, float* scratch /* [256/32] floats */) {
    v = warp_sum(v);
    if (L == 32) return v;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int WPR = L / 32;  // warps per row
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float s = 0.f;
    const int first = (warp / WPR) * WPR;
#pragma unroll
    for (int i = 0; i < WPR; ++i) s += scratch[first + i];
    return s;
}

template <int VPT, int L>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd_out, long long rows,
                   int H, float eps) {
    __shared__ float scratch[8];
    constexpr int RPB = 256 / L;
    const int tl = threadIdx.x % L;
    long long row = (long long)blockIdx.x * RPB + threadIdx.x / L;
    const bool live = row < rows;
    if (!live) row = rows - 1;  // keep every thread in the block-wide reduction
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
    const uint4* rr = res ? reinterpret_cast<const uint4*>(res + row * H) : nullptr;
    float v[VPT][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        unpack8(xr[tl + L * i], v[i]);
        if (rr) {
            float r[8];
            unpack8(rr[tl + L * i], r);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[i][j] = bf16_round(v[i][j] + r[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += v[i][j] * v[i][j];
    }
    ss = row_sum<L>(ss, scratch);
    if (!live) return;
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (tl == 0 && rstd_out) rstd_out[row] = rstd;
    const uint4* wr = reinterpret_cast<const uint4*>(w);
    uint4* yr = reinterpret_cast<uint4*>(y + row * H);
    uint4* hr = h_out ? reinterpret_cast<uint4*>(h_out + row * H) : nullptr;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        if (hr) hr[tl + L * i] = pack8(v[i]);
        float wv[8], o[8];
        unpack8(wr[tl + L * i], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = wv[j] * bf16_round(v[i][j] * rstd);
        yr[tl + L * i] = pack8(o);
    }
}

// RMSNorm backward. dx = rstd * (g*w - xhat * mean(g*w*xhat)) (+ dres); per-block partial dw.
// A fixed grid walks the rows so the partial-sum buffer stays [gridDim.x, H]. Bound by memory (g, h, dres read, dx written):
// rows and weight stay packed in registers and the next row's loads are issued before this row's block-wide sum, so that a
// block always has a row in flight (8,192 rows of 4,096: 95.7 us before, 70 us now; 41 us at the copy rate).
template <int VPT, int L>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ h,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, long long rows, int H) {
    __shared__ float scratch[8];
    constexpr int RPB = 256 / L;
    const int tl = threadIdx.x % L, rg = threadIdx.x / L;
    const uint4* wr = reinterpret_cast<const uint4*>(w);
    uint4 wv[VPT];
    float dwacc[VPT][8];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        wv[i] = wr[tl + L * i];
#pragma unroll
        for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
    }
    const long long step = (long long)gridDim.x * RPB;
    const long long n_iter = (rows + step - 1) / step;
    uint4 gn[VPT], hn[VPT], rn[VPT];
    float rsn = 0.f;
    auto fetch = [&](long long it) {
        long long row = it * step + (long long)blockIdx.x * RPB + rg;
        if (row >= rows) row = rows - 1;                 // keep every thread in the block-wide reduction
        const uint4* gr = reinterpret_cast<const uint4*>(g + row * H);
        const uint4* hr = reinterpret_cast<const uint4*>(h + row * H);
        const uint4* dr = dres ? reinterpret_cast<const uint4*>(dres + row * H) : nullptr;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            gn[i] = gr[tl + L * i];
            hn[i] = hr[tl + L * i];
            if (dr) rn[i] = dr[tl + L * i];
        }
        rsn = rstd[row];
    };
    fetch(0);
    for (long long it = 0; it < n_iter; ++it) {
        const long long row = it * step + (long long)blockIdx.x * RPB + rg;
        const bool live = row < rows;
        uint4 gc[VPT], hc[VPT], rc[VPT];
        const float rs = rsn;
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            gc[i] = gn[i]; hc[i] = hn[i]; rc[i] = rn[i];
        }
        if (it + 1 < n_iter) fetch(it + 1);
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            float gv[8], hv[8], wf[8];
            unpack8(gc[i], gv);
            unpack8(hc[i], hv);
            unpack8(wv[i], wf);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float xh = hv[j] * rs;
                dot += gv[j] * wf[j] * xh;
                if (live) dwacc[i][j] += gv[j] * xh;
            }
        }
        dot = row_sum<L>(dot, scratch) / (float)H;
        if (!live) continue;
        uint4* dxr = reinterpret_cast<uint4*>(dx + row * H);
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            float gv[8], hv[8], wf[8], o[8];
            unpack8(gc[i], gv);
            unpack8(hc[i], hv);
            unpack8(wv[i], wf);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = rs * (gv[j] * wf[j] - hv[j] * rs * dot);
            if (dres) {
                float r[8];
                unpack8(rc[i], r);
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] += r[j];
            }
            dxr[tl + L * i] = pack8(o);
        }
    }
    // fold the RPB row groups of this block, which own the same columns, then write the partial
    __shared__ float red[RPB > 1 ? RPB : 1][L * 8 + 1];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 8; ++j) red[rg][tl * 8 + j] = dwacc[i][j];
        __syncthreads();
        for (int c = threadIdx.x; c < L * 8; c += 256) {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < RPB; ++q) s += red[q][c];
            // column of element (vector tl' + L*i, lane j): (tl' + L*i)*8 + j with c = tl'*8 + j
            dw_partial[(long long)blockIdx.x * H + (long long)i * L * 8 + c] = s;
        }
    }
}

// Column sums of the blocks' partial sums, in a fixed order. A block owns 32 columns and 32 threads share a column: one
// thread per column walked up to 1,184 partials as a chain of dependent loads (54 us for 256 columns, 36 us for 4,096);
// this form takes 4-6 us.
constexpr int kReduceRows = 32;
__global__ void __launch_bounds__(32 * kReduceRows)
reduce_partials_kernel(const float* __restrict__ partial, int n_partials, int H, float* __restrict__ out_f32,
                       __nv_bfloat16* __restrict__ out_bf16, int accumulate) {
    __shared__ float red[kReduceRows][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + tx;
    float s = 0.f;
    if (c < H) {
#pragma unroll 8
        for (int i = ty; i < n_partials; i += kReduceRows) s += partial[(long long)i * H + c];
    }
    red[ty][tx] = s;
    __syncthreads();
    if (ty != 0 || c >= H) return;
    s = 0.f;
#pragma unroll
    for (int i = 0; i < kReduceRows; ++i) s += red[i][tx];
    if (out_f32) out_f32[c] = accumulate ? out_f32[c] + s : s;
    if (out_bf16)
        out_bf16[c] = __float2bfloat16_rn(accumulate ? __bfloat162float(out_bf16[c]) + s : s);
}

// ---------------------------------------------------------------------------------------------
// Rotary table: cos/sin of pos * theta^(-2i/D), i < D/2, rounded to bf16 as the module does.
// ---------------------------------------------------------------------------------------------
__global__ void rope_table_kernel(const int* __restrict__ pos, long long T, int half, float theta,
                                  float2* __restrict__ table) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T * half) return;
    const long long t = i / half;
    const int k = (int)(i % half);
    const float inv = powf(theta, -(float)(2 * k) / (float)(2 * half));
    float s, c;
    sincosf((float)pos[t] * inv, &s, &c);
    table[i] = make_float2(bf16_round(c), bf16_round(s));
}

// q/k RMSNorm over head_dim (=128) + rotate-half RoPE.
//   qkv: [T, (Hq + 2*Hkv) * 128] raw projections;  q_out: [T, Hq*128];  k_out: [T, Hkv*128]
// Bound by memory: every projection is read and written once. Sixteen lanes share a head - lane l owns elements [8 l, 8 l + 8)
// as one 16-byte access, its rotation partner is lane l ^ 8 -, so a warp holds two heads at a time, and it keeps the
// token's 8 cos / sin pairs of its columns in registers over up to kRopePairs pairs of heads, whose loads are issued together.
// (One head per warp with 8-byte accesses and the table re-read for every head measured 585 us forward and 739 us backward
// for 65,536 tokens of 32 + 4 heads, at 0.31 and 0.37 of the copy rate; now 253 and 364 us.)
// A16: every pointer is 16-byte aligned; otherwise rows are read and written in 8-byte halves.
constexpr int kRopePairs = 6;

template <bool A16>
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p) {
    if (A16) return *reinterpret_cast<const uint4*>(p);
    const uint2 a = *reinterpret_cast<const uint2*>(p), b = *reinterpret_cast<const uint2*>(p + 4);
    return make_uint4(a.x, a.y, b.x, b.y);
}
template <bool A16>
__device__ __forceinline__ void store8(__nv_bfloat16* p, const uint4& v) {
    if (A16) {
        *reinterpret_cast<uint4*>(p) = v;
    } else {
        *reinterpret_cast<uint2*>(p) = make_uint2(v.x, v.y);
        *reinterpret_cast<uint2*>(p + 4) = make_uint2(v.z, v.w);
    }
}
template <bool A16>
__device__ __forceinline__ void load_angles(const float2* tab, float (&cs)[8], float (&sn)[8]) {
    if (A16) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 f = reinterpret_cast<const float4*>(tab)[j];
            cs[2 * j] = f.x; sn[2 * j] = f.y; cs[2 * j + 1] = f.z; sn[2 * j + 1] = f.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float2 f = tab[j];
            cs[j] = f.x; sn[j] = f.y;
        }
    }
}
__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ uint4 load_weights8(const __nv_bfloat16* w) {      // no alignment asked of the weight vectors
    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = w[j];
    return *reinterpret_cast<const uint4*>(h);
}
__device__ __forceinline__ float2 unpack2(uint32_t v) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}

// CACHE (sampling): the rotated keys and the values also go to their places in a key/value cache, so that a step needs no
// scatter of its own (two index_put launches a layer before).
struct RopeCache {
    __nv_bfloat16* k;            // one layer's cache, [batch, max_len, Hkv, 128]
    __nv_bfloat16* v;
    const long long* rows;       // [T] sequence and position of every token
    const long long* cols;
    long long batch, max_len;
    int* status;
};

template <bool A16, bool CACHE>
__global__ void __launch_bounds__(256)
qknorm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
                       const __nv_bfloat16* __restrict__ wk, const float2* __restrict__ table,
                       __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ k_out,
                       float* __restrict__ rstd_out, long long T, int Hq, int Hkv, float eps, int use_norm, int splits,
                       const RopeCache cache) {
    const int lane = threadIdx.x & 31, l16 = lane & 15, which = lane >> 4;
    const long long wid = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (wid >= T * splits) return;
    const long long t = wid / splits;
    const int rotated = Hq + Hkv, heads = CACHE ? rotated + Hkv : rotated;
    const int pair0 = (int)(wid % splits) * kRopePairs;
    long long place = -1;        // this token's first cached element
    if (CACHE) {
        long long r = cache.rows[t], c = cache.cols[t];
        if (r < 0) r += cache.batch;                        // counted from the end, as index expressions do
        if (c < 0) c += cache.max_len;
        if (r >= 0 && r < cache.batch && c >= 0 && c < cache.max_len) place = (r * cache.max_len + c) * Hkv * 128 + l16 * 8;
        else if (lane == 0 && cache.status) atomicCAS(cache.status, kStatusOk, kStatusBounds);
    }
    const __nv_bfloat16* src = qkv + t * (long long)(Hq + 2 * Hkv) * 128 + l16 * 8;
    uint4 raw[kRopePairs];
#pragma unroll
    for (int i = 0; i < kRopePairs; ++i) {
        const int hd = 2 * (pair0 + i) + which;
        raw[i] = hd < heads ? load8<A16>(src + (long long)hd * 128) : make_uint4(0, 0, 0, 0);
    }
    float cs[8], sn[8];
    load_angles<A16>(table + t * 64 + (l16 & 7) * 8, cs, sn);
    uint4 wqv = make_uint4(0, 0, 0, 0), wkv = wqv;
    if (use_norm) {
        wqv = load_weights8(wq + l16 * 8);
        wkv = load_weights8(wk + l16 * 8);
    }
#pragma unroll
    for (int i = 0; i < kRopePairs; ++i) {
        if (2 * (pair0 + i) >= heads) break;                // uniform over the warp
        const int hd = 2 * (pair0 + i) + which;
        const bool live = hd < heads, is_q = hd < Hq;
        // the chain of the Hugging Face module, every product and sum rounded to bf16, on packed pairs: what is bf16 already is
        // multiplied by the weight, exchanged with the partner and added two at a time
        uint32_t n[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
        if (use_norm) {
            float v[8], ss = 0.f;
            unpack8(raw[i], v);
#pragma unroll
            for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
            ss = half_warp_sum(ss);
            const float rstd = rsqrtf(ss / 128.f + eps);
            if (l16 == 0 && rstd_out && hd < rotated) rstd_out[t * rotated + hd] = rstd;
            const uint4 w = is_q ? wqv : wkv;
            const uint32_t wp[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) n[j] = mul_bf16x2(wp[j], pack_bf16(v[2 * j] * rstd, v[2 * j + 1] * rstd));
        }
        uint4 out;
        uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // first half: x*cos - partner*sin ; second half: x*cos + partner*sin
            const uint32_t partner = __shfl_xor_sync(0xffffffffu, n[j], 8) ^ (l16 < 8 ? 0x80008000u : 0u);
            const float2 x = unpack2(n[j]), y = unpack2(partner);
            o[j] = add_bf16x2(pack_bf16(x.x * cs[2 * j], x.y * cs[2 * j + 1]), pack_bf16(y.x * sn[2 * j], y.y * sn[2 * j + 1]));
        }
        if (is_q) {
            store8<A16>(q_out + (t * Hq + hd) * 128 + l16 * 8, out);
        } else if (hd < rotated) {
            if (k_out) store8<A16>(k_out + (t * Hkv + (hd - Hq)) * 128 + l16 * 8, out);
            if (CACHE && place >= 0) store8<A16>(cache.k + place + (long long)(hd - Hq) * 128, out);
        } else if (CACHE && live && place >= 0) {
            store8<A16>(cache.v + place + (long long)(hd - rotated) * 128, raw[i]);       // values are stored as they are
        }
    }
}

// Backward: undo the rotation on the incoming gradient, then RMSNorm backward per head; the same mapping of lanes as the
// forward, three pairs of heads in flight, a fixed grid so that the weight gradients end as one partial sum per block.
//   dq: [T, Hq*128], dk: [T, Hkv*128] -> dqkv[:, : (Hq+Hkv)*128]; per-block partial dwq / dwk.
template <bool A16>
__global__ void __launch_bounds__(256, 2)
qknorm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk,
                       const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
                       const __nv_bfloat16* __restrict__ wk, const float2* __restrict__ table,
                       const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dqkv,
                       float* __restrict__ dw_partial, long long T, int Hq, int Hkv, int use_norm, int splits) {
    __shared__ float red[8][2][128];
    constexpr int kFlight = 3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l16 = lane & 15, which = lane >> 4;
    const int heads = Hq + Hkv;
    const long long in_ld = (long long)(Hq + 2 * Hkv) * 128;
    float dwq_acc[8], dwk_acc[8], wqv[8], wkv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) dwq_acc[j] = dwk_acc[j] = 0.f, wqv[j] = wkv[j] = 1.f;
    if (use_norm) {
        unpack8(load_weights8(wq + l16 * 8), wqv);
        unpack8(load_weights8(wk + l16 * 8), wkv);
    }
    const long long total = T * splits;
    for (long long wid = (long long)blockIdx.x * 8 + warp; wid < total; wid += (long long)gridDim.x * 8) {
        const long long t = wid / splits;
        const int pair0 = (int)(wid % splits) * kRopePairs;
        float cs[8], sn[8];
        load_angles<A16>(table + t * 64 + (l16 & 7) * 8, cs, sn);
#pragma unroll 1
        for (int p0 = pair0; p0 < pair0 + kRopePairs && 2 * p0 < heads; p0 += kFlight) {
            uint4 graw[kFlight], xraw[kFlight];
            float rs[kFlight];
#pragma unroll
            for (int i = 0; i < kFlight; ++i) {
                const int hd = 2 * (p0 + i) + which;
                graw[i] = xraw[i] = make_uint4(0, 0, 0, 0);
                rs[i] = 0.f;
                if (hd < heads) {
                    graw[i] = load8<A16>(hd < Hq ? dq + (t * Hq + hd) * 128 + l16 * 8 : dk + (t * Hkv + (hd - Hq)) * 128 + l16 * 8);
                    if (use_norm) {
                        xraw[i] = load8<A16>(qkv + t * in_ld + (long long)hd * 128 + l16 * 8);
                        rs[i] = rstd_in[t * heads + hd];
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < kFlight; ++i) {
                if (2 * (p0 + i) >= heads) break;           // uniform over the warp
                const int hd = 2 * (p0 + i) + which;
                const bool is_q = hd < Hq;
                float gn[8], out[8];
                const uint32_t gp[4] = {graw[i].x, graw[i].y, graw[i].z, graw[i].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    // transpose of the rotation: first half gets +partner*sin, second half -partner*sin
                    const uint32_t partner = __shfl_xor_sync(0xffffffffu, gp[j], 8) ^ (l16 < 8 ? 0u : 0x80008000u);
                    const float2 x = unpack2(gp[j]), y = unpack2(partner);
                    gn[2 * j] = x.x * cs[2 * j] + y.x * sn[2 * j];
                    gn[2 * j + 1] = x.y * cs[2 * j + 1] + y.y * sn[2 * j + 1];
                }
                if (use_norm) {
                    float x[8], gw[8], dot = 0.f;
                    unpack8(xraw[i], x);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        x[j] *= rs[i];
                        gw[j] = gn[j] * (is_q ? wqv[j] : wkv[j]);
                        dot += gw[j] * x[j];
                        const float c = gn[j] * x[j];       // zero for a head past the last one
                        if (is_q) dwq_acc[j] += c;
                        else dwk_acc[j] += c;
                    }
                    dot = half_warp_sum(dot) / 128.f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) out[j] = rs[i] * (gw[j] - x[j] * dot);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) out[j] = gn[j];
                }
                if (hd < heads) store8<A16>(dqkv + t * in_ld + (long long)hd * 128 + l16 * 8, pack8(out));
            }
        }
    }
    if (use_norm && dw_partial) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            // the two half-warps hold the same columns
            dwq_acc[j] += __shfl_xor_sync(0xffffffffu, dwq_acc[j], 16);
            dwk_acc[j] += __shfl_xor_sync(0xffffffffu, dwk_acc[j], 16);
            if (which == 0) {
                red[warp][0][l16 * 8 + j] = dwq_acc[j];
                red[warp][1][l16 * 8 + j] = dwk_acc[j];
            }
        }
        __syncthreads();
        const int row = threadIdx.x >> 7, c = threadIdx.x & 127;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red[w][row][c];
        dw_partial[(long long)blockIdx.x * 256 + row * 128 + c] = s;
    }
}

// ---------------------------------------------------------------------------------------------
// SwiGLU on a packed [rows, 2F] pre-activation (gate | up).
// ---------------------------------------------------------------------------------------------
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ pre, __nv_bfloat16* __restrict__ act,
                                  long long rows, int F) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int vec_per_row = F / 8;
    if (i >= rows * vec_per_row) return;
    const long long r = i / vec_per_row;
    const int c = (int)(i % vec_per_row) * 8;
    float g[8], u[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(pre + r * 2 * F + c), g);
    unpack8(*reinterpret_cast<const uint4*>(pre + r * 2 * F + F + c), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    *reinterpret_cast<uint4*>(act + r * F + c) = pack8(o);
}

__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ pre, const __nv_bfloat16* __restrict__ dact,
                                  __nv_bfloat16* __restrict__ dpre, long long rows, int F) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int vec_per_row = F / 8;
    if (i >= rows * vec_per_row) return;
    const long long r = i / vec_per_row;
    const int c = (int)(i % vec_per_row) * 8;
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(*reinterpret_cast<const uint4*>(pre + r * 2 * F + c), g);
    unpack8(*reinterpret_cast<const uint4*>(pre + r * 2 * F + F + c), u);
    unpack8(*reinterpret_cast<const uint4*>(dact + r * F + c), d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float s = 1.f / (1.f + __expf(-g[j]));
        du[j] = d[j] * g[j] * s;
        dg[j] = d[j] * u[j] * s * (1.f + g[j] * (1.f - s));
    }
    *reinterpret_cast<uint4*>(dpre + r * 2 * F + c) = pack8(dg);
    *reinterpret_cast<uint4*>(dpre + r * 2 * F + F + c) = pack8(du);
}

// ---------------------------------------------------------------------------------------------
// Row statistics of bf16 logits: running maximum, sum of exp(f - max) and, when ENT, sum of exp(f - max) * f.
// A thread takes eight-element vectors, kRowFlight of them at a time so that enough loads are in flight, and rescales its
// sums once per group instead of once per element: the special-function unit then evaluates one exponential per logit,
// which for a 151,936-wide row is just below what reading the row costs.
// ---------------------------------------------------------------------------------------------
constexpr int kRowFlight = 4;

template <bool ENT>
__device__ __forceinline__ void row_stats_add(float& m, float& s, float& ts, const uint4* raw, int n) {
    float lm = m;
#pragma unroll
    for (int i = 0; i < kRowFlight; ++i)
        if (i < n) {
            float f[8];
            unpack8(raw[i], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) lm = fmaxf(lm, f[j]);
        }
    const float sc = __expf(m - lm);                    // exp(-inf) = 0 on the first group
    s *= sc;
    if (ENT) ts *= sc;
    m = lm;
#pragma unroll
    for (int i = 0; i < kRowFlight; ++i)
        if (i < n) {
            float f[8], add = 0.f, tadd = 0.f;
            unpack8(raw[i], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float e = __expf(f[j] - lm);
                add += e;
                if (ENT) tadd += e * f[j];
            }
            s += add;
            if (ENT) ts += tadd;
        }
}

// statistics of one row by the whole block; every thread returns the row's log-sum-exp (and the entropy sum through ts / s).
// V8: the row starts on a 16-byte boundary.
template <bool ENT, int THREADS>
__device__ __forceinline__ void row_stats(const __nv_bfloat16* lr, int V, bool v8, float& m_out, float& s_out, float& ts_out) {
    __shared__ float sm[THREADS / 32], ss[THREADS / 32], st[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nvec = v8 ? V / 8 : 0;
    const uint4* rv = reinterpret_cast<const uint4*>(lr);
    float m = -INFINITY, s = 0.f, ts = 0.f;
    int i = threadIdx.x;
    for (; i + (kRowFlight - 1) * THREADS < nvec; i += kRowFlight * THREADS) {
        uint4 raw[kRowFlight];
#pragma unroll
        for (int k = 0; k < kRowFlight; ++k) raw[k] = rv[i + k * THREADS];
        row_stats_add<ENT>(m, s, ts, raw, kRowFlight);
    }
    if (i < nvec) {
        uint4 raw[kRowFlight];
        int n = 0;
#pragma unroll
        for (int k = 0; k < kRowFlight; ++k)
            if (i + k * THREADS < nvec) {
                raw[k] = rv[i + k * THREADS];
                n = k + 1;
            }
        row_stats_add<ENT>(m, s, ts, raw, n);
    }
    for (int c = nvec * 8 + threadIdx.x; c < V; c += THREADS) {
        const float f = __bfloat162float(lr[c]);
        const float nm = fmaxf(m, f);
        const float sc = __expf(m - nm), e = __expf(f - nm);
        s = s * sc + e;
        if (ENT) ts = ts * sc + e * f;
        m = nm;
    }
    const float wm = warp_max(m);
    const float sc = (m == -INFINITY) ? 0.f : __expf(m - wm);   // a thread (or a whole warp) may own no column
    s = warp_sum(m == -INFINITY ? 0.f : s * sc);
    if (ENT) ts = warp_sum(m == -INFINITY ? 0.f : ts * sc);
    if (lane == 0) { sm[warp] = wm; ss[warp] = s; if (ENT) st[warp] = ts; }
    __syncthreads();
    // every warp folds the warps' results for itself: the same values in the same order everywhere
    float mm = lane < THREADS / 32 ? sm[lane] : -INFINITY;
    float sv = lane < THREADS / 32 ? ss[lane] : 0.f;
    float tv = (ENT && lane < THREADS / 32) ? st[lane] : 0.f;
    const float gm = warp_max(mm);
    const float c2 = (mm == -INFINITY) ? 0.f : __expf(mm - gm);
    s_out = warp_sum(mm == -INFINITY ? 0.f : sv * c2);
    if (ENT) ts_out = warp_sum(mm == -INFINITY ? 0.f : tv * c2);
    m_out = gm;
}

// ---------------------------------------------------------------------------------------------
// Cross-entropy over one logits chunk [rows, V] (bf16), in place: on return the chunk holds
// grad_scale * row_scale[row] * (softmax - onehot) and loss_rows / lse carry the forward results.
// One block per row. Rows whose label is ignore_index get a zero gradient.
// The row is read, read again - out of the L2 cache where it still holds it - and written; the two exponentials per logit
// take 0.28 ms of the special-function units for 4,096 rows of 151,936. That much: 712 us with 512 threads, four blocks an
// SM and one load in flight per thread, 577 us now. (1,024 threads: 649 us with one block an SM, 686 us with two.)
// ---------------------------------------------------------------------------------------------
constexpr int kCeThreads = 512;
__global__ void __launch_bounds__(kCeThreads, 3)
cross_entropy_inplace_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
                             const float* __restrict__ grad_scale, const float* __restrict__ row_scale,
                             float* __restrict__ loss_rows,
                             float* __restrict__ lse_out, long long ld, int V, long long ignore_index) {
    const long long row = blockIdx.x;
    __nv_bfloat16* lr = logits + row * ld;
    const long long label = labels[row];
    const int nvec = V / 8;
    float m, sum, unused;
    row_stats<false, kCeThreads>(lr, V, true, m, sum, unused);
    const float lse = m + logf(sum);
    const bool ignored = (label == ignore_index);
    if (threadIdx.x == 0) {
        if (lse_out) lse_out[row] = lse;
        loss_rows[row] = ignored ? 0.f : lse - __bfloat162float(lr[label]);
    }
    __syncthreads();  // the label logit is read before it is overwritten
    const float gs = ignored ? 0.f : (grad_scale ? *grad_scale : 1.f) * (row_scale ? row_scale[row] : 1.f);
    uint4* rv = reinterpret_cast<uint4*>(lr);
    const int label_vec = label >= 0 && label < V ? (int)(label >> 3) : -1, label_pos = (int)(label & 7);
    auto finish = [&](uint4 raw, int i) {
        float f[8];
        unpack8(raw, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __expf(f[j] - lse) * gs;
        if (i == label_vec) {                           // one vector of the row
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float x[8];
                unpack8(raw, x);
                if (j == label_pos) f[j] = (__expf(x[j] - lse) - 1.f) * gs;
            }
        }
        rv[i] = pack8(f);
    };
    int i = threadIdx.x;
    for (; i + (kRowFlight - 1) * kCeThreads < nvec; i += kRowFlight * kCeThreads) {
        uint4 raw[kRowFlight];
#pragma unroll
        for (int k = 0; k < kRowFlight; ++k) raw[k] = rv[i + k * kCeThreads];
#pragma unroll
        for (int k = 0; k < kRowFlight; ++k) finish(raw[k], i + k * kCeThreads);
    }
    for (; i < nvec; i += kCeThreads) finish(rv[i], i);
    for (int c = nvec * 8 + threadIdx.x; c < V; c += kCeThreads) {
        float p = __expf(__bfloat162float(lr[c]) - lse);
        if ((long long)c == label) p -= 1.f;
        lr[c] = __float2bfloat16_rn(p * gs);
    }
}

// Token log-probabilities and entropy from a logits chunk, no gradient (scoring passes of RL). One block per row, the row
// read once: 2,047 rows of 151,936 took 637 us with two-byte loads and two exponentials per logit, 145 us now (95 us is
// the time of the read).
constexpr int kLogpThreads = 512;
__global__ void __launch_bounds__(kLogpThreads)
logprob_entropy_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
                       float* __restrict__ logp, float* __restrict__ entropy, long long ld, int V,
                       long long ignore_index, int v8) {
    const long long row = blockIdx.x;
    const __nv_bfloat16* lr = logits + row * ld;
    float m, s, ts = 0.f;
    if (entropy) row_stats<true, kLogpThreads>(lr, V, v8 != 0, m, s, ts);
    else row_stats<false, kLogpThreads>(lr, V, v8 != 0, m, s, ts);
    if (threadIdx.x == 0) {
        const float lse = m + logf(s);
        const long long label = labels[row];
        logp[row] = (label == ignore_index) ? 0.f : __bfloat162float(lr[label]) - lse;
        if (entropy) entropy[row] = lse - ts / s;
    }
}

// out[i] = bf16(bf16(x[i]) * bf16(*g)) - gradients that were computed with the forward, times the upstream scalar, in the
// rounding of a bf16 product; without g the fp32 sums are rounded. One pass at the copy rate: 287 us for the sums of a
// 151,936 x 2,048 head and 190 us for their bf16 values, where a conversion and a broadcast product of tensor operations
// took 845 + 200 us.
template <typename T>
__global__ void __launch_bounds__(256)
scale_to_bf16_kernel(const T* __restrict__ x, const float* __restrict__ g, __nv_bfloat16* __restrict__ out, long long n) {
    const float s = g ? bf16_round(*g) : 1.f;
    const long long nvec = n / 8;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
        float f[8];
        if constexpr (sizeof(T) == 4) {
            const float4 a = reinterpret_cast<const float4*>(x)[2 * i], b = reinterpret_cast<const float4*>(x)[2 * i + 1];
            f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
        } else {
            unpack8(reinterpret_cast<const uint4*>(x)[i], f);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = bf16_round(f[j]) * s;
        reinterpret_cast<uint4*>(out)[i] = pack8(f);
    }
    if (blockIdx.x == 0 && threadIdx.x < n - nvec * 8) {
        const long long c = nvec * 8 + threadIdx.x;
        out[c] = __float2bfloat16_rn(bf16_round((float)x[c]) * s);
    }
}

}  // namespace halo

using namespace halo;

extern "C" {

#define HALO_LAUNCH_CHECK() (cudaGetLastError() == cudaSuccess ? 0 : -11)

// Pick the threads-per-row L (32, 128, 256) and vectors-per-thread so that H = 8 * L * VPT, VPT <= 4.
static bool rms_shape(int H, int* L, int* vpt) {
    const int cands[3] = {32, 128, 256};
    for (int i = 0; i < 3; ++i) {
        const int l = cands[i];
        if (H % (8 * l) == 0 && H / (8 * l) <= 4) {
            *L = l;
            *vpt = H / (8 * l);
            return true;
        }
    }
    return false;
}

// The backward keeps a row, the next row and the weight gradient in registers: two vectors per thread fit twice on an SM
// (128 registers), three or four only once, so it takes the narrowest L that gets by with two, else the widest that fits.
static bool rms_bwd_shape(int H, int* L, int* vpt) {
    const int cands[3] = {32, 128, 256};
    bool found = false;
    for (int i = 0; i < 3; ++i) {
        const int l = cands[i];
        if (H % (8 * l) == 0 && H / (8 * l) <= 4) {
            *L = l;
            *vpt = H / (8 * l);
            found = true;
            if (*vpt <= 2) return true;
        }
    }
    return found;
}

#define RMS_DISPATCH(KERNEL, ...)                                                                \
    if (L == 32) {                                                                               \
        switch (vpt) {                                                                           \
            case 1: KERNEL<1, 32><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                      \
            case 2: KERNEL<2, 32><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                      \
            case 3: KERNEL<3, 32><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                      \
            default: KERNEL<4, 32><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                     \
        }                                                                                        \
    } else if (L == 128) {                                                                       \
        switch (vpt) {                                                                           \
            case 1: KERNEL<1, 128><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                     \
            case 2: KERNEL<2, 128><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                     \
            case 3: KERNEL<3, 128><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                     \
            default: KERNEL<4, 128><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                    \
        }                                                                                        \
    } else {                                                                                     \
        switch (vpt) {                                                                           \
            case 1: KERNEL<1, 256><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                     \
            case 2: KERNEL<2, 256><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                     \
            case 3: KERNEL<3, 256><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                     \
            default: KERNEL<4, 256><<<grid, 256, 0, s>>>(__VA_ARGS__); break;                    \
        }                                                                                        \
    }

int halo_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out,
                     float* rstd, long long rows, int H, float eps, void* stream) {
    int L, vpt;
    if (!rms_shape(H, &L, &vpt)) return -1;
    if (rows == 0) return 0;
    const int rpb = 256 / L;
    dim3 grid((unsigned)((rows + rpb - 1) / rpb));
    cudaStream_t s = (cudaStream_t)stream;
    RMS_DISPATCH(rmsnorm_fwd_kernel, (const __nv_bfloat16*)x, (const __nv_bfloat16*)res,
                 (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (__nv_bfloat16*)h_out, rstd, rows, H, eps)
    return HALO_LAUNCH_CHECK();
}

int halo_rmsnorm_supported(int H) {
    int L, vpt;
    return rms_shape(H, &L, &vpt) ? 1 : 0;
}

int halo_rmsnorm_bwd_blocks(long long rows, int H) {
    int L = 32, vpt = 1;
    rms_bwd_shape(H, &L, &vpt);
    const int rpb = 256 / L;
    long long b = (rows + rpb - 1) / rpb;
    static_assert(HALO_NOALLOC_MAX_BLOCKS >= 592, "the built-in scratch must cover the largest grid");
    return (int)(b < 592 ? b : 592);
}

// dw_partial: fp32 scratch of halo_rmsnorm_bwd_blocks(rows, H) * H elements.
int halo_rmsnorm_bwd(const void* g, const void* h, const void* w, const float* rstd,
                     const void* dres, void* dx, float* dw_partial, float* dw_f32, void* dw_bf16,
                     int accumulate, long long rows, int H, void* stream) {
    int L, vpt;
    if (!rms_bwd_shape(H, &L, &vpt)) return -1;
    if (rows == 0) return 0;
    const int blocks = halo_rmsnorm_bwd_blocks(rows, H);
    dim3 grid(blocks);
    cudaStream_t s = (cudaStream_t)stream;
    RMS_DISPATCH(rmsnorm_bwd_kernel, (const __nv_bfloat16*)g, (const __nv_bfloat16*)h,
                 (const __nv_bfloat16*)w, rstd, (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx,
                 dw_partial, rows, H)
    reduce_partials_kernel<<<(H + 31) / 32, 32 * kReduceRows, 0, s>>>(dw_partial, blocks, H, dw_f32,
                                                          (__nv_bfloat16*)dw_bf16, accumulate);
    return HALO_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------------------------
// Allocation-free RMSNorm backward (see halo_noalloc.h). The per-block partial sums live in a
// file-scope device array instead of a caller-provided buffer.
// ---------------------------------------------------------------------------------------------
}  // extern "C"

static __device__ __align__(256) float g_noalloc_scratch[HALO_NOALLOC_MAX_BLOCKS * HALO_NOALLOC_MAX_HIDDEN];

// In host code `g_noalloc_scratch` is only a handle for the runtime, not a device address: the
// address a kernel can use comes from cudaGetSymbolAddress, once per device.
static float* noalloc_scratch_for_current_device() {
    constexpr int kMaxDevices = 64;
    static float* cached[kMaxDevices] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    if (cached[dev] == nullptr) {
        float* ptr = nullptr;
        if (cudaGetSymbolAddress((void**)&ptr, g_noalloc_scratch) != cudaSuccess) return nullptr;
        cached[dev] = ptr;
    }
    return cached[dev];
}

extern "C" {

int halo_rmsnorm_bwd_noalloc(const void* g, const void* h, const void* w, const float* rstd,
                             const void* dres, void* dx, float* dw_f32, void* dw_bf16,
                             int accumulate, long long rows, int H, void* stream) {
    int L, vpt;
    if (!rms_shape(H, &L, &vpt)) return -1;
    if (H > HALO_NOALLOC_MAX_HIDDEN) {
        fprintf(stderr, "halo_rmsnorm_bwd_noalloc: hidden size %d exceeds the built-in scratch (max %d); "
                        "use halo_rmsnorm_bwd with a caller-provided buffer\n", H, HALO_NOALLOC_MAX_HIDDEN);
        return -3;
    }
    if (rows == 0) return 0;
    float* scratch = noalloc_scratch_for_current_device();
    if (scratch == nullptr) return -4;
    // halo_rmsnorm_bwd never launches more than HALO_NOALLOC_MAX_BLOCKS blocks and each block
    // writes H floats, so blocks * H <= the array's size
    return halo_rmsnorm_bwd(g, h, w, rstd, dres, dx, scratch, dw_f32, dw_bf16, accumulate, rows, H, stream);
}

int halo_rope_table(const int* pos, long long T, int head_dim, float theta, void* table,
                    void* stream) {
    const int half = head_dim / 2;
    const long long n = T * half;
    rope_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        pos, T, half, theta, (float2*)table);
    return HALO_LAUNCH_CHECK();
}

static int rope_splits(int heads) { return ((heads + 1) / 2 + kRopePairs - 1) / kRopePairs; }

int halo_qknorm_rope_fwd(const void* qkv, const void* wq, const void* wk, const void* table,
                         void* q_out, void* k_out, float* rstd, long long T, int Hq, int Hkv,
                         int head_dim, float eps, int use_norm, void* stream) {
    if (head_dim != 128) return -1;
    const int splits = rope_splits(Hq + Hkv);
    const unsigned grid = (unsigned)((T * splits + 7) / 8);
    const bool a16 = (((uintptr_t)qkv | (uintptr_t)q_out | (uintptr_t)k_out | (uintptr_t)table) & 15u) == 0;
    auto kernel = a16 ? qknorm_rope_fwd_kernel<true, false> : qknorm_rope_fwd_kernel<false, false>;
    kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk,
        (const float2*)table, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out, rstd, T, Hq, Hkv, eps,
        use_norm, splits, RopeCache{});
    return HALO_LAUNCH_CHECK();
}

// As halo_qknorm_rope_fwd without the statistics, for sampling: the rotated keys and the values go to places (rows[t], cols[t])
// of one layer's cache [batch, max_len, Hkv, 128]; k_out may be null. A place outside the cache is skipped and recorded.
int halo_qknorm_rope_cache(const void* qkv, const void* wq, const void* wk, const void* table, void* q_out, void* k_out,
                           void* k_cache, void* v_cache, const long long* rows, const long long* cols, long long batch,
                           long long max_len, long long T, int Hq, int Hkv, int head_dim, float eps, int use_norm, int* status,
                           void* stream) {
    if (head_dim != 128) return -1;
    const int splits = rope_splits(Hq + 2 * Hkv);
    const unsigned grid = (unsigned)((T * splits + 7) / 8);
    const bool a16 = (((uintptr_t)qkv | (uintptr_t)q_out | (uintptr_t)k_out | (uintptr_t)table | (uintptr_t)k_cache |
                       (uintptr_t)v_cache) & 15u) == 0;
    auto kernel = a16 ? qknorm_rope_fwd_kernel<true, true> : qknorm_rope_fwd_kernel<false, true>;
    const RopeCache cache{(__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, rows, cols, batch, max_len, status};
    kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, (const float2*)table,
        (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out, nullptr, T, Hq, Hkv, eps, use_norm, splits, cache);
    return HALO_LAUNCH_CHECK();
}

int halo_qknorm_rope_bwd_blocks(long long T, int heads) {
    long long b = (T * rope_splits(heads) + 7) / 8;
    return (int)(b < 592 ? b : 592);
}

// dw_partial: fp32 scratch of halo_qknorm_rope_bwd_blocks(...) * 256; dwq/dwk: fp32 [128] outputs.
int halo_qknorm_rope_bwd(const void* dq, const void* dk, const void* qkv, const void* wq,
                         const void* wk, const void* table, const float* rstd, void* dqkv,
                         float* dw_partial, float* dwq, float* dwk, int accumulate, long long T,
                         int Hq, int Hkv, int head_dim, int use_norm, void* stream) {
    if (head_dim != 128) return -1;
    const int blocks = halo_qknorm_rope_bwd_blocks(T, Hq + Hkv);
    cudaStream_t s = (cudaStream_t)stream;
    const bool a16 = (((uintptr_t)dq | (uintptr_t)dk | (uintptr_t)qkv | (uintptr_t)dqkv | (uintptr_t)table) & 15u) == 0;
    auto kernel = a16 ? qknorm_rope_bwd_kernel<true> : qknorm_rope_bwd_kernel<false>;
    kernel<<<blocks, 256, 0, s>>>(
        (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)qkv,
        (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, (const float2*)table, rstd,
        (__nv_bfloat16*)dqkv, dw_partial, T, Hq, Hkv, use_norm, rope_splits(Hq + Hkv));
    if (use_norm) {
        // partial layout per block: [dwq(128) | dwk(128)]
        reduce_partials_kernel<<<256 / 32, 32 * kReduceRows, 0, s>>>(dw_partial, blocks, 256, dwq, nullptr, accumulate);
        (void)dwk;  // dwq points at a [256] buffer: first 128 = q weight grad, last 128 = k weight grad
    }
    return HALO_LAUNCH_CHECK();
}

int halo_swiglu_fwd(const void* pre, void* act, long long rows, int F, void* stream) {
    if (F % 8) return -1;
    const long long n = rows * (F / 8);
    swiglu_fwd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)pre, (__nv_bfloat16*)act, rows, F);
    return HALO_LAUNCH_CHECK();
}

int halo_swiglu_bwd(const void* pre, const void* dact, void* dpre, long long rows, int F,
                    void* stream) {
    if (F % 8) return -1;
    const long long n = rows * (F / 8);
    swiglu_bwd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)pre, (const __nv_bfloat16*)dact, (__nv_bfloat16*)dpre, rows, F);
    return HALO_LAUNCH_CHECK();
}

int halo_cross_entropy_inplace(void* logits, const long long* labels, const float* grad_scale,
                               const float* row_scale, float* loss_rows, float* lse, long long rows, long long ld, int V,
                               long long ignore_index, void* stream) {
    if (rows == 0) return 0;
    if (ld % 8) return -1;
    cross_entropy_inplace_kernel<<<(unsigned)rows, kCeThreads, 0, (cudaStream_t)stream>>>(
        (__nv_bfloat16*)logits, labels, grad_scale, row_scale, loss_rows, lse, ld, V, ignore_index);
    return HALO_LAUNCH_CHECK();
}

int halo_logprob_entropy(const void* logits, const long long* labels, float* logp, float* entropy,
                         long long rows, long long ld, int V, long long ignore_index, void* stream) {
    if (rows == 0) return 0;
    const int v8 = ((uintptr_t)logits & 15u) == 0 && ld % 8 == 0;      // rows on 16-byte boundaries take vector loads
    logprob_entropy_kernel<<<(unsigned)rows, kLogpThreads, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)logits, labels, logp, entropy, ld, V, ignore_index, v8);
    return HALO_LAUNCH_CHECK();
}

// x: n contiguous fp32 (or bf16) values, g: one fp32 value or null, both on the device; x and out 16-byte aligned.
int halo_scale_to_bf16(const void* x, int x_is_f32, const float* g, void* out, long long n, void* stream) {
    if (((uintptr_t)x | (uintptr_t)out) & 15u) return -1;
    if (n <= 0) return 0;
    const long long blocks = (n / 8 + 255) / 256;
    const unsigned grid = (unsigned)(blocks < 1 ? 1 : blocks < 148 * 16 ? blocks : 148 * 16);
    if (x_is_f32)
        scale_to_bf16_kernel<float><<<grid, 256, 0, (cudaStream_t)stream>>>((const float*)x, g, (__nv_bfloat16*)out, n);
    else
        scale_to_bf16_kernel<__nv_bfloat16><<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, g, (__nv_bfloat16*)out, n);
    return HALO_LAUNCH_CHECK();
}

}  // extern "C"

// Fused decode attention over the packed KIVI cache: CUDA-core fp32 kernel.
//
//   out = softmax(q K^T * D^-0.5) V   over [quantized history || residual ring]
// (formula: tests/integration/test_attention_fix.py:40-43; the operand is what
// cache/manager.py:263-286 would serve, but nothing is ever dequantized to
// memory).  Every number is fp32: codes are unpacked in registers, turned into
// k = code*scale + zero, and fed to fp32 FMAs, so this kernel holds the 1e-5
// tolerance of fp32 activations and covers every supported shape.  The
// tensor-core kernel in attn_mma.cu is the fast path for the Llama shape.
//
// Work split: grid = (splits, units).  The quantized history of a unit is cut
// into `nq_splits` runs of whole token groups; the residual ring is one more
// split.  Inside a CTA each warp walks its own groups with a private running
// (max, sum, output); warps are merged through shared memory and the CTA writes
// one partial (max, sum, unnormalised output) per query head to the workspace.
// merge_splits_kernel folds the partials (the only scratch memory of the op).
//
// Per 32-token chunk a warp does: lane = token for the q.k scores (each lane
// walks the D channels of its token), a warp max, exp2, then lane = 4 channels
// for p.V (each lane walks the chunk's tokens).
#include "async_copy.cuh"
#include "cluster_fold.cuh"
#include "kivi_common.cuh"

#include <atomic>

namespace kivi {


namespace {

constexpr int kWarps = 4;

template <int NREP, int DB>
__global__ void __launch_bounds__(kWarps * 32)
attn_fp32_kernel(kivi_layer L, int64_t quant_len, int res_start, int res_len,
                 const void* q, int q_dtype, float scale_log2,
                 int nq_splits, int groups_per_split, int n_splits,
                 float* __restrict__ part_o, float* __restrict__ part_ml) {
    stream_order();
    q = settled(q);
    settle_layer(L);
    const int D = L.head_dim, G = L.group_size, Q = G / 4, W = D < 64 ? D : 64, ng = D / G;
    const int u = blockIdx.y, split = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t max_groups = L.max_tokens / G;

    extern __shared__ __align__(16) float smem[];
    float* q_s = smem;                                   // [NREP][D]
    float* sz_s = q_s + NREP * D + warp * 2 * D;         // per warp: scales[D], zeros[D]
    float* p_s = q_s + NREP * D + kWarps * 2 * D + warp * 32 * NREP;   // per warp [32][NREP]
    float* red_s = q_s + NREP * D + kWarps * 2 * D + kWarps * 32 * NREP;  // [kWarps][NREP][2] + [NREP][DB*128]

    for (int i = threadIdx.x; i < NREP * D; i += blockDim.x)
        q_s[i] = load_as_float(q, q_dtype, (int64_t)u * NREP * D + i);
    __syncthreads();

    float m[NREP], l[NREP], o[NREP][DB][4];
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        m[h] = -INFINITY; l[h] = 0.0f;
#pragma unroll
        for (int b = 0; b < DB; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) o[h][b][i] = 0.0f;
    }

    // softmax update for one chunk of <= 32 tokens whose raw scores sit in acc[]
    auto absorb_scores = [&](float (&acc)[NREP], bool valid) {
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            float s = valid ? acc[h] * scale_log2 : -INFINITY;
            float mx = s;
#pragma unroll
            for (int o_ = 16; o_ > 0; o_ >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o_));
            const float m_new = fmaxf(m[h], mx);            // finite: every chunk has >= 1 token
            const float alpha = exp2f(m[h] - m_new);        // exp2(-inf) = 0 on the first chunk
            const float p = valid ? exp2f(s - m_new) : 0.0f;
            m[h] = m_new;
            l[h] = l[h] * alpha + p;
#pragma unroll
            for (int b = 0; b < DB; ++b)
#pragma unroll
                for (int i = 0; i < 4; ++i) o[h][b][i] *= alpha;
            p_s[lane * NREP + h] = p;
        }
        __syncwarp();
    };

    if (split < nq_splits) {
        const int64_t n_groups = quant_len / G;
        const int64_t g_begin = (int64_t)split * groups_per_split;
        int64_t g_end = g_begin + groups_per_split;
        if (g_end > n_groups) g_end = n_groups;
        for (int64_t g = g_begin + warp; g < g_end; g += kWarps) {
            const int64_t gb = (int64_t)u * max_groups + g;
            const uint8_t* kb = L.k_codes + gb * (D * Q);
            __syncwarp();
            for (int d = lane; d < D; d += 32) {
                sz_s[d] = __ldg(L.k_scales + gb * D + d);
                sz_s[D + d] = __ldg(L.k_zeros + gb * D + d);
            }
            __syncwarp();
            for (int c0 = 0; c0 < G; c0 += 32) {
                const int tt = c0 + lane;
                const bool valid = tt < G;
                float acc[NREP];
#pragma unroll
                for (int h = 0; h < NREP; ++h) acc[h] = 0.0f;
                if (valid) {
                    const int j = tt / 4, e = tt % 4;
                    for (int d0 = 0; d0 < D; d0 += 4) {
                        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(kb + kblock_offset(d0, j, Q, W)));
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float code = (float)((w >> (8 * i + 2 * e)) & 3u);
                            const float k = fmaf(code, sz_s[d0 + i], sz_s[D + d0 + i]);
#pragma unroll
                            for (int h = 0; h < NREP; ++h) acc[h] = fmaf(q_s[h * D + d0 + i], k, acc[h]);
                        }
                    }
                }
                absorb_scores(acc, valid);
                const int ntok = G - c0 < 32 ? G - c0 : 32;
                const int64_t t0 = g * G + c0;
                const uint8_t* vcu = L.v_codes + (int64_t)u * L.max_tokens * (D / 4);
                const float* vsu = L.v_scales + (int64_t)u * L.max_tokens * ng;
                const float* vzu = L.v_zeros + (int64_t)u * L.max_tokens * ng;
                for (int tk = 0; tk < ntok; ++tk) {
                    float p[NREP];
#pragma unroll
                    for (int h = 0; h < NREP; ++h) p[h] = p_s[tk * NREP + h];
#pragma unroll
                    for (int b = 0; b < DB; ++b) {
                        const int byte = lane + 32 * b;
                        if (byte < D / 4) {
                            const uint32_t vb = __ldg(vcu + vcode_offset(t0 + tk, byte, D, G));
                            const int gd = (4 * byte) / G;
                            const int64_t mi = vmeta_index(t0 + tk, gd, D, G);
                            const float s = __ldg(vsu + mi);
                            const float z = __ldg(vzu + mi);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float v = fmaf((float)((vb >> (2 * i)) & 3u), s, z);
#pragma unroll
                                for (int h = 0; h < NREP; ++h) o[h][b][i] = fmaf(p[h], v, o[h][b][i]);
                            }
                        }
                    }
                }
                __syncwarp();
            }
        }
    } else {
        // residual ring, full precision (cache/manager.py:275-278)
        const int R = L.residual_cap;
        for (int c0 = warp * 32; c0 < res_len; c0 += kWarps * 32) {
            const int r = c0 + lane;
            const bool valid = r < res_len;
            float acc[NREP];
#pragma unroll
            for (int h = 0; h < NREP; ++h) acc[h] = 0.0f;
            if (valid) {
                const int slot = (res_start + r) % R;
                const int64_t base = ((int64_t)u * R + slot) * D;
                for (int d = 0; d < D; ++d) {
                    const float k = load_as_float(L.k_res, L.res_dtype, base + d);
#pragma unroll
                    for (int h = 0; h < NREP; ++h) acc[h] = fmaf(q_s[h * D + d], k, acc[h]);
                }
            }
            absorb_scores(acc, valid);
            const int ntok = res_len - c0 < 32 ? res_len - c0 : 32;
            for (int tk = 0; tk < ntok; ++tk) {
                const int slot = (res_start + c0 + tk) % R;
                const int64_t base = ((int64_t)u * R + slot) * D;
                float p[NREP];
#pragma unroll
                for (int h = 0; h < NREP; ++h) p[h] = p_s[tk * NREP + h];
#pragma unroll
                for (int b = 0; b < DB; ++b) {
                    const int byte = lane + 32 * b;
                    if (byte < D / 4) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float v = load_as_float(L.v_res, L.res_dtype, base + 4 * byte + i);
#pragma unroll
                            for (int h = 0; h < NREP; ++h) o[h][b][i] = fmaf(p[h], v, o[h][b][i]);
                        }
                    }
                }
            }
            __syncwarp();
        }
    }

    // ---- merge the warps of this CTA -------------------------------------
    float* ml_s = red_s;                         // [kWarps][NREP][2]
    float* o_s = red_s + kWarps * NREP * 2;      // [NREP][DB*128]
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        float ls = l[h];
#pragma unroll
        for (int o_ = 16; o_ > 0; o_ >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, o_);
        if (lane == 0) { ml_s[(warp * NREP + h) * 2] = m[h]; ml_s[(warp * NREP + h) * 2 + 1] = ls; }
    }
    for (int i = threadIdx.x; i < NREP * DB * 128; i += blockDim.x) o_s[i] = 0.0f;
    __syncthreads();
    float M[NREP];
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        float mm = -INFINITY;
        for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, ml_s[(w * NREP + h) * 2]);
        M[h] = mm;
    }
    for (int w = 0; w < kWarps; ++w) {
        if (warp == w) {
#pragma unroll
            for (int h = 0; h < NREP; ++h) {
                const float f = (m[h] == -INFINITY) ? 0.0f : exp2f(m[h] - M[h]);
#pragma unroll
                for (int b = 0; b < DB; ++b)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        o_s[h * DB * 128 + (lane + 32 * b) * 4 + i] += o[h][b][i] * f;
            }
        }
        __syncthreads();
    }
    const int64_t pbase = ((int64_t)u * n_splits + split) * NREP;
    for (int i = threadIdx.x; i < NREP * D; i += blockDim.x) {
        const int h = i / D, d = i % D;
        part_o[(pbase + h) * D + d] = o_s[h * DB * 128 + d];
    }
    if (threadIdx.x < NREP) {
        const int h = threadIdx.x;
        float ls = 0.0f;
        for (int w = 0; w < kWarps; ++w) {
            const float mw = ml_s[(w * NREP + h) * 2];
            if (mw != -INFINITY) ls += ml_s[(w * NREP + h) * 2 + 1] * exp2f(mw - M[h]);
        }
        part_ml[(pbase + h) * 2] = M[h];
        part_ml[(pbase + h) * 2 + 1] = ls;
    }
}

// ---- fp32 kernel for head_dim 64 and 128 -----------------------------------------
// Same arithmetic (k = code*scale + zero in one fp32 rounding, fp32 FMAs for both
// contractions), organised so that little is left beside the FMAs:
//   * every warp streams its own token groups into a private two-stage ring in shared
//     memory with bulk copies (the six arrays of a group are contiguous runs);
//   * q.k: a lane takes four tokens x D/4 channels, exactly what its 32-bit code
//     words hold (4 tokens x 4 channels), so a code is read once, a dequantized
//     key serves all heads, and a query or scale read serves four tokens; the lanes
//     of a token quad then exchange partial sums and lane l ends with token l;
//   * p.v: a lane takes four channels, a word is again 4 tokens x 4 channels;
//   * a code becomes a float with one byte permute (2^23 + c) and half a packed
//     subtract; dequantization and both contractions are packed two to an instruction
//     (same rate on the FMA pipe, half the issue slots);
//   * a running maximum is only worked out when a score exceeds it.
// What bounds it: no single pipe.  A lane's 256 codes of a group cost one FMA per code and
// head (256 cycles of the SM quarter per head: two per packed instruction, which does two)
// and about 1000 cycles of conversion (a byte permute, half a packed add and half a packed
// FMA per code), so four heads need 2000 of the 3800-4100 cycles a group takes.  Counters
// on 160 units x 8k, four heads: 2060 instructions per group and warp, issue slots 60 %
// busy, FMA pipe 53 %, ALU 43 %, shared-memory pipe (query, weight and scale reads) 46 %,
// with 11 warps on an SM (162 registers) to cover the latencies in between.
// Measured 2150 / 4100 / 6700 cycles per group with 1 / 4 / 8 heads, against 13000 with
// four heads in the generic kernel (dependent 32-bit loads, an integer conversion per
// code).  32 units x 8k tokens, 4 heads: 99 -> 37 us; 32 x 32k, 1 head: 259 -> 67 us;
// 12 units x 712 tokens, head_dim 64: 18.4 -> 5.1 us (with the fold in a cluster).
// Error against 64 bits is about half of the generic kernel's (shorter chains of adds).
template <int D> struct Fp32Tile {
    static constexpr int kBytes = D / 4;               // packed value bytes of a token
    static constexpr int kTokPar = 32 / kBytes;        // token quads a warp takes side by side in p.v (2 for D = 64)
};

// score of one token per lane and head -> weight; running maximum, sum and outputs of the warp
template <int NREP, int NO>
__device__ __forceinline__ void absorb(float (&s)[NREP], bool valid, float* __restrict__ p_slot, float (&m)[NREP], float (&l)[NREP], float2 (&o)[NREP][NO]) {
    bool above = false;
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        s[h] = valid ? s[h] : -INFINITY;
        above |= s[h] > m[h];
    }
    if (__any_sync(0xffffffffu, above)) {
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            float mx = s[h];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float m_new = fmaxf(m[h], mx);
            const float alpha = m_new == -INFINITY ? 1.0f : exp2f(m[h] - m_new);       // 0 on the first chunk
            m[h] = m_new;
            l[h] *= alpha;
#pragma unroll
            for (int i = 0; i < NO; ++i) o[h][i] = mul2(o[h][i], both(alpha));
        }
    }
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        const float p = valid ? exp2f(s[h] - m[h]) : 0.0f;
        l[h] += p;
        p_slot[h] = p;
    }
}

template <int NREP> __device__ __forceinline__ void load_weights(const float* __restrict__ p, float (&w)[NREP]) {
    if constexpr (NREP % 4 == 0) {
#pragma unroll
        for (int h = 0; h < NREP; h += 4) {
            const float4 t = *reinterpret_cast<const float4*>(p + h);
            w[h] = t.x; w[h + 1] = t.y; w[h + 2] = t.z; w[h + 3] = t.w;
        }
    } else if constexpr (NREP % 2 == 0) {
#pragma unroll
        for (int h = 0; h < NREP; h += 2) {
            const float2 t = *reinterpret_cast<const float2*>(p + h);
            w[h] = t.x; w[h + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int h = 0; h < NREP; ++h) w[h] = p[h];
    }
}

// the four 2-bit fields at bits 0-1 of the bytes of t, as floats
__device__ __forceinline__ void codes_to_float(uint32_t t, float2& a, float2& b) {
    const float2 x = make_float2(__uint_as_float(__byte_perm(t, 0x4B000000u, 0x7440)), __uint_as_float(__byte_perm(t, 0x4B000000u, 0x7441)));
    const float2 y = make_float2(__uint_as_float(__byte_perm(t, 0x4B000000u, 0x7442)), __uint_as_float(__byte_perm(t, 0x4B000000u, 0x7443)));
    a = add2(x, both(-8388608.0f));
    b = add2(y, both(-8388608.0f));
}

template <typename T> __device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <> __device__ __forceinline__ void load4<float>(const float* p, float (&v)[4]) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
template <> __device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 t = __ldg(reinterpret_cast<const uint2*>(p));
    v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xffff0000u);
    v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xffff0000u);
}

// window tokens of one warp (every kWarps-th run of 32): lane (tl, cq) scores tokens
// tl + 8j, j = 0..3, over channels cq*D/4 .. ; lane = token tl + 8*cq afterwards
template <int NREP, int D, typename T>
__device__ __forceinline__ void ring_tokens(const T* __restrict__ k_res, const T* __restrict__ v_res, int R, int res_start, int res_len,
                                            const float* __restrict__ q_s, float scale_log2, float* __restrict__ p_s, int lane, int warp,
                                            float (&m)[NREP], float (&l)[NREP], float2 (&o)[NREP][2]) {
    constexpr int kTokPar = Fp32Tile<D>::kTokPar, kBytes = Fp32Tile<D>::kBytes;
    const int tl = lane >> 2, cq = lane & 3;
    for (int t0 = 32 * warp; t0 < res_len; t0 += 32 * kWarps) {
        const int ntok = res_len - t0 < 32 ? res_len - t0 : 32;
        float2 acc[4][NREP];
        const T* row[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int slot = res_start + t0 + (tl + 8 * j < ntok ? tl + 8 * j : 0);
            if (slot >= R) slot -= R;
            row[j] = k_res + (int64_t)slot * D + cq * (D / 4);
#pragma unroll
            for (int h = 0; h < NREP; ++h) acc[j][h] = make_float2(0.0f, 0.0f);
        }
#pragma unroll 2
        for (int c = 0; c < D / 4; c += 4) {
            float kv[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) load4<T>(row[j] + c, kv[j]);
#pragma unroll
            for (int h = 0; h < NREP; ++h) {
                const float4 q4 = *reinterpret_cast<const float4*>(q_s + h * D + cq * (D / 4) + c);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[j][h] = fma2(make_float2(q4.x, q4.y), make_float2(kv[j][0], kv[j][1]), acc[j][h]);
                    acc[j][h] = fma2(make_float2(q4.z, q4.w), make_float2(kv[j][2], kv[j][3]), acc[j][h]);
                }
            }
        }
        float s[NREP];
#pragma unroll
        for (int h = 0; h < NREP; ++h) {
            float a[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                a[j] = acc[j][h].x + acc[j][h].y;
                a[j] += __shfl_xor_sync(0xffffffffu, a[j], 1);
                a[j] += __shfl_xor_sync(0xffffffffu, a[j], 2);
            }
            s[h] = (cq == 0 ? a[0] : cq == 1 ? a[1] : cq == 2 ? a[2] : a[3]) * scale_log2;
        }
        __syncwarp();
        absorb<NREP, 2>(s, tl + 8 * cq < ntok, p_s + (tl + 8 * cq) * NREP, m, l, o);
        __syncwarp();
        const int b = lane % kBytes, tp = lane / kBytes;
        for (int k0 = 0; k0 < ntok; k0 += 8 * kTokPar) {
            float vv[8][4];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int tk = k0 + k * kTokPar + tp;
                int slot = res_start + t0 + (tk < ntok ? tk : 0);
                if (slot >= R) slot -= R;
                load4<T>(v_res + (int64_t)slot * D + 4 * b, vv[k]);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int tk = k0 + k * kTokPar + tp;
                float w[NREP];
                load_weights<NREP>(p_s + (tk < ntok ? tk : 0) * NREP, w);
#pragma unroll
                for (int h = 0; h < NREP; ++h) {
                    const float2 pp = both(tk < ntok ? w[h] : 0.0f);
                    o[h][0] = fma2(pp, make_float2(vv[k][0], vv[k][1]), o[h][0]);
                    o[h][1] = fma2(pp, make_float2(vv[k][2], vv[k][3]), o[h][1]);
                }
            }
        }
    }
}

__device__ int g_fp32_copy_fault = 0;

// Shared memory: warps' stage rings [kWarps][2][stage_bytes] (a warp's ring doubles as
// its [NREP][D] output buffer) | queries [NREP][D] | weights [kWarps][32][NREP] |
// mbarriers [kWarps][2] | (max, sum) [kWarps][NREP][2]
template <int NREP, int D>
__global__ void __launch_bounds__(kWarps * 32, NREP <= 2 ? 4 : NREP <= 6 ? 3 : 2)
attn_fp32_tile_kernel(kivi_layer L, int64_t quant_len, int res_start, int res_len,
                      const void* q, int q_dtype, float scale_log2,
                      int nq_splits, int groups_per_split, int n_splits, int stage_bytes,
                      float* __restrict__ part_o, float* __restrict__ part_ml, ClusterOut direct) {
    constexpr int kBytes = Fp32Tile<D>::kBytes, kTokPar = Fp32Tile<D>::kTokPar;
    const int G = L.group_size, ng = D / G;
    const int u = blockIdx.y, split = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t* ring = smem_raw + warp * 2 * stage_bytes;
    float* q_s = reinterpret_cast<float*>(smem_raw + kWarps * 2 * stage_bytes);
    float* p_s = q_s + NREP * D + warp * 32 * NREP;
    uint64_t* bars = reinterpret_cast<uint64_t*>(q_s + NREP * D + kWarps * 32 * NREP);
    float* ml_s = reinterpret_cast<float*>(bars + kWarps * 2);
    if (direct.out == nullptr) cudaTriggerProgrammaticLaunchCompletion();      // the kernel that folds the partials may become resident (attn_mma.cu)
    stream_order();
    q = settled(q);
    settle_layer(L);

    const bool is_ring = split >= nq_splits;
    const int64_t g_begin = is_ring ? 0 : (int64_t)split * groups_per_split;
    int64_t g_end = is_ring ? 0 : g_begin + groups_per_split;
    if (g_end > quant_len / G) g_end = quant_len / G;
    const int n_my = (int)(g_end - g_begin) > warp ? ((int)(g_end - g_begin) - warp + kWarps - 1) / kWarps : 0;
    // the six pieces of a group: key codes, scales, zeros, value codes, scales, zeros
    const uint32_t code_bytes = (uint32_t)(D * G / 4), meta_bytes = D * 4;
    const uint32_t bar0 = smem_u32(bars + warp * 2), ring0 = smem_u32(ring);
    const uint64_t policy = l2_stream_policy();
    const uint8_t* my_src = nullptr;
    uint32_t my_bytes = 0, my_dst = 0;
    auto issue = [&](int i) {                             // the warp's i-th group
        const uint32_t bar = bar0 + 8 * (i & 1);
        if (lane == 0) mbar_expect_tx(bar, 2 * code_bytes + 4 * meta_bytes);
        __syncwarp();
        if (lane < 6) bulk_g2s(ring0 + (i & 1) * stage_bytes + my_dst, my_src + (int64_t)i * kWarps * my_bytes, my_bytes, bar, policy);
    };
    if (n_my > 0) {
        const uint8_t* base = lane == 0 ? L.k_codes
                            : lane == 1 ? reinterpret_cast<const uint8_t*>(L.k_scales)
                            : lane == 2 ? reinterpret_cast<const uint8_t*>(L.k_zeros)
                            : lane == 3 ? L.v_codes
                            : lane == 4 ? reinterpret_cast<const uint8_t*>(L.v_scales)
                                        : reinterpret_cast<const uint8_t*>(L.v_zeros);
        my_bytes = (lane == 0 || lane == 3) ? code_bytes : meta_bytes;
        my_dst = lane <= 3 ? (lane == 0 ? 0u : code_bytes + (lane - 1) * meta_bytes) : 2 * code_bytes + (lane - 2) * meta_bytes;
        my_src = base + ((int64_t)u * (L.max_tokens / G) + g_begin + warp) * my_bytes;
        if (lane == 0) { mbar_init(bar0, 1); mbar_init(bar0 + 8, 1); mbar_init_fence(); }
        __syncwarp();
        issue(0);
        if (n_my > 1) issue(1);
    }
    for (int i = threadIdx.x; i < NREP * D; i += blockDim.x)
        q_s[i] = load_as_float(q, q_dtype, (int64_t)u * NREP * D + i);
    __syncthreads();

    float m[NREP], l[NREP];
    float2 o[NREP][2];
#pragma unroll
    for (int h = 0; h < NREP; ++h) { m[h] = -INFINITY; l[h] = 0.0f; o[h][0] = make_float2(0.0f, 0.0f); o[h][1] = o[h][0]; }

    if (is_ring) {
        const int64_t r0 = (int64_t)u * L.residual_cap * D;
        if (L.res_dtype == KIVI_BF16)
            ring_tokens<NREP, D, __nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(L.k_res) + r0, reinterpret_cast<const __nv_bfloat16*>(L.v_res) + r0,
                                                L.residual_cap, res_start, res_len, q_s, scale_log2, p_s, lane, warp, m, l, o);
        else
            ring_tokens<NREP, D, float>(reinterpret_cast<const float*>(L.k_res) + r0, reinterpret_cast<const float*>(L.v_res) + r0,
                                        L.residual_cap, res_start, res_len, q_s, scale_log2, p_s, lane, warp, m, l, o);
    } else {
        const int j = lane >> 2, cq = lane & 3;           // q.k: token quad, channels 16*i + 4*cq
        const int b = lane % kBytes, tp = lane / kBytes;  // p.v: packed byte (four channels), token quads tp, tp + kTokPar, ...
        const int gd = 4 * b / G;
        const bool blocks = value_blocks(D, G);
        int i = 0;
        for (; i < n_my; ++i) {
            if (!mbar_wait(bar0 + 8 * (i & 1), (uint32_t)(i >> 1) & 1u)) break;
            __syncwarp();
            const uint8_t* kc = ring + (i & 1) * stage_bytes;
            const float* ks = reinterpret_cast<const float*>(kc + code_bytes);
            const float* kz = ks + D;
            const uint8_t* vc = kc + code_bytes + 2 * meta_bytes;
            const float* vs = reinterpret_cast<const float*>(vc + code_bytes);
            const float* vz = vs + D;
            for (int c0 = 0; c0 < G; c0 += 32) {          // 32 tokens at a time (fewer when G has no 32)
                const int nt = G - c0 < 32 ? G - c0 : 32;
                float2 acc[4][NREP];
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int h = 0; h < NREP; ++h) acc[e][h] = make_float2(0.0f, 0.0f);
                const uint8_t* krow = kc + (c0 / 4 + (4 * j < nt ? j : 0)) * 64 + cq * 16;
#pragma unroll
                for (int hh = 0; hh < D / 64; ++hh) {
                    const uint4 wv = *reinterpret_cast<const uint4*>(krow + hh * 16 * G);
                    const uint32_t w4[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                    for (int mm = 0; mm < 4; ++mm) {
                        const int ch = 64 * hh + 16 * mm + 4 * cq;
                        const float4 s4 = *reinterpret_cast<const float4*>(ks + ch), z4 = *reinterpret_cast<const float4*>(kz + ch);
                        float2 k01[4], k23[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            codes_to_float((w4[mm] >> (2 * e)) & 0x03030303u, k01[e], k23[e]);
                            k01[e] = fma2(k01[e], make_float2(s4.x, s4.y), make_float2(z4.x, z4.y));
                            k23[e] = fma2(k23[e], make_float2(s4.z, s4.w), make_float2(z4.z, z4.w));
                        }
#pragma unroll
                        for (int h = 0; h < NREP; ++h) {
                            const float4 q4 = *reinterpret_cast<const float4*>(q_s + h * D + ch);
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                acc[e][h] = fma2(make_float2(q4.x, q4.y), k01[e], acc[e][h]);
                                acc[e][h] = fma2(make_float2(q4.z, q4.w), k23[e], acc[e][h]);
                            }
                        }
                    }
                }
                // sums over the four lanes of a quad; lane 4j + cq keeps token 4j + cq
                float s[NREP];
#pragma unroll
                for (int h = 0; h < NREP; ++h) {
                    float a[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) a[e] = acc[e][h].x + acc[e][h].y;
                    const bool hi = (cq & 2) != 0, odd = (cq & 1) != 0;
                    const float x0 = (hi ? a[2] : a[0]) + __shfl_xor_sync(0xffffffffu, hi ? a[0] : a[2], 2);
                    const float x1 = (hi ? a[3] : a[1]) + __shfl_xor_sync(0xffffffffu, hi ? a[1] : a[3], 2);
                    s[h] = ((odd ? x1 : x0) + __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 1)) * scale_log2;
                }
                __syncwarp();                             // the weights of the chunk before have been read
                absorb<NREP, 2>(s, lane < nt, p_s + lane * NREP, m, l, o);
                __syncwarp();
                for (int qd = tp; 4 * qd < nt; qd += kTokPar) {
                    const int t = c0 + 4 * qd;            // tokens t .. t+3 of the group
                    uint32_t w;
                    int row, row_step;                    // scale / zero index of token t + n: row + n * row_step
                    if (blocks) {                         // word (gd, kappa, r, c): four tokens of one byte (kivi_common.cuh)
                        w = *reinterpret_cast<const uint32_t*>(vc + ((b >> 3) * 64 + (qd >> 2) * 32 + (b & 7) * 4 + (qd & 3)) * 4);
                        row = (16 * (qd >> 2) + (qd & 3)) * 4 + gd; row_step = 16;
                    } else {                              // one row per token
                        const uint8_t* r0 = vc + t * kBytes + b;
                        w = (uint32_t)r0[0] | ((uint32_t)r0[kBytes] << 8) | ((uint32_t)r0[2 * kBytes] << 16) | ((uint32_t)r0[3 * kBytes] << 24);
                        row = t * ng + gd; row_step = ng;
                    }
                    // v[i]: channel 4b + i of tokens (0, 1) and (2, 3)
                    float2 c01[4], c23[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) codes_to_float((w >> (2 * e)) & 0x03030303u, c01[e], c23[e]);
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        const float sc = vs[row + n * row_step], zc = vz[row + n * row_step];
                        const float2 a = n < 2 ? (n == 0 ? make_float2(c01[0].x, c01[1].x) : make_float2(c01[0].y, c01[1].y))
                                               : (n == 2 ? make_float2(c23[0].x, c23[1].x) : make_float2(c23[0].y, c23[1].y));
                        const float2 c = n < 2 ? (n == 0 ? make_float2(c01[2].x, c01[3].x) : make_float2(c01[2].y, c01[3].y))
                                               : (n == 2 ? make_float2(c23[2].x, c23[3].x) : make_float2(c23[2].y, c23[3].y));
                        const float2 v01 = fma2(a, both(sc), both(zc)), v23 = fma2(c, both(sc), both(zc));
                        float wt[NREP];
                        load_weights<NREP>(p_s + (4 * qd + n) * NREP, wt);
#pragma unroll
                        for (int h = 0; h < NREP; ++h) {
                            o[h][0] = fma2(both(wt[h]), v01, o[h][0]);
                            o[h][1] = fma2(both(wt[h]), v23, o[h][1]);
                        }
                    }
                }
            }
            __syncwarp();
            if (i + 2 < n_my) issue(i + 2);
        }
        if (i < n_my) {
            // A copy did not land within the bound: the ones still under way get a second
            // bounded wait before the ring is reused, then the warp reports nothing.
            if (lane == 0) atomicExch(&g_fp32_copy_fault, 1);
            for (int k = i; k < i + 2 && k < n_my; ++k) mbar_wait(bar0 + 8 * (k & 1), (uint32_t)(k >> 1) & 1u);
#pragma unroll
            for (int h = 0; h < NREP; ++h) { m[h] = -INFINITY; l[h] = 0.0f; o[h][0] = make_float2(0.0f, 0.0f); o[h][1] = o[h][0]; }
        }
    }

    // ---- fold the warps ---------------------------------------------------------------
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], off);
        if (lane == 0) { ml_s[(warp * NREP + h) * 2] = m[h]; ml_s[(warp * NREP + h) * 2 + 1] = l[h]; }
        if constexpr (kTokPar == 2) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                o[h][i].x += __shfl_xor_sync(0xffffffffu, o[h][i].x, 16);
                o[h][i].y += __shfl_xor_sync(0xffffffffu, o[h][i].y, 16);
            }
        }
    }
    __syncthreads();
    float* mine = reinterpret_cast<float*>(ring);
#pragma unroll
    for (int h = 0; h < NREP; ++h) {
        float M = -INFINITY;
#pragma unroll
        for (int w2 = 0; w2 < kWarps; ++w2) M = fmaxf(M, ml_s[(w2 * NREP + h) * 2]);
        const float f = m[h] == -INFINITY ? 0.0f : exp2f(m[h] - M);
        if (lane < kBytes)
            *reinterpret_cast<float4*>(mine + h * D + 4 * lane) = make_float4(f * o[h][0].x, f * o[h][0].y, f * o[h][1].x, f * o[h][1].y);
    }
    __syncthreads();
    const int64_t pbase = ((int64_t)u * n_splits + split) * NREP;
    for (int i = threadIdx.x * 4; i < NREP * D; i += blockDim.x * 4) {
        float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(smem_raw) + i);
#pragma unroll
        for (int w2 = 1; w2 < kWarps; ++w2) {
            const float4 c = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(smem_raw + w2 * 2 * stage_bytes) + i);
            a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
        }
        // (the queries and the weights have been read for the last time)
        *reinterpret_cast<float4*>(direct.out ? q_s + i : part_o + pbase * D + i) = a;
    }
    float* const ml_out = direct.out ? q_s + NREP * D : part_ml + pbase * 2;
    if (threadIdx.x < NREP) {
        const int h = threadIdx.x;
        float M = -INFINITY, ls = 0.0f;
        for (int w2 = 0; w2 < kWarps; ++w2) M = fmaxf(M, ml_s[(w2 * NREP + h) * 2]);
        for (int w2 = 0; w2 < kWarps; ++w2) {
            const float mw = ml_s[(w2 * NREP + h) * 2];
            if (mw != -INFINITY) ls += ml_s[(w2 * NREP + h) * 2 + 1] * exp2f(mw - M);
        }
        ml_out[h * 2] = M;
        ml_out[h * 2 + 1] = ls;
    }
    if (direct.out) cluster_fold(q_s, ml_out, NREP, D, (int64_t)u * NREP, direct);
}

}  // namespace

namespace {

// out[u][h][:] = sum_s o_s * 2^(m_s - M) / sum_s l_s * 2^(m_s - M)
// One warp per output row (row = u*n_rep + h), kMergeWarps rows per CTA; partials
// laid out [(u*n_splits + s)*n_rep + h].  Lane s holds (m_s, l_s) and the weight
// of split s, the maximum and the denominator are warp reductions, and every
// lane folds four channels with 16-byte loads, the weights handed round by
// shuffle.  `sink(index, float4)` receives the four output elements starting at
// index = row*D + d (d a multiple of four; head_dim is a multiple of four).
constexpr int kMergeWarps = 8;

template <typename Sink>
__device__ __forceinline__ void merge_row(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                          int n_splits, int nrep, int64_t row, int D, const Sink& sink,
                                          float* __restrict__ lse) {
    const int lane = threadIdx.x & 31;
    const int64_t u = row / nrep;
    const int h = (int)(row - u * nrep);
    const int64_t row0 = u * n_splits * nrep + h;            // + s*nrep
    float M = -INFINITY;
    for (int s = lane; s < n_splits; s += 32) M = fmaxf(M, part_ml[(row0 + (int64_t)s * nrep) * 2]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    for (int d0 = 0; d0 < D; d0 += 128) {
        const int d = d0 + 4 * lane;
        const bool active = d < D;
        float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
        float den = 0.0f;
        for (int s0 = 0; s0 < n_splits; s0 += 32) {
            const int s = s0 + lane;
            float wgt = 0.0f;
            if (s < n_splits) {
                const float2 ml = *reinterpret_cast<const float2*>(part_ml + (row0 + (int64_t)s * nrep) * 2);
                wgt = (ml.x == -INFINITY) ? 0.0f : exp2f(ml.x - M);
                den = fmaf(wgt, ml.y, den);
            }
            const int cnt = min(32, n_splits - s0);
            const float* src = part_o + (row0 + (int64_t)s0 * nrep) * D + (active ? d : 0);
            // eight partial rows in flight per lane (a unit cut into a hundred pieces
            // would otherwise pay a hundred load latencies in a row); rows past the
            // end are the last row again, with weight zero
            for (int i = 0; i < cnt; i += 8) {
                float4 v[8];
                float w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int k = i + j < cnt ? i + j : cnt - 1;
                    v[j] = *reinterpret_cast<const float4*>(src + (int64_t)k * nrep * D);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float wj = __shfl_sync(0xffffffffu, wgt, (i + j) & 31);
                    w[j] = i + j < cnt ? wj : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    a0.x = fmaf(v[j].x, w[j], a0.x); a0.y = fmaf(v[j].y, w[j], a0.y);
                    a0.z = fmaf(v[j].z, w[j], a0.z); a0.w = fmaf(v[j].w, w[j], a0.w);
                    a1.x = fmaf(v[j + 1].x, w[j + 1], a1.x); a1.y = fmaf(v[j + 1].y, w[j + 1], a1.y);
                    a1.z = fmaf(v[j + 1].z, w[j + 1], a1.z); a1.w = fmaf(v[j + 1].w, w[j + 1], a1.w);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
        const float inv = 1.0f / den;
        // natural-log sum of exponentials of the scaled scores (M and den live in the log2 domain)
        if (lse != nullptr && lane == 0 && d0 == 0) lse[row] = (M + log2f(den)) * 0.6931471805599453f;
        if (active)
            sink(row * D + d, make_float4((a0.x + a1.x) * inv, (a0.y + a1.y) * inv, (a0.z + a1.z) * inv, (a0.w + a1.w) * inv));
    }
}

// The same fold with all kMergeWarps warps of a CTA on ONE row, for rows with
// many partials (few units cut into many pieces): warp w folds pieces w, w + 8,
// ... with eight loads in flight, the warps' sums meet in shared memory and are
// added in warp order.  (A different summation order than merge_row: which of
// the two a call uses depends on its piece count alone.)
constexpr int kMergeWideFrom = 17;            // partials per row from which the CTA-wide fold is used

template <typename Sink>
__device__ __forceinline__ void merge_row_wide(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                               int n_splits, int nrep, int64_t row, int D, const Sink& sink,
                                               float* __restrict__ lse, float (*fold_s)[128]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t u = row / nrep;
    const int h = (int)(row - u * nrep);
    const int64_t row0 = u * n_splits * nrep + h;            // + s*nrep
    // every warp works out the maximum and the denominator itself (same loads, same order, same bits)
    float M = -INFINITY;
    for (int s = lane; s < n_splits; s += 32) M = fmaxf(M, part_ml[(row0 + (int64_t)s * nrep) * 2]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float den = 0.0f;
    for (int s = lane; s < n_splits; s += 32) {
        const float2 ml = *reinterpret_cast<const float2*>(part_ml + (row0 + (int64_t)s * nrep) * 2);
        den = fmaf((ml.x == -INFINITY) ? 0.0f : exp2f(ml.x - M), ml.y, den);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    const float inv = 1.0f / den;
    const int n_mine = warp < n_splits ? (n_splits - warp + kMergeWarps - 1) / kMergeWarps : 0;
    for (int d0 = 0; d0 < D; d0 += 128) {
        const int d = d0 + 4 * lane;
        const bool active = d < D;
        float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
        const float* src = part_o + row0 * D + (active ? d : 0);
        for (int i = 0; i < n_mine; i += 8) {
            float4 v[8];
            float w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int s = warp + kMergeWarps * (i + j < n_mine ? i + j : n_mine - 1);
                v[j] = *reinterpret_cast<const float4*>(src + (int64_t)s * nrep * D);
                const float ms = part_ml[(row0 + (int64_t)s * nrep) * 2];
                w[j] = (i + j < n_mine && ms != -INFINITY) ? exp2f(ms - M) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                a0.x = fmaf(v[j].x, w[j], a0.x); a0.y = fmaf(v[j].y, w[j], a0.y);
                a0.z = fmaf(v[j].z, w[j], a0.z); a0.w = fmaf(v[j].w, w[j], a0.w);
                a1.x = fmaf(v[j + 1].x, w[j + 1], a1.x); a1.y = fmaf(v[j + 1].y, w[j + 1], a1.y);
                a1.z = fmaf(v[j + 1].z, w[j + 1], a1.z); a1.w = fmaf(v[j + 1].w, w[j + 1], a1.w);
            }
        }
        *reinterpret_cast<float4*>(&fold_s[warp][4 * lane]) = make_float4(a0.x + a1.x, a0.y + a1.y, a0.z + a1.z, a0.w + a1.w);
        __syncthreads();
        if (warp == 0) {
            float4 t = *reinterpret_cast<const float4*>(&fold_s[0][4 * lane]);
#pragma unroll
            for (int w2 = 1; w2 < kMergeWarps; ++w2) {
                const float4 b = *reinterpret_cast<const float4*>(&fold_s[w2][4 * lane]);
                t.x += b.x; t.y += b.y; t.z += b.z; t.w += b.w;
            }
            // natural-log sum of exponentials of the scaled scores (M and den live in the log2 domain)
            if (lse != nullptr && lane == 0 && d0 == 0) lse[row] = (M + log2f(den)) * 0.6931471805599453f;
            if (active) sink(row * D + d, make_float4(t.x * inv, t.y * inv, t.z * inv, t.w * inv));
        }
        __syncthreads();                                  // fold_s is rewritten by the next 128 channels
    }
}

struct LocalSink {
    void* out;
    int out_dtype;
    __device__ void operator()(int64_t i, float4 v) const { store_quad(out, out_dtype, i, v); }
};

__global__ void __launch_bounds__(kMergeWarps * 32)
merge_splits_kernel(const float* part_o, const float* part_ml,
                    void* __restrict__ out, int out_dtype, int n_splits, int nrep, int64_t rows, int D,
                    float* __restrict__ lse) {
    // the launch may overlap the tail of the attention kernel, the partials may not
    // be read before that kernel has completed
    __shared__ __align__(16) float fold_s[kMergeWarps][128];
    stream_order();
    part_o = settled(part_o); part_ml = settled(part_ml);
    if (n_splits >= kMergeWideFrom) {                     // grid = rows: the whole CTA on one row
        merge_row_wide(part_o, part_ml, n_splits, nrep, (int64_t)blockIdx.x, D, LocalSink{out, out_dtype}, lse, fold_s);
        return;
    }
    const int64_t row = (int64_t)blockIdx.x * kMergeWarps + (threadIdx.x >> 5);
    if (row < rows) merge_row(part_o, part_ml, n_splits, nrep, row, D, LocalSink{out, out_dtype}, lse);
}

// ---- merge + all-gather over peer memory -------------------------------------------
// The same fold, but every output row is stored into the gathered buffer of
// every rank (plain stores through peer-mapped pointers).  When the last CTA of
// the grid has finished, lane r of its first warp publishes this rank's epoch in
// rank r's flag array and, if asked, waits (bounded) until rank r has published
// it here: one fence, then all flags and all waits side by side.
__device__ unsigned g_gather_done = 0;      // CTAs of the running launch that have stored their row
__device__ int g_gather_fault = 0;

__device__ __forceinline__ void st_relaxed_sys(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

struct PeerSink {
    kivi_peer_gather g;
    int out_dtype;
    int64_t base;              // element offset of this rank's first row in a gathered buffer
    int64_t alt;               // byte offset of the buffer this call writes (device-kept epoch: odd calls)
    __device__ void operator()(int64_t i, float4 v) const {
#pragma unroll
        for (int r = 0; r < KIVI_PEER_MAX_WORLD; ++r)
            if (r < g.world) store_quad(reinterpret_cast<uint8_t*>(g.out_ptrs[r]) + alt, out_dtype, base + i, v);
    }
};

constexpr uint32_t kPeerSpinLimit = 5u << 20;      // default bound: x 200 ns sleeps, about a second

__global__ void __launch_bounds__(kMergeWarps * 32)
merge_gather_kernel(const float* part_o, const float* part_ml,
                    kivi_peer_gather g, int out_dtype, int n_splits, int nrep, int64_t rows, int D) {
    cudaGridDependencySynchronize();
    part_o = settled(part_o); part_ml = settled(part_ml);
    // Epoch kept on the device (a call replayed from a CUDA graph): every CTA
    // reads the counter here; the last CTA stores it back after all CTAs have
    // counted themselves in, that is after all of them have read it.
    uint32_t epoch = g.epoch;
    int64_t alt = 0;
    if (g.epoch_dev != nullptr) {
        epoch = *reinterpret_cast<const volatile uint32_t*>(g.epoch_dev) + 1u;
        alt = (epoch & 1u) ? g.alt_bytes : 0;
    }
    __shared__ __align__(16) float fold_s[kMergeWarps][128];
    const PeerSink sink{g, out_dtype, g.unit_offset * (int64_t)nrep * D, alt};
    if (n_splits >= kMergeWideFrom) {                     // grid = rows: the whole CTA on one row
        merge_row_wide(part_o, part_ml, n_splits, nrep, (int64_t)blockIdx.x, D, sink, nullptr, fold_s);
    } else {
        const int64_t row = (int64_t)blockIdx.x * kMergeWarps + (threadIdx.x >> 5);
        if (row < rows) merge_row(part_o, part_ml, n_splits, nrep, row, D, sink, nullptr);
    }
    __syncthreads();                                  // the CTA's stores are issued
    if (threadIdx.x >= 32) return;                    // warp 0 carries the protocol
    const int lane = threadIdx.x;
    const unsigned total = gridDim.x;
    unsigned last = 0;
    if (lane == 0) {
        __threadfence_system();                       // ... and ordered before the count below, system-wide
        last = atomicAdd(&g_gather_done, 1u) + 1u == total;
        if (last) {
            g_gather_done = 0;                        // re-armed for the next launch (stream order)
            if (g.epoch_dev != nullptr) *g.epoch_dev = epoch;
            __threadfence_system();                   // what the other CTAs published comes before the flags
        }
    }
    __syncwarp();
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    // lane r tells rank r and then waits for rank r: the flags travel, and are polled, side by side
    const bool has_peer = lane < g.world;
    if (has_peer) st_relaxed_sys(g.flag_ptrs[lane] + g.rank, epoch);
    if (!g.wait) return;
    const uint32_t limit = g.spin_limit ? g.spin_limit : kPeerSpinLimit;
    uint64_t t0 = 0;
    if (g.wait_stats && lane == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    if (has_peer) {
        const uint32_t* mine = g.flag_ptrs[g.rank] + lane;
        uint32_t it = 0;
        while ((int32_t)(ld_acquire_sys(mine) - epoch) < 0) {
            if (++it > limit) { atomicOr(&g_gather_fault, 2); break; }
            __nanosleep(200);
        }
    }
    __syncwarp();
    if (g.wait_stats && lane == 0) {
        uint64_t t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        g.wait_stats[0] += t1 - t0;        // one thread of one CTA per launch, launches are stream-ordered
        g.wait_stats[1] += 1;
    }
}

}  // namespace

int fp32_fault_word(int* out) {
    KIVI_CUDA_OK(cudaMemcpyFromSymbol(out, g_fp32_copy_fault, sizeof(int)));
    return KIVI_OK;
}

int fp32_fault_clear() {
    const int zero = 0;
    KIVI_CUDA_OK(cudaMemcpyToSymbol(g_fp32_copy_fault, &zero, sizeof(int)));
    return KIVI_OK;
}

int gather_fault_word(int* out) {
    KIVI_CUDA_OK(cudaMemcpyFromSymbol(out, g_gather_fault, sizeof(int)));
    return KIVI_OK;
}

int gather_fault_clear() {
    const int zero = 0;
    KIVI_CUDA_OK(cudaMemcpyToSymbol(g_gather_fault, &zero, sizeof(int)));
    return KIVI_OK;
}

// merge of the split partials into `out`, or (gather != nullptr) into every
// rank's gathered buffer; queued behind the attention kernel with programmatic
// stream serialization, so its launch latency overlaps that kernel's tail
int run_merge(const float* part_o, const float* part_ml, void* out, const kivi_peer_gather* gather, float* lse,
              int out_dtype, int num_units, int n_rep, int n_splits, int D, cudaStream_t st) {
    const int64_t rows = (int64_t)num_units * n_rep;
    const dim3 grid((unsigned)(n_splits >= kMergeWideFrom ? rows : (rows + kMergeWarps - 1) / kMergeWarps));
    if (gather)
        KIVI_CUDA_OK(launch(merge_gather_kernel, grid, kMergeWarps * 32, 0, st, true, part_o, part_ml, *gather, out_dtype, n_splits, n_rep, rows, D));
    else
        KIVI_CUDA_OK(launch(merge_splits_kernel, grid, kMergeWarps * 32, 0, st, true, part_o, part_ml, out, out_dtype, n_splits, n_rep, rows, D, lse));
    return KIVI_OK;
}

// ---- token shards: combine attention computed over disjoint token ranges -----------
// parts [n_shards][rows][D + 1] fp32: D outputs then the natural-log sum of
// exponentials of the shard (-inf for a shard that attended to nothing).
// out[row] = sum_i out_i * exp(lse_i - LSE) / sum_i exp(lse_i - LSE); one warp per row.
__global__ void __launch_bounds__(128)
merge_token_shards_kernel(const float* __restrict__ parts, int n_shards, int64_t rows, int D,
                          void* __restrict__ out, int out_dtype, float* __restrict__ lse_out) {
    const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const int64_t stride = rows * (D + 1);
    float M = -INFINITY;
    for (int i = 0; i < n_shards; ++i) M = fmaxf(M, parts[i * stride + row * (D + 1) + D]);
    float den = 0.0f;
    for (int i = 0; i < n_shards; ++i) {
        const float l = parts[i * stride + row * (D + 1) + D];
        den += (l == -INFINITY) ? 0.0f : expf(l - M);
    }
    for (int d = lane; d < D; d += 32) {
        float acc = 0.0f;
        for (int i = 0; i < n_shards; ++i) {
            const float l = parts[i * stride + row * (D + 1) + D];
            if (l != -INFINITY) acc = fmaf(parts[i * stride + row * (D + 1) + d], expf(l - M), acc);
        }
        store_from_float(out, out_dtype, row * D + d, acc / den);
    }
    if (lse_out != nullptr && lane == 0) lse_out[row] = M + logf(den);
}

int run_merge_token_shards(const float* parts, int n_shards, int64_t rows, int D, void* out, int out_dtype,
                           float* lse_out, cudaStream_t st) {
    merge_token_shards_kernel<<<(unsigned)((rows + 3) / 4), 128, 0, st>>>(parts, n_shards, rows, D, out, out_dtype, lse_out);
    KIVI_LAUNCH_OK();
    return KIVI_OK;
}

// The tile kernel takes head_dim 64 and 128 with 16-byte aligned arrays and groups of
// whole 16-byte pieces (any group size: D*G/4 bytes of codes are a multiple of 16);
// everything else -- other head_dims, odd alignments -- takes the generic kernel.
bool attn_fp32_tile_head_dim(int head_dim) { return head_dim == 64 || head_dim == 128; }
bool attn_fp32_tile_ok(const kivi_layer* L) {
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    return attn_fp32_tile_head_dim(L->head_dim) && al(L->k_res) && al(L->v_res) && al(L->k_codes) && al(L->k_scales) &&
           al(L->k_zeros) && al(L->v_codes) && al(L->v_scales) && al(L->v_zeros);
}

// Bytes of one stage (one group of a warp): two stages of a warp also hold its [NREP][D] outputs.
template <int NREP, int D> constexpr int tile_stage_bytes(int group_size) {
    const int stage = 2 * (D * group_size / 4) + 4 * D * 4;
    return stage < NREP * D * 2 ? NREP * D * 2 : stage;
}
template <int NREP, int D> constexpr int tile_smem_bytes(int group_size) {
    return kWarps * 2 * tile_stage_bytes<NREP, D>(group_size) + 4 * (NREP * D + kWarps * 32 * NREP) + 8 * kWarps * 2 + 4 * kWarps * NREP * 2;
}

template <int NREP, int D>
static int launch_tile(const kivi_layer* L, int64_t quant_len, int res_start, int res_len, const void* q, int q_dtype, float scale_log2,
                       int nq_splits, int gps, int n_splits, float* part_o, float* part_ml, const ClusterOut& direct, cudaStream_t st) {
    // The limit is set once per device to what the largest group (G = D) takes: threads
    // that come here together with different group sizes all write the same value.
    static std::atomic<bool> limit_set[64];
    const int stage = tile_stage_bytes<NREP, D>(L->group_size), smem = tile_smem_bytes<NREP, D>(L->group_size);
    int dev = 0;
    KIVI_CUDA_OK(cudaGetDevice(&dev));
    KIVI_REQUIRE(dev >= 0 && dev < 64, "device ordinal %d out of range", dev);
    if (smem > 48 * 1024 && !limit_set[dev].load(std::memory_order_acquire)) {
        KIVI_CUDA_OK(cudaFuncSetAttribute(attn_fp32_tile_kernel<NREP, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem_bytes<NREP, D>(D)));
        limit_set[dev].store(true, std::memory_order_release);
    }
    dim3 grid((unsigned)n_splits, (unsigned)L->num_units);
    KIVI_CUDA_OK(launch_cluster(attn_fp32_tile_kernel<NREP, D>, direct.out ? n_splits : 0, grid, kWarps * 32, (size_t)smem, st, true, *L, quant_len, res_start, res_len, q, q_dtype, scale_log2,
                        nq_splits, gps, n_splits, stage, part_o, part_ml, direct));
    return KIVI_OK;
}

template <int NREP>
static int launch_fp32(const kivi_layer* L, int64_t quant_len, int res_start, int res_len,
                       const void* q, int q_dtype, float scale_log2, int nq_splits, int gps,
                       int n_splits, float* part_o, float* part_ml, const ClusterOut& direct, cudaStream_t st) {
    const int D = L->head_dim;
    if (attn_fp32_tile_ok(L))
        return D == 64 ? launch_tile<NREP, 64>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st)
                       : launch_tile<NREP, 128>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
    const int DB = D > 128 ? 2 : 1;
    const size_t smem = sizeof(float) * ((size_t)NREP * D + kWarps * 2 * D + kWarps * 32 * NREP +
                                         kWarps * NREP * 2 + (size_t)NREP * DB * 128);
    dim3 grid((unsigned)n_splits, (unsigned)L->num_units);
    auto kernel = DB == 1 ? attn_fp32_kernel<NREP, 1> : attn_fp32_kernel<NREP, 2>;
    if (smem > 48 * 1024) KIVI_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    KIVI_CUDA_OK(launch(kernel, grid, kWarps * 32, smem, st, true, *L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml));
    return KIVI_OK;
}

int run_attn_fp32(const kivi_layer* L, int64_t quant_len, int res_start, int res_len,
                  const void* q, int q_dtype, int n_rep, float scale_log2, int nq_splits, int gps,
                  int n_splits, float* part_o, float* part_ml, const ClusterOut& direct, cudaStream_t st) {
    switch (n_rep) {
        case 1: return launch_fp32<1>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        case 2: return launch_fp32<2>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        case 3: return launch_fp32<3>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        case 4: return launch_fp32<4>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        case 5: return launch_fp32<5>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        case 6: return launch_fp32<6>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        case 7: return launch_fp32<7>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        case 8: return launch_fp32<8>(L, quant_len, res_start, res_len, q, q_dtype, scale_log2, nq_splits, gps, n_splits, part_o, part_ml, direct, st);
        default: break;
    }
    set_error("n_rep (%d) outside 1..8", n_rep);
    return KIVI_ERR_UNSUPPORTED;
}

}  // namespace kivi

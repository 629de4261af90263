// Fused decode attention over the packed KIVI cache: tensor-core kernel for
// head_dim 128, group_size 32, up to 8 query heads per KV head in blocks of
// four per CTA (sm_100a).
//
// Decode attention over 2-bit codes is instruction-bound before it is HBM-bound:
// one quantized (token, kv_head) is 128 bytes of HBM but 256 codes that each
// feed 4 query heads.  The GQA query-group tile therefore runs on the tensor
// cores (mma.sync m16n8k32, bytes in, exact 32-bit integer sums) with the codes as
// one operand, and everything that depends on scales and zeros is folded into the
// small operand, a fixed-point number cut into bytes:
//
//   q.k   score[t,h] = sum_d (q[h,d]*s[g,d]) * c[d,t]  +  sum_d q[h,d]*z[g,d]
//         A = codes of 16 tokens x 32 channels; a byte of four codes is an operand as
//         it lies, and so is what three masks leave of it (below); B = q*s in 22 bits
//         and a sign of the largest of the group and head, three bytes and a constant (16
//         columns = 4 heads x 4 bytes); the zero term is an fp32 dot product.
//   p.v   out[h,d]   = sum_t (p[h,t]*s[t,gd]) * c[t,d]  +  sum_t p[h,t]*z[t,gd]
//         A = codes of 16 channels x 32 tokens, same encoding; B = p*s in 16 bits of
//         the largest of the stage's tokens, of the same head and channel group (8 columns =
//         4 heads x 2 bytes); the zero term accumulates in fp32.
//   What shares a largest value ends in the same sums: scores of one group, outputs of one
//   channel group.  One for the whole stage cost those beside a louder neighbour their bits
//   (channel groups 32 times apart: 2.9e-3 of the quiet one's largest output, now 1e-4).
//   Two to four times as many warp reductions for that: 64 units x 32k 57.1 -> 60.5 us, 128 x 4k
//   21.8 -> 22.2, one head 32 x 8k 11.7 -> 11.9.
//   Infinities, NaN and negative value scales take an fp32 form of their own.
//
// Bytes instead of fp16 (codes as subnormals, q*s in two parts): 16 codes cost three
// ALU operations instead of nine, and every MMA contracts twice as many.  512 units x
// 32k tokens at boost clocks 416 -> 368 us (5.9 TB/s, 0.90 of a plain copy), under the power
// cap 484 -> 435 (0.76); 32 x 128k 129 -> 117, 128 x 4k 25.1 -> 23.7, and the error against the
// fp32 kernel falls to a seventh.  A group of 32 tokens takes about 510 instructions of a
// warp, 24 of them MMAs.
//
// Data movement: every warp streams its own token groups from HBM into a
// private shared-memory ring with bulk asynchronous copies (cp.async.bulk,
// completion on an mbarrier), two groups (8 KB) per stage, and masks codes in
// registers.  The small operands are made where their scales are read without
// repetition (a lane takes four channels, or one token, for all four heads) and
// travel through 2 KB of shared memory per warp to where the MMA wants them
// (ldmatrix with byte transposition).  Nothing dequantized is ever written anywhere.
// The residual ring (full precision) is handled by extra CTAs with fp32 FMAs.
//
// Every wait on an mbarrier is bounded; on expiry the warp raises the device
// fault word, stops consuming and its partial is written as "empty".
#include "async_copy.cuh"
#include "cluster_fold.cuh"
#include "kivi_common.cuh"

#include <cuda_fp16.h>

#include <atomic>
#include <type_traits>

namespace kivi {
namespace {

constexpr int kD = 128, kG = 32;
constexpr int kWarps = 4;              // warps per CTA, each with a private pipeline
constexpr int kGPS = 2;                // token groups per pipeline stage
constexpr int kStages = 2;
constexpr int kScratchBytes = 2048;    // per warp, for operands on their way from lane to lane
constexpr int kGroupBytes = 4096;      // kc 1024 | ks 512 | kz 512 | vc 1024 | vs 512 | vz 512
constexpr int kStageBytes = kGPS * kGroupBytes;

__device__ int g_fault_word = 0;

// ---- PTX wrappers ------------------------------------------------------------
// accumulator c (+)= codes x digits, both unsigned bytes: exact 32-bit integers
__device__ __forceinline__ void mma_u8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// c = start + codes x digits: `start` stays in four registers of its own for the whole kernel
__device__ __forceinline__ void mma_u8_from(const int (&start)[4], int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(start[0]), "r"(start[1]), "r"(start[2]), "r"(start[3]));
}
// Two 16 x 16 byte matrices, transposed: lane l gives the address of row l (0-15: first
// matrix, 16-31: second); lane (gid, tig) gets, as bytes, rows 4*tig .. 4*tig+3 of column
// gid and of column gid + 8 of the first (r[0], r[1]) and the second (r[2], r[3]).
__device__ __forceinline__ void ldmatrix_t8(uint32_t (&r)[4], uint32_t row_addr) {
    asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(row_addr) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, float x) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(x) : "memory"); }
__device__ __forceinline__ float lds32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// largest magnitude; NaN if any is
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c) {
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(fabsf(a)), "f"(fabsf(b)), "f"(fabsf(c)));
    return d;
}
__device__ __forceinline__ float warp_max_abs_nan(float a) {
    float d;
    asm volatile("redux.sync.max.abs.NaN.f32 %0, %1, 0xffffffff;" : "=f"(d) : "f"(a));
    return d;
}
__device__ __forceinline__ uint32_t warp_max_u32(uint32_t a) {
    uint32_t d;
    asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(d) : "r"(a));
    return d;
}

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// ---- operands ------------------------------------------------------------------
// A byte of packed codes c0 + 4 c1 + 16 c2 + 64 c3 is itself a tensor-core operand, and so
// are the bytes left by masking away c0; c0 and c1; c0, c1 and c2: three ANDs turn a 32-bit
// word (four bytes, four consecutive contraction indices) into four operands.  Neighbouring
// accumulator rows then differ by the sum wanted of one code, times 4^e, which is taken out
// (exactly) at the end.
constexpr uint32_t kFrom1 = 0xfcfcfcfcu, kFrom2 = 0xf0f0f0f0u, kFrom3 = 0xc0c0c0c0u;
constexpr float kRow1 = 0.25f, kRow2 = 0.0625f, kRow3 = 0.015625f;

// The other operand is a fixed-point number cut into bytes, each byte a column of its own.
// x = fma(w, F, M) leaves round(w * F) in the low bits of the float x.
//
// q.k: M = 2^23 + 0x4b0000, |w * F| < 1.6 * 2^21: bytes 0 and 1 are digits, byte 2 is the top
// digit plus 0x4b, byte 3 the constant 0x4b -- whose column is 0x4b * sum of the codes,
// which is what the top digit's bias adds up to.  22 bits and a sign, against 22 bits of
// each single element in an fp16 hi/lo pair whose sums the tensor core truncates at 20.
// p.v: M = 2^23, 0 <= w * F <= 65535: two digits.
// F follows the largest |w| of what goes into the same sums: the bits of a positive float x
// subtracted from those of (1 + c) * 2^n give a float y with x * y between 1 + c and
// (1 + c/2)^2 times a power of two (c = 0: 1 and 1.125).
//
// Integer accumulators start at the bits of 2^23: read as floats they are 2^23 + sum, since
// the sums stay below 2^23 (128 * 255 * 255), and differences of them are exact.
constexpr float kTwo23 = 8388608.0f;
constexpr int kTwo23Bits = 0x4b000000;
constexpr float kMagicK = 8388608.0f + 4915200.0f;        // 2^23 + 0x4b0000
// Queries in fp32 (WIDE) take five digits for q.k and four for p.v: the rest r = w * F - x,
// between -1/2 and 1/2, goes on as fma(r, 2^15, 2^23 + 0x4b00), whose low two bytes are two
// more digits (the upper with the same bias); p.v has w * F < 2^23 and eight bits below that.
// There the codes count from 1.5 (and the zero points from z + 1.5 s, the middle of a group's
// range), or the two halves of a sum would cancel and leave their roundings: a contraction
// with ones gives the sum of each digit, 1.5 times which is taken off the digit's sum.
constexpr float kMiddle = 1.5f;
constexpr uint32_t kOnes = 0x01010101u;
constexpr float kMagicRest = 8388608.0f + 19200.0f;       // 2^23 + 0x4b00
constexpr float kRestV = 255.49f;                         // 0 <= rest < 1 becomes 0 .. 255
constexpr float kSmallest = 7.888609052210118e-31f;       // 2^-100: weights below it count as zero beside it
constexpr uint32_t kExponent = 0x7f800000u, kSmallestBits = 27u << 23;
constexpr uint32_t kInverseK = 275u << 23;                // largest |w * F| is 2^21 .. 1.125 * 2^21
constexpr uint32_t kInverseV = (269u << 23) + 0x6a0000u;  // 1.828 * 2^15 .. 65523
constexpr uint32_t kInverseVWide = kInverseV + (7u << 23);         // 2^7 times that
constexpr uint32_t kLargestScale = 245u << 23;            // 2^118: times a weight (at most 2^8 and a little) still finite
constexpr float kGrowth = 8.0f;                           // weights up to 2^8 are let stand before the running maximum moves

struct WarpState {
    float m, l;            // running max / sum of head `tig` (score layout)
    float o[8][2];         // p.v sums of head tig: channel 32*(t/2) + 4*gid + 2*(t%2) + r, times 4^(2*(t%2) + r)
    float oz[4][4];        // zero-point term [head][channel group] of the tokens this lane weighs
};

// what a lane holds for the whole kernel
struct LaneView {
    int gid, tig, lane;
    float qk[4][4];        // [i][head]: pre-scaled queries of channel k_channel(lane, i)
    float4 qz[4];          // head tig, channels 4 * zero_quad(i, gid) .. + 3
    uint32_t scratch;      // the warp's 2 KB of shared memory for operands on their way from lane to lane
    uint32_t k_rows, v_rows;   // row addresses of ldmatrix_t8 for the q.k and the p.v operand
    uint32_t p_even, p_odd;    // where it leaves the weights of tokens 4*gid + 0, 2 and + 1, 3
    uint32_t p_read, v_write;
    int v_first;               // value words: contraction half read first
    int start[4];              // 2^23 in each accumulator register
    // WIDE:
    uint32_t rest_rows;        // as k_rows, for the third column block (from `spare`)
    uint32_t ones[4];          // operand whose contraction sums the other one
    const float4* q_zero;      // head tig's queries in shared memory, in place of qz
};
// The zero term q.z of a group: lane (gid, tig) takes head tig and the 16 channels 16*gid ..,
// in an order that keeps the lanes of a half-warp off each other's banks.
__device__ __forceinline__ int zero_quad(int i, int gid) { return 4 * gid + ((i + gid) & 3); }
// The q.k operand of a group: one 16-byte row per pair of channels 16 apart (the two halves
// of a 32-channel contraction step) and half of the columns; lane 8*j + y makes the rows of
// step j and channels 2*y, 2*y + 1 of each half.  In odd steps the second half comes first,
// so that the scales are read without bank conflicts.
__device__ __forceinline__ int k_channel(int l, int i) {
    const int j = l >> 3;
    return 32 * j + 16 * ((i >> 1) ^ (j & 1)) + 2 * (l & 7) + (i & 1);
}
// Row of the weights of the token whose scales are row r of the group (kivi_common.cuh:
// token 16*kappa + 4*c + n at row 16*kappa + 4*n + c), for the same reason.
__device__ __forceinline__ int p_row(int r) { return r ^ ((r >> 4) << 2); }

// ---- plain fp32 forms for values that no fixed-point number holds ------------------
// (infinities and NaN in the queries, scales or weights, negative value scales):
// dequantize as the fp32 kernels do, code * scale + zero.
__device__ __noinline__ float4 scores_plain(const uint8_t* kc, const float* ks, const float* kz, const float4* q4, int gid) {
    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
    for (int c4 = 0; c4 < 32; ++c4) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(kc + kblock_offset(4 * c4, gid, 8, 64));
        const float4 s = *reinterpret_cast<const float4*>(ks + 4 * c4), z = *reinterpret_cast<const float4*>(kz + 4 * c4);
        const float4 q = q4[c4];
        const float sv[4] = {s.x, s.y, s.z, s.w}, zv[4] = {z.x, z.y, z.z, z.w}, qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int n = 0; n < 4; ++n) a[n] = fmaf(qv[i], fmaf((float)((w >> (8 * i + 2 * n)) & 3u), sv[i], zv[i]), a[n]);
    }
    return make_float4(a[0], a[1], a[2], a[3]);
}
// channels 32*gd + 4*gid + 0..3 of one head (ONE: the only one, weights in the order of the scales)
template <bool ONE>
__device__ __noinline__ float4 weighted_plain(const uint8_t* vc, const float* vs, const float* vz, const float* p, int gd, int gid, int tig) {
    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
    for (int r = 0; r < 32; ++r) {
        const int kap = r >> 4, n = (r >> 2) & 3, c = r & 3;
        const uint32_t b = vc[(gd * 64 + kap * 32 + gid * 4 + c) * 4 + n];
        const float s = vs[4 * r + gd], z = vz[4 * r + gd], ph = p[ONE ? r : 4 * p_row(r) + tig];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = fmaf(ph, fmaf((float)((b >> (2 * i)) & 3u), s, z), a[i]);
    }
    return make_float4(a[0], a[1], a[2], a[3]);
}

// ---- NG token groups (32 tokens each) in three phases -------------------------------
// q.k: scores of the lane's four tokens (4*gid + n) of each group for head `tig`, log2 domain.
// A score is s, or for WIDE s + fine, where s is a multiple of the top digit's unit,
// so that s less the running maximum, the number exponentiated, keeps all its bits.
// `spare` (WIDE): the stage's key scales and zeros, kGPS * 1024 bytes, which take operands
// once they have been read.
template <int NG, bool WIDE>
__device__ __forceinline__ void qk_phase(const uint8_t* __restrict__ kc, const float* __restrict__ ks, const float* __restrict__ kz,
                                         const LaneView& v, uint8_t* scratch, uint32_t spare, float (&s)[NG][4], float (&fine)[NG][4]) {
    float w[NG][4][4], sv[NG][4], top[NG][4], qz[NG];       // top: largest |q * s| of a head, per group of tokens
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const float2 sa = *reinterpret_cast<const float2*>(ks + 128 * g + k_channel(v.lane, 0)), sb = *reinterpret_cast<const float2*>(ks + 128 * g + k_channel(v.lane, 2));
        sv[g][0] = sa.x; sv[g][1] = sa.y; sv[g][2] = sb.x; sv[g][3] = sb.y;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
#pragma unroll
            for (int i = 0; i < 4; ++i) w[g][i][h] = v.qk[i][h] * sv[g][i];
            top[g][h] = max3_abs_nan(w[g][2][h], w[g][3][h], max3_abs_nan(w[g][0][h], w[g][1][h], kSmallest));
        }
    }
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int h = 0; h < 4; ++h) top[g][h] = warp_max_abs_nan(top[g][h]);
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        float z0 = 0.0f, z1 = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float4 z = *reinterpret_cast<const float4*>(kz + 128 * g + 4 * zero_quad(i, v.gid));
            if constexpr (WIDE) {
                const float4 a = *reinterpret_cast<const float4*>(ks + 128 * g + 4 * zero_quad(i, v.gid));
                z.x = fmaf(kMiddle, a.x, z.x); z.y = fmaf(kMiddle, a.y, z.y); z.z = fmaf(kMiddle, a.z, z.z); z.w = fmaf(kMiddle, a.w, z.w);
            }
            const float4 y = WIDE ? v.q_zero[zero_quad(i, v.gid)] : v.qz[i];
            z0 = fmaf(y.x, z.x, z0); z1 = fmaf(y.y, z.y, z1);
            z0 = fmaf(y.z, z.z, z0); z1 = fmaf(y.w, z.w, z1);
        }
        qz[g] = z0 + z1;
    }
#pragma unroll
    for (int off = 4; off <= 16; off *= 2)
#pragma unroll
        for (int g = 0; g < NG; ++g) qz[g] += __shfl_xor_sync(0xffffffffu, qz[g], off);
    __syncwarp();                                           // the scratch is free
    float largest = top[0][0];
#pragma unroll
    for (int g = 0; g < NG; ++g) largest = max3_abs_nan(top[g][0], top[g][1], max3_abs_nan(top[g][2], top[g][3], largest));
    if (!(largest <= 3.0e38f)) {
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i) sts32(v.scratch + h * 512 + 4 * k_channel(v.lane, i), v.qk[i][h]);
        __syncwarp();
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const float4 r = scores_plain(kc + 1024 * g, ks + 128 * g, kz + 128 * g, reinterpret_cast<const float4*>(scratch) + 32 * v.tig, v.gid);
            s[g][0] = r.x; s[g][1] = r.y; s[g][2] = r.z; s[g][3] = r.w;
            if constexpr (WIDE) {
#pragma unroll
                for (int n = 0; n < 4; ++n) fine[g][n] = 0.0f;
            }
        }
        return;
    }
    if constexpr (WIDE) {                                   // (the products are made again from here on: 32 of them would not stay in registers)
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int i = 0; i < 4; ++i) asm volatile("" : "+f"(sv[g][i]));
    }
    float unit[NG];
    constexpr int kBlocks = WIDE ? 3 : 2;                   // column blocks: digits 0,1 / 2,const / rest 0,1
    constexpr int kDigits = 2 * kBlocks - 1;
    int c[WIDE ? 1 : NG][2][kBlocks][4];                    // [rows of codes 0,1 / 2,3 and up]
    int sum[kBlocks][4];                                    // WIDE: every row the sum of the digits
    auto read_scores = [&](int g) {
        const int cg = WIDE ? 0 : g;
        float below = 0.0f, y[5][kDigits], all[kDigits];    // digits (the biased ones less the constant) of the sums "code n and up"
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const int t = n >> 1, r = 2 * (n & 1);
            y[n][0] = __int_as_float(c[cg][t][0][r]); y[n][1] = __int_as_float(c[cg][t][0][r + 1]);
            y[n][2] = __int_as_float(c[cg][t][1][r]) - __int_as_float(c[cg][t][1][r + 1]);
            if constexpr (WIDE) {
                y[n][3] = __int_as_float(c[cg][t][2][r]);
                y[n][4] = __int_as_float(c[cg][t][2][r + 1]) - __int_as_float(c[cg][t][1][r + 1]);
            }
        }
        y[4][0] = kTwo23; y[4][1] = kTwo23; y[4][2] = 0.0f;
        if constexpr (WIDE) {
            y[4][3] = kTwo23; y[4][4] = 0.0f;
            all[0] = __int_as_float(sum[0][0]) - kTwo23; all[1] = __int_as_float(sum[0][1]) - kTwo23;
            all[2] = __int_as_float(sum[1][0]) - __int_as_float(sum[1][1]);
            all[3] = __int_as_float(sum[2][0]) - kTwo23; all[4] = __int_as_float(sum[2][1]) - __int_as_float(sum[1][1]);
            below = fmaf(fmaf(all[4], 256.0f, all[3]), 0x1p-15f, all[0]);
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const float row = n == 0 ? 1.0f : n == 1 ? kRow1 : n == 2 ? kRow2 : kRow3;
            float d[kDigits];
#pragma unroll
            for (int i = 0; i < kDigits; ++i) d[i] = y[n][i] - y[n + 1][i];
            if constexpr (WIDE) {
                const float off = -kMiddle / row;
                s[g][n] = fmaf(all[2], off, d[2]) * (65536.0f * row) * unit[g];
                const float low = fmaf(below, off, fmaf(fmaf(d[4], 256.0f, d[3]), 0x1p-15f, d[0]));
                fine[g][n] = fmaf(fmaf(fmaf(all[1], off, d[1]), 256.0f, low), unit[g] * row, qz[g]);
            } else {
                s[g][n] = fmaf(fmaf(d[2], 65536.0f, fmaf(d[1], 256.0f, d[0])), unit[g] * row, qz[g]);
            }
        }
    };
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        if (g > 0) __syncwarp();                            // the operand of the group before has been read
        float F[4];
#pragma unroll
        for (int h = 0; h < 4; ++h)                          // (WIDE: a power of two, so that unit = 1 / F exactly)
            F[h] = __uint_as_float(WIDE ? kInverseK - (1u << 23) - (__float_as_uint(top[g][h]) & kExponent) : kInverseK - __float_as_uint(top[g][h]));
        const float own = v.tig == 0 ? F[0] : v.tig == 1 ? F[1] : v.tig == 2 ? F[2] : F[3];
        unit[g] = WIDE ? __uint_as_float((254u << 23) - __float_as_uint(own)) : rcp_approx(own);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            uint32_t x[2][4], rest[2][4];
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int i = 2 * k + e;
                    if constexpr (WIDE) {
                        const float y = v.qk[i][h] * sv[g][i], t = fmaf(y, F[h], kMagicK);
                        x[k][h] = __float_as_uint(t);
                        rest[k][h] = __float_as_uint(fmaf(fmaf(y, F[h], kMagicK - t), 32768.0f, kMagicRest));
                    } else {
                        x[k][h] = __float_as_uint(fmaf(w[g][i][h], F[h], kMagicK));
                    }
                }
            // columns: digits 0 and 1 of the four heads; digit 2 and the constant
            sts128(v.scratch + 512 * e + 16 * v.lane, __byte_perm(x[0][0], x[0][1], 0x5410), __byte_perm(x[0][2], x[0][3], 0x5410),
                   __byte_perm(x[1][0], x[1][1], 0x5410), __byte_perm(x[1][2], x[1][3], 0x5410));
            sts128(v.scratch + 1024 + 512 * e + 16 * v.lane, __byte_perm(x[0][0], x[0][1], 0x7632), __byte_perm(x[0][2], x[0][3], 0x7632),
                   __byte_perm(x[1][0], x[1][1], 0x7632), __byte_perm(x[1][2], x[1][3], 0x7632));
            if constexpr (WIDE)
                sts128(spare + 1024 * g + 512 * e + 16 * v.lane, __byte_perm(rest[0][0], rest[0][1], 0x5410), __byte_perm(rest[0][2], rest[0][3], 0x5410),
                       __byte_perm(rest[1][0], rest[1][1], 0x5410), __byte_perm(rest[1][2], rest[1][3], 0x5410));
        }
        __syncwarp();
        uint32_t b[4][4], br[2][4];                         // step j: both halves of columns 0-7, of columns 8-15; steps 2j, 2j+1 of the rest
        if constexpr (!WIDE) {                              // (WIDE has no registers to spare for all of them)
#pragma unroll
            for (int j = 0; j < 4; ++j) ldmatrix_t8(b[j], v.k_rows + 128 * j);
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint4 wv = *reinterpret_cast<const uint4*>(kc + 1024 * g + half * 512 + v.gid * 64 + v.tig * 16);
            const uint32_t cw[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int m = 0; m < 4; m += 2) {
                const int j = 2 * half + m / 2, cg = WIDE ? 0 : g;
                const uint32_t wa = cw[m + (j & 1)], wb = cw[m + 1 - (j & 1)];
                if constexpr (WIDE) {
                    ldmatrix_t8(b[j], v.k_rows + 128 * j);
                    if (m == 0) ldmatrix_t8(br[half], spare + 1024 * g + v.rest_rows + 256 * half);
                }
#pragma unroll
                for (int d = 0; d < kBlocks; ++d) {
                    const uint32_t b0 = d < 2 ? b[j][2 * d] : br[half][m], b1 = d < 2 ? b[j][2 * d + 1] : br[half][m + 1];
                    if (j == 0) {
                        mma_u8_from(v.start, c[cg][0][d], wa, wa & kFrom1, wb, wb & kFrom1, b0, b1);
                        mma_u8_from(v.start, c[cg][1][d], wa & kFrom2, wa & kFrom3, wb & kFrom2, wb & kFrom3, b0, b1);
                        if constexpr (WIDE) mma_u8_from(v.start, sum[d], v.ones[0], v.ones[1], v.ones[2], v.ones[3], b0, b1);
                    } else {
                        mma_u8(c[cg][0][d], wa, wa & kFrom1, wb, wb & kFrom1, b0, b1);
                        mma_u8(c[cg][1][d], wa & kFrom2, wa & kFrom3, wb & kFrom2, wb & kFrom3, b0, b1);
                        if constexpr (WIDE) mma_u8(sum[d], v.ones[0], v.ones[1], v.ones[2], v.ones[3], b0, b1);
                    }
                }
            }
        }
        if constexpr (WIDE) read_scores(g);                 // (registers: one group's accumulators at a time)
    }
    if constexpr (!WIDE) {
#pragma unroll
        for (int g = 0; g < NG; ++g) read_scores(g);
    }
}

// running max / sum update for NG groups at once; turns scores into weights
template <int NG, bool WIDE>
__device__ __forceinline__ void softmax_phase(float (&s)[NG][4], const float (&fine)[NG][4], WarpState& st) {
    float gmax = -INFINITY;
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) gmax = fmaxf(gmax, WIDE ? s[g][e] + fine[g][e] : s[g][e]);
    if (__any_sync(0xffffffffu, gmax > st.m + kGrowth)) {
        gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 4));
        gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 8));
        gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 16));
        const float m_new = fmaxf(st.m, gmax);
        const float alpha = ex2(st.m - m_new);         // 0 when st.m == -inf
        st.m = m_new;
        st.l *= alpha;
#pragma unroll
        for (int mt = 0; mt < 8; ++mt) { st.o[mt][0] *= alpha; st.o[mt][1] *= alpha; }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const float alpha_h = __shfl_sync(0xffffffffu, alpha, h);
#pragma unroll
            for (int gd = 0; gd < 4; ++gd) st.oz[h][gd] *= alpha_h;
        }
    }
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) { s[g][e] = ex2(WIDE ? (s[g][e] - st.m) + fine[g][e] : s[g][e] - st.m); st.l += s[g][e]; }
}

// p.v of NG groups; p[g][n] = weight of token 4*gid + n of group g for head tig.
// The weights first change hands: a lane comes to hold the four heads of the token whose
// scales are row `lane` of the group, multiplies them with the four scales, and the digits
// go out as rows of 16 bytes -- one per token and pair of channel groups, columns
// [channel group][head][digit] -- that ldmatrix_t8 hands back as tensor-core operands.
// Value block words (kivi_common.cuh): word (gd, kappa, r, c) holds natural byte
// 8*gd + r (channels 32*gd + 4*r + i) of tokens 16*kappa + 4*c + n in bytes n: four
// consecutive contraction indices, as the tensor core wants them.
template <int NG, bool WIDE>
__device__ __forceinline__ void pv_phase(const uint8_t* __restrict__ vc, const float* __restrict__ vs, const float* __restrict__ vz,
                                         const float (&p)[NG][4], const LaneView& v, uint8_t* scratch, uint32_t spare, WarpState& st) {
    __syncwarp();                                           // the scratch is free
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        sts32(v.p_even + 512 * g, p[g][0]); sts32(v.p_even + 512 * g + 128, p[g][2]);
        sts32(v.p_odd + 512 * g, p[g][1]); sts32(v.p_odd + 512 * g + 128, p[g][3]);
    }
    __syncwarp();
    float ph[NG][4], sv[NG][4];                             // weights [head], scales [channel group] of the lane's token
    uint32_t p_bits = 0u, s_bits = 0u;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const float4 p4 = lds128(v.p_read + 512 * g);
        const float4 s4 = *reinterpret_cast<const float4*>(vs + g * 128 + 4 * v.lane);
        ph[g][0] = p4.x; ph[g][1] = p4.y; ph[g][2] = p4.z; ph[g][3] = p4.w;
        sv[g][0] = s4.x; sv[g][1] = s4.y; sv[g][2] = s4.z; sv[g][3] = s4.w;
#pragma unroll
        for (int i = 0; i < 4; ++i) { p_bits = max(p_bits, __float_as_uint(ph[g][i])); s_bits = max(s_bits, __float_as_uint(sv[g][i])); }
    }
    // as integers, the bits of negative numbers, infinities and NaN all lie above those of a finite one
    if (__any_sync(0xffffffffu, p_bits >= kExponent || s_bits >= kLargestScale)) {
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int gd = 0; gd < 4; ++gd) {
                const float4 r = weighted_plain<false>(vc + g * 1024, vs + g * 128, vz + g * 128, reinterpret_cast<const float*>(scratch + 512 * g), gd, v.gid, v.tig);
                st.o[2 * gd][0] += r.x; st.o[2 * gd][1] += 4.0f * r.y;
                st.o[2 * gd + 1][0] += 16.0f * r.z; st.o[2 * gd + 1][1] += 64.0f * r.w;
            }
        return;
    }
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        float4 z4 = *reinterpret_cast<const float4*>(vz + g * 128 + 4 * v.lane);
        if constexpr (WIDE) {
            z4.x = fmaf(kMiddle, sv[g][0], z4.x); z4.y = fmaf(kMiddle, sv[g][1], z4.y);
            z4.z = fmaf(kMiddle, sv[g][2], z4.z); z4.w = fmaf(kMiddle, sv[g][3], z4.w);
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            st.oz[h][0] = fmaf(ph[g][h], z4.x, st.oz[h][0]); st.oz[h][1] = fmaf(ph[g][h], z4.y, st.oz[h][1]);
            st.oz[h][2] = fmaf(ph[g][h], z4.z, st.oz[h][2]); st.oz[h][3] = fmaf(ph[g][h], z4.w, st.oz[h][3]);
        }
    }
    // the products of a channel group and the largest of each head, one group ahead of their use
    float w[2][NG][4], unit[4];
    uint32_t top[2][4];
    auto weigh = [&](int gd) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            uint32_t t = kSmallestBits;
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                w[gd & 1][g][h] = ph[g][h] * sv[g][gd];
                t = max(t, __float_as_uint(w[gd & 1][g][h]));
            }
            top[gd & 1][h] = warp_max_u32(t);
        }
    };
    weigh(0);
    __syncwarp();                                           // every lane has read its weights
    // Rows of 16 bytes per channel group and contraction index k = 4*c + n: the columns
    // [head][digit] of tokens 16*0 + k and 16*1 + k, in the other order for k >= 8 (the writes
    // of a half-warp then touch every bank once; the codes are read in that order too).
#pragma unroll
    for (int gd = 0; gd < 4; ++gd) {
        if (gd < 3) weigh(gd + 1);
        float F[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) F[h] = __uint_as_float((WIDE ? kInverseVWide : kInverseV) - top[gd & 1][h]);
        const float own = v.tig == 0 ? F[0] : v.tig == 1 ? F[1] : v.tig == 2 ? F[2] : F[3];
        unit[gd] = rcp_approx(own);
        if constexpr (WIDE) unit[gd] = fmaf(unit[gd], fmaf(-own, unit[gd], 1.0f), unit[gd]);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            uint32_t x[4];
            if constexpr (WIDE) {                           // below the 23 bits eight more: the rest of a number rounded down
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const float y = w[gd & 1][g][h], t = __fmaf_rz(y, F[h], kTwo23), r = fmaf(fmaf(y, F[h], kTwo23 - t), kRestV, kTwo23);
                    x[h] = __byte_perm(__float_as_uint(r), __float_as_uint(t), 0x6540);
                }
                const uint32_t row = (g == 0 ? v.v_write : v.v_write - v.scratch + spare) + 512 * gd;
                sts64(row, __byte_perm(x[0], x[1], 0x5410), __byte_perm(x[2], x[3], 0x5410));
                sts64(row + 256, __byte_perm(x[0], x[1], 0x7632), __byte_perm(x[2], x[3], 0x7632));
            } else {
#pragma unroll
                for (int h = 0; h < 4; ++h) x[h] = __float_as_uint(fmaf(w[gd & 1][g][h], F[h], kTwo23));
                sts64(v.v_write + 1024 * g + 256 * gd, __byte_perm(x[0], x[1], 0x5410), __byte_perm(x[2], x[3], 0x5410));
            }
        }
    }
    __syncwarp();
    if constexpr (WIDE) {
#pragma unroll
        for (int gd = 0; gd < 4; ++gd) {
            int acc[2][2][4], sum[2][4];                    // [rows of codes 0,1 / 2,3 and up][digits 0,1 / 2,3]; sums of the digits
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                const uint32_t* vw = reinterpret_cast<const uint32_t*>(vc + g * 1024) + v.lane;
                uint32_t b[4];
                ldmatrix_t8(b, (g == 0 ? v.v_rows : v.v_rows - v.scratch + spare) + 512 * gd);
                const uint32_t w0 = vw[gd * 64 + v.v_first], w1 = vw[gd * 64 + (v.v_first ^ 32)];
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    if (g == 0) {
                        mma_u8_from(v.start, acc[0][d], w0, w0 & kFrom1, w1, w1 & kFrom1, b[2 * d], b[2 * d + 1]);
                        mma_u8_from(v.start, acc[1][d], w0 & kFrom2, w0 & kFrom3, w1 & kFrom2, w1 & kFrom3, b[2 * d], b[2 * d + 1]);
                        mma_u8_from(v.start, sum[d], v.ones[0], v.ones[1], v.ones[2], v.ones[3], b[2 * d], b[2 * d + 1]);
                    } else {
                        mma_u8(acc[0][d], w0, w0 & kFrom1, w1, w1 & kFrom1, b[2 * d], b[2 * d + 1]);
                        mma_u8(acc[1][d], w0 & kFrom2, w0 & kFrom3, w1 & kFrom2, w1 & kFrom3, b[2 * d], b[2 * d + 1]);
                        mma_u8(sum[d], v.ones[0], v.ones[1], v.ones[2], v.ones[3], b[2 * d], b[2 * d + 1]);
                    }
                }
            }
            float all[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) all[k] = __int_as_float(sum[k >> 1][k & 1]) - kTwo23;
            const float below = fmaf(all[2], 256.0f, fmaf(all[0], 1.0f / kRestV, all[1]));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int mt = i >> 1, r = 2 * (i & 1), mt1 = i < 3 ? (i + 1) >> 1 : 0, r1 = 2 * ((i + 1) & 1);
                const float off = i == 0 ? -kMiddle : i == 1 ? -4.0f * kMiddle : i == 2 ? -16.0f * kMiddle : -64.0f * kMiddle;
                float d[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    d[k] = __int_as_float(acc[mt][k >> 1][r + (k & 1)]) - (i < 3 ? __int_as_float(acc[mt1][k >> 1][r1 + (k & 1)]) : kTwo23);
                const float low = fmaf(below, off, fmaf(d[2], 256.0f, fmaf(d[0], 1.0f / kRestV, d[1])));
                float& o = st.o[2 * gd + mt][i & 1];
                o = fmaf(fmaf(fmaf(all[3], off, d[3]), 65536.0f, low), unit[gd], o);
            }
        }
        return;
    }
    int acc[8][4];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const uint32_t* vw = reinterpret_cast<const uint32_t*>(vc + g * 1024) + v.lane;
#pragma unroll
        for (int gp = 0; gp < 2; ++gp) {
            uint32_t b[4];
            ldmatrix_t8(b, v.v_rows + 1024 * g + 512 * gp);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int gd = 2 * gp + e;
                const uint32_t w0 = vw[gd * 64 + v.v_first], w1 = vw[gd * 64 + (v.v_first ^ 32)];
                if (g == 0) {
                    mma_u8_from(v.start, acc[2 * gd], w0, w0 & kFrom1, w1, w1 & kFrom1, b[2 * e], b[2 * e + 1]);
                    mma_u8_from(v.start, acc[2 * gd + 1], w0 & kFrom2, w0 & kFrom3, w1 & kFrom2, w1 & kFrom3, b[2 * e], b[2 * e + 1]);
                } else {
                    mma_u8(acc[2 * gd], w0, w0 & kFrom1, w1, w1 & kFrom1, b[2 * e], b[2 * e + 1]);
                    mma_u8(acc[2 * gd + 1], w0 & kFrom2, w0 & kFrom3, w1 & kFrom2, w1 & kFrom3, b[2 * e], b[2 * e + 1]);
                }
            }
        }
    }
#pragma unroll
    for (int gd = 0; gd < 4; ++gd)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int mt = 2 * gd + (i >> 1), r = 2 * (i & 1), mt1 = 2 * gd + ((i + 1) >> 1), r1 = 2 * ((i + 1) & 1);
            const float n0 = i < 3 ? __int_as_float(acc[i < 3 ? mt1 : 0][r1]) : kTwo23, n1 = i < 3 ? __int_as_float(acc[i < 3 ? mt1 : 0][r1 + 1]) : kTwo23;
            const float d0 = __int_as_float(acc[mt][r]) - n0, d1 = __int_as_float(acc[mt][r + 1]) - n1;
            st.o[mt][i & 1] = fmaf(fmaf(d1, 256.0f, d0), unit[gd], st.o[mt][i & 1]);
        }
}

// NG consecutive token groups of one pipeline stage: the softmax update and the reading of
// the p.v accumulators are done once for all NG*32 tokens.
template <int NG, bool WIDE>
__device__ __forceinline__ void process_groups(const uint8_t* __restrict__ sb, const LaneView& v, uint8_t* scratch, WarpState& st) {
    float s[NG][4], fine[NG][4];
    const uint32_t spare = WIDE ? smem_u32(sb + kGPS * 1024) : 0u;
    qk_phase<NG, WIDE>(sb, reinterpret_cast<const float*>(sb + kGPS * 1024), reinterpret_cast<const float*>(sb + kGPS * 1536), v, scratch, spare, s, fine);
    softmax_phase<NG, WIDE>(s, fine, st);
    pv_phase<NG, WIDE>(sb + kGPS * 2048, reinterpret_cast<const float*>(sb + kGPS * 3072), reinterpret_cast<const float*>(sb + kGPS * 3584), s, v, scratch, spare, st);
    // what was written over the stage comes before the copy that fills it again
    if constexpr (WIDE) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- one query head per KV head ------------------------------------------------------
// With one head the columns that four would take hold other things instead: in q.k the two
// groups of the stage (one operand for both, each lane reading the accumulators of its
// group), in p.v the four channel groups (their contractions go to one accumulator, each
// with the columns of the others at zero).  A quarter of the operand work, half of the
// reading of accumulators.  256 units x 4k tokens 40.0 -> 32.8 us with the form for four
// heads before, 512 x 8k 121 (fp16 form) -> 97, 32 x 8k 14.5 -> 11.7.
struct OneView {
    int gid, tig, lane;
    float qk[4];           // pre-scaled query, channel k_channel(lane, i)
    float4 qz[4];          // channels 4 * zero_quad_one(i, gid, tig) .. + 3
    uint32_t scratch, k_rows, v_rows, p_write, v_write;
    int v_first;
    int start[4];
};
struct OneState {
    float m, l;            // running max; sum over the lane's tokens
    float o[4];            // channel 32*tig + 4*gid + i, times 4^i
    float oz[4];           // zero-point term [channel group] of the tokens this lane weighs
};
// Zero term: lane (gid, tig) takes group tig; odd and even tig are two quads apart (bank conflicts).
__device__ __forceinline__ int zero_quad_one(int i, int gid, int tig) { return 4 * gid + ((i + ((gid >> 1) & 1) + 2 * (tig & 1)) & 3); }

// scores of the lane's tokens 4*gid + n of group tig (lanes with tig >= NG: -inf)
template <int NG>
__device__ __forceinline__ void qk_one(const uint8_t* __restrict__ kc, const float* __restrict__ ks, const float* __restrict__ kz,
                                       const OneView& v, uint8_t* scratch, float (&s)[4]) {
    float w[2][4], top[2];                                  // top: largest |q * s| of a group of tokens
#pragma unroll
    for (int g = 0; g < 2; ++g) {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[g][i] = 0.0f;
        top[g] = kSmallest;
        if (g < NG) {
            const float2 sa = *reinterpret_cast<const float2*>(ks + 128 * g + k_channel(v.lane, 0)), sb = *reinterpret_cast<const float2*>(ks + 128 * g + k_channel(v.lane, 2));
            w[g][0] = v.qk[0] * sa.x; w[g][1] = v.qk[1] * sa.y; w[g][2] = v.qk[2] * sb.x; w[g][3] = v.qk[3] * sb.y;
            top[g] = warp_max_abs_nan(max3_abs_nan(w[g][2], w[g][3], max3_abs_nan(w[g][0], w[g][1], kSmallest)));
        }
    }
    const int mine = v.tig < NG ? v.tig : 0;
    float z0 = 0.0f, z1 = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 z = *reinterpret_cast<const float4*>(kz + 128 * mine + 4 * zero_quad_one(i, v.gid, v.tig));
        z0 = fmaf(v.qz[i].x, z.x, z0); z1 = fmaf(v.qz[i].y, z.y, z1);
        z0 = fmaf(v.qz[i].z, z.z, z0); z1 = fmaf(v.qz[i].w, z.w, z1);
    }
    float qz = z0 + z1;
#pragma unroll
    for (int off = 4; off <= 16; off *= 2) qz += __shfl_xor_sync(0xffffffffu, qz, off);
    __syncwarp();                                           // the scratch is free
    if (!(top[0] + top[1] <= 3.0e38f)) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sts32(v.scratch + 4 * k_channel(v.lane, i), v.qk[i]);
        __syncwarp();
        const float4 r = scores_plain(kc + 1024 * mine, ks + 128 * mine, kz + 128 * mine, reinterpret_cast<const float4*>(scratch), v.gid);
        s[0] = r.x; s[1] = r.y; s[2] = r.z; s[3] = r.w;
    } else {
        const float F[2] = {__uint_as_float(kInverseK - __float_as_uint(top[0])), __uint_as_float(kInverseK - __float_as_uint(top[1]))};
        const float unit = rcp_approx(mine ? F[1] : F[0]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            uint32_t x[2][2];
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int g = 0; g < 2; ++g) x[k][g] = __float_as_uint(fmaf(w[g][2 * k + e], F[g], kMagicK));
            // columns: digits 0 and 1 of the two groups; digit 2 and the constant
            sts128(v.scratch + 512 * e + 16 * v.lane, __byte_perm(x[0][0], x[0][1], 0x5410), 0u, __byte_perm(x[1][0], x[1][1], 0x5410), 0u);
            sts128(v.scratch + 1024 + 512 * e + 16 * v.lane, __byte_perm(x[0][0], x[0][1], 0x7632), 0u, __byte_perm(x[1][0], x[1][1], 0x7632), 0u);
        }
        __syncwarp();
        uint32_t b[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) ldmatrix_t8(b[j], v.k_rows + 128 * j);
        int c[NG][2][2][4];
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint4 wv = *reinterpret_cast<const uint4*>(kc + 1024 * g + (j >> 1) * 512 + v.gid * 64 + v.tig * 16);
                const uint32_t wa = j & 1 ? wv.w : wv.x, wb = j & 1 ? wv.z : wv.y;
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    if (j == 0) {
                        mma_u8_from(v.start, c[g][0][d], wa, wa & kFrom1, wb, wb & kFrom1, b[j][2 * d], b[j][2 * d + 1]);
                        mma_u8_from(v.start, c[g][1][d], wa & kFrom2, wa & kFrom3, wb & kFrom2, wb & kFrom3, b[j][2 * d], b[j][2 * d + 1]);
                    } else {
                        mma_u8(c[g][0][d], wa, wa & kFrom1, wb, wb & kFrom1, b[j][2 * d], b[j][2 * d + 1]);
                        mma_u8(c[g][1][d], wa & kFrom2, wa & kFrom3, wb & kFrom2, wb & kFrom3, b[j][2 * d], b[j][2 * d + 1]);
                    }
                }
            }
        float y[5][3];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const int t = n >> 1, r = 2 * (n & 1);
            auto pick = [&](int d, int k) { return __int_as_float(NG == 2 && (v.tig & 1) ? c[NG - 1][t][d][r + k] : c[0][t][d][r + k]); };
            y[n][0] = pick(0, 0); y[n][1] = pick(0, 1); y[n][2] = pick(1, 0) - pick(1, 1);
        }
        y[4][0] = kTwo23; y[4][1] = kTwo23; y[4][2] = 0.0f;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const float row = n == 0 ? 1.0f : n == 1 ? kRow1 : n == 2 ? kRow2 : kRow3;
            s[n] = fmaf(fmaf(y[n][2] - y[n + 1][2], 65536.0f, fmaf(y[n][1] - y[n + 1][1], 256.0f, y[n][0] - y[n + 1][0])), unit * row, qz);
        }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) s[n] = v.tig < NG ? s[n] : -INFINITY;
}

__device__ __forceinline__ void softmax_one(float (&s)[4], OneState& st) {
    float gmax = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
    if (__any_sync(0xffffffffu, gmax > st.m + kGrowth)) {
#pragma unroll
        for (int off = 1; off <= 16; off *= 2) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, off));
        const float m_new = fmaxf(st.m, gmax);
        const float alpha = ex2(st.m - m_new);         // 0 when st.m == -inf
        st.m = m_new;
        st.l *= alpha;
#pragma unroll
        for (int i = 0; i < 4; ++i) { st.o[i] *= alpha; st.oz[i] *= alpha; }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) { s[n] = ex2(s[n] - st.m); st.l += s[n]; }
}

template <int NG>
__device__ __forceinline__ void pv_one(const uint8_t* __restrict__ vc, const float* __restrict__ vs, const float* __restrict__ vz,
                                       const float (&p)[4], const OneView& v, uint8_t* scratch, OneState& st) {
    __syncwarp();                                           // the scratch is free
    if (v.tig < NG) {
#pragma unroll
        for (int n = 0; n < 4; ++n) sts32(v.p_write + 16 * n, p[n]);
    }
    __syncwarp();
    float ph[NG], sv[NG][4];
    uint32_t top[4] = {kSmallestBits, kSmallestBits, kSmallestBits, kSmallestBits};      // largest p * s of a channel group
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        ph[g] = lds32(v.scratch + 128 * g + 4 * v.lane);
        const float4 s4 = *reinterpret_cast<const float4*>(vs + g * 128 + 4 * v.lane);
        sv[g][0] = s4.x; sv[g][1] = s4.y; sv[g][2] = s4.z; sv[g][3] = s4.w;
#pragma unroll
        for (int gd = 0; gd < 4; ++gd) top[gd] = max(top[gd], __float_as_uint(ph[g] * sv[g][gd]));
    }
#pragma unroll
    for (int gd = 0; gd < 4; ++gd) top[gd] = warp_max_u32(top[gd]);
    if (max(max(top[0], top[1]), max(top[2], top[3])) >= kExponent) {
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const float4 r = weighted_plain<true>(vc + g * 1024, vs + g * 128, vz + g * 128, reinterpret_cast<const float*>(scratch + 128 * g), v.tig, v.gid, 0);
            st.o[0] += r.x; st.o[1] += 4.0f * r.y; st.o[2] += 16.0f * r.z; st.o[3] += 64.0f * r.w;
        }
        return;
    }
    float F[4];
#pragma unroll
    for (int gd = 0; gd < 4; ++gd) F[gd] = __uint_as_float(kInverseV - top[gd]);
    const float unit = rcp_approx(v.tig == 0 ? F[0] : v.tig == 1 ? F[1] : v.tig == 2 ? F[2] : F[3]);       // (the lane's columns are of group tig)
    __syncwarp();                                           // every lane has read its weights
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const float4 z4 = *reinterpret_cast<const float4*>(vz + g * 128 + 4 * v.lane);
        st.oz[0] = fmaf(ph[g], z4.x, st.oz[0]); st.oz[1] = fmaf(ph[g], z4.y, st.oz[1]);
        st.oz[2] = fmaf(ph[g], z4.z, st.oz[2]); st.oz[3] = fmaf(ph[g], z4.w, st.oz[3]);
        uint32_t x[4];
#pragma unroll
        for (int gd = 0; gd < 4; ++gd) x[gd] = __float_as_uint(fmaf(ph[g] * sv[g][gd], F[gd], kTwo23));
        sts64(v.v_write + 256 * g, __byte_perm(x[0], x[1], 0x5410), __byte_perm(x[2], x[3], 0x5410));       // columns [channel group][digit]
    }
    __syncwarp();
    uint32_t b[4];
    ldmatrix_t8(b, v.v_rows);                               // one matrix per group
    int acc[2][4];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const uint32_t* vw = reinterpret_cast<const uint32_t*>(vc + g * 1024) + v.lane;
#pragma unroll
        for (int gd = 0; gd < 4; ++gd) {
            const uint32_t w0 = vw[gd * 64 + v.v_first], w1 = vw[gd * 64 + (v.v_first ^ 32)];
            const bool own = (v.gid >> 1) == gd;             // the lane's column is of this channel group
            const uint32_t b0 = own ? b[2 * g] : 0u, b1 = own ? b[2 * g + 1] : 0u;
            if (g == 0 && gd == 0) {
                mma_u8_from(v.start, acc[0], w0, w0 & kFrom1, w1, w1 & kFrom1, b0, b1);
                mma_u8_from(v.start, acc[1], w0 & kFrom2, w0 & kFrom3, w1 & kFrom2, w1 & kFrom3, b0, b1);
            } else {
                mma_u8(acc[0], w0, w0 & kFrom1, w1, w1 & kFrom1, b0, b1);
                mma_u8(acc[1], w0 & kFrom2, w0 & kFrom3, w1 & kFrom2, w1 & kFrom3, b0, b1);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = i >> 1, r = 2 * (i & 1), t1 = i < 3 ? (i + 1) >> 1 : 0, r1 = 2 * ((i + 1) & 1);
        const float d0 = __int_as_float(acc[t][r]) - (i < 3 ? __int_as_float(acc[t1][r1]) : kTwo23);
        const float d1 = __int_as_float(acc[t][r + 1]) - (i < 3 ? __int_as_float(acc[t1][r1 + 1]) : kTwo23);
        st.o[i] = fmaf(fmaf(d1, 256.0f, d0), unit, st.o[i]);
    }
}

template <int NG, bool>
__device__ __forceinline__ void process_groups(const uint8_t* __restrict__ sb, const OneView& v, uint8_t* scratch, OneState& st) {
    float s[4];
    qk_one<NG>(sb, reinterpret_cast<const float*>(sb + kGPS * 1024), reinterpret_cast<const float*>(sb + kGPS * 1536), v, scratch, s);
    softmax_one(s, st);
    pv_one<NG>(sb + kGPS * 2048, reinterpret_cast<const float*>(sb + kGPS * 3072), reinterpret_cast<const float*>(sb + kGPS * 3584), s, v, scratch, st);
}

__device__ __forceinline__ void clear(WarpState& st) {
    st.m = -INFINITY; st.l = 0.0f;
#pragma unroll
    for (int t = 0; t < 8; ++t) { st.o[t][0] = 0.0f; st.o[t][1] = 0.0f; }
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int gd = 0; gd < 4; ++gd) st.oz[h][gd] = 0.0f;
}
__device__ __forceinline__ void clear(OneState& st) {
    st.m = -INFINITY; st.l = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) { st.o[i] = 0.0f; st.oz[i] = 0.0f; }
}

// ---- residual ring: full-precision tokens ---------------------------------------
// CTA `rs` of the residual part handles window tokens [rs*chunk, (rs+1)*chunk).
// A warp takes 32 tokens at a time: lane = (4 tokens, quarter of the channels)
// for q.k (vector loads of 32 channels, 2 shuffles to finish the dot products),
// then lane = 4 channels for p.v.  Result: per warp (m, l, o) for 4 heads, merged
// through shared memory like the quantized splits.
template <typename T> struct RowVec;
template <> struct RowVec<float> {
    __device__ static void load8(const float* p, float (&v)[8]) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    __device__ static void load4(const float* p, float (&v)[4]) {
        const float4 a = *reinterpret_cast<const float4*>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    }
};
template <> struct RowVec<__nv_bfloat16> {
    __device__ static void load8(const __nv_bfloat16* p, float (&v)[8]) {
        const uint4 t = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    }
    __device__ static void load4(const __nv_bfloat16* p, float (&v)[4]) {
        const uint2 t = *reinterpret_cast<const uint2*>(p);
        v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xffff0000u);
        v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xffff0000u);
    }
};

// The queries a lane holds, pre-scaled.  All loads are issued before the first is used
// (absent heads read the last one's again and count as zero): one trip to memory, where a
// branch around each load made twelve (3 us of a CTA's start).
template <typename T>
__device__ __forceinline__ void load_queries(const T* __restrict__ q, int n_heads, float scale_log2, LaneView& v) {
    float a[4][4], b[4][4], z[4][4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const T* row = q + (h < n_heads ? h : n_heads - 1) * kD;
        RowVec<T>::load4(row + (k_channel(v.lane, 0) & ~3), a[h]);
        RowVec<T>::load4(row + (k_channel(v.lane, 2) & ~3), b[h]);
        RowVec<T>::load4(q + (v.tig < n_heads ? v.tig : n_heads - 1) * kD + 4 * zero_quad(h, v.gid), z[h]);
    }
    const bool upper = v.lane & 1;                           // channels 2, 3 of a quad
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const float f = h < n_heads ? scale_log2 : 0.0f, fz = v.tig < n_heads ? scale_log2 : 0.0f;
        v.qk[0][h] = h < n_heads ? f * (upper ? a[h][2] : a[h][0]) : 0.0f; v.qk[1][h] = h < n_heads ? f * (upper ? a[h][3] : a[h][1]) : 0.0f;
        v.qk[2][h] = h < n_heads ? f * (upper ? b[h][2] : b[h][0]) : 0.0f; v.qk[3][h] = h < n_heads ? f * (upper ? b[h][3] : b[h][1]) : 0.0f;
        v.qz[h] = v.tig < n_heads ? make_float4(fz * z[h][0], fz * z[h][1], fz * z[h][2], fz * z[h][3]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

template <typename T>
__device__ __forceinline__ void load_queries(const T* __restrict__ q, int, float scale_log2, OneView& v) {
    float a[4], b[4], z[4][4];
    RowVec<T>::load4(q + (k_channel(v.lane, 0) & ~3), a);
    RowVec<T>::load4(q + (k_channel(v.lane, 2) & ~3), b);
#pragma unroll
    for (int i = 0; i < 4; ++i) RowVec<T>::load4(q + 4 * zero_quad_one(i, v.gid, v.tig), z[i]);
    const bool upper = v.lane & 1;
    v.qk[0] = scale_log2 * (upper ? a[2] : a[0]); v.qk[1] = scale_log2 * (upper ? a[3] : a[1]);
    v.qk[2] = scale_log2 * (upper ? b[2] : b[0]); v.qk[3] = scale_log2 * (upper ? b[3] : b[1]);
#pragma unroll
    for (int i = 0; i < 4; ++i) v.qz[i] = make_float4(scale_log2 * z[i][0], scale_log2 * z[i][1], scale_log2 * z[i][2], scale_log2 * z[i][3]);
}

template <typename T>
__device__ __forceinline__ void residual_part(
    const T* __restrict__ k_res, const T* __restrict__ v_res, int R, int res_start, int res_len,
    int t_begin, int t_end, const float* __restrict__ q_s /* [4][128], pre-scaled */,
    int lane, int warp, float (&m)[4], float (&l)[4], float (&o)[4][4]) {
    const int tl = lane >> 2, cq = lane & 3;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        m[h] = -INFINITY; l[h] = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) o[h][i] = 0.0f;
    }
    // a warp pass covers 32 tokens: lane (tl, cq) holds tokens t0 + tl + 8j, j = 0..3,
    // and channels 32*cq .. 32*cq+31 of each; every q vector read feeds 4 tokens
    for (int t0 = t_begin + 32 * warp; t0 < t_end; t0 += 32 * kWarps) {
        float acc[4][4];
        const T* row[4];
        bool valid[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int t = t0 + tl + 8 * j;
            valid[j] = t < t_end;
            int slot = res_start + (valid[j] ? t : t0);              // both below R
            if (slot >= R) slot -= R;
            row[j] = k_res + (int64_t)slot * kD + 32 * cq;
#pragma unroll
            for (int h = 0; h < 4; ++h) acc[j][h] = 0.0f;
        }
#pragma unroll 2
        for (int c = 0; c < 4; ++c) {
            float kv[4][8];
#pragma unroll
            for (int j = 0; j < 4; ++j) RowVec<T>::load8(row[j] + 8 * c, kv[j]);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const float4 qa = *reinterpret_cast<const float4*>(q_s + h * kD + 32 * cq + 8 * c);
                const float4 qb = *reinterpret_cast<const float4*>(q_s + h * kD + 32 * cq + 8 * c + 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float a = acc[j][h];
                    a = fmaf(kv[j][0], qa.x, a); a = fmaf(kv[j][1], qa.y, a);
                    a = fmaf(kv[j][2], qa.z, a); a = fmaf(kv[j][3], qa.w, a);
                    a = fmaf(kv[j][4], qb.x, a); a = fmaf(kv[j][5], qb.y, a);
                    a = fmaf(kv[j][6], qb.z, a); a = fmaf(kv[j][7], qb.w, a);
                    acc[j][h] = a;
                }
            }
        }
        float p[4][4];     // [j][h]
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float sc = acc[j][h];
                sc += __shfl_xor_sync(0xffffffffu, sc, 1);
                sc += __shfl_xor_sync(0xffffffffu, sc, 2);
                acc[j][h] = valid[j] ? sc : -INFINITY;
                mx = fmaxf(mx, acc[j][h]);
            }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            const float m_new = fmaxf(m[h], mx);          // finite: token t0 is always valid
            const float alpha = ex2(m[h] - m_new);
            m[h] = m_new;
            float ps = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) { p[j][h] = valid[j] ? ex2(acc[j][h] - m_new) : 0.0f; ps += p[j][h]; }
            // the four lanes of a token quad hold the same p: count it once
            l[h] = l[h] * alpha + (cq == 0 ? ps : 0.0f);
#pragma unroll
            for (int i = 0; i < 4; ++i) o[h][i] *= alpha;
        }
        const int ntok = t_end - t0 < 32 ? t_end - t0 : 32;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (8 * j >= ntok) break;
            // eight value rows in flight at once; a token past the end re-reads
            // row t0 and carries p = 0
            float vv[8][4];
#pragma unroll
            for (int tk = 0; tk < 8; ++tk) {
                int slot = res_start + t0 + (8 * j + tk < ntok ? 8 * j + tk : 0);
                if (slot >= R) slot -= R;
                RowVec<T>::load4(v_res + (int64_t)slot * kD + 4 * lane, vv[tk]);
            }
#pragma unroll
            for (int tk = 0; tk < 8; ++tk) {
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const float ph = __shfl_sync(0xffffffffu, p[j][h], 4 * tk);
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[h][i] = fmaf(ph, vv[tk][i], o[h][i]);
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], off);
    }
}

// grid = units * head blocks * (nq_splits + n_res_splits) CTAs in one dimension
// (head blocks = ceil(n_rep / 4): a CTA serves up to four query heads); block =
// kWarps warps.  The first units*nq_splits CTAs are the quantized pieces, unit by unit:
// piece i of a unit covers token groups [i*gps, min((i+1)*gps, n_groups)).  The
// units*n_res_splits CTAs of the residual ring come last: they are short, so
// the long CTAs start first and the short ones fill the end of the grid
// (measured against ring CTAs first: 3.5 % faster at batch 64 x 32k, 7 % at
// batch 16 x 4k).  Partial slots: quantized piece i -> i, residual part r ->
// nq_splits + r.
//
// Shared memory: [kWarps][kStages][kStageBytes] stage rings | [kWarps][kScratchBytes]
// (in ring CTAs the first holds the queries, [4][128] fp32 times sm_scale*log2(e), absent
// rows zero) | mbarriers | (max, sum) of the warps.  When a warp is done, its ring doubles
// as the [4][128] buffer its scaled output goes to; the CTA then adds the warps'
// buffers in warp order (deterministic) and writes one partial.
//
// ONE: one query head per KV head.  WIDE: operands long enough for fp32 accuracy.
// FOLD: the CTAs of a unit and head block are a cluster and fold their partials
// themselves (a template, so that the wide grids keep their registers).
template <bool FOLD, bool WIDE, bool ONE>
__global__ void __launch_bounds__(kWarps * 32, 3)
attn_mma_kernel(kivi_layer L, int64_t quant_len, int res_start, int res_len,
                const void* q, int q_dtype,
                float scale_log2, int n_rep, int gps, int nq_splits, int n_res_splits, int res_chunk,
                float* __restrict__ part_o, float* __restrict__ part_ml, ClusterOut direct) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t* stage_mem = smem_raw;                                               // [kWarps][kStages][kStageBytes]
    uint8_t* scratch_mem = smem_raw + kWarps * kStages * kStageBytes;            // [kWarps][kScratchBytes]
    float* q_s = reinterpret_cast<float*>(scratch_mem);                          // [4][128], ring CTAs
    uint64_t* bars = reinterpret_cast<uint64_t*>(scratch_mem + kWarps * kScratchBytes);   // [kWarps][kStages]
    float* ml_s = reinterpret_cast<float*>(bars + kWarps * kStages);             // [kWarps][4][2]
    float* const zero_s = ml_s + kWarps * 4 * 2;                                 // WIDE: [4][128] queries for the zero term

    // With a fold kernel behind this one, its few small blocks may become resident from
    // here on (it waits for this grid's end).  Without (FOLD), what comes next can be
    // another attention call, whose blocks would take places beside this one's while
    // other SMs stay empty: let in before the fold in the cluster (cluster_fold.cuh).
    if constexpr (!FOLD) cudaTriggerProgrammaticLaunchCompletion();
    stream_order();
    q = settled(q);
    settle_layer(L);

    // grid order: all quantized pieces (unit-major), then all residual-ring CTAs --
    // the long CTAs start first, the short ones fill the end
    // With more than four query heads per KV head a unit is served by two CTAs per
    // piece, one per block of four heads (they run side by side, so the second
    // read of the piece mostly comes from L2).
    const int head_blocks = (n_rep + 3) >> 2;
    const int n_quant_ctas = (int)L.num_units * head_blocks * nq_splits;
    // When the partials are folded inside clusters (FOLD), the CTAs of a unit and
    // head block lie side by side instead: pieces, then ring parts.
    const int n_all = nq_splits + n_res_splits;
    const int in_row = (int)blockIdx.x % n_all;
    const bool is_res = FOLD ? in_row >= nq_splits : (int)blockIdx.x >= n_quant_ctas;
    const int rel = is_res ? (int)blockIdx.x - n_quant_ctas : (int)blockIdx.x;
    const int per_unit = is_res ? n_res_splits : nq_splits;
    const int uv = FOLD ? (int)blockIdx.x / n_all : rel / per_unit;
    const int sub = FOLD ? (is_res ? in_row - nq_splits : in_row) : rel - uv * per_unit;
    const int u = uv / head_blocks, head0 = 4 * (uv - u * head_blocks);
    const int n_heads = n_rep - head0 < 4 ? n_rep - head0 : 4;       // heads of this CTA: head0 .. head0 + n_heads - 1
    const int n_splits_total = nq_splits + n_res_splits;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);      // (known to be the same for all lanes)
    const int gid = lane >> 2, tig = lane & 3;
    uint8_t* wstage = stage_mem + warp * kStages * kStageBytes;
    float* fo = reinterpret_cast<float*>(wstage);                               // [4][128] once the ring is idle
    const int slot = is_res ? nq_splits + sub : sub;

    // ---- quantized split: start the copies before anything else ----------------
    const int64_t n_groups = quant_len / kG;
    const int64_t g_begin = is_res ? 0 : (int64_t)slot * gps;
    int64_t g_end = is_res ? 0 : g_begin + gps;
    if (g_end > n_groups) g_end = n_groups;
    const int n_my_groups = (int)(g_end - g_begin);
    const int n_chunks = (n_my_groups + kGPS - 1) / kGPS;
    const int my_n = n_chunks > warp ? (n_chunks - warp + kWarps - 1) / kWarps : 0;
    const uint32_t bar0 = smem_u32(bars + warp * kStages);
    const uint32_t stage0 = smem_u32(wstage);
    // The six pieces of a chunk (key codes, scales, zeros, value codes, scales, zeros) are
    // contiguous runs of 1024 or 512 bytes per token group.  One elected lane issues them
    // from addresses that are the same for the whole warp (a bulk copy takes its operands
    // from uniform registers: six lanes with an address each cost a loop of some 70
    // instructions).  Chunk c of this warp starts at group g_begin + (warp + kWarps*c)*kGPS.
    if (!is_res) {
        if (elect_one()) {
#pragma unroll
            for (int s = 0; s < kStages; ++s) mbar_init(bar0 + 8 * s, 1);
            mbar_init_fence();
        }
        __syncwarp();
    }
    const uint64_t policy = l2_stream_policy();
    const int64_t gw0 = (int64_t)u * (L.max_tokens / kG) + g_begin + (int64_t)warp * kGPS;
    auto issue = [&](int c) {                 // all lanes call it
        const int goff = (warp + kWarps * c) * kGPS;             // groups from g_begin
        const uint32_t ng = (n_my_groups - goff) < kGPS ? (n_my_groups - goff) : kGPS;
        const int s = c % kStages;
        const uint32_t bar = bar0 + 8 * s, dst = stage0 + s * kStageBytes;
        const int64_t g = gw0 + (int64_t)c * (kWarps * kGPS);
        if (elect_one()) {
            mbar_expect_tx(bar, ng * kGroupBytes);
            bulk_g2s(dst, L.k_codes + g * 1024, ng * 1024, bar, policy);
            bulk_g2s(dst + kGPS * 1024, L.k_scales + g * 128, ng * 512, bar, policy);
            bulk_g2s(dst + kGPS * 1536, L.k_zeros + g * 128, ng * 512, bar, policy);
            bulk_g2s(dst + kGPS * 2048, L.v_codes + g * 1024, ng * 1024, bar, policy);
            bulk_g2s(dst + kGPS * 3072, L.v_scales + g * 128, ng * 512, bar, policy);
            bulk_g2s(dst + kGPS * 3584, L.v_zeros + g * 128, ng * 512, bar, policy);
        }
        __syncwarp();
    };
    for (int c = 0; c < kStages && c < my_n; ++c) issue(c);

    const int64_t q_row = (int64_t)u * n_rep + head0;
    auto stage_queries = [&](float* dst) {                               // [4][128], pre-scaled (absent heads: zeros)
        for (int i = threadIdx.x; i < kD; i += blockDim.x) {
            float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if ((i >> 5) < n_heads) {
                if (q_dtype == KIVI_BF16) RowVec<__nv_bfloat16>::load4(reinterpret_cast<const __nv_bfloat16*>(q) + q_row * kD + 4 * i, t);
                else RowVec<float>::load4(reinterpret_cast<const float*>(q) + q_row * kD + 4 * i, t);
            }
            *reinterpret_cast<float4*>(dst + 4 * i) = make_float4(scale_log2 * t[0], scale_log2 * t[1], scale_log2 * t[2], scale_log2 * t[3]);
        }
    };
    if (is_res) {
        // ---------------- residual ring ----------------
        stage_queries(q_s);
        __syncthreads();
        const int rs = sub;
        const int t_begin = rs * res_chunk;
        const int t_end = t_begin + res_chunk < res_len ? t_begin + res_chunk : res_len;
        float m[4], l[4], o[4][4];
        if (L.res_dtype == KIVI_BF16)
            residual_part<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(L.k_res) + (int64_t)u * L.residual_cap * kD,
                                         reinterpret_cast<const __nv_bfloat16*>(L.v_res) + (int64_t)u * L.residual_cap * kD,
                                         L.residual_cap, res_start, res_len, t_begin, t_end, q_s, lane, warp, m, l, o);
        else
            residual_part<float>(reinterpret_cast<const float*>(L.k_res) + (int64_t)u * L.residual_cap * kD,
                                 reinterpret_cast<const float*>(L.v_res) + (int64_t)u * L.residual_cap * kD,
                                 L.residual_cap, res_start, res_len, t_begin, t_end, q_s, lane, warp, m, l, o);
        if (lane < 4) {
            // lane h publishes head h (m and l are warp-uniform after the reductions)
            float mh = m[0], lh = l[0];
            if (lane == 1) { mh = m[1]; lh = l[1]; }
            if (lane == 2) { mh = m[2]; lh = l[2]; }
            if (lane == 3) { mh = m[3]; lh = l[3]; }
            ml_s[(warp * 4 + lane) * 2] = mh; ml_s[(warp * 4 + lane) * 2 + 1] = lh;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            float M = -INFINITY;
#pragma unroll
            for (int w2 = 0; w2 < kWarps; ++w2) M = fmaxf(M, ml_s[(w2 * 4 + h) * 2]);
            const float f = (m[h] == -INFINITY) ? 0.0f : ex2(m[h] - M);
            *reinterpret_cast<float4*>(fo + h * kD + 4 * lane) = make_float4(f * o[h][0], f * o[h][1], f * o[h][2], f * o[h][3]);
        }
    } else {
        // ---------------- quantized history ----------------
        std::conditional_t<ONE, OneView, LaneView> v;
        v.gid = gid; v.tig = tig; v.lane = lane;
        uint8_t* scratch = scratch_mem + warp * kScratchBytes;
        v.scratch = smem_u32(scratch);
        // row `lane & 15` of matrix `lane >> 4`
        v.k_rows = v.scratch + 1024 * (lane >> 4) + 512 * (lane & 1) + 16 * ((lane >> 1) & 7);
        v.v_rows = v.scratch + 256 * (lane >> 4) + 16 * (lane & 15);
        // contraction index of the token whose scales are row `lane`
        const int kap = gid >> 2, k = 4 * tig + (gid & 3);
        v.v_write = v.scratch + 16 * k + 8 * (kap ^ (k >> 3));
        v.v_first = 32 * (tig >> 1);
        if constexpr (ONE) {
            v.p_write = v.scratch + 128 * (tig & 1) + 4 * (16 * kap + (gid & 3));
        } else {
            v.p_even = v.scratch + 16 * (16 * kap + (gid & 3)) + 64 * kap + 4 * tig;
            v.p_odd = v.scratch + 16 * (16 * kap + (gid & 3)) + 64 * (1 - kap) + 4 * tig;
            v.p_read = v.scratch + 16 * p_row(lane);
            v.rest_rows = 128 * (lane >> 4) + 512 * (lane & 1) + 16 * ((lane >> 1) & 7);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) asm volatile("mov.b32 %0, %1;" : "=r"(v.start[i]) : "n"(kTwo23Bits));
        if (q_dtype == KIVI_BF16) load_queries(reinterpret_cast<const __nv_bfloat16*>(q) + q_row * kD, n_heads, scale_log2, v);
        else load_queries(reinterpret_cast<const float*>(q) + q_row * kD, n_heads, scale_log2, v);

        if constexpr (WIDE) {
#pragma unroll
            for (int i = 0; i < 4; ++i) asm volatile("mov.b32 %0, %1;" : "=r"(v.ones[i]) : "n"(kOnes));
            v.q_zero = reinterpret_cast<const float4*>(zero_s) + 32 * tig;
            stage_queries(zero_s);
            __syncthreads();
        }

        std::conditional_t<ONE, OneState, WarpState> st;
        clear(st);

        bool ok = true;
        int c = 0;
        for (; c < my_n; ++c) {
            const int s = c % kStages;
            if (!__all_sync(0xffffffffu, mbar_wait(bar0 + 8 * s, (uint32_t)(c / kStages) & 1u))) { ok = false; break; }
            const int goff = (warp + kWarps * c) * kGPS;
            const uint8_t* sb = wstage + s * kStageBytes;
            if (n_my_groups - goff >= 2) process_groups<2, WIDE>(sb, v, scratch, st);
            else process_groups<1, WIDE>(sb, v, scratch, st);
            __syncwarp();
            if (c + kStages < my_n) issue(c + kStages);
        }
        if (!ok) {
            // A copy did not land within the bound.  The copies still in flight
            // target this warp's ring: give each of them (chunks c .. c+kStages-1,
            // those that were issued) a second bounded wait on its own phase
            // before the ring is reused, then report an empty partial.
            if (lane == 0) atomicExch(&g_fault_word, 1);
            for (int i = c; i < c + kStages && i < my_n; ++i)
                mbar_wait(bar0 + 8 * (i % kStages), (uint32_t)(i / kStages) & 1u);
            clear(st);
        }

        // ---- fold the warp's lanes ----------------------------------------------
        if constexpr (ONE) {
#pragma unroll
            for (int off = 1; off <= 16; off *= 2) {
                st.l += __shfl_xor_sync(0xffffffffu, st.l, off);
#pragma unroll
                for (int gd = 0; gd < 4; ++gd) st.oz[gd] += __shfl_xor_sync(0xffffffffu, st.oz[gd], off);
            }
            if (lane == 0) { ml_s[warp * 8] = st.m; ml_s[warp * 8 + 1] = st.l; }
            __syncthreads();
            float M = -INFINITY;
#pragma unroll
            for (int w2 = 0; w2 < kWarps; ++w2) M = fmaxf(M, ml_s[w2 * 8]);
            const float f = (st.m == -INFINITY) ? 0.0f : ex2(st.m - M);
            const float z = tig == 0 ? st.oz[0] : tig == 1 ? st.oz[1] : tig == 2 ? st.oz[2] : st.oz[3];
            *reinterpret_cast<float4*>(fo + 32 * tig + 4 * gid) =
                make_float4(f * (st.o[0] + z), f * fmaf(st.o[1], kRow1, z), f * fmaf(st.o[2], kRow2, z), f * fmaf(st.o[3], kRow3, z));
        } else {
            st.l += __shfl_xor_sync(0xffffffffu, st.l, 4);
            st.l += __shfl_xor_sync(0xffffffffu, st.l, 8);
            st.l += __shfl_xor_sync(0xffffffffu, st.l, 16);
            // zero term: every lane holds partial sums of all heads and channel groups
            float* const oz_s = reinterpret_cast<float*>(scratch);                  // [lane][head][channel group]
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 4; ++h) *reinterpret_cast<float4*>(oz_s + 16 * lane + 4 * h) = make_float4(st.oz[h][0], st.oz[h][1], st.oz[h][2], st.oz[h][3]);
            __syncwarp();
            float z = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; ++i) z += oz_s[16 * ((lane & 16) + i) + (lane & 15)];
            z += __shfl_xor_sync(0xffffffffu, z, 16);
            float ozt[4];                                                            // head tig
#pragma unroll
            for (int gd = 0; gd < 4; ++gd) ozt[gd] = __shfl_sync(0xffffffffu, z, 4 * tig + gd);
            if (gid == 0) { ml_s[(warp * 4 + tig) * 2] = st.m; ml_s[(warp * 4 + tig) * 2 + 1] = st.l; }
            __syncthreads();
            float M = -INFINITY;
#pragma unroll
            for (int w2 = 0; w2 < kWarps; ++w2) M = fmaxf(M, ml_s[(w2 * 4 + tig) * 2]);
            const float f = (st.m == -INFINITY) ? 0.0f : ex2(st.m - M);
#pragma unroll
            for (int mt = 0; mt < 8; ++mt) {
                const int gd = mt >> 1;
                const int ch = 32 * gd + 4 * gid + 2 * (mt & 1);
                // code index 2*(mt&1) / 2*(mt&1)+1 of its byte
                const float r0 = (mt & 1) ? kRow2 : 1.0f, r1 = (mt & 1) ? kRow3 : kRow1;
                *reinterpret_cast<float2*>(fo + tig * kD + ch) =
                    make_float2(f * fmaf(st.o[mt][0], r0, ozt[gd]), f * fmaf(st.o[mt][1], r1, ozt[gd]));
            }
        }
    }
    __syncthreads();

    // ---- the CTA's partial: warps added in warp order ------------------------------
    // (for the fold inside a cluster it stays in shared memory, behind the first warp's buffer)
    const int64_t pbase = ((int64_t)u * n_splits_total + slot) * n_rep + head0;
    float* const cta_o = reinterpret_cast<float*>(stage_mem) + 4 * kD;
    for (int i = threadIdx.x; i < kD; i += blockDim.x) {
        const int h = i >> 5, cc = (i & 31) * 4;
        if (h < n_heads) {
            float4 a = *reinterpret_cast<const float4*>(stage_mem + h * kD * 4 + cc * 4);
#pragma unroll
            for (int w2 = 1; w2 < kWarps; ++w2) {
                const float4 b = *reinterpret_cast<const float4*>(stage_mem + w2 * kStages * kStageBytes + h * kD * 4 + cc * 4);
                a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
            }
            *reinterpret_cast<float4*>(FOLD ? cta_o + h * kD + cc : part_o + (pbase + h) * kD + cc) = a;
        }
    }
    float* const ml_out = FOLD ? cta_o + 4 * kD : part_ml + pbase * 2;
    if (threadIdx.x < n_heads) {
        const int h = threadIdx.x;
        float Mh = -INFINITY, ls = 0.0f;
        for (int w2 = 0; w2 < kWarps; ++w2) Mh = fmaxf(Mh, ml_s[(w2 * 4 + h) * 2]);
        for (int w2 = 0; w2 < kWarps; ++w2) {
            const float mw = ml_s[(w2 * 4 + h) * 2];
            if (mw != -INFINITY) ls += ml_s[(w2 * 4 + h) * 2 + 1] * ex2(mw - Mh);
        }
        ml_out[h * 2] = Mh;
        ml_out[h * 2 + 1] = ls;
    }
    if constexpr (FOLD) cluster_fold(cta_o, ml_out, n_heads, kD, (int64_t)u * n_rep + head0, direct);
}

constexpr size_t kSmemBytes = (size_t)kWarps * (kStages * kStageBytes + kScratchBytes) + kWarps * kStages * 8 + kWarps * 4 * 2 * 4;
constexpr size_t kSmemBytesWide = kSmemBytes + 4 * kD * 4;
static_assert(kScratchBytes >= 4 * kD * 4, "ring CTAs keep the queries in the first warp's scratch");
static_assert(kStages * kStageBytes >= 2 * 4 * kD * 4 + 32, "a warp's ring doubles as its [4][128] fold buffer, the first also holds the CTA's partial");
static_assert(kWarps * 32 >= 32, "at least one warp");

}  // namespace

bool attn_mma_supported(const kivi_layer* L, int n_rep, const void* q) {
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    return L->head_dim == kD && L->group_size == kG && n_rep >= 1 && n_rep <= 8 && al(q) &&
           al(L->k_res) && al(L->v_res) && al(L->k_codes) && al(L->k_scales) && al(L->k_zeros) && al(L->v_codes) && al(L->v_scales) && al(L->v_zeros);
}

// number of residual CTAs per unit and tokens per CTA (multiple of 32)
void attn_mma_residual_plan(int res_len, int* n_res_splits, int* res_chunk) {
    int rs = (res_len + 32 * kWarps - 1) / (32 * kWarps);
    if (rs > 8) rs = 8;
    int chunk = rs ? (res_len + rs - 1) / rs : 0;
    chunk = (chunk + 31) / 32 * 32;
    *n_res_splits = chunk ? (res_len + chunk - 1) / chunk : 0;
    *res_chunk = chunk;
}

// the opt-in shared-memory size is a per-device attribute of the kernel
static int ensure_smem_attr(int* dev_out) {
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    KIVI_CUDA_OK(cudaGetDevice(&dev));
    KIVI_REQUIRE(dev >= 0 && dev < 64, "device ordinal %d out of range", dev);
    if (!attr_set[dev].load(std::memory_order_acquire)) {
        for (auto* kernel : {attn_mma_kernel<false, false, false>, attn_mma_kernel<true, false, false>, attn_mma_kernel<false, true, false>,
                             attn_mma_kernel<true, true, false>, attn_mma_kernel<false, false, true>, attn_mma_kernel<true, false, true>})
            KIVI_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytesWide));
        attr_set[dev].store(true, std::memory_order_release);
    }
    if (dev_out) *dev_out = dev;
    return KIVI_OK;
}

// CTAs of the kernel that one SM holds at a time (registers and shared memory
// decide); asked from the runtime once per device.  0 = the query failed.
int attn_mma_ctas_per_sm() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (ensure_smem_attr(&dev) != KIVI_OK) return 0;
    int n = cached[dev].load(std::memory_order_acquire);
    if (n == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, attn_mma_kernel<false, false, false>, kWarps * 32, kSmemBytesWide) != cudaSuccess || n <= 0)
            return 0;
        cached[dev].store(n, std::memory_order_release);
    }
    return n;
}

int run_attn_mma(const kivi_layer* L, int64_t quant_len, int res_start, int res_len,
                 const void* q, int q_dtype, int n_rep, float scale_log2, bool wide, int nq_splits, int gps,
                 int n_res_splits, int res_chunk, float* part_o, float* part_ml, const ClusterOut& direct, cudaStream_t st) {
    if (int rc = ensure_smem_attr(nullptr)) return rc;
    dim3 grid((unsigned)(nq_splits + n_res_splits) * (unsigned)L->num_units * (unsigned)((n_rep + 3) / 4));
    const bool fold = direct.out != nullptr;
    auto* const kernel = wide ? (fold ? attn_mma_kernel<true, true, false> : attn_mma_kernel<false, true, false>)
                       : n_rep == 1 ? (fold ? attn_mma_kernel<true, false, true> : attn_mma_kernel<false, false, true>)
                                    : (fold ? attn_mma_kernel<true, false, false> : attn_mma_kernel<false, false, false>);
    KIVI_CUDA_OK(launch_cluster(kernel, direct.out ? nq_splits + n_res_splits : 0, grid, kWarps * 32, wide ? kSmemBytesWide : kSmemBytes, st, true, *L, quant_len, res_start, res_len, q, q_dtype, scale_log2,
                        n_rep, gps, nq_splits, n_res_splits, res_chunk, part_o, part_ml, direct));
    return KIVI_OK;
}

// ---- self-test: how far below the largest product the tensor core keeps bits -------
// One m16n8k16 MMA per k: C = -1, products {1 * 1, 2^-a * 2^-b} with a + b = k.
// If the unit kept every bit the result would be exactly 2^-k; it aligns the
// addends on their exponent fields and truncates below a fixed distance from the
// largest, so from some k on the small product is lost.  (Why the kernel above
// contracts bytes, whose sums are exact.)
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__global__ void mma_alignment_probe_kernel(int* kept_out) {
    const int lane = threadIdx.x, gid = lane >> 2, tig = lane & 3;
    int kept = 0;
    for (int k = 8; k <= 34; ++k) {
        const int a_exp = k < 14 ? k : 14, b_exp = k - a_exp;          // both factors stay normal fp16 numbers
        // A[row][0] = 1, A[row][1] = 2^-a; B[0][col] = 1, B[1][col] = 2^-b; everything else 0
        const __half2 a01 = __halves2half2(__float2half(1.0f), __float2half(ldexpf(1.0f, -a_exp)));
        const __half2 b01 = __halves2half2(__float2half(1.0f), __float2half(ldexpf(1.0f, -b_exp)));
        uint32_t a[4] = {0u, 0u, 0u, 0u}, b0 = 0u;
        if (tig == 0) {                                                // k-slots 0 and 1 live in lanes with tig == 0
            a[0] = *reinterpret_cast<const uint32_t*>(&a01);
            a[1] = a[0];
            b0 = *reinterpret_cast<const uint32_t*>(&b01);
        }
        float c[4] = {-1.0f, -1.0f, -1.0f, -1.0f};
        mma_f16(c, a, b0, 0u);
        const bool ok = c[0] == ldexpf(1.0f, -k);
        if (__all_sync(0xffffffffu, ok)) kept = k;
    }
    (void)gid;
    if (lane == 0) *kept_out = kept;
}

int run_mma_alignment_probe(int* bits_out) {
    int* d = nullptr;
    KIVI_CUDA_OK(cudaMalloc(&d, sizeof(int)));
    mma_alignment_probe_kernel<<<1, 32>>>(d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(bits_out, d, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) { set_error("tensor-core alignment probe failed: %s", cudaGetErrorString(e)); return KIVI_ERR_CUDA; }
    return KIVI_OK;
}

int attn_mma_fault_word(int* out) {
    KIVI_CUDA_OK(cudaMemcpyFromSymbol(out, g_fault_word, sizeof(int)));
    return KIVI_OK;
}

int attn_mma_fault_clear() {
    const int zero = 0;
    KIVI_CUDA_OK(cudaMemcpyToSymbol(g_fault_word, &zero, sizeof(int)));
    return KIVI_OK;
}

}  // namespace kivi

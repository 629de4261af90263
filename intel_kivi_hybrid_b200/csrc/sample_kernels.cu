// Next-token choice on the device: argmax, or temperature / top-k / multinomial
// sampling over [batch, vocab] logits, one CTA per batch row.
//
// Same arithmetic as the reference's sample_token
// (src/kivi_sycl/generation/sampling.py:10-25): logits / max(temperature, 1e-8),
// everything below the k-th largest scaled logit masked out (ties with the k-th
// are kept, as `logits < kth` does), softmax, one draw.  The draw is the inverse
// CDF in index order of a counter-based uniform number (Philox4x32-10 keyed by
// (seed), counter (step, row)), so a CPU restatement reproduces it without
// sharing any generator state, and the ids never have to leave the device.
#include "kivi_common.cuh"

#include <type_traits>

namespace kivi {
namespace {

// Candidates of a top-k cut that are kept in shared memory, and the largest cut that is
// made that way: the k-th largest of n threads' maxima leaves about n ln(n / (n - k))
// entries of a row of unrelated logits, 0.51 n at k = 2n/5.
__host__ __device__ constexpr int cut_capacity(int threads) { return threads == 1024 ? 640 : 512; }
__host__ __device__ constexpr int cut_limit(int threads) { return threads * 2 / 5; }

// order-preserving map float -> uint32 (larger float, larger key); NaN sorts above +inf
__device__ __forceinline__ uint32_t ordered_key(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b) { return __umulhi(a, b); }

// Philox4x32-10 (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3"):
// returns the first of the four output words
__device__ uint32_t philox_first_word(uint64_t seed, uint64_t step, uint32_t row) {
    uint32_t c0 = (uint32_t)step, c1 = (uint32_t)(step >> 32), c2 = row, c3 = 0u;
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = mulhi32(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        const uint32_t hi1 = mulhi32(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
        c0 = n0; c1 = n1; c2 = n2; c3 = n3;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return c0;
}

struct MaxIdx { float v; int i; };
__device__ __forceinline__ MaxIdx better(MaxIdx a, MaxIdx b) {      // larger value, then smaller index; NaN never wins
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

// The k-th largest of the threads' keys by bisection on the bits from 31 down to
// `last_bit` (the lower bits 0): one barrier per bit, which also counts.  Every thread
// gets the answer; at least k keys are >= it.
__device__ __forceinline__ uint32_t kth_key(uint32_t key, int k, int last_bit) {
    uint32_t t = 0u;
    for (int bit = 31; bit >= last_bit; --bit) {
        const uint32_t probe = t | (1u << bit);
        if (__syncthreads_count(key >= probe) >= k) t = probe;
    }
    return t;
}

// Entries i0, i0 + step, ... of a row below `end`, kFlight loads in flight: whole blocks
// of that many without a bounds test, the last one with.  (Indices are unsigned: a row
// may have 2^31 - 1 entries, and the walk steps past its end.)
template <int kFlight, typename T, typename F>
__device__ __forceinline__ void walk(const T* row, uint32_t i0, uint32_t end, uint32_t step, const F& f) {
    float x[kFlight];
    for (; i0 + (kFlight - 1) * step < end; i0 += kFlight * step) {
#pragma unroll
        for (int j = 0; j < kFlight; ++j) x[j] = (float)row[i0 + j * step];
#pragma unroll
        for (int j = 0; j < kFlight; ++j) f(x[j], i0 + j * step);
    }
    if (i0 < end) {
#pragma unroll
        for (int j = 0; j < kFlight; ++j) x[j] = i0 + j * step < end ? (float)row[i0 + j * step] : 0.0f;
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
            if (i0 + j * step < end) f(x[j], i0 + j * step);
    }
}

// One CTA per row.  A row is a few hundred KB that one SM reads at its share of the
// memory rate, so what counts is how often it is walked and how many loads are in
// flight: one pass for the maximum (strided over the threads, coalesced, eight loads in
// flight), one more to draw.
//
// Top-k cut: at least k entries are >= the k-th largest of the threads' own maxima
// (its upper 16 bits are bound enough), so one pass that collects the entries above
// that bound into shared memory (a few more than k for unrelated logits) leaves a set
// small enough to rank every entry by counting and to draw from without reading the
// row again: an entry is kept when fewer than k are greater, which is what comparing
// it with the k-th value says.  A larger k (cut_limit), more candidates than kCand (long
// runs of equal logits) and rows with NaN take a radix select over the row instead.
// 128 rows x 50257 fp32, top 50: 237 us with seven passes and two serial scans, 15 now.
//
// What a call needs is a kernel of its own (Choice) and so is the number of threads a row
// gets, so that the registers of one way do not cost another its occupancy.
enum class Choice { kArgmax, kDraw, kTopK, kTopKRadix };

template <typename T, int kThreads, Choice kChoice>
__global__ void __launch_bounds__(kThreads, kThreads == 256 ? 8 : kThreads == 512 ? 3 : 1)
sample_kernel(const T* logits, int vocab, int64_t row_stride,
              float temperature, int top_k, uint64_t seed, uint64_t step, int64_t* __restrict__ ids) {
    constexpr int kWarps = kThreads / 32;
    constexpr int kFlight = kThreads == 256 && kChoice != Choice::kArgmax ? 4 : 8;     // (256: 32 registers, so that an SM holds eight rows)
    constexpr int kCand = cut_capacity(kThreads), kPer = (kCand + kThreads - 1) / kThreads;      // candidates; how many of them a thread ranks
    __shared__ float red_f[kWarps];
    __shared__ int red_i[kWarps];
    __shared__ double scan_s[kWarps];
    __shared__ int pick_s;
    stream_order();
    const T* row = settled(logits) + (int64_t)blockIdx.x * row_stride;
    // the reference divides: logits / max(temperature, 1e-8)
    auto scaled = [&](float x) { return __fdiv_rn(x, temperature); };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n_row = (uint32_t)vocab;

    // ---- row maximum and its first index (also the argmax answer) ----------------
    MaxIdx best{-INFINITY, 0x7fffffff};
    bool nan = false;
    walk<kFlight>(row, tid, n_row, kThreads, [&](float x, uint32_t i) {
        best = better(best, MaxIdx{x, (int)i});
        if constexpr (kChoice == Choice::kTopK) nan |= x != x;
    });
    const MaxIdx mine_best = best;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        best = better(best, MaxIdx{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
    if (lane == 0) { red_f[warp] = best.v; red_i[warp] = best.i; }
    if (tid == 0) pick_s = -1;
    const bool row_nan = __syncthreads_or(nan);
    best = MaxIdx{red_f[0], red_i[0]};
    for (int w = 1; w < kWarps; ++w) best = better(best, MaxIdx{red_f[w], red_i[w]});
    if (best.i == 0x7fffffff) best.i = 0;                  // a row of NaNs / -inf
    if constexpr (kChoice == Choice::kArgmax) {
        if (tid == 0) ids[blockIdx.x] = best.i;
        return;
    }
    const float m = scaled(best.v);
    const double u = ((double)philox_first_word(seed, step, blockIdx.x) + 0.5) * (1.0 / 4294967296.0);

    float kth = -INFINITY;
    if constexpr (kChoice == Choice::kTopK) {
        __shared__ float cand_x[kCand];
        __shared__ int cand_i[kCand];
        __shared__ double cand_w[kCand];
        __shared__ int n_cand_s;
        if (tid == 0) n_cand_s = 0;                         // (the barriers of kth_key lie in between)
        // largest scaled logit of this thread as a key; 0 (below every number's key) without one
        const uint32_t my_key = mine_best.i == 0x7fffffff ? 0u : ordered_key(scaled(mine_best.v));
        const uint32_t bound = row_nan ? 0u : kth_key(my_key, top_k, 16);
        if (bound != 0u) {                                  // CTA-uniform
            // compared as a number: -0 counts as +0, as in the cut itself (the keys between 0 and
            // that of -inf are NaN patterns: cutting the lower bits may end there)
            const float least = bound < 0x007fffffu ? -INFINITY : key_to_float(bound);
            // what is clearly below is dropped without a division (a quotient that lost bits in
            // the subnormals does not say what is clear)
            const float clear = fabsf(least) > 1e-30f && fabsf(least) < 1e30f ? (least - fabsf(least) * 1e-5f) * temperature : -INFINITY;
            // ---- collect what is not below the bound -------------------------------
            walk<kFlight>(row, tid, n_row, kThreads, [&](float x, uint32_t i) {
                if (!(x >= clear)) return;
                const float y = scaled(x);
                if (y >= least) {
                    const int at = atomicAdd(&n_cand_s, 1);
                    if (at < kCand) { cand_x[at] = y; cand_i[at] = (int)i; }
                }
            });
            __syncthreads();
            const int n = n_cand_s;
            if (n <= kCand) {
                // an entry's place in index order and how many are greater, by counting
                float x[kPer];
                int idx[kPer], place[kPer], greater[kPer];
#pragma unroll
                for (int e = 0; e < kPer; ++e) {
                    const int at = tid + e * kThreads;
                    x[e] = at < n ? cand_x[at] : 0.0f;
                    idx[e] = at < n ? cand_i[at] : 0;
                    place[e] = greater[e] = 0;
                    if (at < n)
                        for (int c = 0; c < n; ++c) {
                            place[e] += cand_i[c] < idx[e];
                            greater[e] += cand_x[c] > x[e];
                        }
                }
                __syncthreads();                            // all have read the unsorted entries
#pragma unroll
                for (int e = 0; e < kPer; ++e)
                    if (tid + e * kThreads < n) {
                        cand_i[place[e]] = idx[e];
                        cand_w[place[e]] = greater[e] < top_k ? (double)expf(x[e] - m) : 0.0;
                    }
                __syncthreads();
                if (warp == 0) {
                    // running masses in index order, the first one past the target is the draw
                    double total = 0.0;
                    for (int c = 0; c < n; c += 32) total += c + lane < n ? cand_w[c + lane] : 0.0;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
                    const double target = u * total;
                    double run = 0.0;
                    int pick = -1, last_kept = -1;
                    for (int c = 0; c < n && pick < 0; c += 32) {
                        const double w = c + lane < n ? cand_w[c + lane] : 0.0;
                        double incl = w;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) { const double v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
                        const unsigned kept = __ballot_sync(0xffffffffu, w > 0.0);
                        const unsigned past = __ballot_sync(0xffffffffu, w > 0.0 && run + incl > target);
                        if (past) pick = c + __ffs(past) - 1;
                        if (kept) last_kept = c + 31 - __clz(kept);
                        run += __shfl_sync(0xffffffffu, incl, 31);
                    }
                    // (rounding may leave the last running mass at the target: the last kept entry then;
                    // a total that is zero or not a number falls back to the argmax)
                    if (lane == 0) ids[blockIdx.x] = !(total > 0.0) || total == INFINITY ? best.i : pick >= 0 ? cand_i[pick] : last_kept >= 0 ? cand_i[last_kept] : best.i;
                }
                return;
            }
        }
    }
    if constexpr (kChoice == Choice::kTopK || kChoice == Choice::kTopKRadix) {
        __shared__ unsigned hist[256];
        __shared__ uint32_t sel_prefix;
        __shared__ int sel_remaining;
        // ---- radix select on the ordered keys, 8 bits a pass --------------------------
        if (tid == 0) { sel_prefix = 0u; sel_remaining = top_k; }
        for (int pass = 0; pass < 4; ++pass) {
            const int shift = 24 - 8 * pass;
            for (int b = tid; b < 256; b += kThreads) hist[b] = 0u;
            __syncthreads();
            const uint32_t prefix = sel_prefix;
            const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
            walk<kFlight>(row, tid, n_row, kThreads, [&](float x, uint32_t) {
                const uint32_t key = ordered_key(scaled(x));
                if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
            });
            __syncthreads();
            if (tid == 0) {
                int need = sel_remaining, b = 255;
                for (; b > 0; --b) {
                    if ((int)hist[b] >= need) break;
                    need -= (int)hist[b];
                }
                sel_prefix = prefix | ((uint32_t)b << shift);
                sel_remaining = need;
            }
            __syncthreads();
        }
        kth = key_to_float(sel_prefix);
    }

    // ---- softmax weights over the kept entries: a contiguous segment per warp ---------
    const uint32_t seg = (n_row + kWarps - 1) / kWarps;
    const uint32_t s0 = min(n_row, warp * seg), s1 = min(n_row, s0 + seg);
    double mine = 0.0;
    walk<kFlight>(row, s0 + lane, s1, 32, [&](float x, uint32_t) {
        const float y = scaled(x);
        if (y >= kth) mine += (double)expf(y - m);
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0) scan_s[warp] = mine;
    __syncthreads();
    double before = 0.0, total = 0.0;                       // 32 numbers, added in order by every thread
    for (int w = 0; w < kWarps; ++w) { if (w == warp) before = total; total += scan_s[w]; }
    const double target = u * total;
    // exactly one segment has before <= target < before + mine (masses are >= 0 and
    // target < total); it walks its kept entries until the running mass passes the target
    if (mine > 0.0 && before <= target && target < before + mine) {
        double run = before;
        int pick = -1, last_kept = -1;
        uint32_t i0 = s0;
        // blocks of kFlight x 32 entries that end below the target are passed as a whole
        for (; i0 + kFlight * 32 <= s1; i0 += kFlight * 32) {
            float y[kFlight];
#pragma unroll
            for (int j = 0; j < kFlight; ++j) y[j] = (float)row[i0 + 32 * j + lane];
            double block = 0.0;
#pragma unroll
            for (int j = 0; j < kFlight; ++j) {
                const float z = scaled(y[j]);
                if (z >= kth) { block += (double)expf(z - m); last_kept = (int)(i0 + 32 * j + lane); }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) block += __shfl_xor_sync(0xffffffffu, block, o);
            if (run + block > target) break;
            run += block;
        }
        for (; i0 < s1 && pick < 0; i0 += 32) {
            const uint32_t i = i0 + lane;
            const float y = i < s1 ? scaled((float)row[i]) : 0.0f;
            const bool kept = i < s1 && y >= kth;
            double incl = kept ? (double)expf(y - m) : 0.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const double v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
            const unsigned past = __ballot_sync(0xffffffffu, kept && run + incl > target);
            if (past) pick = (int)i0 + __ffs(past) - 1;
            if (kept) last_kept = (int)i;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) last_kept = max(last_kept, __shfl_xor_sync(0xffffffffu, last_kept, o));
        // the walk adds the same numbers in another order than the sum above: should the
        // last bits leave it short of the target, the segment's last kept entry is the draw
        if (lane == 0) pick_s = pick >= 0 ? pick : last_kept;
    }
    __syncthreads();
    // no segment claimed the target (total mass 0 or not finite): fall back to the argmax
    if (tid == 0) ids[blockIdx.x] = pick_s >= 0 ? pick_s : best.i;
}

}  // namespace

// Threads per row.  A CTA of 1024 threads fills an SM, one of 512 a third, one of 256 an
// eighth: up to one row per SM the row's length decides (as many loads in flight as it can
// use; past that, barriers and folds cost more than the walk), with more rows than that
// the rows side by side do.  Measured with 256 / 512 / 1024 threads, us, fp32:
//   1 row, drawn from the whole row: 1000 entries 4.9 / 5.0 / 6.9, 10000 16 / 13 / 15, 50257 44 / 31 / 22
//   256 rows x 32000, the same: 46 / 31 / 37; argmax 8.0 / 7.7 / 10.5
//   1024 rows x 1000: 9.9 / 16 / 39; argmax 4.5 / 7.6 / 19
// A top-k cut from candidates wants 5k/2 threads (64 rows x 2048, k = 200: 18 / 11 / 12,
// k = 400: 27 / 30 / 20) and gets them unless that leaves rows waiting for a place; short
// rows in crowds do as well with the radix select (1024 x 1000, k = 200: 32, and 34 with 512).
static int sample_threads(int batch, int vocab, int cut) {
    const int sms = num_sms();
    const int walk = batch <= sms ? (vocab <= 2048 ? 256 : vocab <= 16384 ? 512 : 1024) : batch <= 3 * sms && vocab > 8192 ? 512 : 256;
    const int ranking = cut <= cut_limit(256) ? 256 : cut <= cut_limit(512) ? 512 : cut <= cut_limit(1024) ? 1024 : 0;
    if (ranking > walk && (batch <= sms || (ranking == 512 && (batch <= 3 * sms || vocab > 2048)))) return ranking;
    return walk;
}

template <typename T, int kThreads>
static cudaError_t launch_sample(const T* logits, int batch, int vocab, int64_t row_stride, float temperature, int top_k, int do_sample,
                                 uint64_t seed, uint64_t step, int64_t* ids, cudaStream_t st) {
    auto go = [&](auto kernel) { return launch(kernel, dim3((unsigned)batch), kThreads, 0, st, true, logits, vocab, row_stride, temperature, top_k, seed, step, ids); };
    if (!do_sample) return go(sample_kernel<T, kThreads, Choice::kArgmax>);
    if (top_k == 0) return go(sample_kernel<T, kThreads, Choice::kDraw>);
    if (top_k <= cut_limit(kThreads)) return go(sample_kernel<T, kThreads, Choice::kTopK>);
    return go(sample_kernel<T, kThreads, Choice::kTopKRadix>);
}

int run_sample(const void* logits, int dtype, int batch, int vocab, int64_t row_stride, float temperature, int top_k,
               int do_sample, uint64_t seed, uint64_t step, int64_t* ids, cudaStream_t st) {
    const float t = temperature > 1e-8f ? temperature : 1e-8f;
    if (!do_sample || top_k >= vocab) top_k = 0;           // no cut
    const int threads = sample_threads(batch, vocab, top_k);
    auto go = [&](auto* p) {
        using T = std::remove_pointer_t<decltype(p)>;
        auto run = threads == 256 ? launch_sample<std::remove_cv_t<T>, 256> : threads == 512 ? launch_sample<std::remove_cv_t<T>, 512> : launch_sample<std::remove_cv_t<T>, 1024>;
        return run(p, batch, vocab, row_stride, t, top_k, do_sample, seed, step, ids, st);
    };
    if (dtype == KIVI_F32) KIVI_CUDA_OK(go(reinterpret_cast<const float*>(logits)));
    else KIVI_CUDA_OK(go(reinterpret_cast<const __nv_bfloat16*>(logits)));
    return KIVI_OK;
}

}  // namespace kivi

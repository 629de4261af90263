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
#include "async_copy.cuh"
#include "kivi_common.cuh"

#include <atomic>
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

// A bound that at least k keys reach, for k up to an eighth of the threads, with two
// barriers instead of sixteen: every warp finds its j-th largest key, and r warps (r j >= k)
// reach the r-th largest of those.  About 1.7 k keys reach it, where the k-th largest is
// reached by k; 1024 threads, k = 50: 2700 cycles by bisection, 600 this way (three bits
// a step with counts by ballot and shared-memory atomics took 5000).
template <int kWarps>
__device__ __forceinline__ uint32_t bound_key(uint32_t key, int k, uint32_t* warp_s) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = (k + kWarps * 5 / 8 - 1) / (kWarps * 5 / 8), r = (k + j - 1) / j;
    uint32_t largest = 0u;
    for (int i = 0; i < j; ++i) {
        largest = __reduce_max_sync(0xffffffffu, key);
        const unsigned who = __ballot_sync(0xffffffffu, key == largest);
        if (lane == __ffs(who) - 1) key = 0u;                // one of them is counted
    }
    if (lane == 0) warp_s[warp] = largest;
    __syncthreads();
    if (warp == 0) {                                        // (one warp: thirty-two would wait for each other's shuffles)
        const uint32_t mine = lane < kWarps ? warp_s[lane] : 0u;
        int before = 0;                                     // warps whose key comes before this lane's
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t other = __shfl_sync(0xffffffffu, mine, w);
            before += other > mine || (other == mine && w < lane);
        }
        if (lane < kWarps && before == r - 1) warp_s[kWarps] = mine;
    }
    __syncthreads();
    return warp_s[kWarps];
}

__device__ __forceinline__ float max_nan(float a, float b) {              // NaN if either is
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float warp_max_nan(float a) {
    float d;
    asm volatile("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(d) : "f"(a));
    return d;
}
// the entries of an aligned 16 bytes
template <typename T> struct Granule;
template <> struct Granule<float> {
    static constexpr int kSize = 4;
    __device__ static void load(const unsigned char* p, float (&x)[4]) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    }
};
template <> struct Granule<__nv_bfloat16> {
    static constexpr int kSize = 8;
    __device__ static void load(const unsigned char* p, float (&x)[8]) {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { x[2 * i] = __uint_as_float(w[i] << 16); x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    }
};
template <int N> __device__ __forceinline__ float largest(const float (&x)[N]) {
    float m = max_nan(x[0], x[1]);
#pragma unroll
    for (int i = 2; i < N; i += 2) m = max_nan(m, max_nan(x[i], x[i + 1]));
    return m;
}

__device__ int g_sample_fault = 0;
constexpr int kChunks = 4;                 // pieces a staged row arrives in

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

// One CTA per row.  What a row costs is latency: how often it is walked, how many bytes are
// in flight, and the barriers in between.  kStaged (long rows that fit shared memory, one row
// per SM): bulk copies bring the whole row into shared memory, everything in flight at once,
// and both passes read it there, 16 bytes at a time: the maximum as the pieces arrive, then
// the candidates or the draw.  Otherwise both passes read memory, strided over the threads.
//
// Top-k cut: at least k entries are >= the k-th largest of the threads' own maxima
// (its upper 16 bits are bound enough), so one pass that collects the entries above
// that bound into shared memory (a few more than k for unrelated logits) leaves a set
// small enough to rank every entry by counting and to draw from without reading the
// row again: an entry is kept when fewer than k are greater, which is what comparing
// it with the k-th value says.  A larger k (cut_limit), more candidates than kCand (long
// runs of equal logits) and rows with NaN take a radix select over the row instead.
// 128 rows x 50257 fp32, top 50: 237 us with seven passes and two serial scans, 14.2 with two
// passes over memory, bisection and one thread to a candidate, 10.6 now.
//
// What a call needs is a kernel of its own (Choice) and so is the number of threads a row
// gets, so that the registers of one way do not cost another its occupancy.
enum class Choice { kArgmax, kDraw, kTopK, kTopKRadix };

template <typename T, int kThreads, Choice kChoice, bool kStaged>
__global__ void __launch_bounds__(kThreads, kThreads == 256 ? 8 : kThreads == 512 && !kStaged ? 3 : 1)
sample_kernel(const T* logits, int vocab, int64_t row_stride,
              float temperature, int top_k, uint64_t seed, uint64_t step, int64_t* __restrict__ ids) {
    constexpr int kWarps = kThreads / 32;
    constexpr int kFlight = kThreads == 256 && kChoice != Choice::kArgmax ? 4 : 8;     // (256: 32 registers, so that an SM holds eight rows)
    constexpr int kCand = cut_capacity(kThreads), kPer = (kCand + kThreads - 1) / kThreads;      // candidates; how many of them a thread ranks
    constexpr bool kArg = kChoice == Choice::kArgmax;
    __shared__ float red_f[kWarps];
    __shared__ int red_i[kWarps];
    __shared__ double scan_s[kWarps];
    __shared__ int pick_s;
    extern __shared__ __align__(128) unsigned char staged_s[];          // kStaged: the row at its own offset from a 16-byte boundary
    // the reference divides: logits / max(temperature, 1e-8)
    auto scaled = [&](float x) { return __fdiv_rn(x, temperature); };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n_row = (uint32_t)vocab;
    // (staged: worked out while the row is under way; else later, or it costs registers in the walk)
    auto uniform = [&]() { return ((double)philox_first_word(seed, step, blockIdx.x) + 0.5) * (1.0 / 4294967296.0); };
    double u = 0.0;
    if constexpr (kStaged) u = uniform();
    if (tid == 0) pick_s = -1;
    stream_order();
    const T* const given = settled(logits) + (int64_t)blockIdx.x * row_stride;
    const uint32_t skew = kStaged ? (uint32_t)(reinterpret_cast<uintptr_t>(given) & 15u) : 0u;
    const T* const row = kStaged ? reinterpret_cast<const T*>(staged_s + skew) : given;

    // largest entry and its first index; NaN does not count (a row of NaN: index 0)
    auto find_best = [&](const T* from) {
        MaxIdx best{-INFINITY, 0x7fffffff};
        walk<kFlight>(from, tid, n_row, kThreads, [&](float x, uint32_t i) { best = better(best, MaxIdx{x, (int)i}); });
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            best = better(best, MaxIdx{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
        if (lane == 0) { red_f[warp] = best.v; red_i[warp] = best.i; }
        __syncthreads();
        if constexpr (kWarps <= 8) {                        // (side by side eight reads cost less than five exchanges: 32 x 2048 1.56 us, not 1.66)
            best = MaxIdx{red_f[0], red_i[0]};
#pragma unroll
            for (int w = 1; w < kWarps; ++w) best = better(best, MaxIdx{red_f[w], red_i[w]});
        } else {
            best = lane < kWarps ? MaxIdx{red_f[lane], red_i[lane]} : MaxIdx{-INFINITY, 0x7fffffff};
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                best = better(best, MaxIdx{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
        }
        if (best.i == 0x7fffffff) best.i = 0;
        return best;
    };
    if constexpr (kArg) {
        const MaxIdx best = find_best(row);
        if (tid == 0) ids[blockIdx.x] = best.i;
        return;
    } else {
    __shared__ uint32_t warp_key_s[kWarps + 1];
    constexpr bool kCut = kChoice == Choice::kTopK;
    __shared__ __align__(16) float cand_x[kCut ? kCand : 4];
    __shared__ __align__(16) int cand_i[kCut ? kCand : 4];
    __shared__ double cand_w[kCut ? kCand : 1];
    __shared__ int n_cand_s;
    if (kCut && tid == 0) n_cand_s = 0;                     // (barriers lie between this and its use)

    // ---- largest entry of each thread and of the row (NaN if the row has one) ----------
    float top = -INFINITY;
    constexpr int kG = Granule<T>::kSize;
    const uint32_t n_granules = (skew + n_row * (uint32_t)sizeof(T) + 15u) / 16u;       // kStaged
    if constexpr (kStaged) {
        __shared__ uint64_t bars[kChunks];
        const uint32_t bar0 = smem_u32(bars);
        const unsigned char* const base = reinterpret_cast<const unsigned char*>(given) - skew;
        // granules that lie in the row as a whole are copied in kChunks pieces; the ragged
        // ends are loaded entry by entry, places outside the row hold -inf
        const uint32_t g0 = skew ? 1u : 0u, g1 = (skew + n_row * (uint32_t)sizeof(T)) / 16u;
        const uint32_t per = g1 > g0 ? (g1 - g0 + kChunks - 1) / kChunks : 0u;
        if (__shfl_sync(0xffffffffu, warp, 0) == 0 && elect_one()) {     // (operands of a bulk copy are the warp's, not a thread's)
            const uint64_t policy = l2_stream_policy();
#pragma unroll
            for (int c = 0; c < kChunks; ++c) mbar_init(bar0 + 8 * c, 1);
            mbar_init_fence();
#pragma unroll
            for (int c = 0; c < kChunks; ++c) {
                const uint32_t from = g0 + c * per, to = min(from + per, g1);
                if (from < to) {
                    mbar_expect_tx(bar0 + 8 * c, (to - from) * 16u);
                    bulk_g2s(smem_u32(staged_s) + from * 16u, base + (size_t)from * 16u, (to - from) * 16u, bar0 + 8 * c, policy);
                }
            }
        }
        for (int e = tid; e < 2 * kG; e += kThreads) {
            const uint32_t g = e < kG ? 0u : n_granules - 1u;
            if (e < kG ? g0 == 1u : (g1 < n_granules && (n_granules > 1u || g0 == 0u))) {
                const int64_t i = (int64_t)(g * kG) + (e % kG) - (int64_t)(skew / sizeof(T));
                const T x = i >= 0 && i < (int64_t)n_row ? given[i] : (T)(-INFINITY);
                reinterpret_cast<T*>(staged_s)[g * kG + e % kG] = x;
                top = max_nan(top, (float)x);
            }
        }
        __syncthreads();                                    // the barriers are set up
        bool arrived = true;
        for (int c = 0; c < kChunks; ++c) {
            const uint32_t from = g0 + c * per, to = min(from + per, g1);
            if (from >= to) break;
            if (!mbar_wait(bar0 + 8 * c, 0u)) { arrived = false; break; }
            // (thread t takes granules t, t + kThreads, ... whatever the pieces)
            for (uint32_t g = from + ((tid - from) & (kThreads - 1)); g < to; g += kThreads) {
                float x[kG];
                Granule<T>::load(staged_s + 16u * g, x);
                top = max_nan(top, largest<kG>(x));
            }
        }
        if (!__syncthreads_and(arrived)) {
            // a copy did not land within the bound: raise the fault word, give all of them a
            // second bounded wait, and read the row the plain way
            if (tid == 0) atomicExch(&g_sample_fault, 1);
            for (int c = 0; c < kChunks; ++c)
                if (g0 + c * per < g1) mbar_wait(bar0 + 8 * c, 0u);
            __syncthreads();
            top = -INFINITY;
            for (uint32_t i = tid; i < n_row; i += kThreads) {
                const_cast<T*>(row)[i] = given[i];
                top = max_nan(top, (float)given[i]);
            }
            __syncthreads();
        }
    } else {
        walk<kFlight>(row, tid, n_row, kThreads, [&](float x, uint32_t) { top = max_nan(top, x); });
    }
    const float mine_top = top;
    top = warp_max_nan(top);
    if (lane == 0) red_f[warp] = top;
    __syncthreads();
    top = warp_max_nan(lane < kWarps ? red_f[lane] : -INFINITY);
    const bool row_nan = top != top;                        // the same for all threads
    if (row_nan) {
        __syncthreads();
        top = find_best(row).v;
    }
    const float m = scaled(top);
    if constexpr (!kStaged) u = uniform();
    // the fallback of a draw that finds no mass, called by one warp: first index of the maximum
    auto argmax_index = [&]() {
        int at = 0x7fffffff;
        for (uint32_t i = lane; i < n_row && at == 0x7fffffff; i += 32)
            if ((float)row[i] == top) at = (int)i;
        at = __reduce_min_sync(0xffffffffu, at);
        return at == 0x7fffffff ? 0 : at;
    };

    float kth = -INFINITY;
    if constexpr (kCut) {
        // A thread's largest logit as a key, of the logit itself: division by the temperature
        // keeps the order.  (A thread without one: the key of -inf; fewer than k threads have
        // one then, or the bound is no higher.)
        const uint32_t my_key = ordered_key(mine_top);
        const uint32_t bound = row_nan ? 0u : top_k <= kThreads / 8 ? bound_key<kWarps>(my_key, top_k, warp_key_s) : kth_key(my_key, top_k, 16);
        if (bound != 0u) {                                  // CTA-uniform
            // Entries that the division rounds to the bound's quotient count too: the margin
            // takes them in where quotients are normal numbers, else everything is taken (the
            // keys between 0 and that of -inf are NaN patterns: cutting the lower bits may end there).
            const float least = bound < 0x007fffffu ? -INFINITY : key_to_float(bound);
            const float clear = fabsf(least) > 1e-20f && fabsf(least) < 1e20f && temperature < 1e8f ? least - fabsf(least) * 1e-5f : -INFINITY;
            // ---- collect what is not below the bound -------------------------------
            auto collect = [&](float x, uint32_t i) {
                if (!(x >= clear)) return;
                const int at = atomicAdd(&n_cand_s, 1);
                if (at < kCand) { cand_x[at] = x; cand_i[at] = (int)i; }
            };
            if constexpr (kStaged) {
                const uint32_t off = skew / (uint32_t)sizeof(T);
#pragma unroll 4
                for (uint32_t g = tid; g < n_granules; g += kThreads) {
                    float x[kG];
                    Granule<T>::load(staged_s + 16u * g, x);
                    if (largest<kG>(x) >= clear) {
#pragma unroll
                        for (int e = 0; e < kG; ++e)
                            if (g * kG + e - off < n_row) collect(x[e], g * kG + e - off);      // (unsigned: below the row counts as beyond)
                    }
                }
            } else {
                walk<kFlight>(row, tid, n_row, kThreads, collect);
            }
            __syncthreads();
            const int n = n_cand_s;
            if (n <= kCand) {
                // Scaled as the reference does; what only `clear` let through is below at least k
                // others and falls out with them.
                for (int c = tid; c < n; c += kThreads) cand_x[c] = scaled(cand_x[c]);
                const int n4 = (n + 3) & ~3;                // (whole fours: beyond n is below everything)
                if (tid < n4 - n) { cand_x[n + tid] = -INFINITY; cand_i[n + tid] = 0x7fffffff; }
                __syncthreads();
                // An entry's place in index order and how many are greater, by counting: as many
                // threads to an entry as there are, each taking every `share`-th four others.
                int share = 32;
                while (share > 1 && (n * share > kThreads || 2 * share > n)) share >>= 1;
                const int sub = tid & (share - 1), per_round = kThreads / share;
                int idx[kPer], tally[kPer];                 // place | greater << 16
                float w[kPer];
#pragma unroll
                for (int e = 0; e < kPer; ++e) {
                    const int at = tid / share + e * per_round;
                    const bool valid = at < n;
                    const float x = valid ? cand_x[at] : INFINITY;
                    idx[e] = valid ? cand_i[at] : 0;
                    int t = 0;
                    if (valid) {
#pragma unroll 2
                        for (int c = 4 * sub; c < n; c += 4 * share) {
                            const float4 xs = *reinterpret_cast<const float4*>(cand_x + c);
                            const int4 is = *reinterpret_cast<const int4*>(cand_i + c);
                            t += (is.x < idx[e]) + (is.y < idx[e]) + (is.z < idx[e]) + (is.w < idx[e]);
                            t += (xs.x > x ? 65536 : 0) + (xs.y > x ? 65536 : 0) + (xs.z > x ? 65536 : 0) + (xs.w > x ? 65536 : 0);
                        }
                    }
                    for (int o = share >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                    tally[e] = t;
                    w[e] = x;
                }
                __syncthreads();                            // all have read the unsorted entries
#pragma unroll
                for (int e = 0; e < kPer; ++e)
                    if (sub == 0 && tid / share + e * per_round < n) {
                        cand_i[tally[e] & 0xffff] = idx[e];
                        cand_w[tally[e] & 0xffff] = (tally[e] >> 16) < top_k ? (double)expf(w[e] - m) : 0.0;
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
                    const int at = !(total > 0.0) || total == INFINITY ? -1 : pick >= 0 ? pick : last_kept;
                    const int id = at >= 0 ? cand_i[at] : argmax_index();                       // (the same for the whole warp)
                    if (lane == 0) ids[blockIdx.x] = id;
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
    if (warp == 0) {
        const int id = pick_s >= 0 ? pick_s : argmax_index();
        if (lane == 0) ids[blockIdx.x] = id;
    }
    }
}

}  // namespace

// Threads per row.  A CTA of 1024 threads fills an SM, one of 512 a third, one of 256 an
// eighth: up to one row per SM the row's length decides (as many loads in flight as it can
// use; past that, barriers and folds cost more than the walk), with more rows than that
// the rows side by side do.  Measured with 256 / 512 / 1024 threads, us, fp32:
//   1 row, drawn from the whole row: 1000 entries 4.0 / 3.7 / 4.1, 10000 12 / 7.6 / 8.4, 50257 41 / 16 / 15
//   256 rows x 32000, the same: 41 / 27 / 31; argmax 7.0 / 6.4 / 7.3
//   1024 rows x 1000: 7.9 / 12 / 26; argmax 3.5 / 5.2 / 11
// A top-k cut from candidates wants 5k/2 threads (64 rows x 2048, k = 200: 23 / 9.5 / 9.1,
// k = 400: 25 / 25 / 17) and gets them unless that leaves rows waiting for a place; short
// rows in crowds do as well with the radix select (1024 x 1000, k = 200: 31, and 30 with 512).
static int sample_threads(int batch, int vocab, int cut) {
    const int sms = num_sms();
    const int walk = batch <= sms ? (vocab <= 2048 ? 256 : vocab <= 16384 ? 512 : 1024) : batch <= 3 * sms && vocab > 8192 ? 512 : 256;
    const int ranking = cut <= cut_limit(256) ? 256 : cut <= cut_limit(512) ? 512 : cut <= cut_limit(1024) ? 1024 : 0;
    if (ranking > walk && (batch <= sms || (ranking == 512 && (batch <= 3 * sms || vocab > 2048)))) return ranking;
    return walk;
}

// Rows that fit the shared memory of an SM are staged there when every row has an SM of its
// own and the row is long enough.  Threads take a staged row 16 bytes at a time, so a short one
// leaves threads without an entry, and with fewer maxima than the cut keeps there is no bound:
// every entry is a candidate.  us for 32 rows, staged / from memory: k = 20 of 2049 bf16 entries
// 30.3 / 4.8, k = 300 of 1000 28.1 / 10.8.  Where there is a bound, waiting for the copies
// costs more than loads in flight until the row outgrows those: k = 50 of 24000 fp32 entries
// 9.05 / 8.37, of 40000 9.44 / 9.50, of 106000 bf16 a tenth less.  Draws and the radix select,
// which walk the row more often: 2049 entries 5.06 / 4.73, 4500 7.4 / 7.4, 13000 10.8 / 11.7.
constexpr size_t kStagedBytes = 208 * 1024;
constexpr int kStagedFromCut = 40000, kStagedFrom = 4096;

template <typename T, int kThreads, Choice kChoice>
static cudaError_t allow_staged() {
    static std::atomic<bool> done[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    e = cudaFuncSetAttribute(sample_kernel<T, kThreads, kChoice, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStagedBytes);
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    return e;
}

template <typename T, int kThreads>
static cudaError_t launch_sample(const T* logits, int batch, int vocab, int64_t row_stride, float temperature, int top_k, int do_sample,
                                 uint64_t seed, uint64_t step, int64_t* ids, cudaStream_t st) {
    auto go = [&](auto kernel, size_t smem) { return launch(kernel, dim3((unsigned)batch), kThreads, smem, st, true, logits, vocab, row_stride, temperature, top_k, seed, step, ids); };
    if (!do_sample) return go(sample_kernel<T, kThreads, Choice::kArgmax, false>, 0);
    auto pick = [&](auto choice) {
        constexpr Choice c = decltype(choice)::value;
        if constexpr (kThreads > 256) {
            const size_t bytes = ((size_t)vocab * sizeof(T) + 32) / 16 * 16;           // whole 16 bytes at any offset
            if (batch <= num_sms() && bytes <= kStagedBytes && vocab >= (c == Choice::kTopK ? kStagedFromCut : kStagedFrom)) {
                if (cudaError_t e = allow_staged<T, kThreads, c>(); e != cudaSuccess) return e;
                return go(sample_kernel<T, kThreads, c, true>, bytes);
            }
        }
        return go(sample_kernel<T, kThreads, c, false>, 0);
    };
    if (top_k == 0) return pick(std::integral_constant<Choice, Choice::kDraw>{});
    if (top_k <= cut_limit(kThreads)) return pick(std::integral_constant<Choice, Choice::kTopK>{});
    return pick(std::integral_constant<Choice, Choice::kTopKRadix>{});
}

int sample_fault_word(int* out) {
    KIVI_CUDA_OK(cudaMemcpyFromSymbol(out, g_sample_fault, sizeof(int)));
    return KIVI_OK;
}
int sample_fault_clear() {
    const int zero = 0;
    KIVI_CUDA_OK(cudaMemcpyToSymbol(g_sample_fault, &zero, sizeof(int)));
    return KIVI_OK;
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

// bsg_swaptions.cu -- sm_103a kernels of the swaption Monte Carlo (HJM).
//
// P3ARSEC's swaptions application prices every swaption with
// HJM_Swaption_Blocking (parsec-ff/pkgs/apps/swaptions/src/
// HJM_Swaption_Blocking.cpp:19-223), one swaption per FastFlow worker
// iteration (HJM_Securities.cpp:312-323), trials in blocks on one core.  Here
// one launch prices every swaption: persistent blocks whose warps take the next
// paths of the next swaption from a queue, one path a lane at a time, in 64-bit
// fixed point and doubles, to the double precision of the reference's FTYPE.
//
// Per path (the driver's arithmetic, HJM_Swaption_Blocking.cpp:160-204, on
// a discrete HJM model in the time-to-maturity parameterisation):
//   f(t_{i+1}, t_{i+1+m}) = f(t_i, t_{i+1+m}) + mu[m] h + sqrt(h) sum_k v_k[m] z_ik
//   D     = exp(-h sum_{i<s} f(t_i, t_i))               discount to maturity t_s
//   V     = sum_l pay[l] exp(-h sum_{m<l} f(t_s, t_{s+m}))   fixed leg at t_s
//   price = mean of max(V - 1, 0) D,  error = the reference's standard error
// with mu[m] = (h/2) sum_k (S_k(m)^2 - S_k(m-1)^2) (S_k: running sums of
// factor k's vols), the drift that makes discounted bonds martingales.
//
// The path rows are linear in the variates, so the rows themselves are not
// formed: the exponent of each payment's discount factor (and of D) is a
// constant plus a coefficient times each variate up to maturity, the
// coefficients differences of the S_k (swaption_setup in bsg_api.cu).  The
// variates are the ones a full-path simulation with the same stream draws:
// a counter-based generator (Philox4x32-10, Salmon et al., SC'11) keyed by
// (seed, trial, index), turned normal by Box-Muller.
//
// What bounds it: in doubles the FP64 rate (2 operations a clock and SM):
// 33.1 ms for 128 swaptions x 1M paths with 130 FP64 operations a path, that
// pipe 85 % busy.  So the variates, the exponents and the powers of two are
// 64-bit fixed point (bsg_swmath.h), and FP64 is left with a payment's
// multiply-add, the floor and the two sums, 4 to 6 operations a path: 5.28 ms.
// Its bound is the pipe that takes the integer multiply-adds (two thirds busy,
// 170 of them a path, 40 in the generator).  Four blocks of 64 registers an SM:
// 5.34 ms, three of 80 5.53, two of 128 5.54.  With warps that take their own
// work (below) instead of blocks: 4.74 ms.
//
// Reduction: each warp reduces its paths' sums (sum and sum of squares of
// the discounted payoff) in a fixed order to one part; the warp that finishes
// a group of parts, and then a swaption, last adds them up in a fixed order.
// Which paths a part covers and how parts are grouped depends on the number of
// trials alone: two runs, and a swaption alone or among others, give the same
// bits.
#include "bsg_internal.h"
#include "bsg_swmath.h"

#include <math.h>

#include <algorithm>
#include <type_traits>

namespace bsg {

namespace {

constexpr int kSwThreads = 256;
constexpr int kSwWarps = kSwThreads / 32;

// How many of a swaption's parts one warp adds up before the swaption's last
// warp adds up the groups' sums: all of up to 256 (eight loads a lane, at once),
// else 32.  16 swaptions x 5,000 paths (160 parts): 38.9 us in groups of 32,
// 37.9 in one; x 20,000 (632): 52.0 in groups of 32, 53.8 of 256.
__host__ __device__ __forceinline__ unsigned group_size(uint64_t parts) { return parts <= 256 ? 256 : 32; }
__host__ __device__ __forceinline__ uint64_t group_count(uint64_t parts) {
    return parts <= 256 ? 1 : (parts + 31) / 32;
}
constexpr int kHeadWords = sizeof(SwHead) / sizeof(uint64_t);

__device__ __forceinline__ void philox4x32_10(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                              uint32_t k0, uint32_t k1, uint32_t out[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * x0, hi0 = __umulhi(0xD2511F53u, x0);
        const uint32_t lo1 = 0xCD9E8D57u * x2, hi1 = __umulhi(0xCD9E8D57u, x2);
        const uint32_t y0 = hi1 ^ x1 ^ k0, y2 = hi0 ^ x3 ^ k1;
        x0 = y0;
        x1 = lo1;
        x2 = y2;
        x3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    out[0] = x0;
    out[1] = x1;
    out[2] = x2;
    out[3] = x3;
}

__device__ const bsg_sw::Tables kSwTables = BSG_SW_TABLES;

// Copies the tables of bsg_swmath.h into shared memory (all threads of the block).
__device__ __forceinline__ void load_tables(bsg_sw::Tables& dst) {
    static_assert(sizeof(bsg_sw::Tables) % sizeof(double2) == 0, "copied in 16-byte words");
    const double2* src = reinterpret_cast<const double2*>(&kSwTables);
    double2* d = reinterpret_cast<double2*>(&dst);
    for (int i = threadIdx.x; i < (int)(sizeof(bsg_sw::Tables) / sizeof(double2)); i += blockDim.x)
        d[i] = src[i];
}

// What a block keeps in shared memory: the tables, and the swaptions when
// they came with the launch.
template <bool INLINE>
struct SwShared {
    bsg_sw::Tables nt;
    uint64_t words[INLINE ? kSwInlineWords : 1];
};

__device__ __forceinline__ double as_double(uint64_t u) { return __longlong_as_double((long long)u); }

// The payoff of trial t of the swaption with head hd and these words (pays,
// constants, coefficients; bsg_internal.h), less its constant discount.
// NP: the number of exponents, or with GUARD an upper bound of it.
template <int NP, bool GUARD>
__device__ __forceinline__ double path_payoff(const bsg_sw::Tables& nt, const SwHead& hd,
                                              const uint64_t* words, uint64_t t) {
    const int np = GUARD ? hd.n_exp : NP;
    const uint64_t* c0 = words + np;
    const uint64_t* g = words + 2 * np;
    uint64_t x[NP], half = 0;
#pragma unroll
    for (int l = 0; l < NP; ++l) x[l] = (!GUARD || l < np) ? c0[l] : 0;
    // coefficients g = G 2^-63 and variates z = Z 2^-58 enter as G + 2^63 and
    // Z + 2^62 (swaption_setup's constants take that out again)
    auto take = [&](int64_t z) {
        const uint64_t zu = (uint64_t)z + (1ull << 62);
        half += zu >> 1;
#pragma unroll
        for (int l = 0; l < NP; ++l)
            if (!GUARD || l < np) x[l] += bsg_sw::mulhi(g[l], zu);
        g += np;
    };
    const int nz = hd.n_normals;
#pragma unroll 1
    for (int i = 0; i < nz; i += 2) {
        uint32_t w[4];
        philox4x32_10((uint32_t)t, (uint32_t)(t >> 32), (uint32_t)(i >> 1), 0u, (uint32_t)hd.seed,
                      (uint32_t)(hd.seed >> 32), w);
        int64_t z0, z1;
        if (i + 1 < nz) {
            bsg_sw::normal_pair_fixed<true>(nt, w[0], w[1], w[2], w[3], &z0, &z1);
            take(z0);
            take(z1);
        } else {
            bsg_sw::normal_pair_fixed<false>(nt, w[0], w[1], w[2], w[3], &z0, &z1);
            take(z0);
        }
    }
    // the payments' discount factors, then the path's own if it varies
    const int pays = hd.n_exp - hd.disc_varies;
    double v = -1.0, disc = 1.0;
#pragma unroll
    for (int l = 0; l < NP; ++l)
        if (!GUARD || l < np) {
            const double y = bsg_sw::exp2_fixed(nt, (int64_t)(x[l] - half));
            if (l < pays) v = __fma_rn(as_double(words[l]), y, v);
            else disc = y;
        }
    return v > 0.0 ? __dmul_rn(v, disc) : 0.0;
}

// The same in double precision, for exponents outside the fixed-point range:
// words hold the constants and coefficients as doubles, natural exponents.
__device__ __noinline__ double path_payoff_wide(const bsg_sw::Tables& nt, const SwHead& hd,
                                                const uint64_t* words, uint64_t t) {
    const int np = hd.n_exp, nz = hd.n_normals, pays = np - hd.disc_varies;
    double v = -1.0, disc = 1.0;
    for (int l = 0; l < np; ++l) {
        double x = as_double(words[np + l]), z[2];
        for (int i = 0; i < nz; ++i) {
            if ((i & 1) == 0) {
                uint32_t w[4];
                philox4x32_10((uint32_t)t, (uint32_t)(t >> 32), (uint32_t)(i >> 1), 0u,
                              (uint32_t)hd.seed, (uint32_t)(hd.seed >> 32), w);
                bsg_sw::normal_pair(nt, w[0], w[1], w[2], w[3], &z[0], &z[1]);
            }
            x = __fma_rn(as_double(words[2 * np + i * np + l]), z[i & 1], x);
        }
        const double y = bsg_sw::exp_(nt, x);
        if (l < pays) v = __fma_rn(as_double(words[l]), y, v);
        else disc = y;
    }
    return v > 0.0 ? __dmul_rn(v, disc) : 0.0;
}

// A warp's two sums in a fixed order: the lower half of the warp adds up a,
// the upper half b.
__device__ __forceinline__ double2 warp_sums(double a, double b) {
    const bool low = (threadIdx.x & 31) < 16;
    const double give = low ? b : a, keep = low ? a : b;
    double v = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, 16));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    return make_double2(v, __shfl_sync(0xffffffffu, v, 16));  // lane 0's are the sums
}

// The sums of a warp's per_thread paths a lane from trial t on, kSwThreads apart.
template <int NP, bool GUARD, bool WIDE>
__device__ __forceinline__ double2 sum_paths(const bsg_sw::Tables& nt, const SwHead& hd, const uint64_t* words,
                                             uint64_t t, int per_thread, uint64_t trials) {
    double sum = 0.0, sum_sq = 0.0;
#pragma unroll 1
    for (int q = 0; q < per_thread && t < trials; ++q, t += kSwThreads) {
        const double dp = WIDE ? path_payoff_wide(nt, hd, words, t) : path_payoff<NP, GUARD>(nt, hd, words, t);
        sum = __dadd_rn(sum, dp);
        sum_sq = __fma_rn(dp, dp, sum_sq);
    }
    __syncwarp();
    return warp_sums(sum, sum_sq);
}

// Lane 0's value v to *at; true in the warp that is the last of `of` to come
// here with this counter, which then sees all their values and leaves it zero.
__device__ __forceinline__ bool last_of(unsigned lane, double2* at, double2 v, unsigned* counter, unsigned of) {
    unsigned before = 0;
    if (lane == 0) {
        *at = v;
        __threadfence();
        before = atomicAdd(counter, 1u);
        if (before == of - 1) *counter = 0;
    }
    if (__shfl_sync(0xffffffffu, before, 0) != of - 1) return false;
    __threadfence();
    return true;
}

// The sum of p[0 .. n) in a fixed order, eight loads a lane in flight.
__device__ __forceinline__ double2 sum_parts(unsigned lane, const double2* p, unsigned n) {
    double a = 0.0, b = 0.0;
#pragma unroll 8
    for (unsigned i = lane; i < n; i += 32) {
        const double2 v = __ldcg(p + i);
        a = __dadd_rn(a, v.x);
        b = __dadd_rn(b, v.y);
    }
    return warp_sums(a, b);
}

// Persistent blocks whose warps each take the next 32 x per_thread paths from
// a queue: no warp waits for another, and what is left over at the end is a
// part's work, not a block's.  Blocks that took 256 x per_thread paths at a
// time, with a barrier on either side, spent a quarter of a round of one path
// per thread outside the paths, and a round more for a remainder: 16 swaptions
// x 20,000 paths 56 -> 52 us, x 80,000 139 -> 93, 64 x 100,000 494 -> 361, 128 x
// 1M 5.17 -> 4.74 ms.  (Counting a part only when the next is done, so that the
// warp does not wait for its store, took more registers: 4.88 ms.)
// LARGE: also swaptions of more than four exponents or outside the fixed-point
// range (their registers would cost the others two blocks per SM).  INLINE:
// the table came in the launch's parameters.
template <bool LARGE, bool INLINE>
__global__ void __launch_bounds__(kSwThreads, LARGE ? 2 : 4) swaption_paths_kernel(
    const __grid_constant__ SwInline in, const uint64_t* __restrict__ table, int nsw, uint64_t trials,
    int per_thread, uint64_t nparts, double2* __restrict__ partial, unsigned* __restrict__ done,
    unsigned long long* queue, double2* __restrict__ sums, unsigned* count, unsigned* flag, unsigned seq) {
    __shared__ SwShared<INLINE> sh;
    load_tables(sh.nt);
    if (INLINE)
        for (int i = threadIdx.x; i < kSwInlineWords; i += kSwThreads) sh.words[i] = in.words[i];
    __syncthreads();
    const uint64_t* tab = INLINE ? sh.words : table;
    const unsigned lane = threadIdx.x & 31;
    // an item: 32 x per_thread paths, one part of one swaption's sums
    using Item = typename std::conditional<LARGE, uint64_t, uint32_t>::type;
    using Take = typename std::conditional<LARGE, unsigned long long, unsigned>::type;
    const Item parts = (Item)nparts, items = parts * (Item)nsw;
    for (Item item = blockIdx.x * kSwWarps + (threadIdx.x >> 5); item < items;) {
        // asked for now, looked at when this item is done
        Item next = 0;
        if (lane == 0) next = (Item)atomicAdd(reinterpret_cast<Take*>(queue), (Take)1);
        const uint64_t* words;
        uint64_t t;
        {
            const Item sw = item / parts, part = item - sw * parts;
            t = (uint64_t)(part / kSwWarps) * per_thread * kSwThreads + (part % kSwWarps) * 32 + lane;
            words = tab + (uint64_t)sw * kHeadWords;
        }
        const SwHead& hd = *reinterpret_cast<const SwHead*>(words);
        words = tab + hd.words_at;
        double2 v;
        if (LARGE && hd.wide) {
            v = sum_paths<1, true, true>(sh.nt, hd, words, t, per_thread, trials);
        } else {
            switch (hd.n_exp) {
                case 1: v = sum_paths<1, false, false>(sh.nt, hd, words, t, per_thread, trials); break;
                case 2: v = sum_paths<2, false, false>(sh.nt, hd, words, t, per_thread, trials); break;
                case 3: v = sum_paths<3, false, false>(sh.nt, hd, words, t, per_thread, trials); break;
                default:
                    if (!LARGE || hd.n_exp == 4)
                        v = sum_paths<4, false, false>(sh.nt, hd, words, t, per_thread, trials);
                    else if (hd.n_exp <= 8)
                        v = sum_paths<8, true, false>(sh.nt, hd, words, t, per_thread, trials);
                    else
                        v = sum_paths<kSwMaxExp, true, false>(sh.nt, hd, words, t, per_thread, trials);
            }
        }
        v = make_double2(__dmul_rn(v.x, hd.disc), __dmul_rn(v.y, __dmul_rn(hd.disc, hd.disc)));
        const Item sw = item / parts, part = item - sw * parts;
        // the warp that finishes a group of parts adds them up, the one that
        // finishes a swaption's last group adds the groups up
        const unsigned size = group_size(parts);
        const Item groups = (Item)group_count(parts), group = part / size;
        double2* mine = partial + (uint64_t)sw * (parts + groups);
        unsigned* left = done + (uint64_t)sw * (groups + 1);
        const unsigned in_group = group + 1 < groups ? size : (unsigned)(parts - size * group);
        item = (Item)(gridDim.x * kSwWarps) + __shfl_sync(0xffffffffu, next, 0);
        if (!last_of(lane, mine + part, v, left + group, in_group)) continue;
        v = sum_parts(lane, mine + size * group, in_group);
        if (groups > 1) {
            if (!last_of(lane, mine + parts + group, v, left + groups, (unsigned)groups)) continue;
            v = sum_parts(lane, mine + parts, (unsigned)groups);
        }
        if (lane == 0) {
            sums[sw] = v;
            signal_host(count, (unsigned)nsw, flag, seq, queue);
        }
    }
}

__global__ void __launch_bounds__(kSwThreads) swaption_normals_kernel(const uint32_t* __restrict__ words,
                                                                      uint64_t n, double* __restrict__ z) {
    __shared__ bsg_sw::Tables nt;
    load_tables(nt);
    __syncthreads();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        bsg_sw::normal_pair(nt, words[4 * i], words[4 * i + 1], words[4 * i + 2], words[4 * i + 3],
                            &z[2 * i], &z[2 * i + 1]);
}

}  // namespace

cudaError_t launch_swaption_normals(const uint32_t* words, uint64_t n, double* z, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const uint64_t blocks = std::min<uint64_t>((n + kSwThreads - 1) / kSwThreads, 4096);
    swaption_normals_kernel<<<(unsigned)blocks, kSwThreads, 0, st>>>(words, n, z);
    return cudaGetLastError();
}

int swaption_per_thread(uint64_t trials) {
    int q = 1;
    while (q < 1024 && (trials + 2 * q * kSwThreads - 1) / ((uint64_t)2 * q * kSwThreads) >= 304) q *= 2;
    return q;
}

uint64_t swaption_chunks(uint64_t trials) {
    const uint64_t per_block = (uint64_t)swaption_per_thread(trials) * kSwThreads;
    return (trials + per_block - 1) / per_block;
}

size_t swaption_partial_bytes(int nsw, uint64_t trials) {
    const size_t parts = swaption_chunks(trials) * kSwWarps;
    return (size_t)nsw * (parts + group_count(parts)) * sizeof(double2);
}

size_t swaption_counters(int nsw, uint64_t trials) {
    return (size_t)nsw * (group_count(swaption_chunks(trials) * kSwWarps) + 1);
}

cudaError_t launch_swaptions(const SwInline& in, const uint64_t* table, int nsw, bool large,
                             uint64_t trials, void* partial, unsigned* done, unsigned long long* queue,
                             double2* sums, unsigned* count, unsigned* flag, unsigned seq, int sm_count,
                             cudaStream_t st) {
    if (nsw <= 0 || trials < 2) return cudaErrorInvalidValue;
    const uint64_t chunks = swaption_chunks(trials);
    large = large || chunks * kSwWarps * nsw >> 31;  // counts items in 64 bits
    const unsigned grid = (unsigned)std::min<uint64_t>(chunks * nsw, (uint64_t)sm_count * (large ? 2 : 4));
    auto* kernel = large ? (table ? swaption_paths_kernel<true, false> : swaption_paths_kernel<true, true>)
                         : (table ? swaption_paths_kernel<false, false> : swaption_paths_kernel<false, true>);
    kernel<<<grid, kSwThreads, 0, st>>>(in, table, nsw, trials, swaption_per_thread(trials),
                                        chunks * kSwWarps, static_cast<double2*>(partial), done, queue, sums,
                                        count, flag, seq);
    return cudaGetLastError();
}

}  // namespace bsg

// bsg_swaptions.cu -- sm_103a kernels of the swaption Monte Carlo (HJM).
//
// P3ARSEC's swaptions application prices every swaption with
// HJM_Swaption_Blocking (parsec-ff/pkgs/apps/swaptions/src/
// HJM_Swaption_Blocking.cpp:19-223), one swaption per FastFlow worker
// iteration (HJM_Securities.cpp:312-323), trials in blocks on one core.  Here
// one launch prices every swaption: a grid of (trial chunk, swaption) blocks,
// one path per thread at a time, in double precision as the reference's
// FTYPE.
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
// 5.34 ms, three of 80 5.53, two of 128 5.54.
//
// Reduction: each warp reduces its paths' sums (sum and sum of squares of
// the discounted payoff) in a fixed order and writes one partial; the block
// that finishes a swaption last adds its partials in a fixed order.  Which
// paths a partial covers depends on the number of trials alone: two runs, and
// a swaption alone or among others, give the same bits.
#include "bsg_internal.h"
#include "bsg_swmath.h"

#include <math.h>

#include <algorithm>

namespace bsg {

namespace {

constexpr int kSwThreads = 256;
constexpr int kSwWarps = kSwThreads / 32;

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

// One swaption in shared memory: its head and its words (pays, constants,
// coefficients; bsg_internal.h).  Swaptions of up to four exponents have at
// most 4 (2 + 8 x 31) words.
template <bool LARGE>
struct SwShared {
    bsg_sw::Tables nt;
    SwHead head;
    uint64_t words[LARGE ? kSwMaxWords : 1000];
    double red[2][kSwWarps];
    int last;
};

__device__ __forceinline__ double as_double(uint64_t u) { return __longlong_as_double((long long)u); }

// The payoff of trial t of the swaption in sh, less its constant discount.
// NP: the number of exponents, or with GUARD an upper bound of it.
template <int NP, bool GUARD, typename Sh>
__device__ __forceinline__ double path_payoff(const Sh& sh, uint64_t t) {
    const SwHead& hd = sh.head;
    const int np = GUARD ? hd.n_exp : NP;
    const uint64_t* c0 = sh.words + np;
    const uint64_t* g = sh.words + 2 * np;
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
            bsg_sw::normal_pair_fixed<true>(sh.nt, w[0], w[1], w[2], w[3], &z0, &z1);
            take(z0);
            take(z1);
        } else {
            bsg_sw::normal_pair_fixed<false>(sh.nt, w[0], w[1], w[2], w[3], &z0, &z1);
            take(z0);
        }
    }
    // the payments' discount factors, then the path's own if it varies
    const int pays = hd.n_exp - hd.disc_varies;
    double v = -1.0, disc = 1.0;
#pragma unroll
    for (int l = 0; l < NP; ++l)
        if (!GUARD || l < np) {
            const double y = bsg_sw::exp2_fixed(sh.nt, (int64_t)(x[l] - half));
            if (l < pays) v = __fma_rn(as_double(sh.words[l]), y, v);
            else disc = y;
        }
    return v > 0.0 ? __dmul_rn(v, disc) : 0.0;
}

// The same in double precision, for exponents outside the fixed-point range:
// words hold the constants and coefficients as doubles, natural exponents.
template <typename Sh>
__device__ __noinline__ double path_payoff_wide(const Sh& sh, uint64_t t) {
    const SwHead& hd = sh.head;
    const int np = hd.n_exp, nz = hd.n_normals, pays = np - hd.disc_varies;
    double v = -1.0, disc = 1.0;
    for (int l = 0; l < np; ++l) {
        double x = as_double(sh.words[np + l]), z[2];
        for (int i = 0; i < nz; ++i) {
            if ((i & 1) == 0) {
                uint32_t w[4];
                philox4x32_10((uint32_t)t, (uint32_t)(t >> 32), (uint32_t)(i >> 1), 0u,
                              (uint32_t)hd.seed, (uint32_t)(hd.seed >> 32), w);
                bsg_sw::normal_pair(sh.nt, w[0], w[1], w[2], w[3], &z[0], &z[1]);
            }
            x = __fma_rn(as_double(sh.words[2 * np + i * np + l]), z[i & 1], x);
        }
        const double y = bsg_sw::exp_(sh.nt, x);
        if (l < pays) v = __fma_rn(as_double(sh.words[l]), y, v);
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

// Chunks [chunk, end) of the swaption in sh: one partial per warp and chunk.
template <int NP, bool GUARD, bool WIDE, typename Sh>
__device__ __forceinline__ void sum_chunks(const Sh& sh, uint64_t chunk, uint64_t end, int per_thread,
                                           uint64_t trials, double2* partial) {
#pragma unroll 1
    for (; chunk < end; ++chunk) {
        double sum = 0.0, sum_sq = 0.0;
        uint64_t t = chunk * per_thread * kSwThreads + threadIdx.x;
#pragma unroll 1
        for (int q = 0; q < per_thread && t < trials; ++q, t += kSwThreads) {
            const double dp = WIDE ? path_payoff_wide(sh, t) : path_payoff<NP, GUARD>(sh, t);
            sum = __dadd_rn(sum, dp);
            sum_sq = __fma_rn(dp, dp, sum_sq);
        }
        const double2 v = warp_sums(sum, sum_sq);
        const double d = sh.head.disc;
        if ((threadIdx.x & 31) == 0)
            partial[chunk * kSwWarps + (threadIdx.x >> 5)] =
                make_double2(__dmul_rn(v.x, d), __dmul_rn(v.y, __dmul_rn(d, d)));
    }
}

// Persistent blocks over (swaption, `span` consecutive chunks of per_thread x
// 256 paths).  LARGE: also swaptions of more than four exponents or outside
// the fixed-point range (their registers would cost the others a block per SM).
template <bool LARGE>
__global__ void __launch_bounds__(kSwThreads, LARGE ? 2 : 4) swaption_paths_kernel(
    const __grid_constant__ SwInline in, const uint64_t* __restrict__ table, int nsw, uint64_t trials,
    int per_thread, uint64_t chunks, unsigned span, double2* __restrict__ partial,
    unsigned* __restrict__ done, double* __restrict__ out, unsigned* count, unsigned* flag, unsigned seq) {
    __shared__ SwShared<LARGE> sh;
    load_tables(sh.nt);
    const uint64_t spans = (chunks + span - 1) / span, items = spans * (uint64_t)nsw;
    for (uint64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint64_t sw = item / spans, chunk = (item - sw * spans) * span;
        const uint64_t end = chunk + span < chunks ? chunk + span : chunks;
        __syncthreads();  // the previous item's reads of sh are done
        {
            // head, then its words (from the launch's parameters when they all fit there)
            constexpr int hw = (int)(sizeof(SwHead) / 8);
            const uint64_t* tab = table ? table : in.words;
            uint64_t* hd = reinterpret_cast<uint64_t*>(&sh.head);
            if (threadIdx.x < hw) hd[threadIdx.x] = tab[sw * hw + threadIdx.x];
            __syncthreads();
            const uint64_t* src = tab + sh.head.words_at;
            for (int i = threadIdx.x; i < sh.head.n_words; i += kSwThreads) sh.words[i] = src[i];
        }
        __syncthreads();
        double2* part = partial + sw * chunks * kSwWarps;
        if (LARGE && sh.head.wide) {
            sum_chunks<1, true, true>(sh, chunk, end, per_thread, trials, part);
        } else {
            switch (sh.head.n_exp) {
                case 1: sum_chunks<1, false, false>(sh, chunk, end, per_thread, trials, part); break;
                case 2: sum_chunks<2, false, false>(sh, chunk, end, per_thread, trials, part); break;
                case 3: sum_chunks<3, false, false>(sh, chunk, end, per_thread, trials, part); break;
                case 4: sum_chunks<4, false, false>(sh, chunk, end, per_thread, trials, part); break;
                default:
                    if constexpr (LARGE) {
                        if (sh.head.n_exp <= 8)
                            sum_chunks<8, true, false>(sh, chunk, end, per_thread, trials, part);
                        else
                            sum_chunks<kSwMaxExp, true, false>(sh, chunk, end, per_thread, trials, part);
                    }
            }
        }
        // the block that finishes the swaption's last chunk adds the partials up
        if ((threadIdx.x & 31) == 0) __threadfence();
        __syncthreads();
        if (threadIdx.x == 0)
            sh.last = atomicAdd(&done[sw], (unsigned)(end - chunk)) + (unsigned)(end - chunk) == (unsigned)chunks;
        __syncthreads();
        if (!sh.last) continue;
        __threadfence();
        double ta = 0.0, tb = 0.0;
        for (uint64_t i = threadIdx.x; i < chunks * kSwWarps; i += kSwThreads) {
            const double2 v = __ldcg(part + i);
            ta = __dadd_rn(ta, v.x);
            tb = __dadd_rn(tb, v.y);
        }
        const double2 v = warp_sums(ta, tb);
        if ((threadIdx.x & 31) == 0) {
            sh.red[0][threadIdx.x >> 5] = v.x;
            sh.red[1][threadIdx.x >> 5] = v.y;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double s1 = sh.red[0][0], s2 = sh.red[1][0];
            for (int w = 1; w < kSwWarps; ++w) {
                s1 = __dadd_rn(s1, sh.red[0][w]);
                s2 = __dadd_rn(s2, sh.red[1][w]);
            }
            // the mean and the reference's standard error (HJM_Swaption_Blocking.cpp:212-214)
            const double m = (double)trials;
            out[2 * sw] = s1 / m;
            out[2 * sw + 1] = sqrt((s2 - s1 * s1 / m) / (m - 1.0)) / sqrt(m);
            done[sw] = 0;  // ready for the next call
            signal_host(count, (unsigned)nsw, flag, seq);
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
    return (size_t)nsw * swaption_chunks(trials) * kSwWarps * sizeof(double2);
}

cudaError_t launch_swaptions(const SwInline& in, const uint64_t* table, int nsw, bool large,
                             uint64_t trials, void* partial, unsigned* done, double* out, unsigned* count,
                             unsigned* flag, unsigned seq, int sm_count, cudaStream_t st) {
    if (nsw <= 0 || trials < 2) return cudaErrorInvalidValue;
    const uint64_t chunks = swaption_chunks(trials), items = chunks * (uint64_t)nsw;
    const uint64_t room = (uint64_t)sm_count * (large ? 2 : 4);
    const int per_thread = swaption_per_thread(trials);
    // chunks per visit of a block: the fewer the better for the last wave, so
    // the most that leave 16 visits per block
    const unsigned span = (unsigned)std::min<uint64_t>(std::max<uint64_t>(items / (16 * room), 1), 16);
    const unsigned grid = (unsigned)std::min<uint64_t>((chunks + span - 1) / span * (uint64_t)nsw, room);
    double2* part = static_cast<double2*>(partial);
    if (large)
        swaption_paths_kernel<true><<<grid, kSwThreads, 0, st>>>(in, table, nsw, trials, per_thread, chunks,
                                                                 span, part, done, out, count, flag, seq);
    else
        swaption_paths_kernel<false><<<grid, kSwThreads, 0, st>>>(in, table, nsw, trials, per_thread, chunks,
                                                                  span, part, done, out, count, flag, seq);
    return cudaGetLastError();
}

}  // namespace bsg

// bsg_kernels.cu -- sm_103a kernels of the Black-Scholes map.
//
// The hot path is an HBM-bound elementwise map: 28 bytes per option per run
// (five float inputs, one int32 otype, one float price) against ~86 issued
// instructions (the FAST arithmetic runs two options per packed f32x2
// instruction).  Design:
//  * SoA streams read with 128-bit (v4) or 256-bit (v8) non-coherent loads
//    that do not allocate in L1, optionally inserted into L2 as evict_first
//    (a cyclic scan of a working set larger than L2 then keeps a slice of it
//    resident between passes), or with a prefix of the book (a tuned
//    fraction of the L2, inputs and prices) evict_last and the rest evict_first, so that
//    the prefix stays resident from pass to pass; prices stored with
//    streaming stores (or with the prefix's policy).
//  * Each thread loads VPT vector groups of all six arrays before computing,
//    so a warp keeps 6 * VPT independent 512/1024-byte requests in flight.
//  * Grid: one block per tile, or a persistent grid-stride loop sized in
//    multiples of the SM count (chosen by the autotuner).
//  * No shared memory, no tensor cores: there is no reuse to stage and no
//    contraction to run.
#include "bsg_fx64.h"
#include "bsg_internal.h"
#include "bsg_math.cuh"

#include <atomic>

namespace bsg {

// ------------------------------------------------------------ memory access
__device__ __forceinline__ unsigned long long evict_first_policy() {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ unsigned long long evict_last_policy() {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

template <int W>
struct Raw {
    uint32_t v[W];
};

// Load paths of the vector kernel: LP 0/2: ld.global.nc.L1::no_allocate
// (v4 / v8); LP 1 / 6: the same v4 / v8 loads with an L2 evict_first cache
// policy; LP 7: v8 loads and stores of a resident prefix of the book (the
// first `gres` groups, a tuned fraction of the L2) with an evict_last
// policy, the rest evict_first -- the prefix then stays in L2 from pass to
// pass while the rest streams through.
// LP 8: the v8 loads of LP 2 and stores with the default L2 policy, every
// other pass in reverse tile order (the L2 keeps what it saw last).
__host__ __device__ constexpr bool lp_resident(int lp) { return lp == 7; }
__host__ __device__ constexpr bool lp_hinted(int lp) { return lp == 1 || lp == 6 || lp == 7; }
__host__ __device__ constexpr bool lp_evict_first(int lp) { return lp == 1 || lp == 6; }
__host__ __device__ constexpr bool lp_v8(int lp) { return lp == 2 || lp == 6 || lp == 7 || lp == 8; }
__host__ __device__ constexpr bool lp_alternating(int lp) { return lp == 8; }

template <int W, int LP>
__device__ __forceinline__ Raw<W> ld_group(const void* p, unsigned long long pol) {
    Raw<W> r;
    if constexpr (W == 4) {
        if constexpr (LP == 1) {
            asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
                : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3])
                : "l"(p), "l"(pol));
        } else {
            (void)pol;
            asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3])
                : "l"(p));
        }
    } else if constexpr (lp_hinted(LP)) {
        asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;"
            : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]),
              "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
            : "l"(p), "l"(pol));
    } else {
        (void)pol;
        asm("ld.global.nc.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]),
              "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
            : "l"(p));
    }
    return r;
}

template <int W, int LP>
__device__ __forceinline__ void st_group(float* p, const float (&x)[W], unsigned long long pol) {
    if constexpr (W == 8 && lp_resident(LP)) {
        asm volatile("st.global.L2::cache_hint.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8}, %9;"
                     :: "l"(p), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]),
                        "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7]), "l"(pol)
                     : "memory");
    } else if constexpr (W == 8 && lp_alternating(LP)) {
        (void)pol;
        asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                     :: "l"(p), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]),
                        "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7])
                     : "memory");
    } else if constexpr (W == 4) {
        (void)pol;
        asm volatile("st.global.cs.v4.f32 [%0], {%1,%2,%3,%4};"
                     :: "l"(p), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3])
                     : "memory");
    } else {
        asm volatile("st.global.cs.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                     :: "l"(p), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]),
                        "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7])
                     : "memory");
    }
}


template <int M>
__device__ __forceinline__ void price_scalar(const SoA& a, int64_t i) {
    a.out[i] = price<M>(__ldg(a.s + i), __ldg(a.k + i), __ldg(a.r + i),
                        __ldg(a.v + i), __ldg(a.t + i), __ldg(a.ot + i));
}

// Prices vector groups [g0, g1) (group = W options) as thread `tid` of `bd`
// that share them: each loads VPT groups (stride bd) of all six arrays, then
// computes and stores them.  pol is the L2 policy of the hinted load paths;
// for LP 7, groups below gres use pol_res instead.
template <int M, int W, int VPT, int LP>
__device__ __forceinline__ void price_groups(const SoA& a, int64_t g0, int64_t g1,
                                             unsigned long long pol,
                                             unsigned long long pol_res, int64_t gres,
                                             unsigned tid, unsigned bd) {
    for (int64_t base = g0; base < g1; base += bd * VPT) {
        Raw<W> S[VPT], K[VPT], R[VPT], V[VPT], T[VPT], O[VPT];
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const int64_t g = base + tid + (int64_t)j * bd;
            if (g < g1) {
                const int64_t o = g * W;
                const unsigned long long pl = (lp_resident(LP) && g < gres) ? pol_res : pol;
                S[j] = ld_group<W, LP>(a.s + o, pl);
                K[j] = ld_group<W, LP>(a.k + o, pl);
                R[j] = ld_group<W, LP>(a.r + o, pl);
                V[j] = ld_group<W, LP>(a.v + o, pl);
                T[j] = ld_group<W, LP>(a.t + o, pl);
                O[j] = ld_group<W, LP>(a.ot + o, pl);
            }
        }
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const int64_t g = base + tid + (int64_t)j * bd;
            if (g < g1) {
                float p[W];
#pragma unroll
                for (int e = 0; e < W; e += 4) {
                    const float4 q = price4<M>(
                        make_float4(__uint_as_float(S[j].v[e]), __uint_as_float(S[j].v[e + 1]),
                                    __uint_as_float(S[j].v[e + 2]), __uint_as_float(S[j].v[e + 3])),
                        make_float4(__uint_as_float(K[j].v[e]), __uint_as_float(K[j].v[e + 1]),
                                    __uint_as_float(K[j].v[e + 2]), __uint_as_float(K[j].v[e + 3])),
                        make_float4(__uint_as_float(R[j].v[e]), __uint_as_float(R[j].v[e + 1]),
                                    __uint_as_float(R[j].v[e + 2]), __uint_as_float(R[j].v[e + 3])),
                        make_float4(__uint_as_float(V[j].v[e]), __uint_as_float(V[j].v[e + 1]),
                                    __uint_as_float(V[j].v[e + 2]), __uint_as_float(V[j].v[e + 3])),
                        make_float4(__uint_as_float(T[j].v[e]), __uint_as_float(T[j].v[e + 1]),
                                    __uint_as_float(T[j].v[e + 2]), __uint_as_float(T[j].v[e + 3])),
                        make_int4((int)O[j].v[e], (int)O[j].v[e + 1], (int)O[j].v[e + 2],
                                  (int)O[j].v[e + 3]));
                    p[e] = q.x;
                    p[e + 1] = q.y;
                    p[e + 2] = q.z;
                    p[e + 3] = q.w;
                }
                const unsigned long long pst = (lp_resident(LP) && g < gres) ? pol_res : pol;
                st_group<W, LP>(a.out + g * W, p, pst);
            }
        }
    }
}

// ------------------------------------------------------------- plain map
// Vector kernel: options [0, n - n % W) in groups of W; the last n % W
// options, and the `head` options before the (aligned) pointers, by block 0.  blocks_per_sm == 0: each block prices one tile of
// blockDim.x * VPT groups; otherwise blocks stride over tiles.
// Programmatic dependent launch: every block lets the next pass launch as
// soon as it starts (the next pass reads only the inputs, which no pass
// writes), and waits for the previous pass to complete only after its own
// stores, so a pass still completes after the one before it.  Both
// instructions are no-ops for a launch without the PDL attribute.
// Registers: one-group shapes (VPT = 1) are held to 64 per thread (1024
// threads per SM, no spills); more groups per thread need up to 128.  The
// reference-order libm mode (compute-bound, float-float exp/log) runs blocks of
// up to 256 threads (untuned contexts: 128), 1024 threads per SM (59
// registers, no spills).
__device__ __forceinline__ void pdl_trigger() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int M, int W, int VPT, int LP>
__global__ void __launch_bounds__(M == MODE_LIBM_REF ? 256 : 512,
                                  M == MODE_LIBM_REF ? 4 : (VPT == 1 ? 2 : 1))
    map_vec_kernel(SoA a, int64_t n, int head, int64_t gres, int rev) {
    pdl_trigger();
    const unsigned long long pol =
        (lp_evict_first(LP) || lp_resident(LP)) ? evict_first_policy() : 0ull;
    const unsigned long long pol_res = lp_resident(LP) ? evict_last_policy() : 0ull;
    const int64_t ngroups = n / W;
    const int64_t tile = (int64_t)blockDim.x * VPT;
    const int64_t ntiles = (ngroups + tile - 1) / tile;
    for (int64_t ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
        // LP 8's odd passes take the tiles from the last to the first
        const int64_t t0 = (lp_alternating(LP) && rev ? ntiles - 1 - ti : ti) * tile;
        const int64_t t1 = (t0 + tile < ngroups) ? t0 + tile : ngroups;
        price_groups<M, W, VPT, LP>(a, t0, t1, pol, pol_res, gres, threadIdx.x, blockDim.x);
    }
    if (blockIdx.x == 0) {
        const int64_t i = ngroups * W + threadIdx.x;
        if (i < n) price_scalar<M>(a, i);
        if ((int)threadIdx.x < head) price_scalar<M>(a, (int64_t)threadIdx.x - head);
    }
    pdl_wait();
}

// -------------------------------------------- several passes in one launch
// Short books: all `runs` passes of a book in one launch.  Each thread owns W
// neighbouring options and makes every pass over them in order, as a worker
// of the reference's bs_thread does over its range (blackscholes.c:607-658:
// NUM_RUNS over [start, end), no barrier between runs).  Every pass loads its
// inputs again (volatile loads; from L1 after the first), evaluates them and
// stores its prices.  U passes are in flight at once: their loads are issued
// together, then the U evaluations, whose chains of dependent operations
// (about 500 clocks each) overlap.
// What bounds a short book is that chain and the interval between dependent
// launches, not its bytes (65,536 options: 1.8 MB).  The whole call, 65,536
// options x 100 passes: 41 us (two options a thread and four passes in flight
// 45, one pass 58), 91 as a graph of programmatic launches, 212 as a graph of
// plain ones; 100 options: 27 (31, 47), 78, 155.  Of a host book of 65,536 pinned
// options x 100 passes a launch that first gathered it (14 us), the passes (29)
// and a copy of the prices took 65; with HOST, the kernel that does all three,
// 49; x 2, 40 and 30.
template <int W, bool OWN>  // OWN: written by this thread before
__device__ __forceinline__ Raw<W> ld_again(const void* p) {
    Raw<W> r;
    if constexpr (W == 1 && OWN)
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(r.v[0]) : "l"(p) : "memory");
    else if constexpr (W == 1)
        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(r.v[0]) : "l"(p));
    else if constexpr (W == 2 && OWN)
        asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(r.v[0]), "=r"(r.v[1]) : "l"(p) : "memory");
    else if constexpr (W == 2)
        asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(r.v[0]), "=r"(r.v[1]) : "l"(p));
    else if constexpr (OWN)
        asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]) : "l"(p) : "memory");
    else
        asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]) : "l"(p));
    return r;
}

template <int M>
__device__ __forceinline__ float2 price2(float2 s, float2 k, float2 r, float2 v, float2 t, int o0, int o1) {
    if constexpr (M == MODE_FAST) return price_fast2(s, k, r, v, t, o0, o1);
    else if constexpr (M == MODE_LIBM_REF) return price_libm_ref2(s, k, r, v, t, o0, o1);
    else return make_float2(price<M>(s.x, k.x, r.x, v.x, t.x, o0), price<M>(s.y, k.y, r.y, v.y, t.y, o1));
}

// W words from host memory (s + o) to device memory (d + o).
template <int W>
__device__ __forceinline__ void take_words(const void* s, const void* d, int64_t o) {
    using V = typename std::conditional<W == 1, uint32_t, typename std::conditional<W == 2, uint2, uint4>::type>::type;
    const uint32_t* from = static_cast<const uint32_t*>(s) + o;
    uint32_t* to = const_cast<uint32_t*>(static_cast<const uint32_t*>(d)) + o;
    if ((reinterpret_cast<uintptr_t>(s) & (4 * W - 1)) == 0) {
        *reinterpret_cast<V*>(to) = __ldg(reinterpret_cast<const V*>(from));
    } else {
        uint32_t x[W];
#pragma unroll
        for (int i = 0; i < W; ++i) x[i] = __ldg(from + i);
#pragma unroll
        for (int i = 0; i < W; ++i) to[i] = x[i];
    }
}

template <int W>
__device__ __forceinline__ void give_words(float* to, const float* p) {
    if ((reinterpret_cast<uintptr_t>(to) & (4 * W - 1)) == 0) {
        if constexpr (W == 1) *to = p[0];
        else if constexpr (W == 2) *reinterpret_cast<float2*>(to) = make_float2(p[0], p[1]);
        else *reinterpret_cast<float4*>(to) = make_float4(p[0], p[1], p[2], p[3]);
    } else {
#pragma unroll
        for (int i = 0; i < W; ++i) to[i] = p[i];
    }
}

// HOST: the book is the host's: each thread first brings its options into a
// (device arrays, aligned), and the last pass's prices go to the host too.
template <int M, int W, int U, bool HOST>
__global__ void __launch_bounds__(512, 1) map_runs_kernel(SoA a, int64_t n, int head, int runs,
                                                                        SoA host, Signal sig) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t o = g * W;
    if (o + W <= n) {
        if constexpr (HOST) {
            take_words<W>(host.s, a.s, o);
            take_words<W>(host.k, a.k, o);
            take_words<W>(host.r, a.r, o);
            take_words<W>(host.v, a.v, o);
            take_words<W>(host.t, a.t, o);
            take_words<W>(host.ot, a.ot, o);
        }
        for (int j = 0; j < runs; j += U) {
            Raw<W> S[U], K[U], R[U], V[U], T[U], O[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u < runs) {
                    S[u] = ld_again<W, HOST>(a.s + o);
                    K[u] = ld_again<W, HOST>(a.k + o);
                    R[u] = ld_again<W, HOST>(a.r + o);
                    V[u] = ld_again<W, HOST>(a.v + o);
                    T[u] = ld_again<W, HOST>(a.t + o);
                    O[u] = ld_again<W, HOST>(a.ot + o);
                }
            float p[U][W];
            // two evaluations at a time: neighbouring options, or (W = 1) an
            // option's neighbouring passes
            constexpr int kPassStep = W == 1 ? 2 : 1;
#pragma unroll
            for (int u = 0; u < U; u += kPassStep) {
#pragma unroll
                for (int e = 0; e < W; e += 2) {
                    const int u2 = W == 1 ? u + 1 : u, e2 = W == 1 ? e : e + 1;
                    auto two = [&](const Raw<W>* x) {
                        return make_float2(__uint_as_float(x[u].v[e]), __uint_as_float(x[u2].v[e2]));
                    };
                    const float2 q = price2<M>(two(S), two(K), two(R), two(V), two(T), (int)O[u].v[e], (int)O[u2].v[e2]);
                    p[u][e] = q.x;
                    p[u2][e2] = q.y;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u < runs) {
                    if constexpr (W == 1)
                        asm volatile("st.global.f32 [%0], %1;" :: "l"(a.out + o), "f"(p[u][0]) : "memory");
                    else if constexpr (W == 2)
                        asm volatile("st.global.v2.f32 [%0], {%1,%2};"
                                     :: "l"(a.out + o), "f"(p[u][0]), "f"(p[u][1]) : "memory");
                    else
                        asm volatile("st.global.v4.f32 [%0], {%1,%2,%3,%4};"
                                     :: "l"(a.out + o), "f"(p[u][0]), "f"(p[u][1]), "f"(p[u][2]), "f"(p[u][3])
                                     : "memory");
                    if (HOST && j + u == runs - 1) give_words<W>(host.out + o, p[u]);
                }
        }
    }
    // the options before the first vector and after the last: two warps of the
    // last block, which has no others then
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x < 64) {
        const int64_t i = threadIdx.x < 32 ? n / W * W + threadIdx.x : (int64_t)threadIdx.x - 32 - head;
        if (threadIdx.x < 32 ? i < n : i < 0) {
            if constexpr (HOST) {
                const_cast<float*>(a.s)[i] = host.s[i];
                const_cast<float*>(a.k)[i] = host.k[i];
                const_cast<float*>(a.r)[i] = host.r[i];
                const_cast<float*>(a.v)[i] = host.v[i];
                const_cast<float*>(a.t)[i] = host.t[i];
                const_cast<int32_t*>(a.ot)[i] = host.ot[i];
            }
            auto f = [&](const float* x) { return *const_cast<const volatile float*>(x + i); };
            constexpr int kTail = 4;  // passes in flight
            float p = 0.0f;
            for (int j = 0; j < runs; j += kTail) {
                float in[kTail][5], q[kTail];
                int ot[kTail];
#pragma unroll
                for (int u = 0; u < kTail; ++u) {
                    in[u][0] = f(a.s);
                    in[u][1] = f(a.k);
                    in[u][2] = f(a.r);
                    in[u][3] = f(a.v);
                    in[u][4] = f(a.t);
                    ot[u] = *const_cast<const volatile int32_t*>(a.ot + i);
                }
#pragma unroll
                for (int u = 0; u < kTail; ++u)
                    q[u] = price<M>(in[u][0], in[u][1], in[u][2], in[u][3], in[u][4], ot[u]);
#pragma unroll
                for (int u = 0; u < kTail; ++u)
                    if (j + u < runs) *const_cast<volatile float*>(a.out + i) = p = q[u];
            }
            if constexpr (HOST) host.out[i] = p;
        }
    }
    if (sig.flag) {
        __syncthreads();
        if (threadIdx.x == 0) signal_host(sig.count, gridDim.x, sig.flag, sig.seq);
    }
}

// One pass over a short book, in device memory or staged by the host (16-byte
// aligned arrays), which tells the host itself that it is done: the block that
// finishes last stores the call's number to a word in pinned memory, after every
// price is there.  The host polls that word: a call of 16 options takes 11.7 us,
// 13.7 with a stream synchronisation.
constexpr int kStageThreads = 128;

template <int M, bool HEAD>  // (HEAD's code alone costs a call without one 0.4 us)
__global__ void __launch_bounds__(kStageThreads) map_stage_kernel(SoA a, int n, int head, Signal sig) {
    const int g = blockIdx.x * kStageThreads + threadIdx.x;
    if (4 * g + 4 <= n) {
        const float4 q = price4<M>(__ldg(reinterpret_cast<const float4*>(a.s) + g),
                                   __ldg(reinterpret_cast<const float4*>(a.k) + g),
                                   __ldg(reinterpret_cast<const float4*>(a.r) + g),
                                   __ldg(reinterpret_cast<const float4*>(a.v) + g),
                                   __ldg(reinterpret_cast<const float4*>(a.t) + g),
                                   __ldg(reinterpret_cast<const int4*>(a.ot) + g));
        reinterpret_cast<float4*>(a.out)[g] = q;
    } else {
        for (int i = 4 * g; i < n; ++i) price_scalar<M>(a, i);
    }
    // the options before the vectors: a block of their own, the last
    if (HEAD && blockIdx.x == gridDim.x - 1 && (int)threadIdx.x < head) price_scalar<M>(a, (int)threadIdx.x - head);
    __syncthreads();
    if (threadIdx.x == 0) signal_host(sig.count, gridDim.x, sig.flag, sig.seq);
}

// Host arrays into device arrays: blockIdx.y picks the array, so that the link
// carries all six at once; 16-byte words where the source allows (dst is
// aligned), four in flight per thread.
__global__ void __launch_bounds__(256) gather_kernel(SoA src, SoA dst, int64_t n) {
    const void* ps[6] = {src.s, src.k, src.r, src.v, src.t, src.ot};
    const void* pd[6] = {dst.s, dst.k, dst.r, dst.v, dst.t, dst.ot};
    const uint32_t* s = static_cast<const uint32_t*>(ps[blockIdx.y]);
    uint32_t* d = const_cast<uint32_t*>(static_cast<const uint32_t*>(pd[blockIdx.y]));
    const int64_t n4 = (reinterpret_cast<uintptr_t>(s) & 15) == 0 ? n / 4 : 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t i = i0;
    for (; i + 3 * stride < n4; i += 4 * stride) {
        uint4 x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = __ldg(reinterpret_cast<const uint4*>(s) + i + j * stride);
#pragma unroll
        for (int j = 0; j < 4; ++j) reinterpret_cast<uint4*>(d)[i + j * stride] = x[j];
    }
    for (; i < n4; i += stride) reinterpret_cast<uint4*>(d)[i] = __ldg(reinterpret_cast<const uint4*>(s) + i);
    for (int64_t k = 4 * n4 + i0; k < n; k += stride) d[k] = __ldg(s + k);
}

cudaError_t launch_gather(const SoA& src, const SoA& dst, int64_t n, int sm_count, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int64_t gx = (n / 4 + 255) / 256;
    if (gx > sm_count) gx = sm_count;
    if (gx < 1) gx = 1;
    gather_kernel<<<dim3((unsigned)gx, 6), 256, 0, st>>>(src, dst, n);
    return cudaGetLastError();
}

// Scalar kernel: any 4-byte aligned pointers.
template <int M>
__global__ void __launch_bounds__(256) map_scalar_kernel(SoA a, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        price_scalar<M>(a, i);
}

// ------------------------------------------------- TMA bulk-staged variant
// Each persistent CTA streams whole tiles (256 threads x OPT options) through
// a STAGES-deep ring in shared memory: one thread issues six 1D bulk copies
// (cp.async.bulk, one per input array) per tile, completing on the stage's
// mbarrier with a transaction count; every thread waits on the barrier,
// prices OPT options from shared memory and stores them with streaming
// stores.  A stage is refilled after a block barrier and a proxy fence.
// Waits are bounded: on expiry the CTA records kErrBulkTimeout in
// g_bulk_err, waits (bounded) for its copies in flight and returns.
// Shapes: <8, 3> 144 KB per CTA (1 per SM), <4, 4> 96 KB (2 per SM),
// <4, 3> 72 KB (3 per SM).
constexpr int kBulkThreads = 256;
constexpr unsigned kErrBulkTimeout = 1u;
constexpr uint64_t kBulkWaitNs = 1000000000ull;  // bound of one wait: 1 s

// Error word of the bulk kernels (kErrBulkTimeout); read and cleared by the
// host with bulk_error_take().
__device__ unsigned g_bulk_err;

template <int OPT, int STAGES>
struct BulkShape {
    static constexpr int tile = kBulkThreads * OPT;
    static constexpr int stage_bytes = 6 * tile * 4;
    static constexpr int smem = STAGES * stage_bytes;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the phase of `bar` with parity `parity` for at most limit_ns of
// wall time (the GPU's global timer); false when the bound expired.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

// One 1D bulk copy of `bytes` (16-byte aligned at both ends, a multiple of
// 16) into shared memory, completing on `bar`, with L2 cache policy `pol`
// (evict_first: the cyclic scan then keeps a slice of the inputs in L2 from
// pass to pass, as the evict_first load paths do).
__device__ __forceinline__ void bulk_copy(char* dst, const char* src, int bytes, uint32_t bar,
                                          unsigned long long pol) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1], %2, [%3], %4;"
        :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(bar), "l"(pol) : "memory");
}

// Issues the six copies of tile `tile` into stage memory `st` (thread 0).
// tx_extra (0 in production) raises the barrier's expected byte count above
// what the copies deliver, so that its phase can never complete: the
// self-test of the bounded waits.
template <int TILE>
__device__ __forceinline__ void bulk_issue(const SoA& a, int64_t tile, char* st, uint32_t bar,
                                           uint32_t tx_extra) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(bar), "r"(6 * TILE * 4 + tx_extra) : "memory");
    const size_t off = (size_t)tile * TILE * 4;
    const unsigned long long pol = evict_first_policy();
    bulk_copy(st + 0 * TILE * 4, reinterpret_cast<const char*>(a.s) + off, TILE * 4, bar, pol);
    bulk_copy(st + 1 * TILE * 4, reinterpret_cast<const char*>(a.k) + off, TILE * 4, bar, pol);
    bulk_copy(st + 2 * TILE * 4, reinterpret_cast<const char*>(a.r) + off, TILE * 4, bar, pol);
    bulk_copy(st + 3 * TILE * 4, reinterpret_cast<const char*>(a.v) + off, TILE * 4, bar, pol);
    bulk_copy(st + 4 * TILE * 4, reinterpret_cast<const char*>(a.t) + off, TILE * 4, bar, pol);
    bulk_copy(st + 5 * TILE * 4, reinterpret_cast<const char*>(a.ot) + off, TILE * 4, bar, pol);
}

template <int M, int OPT, int STAGES>
__global__ void __launch_bounds__(kBulkThreads) map_bulk_kernel(SoA a, int64_t n, uint64_t wait_ns,
                                                                 uint32_t tx_extra) {
    using B = BulkShape<OPT, STAGES>;
    constexpr int TILE = B::tile;
    extern __shared__ __align__(128) char smem[];
    __shared__ __align__(8) unsigned long long bars[STAGES];
    __shared__ int sh_abort;
    pdl_trigger();
    const int64_t ntiles = n / TILE;
    // tiles of this CTA: blockIdx.x + k * gridDim.x
    const int64_t mine = (ntiles > blockIdx.x) ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&bars[s])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sh_abort = 0;
        for (int s = 0; s < STAGES && s < mine; ++s)
            bulk_issue<TILE>(a, blockIdx.x + (int64_t)s * gridDim.x, smem + s * B::stage_bytes,
                             smem_u32(&bars[s]), tx_extra);
    }
    __syncthreads();
    int64_t k = 0;
    for (; k < mine; ++k) {
        const int s = (int)(k % STAGES);
        const uint32_t parity = (uint32_t)((k / STAGES) & 1);
        const bool ok = mbar_wait_bounded(smem_u32(&bars[s]), parity, wait_ns);
        if (!ok) sh_abort = 1;  // benign race: every writer stores 1
        __syncthreads();
        if (sh_abort) break;
        const char* st = smem + s * B::stage_bytes;
        const int64_t tile = blockIdx.x + k * gridDim.x;
        // thread t prices options 4t..4t+3 of each 1024-option slice, so each
        // 128-bit shared load and global store of a warp covers 512
        // contiguous bytes (no bank conflicts)
        float p[OPT / 4][4];
#pragma unroll
        for (int h = 0; h < OPT / 4; ++h) {
            const int o = (4 * threadIdx.x + 1024 * h) * 4;
            const float4 S = *reinterpret_cast<const float4*>(st + 0 * TILE * 4 + o);
            const float4 K = *reinterpret_cast<const float4*>(st + 1 * TILE * 4 + o);
            const float4 R = *reinterpret_cast<const float4*>(st + 2 * TILE * 4 + o);
            const float4 V = *reinterpret_cast<const float4*>(st + 3 * TILE * 4 + o);
            const float4 T = *reinterpret_cast<const float4*>(st + 4 * TILE * 4 + o);
            const int4 O = *reinterpret_cast<const int4*>(st + 5 * TILE * 4 + o);
            const float4 q = price4<M>(S, K, R, V, T, O);
            p[h][0] = q.x;
            p[h][1] = q.y;
            p[h][2] = q.z;
            p[h][3] = q.w;
        }
        __syncthreads();  // every thread has read stage s
        if (threadIdx.x == 0 && k + STAGES < mine) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bulk_issue<TILE>(a, blockIdx.x + (k + STAGES) * gridDim.x, smem + s * B::stage_bytes,
                             smem_u32(&bars[s]), tx_extra);
        }
#pragma unroll
        for (int h = 0; h < OPT / 4; ++h)
            st_group<4, 0>(a.out + tile * TILE + 1024 * h + 4 * threadIdx.x, p[h], 0ull);
    }
    if (k < mine) {
        // timed out: record it, let this CTA's copies in flight land (bounded)
        if (threadIdx.x == 0) {
            atomicOr(&g_bulk_err, kErrBulkTimeout);
            for (int64_t q = k; q < mine && q < k + STAGES; ++q)
                mbar_wait_bounded(smem_u32(&bars[q % STAGES]), (uint32_t)((q / STAGES) & 1), wait_ns);
        }
        __syncthreads();
        return;
    }
    // options past the last whole tile: the last CTA, one per thread
    if (blockIdx.x == gridDim.x - 1)
        for (int64_t i = ntiles * TILE + threadIdx.x; i < n; i += kBulkThreads)
            price_scalar<M>(a, i);
    pdl_wait();
}

unsigned bulk_error_take() {
    unsigned v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_bulk_err, sizeof v) != cudaSuccess ||
        cudaMemcpyToSymbol(g_bulk_err, &zero, sizeof zero) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return v;
}

static bool aligned(const void* p, uintptr_t al) {
    return (reinterpret_cast<uintptr_t>(p) & (al - 1)) == 0;
}

// Moves the pointers up to the next `al`-byte boundary when all seven are
// the same number of options past one (a slice of a book): the options
// passed over, or -1 when no such move exists or the book ends before it.
static int peel(SoA* a, int64_t* n, uintptr_t al) {
    const uintptr_t m = reinterpret_cast<uintptr_t>(a->s) & (al - 1);
    const void* p[6] = {a->k, a->r, a->v, a->t, a->ot, a->out};
    for (const void* q : p)
        if ((reinterpret_cast<uintptr_t>(q) & (al - 1)) != m) return -1;
    const int h = m ? (int)((al - m) / 4) : 0;
    if (h > *n) return -1;
    a->s += h;
    a->k += h;
    a->r += h;
    a->v += h;
    a->t += h;
    a->ot += h;
    a->out += h;
    *n -= h;
    return h;
}

bool map_vectorizable(const SoA& a, const MapCfg& cfg) {
    // 256-bit loads for LP 2 and 6, and for the bulk paths' small-n fallback
    const uintptr_t al = (cfg.load_path >= 2) ? 32 : 16;
    return aligned(a.s, al) && aligned(a.k, al) && aligned(a.r, al) &&
           aligned(a.v, al) && aligned(a.t, al) && aligned(a.ot, al) &&
           aligned(a.out, al);
}

// Opts kernel K in to `bytes` of dynamic shared memory, once per device
// (contexts on several host threads may race here: setting the attribute
// twice is harmless, the bit mask is atomic).
template <auto* K>
static cudaError_t opt_in_smem(size_t bytes) {
    static std::atomic<unsigned long long> opted{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(opted.load(std::memory_order_acquire) & (1ull << dev))) {
        e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        if (dev < 64) opted.fetch_or(1ull << dev, std::memory_order_release);
    }
    return cudaSuccess;
}

template <int M, int OPT, int STAGES>
static cudaError_t launch_map_bulk(const SoA& a, int64_t n, const MapCfg& cfg, int sm_count,
                                  cudaStream_t st, uint64_t wait_ns = kBulkWaitNs,
                                  uint32_t tx_extra = 0) {
    using B = BulkShape<OPT, STAGES>;
    cudaError_t e = opt_in_smem<map_bulk_kernel<M, OPT, STAGES>>(B::smem);
    if (e != cudaSuccess) return e;
    const int64_t ntiles = n / B::tile;
    int64_t grid = (int64_t)sm_count * (220 * 1024 / B::smem);  // CTAs that fit per SM
    if (grid > ntiles) grid = ntiles;
    if (grid < 1) grid = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)grid);
    lc.blockDim = dim3(kBulkThreads);
    lc.dynamicSmemBytes = B::smem;
    lc.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = cfg.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&lc, map_bulk_kernel<M, OPT, STAGES>, a, n, wait_ns, tx_extra);
}

// The current device's L2 size in bytes (0 if unknown), cached per device.
static int64_t device_l2_bytes() {
    static std::atomic<int64_t> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int64_t v = cache[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        int b = 0;
        if (cudaDeviceGetAttribute(&b, cudaDevAttrL2CacheSize, dev) != cudaSuccess) return 0;
        v = b;
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

template <int M>
static cudaError_t launch_map_mode(const SoA& a_in, int64_t n, const MapCfg& cfg_in,
                                   int sm_count, cudaStream_t st) {
    MapCfg cfg = cfg_in;
    SoA a = a_in;
    if constexpr (M == MODE_LIBM_REF) {
        // compute-bound (float-float exp/log): 128-bit loads and one block of
        // up to 256 threads per tile (1024 threads resident per SM), whatever
        // shape the memory-bound tuning chose
        cfg.load_path = 0;
        cfg.vpt = 1;
        cfg.blocks_per_sm = 0;
        if (cfg.block > 256) cfg.block = 256;
    }
    const int block = cfg.block;
    // 256-bit loads for load paths 2 and up where a common boundary is that
    // far, else 128-bit; a slice of a book (all seven pointers equally far
    // from one) starts with up to 7 single options.  From
    // option 3 of a book 10M x 100 passes take 3.48 ms, 5.25 with the scalar kernel;
    // 45M once 194 us, 237.
    int head = peel(&a, &n, cfg.load_path >= 2 ? 32 : 16);
    if (head < 0 && cfg.load_path >= 2 && (head = peel(&a, &n, 16)) >= 0) {
        cfg.load_path = 0;
        cfg.vpt = 1;
    }
    if (head < 0) {
        int64_t grid = (n + 255) / 256;
        const int64_t cap = (int64_t)sm_count * 8;
        if (grid > cap) grid = cap;
        if (grid < 1) grid = 1;
        map_scalar_kernel<M><<<(unsigned)grid, 256, 0, st>>>(a, n);
        return cudaGetLastError();
    }
    if (cfg.load_path >= 3 && cfg.load_path <= 5) {
        if constexpr (M == MODE_FAST) if (head == 0) {
            // 3: <8 options, 3 stages>, 4: <4, 4>, 5: <4, 3>
            if (cfg.load_path == 3 && n >= BulkShape<8, 3>::tile)
                return launch_map_bulk<M, 8, 3>(a, n, cfg, sm_count, st);
            if (cfg.load_path == 4 && n >= BulkShape<4, 4>::tile)
                return launch_map_bulk<M, 4, 4>(a, n, cfg, sm_count, st);
            if (cfg.load_path == 5 && n >= BulkShape<4, 3>::tile)
                return launch_map_bulk<M, 4, 3>(a, n, cfg, sm_count, st);
        }
        MapCfg v8 = cfg;  // too small for a whole tile (or another mode): 256-bit loads
        v8.load_path = 2;
        v8.vpt = 1;
        return launch_map_mode<M>(a_in, n + head, v8, sm_count, st);
    }
    const int W = lp_v8(cfg.load_path) ? 8 : 4;
    const int64_t ngroups = n / W;
    // LP 7: the first gres groups (res32 32nds of the L2 in inputs and
    // prices, 28 bytes an option) are kept resident across passes
    int64_t gres = 0;
    if (lp_resident(cfg.load_path)) {
        const int res32 = (cfg.res32 >= 1 && cfg.res32 <= 24) ? cfg.res32 : 15;
        gres = device_l2_bytes() * res32 / 32 / (28 * W);
        if (gres > ngroups) gres = ngroups;
    }
    const int64_t tile = (int64_t)block * cfg.vpt;
    int64_t ntiles = (ngroups + tile - 1) / tile;
    int64_t grid = ntiles;
    if (cfg.blocks_per_sm > 0) {
        const int64_t cap = (int64_t)cfg.blocks_per_sm * sm_count;
        if (grid > cap) grid = cap;
    }
    if (grid > 0x7fffffff) grid = 0x7fffffff;
    if (grid < 1) grid = 1;
    const dim3 g((unsigned)grid), b((unsigned)block);

    cudaLaunchConfig_t lc = {};
    lc.gridDim = g;
    lc.blockDim = b;
    lc.dynamicSmemBytes = 0;
    lc.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = cfg.pdl ? 1 : 0;
    cudaError_t le = cudaSuccess;
#define BSG_LAUNCH(W_, V_, L_) \
    le = cudaLaunchKernelEx(&lc, map_vec_kernel<M, W_, V_, L_>, a, n, head, gres, cfg.rev)
    if constexpr (M == MODE_FAST) {
        switch (cfg.load_path * 10 + cfg.vpt) {
            case 1: BSG_LAUNCH(4, 1, 0); break;
            case 2: BSG_LAUNCH(4, 2, 0); break;
            case 4: BSG_LAUNCH(4, 4, 0); break;
            case 11: BSG_LAUNCH(4, 1, 1); break;
            case 12: BSG_LAUNCH(4, 2, 1); break;
            case 14: BSG_LAUNCH(4, 4, 1); break;
            case 21: BSG_LAUNCH(8, 1, 2); break;
            case 22: BSG_LAUNCH(8, 2, 2); break;
            case 61: BSG_LAUNCH(8, 1, 6); break;
            case 62: BSG_LAUNCH(8, 2, 6); break;
            case 71: BSG_LAUNCH(8, 1, 7); break;
            case 72: BSG_LAUNCH(8, 2, 7); break;
            case 81: BSG_LAUNCH(8, 1, 8); break;
            case 82: BSG_LAUNCH(8, 2, 8); break;
            default: return cudaErrorInvalidValue;
        }
    } else {
        // reference-order paths are validation variants: one shape each.
        if constexpr (M == MODE_LIBM_REF) BSG_LAUNCH(4, 1, 0);
        else if (lp_v8(cfg.load_path)) BSG_LAUNCH(8, 1, 2);
        else BSG_LAUNCH(4, 1, 0);
    }
#undef BSG_LAUNCH
    if (le != cudaSuccess) return le;
    return cudaGetLastError();
}

cudaError_t launch_bulk_wait_selftest(const SoA& a, int64_t n, int sm_count, uint64_t wait_ns,
                                      cudaStream_t st) {
    if (n < BulkShape<4, 4>::tile) return cudaErrorInvalidValue;
    const MapCfg cfg{1, kBulkThreads, 0, 4, 0};
    return launch_map_bulk<MODE_FAST, 4, 4>(a, n, cfg, sm_count, st, wait_ns, 16u);
}

cudaError_t launch_map(const SoA& a, int64_t n, int mode, const MapCfg& cfg,
                       int sm_count, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (cfg.block < 32 || cfg.block > 512 || (cfg.block & 31)) return cudaErrorInvalidValue;
    switch (mode) {
        case MODE_FAST: return launch_map_mode<MODE_FAST>(a, n, cfg, sm_count, st);
        case MODE_SFU_REF: return launch_map_mode<MODE_SFU_REF>(a, n, cfg, sm_count, st);
        case MODE_LIBM_REF: return launch_map_mode<MODE_LIBM_REF>(a, n, cfg, sm_count, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int M>
static cudaError_t launch_runs_mode(SoA a, int64_t n, int runs, int sm_count, cudaStream_t st, const Signal& sig,
                                    const SoA* host) {
    // one, then two options per thread while that needs no more than 512 threads
    // an SM: 40,000 options x 100 36 us with one, 44 with two (half the warps);
    // 155,000 57 with two.  One option's passes are evaluated in pairs, four in
    // flight (two 40, eight 39).
    const int w = n <= (int64_t)sm_count * 512 ? 1 : n <= (int64_t)sm_count * 1024 ? 2 : 4;
    const int head = w == 1 ? 0 : peel(&a, &n, 16);
    if (head < 0 || (host && head)) return cudaErrorInvalidValue;
    const int64_t ngroups = n / w;
    int64_t block = (((ngroups + sm_count - 1) / sm_count) + 31) / 32 * 32;
    block = block < 64 ? 64 : block > 512 ? 512 : block;
    // (a block of its own for the options before and after the vectors, so that
    // their passes run beside the others': 20,001 options x 100 on the device 49 us without)
    const bool odd = head || n % w;
    int64_t grid = (ngroups + block - 1) / block + odd;
    if (grid < 1) grid = 1;
    const SoA h = host ? *host : SoA{};
    void (*kernel)(SoA, int64_t, int, int, SoA, Signal) = nullptr;
    constexpr int kPairs = M == MODE_LIBM_REF ? 2 : 4;  // passes of two options in flight
    if (w == 1) kernel = host ? map_runs_kernel<M, 1, 4, true> : map_runs_kernel<M, 1, 4, false>;
    else if (w == 2) kernel = host ? map_runs_kernel<M, 2, kPairs, true> : map_runs_kernel<M, 2, kPairs, false>;
    else if constexpr (M != MODE_LIBM_REF) kernel = host ? map_runs_kernel<M, 4, 2, true> : map_runs_kernel<M, 4, 2, false>;
    if (!kernel) return cudaErrorInvalidValue;
    kernel<<<(unsigned)grid, (unsigned)block, 0, st>>>(a, n, head, runs, h, sig);
    return cudaGetLastError();
}

cudaError_t launch_map_stage(SoA a, int64_t n, int mode, const Signal& sig, cudaStream_t st) {
    if (n <= 0 || n > 1 << 30 || !sig.flag) return cudaErrorInvalidValue;
    const int head = peel(&a, &n, 16);
    if (head < 0) return cudaErrorNotSupported;
    const unsigned grid = (unsigned)((n + 4 * kStageThreads - 1) / (4 * kStageThreads)) + (head > 0);
    void (*kernel)(SoA, int, int, Signal) = nullptr;
    switch (mode) {
        case MODE_FAST: kernel = head ? map_stage_kernel<MODE_FAST, true> : map_stage_kernel<MODE_FAST, false>; break;
        case MODE_SFU_REF: kernel = head ? map_stage_kernel<MODE_SFU_REF, true> : map_stage_kernel<MODE_SFU_REF, false>; break;
        case MODE_LIBM_REF: kernel = head ? map_stage_kernel<MODE_LIBM_REF, true> : map_stage_kernel<MODE_LIBM_REF, false>; break;
        default: return cudaErrorInvalidValue;
    }
    kernel<<<grid, kStageThreads, 0, st>>>(a, (int)n, head, sig);
    return cudaGetLastError();
}

// Whether the n prices share memory with an input array.
bool in_place(const SoA& a, int64_t n) {
    const uintptr_t o = reinterpret_cast<uintptr_t>(a.out), b = (uintptr_t)n * 4;
    const void* p[6] = {a.s, a.k, a.r, a.v, a.t, a.ot};
    for (const void* q : p) {
        const uintptr_t x = reinterpret_cast<uintptr_t>(q);
        if (x < o + b && o < x + b) return true;
    }
    return false;
}

// Up to 2048 options an SM (4 options a thread, 512 threads): 311,000 options x
// 100 passes take 100 us, 117 as programmatic launches; at 622,592 both took
// 222.  The reference-order libm mode up to 1024 (2 a thread): 155,648 options
// 128 us against 141, 65,536 75 against 96, 1,000 42 against 70; at 200,000, four
// a thread, 184 against 170.  (The kernel's pass counter runs a step past `runs`.)
bool map_runs_fit(const SoA& a, int64_t n, int mode, int runs, int sm_count) {
    SoA b = a;
    int64_t m = n;
    return runs > 1 && runs <= 1 << 30 && n <= (int64_t)sm_count * (mode == MODE_LIBM_REF ? 1024 : 2048) && !in_place(a, n) &&
           peel(&b, &m, 16) >= 0;
}

cudaError_t launch_map_runs(const SoA& a, int64_t n, int mode, int runs, int sm_count, cudaStream_t st,
                            const Signal& sig, const SoA* host) {
    if (n <= 0 || runs <= 0) return host || sig.flag ? cudaErrorInvalidValue : cudaSuccess;
    switch (mode) {
        case MODE_FAST: return launch_runs_mode<MODE_FAST>(a, n, runs, sm_count, st, sig, host);
        case MODE_SFU_REF: return launch_runs_mode<MODE_SFU_REF>(a, n, runs, sm_count, st, sig, host);
        case MODE_LIBM_REF: return launch_runs_mode<MODE_LIBM_REF>(a, n, runs, sm_count, st, sig, host);
        default: return cudaErrorInvalidValue;
    }
}

MapCfg map_default_cfg(const SoA& a, int64_t n, int runs) {
    if (in_place(a, n)) return MapCfg{1, 256, 0, 0, 0};  // passes in strict order
    const int64_t l2 = device_l2_bytes(), bytes = n * 28;
    // One pass: 256-bit loads, a 128-thread block per tile (2^28 options:
    // 1047 us against 1119 with 128-bit loads; the same within 2 % below 20M).
    if (runs == 1) return MapCfg{1, 128, 0, 2, 0};
    // Passes launch programmatically, each while the previous one drains.  A
    // book in half the L2: the same shape (1M x 100: 339 us, 351 with a
    // persistent grid, 533 without programmatic launches).  Up to 2.5 L2: the
    // resident prefix (10M x 100: 3.31 ms, 3.57 persistent, 3.82 one block per
    // tile, 4.16 without; 4M: 1.33, 1.33, 1.42; 15M: 5.54, 5.47, 5.80).  Up to 6
    // L2: the persistent grid (22M: 8.44, 8.45 one block per tile).  Beyond,
    // two groups a thread (120M x 100: 45.7 ms, 45.9 with one, 46.4 persistent,
    // 50.0 without).
    if (bytes <= l2 / 2) return MapCfg{1, 128, 0, 2, 1};
    if (bytes <= l2 * 5 / 2) {
        MapCfg c{1, 128, 4, 7, 1};
        c.res32 = 10;
        return c;
    }
    if (bytes <= 6 * l2) return MapCfg{1, 256, 2, 2, 1};
    return MapCfg{2, 128, 0, 2, 1};
}

// ------------------------------------------------------------------ FP64
// Double prices: double storage in and out (the SIMD variant's NCO = 2
// types, 52 bytes per option), or float storage in (the validation oracle).
// In double arithmetic the kernel is bound by GB300's FP64 rate (177
// operations an option, that pipe 85 % busy: 4M options in 1.38 ms against
// 32 us of HBM traffic), so the elementary functions are fixed point
// (bsg_fx64.h).  The few options that are left to the double evaluation go
// into a queue of the block's: the warp whose option is a 32nd prices 32 of
// them together, between the other warps' integer work, and the block the rest
// at the end.  In place, one such option would hold its warp for a whole
// double evaluation.  4M options: 124 us, bound by the pipe of the integer
// multiply-adds (173 us before N came from a table).
//
// One block of 32 warps an SM; each warp takes the SM's next 32 options when it
// is done with its last, and has the ones after copied into shared memory
// meanwhile.  With a fixed share per warp (256-thread blocks, four an SM) the
// scheduler, which prefers older warps, left the younger ones alone at the
// end (25 of 32 warps resident on average), a fifth of the stalls were for
// loads, and the queue waited for the end: 136 us, 155 where 3 % go into the
// queue (now 136), 16M of those 533 (446).
constexpr int kF64Threads = 1024;
constexpr int kF64Warps = kF64Threads / 32;
constexpr int kF64Queue = 1024;
constexpr uint32_t kEmpty = 0xFFFFFFFFu;

__device__ const bsg_sw::Tables kFxTables = BSG_SW_TABLES;
__device__ const bsg_fx::TailTable kFxTails = BSG_FX_TAILS;

// One warp's options on their way in.
template <typename T>
struct F64Slot {
    T s[32], k[32], r[32], v[32], t[32];
    int32_t ot[32];
};

// The block's copy of the tables the price reads (48,640 bytes), two slots a
// warp, and the options left to the double evaluation: dynamic shared memory.
template <typename T>
struct F64Shared {
    bsg_sw::LogEntry lg[512];
    bsg_sw::SeedEntry rs[384];
    uint64_t e2[1024];
    bsg_fx::TailTable tails;
    F64Slot<T> slot[2][kF64Warps];
    uint32_t queue[kF64Queue];
    uint32_t queued, next;
};

template <typename T>
__device__ __forceinline__ void copy_table(T& dst, const T& src) {
    static_assert(sizeof(T) % 16 == 0, "copied in 16-byte words");
    for (int i = threadIdx.x; i < (int)(sizeof(T) / 16); i += kF64Threads)
        reinterpret_cast<uint4*>(&dst)[i] = __ldg(reinterpret_cast<const uint4*>(&src) + i);
}

__device__ __noinline__ double price_fp64_call(double s, double k, double r, double v, double t, int ot) {
    return price_fp64(s, k, r, v, t, ot);
}

__device__ __forceinline__ uint64_t dbits(double d) { return (uint64_t)__double_as_longlong(d); }

template <typename T>
struct F64View {
    const T* s;
    const T* k;
    const T* r;
    const T* v;
    const T* t;
    const int32_t* ot;
    double* out;
};

template <typename T>
__device__ __forceinline__ void copy_async(T* dst, const T* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(sizeof(T))
                 : "memory");
}

template <typename T>
__global__ void __launch_bounds__(kF64Threads, 1) map_f64_kernel(F64View<T> a, int64_t n, Signal sig) {
    extern __shared__ __align__(16) char f64_smem[];
    F64Shared<T>& sh = *reinterpret_cast<F64Shared<T>*>(f64_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the block's j-th 32 options begin here
    auto begin = [&](uint32_t j) { return ((int64_t)j * gridDim.x + blockIdx.x) * 32; };
    auto fetch = [&](uint32_t j, int b) {
        const int64_t i = begin(j) + lane;
        if (i < n) {
            F64Slot<T>& d = sh.slot[b][warp];
            copy_async(&d.s[lane], a.s + i);
            copy_async(&d.k[lane], a.k + i);
            copy_async(&d.r[lane], a.r + i);
            copy_async(&d.v[lane], a.v + i);
            copy_async(&d.t[lane], a.t + i);
            copy_async(&d.ot[lane], a.ot + i);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint32_t j = warp;
    int b = 0;
    fetch(j, b);
    copy_table(sh.lg, kFxTables.lg);
    copy_table(sh.rs, kFxTables.rs);
    copy_table(sh.e2, kFxTables.e2);
    copy_table(sh.tails, kFxTails);
    for (int q = threadIdx.x; q < kF64Queue; q += kF64Threads) sh.queue[q] = kEmpty;
    if (threadIdx.x == 0) {
        sh.queued = 0;
        sh.next = kF64Warps;
    }
    __syncthreads();
    auto price_left = [&](uint32_t at) {
        const int64_t i = begin(at / 32) + at % 32;
        a.out[i] = price_fp64_call(__ldg(a.s + i), __ldg(a.k + i), __ldg(a.r + i), __ldg(a.v + i),
                                   __ldg(a.t + i), __ldg(a.ot + i));
    };
    while (begin(j) < n) {
        uint32_t after = 0;
        if (lane == 0) after = atomicAdd(&sh.next, 1u);
        after = __shfl_sync(0xffffffffu, after, 0);
        fetch(after, b ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // each lane reads what it copied itself
        const int64_t i = begin(j) + lane;
        bool done = true;
        if (i < n) {
            const F64Slot<T>& d = sh.slot[b][warp];
            const uint64_t s = dbits(d.s[lane]), k = dbits(d.k[lane]), r = dbits(d.r[lane]),
                           v = dbits(d.v[lane]), t = dbits(d.t[lane]);
            double p;
            done = bsg_fx::fx64_domain(s, k, r, v, t);
            if (done) done = bsg_fx::price_fx64(sh, sh.tails, s, k, r, v, t, d.ot[lane], &p);
            if (done) a.out[i] = p;
        }
        uint32_t q = 0;
        if (!done) {
            q = atomicAdd(&sh.queued, 1u);
            if (atomicCAS(&sh.queue[q % kF64Queue], kEmpty, j * 32 + lane) != kEmpty) price_left(j * 32 + lane);
        }
        // whoever fills up 32 entries prices those that are there (one whose
        // writer is not that far yet stays until the end), unless the block is
        // nearly through: then the rest is priced side by side at the end
        const bool fills = q % 32 == 31 && begin(j + 4 * kF64Warps) < n;
        for (unsigned full = __ballot_sync(0xffffffffu, fills); full; full &= full - 1) {
            const uint32_t last = __shfl_sync(0xffffffffu, q, __ffs(full) - 1);
            const uint32_t at = atomicExch(&sh.queue[(last - lane) % kF64Queue], kEmpty);
            if (at != kEmpty) price_left(at);
            __syncwarp();
        }
        j = after;
        b ^= 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int q = threadIdx.x; q < kF64Queue; q += kF64Threads)
        if (sh.queue[q] != kEmpty) price_left(sh.queue[q]);
    if (sig.flag) {
        __syncthreads();
        if (threadIdx.x == 0) signal_host(sig.count, gridDim.x, sig.flag, sig.seq);
    }
}

template <typename T>
static cudaError_t launch_f64_view(const F64View<T>& a, int64_t n, int sm_count, cudaStream_t st, const Signal& sig) {
    if (n <= 0) return cudaSuccess;
    cudaError_t e = opt_in_smem<map_f64_kernel<T>>(sizeof(F64Shared<T>));
    if (e != cudaSuccess) return e;
    const int64_t grid = std::min<int64_t>((n + 31) / 32, sm_count);
    map_f64_kernel<T><<<(unsigned)grid, kF64Threads, sizeof(F64Shared<T>), st>>>(a, n, sig);
    return cudaGetLastError();
}

cudaError_t launch_map_f64(const SoA64& a, int64_t n, int sm_count, cudaStream_t st, const Signal& sig) {
    return launch_f64_view(F64View<double>{a.s, a.k, a.r, a.v, a.t, a.ot, a.out}, n, sm_count, st, sig);
}

cudaError_t launch_fp64(const SoA& a, double* out, int64_t n, int sm_count, cudaStream_t st, const Signal& sig) {
    return launch_f64_view(F64View<float>{a.s, a.k, a.r, a.v, a.t, a.ot, out}, n, sm_count, st, sig);
}

// ------------------------------------------------------------ batched books
// A tile is 8192 options; a block covers it in passes of kBatchBlock
// threads x kBatchVpt v4 groups.
constexpr int kBatchVpt = 1;

// Prices options [b, e) of the pool as thread `tid` of `nt` that share them: an
// unaligned head and tail one option per thread, the aligned body in groups of
// W options (W = 4: 16-byte loads; W = 8: 256-bit loads).
template <int M, int W>
__device__ __forceinline__ void price_range(const SoA& pool, uint64_t b, uint64_t e, unsigned tid, unsigned nt) {
    constexpr uint64_t mask = W - 1;
    const uint64_t head_end = ((b + mask) & ~mask) < e ? ((b + mask) & ~mask) : e;
    const uint64_t body_end = (e & ~mask) > head_end ? (e & ~mask) : head_end;
    const uint64_t i_head = b + tid;
    if (i_head < head_end) price_scalar<M>(pool, (int64_t)i_head);
    price_groups<M, W, W == 8 ? 1 : kBatchVpt, W == 8 ? 2 : 0>(
        pool, (int64_t)(head_end / W), (int64_t)(body_end / W), 0ull, 0ull, 0, tid, nt);
    const uint64_t i_tail = body_end + tid;
    if (i_tail < e) price_scalar<M>(pool, (int64_t)i_tail);
}

// Persistent kernel over a table of tiles ([b, e) in the pool, two words
// each): each block takes the next tile from the device work counter and
// prices it.  The claim of the next tile is issued before the current one is
// priced, so the counter's round trip overlaps the pricing.  No block ever
// waits on another; the loop ends when the counter passes the last tile.
// (Four blocks per SM hold the registers to 64; the libm mode's float-float
// exp/log get up to 128.)
template <int M, int W>
__global__ void __launch_bounds__(kBatchBlock, M == MODE_LIBM_REF ? 2 : 4) batch_kernel(
    SoA pool, const uint64_t* __restrict__ tiles, uint64_t ntiles, unsigned long long* cursor, Signal sig) {
    __shared__ uint64_t sh_b, sh_e;
    __shared__ int sh_done;
    pdl_trigger();
    unsigned long long next = 0;
    if (threadIdx.x == 0) next = atomicAdd(cursor, 1ull);
    for (;;) {
        if (threadIdx.x == 0) {
            const unsigned long long tile = next;
            sh_done = tile >= ntiles;
            if (!sh_done) {
                next = atomicAdd(cursor, 1ull);  // travels while this tile is priced
                sh_b = tiles[2 * tile];
                sh_e = tiles[2 * tile + 1];
            }
        }
        __syncthreads();
        const int done = sh_done;
        const uint64_t b = sh_b, e = sh_e;
        __syncthreads();
        if (done) break;
        price_range<M, W>(pool, b, e, threadIdx.x, kBatchBlock);
    }
    // (the barriers above are behind every price of the block)
    if (sig.flag && threadIdx.x == 0) signal_host(sig.count, gridDim.x, sig.flag, sig.seq);
    pdl_wait();
}

// The same over a table of segments (the serving loop's unfused path, whose
// tiles have no table): thread 0 finds a tile's segment by a binary search of
// the tile prefix.
template <int M, int W>
__global__ void __launch_bounds__(kBatchBlock, M == MODE_LIBM_REF ? 2 : 4) batch_segments_kernel(
    SoA pool, const uint64_t* __restrict__ seg_off, const uint64_t* __restrict__ seg_len,
    const uint64_t* __restrict__ tile_prefix, int nseg, uint64_t ntiles, uint64_t topt,
    unsigned long long* cursor) {
    __shared__ uint64_t sh_b, sh_e;
    __shared__ int sh_done;
    unsigned long long next = 0;
    if (threadIdx.x == 0) next = atomicAdd(cursor, 1ull);
    for (;;) {
        if (threadIdx.x == 0) {
            const unsigned long long tile = next;
            sh_done = tile >= ntiles;
            if (!sh_done) {
                next = atomicAdd(cursor, 1ull);  // travels while this tile is priced
                int lo = 0, hi = nseg - 1;
                while (lo < hi) {  // largest segment whose first tile <= tile
                    const int mid = (lo + hi + 1) >> 1;
                    if (tile_prefix[mid] <= tile) lo = mid; else hi = mid - 1;
                }
                const uint64_t b = seg_off[lo] + (tile - tile_prefix[lo]) * topt;
                const uint64_t send = seg_off[lo] + seg_len[lo];
                sh_b = b;
                sh_e = (b + topt < send) ? b + topt : send;
            }
        }
        __syncthreads();
        const int done = sh_done;
        const uint64_t b = sh_b, e = sh_e;
        __syncthreads();
        if (done) break;
        price_range<M, W>(pool, b, e, threadIdx.x, kBatchBlock);
    }
}

int batch_blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel<MODE_FAST, 8>, kBatchBlock, 0) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return n > 0 ? n : 1;
}

// 256-bit loads need every pool array 32-byte aligned; the libm mode keeps
// 128-bit loads (fewer registers: it is compute-bound)
static bool batch_w8(const SoA& pool, int mode) {
    return mode != MODE_LIBM_REF && map_vectorizable(pool, MapCfg{1, kBatchBlock, 0, 2, 0});
}

cudaError_t launch_batch(const SoA& pool, const uint64_t* tiles, uint64_t ntiles,
                         unsigned long long* cursor, int mode, int grid, int pdl, cudaStream_t st,
                         const Signal& sig) {
    if (ntiles == 0) return sig.flag ? cudaErrorInvalidValue : cudaSuccess;
    if ((uint64_t)grid > ntiles) grid = (int)ntiles;  // no block without a tile
    if (grid < 1) grid = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)grid);
    lc.blockDim = dim3(kBatchBlock);
    lc.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = pdl ? 1 : 0;
    const bool w8 = batch_w8(pool, mode);
#define BSG_BATCH(M_) \
    (w8 ? cudaLaunchKernelEx(&lc, batch_kernel<M_, 8>, pool, tiles, ntiles, cursor, sig) \
        : cudaLaunchKernelEx(&lc, batch_kernel<M_, 4>, pool, tiles, ntiles, cursor, sig))
    switch (mode) {
        case MODE_FAST: return BSG_BATCH(MODE_FAST);
        case MODE_SFU_REF: return BSG_BATCH(MODE_SFU_REF);
        case MODE_LIBM_REF: return BSG_BATCH(MODE_LIBM_REF);
        default: return cudaErrorInvalidValue;
    }
#undef BSG_BATCH
}

cudaError_t launch_batch_segments(const SoA& pool, const uint64_t* seg_off, const uint64_t* seg_len,
                                  const uint64_t* tile_prefix, int nseg, uint64_t ntiles, uint64_t tile_opts,
                                  unsigned long long* cursor, int mode, int grid, cudaStream_t st) {
    if (ntiles == 0 || nseg <= 0) return cudaSuccess;
    if (tile_opts == 0) return cudaErrorInvalidValue;
    if ((uint64_t)grid > ntiles) grid = (int)ntiles;  // no block without a tile
    if (grid < 1) grid = 1;
    const bool w8 = batch_w8(pool, mode);
#define BSG_BATCH(M_) \
    do { \
        if (w8) batch_segments_kernel<M_, 8><<<grid, kBatchBlock, 0, st>>>(pool, seg_off, seg_len, tile_prefix, \
                                                                          nseg, ntiles, tile_opts, cursor); \
        else batch_segments_kernel<M_, 4><<<grid, kBatchBlock, 0, st>>>(pool, seg_off, seg_len, tile_prefix, \
                                                                       nseg, ntiles, tile_opts, cursor); \
    } while (0)
    switch (mode) {
        case MODE_FAST: BSG_BATCH(MODE_FAST); break;
        case MODE_SFU_REF: BSG_BATCH(MODE_SFU_REF); break;
        case MODE_LIBM_REF: BSG_BATCH(MODE_LIBM_REF); break;
        default: return cudaErrorInvalidValue;
    }
#undef BSG_BATCH
    return cudaGetLastError();
}

// ---------------------------------------------------------- error report
__global__ void __launch_bounds__(256) err_kernel(SoA a, const float* __restrict__ prices,
                                                  int64_t n, const double* __restrict__ edges,
                                                  int nb, double rel_floor, ErrAcc* acc) {
    __shared__ ErrAcc sh[kMaxErrBuckets];
    __shared__ double sh_edges[kMaxErrBuckets + 1];
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        sh[i].count = 0;
        sh[i].max_abs_bits = 0;
        sh[i].max_rel_bits = 0;
        sh[i].max_price_bits = 0;
        sh[i].sum_sq = 0.0;
    }
    for (int i = threadIdx.x; i <= nb; i += blockDim.x) sh_edges[i] = edges[i];
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double s = a.s[i], k = a.k[i], r = a.r[i], v = a.v[i], t = a.t[i];
        const double o = price_fp64(s, k, r, v, t, a.ot[i]);
        const double d1 = fabs(d1_fp64(s, k, r, v, t));
        int bk = 0;
        while (bk < nb - 1 && !(d1 < sh_edges[bk + 1])) ++bk;  // NaN -> last
        const double err = fabs((double)prices[i] - o);
        const double den = fabs(o) > rel_floor ? fabs(o) : rel_floor;
        const double rel = err / den;
        atomicAdd(&sh[bk].count, 1ull);
        atomicMax(&sh[bk].max_abs_bits, (unsigned long long)__double_as_longlong(err));
        atomicMax(&sh[bk].max_rel_bits, (unsigned long long)__double_as_longlong(rel));
        atomicMax(&sh[bk].max_price_bits, (unsigned long long)__double_as_longlong(fabs(o)));
        atomicAdd(&sh[bk].sum_sq, err * err);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        if (sh[i].count == 0) continue;
        atomicAdd(&acc[i].count, sh[i].count);
        atomicMax(&acc[i].max_abs_bits, sh[i].max_abs_bits);
        atomicMax(&acc[i].max_rel_bits, sh[i].max_rel_bits);
        atomicMax(&acc[i].max_price_bits, sh[i].max_price_bits);
        atomicAdd(&acc[i].sum_sq, sh[i].sum_sq);
    }
}

cudaError_t launch_err_report(const SoA& a, const float* prices, int64_t n,
                              const double* edges, int nbuckets, double rel_floor,
                              ErrAcc* acc, int sm_count, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (nbuckets < 1 || nbuckets > kMaxErrBuckets) return cudaErrorInvalidValue;
    int64_t grid = (n + 255) / 256;
    const int64_t cap = (int64_t)sm_count * 4;
    if (grid > cap) grid = cap;
    err_kernel<<<(unsigned)grid, 256, 0, st>>>(a, prices, n, edges, nbuckets, rel_floor, acc);
    return cudaGetLastError();
}

// -------------------------------------------------------------- fill (tuning)
__device__ __forceinline__ float hash_unit(uint64_t x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
    return (float)(x >> 40) * (1.0f / 16777216.0f);
}

__global__ void fill_kernel(SoA a, int64_t n, uint32_t seed) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t b = ((uint64_t)seed << 40) ^ ((uint64_t)i * 8);
        const float s = 10.0f + 190.0f * hash_unit(b + 1);
        float* ms = const_cast<float*>(a.s);
        float* mk = const_cast<float*>(a.k);
        float* mr = const_cast<float*>(a.r);
        float* mv = const_cast<float*>(a.v);
        float* mt = const_cast<float*>(a.t);
        int32_t* mo = const_cast<int32_t*>(a.ot);
        ms[i] = s;
        mk[i] = s * (0.5f + hash_unit(b + 2));
        mr[i] = 0.01f + 0.09f * hash_unit(b + 3);
        mv[i] = 0.05f + 0.6f * hash_unit(b + 4);
        mt[i] = 0.05f + 1.95f * hash_unit(b + 5);
        mo[i] = hash_unit(b + 6) < 0.5f ? 1 : 0;
    }
}

cudaError_t launch_fill(const SoA& a, int64_t n, uint32_t seed, int sm_count,
                        cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int64_t grid = (n + 255) / 256;
    const int64_t cap = (int64_t)sm_count * 8;
    if (grid > cap) grid = cap;
    fill_kernel<<<(unsigned)grid, 256, 0, st>>>(a, n, seed);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Debug guards (contexts created with BSG_DEBUG set): one CTA row per array.

__global__ void guard_check_kernel(const uint32_t* __restrict__ base, int64_t stride,
                                   int64_t cap, int64_t out_lo, uint32_t pattern,
                                   unsigned long long* res) {
    const int64_t a = blockIdx.y;
    const int64_t lo = a == 6 ? out_lo : cap;
    unsigned long long cnt = 0, first = ~0ull;
    for (int64_t i = lo + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < stride;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (base[a * stride + i] != pattern) {
            ++cnt;
            first = min(first, (unsigned long long)(a * stride + i));
        }
    }
    if (cnt) {
        atomicAdd(&res[0], cnt);
        atomicMin(&res[1], first);
    }
}

cudaError_t launch_guard_check(const uint32_t* base, int64_t stride, int64_t cap,
                               int64_t out_lo, uint32_t pattern, unsigned long long* res,
                               int sm_count, cudaStream_t st) {
    if (cap > stride || out_lo > stride || cap < 0 || out_lo < 0) return cudaErrorInvalidValue;
    const int64_t span = stride - (cap < out_lo ? cap : out_lo);
    int64_t gx = (span + 255) / 256;
    if (gx > 4LL * sm_count) gx = 4LL * sm_count;
    if (gx < 1) gx = 1;
    guard_check_kernel<<<dim3((unsigned)gx, 7), 256, 0, st>>>(base, stride, cap, out_lo,
                                                              pattern, res);
    return cudaGetLastError();
}

}  // namespace bsg

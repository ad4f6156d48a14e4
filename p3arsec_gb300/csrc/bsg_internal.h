// bsg_internal.h -- launch interface between the C ABI (bsg_api.cu) and the
// kernels (bsg_kernels.cu).  Not installed; no torch types anywhere.
#pragma once
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>

namespace bsg {

// Arithmetic of the map (see bsg_math.cuh).
enum Mode : int { MODE_FAST = 0, MODE_SFU_REF = 1, MODE_LIBM_REF = 2 };

// One SoA view: the reference's five float arrays, int32 otype, float out.
struct SoA {
    const float* s;
    const float* k;
    const float* r;
    const float* v;
    const float* t;
    const int32_t* ot;
    float* out;
};

// The FP64 product mode's SoA: double storage (otype int32).
struct SoA64 {
    const double* s;
    const double* k;
    const double* r;
    const double* v;
    const double* t;
    const int32_t* ot;
    double* out;
};

// Plain-map launch shape (see bsg_tune in bsg.h).
struct MapCfg {
    int vpt;           // vector groups per thread per tile: 1, 2, 4
    int block;         // threads per block
    int blocks_per_sm; // 0: one block per tile; else grid = blocks_per_sm * SMs
    int load_path;     // 0: v4 nc; 1: v4 + L2 evict_first; 2: v8 (256-bit) nc;
                       // 3, 4, 5: TMA bulk copies into a shared-memory ring;
                       // 6: v8 + L2 evict_first; 7: v8, a prefix of the book
                       // (res32 32nds of the L2) evict_last, the rest evict_first;
                       // 8: v8, every other pass in reverse tile order
    int pdl;           // 1: launch with programmatic stream serialization
    int res32 = 15;    // LP 7: the resident prefix, in 32nds of the L2 (1..24)
    int rev = 0;       // LP 8: this pass walks the tiles from the last to the first
};

// Accumulators of one error bucket (device scratch, zeroed per report).
struct ErrAcc {
    unsigned long long count;
    unsigned long long max_abs_bits;   // non-negative doubles order as u64
    unsigned long long max_rel_bits;
    unsigned long long max_price_bits;
    double sum_sq;
};

constexpr int kMaxErrBuckets = 32;
constexpr int kBatchBlock = 256;

// Launches one pass of the plain map over n options.  Picks the vector kernel
// when all pointers are equally far from a boundary of the configured width
// (the options before it are priced one by one), or else of 16 bytes, and
// otherwise the scalar kernel.  Returns the launch error.
cudaError_t launch_map(const SoA& a, int64_t n, int mode, const MapCfg& cfg,
                       int sm_count, cudaStream_t st);
// The shape of pass j of `runs` consecutive passes over the same book.  The
// resident-prefix load path (7) marks part of the book evict_last so that it
// stays in L2 for the next pass.  The last pass runs the same loads with
// evict_first (6): it still hits the resident lines, and an access with an
// explicit policy sets the line's priority, so no evict_last line is left
// behind the call.  A single pass therefore never marks lines evict_last.
// The alternating load path (8) walks odd passes from the book's last tile
// to its first, so each pass starts on the lines the previous pass touched
// last, which the L2 still holds.
// Pass 0 is never a programmatic launch: a kernel with that attribute loads its
// inputs, and stores prices, while the kernel before it on the stream may still
// be writing (map_vec_kernel and batch_kernel let their dependents start at
// once).  Passes of one book may overlap; the first waits for whatever the
// stream holds: a call that wrote its inputs or writes the same prices, a
// gather, the caller's own kernels.
inline MapCfg pass_cfg(MapCfg c, int j, int runs) {
    if (j == 0) c.pdl = 0;
    if (c.load_path == 7 && j == runs - 1) c.load_path = 6;
    c.rev = (c.load_path == 8) ? (j & 1) : 0;
    return c;
}
// The shape of a context that was never tuned, by the book's size and the
// number of passes.
MapCfg map_default_cfg(const SoA& a, int64_t n, int runs);
// Whether launch_map_runs takes `runs` passes of this book (in one launch).
bool map_runs_fit(const SoA& a, int64_t n, int mode, int runs, int sm_count);
// How a kernel tells the host that it is done (signal_host): a device counter,
// zero, left zero, and a word in pinned memory that gets seq.  flag NULL: not.
struct Signal {
    unsigned* count;
    unsigned* flag;
    unsigned seq;
};
// All passes in one launch; with `host` (the device's addresses of a host book)
// over that book, by way of the device arrays a (16-byte aligned).
cudaError_t launch_map_runs(const SoA& a, int64_t n, int mode, int runs, int sm_count, cudaStream_t st,
                            const Signal& sig = Signal{}, const SoA* host = nullptr);
// Whether the n prices share memory with an input array.
bool in_place(const SoA& a, int64_t n);
#if defined(__CUDACC__)
// One thread of each of `parts` parts of a kernel, once the part's stores are
// made (and seen by this thread): the last one zeroes the count and stores seq
// (and zeroes *queue if there is one: no part takes from it any more) to *flag
// in pinned host memory, where the host then sees every part's stores.
__device__ __forceinline__ void signal_host(unsigned* count, unsigned parts, unsigned* flag, unsigned seq,
                                            unsigned long long* queue = nullptr) {
    __threadfence_system();
    if (atomicAdd(count, 1u) != parts - 1) return;
    *count = 0;
    if (queue) *queue = 0;
    __threadfence_system();
    asm volatile("st.release.sys.global.u32 [%0], %1;" :: "l"(flag), "r"(seq) : "memory");
}
#endif

// One pass over n options of arrays equally far from a 16-byte boundary (else
// cudaErrorNotSupported), in device memory or pinned host memory (its device
// addresses).
cudaError_t launch_map_stage(SoA a, int64_t n, int mode, const Signal& sig, cudaStream_t st);
// Copies n options' six input arrays from src (pinned host memory, its device
// addresses) into dst's, by one kernel.
cudaError_t launch_gather(const SoA& src, const SoA& dst, int64_t n, int sm_count, cudaStream_t st);
// Reads and clears the bulk-staged kernel's error word (non-zero: a bounded
// wait expired and some tiles were not priced).
unsigned bulk_error_take();
// Launches the bulk-staged kernel with every barrier expecting 16 bytes more
// than its copies deliver, so each wait expires after wait_ns (self-test of
// the bounded waits; the copies themselves complete normally).
cudaError_t launch_bulk_wait_selftest(const SoA& a, int64_t n, int sm_count, uint64_t wait_ns,
                                      cudaStream_t st);
// True when every pointer is aligned for cfg's load path (the batch kernel's
// choice of 256-bit loads).
bool map_vectorizable(const SoA& a, const MapCfg& cfg);

cudaError_t launch_fp64(const SoA& a, double* out, int64_t n, int sm_count, cudaStream_t st,
                        const Signal& sig = Signal{});
// One pass of the FP64 product mode over n options.
cudaError_t launch_map_f64(const SoA64& a, int64_t n, int sm_count, cudaStream_t st, const Signal& sig = Signal{});

// Persistent batched pricing over a device table of ntiles tiles, each its
// [begin, end) in the pool.  cursor is a device counter that must be 0 at
// launch.  pdl: launch with programmatic stream serialization (the next pass
// may start while this one drains; it must use its own cursor).
cudaError_t launch_batch(const SoA& pool, const uint64_t* tiles, uint64_t ntiles,
                         unsigned long long* cursor, int mode, int grid, int pdl, cudaStream_t st,
                         const Signal& sig = Signal{});
// The same over device arrays of nseg segments (tile_prefix: nseg + 1 entries,
// exclusive prefix of tiles of tile_opts options per segment).
cudaError_t launch_batch_segments(const SoA& pool, const uint64_t* seg_off, const uint64_t* seg_len,
                                  const uint64_t* tile_prefix, int nseg, uint64_t ntiles, uint64_t tile_opts,
                                  unsigned long long* cursor, int mode, int grid, cudaStream_t st);
// Resident blocks per SM of the batch kernel (its persistent grid = this x SMs).
int batch_blocks_per_sm();

cudaError_t launch_err_report(const SoA& a, const float* prices, int64_t n,
                              const double* edges, int nbuckets,
                              double rel_floor, ErrAcc* acc, int sm_count,
                              cudaStream_t st);

// NVTX range for the lifetime of a scope (header-only NVTX3: a no-op unless a
// profiler injects itself), so profiler timelines show the library's calls.
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&) = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};

// Where [p, p + bytes) lies: kExtentOk when it is device memory of `device`
// (or managed memory) inside one allocation, or across consecutive pieces
// that the virtual memory API mapped into one range with read-write access
// for `device` (pool allocators that grow in place map memory piece by
// piece).  Ordinary allocations are never joined with their neighbours, so
// a size that runs past one is kExtentOverrun.
enum Extent : int {
    kExtentOk = 0,
    kExtentNotDevice = 1,
    kExtentOtherDevice = 2,
    kExtentUnknown = 3,
    kExtentOverrun = 4,
};
// *alloc (optional): on kExtentOk within one allocation, its [begin, end).
struct Range { uintptr_t b = 0, e = 0; };
int device_extent(const void* p, size_t bytes, int device, Range* alloc = nullptr);

// ---- swaptions (HJM Monte Carlo) -------------------------------------------
constexpr int kSwMaxSteps = 32;    // grid points of the HJM path (iN)
constexpr int kSwMaxFactors = 8;   // volatility factors (iFactors)

constexpr int kSwMaxExp = kSwMaxSteps;  // payments, and the path's own discount factor

// One swaption as the path kernel reads it.  A path is linear in its normal
// variates, so each exponential the payoff needs -- the discount factor of
// each payment, then (disc_varies) the path's own down to maturity -- has an
// exponent of a constant plus one coefficient per variate.  Its words, from
// words_at of the table on: n_exp payments (doubles), n_exp constants, then
// n_exp coefficients per variate.  Constants and coefficients are in powers
// of two, fixed point (swaption_setup in bsg_api.cu), or (wide: some exponent
// may leave the fixed-point range) natural exponents as doubles.
struct SwHead {
    uint64_t seed;            // the paths' random stream
    double disc;              // the path's discount factor where it is a constant, else 1
    uint32_t words_at, n_words;
    int n_normals;            // variates up to maturity: grid steps x factors
    int n_exp;
    int disc_varies;          // 0, 1
    int wide;                 // 0, 1
};
// A table small enough to travel with the launch (a copy before the kernel
// costs 3 us of a 20 us call).
constexpr int kSwInlineWords = 480;
struct SwInline {
    uint64_t words[kSwInlineWords];
};

// Paths per thread and blocks of paths per swaption for `trials` paths: a
// rule of the trials alone, so that the order of a swaption's sums is too.
int swaption_per_thread(uint64_t trials);
uint64_t swaption_chunks(uint64_t trials);
size_t swaption_partial_bytes(int nsw, uint64_t trials);
size_t swaption_counters(int nsw, uint64_t trials);
// Runs nsw swaptions with `trials` paths each: sums[i] = the sums of the
// discounted payoffs and of their squares (pinned or device memory).  The
// table: nsw heads, then their words, at `table` (device memory) or in `in`
// (table NULL).  large: some swaption has more than four exponents or is
// wide.  partial: device scratch of swaption_partial_bytes; done:
// swaption_counters device counters, and queue another: zero, left zero.
// At the end it stores seq to *flag in pinned memory (signal_host over count).
cudaError_t launch_swaptions(const SwInline& in, const uint64_t* table, int nsw, bool large,
                             uint64_t trials, void* partial, unsigned* done, unsigned long long* queue,
                             double2* sums, unsigned* count, unsigned* flag, unsigned seq, int sm_count,
                             cudaStream_t st);

// z[2 i], z[2 i + 1] = the swaption kernel's normal pair of words[4 i .. 4 i + 3]
// (device arrays), i < n.
cudaError_t launch_swaption_normals(const uint32_t* words, uint64_t n, double* z, cudaStream_t st);

// Fills n options with a deterministic plausible book (autotuning input).
cudaError_t launch_fill(const SoA& a, int64_t n, uint32_t seed, int sm_count,
                        cudaStream_t st);

// Debug guards of a resident set: seven arrays of `stride` words from `base`;
// the guard of input array a < 6 is words [cap, stride), that of the price
// array words [out_lo, stride).  Adds the number of guard words that differ
// from `pattern` to res[0] and lowers res[1] to the smallest differing word's
// index from `base` (res must hold {0, ~0} beforehand).
cudaError_t launch_guard_check(const uint32_t* base, int64_t stride, int64_t cap,
                               int64_t out_lo, uint32_t pattern, unsigned long long* res,
                               int sm_count, cudaStream_t st);

}  // namespace bsg

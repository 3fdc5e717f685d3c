// cbl_internal.h - shared between the kernels (cbl_kernels.cu) and the host
// library (cbl_host.cu). Not part of the public ABI.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>
#include <new>

// Every int-returning entry point runs inside this guard, so no C++ exception
// crosses the C ABI: a failed host allocation returns CBL_E_NOMEM, anything
// else CBL_E_ARG.
#define CBL_GUARD_BEGIN try {
#define CBL_GUARD_END                                                                   \
    }                                                                                   \
    catch (const std::bad_alloc &) { return CBL_E_NOMEM; }                              \
    catch (...) { return CBL_E_ARG; }

namespace cbl {

// The 7 series (KernelFuncs.as:9-12).
constexpr int kNumer[7] = {32, 1, 256, 64, 4, 4, 1};
constexpr int kNumerLog2[7] = {5, 0, 8, 6, 2, 2, 0};
constexpr int kSign[7] = {1, 1, 0, 1, 1, 1, 0};      // 1 = minus
constexpr uint32_t kDen0[7] = {4, 4, 10, 10, 10, 10, 10};
constexpr uint32_t kDen1[7] = {1, 3, 1, 3, 5, 7, 9};

// Residue-width limits of the term kernels (m odd, m >= 3).
constexpr uint64_t kW1Max = 1ull << 28;   // width 1 (one 32-bit word) for m < 2^28
constexpr uint64_t kW1L3Min = 1ull << 17; // lazy width-1 steps, started from three exponent bits, ...
constexpr uint64_t kW1L4Min = 1ull << 25; // ... from four, ...
constexpr uint64_t kW1LMax = 1ull << 29;  // ... up to here, in width-1 and middle tiles
constexpr uint64_t kW1MMax = 1ull << 31;  // middle width 1 for 2^28 <= m < 2^31
constexpr uint64_t kW1SMax = 1ull << 32;  // strict width 1 for 2^31 <= m < 2^32
constexpr uint64_t kW2FLow = 15ull << 34; // float-quotient steps without an offset for 2^32 <= m < 15 * 2^34
constexpr uint64_t kW2FMax = 94ull << 32; // float-quotient steps for 2^32 <= m < 94 * 2^32, inside short width 2
constexpr uint64_t kW2FExp = 1ull << 48;  // ... in tiles whose exponents are below 2^48 (the short kind's steps above)
constexpr uint64_t kW2SMax = 1ull << 44;  // short width 2 for 2^32 <= m < 2^44
constexpr uint64_t kW2SWide = 39ull << 40; // the short kind's steps also serve width-2 tiles up to here
constexpr uint64_t kW2Max = 1ull << 60;   // width 2 (two words, residues < 4m) for m < 2^60
constexpr uint64_t kW2XMax = 1ull << 62;  // wide width 2 (residues < 2m) for 2^60 <= m < 2^62

constexpr int kTail192 = 20;   // tail terms k = d..d+19 (Bellard.cl:1164-1239)
constexpr int kTailDD = 10;    // tail terms k = d..d+9  (Bellard.cl:1125)
constexpr int kEndDD = 6;      // terms before d with 2^(10(d-k)) < 2^62, which may be below every modulus
static_assert(kEndDD + kTailDD <= 32, "a lane each");

// One contiguous k-range of one series at one position, within one residue
// width. Tiles of `tile_k` consecutive k are handed to warps in order of the
// global tile index; tile0 is this segment's first tile.
struct Seg {
    uint64_t d;
    uint64_t k0, k1;       // [k0, k1); k >= d are tail terms 2^(-10(k-d))/m
    uint64_t tile0;
    uint32_t den0, den1;
    uint32_t slot;         // accumulator slot (6 x u64 digit sums)
    uint32_t flags;        // bit 0: series sign (1 = minus), bits 4-7: residue kind 1..6
};
static_assert(sizeof(Seg) == 48, "Seg layout");

constexpr uint32_t kFlagSign = 1u;
inline uint32_t seg_flags(int sign, int width) { return (uint32_t)(sign & 1) | ((uint32_t)width << 4); }

// Programmatic dependent launches: a kernel launched as the dependent of the stream's last
// kernel may be scheduled once every block of that one has passed allow_dependent() or
// ended, and waits for its end, memory included, in await_predecessor() (which returns at
// once in a plain launch).
__device__ __forceinline__ void await_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependent() { asm volatile("griddepcontrol.launch_dependents;"); }

// Instantiation of the term kernel for a table whose moduli lie in [min_m, max_m]:
// 0 the width-1 and lazy kinds only (m < 2^29), 1 all one-word kinds (m < 2^32), 2 also
// the float-quotient and short two-word kinds (m < 2^44), 3 any kind but without the
// float-quotient steps (moduli below 94 * 2^32 take the short kind's there). A kernel's
// registers and code follow its widest kind: one-word terms ran 5 % slower beside the
// float-quotient steps, and short two-word terms are 2 % faster at level 3 than
// beside the float-quotient steps, so a table without moduli for those takes level 3.
constexpr int kTermLevels = 4;
__host__ __device__ inline int term_level(uint64_t min_m, uint64_t max_m)
{
    return max_m < kW1LMax ? 0 : max_m < kW1SMax ? 1 : max_m < kW2SMax && min_m < kW2FMax ? 2 : 3;
}

constexpr int kBlock192 = 128;            // threads of the term kernel's blocks

// How a pass without a time budget deals its tiles out: from the tile counter, or
// (fixed) as 2^log2_parts parts of part_k terms each, one contiguous share a block.
struct TileSplit {
    uint32_t log2_parts, fixed, part_k;
};

// A pass with fewer tiles than resident warps leaves most of the GPU idle and its
// lanes a long serial run (position 1e6: 1367 tiles for 6080 warps, 64 terms a
// lane). Its tiles are cut into parts of down to 64 terms, about four a warp, and
// every block takes one contiguous share: no counter to wait for, and one slot
// update a block instead of one a part (those queue at three cache lines: 141 us
// at 1e6). Measured, term kernel: 1e4 24.5 -> 8 us, 1e5 39 -> 10.4 us, 1e6 52 -> 39 us,
// 2^20 terms at 1e11 187 -> 64 us. From one tile a warp on, contiguous shares lose to
// the counter (1e7 268 -> 274 us, 1e8 2.61 -> 2.82 ms): costs differ along the table.
inline TileSplit tile_split(uint64_t ntiles, uint32_t tile_k, int grid)
{
    const uint64_t warps = (uint64_t)grid * (kBlock192 / 32);
    TileSplit sp{0, 0, tile_k};
    if (ntiles >= warps) return sp;
    sp.fixed = 1;
    while (sp.part_k > 64 && (ntiles << sp.log2_parts) < 4 * warps) {
        ++sp.log2_parts;
        const uint64_t unit = 64ull << sp.log2_parts;              // rounded up: the parts cover the tile
        sp.part_k = (uint32_t)((tile_k + unit - 1) / unit) * 64;
    }
    return sp;
}

// cbl_set_tuning, the autotuner with its cache file, and cbl_prepared_info count CTAs of
// 256 threads, whatever blocks the kernels run in: resident warps, and so the meaning of a
// stored or written setting, do not change with the kernels' block size. Blocks an SM for
// a setting (0 = as many as are resident, which is also the most: one wave at every level).
constexpr int kCtaThreads = 256;
inline int tuned_blocks(int ctas, int resident)
{
    return ctas > 0 && ctas < resident && ctas * (kCtaThreads / kBlock192) < resident
               ? ctas * (kCtaThreads / kBlock192) : resident;
}
inline int blocks_to_ctas(int blocks) { return (blocks + kCtaThreads / kBlock192 - 1) / (kCtaThreads / kBlock192); }

// Most flushes into one slot that a pass can make: a warp or block flushes only sums of
// tiles of its own or, in the fixed form, of parts of its own (one 2048-term tile is up to
// 32 parts in as many blocks, each with its flush).
inline uint64_t flush_bound(uint64_t ntiles, uint32_t tile_k, int grid)
{
    return ntiles << tile_split(ntiles, tile_k, grid).log2_parts;
}

// Resident blocks (of one SM, or of a grid) of the term kernel's two forms.
struct TermGrid {
    int tiles = 0;         // tiles from the counter
    int shares = 0;        // fixed shares
};

// Launch wrappers (cbl_kernels.cu).
// budget_ns = 0: run to the end; else warps stop taking tiles after budget_ns
// and the finished tiles are [0, *counter).
// reset_counter: zero the tile counter first, where the launch uses it.
// carry: the slots' digit sums may wrap past 2^64 (a slot can receive 2^31 or
// more flushes since it was zeroed, or it started from a preset); the flushes
// then carry each wrap into the digit sum two places up (exact mod 2^192).
// slot_needs_carry() decides it from flush_bound().
// dependent: the stream's last operation is the kernel that wrote segs; the launch is its
// programmatic dependent (cbl_kernels.cu).
cudaError_t launch_terms192(int level, const Seg *segs, int nseg, uint64_t ntiles, uint32_t tile_k,
                            unsigned long long *counter, unsigned long long *slots, const TermGrid &grids,
                            cudaStream_t st, uint64_t budget_ns, bool carry, bool reset_counter,
                            bool dependent = false);
constexpr uint64_t kCarryFlushes = 1ull << 31;
inline bool slot_needs_carry(uint64_t max_flushes) { return max_flushes >= kCarryFlushes; }
// slots (nslot x 6 digit sums) of position i, series f = slots[(7 i + f) * 6 ..]:
// out3[3i..3i+2] (word 0 most significant) = sum_f (S_f << (numer_log2[f] + shift[i])).
// The same words also go to copy3 (n positions, may be pinned host memory) and, for
// position 0, to first3, where those are not null. dependent: as in launch_terms192.
cudaError_t launch_combine(const unsigned long long *slots, int npos, const int *shift,
                           uint64_t *out3, uint64_t *copy3, uint64_t *first3, cudaStream_t st,
                           bool dependent = false);
// slots[0 .. 6*nslot) <- preset[j % 6] (device array of 6), instead of zero.
cudaError_t launch_slot_fill(unsigned long long *slots, int nslot, const unsigned long long *preset,
                             cudaStream_t st);
// Reference-style single-series pieces on 192-bit buffers:
//  normalise slot 0 into partial[3] (Ssum_192)
cudaError_t launch_ssum192(const unsigned long long *slots, uint64_t *partial, cudaStream_t st);
//  partial <- partial << log2(numer); ans += partial (Sum7_192)
cudaError_t launch_sum7_192(uint64_t *partial, uint64_t *ans, int numer_log2, cudaStream_t st);
// Per-term evaluation (diagnostics and per-term parity).
cudaError_t launch_terms_each(uint64_t d, uint32_t den0, uint32_t den1, int sign, const uint64_t *k,
                              int n, uint64_t *out3n, cudaStream_t st);

// Double-double (mode 0) kernels. bigSum is kDDBlocks 192-bit fractions mod 1
// (little-endian words, three uint2 each), of which the first *used hold sums.
// launch_dd_terms runs at most `grid` blocks (one wave), block i adding into entry i, or
// setting it from *used on, and raises *used; k in [k0, k1) with k1 <= d, and the end_n
// (at most kEndDD + kTailDD) terms from end0 >= d - kEndDD on.
cudaError_t launch_dd_terms(int level, uint2 *bigsum, int grid, int *used, uint64_t k0, uint64_t k1, uint64_t d,
                            int sign, uint32_t den0, uint32_t den1, uint64_t end0, int end_n, cudaStream_t st);
int dd_terms_max_ctas_per_sm(int level);
cudaError_t launch_dd_ssum(const uint2 *bigsum, int nblk, double2 *partial, cudaStream_t st);
cudaError_t launch_dd_sum7(double2 *partial, double2 *ans, int numer, cudaStream_t st);

// Throughput probe: grid x block threads each run `iters` rounds of 16
// independent dependent mad.lo.u32 chains; *ops = multiply halves issued.
cudaError_t launch_probe_imad(uint32_t *sink, int grid, int block, int iters, uint64_t *ops, cudaStream_t st);
int probe_imad_grid(int sm_count);   // one full wave of probe CTAs

int device_sm_count(int device);
TermGrid terms192_ctas_per_sm(int level);

}  // namespace cbl

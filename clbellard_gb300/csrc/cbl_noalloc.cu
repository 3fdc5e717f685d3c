// cbl_noalloc.cu - an entry point for callers that may not allocate device
// memory: cbl_batch_noalloc. It evaluates up to CBL_NOALLOC_MAX_POSITIONS
// reference positions in 192-bit mode with the same persistent term kernel
// and combine kernel as cbl_batch, but every piece of scratch those kernels
// need (tile counter, per-series digit sums, per-position shifts, the tile
// table) lives in one fixed-size array defined in this file. The caller passes
// the positions and a device output buffer it already owns.
//
// The positions travel to the GPU as a kernel parameter, and a one-block
// kernel builds the tile table in the array, so a call issues no host-to-device
// copy: it enqueues three kernels on the caller's stream (the second and third as
// programmatic dependents, so they are in place when their predecessor ends) and
// returns without waiting for them.
#include "../../include/clbellard.h"
#include "cbl_internal.h"

#include <mutex>

using namespace cbl;

namespace {

constexpr int kMaxPos = CBL_NOALLOC_MAX_POSITIONS;
// One series covers k in [0, d + 20), cut at d (main body / tail) and at the
// five residue-kind boundaries m = 2^28, 2^31, 2^32, 2^44, 2^60: at most 7 pieces.
constexpr int kMaxPieces = 7;
constexpr int kMaxSegs = kMaxPos * 7 * kMaxPieces;
constexpr int kBuckets = 12;                      // (main, tail) x 6 residue kinds, costliest first
constexpr uint64_t kTileTerms = 2048;

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kOffCounter = 0;                                          // 8 bytes
constexpr size_t kOffSlots = 256;                                          // 7 x 6 digit sums per position
constexpr size_t kOffShift = align256(kOffSlots + (size_t)kMaxPos * 7 * 6 * 8);
constexpr size_t kOffSegs = align256(kOffShift + (size_t)kMaxPos * sizeof(int));
constexpr size_t kScratchBytes = align256(kOffSegs + (size_t)kMaxSegs * sizeof(Seg));
static_assert(kScratchBytes == CBL_NOALLOC_SCRATCH_BYTES, "scratch size documented in clbellard.h");

typedef unsigned __int128 u128;

// The 7 series (KernelFuncs.as:9-12) packed for host and device code alike.
__host__ __device__ __forceinline__ uint32_t series_den0(int f) { return f < 2 ? 4u : 10u; }
__host__ __device__ __forceinline__ uint32_t series_den1(int f) { return (0x9753131u >> (4 * f)) & 15u; }
__host__ __device__ __forceinline__ int series_sign(int f) { return (0x3Bu >> f) & 1u; }

// First k with den0 k + den1 >= limit; with den0 and den1 known the division folds away.
constexpr uint64_t first_k(uint64_t limit, uint64_t den0, uint64_t den1) { return (limit - den1 + den0 - 1) / den0; }

struct KindCuts {
    uint64_t k[7][5];
};

// Where each series passes the residue-kind boundaries 2^28, 2^31, 2^32, 2^44 and 2^60.
constexpr KindCuts make_kind_cuts()
{
    KindCuts c{};
    const uint64_t limit[5] = {kW1Max, kW1MMax, kW1SMax, kW2SMax, kW2Max};
    for (int f = 0; f < 7; ++f)
        for (int i = 0; i < 5; ++i) c.k[f][i] = first_k(limit[i], f < 2 ? 4 : 10, (0x9753131u >> (4 * f)) & 15u);
    return c;
}

[[maybe_unused]] constexpr KindCuts kCuts = make_kind_cuts();
__constant__ KindCuts d_cuts = make_kind_cuts();

// A piece's terms k in [k0, k1); empty where k0 >= k1.
struct Piece {
    uint64_t k0, k1;
};

// The part of series f at position d in residue kind q (0 .. 5, in order of m), main body
// or tail. k = 0 of a series with den1 = 1 has m = 1 and contributes exactly 0, so it is
// left out.
__host__ __device__ __forceinline__ Piece series_piece(uint64_t d, int f, int q, bool tail)
{
#ifdef __CUDA_ARCH__
    const uint64_t *cut = d_cuts.k[f];
#else
    const uint64_t *cut = kCuts.k[f];
#endif
    Piece p;
    p.k0 = q > 0 ? cut[q - 1] : series_den1(f) == 1 ? 1 : 0;
    p.k1 = tail ? d + kTail192 : d;
    if (tail && p.k0 < d) p.k0 = d;
    if (q < 5 && cut[q] < p.k1) p.k1 = cut[q];
    return p;
}

__host__ __device__ __forceinline__ uint64_t piece_tiles(const Piece &p)
{
    return p.k0 < p.k1 ? (p.k1 - p.k0 + kTileTerms - 1) / kTileTerms : 0;
}

struct PositionArgs {
    uint64_t d[kMaxPos];
    int n;
};

}  // namespace

// The scratch array. Every GPU that loads this library holds it until the
// process exits; all calls on a device share it.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// A piece's place among its position's series, in the eight lanes that hold them: the
// segments and tiles of the series before it, and of all of them (in lane 7's next).
struct Place {
    uint32_t seg, next_seg;
    uint64_t tile, next_tile;
};

__device__ __forceinline__ Place place_among_series(uint64_t tiles, int f)
{
    uint32_t s = tiles != 0;
    uint64_t t = tiles;
#pragma unroll
    for (int w = 1; w < 8; w *= 2) {
        const uint32_t us = __shfl_up_sync(0xffffffffu, s, w, 8);
        const uint64_t ut = __shfl_up_sync(0xffffffffu, t, w, 8);
        if (f >= w) {
            s += us;
            t += ut;
        }
    }
    return Place{s - (tiles != 0), s, t - tiles, t};
}

// One block, eight lanes a position (of kMaxPos), lane f for series f. The table is
// ordered costliest tiles first: by bucket (main body before tail, then the costlier
// residue kind), then by d (larger first, ties by position index), then by series; a
// series has at most one piece per bucket. The lanes of a position count its pieces and
// tiles per bucket under its rank in that d order, two warps scan the counts
// (bucket-major, then rank) into offsets, 12 cells a thread, then every lane writes
// its segments. The zeros for the kernels behind it go first. What bounds it is latency:
// loads, fetches of code that no warp has run yet and barriers in sequence, which is why a
// series is a lane and no loop is unrolled. With one thread a position, a memset of its own
// and plain launches behind it a call of one position at 1e4 took 26.4 us (calls in a
// row) and 64 positions at 1e4 53 us; now 19.1 and 44 us.
__global__ void __launch_bounds__(8 * kMaxPos) noalloc_table_kernel(const __grid_constant__ PositionArgs a, Seg *segs,
                                                                    uint4 *zero)
{
    __shared__ uint64_t sd[kMaxPos];
    __shared__ uint32_t seg_off[kBuckets * kMaxPos];
    __shared__ uint64_t tile_off[kBuckets * kMaxPos];
    __shared__ uint32_t warp_segs;
    __shared__ uint64_t warp_tiles;
    static_assert(kMaxPos == 64, "two warps scan");
    allow_dependent();
    const int tid = threadIdx.x, i = tid >> 3, f = tid & 7;
#pragma unroll 1
    for (int z = tid; z < (int)(kOffSegs / sizeof(uint4)); z += 8 * kMaxPos) zero[z] = make_uint4(0, 0, 0, 0);
    if (tid < kMaxPos) sd[tid] = a.d[tid];
    __syncthreads();
    const bool used = i < a.n;
    const uint64_t d = used ? sd[i] : 0;
    int rank = 0;                                           // unused positions keep their own cells, empty
#pragma unroll 1
    for (int j = f; j < a.n; j += 8) rank += sd[j] > d || (sd[j] == d && j < i);
#pragma unroll
    for (int w = 1; w < 8; w *= 2) rank += __shfl_xor_sync(0xffffffffu, rank, w);
    if (!used) rank = i;
#pragma unroll 1
    for (int b = 0; b < kBuckets; ++b) {
        const uint64_t tiles = used && f < 7 ? piece_tiles(series_piece(d, f, 5 - b % 6, b >= 6)) : 0;
        const Place at = place_among_series(tiles, f);
        if (f == 7) {
            seg_off[b * kMaxPos + rank] = at.next_seg;
            tile_off[b * kMaxPos + rank] = at.next_tile;
        }
    }
    __syncthreads();
    if (tid < 64) {                                         // exclusive scan over cells 12 tid .. 12 tid + 11
        uint32_t s = 0;
        uint64_t t = 0;
#pragma unroll 1
        for (int c = kBuckets * tid; c < kBuckets * (tid + 1); ++c) {
            s += seg_off[c];
            t += tile_off[c];
        }
        const uint32_t own_s = s;
        const uint64_t own_t = t;
        for (int w = 1; w < 32; w *= 2) {
            const uint32_t us = __shfl_up_sync(0xffffffffu, s, w);
            const uint64_t ut = __shfl_up_sync(0xffffffffu, t, w);
            if ((tid & 31) >= w) {
                s += us;
                t += ut;
            }
        }
        if (tid == 31) {
            warp_segs = s;
            warp_tiles = t;
        }
        asm volatile("bar.sync 1, 64;" ::: "memory");       // the two scanning warps
        s += (tid >= 32 ? warp_segs : 0) - own_s;
        t += (tid >= 32 ? warp_tiles : 0) - own_t;
#pragma unroll 1
        for (int c = kBuckets * tid; c < kBuckets * (tid + 1); ++c) {
            const uint32_t cs = seg_off[c];
            const uint64_t ct = tile_off[c];
            seg_off[c] = s;
            tile_off[c] = t;
            s += cs;
            t += ct;
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int b = 0; b < kBuckets; ++b) {
        const int q = 5 - b % 6;
        const Piece p = series_piece(d, f < 7 ? f : 0, q, b >= 6);
        const uint64_t tiles = used && f < 7 ? piece_tiles(p) : 0;
        const Place at = place_among_series(tiles, f);
        if (tiles == 0) continue;
        Seg s;
        s.d = d;
        s.k0 = p.k0;
        s.k1 = p.k1;
        s.tile0 = tile_off[b * kMaxPos + rank] + at.tile;
        s.den0 = series_den0(f);
        s.den1 = series_den1(f);
        s.slot = (uint32_t)(i * 7 + f);
        s.flags = (uint32_t)series_sign(f) | (((0x624351u >> (4 * q)) & 15u) << 4);     // kinds 1, 5, 3, 4, 2, 6
        segs[seg_off[b * kMaxPos + rank] + at.seg] = s;
    }
}

namespace {

struct DeviceSetup {
    bool ready = false;
    unsigned char *scratch = nullptr;   // device address of g_noalloc_scratch on this device
    TermGrid grid[kTermLevels];
};

constexpr int kMaxDevices = 64;
DeviceSetup g_setup[kMaxDevices];
std::mutex g_setup_mu;

// Once per device, with that device current: resolve the array's device
// address (the host-side name is only a stand-in), size the persistent grid,
// and load the table kernel, so later calls only enqueue work.
int setup_device(int dev, DeviceSetup **out)
{
    if (dev < 0 || dev >= kMaxDevices) return CBL_E_NODEVICE;
    std::lock_guard<std::mutex> lk(g_setup_mu);
    DeviceSetup &s = g_setup[dev];
    if (!s.ready) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) return CBL_E_CUDA;
        const int sms = device_sm_count(dev);
        if (sms <= 0) return CBL_E_CUDA;
        cudaFuncAttributes attr;
        if (cudaFuncGetAttributes(&attr, noalloc_table_kernel) != cudaSuccess) return CBL_E_CUDA;
        s.scratch = static_cast<unsigned char *>(p);
        for (int l = 0; l < kTermLevels; ++l) {
            const TermGrid per = terms192_ctas_per_sm(l);
            s.grid[l] = TermGrid{sms * per.tiles, sms * per.shares};
        }
        s.ready = true;
    }
    *out = &s;
    return CBL_OK;
}

}  // namespace

extern "C" int cbl_batch_noalloc(const uint64_t *pos, int n, uint64_t *d_out3n, void *stream)
{
    CBL_GUARD_BEGIN
    if (n < 0 || (n > 0 && (!pos || !d_out3n))) return CBL_E_ARG;
    if (n > kMaxPos) return CBL_E_LIMIT;
    if (n == 0) return CBL_OK;
    // positions as a kernel parameter; segment and tile counts from the same
    // piece arithmetic the table kernel runs
    PositionArgs args;
    args.n = n;
    int nseg = 0;
    uint64_t ntiles = 0, max_series_tiles = 0, max_m = 0;
    for (int i = 0; i < n; ++i) {
        uint64_t d = 0;
        const int rc = cbl_pos_to_d(pos[i], &d, nullptr);
        if (rc) return rc;
        if ((u128)10 * (d + kTail192 - 1) + 9 >= (u128)kW2XMax) return CBL_E_POSITION;
        args.d[i] = d;
        const uint64_t m_last = 10 * (d + kTail192 - 1) + 9;
        max_m = max_m > m_last ? max_m : m_last;
        for (int f = 0; f < 7; ++f) {
            uint64_t series_tiles = 0;
            for (int q = 0; q < 6 && (q == 0 || kCuts.k[f][q - 1] < d + kTail192); ++q)
                for (int tail = 0; tail < 2; ++tail) {
                    const uint64_t tiles = piece_tiles(series_piece(d, f, q, tail != 0));
                    nseg += tiles != 0;
                    series_tiles += tiles;
                }
            ntiles += series_tiles;
            max_series_tiles = max_series_tiles > series_tiles ? max_series_tiles : series_tiles;
        }
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return CBL_E_NODEVICE;
    DeviceSetup *ds = nullptr;
    const int rc = setup_device(dev, &ds);
    if (rc) return rc;

    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned char *base = ds->scratch;
    auto *counter = reinterpret_cast<unsigned long long *>(base + kOffCounter);
    auto *slots = reinterpret_cast<unsigned long long *>(base + kOffSlots);
    auto *shift = reinterpret_cast<int *>(base + kOffShift);
    auto *dsegs = reinterpret_cast<Seg *>(base + kOffSegs);
    // the array keeps the previous call's contents: the table kernel zeroes the counter, the
    // digit sums and the shifts and overwrites the first nseg segments
    noalloc_table_kernel<<<1, 8 * kMaxPos, 0, st>>>(args, dsegs, reinterpret_cast<uint4 *>(base));
    if (cudaGetLastError() != cudaSuccess) return CBL_E_CUDA;
    const int level = term_level(0, max_m);
    if (launch_terms192(level, dsegs, nseg, ntiles, (uint32_t)kTileTerms, counter, slots, ds->grid[level], st, 0,
                        slot_needs_carry(max_series_tiles), false, true) != cudaSuccess)
        return CBL_E_CUDA;
    if (launch_combine(slots, n, shift, d_out3n, nullptr, nullptr, st, true) != cudaSuccess) return CBL_E_CUDA;
    return CBL_OK;
    CBL_GUARD_END
}

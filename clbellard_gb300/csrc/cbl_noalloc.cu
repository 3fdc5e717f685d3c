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
// copy: it enqueues a memset and three kernels on the caller's stream and
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

struct Piece {
    uint64_t k0, k1;
    uint32_t kind;     // residue kind 1..6 (cbl_internal.h)
};

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

// The pieces of series f at position d, in increasing k. k = 0 of a series
// with den1 = 1 has m = 1 and contributes exactly 0, so it is left out.
__host__ __device__ inline int series_pieces(uint64_t d, int f, Piece out[kMaxPieces])
{
#ifdef __CUDA_ARCH__
    const uint64_t *cut = d_cuts.k[f];
#else
    const uint64_t *cut = kCuts.k[f];
#endif
    constexpr uint32_t kind[6] = {1, 5, 3, 4, 2, 6};
    uint64_t k = series_den1(f) == 1 ? 1 : 0;
    const uint64_t k1 = d + kTail192;
    int n = 0;
    for (int i = 0; i < 6; ++i) {                                    // main body and tail of each kind's range
        const uint64_t end = i < 5 && cut[i] < k1 ? cut[i] : k1;
        const uint64_t body = end < d ? end : d;
        if (k < body) {
            out[n++] = Piece{k, body, kind[i]};
            k = body;
        }
        if (k < end) {
            out[n++] = Piece{k, end, kind[i]};
            k = end;
        }
    }
    return n;
}

// Bucket of a piece: main body before tail, then the costlier residue kind
// first (wide width 2, width 2, short width 2, strict, middle, width 1).
__host__ __device__ __forceinline__ int piece_bucket(const Piece &p, uint64_t d)
{
    const int order = p.kind == 6 ? 0 : p.kind == 2 ? 1 : p.kind == 4 ? 2 : p.kind == 3 ? 3 : p.kind == 5 ? 4 : 5;
    return (p.k0 >= d ? 6 : 0) + order;
}

__host__ __device__ __forceinline__ uint64_t piece_tiles(const Piece &p)
{
    return (p.k1 - p.k0 + kTileTerms - 1) / kTileTerms;
}

struct PositionArgs {
    uint64_t d[kMaxPos];
    int n;
};

}  // namespace

// The scratch array. Every GPU that loads this library holds it until the
// process exits; all calls on a device share it.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// One block, thread i for position i (of kMaxPos). The table is ordered
// costliest tiles first: by bucket, then by d (larger first, ties by position
// index), then by series; a series has at most one piece per bucket. Thread i
// counts its pieces and tiles per bucket under its rank in that d order, the block
// scans the counts (bucket-major, then rank) into offsets, 12 cells a thread, then
// every thread writes its segments. One thread doing the scan, and 64-bit divisions
// for the cuts, made this 34 us of a 1.46 ms call.
__global__ void __launch_bounds__(kMaxPos) noalloc_table_kernel(PositionArgs a, Seg *segs)
{
    __shared__ uint32_t seg_off[kBuckets * kMaxPos];
    __shared__ uint64_t tile_off[kBuckets * kMaxPos];
    __shared__ uint32_t warp_segs;
    __shared__ uint64_t warp_tiles;
    static_assert(kMaxPos == 64, "two warps scan");
    const int i = threadIdx.x;
    for (int b = 0; b < kBuckets; ++b) {
        seg_off[b * kMaxPos + i] = 0;
        tile_off[b * kMaxPos + i] = 0;
    }
    __syncthreads();
    int rank = 0;
    uint64_t d = 0;
    Piece p[kMaxPieces];
    if (i < a.n) {
        d = a.d[i];
        for (int j = 0; j < a.n; ++j)
            if (a.d[j] > d || (a.d[j] == d && j < i)) ++rank;
        for (int f = 0; f < 7; ++f) {
            const int np = series_pieces(d, f, p);
            for (int q = 0; q < np; ++q) {
                const int c = piece_bucket(p[q], d) * kMaxPos + rank;
                seg_off[c] += 1;
                tile_off[c] += piece_tiles(p[q]);
            }
        }
    }
    __syncthreads();
    uint32_t s = 0;                                         // exclusive scan over cells 12 i .. 12 i + 11
    uint64_t t = 0;
    for (int c = kBuckets * i; c < kBuckets * (i + 1); ++c) {
        s += seg_off[c];
        t += tile_off[c];
    }
    const uint32_t own_s = s;
    const uint64_t own_t = t;
    for (int w = 1; w < 32; w *= 2) {
        const uint32_t us = __shfl_up_sync(0xffffffffu, s, w);
        const uint64_t ut = __shfl_up_sync(0xffffffffu, t, w);
        if ((i & 31) >= w) {
            s += us;
            t += ut;
        }
    }
    if (i == 31) {
        warp_segs = s;
        warp_tiles = t;
    }
    __syncthreads();
    s += (i >= 32 ? warp_segs : 0) - own_s;
    t += (i >= 32 ? warp_tiles : 0) - own_t;
    for (int c = kBuckets * i; c < kBuckets * (i + 1); ++c) {
        const uint32_t cs = seg_off[c];
        const uint64_t ct = tile_off[c];
        seg_off[c] = s;
        tile_off[c] = t;
        s += cs;
        t += ct;
    }
    __syncthreads();
    if (i >= a.n) return;
    for (int f = 0; f < 7; ++f) {
        const int np = series_pieces(d, f, p);
        for (int q = 0; q < np; ++q) {
            const int c = piece_bucket(p[q], d) * kMaxPos + rank;
            Seg s;
            s.d = d;
            s.k0 = p[q].k0;
            s.k1 = p[q].k1;
            s.tile0 = tile_off[c];
            s.den0 = series_den0(f);
            s.den1 = series_den1(f);
            s.slot = (uint32_t)(i * 7 + f);
            s.flags = (uint32_t)series_sign(f) | (p[q].kind << 4);
            segs[seg_off[c]] = s;
            seg_off[c] += 1;                                // this (bucket, rank) cell is this thread's alone
            tile_off[c] += piece_tiles(p[q]);
        }
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
        Piece p[kMaxPieces];
        for (int f = 0; f < 7; ++f) {
            const int np = series_pieces(d, f, p);
            nseg += np;
            uint64_t series_tiles = 0;
            for (int q = 0; q < np; ++q) series_tiles += piece_tiles(p[q]);
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
    // the array keeps the previous call's contents: zero the counter, the digit
    // sums and the shifts; the table kernel overwrites the first nseg segments
    if (cudaMemsetAsync(base, 0, kOffSegs, st) != cudaSuccess) return CBL_E_CUDA;
    noalloc_table_kernel<<<1, kMaxPos, 0, st>>>(args, dsegs);
    if (cudaGetLastError() != cudaSuccess) return CBL_E_CUDA;
    const int level = term_level(0, max_m);
    if (launch_terms192(level, dsegs, nseg, ntiles, (uint32_t)kTileTerms, counter, slots, ds->grid[level], st, 0,
                        slot_needs_carry(max_series_tiles), false) != cudaSuccess)
        return CBL_E_CUDA;
    if (launch_combine(slots, n, shift, d_out3n, nullptr, nullptr, st) != cudaSuccess) return CBL_E_CUDA;
    return CBL_OK;
    CBL_GUARD_END
}

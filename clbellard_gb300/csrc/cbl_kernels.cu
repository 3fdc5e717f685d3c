// cbl_kernels.cu - sm_103a kernels of the Bellard hot path.
//
//   terms192_kernel  persistent, work-stealing over warp tiles of (position,
//                    series, k-range): the 192-bit integer term sum that
//                    replaces Sglobal32mtg_192 / Sglobal64mtg_192(_Refresh) /
//                    Sglobal_after_192 (Bellard.cl:771-823, 992-1092, 1153-1253;
//                    Bellard_div2by1.cl:313-359) and their shared-memory
//                    reductions (Bellard.cl:601-675).
//   combine_kernel   Ssum_192 + Sum7_192 for every position (Bellard.cl:1300-1398).
//   dd_*             the 106-bit double-double mode (Bellard.cl:729-763, 914-982,
//                    1118-1144, 1274-1353): fractions summed as integers,
//                    double-doubles from Ssum on (the only FP64 on the GPU).
#include "cbl_arith.cuh"
#include "cbl_internal.h"
#include <algorithm>

namespace cbl {

// Programmatic dependents (cbl_internal.h) are the one-block kernels behind a term kernel
// (Ssum, Sum7), the mode-0 term kernel, and the term and combine kernels of an
// allocation-free call; each waits before it touches anything that its predecessor
// wrote or reads. Seven series at 1e7 in mode 0: 392 us with plain launches, 362 us with
// dependent Ssum and Sum7, 264 us with the term kernel too, whose terms of one series
// run beside Ssum and Sum7 of the one before.
template <typename... Params, typename... Args>
static cudaError_t launch_dependent(void (*kernel)(Params...), int grid, int block, cudaStream_t st, Args... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// numer of series f as a shift (KernelFuncs.as:9): 32,1,256,64,4,4,1
__device__ __forceinline__ int numer_log2(int f)
{
    return (int)((0x0226805u >> (4 * f)) & 15u);
}

// ---------------------------------------------------------------- helpers --
// q >>= s on N 32-bit digits (digit 0 least significant), with static register
// indexing only.
template <int N>
__device__ __forceinline__ void shr_digits(uint32_t q[N], int s)
{
    if (s >= 32 * N) {
#pragma unroll
        for (int j = 0; j < N; ++j) q[j] = 0;
        return;
    }
    const int ws = s >> 5, bs = s & 31;
#pragma unroll
    for (int t = 0; t < N - 1; ++t) {
        if (t < ws) {
#pragma unroll
            for (int j = 0; j < N - 1; ++j) q[j] = q[j + 1];
            q[N - 1] = 0;
        }
    }
#pragma unroll
    for (int j = 0; j < N - 1; ++j) q[j] = __funnelshift_r(q[j], q[j + 1], bs);
    q[N - 1] >>= bs;
}

// One term's N quotient digits: k < d gives frac(2^(10(d-k))/m), k >= d the
// tail value 2^(-10(k-d))/m (digits of 1/m shifted right by 10(k-d)).
// KIND: 1 = width 1 (m < 2^28), 9 and 10 = lazy width 1 with a start of three (2^17 <= m
// < 2^29) and four bits (2^25 <= m < 2^29), 5 = middle width 1 (2^25 <= m < 2^31),
// 3 = strict width 1 (2^31 <= m < 2^32), 7 and 8 = float-quotient width 2 (2^32 <= m
// < 15 * 2^34 and < 94 * 2^32), 4 = short width 2 (2^32 <= m < 39 * 2^40),
// 2 = width 2 (2^44 <= m < 2^60), 6 = wide width 2 (2^60 <= m < 2^62).
template <int KIND, bool TAIL, int N>
__device__ __forceinline__ void term_digits(uint64_t d, uint64_t k, uint64_t m, uint32_t q[N])
{
    const uint32_t mp = neg_inv32((uint32_t)m);
    const uint64_t E = TAIL ? 32ull * N : 10ull * (d - k) + 32ull * N;
    if (KIND == 1) {
        const uint32_t r = w1_pow2(E, (uint32_t)m, mp);
        w1_digits<N>(r, (uint32_t)m, mp, q);
    } else if (KIND == 9 || KIND == 10) {
        const uint32_t r = w1l_pow2<KIND == 9 ? 3 : 4>(E, (uint32_t)m, mp);
        w1_digits<N>(r, (uint32_t)m, mp, q);
    } else if (KIND == 5) {
        const uint32_t r = w1m_pow2(E, (uint32_t)m, mp);
        w1_digits<N>(r, (uint32_t)m, mp, q);
    } else if (KIND == 3) {
        const uint32_t r = w1s_pow2(E, (uint32_t)m, mp);
        w1_digits<N>(r, (uint32_t)m, mp, q);
    } else if (KIND == 7 || KIND == 8) {
        const uint64_t r = w2f_pow2<KIND == 8>(E, m, mp);
        w2_redc_down<N>(r, m, mp, q);
    } else if (KIND == 4) {
        const uint64_t r = w2s_pow2(E, m, mp);
        w2_redc_down<N>(r, m, mp, q);
    } else if (KIND == 6) {
        const uint64_t r = w2x_pow2(E, m, mp);
        w2_redc_down<N>(r, m, mp, q);
    } else {
        const uint64_t r = w2_pow2(E, m, mp);
        w2_redc_down<N>(r, m, mp, q);
    }
    if (TAIL) shr_digits<N>(q, (int)(10 * (k - d)));
}

// Two terms (exponents Ea and Ea - 320) of a lane per iteration, their ladders in
// turn. e_max is the largest exponent of the warp's 64. One ladder a lane measured
// 40.7 against 46.9e9 terms/s (float-quotient kinds), 21.6 against 23.1e9 (width 2 at
// 1e14), 12.1 against 13.0e9 (wide width 2 at 9e17); three and four lose again
// (terms192_kernel).
template <int KIND, int N>
__device__ __forceinline__ void term_pair(uint64_t Ea, uint64_t e_max, uint64_t ma, uint64_t mb, uint32_t qa[N],
                                          uint32_t qb[N])
{
    const uint32_t mpab = neg_inv32((uint32_t)ma * (uint32_t)mb);      // one inverse for both
    const uint32_t mpa = mpab * (uint32_t)mb, mpb = mpab * (uint32_t)ma;
    const uint64_t Eb = Ea - 320ull;
    if (KIND == 7 || KIND == 8) {
        uint64_t ra, rb;
        w2f_pow2_pair<KIND == 8>(Ea, ma, mpa, Eb, mb, mpb, e_max, ra, rb);
        w2_redc_down<N>(ra, ma, mpa, qa);
        w2_redc_down<N>(rb, mb, mpb, qb);
    } else if (KIND == 4) {
        W2SState A{0, 0, (uint32_t)ma, (uint32_t)(ma >> 32), mpa}, B{0, 0, (uint32_t)mb, (uint32_t)(mb >> 32), mpb};
        walk_bits_group<4, true>(Ea - 50, Eb - 50, e_max - 50, A, B, W2Start<50>{});     // R = 2^50
        w2_redc_down<N>(lazy_residue(A), ma, mpa, qa);
        w2_redc_down<N>(lazy_residue(B), mb, mpb, qb);
    } else if (KIND == 2) {
        W2State A{0, 0, (uint32_t)ma, (uint32_t)(ma >> 32), mpa}, B{0, 0, (uint32_t)mb, (uint32_t)(mb >> 32), mpb};
        walk_bits_group<4>(Ea - 64, Eb - 64, e_max - 64, A, B, W2Start<64>{});
        w2_redc_down<N>(lazy_residue(A), ma, mpa, qa);
        w2_redc_down<N>(lazy_residue(B), mb, mpb, qb);
    } else if (KIND == 6) {
        W2XState A = w2x_state(ma, mpa), B = w2x_state(mb, mpb);
        walk_bits_group<4>(Ea - 64, Eb - 64, e_max - 64, A, B, W2Start<64>{});
        const uint64_t ra = two_words(A.y0, A.y1), rb = two_words(B.y0, B.y1);     // below 2m
        w2_redc_down<N>(min(ra, ra - ma), ma, mpa, qa);
        w2_redc_down<N>(min(rb, rb - mb), mb, mpb, qb);
    } else if (KIND == 1) {
        W1State A{0, (uint32_t)ma, mpa}, B{0, (uint32_t)mb, mpb};
        walk_bits_group<1>(Ea - 32, Eb - 32, e_max - 32, A, B, W1Start1{});
        uint32_t ya = A.y, yb = B.y;
        ya = min(ya, ya - 2u * (uint32_t)ma);
        ya = min(ya, ya - (uint32_t)ma);
        yb = min(yb, yb - 2u * (uint32_t)mb);
        yb = min(yb, yb - (uint32_t)mb);
        w1_digits<N>(ya, (uint32_t)ma, mpa, qa);
        w1_digits<N>(yb, (uint32_t)mb, mpb, qb);
    } else if (KIND == 9 || KIND == 10) {
        W1LState A{0, (uint32_t)ma, mpa}, B{0, (uint32_t)mb, mpb};
        walk_bits_group<KIND == 9 ? 3 : 4>(Ea - 32, Eb - 32, e_max - 32, A, B, W1LStart{});
        w1_digits<N>(A.residue(), (uint32_t)ma, mpa, qa);
        w1_digits<N>(B.residue(), (uint32_t)mb, mpb, qb);
    } else if (KIND == 5) {
        W1MState A{0, (uint32_t)ma, mpa}, B{0, (uint32_t)mb, mpb};
        walk_bits_group<4>(Ea - 32, Eb - 32, e_max - 32, A, B, W1MStart{});
        w1_digits<N>(A.y, (uint32_t)ma, mpa, qa);
        w1_digits<N>(B.y, (uint32_t)mb, mpb, qb);
    } else {
        W1SState A{0, (uint32_t)ma, 0u - mpa}, B{0, (uint32_t)mb, 0u - mpb};
        walk_bits_group<4>(Ea - 32, Eb - 32, e_max - 32, A, B, W1SStart{});
        w1_digits<N>(A.y, (uint32_t)ma, mpa, qa);
        w1_digits<N>(B.y, (uint32_t)mb, mpb, qb);
    }
}

template <int KIND, bool TAIL, int N>
__device__ __forceinline__ void run_tile(const Seg &s, uint64_t kb, uint64_t ke, int lane, Acc<N> &acc,
                                         uint32_t &cnt)
{
    uint64_t k = kb + lane;
    if (!TAIL) {
        constexpr bool wide = KIND == 2 || KIND == 4 || KIND == 6 || KIND == 7 || KIND == 8;
        uint64_t ea = 10ull * (s.d - k) + 32ull * N, ma = (uint64_t)s.den0 * k + s.den1;
        uint64_t e_max = ea + 10u * lane;
        const uint64_t m32 = 32ull * s.den0;
        for (uint32_t n = (uint32_t)(ke - kb) >> 6; n > 0; --n) {   // terms k and k+32 together
            uint32_t qa[N], qb[N];
            // e_max kept in registers cost the two-word kinds more than its two adds
            // (1e10: 550.1 against 542.6 ms) and gained on the one-word kinds (1e9: 32.7 to 32.2 ms)
            term_pair<KIND, N>(ea, wide ? ea + 10u * lane : e_max, ma, ma + m32, qa, qb);
            e_max -= 640;
            ma += 2 * m32;
            ea -= 640;
            k += 64;
            acc_add(acc, qa);
            acc_add(acc, qb);
            cnt += 2;
        }
    }
    for (; k < ke; k += 32) {
        const uint64_t m = (uint64_t)s.den0 * k + s.den1;
        uint32_t q[N];
        term_digits<KIND, TAIL, N>(s.d, k, m, q);
        acc_add(acc, q);
        ++cnt;
    }
}

// Add v to element j of a slot (six 64-bit digit sums, element j weighing
// 2^(32j)), exactly mod 2^192 however many tiles land in the slot. An add that
// wraps element j past 2^64 drops 2^64 * 2^(32j) = one unit of element j+2, so
// that unit is added there (and again on the rare wrap of that add); from
// element 6 on the weight is >= 2^192 and vanishes. Each wrap is seen by
// exactly the atomic that crossed 2^64, so concurrent flushes stay exact.
__device__ __forceinline__ void slot_add(unsigned long long *slot6, int j, unsigned long long v)
{
    for (;;) {
        const unsigned long long old = atomicAdd(slot6 + j, v);
        if (old + v >= old) return;
        j += 2;
        v = 1ull;
        if (j >= 6) return;
    }
}

// Digit sums S (each below 2^56), normalised, added into a slot's six 64-bit
// digit sums. Each add is < 2^32, so a slot that receives fewer than
// 2^32 flushes from zero cannot wrap and takes plain fire-and-forget adds;
// with carry set (a slot that may receive 2^31 or more flushes, or a preset
// start value) slot_add carries the wraps, and the number of flushes per slot
// is unbounded.
__device__ __forceinline__ void add_digits(const uint64_t S[6], unsigned long long *slot6, int carry)
{
    uint64_t c = 0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const uint64_t t = S[j] + c;
        const uint32_t dj = (uint32_t)t;
        c = t >> 32;
        if (dj) {
            if (carry) slot_add(slot6, j, (unsigned long long)dj);
            else atomicAdd(slot6 + j, (unsigned long long)dj);
        }
    }
}

// Sums over a warp's lanes of the low and high halves of digit j.
__device__ __forceinline__ uint32_t warp_low(const Acc192 &acc, int j)
{
    return __reduce_add_sync(0xffffffffu, acc.w[j] & 0xffffu);
}

__device__ __forceinline__ uint32_t warp_high(const Acc192 &acc, int j)
{
    return __reduce_add_sync(0xffffffffu, acc.w[j] >> 16);
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ------------------------------------------------------- terms192 kernel --
// Fold a warp's accumulated terms of one segment and add them into its slot.
// Every k of a lane has the parity of seg.k0 + lane (tiles hold an even number
// of terms), so the lane's sign (-1)^(k + sign) is fixed for the segment.
__device__ __forceinline__ void fold_sign(const Seg &s, int lane, Acc192 &acc, uint32_t cnt)
{
    if (((s.k0 + (uint64_t)lane + (s.flags & kFlagSign)) & 1ull) != 0) acc_negate_minus(acc, cnt);
}

__device__ __forceinline__ void flush_segment(const Seg &s, int lane, Acc192 &acc, uint32_t cnt,
                                              unsigned long long *slots, int carry)
{
    fold_sign(s, lane, acc, cnt);
    uint64_t S[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) S[j] = (uint64_t)warp_low(acc, j) + ((uint64_t)warp_high(acc, j) << 16);
    if (lane == 0) add_digits(S, slots + (size_t)s.slot * 6, carry);
}

// The last flush of a block whose warps shared one run of tiles: warps still
// in warp 0's segment add up in shared memory first, so the block updates the slot once.
__device__ __forceinline__ void flush_block(const Seg *segs, int cur, int lane, Acc192 &acc, uint32_t cnt,
                                            unsigned long long *slots, int carry)
{
    __shared__ uint32_t half[12];
    __shared__ int seg0;
    if (threadIdx.x < 12) half[threadIdx.x] = 0;
    if (threadIdx.x == 0) seg0 = cur;
    __syncthreads();
    if (cur >= 0 && cur != seg0) flush_segment(segs[cur], lane, acc, cnt, slots, carry);
    else if (cur >= 0) {
        fold_sign(segs[cur], lane, acc, cnt);
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const uint32_t lo = warp_low(acc, j), hi = warp_high(acc, j);
            if (lane == 0) {
                atomicAdd(&half[2 * j], lo);
                atomicAdd(&half[2 * j + 1], hi);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && seg0 >= 0) {
        uint64_t S[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) S[j] = (uint64_t)half[2 * j] + ((uint64_t)half[2 * j + 1] << 16);
        add_digits(S, slots + (size_t)segs[seg0].slot * 6, carry);
    }
}

// One tile's terms, by residue kind and main body / tail. LEVEL limits the kinds
// that a launch can meet (term_level): the kernel's registers and code follow its
// widest kind, and the one-word kinds ran 5 % slower beside the two-word ones
// (1e9: 36.8 ms alone in the kernel, 38.8 ms with the float-quotient steps there).
template <int LEVEL, bool TAIL, int N>
__device__ __forceinline__ void run_tile_kind(const Seg &s, uint64_t kb, uint64_t ke, int lane, Acc<N> &acc,
                                              uint32_t &cnt)
{
    const int width = (int)((s.flags >> 4) & 15u);
    const uint64_t m_first = (uint64_t)s.den0 * kb + s.den1, m_last = (uint64_t)s.den0 * (ke - 1) + s.den1;
    if (LEVEL == 2 && width == 4) {
        const bool fq = TAIL || 10 * (s.d - kb) + 32 * N < kW2FExp;
        if (fq && m_last < kW2FLow) run_tile<7, TAIL>(s, kb, ke, lane, acc, cnt);
        else if (fq && m_last < kW2FMax) run_tile<8, TAIL>(s, kb, ke, lane, acc, cnt);
        else run_tile<4, TAIL>(s, kb, ke, lane, acc, cnt);
    } else if (LEVEL == 3 && (width == 4 || (width == 2 && m_last < kW2SWide))) {
        run_tile<4, TAIL>(s, kb, ke, lane, acc, cnt);
    } else if (LEVEL == 3 && width == 2) run_tile<2, TAIL>(s, kb, ke, lane, acc, cnt);
    else if (LEVEL == 3 && width == 6) run_tile<6, TAIL>(s, kb, ke, lane, acc, cnt);
    else if (LEVEL >= 1 && width == 3) run_tile<3, TAIL>(s, kb, ke, lane, acc, cnt);
    else if (LEVEL >= 1 && m_last >= kW1LMax) run_tile<5, TAIL>(s, kb, ke, lane, acc, cnt);
    else if (m_first >= kW1L4Min) run_tile<10, TAIL>(s, kb, ke, lane, acc, cnt);
    else if (m_first >= kW1L3Min) run_tile<9, TAIL>(s, kb, ke, lane, acc, cnt);
    else run_tile<1, TAIL>(s, kb, ke, lane, acc, cnt);
}

// With budget_ns != 0 a warp takes no new tile once budget_ns have passed
// since it started. The deadline is checked before the tile counter is
// incremented, so every tile taken is finished and the finished tiles are
// exactly [0, counter): a later launch continues from there.
// A warp keeps its lanes' sums across consecutive tiles of one segment and
// flushes them when it moves to another segment, when a lane's term count
// reaches 2^30, and before it exits: one slot update per run of tiles
// instead of one per tile. (split: see tile_split.)
// Registers and blocks: 128-thread blocks let ptxas have 56 registers at 9 blocks an SM
// for one-word kinds (512 positions below 1e8: 108.9 ms; 110.7 ms at 46 registers and 40
// warps in blocks of 256, 125.8 ms at 11 blocks) and 72 at 7 for the float-quotient
// kinds (1e10: 541.4 ms; 543.6 at 8, 547 at 9, 569 at 10 with spills). Three and four
// ladders a lane, with 80 and 96 registers, ran those at 548 and 595 ms, one at 613 ms.
// segs is not __restrict__: as a dependent the kernel starts while its predecessor still
// writes the table, so loads of it must stay coherent and behind await_predecessor().
template <int LEVEL, bool FIXED>
__global__ void __launch_bounds__(kBlock192, LEVEL == 2 ? 7 : 9) terms192_kernel(const Seg *segs, int nseg,
                                                             uint64_t ntiles, uint32_t tile_k, TileSplit split,
                                                             unsigned long long *counter,
                                                             unsigned long long *slots, uint64_t budget_ns,
                                                             int carry)
{
    const int lane = threadIdx.x & 31;
    allow_dependent();
    await_predecessor();                            // the tile table's kernel, where one precedes
    const uint64_t t_start = budget_ns ? global_ns() : 0;
    uint64_t nitems = ntiles, item = 0;
    if (FIXED) {                                    // this block's share, dealt to its warps in turn
        nitems <<= split.log2_parts;
        item = nitems * blockIdx.x / gridDim.x + (threadIdx.x >> 5);
        nitems = nitems * (blockIdx.x + 1) / gridDim.x;
    }
    int cur = -1;                                   // segment of the sums held in acc
    int seg = 0;                                    // segment of the last item
    Acc192 acc;
    acc_zero(acc);
    uint32_t cnt = 0;
    for (;; item += kBlock192 / 32) {
        if (!FIXED) {
            unsigned long long t = 0;
            if (lane == 0) {
                if (budget_ns && global_ns() - t_start > budget_ns) t = ~0ull;
                else t = atomicAdd(counter, 1ull);
            }
            item = __shfl_sync(0xffffffffu, t, 0);
        }
        if (item >= nitems) break;
        const uint64_t t = FIXED ? item >> split.log2_parts : item;
        // items come in order: in a share mostly this segment's or the next one's, or a
        // part past its tile's end (64 positions below 1e5: 104 -> 96 us; the counter's
        // few, larger items gain nothing)
        int lo = 0, hi = nseg - 1;
        if (FIXED) {
            lo = seg;
            if (lo + 1 < nseg && segs[lo + 1].tile0 <= t) ++lo;
            if (lo + 1 >= nseg || segs[lo + 1].tile0 > t) hi = lo;
        }
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (segs[mid].tile0 <= t) lo = mid; else hi = mid - 1;
        }
        if (FIXED) {                                // parts past the end of their tile
            seg = lo;
            const uint64_t off = (t - segs[lo].tile0) * tile_k +
                                 ((uint32_t)item & ((1u << split.log2_parts) - 1u)) * split.part_k;
            if (segs[lo].k0 + off >= segs[lo].k1) continue;
        }
        if (lo != cur || __any_sync(0xffffffffu, cnt >= (1u << 30))) {
            if (cur >= 0) flush_segment(segs[cur], lane, acc, cnt, slots, carry);
            acc_zero(acc);
            cnt = 0;
            cur = lo;
        }
        const Seg s = segs[lo];
        uint64_t kb = s.k0 + (t - s.tile0) * tile_k, ke = min(s.k1, kb + tile_k);
        if (FIXED) {
            kb += ((uint32_t)item & ((1u << split.log2_parts) - 1u)) * split.part_k;
            ke = min(ke, kb + split.part_k);        // a last part may start past the tile's end
            if (kb >= ke) continue;
        }
        if (kb >= s.d) run_tile_kind<LEVEL, true>(s, kb, ke, lane, acc, cnt);
        else run_tile_kind<LEVEL, false>(s, kb, ke, lane, acc, cnt);
    }
    if (FIXED) flush_block(segs, cur, lane, acc, cnt, slots, carry);
    else if (cur >= 0) flush_segment(segs[cur], lane, acc, cnt, slots, carry);
}

typedef void (*Terms192Fn)(const Seg *, int, uint64_t, uint32_t, TileSplit, unsigned long long *, unsigned long long *,
                           uint64_t, int);

template <bool FIXED>
static Terms192Fn terms192_fn(int level)
{
    static const Terms192Fn fn[kTermLevels] = {terms192_kernel<0, FIXED>, terms192_kernel<1, FIXED>,
                                               terms192_kernel<2, FIXED>, terms192_kernel<3, FIXED>};
    return fn[level];
}

cudaError_t launch_terms192(int level, const Seg *segs, int nseg, uint64_t ntiles, uint32_t tile_k,
                            unsigned long long *counter, unsigned long long *slots, const TermGrid &grids,
                            cudaStream_t st, uint64_t budget_ns, bool carry, bool reset_counter, bool dependent)
{
    // a budgeted pass stops and resumes at whole tiles
    const TileSplit sp = budget_ns ? TileSplit{0, 0, tile_k} : tile_split(ntiles, tile_k, grids.tiles);
    const int grid = sp.fixed ? (int)std::min<uint64_t>(grids.shares, ntiles << sp.log2_parts) : grids.tiles;
    if (reset_counter && !sp.fixed) {
        const cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);
        if (e != cudaSuccess) return e;
    }
    const Terms192Fn fn = sp.fixed ? terms192_fn<true>(level) : terms192_fn<false>(level);
    if (dependent)
        return launch_dependent(fn, grid, kBlock192, st, segs, nseg, ntiles, tile_k, sp, counter, slots, budget_ns,
                                carry ? 1 : 0);
    fn<<<grid, kBlock192, 0, st>>>(segs, nseg, ntiles, tile_k, sp, counter, slots, budget_ns, carry ? 1 : 0);
    return cudaGetLastError();
}

template <typename Kernel>
static int max_ctas_per_sm(Kernel fn, int block)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, block, 0) != cudaSuccess) return 1;
    return n > 0 ? n : 1;
}

TermGrid terms192_ctas_per_sm(int level)
{
    return TermGrid{max_ctas_per_sm(terms192_fn<false>(level), kBlock192),
                    max_ctas_per_sm(terms192_fn<true>(level), kBlock192)};
}

int device_sm_count(int device)
{
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    return n;
}

// ------------------------------------------------------ 192-bit combine --
// Six 64-bit digit sums (digit j weighs 2^(32j)) -> 192 bits as 3 little-endian words.
__device__ __forceinline__ void normalise6(const unsigned long long *s6, uint64_t w[3])
{
    uint32_t dgt[6];
    uint64_t c = 0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const uint64_t v = s6[j];
        const uint64_t lo = (v & 0xffffffffull) + c;
        dgt[j] = (uint32_t)lo;
        c = (v >> 32) + (lo >> 32);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = ((uint64_t)dgt[2 * i + 1] << 32) | dgt[2 * i];
}

__device__ __forceinline__ void shl192(uint64_t w[3], int s)   // 0 <= s < 64, mod 2^192
{
    if (s == 0) return;
    w[2] = (w[2] << s) | (w[1] >> (64 - s));
    w[1] = (w[1] << s) | (w[0] >> (64 - s));
    w[0] <<= s;
}

__device__ __forceinline__ void add192(uint64_t a[3], const uint64_t b[3])
{
    uint64_t c = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint64_t s = a[i] + b[i];
        const uint64_t c1 = s < a[i];
        a[i] = s + c;
        c = c1 | (a[i] < s);
    }
}

// Every slot's six digit sums <- preset[0..6) (a test hook: presets near 2^64
// make the sums wrap within a few tiles).
__global__ void slot_fill_kernel(unsigned long long *slots, int nslot, const unsigned long long *preset)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nslot * 6) slots[i] = preset[i % 6];
}

cudaError_t launch_slot_fill(unsigned long long *slots, int nslot, const unsigned long long *preset,
                             cudaStream_t st)
{
    const int b = 256;
    slot_fill_kernel<<<(nslot * 6 + b - 1) / b, b, 0, st>>>(slots, nslot, preset);
    return cudaGetLastError();
}

__global__ void combine_kernel(const unsigned long long *slots, int npos, const int *shift, uint64_t *out3,
                               uint64_t *copy3, uint64_t *first3)
{
    await_predecessor();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npos) return;
    uint64_t ans[3] = {0, 0, 0};
    const int sh = shift ? shift[i] : 0;
#pragma unroll                                          // all 42 loads in flight at once
    for (int f = 0; f < 7; ++f) {
        uint64_t w[3];
        normalise6(slots + ((size_t)i * 7 + f) * 6, w);
        shl192(w, numer_log2(f) + sh);
        add192(ans, w);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        out3[3 * (size_t)i + j] = ans[2 - j];
        if (copy3) copy3[3 * (size_t)i + j] = ans[2 - j];
        if (first3 && i == 0) first3[j] = ans[2 - j];
    }
}

cudaError_t launch_combine(const unsigned long long *slots, int npos, const int *shift, uint64_t *out3,
                           uint64_t *copy3, uint64_t *first3, cudaStream_t st, bool dependent)
{
    const int b = 128;
    if (dependent)
        return launch_dependent(combine_kernel, (npos + b - 1) / b, b, st, slots, npos, shift, out3, copy3, first3);
    combine_kernel<<<(npos + b - 1) / b, b, 0, st>>>(slots, npos, shift, out3, copy3, first3);
    return cudaGetLastError();
}

__global__ void ssum192_kernel(const unsigned long long *slots, uint64_t *partial)
{
    allow_dependent();
    await_predecessor();
    uint64_t w[3];
    normalise6(slots, w);
    partial[0] = w[2]; partial[1] = w[1]; partial[2] = w[0];
}

cudaError_t launch_ssum192(const unsigned long long *slots, uint64_t *partial, cudaStream_t st)
{
    return launch_dependent(ssum192_kernel, 1, 1, st, slots, partial);
}

__global__ void sum7_192_kernel(uint64_t *partial, uint64_t *ans, int sh)
{
    await_predecessor();
    uint64_t w[3] = {partial[2], partial[1], partial[0]};
    shl192(w, sh);
    partial[0] = w[2]; partial[1] = w[1]; partial[2] = w[0];
    uint64_t a[3] = {ans[2], ans[1], ans[0]};
    add192(a, w);
    ans[0] = a[2]; ans[1] = a[1]; ans[2] = a[0];
}

cudaError_t launch_sum7_192(uint64_t *partial, uint64_t *ans, int numer_log2, cudaStream_t st)
{
    return launch_dependent(sum7_192_kernel, 1, 1, st, partial, ans, numer_log2);
}

// ---------------------------------------------------------- per-term kernel --
__global__ void terms_each_kernel(uint64_t d, uint32_t den0, uint32_t den1, int sign, const uint64_t *ks, int n,
                                  uint64_t *out3n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t k = ks[i];
    const uint64_t m = (uint64_t)den0 * k + den1;
    uint32_t q[6] = {0, 0, 0, 0, 0, 0};
    if (m != 1) {
        if (k < d) {
            if (m < kW1L3Min) term_digits<1, false, 6>(d, k, m, q);
            else if (m < kW1L4Min) term_digits<9, false, 6>(d, k, m, q);
            else if (m < kW1LMax) term_digits<10, false, 6>(d, k, m, q);
            else if (m < kW1MMax) term_digits<5, false, 6>(d, k, m, q);
            else if (m < kW1SMax) term_digits<3, false, 6>(d, k, m, q);
            else if (m < kW2FLow) term_digits<7, false, 6>(d, k, m, q);
            else if (m < kW2FMax) term_digits<8, false, 6>(d, k, m, q);
            else if (m < kW2SWide) term_digits<4, false, 6>(d, k, m, q);
            else if (m < kW2Max) term_digits<2, false, 6>(d, k, m, q);
            else term_digits<6, false, 6>(d, k, m, q);
        } else {
            if (m < kW1L3Min) term_digits<1, true, 6>(d, k, m, q);
            else if (m < kW1L4Min) term_digits<9, true, 6>(d, k, m, q);
            else if (m < kW1LMax) term_digits<10, true, 6>(d, k, m, q);
            else if (m < kW1MMax) term_digits<5, true, 6>(d, k, m, q);
            else if (m < kW1SMax) term_digits<3, true, 6>(d, k, m, q);
            else if (m < kW2SWide) term_digits<4, true, 6>(d, k, m, q);
            else if (m < kW2Max) term_digits<2, true, 6>(d, k, m, q);
            else term_digits<6, true, 6>(d, k, m, q);
        }
        if ((k + (uint64_t)sign) & 1ull)
            for (int j = 0; j < 6; ++j) q[j] = ~q[j];
    }
    out3n[3 * (size_t)i + 0] = ((uint64_t)q[5] << 32) | q[4];
    out3n[3 * (size_t)i + 1] = ((uint64_t)q[3] << 32) | q[2];
    out3n[3 * (size_t)i + 2] = ((uint64_t)q[1] << 32) | q[0];
}

cudaError_t launch_terms_each(uint64_t d, uint32_t den0, uint32_t den1, int sign, const uint64_t *k, int n,
                              uint64_t *out3n, cudaStream_t st)
{
    const int b = 128;
    terms_each_kernel<<<(n + b - 1) / b, b, 0, st>>>(d, den0, den1, sign, k, n, out3n);
    return cudaGetLastError();
}

// ------------------------------------------------------ double-double mode --
struct DD {
    double hi, lo;
};

__device__ __forceinline__ DD two_sum(double a, double b)
{
    const double s = a + b;
    const double bb = s - a;
    return DD{s, (a - (s - bb)) + (b - bb)};
}

__device__ __forceinline__ DD dd_add(DD a, DD b)
{
    DD s = two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return two_sum(s.hi, s.lo);
}

// Into (-1, 1): drop the integer part of hi (sumfix2, Bellard.cl:472-488).
__device__ __forceinline__ DD dd_frac(DD a)
{
    const double t = trunc(a.hi);
    return (t != 0.0) ? two_sum(a.hi - t, a.lo) : a;
}

constexpr int kBlockDD = 128;
constexpr int kBlockSsum = 256;

// 192-bit fraction, mod 1 and taken in [-1/2, 1/2), as a double-double: the magnitude is
// shifted up to its leading bit, so a small fraction keeps its own bits; 53 of them are the
// high double, exactly, the next 64 the low one, rounded. Integers and one addition: a
// chain of double-double additions over the words made Ssum 1 us longer (seven series
// kernel by kernel: 56 us at 1e4 and 76.6 at 1e6; 46 and 66.1 us so).
__device__ __forceinline__ DD dd_from_fraction(const uint32_t w[6])
{
    uint64_t a = ((uint64_t)w[5] << 32) | w[4], b = ((uint64_t)w[3] << 32) | w[2], c = ((uint64_t)w[1] << 32) | w[0];
    const bool minus = (int64_t)a < 0;
    if (minus) {
        c = 0ull - c;
        b = ~b + (c == 0);
        a = ~a + (b == 0 && c == 0);
    }
    int e = 0;
#pragma unroll 1
    while (a == 0 && e < 128) {
        a = b;
        b = c;
        c = 0;
        e += 64;
    }
    if (a == 0) return DD{0.0, 0.0};
    const int s = __clzll((long long)a);
    if (s > 0) {
        a = (a << s) | (b >> (64 - s));
        b = (b << s) | (c >> (64 - s));
    }
    e += s;
    const double scale = __hiloint2double((int)((uint32_t)(1023 - 53 - e) << 20 | (minus ? 0x80000000u : 0u)), 0);
    return two_sum(__ull2double_rn(a >> 11) * scale, __ull2double_rn((a << 53) | (b >> 11)) * (scale * 0x1p-64));
}

// Residue kind of a modulus (Seg::flags), and the first k of the next kind.
__device__ __forceinline__ uint32_t modulus_kind(uint64_t m, uint64_t &limit)
{
    if (m < kW1Max) { limit = kW1Max; return 1; }
    if (m < kW1MMax) { limit = kW1MMax; return 5; }
    if (m < kW1SMax) { limit = kW1SMax; return 3; }
    if (m < kW2SMax) { limit = kW2SMax; return 4; }
    if (m < kW2Max) { limit = kW2Max; return 2; }
    limit = kW2XMax;
    return 6;
}

// Add a warp's lanes' accumulators, as the top N of six digits, into half: 12 words of
// shared memory, the sums of the digits' 16-bit halves.
template <int N>
__device__ __forceinline__ void add_halves(const Acc<N> &acc, uint32_t *half)
{
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t lo = __reduce_add_sync(0xffffffffu, acc.w[j] & 0xffffu);
        const uint32_t hi = __reduce_add_sync(0xffffffffu, acc.w[j] >> 16);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&half[2 * (6 - N + j)], lo);
            atomicAdd(&half[2 * (6 - N + j) + 1], hi);
        }
    }
}

// The halves' sums, mod 1.
__device__ __forceinline__ void fraction_of(const uint32_t *half, uint32_t w[6])
{
    uint64_t c = 0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        c += (uint64_t)half[2 * j] + ((uint64_t)half[2 * j + 1] << 16);
        w[j] = (uint32_t)c;
        c >>= 32;
    }
}

// Signed fraction of one term next to d (d - k <= kEndDD) or of the tail (k >= d) in
// 192 bits: 2^(10(d-k)) / m is small there, and 128 bits would keep few of its own (66 of a
// tail at the position limit). Long division, in one warp a launch.
__device__ __forceinline__ Acc<6> end_fraction(uint64_t d, uint64_t k, uint64_t m, int sign)
{
    uint64_t r = k < d ? (1ull << 10 * (d - k)) % m : 1, top = 0, mid = 0, low = 0;
#pragma unroll 1
    for (int j = 0; j < 3; ++j) {
        const unsigned __int128 n = (unsigned __int128)r << 64;
        top = mid;
        mid = low;
        low = (uint64_t)(n / m);
        r = (uint64_t)n - low * m;
    }
    Acc<6> x{{(uint32_t)low, (uint32_t)(low >> 32), (uint32_t)mid, (uint32_t)(mid >> 32), (uint32_t)top,
              (uint32_t)(top >> 32)}};
    if (k > d) shr_digits<6>(x.w, (int)(10 * (k - d)));
    if ((k + (uint64_t)sign) & 1) acc_negate_minus(x, 0);
    return x;
}

// Terms k in [k0, k1) of one series, k1 <= d, and the terms k = end0 .. end0 + end_n - 1
// next to d and behind it. A term's fraction enters the sum as its first 128 bits: the
// ladder runs to 2^(10(d-k) + 128) and four REDC steps give them as quotient digits, as in
// the 192-bit mode. Lanes add 128-bit integers mod 1, blocks and bigSum 192-bit ones, and
// Ssum makes one double-double of the sum: FP64 (1.6 operations a clock and SM here) is left
// to Ssum and Sum7, where the terms took two divisions and 25 operations each (2^25
// terms at 1e10: 3.25 ms; 0.74 ms so). The truncations (below 2^-128 a term, of either
// sign) stay under the rounding of one double-double addition of terms of their size; the
// terms at the end, which are small by nature, come in 192 bits (end_fraction).
// Warps take tiles of tile_k terms (a multiple of 64) in turn; the last warp, which has a
// tile less than others unless they come out even, takes the end.
template <int LEVEL>
__global__ void __launch_bounds__(kBlockDD, LEVEL == 2 ? 7 : 9) dd_terms_kernel(uint2 *bigsum, uint64_t k0, uint64_t k1,
                                                                             uint64_t d, int sign, uint32_t den0,
                                                                             uint32_t den1, uint64_t tile_k,
                                                                             uint64_t end0, int end_n, int used)
{
    __shared__ uint32_t half[12];
    const int lane = threadIdx.x & 31;
    const uint64_t step = (uint64_t)gridDim.x * (kBlockDD / 32) * tile_k;
    allow_dependent();
    if (threadIdx.x < 12) half[threadIdx.x] = 0;
    __syncthreads();
    if (end_n > 0 && blockIdx.x == gridDim.x - 1 && threadIdx.x >= kBlockDD - 32) {
        const uint64_t k = end0 + lane, m = (uint64_t)den0 * k + den1;
        Acc<6> x;
        acc_zero(x);
        if (lane < end_n && m != 1) x = end_fraction(d, k, m, sign);
        add_halves<6>(x, half);
    }
    Acc<4> acc;
    acc_zero(acc);
    uint64_t odd = k0 & 1;                              // acc holds terms of lanes whose k has parity odd + lane
    uint32_t cnt = 0;
    for (uint64_t kb = k0 + ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * tile_k; kb < k1; kb += step) {
        const uint64_t ke = min(k1, kb + tile_k);
        for (uint64_t a = kb, b; a < ke; a = b) {       // one run per residue kind
            uint64_t limit;
            const Seg s{d, a, ke, 0, den0, den1, 0, modulus_kind((uint64_t)den0 * a + den1, limit) << 4};
            b = min(ke, (limit - den1 + den0 - 1) / den0);
            if ((a & 1) != odd) {
                acc_negate(acc);
                odd ^= 1;
            }
            run_tile_kind<LEVEL, false>(s, a, b, lane, acc, cnt);
        }
    }
    if ((odd + lane + sign) & 1) acc_negate(acc);
    add_halves<4>(acc, half);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t q[6];
        fraction_of(half, q);
        await_predecessor();
        Acc<6> v;
        acc_zero(v);
        uint2 *own = bigsum + 3 * blockIdx.x;
        if ((int)blockIdx.x < used) {                   // entries from `used` on hold nothing yet
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const uint2 o = own[j];
                v.w[2 * j] = o.x;
                v.w[2 * j + 1] = o.y;
            }
        }
        acc_add(v, q);
#pragma unroll
        for (int j = 0; j < 3; ++j) own[j] = make_uint2(v.w[2 * j], v.w[2 * j + 1]);
    }
}

typedef void (*DDTermsFn)(uint2 *, uint64_t, uint64_t, uint64_t, int, uint32_t, uint32_t, uint64_t, uint64_t, int,
                          int);

static DDTermsFn dd_terms_fn(int level)
{
    static const DDTermsFn fn[kTermLevels] = {dd_terms_kernel<0>, dd_terms_kernel<1>, dd_terms_kernel<2>,
                                              dd_terms_kernel<3>};
    return fn[level];
}

int dd_terms_max_ctas_per_sm(int level) { return max_ctas_per_sm(dd_terms_fn(level), kBlockDD); }

cudaError_t launch_dd_terms(int level, uint2 *bigsum, int grid, int *used, uint64_t k0, uint64_t k1, uint64_t d,
                            int sign, uint32_t den0, uint32_t den1, uint64_t end0, int end_n, cudaStream_t st)
{
    // eight tiles a resident warp: their costs fall along k, and each warp takes every eighth part
    const uint64_t warps = (uint64_t)grid * (kBlockDD / 32), n = k1 > k0 ? k1 - k0 : 0;
    const uint64_t tile_k = std::max<uint64_t>(1, (n + 8 * 64 * warps - 1) / (8 * 64 * warps)) * 64;
    const int blocks = (int)std::min<uint64_t>(grid, std::max<uint64_t>(1, (n + tile_k - 1) / tile_k));
    const cudaError_t e = launch_dependent(dd_terms_fn(level), blocks, kBlockDD, st, bigsum, k0, k0 + n, d, sign, den0,
                                           den1, tile_k, end0, end_n, *used);
    if (e == cudaSuccess) *used = std::max(*used, blocks);
    return e;
}

__global__ void __launch_bounds__(kBlockSsum) dd_ssum_kernel(const uint2 *bigsum, int nblk, double2 *partial)
{
    __shared__ uint32_t half[12];
    allow_dependent();
    if (threadIdx.x < 12) half[threadIdx.x] = 0;
    __syncthreads();
    await_predecessor();
    Acc<6> acc;
    acc_zero(acc);
    for (int i = threadIdx.x; i < nblk; i += kBlockSsum) {
        const uint2 a = bigsum[3 * i], b = bigsum[3 * i + 1], c = bigsum[3 * i + 2];
        const uint32_t q[6] = {a.x, a.y, b.x, b.y, c.x, c.y};
        acc_add(acc, q);
    }
    add_halves<6>(acc, half);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t w[6];
        fraction_of(half, w);
        const DD v = dd_from_fraction(w);
        *partial = make_double2(v.hi, v.lo);
    }
}

cudaError_t launch_dd_ssum(const uint2 *bigsum, int nblk, double2 *partial, cudaStream_t st)
{
    return launch_dependent(dd_ssum_kernel, 1, kBlockSsum, st, bigsum, nblk, partial);
}

__device__ __forceinline__ DD dd_unit(DD a)   // into [0, 1)
{
    a = dd_frac(a);
    if (a.hi < 0.0 || (a.hi == 0.0 && a.lo < 0.0)) a = dd_add(a, DD{1.0, 0.0});
    if (a.hi >= 1.0) a = dd_add(a, DD{-1.0, 0.0});
    return a;
}

// Sum7 (Bellard.cl:1324-1353): weight by numer, keep the fraction, write back,
// add into the answer.
__global__ void dd_sum7_kernel(double2 *partial, double2 *ans, int numer)
{
    allow_dependent();
    await_predecessor();
    DD a = dd_unit(DD{partial->x, partial->y});
    a.hi *= (double)numer;
    a.lo *= (double)numer;
    a = dd_unit(a);
    *partial = make_double2(a.hi, a.lo);
    const DD s = dd_unit(dd_add(DD{ans->x, ans->y}, a));
    *ans = make_double2(s.hi, s.lo);
}

cudaError_t launch_dd_sum7(double2 *partial, double2 *ans, int numer, cudaStream_t st)
{
    return launch_dependent(dd_sum7_kernel, 1, 1, st, partial, ans, numer);
}

}  // namespace cbl

namespace cbl {

// ------------------------------------------------------------ IMAD probe --
// 16 independent dependent chains of mad.lo.u32 per thread, one multiply half
// per instruction: the full issue rate of the FMA-heavy pipe, which is the
// peak of the term kernels' algorithmic work unit (a multiply half).
__global__ void __launch_bounds__(256) probe_imad_kernel(uint32_t *sink, int iters)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t x[16], a[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        a[j] = t * 2654435761u + 7919u * j;
        x[j] = (t ^ (0x9e3779b9u * (j + 1))) | 1u;
    }
    const uint32_t k1 = 0x7feb352du;
    // 16 independent chains x = x k1 + a: each multiply needs the previous
    // one's result, so none can be hoisted out of the loop, and 16 chains per
    // thread hide the latency: the issue rate of mad.lo.u32 (one multiply half
    // each) is measured. A full 32x32 product (two halves) issues at half this
    // rate, so the rate of halves is the same for wide products.
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 16; ++j) asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(x[j]) : "r"(k1), "r"(a[j]));
    }
    uint32_t r = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) r ^= x[j];
    sink[t] = r;
}

int probe_imad_grid(int sm_count)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, probe_imad_kernel, 256, 0) != cudaSuccess || n < 1) n = 1;
    return sm_count * n;
}

cudaError_t launch_probe_imad(uint32_t *sink, int grid, int block, int iters, uint64_t *ops, cudaStream_t st)
{
    (void)block;
    probe_imad_kernel<<<grid, 256, 0, st>>>(sink, iters);
    if (ops) *ops = (uint64_t)grid * block * (uint64_t)iters * 16ull;   // one half per mad.lo
    return cudaGetLastError();
}

}  // namespace cbl

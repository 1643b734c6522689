// count_kernel.cuh -- the tcgen05 counting kernel: contingency counts of SNP
// pairs or triplets, scored (or stored) without the counts ever forming a
// table in memory.
//
// One tile is 128 A SNPs x NZ B SNPs (256 x 2 NZ operand rows, one row per
// {SNP, genotype plane}).  A CTA pair multiplies it with
// tcgen05.mma.cta_group::2.kind::mxf4, M = 256, N = 2 NZ, one *segment* of the
// K range at a time:
//   pairs:    {cases, controls};
//   triplets: {cases, controls} x {X genotype a, X genotype b}.
// The 512 TMEM columns hold two accumulators of 2 NZ columns (and the block
// scales), used in turn: while one segment is multiplied the previous one is
// drained.  Per CTA (448 threads, one CTA per SM, persistent over the tiles):
//   warp 0       TMA producer, kStages K blocks in flight;
//   warp 1       MMA issuer (even CTA of the pair), never waits for scoring;
//   warps 2-5    drain: tcgen05.ld of a finished segment, counts packed to 16
//                bits, written to a two-tile ring in global memory (L2);
//   warps 6-13   scoring: read the tile's counts back, one set per lane, bound
//                every score, score the survivors.
//
// Why this split (measured on a B200): the MMA itself takes N / 2 clocks (56 for
// N = 112, 112 for N = 224) whatever the number of MMAs per commit, 4470 TMAC/s
// on the chip (nvidia-smi at 1965 MHz, the SM's cycle counter at 1845), so the
// tensor pipe wants MMAs back to back and operands at 64 bytes per clock and SM.
// A tile of N = 112 needs 103 (4 KB of A and 1.75 KB of B per 56 clocks), one of
// N = 224 needs 67.  With all four segments of a triplet tile in TMEM at once N cannot
// pass 112, and the scoring of a tile holds its accumulators; moving finished
// segments out costs 57 KB of L2 traffic each (against 1 to 4 MB of operands)
// and frees both N and the issuer.  One eighth of the 4096 x 262144 K2 search: 531
// ms with four segments in TMEM and exact scoring beside them, 259 ms so; one
// sixteenth of the 8192 x 65536 MI search 750 -> 320 ms; 1536 SNPs x 40000 samples
// K2 132 -> 40 ms; all pairs of 16384 SNPs x 32768 samples MI 12.1 -> 6.1 ms
// (repeated for seconds, under the power cap).
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "device_data.cuh"
#include "tc_ptx.cuh"

namespace episdet {
namespace tc {

constexpr int kTileA = 128;                 // A SNPs of a tile (64 per CTA)
constexpr int kCtaRows = 128;               // A rows of a CTA
constexpr int kKB = 128;                    // bytes of one K block of a row
constexpr int kF4PerKB = 2 * kKB;           // packed e2m1 samples of a K block
constexpr int kABytes = kCtaRows * kKB;
// Packed samples per class region of a regrouped row: two segments padded to
// whole K blocks need at most n + 2 * (kF4PerKB - 1) <= Kc + kClassPad.
constexpr int kClassPad = 2 * kF4PerKB;
constexpr int kDrainWarps = 4;
constexpr int kScoreWarps = 8;
constexpr int kScoreThreads = 32 * kScoreWarps;
constexpr int kThreads = 64 + 32 * kDrainWarps + kScoreThreads;
constexpr int kMaxGroup = 64;               // first SNPs of a launch at most
constexpr int kWideZ = 112, kNarrowZ = 56;  // B SNPs of a tile
// Candidate list of a CTA (global memory): its fill is checked once per tile,
// so it holds k entries and a whole tile of offers.
constexpr int kCapG = 16384;
static_assert((kTileA / 2) * kNarrowZ % kScoreThreads == 0, "every scoring thread has the same number of sets of a tile");
static_assert((kTileA / 2) * kWideZ / kScoreThreads <= 32, "a thread's sets of a tile are bits of a word");
static_assert(kMaxTopK + (kTileA / 2) * kWideZ <= kCapG, "candidate list too small for one tile of offers");

// Waits for work (operand copies, MMA commits, drained segments) give up after
// CountParams::wait_ns.  Drains before exit wait for the copies and MMAs still
// in flight: up to kDrainLimitNs, or kAbortDrainNs once the CTA is aborting (a
// copy the peer CTA never issued must not hold the drain up; the pause before
// exit covers copies still landing).
constexpr uint64_t kDrainLimitNs = 4000000000ull;
constexpr uint64_t kAbortDrainNs = 2000000ull;
constexpr uint64_t kAbortPauseNs = 200000ull;

enum Mode { kStore = 0, kPairs = 1, kTriplets = 2 };

struct Seg {
    int kb0, kb1;  // K-block range [kb0, kb1)
};

// Per-X sample regrouping: genotypes ga and gb of X are kept, gd (the most
// frequent) is derived.
struct XInfo {
    int gd, ga, gb, pad;
    int len[2][2];  // [class][kept genotype] samples
    Seg seg[4];     // [class*2 + kept genotype]
};

// A window of the pair table: the AND cells (00, 01, 10, 11) x (cases,
// controls) of pair (r, col) as 8 floats at p + 8 * ((r - r0) * ld + col - c0),
// rows r >= r0, columns col > r.
struct PairView {
    const float* p;
    int r0, c0;
    long ld;
};

struct CountParams {
    ScoreTables T;
    Slots S;
    int M;
    int ngroup, ntiles;  // members (first SNPs) of this launch, tiles over all of them
    int x0;              // member g's first SNP is x0 + g (triplets)
    int rows_member;     // operand rows between members
    const int2* tiles;   // (A tile, B tile)
    int list_off[kMaxGroup], cum[kMaxGroup];  // member g: tiles[list_off[g] ..], tile numbers from cum[g]
    const uint8_t* xinfo;  // XInfo of member g at xinfo + g * xstride (triplets)
    size_t xstride;
    Seg seg2[2];  // pairs
    int first_begin, first_end;
    // Counts of derived cells: (cases, controls) of the marginal m[h] (pairs)
    // or of the pair cell (X = kept/derived genotype i, genotype h) (triplets,
    // 3 i + h), each plus tab_off, at rt + ((g * 9) + 3 i + h) * rt_ld + snp.
    const float2* rt;
    int rt_ld;
    float tab_off;
    PairView yv;        // triplets: pairs of the second and third SNP
    const float4* tot;  // label mode: [M][M] AND cells over all samples; controls = these - cases
    float* out;         // store mode: pair (r, col) at out + out_n * ((r - out_r0) * out_ld + col - out_c0)
    int out_n, out_r0, out_c0;
    long out_ld;
    uint4* stash;       // per CTA: two tiles of drained segments
    size_t stash_cta, stash_slot;
    uint32_t* seeds;    // seed pass: [grid][kScoreThreads] keys, one tile per CTA pair, no offers
    // A set whose bound L (below) is less than thr * cut_mul + cut_add scores
    // worse than thr; a set's score is at most (worse than) (L + seed_add) * seed_mul.
    double cut_mul, cut_add, seed_mul, seed_add;
    int filter;         // 0: every set is scored exactly
    int wide;           // pairs: counts do not fit 16 bits
    int one_class;      // pairs: no second segment (label mode, or the totals of one plane set)
    int* err;
    uint64_t wait_ns;   // limit of every wait for work
    const int* hold;    // failure-detection test: a word the scoring warps wait for (nothing sets it), or null
};

// Shared-memory layout.
template <int NZ>
struct Cfg {
    static constexpr int kN = 2 * NZ;               // accumulator columns of a segment
    static constexpr int kSegWords = (kTileA / 2) * NZ;  // sets of a CTA's tile: 8 (narrow) or 16 bytes of counts per segment
    static constexpr int kKbBytes = kABytes + NZ * kKB;  // one K block: 128 A rows, NZ of the pair's 2 NZ B rows
    static constexpr int kStages = NZ == kWideZ ? 6 : 8;
    static constexpr size_t kSmemBars = (size_t)kStages * kKbBytes;
    static constexpr int kNumBars = 2 * kStages + 9;  // full, empty, tfull[2], tempty[2], sfull[2], sempty[2], drain
    static constexpr size_t kSmemMisc = kSmemBars + ((kNumBars * sizeof(uint64_t) + 63) & ~size_t(63));
    static constexpr size_t kSmemGroup = kSmemMisc + 64;
    // The tile's row of each derived-cell table: [9][NZ] for the B SNPs, [6][64]
    // for the A SNPs.
    static constexpr size_t kSmemXz = kSmemGroup + (size_t)kMaxGroup * 48;
    static constexpr size_t kSmemXy = kSmemXz + (size_t)9 * NZ * 8;
    static constexpr size_t kSmemLevel = kSmemXy + (size_t)6 * (kTileA / 2) * 8;
    static constexpr size_t kSmemTotal = kSmemLevel + kLevels * sizeof(uint32_t) + 1024;
    static_assert(kSmemTotal <= 232448, "count_kernel shared memory exceeds 227 KB");
    static_assert(kKbBytes % 1024 == 0, "operand tiles must stay 1024-byte aligned");
    static_assert(2 * kN <= 448, "two accumulators and the block scales in 512 TMEM columns");
};
constexpr uint32_t kSfCol = 448;  // block scales (every byte 1.0 = UE8M0 127) in columns 448 .. 511

struct GroupSm {
    Seg seg[4];
    int ga, gb;
    int empty_mask;  // segments without samples
    int wide;        // a segment's counts may not fit 16 bits
};
static_assert(sizeof(GroupSm) == 48, "group table size");

__device__ __forceinline__ void record_error(int* err, int code) { atomicCAS(err, 0, code); }

// Waits until *word != 0; false after limit_ns.
__device__ __forceinline__ bool wait_word(const int* word, uint64_t limit_ns) {
    const uint64_t t0 = ptx::globaltimer();
    while (*(const volatile int*)word == 0) {
        if (ptx::globaltimer() - t0 > limit_ns) return false;
        __nanosleep(2000);
    }
    return true;
}

// Drain wait for copies or MMAs in flight: gives up after kDrainLimitNs, or
// after kAbortDrainNs once *abort is set.
__device__ __forceinline__ bool drain_wait(uint64_t* bar, uint32_t parity, volatile int* abort) {
    if (ptx::mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = ptx::globaltimer();
    for (uint32_t it = 1;; ++it) {
        if (ptx::mbar_try_wait(bar, parity)) return true;
        if ((it & 255) == 0) {
            const uint64_t dt = ptx::globaltimer() - t0;
            if (dt > kDrainLimitNs || (*abort && dt > kAbortDrainNs)) return false;
        }
    }
}

__device__ __forceinline__ int group_of(const CountParams& P, int t) {
    int lo = 0, hi = P.ngroup;  // the last g with cum[g] <= t
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (P.cum[mid] <= t)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// ------------------------------------------------------------ score bound
// Both scores are, up to a constant, monotone in
//   L = sum over cells of n lg n + m lg m - T lg T   (n cases, m controls)
// taken at n, m, T = n + m for MI (score = H(Y) + L / N, maximised) and at
// n + 1/2, m + 1/2, T + 3/2 for K2: by Burnside's form of Stirling's series,
//   ln v! = z ln z - z + ln(2 pi) / 2 - e(v), z = v + 1/2,
// with e positive and decreasing, and e(n) + e(m) - e(n + m + 1) > 0, so
//   score >= -(ln 2 L + 27 or 9 cells x (1/2 + ln(2 pi) / 2)),
// too small by at most 0.1176 a cell (2 e(0) - e(1) = 0.11759).  A set is scored
// exactly only if this bound, less the rounding of both sums (bound_coefficients
// in tensor.cu, checked against scores by tests/test_score_bound_cpu.py), does not rule
// it out of the list.  27 x 3 logarithms on the MUFU pipe bound the scoring: 8
// clocks a warp instruction, 648 of the 32 triplets' clocks on an SM quarter.
using f2 = unsigned long long;  // (cases, controls)
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, pack2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float lg2(float x) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Offset of a directly counted cell, and of the pair cells and marginals other
// cells are derived from (each derived cell then carries kCellOff too).
template <int SC>
constexpr float kCellOff = SC == 0 ? 0.5f : 0.0f;
constexpr float kTiny = 1e-30f;  // MI: 0 lg 0 = 0; added to a count of 1 or more it is lost

struct Bound {
    f2 acc = 0;        // (cases', controls') part of L
    float tsum = 0.0f;  // K2: sum of lg (T + 3/2), each counted half
};

template <int SC>
__device__ __forceinline__ void bound_cell(Bound& b, f2 z) {
    if (SC == 1) z = add2(z, pack2(kTiny, kTiny));
    float n, m;
    unpack2(z, n, m);
    const float t = SC == 0 ? (n + m) + 0.5f : n + m;
    const float lt = lg2(t);
    b.acc = fma2(z, sub2(pack2(lg2(n), lg2(m)), pack2(lt, lt)), b.acc);
    if (SC == 0) b.tsum += lt;
}

// The nine cells of one genotype of X (triplets) or of the whole table (pairs)
// from the four counted ones: xy the cells summed over the B genotype, xz over
// the A genotype.
template <int SC>
__device__ __forceinline__ void bound_slice(Bound& b, const f2 (&c)[2][2], f2 xy0, f2 xy1, f2 xz0, f2 xz1, f2 xz2) {
    const f2 c02 = sub2(sub2(xy0, c[0][0]), c[0][1]), c12 = sub2(sub2(xy1, c[1][0]), c[1][1]);
    bound_cell<SC>(b, c[0][0]);
    bound_cell<SC>(b, c[0][1]);
    bound_cell<SC>(b, c[1][0]);
    bound_cell<SC>(b, c[1][1]);
    bound_cell<SC>(b, c02);
    bound_cell<SC>(b, c12);
    bound_cell<SC>(b, sub2(sub2(xz0, c[0][0]), c[1][0]));
    bound_cell<SC>(b, sub2(sub2(xz1, c[0][1]), c[1][1]));
    bound_cell<SC>(b, sub2(sub2(xz2, c02), c12));
}

template <int SC>
__device__ __forceinline__ float bound_value(const Bound& b) {
    float n, m;
    unpack2(b.acc, n, m);
    return SC == 0 ? fmaf(-0.5f, b.tsum, n + m) : n + m;
}

// ------------------------------------------------------------ the stash
// A drained segment, [A SNP][B SNP]: narrow, two words of 16-bit counts (A plane
// 0, 1), each B planes 0 and 1; wide, four FP32 counts in the same order.
// 16-bit values come and go by adding 2^23 (exact for any count below it).
__device__ __forceinline__ uint32_t pack16(uint32_t lo, uint32_t hi) {
    const uint32_t a = __float_as_uint(__uint_as_float(lo) + 8388608.0f);
    const uint32_t b = __float_as_uint(__uint_as_float(hi) + 8388608.0f);
    return __byte_perm(a, b, 0x5410);
}
__device__ __forceinline__ float unpack16(uint32_t w, int hi, float off) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, hi ? 0x7632 : 0x7610)) - (8388608.0f - off);
}

// The counts [A plane][B plane] of set `idx` = yl * NZ + z in segment s, exact.
template <int NZ>
__device__ __forceinline__ float4 stash_counts(const uint4* slot, int wide, int s, int idx) {
    if (wide) return __ldcg(reinterpret_cast<const float4*>(slot) + (size_t)s * Cfg<NZ>::kSegWords + idx);
    const uint2 w = __ldcg(reinterpret_cast<const uint2*>(slot) + (size_t)s * Cfg<NZ>::kSegWords + idx);
    return make_float4((float)(w.x & 0xFFFFu), (float)(w.x >> 16), (float)(w.y & 0xFFFFu), (float)(w.y >> 16));
}

// ------------------------------------------------------------ exact score
// FP32 score of one set from its exact counts, in the reference's cell order.
// Rare (the bound rules out nearly every set): everything is read again.
template <int MODE, int SC, int NZ>
__device__ __noinline__ float exact_score(const CountParams& P, const uint4* slot, int wide, int ga, int gb, int g,
                                          int idx, int arow, int bsnp) {
    constexpr int NS = MODE == kTriplets ? 3 : 1;  // genotypes of X
    constexpr int NC = MODE == kTriplets ? 27 : 9;
    int tab[2][NC];
    const int gi[3] = {MODE == kTriplets ? ga : 0, gb, 3 - ga - gb};
    int sum[2][2][2] = {};  // [class][A plane][B plane], over the kept genotypes of X
    const float* yz = MODE == kTriplets
                          ? P.yv.p + 8 * ((size_t)(arow - P.yv.r0) * (size_t)P.yv.ld + (size_t)(bsnp - P.yv.c0))
                          : nullptr;
    for (int i = 0; i < NS; ++i) {
        int c4[2][2][2];
        for (int c = 0; c < 2; ++c) {
            int v[4];
            if (i == 2) {
                for (int e = 0; e < 4; ++e) v[e] = (int)yz[2 * e + c] - sum[c][e >> 1][e & 1];
            } else if (MODE == kPairs && P.tot && c == 1) {
                const float4 t = __ldg(P.tot + (size_t)arow * P.M + bsnp);
                v[0] = (int)t.x - c4[0][0][0], v[1] = (int)t.y - c4[0][0][1];
                v[2] = (int)t.z - c4[0][1][0], v[3] = (int)t.w - c4[0][1][1];
            } else {
                const float4 t = stash_counts<NZ>(slot, wide, MODE == kTriplets ? 2 * c + i : c, idx);
                v[0] = (int)t.x, v[1] = (int)t.y, v[2] = (int)t.z, v[3] = (int)t.w;
            }
            for (int e = 0; e < 4; ++e) {
                c4[c][e >> 1][e & 1] = v[e];
                sum[c][e >> 1][e & 1] += v[e];
            }
        }
        const float2* rt = P.rt + (size_t)(g * 9 + 3 * i) * P.rt_ld;
        for (int c = 0; c < 2; ++c) {
            auto at = [&](int h, int snp) {
                const float2 v = rt[(size_t)h * P.rt_ld + snp];
                return (int)((c ? v.y : v.x) - P.tab_off);
            };
            int* t = tab[c] + gi[i] * 9;
            t[0] = c4[c][0][0];
            t[1] = c4[c][0][1];
            t[3] = c4[c][1][0];
            t[4] = c4[c][1][1];
            t[2] = at(0, arow) - (t[0] + t[1]);
            t[5] = at(1, arow) - (t[3] + t[4]);
            t[6] = at(0, bsnp) - (t[0] + t[3]);
            t[7] = at(1, bsnp) - (t[1] + t[4]);
            t[8] = at(2, bsnp) - (t[2] + t[5]);
        }
    }
    return score32<NC, SC>(P.T, tab[0], tab[1]);
}

// Counts a scored set of this key at the lowest level it reaches, and lowers
// the search-wide key to the lowest level that k sets have reached.
__device__ __noinline__ void reach_level(const Slots& S, const uint32_t* s_level, uint32_t key) {
    if (key > s_level[0]) return;
    int j = 0;
    while (j + 1 < kLevels && key <= s_level[j + 1]) ++j;
    atomicAdd(&S.level_count[j], 1);
    // (All counts at once: one trip to L2.  Their order does not matter, since
    // each only grows.)
    int4 c[kLevels / 4];
#pragma unroll
    for (int i = 0; i < kLevels / 4; ++i) c[i] = __ldcg(reinterpret_cast<const int4*>(S.level_count) + i);
    int below = 0;
#pragma unroll
    for (int i = kLevels / 4 - 1; i >= 0; --i) {
        const int v[4] = {c[i].x, c[i].y, c[i].z, c[i].w};
#pragma unroll
        for (int e = 3; e >= 0; --e) {
            below += v[e];
            if (below >= S.k) {
                atomicMin(S.gkey, s_level[4 * i + e]);
                return;
            }
        }
    }
}

// ------------------------------------------------------------------ kernel
// MODE kStore (pair table), kPairs (2-way search) or kTriplets; SC the score (0
// = K2, 1 = MI); NZ the B SNPs of a tile.
template <int MODE, int SC, int NZ>
__global__ void __launch_bounds__(kThreads, 1)
    count_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const __grid_constant__ CountParams P) {
    using C = Cfg<NZ>;
    constexpr int kStages = C::kStages;
    constexpr int kKbBytes = C::kKbBytes;
    constexpr int NSEG = MODE == kTriplets ? 4 : 2;
    constexpr uint32_t kIdesc = ptx::idesc_mxf4(C::kN, 256);
    // Without a second class (pair totals, label mode) there is one segment.
    const int nseg = MODE != kTriplets && P.one_class ? 1 : NSEG;
    extern __shared__ uint8_t smem_raw[];
    // A launch with less dynamic shared memory than the layout needs is
    // refused before anything touches it (uniform over the pair, so no barrier
    // is left waiting).
    {
        uint32_t dyn;
        asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (dyn < (uint32_t)C::kSmemTotal) {
            if (threadIdx.x == 0) record_error(P.err, 7);
            return;
        }
    }
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kSmemBars);
    uint64_t* empty = full + kStages;
    uint64_t* tfull = empty + kStages;   // accumulator multiplied
    uint64_t* tempty = tfull + 2;        // accumulator drained (by both CTAs; the even CTA's counts)
    uint64_t* sfull = tempty + 2;        // tile in the stash
    uint64_t* sempty = sfull + 2;        // tile scored
    uint64_t* drain = sempty + 2;
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + C::kSmemMisc);
    int* s_abort = reinterpret_cast<int*>(smem + C::kSmemMisc + 4);
    int* s_never = reinterpret_cast<int*>(smem + C::kSmemMisc + 8);  // stays 0: drain waits ignore aborts
    int* s_count = reinterpret_cast<int*>(smem + C::kSmemMisc + 16);
    Cand* s_thr = reinterpret_cast<Cand*>(smem + C::kSmemMisc + 32);
    GroupSm* s_grp = reinterpret_cast<GroupSm*>(smem + C::kSmemGroup);
    f2* s_xz = reinterpret_cast<f2*>(smem + C::kSmemXz);
    f2* s_xy = reinterpret_cast<f2*>(smem + C::kSmemXy);
    uint32_t* s_level = reinterpret_cast<uint32_t*>(smem + C::kSmemLevel);
    volatile int* abort = s_abort;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < P.ngroup) {
        GroupSm gs;
        gs.wide = P.wide;
        if (MODE == kTriplets) {
            const XInfo* xi = reinterpret_cast<const XInfo*>(P.xinfo + threadIdx.x * P.xstride);
            for (int s = 0; s < 4; ++s) {
                gs.seg[s] = xi->seg[s];
                if (xi->len[s >> 1][s & 1] > 65535) gs.wide = 1;
            }
            gs.ga = xi->ga;
            gs.gb = xi->gb;
        } else {
            gs.seg[0] = P.seg2[0];
            gs.seg[1] = P.seg2[1];
            gs.seg[2] = gs.seg[3] = Seg{0, 0};
            gs.ga = 0;
            gs.gb = 1;
        }
        gs.empty_mask = 0;
        for (int s = 0; s < 4; ++s)
            if (gs.seg[s].kb1 <= gs.seg[s].kb0) gs.empty_mask |= 1 << s;
        s_grp[threadIdx.x] = gs;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            ptx::mbar_init(&full[i], 1);
            ptx::mbar_init(&empty[i], 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(&tfull[b], 1);
            ptx::mbar_init(&tempty[b], 2 * kDrainWarps);
            ptx::mbar_init(&sfull[b], kDrainWarps);
            ptx::mbar_init(&sempty[b], kScoreWarps);
        }
        ptx::mbar_init(drain, 1);
        *s_abort = 0;
        *s_never = 0;
        ptx::fence_barrier_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc_pair(s_tmem, 512);
        ptx::tmem_relinquish_pair();
    }
    if (warp == 0 && lane == 0) {
        ptx::prefetch_tmap(&tma_a);
        ptx::prefetch_tmap(&tma_b);
    }
    // The pair's barriers must be initialised before either CTA touches the other's.
    ptx::tc_fence_before();
    ptx::cluster_sync();
    ptx::tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const int rank = (int)ptx::cluster_ctarank();
    const int ncl = (int)ptx::nclusters_x();
    // Seed pass: one tile per CTA pair, spread over the launch's tiles.
    const int t_first = P.seeds ? (int)((long)ptx::cluster_id_x() * P.ntiles / ncl) : (int)ptx::cluster_id_x();
    const int t_step = P.seeds ? P.ntiles : ncl;
    // Block scale factors of every MMA, written before any MMA is issued.
    if (warp >= 2 && warp < 2 + kDrainWarps) {
        const uint32_t sf = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kSfCol;
#pragma unroll
        for (int c = 0; c < 64; c += 8) ptx::tmem_st8_fill(sf + (uint32_t)c, 0x7F7F7F7Fu);
        ptx::tmem_wait_st();
    }
    ptx::tc_fence_before();
    ptx::cluster_sync();
    ptx::tc_fence_after();

    if (warp == 0) {
        // ---------------------------------------------------- TMA producer
        if (lane == 0) {
            uint32_t stage = 0, phase = 0, pend = 0, pend_phase = 0;  // bit i: stage i
            bool ok = true;
            // The even CTA arms each stage's full barrier for both CTAs' bytes;
            // the odd CTA's copies count on that barrier too.
            const uint32_t full0 = ptx::mapa(full, 0);
            for (int t = t_first; ok && t < P.ntiles; t += t_step) {
                const int g = group_of(P, t);
                const int2 tl = P.tiles[P.list_off[g] + t - P.cum[g]];
                const int arow = g * P.rows_member + tl.x * 2 * kTileA + rank * kCtaRows;
                const int brow = g * P.rows_member + tl.y * C::kN + rank * NZ;
                for (int s = 0; ok && s < nseg; ++s) {
                    const Seg seg = s_grp[g].seg[s];
                    for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
                        if (!ptx::mbar_wait(&empty[stage], phase ^ 1, abort, P.wait_ns)) {
                            ok = false;
                            break;
                        }
                        uint8_t* sa = smem + stage * kKbBytes;
                        if (rank == 0) {
                            ptx::mbar_arrive_expect_tx(&full[stage], (uint32_t)(2 * kKbBytes));
                            // Completions land on the even CTA's barriers.
                            pend |= 1u << stage;
                            pend_phase = (pend_phase & ~(1u << stage)) | (phase << stage);
                        }
                        const uint32_t fb = full0 + stage * (uint32_t)sizeof(uint64_t);
                        ptx::tma_load_2d_pair(sa, &tma_a, kb * kKB, arow, fb);
                        ptx::tma_load_2d_pair(sa + kABytes, &tma_b, kb * kKB, brow, fb);
                        if (++stage == (uint32_t)kStages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
            if (!ok) {
                record_error(P.err, 1);
                *s_abort = 1;
            }
            // Never leave with a copy in flight: the even CTA's barriers count
            // both CTAs' copies; the odd CTA's copies of a stage the even CTA
            // never armed land during the pause before exit (see the end).
            for (int i = 0; i < kStages; ++i)
                if (((pend >> i) & 1u) && !drain_wait(&full[i], (pend_phase >> i) & 1u, abort)) record_error(P.err, 2);
        }
    } else if (warp == 1) {
        // ---------------------------------------------------- MMA issuer
        // The even CTA issues every MMA of the pair.  The warp walks the tiles
        // together and one elected lane issues, so that descriptors stay in
        // uniform registers (an issue loop under a one-lane branch took about
        // 100 clocks an MMA).
        if (rank == 0) {
            uint32_t stage = 0, phase = 0, job = 0;
            bool ok = true;
            const uint64_t desc0 = ptx::smem_desc_sw128(ptx::smem_u32(smem));
            for (int t = t_first; ok && t < P.ntiles; t += t_step) {
                const int g = group_of(P, t);
                for (int s = 0; ok && s < nseg; ++s, ++job) {
                    const uint32_t b = job & 1u, use = job >> 1;
                    const Seg seg = s_grp[g].seg[s];
                    bool w = ptx::mbar_wait_cluster(&tempty[b], (use & 1) ^ 1, abort, P.wait_ns);
                    if (!__all_sync(0xFFFFFFFFu, w)) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t d = tmem + b * (uint32_t)C::kN;
                    uint32_t acc = 0;
                    for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
                        w = ptx::mbar_wait(&full[stage], phase, abort, P.wait_ns);
                        if (!__all_sync(0xFFFFFFFFu, w)) {
                            ok = false;
                            break;
                        }
                        ptx::tc_fence_after();
                        const uint64_t ad = desc0 + (uint64_t)((stage * (uint32_t)kKbBytes) >> 4);
                        const uint64_t bd = ad + (uint64_t)(kABytes >> 4);
                        if (ptx::elect_one()) {
                            ptx::mma_mxf4_pair(d, ad, bd, kIdesc, tmem + kSfCol, tmem + kSfCol + 32, acc);
#pragma unroll
                            for (int kk = 1; kk < kKB / 32; ++kk)
                                ptx::mma_mxf4_pair(d, ad + 2 * kk, bd + 2 * kk, kIdesc, tmem + kSfCol,
                                                   tmem + kSfCol + 32, 1u);
                            ptx::mma_commit_pair_mc(&empty[stage], 0x3);  // frees the stage in both CTAs
                        }
                        __syncwarp();
                        acc = 1;
                        if (++stage == (uint32_t)kStages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                    if (ok && ptx::elect_one()) ptx::mma_commit_pair_mc(&tfull[b], 0x3);
                    __syncwarp();
                }
            }
            if (!ok && lane == 0) {
                record_error(P.err, 3);
                *s_abort = 1;
            }
            // Every MMA this warp issued completes before TMEM is released.
            if (ptx::elect_one()) ptx::mma_commit_pair_mc(drain, 0x1);
            __syncwarp();
            if (lane == 0 && !ptx::mbar_wait(drain, 0, s_never, kDrainLimitNs)) record_error(P.err, 4);
        }
    } else if (warp < 2 + kDrainWarps) {
        // ---------------------------------------------------- drain
        const int row = (warp & 3) * 32 + lane;  // the TMEM lane quarter this warp may access
        const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t tempty0 = ptx::mapa(tempty, 0);
        uint32_t job = 0;
        int local = 0;
        bool ok = true;
        for (int t = t_first; ok && t < P.ntiles; t += t_step, ++local) {
            const int g = group_of(P, t);
            const int emask = s_grp[g].empty_mask, wide = s_grp[g].wide;
            if constexpr (MODE == kTriplets) {
                // The tile's pair-table rows into L2 while its MMAs run: one
                // row of this CTA's 64 A SNPs per thread, columns past the row
                // only (the view holds no others).
                const int2 tl = P.tiles[P.list_off[g] + t - P.cum[g]];
                const int r = tl.x * kTileA + rank * (kTileA / 2) + row;
                const int z0 = max(tl.y * NZ, r + 1), nz = min(tl.y * NZ + NZ, P.M) - z0;
                if (row < kTileA / 2 && r < P.M && nz > 0)
                    ptx::prefetch_l2(P.yv.p + 8 * ((size_t)(r - P.yv.r0) * (size_t)P.yv.ld + (size_t)(z0 - P.yv.c0)),
                                     (uint32_t)nz * 32u);
            }
            uint4* slot = P.stash + (size_t)blockIdx.x * P.stash_cta + (size_t)(local & 1) * P.stash_slot;
            bool w = ptx::mbar_wait(&sempty[local & 1], ((local >> 1) & 1) ^ 1, abort, P.wait_ns);
            if (!__all_sync(0xFFFFFFFFu, w)) {
                ok = false;
                break;
            }
#pragma unroll 1
            for (int s = 0; s < nseg; ++s, ++job) {
                const uint32_t b = job & 1u;
                w = ptx::mbar_wait(&tfull[b], (job >> 1) & 1u, abort, P.wait_ns);
                if (!__all_sync(0xFFFFFFFFu, w)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                const bool zero = (emask >> s) & 1;
                const int odd = lane & 1;
                const size_t o = (size_t)s * C::kSegWords + (size_t)(row >> 1) * NZ;  // set of this lane's A SNP, B SNP 0
#pragma unroll 2
                for (int c = 0; c < C::kN; c += 16) {
                    uint32_t v[16];
                    ptx::tmem_ld16(trow + b * (uint32_t)C::kN + (uint32_t)c, v);
                    ptx::tmem_wait_ld();
                    ptx::tmem_regs_ready16(v);
                    if (zero) {
#pragma unroll
                        for (int e = 0; e < 16; ++e) v[e] = 0;
                    }
                    if (wide) {
                        uint2* out = reinterpret_cast<uint2*>(slot) + 2 * (o + c / 2) + odd;
#pragma unroll
                        for (int q = 0; q < 8; ++q) __stcg(out + 2 * q, make_uint2(v[2 * q], v[2 * q + 1]));
                    } else {
                        // The lanes of an A SNP's two planes swap halves: of each
                        // four B SNPs the even one writes the first two.
                        uint2* out = reinterpret_cast<uint2*>(slot) + o + c / 2 + 2 * odd;
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const uint32_t w0 = pack16(v[8 * q], v[8 * q + 1]), w1 = pack16(v[8 * q + 2], v[8 * q + 3]);
                            const uint32_t w2 = pack16(v[8 * q + 4], v[8 * q + 5]), w3 = pack16(v[8 * q + 6], v[8 * q + 7]);
                            const uint32_t r0 = __shfl_xor_sync(0xFFFFFFFFu, odd ? w0 : w2, 1);
                            const uint32_t r1 = __shfl_xor_sync(0xFFFFFFFFu, odd ? w1 : w3, 1);
                            __stcg(reinterpret_cast<uint4*>(out + 4 * q),
                                   odd ? make_uint4(r0, w2, r1, w3) : make_uint4(w0, r0, w1, r1));
                        }
                    }
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive_cluster(tempty0 + b * (uint32_t)sizeof(uint64_t));
            }
            if (ok && lane == 0) ptx::mbar_arrive(&sfull[local & 1]);
            __syncwarp();
        }
        if (!ok && lane == 0) {
            record_error(P.err, 5);
            *s_abort = 1;
        }
    } else {
        // ---------------------------------------------------- scoring
        const int etid = threadIdx.x - (64 + 32 * kDrainWarps);
        const BarNamed bar{1, kScoreThreads};
        const int M = P.M;
        LocalTopK<kCapG, kScoreThreads> tk{P.S.lists + (size_t)blockIdx.x * P.S.ld, s_count, s_thr, P.S.k, etid, P.S.gkey};
        if (MODE != kStore && etid == 0) {
            *s_count = P.S.counts[blockIdx.x];
            *s_thr = P.S.thr[blockIdx.x];
        }
        if (MODE != kStore && etid < kLevels) s_level[etid] = P.seeds ? 0 : P.S.level[etid];
        bar();
        float best = -INFINITY;  // seed pass: this thread's largest bound
        bool ok = true;
        int local = 0;
        for (int t = t_first; t < P.ntiles; t += t_step, ++local) {
            const int g = group_of(P, t);
            const int2 tl = P.tiles[P.list_off[g] + t - P.cum[g]];
            const int wide = s_grp[g].wide;
            const int arow0 = tl.x * kTileA + rank * (kTileA / 2);
            const int X = MODE == kTriplets ? P.x0 + g : -1;
            const float2* rt = P.rt + (size_t)(g * 9) * P.rt_ld;
            constexpr int NS = MODE == kTriplets ? 3 : 1;
            // This tile's derived-cell rows, on their way to shared memory.
            constexpr int kXz = 3 * NS * NZ, kXy = 2 * NS * (kTileA / 2);
            f2 tx[(kXz + kScoreThreads - 1) / kScoreThreads], ty[(kXy + kScoreThreads - 1) / kScoreThreads];
            if (MODE != kStore) {
#pragma unroll
                for (int e = 0; e * kScoreThreads < kXz; ++e) {
                    const int i = etid + e * kScoreThreads, h = i / NZ, snp = tl.y * NZ + i % NZ;
                    tx[e] = i < kXz && snp < M ? __ldg(reinterpret_cast<const f2*>(rt + (size_t)h * P.rt_ld + snp)) : 0;
                }
#pragma unroll
                for (int e = 0; e * kScoreThreads < kXy; ++e) {
                    const int i = etid + e * kScoreThreads, h = i / (kTileA / 2);
                    const int snp = arow0 + i % (kTileA / 2);
                    ty[e] = i < kXy && snp < M
                                ? __ldg(reinterpret_cast<const f2*>(rt + (size_t)(h / 2 * 3 + h % 2) * P.rt_ld + snp))
                                : 0;
                }
            }
            // The decision to leave must be uniform over the scoring warps
            // (they meet at a named barrier), so it is taken at one.
            bool w = true;
            if (local == 0 && P.hold) w = wait_word(P.hold, P.wait_ns);
            if (w) w = ptx::mbar_wait(&sfull[local & 1], (local >> 1) & 1, abort, P.wait_ns);
            if (bar.any(!w)) {
                ok = false;
                break;
            }
            if (MODE != kStore) {
#pragma unroll
                for (int e = 0; e * kScoreThreads < kXz; ++e)
                    if (etid + e * kScoreThreads < kXz) s_xz[etid + e * kScoreThreads] = tx[e];
#pragma unroll
                for (int e = 0; e * kScoreThreads < kXy; ++e)
                    if (etid + e * kScoreThreads < kXy) s_xy[etid + e * kScoreThreads] = ty[e];
                bar();
            }
            const uint4* slot = P.stash + (size_t)blockIdx.x * P.stash_cta + (size_t)(local & 1) * P.stash_slot;
            // The smaller of this CTA's and the search-wide k-th best key so far.
            const Cand thr = MODE == kStore ? cand_worst() : *s_thr;
            const uint32_t lim_key = MODE == kStore ? 0 : min(thr.key, *(volatile uint32_t*)P.S.gkey);
            float cut = -INFINITY;
            if (MODE != kStore && P.filter && !P.seeds) {
                const uint32_t key = lim_key;
                if (key != 0xFFFFFFFFu) cut = __double2float_rd((double)key_score(key, SC == 1) * P.cut_mul + P.cut_add);
            }
            int hi = 0;
            uint32_t keep = 0;  // this thread's sets to score exactly, bit = step
            // Set `etid + step * kScoreThreads` of the tile is A SNP yl, B SNP z.
            struct Item {
                int yl, z;
            };
            auto next = [](Item it) {
                it.yl += kScoreThreads / NZ;
                it.z += kScoreThreads % NZ;
                if (it.z >= NZ) it.z -= NZ, ++it.yl;
                return it;
            };
            auto valid = [&](Item it) {
                const int arow = arow0 + it.yl, bsnp = tl.y * NZ + it.z;
                return bsnp > arow && bsnp < M && (MODE != kTriplets || arow > X) &&
                       (MODE != kPairs || (arow >= P.first_begin && arow < P.first_end));
            };
            // What a step reads from L2, fetched kAhead steps ahead (loads took 1
            // to 2 thousand clocks while operands stream; a step of a triplet
            // tile takes about 1300, of a pairs tile 430): the packed counts
            // (narrow stash) and the set's pair-table cells, both contiguous over
            // the lanes.  (With a lane per A SNP the pair-table reads of a warp
            // touched 32 rows and took a third of the time.)  A thread without a
            // set to score there reads other valid memory.
            struct Fetched {
                uint2 u[NSEG];
                float4 y0, y1;
            };
            auto fetch = [&](Fetched& f, Item it, int step) {
                if (!wide) {
#pragma unroll
                    for (int s = 0; s < NSEG; ++s)
                        f.u[s] = s < nseg ? __ldcg(reinterpret_cast<const uint2*>(slot) + s * C::kSegWords + etid + step * kScoreThreads)
                                          : make_uint2(0, 0);
                }
                if constexpr (MODE == kTriplets) {
                    const size_t o = valid(it) ? (size_t)(arow0 + it.yl - P.yv.r0) * (size_t)P.yv.ld +
                                                     (size_t)(tl.y * NZ + it.z - P.yv.c0)
                                               : 0;
                    ptx::ld_stream8(P.yv.p + 8 * o, f.y0, f.y1);
                }
                if (MODE == kPairs && P.tot)
                    f.y0 = __ldg(P.tot + (valid(it) ? (size_t)(arow0 + it.yl) * M + tl.y * NZ + it.z : 0));
            };
            constexpr int kSteps = C::kSegWords / kScoreThreads;
            constexpr int kAhead = MODE == kTriplets ? 2 : 4;
            Item it{etid / NZ, etid % NZ}, ahead = it;
            Fetched ring[kAhead];
#pragma unroll
            for (int e = 0; e < kAhead; ++e, ahead = next(ahead)) fetch(ring[e], ahead, e);
#pragma unroll 1
            for (int step = 0; step < kSteps; step += kAhead) {
#pragma unroll
                for (int half = 0; half < kAhead; ++half, it = next(it), ahead = next(ahead)) {
                    if (kSteps % kAhead != 0 && step + half >= kSteps) break;
                    const Fetched f = ring[half];
                    if (step + half + kAhead < kSteps) fetch(ring[half], ahead, step + half + kAhead);
                    const bool here = valid(it);
                    if (!__any_sync(0xFFFFFFFFu, here)) continue;
                    const int yl = it.yl, arow = arow0 + yl, bsnp = tl.y * NZ + it.z;
                    // Counted cells (cases, controls), plus the score's offset.
                    constexpr float off = MODE == kStore ? 0.0f : kCellOff<SC>;
                    f2 c[NSEG / 2][2][2];
                    if (wide) {
#pragma unroll
                        for (int i = 0; i < NSEG / 2; ++i) {
                            const int idx = etid + (step + half) * kScoreThreads;
                            const float4 a = stash_counts<NZ>(slot, 1, i, idx);
                            const float4 b = nseg == NSEG ? stash_counts<NZ>(slot, 1, NSEG / 2 + i, idx) : make_float4(0, 0, 0, 0);
                            c[i][0][0] = pack2(a.x + off, b.x + off);
                            c[i][0][1] = pack2(a.y + off, b.y + off);
                            c[i][1][0] = pack2(a.z + off, b.z + off);
                            c[i][1][1] = pack2(a.w + off, b.w + off);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < NSEG / 2; ++i) {
                            const uint2 a = f.u[i], b = f.u[NSEG / 2 + i];
                            c[i][0][0] = pack2(unpack16(a.x, 0, off), unpack16(b.x, 0, off));
                            c[i][0][1] = pack2(unpack16(a.x, 1, off), unpack16(b.x, 1, off));
                            c[i][1][0] = pack2(unpack16(a.y, 0, off), unpack16(b.y, 0, off));
                            c[i][1][1] = pack2(unpack16(a.y, 1, off), unpack16(b.y, 1, off));
                        }
                    }
                    if constexpr (MODE == kStore) {
                        if (here) {
                            float* o = P.out + (size_t)P.out_n * ((size_t)(arow - P.out_r0) * (size_t)P.out_ld +
                                                                  (size_t)(bsnp - P.out_c0));
                            float v[8];
#pragma unroll
                            for (int j = 0; j < 2; ++j)
#pragma unroll
                                for (int k = 0; k < 2; ++k) unpack2(c[0][j][k], v[4 * j + 2 * k], v[4 * j + 2 * k + 1]);
                            if (P.out_n == 8) {
                                reinterpret_cast<float4*>(o)[0] = make_float4(v[0], v[1], v[2], v[3]);
                                reinterpret_cast<float4*>(o)[1] = make_float4(v[4], v[5], v[6], v[7]);
                            } else {
                                reinterpret_cast<float4*>(o)[0] = make_float4(v[0], v[2], v[4], v[6]);
                            }
                        }
                        continue;
                    }
                    Bound bd;
                    auto xz = [&](int i, int h) { return s_xz[(3 * i + h) * NZ + it.z]; };
                    auto xy = [&](int i, int h) { return s_xy[(2 * i + h) * (kTileA / 2) + yl]; };
                    if constexpr (MODE == kTriplets) {
                        bound_slice<SC>(bd, c[0], xy(0, 0), xy(0, 1), xz(0, 0), xz(0, 1), xz(0, 2));
                        bound_slice<SC>(bd, c[1], xy(1, 0), xy(1, 1), xz(1, 0), xz(1, 1), xz(1, 2));
                        const f2 o3 = pack2(3.0f * off, 3.0f * off);
                        const f2 yz[2][2] = {{pack2(f.y0.x, f.y0.y), pack2(f.y0.z, f.y0.w)},
                                             {pack2(f.y1.x, f.y1.y), pack2(f.y1.z, f.y1.w)}};
                        f2 d[2][2];
#pragma unroll
                        for (int j = 0; j < 2; ++j)
#pragma unroll
                            for (int k = 0; k < 2; ++k)
                                d[j][k] = sub2(sub2(add2(yz[j][k], o3), c[0][j][k]), c[1][j][k]);
                        bound_slice<SC>(bd, d, xy(2, 0), xy(2, 1), xz(2, 0), xz(2, 1), xz(2, 2));
                    } else {
                        if (P.tot) {
                            // Label mode: controls = all samples - cases.
                            const float tv[2][2] = {{f.y0.x, f.y0.y}, {f.y0.z, f.y0.w}};
#pragma unroll
                            for (int j = 0; j < 2; ++j)
#pragma unroll
                                for (int k = 0; k < 2; ++k) {
                                    float a, b;
                                    unpack2(c[0][j][k], a, b);
                                    c[0][j][k] = pack2(a, (tv[j][k] + 2.0f * off) - a);
                                }
                        }
                        bound_slice<SC>(bd, c[0], xy(0, 0), xy(0, 1), xz(0, 0), xz(0, 1), xz(0, 2));
                    }
                    const float L = MODE == kStore ? 0.0f : bound_value<SC>(bd);
                    if (MODE == kStore || !here) continue;
                    if (P.seeds) {
                        best = fmaxf(best, L);
                        continue;
                    }
                    // (Otherwise provably worse than the k-th candidate.)
                    if (!(L < cut)) keep |= 1u << (step + half);
                }
            }
            // The sets that may enter the list, scored exactly.
            if constexpr (MODE != kStore) {
                while (__any_sync(0xFFFFFFFFu, keep != 0)) {
                    if (keep == 0) continue;
                    const int e = __ffs((int)keep) - 1;
                    keep &= keep - 1;
                    const int idx = etid + e * kScoreThreads, arow = arow0 + idx / NZ, bsnp = tl.y * NZ + idx % NZ;
                    Cand cd;
                    cd.key = score_key(
                        exact_score<MODE, SC, NZ>(P, slot, wide, s_grp[g].ga, s_grp[g].gb, g, idx, arow, bsnp), SC == 1);
                    if (cd.key > lim_key) continue;
                    reach_level(P.S, s_level, cd.key);
                    cd.pad = 0;
                    cd.set = MODE == kTriplets ? set_key3((uint32_t)X, (uint32_t)arow, (uint32_t)bsnp)
                                               : set_key2((uint32_t)arow, (uint32_t)bsnp);
                    tk.offer(cd, thr, hi);
                }
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&sempty[local & 1]);
            if (MODE != kStore && !P.seeds) tk.check(hi, kCapG - (kTileA / 2) * NZ, bar);
        }
        if (!ok) {
            if (etid == 0) record_error(P.err, 6);
            *s_abort = 1;
        } else if (MODE != kStore) {
            if (P.seeds) {
                // The key of a score this set is at least as good as.
                P.seeds[(size_t)blockIdx.x * kScoreThreads + etid] =
                    best == -INFINITY ? 0xFFFFFFFFu
                                      : score_key((float)(((double)best + P.seed_add) * P.seed_mul), SC == 1);
            } else {
                bar();  // every offer has landed
                if (etid == 0) {
                    P.S.counts[blockIdx.x] = *s_count;
                    P.S.thr[blockIdx.x] = *s_thr;
                }
            }
        }
    }
    // Neither CTA of a pair may release TMEM or leave while the pair's MMAs
    // can still read its shared memory or write its accumulators.
    __syncwarp();
    ptx::tc_fence_before();
    ptx::cluster_sync();
    // After an abort, copies that no barrier of this CTA tracks (its half of a
    // stage the peer never armed) complete within microseconds: pause before
    // either CTA of the pair leaves.
    if (threadIdx.x == 0 && *abort) {
        const uint64_t t0 = ptx::globaltimer();
        while (ptx::globaltimer() - t0 < kAbortPauseNs) __nanosleep(1000);
    }
    __syncwarp();
    ptx::cluster_sync();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem, 512);
    }
}

}  // namespace tc
}  // namespace episdet

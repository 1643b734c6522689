// tensor.cu -- tcgen05 (5th-generation tensor core) counting engine.
//
// Counting is a matrix product over 0/1 operand rows: for rows a, b (one per
// {SNP, genotype} bit plane) sum_s a[s]*b[s] is the AND-popcount the reference
// computes as (popc a + popc b - popc(a^b))/2 from its CUTLASS XOR GEMM
// (src/helper.cu:636-637, :484-485, :714-750).  Operands are packed e2m1 (1.0 =
// nibble 2, two samples per byte), multiplied by
// tcgen05.mma.cta_group::2.kind::mxf4 with unit block scales and FP32
// accumulation (exact below 2^24).  The kernel (count_kernel.cuh) serves the
// 3-way pair table, the 2-way search and the triplet search; this file holds
// the kernels that prepare its operands and the host side.
//
// For triplets the sample columns are regrouped per first SNP X by X's
// genotype (xinfo/transpose/regroup kernels below), keeping the two genotypes
// of X with the fewest samples; the third is recovered from the Y-Z pair table
// exactly as the reference recovers genotype 2 (src/helper.cu:494-548).  This
// replaces the materialised X AND Y operand of src/helper.cu:396-425 and
// reduces the tensor work per triplet from 8 N to 4 (N - max_g count(X=g)) MACs.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "count_kernel.cuh"
#include "device_data.cuh"
#include "host_util.h"
#include "kernels.h"
#include "search_internal.h"

namespace episdet {
namespace tc {

// ------------------------------------------------------------ operand prep
// 32 samples of one row as packed e2m1.  The order of samples inside a K block
// is free as long as every row of a launch has the same one, so nibble k of
// word j takes bit 4 k + j: two instructions a word.
__device__ __forceinline__ uint4 e2m1_word(uint32_t w) {
    return make_uint4((w << 1) & 0x22222222u, w & 0x22222222u, (w >> 1) & 0x22222222u, (w >> 2) & 0x22222222u);
}

// Packed planes -> packed e2m1 operand rows, in the class-region layout of the
// regrouped triplet rows (no regrouping): row r = 2*snp + g holds the cases
// from packed sample 0 and the controls from packed sample Kc + kClassPad.
// Bits past a class's samples are left out (a cohort's may be set: its pair
// totals count the samples that the labels split, no more).  One thread per
// source word.
__global__ void __launch_bounds__(256) pack_f4_kernel(DevData D, uint8_t* __restrict__ out, int rows, int pitch) {
    const int W0 = D.W[0], W1 = D.W[1], wpr = W0 + W1;
    const int base1 = (W0 * 32 + kClassPad) / 2;  // byte offset of the controls' region
    const long total = (long)rows * wpr;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
        const int r = (int)(t / wpr), w = (int)(t % wpr);
        const int c = w < W0 ? 0 : 1;
        const int ww = w - (c ? W0 : 0);
        const int left = D.n[c] - 32 * ww;  // samples from this word on
        const uint32_t valid = left >= 32 ? ~0u : left > 0 ? ~0u << (32 - left) : 0u;
        const uint32_t word = __ldg(D.bits[c] + (size_t)r * D.W[c] + ww) & valid;
        *reinterpret_cast<uint4*>(out + (size_t)r * pitch + (c ? base1 : 0) + (size_t)ww * 16) = e2m1_word(word);
    }
}

// Counts that cells are derived from, as (cases, controls) floats plus `off`:
// the marginals m[h] of every SNP, rt[h * ld + snp] (2-way), ...
__global__ void __launch_bounds__(256) marginal_rows_kernel(DevData D, float2* __restrict__ rt, int ld, float off) {
    const int snp = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (snp >= D.M) return;
#pragma unroll
    for (int h = 0; h < 3; ++h)
        rt[(size_t)h * ld + snp] = make_float2((float)__ldg(D.marg[0] + h * D.M + snp) + off,
                                               (float)__ldg(D.marg[1] + h * D.M + snp) + off);
}

// ... or the 3 x 3 pair cells of the launch's first SNPs X = x0 + g with every
// later SNP, rt[(9 g + 3 i + h) * ld + snp], i over X's genotypes (a, b,
// derived) and h over the other SNP's (the 2-way derivation of
// src/helper.cu:645-662 from the pair's AND cells and the marginals).
__global__ void __launch_bounds__(256) pair_rows_kernel(DevData D, PairView xv, const uint8_t* __restrict__ xinfo,
                                                        size_t xstride, int x0, float2* __restrict__ rt, int ld,
                                                        float off) {
    const int snp = (int)(blockIdx.x * blockDim.x + threadIdx.x), g = (int)blockIdx.y, X = x0 + g;
    if (snp >= D.M || snp <= X) return;
    const XInfo* xi = reinterpret_cast<const XInfo*>(xinfo + g * xstride);
    const int order[3] = {xi->ga, xi->gb, xi->gd};
    const float* p = xv.p + 8 * ((size_t)(X - xv.r0) * (size_t)xv.ld + (size_t)(snp - xv.c0));
    int t[2][9];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        int mx[3], ms[3];
        load_marg3(D.marg[c], D.M, X, mx);
        load_marg3(D.marg[c], D.M, snp, ms);
        pair9_from4(t[c], make_uint4((uint32_t)p[c], (uint32_t)p[2 + c], (uint32_t)p[4 + c], (uint32_t)p[6 + c]), mx, ms);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            const int o = order[i];
            const int a = o == 0 ? t[0][h] : o == 1 ? t[0][3 + h] : t[0][6 + h];
            const int b = o == 0 ? t[1][h] : o == 1 ? t[1][3 + h] : t[1][6 + h];
            rt[(size_t)(9 * g + 3 * i + h) * ld + snp] = make_float2((float)a + off, (float)b + off);
        }
}

// Block-wide exclusive scan of one int per thread (at most 1024 threads).
__device__ __forceinline__ int block_exclusive_scan(int v, int* s_warp, int* total) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
        int z = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xFFFFFFFFu, z, o);
            if (lane >= o) z += y;
        }
        s_warp[lane] = z - w;
        if (lane == 31) *total = z;
    }
    __syncthreads();
    int r = s_warp[warp] + x - v;
    __syncthreads();
    return r;
}

// Per first SNP X and class: which genotype of X to derive (the most frequent
// over both classes), and the ascending sample indices of the two kept ones.
// Regrouping work of the first SNPs X0 .. X0 + gridDim.y - 1 of one launch: member
// m = blockIdx.y owns the XInfo and index lists at base + m * stride bytes.
struct XWork {
    uint8_t* base;     // member 0's XInfo, its index lists info_bytes after it
    size_t stride;     // bytes between members
    size_t info_bytes;
    int x0;
    int max_n;
    int* err;
    __device__ __forceinline__ XInfo* info(int m) const { return reinterpret_cast<XInfo*>(base + m * stride); }
    __device__ __forceinline__ int* idx(int m) const { return reinterpret_cast<int*>(base + m * stride + info_bytes); }
};

constexpr int kXinfoThreads = 1024;
__global__ void __launch_bounds__(kXinfoThreads) xinfo_kernel(DevData D, XWork xw) {
    __shared__ int s_warp[32];
    __shared__ int s_total;
    const int c = blockIdx.x;
    const int X = xw.x0 + (int)blockIdx.y;
    XInfo* info = xw.info(blockIdx.y);
    int* idx = xw.idx(blockIdx.y);
    const int max_n = xw.max_n;
    const int M = D.M;
    int tot[3];
#pragma unroll
    for (int g = 0; g < 3; ++g) tot[g] = __ldg(D.marg[0] + g * M + X) + __ldg(D.marg[1] + g * M + X);
    int gd = 0;
    if (tot[1] > tot[gd]) gd = 1;
    if (tot[2] > tot[gd]) gd = 2;
    // Kept genotypes, the larger group first.
    const int o1 = gd == 0 ? 1 : 0, o2 = gd == 2 ? 1 : 2;
    const int ga = tot[o2] > tot[o1] ? o2 : o1, gb = ga == o1 ? o2 : o1;
    const int W = D.W[c], n = D.n[c];
    const uint32_t* p0 = D.bits[c] + (size_t)X * 2 * W;
    const uint32_t* p1 = p0 + W;
    const int per = (W + blockDim.x - 1) / blockDim.x;
    const int w0 = threadIdx.x * per, w1 = min(W, w0 + per);
    // Class 1's region starts after class 0's Kc + kClassPad packed samples.
    const int base_kb = c == 0 ? 0 : (D.W[0] * 32 + kClassPad) / kF4PerKB;
    const int end_kb = base_kb + (W * 32 + kClassPad) / kF4PerKB;
    int kb = base_kb;
    for (int s = 0; s < 2; ++s) {
        const int g = s == 0 ? ga : gb;
        int cnt = 0;
        for (int w = w0; w < w1; ++w) {
            uint32_t m = g == 0 ? p0[w] : (g == 1 ? p1[w] : ~(p0[w] | p1[w]));
            int lo = w * 32;
            uint32_t valid = (lo + 32 <= n) ? 0xFFFFFFFFu : (lo >= n ? 0u : (0xFFFFFFFFu << (32 - (n - lo))));
            cnt += __popc(m & valid);
        }
        int off = block_exclusive_scan(cnt, s_warp, &s_total);
        int* out = idx + ((size_t)c * 2 + s) * max_n;
        for (int w = w0; w < w1; ++w) {
            uint32_t m = g == 0 ? p0[w] : (g == 1 ? p1[w] : ~(p0[w] | p1[w]));
            int lo = w * 32;
            uint32_t valid = (lo + 32 <= n) ? 0xFFFFFFFFu : (lo >= n ? 0u : (0xFFFFFFFFu << (32 - (n - lo))));
            m &= valid;
            while (m) {
                int lz = __clz(m);
                out[off++] = lo + lz;
                m &= ~(0x80000000u >> lz);
            }
        }
        int len = s_total;
        // The two kept genotypes of disjoint planes fit the class's region.
        if (kb + (len + kF4PerKB - 1) / kF4PerKB > end_kb) {
            len = 0;
            if (threadIdx.x == 0) record_error(xw.err, kErrPlanes);
        }
        if (threadIdx.x == 0) {
            info->len[c][s] = len;
            info->seg[c * 2 + s].kb0 = kb;
            info->seg[c * 2 + s].kb1 = kb + (len + kF4PerKB - 1) / kF4PerKB;
        }
        kb += (len + kF4PerKB - 1) / kF4PerKB;
        __syncthreads();
    }
    if (c == 0 && threadIdx.x == 0) {
        info->gd = gd;
        info->ga = ga;
        info->gb = gb;
        info->pad = 0;
    }
}

// Genotype counts of a whole cohort, [3][M], over its n samples: one warp per
// SNP.  *bad is set when a sample has both genotype planes.
__global__ void __launch_bounds__(256) cohort_marginals_kernel(const uint32_t* __restrict__ planes, int M, int n, int W,
                                                               int* __restrict__ marg, int* __restrict__ bad) {
    const int snp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (snp >= M) return;
    const uint32_t* p0 = planes + (size_t)snp * 2 * W;
    const uint32_t* p1 = p0 + W;
    int c0 = 0, c1 = 0;
    uint32_t over = 0;
    for (int w = lane; w < W; w += 32) {
        const int lo = w * 32;
        const uint32_t valid = (lo + 32 <= n) ? 0xFFFFFFFFu : (lo >= n ? 0u : (0xFFFFFFFFu << (32 - (n - lo))));
        const uint32_t a = __ldg(p0 + w) & valid, b = __ldg(p1 + w) & valid;
        c0 += __popc(a);
        c1 += __popc(b);
        over |= a & b;
    }
    c0 = __reduce_add_sync(0xFFFFFFFFu, c0);
    c1 = __reduce_add_sync(0xFFFFFFFFu, c1);
    if (over) atomicOr(bad, 1);
    if (lane == 0) {
        marg[snp] = c0;
        marg[M + snp] = c1;
        marg[2 * M + snp] = n - c0 - c1;
    }
}

// One label: the ascending case samples (as member 0's first segment of class
// 0, the form the regrouping reads) and the two classes' masks.  The operand
// rows are sized for the nc cases that the host counted: a label whose words
// have changed since is an error, and no more than nc samples are regrouped.
__global__ void __launch_bounds__(kXinfoThreads) label_lists_kernel(const uint32_t* __restrict__ label, int n, int W,
                                                                    int nc, XWork xw, uint32_t* __restrict__ mask) {
    __shared__ int s_warp[32];
    __shared__ int s_total;
    const int per = (W + kXinfoThreads - 1) / kXinfoThreads;
    const int w0 = threadIdx.x * per, w1 = min(W, w0 + per);
    int cnt = 0;
    for (int w = w0; w < w1; ++w) {
        const int lo = w * 32;
        const uint32_t valid = (lo + 32 <= n) ? 0xFFFFFFFFu : (lo >= n ? 0u : (0xFFFFFFFFu << (32 - (n - lo))));
        const uint32_t m = __ldg(label + w) & valid;
        mask[w] = m;
        mask[W + w] = ~m & valid;
        cnt += __popc(m);
    }
    int off = block_exclusive_scan(cnt, s_warp, &s_total);
    int* out = xw.idx(0);
    for (int w = w0; w < w1; ++w) {
        uint32_t m = mask[w];
        while (m) {
            const int lz = __clz(m);
            out[off++] = w * 32 + lz;
            m &= ~(0x80000000u >> lz);
        }
    }
    if (threadIdx.x == 0) {
        XInfo* info = xw.info(0);
        info->len[0][0] = min(s_total, nc);
        if (s_total != nc) record_error(xw.err, kErrLabelChanged);
        info->len[0][1] = info->len[1][0] = info->len[1][1] = 0;
    }
}

// Genotype counts of the label's cases, and of the controls as the cohort's
// minus those: one warp per SNP.
__global__ void __launch_bounds__(256) label_marginals_kernel(const uint32_t* __restrict__ planes, int M, int W,
                                                              const uint32_t* __restrict__ mask, int nc,
                                                              const int* __restrict__ total, int* __restrict__ cases,
                                                              int* __restrict__ controls) {
    const int snp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (snp >= M) return;
    const uint4* p0 = reinterpret_cast<const uint4*>(planes + (size_t)snp * 2 * W);
    const uint4* p1 = p0 + W / 4;
    const uint4* mk = reinterpret_cast<const uint4*>(mask);
    int c0 = 0, c1 = 0;
    for (int w = lane; w < W / 4; w += 32) {
        const uint4 a = __ldg(p0 + w), b = __ldg(p1 + w), m = __ldg(mk + w);
        c0 += __popc(a.x & m.x) + __popc(a.y & m.y) + __popc(a.z & m.z) + __popc(a.w & m.w);
        c1 += __popc(b.x & m.x) + __popc(b.y & m.y) + __popc(b.z & m.z) + __popc(b.w & m.w);
    }
    c0 = __reduce_add_sync(0xFFFFFFFFu, c0);
    c1 = __reduce_add_sync(0xFFFFFFFFu, c1);
    if (lane < 3) {
        const int v = lane == 0 ? c0 : lane == 1 ? c1 : nc - c0 - c1;
        cases[lane * M + snp] = v;
        controls[lane * M + snp] = total[lane * M + snp] - v;
    }
}

// Regrouped operand rows for one X: row r, class c, segment s holds the e2m1
// value bit(r, idx[c][s][k]) at packed sample position seg.kb0*256 + k (in
// e2m1_word's order within each 32; zero past the segment's length up to its
// 256-sample end).  Rows below row0 are not needed by X.
//
// Output rows of the members of one launch: member m writes rows
// [row0[m], nrows_total) at out + m * stride.
struct CmpOut {
    uint8_t* out;
    size_t stride;
    int row0[kMaxGroup];
};

// ------------------------------------------------- sample-major regrouping
// Gathering single bits of the plane rows costs about ten instructions per
// output byte, and a kernel doing that beside the counting kernel slowed it by
// 15 %.  Instead the planes are transposed once per search into sample-major
// words (tt[c][s][q]: bit 31 - i is row 32 q + i at sample s), so that
// gathering a sample is a 128-byte copy, and the gathered block is turned
// back into rows by a 32 x 32 bit transpose in registers (five shuffle
// stages).

// Rows padded to whole 256-row tiles in the sample-major layout.
constexpr int kTtRows = 256;
__host__ __device__ inline int tt_row_words(int rows) { return (rows + kTtRows - 1) / kTtRows * (kTtRows / 32); }

// Planes of class c -> tt (one warp per 256 rows x 256 samples: eight
// 32-byte reads of eight rows' words per lane, eight 32-byte writes).
constexpr int kTtThreads = 256;
__global__ void __launch_bounds__(kTtThreads) transpose_planes_kernel(DevData D, int c, uint32_t* __restrict__ tt,
                                                                      int rows, int rwp) {
    const int lane = threadIdx.x & 31;
    const int warp = (int)(blockIdx.x * (kTtThreads / 32) + threadIdx.x / 32);
    const int W = D.W[c];
    const int nqb = rwp / 8, nsb = W / 8;
    if (warp >= nqb * nsb) return;  // uniform over the warp
    const int qb = warp % nqb, sb = warp / nqb;
    const uint32_t* __restrict__ bits = D.bits[c];
    uint32_t out[8][8];  // [sample word][row word]
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int r = (qb * 8 + q) * 32 + lane;
        uint4 v0 = make_uint4(0, 0, 0, 0), v1 = v0;
        if (r < rows) {
            const uint4* src = reinterpret_cast<const uint4*>(bits + (size_t)r * W + sb * 8);
            v0 = __ldg(src);
            v1 = __ldg(src + 1);
        }
        const uint32_t v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) out[e][q] = warp_transpose32(v[e], lane);
    }
    // Lane k now holds, for sample 32 (sb*8 + e) + k, the words of rows
    // 32 (qb*8 + q) .. + 31 (bit 31 - i = row 32 (qb*8 + q) + i).
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        uint4* dst = reinterpret_cast<uint4*>(tt + (size_t)((sb * 8 + e) * 32 + lane) * rwp + qb * 8);
        dst[0] = make_uint4(out[e][0], out[e][1], out[e][2], out[e][3]);
        dst[1] = make_uint4(out[e][4], out[e][5], out[e][6], out[e][7]);
    }
}

// Regrouped operand rows for the members of one launch (the layout above),
// from tt: a work item is kRgRows rows x 256 packed sample positions (one K
// block) of one class region of one member.  Each thread copies the 128 bytes
// of its position's source sample (these rows: one cache line) into shared
// memory; then each lane transposes one 32 rows x 32 positions block in its own
// registers (no shuffles) and writes its 32 rows' 16 bytes, the eight lanes of
// the same rows writing whole 128-byte lines.
//
// The bound is DRAM (an eighth of the written bytes read, half a byte per row
// and kept sample written).  It does not run beside the counting kernel: in a
// form that fitted there (128 threads, 64 registers) its writes evicted the
// operands being counted and cost the counting launches of the 4096 x 262144
// search 1.1 ms for every 0.5 ms saved.
constexpr int kRgThreads = 256;
constexpr int kRgRows = 1024;
constexpr int kRgWords = kRgRows / 32;  // row words per position
constexpr int kRgCtas = 4;              // per SM
// [position][row word] with 36 words a position and 4 more each 32 positions:
// 16-byte copies stay aligned, and the per-block column reads (lanes of 4 row
// words x 8 position blocks) are free of bank conflicts.
__host__ __device__ constexpr int rg_slot(int pos, int q) { return pos * (kRgWords + 4) + 4 * (pos >> 5) + q; }
constexpr int kRgSlots = rg_slot(kRgThreads - 1, kRgWords - 1) + 1;
static_assert(kRgThreads == kF4PerKB, "an item is one K block");
static_assert(kRgSlots * 4 <= 40 * 1024, "regroup tile");

// 32 x 32 bit transpose of a[0..31] in place: afterwards bit 31 - l of a[k]
// is what bit 31 - k of a[l] was (the block-swap transpose of H. S. Warren,
// Hacker's Delight, 2nd ed., section 7-3).
__device__ __forceinline__ void transpose32(uint32_t (&a)[32]) {
    uint32_t m = 0x0000FFFFu;
#pragma unroll
    for (int j = 16; j != 0; j >>= 1, m ^= m << j) {
#pragma unroll
        for (int k = 0; k < 32; k = (k + j + 1) & ~j) {
            const uint32_t t = (a[k] ^ (a[k + j] >> j)) & m;
            a[k] ^= t;
            a[k + j] ^= t << j;
        }
    }
}

// Persistent: CTA i takes items i, i + gridDim.x, ... of the launch's list, in
// member order, each member's K blocks x its row tiles from row0 on.
__global__ void __launch_bounds__(kRgThreads, kRgCtas)
    regroup_kernel(DevData D, XWork xw, CmpOut co, const uint32_t* __restrict__ tt0, const uint32_t* __restrict__ tt1,
                   int rwp, int rows_total, int pitch, int nmem) {
    __shared__ __align__(16) uint32_t s_t[kRgSlots];  // rg_slot(position, row word)
    __shared__ int s_len[kMaxGroup][2][2];            // [member][class][segment]: samples
    __shared__ int s_first[kMaxGroup + 1];            // first item of each member
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int i = t; i < 4 * nmem; i += kRgThreads) {
        const int m = i >> 2, c = (i >> 1) & 1, sg = i & 1;
        s_len[m][c][sg] = xw.info(m)->len[c][sg];
    }
    __syncthreads();
    const int RT = (rows_total + kRgRows - 1) / kRgRows;
    // Positions of a class region: both segments padded to whole K blocks.
    auto padded = [&](int m, int c, int sg) { return (s_len[m][c][sg] + kF4PerKB - 1) / kF4PerKB * kF4PerKB; };
    auto blocks = [&](int m, int c) { return (padded(m, c, 0) + padded(m, c, 1)) / kRgThreads; };
    if (t == 0) {
        int n = 0;
        for (int m = 0; m < nmem; ++m) {
            s_first[m] = n;
            n += (blocks(m, 0) + blocks(m, 1)) * (RT - co.row0[m] / kRgRows);
        }
        s_first[nmem] = n;
    }
    __syncthreads();
    // This lane's block: row word q (rows 32 q .. 32 q + 31 of the tile) and
    // positions 32 j .. 32 j + 31.
    const int q = 4 * w + (lane >> 3), j = lane & 7;
    int m = 0;
    for (int i = blockIdx.x; i < s_first[nmem]; i += gridDim.x) {
        while (i >= s_first[m + 1]) ++m;
        const int row0 = co.row0[m], rt0 = row0 / kRgRows, nrt = RT - rt0;
        const int rt = rt0 + (i - s_first[m]) % nrt, kt = (i - s_first[m]) / nrt;
        const int b0 = blocks(m, 0), c = kt < b0 ? 0 : 1;
        const int k0 = (kt - (c ? b0 : 0)) * kRgThreads;
        {
            const int la = s_len[m][c][0], pa = padded(m, c, 0), lb = s_len[m][c][1], k = k0 + t;
            const int* __restrict__ idx = xw.idx(m) + (size_t)c * 2 * xw.max_n;
            int src = -1;
            if (k < pa) {
                if (k < la) src = __ldg(idx + k);
            } else if (k - pa < lb) {
                src = __ldg(idx + xw.max_n + (k - pa));
            }
            // Row words past the padded row count (the last tile) are zero, as
            // are positions without a sample.
            const int nw = src >= 0 ? min(kRgWords, rwp - rt * kRgWords) : 0;
            const uint32_t* p = (c ? tt1 : tt0) + (size_t)max(src, 0) * rwp + rt * kRgWords;
            const uint32_t d = ptx::smem_u32(s_t + rg_slot(t, 0));
#pragma unroll
            for (int e = 0; e < kRgWords / 4; ++e) ptx::cp_async16(d + 16 * e, 4 * e < nw ? p + 4 * e : p, 4 * e < nw);
            ptx::cp_async_wait_all();
        }
        __syncthreads();
        uint32_t a[32];
        // a[p]: bit 31 - r is row 32 q + r at position 32 j + p.
#pragma unroll
        for (int p = 0; p < 32; ++p) a[p] = s_t[rg_slot(32 * j + p, q)];
        __syncthreads();  // s_t may be refilled
        transpose32(a);   // a[r]: bit 31 - p is row 32 q + r at position 32 j + p
        uint8_t* __restrict__ out = co.out + (size_t)m * co.stride +
                                    ((c ? D.W[0] * 32 + kClassPad : 0) + k0) / 2 + 16 * j;
        const int rbase = rt * kRgRows + 32 * q;
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            const int row = rbase + r;
            if (row >= row0 && row < rows_total) *reinterpret_cast<uint4*>(out + (size_t)row * pitch) = e2m1_word(a[r]);
        }
    }
}

}  // namespace tc

// ------------------------------------------------------------------ host
using namespace tc;

// Coefficients of the score bound (count_kernel.cuh) for `cells` cells:
// `margin` bounds |the value of the bound computed in the kernel - its exact
// value| + |the FP32 score - the exact score|.  u = 2^-24; lg2.approx.ftz is
// within 2^-22 of the logarithm, absolutely in (1/2, 2) and relatively outside
// (PTX ISA).  L: 2 N' logarithm errors weighted by the counts, one subtraction
// and a cell-long chain of multiply-adds per class over partial sums of at
// most 1.1 N' (each cell adds at most T' times a binary entropy).  FP32 K2:
// table entries rounded once; the first addition of a cell at most u times
// the tables, sum of lnG(n_c + 1) <= lnG(n + 1) per class (superadditivity of
// ln n!); cell term |b_c| <= (n_c + m_c) ln 2 + ln(N + 1) + 3 and the running
// sum at most sum of the |b_c|.  FP32 MI: p's two roundings and the table's
// against an entropy of at most lg 54, 81 multiply-adds on partial sums of at
// most that.
static void bound_coefficients(int score, double hy64, int nc, int nn, int cells, CountParams* p) {
    const double u = std::ldexp(1.0, -24), N = (double)nc + nn, Np = N + 1.5 * cells, ln2 = std::log(2.0);
    const double lgN = std::log2(N + 2.0);
    const double dl = std::ldexp(1.0, -22) * std::max(1.0, lgN);
    const double r = (2.0 * dl * Np + u * Np * (1.1 * cells + 4.0) + u * cells * cells * lgN + 0.5 * cells * dl) * 1.05;
    if (score == EPISDET_SCORE_K2) {
        const double lg = std::lgamma(nc + 1.0) + std::lgamma(nn + 1.0);
        const double bt = N * ln2 + cells * (std::log(N + 2.0) + 3.0);
        const double s32 = u * (2.0 * lg + std::lgamma(N + 2.0 * cells + 2.0) + (cells + 1.0) * bt) * 1.05;
        const double margin = ln2 * r + s32 + 1e-4 + 4.0 * u * bt;
        const double c = cells * (0.5 + 0.5 * std::log(2.0 * M_PI));
        p->cut_mul = -1.0 / ln2;
        p->cut_add = -(margin + c) / ln2;
        p->seed_mul = -ln2;
        p->seed_add = (c - margin - 0.1176 * cells) / ln2;
    } else {
        const double s32 = u * (2.0 * (lgN + 1.5) + 2.0 * 12.0 + 3.0 * cells * 6.0 + 16.0);
        const double margin = r / N + s32 + 1e-7;
        p->cut_mul = N;
        p->cut_add = -(margin + hy64) * N;
        p->seed_mul = 1.0 / N;
        p->seed_add = (hy64 - margin) * N;
    }
}

static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

static episdet_status get_encoder() {
    if (g_encode) return EPISDET_OK;
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
        return set_error(EPISDET_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    return EPISDET_OK;
}

// rows x pitch bytes, row-major, boxes of box_rows x 128 bytes, 128-byte swizzle.
static episdet_status make_tmap(CUtensorMap* m, void* base, uint64_t rows, uint64_t pitch, uint32_t box_rows) {
    cuuint64_t dims[2] = {pitch, rows};
    cuuint64_t strides[1] = {pitch};
    cuuint32_t box[2] = {kKB, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, base, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(EPISDET_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return EPISDET_OK;
}

static int grid_for(long work, int threads) {
    long b = (work + threads - 1) / threads;
    return (int)std::min<long>(std::max<long>(b, 1), 148L * 64);
}

// One instance of the counting kernel.
struct Instance {
    void (*kern)(const CUtensorMap, const CUtensorMap, const CountParams);
    int mode, nz;
    size_t smem;
};

enum { kIStore = 0, kIPairs = 1, kITriplets = 5, kInstances = 9 };  // kIPairs + 2 * score + (narrow), same for triplets

template <int MODE, int SC, int NZ>
static constexpr Instance instance() {
    return Instance{count_kernel<MODE, SC, NZ>, MODE, NZ, Cfg<NZ>::kSmemTotal};
}

static const Instance& instance_at(int i) {
    static const Instance all[kInstances] = {
        instance<kStore, 0, kWideZ>(),
        instance<kPairs, 0, kWideZ>(),    instance<kPairs, 0, kNarrowZ>(),
        instance<kPairs, 1, kWideZ>(),    instance<kPairs, 1, kNarrowZ>(),
        instance<kTriplets, 0, kWideZ>(), instance<kTriplets, 0, kNarrowZ>(),
        instance<kTriplets, 1, kWideZ>(), instance<kTriplets, 1, kNarrowZ>(),
    };
    return all[i];
}

static cudaLaunchConfig_t cluster_config(const Instance& k, int ctas, cudaStream_t st, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = 2;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = k.smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// CTA pairs of an instance that can be resident at once (asked for once).
static episdet_status resident_pairs(Workspace* w, int inst, int* pairs) {
    static_assert(kInstances <= sizeof(w->pairs) / sizeof(w->pairs[0]), "instances");
    if (w->pairs[inst] == 0) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = cluster_config(instance_at(inst), 2 * (w->sms / 2), w->st, &attr);
        int n = 0;
        CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, instance_at(inst).kern, &cfg));
        w->pairs[inst] = std::min(n, w->sms / 2);
    }
    if (w->pairs[inst] < 1)
        return set_error(EPISDET_ERR_UNSUPPORTED, "no CTA pair of the counting kernel fits on the device");
    *pairs = w->pairs[inst];
    return EPISDET_OK;
}

// Launches an instance over p.ntiles tiles (no more CTA pairs than tiles: SMs
// left idle stay free for concurrent work).
static episdet_status launch_count(Workspace* w, int inst, const CUtensorMap& ta, const CUtensorMap& tb,
                                   const CountParams& p) {
    int pairs = 0;
    episdet_status st = resident_pairs(w, inst, &pairs);
    if (st != EPISDET_OK) return st;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg =
        cluster_config(instance_at(inst), 2 * std::max(1, std::min(pairs, p.ntiles)), w->st, &attr);
    CUDA_TRY(cudaLaunchKernelEx(&cfg, instance_at(inst).kern, ta, tb, p));
    CHECK_LAUNCH();
    return EPISDET_OK;
}

// 16-byte words of one tile's drained segments.
static size_t stash_slot(int nz, int nseg, bool wide) {
    return (size_t)nseg * nz * (kTileA / 2) / 2 * (wide ? 2 : 1);
}

// Room for two tiles of drained segments per CTA.
static episdet_status prepare_stash(Workspace* w, int nz, int nseg, bool wide, CountParams* p) {
    p->stash_slot = stash_slot(nz, nseg, wide);
    p->stash_cta = 2 * p->stash_slot;
    CUDA_TRY(w->stash.ensure(sizeof(uint4) * p->stash_cta * w->sms));
    p->stash = (uint4*)w->stash.p;
    return EPISDET_OK;
}

// Seed pass: bounds on one set per scoring thread over one tile per CTA pair
// give a first search-wide threshold (the k-th best of some 38,000 sets that
// are each the best of 28), so that from the first tile on at most about one
// set in a thousand is scored exactly and offered; the better seeds are levels
// that the counting kernel tightens the threshold to as sets reach them.
static episdet_status seed_threshold(Workspace* w, int inst, const CUtensorMap& ta, const CUtensorMap& tb,
                                     CountParams p, uint64_t* launches) {
    int pairs = 0;
    episdet_status st = resident_pairs(w, inst, &pairs);
    if (st != EPISDET_OK) return st;
    const int n = 2 * std::max(1, std::min(pairs, p.ntiles)) * kScoreThreads;
    CUDA_TRY(w->seeds.ensure(sizeof(uint32_t) * (size_t)n));
    p.seeds = (uint32_t*)w->seeds.p;
    st = launch_count(w, inst, ta, tb, p);
    if (st != EPISDET_OK) return st;
    seed_levels_kernel<<<1, kMergeBlockThreads, 0, w->st>>>(p.S, p.seeds, n);
    CHECK_LAUNCH();
    *launches += 2;
    return EPISDET_OK;
}

// A tile's counts fit 16 bits in the stash.
static bool counts_wide(int nc, int nn) { return std::max(nc, nn) > 65535; }

// First B tile of nz SNPs that reaches past the first SNP of A tile a.
static int first_b(int a, int nz) { return (kTileA * a) / nz; }

// Tiles of the pairs (r, col > r) with r in A tiles [a0, a1), every B tile that
// reaches past the A tile's first SNP, in bands of about 1024 x 1008 SNPs: the 74
// tiles that run at once then read 8 + 9 row panels instead of 1 + 74 (all pairs
// of 16384 SNPs x 32768 samples, whose rows are 537 MB: row by row 5.98 ms,
// in bands 4.89).
static void pair_tiles(int M, int a0, int a1, int nz, std::vector<int2>& out) {
    constexpr int kBandA = 8;
    const int band_b = 9 * kWideZ / nz, ntb = (M + nz - 1) / nz;
    for (int ba = a0; ba < a1; ba += kBandA)
        for (int bb = first_b(ba, nz); bb < ntb; bb += band_b)
            for (int a = ba; a < std::min(a1, ba + kBandA); ++a)
                for (int b = std::max(first_b(a, nz), bb); b < std::min(ntb, bb + band_b); ++b)
                    out.push_back(make_int2(a, b));
}

static int a_tiles(int M) { return (M + kTileA - 1) / kTileA; }

// Packed e2m1 rows of the planes in D, and their tensor maps.
static episdet_status pack_rows(Workspace* w, DevBuf* buf, const DevData& D, int pitch, int nz, CUtensorMap* ta,
                                CUtensorMap* tb) {
    const int rows = 2 * D.M;
    CUDA_TRY(buf->ensure((size_t)rows * pitch));
    pack_f4_kernel<<<grid_for((long)rows * (D.W[0] + D.W[1]), 256), 256, 0, w->st>>>(D, (uint8_t*)buf->p, rows, pitch);
    CHECK_LAUNCH();
    episdet_status st = make_tmap(ta, buf->p, (uint64_t)rows, (uint64_t)pitch, kCtaRows);
    if (st == EPISDET_OK) st = make_tmap(tb, buf->p, (uint64_t)rows, (uint64_t)pitch, nz);
    return st;
}

// Label-free AND cells of every SNP pair over the n samples of one plane set
// ([M][2][W] words, on the device) into out ([M][M] float4, pairs a < b).
episdet_status tensor_pair_totals(Workspace* w, const uint32_t* d_planes, int M, int n, float4* out) {
    episdet_status st = get_encoder();
    if (st != EPISDET_OK) return st;
    CUDA_TRY(w->tensor_flag.ensure(sizeof(int) * 4));
    CUDA_TRY(cudaMemsetAsync(w->tensor_flag.p, 0, sizeof(int) * 4, w->st));
    DevData D;
    memset(&D, 0, sizeof(D));
    D.M = M;
    D.bits[0] = D.bits[1] = d_planes;  // no second class: W[1] = 0
    D.n[0] = n;
    D.W[0] = episdet_class_words(n);
    const int pitch = (D.W[0] * 32 + kClassPad) / 2;
    CUtensorMap ta, tb;
    st = pack_rows(w, &w->frows, D, pitch, kWideZ, &ta, &tb);
    if (st != EPISDET_OK) return st;
    std::vector<int2> tiles;
    pair_tiles(M, 0, a_tiles(M), kWideZ, tiles);
    CUDA_TRY(w->tiles.ensure(sizeof(int2) * tiles.size()));
    CUDA_TRY(cudaMemcpyAsync(w->tiles.p, tiles.data(), sizeof(int2) * tiles.size(), cudaMemcpyHostToDevice, w->st));
    CountParams p;
    memset(&p, 0, sizeof(p));
    p.M = M;
    p.err = (int*)w->tensor_flag.p;
    p.wait_ns = 4000ull * 1000000ull;
    p.ngroup = 1;
    p.tiles = (const int2*)w->tiles.p;
    p.ntiles = (int)tiles.size();
    p.seg2[0] = Seg{0, (n + kF4PerKB - 1) / kF4PerKB};
    p.wide = counts_wide(n, 0);
    p.one_class = 1;
    p.out = (float*)out;
    p.out_n = 4;
    p.out_ld = M;
    st = prepare_stash(w, kWideZ, 2, p.wide != 0, &p);
    if (st == EPISDET_OK) st = launch_count(w, kIStore, ta, tb, p);
    if (st != EPISDET_OK) return st;
    int err = 0;
    CUDA_TRY(cudaMemcpyAsync(&err, w->tensor_flag.p, sizeof(int), cudaMemcpyDeviceToHost, w->st));
    CUDA_TRY(cudaStreamSynchronize(w->st));  // the tile list is reused by the next search
    if (err) return set_error(EPISDET_ERR_TIMEOUT, "a bounded device wait gave up (code %d)", err);
    return EPISDET_OK;
}

static episdet_status transpose_planes(Workspace* w, const DevData& D, int c, DevBuf* buf) {
    const int rows = 2 * D.M, rwp = tt_row_words(rows);
    CUDA_TRY(buf->ensure(sizeof(uint32_t) * (size_t)D.W[c] * 32 * rwp));
    const int warps = (rwp / 8) * (D.W[c] / 8);
    transpose_planes_kernel<<<(warps + kTtThreads / 32 - 1) / (kTtThreads / 32), kTtThreads, 0, w->st>>>(
        D, c, (uint32_t*)buf->p, rows, rwp);
    CHECK_LAUNCH();
    return EPISDET_OK;
}

episdet_status tensor_label_cohort(Workspace* w, LabelCohort* c, bool validate) {
    DevData D;
    memset(&D, 0, sizeof(D));
    D.M = c->M;
    D.bits[0] = c->planes;
    D.W[0] = c->W;
    D.n[0] = c->n;
    CUDA_TRY(w->perm_marg.ensure(sizeof(int) * 3 * (size_t)c->M));
    CUDA_TRY(w->flag.ensure(sizeof(int) * 4));
    CUDA_TRY(cudaMemsetAsync(w->flag.p, 0, sizeof(int) * 4, w->st));
    cohort_marginals_kernel<<<(c->M + 7) / 8, 256, 0, w->st>>>(c->planes, c->M, c->n, c->W, (int*)w->perm_marg.p,
                                                               (int*)w->flag.p);
    CHECK_LAUNCH();
    int bad = 0;
    CUDA_TRY(cudaMemcpyAsync(&bad, w->flag.p, sizeof(int), cudaMemcpyDeviceToHost, w->st));
    CUDA_TRY(cudaStreamSynchronize(w->st));
    if (bad && validate)
        return set_error(EPISDET_ERR_INVALID_INPUT, "input planes have overlapping genotype-0/1 planes");
    episdet_status st = transpose_planes(w, D, 0, &w->perm_tt);
    if (st != EPISDET_OK) return st;
    CUDA_TRY(w->perm_tot.ensure(sizeof(float4) * (size_t)c->M * c->M));
    st = tensor_pair_totals(w, c->planes, c->M, c->n, (float4*)w->perm_tot.p);  // ends with a synchronise
    c->tt = (const uint32_t*)w->perm_tt.p;
    c->marg = (const int*)w->perm_marg.p;
    c->tot = (const float4*)w->perm_tot.p;
    return st;
}

episdet_status tensor_label_rows(Workspace* w, const LabelCohort& c, const uint32_t* d_label, int nc, DevData* D,
                                 uint64_t* launches) {
    memset(D, 0, sizeof(*D));
    D->M = c.M;
    D->n[0] = nc;
    D->n[1] = c.n - nc;
    CUDA_TRY(w->perm_mask.ensure(sizeof(uint32_t) * 2 * (size_t)c.W));
    uint32_t* mask = (uint32_t*)w->perm_mask.p;
    for (int k = 0; k < 2; ++k) {
        D->bits[k] = c.planes;
        D->W[k] = c.W;
        D->mask[k] = mask + (size_t)k * c.W;
        CUDA_TRY(w->marg[k].ensure(sizeof(int) * 3 * (size_t)c.M));
        D->marg[k] = (const int*)w->marg[k].p;
    }
    CUDA_TRY(w->tensor_flag.ensure(sizeof(int) * 4));
    CUDA_TRY(cudaMemsetAsync(w->tensor_flag.p, 0, sizeof(int) * 4, w->st));
    XWork xw;
    xw.info_bytes = 256;
    xw.stride = (xw.info_bytes + sizeof(int) * 4 * (size_t)c.n + 255) & ~size_t(255);
    xw.max_n = c.n;
    xw.x0 = 0;
    xw.err = (int*)w->tensor_flag.p;
    CUDA_TRY(w->xinfo.ensure(xw.stride));
    xw.base = (uint8_t*)w->xinfo.p;
    label_lists_kernel<<<1, kXinfoThreads, 0, w->st>>>(d_label, c.n, c.W, nc, xw, mask);
    CHECK_LAUNCH();
    label_marginals_kernel<<<(c.M + 7) / 8, 256, 0, w->st>>>(c.planes, c.M, c.W, mask, nc, c.marg, (int*)w->marg[0].p,
                                                             (int*)w->marg[1].p);
    CHECK_LAUNCH();
    // Case operand rows: one member whose only segment is the cases.
    const int rows = 2 * c.M, pitch = (episdet_class_words(nc) * 32 + kClassPad) / 2;
    CUDA_TRY(w->frows.ensure((size_t)rows * pitch));
    CmpOut co;
    memset(&co, 0, sizeof(co));
    co.out = (uint8_t*)w->frows.p;
    regroup_kernel<<<kRgCtas * w->sms, kRgThreads, 0, w->st>>>(*D, xw, co, c.tt, c.tt, tt_row_words(rows), rows, pitch, 1);
    CHECK_LAUNCH();
    *launches += 3;
    return EPISDET_OK;
}

episdet_status tensor_init_attributes() {
    for (int i = 0; i < kInstances; ++i)
        CUDA_TRY(cudaFuncSetAttribute(instance_at(i).kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)instance_at(i).smem));
    return get_encoder();
}

// 2-way search: packed e2m1 rows of every SNP plane, one launch over the tiles
// of the slab.  Label mode (w->label_tot): operand rows of the cases only,
// already in w->frows (tensor_label_rows); the controls' cells come from the
// label-free pair totals.
static episdet_status run_pairs(Workspace* w, const DevData& D, const episdet_options& o, int fb, int fe,
                                CountParams& p, uint64_t* launches, bool progress) {
    const int M = D.M, Kc = D.W[0] * 32, Kn = D.W[1] * 32;
    const bool label = w->label_tot != nullptr;
    const int a0 = fb / kTileA, a1 = (fe - 1) / kTileA + 1;
    // Narrow tiles when wide ones would leave CTA pairs without work (512 SNPs:
    // counting launch 33 us narrow, 48 us wide; 1000 SNPs 33 and 37).
    std::vector<int2> tiles;
    pair_tiles(M, a0, a1, kWideZ, tiles);
    const bool narrow = (int)tiles.size() < w->sms / 2;
    const int nz = narrow ? kNarrowZ : kWideZ;
    if (narrow) {
        tiles.clear();
        pair_tiles(M, a0, a1, nz, tiles);
    }
    const int inst = kIPairs + 2 * p.T.score + (narrow ? 1 : 0);
    CUtensorMap ta, tb;
    episdet_status st;
    if (label) {
        const int pitch = (episdet_class_words(D.n[0]) * 32 + kClassPad) / 2;
        st = make_tmap(&ta, w->frows.p, (uint64_t)2 * M, (uint64_t)pitch, kCtaRows);
        if (st == EPISDET_OK) st = make_tmap(&tb, w->frows.p, (uint64_t)2 * M, (uint64_t)pitch, nz);
    } else {
        st = pack_rows(w, &w->frows, D, (Kc + kClassPad) / 2 + (Kn + kClassPad) / 2, nz, &ta, &tb);
        ++*launches;
    }
    if (st != EPISDET_OK) return st;
    p.rt_ld = (M + 3) & ~3;
    CUDA_TRY(w->rtab.ensure(sizeof(float2) * 9 * (size_t)p.rt_ld));
    p.rt = (const float2*)w->rtab.p;
    marginal_rows_kernel<<<(M + 255) / 256, 256, 0, w->st>>>(D, (float2*)w->rtab.p, p.rt_ld, p.tab_off);
    CHECK_LAUNCH();
    ++*launches;
    CUDA_TRY(w->tiles.ensure(sizeof(int2) * tiles.size()));
    CUDA_TRY(cudaMemcpyAsync(w->tiles.p, tiles.data(), sizeof(int2) * tiles.size(), cudaMemcpyHostToDevice, w->st));
    w->h2d += (int64_t)(sizeof(int2) * tiles.size());
    if (progress)
        for (int i = 0; i < (M + 255) / 256; ++i) printf("Outer loop iteration %d out of %d\n", i, (M + 255) / 256);
    const int kb1 = (Kc + kClassPad) / kF4PerKB;
    p.seg2[0] = Seg{0, (D.n[0] + kF4PerKB - 1) / kF4PerKB};
    p.seg2[1] = label ? Seg{kb1, kb1} : Seg{kb1, kb1 + (D.n[1] + kF4PerKB - 1) / kF4PerKB};
    p.tot = w->label_tot;
    p.one_class = label;
    p.ngroup = 1;
    p.tiles = (const int2*)w->tiles.p;
    p.ntiles = (int)tiles.size();
    p.wide = counts_wide(D.n[0], label ? 0 : D.n[1]);
    st = prepare_stash(w, nz, 2, p.wide != 0, &p);
    if (st != EPISDET_OK) return st;
    if (p.filter) {
        st = seed_threshold(w, inst, ta, tb, p, launches);
        if (st != EPISDET_OK) return st;
    }
    CUDA_TRY(timer_begin(w));
    st = launch_count(w, inst, ta, tb, p);
    if (st != EPISDET_OK) return st;
    CUDA_TRY(timer_end(w));
    ++*launches;
    if (w->timing)
        w->executed_macs = (double)tiles.size() * 4.0 * kTileA * nz *
                           (double)(p.seg2[0].kb1 - p.seg2[0].kb0 + p.seg2[1].kb1 - p.seg2[1].kb0) * kF4PerKB;
    return EPISDET_OK;
}

episdet_status run_tensor(Workspace* w, DevData& D, const ScoreTables& T, const episdet_options& o, int fb, int fe,
                          Slots* S, uint64_t* launches, bool progress) {
    episdet_status st = get_encoder();
    if (st != EPISDET_OK) return st;
    const int M = D.M;
    const int grid = w->sms;
    CUDA_TRY(w->cbuf.ensure(sizeof(Cand) * (size_t)kCapG * grid));
    st = prepare_slots(w, grid, o.top_k, S);
    if (st != EPISDET_OK) return st;
    S->lists = (Cand*)w->cbuf.p;
    S->ld = kCapG;
    CUDA_TRY(w->tensor_flag.ensure(sizeof(int) * 4));
    int* d_err = (int*)w->tensor_flag.p;

    CountParams p;
    memset(&p, 0, sizeof(p));
    p.M = M;
    p.T = T;
    p.S = *S;
    p.first_begin = fb;
    p.first_end = fe;
    p.err = d_err;
    p.wait_ns = (uint64_t)(o.wait_limit_ms > 0 ? o.wait_limit_ms : 4000) * 1000000ull;
    p.hold = (o.flags & EPISDET_FLAG_INJECT_STALL) ? d_err + 3 : nullptr;
    // The bound adds 1/2 and 3/2 to counts in FP32, exact up to 2^22; classes
    // past that are scored exactly throughout.
    p.filter = (o.flags & EPISDET_FLAG_FILTER_OFF) == 0 && std::max(D.n[0], D.n[1]) <= (1 << 22);
    p.tab_off = p.filter && T.score == EPISDET_SCORE_K2 ? 3.0f * kCellOff<0> : 0.0f;
    bound_coefficients(T.score, T.hy64, D.n[0], D.n[1], o.order == 2 ? 9 : 27, &p);

    if (o.order == 2) return run_pairs(w, D, o, fb, fe, p, launches, progress);

    const int Kc = D.W[0] * 32, Kn = D.W[1] * 32;
    const int rows = 2 * M;
    const int bs_lines = (M + 255) / 256;
    // Triplet tiles: narrow for panels of few B tiles and few samples
    // (w->stage_override: the autotuner's choice).
    const bool narrow = w->stage_override >= 0
                            ? w->stage_override == 0
                            : M <= kNarrowTileSnps && D.n[0] + D.n[1] <= kNarrowTileSamples;
    const int nz = narrow ? kNarrowZ : kWideZ;
    const int inst = kITriplets + 2 * T.score + (narrow ? 1 : 0);

    // 3-way pair table.  Whole: every pair whose first SNP lies in a tile >=
    // fb's, an [M][M] window, filled once.  Y-blocked (when the whole table
    // does not fit beside the other buffers, or as o.pair_block_snps asks): the
    // rows of one block of second SNPs Y at a time ([BY][M - y0] from column
    // y0), plus the rows of the current first SNPs X ([128][M - xt0]); the first
    // SNPs are then swept once per Y block, each pass counting only the
    // triplets whose Y lies in the block (the reference keeps
    // [9][BLOCK_SIZE][M] pair counts per Y block, src/search-triplets.cu:173-176).
    const int nt2 = a_tiles(M);
    const int ntb = (M + nz - 1) / nz;
    const int a_first = (fb + 1) / kTileA;
    const int xend = std::min(fe, M - 2);
    // Rows of both classes' packed e2m1 regions, 2 samples per byte.
    const int pitch = (Kc + kClassPad) / 2 + (Kn + kClassPad) / 2;
    const int max_n = std::max(D.n[0], D.n[1]);
    const size_t info_bytes = 256;
    const size_t xstride = (info_bytes + sizeof(int) * 4 * (size_t)max_n + 255) & ~size_t(255);
    // First SNPs of a launch: as many as give every CTA pair kGroupTiles tiles,
    // at least kXGroup, with at most kGroupBytes of regrouped rows (or kXGroup's),
    // and no more than the device has room for beside the pair table.
    const size_t member_bytes = (size_t)rows * pitch;
    int gmax = (int)std::min<size_t>(kMaxGroup, std::max<size_t>(kXGroup, kGroupBytes / member_bytes));
    const int all_tiles = nt2 - a_first;
    int blk_tiles = all_tiles;  // A pair tiles (128 Y SNPs) per Y block
    if (o.pair_block_snps > 0) blk_tiles = std::min(blk_tiles, (o.pair_block_snps + kTileA - 1) / kTileA);
    p.rt_ld = (M + 3) & ~3;
    {
        const size_t row_bytes = 8 * sizeof(float) * (size_t)M;  // one table row, both classes
        const size_t xrows_bytes = row_bytes * kTileA;
        const bool wide = counts_wide(D.n[0], D.n[1]);
        // The buffers of the search but for the pair table.
        struct Need {
            DevBuf* buf;
            size_t bytes;
        };
        auto needs = [&](int g) {
            std::vector<Need> v = {{&w->frows, (size_t)rows * pitch},
                                   {&w->xinfo, (size_t)kXSets * g * xstride},
                                   {&w->rtab, sizeof(float2) * 9 * (size_t)p.rt_ld * g},
                                   {&w->stash, sizeof(uint4) * 2 * stash_slot(nz, 4, wide) * w->sms}};
            for (DevBuf& d : w->xsub) v.push_back({&d, member_bytes * g});
            for (int c = 0; c < 2; ++c)
                v.push_back({&w->planes_t[c], sizeof(uint32_t) * (size_t)D.W[c] * 32 * tt_row_words(rows)});
            return v;
        };
        // Device memory they still take (a buffer is replaced when it grows).
        auto growth = [&](int g) {
            size_t more = 0;
            for (const Need& d : needs(g)) more += d.bytes > d.buf->cap ? d.bytes - d.buf->cap : 0;
            return more;
        };
        auto table_bytes = [&] { return row_bytes * (blk_tiles < all_tiles ? (size_t)blk_tiles * kTileA : (size_t)M); };
        auto keep_limit = [&](int top) {
            w->limit_bytes = member_bytes;
            w->limit = gmax;
            w->limit_uses = gmax < top ? 64 : 0;
        };
        // Chooses gmax and, unless asked for, the pair table's blocks.  (Free
        // memory is asked for only when something has to grow: on some hosts the
        // driver takes 9 ms to answer, more than a small search.)
        auto plan = [&]() -> episdet_status {
            const int top = gmax;
            const bool asked = blk_tiles < all_tiles;
            const bool held_all = w->ptab.cap >= table_bytes() && (!asked || w->ptabx.cap >= xrows_bytes);
            if (held_all && growth(gmax) == 0) return EPISDET_OK;
            // A launch size that memory limited lately is kept for searches with the same rows.
            if (held_all && w->limit_bytes == member_bytes && w->limit_uses > 0 && growth(std::min(gmax, w->limit)) == 0) {
                --w->limit_uses;
                gmax = std::min(gmax, w->limit);
                return EPISDET_OK;
            }
            size_t fr = 0, tot = 0;
            CUDA_TRY(cudaMemGetInfo(&fr, &tot));
            // Left for the tile lists, slots, merge buffers and the driver.
            const size_t reserve = std::max<size_t>(tot / 32, (size_t)1 << 30);
            const size_t table = held_all ? 0 : table_bytes() + (asked ? xrows_bytes : 0);
            // The pair-table buffers are replaced when they grow, so their memory counts as free.
            size_t held = held_all ? 0 : w->ptab.cap + w->ptabx.cap;
            const size_t least = reserve + table + growth(kXGroup);
            if (fr + held >= least) {
                // Larger launches hold a small part of what is left beside the smallest,
                // so that they narrow nothing for the other lanes of a batch or other
                // processes; what they hold already is part of what is left.
                size_t spare = fr + held - least;
                for (const Need& d : needs(kXGroup)) spare += d.buf->cap > d.bytes ? d.buf->cap - d.bytes : 0;
                auto total = [&](int g) {
                    size_t b = 0;
                    for (const Need& d : needs(g)) b += d.bytes;
                    return b;
                };
                while (gmax > kXGroup && growth(gmax) > 0 && total(gmax) > total(kXGroup) + spare / 16)
                    gmax = std::max(kXGroup, gmax * 3 / 4);
                keep_limit(top);
                return EPISDET_OK;
            }
            // Little memory left: the smallest launches, and what earlier searches'
            // larger ones hold goes back.
            gmax = kXGroup;
            keep_limit(top);
            for (const Need& d : needs(gmax))
                if (d.buf->cap > d.bytes) d.buf->release();
            if (asked || held_all) return EPISDET_OK;
            CUDA_TRY(cudaMemGetInfo(&fr, &tot));
            const size_t taken = reserve + growth(gmax);
            const size_t avail = fr + held > taken ? fr + held - taken : 0;
            if (row_bytes * (size_t)M > avail) {
                const size_t left = avail > xrows_bytes ? avail - xrows_bytes : 0;
                blk_tiles = (int)std::min<size_t>((size_t)blk_tiles, left / (row_bytes * kTileA));
                if (blk_tiles < 1)
                    return set_error(EPISDET_ERR_OUT_OF_MEMORY,
                                     "3-way search of %d SNPs: no 128-row block of the pair table fits in the %.1f GB "
                                     "left beside the operand buffers",
                                     M, (double)avail / 1e9);
            }
            return EPISDET_OK;
        };
        auto allocate = [&]() -> cudaError_t {
            for (const Need& d : needs(gmax)) {
                const cudaError_t e = d.buf->ensure(d.bytes);
                if (e != cudaSuccess) return e;
            }
            // (A table that grows takes the memory of the buffer it no longer needs.)
            const bool blocked = blk_tiles < all_tiles;
            if (!blocked && w->ptab.cap < table_bytes()) w->ptabx.release();
            if (blocked && w->ptabx.cap < xrows_bytes && w->ptab.cap > table_bytes()) w->ptab.release();
            cudaError_t e = w->ptab.ensure(table_bytes());
            if (e == cudaSuccess && blocked) e = w->ptabx.ensure(xrows_bytes);
            return e;
        };
        for (;;) {
            st = plan();
            if (st != EPISDET_OK) return st;
            const cudaError_t e = allocate();
            if (e == cudaSuccess) break;
            if (e != cudaErrorMemoryAllocation || gmax == kXGroup) return cuda_fail(e, "3-way search buffers");
            // Less memory than it seemed (another lane or process): once more with
            // the smallest launches.
            gmax = kXGroup;
            for (const Need& d : needs(gmax))
                if (d.buf->cap > d.bytes) d.buf->release();
        }
        st = prepare_stash(w, nz, 4, wide, &p);
        if (st != EPISDET_OK) return st;
    }
    const bool blocked = blk_tiles < nt2 - a_first;
    const int nblk = (nt2 - a_first + blk_tiles - 1) / blk_tiles;
    p.rt = (const float2*)w->rtab.p;

    // Operand rows of the pair table, and its tiles: one list per Y block (all
    // rows from the slab's first on when whole) and, Y-blocked, one per A tile
    // that holds first SNPs.
    CUtensorMap fa, fbm;
    st = pack_rows(w, &w->frows, D, pitch, kWideZ, &fa, &fbm);
    if (st != EPISDET_OK) return st;
    ++*launches;
    std::vector<int2> lists;
    std::vector<size_t> blk_off((size_t)nblk + 1, 0), row_off((size_t)nt2 + 1, 0);
    for (int blk = 0; blk < nblk; ++blk) {
        const int ya0 = blocked ? a_first + blk * blk_tiles : fb / kTileA;
        pair_tiles(M, ya0, blocked ? std::min(nt2, ya0 + blk_tiles) : nt2, kWideZ, lists);
        blk_off[blk + 1] = lists.size();
    }
    for (int a = 0; a < nt2; ++a) {
        row_off[a] = lists.size();
        if (blocked && a >= fb / kTileA && a <= (xend - 1) / kTileA) pair_tiles(M, a, a + 1, kWideZ, lists);
    }
    row_off[nt2] = lists.size();
    // Triplet tile lists, one per (Y block, first A tile a0 = (X+1)/128): every
    // (A tile a, B tile b) with max(a0, first tile of the block) <= a < end of
    // the block, whose Z range reaches past the tile's first Y, ordered in
    // bands of about 768 x 784 SNPs so that a wave of concurrent tiles shares
    // few A and B row panels in L2.  First SNPs below the block share one
    // list; lists are built only for the first SNPs of this call's slab.
    const int band_a = 6, band_b = 14 * kNarrowZ / nz;
    const int a_last = std::min(nt2 - 1, xend / kTileA);  // a0 of the slab's last first SNP
    std::vector<size_t> list_off((size_t)nblk * (nt2 + 1), 0);
    std::vector<int> list_len((size_t)nblk * (nt2 + 1), 0);
    for (int blk = 0; blk < nblk; ++blk) {
        const int ya0 = a_first + blk * blk_tiles, ya1 = std::min(nt2, ya0 + blk_tiles);
        for (int a0 = a_first; a0 < std::min(ya1, a_last + 1); ++a0) {
            const size_t li = (size_t)blk * (nt2 + 1) + a0;
            if (a0 < ya0 && a0 > a_first) {  // same list as the block's first a0
                list_off[li] = list_off[li - 1];
                list_len[li] = list_len[li - 1];
                continue;
            }
            list_off[li] = lists.size();
            for (int ba = std::max(a0, ya0); ba < ya1; ba += band_a)
                for (int bb = first_b(ba, nz); bb < ntb; bb += band_b)
                    for (int a = ba; a < std::min(ya1, ba + band_a); ++a)
                        for (int b = std::max(first_b(a, nz), bb); b < std::min(ntb, bb + band_b); ++b)
                            lists.push_back(make_int2(a, b));
            list_len[li] = (int)(lists.size() - list_off[li]);
        }
    }
    if (lists.size() > (size_t)INT32_MAX) return set_error(EPISDET_ERR_UNSUPPORTED, "too many tiles");
    CUDA_TRY(w->tiles.ensure(sizeof(int2) * lists.size()));
    CUDA_TRY(cudaMemcpyAsync(w->tiles.p, lists.data(), sizeof(int2) * lists.size(), cudaMemcpyHostToDevice, w->st));
    w->h2d += (int64_t)(sizeof(int2) * lists.size());
    p.tiles = (const int2*)w->tiles.p;

    // Counts of the pairs of SNP rows from r0 on (128-aligned) with every later
    // SNP, by the tiles [t0, t1) of the lists, stored at pair (row - r0) *
    // (M - r0) + (col - r0) of out (or at row * M + col when whole).
    CountParams ps = p;
    ps.seg2[0] = Seg{0, (D.n[0] + kF4PerKB - 1) / kF4PerKB};
    const int kbn = (Kc + kClassPad) / kF4PerKB;
    ps.seg2[1] = Seg{kbn, kbn + (D.n[1] + kF4PerKB - 1) / kF4PerKB};
    ps.wide = counts_wide(D.n[0], D.n[1]);
    ps.ngroup = 1;
    ps.out_n = 8;
    ps.hold = nullptr;
    st = prepare_stash(w, kWideZ, 2, ps.wide != 0, &ps);
    if (st != EPISDET_OK) return st;
    p.stash = ps.stash;
    auto store_pairs = [&](float* out, size_t t0, size_t t1, int r0, bool whole) -> episdet_status {
        ps.list_off[0] = (int)t0;
        ps.ntiles = (int)(t1 - t0);
        ps.out = out;
        ps.out_r0 = ps.out_c0 = whole ? 0 : r0;
        ps.out_ld = whole ? M : M - r0;
        ++*launches;
        return launch_count(w, kIStore, fa, fbm, ps);
    };
    PairView xv{};
    if (!blocked) {
        st = store_pairs((float*)w->ptab.p, 0, blk_off[1], 0, true);
        if (st != EPISDET_OK) return st;
        p.yv = xv = PairView{(const float*)w->ptab.p, 0, 0, M};
    }

    // kXSets sets of regrouped operands and segment tables: the regrouping of
    // group g + 1 (on aux_st) is queued while the counting launch of group g
    // (on st) runs.
    CUtensorMap tmx[kXSets][2];
    XWork xw[kXSets];
    CmpOut co[kXSets];
    memset(co, 0, sizeof(co));
    for (int b = 0; b < kXSets; ++b) {
        xw[b].base = (uint8_t*)w->xinfo.p + (size_t)b * gmax * xstride;
        xw[b].stride = xstride;
        xw[b].info_bytes = info_bytes;
        xw[b].max_n = max_n;
        xw[b].err = d_err;
        st = make_tmap(&tmx[b][0], w->xsub[b].p, (uint64_t)rows * gmax, (uint64_t)pitch, kCtaRows);
        if (st == EPISDET_OK) st = make_tmap(&tmx[b][1], w->xsub[b].p, (uint64_t)rows * gmax, (uint64_t)pitch, nz);
        if (st != EPISDET_OK) return st;
        co[b].out = (uint8_t*)w->xsub[b].p;
        co[b].stride = member_bytes;
    }
    p.rows_member = rows;
    p.xstride = xstride;
    int pairs = 0;
    st = resident_pairs(w, inst, &pairs);
    if (st != EPISDET_OK) return st;
    // Sample-major planes for the regrouping.
    const int rwp = tt_row_words(rows);
    for (int c = 0; c < 2; ++c) {
        st = transpose_planes(w, D, c, &w->planes_t[c]);
        if (st != EPISDET_OK) return st;
        ++*launches;
    }
    // The regrouping reads the planes, their transposes and the marginals staged on st.
    CUDA_TRY(cudaEventRecord(w->ev_ready, w->st));
    CUDA_TRY(cudaStreamWaitEvent(w->aux_st, w->ev_ready, 0));
    // Tiles each first SNP was counted against, per launch (for the MAC count).
    struct LaunchTiles {
        int x0, gn;
        int len[kMaxGroup];
    };
    std::vector<LaunchTiles> launch_tiles;
    int gi = 0;
    int xt0 = -1;  // first row held in ptabx (Y-blocked)
    for (int blk = 0; blk < nblk; ++blk) {
        const int ya0 = a_first + blk * blk_tiles, ya1 = std::min(nt2, ya0 + blk_tiles);
        const int y0 = ya0 * kTileA, y1 = std::min(M, ya1 * kTileA);
        if (blocked) {
            // Y-Z rows of this block (the previous block's launches, on the
            // same stream, have read theirs).
            st = store_pairs((float*)w->ptab.p, blk_off[blk], blk_off[blk + 1], y0, false);
            if (st != EPISDET_OK) return st;
            p.yv = PairView{(const float*)w->ptab.p, y0, y0, M - y0};
        }
        const int xe = std::min(xend, y1 - 1);  // X < Y < y1
        int gn = 0;
        for (int x0 = fb; x0 < xe; x0 += gn) {
            const int b = gi % kXSets;
            LaunchTiles lt;
            lt.x0 = x0;
            int cum = 0;
            for (gn = 0; gn < gmax && x0 + gn < xe && (gn < kXGroup || cum < kGroupTiles * pairs); ++gn) {
                const int x = x0 + gn;
                // X rows of a Y-blocked launch are within one 128-row window.
                if (blocked && gn > 0 && x / kTileA != x0 / kTileA) break;
                if (progress && x % 256 == 0 && x + 1 >= y0) printf("Outer loop iteration %d out of %d\n", x / 256, bs_lines);
                const size_t li = (size_t)blk * (nt2 + 1) + (x + 1) / kTileA;
                p.list_off[gn] = (int)list_off[li];
                p.cum[gn] = cum;
                lt.len[gn] = list_len[li];
                cum += list_len[li];
                co[b].row0[gn] = 2 * nz * first_b(std::max((x + 1) / kTileA, ya0), nz);
            }
            lt.gn = gn;
            if (cum == 0) continue;
            if (w->timing) launch_tiles.push_back(lt);
            ++gi;
            if (blocked && xt0 != x0 / kTileA * kTileA) {
                // X-Y and X-Z rows of this group's first SNPs (and the next ones').
                xt0 = x0 / kTileA * kTileA;
                st = store_pairs((float*)w->ptabx.p, row_off[xt0 / kTileA], row_off[xt0 / kTileA + 1], xt0, false);
                if (st != EPISDET_OK) return st;
                xv = PairView{(const float*)w->ptabx.p, xt0, xt0, M - xt0};
            }
            // Index lists and regrouped rows of the gn first SNPs, one launch each,
            // into buffer set b once the counting launch that last read it is done.
            if (gi > kXSets) CUDA_TRY(cudaStreamWaitEvent(w->aux_st, w->ev_tc[b], 0));
            xw[b].x0 = x0;
            xinfo_kernel<<<dim3(2, gn), kXinfoThreads, 0, w->aux_st>>>(D, xw[b]);
            CHECK_LAUNCH();
            regroup_kernel<<<kRgCtas * grid, kRgThreads, 0, w->aux_st>>>(
                D, xw[b], co[b], (const uint32_t*)w->planes_t[0].p, (const uint32_t*)w->planes_t[1].p, rwp, rows,
                pitch, gn);
            CHECK_LAUNCH();
            CUDA_TRY(cudaEventRecord(w->ev_cmp[b], w->aux_st));
            CUDA_TRY(cudaStreamWaitEvent(w->st, w->ev_cmp[b], 0));
            pair_rows_kernel<<<dim3((M + 255) / 256, gn), 256, 0, w->st>>>(D, xv, xw[b].base, xstride, x0,
                                                                          (float2*)w->rtab.p, p.rt_ld, p.tab_off);
            CHECK_LAUNCH();
            *launches += 3;
            p.ngroup = gn;
            p.ntiles = cum;
            p.x0 = x0;
            p.xinfo = xw[b].base;
            if (gi == 1 && p.filter) {
                st = seed_threshold(w, inst, tmx[b][0], tmx[b][1], p, launches);
                if (st != EPISDET_OK) return st;
            }
            CUDA_TRY(timer_begin(w));
            st = launch_count(w, inst, tmx[b][0], tmx[b][1], p);
            if (st != EPISDET_OK) return st;
            CUDA_TRY(timer_end(w));
            CUDA_TRY(cudaEventRecord(w->ev_tc[b], w->st));
            *launches += 1;
        }
    }
    if (w->timing) {
        // Tensor MACs issued: per X, tiles x 256 x 2 nz x the regrouped K extent,
        // which follows from X's genotype counts exactly as xinfo_kernel derives it.
        std::vector<int> mg[2];
        for (int c = 0; c < 2; ++c) {
            mg[c].resize((size_t)3 * M);
            CUDA_TRY(cudaMemcpyAsync(mg[c].data(), D.marg[c], sizeof(int) * 3 * M, cudaMemcpyDeviceToHost, w->st));
        }
        CUDA_TRY(cudaStreamSynchronize(w->st));
        w->d2h += (int64_t)(2 * sizeof(int) * 3 * M);
        auto kext_of = [&](int x) {
            int tot[3];
            for (int g = 0; g < 3; ++g) tot[g] = mg[0][(size_t)g * M + x] + mg[1][(size_t)g * M + x];
            int gd = 0;
            if (tot[1] > tot[gd]) gd = 1;
            if (tot[2] > tot[gd]) gd = 2;
            long kext = 0;
            for (int c = 0; c < 2; ++c)
                for (int g = 0; g < 3; ++g)
                    if (g != gd) kext += ((mg[c][(size_t)g * M + x] + kF4PerKB - 1) / kF4PerKB) * (long)kF4PerKB;
            return kext;
        };
        double macs = 0.0;
        for (const LaunchTiles& lt : launch_tiles) {
            double m = 0.0;
            for (int g = 0; g < lt.gn; ++g) m += (double)lt.len[g] * 4 * kTileA * nz * (double)kext_of(lt.x0 + g);
            w->launch_macs.push_back(m);
            macs += m;
        }
        w->executed_macs = macs;
    }
    return EPISDET_OK;
}

}  // namespace episdet

extern "C" void episdet_test_bound_coefficients(int32_t order, int32_t score, int32_t num_cases, int32_t num_controls,
                                                double* out) {
    const double n = (double)num_cases + num_controls, a = num_cases / n, b = num_controls / n;
    episdet::tc::CountParams p;
    episdet::bound_coefficients(score, -a * std::log2(a) - b * std::log2(b), num_cases, num_controls,
                                order == 2 ? 9 : 27, &p);
    out[0] = p.cut_mul, out[1] = p.cut_add, out[2] = p.seed_mul, out[3] = p.seed_add;
}

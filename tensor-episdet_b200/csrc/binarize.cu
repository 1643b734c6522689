// binarize.cu -- genotype matrix -> the reference's per-class bit planes.
//
// hiperbio/tensor-episdet reads datasets that are already binarized: per class,
// [SNP][genotype 0/1][W] 32-bit words, MSB first, each row zero-padded to a
// multiple of 1024 bits (src/tensor-episdet.cu:58-148, README.md:48-50).  This
// builds that layout on the GPU from a dense [SNP][sample] matrix of 0/1/2
// genotype bytes and a case flag per sample.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "common.cuh"
#include "episdet.h"
#include "host_util.h"
#include "search_internal.h"

namespace episdet {

// Sample lists, cases then controls, each in sample order, and *num_cases.
// One CTA: every warp counts, then lists, one stretch of samples, a lane each.
constexpr int kListThreads = 1024;
__global__ void __launch_bounds__(kListThreads) class_lists_kernel(const uint8_t* __restrict__ is_case, int n,
                                                                   int* __restrict__ idx, int* __restrict__ num_cases) {
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // (n may be close to 2^31: unsigned positions hold the sums past it.)
    const uint32_t per = ((uint32_t)n + kListThreads - 1) / kListThreads * 32;  // samples of a warp
    const uint32_t s0 = min((uint32_t)n, warp * per), s1 = min((uint32_t)n, s0 + per);
    int cnt = 0;
#pragma unroll 8
    for (uint32_t i = s0; i < s1; i += 32)
        cnt += __popc(__ballot_sync(0xFFFFFFFFu, i + lane < s1 && __ldg(is_case + i + lane) != 0));
    if (lane == 0) s_warp[warp] = cnt;
    __syncthreads();
    int below = 0, total = 0;
    for (int i = 0; i < 32; ++i) {
        below += i < warp ? s_warp[i] : 0;
        total += s_warp[i];
    }
    int ic = below, in = total + (int)s0 - below;
#pragma unroll 8
    for (uint32_t i = s0; i < s1; i += 32) {
        const bool here = i + lane < s1, is = here && __ldg(is_case + i + lane) != 0;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, is), v = __ballot_sync(0xFFFFFFFFu, here);
        const uint32_t lower = (1u << lane) - 1u;
        if (here) idx[is ? ic + __popc(m & lower) : in + __popc(~m & lower)] = (int)i + lane;
        ic += __popc(m);
        in += __popc(v & ~m);
    }
    if (threadIdx.x == 0) *num_cases = total;
}

// The matrix is packed first, 16 SNPs of a sample to a word (bits 2 s and 2 s + 1:
// genotype of SNP s is 0, 1), so that a class's samples are gathered a word at a
// time and a 32 x 32 bit transpose of 32 samples gives the plane words of all 16
// SNPs.  The bound is reading the bytes (79 us for 8192 x 50001 at the copy rate,
// and a quarter of them written and read as words); a thread per output word,
// each reading its own 32 samples, took 1700 us there, two ballots per SNP and
// word 421 us.
constexpr int kBinSnps = 16;

// Four samples of 16 SNPs a thread.
__global__ void __launch_bounds__(256) pack_genotypes_kernel(const uint8_t* __restrict__ geno, int M, int n,
                                                             uint32_t* __restrict__ packed, size_t pitch,
                                                             int* __restrict__ bad) {
    const uint32_t i0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);  // below 2^31 + 1024
    const int snp0 = (int)blockIdx.y * kBinSnps;
    if (i0 >= (uint32_t)n) return;
    const int ns = min(kBinSnps, M - snp0);
    uint32_t acc[4] = {0, 0, 0, 0}, over = 0;
    auto add = [&](int s, uint32_t x) {
        over |= (x & 0xFCFCFCFCu) | (x & (x >> 1) & 0x01010101u);
        const uint32_t code = (~(x | (x >> 1)) & 0x01010101u) | ((x & 0x01010101u) << 1);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[e] |= ((code >> (8 * e)) & 3u) << (2 * s);
    };
    // Four bytes at any alignment are two aligned words, where those lie in the
    // matrix for all 16 rows; else one byte at a time (2 past the row's end).
    const uint8_t* first = geno + (size_t)snp0 * n + i0;
    if (ns == kBinSnps && i0 + 4 <= (uint32_t)n && first - geno >= 3 &&
        first + (size_t)(kBinSnps - 1) * n + 8 <= geno + (size_t)M * n) {
        uint32_t lo[kBinSnps], hi[kBinSnps];
#pragma unroll
        for (int s = 0; s < kBinSnps; ++s) {
            const uint8_t* p = first + (size_t)s * n;
            const uint32_t* base = reinterpret_cast<const uint32_t*>(p - ((uintptr_t)p & 3));
            lo[s] = __ldg(base);
            hi[s] = __ldg(base + 1);
        }
#pragma unroll
        for (int s = 0; s < kBinSnps; ++s)
            add(s, __funnelshift_r(lo[s], hi[s], 8 * (int)((uintptr_t)(first + (size_t)s * n) & 3)));
    } else {
        for (int s = 0; s < ns; ++s) {
            const uint8_t* p = first + (size_t)s * n;
            uint32_t x = 0;
            for (int e = 0; e < 4; ++e) x |= (uint32_t)(i0 + e < (uint32_t)n ? p[e] : 2) << (8 * e);
            add(s, x);
        }
    }
    *reinterpret_cast<uint4*>(packed + blockIdx.y * pitch + i0) = make_uint4(acc[0], acc[1], acc[2], acc[3]);
    if (over) atomicExch(bad, 1);
}

// One warp per 16 SNPs x 8 output words of a class: lane l gathers the word's
// sample l and, after the transpose, holds row l (SNP l / 2, plane l % 2); eight
// words make its 32-byte store.
struct BinClass {
    const int* idx;  // samples of the class
    uint32_t* out;   // [M][2][W]
    int n, W;
};
__global__ void __launch_bounds__(256) planes_kernel(const uint32_t* __restrict__ packed, size_t pitch, int M, BinClass a,
                                                     BinClass b) {
    const int lane = threadIdx.x & 31, wa = a.W / 8, wb = b.W / 8;
    const int chunk = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), snp0 = (int)blockIdx.y * kBinSnps;
    if (chunk >= wa + wb) return;  // uniform over the warp
    const bool second = chunk >= wa;
    const int* __restrict__ idx = second ? b.idx : a.idx;
    uint32_t* __restrict__ out = second ? b.out : a.out;
    const int nk = second ? b.n : a.n, W = second ? b.W : a.W;
    const int w0 = (second ? chunk - wa : chunk) * 8;
    const uint32_t* __restrict__ p = packed + blockIdx.y * pitch;
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int i = (w0 + k) * 32 + lane;
        v[k] = i < nk ? __ldg(p + __ldg(idx + i)) : 0u;
    }
    // warp_transpose32 gives lane l the words' bits 31 - l, first lane first.
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = warp_transpose32(v[k], lane);
    const int bit = 31 - lane, snp = snp0 + bit / 2;
    if (snp < M) {
        uint32_t* o = out + ((size_t)snp * 2 + bit % 2) * W + w0;
        if (((uintptr_t)o & 15) == 0) {
            reinterpret_cast<uint4*>(o)[0] = make_uint4(v[0], v[1], v[2], v[3]);
            reinterpret_cast<uint4*>(o)[1] = make_uint4(v[4], v[5], v[6], v[7]);
        } else {  // the caller's array
#pragma unroll
            for (int k = 0; k < 8; ++k) o[k] = v[k];
        }
    }
}

}  // namespace episdet

using namespace episdet;

extern "C" episdet_status episdet_binarize(const uint8_t* genotypes, int32_t num_snps, int32_t num_samples,
                                           const uint8_t* is_case, uint32_t* cases, uint32_t* controls,
                                           int32_t memory, int32_t device) {
    clear_error();
    if (!genotypes || !is_case || !cases || !controls)
        return set_error(EPISDET_ERR_INVALID_ARGUMENT, "binarize needs genotypes, case flags and two outputs");
    if (memory != EPISDET_HOST && memory != EPISDET_DEVICE)
        return set_error(EPISDET_ERR_INVALID_ARGUMENT, "unknown memory kind");
    const int M = num_snps, n = num_samples;
    if (M < 1 || n < 2 || (int64_t)M * n > ((int64_t)1 << 40))
        return set_error(EPISDET_ERR_INVALID_ARGUMENT, "bad matrix size %d x %d", M, n);
    Workspace* w = nullptr;
    episdet_status st = get_workspace(device, &w);
    if (st != EPISDET_OK) return st;
    std::lock_guard<std::mutex> lock(w->mu);
    CUDA_TRY(cudaSetDevice(device));
    cudaStream_t s = w->own_st;
    CUDA_TRY(w->bin_idx.ensure(sizeof(int) * (size_t)n + (size_t)n));
    int* d_idx = (int*)w->bin_idx.p;
    CUDA_TRY(w->flag.ensure(sizeof(int) * 4));
    int* d_flag = (int*)w->flag.p;  // [0] a genotype above 2, [1] number of cases
    CUDA_TRY(cudaMemsetAsync(d_flag, 0, sizeof(int) * 2, s));
    const uint8_t* d_case = is_case;
    if (memory == EPISDET_HOST) {
        uint8_t* f = (uint8_t*)(d_idx + n);
        CUDA_TRY(cudaMemcpyAsync(f, is_case, (size_t)n, cudaMemcpyHostToDevice, s));
        d_case = f;
    }
    class_lists_kernel<<<1, kListThreads, 0, s>>>(d_case, n, d_idx, d_flag + 1);
    CHECK_LAUNCH();
    int nc = 0;
    CUDA_TRY(cudaMemcpyAsync(&nc, d_flag + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    const int nn = n - nc;
    if (nc < 1 || nn < 1) return set_error(EPISDET_ERR_INVALID_ARGUMENT, "the case flags leave a class empty");
    const int Wc = episdet_class_words(nc), Wn = episdet_class_words(nn);
    const size_t geno_bytes = (size_t)M * n;
    const size_t out_words[2] = {(size_t)M * 2 * Wc, (size_t)M * 2 * Wn};
    const uint8_t* d_geno = genotypes;
    uint32_t* d_out[2] = {cases, controls};
    if (memory == EPISDET_HOST) {
        CUDA_TRY(w->bin_geno.ensure(geno_bytes));
        CUDA_TRY(cudaMemcpyAsync(w->bin_geno.p, genotypes, geno_bytes, cudaMemcpyHostToDevice, s));
        d_geno = (const uint8_t*)w->bin_geno.p;
        for (int c = 0; c < 2; ++c) {
            CUDA_TRY(w->bin_out[c].ensure(sizeof(uint32_t) * out_words[c]));
            d_out[c] = (uint32_t*)w->bin_out[c].p;
        }
    }
    const int groups = (int)((M + kBinSnps - 1L) / kBinSnps);
    const size_t pitch = ((size_t)n + 3) & ~(size_t)3;
    const BinClass ca{d_idx, d_out[0], nc, Wc}, cb{d_idx + nc, d_out[1], nn, Wn};
    // SNP groups in batches of at most 64 MB of words (and of the grid's second dimension).
    const int batch = (int)std::max<size_t>(1, std::min<size_t>(32768, ((size_t)64 << 20) / (sizeof(uint32_t) * pitch)));
    CUDA_TRY(w->bin_pack.ensure(sizeof(uint32_t) * std::min(groups, batch) * pitch));
    uint32_t* d_pack = (uint32_t*)w->bin_pack.p;
    for (int g0 = 0; g0 < groups; g0 += batch) {
        const int ng = std::min(batch, groups - g0);
        const long r0 = (long)g0 * kBinSnps;
        const int rows = (int)std::min(M - r0, (long)ng * kBinSnps);
        pack_genotypes_kernel<<<dim3((unsigned)((pitch / 4 + 255) / 256), (unsigned)ng), 256, 0, s>>>(
            d_geno + (size_t)r0 * n, rows, n, d_pack, pitch, d_flag);
        CHECK_LAUNCH();
        BinClass ga = ca, gb = cb;
        ga.out += (size_t)r0 * 2 * Wc;
        gb.out += (size_t)r0 * 2 * Wn;
        planes_kernel<<<dim3((unsigned)((Wc / 8 + Wn / 8 + 7) / 8), (unsigned)ng), 256, 0, s>>>(d_pack, pitch, rows, ga, gb);
        CHECK_LAUNCH();
    }
    int bad = 0;
    CUDA_TRY(cudaMemcpyAsync(&bad, w->flag.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    if (memory == EPISDET_HOST) {
        CUDA_TRY(cudaMemcpyAsync(cases, d_out[0], sizeof(uint32_t) * out_words[0], cudaMemcpyDeviceToHost, s));
        CUDA_TRY(cudaMemcpyAsync(controls, d_out[1], sizeof(uint32_t) * out_words[1], cudaMemcpyDeviceToHost, s));
    }
    CUDA_TRY(cudaStreamSynchronize(s));
    if (bad) return set_error(EPISDET_ERR_INVALID_INPUT, "a genotype value is above 2");
    return EPISDET_OK;
}

// binarize.cu -- genotype matrix -> the reference's per-class bit planes.
//
// hiperbio/tensor-episdet reads datasets that are already binarized: per class,
// [SNP][genotype 0/1][W] 32-bit words, MSB first, each row zero-padded to a
// multiple of 1024 bits (src/tensor-episdet.cu:58-148, README.md:48-50).  This
// builds that layout on the GPU from a dense [SNP][sample] matrix of 0/1/2
// genotype bytes and a case flag per sample.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "episdet.h"
#include "host_util.h"
#include "search_internal.h"
#include "tc_ptx.cuh"

namespace episdet {

// Sample lists, cases then controls, each in sample order, and *num_cases.
// One CTA: every thread counts, then lists, one stretch of samples.
constexpr int kListThreads = 1024;
__global__ void __launch_bounds__(kListThreads) class_lists_kernel(const uint8_t* __restrict__ is_case, int n,
                                                                   int* __restrict__ idx, int* __restrict__ num_cases) {
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (n + kListThreads - 1) / kListThreads;
    const int s0 = min(n, (int)threadIdx.x * per), s1 = min(n, s0 + per);
    int cnt = 0;
    for (int i = s0; i < s1; ++i) cnt += __ldg(is_case + i) != 0;
    int x = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    int below = 0, total = 0;
    for (int i = 0; i < 32; ++i) {
        below += i < warp ? s_warp[i] : 0;
        total += s_warp[i];
    }
    int ic = below + x - cnt, in = total + s0 - ic;
    for (int i = s0; i < s1; ++i) idx[__ldg(is_case + i) != 0 ? ic++ : in++] = i;
    if (threadIdx.x == 0) *num_cases = total;
}

// One warp per kBinSnps SNPs x 32 output words of a class.  The 1,024 samples of
// those words lie in one stretch of each genotype row: the warp copies the
// stretch into shared memory (kBinSpan bytes at most; a class so sparse that it
// is longer reads the row instead), and for each word the lanes read its 32
// samples' bytes and two ballots make the plane words; lane k keeps word k, so
// the stores are whole lines.  The bound is reading every genotype byte once
// per class (8192 x 50001: 79 us for once at the copy rate); a thread per word,
// each reading its own 32 samples, took 1700 us there, ballots over global
// bytes 421 us, this BIN_US us.
constexpr int kBinSnps = 16;
constexpr int kBinSpan = 4096;
constexpr int kBinWarps = 4;
struct BinClass {
    const int* idx;  // samples of the class
    uint32_t* out;   // [M][2][W]
    int n, W;
};
__global__ void __launch_bounds__(32 * kBinWarps) binarize_kernel(const uint8_t* __restrict__ geno, int M, int n,
                                                                  BinClass a, BinClass b, int* __restrict__ bad) {
    __shared__ __align__(16) uint8_t s_row[kBinWarps][2][kBinSpan + 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wa = a.W / 32, wb = b.W / 32;
    const long unit = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // both classes of an SNP group together
    const long group = unit / (wa + wb);
    const int chunk = (int)(unit % (wa + wb));
    if (group * kBinSnps >= M) return;
    const bool second = chunk >= wa;
    const int* __restrict__ idx = second ? b.idx : a.idx;
    uint32_t* __restrict__ out = second ? b.out : a.out;
    const int nk = second ? b.n : a.n, W = second ? b.W : a.W;
    const int w0 = (second ? chunk - wa : chunk) * 32, i0 = w0 * 32;
    const int snp0 = (int)group * kBinSnps, ns = min(kBinSnps, M - snp0);
    // The stretch [lo, hi) of a row (empty when the words are all padding).
    const int lo = i0 < nk ? __ldg(idx + i0) : 0, hi = i0 < nk ? __ldg(idx + min(nk, i0 + 1024) - 1) + 1 : 0;
    const bool staged = hi - lo <= kBinSpan;
    uint16_t rel[32];  // this lane's sample of each word, from lo
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const int i = i0 + k * 32 + lane;
        rel[k] = staged && i < nk ? (uint16_t)(__ldg(idx + i) - lo) : 0xFFFFu;
    }
    // Copies a row's stretch: whole aligned 16 bytes, byte by byte where they
    // would leave the row.  Returns where the stretch begins in the buffer.
    auto copy = [&](int s) {
        const uint8_t* g0 = geno + (size_t)(snp0 + s) * n;
        const uint8_t* from = g0 + lo;
        const int skew = (int)((uintptr_t)from & 15);
        const uint8_t* base = from - skew;
        uint8_t* row = s_row[warp][s & 1];
        for (int o = 16 * lane; o < hi - lo + skew; o += 512) {
            const uint8_t* p = base + o;
            if (p >= g0 && p + 16 <= g0 + n) {
                ptx::cp_async16(ptx::smem_u32(row + o), p, true);
            } else {
                for (int e = 0; e < 16; ++e)
                    if (p + e >= from && p + e < g0 + hi) row[o + e] = p[e];
            }
        }
        ptx::cp_async_commit();
        return skew;
    };
    bool over = false;
    int skew = 0, skew_next = staged ? copy(0) : 0;
    for (int s = 0; s < ns; ++s) {
        const uint8_t* g0 = geno + (size_t)(snp0 + s) * n;
        uint32_t p0 = 0, p1 = 0;
        skew = skew_next;
        if (staged) {
            // The next row's copy is in flight while this one is read.
            if (s + 1 < ns) {
                skew_next = copy(s + 1);
                ptx::cp_async_wait<1>();
            } else {
                ptx::cp_async_wait<0>();
            }
            __syncwarp();
            const uint8_t* row = s_row[warp][s & 1] + skew;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const uint32_t g = rel[k] != 0xFFFFu ? row[rel[k]] : 2u;
                const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, g == 0), m1 = __ballot_sync(0xFFFFFFFFu, g == 1);
                over |= g > 2;
                if (lane == k) p0 = m0, p1 = m1;
            }
            __syncwarp();  // before the buffer's next copy
        } else {
            for (int k = 0; k < 32; ++k) {
                const int i = i0 + k * 32 + lane;
                const uint32_t g = i < nk ? __ldg(g0 + __ldg(idx + i)) : 2u;
                const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, g == 0), m1 = __ballot_sync(0xFFFFFFFFu, g == 1);
                over |= g > 2;
                if (lane == k) p0 = m0, p1 = m1;
            }
        }
        uint32_t* o = out + (size_t)(snp0 + s) * 2 * W + w0 + lane;
        o[0] = __brev(p0);
        o[W] = __brev(p1);
    }
    if (__any_sync(0xFFFFFFFFu, over) && lane == 0) atomicExch(bad, 1);
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
    const BinClass ca{d_idx, d_out[0], nc, Wc}, cb{d_idx + nc, d_out[1], nn, Wn};
    const long warps = (long)((M + kBinSnps - 1) / kBinSnps) * (Wc / 32 + Wn / 32);
    binarize_kernel<<<(unsigned)((warps + kBinWarps - 1) / kBinWarps), 32 * kBinWarps, 0, s>>>(d_geno, M, n, ca, cb, d_flag);
    CHECK_LAUNCH();
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

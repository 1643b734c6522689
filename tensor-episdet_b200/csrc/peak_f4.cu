// peak_f4.cu -- exactness check and rate of tcgen05.mma kind::mxf4 on B200.
//
//   episdet-peak-f4 [MMAs per CTA pair]
//
// The counting engine can hold its 0/1 operand rows as packed e2m1 values
// (0.0 and 1.0, four bits each) instead of unsigned bytes: half the bytes per
// sample and twice the MACs per instruction.  The block scale factors are all
// 1.0 (UE8M0 127), accumulation is FP32, so a count is exact while it stays
// below 2^24.  This program checks that on the device and measures the rate:
//
//  * check: A row i is all 1.0 when i % 3 == 1, B row j all 1.0 when j % 4 != 0
//    (every other value 0), so every D[i][j] must equal the K length or 0 --
//    independent of the swizzle and of the nibble order inside a byte, which A
//    and B share; in both instruction forms, cta_group::1 (M = 128, one CTA) and
//    cta_group::2 (M = 256 over a cluster of two CTAs, each holding 128 A rows
//    and N/2 B rows, the even one issuing: the counting engine's form);
//  * rate: back-to-back MMAs of the pair form on resident tiles, over N, the
//    MMAs per commit (or none) and how they are issued: by one elected lane of a
//    converged warp (the engine's way), or under a one-lane branch.  The loops
//    are unrolled over a commit group, so that descriptors are ready in uniform
//    registers: with run-time loops and one-lane branches an MMA takes about 100
//    clocks to issue, more than the 56 that N = 112 takes to run.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <string>

#include "tc_ptx.cuh"

using namespace episdet;

namespace {

constexpr int kThreads = 128;
constexpr uint64_t kLimitNs = 2000000000ull;
constexpr int kInFlight = 64;  // MMAs in flight at most
constexpr int kMaxRing = 16;   // commit groups in flight (commit_every >= 4)

__device__ int g_err;
__device__ unsigned long long g_bad;

__device__ __forceinline__ void mma_mxf4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(
            d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
}

template <int N, bool PAIR>
constexpr size_t smem_bytes() {
    return 1024 + 16384 + (size_t)(PAIR ? N / 2 : N) * 128 + (kMaxRing + 1) * 8 + 16 + 256;
}

// `groups` groups of `cper` MMAs, one commit per group.  check != 0: the
// exactness check (one accumulator, K = 64 * groups * cper values).
template <int N, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
    f4_kernel(int groups, int cper, int check, unsigned long long* cycles) {
    constexpr int kBRows = PAIR ? N / 2 : N;
    // Scale factors: columns sf0 .. 511 of every lane hold bytes of 127 (2^0);
    // the pair form uses the engine's columns 448 .. 511.
    constexpr uint32_t sf0 = PAIR ? 448u : 496u;
    constexpr uint32_t sfb_off = PAIR ? 32u : 8u;
    extern __shared__ uint8_t raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    uint8_t* a = sm;          // 128 rows x 128 bytes
    uint8_t* b = sm + 16384;  // kBRows rows x 128 bytes
    uint64_t* bars = reinterpret_cast<uint64_t*>(b + kBRows * 128);  // [0, kMaxRing) ring, [kMaxRing] drain
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + kMaxRing + 1);
    int* s_abort = reinterpret_cast<int*>(s_tmem + 1);
    int* s_never = s_abort + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = PAIR ? (int)ptx::cluster_ctarank() : 0;
    // Row-constant operands (a byte holds two e2m1 values: 0x22 = two 1.0).
    // B row j of the pair's N rows is row j - rank * N/2 of CTA `rank`.
    for (int i = threadIdx.x; i < 128 * 128; i += kThreads) a[i] = ((i >> 7) % 3 == 1) ? 0x22 : 0x00;
    for (int i = threadIdx.x; i < kBRows * 128; i += kThreads)
        b[i] = ((rank * kBRows + (i >> 7)) % 4 != 0) ? 0x22 : 0x00;
    if (threadIdx.x == 0) {
        for (int i = 0; i <= kMaxRing; ++i) ptx::mbar_init(&bars[i], 1);
        *s_abort = 0;
        *s_never = 0;
        ptx::fence_barrier_init();
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) {
        if constexpr (PAIR) {
            ptx::tmem_alloc_pair(s_tmem, 512);
            ptx::tmem_relinquish_pair();
        } else {
            ptx::tmem_alloc(s_tmem, 512);
            ptx::tmem_relinquish();
        }
    }
    ptx::tc_fence_before();
    if constexpr (PAIR)
        ptx::cluster_sync();
    else
        __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    for (uint32_t c = sf0; c < 512u; c += 8) ptx::tmem_st8_fill(lane_base + c, 0x7F7F7F7Fu);
    ptx::tmem_wait_st();
    // Both CTAs' operands and scale factors are in place before the first MMA.
    ptx::tc_fence_before();
    if constexpr (PAIR)
        ptx::cluster_sync();
    else
        __syncthreads();
    ptx::tc_fence_after();
    volatile int* abort = s_abort;
    if (warp == 0 && lane == 0) {
        if (rank == 0) {
            const uint32_t idesc = ptx::idesc_mxf4(N, PAIR ? 256 : 128);
            const uint64_t ad = ptx::smem_desc_sw128(ptx::smem_u32(a)), bd = ptx::smem_desc_sw128(ptx::smem_u32(b));
            const uint32_t sfa = tmem + sf0, sfb = tmem + sf0 + sfb_off;
            const int ring = kInFlight / cper;
            long long t0 = clock64();
            uint32_t ph = 0;
            uint32_t gm = 0;
            for (int g = 0; g < groups; ++g) {
                const int slot = g % ring;
                if (g >= ring) {
                    if (!ptx::mbar_wait(&bars[slot], (ph >> slot) & 1u, abort, kLimitNs)) {
                        atomicExch(&g_err, 1);
                        *s_abort = 1;
                        break;
                    }
                    ph ^= 1u << slot;
                }
                for (int m = 0; m < cper; ++m, ++gm) {
                    const int kk = gm & 3;  // 4 MMAs of K = 64 cover one 128-byte block
                    // Two accumulator regions below the scale factors (one for N = 256).
                    const uint32_t acc = (check || N > 224) ? 0u : ((gm >> 2) & 1u) * (uint32_t)N;
                    const uint32_t first = (check && gm == 0) ? 0u : 1u;
                    if constexpr (PAIR)
                        ptx::mma_mxf4_pair(tmem + acc, ad + 2 * kk, bd + 2 * kk, idesc, sfa, sfb, first);
                    else
                        mma_mxf4(tmem + acc, ad + 2 * kk, bd + 2 * kk, idesc, sfa, sfb, first);
                }
                if constexpr (PAIR)
                    ptx::mma_commit_pair_mc(&bars[slot], 0x3);  // as the engine: both CTAs' barriers
                else
                    ptx::mma_commit(&bars[slot]);
            }
            if constexpr (PAIR)
                ptx::mma_commit_pair_mc(&bars[kMaxRing], 0x3);
            else
                ptx::mma_commit(&bars[kMaxRing]);
            if (!ptx::mbar_wait(&bars[kMaxRing], 0, s_never, kLimitNs)) atomicExch(&g_err, 2);
            cycles[blockIdx.x] = (unsigned long long)(clock64() - t0);
        } else if (!ptx::mbar_wait(&bars[kMaxRing], 0, s_never, kLimitNs)) {
            atomicExch(&g_err, 3);  // the odd CTA: its accumulators are complete
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const int unit = PAIR ? (int)ptx::cluster_id_x() : (int)blockIdx.x;
    if (check && unit == 0) {
        const float want_one = 64.0f * (float)groups * (float)cper;
        const int row = warp * 32 + lane;
        unsigned long long bad = 0;
        for (int c0 = 0; c0 < N; c0 += 8) {
            uint32_t v[8];
            ptx::tmem_ld8(lane_base + (uint32_t)c0, v);
            ptx::tmem_wait_ld();
            ptx::tmem_regs_ready(v);
            for (int e = 0; e < 8; ++e) {
                const int col = c0 + e;
                const float want = (row % 3 == 1 && col % 4 != 0) ? want_one : 0.0f;
                if (__uint_as_float(v[e]) != want) ++bad;
            }
        }
        if (bad) atomicAdd(&g_bad, bad);
    }
    // Neither CTA of a pair releases TMEM or leaves while the pair's MMAs may
    // still read its shared memory.
    ptx::tc_fence_before();
    if constexpr (PAIR)
        ptx::cluster_sync();
    else
        __syncthreads();
    if (warp == 0) {
        ptx::tc_fence_after();
        if constexpr (PAIR)
            ptx::tmem_dealloc_pair(tmem, 512);
        else
            ptx::tmem_dealloc(tmem, 512);
    }
}


// Issue-rate kernel: `groups` groups of CPER MMAs, a commit after each (nothing
// waits on it) when COMMIT; ELECT: the warp walks the groups together and one
// elected lane issues, else one lane walks alone.
template <int N, int CPER, bool ELECT, bool COMMIT>
__global__ void __launch_bounds__(kThreads, 1) issue_kernel(int groups, unsigned long long* cycles) {
    constexpr int kBBytes = (N / 2) * 128;
    extern __shared__ uint8_t raw[];
    uint8_t* a = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));  // 4 K blocks
    uint8_t* b = a + 4 * 16384;
    uint64_t* bars = reinterpret_cast<uint64_t*>(b + 4 * kBBytes);  // sink, drain
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 2);
    int* s_never = reinterpret_cast<int*>(s_tmem + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)ptx::cluster_ctarank();
    for (int i = threadIdx.x; i < 4 * (16384 + kBBytes); i += kThreads) a[i] = (uint8_t)((i * 2654435761u >> 20) & 0x22);
    if (threadIdx.x == 0) {
        ptx::mbar_init(&bars[0], 1);
        ptx::mbar_init(&bars[1], 1);
        *s_never = 0;
        ptx::fence_barrier_init();
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) {
        ptx::tmem_alloc_pair(s_tmem, 512);
        ptx::tmem_relinquish_pair();
    }
    ptx::tc_fence_before();
    ptx::cluster_sync();
    ptx::tc_fence_after();
    const uint32_t tmem = *s_tmem;
    for (uint32_t c = 448; c < 512u; c += 8) ptx::tmem_st8_fill(tmem + ((uint32_t)(warp * 32) << 16) + c, 0x7F7F7F7Fu);
    ptx::tmem_wait_st();
    ptx::tc_fence_before();
    ptx::cluster_sync();
    ptx::tc_fence_after();
    const uint32_t idesc = ptx::idesc_mxf4(N, 256);
    uint64_t ad[4], bd[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        ad[i] = ptx::smem_desc_sw128(ptx::smem_u32(a + i * 16384));
        bd[i] = ptx::smem_desc_sw128(ptx::smem_u32(b + i * kBBytes));
    }
    auto group = [&](int g) {
#pragma unroll
        for (int m = 0; m < CPER; ++m)
            ptx::mma_mxf4_pair(tmem + (uint32_t)((g & 1) * (N > 224 ? 0 : N)), ad[(m >> 2) & 3] + 2 * (m & 3),
                               bd[(m >> 2) & 3] + 2 * (m & 3), idesc, tmem + 448, tmem + 480, 1u);
        if (COMMIT) ptx::mma_commit_pair_mc(&bars[0], 0x3);
    };
    if (warp == 0) {
        const long long t0 = clock64();
        if (rank == 0) {
            if (ELECT) {
                for (int g = 0; g < groups; ++g) {
                    if (ptx::elect_one()) group(g);
                    __syncwarp();
                }
                if (ptx::elect_one()) ptx::mma_commit_pair_mc(&bars[1], 0x3);
            } else if (lane == 0) {
                for (int g = 0; g < groups; ++g) group(g);
                ptx::mma_commit_pair_mc(&bars[1], 0x3);
            }
            __syncwarp();
        }
        if (lane == 0) {
            if (!ptx::mbar_wait(&bars[1], 0, s_never, kLimitNs)) atomicExch(&g_err, 9);
            cycles[blockIdx.x] = (unsigned long long)(clock64() - t0);
        }
        __syncwarp();
    }
    ptx::tc_fence_before();
    ptx::cluster_sync();
    if (warp == 0) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem, 512);
    }
}

}  // namespace

#define CK(x)                                                                               \
    do {                                                                                    \
        cudaError_t e_ = (x);                                                               \
        if (e_ != cudaSuccess) {                                                            \
            fprintf(stderr, "%s:%d %s: %s\n", __FILE__, __LINE__, #x, cudaGetErrorString(e_)); \
            return 1;                                                                       \
        }                                                                                   \
    } while (0)

template <int N, bool PAIR>
static int launch(int grid, int groups, int cper, int check, unsigned long long* d_cyc) {
    const size_t smem = smem_bytes<N, PAIR>();
    CK(cudaFuncSetAttribute(f4_kernel<N, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = PAIR ? 2 : 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CK(cudaLaunchKernelEx(&cfg, f4_kernel<N, PAIR>, groups, cper, check, d_cyc));
    CK(cudaGetLastError());
    return 0;
}

// The exactness check on one CTA or pair: groups of cper MMAs, iters x 16 in all.
template <int N, bool PAIR>
static int run(int sms, int iters, int cper, int check, unsigned long long* d_cyc) {
    const int unit = PAIR ? 2 : 1;
    const int grid = check ? unit : (sms / unit) * unit;
    const int groups = iters * 16 / cper;
    if (!check) {
        if (launch<N, PAIR>(grid, 64 * 16 / cper, cper, 0, d_cyc)) return 1;  // warm-up
        CK(cudaDeviceSynchronize());
    }
    unsigned long long zero = 0;
    CK(cudaMemcpyToSymbol(g_bad, &zero, sizeof(zero)));
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    CK(cudaEventRecord(e0));
    if (launch<N, PAIR>(grid, groups, cper, check, d_cyc)) return 1;
    CK(cudaEventRecord(e1));
    CK(cudaEventSynchronize(e1));
    int err = 0;
    unsigned long long bad = 0, cyc = 0;
    CK(cudaMemcpyFromSymbol(&err, g_err, sizeof(int)));
    CK(cudaMemcpyFromSymbol(&bad, g_bad, sizeof(bad)));
    CK(cudaMemcpy(&cyc, d_cyc, sizeof(cyc), cudaMemcpyDeviceToHost));
    float ms = 0.0f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    CK(cudaEventDestroy(e0));
    CK(cudaEventDestroy(e1));
    // MACs of one SM: its 128 rows of D (the pair's M = 256 is split over two SMs).
    const double per_sm = (double)groups * cper * 128.0 * N * 64.0;
    const char* form = PAIR ? "pair" : "cta1";
    if (check)
        printf("{\"form\": \"%s\", \"n\": %d, \"mode\": \"check\", \"k_values\": %d, \"bad_cells\": %llu, "
               "\"err\": %d}\n",
               form, N, groups * cper * 64, bad, err);
    else
        printf("{\"form\": \"%s\", \"n\": %d, \"commit_every\": %d, \"mode\": \"rate\", \"ms\": %.3f, "
               "\"tmacs_per_s\": %.1f, \"mac_per_clk_per_sm\": %.0f, \"err\": %d}\n",
               form, N, cper, ms, per_sm * grid / (ms * 1e-3) / 1e12, per_sm / (double)cyc, err);
    return err || bad ? 1 : 0;
}

// One rate point: a CTA pair on every two SMs, `total` MMAs per pair.
template <int N, int CPER, bool ELECT, bool COMMIT>
static int rate(int sms, int total, unsigned long long* d_cyc) {
    const size_t smem = 1024 + 4 * 16384 + 4 * (size_t)(N / 2) * 128 + 256;
    auto* const kern = issue_kernel<N, CPER, ELECT, COMMIT>;
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((sms / 2) * 2);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int groups = total / CPER;
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    float best = 1e30f;
    for (int r = 0; r < 3; ++r) {  // the first is the warm-up
        CK(cudaEventRecord(e0));
        CK(cudaLaunchKernelEx(&cfg, kern, groups, d_cyc));
        CK(cudaEventRecord(e1));
        CK(cudaEventSynchronize(e1));
        float ms = 0.0f;
        CK(cudaEventElapsedTime(&ms, e0, e1));
        if (r > 0 && ms < best) best = ms;
    }
    int err = 0;
    unsigned long long cyc = 0;
    CK(cudaMemcpyFromSymbol(&err, g_err, sizeof(int)));
    CK(cudaMemcpy(&cyc, d_cyc, sizeof(cyc), cudaMemcpyDeviceToHost));
    CK(cudaEventDestroy(e0));
    CK(cudaEventDestroy(e1));
    const double n = (double)groups * CPER;
    printf("{\"form\": \"pair\", \"n\": %d, \"mma_per_commit\": %d, \"issue\": \"%s\", \"ns_per_mma\": %.1f, "
           "\"clk_per_mma\": %.1f, \"tmacs_per_s\": %.1f, \"sm_mhz\": %.0f, \"err\": %d}\n",
           N, COMMIT ? CPER : 0, ELECT ? "elected" : "one lane", best * 1e6 / n, cyc / n,
           n * (sms / 2) * 256.0 * N * 64.0 / (best * 1e-3) / 1e12, cyc / (best * 1e3), err);  // the clock it ran at
    return err ? 1 : 0;
}

int main(int argc, char** argv) {
    int total = argc > 1 ? atoi(argv[1]) : 60000;
    if (total < 1024 || total > 100000000) total = 60000;
    cudaDeviceProp p;
    CK(cudaGetDeviceProperties(&p, 0));
    if (p.major != 10) {
        fprintf(stderr, "needs an sm_100 device\n");
        return 1;
    }
    printf("{\"gpu\": \"%s\", \"sms\": %d}\n", p.name, p.multiProcessorCount);
    const int sms = p.multiProcessorCount;
    unsigned long long* d_cyc = nullptr;
    CK(cudaMalloc(&d_cyc, sizeof(unsigned long long) * sms));
    int rc = 0;
    // Exactness first (4096 x 16 MMAs = 4,194,304 values per count).
    rc |= run<128, false>(sms, 4096, 16, 1, d_cyc);
    rc |= run<112, false>(sms, 4096, 16, 1, d_cyc);
    rc |= run<256, false>(sms, 64, 16, 1, d_cyc);
    rc |= run<112, true>(sms, 4096, 16, 1, d_cyc);
    rc |= run<224, true>(sms, 4096, 16, 1, d_cyc);
    rc |= run<256, true>(sms, 64, 16, 1, d_cyc);
    if (rc) return rc;
    rc |= rate<112, 4, true, true>(sms, total, d_cyc);
    rc |= rate<112, 4, false, true>(sms, total, d_cyc);
    rc |= rate<112, 16, true, true>(sms, total, d_cyc);
    rc |= rate<112, 16, true, false>(sms, total, d_cyc);
    rc |= rate<224, 4, true, true>(sms, total, d_cyc);
    rc |= rate<224, 4, false, true>(sms, total, d_cyc);
    rc |= rate<224, 8, true, true>(sms, total, d_cyc);
    rc |= rate<224, 16, true, false>(sms, total, d_cyc);
    rc |= rate<256, 4, true, true>(sms, total, d_cyc);
    rc |= rate<256, 16, true, false>(sms, total, d_cyc);
    CK(cudaFree(d_cyc));
    return rc;
}

// search_internal.h -- host-side workspace and helpers shared by the engines.
#pragma once
#include <cuda_runtime.h>

#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "device_data.cuh"
#include "episdet.h"

namespace episdet {

episdet_status cuda_fail(cudaError_t e, const char* what);

#define CUDA_TRY(x)                                     \
    do {                                                \
        cudaError_t e_ = (x);                           \
        if (e_ != cudaSuccess) return cuda_fail(e_, #x); \
    } while (0)

// Launch-error check naming the launch site.
#define CHECK_LAUNCH()                                                         \
    do {                                                                       \
        cudaError_t e_ = cudaGetLastError();                                   \
        if (e_ != cudaSuccess) return cuda_fail(e_, "launch at " __FILE__ ":" EPI_STR(__LINE__)); \
    } while (0)
#define EPI_STR2(x) #x
#define EPI_STR(x) EPI_STR2(x)

// Grow-only device allocation kept between calls.
struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes);
    void release();
};

// The same in pinned host memory.
struct HostBuf {
    void* p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes);
    void release();
};

// Sets of regrouped operand buffers of the triplet engine: the regrouping of
// group g + kXSets - 1 (second stream) overlaps the counting launch of group g.
constexpr int kXSets = 2;
constexpr int kXGroup = 4;  // first SNPs per triplet launch at least
// Tiles per CTA pair that a triplet launch should have (1536 SNPs x 40000
// samples: 8 39.8 ms, 16 39.0, 32 38.7 at twice the rows).
constexpr int kGroupTiles = 16;
constexpr size_t kGroupBytes = (size_t)2 << 30;   // regrouped rows a launch may take for them
// Panels up to this size use narrow triplet tiles, whose last tile of a row is a
// smaller share of the work, up to a number of samples: past it a tile takes as
// long as its MMAs, and a narrow one's need 103 operand bytes a clock instead of
// 67.  Narrow against wide, K2, ms:
//   samples     4,000        40,000       56,000        90,000       262,144
//   200 SNPs    0.61  0.62   0.94  0.97    1.13  1.13    1.55  1.47    3.9   3.6
//   400         1.44  1.39   2.51  2.35    3.20  2.83    4.71  4.06   13.0  10.9
//   600         2.82  2.92   5.04  5.00    6.51  6.19    9.98  9.39   28.2  25.6
//   704         4.10  4.14   7.01  7.14    9.04  8.68   13.90 13.26   37.8  34.5
//   1024       10.54 10.20  15.57 15.90                               83.5  74.2
//   1250       18.22 17.44  25.63 25.94
// (MI the same within 3 %; above 704 SNPs neither is ahead at few samples.)
constexpr int kNarrowTileSnps = 704;
constexpr int kNarrowTileSamples = 48000;

struct Workspace {
    int device = 0;
    int sms = 0;
    cudaStream_t st = nullptr;      // stream of the current call (own_st or the caller's)
    cudaStream_t own_st = nullptr;  // the library's own stream
    cudaStream_t aux_st = nullptr;  // operand regrouping, overlapped with the counting launches
    cudaEvent_t ev_ready = nullptr, ev_cmp[kXSets] = {}, ev_tc[kXSets] = {};  // ordering between st and aux_st
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    std::mutex mu;
    DevBuf bits[2], marg[2], pair4[2], t32, t64, slots, counts, tiles, merged, flag;
    HostBuf results;      // a search's result lists on the host
    DevBuf ptab, ptabx;   // 3-way tensor engine: pair table, and (Y-blocked) the rows of the current first SNPs
    DevBuf frows;         // packed e2m1 operand rows of the planes (2-way and pair table)
    DevBuf rtab;          // counts that cells are derived from, per SNP (tensor engine)
    DevBuf stash;         // drained count segments (tensor engine)
    DevBuf seeds;         // seed pass: one key per scoring thread (tensor engine)
    DevBuf planes_t[2];   // sample-major transposed planes per class (3-way tensor engine's regrouping)
    DevBuf xsub[kXSets];  // sample-regrouped operand rows of one launch's first SNPs (tensor engine)
    DevBuf xinfo;         // per-X segment tables (tensor engine)
    DevBuf tensor_flag;   // device error / progress words of the tensor engine
    DevBuf cbuf;          // per-CTA candidate lists (tensor engine)
    DevBuf perm_tot;      // label-free pair totals of a permutation batch's cohort
    DevBuf perm_tt, perm_marg, perm_labels, perm_mask;  // label mode: transposed planes, genotype counts, labels, class masks
    const float4* label_tot = nullptr;  // set during a label-mode 2-way search (episdet_search_perm)
    DevBuf perm_planes, perm_cls[2], perm_idx;  // phenotype-permutation staging
    DevBuf bin_geno, bin_idx, bin_pack, bin_out[2];       // genotype-matrix binarizer staging
    // Per-call accounting.
    int64_t h2d = 0, d2h = 0;
    bool timing = false;
    std::vector<cudaEvent_t> tev;  // event pool: (start, end) around each counting launch
    int tev_used = 0;
    int64_t count_launches = 0;
    double executed_macs = 0.0;
    std::vector<double> launch_ms, launch_macs;  // EPISDET_FLAG_TIMING: per counting launch of the last call
    int tab_score = -1, tab_size = 0, tab_nc = -1, tab_nn = -1;
    int stage_override = -1;  // triplet tiles: -1 by the panel-size rule, 0 narrow, 1 wide
    // The first SNPs of a launch that memory last allowed, for regrouped rows of
    // limit_bytes a first SNP; asked again after limit_uses searches.
    size_t limit_bytes = 0;
    int limit = 0, limit_uses = 0;
    int pairs[16] = {};       // resident CTA pairs of each counting-kernel instance (0: not asked yet)
    float inv32 = 0.0f, hy32 = 0.0f;
    double inv64 = 0.0, hy64 = 0.0;

    void release_all() {
        for (DevBuf& b : xsub) b.release();
        DevBuf* all[] = {&bits[0], &bits[1], &marg[0], &marg[1], &pair4[0], &pair4[1], &ptab, &ptabx, &t32,
                         &t64, &slots,
                         &counts, &tiles, &merged, &flag, &frows, &rtab, &stash, &seeds, &planes_t[0], &planes_t[1],
                         &xinfo,
                         &tensor_flag, &cbuf, &perm_tot, &perm_tt, &perm_marg, &perm_labels, &perm_mask, &perm_planes, &perm_cls[0], &perm_cls[1], &perm_idx,
                         &bin_geno, &bin_idx, &bin_pack, &bin_out[0], &bin_out[1]};
        for (DevBuf* b : all) b->release();
        results.release();
        limit_uses = 0;
        tab_score = tab_nc = tab_nn = -1;
    }
};

constexpr int kMaxLanes = 4;  // concurrent cohorts of one batched call
episdet_status get_workspace(int device, Workspace** out);
episdet_status get_workspace_lane(int device, int lane, Workspace** out);
episdet_status build_tables(Workspace* w, int score, int nc, int nn, ScoreTables* T);
episdet_status stage_dataset(Workspace* w, const episdet_dataset* d, bool validate, DevData* D, uint64_t* launches);
episdet_status prepare_slots(Workspace* w, int nslots, int k, Slots* S);
episdet_status check_options(const episdet_options* in, int M, episdet_options* o);
episdet_status check_dataset(const episdet_dataset* d, int order);
// Largest class the tensor engine counts exactly (FP32 accumulators: 2^24).
constexpr int kTensorMaxClass = 1 << 24;
// Largest label-free pair table (M x M x 16 bytes) a permutation batch builds
// for its label mode; beyond it every label runs as a two-class search.
constexpr long long kLabelTotalsMaxBytes = 32ll << 30;
// H(Y) of the FP32 MI score as include/scoring.hpp:29-30 evaluates it on the
// device: each class's p = n * (1/N) is a float product; the first term is a
// double product rounded to float, the second a double multiply-add (nvcc
// contracts `entropyY += (-1.0) * p * t` into one fused operation) rounded to
// float.  t32 is the FP32 log2 table, indexed by count.
inline float mi_hy32(int nc, int nn, float inv32, const float* t32) {
    float p1 = (float)nc * inv32;
    float hy = (float)(-((double)p1 * (double)t32[nc]));
    float p2 = (float)nn * inv32;
    return (float)std::fma(-(double)p2, (double)t32[nn], (double)hy);
}

bool tensor_exact_for(const episdet_dataset* d);
episdet_status check_engine(const episdet_dataset* d, const episdet_options& o);

// Brackets one counting-kernel launch with events when timing is on.
cudaError_t timer_begin(Workspace* w);
cudaError_t timer_end(Workspace* w);

// Selects the stream of this call and resets the per-call accounting.
void begin_call(Workspace* w, const episdet_options& o);

// One search; the caller holds w->mu and has validated the options.
episdet_status search_locked(Workspace* w, const episdet_dataset* data, const episdet_options& o,
                             episdet_result* result);

void reset_result(episdet_result* result);
episdet_status search_staged(Workspace* w, DevData& D, const episdet_options& o, bool simt, uint64_t launches,
                             std::chrono::steady_clock::time_point t0, episdet_result* result);

// What every label of a label-mode permutation batch shares: the cohort's
// planes, their sample-major transpose, its genotype counts [3][M] and its pair
// totals, all in lane 0's workspace.
struct LabelCohort {
    const uint32_t* planes;
    int M, n, W;
    const uint32_t* tt;
    const int* marg;
    const float4* tot;
};
// Fills tt, marg and tot on lane 0 (tensor.cu); EPISDET_ERR_INVALID_INPUT if
// `validate` and the genotype planes of a sample overlap.
episdet_status tensor_label_cohort(Workspace* w, LabelCohort* c, bool validate);
// Class masks, marginals and case operand rows of one label (device words) of
// nc cases, on w->st; D describes the two classes afterwards (tensor.cu).
episdet_status tensor_label_rows(Workspace* w, const LabelCohort& c, const uint32_t* d_label, int nc, DevData* D,
                                 uint64_t* launches);

// Label-free AND cells of every pair of one plane set (tensor.cu), for the
// label-mode 2-way permutation search.
episdet_status tensor_pair_totals(Workspace* w, const uint32_t* d_planes, int M, int n, float4* out);

// Sets the tensor engine's kernel attributes on the current device.
episdet_status tensor_init_attributes();

// Tensor-core engine (tensor.cu).  Fills S with the per-CTA candidate lists.
episdet_status run_tensor(Workspace* w, DevData& D, const ScoreTables& T, const episdet_options& o, int fb, int fe,
                          Slots* S, uint64_t* launches, bool progress);

}  // namespace episdet

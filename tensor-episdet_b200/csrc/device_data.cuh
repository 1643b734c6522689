// device_data.cuh -- the resident per-search device state shared by all engines.
#pragma once
#include <cstdint>
#include "common.cuh"

namespace episdet {

// Class 0 = cases, class 1 = controls (the reference's two .bin arrays).
struct DevData {
    const uint32_t* bits[2];  // [M][2][W[c]] packed planes, reference layout
    int W[2];                 // words per plane row
    int n[2];                 // samples per class
    int M;                    // SNPs
    const int* marg[2];       // [3][M] genotype counts (g2 = n - g0 - g1)
    // Label mode: both classes are columns of one plane set (bits[0] = bits[1],
    // W[0] = W[1]), class c the samples of mask[c] [W]; null otherwise.
    const uint32_t* mask[2];
    const uint4* pair4[2];    // [M][M] AND cells (00,01,10,11) of SNP pair (a<b); 3-way SIMT engine only
};

// Search slot lists: one persistent candidate list per CTA, kept in global
// memory between launches of the same search.
struct Slots {
    Cand* lists;     // [nslots][ld]; SIMT engine: ld = k, sorted
    int ld;
    Cand* thr;       // [nslots] tensor engine: each list's k-th best entry at its last compaction
    int* counts;     // [nslots]
    int nslots;
    int k;
    // The smallest k-th best key any CTA has held in this search (0xFFFFFFFF
    // until one held k candidates): a set whose key is larger has k better
    // sets and cannot be in the search's top k.
    uint32_t* gkey;
    // Tensor engine: descending keys level[0 .. kLevels) below the first
    // threshold (0 = none) and, from level_count, how many scored sets had a
    // key in (level[j + 1], level[j]]: once k sets are at or below level[j],
    // that is the search-wide key.
    uint32_t* level;
    int* level_count;
};
constexpr int kLevels = 16;

// Codes of the tensor engine's error word; 1 to 7 are waits that gave up and
// refused launches (count_kernel.cuh).
constexpr int kErrLabelChanged = 8;  // a label is not the one its cases were counted from
constexpr int kErrPlanes = 9;        // overlapping planes: a first SNP keeps more samples than its rows hold

__device__ __forceinline__ void load_marg3(const int* m, int M, int snp, int out[3]) {
    out[0] = __ldg(m + snp);
    out[1] = __ldg(m + M + snp);
    out[2] = __ldg(m + 2 * M + snp);
}

}  // namespace episdet

// ism_moment.cuh -- launch descriptors of the fractional-delay moment kernel (ism_moment.cu).
#pragma once

#include <vector>

#include "gpurir_internal.cuh"

namespace gpurir {

constexpr int kMPairs = 7;                // (even, odd) pairs of Chebyshev moments per cell
constexpr int kMBasis = 6;                // pairs of the filter's basis
constexpr double kMomFar = 12.6;          // taps beyond this many samples use basis pairs 0 and 1
constexpr double kMomNear = 4.6;          // taps beyond this one pairs 0 to 2
constexpr int kMomMinTw = 48;             // window lengths the moment path is used for
constexpr int kMomMaxTw = 400;
constexpr int kMomCells = 768;            // most cells of a segment
constexpr int kMomLarge = 384, kMomSmall = 256;   // threads of a block: two per SM, three per SM
constexpr int kMomSmallCells = 624;               // most cells of a segment with the latter
constexpr int kMomTabSmem = 256;           // per-axis entries of a launch held in shared memory
constexpr int kMomRuns = 18;               // three per pair

// Quads (groups of four cell taps) of one basis pair.
struct MomRun {
    int pair, first, quads;
};

// Basis and filter of one window length (moment_basis).
struct MomBasis {
    int tw = 0, lead = 0;                 // window; first sample of an output's first cell is `lead` before it
    int taps = 0, quads = 0;              // cells that reach an output, in groups of four
    float2 S[kMBasis][kMPairs];           // moments -> basis
    MomRun run[kMomRuns];
    int n_runs = 0, n_quads = 0;          // over all runs
    unsigned char cut[2][2][kMomLarge / 32 + 1];   // large, small blocks: the warps' ranges of quads, for one tile and two
    std::vector<float2> coef;             // 8 n_quads: per quad, tap by tap, two output phases
};

struct MomLaunch {
    const RoomDesc *rooms;
    const IsmItem *items;             // i_lo, i_hi: this item's share of the image rows (rows i_lo mod i_hi)
    int n_items;
    const float *pos_src, *pos_rcv, *orv_src, *orv_rcv;
    float *out, *partial;
    int *work_counter, *status;
    float4 *axis_tab;                 // per block: two tables of axis_cap entries
    int axis_cap;
    int T;                            // longest segment
    int win;                          // shortest last segment of an item (holds the envelope window)
    int lead, taps, quads;            // as in MomBasis
    const float2 *coef;
    MomRun run[kMomRuns];
    int n_quads;
    unsigned char cut[2][kMomLarge / 32 + 1];
    float2 S[kMBasis][kMPairs];
    // diffuse tail of the RIRs whose last segment is one item (TailArgs)
    uint64_t seed, offset;
    const uint64_t *offset_ptr;
    int noise_kind;
    float *env_out;
    int fuse_tail;
    const unsigned char *tail_pre;
};

const MomBasis &moment_basis_cached(int tw);
int moment_cells(int T, const MomBasis &B);
size_t moment_smem_bytes(int threads, int axis_cap, const MomBasis &B);
int moment_blocks_per_sm(int threads, size_t smem);
cudaError_t moment_launch(const MomLaunch &p, int threads, size_t smem, int grid, cudaStream_t st);

}  // namespace gpurir

// chem_launch.h -- kernel argument blocks and launchers (internal to the library).
#pragma once
#include <cuda_runtime.h>

namespace gdtk {

enum { CHEM_FLAG_UPDATE_THERMO = 1, CHEM_FLAG_RETRY = 2, CHEM_FLAG_REFERENCE_ORDER = 4 };

// All pointers are device pointers.  Mass fractions are species-major: massf[isp * ncell + cell].
struct ChemUpdateArgs {
    const int* mech_i;
    const double* mech_d;
    int n_mech_i, n_mech_d;
    int ncell;
    const double* rho;
    const double* u;
    double* T;
    double* p;
    double* massf;
    double* dt_chem;
    int* status;              // may be null
    double t_interval;
    double T_frozen;
    int flags;
    unsigned* counter;        // work counter, zero at launch
    const int* order;         // cell of each work index, or null
    int* cell_counters;       // optional [6][ncell]: step attempts, rhs, rate-constant evals, Newton
                              // iterations, rejected attempts, initial step-size estimates
    unsigned long long* totals;   // optional [6], same quantities summed
};

struct GasServiceArgs {
    const int* mech_i;
    const double* mech_d;
    int n_mech_i, n_mech_d;
    int nsp_hint, nr_hint, neff_hint;
    int ncell;
    int mode;
    int clip;
    double* rho;
    double* u;
    double* T;
    double* p;
    const double* massf;
    double* out1;
    double* out2;
    int* status;
    double* gscratch;   // set by the launcher when a thread's vectors do not fit in shared memory
};

struct LaunchInfo {
    int grid, block, smem, blocks_per_sm;
};

int chem_scratch_doubles(int nsp, int nr, int neff, int method);
cudaError_t launch_chem_update(const ChemUpdateArgs& a, int method, int scratch_doubles, int sm_count,
                               cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_gas_service(const GasServiceArgs& a, int sm_count, cudaStream_t stream);
// One, two or four warps per cell (mechanisms too large for the thread-per-cell kernels): the reference-order update
// with species and reactions over the lanes.  Its tables (built by the host from the packed mechanism, one set for each
// number of warps):
//   ints [0, n_smem_ints), staged in shared memory by every block:
//     [4 k]              reaction at position k: up to four reactant and four product factors, 16 bits each, species |
//                        coeff << 8; the reactions are sorted by their numbers of factors and third bodies
//     [off_rxm + k]      efficiency list of its third body + 1, or 0; with RX_LONG (more factors, or larger coefficients)
//                        its number among the long reactions << 16 as well
//     [off_M + 2 i]      molar mass of species i (a double)
//     [off_lane + l]     first gather task of lane l (one entry more than lanes)
//     [off_task + t]     task t: target | number of entries << 16.  Targets: q of each species, L of each, partial sums.
//                        A species' q or L of more than a 128th of all entries is split into parts, the later ones
//                        partial sums; the tasks are dealt to the lanes, longest first
//     [off_ent]          16-bit entries [k][lane], a lane's tasks one after the other: index | shift << 13, adding element
//                        `index` of w_f[nr], w_b[nr] (end to end) times 2^shift.  Ascending reaction order
//     [off_comb + 2 k]   split task k: target | first partial sum << 16, and their number
//     [off_eff + 2 (s nsp + i)]   efficiency of species i in list s (doubles); read from global memory if they lie past
//                        n_smem_ints
//   ints read from global memory:
//     [off_perm + k]     the reaction at position k
//     [off_lstart + 3 j] long reaction j: its first term, its first product term, its end
//     [off_lterms + k]   term: species | coeff << 8
struct WarpTables {
    const int* gi;
    int n_smem_ints, npart, ncomb;
    int off_rxm, off_M, off_lane, off_task, off_ent, off_comb, off_eff, off_perm, off_lstart, off_lterms;
};
constexpr int RX_LONG = 1 << 30;
constexpr int WARP_VARIANTS = 3;   // 1, 2, 4 warps per cell
// Shared-memory doubles of one cell's vectors.
int chem_warp_doubles(int nsp, int nr, int neff, int method, int npart);
// Cells that are resident at once in a batch of ncell (0: the mechanism does not fit).  width: the larger of the mechanism's
// numbers of species and reactions.
int chem_warp_resident(int ncell, int width, int method, const WarpTables* tabs, int warp_doubles, int sm_count);
// A cost key of each cell, for launch_bucket_order: about proportional to its steps.
cudaError_t launch_chem_warp_cost(const ChemUpdateArgs& a, int method, const WarpTables* tabs, int warp_doubles,
                                  int sm_count, float* key, cudaStream_t stream);
cudaError_t launch_chem_update_warp(const ChemUpdateArgs& a, int width, int method, const WarpTables* tabs, int warp_doubles,
                                    int sm_count, cudaStream_t stream, LaunchInfo* info);
// Cost buckets of the longest-first ordering: launch_bucket_order's hist scratch holds this many ints.
constexpr int ORDER_BUCKETS = 256;

// Counting sort of n cells by cost key (descending) into order[n]; hist is ORDER_BUCKETS ints of scratch.
cudaError_t launch_bucket_order(const float* key, int n, int* order, int* hist, int sm_count, cudaStream_t stream);

}  // namespace gdtk

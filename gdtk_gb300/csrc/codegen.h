// codegen.h -- mechanism-specialised kernels: source generation, NVRTC compilation, launch.
#pragma once
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>
#include <vector>

#include "mechanism.h"

namespace gdtk {

// Host mirrors of gdtk_fast::CellBlock / FastArgs (chem_fast.cuh); the layouts must agree.
enum { FAST_MAX_BLOCKS = 128 };

struct CellBlock {
    int ncell;
    int first;
    double t_interval;
    const double* rho;
    const double* u;
    double* T;
    double* p;
    double* massf;
    double* dt_chem;
    int* status;
};

struct FastArgs {
    const double* thermo;
    const uint64_t* exp_table;
    int nblocks;
    int total;
    int flags;
    int refill_chunk;   // visit positions a warp reserves per atomic (<= 1: exactly the lanes that need a cell)
    double T_frozen;
    unsigned* counter;
    int* cell_counters;
    unsigned long long* totals;
    const int* order;
    unsigned long long* lane_stats;
    CellBlock blocks[FAST_MAX_BLOCKS];
};

// Shared memory of the kernel with a group of lanes per cell (chem_group.cuh), in doubles; 0: not built.
struct GroupShape {
    int table_doubles = 0;   // of a block
    int cell_doubles = 0;    // of a cell
};

struct FastKernel {
    void* module = nullptr;     // CUmodule
    void* function = nullptr;   // CUfunction
    void* cost_function = nullptr;   // CUfunction of the cost pre-pass
    void* source_function = nullptr; // CUfunction of the source terms
    int block = 0;              // threads per block the kernel was compiled for
    int min_blocks = 1;
    int method = 0;
    int per_thread_doubles = 0;
    int table_doubles = 0;
    int blocks_per_sm = 0;      // occupancy at full block size
    void* group_function = nullptr;  // CUfunction of chem_group.cuh, null where it does not take the mechanism
    GroupShape group;
    int group_warps[4] = {0, 0, 0, 0};   // warps of an SM with 4, 8, 16, 32 lanes per cell
    double* d_thermo = nullptr;
    uint64_t* d_exp = nullptr;
    std::string log;            // NVRTC/ptxas log
    std::string source;
    ~FastKernel();
};

// No mechanism-specialised kernel can be built for the mechanism, whatever the state of the machine.
struct NoFastKernel : std::runtime_error {
    using std::runtime_error::runtime_error;
};
// Thermo table of chem_fast.cuh (120 doubles per species).
std::vector<double> fast_thermo_table(const GasModelHost& gm);
// CUDA source of the generated prologue + kernel for one mechanism.
std::string generate_fast_source(const GasModelHost& gm, const MechanismHost& mh, int block, int min_blocks,
                                 GroupShape* group_shape = nullptr);
// Compiles the generated source for compute capability major.minor without loading it
// (no GPU needed); returns the NVRTC/ptxas log, throws on a compilation error.
std::string compile_fast_check(const GasModelHost& gm, const MechanismHost& mh, int major, int minor);
// Compiles (or fetches from the in-process / on-disk cache) and loads the fast kernel.
// block/min_blocks <= 0: chosen from the shared-memory budget.
FastKernel* build_fast_kernel(const GasModelHost& gm, const MechanismHost& mh, int block = 0, int min_blocks = 0);
// Launches it; `info` receives the launch shape.
cudaError_t launch_fast(FastKernel& k, FastArgs& a, int sm_count, cudaStream_t stream, int* grid_out, int* block_out,
                        int* smem_out);
// Lanes per cell that suit a batch (4, 8, 16 or 32), or 0 for the one-thread-per-cell kernel.
int group_lanes(const FastKernel& k, long long total, int sm_count);
// Launches the kernel with a group of `lanes` lanes per cell.
cudaError_t launch_group(FastKernel& k, FastArgs& a, int lanes, int sm_count, cudaStream_t stream, int* grid_out,
                         int* block_out, int* smem_out);
// Species source terms of n cells.
cudaError_t launch_source(FastKernel& k, int n, const double* rho, const double* T, const double* massf, double* source,
                          int* status, int sm_count, cudaStream_t stream);
// Longest-first visit order: cost pre-pass into key[total], then a bucket sort into order[total]
// (hist: 257 ints of scratch).  All on `stream`.
cudaError_t launch_order(FastKernel& k, FastArgs& a, int sm_count, float* key, int* order, int* hist,
                         cudaStream_t stream);

}  // namespace gdtk

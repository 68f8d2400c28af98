// Kernel declarations shared by the step orchestration (driver.cu) and the kernel files.
#pragma once

#include "device.cuh"

namespace mdelast {

// The kernels of a step are launched as a chain of programmatic dependents: each starts (its
// blocks resident, its parameters read) while the one before it drains, and waits in
// chain_begin() until that one has completed and its writes are visible. chain_begin() comes
// before every other access to memory and lets the next kernel of the chain do the same; a
// kernel launched with launch_chain must call it first. It costs nothing in a plain launch.
//
// A grid of more than kChainBlocks blocks (4 per SM) is launched plainly: its first blocks would
// start on SMs that still hold the previous kernel, with the split of L1 and shared memory that one
// asked for. One 500-atom cell: 0.063 ms per step plain, 0.0505 chained.
constexpr unsigned kChainBlocks = 148 * 4;
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}
template <typename... P, typename... V>
inline cudaError_t launch_chain_up_to(unsigned blocks, void (*kernel)(P...), dim3 grid, dim3 block,
                                      size_t smem, cudaStream_t s, V const &...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = grid.x * grid.y <= blocks ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... V>
inline cudaError_t launch_chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                                cudaStream_t s, V const &...args) {
    return launch_chain_up_to(kChainBlocks, kernel, grid, block, smem, s, args...);
}

// A pair pass with tpa lanes per atom is bound by the L1 and by its longest SM, and loses more to that
// split and to blocks crowded onto the SMs that were free first than a launch costs, unless it is
// latency alone: a warp per atom, or up to a block per SM of 16 lanes. Steps in ms, passes chained up
// to 592 blocks / by this rule:
//   atoms     FP64              mixed             FP64, 1 lane      mixed, 1 lane
//   500       0.0381 / 0.0381   0.0379 / 0.0379   -                 -
//   4,000     0.0625 / 0.0605   0.0505 / 0.0481   0.160 / 0.161     0.098 / 0.097
//   8,788     0.0946 / 0.0894   0.0721 / 0.0684   -                 -
//   13,500    0.0961 / 0.0959   0.0811 / 0.0812   0.226 / 0.178     0.153 / 0.115
//   32,000    0.164 / 0.164     0.109 / 0.108     0.258 / 0.192     0.180 / 0.127
// (64 x 2,048 atoms, mixed: 0.440 chained throughout, 0.404 plain.) With 4 or 8 lanes, 2,048 atoms
// mixed 0.0517 / 0.0498 and 0.0453 / 0.0434. A warp per atom, 2 x 500 atoms FP64 (256
// blocks): 0.0401 chained, 0.0404 to 0.0415 not; 1,372 atoms 0.0426 both.
constexpr unsigned kChainPassBlocks = 148;
template <typename... P, typename... V>
inline cudaError_t launch_pass(int tpa, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t s, V const &...args) {
    unsigned const most = tpa == 32 ? kChainBlocks : (tpa == 16 ? kChainPassBlocks : 0);
    return launch_chain_up_to(most, kernel, grid, block, smem, s, args...);
}

// scalar-kernel modes
enum PostMode : int { POST_INIT = 0, POST_STEP = 1 };

__global__ void k_cell_bin(AtomsView A);
__global__ void k_cell_sort(AtomsView A);
__global__ void k_nbr_build(AtomsView A, int cells_done);
__global__ void k_nbr_cells(AtomsView A);
size_t nbr_cells_smem(int cell_cap); // dynamic shared memory of k_nbr_cells
constexpr int kCellSortWarps = 8;      // half cells per k_cell_sort block (one warp each)
constexpr int kNbrCellsThreads = 256;   // threads of a k_nbr_cells block (one 2x2x2 half-cell group)
constexpr size_t kNbrCellsStaticSmem = 4 * 1024; // bound on k_nbr_cells' static shared memory
// launchers of the templated pair kernels (defined beside them); tpa = lanes per atom,
// one of 1, 4, 8, 16 (valid_tpa: what callers may name) or 32
bool valid_tpa(int tpa);
void launch_density(bool obs, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                    TablesView const &T);
void launch_force(bool obs, bool kick, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                  TablesView const &T);
// the same passes with FP32 pair math (mixed precision)
void launch_density_mx(bool obs, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                       TablesView const &T);
void launch_force_mx(bool obs, bool kick, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                     TablesView const &T);
// the mixed force pass with the quintic tables staged in shared memory (T.st_n > 0; tpa 4, 8,
// 16 or 32; blocks of kStagedBlock threads); prepare_force_mx_staged raises the kernels'
// dynamic shared-memory limit (to the staging budget) before any launch or capture
constexpr int kStagedBlock = 512;
void launch_force_mx_staged(bool obs, bool kick, int tpa, int grid, cudaStream_t s,
                            AtomsView const &A, TablesView const &T);
cudaError_t prepare_force_mx_staged(int smem_bytes);
__global__ void k_posf(AtomsView A);
__global__ void k_kick_drift(AtomsView A, TablesView T);
__global__ void k_pre(AtomsView A);
__global__ void k_reduce(AtomsView A);
__global__ void k_post(AtomsView A, int mode, int obs, mdelast_observables *host);
__global__ void k_samples_reset(AtomsView A, int what);
// the pair-list refresh, with sublist_smem(maxn) bytes of dynamic shared memory
void launch_sublist(int grid, size_t smem, cudaStream_t s, AtomsView const &A);
// k_sublist's dynamic shared memory for rows of capacity maxn (0: rows keep list order)
constexpr size_t kSublistSortMax = 150 * 1024;
__host__ __device__ size_t sublist_smem(int maxn);
__global__ void k_sub_invalidate(AtomsView A);
__global__ void k_readout(AtomsView A, TablesView T, int r, int field, int first, int n, double *out,
                          const double *pos0, int stepped);
__global__ void k_half_list_counts(AtomsView A, int r, int *counts);
__global__ void k_half_list_fill(AtomsView A, int r, const int *point, int *out);
__global__ void k_status_and(AtomsView A, unsigned mask);
__global__ void k_clear_counts(AtomsView A);
__global__ void k_table_eval(TablesView T, int which, int s, const double *x, int n,
                             double *out);

} // namespace mdelast

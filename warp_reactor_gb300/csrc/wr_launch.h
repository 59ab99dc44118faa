// wr_launch.h -- host-side launchers of the advance kernel, one translation unit
// per math policy (the advance kernel is the large one; compiling the policies in
// parallel keeps the build short).
#pragma once

#include <cuda_runtime.h>

#include "wr_kernels.cuh"

namespace wr {

constexpr int kPrepareThreads = 256;

// Advance kernel configurations, selected per context (wr_set_advance_variant):
//   0  128 threads x 1 block per SM, iteration matrix in shared memory (225 KiB)
//   1  128 threads x 2 blocks per SM, iteration matrix in a global lane array
//   2  256 threads x 1 block per SM, iteration matrix in a global lane array
//   3  precision form: 256 threads x 1 block per SM, FP32 factorisation in shared
//      memory (900 B per lane) with one FP64 residual refinement per stage solve
//   4  384 threads x 1 block per SM (at most 168 registers per thread: more spills,
//      twelve warps per SM to hide them)
//   5  cooperative advance (wr_coop.cuh), 8 lanes per cell
//   6  cooperative advance, 16 lanes per cell
//   7  cooperative advance, 32 lanes per cell
//   (cooperative advance: one block per SM, as many warps as the cells' slot
//   arrays fit in its shared memory, kWarps of generated/coop_prog_g<G>.h)
constexpr int kAdvanceVariants = 8;
constexpr int kPrecisionVariant = 3;
constexpr int kDefaultVariant = 6;   // 16 lanes per cell: the most cells per second
constexpr int kLatencyVariant = 7;   // 32 lanes per cell: the shortest attempt
// Cells per SM up to which a context takes 32 lanes per cell.  A block holds 16 cells
// at 32 lanes and 32 at 16: while every cell has its warp at once, an outer step lasts
// as long as its longest burn, and a 32-lane attempt is shorter (one outer step on GB300,
// CUDA math: 512 cells 2.01 ms at 32 lanes, 2.24 ms at 16; 2,432 cells, 16 per SM, 2.52
// and 3.21 ms); beyond that the 16-lane shape's rate decides (3,000 cells 3.43 and 3.34 ms,
// 20,011 cells 16.3 and 12.4 ms).
constexpr int kLatencyCellsPerSm = 16;
struct AdvanceShape {
    int threads;    // lane-per-cell shapes (0 for the cooperative advance)
    int blocks_per_sm;
    bool smem_matrix;
    int precision;  // 0 FP64 factorisation, 1 FP32 factorisation + FP64 refinement
    int coop_lanes; // lanes per cell of the cooperative advance (0: one lane per cell)
};
constexpr AdvanceShape kAdvanceShapes[kAdvanceVariants] = {
    {128, 1, true, 0, 0},  {128, 2, false, 0, 0}, {256, 1, false, 0, 0},  {256, 1, true, 1, 0},
    {384, 1, false, 0, 0}, {0, 1, false, 0, 8}, {0, 1, false, 0, 16}, {0, 1, false, 0, 32}};
constexpr int default_variant(int cells, int sms) {
    return cells <= sms * kLatencyCellsPerSm ? kLatencyVariant : kDefaultVariant;
}
constexpr bool is_coop(int variant) { return kAdvanceShapes[variant].coop_lanes != 0; }

constexpr size_t advance_smem_bytes(int variant) {
    return kAdvanceShapes[variant].smem_matrix && !is_coop(variant)
               ? static_cast<size_t>(NEQ) * NEQ * kAdvanceShapes[variant].threads *
                     (kAdvanceShapes[variant].precision ? sizeof(float) : sizeof(double))
               : 0;
}

cudaError_t launch_advance_portable(int variant, int blocks, cudaStream_t stream, DevState s, StepCtl* ctl,
                                    double* jbackup, double* ebuf);
cudaError_t launch_advance_cuda(int variant, int blocks, cudaStream_t stream, DevState s, StepCtl* ctl,
                                double* jbackup, double* ebuf);
cudaError_t configure_advance_portable();
// gridwide-structured-cta32 policy (wr_coop_cta32.cuh): a tile of 32 cells on a cluster
// of `cluster` SMs at `lanes` lanes per cell.  A trial's latency sets the time while
// there are SMs to spare, so a tile spreads over four SMs (8 cells each) or two as long
// as the device runs all clusters at once; beyond that one SM per tile at 16 lanes per
// cell.  fit4 and fit2 are the clusters that fit (cta32_clusters): the blocks of one lie
// in one GPC, so of 152 SMs 36 clusters of four, not 38 (one outer step of like tiles:
// up to 36 tiles 8.6 ms, 37 and 38 tiles 16.9 ms in two waves of them, 11.9 ms on
// clusters of two, which take up to 76; from 77 on 15.2 ms on one SM per tile).
struct Cta32Shape {
    int lanes, cluster;
};
constexpr Cta32Shape cta32_shape(int tiles, int fit4, int fit2) {
    return tiles <= fit4 ? Cta32Shape{32, 4} : tiles <= fit2 ? Cta32Shape{32, 2} : Cta32Shape{16, 1};
}
// clusters of 4 or 2 blocks of the 32-lane kernel that the current device runs at once
cudaError_t cta32_clusters(int math_cuda, int cluster, int* fit);
cudaError_t launch_advance_cta32_16(int math_cuda, int cluster, int tiles, int sms, cudaStream_t stream, DevState s,
                                    StepCtl* ctl);
cudaError_t launch_advance_cta32_32(int math_cuda, int cluster, int tiles, int sms, cudaStream_t stream, DevState s,
                                    StepCtl* ctl);
cudaError_t configure_advance_cuda();
// cooperative advance (wr_adv_coop<G>.cu): G lanes per cell, one block per SM
cudaError_t configure_advance_coop8();
cudaError_t configure_advance_coop16();
cudaError_t configure_advance_coop32();
cudaError_t launch_advance_coop8(int math_cuda, int blocks, cudaStream_t stream, DevState s, StepCtl* ctl,
                                  unsigned long long* phases);
cudaError_t launch_advance_coop16(int math_cuda, int blocks, cudaStream_t stream, DevState s, StepCtl* ctl,
                                  unsigned long long* phases);
cudaError_t launch_advance_coop32(int math_cuda, int blocks, cudaStream_t stream, DevState s, StepCtl* ctl,
                                  unsigned long long* phases);
// around the cooperative advance (wr_capi.cu): the queue with the advance's prologue,
// and the commit of the cells it burned
cudaError_t launch_order_preburn(cudaStream_t stream, DevState s, StepCtl* ctl);
cudaError_t launch_commit(cudaStream_t stream, DevState s, StepCtl* ctl);
// kernels launched outside wr_capi.cu, for wr_kernel_launch_count
void count_launches(int n);
// diagnostics of the cooperative programs and LU on device buffers (wr_diag.cu)
cudaError_t diag_coop_network8(int math_cuda, int n, const double* y, double* J, double* f, double* f2);
cudaError_t diag_coop_network16(int math_cuda, int n, const double* y, double* J, double* f, double* f2);
cudaError_t diag_coop_network32(int math_cuda, int n, const double* y, double* J, double* f, double* f2);
cudaError_t diag_coop_lu8(int n, const double* A, const double* b, double* LU, int* ipvt, int* info, double* x);
cudaError_t diag_coop_lu16(int n, const double* A, const double* b, double* LU, int* ipvt, int* info, double* x);
cudaError_t diag_coop_lu32(int n, const double* A, const double* b, double* LU, int* ipvt, int* info, double* x);

}  // namespace wr

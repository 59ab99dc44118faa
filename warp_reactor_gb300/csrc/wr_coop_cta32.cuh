// wr_coop_cta32.cuh -- advance kernel of the gridwide-structured-cta32 policy.
//
// The reference's other GPU policy (advance_collapse_gridwide_structured_kernel,
// structured_cuda.cuh:393-782; selected by PRIMORDIAL_ROS2S_CUDA_STRUCTURED,
// reproducer.cpp:7845-7916): the grid is cut into tiles of 32 consecutive cells and
// each tile advances its participating cells with ONE ROS2S controller -- a common
// step h, the tile error = maximum over its participating cells of their error
// norms (a non-finite norm counts as DBL_MAX), the Jacobian kept across rejected
// trials, the common
// final-step truncation and the commit of every participating cell on success.  The
// prepare kernel and the grid minimum are the gridwide-independent ones.
//
// GB300 mapping: the attempts are the cooperative advance's (wr_coop.cuh), G lanes per
// cell, and a tile is one thread block, or a cluster of CL blocks on as many SMs with
// 32 / CL cells each.  The cells' error norms meet in shared memory (read across the
// cluster); one warp of each block runs the tile's controller on all 32 and hands the
// next step to its block, so the blocks of a cluster decide alike without exchanging
// anything else.  A tile's trials are serial, so with few tiles the time is a trial's
// latency: 32 cells on one SM share its FP64 pipes, 8 cells on each of four SMs at 32
// lanes per cell run a trial in half the time (the choice is cta32_shape's).  Measured
// on GB300, 1,000 cells over the last eight outer steps of a collapse: 87 ms; one lane
// per cell and one warp per tile, as this kernel was before, 1,159 ms.
#pragma once

#include <cooperative_groups.h>

#include "wr_coop.cuh"

namespace wr {

constexpr int kTileCells = 32;

template <class M>
__device__ __forceinline__ double cbrt_nonnegative(double v) {  // structured_cuda.cuh:88-93
    if (v == 0.0) return 0.0;
    return coop::StepMath<M>::exp(ddiv(coop::StepMath<M>::log(v), 3.0));
}

// one block's part of a tile: its cells' error norms (-1: singular matrix; two sets, so
// that a block may go on while another still reads), its participating cells, and what
// its controller decided
template <int CELLS>
struct TileCtl {
    double err[2][CELLS];
    double h;
    unsigned int part;
    int run, accept, status, tile;
};

template <class M, int G, int CL, class Tab>
__global__ void __launch_bounds__(kTileCells / CL * G, 1) k_advance_cta32(DevState s, StepCtl* ctl) {
    using namespace coop;
    namespace cg = cooperative_groups;
    constexpr int CELLS = kTileCells / CL;
    constexpr int K = (NEQ + G - 1) / G;
    constexpr int SLOTS = 32 / G;
    extern __shared__ uint64_t sm[];
    __shared__ TileCtl<CELLS> tc;
    StepCtl* c = ctl;
    if (c->stop) return;  // set before this launch: uniform over the grid
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = lane / G, gl = lane % G;
    const int mine = warp * SLOTS + slot;  // the group's cell of the block's CELLS
    uint64_t* V = sm + static_cast<size_t>(mine) * Tab::kNV;
    init_reserved<M, G, Tab>(V, gl);
    const int n = s.n;
    const int tiles = (n + kTileCells - 1) / kTileCells;
    const int rank = CL > 1 ? static_cast<int>(blockIdx.x) % CL : 0;
    const int cgs = c->cgs;
    const double grid_time = c->grid_time;
    const double dt_grid = c->dt_grid;
    const double next_grid_time = c->next_grid_time;
    auto remote = [&](int r) -> const TileCtl<CELLS>* {
        if constexpr (CL > 1) return cg::this_cluster().map_shared_rank(&tc, r);
        else return &tc;
    };
    auto tile_sync = [&]() {
        if constexpr (CL > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    PhaseClock<false> pc;

    int tile = CL > 1 ? static_cast<int>(blockIdx.x) / CL : 0;
    const int stride = CL > 1 ? static_cast<int>(gridDim.x) / CL : 0;
    while (true) {
        if constexpr (CL == 1) {  // tiles differ in length: the next free one
            if (threadIdx.x == 0) tc.tile = static_cast<int>(atomicAdd(&ctl->queue, 1u));
            __syncthreads();
            tile = tc.tile;
        }
        if (tile >= tiles) break;
        const int first = tile * kTileCells + rank * CELLS;

        // ---- per-cell prologue, structured_cuda.cuh:410-450, one lane per cell
        if (warp == 0) {
            const int cell = first + lane;
            bool part = false;
            if (lane < CELLS && cell < n && s.steps[cell] == cgs) {
                if (s.time[cell] != grid_time) {
                    record_failure(c, WR_BAD_INPUTS);
                } else {
                    double xn[NS];
#pragma unroll
                    for (int k = 0; k < NS; ++k) xn[k] = s.xn[k * n + cell];
                    const double local_dt = collapse_timestep(xn);
                    if (local_dt >= 10.0) {
                        const double old_density = s.driver[cell];
                        const double driver = old_density + ddiv(dt_grid * old_density, ddiv(local_dt, kTffReduc));
                        s.driver[cell] = driver;
                        if (valid_positive(driver) && driver <= kDriverLimit) {
                            const double ratio = ddiv(driver, old_density);
#pragma unroll
                            for (int k = 0; k < NS; ++k) xn[k] *= ratio;
                            s.rho[cell] = s.rho[cell] * ratio;
                            s.e[cell] = eos_e_from_T(xn, s.T[cell]);
#pragma unroll
                            for (int k = 0; k < NS; ++k) s.xn[k * n + cell] = xn[k];
                            part = true;
                        }
                    }
                }
            }
            const unsigned int pm = __ballot_sync(kWarp, part);
            if (lane == 0) tc.part = pm;
        }
        tile_sync();
        int count = 0;
#pragma unroll
        for (int r = 0; r < CL; ++r) count += __popc(remote(r)->part);
        if (count != 0) {
            const int cell = first + mine;
            const bool have = (tc.part >> mine) & 1u;
            const unsigned holders = __ballot_sync(kWarp, have);
            // a group without a cell follows one of its warp that has one
            const int from = holders ? (__ffs(holders) - 1) / G * G + gl : lane;
            double y[K];
#pragma unroll
            for (int t = 0; t < K; ++t) {
                const int q = gl + t * G;
                y[t] = !have ? 0.0 : q < NS ? s.xn[q * n + cell] : (q == NS ? s.e[cell] : 0.0);
                const double o = __shfl_sync(kWarp, y[t], from);
                y[t] = have ? y[t] : o;
            }
            int regime = have ? regime_of<Tab>(bits(s.T[cell])) : 0;
            const int og = __shfl_sync(kWarp, regime, from);
            regime = have ? regime : og;

            // ---- the tile's controller, structured_cuda.cuh:468-733, in every block's
            // first warp (all lanes alike)
            double h = dt_grid, x = 0.0, hacc = 0.0, erracc = 1.0;
            bool reject = false, jac_valid = false, final_trial = false;
            int nsing = 0, n_step = 0, n_accept = 0, n_jac = 0, n_rej = 0;
            int status = WR_SUCCESS;
            auto next_trial = [&]() {  // the checks before a trial; tells the block
                bool run = false;
                if (status == WR_SUCCESS && !(x >= dt_grid)) {
                    if (n_step > kMaxSteps) {
                        status = WR_TOO_MANY_STEPS;
                    } else if (0.1 * ::fabs(h) <= ::fabs(x) * kUround) {
                        status = WR_DT_UNDERFLOW;
                    } else {
                        final_trial = false;
                        if (x + h * 1.0001 >= dt_grid) {
                            h = dt_grid - x;
                            final_trial = true;
                        }
                        run = true;
                    }
                }
                if (lane == 0) {
                    tc.h = h;
                    tc.run = run ? 1 : 0;
                    tc.status = status;
                }
            };
            if (warp == 0) next_trial();
            __syncthreads();
            int set = 0;
            bool again = false;  // the last trial was not accepted: the same states
            Kept<G, K> kept;
            while (tc.run) {
                double ynew[K], err = 0.0;
                int info = 0;
                if (holders) info = ros2s_attempt<M, G, Tab, true, K>(V, y, tc.h, regime, gl, pc, again, kept, ynew, err);
                if (gl == 0) tc.err[set][mine] = !have ? 0.0 : info != 0 ? -1.0 : isfinite(err) ? err : DBL_MAX;
                tile_sync();
                if (warp == 0) {
                    double ev = remote(lane / CELLS)->err[set][lane % CELLS];
                    if (!jac_valid) n_jac += 1;
                    jac_valid = true;
                    bool accept = false;
                    if (__any_sync(kWarp, ev < 0.0)) {
                        ++nsing;
                        if (nsing >= 5) {
                            status = WR_LU_DECOMPOSITION_ERROR;
                        } else {
                            h = h * 0.5;
                            reject = true;
                        }
                    } else {
#pragma unroll
                        for (int off = 16; off > 0; off >>= 1) ev = ::fmax(ev, __shfl_xor_sync(kWarp, ev, off));
                        const double err_tile = ev;
                        ++n_step;
                        double hnew, hgus;
                        step_sizes<32, true>(err_tile, erracc, hacc, h, lane, cbrt_nonnegative<M>, hnew, hgus);
                        accept = err_tile <= 1.0;
                        if (accept) {
                            ++n_accept;
                            if (n_accept > 1) hnew = hgus;
                            hacc = h;
                            erracc = ::fmax(1.0e-2, err_tile);
                            x = final_trial ? dt_grid : x + h;
                            hnew = ::fmin(::fabs(hnew), dt_grid);
                            if (reject) hnew = ::fmin(hnew, ::fabs(h));
                            reject = false;
                            h = hnew;
                            jac_valid = false;
                        } else {
                            if (n_accept >= 1) ++n_rej;
                            reject = true;
                            h = hnew;
                        }
                    }
                    next_trial();
                    if (lane == 0) tc.accept = accept ? 1 : 0;
                }
                __syncthreads();
                if (tc.accept && holders) {
#pragma unroll
                    for (int t = 0; t < K; ++t) y[t] = ynew[t];
                }
                again = tc.accept == 0;
                set ^= 1;
            }

            // ---- commit, structured_cuda.cuh:737-778
            if (tc.status == WR_SUCCESS) {
                if (have) {
#pragma unroll
                    for (int t = 0; t < K; ++t) {
                        const int q = gl + t * G;
                        if (q < NS) s.xn[q * n + cell] = y[t];
                        else if (q == NS) s.e[cell] = y[t];
                    }
                }
                __syncthreads();
                if (warp == 0 && ((tc.part >> lane) & 1u)) {
                    const int i = first + lane;
                    double xn[NS];
#pragma unroll
                    for (int k = 0; k < NS; ++k) xn[k] = s.xn[k * n + i];
                    renormalize(xn, s.rho[i]);
                    s.T[i] = eos_T_from_e(xn, s.e[i]);
#pragma unroll
                    for (int k = 0; k < NS; ++k) s.xn[k * n + i] = xn[k];
                    s.time[i] = next_grid_time;
                    s.steps[i] = cgs + 1;
                    const uint64_t st[7] = {static_cast<uint64_t>(n_step), static_cast<uint64_t>(3 * n_step),
                                            static_cast<uint64_t>(n_jac), static_cast<uint64_t>(n_step),
                                            static_cast<uint64_t>(3 * n_step), static_cast<uint64_t>(n_accept),
                                            static_cast<uint64_t>(n_rej)};
#pragma unroll
                    for (int k = 0; k < 7; ++k) s.stats[k * n + i] += st[k];
                }
                if (rank == 0 && threadIdx.x == 0) atomicAdd(&c->integrated, count);
            } else if (rank == 0 && threadIdx.x == 0) {
                record_failure(c, status);
            }
        }
        tile_sync();  // the tile's shared words are read: the next tile may write them
        tile += stride;
    }
    // no block of the cluster leaves while another may still read its shared memory:
    // the last tile_sync above
}

}  // namespace wr

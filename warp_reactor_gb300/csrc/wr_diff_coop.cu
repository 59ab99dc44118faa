// wr_diff_coop.cu -- differentiation form: the forward and adjoint kernels (the map
// and its storage are described in wr_diff.cuh).
//
// One warp per cell, in the manner of the cooperative advance (wr_coop.cuh): the
// network's Jacobian, its RHS with multipliers and both vector-Jacobian products are
// generated vector programs (gen/coop_adj.py) on the cell's slot array in shared
// memory, the factorisation and the solves are warp-cooperative, a 15-vector lies
// one component per lane; the per-step scalar pieces (perturbation, equation of state,
// normalisation and their adjoints) run alike in every lane.  Warps take cells from a
// counter: a cell's whole schedule is one piece of work.
//
// What bounds it: a cell is a serial chain of attempts (forward) or steps (adjoint), and
// the workloads have a few thousand cells, so the latency of an attempt decides, and
// how many cells an SM holds at once: 16 slot arrays of the forward programs, 10 or
// more of the adjoint's, which keep most values of the Jacobian's evaluation alive.
// One lane per cell, as these kernels were before, kept 128 warps of divergent lanes
// and local-memory arrays on 152 SMs for 4,096 cells.  Measured on GB300 (forward and
// adjoint of 4,096 cells over four outer steps, and of 64 cells over eight): 163 ms and
// 566 ms before, 47 ms and 50 ms now, with the same bits (at 65,536 cells over four outer
// steps 296 + 892 ms before, 223 + 448 ms now).
#include "generated/coop_diff.h"
#include "wr_coop.cuh"
#include "wr_diff.cuh"

namespace wr {
namespace diff {

namespace {

namespace cd = wr::coop_diff;
using CM = PortableMathCall;

struct Tab {
    static constexpr int kNV = cd::kNV;
    static constexpr int kNR = cd::kNR;
    static constexpr int kNF = cd::kNF;
    static constexpr int kRegimes = cd::kRegimes;
    static constexpr bool kAdjoint = true;
    static __device__ __forceinline__ const uint64_t* vconst() { return cd::kVConst; }
    static __device__ __forceinline__ const ulonglong2* vfun() { return cd::kVFun; }
    static __device__ __forceinline__ const ulonglong2* prog() { return cd::kProg; }
    static __device__ __forceinline__ const uint64_t* lit() { return cd::kLit; }
    static __device__ __forceinline__ uint32_t ctl(int i) { return cd::kCtl[i]; }
    static __device__ __forceinline__ int first(int w) { return cd::kProgStep[w][0]; }
    static __device__ __forceinline__ int steps(int w) { return cd::kProgStep[w][1]; }
    // the vector-Jacobian programs lie on the adjoint's larger slot array: kNV - 1 is one of
    // their ordinary slots
    static __device__ __forceinline__ int sink(int w) { return (w < 2 * kRegimes ? cd::kNV : cd::kNVA) - 1; }
    static __device__ __forceinline__ uint64_t regime(int k, int i) { return cd::kRegimeT[k][i]; }
    static __device__ __forceinline__ const uint16_t* out(int w) { return cd::kOut[w]; }
    static __device__ __forceinline__ const uint16_t* jac(int r) { return cd::kJac[r]; }
};
static_assert(cd::kMult + NP <= cd::kNV && cd::kFbar + NEQ <= cd::kNV, "inputs lie inside the slot array");
static_assert(cd::kNumMult == NP, "rate multiplier count");

constexpr int G = 32;
constexpr int kMaxSmem = 232448;
constexpr int warps_of(int slots) {
    const int w = kMaxSmem / (slots * 8);
    return w < 16 ? w : 16;
}
constexpr int kFwdWarps = warps_of(cd::kNV);
constexpr int kBwdWarps = warps_of(cd::kNVA);
constexpr size_t kFwdSmem = static_cast<size_t>(kFwdWarps) * cd::kNV * 8;
constexpr size_t kBwdSmem = static_cast<size_t>(kBwdWarps) * cd::kNVA * 8;
// scratch of the adjoint between programs: six 15-vectors in the last slots
constexpr int kTmp = cd::kNVA - 6 * 16;
static_assert(kTmp > cd::kFbar + NEQ, "the scratch vectors lie above the inputs");

__device__ __forceinline__ void init_slots(uint64_t* V, const Args& a, int lane) {
    coop::init_reserved<CM, G, Tab>(V, lane);
    for (int r = lane; r < NP; r += G) V[cd::kMult + r] = coop::bits(a.mult[r]);
    __syncwarp();
}

// the next cell of the launch, the same in every lane; a.n when there is none
__device__ __forceinline__ int next_cell(const Args& a, int lane) {
    int i = 0;
    if (lane == 0) i = atomicAdd(a.queue, 1);
    i = __shfl_sync(coop::kWarp, i, 0);
    return i < a.n ? i : a.n;
}

// a 15-vector that every lane holds whole <-> one component per lane
__device__ __forceinline__ double spread(uint64_t* V, const double* y, int lane) {
    __syncwarp();
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) V[coop::kY + k] = coop::bits(y[k]);
    }
    __syncwarp();
    return lane < NEQ ? coop::dbl(V[coop::kY + lane]) : 0.0;
}
__device__ __forceinline__ void collect(uint64_t* V, double yl, double* y, int lane) {
    __syncwarp();
    if (lane < NEQ) V[coop::kY + lane] = coop::bits(yl);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NEQ; ++k) y[k] = coop::dbl(V[coop::kY + k]);
}

// RODAS::integrate with the configure_ros2s settings (:7205-7347, :7582-7590) on the
// warp's cell, appending accepted step sizes to h_out (at most cap_left).  Returns the
// IntegratorResult; *count = accepted steps.
__device__ __noinline__ int burn_record(uint64_t* V, double& yl, double tout, double* h_out, int cap_left, int* count,
                                        int& regime, int lane) {
    const double hmaxn = tout;
    double h = tout;
    if (::fabs(h) <= 10.0 * kUround) h = 1.e-6;
    h = smin(::fabs(h), hmaxn);
    bool reject = false, last = false, fresh = true;
    int nsing = 0, n_step = 0, n_accept = 0;
    double hacc = 0.0, erracc = 1.0, x = 0.0;
    *count = 0;
    PhaseClock<false> pc;
    coop::Kept<G, 1> kept;
#pragma unroll 1
    for (;;) {
        __syncwarp();  // every lane is done with the last attempt's factors and outputs in V
        const bool again = !fresh;  // the same state as the last attempt's
        if (fresh) {
            if (n_step > kMaxSteps) return WR_TOO_MANY_STEPS;
            if (0.1 * ::fabs(h) <= ::fabs(x) * kUround) return WR_DT_UNDERFLOW;
            if (last) return WR_SUCCESS;
            if (x + h * 1.0001 >= tout) {
                h = tout - x;
                last = true;
            }
            fresh = false;
        }
        const double y[1] = {yl};
        double k1[1], k2[1], k3[1], ynew[1], err;
        uint64_t ip;
        const int info = ros2s_stages<CM, G, Tab, 1>(V, y, h, regime, lane, pc, again, kept, ip, k1, k2, k3);
        if (info != 0) {
            nsing += 1;
            if (nsing >= 5) return WR_LU_DECOMPOSITION_ERROR;
            h = h * 0.5;
            reject = true;
            last = false;
            continue;
        }
        ros2s_candidate<G, false, 1>(y, k1, k2, k3, lane, ynew, err);
        n_step += 1;
        double hnew, hgus;
        step_sizes<G, false>(err, erracc, hacc, h, lane, coop::StepMath<CM>::cbrt, hnew, hgus);
        if (err <= 1.0) {
            n_accept += 1;
            if (n_accept > 1) hnew = hgus;
            hacc = h;
            erracc = smax(1.e-2, err);
            if (*count >= cap_left) return WR_TOO_MANY_STEPS;
            if (lane == 0) h_out[*count] = h;
            *count += 1;
            yl = ynew[0];
            x += h;
            if (::fabs(hnew) > hmaxn) hnew = hmaxn;
            if (reject) hnew = smin(::fabs(hnew), ::fabs(h));
            reject = false;
            h = hnew;
            fresh = true;
        } else {
            reject = true;
            last = false;
            h = hnew;
            if (hnew == 0.0) return WR_DT_UNDERFLOW;  // the reject loop's only other exit
        }
    }
}

__global__ void __launch_bounds__(kFwdWarps * 32, 1) k_diff_forward(Args a) {
    extern __shared__ uint64_t sm[];
    const int lane = threadIdx.x & 31;
    uint64_t* V = sm + static_cast<size_t>(threadIdx.x >> 5) * cd::kNV;
    init_slots(V, a, lane);
#pragma unroll 1
    for (int i = next_cell(a, lane); i < a.n; i = next_cell(a, lane)) {
        CellS c;
        {
            const wr_collapse_state& st = a.cells[i];
#pragma unroll
            for (int k = 0; k < NS; ++k) c.xn[k] = a.u ? a.u[15 * i + k] : st.xn[k];
            c.T = a.u ? a.u[15 * i + NS] : st.T;
            c.e = st.e;
            c.rho = st.rho;
            c.driver = st.density_driver;
        }
        double* hrow = a.hbuf + static_cast<size_t>(i) * a.cap;
        int used = 0, status = WR_SUCCESS;
        int regime = coop::regime_of<Tab>(coop::bits(c.T));
        bool live = true;
#pragma unroll 1
        for (int s = 0; s < a.nsteps; ++s) {
            unsigned char kind = 0;
            int cnt = 0;
            if (live) {
                if (lane == 0) save_ckpt(a, s, i, c);
                double dt;
                int k = prepare_part(a, s, i, c, dt);
                if (k == 3) {
                    double y[NEQ];
                    k = advance_part(a.dt_hist[s], dt, c, y);
                    if (k == 3) {
                        double yl = spread(V, y, lane);
                        const int r = burn_record(V, yl, a.dt_hist[s], hrow + used, a.cap - used, &cnt, regime, lane);
                        if (r != WR_SUCCESS) {
                            status = r;
                            live = false;
                        } else {
                            collect(V, yl, y, lane);
                            commit_part(c, y);
                            used += cnt;
                        }
                    }
                }
                if (k < 0) {
                    status = WR_BAD_INPUTS;
                    live = false;
                } else {
                    kind = static_cast<unsigned char>(k);
                    if (k != 3) live = false;
                }
            }
            if (lane == 0) {
                a.kind[static_cast<size_t>(s) * a.n + i] = kind;
                a.counts[static_cast<size_t>(s) * a.n + i] = cnt;
            }
        }
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < NS; ++k) a.q[15 * i + k] = c.xn[k];
            a.q[15 * i + NS] = c.T;
            a.status[i] = status;
        }
    }
}

// ---------------------------------------------------------------- adjoint pieces
// The adjoints below differentiate the mathematical form of each operation (the
// forward values are the exact IEEE sequence).  A stiff step's adjoint cancels ten
// digits and more, so the order of its operations is part of its result: where lanes
// share a sum, they add in index order.

// eos_re: T = e * A / (R mp B), A = sum m x, B = sum x/(gamma-1)
__device__ __forceinline__ void eos_T_adj(const double* x, double e, double Tbar, double* xbar, double& ebar) {
    double A = 0.0, B = 0.0;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        A += mass(n) * x[n];
        B += x[n] * inv_gm1(n);
    }
    const double T = e * A / (kGasConstant * kMp * B);
    ebar += Tbar * A / (kGasConstant * kMp * B);
#pragma unroll
    for (int n = 0; n < NS; ++n) xbar[n] += Tbar * T * (mass(n) / A - inv_gm1(n) / B);
}

// eos_rt: e = R mp T B / A
__device__ __forceinline__ void eos_e_adj(const double* x, double T, double ebar, double* xbar, double& Tbar) {
    double A = 0.0, B = 0.0;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        A += mass(n) * x[n];
        B += x[n] * inv_gm1(n);
    }
    const double e = kGasConstant * kMp * T * B / A;
    Tbar += ebar * kGasConstant * kMp * B / A;
#pragma unroll
    for (int n = 0; n < NS; ++n) xbar[n] += ebar * e * (inv_gm1(n) / B - mass(n) / A);
}

// floor_and_normalize: out = max(x, F) * rho / S, S = sum m max(x, F)
__device__ __forceinline__ void fn_adj(const double* x, double rho, const double* obar, double* xbar, double& rhobar) {
    double xf[NS], S = 0.0, c = 0.0;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        xf[n] = smax(x[n], kFloor);
        S += mass(n) * xf[n];
        c += obar[n] * xf[n];
    }
    rhobar += c / S;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const double g = obar[n] * rho / S - mass(n) * rho * c / (S * S);
        xbar[n] = (x[n] < kFloor) ? 0.0 : g;
    }
}

// renormalize = floor_and_normalize, balance_charge, floor_and_normalize;
// xbar receives (overwrites) the adjoint of x
__device__ __noinline__ void renorm_adj(const double* x, double rho, const double* obar, double* xbar, double& rhobar) {
    double x1[NS], l2[NS], l1[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) x1[n] = x[n];
    floor_and_normalize(x1, rho);
    balance_charge(x1);  // x1 is now x2, the input of the second normalisation
    fn_adj(x1, rho, obar, l2, rhobar);
    // balance_charge: x2[0] = -x3 - x7 + x1 + x12 + x6 + x4 + x9 + 2 x11
#pragma unroll
    for (int n = 0; n < NS; ++n) l1[n] = l2[n];
    l1[0] = 0.0;
    l1[3] -= l2[0];
    l1[7] -= l2[0];
    l1[1] += l2[0];
    l1[12] += l2[0];
    l1[6] += l2[0];
    l1[4] += l2[0];
    l1[9] += l2[0];
    l1[11] += 2.0 * l2[0];
    fn_adj(x, rho, l1, xbar, rhobar);
}

// x <- E^-T x with the LU of E (LINPACK dgesl, transposed job), x over the lanes.  U^T:
// as its unknowns come, each lane adds its own component's products, in index order.
// L^T: the products of an unknown's sum lie over the lanes, added in index order.
__device__ __noinline__ double solve_t_coop(const double* LU, uint64_t ip, uint64_t rY, double x, int lane) {
    using namespace coop;
    double xx[1] = {x}, t = 0.0;
    const uint64_t yy[1] = {rY};
#pragma unroll 1
    for (int k = 0; k < NEQ; ++k) {
        const double u = lane < NEQ ? LU[k * NEQ + lane] : 0.0;
        const double v[1] = {xx[0] - t};
        const double q = wr_div_finish(get<G, 1>(v, k), LU[k * NEQ + k], get<G, 1>(yy, k));
        if (lane == k) xx[0] = q;
        if (lane > k) t += u * q;
    }
#pragma unroll 1
    for (int k = NEQ - 2; k >= 0; --k) {
        const double p[1] = {lane < NEQ ? LU[lane * NEQ + k] * xx[0] : 0.0};
        double sum = 0.0;
#pragma unroll 1
        for (int i = k + 1; i < NEQ; ++i) sum += get<G, 1>(p, i);
        if (lane == k) xx[0] += sum;
        const int l = static_cast<int>((ip >> (4 * k)) & 15);
        if (l != k) {
            const double xk = get<G, 1>(xx, k), xl = get<G, 1>(xx, l);
            xx[0] = lane == k ? xl : lane == l ? xk : xx[0];
        }
    }
    return xx[0];
}

// A vector-Jacobian product program at state ys (kind 0: of the RHS, 1: of the Jacobian);
// its seeds are in their slots.  Like an evaluation, it guesses the temperature's regime
// and runs the general program where the guess was wrong.  Returns the regime whose
// output table holds.
__device__ __noinline__ int run_vjp(uint64_t* V, int kind, double ys, int& regime, int lane) {
    using namespace coop;
    int r = regime;
#pragma unroll 1
    while (true) {
        if (lane < NEQ) V[kY + lane] = bits(ys);
        __syncwarp();
        run_prog<CM, G, Tab>(2 * Tab::kRegimes + 2 * r + kind, lane, V);
        const uint64_t T = fetch(V, kind == 0 ? cd::kRhsVjpOut[r][NEQ + NP] : cd::kJacVjpOut[r][NEQ]);
        regime = regime_of<Tab>(T);
        if (r == 0 || (T > Tab::regime(r, 0) && T <= Tab::regime(r, 1))) return r;
        __syncwarp();  // every lane has read T
        r = 0;
    }
}

// f-VJP at state ys: fb over the lanes -> its part of the adjoint of ys over the lanes;
// multiplier adjoints accumulate into m0 (multiplier `lane`) and m1 (`lane` + 32)
__device__ __noinline__ double rhs_adj_at(uint64_t* V, double ys, double fb, double& m0, double& m1, int& regime,
                                          int lane) {
    using namespace coop;
    __syncwarp();
    if (lane < NEQ) V[cd::kFbar + lane] = bits(fb);
    const uint16_t* out = cd::kRhsVjpOut[run_vjp(V, 0, ys, regime, lane)];
    const double yb = lane < NEQ ? dbl(fetch(V, out[lane])) : 0.0;
    m0 += dbl(fetch(V, out[NEQ + lane]));
    if (lane + 32 < NP) m1 += dbl(fetch(V, out[NEQ + 32 + lane]));
    __syncwarp();
    return yb;
}

// one accepted step of the frozen controller; with st != nullptr it also stores what
// the step's adjoint needs: the factorised matrix, pivots and stage vectors
__device__ __noinline__ double step_replay(uint64_t* V, double yl, double h, double* st, int& regime, int lane) {
    const double y[1] = {yl};
    double k1[1], k2[1], k3[1];
    uint64_t ip;
    PhaseClock<false> pc;
    coop::KeepNothing none;
    ros2s_stages<CM, G, Tab, 1>(V, y, h, regime, lane, pc, false, none, ip, k1, k2, k3);
    if (st != nullptr) {
        for (int k = lane; k < NEQ * NEQ; k += G) st[k] = coop::dbl(V[coop::kE + k]);
        if (lane == 0) st[kStageIp] = __longlong_as_double(static_cast<long long>(ip));
        if (lane < NEQ) {
            st[kStageK1 + lane] = k1[0];
            st[kStageK2 + lane] = k2[0];
            st[kStageK3 + lane] = k3[0];
        }
    }
    __syncwarp();
    return yl + kB1 * k1[0] + kB2 * k2[0] + k3[0];
}

// Adjoint of one accepted step y -> ynew with step h: lam is the adjoint of ynew, the
// result that of y; multiplier adjoints accumulate into m0 and m1.
__device__ __noinline__ double step_adj(uint64_t* V, double y, double h, double lam, double& m0, double& m1,
                                        const double* st, int& regime, int lane) {
    using namespace coop;
    double* E = reinterpret_cast<double*>(V + kE);
    const bool in = lane < NEQ;
    __syncwarp();
    for (int k = lane; k < NEQ * NEQ; k += G) E[k] = st[k];
    const uint64_t ip = static_cast<uint64_t>(__double_as_longlong(st[kStageIp]));
    const double k1 = in ? st[kStageK1 + lane] : 0.0;
    const double k2 = in ? st[kStageK2 + lane] : 0.0;
    const double k3 = in ? st[kStageK3 + lane] : 0.0;
    __syncwarp();
    const uint64_t rY = in ? wr_div_recip(E[lane * NEQ + lane]) : 0;
    const double ih = ddiv(1.0, h);
    double yb = lam, kb1 = kB1 * lam, kb2 = kB2 * lam;
    // stage 3: k3 = E^-1 (f(y3) + (c31 k1 + c32 k2)/h), y3 = y + a31 k1 + a32 k2
    const double r3 = solve_t_coop(E, ip, rY, lam, lane);
    kb1 += kC31 * ih * r3;
    kb2 += kC32 * ih * r3;
    const double y3b = rhs_adj_at(V, y + kA31 * k1 + kA32 * k2, r3, m0, m1, regime, lane);
    yb += y3b;
    kb1 += kA31 * y3b;
    kb2 += kA32 * y3b;
    // stage 2: k2 = E^-1 (f(y2) + (c21/h) k1), y2 = y + a21 k1
    const double r2 = solve_t_coop(E, ip, rY, kb2, lane);
    kb1 += kC21 * ih * r2;
    const double y2b = rhs_adj_at(V, y + kA21 * k1, r2, m0, m1, regime, lane);
    yb += y2b;
    kb1 += kA21 * y2b;
    // stage 1: k1 = E^-1 f(y)
    const double r1 = solve_t_coop(E, ip, rY, kb1, lane);
    yb += rhs_adj_at(V, y, r1, m0, m1, regime, lane);
    // E = fac I - J(y): Jbar = sum_i rbar_i k_i^T, into the matrix slots
    double* tmp = reinterpret_cast<double*>(V + kTmp);
    if (in) {
        tmp[lane] = r3;
        tmp[16 + lane] = r2;
        tmp[32 + lane] = r1;
        tmp[48 + lane] = k3;
        tmp[64 + lane] = k2;
        tmp[80 + lane] = k1;
    }
    __syncwarp();
    for (int k = lane; k < NEQ * NEQ; k += G) {
        const int a = k / NEQ, b = k % NEQ;
        E[k] = tmp[a] * tmp[48 + b] + tmp[16 + a] * tmp[64 + b] + tmp[32 + a] * tmp[80 + b];
    }
    __syncwarp();
    const int r = run_vjp(V, 1, y, regime, lane);
    if (in) yb += dbl(fetch(V, cd::kJacVjpOut[r][lane]));
    __syncwarp();
    return yb;
}

// Burn replay for the adjoint: the state at the start of every 32-step segment into
// segck, the states before each step of the last segment and its step records into ys
// and stage (it is reversed first).  Returns the burn's final state.
__device__ __noinline__ double burn_checkpoint(uint64_t* V, double yl, const double* hs, int count, double* segck,
                                               double* ys, double* stage, int& regime, int lane) {
    const int nseg = (count + kSeg - 1) / kSeg;
#pragma unroll 1
    for (int k = 0; k < count; ++k) {
        const int g = k / kSeg, at = k % kSeg;
        const bool last = g == nseg - 1;
        if (lane < NEQ) {
            if (at == 0) segck[g * NEQ + lane] = yl;
            if (last) ys[at * NEQ + lane] = yl;
        }
        yl = step_replay(V, yl, hs[k], last ? stage + static_cast<size_t>(at) * kStage : nullptr, regime, lane);
    }
    return yl;
}

// Adjoint of the burn recorded by burn_checkpoint: lam is the adjoint of the final state,
// the result that of y0; each segment but the last (already in ys) is recomputed into
// ys from its checkpoint, then reversed step by step.
__device__ __noinline__ double burn_reverse(uint64_t* V, const double* hs, int count, double lam, double& m0, double& m1,
                                            const double* segck, double* ys, double* stage, int& regime, int lane) {
    const int nseg = (count + kSeg - 1) / kSeg;
#pragma unroll 1
    for (int g = nseg - 1; g >= 0; --g) {
        const int k0 = g * kSeg;
        const int k1 = (k0 + kSeg < count) ? k0 + kSeg : count;
        if (g != nseg - 1) {
            double yl = lane < NEQ ? segck[g * NEQ + lane] : 0.0;
#pragma unroll 1
            for (int k = k0; k < k1; ++k) {
                if (lane < NEQ) ys[(k - k0) * NEQ + lane] = yl;
                yl = step_replay(V, yl, hs[k], stage + static_cast<size_t>(k - k0) * kStage, regime, lane);
            }
        }
        __syncwarp();  // the records are read by other lanes than those that wrote them
#pragma unroll 1
        for (int k = k1 - 1; k >= k0; --k) {
            const double y = lane < NEQ ? ys[(k - k0) * NEQ + lane] : 0.0;
            lam = step_adj(V, y, hs[k], lam, m0, m1, stage + static_cast<size_t>(k - k0) * kStage, regime, lane);
        }
        __syncwarp();
    }
    return lam;
}

struct CellAdj {
    double xn[NS], T, e, rho, driver;
};

__global__ void __launch_bounds__(kBwdWarps * 32, 1) k_diff_backward(Args a) {
    extern __shared__ uint64_t sm[];
    const int lane = threadIdx.x & 31;
    uint64_t* V = sm + static_cast<size_t>(threadIdx.x >> 5) * cd::kNVA;
    init_slots(V, a, lane);
#pragma unroll 1
    for (int i = next_cell(a, lane); i < a.n; i = next_cell(a, lane)) {
        double* hrow = a.hbuf + static_cast<size_t>(i) * a.cap;
        double* segck = a.segck + static_cast<size_t>(i) * a.nseg * NEQ;
        double* ys = a.ys + static_cast<size_t>(i) * kSeg * NEQ;
        double* stage = a.stage + static_cast<size_t>(i) * kSeg * kStage;
        double m0 = 0.0, m1 = 0.0;
        CellAdj L;
#pragma unroll
        for (int k = 0; k < NS; ++k) L.xn[k] = a.qbar[15 * i + k];
        L.T = a.qbar[15 * i + NS];
        L.e = 0.0;
        L.rho = 0.0;
        L.driver = 0.0;
        int hend = 0;
        for (int s = lane; s < a.nsteps; s += 32) hend += a.counts[static_cast<size_t>(s) * a.n + i];
        hend = __reduce_add_sync(coop::kWarp, hend);
        int regime = 0;
#pragma unroll 1
        for (int s = a.nsteps - 1; s >= 0; --s) {
            const int kind = a.kind[static_cast<size_t>(s) * a.n + i];
            if (kind == 0) continue;
            const int cnt = a.counts[static_cast<size_t>(s) * a.n + i];
            const int hbeg = hend - cnt;
            // ---- recompute the step's forward pieces from its checkpoint
            CellS c0;
            load_ckpt(a, s, i, c0);
            const bool pert = a.perturb && s != 0 && s % kPerturbInterval == 0;
            const double f = pert ? perturbation_factor(i, s) : 1.0;
            CellS c1 = c0;  // after the perturbation
            if (pert) {
                c1.driver *= f;
                c1.rho = c1.rho * f;
#pragma unroll
                for (int k = 0; k < NS; ++k) c1.xn[k] *= f;
                renormalize(c1.xn, c1.rho);
                c1.T = eos_T_from_e(c1.xn, c1.e);
            }
            const double dt = collapse_timestep(c1.xn);
            double rho_n = 0.0;  // density of c1.xn
#pragma unroll
            for (int k = 0; k < NS; ++k) rho_n += mass(k) * c1.xn[k];
            double lam_dt = 0.0, lam_drv1 = 0.0;
            // adjoint of the state after the step, mapped back to c1 (and dt)
            double lx1[NS], lT1 = 0.0, le1 = 0.0, lrho1 = 0.0;
            if (kind == 1) {
                // driver += dt * driver / (dt / 0.1) ; xn, T, e, rho unchanged
                const double tff = dt / kTffReduc;
                lam_drv1 = L.driver * (1.0 + dt / tff);
                lam_dt = L.driver * c1.driver * (1.0 / tff - dt / (tff * tff * kTffReduc));
#pragma unroll
                for (int k = 0; k < NS; ++k) lx1[k] = L.xn[k];
                lT1 = L.T;
                le1 = L.e;
                lrho1 = L.rho;
            } else {
                const double dtg = a.dt_hist[s];
                const double tff = dt / kTffReduc;
                // drv2 = drv1 + dtg * drv1 / tff
                double lam_drv2 = L.driver;
                if (kind == 2) {
#pragma unroll
                    for (int k = 0; k < NS; ++k) lx1[k] = L.xn[k];
                    lT1 = L.T;
                    le1 = L.e;
                    lrho1 = L.rho;
                } else {
                    // forward: c2 = c1 scaled by the driver ratio, burn, commit
                    CellS c2 = c1;
                    double y0[NEQ];
                    advance_part(dtg, dt, c2, y0);
                    const double ratio = c2.driver / c1.driver;
                    if (regime == 0) regime = coop::regime_of<Tab>(coop::bits(c1.T));
                    double yN[NEQ];
                    const double yl =
                        burn_checkpoint(V, spread(V, y0, lane), hrow + hbeg, cnt, segck, ys, stage, regime, lane);
                    collect(V, yl, yN, lane);
                    // commit: xd = renormalize(yN, rho2), e3 = yN[14], T3 = eos_re(xd, e3)
                    double xd[NS];
#pragma unroll
                    for (int k = 0; k < NS; ++k) xd[k] = yN[k];
                    renormalize(xd, c2.rho);
                    double lxd[NS], le3 = L.e;
#pragma unroll
                    for (int k = 0; k < NS; ++k) lxd[k] = L.xn[k];
                    eos_T_adj(xd, yN[NS], L.T, lxd, le3);
                    double lam[NEQ], lrho2 = L.rho;
                    renorm_adj(yN, c2.rho, lxd, lam, lrho2);
                    lam[NS] = le3;
                    const double ll = burn_reverse(V, hrow + hbeg, cnt, spread(V, lam, lane), m0, m1, segck, ys, stage,
                                                   regime, lane);
                    collect(V, ll, lam, lane);
                    // y0 = (xc, e2), e2 = eos_rt(xc, T1), xc = x1 * ratio, rho2 = rho1 * ratio
                    double lratio = 0.0;
                    eos_e_adj(y0, c1.T, lam[NS], lam, lT1);
#pragma unroll
                    for (int k = 0; k < NS; ++k) {
                        lx1[k] = lam[k] * ratio;
                        lratio += lam[k] * c1.xn[k];
                    }
                    lrho1 = lrho2 * ratio;
                    lratio += lrho2 * c1.rho;
                    // ratio = drv2 / drv1
                    lam_drv2 += lratio / c1.driver;
                    lam_drv1 -= lratio * c2.driver / (c1.driver * c1.driver);
                    le1 = 0.0;  // e is recomputed from T before the burn
                }
                lam_drv1 += lam_drv2 * (1.0 + dtg / tff);
                lam_dt += lam_drv2 * (-dtg * c1.driver / (tff * tff)) / kTffReduc;
            }
            // dt = 0.1 sqrt(3 pi / (32 G rho)), rho = sum m x1
#pragma unroll
            for (int k = 0; k < NS; ++k) lx1[k] += lam_dt * (-0.5 * dt * mass(k) / rho_n);
            // ---- through the perturbation
            if (pert) {
                // T1 = eos_re(x1, e0)
                double le0 = le1, xa[NS], lxa[NS];
                eos_T_adj(c1.xn, c0.e, lT1, lx1, le0);
#pragma unroll
                for (int k = 0; k < NS; ++k) xa[k] = c0.xn[k] * f;
                renorm_adj(xa, c1.rho, lx1, lxa, lrho1);
#pragma unroll
                for (int k = 0; k < NS; ++k) L.xn[k] = lxa[k] * f;
                L.T = 0.0;
                L.e = le0;
                L.rho = lrho1 * f;
                L.driver = lam_drv1 * f;
            } else {
#pragma unroll
                for (int k = 0; k < NS; ++k) L.xn[k] = lx1[k];
                L.T = lT1;
                L.e = le1;
                L.rho = lrho1;
                L.driver = lam_drv1;
            }
            hend = hbeg;
        }
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < NS; ++k) a.ubar[15 * i + k] = L.xn[k];
            a.ubar[15 * i + NS] = L.T;
        }
        double* mbar = a.mbar + static_cast<size_t>(i) * NP;
        mbar[lane] = m0;
        if (lane + 32 < NP) mbar[lane + 32] = m1;
    }
}

template <class KernelT>
cudaError_t launch(KernelT k, int warps, size_t smem, Args a, int sms, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(k), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e == cudaSuccess) e = cudaMemsetAsync(a.queue, 0, sizeof(int), stream);
    if (e != cudaSuccess) return e;
    // every SM takes part as long as there are cells: with fewer cells than warps they
    // spread over the SMs one by one (blocks of fewer warps)
    const int per_sm = (a.n + sms - 1) / sms;
    const int w = per_sm < warps ? per_sm : warps;
    const int blocks = (a.n + w - 1) / w < sms ? (a.n + w - 1) / w : sms;
    k<<<blocks, w * 32, smem, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_diff_forward(Args a, int sms, cudaStream_t stream) {
    return launch(k_diff_forward, kFwdWarps, kFwdSmem, a, sms, stream);
}
cudaError_t launch_diff_backward(Args a, int sms, cudaStream_t stream) {
    return launch(k_diff_backward, kBwdWarps, kBwdSmem, a, sms, stream);
}

}  // namespace diff
}  // namespace wr

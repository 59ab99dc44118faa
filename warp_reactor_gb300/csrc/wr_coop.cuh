// wr_coop.cuh -- the cooperative advance: G lanes per cell (G = 8, 16 or 32).
//
// advance_collapse_gridwide_kernel (reproducer.cpp:7736-7785) runs one thread per
// cell.  On GB300 a warp issues one FP64 instruction every ~64-76 cycles, so an
// FP64 instruction executed with few active lanes wastes the scarce pipe, and a
// lane-per-cell kernel whose lanes sit in different phases, or idle at the end of
// an outer step while the stiffest cells still iterate, runs far below the FP64
// rate.  Here a group of G lanes owns one cell and every lane of the warp executes
// the same instruction stream:
//
//  * the network (burn_state_from_y, the analytic Jacobian and the RHS) is a
//    generated vector program (gen/coop.py): each step every lane computes one DAG
//    node from operands in the cell's shared-memory slot array V; all add/sub/mul
//    are one fused-multiply-add class with exact neutral operands, so one FP64
//    instruction serves G nodes; comparisons, selects and boolean logic ride on
//    the integer pipe in the same steps;
//  * the 15x15 factorisation (lu_decomposition, reproducer.cpp:96-151) is
//    warp-cooperative: pivot search by a __shfl_xor_sync argmax over the group,
//    row interchange, scaling and the rank-1 update spread over the G lanes, the
//    matrix staged in shared memory (V[0..225));
//  * the triangular solves (lu_solve, :154-181) keep the vector distributed over
//    the group's lanes and broadcast each pivot element with __shfl_sync;
//  * stage combinations, the error norm and the step-size controller
//    (RODAS::integrate, :7205-7347) run per component on the lanes; scalars are
//    replicated in every lane of the group.
//
// A rejected attempt is retried from the same state: where every cell of the warp
// retries, the Jacobian and RHS of the attempt before are used again (Kept); where one
// is at a new state, the program runs for all of them and gives the retrying ones the
// same values (same operations on the same operands), so the warp stays in one
// instruction stream.  The Jacobian counter follows the reference's rule.  Every
// value is the same binary64 operation on the same operands as in the reference
// and the CPU oracle, so results are bit-identical.
//
// The prologue of the advance (driver update, density scaling, e from T) and the
// commit after a successful burn (renormalisation, T from e) are cell-parallel
// kernels around the burn (k_order_preburn, k_commit): lane-per-cell work at full
// SIMD width, out of the cooperative kernel's instruction stream.
#pragma once

#include <climits>

#include "wr_kernels.cuh"

namespace wr {

// qbucket states after k_order_preburn (>= 0 is a queue bucket, -1 not queued)
constexpr int kQSkip = -2;     // queued, but the prologue ended the cell's step
constexpr int kQBurn = -3;     // to be burned by the advance
constexpr int kQBurnOK = -4;   // burned successfully: k_commit commits it

namespace coop {

enum { C_NONE = 0, C_FMA = 1, C_EXP = 2, C_LOG = 3, C_SQRT = 4, C_DIV = 5 };
// classes of derivative programs only (tables with Tab::kAdjoint): V[X] V[Y] and
// V[X] / V[Y], which are 0 where V[X] is zero, whatever V[Y] holds
enum { C_GMUL = 6, C_GDIV = 7 };
enum { I_SEL = 0, I_LE = 1, I_LT = 2, I_SGN = 3 };
// control byte of a step: class | CTL_INT (it has integer nodes) | CTL_SPECIAL (they
// include comparisons or sign operations) | CTL_FLUSH (its main results are stored in
// the step itself)
enum : uint32_t { CTL_CLASS = 7u, CTL_INT = 8u, CTL_SPECIAL = 16u, CTL_FLUSH = 32u };
// flags in the low three bits of the 16-bit destination fields of a step
enum : uint32_t {
    DV_NEG = 1u, DV_ABS = 2u, DV_SWAP = 4u,  // D: argument modifiers; divide V[Y] ^ L by V[X]
    FL_SABS = 4u                             // D2 of I_SGN: clear the sign (else flip)
};
constexpr int kE = 0;        // iteration matrix slots [0, 225)
constexpr int kY = 225;      // program inputs y[0..14]
constexpr int kRes = 240;    // reserved constants [240, 240 + Tab::kNR + Tab::kNF)
constexpr uint32_t kOff = 0xfff8u;
constexpr unsigned kWarp = 0xffffffffu;
constexpr uint64_t kSign = 0x8000000000000000ULL;
constexpr uint64_t kAbs = 0x7fffffffffffffffULL;
constexpr uint64_t kInfBits = 0x7ff0000000000000ULL;

__device__ __forceinline__ double dbl(uint64_t u) { return __longlong_as_double(static_cast<long long>(u)); }
__device__ __forceinline__ uint64_t bits(double d) { return static_cast<uint64_t>(__double_as_longlong(d)); }

// output operand (the RHS and Jacobian tables): slot (12 bits) | negate (bit 13) |
// abs (bit 14); constants sit in reserved slots
__device__ __forceinline__ uint64_t fetch(const uint64_t* V, uint32_t op) {
    uint64_t v = V[op & 0xfffu];
    v = (op & 0x4000u) ? (v & kAbs) : v;
    v = (op & 0x2000u) ? (v ^ kSign) : v;
    return v;
}

// Shared-memory access by 32-bit shared-window addresses (the interpreter runs out
// of line, where generic pointers would lose their address space).
__device__ __forceinline__ uint64_t lds64(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts64(uint32_t addr, uint64_t v) {
    asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
// base + the low (high) 16-bit field of w: one integer dot-product instruction
// instead of a mask (shift) and an add
__device__ __forceinline__ uint32_t addr_lo(uint32_t w, uint32_t base) { return __dp2a_lo(w, 0x0001u, base); }
__device__ __forceinline__ uint32_t addr_hi(uint32_t w, uint32_t base) { return __dp2a_lo(w, 0x0100u, base); }

// IEEE a <= b (le) or a < b on bit patterns: false when either is NaN, -0 == +0.  a <= b
// is the negation of b < a; as signed integers, two patterns order like their values
// unless both are negative.
__device__ __forceinline__ uint64_t compare(uint64_t a, uint64_t b, bool le) {
    const int64_t x = static_cast<int64_t>(le ? b : a), y = static_cast<int64_t>(le ? a : b);
    const bool lt = ((x & y) < 0 ? y < x : x < y) && ((x | y) & static_cast<int64_t>(kAbs)) != 0;
    const bool nan = (a & kAbs) > kInfBits || (b & kAbs) > kInfBits;
    return (lt != le) && !nan ? 1ULL : 0ULL;
}

// Transcendentals are one out-of-line copy each (CUDA's own functions inside for
// CudaMath), as are the solve and the evaluation: the attempt's code has to stay near
// the instruction cache's size, with 16 warps in different phases of it.
template <class M>
struct StepMath {
    static __device__ __noinline__ double exp(double x) { return M::exp(x); }
    static __device__ __noinline__ double log(double x) { return M::log(x); }
    static __device__ __noinline__ double sqrt(double x) { return M::sqrt(x); }
    static __device__ __noinline__ double cbrt(double x) { return M::cbrt(x); }
};

// main result of a division, exp, log or sqrt step: x = V[X], y = V[Y] ^ L, fl the
// modifier flags of D
template <class M>
__device__ __noinline__ uint64_t slow_step(uint32_t cls, uint64_t x, uint64_t y, uint32_t fl) {
    if (cls == C_DIV || cls == C_GDIV) {
        if (cls == C_GDIV && (x & kAbs) == 0) return 0;
        x = (fl & DV_ABS) ? (x & kAbs) : x;
        x = (fl & DV_NEG) ? (x ^ kSign) : x;
        const bool sw = (fl & DV_SWAP) != 0;
        return bits(ddiv(dbl(sw ? y : x), dbl(sw ? x : y)));
    }
    y = (fl & DV_ABS) ? (y & kAbs) : y;
    y = (fl & DV_NEG) ? (y ^ kSign) : y;
    if (cls == C_EXP) return bits(StepMath<M>::exp(dbl(y)));
    if (cls == C_LOG) return bits(StepMath<M>::log(dbl(y)));
    return bits(StepMath<M>::sqrt(dbl(y)));
}

// the integer node of a step: iw = A | B | C | D2
__device__ __forceinline__ void int_step(uint32_t c, uint64_t iw, uint32_t vb) {
    const uint32_t i0 = static_cast<uint32_t>(iw), i1 = static_cast<uint32_t>(iw >> 32);
    const uint64_t A = lds64(addr_lo(i0, vb)), B = lds64(addr_hi(i0, vb)), C = lds64(addr_lo(i1, vb));
    uint64_t v = A != 0 ? B : C;
    if (c & CTL_SPECIAL) {  // comparisons or sign operations
        const uint32_t d2 = i1 >> 16, iop = d2 & 3u;
        const uint64_t s = (d2 & FL_SABS) ? (A & kAbs) : (A ^ kSign);
        v = iop == I_SEL ? v : iop == I_SGN ? s : compare(A, B, iop == I_LE);
    }
    sts64(addr_hi(i1, vb) & ~7u, v);
}

// One generated program on the warp's cells, every lane in step.
//
// Step words of one lane: e.x = X | Y | Z | D and e.y = A | B | C | D2, 16-bit byte
// offsets into the cell's slot array at shared address vb (flags in the low bits of
// D and D2), and the lane's literal, XOR-ed into V[Y].  Main node V[D] =
// fma(V[X], V[Y] ^ L, V[Z]) or the step's other class; integer node V[D2] =
// V[A] != 0 ? V[B] : V[C] or a comparison or sign operation.  A step's class is the
// same for all lanes and comes from a control byte in constant memory, so its tests
// are uniform branches.
//
// A lone warp needs ~500 cycles for an FMA step when each step loads, computes,
// stores and synchronises before the next begins: decode, 30 cycles of shared
// memory, 64+ of FP64, store and barrier in one chain.  So the steps overlap: step s
// issues its FP64 instruction on operands loaded during step s - 1, then the
// results of step s - 1 are stored and the operands of step s + 1 loaded while it
// runs.  The generator keeps a main result MAIN_DELAY = 2 steps from its first use
// (or marks its step CTL_FLUSH), an integer node's INT_DELAY = 1.
//
// The loop runs four steps per iteration and loads the words of the next four at its
// top, in one batch.  A load per step, four
// steps ahead, made every step wait for the L2 latency of the newest one, since the
// few scoreboards of a warp are shared with the operand loads (Jacobian program at 16
// lanes, CUDA math, 16 warps in one block: 345 k cycles a run, 264 k in batches; a
// lone warp 211 k and 173 k).  The next four steps' control word is read with them: read
// at its first use, its constant-cache latency stood in every iteration (a lone warp at 32
// lanes 97.3 k and 90.9 k).  The integer node is part of the loop (a call per node: 90.9 k
// and 85.5 k).  The tables carry four idle steps past the end.  One out-of-line copy
// serves every call site: the instruction cache holds one loop.
__device__ __forceinline__ ulonglong2 ld_words(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint64_t ld_lit(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
template <int G>
struct StepWords {
    ulonglong2 e[4];
    uint64_t l[4];
    __device__ __forceinline__ void load(const ulonglong2* p, const uint64_t* q) {
#pragma unroll
        for (int k = 0; k < 4; ++k) e[k] = ld_words(p + k * G);
#pragma unroll
        for (int k = 0; k < 4; ++k) l[k] = ld_lit(q + k * G);
    }
};
template <class M, int G, class Tab>
__device__ __noinline__ void run_prog(int which, int gl, uint64_t* V) {
    const uint32_t vb = static_cast<uint32_t>(__cvta_generic_to_shared(V));
    which = __shfl_sync(kWarp, which, 0);  // uniform over the warp
    const int first = Tab::first(which), nsteps = Tab::steps(which), ctl0 = first / 4;
    const ulonglong2* p = Tab::prog() + first * G + gl;
    const uint64_t* q = Tab::lit() + first * G + gl;
    StepWords<G> a, b;
    a.load(p, q);
    uint64_t x, y, z;
    auto operands = [&](const ulonglong2 e, const uint64_t l) {
        const uint32_t w0 = static_cast<uint32_t>(e.x), w1 = static_cast<uint32_t>(e.x >> 32);
        x = lds64(addr_lo(w0, vb));
        y = lds64(addr_hi(w0, vb)) ^ l;
        z = lds64(addr_lo(w1, vb));
    };
    uint32_t c0 = Tab::ctl(ctl0);
    operands(a.e[0], a.l[0]);
    uint64_t res = 0;                          // the last step's main results,
    uint32_t dst = vb + Tab::sink(which) * 8;  // stored while this step's run
    auto step = [&](const ulonglong2 e, uint32_t c, const ulonglong2 en, const uint64_t ln) {
        const uint32_t w1 = static_cast<uint32_t>(e.x >> 32);
        const uint32_t cls = c & CTL_CLASS;
        uint64_t r = 0;
        if (cls == C_FMA)
            r = bits(__fma_rn(dbl(x), dbl(y), dbl(z)));
        else if (Tab::kAdjoint && cls == C_GMUL)
            r = (x & kAbs) == 0 ? 0 : bits(__fma_rn(dbl(x), dbl(y), dbl(z)));
        else if (cls != C_NONE)
            r = slow_step<M>(cls, x, y, w1 >> 16);
        if (c & CTL_INT) int_step(c, e.y, vb);
        if (c & CTL_FLUSH) sts64(addr_hi(w1, vb) & ~7u, r);
        sts64(dst, res);
        __syncwarp();
        operands(en, ln);
        res = r;
        dst = addr_hi(w1, vb) & ~7u;
    };
#pragma unroll 1
    for (int s = 0; s < nsteps; s += 4) {
        const uint32_t cn = Tab::ctl(ctl0 + s / 4 + 1);
        p += 4 * G;
        q += 4 * G;
        b.load(p, q);
        step(a.e[0], c0, a.e[1], a.l[1]);
        step(a.e[1], c0 >> 8, a.e[2], a.l[2]);
        step(a.e[2], c0 >> 16, a.e[3], a.l[3]);
        step(a.e[3], c0 >> 24, b.e[0], b.l[0]);
        a = b;
        c0 = cn;
    }
    sts64(dst, res);
    __syncwarp();
}

// The programs of a state (Jacobian program at 16 lanes, CUDA math, a block of 16
// warps: 285 k cycles for the general one, 238 k for a regime's; the RHS program 127 k
// and 102 k): regime 0 is right for every state; the others are the
// network specialised to a range of temperatures (fewer nodes, the same bits where T
// lies in the range).  T is a result of the program itself, so the regime is a guess,
// the cell's regime at its last evaluation, checked afterwards: the general program
// runs again where a cell's T lies outside.  The warp's cells share one program: where
// their guesses differ, the last regime, which spans all others.
template <class Tab>
__device__ __forceinline__ int regime_of(uint64_t T) {
    int r = 0;
#pragma unroll
    for (int k = Tab::kRegimes - 1; k > 0; --k)
        if (T > Tab::regime(k, 0) && T <= Tab::regime(k, 1)) r = k;
    return r;
}

// the reserved constants of the programs into the group's slot array (once per
// launch: no program writes them), then the exp/log/sqrt of constants, evaluated
// here with the kernel's own functions so that they are the bits a program step
// would compute
template <class M, int G, class Tab>
__device__ __forceinline__ void init_reserved(uint64_t* V, int gl) {
    for (int i = gl; i < Tab::kNR; i += G) V[kRes + i] = Tab::vconst()[i];
    for (int i = gl; i < Tab::kNF; i += G) {
        const ulonglong2 f = Tab::vfun()[i];
        const double a = dbl(f.y);
        const double r = f.x == C_EXP ? StepMath<M>::exp(a) : f.x == C_LOG ? StepMath<M>::log(a) : StepMath<M>::sqrt(a);
        V[kRes + Tab::kNR + i] = bits(r);
    }
    __syncwarp();
}

// lu_decomposition<15> (reproducer.cpp:96-151) by the G lanes of a group on the
// matrix E[r*15 + c] in shared memory: the same pivot (first strictly largest
// |a_ik|, a NaN diagonal keeps its row), the same row interchange, negated
// multipliers and rank-1 update, each element the same two roundings.  The warp's
// groups stay in step (a group with a zero pivot idles through the column), and a
// lane updates four elements at a time: their loads and FP64 latencies overlap.
template <int G>
__device__ __forceinline__ int lu_coop(double* E, int gl, uint64_t& ip) {
    constexpr int K = (NEQ + G - 1) / G;
    constexpr int U = 4;
    int info = 0;
    uint64_t piv = 0;
#pragma unroll 1
    for (int k = 0; k < NEQ - 1; ++k) {
        long long key = -1;
        int idx = NEQ;
#pragma unroll
        for (int t = 0; t < K; ++t) {
            const int r = gl + t * G;
            if (r >= k && r < NEQ) {
                const uint64_t u = bits(E[r * NEQ + k]) & kAbs;
                const long long kk = u > kInfBits ? (r == k ? LLONG_MAX : -1LL) : static_cast<long long>(u);
                if (kk > key) {
                    key = kk;
                    idx = r;
                }
            }
        }
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) {
            const long long ok = __shfl_xor_sync(kWarp, key, off, G);
            const int oi = __shfl_xor_sync(kWarp, idx, off, G);
            if (ok > key || (ok == key && oi < idx)) {
                key = ok;
                idx = oi;
            }
        }
        const int p = idx;
        piv |= static_cast<uint64_t>(p) << (4 * k);
        const double pivot = E[p * NEQ + k];
        const bool nz = pivot != 0.0;
        double rk[K], rp[K];
#pragma unroll
        for (int t = 0; t < K; ++t) {
            const int j = k + gl + t * G;
            rk[t] = j < NEQ ? E[k * NEQ + j] : 0.0;
            rp[t] = j < NEQ ? E[p * NEQ + j] : 0.0;
        }
        __syncwarp();
        if (nz && p != k) {
#pragma unroll
            for (int t = 0; t < K; ++t) {
                const int j = k + gl + t * G;
                if (j < NEQ) {
                    E[p * NEQ + j] = rk[t];
                    E[k * NEQ + j] = rp[t];
                }
            }
        }
        __syncwarp();
        if (!nz) info = k + 1;
        const double mult = ddiv(-1.0, pivot);
#pragma unroll
        for (int t = 0; t < K; ++t) {
            const int i = k + 1 + gl + t * G;
            if (nz && i < NEQ) E[i * NEQ + k] = E[i * NEQ + k] * mult;
        }
        __syncwarp();
        const int m = NEQ - 1 - k;
        const unsigned cm = (65536u + static_cast<unsigned>(m) - 1u) / static_cast<unsigned>(m);
        const int last = nz ? m * m : 0;
#pragma unroll 1
        for (int e0 = gl; e0 - gl < m * m; e0 += U * G) {
            double aij[U], akj[U], aik[U];
            int at[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + u * G;
                const int ii = static_cast<int>((static_cast<unsigned>(e) * cm) >> 16);
                const int i = k + 1 + ii;
                const int j = k + 1 + (e - ii * m);
                at[u] = i * NEQ + j;
                if (e < last) {
                    aij[u] = E[at[u]];
                    akj[u] = E[k * NEQ + j];
                    aik[u] = E[i * NEQ + k];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (e0 + u * G < last) E[at[u]] = aij[u] + akj[u] * aik[u];
        }
        __syncwarp();
    }
    piv |= static_cast<uint64_t>(NEQ - 1) << (4 * (NEQ - 1));
    if (E[(NEQ - 1) * NEQ + NEQ - 1] == 0.0) info = NEQ;
    ip = piv;
    return info;
}

// component c of a vector distributed over the group: lane c % G, register c / G
// (c is uniform over the group; the register is picked by a select, so the
// array stays in registers)
template <int G, int K, class T>
__device__ __forceinline__ T get(const T (&x)[K], int c) {
    T v = x[0];
#pragma unroll
    for (int t = 1; t < K; ++t) v = (c / G == t) ? x[t] : v;
    return __shfl_sync(kWarp, v, c % G, G);
}

// the reciprocals of the factorisation's diagonal for the back substitutions
// (wr_div_recip of U(c, c), distributed like a vector): the three stage solves
// of an attempt divide by the same 15 pivots
template <int G, int K>
__device__ __forceinline__ void diag_recips(const double* LU, uint64_t (&rY)[K], int gl) {
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        rY[t] = c < NEQ ? wr_div_recip(LU[c * NEQ + c]) : 0;
    }
}

// lu_solve<15> (reproducer.cpp:154-181) with x distributed over the group; the
// back substitution's quotients use the pivots' precomputed reciprocals (the same
// IEEE quotients as a division), inline (a call for each: 32.1 k cycles for a lone cell's
// three solves, 29.4 k without).  The next column's factors are loaded while a column's
// chain (broadcast, quotient, multiply, add) runs.
template <int K>
struct Vec {
    double v[K];
};
template <int G, int K>
__device__ __noinline__ Vec<K> solve_copy(const double* LU, uint64_t ip, uint64_t r0, uint64_t r1, Vec<K> b, int gl) {
    const uint64_t rY2[2] = {r0, r1};
    uint64_t rY[K];
#pragma unroll
    for (int t = 0; t < K; ++t) rY[t] = rY2[t];
    double(&x)[K] = b.v;
    const double* row[K];
#pragma unroll
    for (int t = 0; t < K; ++t) row[t] = LU + (gl + t * G < NEQ ? gl + t * G : 0) * NEQ;
    double l[K], ln[K];
#pragma unroll
    for (int t = 0; t < K; ++t) l[t] = row[t][0];
#pragma unroll 1
    for (int k = 0; k < NEQ - 1; ++k) {
#pragma unroll
        for (int t = 0; t < K; ++t) ln[t] = row[t][k + 1];
        const int p = static_cast<int>((ip >> (4 * k)) & 15);
        double tk = get<G, K>(x, k);
        if (__any_sync(kWarp, p != k)) {
            double v = x[0];
#pragma unroll
            for (int t = 1; t < K; ++t) v = (p / G == t) ? x[t] : v;
            const double xp = __shfl_sync(kWarp, v, p % G, G);
#pragma unroll
            for (int t = 0; t < K; ++t) {
                const int c = gl + t * G;
                x[t] = c == k ? xp : (c == p ? tk : x[t]);
            }
            tk = xp;
        }
#pragma unroll
        for (int t = 0; t < K; ++t) {
            const int c = gl + t * G;
            if (c > k && c < NEQ) x[t] = x[t] + tk * l[t];
            l[t] = ln[t];
        }
    }
    // l holds column NEQ - 1
    double d = LU[(NEQ - 1) * NEQ + NEQ - 1];
#pragma unroll 1
    for (int k = NEQ - 1; k >= 0; --k) {
        const int kn = k > 0 ? k - 1 : 0;
#pragma unroll
        for (int t = 0; t < K; ++t) ln[t] = row[t][kn];
        const double dn = LU[kn * NEQ + kn];
        const uint64_t yk = get<G, K>(rY, k);
        const double q = wr_div_finish(get<G, K>(x, k), d, yk);
        const double tk = -q;
#pragma unroll
        for (int t = 0; t < K; ++t) {
            const int c = gl + t * G;
            if (c == k) x[t] = q;
            if (c < k) x[t] = x[t] + tk * l[t];
            l[t] = ln[t];
        }
        d = dn;
    }
    return b;
}
template <int G, int K>
__device__ __forceinline__ void solve_coop(const double* LU, uint64_t ip, const uint64_t (&rY)[K], double (&x)[K],
                                           int gl) {
    static_assert(K <= 2, "15 unknowns on at least 8 lanes");
    Vec<K> b;
#pragma unroll
    for (int t = 0; t < K; ++t) b.v[t] = x[t];
    b = solve_copy<G, K>(LU, ip, rY[0], rY[K - 1], b, gl);
#pragma unroll
    for (int t = 0; t < K; ++t) x[t] = b.v[t];
}

template <int G, int K>
__device__ __forceinline__ void store_inputs(uint64_t* V, const double (&v)[K], int gl) {
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        if (c < NEQ) V[kY + c] = bits(v[t]);
    }
}

template <int G, int K>
__device__ __forceinline__ void load_outputs(const uint64_t* V, const uint16_t* out, double (&v)[K], int gl) {
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        v[t] = c < NEQ ? dbl(fetch(V, out[c])) : 0.0;
    }
}

// one evaluation of the network at v (kind 0: Jacobian and RHS, 1: RHS): the
// program's index, whose output tables hold; regime is the group's guess, replaced by
// the regime of the temperature found
// (returned: the index in the low half, the regime in the high half)
template <class M, int G, class Tab, int K>
__device__ __noinline__ int evaluate_copy(int kind, Vec<K> b, int regime, int gl, uint64_t* V) {
    double(&v)[K] = b.v;
    int r = __shfl_sync(kWarp, regime, 0);
    if (__any_sync(kWarp, regime != r)) r = __any_sync(kWarp, regime == 0) ? 0 : Tab::kRegimes - 1;
#pragma unroll 1
    while (true) {
        store_inputs<G, K>(V, v, gl);
        __syncwarp();
        run_prog<M, G, Tab>(2 * r + kind, gl, V);
        const uint64_t T = fetch(V, Tab::out(2 * r + kind)[NEQ]);
        regime = regime_of<Tab>(T);
        const bool fits = r == 0 || (T > Tab::regime(r, 0) && T <= Tab::regime(r, 1));
        if (__all_sync(kWarp, fits)) break;
        __syncwarp();  // every lane has read T
        r = 0;
    }
    return (2 * r + kind) | regime << 16;
}
template <class M, int G, class Tab, int K>
__device__ __forceinline__ int evaluate(int kind, const double (&v)[K], int& regime, int gl, uint64_t* V) {
    Vec<K> b;
#pragma unroll
    for (int t = 0; t < K; ++t) b.v[t] = v[t];
    const int w = evaluate_copy<M, G, Tab, K>(kind, b, regime, gl, V);
    regime = w >> 16;
    return w & 0xffff;
}

// E = -J into the matrix slots after the Jacobian program.  The program uses the
// matrix slots as scratch and keeps its results (the Jacobian entries and the
// RHS) above them; the generated table names, per matrix entry r * 15 + c, the
// slot (a reserved one for a constant entry) that holds J(r, c) with the negation
// as an operand modifier.
template <int G>
__device__ __forceinline__ void gather_matrix(uint64_t* V, const uint16_t* jac, int gl) {
#pragma unroll 5
    for (int i = gl; i < NEQ * NEQ; i += G) V[kE + i] = fetch(V, jac[i]);
    __syncwarp();
}

// E and the RHS of a state, kept in the lanes' local memory for the attempts that
// retry it with another step size (shared memory has no room for a second matrix at
// 16 lanes and 16 warps).  A collapse of one cell rejects 27 % of its attempts, one of
// 64^3 cells 14 %, and the Jacobian program is a third of an attempt: the collapse of one
// cell 219 -> 198 ms, a step of 16^3 cells 22.3 -> 20.0 ms, of 64^3 234 -> 221 ms.
template <int G, int K>
struct Kept {
    static constexpr bool kOn = true;
    static constexpr int kRows = (NEQ * NEQ + G - 1) / G;
    uint64_t m[kRows];
    double f[K];
    __device__ __forceinline__ void save(const uint64_t* V, const double (&rhs)[K], int gl) {
#pragma unroll 4
        for (int t = 0; t < kRows; ++t)
            if (gl + t * G < NEQ * NEQ) m[t] = V[kE + gl + t * G];
#pragma unroll
        for (int t = 0; t < K; ++t) f[t] = rhs[t];
        __syncwarp();  // the caller changes the diagonal, whose entries other lanes have read here
    }
    __device__ __forceinline__ void restore(uint64_t* V, double (&rhs)[K], int gl) const {
#pragma unroll 4
        for (int t = 0; t < kRows; ++t)
            if (gl + t * G < NEQ * NEQ) V[kE + gl + t * G] = m[t];
#pragma unroll
        for (int t = 0; t < K; ++t) rhs[t] = f[t];
        __syncwarp();
    }
};
struct KeepNothing {  // for a caller that never retries
    static constexpr bool kOn = false;
};

// Generated tables of one G, supplied by the translation unit that includes the
// generated header (one unit per G keeps the large initialisers apart).
//   Tab::kNV, Tab::kNR, Tab::kNF, Tab::kRegimes, Tab::kAdjoint and device accessors vconst(),
//   vfun(), prog(), lit(), ctl(i) (control bytes of four steps), first(w), steps(w) and
//   sink(w) (the slot that nothing reads) of program w = 2 * regime + kind, out(w) (RHS
//   operands, then T), jac(regime) and regime(k, 0 or 1) (the temperatures between which
//   regime k holds).

}  // namespace coop

// Phase counters (a diagnostic, wr_diag_coop_phases): the instrumented
// instantiation adds, per warp, the clock64 cycles of each phase of its attempts
// into 16 device counters: [0] queue, prologue and epilogue, [1] Jacobian+RHS
// program, [2] output loads, Jacobian gather, diagonal and stage combinations,
// [3] LU, [4] stage solves, [5] RHS programs, [6] error norm and controller,
// [7] attempts, [8] cycles from start to exit, [9] warps.  The plain
// instantiation compiles every call to nothing.
enum { PH_QUEUE = 0, PH_JPROG = 1, PH_MISC = 2, PH_LU = 3, PH_SOLVE = 4, PH_RPROG = 5, PH_CTL = 6 };
__device__ __forceinline__ long long phase_now() {
#if defined(__CUDA_ARCH__)
    return clock64();
#else
    return 0;
#endif
}
template <bool ON>
struct PhaseClock {
    __device__ __forceinline__ void mark(int) {}
    __device__ __forceinline__ void attempt() {}
    __device__ __forceinline__ void flush(unsigned long long*, int) {}
};
template <>
struct PhaseClock<true> {
    long long acc[7] = {0, 0, 0, 0, 0, 0, 0};
    long long t0, t, attempts = 0;
    __device__ __forceinline__ PhaseClock() : t0(phase_now()), t(t0) {}
    __device__ __forceinline__ void mark(int k) {
        const long long now = phase_now();
        acc[k] += now - t;
        t = now;
    }
    __device__ __forceinline__ void attempt() { ++attempts; }
    __device__ __forceinline__ void flush(unsigned long long* out, int lane) {
        mark(PH_QUEUE);
        if (lane != 0 || out == nullptr) return;
#pragma unroll
        for (int k = 0; k < 7; ++k) atomicAdd(out + k, static_cast<unsigned long long>(acc[k]));
        atomicAdd(out + 7, static_cast<unsigned long long>(attempts));
        atomicAdd(out + 8, static_cast<unsigned long long>(phase_now() - t0));
        atomicAdd(out + 9, 1ULL);
    }
};

// The stages of one ROS2S attempt (reproducer.cpp:7259-7304) of the warp's cells from y
// with step h: the factorised iteration matrix in the matrix slots, its pivots, k1, k2
// and k3.  Returns the factorisation's info (0: regular; the rest means nothing
// otherwise).  again (the same for the whole warp): each cell's y is the one of its
// last attempt, whose Jacobian and RHS stand in kept; the program does not run.
template <class M, int G, class Tab, int K, class PC, class Keep>
__device__ __forceinline__ int ros2s_stages(uint64_t* V, const double (&y)[K], double h, int& regime, int gl, PC& pc,
                                            bool again, Keep& kept, uint64_t& ip, double (&ak1)[K], double (&ak2)[K],
                                            double (&w)[K]) {
    using namespace coop;
    double* E = reinterpret_cast<double*>(V + kE);
    if (!Keep::kOn || !again) {
        const int jw = evaluate<M, G, Tab, K>(0, y, regime, gl, V);
        pc.mark(PH_JPROG);
        load_outputs<G, K>(V, Tab::out(jw), ak1, gl);
        gather_matrix<G>(V, Tab::jac(jw / 2), gl);
        if constexpr (Keep::kOn) kept.save(V, ak1, gl);
    } else if constexpr (Keep::kOn) {
        kept.restore(V, ak1, gl);
    }
    const double fac = ddiv(1.0, h * kGamma);
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        if (c < NEQ) E[c * NEQ + c] = E[c * NEQ + c] + fac;
    }
    __syncwarp();
    pc.mark(PH_MISC);
    ip = 0;
    const int info = lu_coop<G>(E, gl, ip);
    uint64_t rY[K];
    diag_recips<G, K>(E, rY, gl);
    pc.mark(PH_LU);
    solve_coop<G, K>(E, ip, rY, ak1, gl);
    pc.mark(PH_SOLVE);
    // stage 2
    {
        double yn[K];
        const double c21h = ddiv(kC21, h);
#pragma unroll
        for (int t = 0; t < K; ++t) {
            yn[t] = y[t] + kA21 * ak1[t];
            w[t] = c21h * ak1[t];
        }
        pc.mark(PH_MISC);
        const int rw = evaluate<M, G, Tab, K>(1, yn, regime, gl, V);
        pc.mark(PH_RPROG);
        double dy[K];
        load_outputs<G, K>(V, Tab::out(rw), dy, gl);
#pragma unroll
        for (int t = 0; t < K; ++t) w[t] += dy[t];
        pc.mark(PH_MISC);
        solve_coop<G, K>(E, ip, rY, w, gl);
        pc.mark(PH_SOLVE);
#pragma unroll
        for (int t = 0; t < K; ++t) ak2[t] = w[t];
    }
    // stage 3
    {
        double yn[K];
#pragma unroll
        for (int t = 0; t < K; ++t) {
            yn[t] = y[t] + kA31 * ak1[t] + kA32 * ak2[t];
            w[t] = ddiv(kC31 * ak1[t] + kC32 * ak2[t], h);
        }
        __syncwarp();  // every lane has read the stage-2 outputs
        pc.mark(PH_MISC);
        const int rw = evaluate<M, G, Tab, K>(1, yn, regime, gl, V);
        pc.mark(PH_RPROG);
        double dy[K];
        load_outputs<G, K>(V, Tab::out(rw), dy, gl);
#pragma unroll
        for (int t = 0; t < K; ++t) w[t] += dy[t];
        pc.mark(PH_MISC);
        solve_coop<G, K>(E, ip, rY, w, gl);
        pc.mark(PH_SOLVE);
    }
    return info;
}

// The candidate state from the stages and its error norm (reproducer.cpp:7299-7304).
// FMAX: the error scale's maximum by fmax, which drops a NaN (the structured policy),
// instead of std::max.
template <int G, bool FMAX, int K>
__device__ __forceinline__ void ros2s_candidate(const double (&y)[K], const double (&ak1)[K], const double (&ak2)[K],
                                                const double (&ak3)[K], int gl, double (&ynew)[K], double& err) {
    using namespace coop;
    double sq[K];
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        ynew[t] = y[t] + kB1 * ak1[t] + kB2 * ak2[t] + ak3[t];
        const double wi = kE1 * ak1[t] + kE2 * ak2[t] + kE3 * ak3[t];
        const double rtol = c < NS ? kRtolSpec : kRtolEnergy;
        const double atol = c < NS ? kAtolSpec : kAtolEnergy;
        const double a = ::fabs(y[t]), b = ::fabs(ynew[t]);
        const double sk = atol + rtol * (FMAX ? ::fmax(a, b) : smax(a, b));
        const double term = ddiv(wi, sk);
        sq[t] = term * term;
    }
    // err = sum over components in index order (0.0 + sq[0] == sq[0]: a square)
    err = get<G, K>(sq, 0);
#pragma unroll
    for (int c = 1; c < NEQ; ++c) err = err + get<G, K>(sq, c);
    err = ::sqrt(ddiv(err, 15.0));
}

// One attempt: candidate state, error norm, and the factorisation's info
template <class M, int G, class Tab, bool FMAX, int K, class PC, class Keep>
__device__ __forceinline__ int ros2s_attempt(uint64_t* V, const double (&y)[K], double h, int& regime, int gl, PC& pc,
                                             bool again, Keep& kept, double (&ynew)[K], double& err) {
    uint64_t ip;
    double ak1[K], ak2[K], ak3[K];
    const int info = ros2s_stages<M, G, Tab, K>(V, y, h, regime, gl, pc, again, kept, ip, ak1, ak2, ak3);
    ros2s_candidate<G, FMAX, K>(y, ak1, ak2, ak3, gl, ynew, err);
    return info;
}

// The controller's next step sizes (reproducer.cpp:7308-7327) after a step h with error
// norm err: hnew from err alone, hgus with the Gustafsson factor.  Their two chains
// (quotient, cube root, quotient, limits, quotient) run side by side, hnew's in the even
// lanes and hgus's in the odd ones: one cube root and three quotients of latency instead
// of two and five (a step of 20,011 cells in portable math 20.1 -> 19.5 ms, the structured
// policy on 1,000 cells 89.2 -> 86.9 ms).  FMAX: limits by fmax and fmin (the structured
// policy).
template <int G, bool FMAX, class Cbrt>
__device__ __forceinline__ void step_sizes(double err, double erracc, double hacc, double h, int gl, Cbrt cbrt,
                                           double& hnew, double& hgus) {
    using coop::kWarp;
    const bool odd = (gl & 1) != 0;
    // before the first accepted step (hacc 0) hgus is not used, and a zero would take the
    // odd lanes through the division's native fallback beside the even lanes' quotient: 7 k
    // cycles of every first attempt, a 64^3 collapse 23.56 s instead of 23.20 s
    const double q = ddiv(odd ? (hacc == 0.0 ? h : hacc) : err * err, odd ? h : erracc);
    const double e2 = __shfl_sync(kWarp, q, 0, G), ratio = __shfl_sync(kWarp, q, 1, G);
    const double c = cbrt(odd ? e2 : err);
    const double raw = ddiv(odd ? ratio * c : c, kSafe);
    const double f = FMAX ? ::fmax(1.0 / kFacMax, ::fmin(1.0 / kFacMin, raw))
                          : smax(1.0 / kFacMax, smin(1.0 / kFacMin, raw));
    const double fs = __shfl_sync(kWarp, f, 0, G), fg = __shfl_sync(kWarp, f, 1, G);
    const double both = FMAX ? ::fmax(fs, fg) : smax(fs, fg);
    const double hn = ddiv(h, odd ? both : fs);
    hnew = __shfl_sync(kWarp, hn, 0, G);
    hgus = __shfl_sync(kWarp, hn, 1, G);
}

// The cooperative burn: persistent blocks of W warps, G lanes per cell, each group
// taking cells from the work queue until it is empty.  PH: the phase-counting
// instantiation (phases: its 16 counters).
template <class M, int G, int W, class Tab, bool PH = false>
__global__ void __launch_bounds__(W * 32, 1) k_advance_coop(DevState s, StepCtl* ctl, unsigned long long* phases) {
    using namespace coop;
    constexpr int K = (NEQ + G - 1) / G;
    constexpr int SLOTS = 32 / G;
    extern __shared__ uint64_t sm[];
    if (ctl->all_stop) return;
    const int lane = threadIdx.x & 31;
    const int slot = lane / G;
    const int gl = lane % G;
    const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (slot * G));
    uint64_t* V = sm + static_cast<size_t>((threadIdx.x >> 5) * SLOTS + slot) * Tab::kNV;
    init_reserved<M, G, Tab>(V, gl);
    const int n = s.n;
    const unsigned int queued = ctl->queued;

    PhaseClock<PH> pc;
    Lane L;
    int cell = INT_MIN, g = 0;  // without a cell: -1 - (the group it follows)
    bool have = false;     // the group holds a cell
    bool drained = false;  // it has seen the queue's end
    int regime = 0;        // the temperature regime of its last evaluation
    double y[K];
    Kept<G, K> kept;
#pragma unroll
    for (int t = 0; t < K; ++t) y[t] = 0.0;

#pragma unroll 1
    while (true) {
        // ---- bring the group's cell to "ready for an attempt" (per group)
#pragma unroll 1
        while (true) {
            if (!have) {
                if (drained) break;
                unsigned int q = 0;
                if (gl == 0) q = atomicAdd(&ctl->queue, 1u);
                q = __shfl_sync(gmask, q, 0, G);
                if (q >= queued) {
                    drained = true;
                    break;
                }
                cell = s.order[q];
                if (s.qbucket[cell] != kQBurn) continue;
                g = s.grid_of ? s.grid_of[cell] : 0;
                const double dt_grid = s.local_dt ? s.local_dt[cell] : ctl[g].dt_grid;
#pragma unroll
                for (int t = 0; t < K; ++t) {
                    const int c = gl + t * G;
                    y[t] = c < NS ? s.xn[c * n + cell] : (c == NS ? s.e[cell] : 0.0);
                }
                // RODAS::integrate prologue, reproducer.cpp:7218-7235
                L.tout = dt_grid;
                L.x = 0.0;
                double h0 = dt_grid;
                if (::fabs(h0) <= 10.0 * kUround) h0 = 1.e-6;
                L.h = smin(::fabs(h0), dt_grid);
                L.reject = false;
                L.last = false;
                L.nsing = 0;
                L.hacc = 0.0;
                L.erracc = 1.0;
                L.hopt = L.h;
                L.n_step = L.n_accept = L.n_reject = L.n_jac = L.n_decomp = 0;
                L.fresh = true;
                have = true;
                regime = regime_of<Tab>(bits(s.T[cell]));
            }
            if (!L.fresh) break;
            // outer-loop checks, reproducer.cpp:7236-7255
            int code = 0;
            if (L.n_step > kMaxSteps) code = WR_TOO_MANY_STEPS;
            else if (0.1 * ::fabs(L.h) <= ::fabs(L.x) * kUround) code = WR_DT_UNDERFLOW;
            else if (L.last) code = WR_SUCCESS;
            if (code != 0) {
                // burn_ros2s epilogue: counters, then the state (success) or the code
                if (gl == 0) {
                    const uint64_t st[7] = {
                        static_cast<uint64_t>(L.n_step), static_cast<uint64_t>(3 * L.n_step),
                        static_cast<uint64_t>(L.n_jac), static_cast<uint64_t>(L.n_decomp),
                        static_cast<uint64_t>(3 * L.n_step), static_cast<uint64_t>(L.n_accept),
                        static_cast<uint64_t>(L.n_reject)};
#pragma unroll
                    for (int k = 0; k < 7; ++k) s.stats[k * n + cell] += st[k];
                    s.cost[cell] = L.n_step;
                    if (code != WR_SUCCESS) record_failure(ctl + g, code);
                }
                if (code == WR_SUCCESS) {
#pragma unroll
                    for (int t = 0; t < K; ++t) {
                        const int c = gl + t * G;
                        if (c < NS) s.xn[c * n + cell] = y[t];
                        else if (c == NS) s.e[cell] = y[t];
                    }
                    if (gl == 0) s.qbucket[cell] = kQBurnOK;
                }
                have = false;
                continue;
            }
            L.hopt = L.h;
            if (L.x + L.h * 1.0001 >= L.tout) {
                L.h = L.tout - L.x;
                L.last = true;
            }
            break;
        }
        __syncwarp();
        // the warp's groups run every attempt in step; a group without a cell
        // follows one that has one (same state, same branches) and commits nothing
        const unsigned holders = __ballot_sync(kWarp, have);
        if (holders == 0) break;
        const int leader = (__ffs(holders) - 1) / G;
        {
            const int from = leader * G + gl;
#pragma unroll
            for (int t = 0; t < K; ++t) {
                const double o = __shfl_sync(kWarp, y[t], from);
                y[t] = have ? y[t] : o;
            }
            const double oh = __shfl_sync(kWarp, L.h, from);
            L.h = have ? L.h : oh;
            const int og = __shfl_sync(kWarp, regime, from);
            regime = have ? regime : og;
        }
        pc.mark(PH_QUEUE);
        pc.attempt();

        // a rejected attempt is retried from the same state: where no cell of the warp is
        // at a new one, the Jacobian and the RHS of the last attempt stand.  A group that has
        // begun to follow another has its own last cell's: from them its stages would go
        // elsewhere, out of the temperature regime, and the warp's vote would run the general
        // program for everyone at every retry.
        const bool joins = !have && cell != -1 - leader;
        const bool again = !__any_sync(kWarp, have ? L.fresh : joins);
        if (joins) cell = -1 - leader;
        if (L.fresh) L.n_jac += 1;
        L.fresh = false;
        const double h = L.h;
        double ynew[K], err;
        const int info = ros2s_attempt<M, G, Tab, false, K>(V, y, h, regime, gl, pc, again, kept, ynew, err);
        // step-size controller, reproducer.cpp:7308-7344
        double hnew, hgus;
        step_sizes<G, false>(err, L.erracc, L.hacc, h, gl, StepMath<M>::cbrt, hnew, hgus);
        int code = 0;  // a failure that ends the cell's burn
        if (info != 0) {  // singular: the attempt counts for nothing (reproducer.cpp:7268-7277)
            L.nsing += 1;
            if (L.nsing >= 5) {
                code = WR_LU_DECOMPOSITION_ERROR;
            } else {
                L.h = h * 0.5;
                L.reject = true;
                L.last = false;
            }
        } else if (err <= 1.0) {
            L.n_decomp += 1;
            L.n_step += 1;
            L.n_accept += 1;
            if (L.n_accept > 1) hnew = hgus;
            L.hacc = h;
            L.erracc = smax(1.e-2, err);
#pragma unroll
            for (int t = 0; t < K; ++t) y[t] = ynew[t];
            L.x += h;
            const double hmaxn = L.tout;
            if (::fabs(hnew) > hmaxn) hnew = hmaxn;
            if (L.reject) hnew = smin(::fabs(hnew), ::fabs(h));
            L.reject = false;
            L.h = hnew;
            L.fresh = true;
        } else {
            L.n_decomp += 1;
            L.n_step += 1;
            L.reject = true;
            L.last = false;
            L.h = hnew;
            if (L.n_accept >= 1) L.n_reject += 1;
            // the reject loop's only exit besides acceptance: a step size that has
            // underflowed to zero ends the cell with the reference's DT_UNDERFLOW
            // (reproducer.cpp:7240) instead of retrying forever
            if (hnew == 0.0) code = WR_DT_UNDERFLOW;
        }
        if (have && code != 0) {
            if (gl == 0) {
                const uint64_t st[7] = {
                    static_cast<uint64_t>(L.n_step), static_cast<uint64_t>(3 * L.n_step),
                    static_cast<uint64_t>(L.n_jac), static_cast<uint64_t>(L.n_decomp),
                    static_cast<uint64_t>(3 * L.n_step), static_cast<uint64_t>(L.n_accept),
                    static_cast<uint64_t>(L.n_reject)};
#pragma unroll
                for (int k = 0; k < 7; ++k) s.stats[k * n + cell] += st[k];
                s.cost[cell] = L.n_step;
                record_failure(ctl + g, code);
            }
            have = false;
        }
        __syncwarp();  // the next attempt overwrites V: every lane is done with it
        pc.mark(PH_CTL);
    }
    pc.flush(phases, lane);
}

// ---------------------------------------------------------------- diagnostics
// The generated programs and the cooperative LU/solve on caller-supplied inputs
// (include/warp_reactor_diag.h), one group of G lanes per case.
template <class M, int G, class Tab>
__global__ void k_diag_coop_network(int n, const double* __restrict__ y, double* J, double* f, double* f2) {
    using namespace coop;
    constexpr int K = (NEQ + G - 1) / G;
    constexpr int SLOTS = 32 / G;
    extern __shared__ uint64_t sm[];
    const int lane = threadIdx.x & 31, slot = lane / G, gl = lane % G;
    const int warp = threadIdx.x >> 5;
    // the warp's groups run in step: one past the end repeats the last case
    const int cell = min((blockIdx.x * static_cast<int>(blockDim.x >> 5) + warp) * SLOTS + slot, n - 1);
    uint64_t* V = sm + static_cast<size_t>(warp * SLOTS + slot) * Tab::kNV;
    const double* E = reinterpret_cast<const double*>(V + kE);
    init_reserved<M, G, Tab>(V, gl);
    double yy[K], out[K];
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        yy[t] = c < NEQ ? y[static_cast<size_t>(cell) * NEQ + c] : 0.0;
    }
    // the first run finds the temperature's regime, so the two that count run its programs
    int regime = 0;
    evaluate<M, G, Tab, K>(1, yy, regime, gl, V);
    __syncwarp();
    const int jw = evaluate<M, G, Tab, K>(0, yy, regime, gl, V);
    load_outputs<G, K>(V, Tab::out(jw), out, gl);
    gather_matrix<G>(V, Tab::jac(jw / 2), gl);
    for (int i = gl; i < NEQ * NEQ; i += G) J[static_cast<size_t>(cell) * NEQ * NEQ + i] = -E[i];
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        if (c < NEQ) f[static_cast<size_t>(cell) * NEQ + c] = out[t];
    }
    __syncwarp();
    const int rw = evaluate<M, G, Tab, K>(1, yy, regime, gl, V);
    load_outputs<G, K>(V, Tab::out(rw), out, gl);
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        if (c < NEQ) f2[static_cast<size_t>(cell) * NEQ + c] = out[t];
    }
}

template <int G>
__global__ void k_diag_coop_lu(int n, const double* __restrict__ A, const double* __restrict__ b, double* LU,
                               int* ipvt, int* info, double* x) {
    using namespace coop;
    constexpr int K = (NEQ + G - 1) / G;
    constexpr int SLOTS = 32 / G;
    extern __shared__ uint64_t sm[];
    const int lane = threadIdx.x & 31, slot = lane / G, gl = lane % G;
    const int warp = threadIdx.x >> 5;
    // the warp's groups run in step: one past the end repeats the last case
    const int cell = min((blockIdx.x * static_cast<int>(blockDim.x >> 5) + warp) * SLOTS + slot, n - 1);
    double* E = reinterpret_cast<double*>(sm) + static_cast<size_t>(warp * SLOTS + slot) * NEQ * NEQ;
    for (int i = gl; i < NEQ * NEQ; i += G) E[i] = A[static_cast<size_t>(cell) * NEQ * NEQ + i];
    __syncwarp();
    uint64_t ip = 0;
    const int inf = lu_coop<G>(E, gl, ip);
    double v[K];
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        v[t] = c < NEQ ? b[static_cast<size_t>(cell) * NEQ + c] : 0.0;
    }
    uint64_t rY[K];
    diag_recips<G, K>(E, rY, gl);
    double v2[K];
#pragma unroll
    for (int t = 0; t < K; ++t) v2[t] = v[t];
    solve_coop<G, K>(E, ip, rY, v2, gl);
#pragma unroll
    for (int t = 0; t < K; ++t) v[t] = inf == 0 ? v2[t] : v[t];
    __syncwarp();
    for (int i = gl; i < NEQ * NEQ; i += G) LU[static_cast<size_t>(cell) * NEQ * NEQ + i] = E[i];
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const int c = gl + t * G;
        if (c < NEQ) {
            x[static_cast<size_t>(cell) * NEQ + c] = v[t];
            ipvt[static_cast<size_t>(cell) * NEQ + c] = static_cast<int>((ip >> (4 * c)) & 15);
        }
    }
    if (gl == 0) info[cell] = inf;
}

}  // namespace wr

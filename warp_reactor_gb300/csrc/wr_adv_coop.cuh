// wr_adv_coop.cuh -- one translation unit per lanes-per-cell count G: the
// generated vector programs of that G (coop_prog_g<G>.h, large initialisers) and
// the cooperative advance kernel instantiated for both math policies.  The unit
// defines WR_COOP_G and includes generated/coop_prog_g<G>.h (which sets the warps
// per block: as many as the block's shared memory holds) before this file.
#include "wr_launch.h"
#include "wr_coop.cuh"
#include "wr_coop_cta32.cuh"

#define WR_CAT2(a, b) a##b
#define WR_CAT(a, b) WR_CAT2(a, b)

namespace wr {

namespace {
namespace cp = WR_CAT(coop, WR_COOP_G);

struct Tab {
    static constexpr int kNV = cp::kNV;
    static constexpr int kNR = cp::kNR;
    static constexpr int kNF = cp::kNF;
    static constexpr int kRegimes = cp::kRegimes;
    static constexpr bool kAdjoint = false;
    static __device__ __forceinline__ const uint64_t* vconst() { return cp::kVConst; }
    static __device__ __forceinline__ const ulonglong2* vfun() { return cp::kVFun; }
    static __device__ __forceinline__ const ulonglong2* prog() { return cp::kProg; }
    static __device__ __forceinline__ const uint64_t* lit() { return cp::kLit; }
    static __device__ __forceinline__ uint32_t ctl(int i) { return cp::kCtl[i]; }
    static __device__ __forceinline__ int first(int w) { return cp::kProgStep[w][0]; }
    static __device__ __forceinline__ int steps(int w) { return cp::kProgStep[w][1]; }
    static __device__ __forceinline__ int sink(int) { return kNV - 1; }
    static __device__ __forceinline__ uint64_t regime(int k, int i) { return cp::kRegimeT[k][i]; }
    static __device__ __forceinline__ const uint16_t* out(int w) { return cp::kOut[w]; }
    static __device__ __forceinline__ const uint16_t* jac(int r) { return cp::kJac[r]; }
};
static_assert(coop::kRes + Tab::kNR + Tab::kNF <= Tab::kNV, "reserved constants lie inside the slot array");

constexpr int kG = WR_COOP_G;
constexpr int kW = cp::kWarps;
constexpr size_t kSmem = static_cast<size_t>(kW) * (32 / kG) * Tab::kNV * 8;
static_assert(kSmem <= 232448, "cooperative advance: shared memory of one block exceeds 227 KiB");
}  // namespace

cudaError_t WR_CAT(configure_advance_coop, WR_COOP_G)() {
    const void* kernels[4] = {reinterpret_cast<const void*>(k_advance_coop<PortableMathCall, kG, kW, Tab, false>),
                              reinterpret_cast<const void*>(k_advance_coop<CudaMath, kG, kW, Tab, false>),
                              reinterpret_cast<const void*>(k_advance_coop<PortableMathCall, kG, kW, Tab, true>),
                              reinterpret_cast<const void*>(k_advance_coop<CudaMath, kG, kW, Tab, true>)};
    for (const void* k : kernels) {
        const cudaError_t e =
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// phases: the 16 phase counters of the instrumented instantiation (nullptr: the
// plain kernel)
cudaError_t WR_CAT(launch_advance_coop, WR_COOP_G)(int math_cuda, int blocks, cudaStream_t stream, DevState s,
                                                   StepCtl* ctl, unsigned long long* phases) {
    if (phases) {
        if (math_cuda)
            k_advance_coop<CudaMath, kG, kW, Tab, true><<<blocks, kW * 32, kSmem, stream>>>(s, ctl, phases);
        else
            k_advance_coop<PortableMathCall, kG, kW, Tab, true><<<blocks, kW * 32, kSmem, stream>>>(s, ctl, phases);
    } else if (math_cuda) {
        k_advance_coop<CudaMath, kG, kW, Tab, false><<<blocks, kW * 32, kSmem, stream>>>(s, ctl, nullptr);
    } else {
        k_advance_coop<PortableMathCall, kG, kW, Tab, false><<<blocks, kW * 32, kSmem, stream>>>(s, ctl, nullptr);
    }
    return cudaGetLastError();
}

// the structured policy's advance at this lane width, a tile on `cluster` SMs
// (wr_launch.h: cta32_shape picks the pair)
namespace {
template <class M, int CL>
struct Cta32Launch {
    void (*kernel)(DevState, StepCtl*) = k_advance_cta32<M, kG, CL, Tab>;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cudaError_t configured;
    explicit Cta32Launch(int blocks) {
        constexpr size_t smem = static_cast<size_t>(kTileCells / CL) * Tab::kNV * 8;
        static_assert(smem + sizeof(TileCtl<kTileCells / CL>) <= 232448,
                      "a tile's block exceeds 227 KiB of shared memory");
        configured = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        cfg.gridDim = dim3(static_cast<unsigned>(blocks));
        cfg.blockDim = dim3(kTileCells / CL * kG);
        cfg.dynamicSmemBytes = smem;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = CL;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = CL > 1 ? 1 : 0;
    }
    Cta32Launch(const Cta32Launch&) = delete;
};
template <class M, int CL>
cudaError_t launch_cta32(int tiles, int sms, cudaStream_t stream, DevState s, StepCtl* ctl) {
    Cta32Launch<M, CL> l(CL == 1 ? (tiles < sms ? tiles : sms) : tiles * CL);
    if (l.configured != cudaSuccess) return l.configured;
    l.cfg.stream = stream;
    const cudaError_t e = cudaLaunchKernelEx(&l.cfg, l.kernel, s, ctl);
    return e == cudaSuccess ? cudaGetLastError() : e;
}
#if WR_COOP_G == 32
template <class M, int CL>
cudaError_t clusters_cta32(int* fit) {
    Cta32Launch<M, CL> l(CL);
    if (l.configured != cudaSuccess) return l.configured;
    return cudaOccupancyMaxActiveClusters(fit, l.kernel, &l.cfg);
}
#endif
}  // namespace
#if WR_COOP_G != 8
cudaError_t WR_CAT(launch_advance_cta32_, WR_COOP_G)(int math_cuda, int cluster, int tiles, int sms,
                                                     cudaStream_t stream, DevState s, StepCtl* ctl) {
#if WR_COOP_G == 16
    (void)cluster;
    return math_cuda ? launch_cta32<CudaMath, 1>(tiles, sms, stream, s, ctl)
                     : launch_cta32<PortableMathCall, 1>(tiles, sms, stream, s, ctl);
#else
    if (cluster == 4)
        return math_cuda ? launch_cta32<CudaMath, 4>(tiles, sms, stream, s, ctl)
                         : launch_cta32<PortableMathCall, 4>(tiles, sms, stream, s, ctl);
    return math_cuda ? launch_cta32<CudaMath, 2>(tiles, sms, stream, s, ctl)
                     : launch_cta32<PortableMathCall, 2>(tiles, sms, stream, s, ctl);
#endif
}
#endif
#if WR_COOP_G == 32
cudaError_t cta32_clusters(int math_cuda, int cluster, int* fit) {
    if (cluster == 4) return math_cuda ? clusters_cta32<CudaMath, 4>(fit) : clusters_cta32<PortableMathCall, 4>(fit);
    return math_cuda ? clusters_cta32<CudaMath, 2>(fit) : clusters_cta32<PortableMathCall, 2>(fit);
}
#endif

namespace {
constexpr int kDiagWarps = 4;
constexpr size_t kDiagNetSmem = static_cast<size_t>(kDiagWarps) * (32 / kG) * Tab::kNV * 8;
constexpr size_t kDiagLuSmem = static_cast<size_t>(kDiagWarps) * (32 / kG) * NEQ * NEQ * 8;
}  // namespace

// diagnostics on device buffers (wr_diag.cu owns the host side)
cudaError_t WR_CAT(diag_coop_network, WR_COOP_G)(int math_cuda, int n, const double* y, double* J, double* f,
                                                 double* f2) {
    const int per_block = kDiagWarps * (32 / kG);
    const int blocks = (n + per_block - 1) / per_block;
    cudaError_t e;
    if (math_cuda) {
        e = cudaFuncSetAttribute(k_diag_coop_network<CudaMath, kG, Tab>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kDiagNetSmem));
        if (e != cudaSuccess) return e;
        k_diag_coop_network<CudaMath, kG, Tab><<<blocks, kDiagWarps * 32, kDiagNetSmem>>>(n, y, J, f, f2);
    } else {
        e = cudaFuncSetAttribute(k_diag_coop_network<PortableMathCall, kG, Tab>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kDiagNetSmem));
        if (e != cudaSuccess) return e;
        k_diag_coop_network<PortableMathCall, kG, Tab><<<blocks, kDiagWarps * 32, kDiagNetSmem>>>(n, y, J, f, f2);
    }
    return cudaGetLastError();
}

cudaError_t WR_CAT(diag_coop_lu, WR_COOP_G)(int n, const double* A, const double* b, double* LU, int* ipvt, int* info,
                                            double* x) {
    const int per_block = kDiagWarps * (32 / kG);
    k_diag_coop_lu<kG><<<(n + per_block - 1) / per_block, kDiagWarps * 32, kDiagLuSmem>>>(n, A, b, LU, ipvt, info, x);
    return cudaGetLastError();
}

}  // namespace wr

// The cooperative advance (csrc/wr_coop.cuh: k_advance_coop) on the CPU, one warp of
// 8, 16 or 32 lanes per cell.  advance <in> <out>: records of 16 doubles (14 number
// densities, T, the timestep) -> records of 23: the burned number densities and energy, the
// seven counters and the launch's failure code.  The programs that the warp ran, in order,
// go to standard output.
#include "warp_threads.h"

// called by Tab::first, which the test has report the program it starts
inline void started(int program) {
    if (threadIdx.x == 0) std::printf("%d\n", program);
}

#include "device_code.h"

namespace wr {
uint64_t sm[64 * 1200];
}

int main(int argc, char** argv) {
    using namespace wr;
    constexpr int G = cp::kG;
    if (argc != 3) return 2;
    FILE* f = std::fopen(argv[1], "rb");
    std::vector<double> in(16 * 1024);
    const int n = static_cast<int>(std::fread(in.data(), 16 * sizeof(double), 1024, f));
    std::fclose(f);
    std::vector<double> T(n), e(n), xn(NS * n), dt(n);
    std::vector<int> order(n), bucket(n, kQBurn), cost(n);
    std::vector<uint64_t> stats(7 * n);
    for (int i = 0; i < n; ++i) {
        double x[NS];
        for (int k = 0; k < NS; ++k) x[k] = xn[k * n + i] = in[16 * i + k];
        T[i] = in[16 * i + NS];
        dt[i] = in[16 * i + NS + 1];
        e[i] = eos_e_from_T(x, T[i]);
        order[i] = i;
    }
    DevState s{};
    s.T = T.data(), s.e = e.data(), s.xn = xn.data(), s.local_dt = dt.data();
    s.order = order.data(), s.qbucket = bucket.data(), s.cost = cost.data(), s.stats = stats.data();
    s.n = n;
    StepCtl ctl{};
    ctl.queued = static_cast<unsigned>(n);
    ctl.failure = WR_SUCCESS;
    slots = sm;
    warp::is_sink = [](uint32_t addr) { return addr / 8 % Tab::kNV == Tab::kNV - 1; };
    warp::launch([&] { k_advance_coop<PortableMathCall, G, 1, Tab>(s, &ctl, nullptr); });
    f = std::fopen(argv[2], "wb");
    for (int i = 0; i < n; ++i) {
        double out[23];
        for (int k = 0; k < NS; ++k) out[k] = xn[k * n + i];
        out[NS] = e[i];
        for (int k = 0; k < 7; ++k) out[NS + 1 + k] = static_cast<double>(stats[k * n + i]);
        out[22] = ctl.failure;
        std::fwrite(out, sizeof(double), 23, f);
    }
    std::fclose(f);
    return 0;
}

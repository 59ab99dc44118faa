// The structured policy's advance (csrc/wr_coop_cta32.cuh: k_advance_cta32) on the CPU, one
// block of 16 warps, 16 lanes per cell, a tile of 32 cells after the other.
// tiles <dt> <in> <out>: the cells' records, advanced by one outer step of dt; then the
// failure code and the number of cells integrated on standard output.
#include "warp_threads.h"

#include "device_code.h"

namespace wr {
uint64_t sm[32 * 1024];
}

int main(int argc, char** argv) {
    using namespace wr;
    if (argc != 4) return 2;
    std::vector<wr_collapse_state> c(1024);
    FILE* f = std::fopen(argv[2], "rb");
    const int n = static_cast<int>(std::fread(c.data(), sizeof c[0], c.size(), f));
    std::fclose(f);
    std::vector<double> rho(n), T(n), e(n), xn(NS * n), time(n), driver(n);
    std::vector<int> steps(n);
    std::vector<uint64_t> stats(7 * n);
    for (int i = 0; i < n; ++i) {
        rho[i] = c[i].rho, T[i] = c[i].T, e[i] = c[i].e, time[i] = c[i].time, driver[i] = c[i].density_driver;
        steps[i] = c[i].completed_steps;
        for (int k = 0; k < NS; ++k) xn[k * n + i] = c[i].xn[k];
    }
    DevState s{};
    s.n = n;
    s.rho = rho.data(), s.T = T.data(), s.e = e.data(), s.xn = xn.data(), s.time = time.data();
    s.driver = driver.data(), s.steps = steps.data(), s.stats = stats.data();
    StepCtl ctl{};
    ctl.failure = WR_SUCCESS;
    ctl.dt_grid = ctl.next_grid_time = std::strtod(argv[1], nullptr);
    slots = sm;
    warp::is_sink = [](uint32_t addr) { return addr / 8 % Tab::kNV == Tab::kNV - 1; };
    warp::launch([&] { k_advance_cta32<PortableMathCall, 16, 1, Tab>(s, &ctl); }, 16);
    f = std::fopen(argv[3], "wb");
    for (int i = 0; i < n; ++i) {
        c[i].rho = rho[i], c[i].T = T[i], c[i].e = e[i], c[i].time = time[i], c[i].density_driver = driver[i];
        c[i].completed_steps = steps[i];
        for (int k = 0; k < NS; ++k) c[i].xn[k] = xn[k * n + i];
        const uint64_t* st = &stats[i];
        c[i].stats = {st[0], st[n], st[2 * n], st[3 * n], st[4 * n], st[5 * n], st[6 * n]};
        std::fwrite(&c[i], sizeof c[i], 1, f);
    }
    std::fclose(f);
    std::printf("%d %d\n", ctl.failure, ctl.integrated);
    return 0;
}

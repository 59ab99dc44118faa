// The differentiation form's kernels (csrc/wr_diff_coop.cu: k_diff_forward and, with
// "adjoint", k_diff_backward) on the CPU, one warp.  gradient forward|adjoint <in> <out>:
// n, the number of outer steps, the timesteps, the multipliers, the cells' records and qbar
// (n x 15) -> per cell q (15), the adjoint of u (15) and of the multipliers.
#include "warp_threads.h"

// the lane's running program, which the test has Tab::first report
inline thread_local int program;

#include "device_code.h"

namespace wr {
namespace diff {
namespace {
uint64_t sm[4096];
}
}  // namespace diff
}  // namespace wr

int main(int argc, char** argv) {
    using namespace wr::diff;
    if (argc != 4) return 2;
    const bool adjoint = std::strcmp(argv[1], "adjoint") == 0;
    FILE* f = std::fopen(argv[2], "rb");
    int head[2];
    bool ok = std::fread(head, sizeof head, 1, f) == 1;
    const int n = head[0], steps = head[1], cap = 256;
    std::vector<double> dt(steps), mult(NP);
    std::vector<wr_collapse_state> cells(n);
    ok = ok && std::fread(dt.data(), sizeof(double), steps, f) == dt.size();
    ok = ok && std::fread(mult.data(), sizeof(double), NP, f) == mult.size();
    ok = ok && std::fread(cells.data(), sizeof(wr_collapse_state), n, f) == cells.size();
    std::vector<double> qbar(15 * n);
    ok = ok && std::fread(qbar.data(), sizeof(double), 15 * n, f) == qbar.size();
    std::fclose(f);
    if (!ok) return 3;
    Args a{};
    a.cells = cells.data(), a.mult = mult.data(), a.dt_hist = dt.data();
    a.nsteps = steps, a.n = n, a.cap = cap, a.nseg = cap / kSeg + 1;
    std::vector<double> ckpt(steps * kFields * n), hbuf(n * cap), q(15 * n), ubar(15 * n),
        segck(n * a.nseg * wr::NEQ), ys(n * kSeg * wr::NEQ), stage(n * kSeg * kStage), mbar(n * NP);
    std::vector<int> counts(steps * n), status(n);
    std::vector<unsigned char> kind(steps * n);
    int queue = 0;
    a.ckpt = ckpt.data(), a.counts = counts.data(), a.kind = kind.data(), a.hbuf = hbuf.data();
    a.q = q.data(), a.status = status.data(), a.queue = &queue, a.qbar = qbar.data(), a.ubar = ubar.data();
    a.segck = segck.data(), a.ys = ys.data(), a.stage = stage.data(), a.mbar = mbar.data();
    slots = sm;
    warp::is_sink = [](uint32_t addr) { return addr / 8 == Tab::kNV - 1; };
    warp::launch([&] { k_diff_forward(a); });
    for (int s : status)
        if (s != WR_SUCCESS) return 4;
    if (adjoint) {
        queue = 0;
        // the burn's replay runs the forward programs, whose sink is the smaller array's
        warp::is_sink = [](uint32_t addr) {
            return addr / 8 == (program < 2 * Tab::kRegimes ? Tab::kNV : cd::kNVA) - 1;
        };
        warp::launch([&] { k_diff_backward(a); });
    }
    f = std::fopen(argv[3], "wb");
    for (int i = 0; i < n; ++i) {
        std::fwrite(&q[15 * i], sizeof(double), 15, f);
        std::fwrite(&ubar[15 * i], sizeof(double), 15, f);
        std::fwrite(&mbar[NP * i], sizeof(double), NP, f);
    }
    std::fclose(f);
    return 0;
}

// The step-size controller (csrc/wr_coop.cuh: step_sizes) on the CPU, one warp, one cell.
// controller <err> <erracc> <hacc> <h>: the two step sizes and the lanes' divisions that
// left the integer path.
#include "warp_threads.h"

#include "wr_coop.cuh"

int main(int argc, char** argv) {
    if (argc != 5) return 2;
    double in[4], hnew[2][32], hgus[2][32];
    for (int k = 0; k < 4; ++k) in[k] = std::strtod(argv[k + 1], nullptr);
    std::atomic<int> native{0};
    warp::launch([&] {
        const int l = warp::lane();
        wr::step_sizes<16, false>(in[0], in[1], in[2], in[3], l % 16, wr::PortableMathCall::cbrt, hnew[0][l], hgus[0][l]);
        wr::step_sizes<32, true>(in[0], in[1], in[2], in[3], l, wr::PortableMathCall::cbrt, hnew[1][l], hgus[1][l]);
        native += native_divisions;
    });
    for (int k = 0; k < 2; ++k)
        for (int l = 0; l < 32; ++l) std::printf("%a %a\n", hnew[k][l], hgus[k][l]);
    std::printf("%d\n", native.load());
    return 0;
}

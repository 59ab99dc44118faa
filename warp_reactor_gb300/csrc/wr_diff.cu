// wr_diff.cu -- differentiation form: C ABI (the map and its storage are described in
// wr_diff.cuh, the kernels are in wr_diff_coop.cu).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>

#include "wr_diff.cuh"
#include "wr_launch.h"

namespace wr {
namespace diff {

__global__ void k_diff_mult(const double* logm, double* mult) {
    const int r = threadIdx.x;
    if (r < NP) mult[r] = logm ? M::exp(logm[r]) : 1.0;
}

// pbar[r] = mult[r] * sum over cells (in cell order) of mbar[cell][r]
__global__ void k_diff_reduce(const double* mbar, const double* mult, int n, double* pbar) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= NP) return;
    double acc = 0.0;
#pragma unroll 16  // the sums are serial, their loads need not be
    for (int i = 0; i < n; ++i) acc += mbar[static_cast<size_t>(i) * NP + r];
    pbar[r] = acc * mult[r];
}

}  // namespace diff
}  // namespace wr

// ------------------------------------------------------------------ C-ABI
struct wr_diff {
    int n = 0, max_steps = 0, cap = 0, nseg = 0, device = 0;
    int nsteps = 0, perturb = 0, sms = 1;
    bool have_forward = false;
    cudaStream_t stream = nullptr;
    double* ckpt = nullptr;
    int* counts = nullptr;
    unsigned char* kind = nullptr;
    double* hbuf = nullptr;
    double* segck = nullptr;
    double* ys = nullptr;
    double* stage = nullptr;
    double* mbar = nullptr;
    double* mult = nullptr;
    double* dt_hist = nullptr;
    int* status = nullptr;
    int* queue = nullptr;
    const wr_collapse_state* cells = nullptr;  // the caller's records of the last forward
    const double* u = nullptr;
    std::string error;
};

namespace {

int fail(wr_diff* d, const std::string& msg, int code = WR_BAD_INPUTS) {
    if (d) d->error = msg;
    return code;
}

bool cuda_ok(wr_diff* d, cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    cudaGetLastError();  // reported here: not the next launch check's
    if (d) d->error = std::string(what) + ": " + cudaGetErrorString(e);
    return false;
}

wr::diff::Args make_args(wr_diff* d) {
    wr::diff::Args a{};
    a.cells = d->cells;
    a.u = d->u;
    a.mult = d->mult;
    a.dt_hist = d->dt_hist;
    a.nsteps = d->nsteps;
    a.perturb = d->perturb;
    a.n = d->n;
    a.cap = d->cap;
    a.nseg = d->nseg;
    a.ckpt = d->ckpt;
    a.counts = d->counts;
    a.kind = d->kind;
    a.hbuf = d->hbuf;
    a.segck = d->segck;
    a.ys = d->ys;
    a.stage = d->stage;
    a.mbar = d->mbar;
    a.status = d->status;
    a.queue = d->queue;
    return a;
}

}  // namespace

extern "C" {

int wr_diff_num_multipliers(void) { return wr::diff::NP; }

wr_diff* wr_diff_create(int num_cells, int max_outer_steps, int max_accepted_per_cell, int device) {
    if (num_cells <= 0 || max_outer_steps <= 0 || max_accepted_per_cell <= 0) return nullptr;
    wr_diff* d = new wr_diff();
    d->n = num_cells;
    d->max_steps = max_outer_steps;
    d->cap = max_accepted_per_cell;
    d->nseg = (max_accepted_per_cell + wr::diff::kSeg - 1) / wr::diff::kSeg + 1;
    d->device = device;
    const size_t n = static_cast<size_t>(num_cells);
    const size_t S = static_cast<size_t>(max_outer_steps);
    bool ok = cuda_ok(d, cudaSetDevice(device), "cudaSetDevice") &&
              cuda_ok(d, cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking), "cudaStreamCreate") &&
              cuda_ok(d, cudaMalloc(&d->ckpt, S * wr::diff::kFields * n * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->counts, S * n * sizeof(int)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->kind, S * n), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->hbuf, n * d->cap * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->segck, n * d->nseg * wr::NEQ * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->ys, n * wr::diff::kSeg * wr::NEQ * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->stage, n * wr::diff::kSeg * wr::diff::kStage * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->mbar, n * wr::diff::NP * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->mult, wr::diff::NP * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->dt_hist, S * sizeof(double)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->status, n * sizeof(int)), "cudaMalloc") &&
              cuda_ok(d, cudaMalloc(&d->queue, sizeof(int)), "cudaMalloc") &&
              cuda_ok(d, cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, device), "device query");
    if (!ok) {
        fprintf(stderr, "wr_diff_create: %s\n", d->error.c_str());
        wr_diff_destroy(d);
        return nullptr;
    }
    return d;
}

void wr_diff_destroy(wr_diff* d) {
    if (!d) return;
    cudaFree(d->ckpt);
    cudaFree(d->counts);
    cudaFree(d->kind);
    cudaFree(d->hbuf);
    cudaFree(d->segck);
    cudaFree(d->ys);
    cudaFree(d->stage);
    cudaFree(d->mbar);
    cudaFree(d->mult);
    cudaFree(d->dt_hist);
    cudaFree(d->status);
    cudaFree(d->queue);
    if (d->stream) cudaStreamDestroy(d->stream);
    delete d;
}

const char* wr_diff_last_error(wr_diff* d) { return d ? d->error.c_str() : "null context"; }

int wr_diff_forward(wr_diff* d, const wr_collapse_state* d_cells, const double* d_u, const double* d_log_mult,
                    const double* dt_hist, int nsteps, int perturb, double* d_q) {
    if (!d) return WR_BAD_INPUTS;
    if (!d_cells || !dt_hist || !d_q) return fail(d, "null pointer argument");
    if (nsteps <= 0 || nsteps > d->max_steps) return fail(d, "nsteps outside 1..max_outer_steps");
    for (int s = 0; s < nsteps; ++s)
        if (!(dt_hist[s] > 0.0) || !std::isfinite(dt_hist[s])) return fail(d, "dt_hist holds a non-positive step");
    if (!cuda_ok(d, cudaSetDevice(d->device), "cudaSetDevice")) return WR_BAD_INPUTS;
    d->cells = d_cells;
    d->u = d_u;
    d->nsteps = nsteps;
    d->perturb = perturb ? 1 : 0;
    d->have_forward = false;
    if (!cuda_ok(d, cudaMemcpyAsync(d->dt_hist, dt_hist, nsteps * sizeof(double), cudaMemcpyHostToDevice,
                                    d->stream), "cudaMemcpyAsync"))
        return WR_BAD_INPUTS;
    wr::diff::k_diff_mult<<<1, 64, 0, d->stream>>>(d_log_mult, d->mult);
    wr::diff::Args a = make_args(d);
    a.q = d_q;
    if (!cuda_ok(d, wr::diff::launch_diff_forward(a, d->sms, d->stream), "k_diff_forward launch")) return WR_BAD_INPUTS;
    wr::count_launches(2);
    if (!cuda_ok(d, cudaStreamSynchronize(d->stream), "k_diff_forward")) return WR_BAD_INPUTS;
    // first failing cell in index order decides the result
    int* st = new int[d->n];
    const bool got = cuda_ok(d, cudaMemcpy(st, d->status, d->n * sizeof(int), cudaMemcpyDeviceToHost), "cudaMemcpy");
    int result = got ? WR_SUCCESS : WR_BAD_INPUTS;
    for (int i = 0; got && i < d->n; ++i)
        if (st[i] != WR_SUCCESS) {
            result = st[i];
            d->error = "cell " + std::to_string(i) + " failed with code " + std::to_string(st[i]);
            break;
        }
    delete[] st;
    d->have_forward = result == WR_SUCCESS;
    return result;
}

int wr_diff_backward(wr_diff* d, const double* d_qbar, double* d_ubar, double* d_pbar) {
    if (!d) return WR_BAD_INPUTS;
    if (!d->have_forward) return fail(d, "wr_diff_backward needs a successful wr_diff_forward first");
    if (!d_qbar || !d_ubar || !d_pbar) return fail(d, "null pointer argument");
    if (!cuda_ok(d, cudaSetDevice(d->device), "cudaSetDevice")) return WR_BAD_INPUTS;
    wr::diff::Args a = make_args(d);
    a.qbar = d_qbar;
    a.ubar = d_ubar;
    if (!cuda_ok(d, wr::diff::launch_diff_backward(a, d->sms, d->stream), "k_diff_backward launch"))
        return WR_BAD_INPUTS;
    wr::diff::k_diff_reduce<<<1, 64, 0, d->stream>>>(d->mbar, d->mult, d->n, d_pbar);
    wr::count_launches(2);
    if (!cuda_ok(d, cudaStreamSynchronize(d->stream), "k_diff_backward")) return WR_BAD_INPUTS;
    return WR_SUCCESS;
}

int wr_diff_record(wr_diff* d, double* h_hbuf, int* h_counts) {
    if (!d || !d->have_forward || !h_hbuf || !h_counts) return WR_BAD_INPUTS;
    const size_t n = static_cast<size_t>(d->n);
    if (!cuda_ok(d, cudaMemcpy(h_hbuf, d->hbuf, n * d->cap * sizeof(double), cudaMemcpyDeviceToHost), "cudaMemcpy"))
        return WR_BAD_INPUTS;
    // counts are stored [S][n]; the host copy is [n][S]
    int* tmp = new int[static_cast<size_t>(d->nsteps) * n];
    const bool ok = cuda_ok(d, cudaMemcpy(tmp, d->counts, static_cast<size_t>(d->nsteps) * n * sizeof(int),
                                          cudaMemcpyDeviceToHost), "cudaMemcpy");
    if (ok)
        for (size_t i = 0; i < n; ++i)
            for (int s = 0; s < d->nsteps; ++s) h_counts[i * d->nsteps + s] = tmp[static_cast<size_t>(s) * n + i];
    delete[] tmp;
    return ok ? WR_SUCCESS : WR_BAD_INPUTS;
}

}  // extern "C"


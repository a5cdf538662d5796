// resident.cuh -- a whole CG / BiCGSTAB solve (FP64 or mixed) in one cooperative
// launch, for systems whose product and ring fit the SMs' shared memory.
// Implemented in resident.cu.
#pragma once

#include <mutex>

#include "krylov.cuh"

namespace pfg {

// Scalars of a resident solve between two launches (a launch stops after
// `budget` iterations so that no kernel runs for seconds).
struct ResState {
    int phase;    // 0: start from the residual of x, 1: inside the iteration, 2: finished
    int status;   // PFG_OK, PFG_E_BREAKDOWN, PFG_E_NONFINITE, PFG_W_NOT_CONVERGED
    int fallback; // mixed: the caller finishes in FP64
    int iter, restart, replacements, breakdowns, poisoned, failures, stall, first, parity;
    double rho, beta, c2, c3, rr, rr1, bb, true_rr;
    double rel, prev_rel, best_rel;
    float rmax32, rmin32;
    int err;         // raised when a wait runs out
    unsigned round;  // exchanges made by the last launch and those whose slots it took over
};

// What every resident kernel reads: matrices, the published (gathered) vectors
// and the vectors that outlive a launch, all in global memory.
struct ResArgs {
    SellView<double> A64;
    SellView<float> A32;
    const int *bounds;  // first slice of each CTA's share (ctas + 1)
    const double *b;
    double *x, *xb;
    // published vectors, 4 entries per block row of a 3x3-block system: FP64 p (CG)
    // or M^-1 p and M^-1 e; FP32 z and the two p in turn (CG) or M^-1 p and M^-1 e
    double *pub64[2];
    float *pub32[3];
    void *home;  // own vectors of every CTA, those not in shared memory
    const double *dinv64;
    const float *dinv32;
    ResState *st;
    double *slots;   // set by run_resident_kernel, as is:
    unsigned round;  // the first round of the launch
    int pc, stop_rule, itrmax, budget, stages, near;
    double er0, tol, delta;
};

// The shared memory of a resident solve: `stages` ring stages per warp and the
// first `near` of its own vectors.  ctas == 0: it does not fit.
struct ResPlan {
    int ctas = 0, stages = 0, near = 0, vectors = 0;
    size_t smem = 0, home_bytes = 0;
};

constexpr int kResRounds = 8;    // exchange buffers in rotation
constexpr int kResValues = 2;    // most values of one exchange
constexpr int kResMaxCtas = 160;
constexpr size_t kResSlots = (size_t)kResRounds * kResValues * kResMaxCtas * kResMaxCtas;

// What the resident solves of a device share: the exchange slots, 3.3 MB, and their order.
// One grid whose CTAs wait for one another at a time (each fills the device: two that
// held half the SMs each would wait until their limits).  The order is made on the
// device, launch by launch: a launch waits in its stream for the end of the one before,
// whichever thread's that was, and no thread waits for another solve on the host.  Several
// threads' solves so alternate after at most one launch each (4,096 iterations), and
// those on different devices do not meet.  Held by the handles that have solved resident;
// the last one gives it back.
struct ResDevice {
    std::mutex mu;
    cudaEvent_t last = nullptr;  // end of the last launch
    int in_flight = 0;           // launches whose threads have not seen their end
    uint64_t launches = 0;
    DevBuf<double> slots;
    // what the last launch left: inboxes ready for this round of a grid of as many CTAs
    // (0: not known, or not well)
    int ready_ctas = 0;
    unsigned ready_round = 0;
    ~ResDevice()
    {
        if (last) cudaEventDestroy(last);
    }
    static std::shared_ptr<ResDevice> current();
};

// Cuts the sliced matrix into one run of slices per CTA with about equal work
// (once per pattern and number of CTAs: A.share, A.share_ctas, A.share_max).  ctas 0: one
// for every SM.
void share_slices(DevMatrix &A, int ctas, cudaStream_t st);

ResPlan plan_resident(const DevMatrix &A, int algorithm, bool mixed, bool precond);

// Runs the solve from the state *host (page-locked; copied to a.st) until it is
// finished, several launches if need be; *host then holds the final state.
// Returns the launches made; 0 where the device does not hold the grid at once (it may
// give a process fewer SMs than it has): x is as it was.  debug: the state after each
// launch on stderr.
int run_resident_kernel(ResDevice &dev, const ResPlan &pl, ResArgs a, int bs, int algorithm, bool mixed,
                        ResState *host, bool debug, cudaStream_t st);

}  // namespace pfg

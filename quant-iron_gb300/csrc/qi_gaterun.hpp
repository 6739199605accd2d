// qi_gaterun.hpp — runs of per-gate operations applied many to a pass (qi_gaterun.cu).
#pragma once
#include "qi_plan.hpp"

#include <complex>
#include <vector>

namespace qi {

// Whether the passes can apply this gate or Pauli exponential.
bool run_supported(int n, int prec, const Elem &e);
// Schedule elems (all run_supported) into passes appended to seg, their programs to prog.
void schedule_run(int n, int prec, const std::vector<const Elem *> &elems, RunSegment &seg, std::vector<uint8_t> &prog);
Status launch_run_pass(qi_state *s, const RunPass &p, const void *d_prog);

// Reverse sweep of an adjoint gradient (qi_adjrun.cu): gates in sweep order, each un-applied to psi and
// lambda; a parametric one first adds its derivative term.
enum SweepDer : int { kDerX = 1, kDerY = 2, kDerZ = 3, kDerP = 4 };
constexpr int kSweepTerms = 128;    // derivative terms of a pass
constexpr int kSweepPhases = 24;
struct SweepGate {
    const GateMatrix *g;
    int slot;                       // of the derivative term, -1: fixed gate
};
struct SweepPass {
    RunPass run;
    std::vector<int32_t> slot;      // of each term, in program order
    std::vector<double> size2;      // |scale|^2 of what the terms leave out
};
bool sweep_supported(int n, int prec, const GateMatrix &g, int nparams);
void schedule_sweep(int n, int prec, const std::vector<SweepGate> &gates, std::vector<SweepPass> &passes,
                    std::vector<uint8_t> &prog);
// One pass on psi and lambda; the terms' sums (Re <lambda| dU U^dagger |psi> = factor * sum) go to
// out[0 .. terms), partials: workspace of kSweepBlocks * kSweepTerms doubles.
constexpr int kSweepBlocks = 608;
Status launch_sweep_pass(qi_state *psi, void *lam, const SweepPass &p, const void *d_prog, double *partials, double *out);

// Host execution of a pass's FP64 program on 2^n amplitudes (a check of schedule and program).
void replay_run_pass(int n, const RunPass &p, const uint8_t *prog, std::complex<double> *amps);

}  // namespace qi

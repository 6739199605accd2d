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
// Host execution of a pass's FP64 program on 2^n amplitudes (a check of schedule and program).
void replay_run_pass(int n, const RunPass &p, const uint8_t *prog, std::complex<double> *amps);

}  // namespace qi

// qi_plan.hpp — plan structures shared by the planner, the cost model and
// the adjoint-gradient driver.
#pragma once
#include "qi_internal.hpp"

#include <complex>
#include <cstdint>
#include <mutex>
#include <vector>

namespace qi {

// A validated gate (or Pauli exponential) as the fuser sees it.
struct Elem {
    GateMatrix gm;
    uint64_t mask = 0;      // support: targets and controls
    bool diagonal = false;
    bool fusable = false;   // may join a dense block
    bool pauli = false;
    int src = -1;           // index in the caller's gate list
};

struct Block {
    std::vector<int> members;   // element indices, in application order
    uint64_t mask = 0;          // qubits of the block
    bool single = false;        // lowered as one per-gate op
    bool perm = false;          // a run of SWAP / X gates lowered as one qubit permutation
};

std::vector<Block> greedy_partition(const std::vector<Elem> &elems, int n, int kmax);
// Greedy over candidate blocks: the light-cone block of the first remaining element
// (taken as is when it is all-diagonal), and everything each window of kmax
// consecutive qubits can absorb; the candidate with the most elements wins.
std::vector<Block> window_partition(const std::vector<Elem> &elems, int n, int kmax);
// The light-cone block of the first remaining element (at most kmax qubits), and everything the
// qubit window W can absorb from the remaining elements (order and commutation respected).
Block light_cone_block(const std::vector<Elem> &elems, const std::vector<int> &remaining, int n, int kmax);
Block window_block(const std::vector<Elem> &elems, const std::vector<int> &remaining, uint64_t W);
void compose_block(const std::vector<Elem> &elems, const Block &b, std::vector<int> &qubits,
                   std::vector<std::complex<double>> &B);

// One pass of a run of per-gate operations (qi_gaterun.cu): the local qubits (ascending) and the
// byte range of its program.
struct RunPass {
    int32_t tbits = 0;          // local amplitude bits (tile of 2^tbits amplitudes)
    int32_t low = 0;            // qubits 0 .. low-1 are local: contiguous runs of 2^low amplitudes
    int8_t pos[16] = {0};
    int32_t nphase = 0;
    int32_t prog_off = 0, prog_bytes = 0;   // into the plan's run program (16-byte multiples)
    std::vector<uint16_t> slot_at;          // 16-byte units (from prog_off) of the operations with a tile factor
};
// A step of a per-gate plan's execution: the passes of a run of operations, or one operation.
struct RunSegment {
    int32_t op = -1;            // index into the plan's ops; -1: passes
    std::vector<RunPass> passes;
};

// Blocks composed on the device (qi_compose.cu): a matrix per block, members multiplied on from the left.
struct ComposeMember {
    uint32_t off;               // its matrix: 2^m x 2^m complex numbers from this one of the data
    uint8_t m, pos[6];          // local bits of the block it acts on
    uint8_t pad[5];
};
struct ComposeBlock {
    uint64_t tc;                // operand blocks: word of the plan's device words
    uint32_t first, count;      // members
    uint32_t k, pad;
};
static_assert(sizeof(ComposeMember) == 16 && sizeof(ComposeBlock) == 24, "read as such by the device");
struct ComposeJobs {
    std::vector<ComposeBlock> blocks;
    std::vector<ComposeMember> members;
    std::vector<std::complex<double>> data;
    std::vector<size_t> ops;    // the blocks' ops
    size_t at_blocks = 0, at_members = 0, at_data = 0;   // words
    size_t words = 0;           // of the operand blocks
};

}  // namespace qi

struct qi_plan {
    int32_t n = 0;
    int32_t prec = QI_F32;
    qi_exec_options opts = {QI_FUSION_NONE, 0, 0, 0};
    std::vector<qi::Op> ops;
    std::vector<std::complex<double>> mats;   // block matrices / phase tables (host copy, FP64)
    void *d_mats = nullptr;                   // same, in the plan's precision
    std::vector<float> tc;                    // FP32 device blocks: tensor-core operands (fused ops, k >= 5)
                                              // and phase-polynomial blocks, as raw 32-bit words
    void *d_tc = nullptr;
    // A plan for one state's use in one call: operand blocks are composed on the device, before the first
    // execution; its ops have no host matrices.
    bool device_blocks = false, composed = false;
    qi::ComposeJobs compose;
    std::vector<qi::PhasePoly> polys;         // host copy of each OP_PHASE_POLY op (op.mat_offset indexes it)
    // Per-gate plans: how the ops are executed (several to a pass), and the passes' programs.
    std::vector<qi::RunSegment> sched;
    std::vector<uint8_t> run_prog;
    void *d_run = nullptr;        // the programs on device run_device, once executed there
    bool run_normalise = false;   // a renormalisation follows the runs
    // ops not made yet (every op is in a run): what they are made from
    bool lazy = false;
    int32_t run_min = 10, run_max = 12;   // qubits of an FP32 fused plan that executes as gate runs
    std::vector<qi::Elem> lazy_elems;
    std::vector<qi::Block> lazy_blocks;
    int32_t run_device = -1;
    bool run_borrowed = false;    // d_run is a state's workspace
    std::mutex run_mu;            // first use
    qi_plan_stats stats = {};
    std::vector<qi::Block> partition_override;   // set by callers that chose the partition
    bool learned_blocks = false;                 // QI_FUSION_LEARNED chose the model-scored partition
};

namespace qi {
Status build_plan(qi_plan *p, std::vector<Elem> &elems);
Status upload_plan(qi_plan *p);
void finish_compose(qi_plan *p);
Status launch_compose(qi_plan *p, qi_state *s);
void release_runs(qi_plan *p);
Status plan_execute(qi_plan *p, qi_state *s);
Status plan_elems_from_gates(int n, const qi_gate *gates, int64_t ng, const double *theta, int64_t ntheta,
                             std::vector<Elem> &elems);
// Partition choice for QI_FUSION_GREEDY / QI_FUSION_LEARNED (qi_costmodel.cu).
std::vector<Block> choose_partition(qi_plan *p, const std::vector<Elem> &elems, int kmax);
// QI_FUSION_LEARNED: best (k, tensor cores) by the trained cost model (k = 1: one kernel per gate);
// false when no trained model is loaded.  *ms_out = predicted device time of the chosen plan.
bool learned_choice(qi_plan *p, const std::vector<Elem> &elems, int kmax, int *k_out, int *tc_out, double *ms_out);
Elem pauli_exp_elem(const qi_pauli_term &t, double far, double fai, int src);
// Plan element of one gate matrix (support, diagonal and fusable flags).
Elem make_elem_from_gate(const GateMatrix &gm, int src);
}  // namespace qi

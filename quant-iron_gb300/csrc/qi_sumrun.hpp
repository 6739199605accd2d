// qi_sumrun.hpp — SumOp expectation and apply, many X-mask groups to a pass (qi_sumrun.cu).
#pragma once
#include "qi_plan.hpp"

#include <vector>

namespace qi {

struct SumTerm {
    uint64_t z;
    double re, im;   // coefficient times (-i)^(number of Y)
};
struct SumGroup {    // terms that share an X mask
    uint64_t x;
    std::vector<SumTerm> terms;
};

struct SumPass {
    RunPass tile;                   // tile.prog_off / prog_bytes: the pass's program
    int32_t ndiag = 0;              // distinct local Z masks of the diagonal terms
    int32_t nterm = 0;              // diagonal terms
    int32_t diag_at = 0;            // 16-byte unit of their table (from prog_off)
    bool complex_out = false;       // an expectation with an imaginary part
    bool diag_complex = false;      // its diagonal terms have one
};
// Schedule the groups; false when some group cannot be part of a pass (its index is appended to `left`
// when that is given, and the others are scheduled).
bool schedule_sum(int n, int prec, bool apply, const std::vector<SumGroup> &groups, std::vector<SumPass> &passes,
                  std::vector<uint8_t> &prog, std::vector<int> *left);
// One pass: *partials rows of block sums in s->d_partials (stride 4).
Status launch_sum_expect(qi_state *s, const SumPass &p, const void *d_prog, unsigned *nblocks);
// One pass: out (+)= sum of the pass's groups applied to in (`add`: out holds earlier passes' sums).
Status launch_sum_apply(qi_state *out, const qi_state *in, const SumPass &p, const void *d_prog, bool add);

}  // namespace qi

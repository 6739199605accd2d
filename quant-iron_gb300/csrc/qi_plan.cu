// qi_plan.cu — circuit plans: validation, the gate-fusion pass and execution.
//
// Reference: Circuit::execute (src/circuit.rs:160-172) applies gates one by
// one, each a full copy of the state (Gate::apply, src/components/gate.rs:99-122).
// A plan validates the whole gate list first (so an invalid gate leaves the
// state untouched, as the reference's functional execute does), then lowers
// it to device operations:
//   QI_FUSION_NONE   per gate (the plain per-gate method): one op per gate; runs of
//                    them execute several to a pass, each with its own arithmetic
//                    (qi_gaterun.cu);
//   QI_FUSION_GREEDY the greedy fuser below with block width k;
//   QI_FUSION_LEARNED candidate partitions scored by the learned cost model
//                    (qi_costmodel.cu), greedy as the fallback;
//   QI_FUSION_PAULI_GROUPS per gate, but runs of Pauli exponentials with X-masks
//                    in {0, X} become one grouped pass each (qi_pauli.cu).
//
// Greedy fuser ("light-cone" absorption).  A block starts empty; the
// remaining gates are scanned in order.  A gate joins the block when its
// qubits fit (|Q u S| <= k) and it does not depend on a gate that was passed
// over: passed-over gates block their qubits, except that diagonal gates
// commute with each other, so a diagonal gate may pass over a diagonal gate.
// Every absorbed gate therefore commutes with every passed-over gate it
// overtakes, and the block can run before all of them.
//
// The partition takes, at each step, the best of several such blocks: the
// light-cone block of the first remaining gate, and for every window of k
// consecutive qubits the block of all remaining gates inside the window that
// the same rule admits (window_partition).  The first remaining gate's block
// when it is all-diagonal is kept as is (consecutive diagonal blocks become one
// phase-polynomial pass); otherwise the candidate with the most gates wins.  On
// brickwork circuits the windows grow light-cone diamonds instead of the first
// gate's triangles: the 30-qubit 40-layer benchmark circuit needs 80 dense
// blocks and 8 diagonal runs instead of 142 and 9.
#include "qi_internal.hpp"
#include "qi_plan.hpp"
#include "qi_gaterun.hpp"

#include <algorithm>
#include <cmath>
#include <complex>
#include <thread>

namespace qi {

using cd = std::complex<double>;

// ------------------------------------------------------------ elements ---
Elem make_elem_from_gate(const GateMatrix &gm, int src) {
    Elem e;
    e.src = src;
    e.gm = gm;
    if (gm.measure) {   // a barrier: nothing is fused or reordered across a measurement
        e.mask = ~0ull;
        e.diagonal = false;
        e.fusable = false;
        return e;
    }
    if (gm.pauli) {
        const uint64_t sup = gm.xmask | gm.zmask;
        e.mask = gm.normalise_after ? ~0ull : sup;
        e.diagonal = gm.xmask == 0 && !gm.normalise_after;
        e.fusable = false;   // decided later (dense only if narrow enough)
        e.pauli = true;
        return e;
    }
    uint64_t m = 0;
    for (int j = 0; j < gm.nt; ++j) m |= 1ull << gm.t[j];
    for (int32_t c : gm.controls) m |= 1ull << c;
    e.mask = m;
    e.diagonal = gm.diagonal;
    e.fusable = gm.nt > 0;
    return e;
}

// Dense matrix of an element on its support (sorted qubits of e.mask).
static void dense_of(const Elem &e, std::vector<int> &sup, std::vector<cd> &D) {
    sup.clear();
    for (int q = 0; q < 64; ++q)
        if ((e.mask >> q) & 1ull) sup.push_back(q);
    const int s = (int)sup.size();
    const int dim = 1 << s;
    D.assign((size_t)dim * dim, cd(0, 0));
    auto local = [&](int q) { return (int)(std::find(sup.begin(), sup.end(), q) - sup.begin()); };
    if (e.pauli) {
        // cosh(a) I + sinh(a) P on the support
        uint32_t lx = 0, lz = 0;
        for (int j = 0; j < s; ++j) {
            if ((e.gm.xmask >> sup[j]) & 1ull) lx |= 1u << j;
            if ((e.gm.zmask >> sup[j]) & 1ull) lz |= 1u << j;
        }
        const int ny = __builtin_popcount(lx & lz);
        const cd mi_pow[4] = {cd(1, 0), cd(0, -1), cd(-1, 0), cd(0, 1)};
        const double ar = e.gm.alpha_re, ai = e.gm.alpha_im;
        const cd ch(std::cosh(ar) * std::cos(ai), std::sinh(ar) * std::sin(ai));
        const cd sh(std::sinh(ar) * std::cos(ai), std::cosh(ar) * std::sin(ai));
        for (int o = 0; o < dim; ++o) {
            D[(size_t)o * dim + o] += ch;
            const double sg = (__builtin_popcount(o & lz) & 1) ? -1.0 : 1.0;
            D[(size_t)o * dim + (o ^ lx)] += sh * mi_pow[ny & 3] * sg;
        }
        return;
    }
    const GateMatrix &g = e.gm;
    uint32_t cmask = 0;
    for (int32_t c : g.controls) cmask |= 1u << local(c);
    int tl[2] = {0, 0};
    for (int j = 0; j < g.nt; ++j) tl[j] = local(g.t[j]);
    const int td = 1 << g.nt;
    for (int col = 0; col < dim; ++col) {
        if ((col & cmask) != cmask) { D[(size_t)col * dim + col] = cd(1, 0); continue; }
        int tin = 0;
        for (int j = 0; j < g.nt; ++j) tin |= ((col >> tl[j]) & 1) << j;
        int rest = col;
        for (int j = 0; j < g.nt; ++j) rest &= ~(1 << tl[j]);
        for (int tout = 0; tout < td; ++tout) {
            int row = rest;
            for (int j = 0; j < g.nt; ++j) row |= ((tout >> j) & 1) << tl[j];
            D[(size_t)row * dim + col] = cd(g.m[2 * (tout * td + tin)], g.m[2 * (tout * td + tin) + 1]);
        }
    }
}

// B <- G_embedded * B, B row-major 2^nq x 2^nq, G dense on local positions pos[].
static void left_multiply(std::vector<cd> &B, int nq, const std::vector<int> &pos, const std::vector<cd> &G) {
    const int dim = 1 << nq, s = (int)pos.size(), gd = 1 << s;
    uint32_t smask = 0;
    for (int p : pos) smask |= 1u << p;
    std::vector<int> offs(gd);
    for (int r = 0; r < gd; ++r) {
        int o = 0;
        for (int j = 0; j < s; ++j) o |= ((r >> j) & 1) << pos[j];
        offs[r] = o;
    }
    std::vector<cd> in(gd), out(gd);
    for (int base = 0; base < dim; ++base) {
        if (base & (int)smask) continue;
        for (int col = 0; col < dim; ++col) {
            for (int r = 0; r < gd; ++r) in[r] = B[(size_t)(base | offs[r]) * dim + col];
            for (int r = 0; r < gd; ++r) {
                cd acc(0, 0);
                for (int c = 0; c < gd; ++c) acc += G[(size_t)r * gd + c] * in[c];
                out[r] = acc;
            }
            for (int r = 0; r < gd; ++r) B[(size_t)(base | offs[r]) * dim + col] = out[r];
        }
    }
}

// ---------------------------------------------------------------- fuser ---
// The light-cone block of the first remaining element: scan the remaining
// elements in order, absorbing every one that fits (|Q u S| <= k) and depends
// on no passed-over element.
Block light_cone_block(const std::vector<Elem> &elems, const std::vector<int> &remaining, int n, int kmax) {
    Block b;
    const uint64_t all = n >= 64 ? ~0ull : ((1ull << n) - 1);
    const Elem &first = elems[remaining[0]];
    if (!first.fusable || __builtin_popcountll(first.mask) > kmax) {
        b.members.push_back(remaining[0]);
        b.mask = first.mask;
        b.single = true;
        return b;
    }
    uint64_t Q = 0, blocked_any = 0, blocked_diag = 0;
    for (int idx : remaining) {
        const Elem &e = elems[idx];
        const uint64_t S = e.mask;
        bool can = e.fusable && __builtin_popcountll(S) <= kmax;
        if (can) {
            if (S & blocked_any) can = false;
            else if (!e.diagonal && (S & blocked_diag)) can = false;
            else if (__builtin_popcountll(Q | S) > kmax) can = false;
        }
        if (can) {
            Q |= S;
            b.members.push_back(idx);
        } else {
            if (e.diagonal && e.fusable) blocked_diag |= S;
            else blocked_any |= S;
            if ((blocked_any & all) == all) break;
        }
    }
    b.mask = Q;
    b.single = b.members.size() == 1;
    return b;
}

// Everything the window W can absorb: the remaining elements on qubits inside W
// that depend on no passed-over element (same blocking rule as above).
Block window_block(const std::vector<Elem> &elems, const std::vector<int> &remaining, uint64_t W) {
    Block b;
    uint64_t blocked_any = 0, blocked_diag = 0;
    for (int idx : remaining) {
        const Elem &e = elems[idx];
        const uint64_t S = e.mask;
        bool can = e.fusable && S != 0 && (S & ~W) == 0;
        if (can) {
            if (S & blocked_any) can = false;
            else if (!e.diagonal && (S & blocked_diag)) can = false;
        }
        if (can) {
            b.mask |= S;
            b.members.push_back(idx);
        } else {
            if (e.diagonal && e.fusable) blocked_diag |= S;
            else blocked_any |= S;
            if ((blocked_any & W) == W) break;   // nothing further can enter the window
        }
    }
    b.single = b.members.size() == 1;
    return b;
}

template <typename Pick>
static std::vector<Block> partition_with(const std::vector<Elem> &elems, int n, int kmax, Pick pick) {
    std::vector<Block> blocks;
    std::vector<int> remaining(elems.size());
    for (size_t i = 0; i < elems.size(); ++i) remaining[i] = (int)i;
    std::vector<char> taken(elems.size(), 0);
    while (!remaining.empty()) {
        Block b = pick(remaining);
        for (int idx : b.members) taken[idx] = 1;
        std::vector<int> rest;
        rest.reserve(remaining.size());
        for (int idx : remaining)
            if (!taken[idx]) rest.push_back(idx);
        remaining.swap(rest);
        blocks.push_back(std::move(b));
    }
    return blocks;
}

std::vector<Block> greedy_partition(const std::vector<Elem> &elems, int n, int kmax) {
    return partition_with(elems, n, kmax,
                          [&](const std::vector<int> &rem) { return light_cone_block(elems, rem, n, kmax); });
}

std::vector<Block> window_partition(const std::vector<Elem> &elems, int n, int kmax) {
    return partition_with(elems, n, kmax, [&](const std::vector<int> &rem) {
        Block best = light_cone_block(elems, rem, n, kmax);
        if (best.single) return best;
        bool diag = true;
        for (int idx : best.members) diag = diag && elems[idx].diagonal;
        if (diag) return best;   // joins (or starts) a run of diagonal blocks: one phase-polynomial pass
        const uint64_t win = (1ull << kmax) - 1;
        for (int a = 0; a + kmax <= n; ++a) {
            Block w = window_block(elems, rem, win << a);
            if (w.members.size() > best.members.size()) best = std::move(w);
        }
        return best;
    });
}

// A block's members for the device's composition, on its qubits and those of `padded`.
static void compose_job(const std::vector<Elem> &elems, const Block &b, uint64_t padded, ComposeJobs &jobs) {
    ComposeBlock job = {};
    job.first = (uint32_t)jobs.members.size();
    job.count = (uint32_t)b.members.size();
    job.k = (uint32_t)__builtin_popcountll(padded);
    job.tc = jobs.words;
    std::vector<int> sup;
    std::vector<cd> D;
    for (int idx : b.members) {
        dense_of(elems[idx], sup, D);
        ComposeMember m = {};
        m.off = (uint32_t)jobs.data.size();
        m.m = (uint8_t)sup.size();
        for (size_t j = 0; j < sup.size(); ++j) m.pos[j] = (uint8_t)__builtin_popcountll(padded & ((1ull << sup[j]) - 1));
        jobs.members.push_back(m);
        jobs.data.insert(jobs.data.end(), D.begin(), D.end());
    }
    jobs.blocks.push_back(job);
    jobs.words += (size_t)6 << (2 * job.k);
}

// Dense (or diagonal) matrix of a block on its sorted qubits.
void compose_block(const std::vector<Elem> &elems, const Block &b, std::vector<int> &qubits, std::vector<cd> &B) {
    qubits.clear();
    for (int q = 0; q < 64; ++q)
        if ((b.mask >> q) & 1ull) qubits.push_back(q);
    const int nq = (int)qubits.size();
    const int dim = 1 << nq;
    B.assign((size_t)dim * dim, cd(0, 0));
    for (int i = 0; i < dim; ++i) B[(size_t)i * dim + i] = cd(1, 0);
    std::vector<int> sup, pos;
    std::vector<cd> D;
    for (int idx : b.members) {
        dense_of(elems[idx], sup, D);
        pos.clear();
        for (int q : sup) pos.push_back((int)(std::find(qubits.begin(), qubits.end(), q) - qubits.begin()));
        left_multiply(B, nq, pos, D);
    }
}

// ------------------------------------------------------------------ plan ---
// Runs of at least kPermMinSwaps uncontrolled SWAPs (X gates may sit between them) whose
// qubits do not fit one fused block: one qubit permutation (a tiled transpose, one pass)
// instead of the blocks a partition would spend on pure data movement (the SWAP network
// at the end of a QFT on n qubits fills n / 6 blocks).
constexpr int kPermMinSwaps = 3;

static bool perm_elem(const Elem &e) {
    const GateMatrix &g = e.gm;
    if (e.pauli || !g.controls.empty()) return false;
    return g.kind == QI_GATE_SWAP || (g.kind == QI_GATE_X && g.nt == 1);
}

static std::vector<Block> partition_with_permutations(qi_plan *p, const std::vector<Elem> &elems, int kmax) {
    std::vector<Block> out;
    size_t seg = 0;   // first element not yet partitioned
    auto take_segment = [&](size_t end) {
        if (end <= seg) return;
        std::vector<Elem> sub(elems.begin() + (long)seg, elems.begin() + (long)end);
        std::vector<Block> bs = choose_partition(p, sub, kmax);
        for (Block &b : bs) {
            for (int &m : b.members) m += (int)seg;
            out.push_back(std::move(b));
        }
    };
    for (size_t i = 0; i < elems.size();) {
        if (!perm_elem(elems[i])) {
            ++i;
            continue;
        }
        size_t j = i;
        int swaps = 0;
        uint64_t support = 0;
        for (; j < elems.size() && perm_elem(elems[j]); ++j) {
            swaps += elems[j].gm.kind == QI_GATE_SWAP;
            support |= elems[j].mask;
        }
        if (swaps >= kPermMinSwaps && __builtin_popcountll(support) > kmax) {
            take_segment(i);
            Block b;
            b.perm = true;
            b.mask = support;
            for (size_t k = i; k < j; ++k) b.members.push_back((int)k);
            out.push_back(std::move(b));
            seg = j;
        }
        i = j;
    }
    take_segment(elems.size());
    return out;
}

// The run's gather: applying gates G_1..G_m is out[j] = in[s(j)] with s the inverse of their
// index map, i.e. the gates' own (self-inverse) maps composed in reverse order.
static Op bitperm_op(const std::vector<Elem> &elems, const Block &b) {
    AffineMap g;
    affine_identity(g);
    for (auto it = b.members.rbegin(); it != b.members.rend(); ++it) affine_compose(g, elems[(size_t)*it].gm);
    Op op;
    op.kind = OP_BITPERM;
    op.k = (int32_t)b.members.size();
    op.xmask = g.b;
    for (int m = 0; m < 64; ++m)   // row m of g is the single bit j_k: source bit m <- output bit k
        if (g.row[m]) op.perm[__builtin_ctzll(g.row[m])] = (int8_t)m;
    return op;
}

// Widen a dense k-qubit block (k < 5; local bit j <-> op.targets[j], ascending) to 5 qubits: the
// lowest qubits outside it join as identity factors.  op.targets / op.k and the matrix M are
// rewritten in place (local bits again ascending by qubit).
static uint64_t padded_to_5(int n, uint64_t mask) {
    uint64_t sel = mask;
    for (int q = 0, need = 5 - __builtin_popcountll(mask); q < n && need > 0; ++q)
        if (!((mask >> q) & 1ull)) {
            sel |= 1ull << q;
            --need;
        }
    return sel;
}
static void pad_block_to_5(int n, Op &op, std::vector<cd> &M) {
    const int k = op.k;
    uint64_t mask = 0;
    for (int j = 0; j < k; ++j) mask |= 1ull << op.targets[j];
    const uint64_t sel = padded_to_5(n, mask);
    int qs[5], nq = 0;
    for (int q = 0; q < 64 && nq < 5; ++q)
        if ((sel >> q) & 1ull) qs[nq++] = q;
    int src[5];   // new local bit -> old local bit, or -1 for a padding qubit
    for (int j = 0; j < 5; ++j) {
        src[j] = -1;
        for (int i = 0; i < k; ++i)
            if (op.targets[i] == qs[j]) src[j] = i;
    }
    const int od = 1 << k;
    std::vector<cd> W((size_t)32 * 32, cd(0, 0));
    for (int r = 0; r < 32; ++r)
        for (int c = 0; c < 32; ++c) {
            int ro = 0, co = 0;
            bool same = true;
            for (int j = 0; j < 5; ++j) {
                const int rb = (r >> j) & 1, cb = (c >> j) & 1;
                if (src[j] < 0) same = same && rb == cb;
                else {
                    ro |= rb << src[j];
                    co |= cb << src[j];
                }
            }
            if (same) W[(size_t)r * 32 + c] = M[(size_t)ro * od + co];
        }
    M.swap(W);
    op.k = 5;
    for (int j = 0; j < 5; ++j) op.targets[j] = qs[j];
}

// The execution of a per-gate plan: every maximal run of two or more ops whose elements the passes
// of qi_gaterun.cu can apply becomes one segment; any other op, and a run of one (the streaming
// per-gate kernels touch the state as often as a pass would), its own.  first[i] is the first
// element of op i (first[nops] = the element count).
static void build_schedule(qi_plan *p, const std::vector<Elem> &elems, const std::vector<size_t> &first) {
    const size_t nops = p->ops.size();
    auto runnable = [&](size_t i) {
        for (size_t e = first[i]; e < first[i + 1]; ++e)
            if (!run_supported(p->n, p->prec, elems[e])) return false;
        return true;
    };
    for (size_t i = 0; i < nops;) {
        size_t j = i;
        while (j < nops && runnable(j)) ++j;
        if (j - i < 2) {
            RunSegment seg;
            seg.op = (int32_t)i++;
            p->sched.push_back(std::move(seg));
            continue;
        }
        std::vector<const Elem *> run;
        for (size_t e = first[i]; e < first[j]; ++e) run.push_back(&elems[e]);
        RunSegment seg;
        schedule_run(p->n, p->prec, run, seg, p->run_prog);
        p->sched.push_back(std::move(seg));
        i = j;
    }
}

// Plans that execute as gate runs from end to end, without looking at their ops: per-gate plans whose
// every element a pass can apply, and FP32 fused plans of run_min to run_max qubits for which the
// caller chose neither block size nor tensor cores.  Below 13 qubits blocks of six do not fit the
// tensor-core kernel's tiles; 40 layers + QFT, fused blocks / gate runs, among others and alone (us): 10 qubits
// 103 / 71, 264 / 220; 12 qubits 193 / 97, 560 / 300; 13 qubits 76 / 107, 210 / 322; 15 qubits 100 / 128, 266 /
// 376; 17 qubits 115 / 164, 307 / 433 (8 and 9 qubits, where a block covers most of the state, about even).
// Error, relative to blocks: a run rounds every gate, a block of six qubits on the CUDA cores (below 13) every
// sum of 64 products, a tensor-core block truncates.  1 to 30 layers of the benchmark family, of an RY / RZ / CNOT
// ansatz and of a QAOA ansatz: 4 qubits 0.7-4.0, 6 qubits 0.5-2.5 (one block holds the state), 7 to 12 qubits
// 0.47-0.87, 13 to 18 qubits 0.18-0.31.  Pauli exponentials of a time step are near the identity and cost a block
// less: 1.4-1.9 on 7 to 12 qubits (0.2-0.34 from 13 on), so circuits with some keep blocks there.  The
// ops (with the fused blocks' matrices, most of a plan's build time) are made when something asks for them.

// Whether some of an FP32 plan's blocks run on the tensor cores.
static bool any_tc_block(int n, const std::vector<Elem> &elems, const std::vector<Block> &blocks) {
    for (const Block &b : blocks) {
        const int k = __builtin_popcountll(b.mask);
        bool diag = true;
        for (int i : b.members) diag = diag && elems[(size_t)i].diagonal;
        if (!b.single && !b.perm && !diag && ((k >= 3 && k <= 5 && n >= 12) || (k == 6 && n >= 13))) return true;
    }
    return false;
}

// Pauli exponentials narrow enough become dense elements when fusing.
static void fuse_narrow_exponentials(std::vector<Elem> &elems, int kmax) {
    for (Elem &e : elems)
        if (e.pauli && !e.gm.normalise_after && __builtin_popcountll(e.mask) <= kmax) e.fusable = true;
}

static bool build_runs(qi_plan *p, const std::vector<Elem> &elems, int fusion, int kmax) {
    p->lazy = false;
    p->run_normalise = false;
    const bool per_gate = fusion == QI_FUSION_NONE || fusion == QI_FUSION_PAULI_GROUPS;
    const bool small_fused = fusion == QI_FUSION_GREEDY && p->opts.fusion == QI_FUSION_GREEDY && p->prec == QI_F32 &&
                             p->opts.use_tensor_cores == 0 && p->opts.max_block_qubits == 0 &&
                             p->partition_override.empty() && p->n >= p->run_min && p->n <= p->run_max;
    if (!per_gate && !small_fused) return false;
    int64_t count = 0;
    for (const Elem &e : elems) {
        if (!run_supported(p->n, p->prec, e) || (small_fused && p->n < 13 && e.pauli)) return false;
        count += e.gm.pauli || e.gm.nt > 0;
    }
    if (count < 2) return false;
    if (small_fused) {
        // the state is renormalised at the end when tensor-core blocks would have run (build_plan)
        p->lazy_blocks = partition_with_permutations(p, elems, kmax);
        p->run_normalise = p->opts.renorm_every >= 0 && any_tc_block(p->n, elems, p->lazy_blocks);
    }
    std::vector<const Elem *> run;
    for (const Elem &e : elems) run.push_back(&e);
    RunSegment seg;
    schedule_run(p->n, p->prec, run, seg, p->run_prog);
    p->sched.push_back(std::move(seg));
    p->lazy_elems = elems;
    p->lazy = true;
    return true;
}

static Status build_plan_ops(qi_plan *p, std::vector<Elem> &elems, bool ops);
Status build_plan(qi_plan *p, std::vector<Elem> &elems) { return build_plan_ops(p, elems, false); }

// The ops of a plan that executes as gate runs, made on first request.
static Status ensure_ops(const qi_plan *cp) {
    qi_plan *p = const_cast<qi_plan *>(cp);
    std::lock_guard<std::mutex> lk(p->run_mu);
    if (!p->lazy) return ok_status();
    qi_plan q;   // built apart: the runs may be executing
    q.n = p->n;
    q.prec = p->prec;
    q.opts = p->opts;
    q.partition_override = p->lazy_blocks;
    Status st = build_plan_ops(&q, p->lazy_elems, true);
    if (!st.ok()) return st;
    p->ops.swap(q.ops);
    p->mats.swap(q.mats);
    p->tc.swap(q.tc);
    p->polys.swap(q.polys);
    p->stats = q.stats;
    p->lazy = false;
    p->lazy_elems.clear();
    return ok_status();
}

// ops: make the ops and nothing else.
static Status build_plan_ops(qi_plan *p, std::vector<Elem> &elems, bool ops) {
    const int n = p->n;
    int fusion = p->opts.fusion;
    int kmax = p->opts.max_block_qubits > 0 ? p->opts.max_block_qubits : 6;
    kmax = std::min(kmax, std::min(6, n));
    if (p->prec == QI_F64) kmax = std::min(kmax, 5);
    int use_tc = p->opts.use_tensor_cores != 2;
    p->ops.clear();
    p->mats.clear();
    p->tc.clear();
    p->compose = ComposeJobs();
    p->polys.clear();
    p->sched.clear();
    p->run_prog.clear();
    int tc_blocks_since = 0, tc_total = 0;
    std::fill(std::begin(p->stats.n_blocks_by_k), std::end(p->stats.n_blocks_by_k), 0);
    p->stats.n_gates = (int64_t)elems.size();
    p->stats.predicted_us = 0.0;
    if (fusion == QI_FUSION_LEARNED && p->partition_override.empty()) {
        // the cost model picks per-gate vs greedy k (and tensor cores); greedy k = kmax without a model
        int kbest = kmax, tcbest = use_tc;
        double ms = 0.0;
        if (learned_choice(p, elems, kmax, &kbest, &tcbest, &ms)) {
            p->stats.predicted_us = ms * 1e3;
            if (kbest <= 1) fusion = QI_FUSION_NONE;
            kmax = std::max(2, kbest);
            use_tc = tcbest;
        }
    }
    if (fusion != QI_FUSION_NONE) fuse_narrow_exponentials(elems, kmax);
    if (!ops && build_runs(p, elems, fusion, kmax)) return ok_status();
    auto lower_single = [&](const Elem &e) {
        Op op = lower_gate(n, e.gm);
        if (op.kind == OP_PAULI_EXP) {
            const double ar = op.alpha_re, ai = op.alpha_im;
            op.cre = std::cosh(ar) * std::cos(ai);
            op.cim = std::sinh(ar) * std::sin(ai);
            op.sre = std::sinh(ar) * std::cos(ai);
            op.sim = std::cosh(ar) * std::sin(ai);
        }
        if (op.kind != OP_NOP) {
            p->ops.push_back(op);
            p->stats.n_blocks_by_k[0]++;
        }
    };
    if (fusion == QI_FUSION_NONE || fusion == QI_FUSION_PAULI_GROUPS) {
        auto groupable = [&](const Elem &e) {
            return fusion == QI_FUSION_PAULI_GROUPS && e.pauli && !e.gm.normalise_after;
        };
        std::vector<size_t> first;   // element each op starts at
        auto note = [&](size_t e) {
            if (first.size() < p->ops.size()) first.push_back(e);
        };
        for (size_t i = 0; i < elems.size();) {
            if (!groupable(elems[i])) {
                lower_single(elems[i]);
                note(i++);
                continue;
            }
            std::vector<const GateMatrix *> run;
            size_t j = i;
            for (; j < elems.size() && groupable(elems[j]); ++j) run.push_back(&elems[j].gm);
            for (size_t used = 0; used < run.size();) {
                Op op;
                const size_t took = pauli_group_op(run, used, op, p->mats);
                if (took == 1) {
                    lower_single(elems[i + used]);
                } else {
                    p->ops.push_back(op);
                    p->stats.n_blocks_by_k[0]++;
                }
                note(i + used);
                used += took;
            }
            i = j;
        }
        first.push_back(elems.size());
        if (!ops) build_schedule(p, elems, first);
    } else {
        std::vector<Block> blocks = p->partition_override.empty() ? partition_with_permutations(p, elems, kmax)
                                                                  : p->partition_override;
        // compose block matrices in parallel (independent)
        std::vector<std::vector<int>> qb(blocks.size());
        std::vector<std::vector<cd>> mb(blocks.size());
        // ... those the device does not compose: tensor-core blocks of a plan for one call
        std::vector<uint64_t> on_device(blocks.size(), 0);   // the block's qubits, padded
        size_t on_host = 0;
        for (size_t bi = 0; bi < blocks.size(); ++bi) {
            const Block &b = blocks[bi];
            if (b.single || b.perm) continue;
            bool diag = true;
            for (int idx : b.members) diag = diag && elems[idx].diagonal;
            const int k = __builtin_popcountll(b.mask);
            const uint64_t padded = k == 3 || k == 4 ? (n >= 12 ? padded_to_5(n, b.mask) : 0) : k >= 5 ? b.mask : 0;
            if (p->device_blocks && !ops && use_tc && p->prec == QI_F32 && !diag && padded &&
                n >= __builtin_popcountll(padded) + 7)
                on_device[bi] = padded;
            else
                ++on_host;
        }
        const unsigned nth = (unsigned)std::min<size_t>({on_host, 16, std::max(1u, std::thread::hardware_concurrency())});
        std::vector<std::thread> th;
        for (unsigned w = 0; w < nth; ++w) {
            th.emplace_back([&, w] {
                for (size_t bi = w; bi < blocks.size(); bi += nth)
                    if (!blocks[bi].single && !blocks[bi].perm && !on_device[bi]) compose_block(elems, blocks[bi], qb[bi], mb[bi]);
            });
        }
        for (auto &t : th) t.join();
        // FP32 plans: a run of consecutive diagonal blocks whose phases are
        // polynomials of degree <= 2 is applied as one phase polynomial (one pass;
        // also a run of one block of three or more qubits, where the polynomial pass
        // is faster than the table kernel: 2.6 vs 3.0 ms at 30 qubits).
        const bool poly_ok = p->prec == QI_F32;
        PhasePoly pending;
        std::vector<Op> pending_ops;
        if (poly_ok) pending.init(n);
        auto flush = [&]() {
            if (pending_ops.size() >= 2 || (pending_ops.size() == 1 && pending_ops[0].k >= 3)) {
                Op op;
                op.kind = OP_PHASE_POLY;
                op.k = (int32_t)pending_ops.size();
                for (const Op &d : pending_ops)
                    for (int j = 0; j < d.k; ++j) op.zmask |= 1ull << d.targets[j];
                op.mat_offset = (int64_t)p->polys.size();
                op.tc_offset = (int64_t)p->tc.size();
                p->polys.push_back(pending);
                Op *prev = p->ops.empty() ? nullptr : &p->ops.back();
                if (prev && prev->kind == OP_FUSED && prev->tc_offset >= 0 && prev->poly_tc < 0 &&
                    tc_phase_table(pending, prev->k, prev->targets, p->tc)) {
                    // right after a tensor-core block: its epilogue applies the phases (no extra pass)
                    prev->poly_tc = op.tc_offset;
                    prev->poly_idx = op.mat_offset;
                } else {
                    phase_poly_device_block(pending, p->tc);
                    p->ops.push_back(op);
                }
            } else if (pending_ops.size() == 1) {
                p->ops.push_back(pending_ops[0]);
            }
            pending_ops.clear();
            if (poly_ok) pending.init(n);
        };
        auto emit = [&](const Op &op) {
            p->ops.push_back(op);
            p->stats.n_blocks_by_k[op.k]++;
            if (op.tc_offset >= 0) {
                ++tc_blocks_since;
                ++tc_total;
                if (p->opts.renorm_every > 0 && tc_blocks_since >= p->opts.renorm_every) {
                    Op nrm;
                    nrm.kind = OP_NORMALISE;
                    p->ops.push_back(nrm);
                    tc_blocks_since = 0;
                }
            }
        };
        for (size_t bi = 0; bi < blocks.size(); ++bi) {
            const Block &b = blocks[bi];
            if (b.single) {
                flush();
                lower_single(elems[b.members[0]]);
                continue;
            }
            if (b.perm) {
                flush();
                p->ops.push_back(bitperm_op(elems, b));
                p->stats.n_blocks_by_k[0]++;
                continue;
            }
            if (on_device[bi]) {
                flush();
                Op op;
                op.kind = OP_FUSED;
                op.mode = use_tc;
                op.mat_offset = 0;
                for (uint64_t m = on_device[bi]; m; m &= m - 1) op.targets[op.k++] = __builtin_ctzll(m);
                op.tc_offset = (int64_t)p->compose.words;
                p->compose.ops.push_back(p->ops.size());
                compose_job(elems, b, on_device[bi], p->compose);
                emit(op);
                continue;
            }
            bool diag = true;
            for (int idx : b.members) diag = diag && elems[idx].diagonal;
            const int k = (int)qb[bi].size();
            Op op;
            op.k = k;
            for (int j = 0; j < k; ++j) op.targets[j] = qb[bi][j];
            op.mat_offset = (int64_t)p->mats.size();
            const int dim = 1 << k;
            if (diag) {
                op.kind = OP_DIAGK;
                std::vector<cd> table((size_t)dim);
                for (int r = 0; r < dim; ++r) table[(size_t)r] = mb[bi][(size_t)r * dim + r];
                p->mats.insert(p->mats.end(), table.begin(), table.end());
                if (poly_ok && phase_poly_add_table(pending, k, op.targets, table.data())) {
                    pending_ops.push_back(op);
                    p->stats.n_blocks_by_k[k]++;
                    continue;
                }
                flush();
            } else {
                flush();
                op.kind = OP_FUSED;
                op.mode = use_tc;
                if (op.mode && p->prec == QI_F32 && (k == 3 || k == 4) && n >= 12) {
                    // a 3- or 4-qubit block runs faster on the tensor cores as a 5-qubit block with the
                    // identity on the lowest free qubits (30 qubits: 3.5 ms on the CUDA cores, 2.6-2.9 ms
                    // padded; low padding qubits give the tile long row runs)
                    pad_block_to_5(n, op, mb[bi]);
                }
                const int kk = op.k, dd = 1 << kk;
                for (size_t i = 0; i < (size_t)dd * dd; ++i) p->mats.push_back(mb[bi][i]);
                if (op.mode && p->prec == QI_F32 && kk >= 5 && n >= kk + 7) {
                    op.tc_offset = (int64_t)p->tc.size();
                    tc_blocks(kk, reinterpret_cast<const double *>(mb[bi].data()), p->tc);
                }
            }
            emit(op);
        }
        flush();
    }
    // Tensor-core accumulation rounds toward zero: renormalise once at the end
    // (unless disabled, or the last op already did).
    if (tc_total > 0 && p->opts.renorm_every >= 0 && (p->ops.empty() || p->ops.back().kind != OP_NORMALISE)) {
        Op nrm;
        nrm.kind = OP_NORMALISE;
        p->ops.push_back(nrm);
    }
    finish_compose(p);
    p->stats.n_kernels = (int64_t)p->ops.size();
    return ok_status();
}

static bool not_uploaded(const qi_plan *p) {
    return (!p->d_mats && !p->mats.empty()) || (!p->d_tc && !p->tc.empty());
}

// A copy that has arrived when it returns: cudaMemcpy of pageable memory may return while its last part is
// still on its way in the default stream, which the states' (non-blocking) streams do not wait for.
static cudaError_t copy_in(void *d, const void *h, size_t bytes) {
    const cudaError_t e = cudaMemcpy(d, h, bytes, cudaMemcpyHostToDevice);
    return e == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : e;
}

Status upload_plan(qi_plan *p) {
    if (p->d_mats) { cudaFree(p->d_mats); p->d_mats = nullptr; }
    if (p->d_tc) { cudaFree(p->d_tc); p->d_tc = nullptr; }
    if (!p->tc.empty()) {
        QI_CUDA(device_malloc(&p->d_tc, (p->tc.size() + p->compose.words) * sizeof(float)));
        p->composed = false;
        QI_CUDA(copy_in(p->d_tc, p->tc.data(), p->tc.size() * sizeof(float)));
    }
    if (p->mats.empty()) return ok_status();
    const size_t cnt = p->mats.size();
    if (p->prec == QI_F32) {
        std::vector<float2> h(cnt);
        for (size_t i = 0; i < cnt; ++i) h[i] = make_float2((float)p->mats[i].real(), (float)p->mats[i].imag());
        QI_CUDA(device_malloc(&p->d_mats, cnt * sizeof(float2)));
        QI_CUDA(copy_in(p->d_mats, h.data(), cnt * sizeof(float2)));
    } else {
        std::vector<double2> h(cnt);
        for (size_t i = 0; i < cnt; ++i) h[i] = make_double2(p->mats[i].real(), p->mats[i].imag());
        QI_CUDA(device_malloc(&p->d_mats, cnt * sizeof(double2)));
        QI_CUDA(copy_in(p->d_mats, h.data(), cnt * sizeof(double2)));
    }
    return ok_status();
}

Status plan_elems_from_gates(int n, const qi_gate *gates, int64_t ng, const double *theta, int64_t ntheta,
                             std::vector<Elem> &elems) {
    elems.clear();
    elems.reserve((size_t)ng);
    for (int64_t k = 0; k < ng; ++k) {
        qi_gate g = gates[k];
        for (int j = 0; j < 3; ++j) {
            if (g.param_ids[j] >= 0) {
                if (!theta || g.param_ids[j] >= ntheta)
                    return err(QI_ERR_MISMATCHED_NUMBER_OF_PARAMETERS, g.param_ids[j] + 1, ntheta);
                g.params[j] = theta[g.param_ids[j]];
            }
        }
        GateMatrix gm;
        Status st = gate_to_matrix(n, g, &gm);
        if (!st.ok()) {
            st.msg = "gate " + std::to_string(k) + (st.msg.empty() ? "" : ": " + st.msg);
            return st;
        }
        elems.push_back(make_elem_from_gate(gm, (int)k));
    }
    return ok_status();
}

// Whether the plan's runs can execute on s: their program goes to s's device on first use.  Where that
// is not possible (the stream is being captured, the program is on another device, no memory), the
// plan's ops run one kernel each instead.
static bool runs_ready(qi_plan *p, qi_state *s) {
    if (p->run_prog.empty()) return false;
    std::lock_guard<std::mutex> lk(p->run_mu);
    if (p->d_run) return p->run_device == s->device;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return false;
    }
    void *d = nullptr;
    if (device_malloc(&d, p->run_prog.size()) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    if (copy_in(d, p->run_prog.data(), p->run_prog.size()) != cudaSuccess) {
        (void)cudaGetLastError();
        cudaFree(d);
        return false;
    }
    p->d_run = d;
    p->run_device = s->device;
    return true;
}

// The same for plans that live for one call on one state: their programs are copied into the state's
// program space, in stream order (the caller waits for the stream before it lets go of the state).
static void borrow_runs(std::initializer_list<qi_plan *> plans, qi_state *s) {
    size_t total = 0;
    for (qi_plan *p : plans) total += (p->run_prog.size() + 15) / 16 * 16;
    void *d = nullptr;
    if (total == 0 || !state_workspace(s, total, &d, true).ok()) return;
    char *at = static_cast<char *>(d);
    for (qi_plan *p : plans) {
        if (p->run_prog.empty()) continue;
        if (cudaMemcpyAsync(at, p->run_prog.data(), p->run_prog.size(), cudaMemcpyHostToDevice, s->stream) != cudaSuccess) {
            (void)cudaGetLastError();
            return;
        }
        p->d_run = at;
        p->run_device = s->device;
        p->run_borrowed = true;
        at += (p->run_prog.size() + 15) / 16 * 16;
    }
}

void release_runs(qi_plan *p) {
    if (p->d_run && !p->run_borrowed) cudaFree(p->d_run);
    p->d_run = nullptr;
}

// Launches a plan's ops on a state.  OP_BITPERM writes out of place: the amplitudes move to
// the state's second buffer and back (the next renormalisation writes into the state's own
// buffer; otherwise one copy at the end), so the state's device pointer never changes.
struct PlanRunner {
    qi_plan *p;
    qi_state *s;
    void *home;
    unsigned norm_nb = 0;   // norm partials of the current amplitudes are in s->d_partials (rows)
    PlanRunner(qi_plan *p_, qi_state *s_) : p(p_), s(s_), home(s_->amps) {}
    Status op(const Op &o, int next_kind) {
        const unsigned have_norm = norm_nb;   // left by the op before this one
        norm_nb = 0;
        if (o.kind == OP_BITPERM) {
            void *scratch = nullptr;
            if (s->amps == home && !state_scratch(s, &scratch).ok())
                return bitperm_in_place_async(s, o.perm, o.xmask);   // no room for a second buffer
            void *dst = s->amps == home ? scratch : home;
            // a renormalisation next: the permutation sums the norm as it writes
            unsigned nb = 0;
            Status st = bitperm_async(s, dst, s->amps, o.perm, o.xmask, next_kind == OP_NORMALISE ? &nb : nullptr);
            if (st.ok()) {
                s->amps = dst;
                norm_nb = nb;
            }
            return st;
        }
        if (o.kind == OP_MEASURE && s->amps != home) {   // measure the amplitudes in the state's own buffer
            Status st = finish(ok_status());
            if (!st.ok()) return st;
        }
        if (o.kind == OP_NORMALISE && s->amps != home) {
            Status st = have_norm ? state_normalise_to_from_partials_async(s, home, s->amps, have_norm)
                                  : state_normalise_device_to_async(s, home, s->amps);
            if (st.ok()) s->amps = home;
            return st;
        }
        return launch_op(s, o, p->d_mats, p->d_tc);
    }
    Status finish(Status st) {   // the amplitudes back in the state's own buffer
        if (s->amps != home) {
            if (st.ok()) {
                cudaError_t e = cudaMemcpyAsync(home, s->amps, s->bytes(), cudaMemcpyDeviceToDevice, s->stream);
                if (e != cudaSuccess) st = cuda_status(e, "copy back after qubit permutation");
            }
            s->amps = home;
        }
        return st;
    }
};

Status plan_execute(qi_plan *p, qi_state *s) {
    if (s->n != p->n) return err(QI_ERR_INVALID_NUMBER_OF_QUBITS, s->n);   // circuit.rs:161-163
    if (s->prec != p->prec) return err(QI_ERR_UNSUPPORTED, -1, -1, "plan precision differs from state");
    const bool runs = runs_ready(p, s);
    bool matrices = !runs;   // only operations outside the runs need them
    for (size_t i = 0; !matrices && i < p->sched.size(); ++i)
        matrices = p->sched[i].op >= 0 && p->ops[(size_t)p->sched[i].op].mat_offset >= 0;
    if (!runs) {
        Status have = ensure_ops(p);
        if (!have.ok()) return have;
    }
    if (matrices && not_uploaded(p)) {   // they go to the device on first use
        Status up = upload_plan(p);
        if (!up.ok()) return up;
    }
    bool has_norm = false;
    const bool compose = !runs && !p->compose.blocks.empty() && !p->composed;
    if (compose) {
        Status st = launch_compose(p, s);
        if (!st.ok()) return st;
        p->ops[p->compose.ops[0]].fresh_tc = p->composed = true;
    }
    PlanRunner run(p, s);
    for (size_t i = 0; runs && i < p->sched.size(); ++i) {
        const RunSegment &seg = p->sched[i];
        if (seg.op >= 0) {
            const Op &op = p->ops[(size_t)seg.op];
            Status st = run.op(op, -1);
            if (!st.ok()) return run.finish(st);
            has_norm = has_norm || op.kind == OP_PAULI_NORM;
        }
        for (const RunPass &pass : seg.passes) {
            Status st = launch_run_pass(s, pass, p->d_run);
            if (!st.ok()) return run.finish(st);
        }
    }
    if (runs && p->run_normalise) {
        Status st = state_normalise_device_async(s);
        if (!st.ok()) return run.finish(st);
    }
    for (size_t i = 0; !runs && i < p->ops.size(); ++i) {
        const Op &op = p->ops[i];
        Status st = run.op(op, i + 1 < p->ops.size() ? p->ops[i + 1].kind : -1);
        if (!st.ok()) return run.finish(st);
        has_norm = has_norm || op.kind == OP_PAULI_NORM;
    }
    if (compose) p->ops[p->compose.ops[0]].fresh_tc = false;
    {
        Status st = run.finish(ok_status());
        if (!st.ok()) return st;
    }
    if (has_norm) {
        int flag = 0;
        Status st = state_read_flag(s, &flag);
        if (!st.ok()) return st;
        if (flag) return err(QI_ERR_ZERO_NORM);
    }
    return ok_status();
}

Elem pauli_exp_elem(const qi_pauli_term &t, double far, double fai, int src) {
    GateMatrix gm;
    gm.kind = QI_GATE_PAULI_EVOLUTION;
    gm.pauli = true;
    gm.xmask = t.xmask;
    gm.zmask = t.zmask;
    gm.alpha_re = t.coeff_re * far - t.coeff_im * fai;
    gm.alpha_im = t.coeff_re * fai + t.coeff_im * far;
    return make_elem_from_gate(gm, src);
}

Status sumop_expectation(qi_state *s, const qi_pauli_term *terms, int64_t nt, double out[2]);

}  // namespace qi

using namespace qi;

extern "C" {

static qi_status plan_create(int32_t num_qubits, int32_t precision, const qi_gate *gates, int64_t n_gates,
                             const double *theta, int64_t n_theta, const qi_exec_options *opts, bool one_call,
                             qi_plan **out) {
    if (!out || (!gates && n_gates > 0)) return publish(err(QI_ERR_NULL_ARGUMENT));
    *out = nullptr;
    if (num_qubits <= 0 || num_qubits > 40) return publish(err(QI_ERR_INVALID_NUMBER_OF_QUBITS, num_qubits));
    if (precision != QI_F32 && precision != QI_F64) return publish(err(QI_ERR_INVALID_INPUT_VALUE, precision));
    qi_plan *p = new qi_plan();
    p->n = num_qubits;
    p->prec = precision;
    if (opts) p->opts = *opts;
    p->device_blocks = one_call;
    std::vector<Elem> elems;
    Status st = plan_elems_from_gates(num_qubits, gates, n_gates, theta, n_theta, elems);
    // The plan's build counts too, 1.3-1.7 ms for blocks, so gate runs win until their slower passes have cost
    // as much: 4 / 10 / 20 / 40 layers, runs and (blocks), us: 20 qubits 486 / 720 / 1159 / 1981 (1661 / 1868 /
    // 2183 / 2726); 21 qubits 640 / 1018 / 1628 / 2829 (1764 / 1848 / 2195 / 2781); 22 qubits 927 / 1463 / 2371 /
    // 4156 (1860 / 2055 / 2486 / 3226); 23 qubits 1559 / 2458 / 4054 / 7189 (2172 / 2386 / 3129 / 3976): even at
    // about 1700 gates of 21 qubits (40 layers), half as many a qubit more.  Below 7 qubits blocks are more exact
    // (build_runs).
    if (one_call) {
        p->run_min = 7;
        if (num_qubits <= 23 && std::ldexp((double)elems.size(), num_qubits - 21) <= 1700.0) p->run_max = 23;
    }
    if (st.ok()) st = build_plan(p, elems);
    if (!st.ok()) { delete p; return publish(st); }
    *out = p;
    return publish(ok_status());
}

qi_status qi_plan_create(int32_t num_qubits, int32_t precision, const qi_gate *gates, int64_t n_gates,
                         const double *theta, int64_t n_theta, const qi_exec_options *opts, qi_plan **out) {
    return plan_create(num_qubits, precision, gates, n_gates, theta, n_theta, opts, false, out);
}

qi_status qi_plan_execute(qi_plan *p, qi_state *s) {
    if (!p || !s) return publish(err(QI_ERR_NULL_ARGUMENT));
    std::lock_guard<std::recursive_mutex> lk(s->mu);
    cudaError_t e = cudaSetDevice(s->device);
    if (e != cudaSuccess) return publish(cuda_status(e, "cudaSetDevice"));
    return publish(plan_execute(p, s));
}

qi_status qi_plan_stats_get(const qi_plan *p, qi_plan_stats *out) {
    if (!p || !out) return publish(err(QI_ERR_NULL_ARGUMENT));
    Status st = ensure_ops(p);
    if (!st.ok()) return publish(st);
    *out = p->stats;
    return publish(ok_status());
}

qi_status qi_plan_profile(qi_plan *p, qi_state *s, float *ms_out) {
    if (!p || !s || !ms_out) return publish(err(QI_ERR_NULL_ARGUMENT));
    std::lock_guard<std::recursive_mutex> lk(s->mu);
    cudaError_t e = cudaSetDevice(s->device);
    if (e != cudaSuccess) return publish(cuda_status(e, "cudaSetDevice"));
    if (s->n != p->n || s->prec != p->prec) return publish(err(QI_ERR_INVALID_NUMBER_OF_QUBITS, s->n));
    {
        Status have = ensure_ops(p);
        if (!have.ok()) return publish(have);
    }
    if (not_uploaded(p)) {
        Status up = upload_plan(p);
        if (!up.ok()) return publish(up);
    }
    const size_t nops = p->ops.size();
    std::vector<cudaEvent_t> ev(nops + 1);
    for (auto &x : ev) {
        e = cudaEventCreate(&x);
        if (e != cudaSuccess) return publish(cuda_status(e, "cudaEventCreate"));
    }
    Status st = ok_status();
    PlanRunner run(p, s);
    cudaEventRecord(ev[0], s->stream);
    for (size_t i = 0; i < nops && st.ok(); ++i) {
        st = run.op(p->ops[i], i + 1 < nops ? p->ops[i + 1].kind : -1);
        cudaEventRecord(ev[i + 1], s->stream);
    }
    st = run.finish(st);
    e = cudaStreamSynchronize(s->stream);
    if (st.ok() && e != cudaSuccess) st = cuda_status(e, "profile");
    for (size_t i = 0; i < nops && st.ok(); ++i) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ev[i], ev[i + 1]);
        ms_out[i] = ms;
    }
    for (auto &x : ev) cudaEventDestroy(x);
    return publish(st);
}

qi_status qi_apply_matrix(qi_state *s, const int32_t *targets, int32_t k, const double *matrix,
                          int32_t use_tensor_cores) {
    if (!s || !targets || !matrix) return publish(err(QI_ERR_NULL_ARGUMENT));
    std::lock_guard<std::recursive_mutex> lk(s->mu);
    cudaError_t e = cudaSetDevice(s->device);
    if (e != cudaSuccess) return publish(cuda_status(e, "cudaSetDevice"));
    if (k < 1 || k > 6) return publish(err(QI_ERR_INVALID_NUMBER_OF_QUBITS, k));
    const int n = s->n;
    for (int j = 0; j < k; ++j) {
        if (targets[j] < 0 || targets[j] >= n) return publish(err(QI_ERR_INVALID_QUBIT_INDEX, targets[j], n));
        for (int i = 0; i < j; ++i)
            if (targets[i] == targets[j]) return publish(err(QI_ERR_INVALID_QUBIT_INDEX, targets[j], n));
    }
    // sort targets and permute the matrix to the sorted local order
    std::vector<int> order(k);
    for (int j = 0; j < k; ++j) order[j] = j;
    std::sort(order.begin(), order.end(), [&](int x, int y) { return targets[x] < targets[y]; });
    const int dim = 1 << k;
    auto remap = [&](int idx) {   // sorted-local index -> caller-local index
        int o = 0;
        for (int j = 0; j < k; ++j) o |= ((idx >> j) & 1) << order[j];
        return o;
    };
    std::vector<cd> U((size_t)dim * dim);
    for (int r = 0; r < dim; ++r)
        for (int c = 0; c < dim; ++c) {
            const size_t src = (size_t)remap(r) * dim + remap(c);
            U[(size_t)r * dim + c] = cd(matrix[2 * src], matrix[2 * src + 1]);
        }
    qi_plan plan;
    plan.n = n;
    plan.prec = s->prec;
    Op op;
    op.kind = OP_FUSED;
    op.k = k;
    for (int j = 0; j < k; ++j) op.targets[j] = targets[order[j]];
    op.mat_offset = 0;
    op.mode = use_tensor_cores != 2;
    plan.mats = U;
    if (op.mode && s->prec == QI_F32 && k >= 5 && n >= k + 7) {
        op.tc_offset = 0;
        tc_blocks(k, reinterpret_cast<const double *>(U.data()), plan.tc);
    }
    if (s->prec == QI_F64 && k > 5) return publish(err(QI_ERR_UNSUPPORTED, k, -1, "FP64 blocks are limited to k <= 5"));
    plan.ops.push_back(op);
    Status st = upload_plan(&plan);
    if (st.ok()) st = plan_execute(&plan, s);
    if (st.ok()) {
        e = cudaStreamSynchronize(s->stream);
        if (e != cudaSuccess) st = cuda_status(e, "apply_matrix");
    }
    if (st.ok()) {
        int flag = 0;
        st = state_read_flag(s, &flag);
        if (st.ok() && flag == 2) st = err(QI_ERR_TIMEOUT, -1, -1, "tensor-core kernel wait timed out");
    }
    if (plan.d_mats) cudaFree(plan.d_mats);
    if (plan.d_tc) cudaFree(plan.d_tc);
    plan.d_mats = plan.d_tc = nullptr;
    return publish(st);
}

qi_status qi_plan_num_ops(const qi_plan *p, int64_t *out) {
    if (!p || !out) return publish(err(QI_ERR_NULL_ARGUMENT));
    Status st = ensure_ops(p);
    if (!st.ok()) return publish(st);
    *out = (int64_t)p->ops.size();
    return publish(ok_status());
}

qi_status qi_plan_run_info(const qi_plan *p, int64_t *n_passes, int64_t *n_phases, int64_t *n_single) {
    if (!p || !n_passes || !n_phases || !n_single) return publish(err(QI_ERR_NULL_ARGUMENT));
    *n_passes = *n_phases = *n_single = 0;
    for (const RunSegment &seg : p->sched) {
        *n_single += seg.op >= 0;
        for (const RunPass &pass : seg.passes) {
            ++*n_passes;
            *n_phases += pass.nphase;
        }
    }
    return publish(ok_status());
}

qi_status qi_plan_run_replay(const qi_plan *p, double *amps) {
    if (!p || !amps) return publish(err(QI_ERR_NULL_ARGUMENT));
    if (p->prec != QI_F64) return publish(err(QI_ERR_UNSUPPORTED, p->prec, -1, "replay is of FP64 plans"));
    for (const RunSegment &seg : p->sched)
        if (seg.op >= 0) return publish(err(QI_ERR_UNSUPPORTED, seg.op, -1, "operation outside a run"));
    for (const RunSegment &seg : p->sched)
        for (const RunPass &pass : seg.passes)
            replay_run_pass(p->n, pass, p->run_prog.data(), reinterpret_cast<cd *>(amps));
    return publish(ok_status());
}

qi_status qi_plan_op_phase_poly(const qi_plan *p, int64_t i, uint64_t *c0, uint64_t *a, uint64_t *b) {
    if (!p || !c0 || !a || !b) return publish(err(QI_ERR_NULL_ARGUMENT));
    {
        Status have = ensure_ops(p);
        if (!have.ok()) return publish(have);
    }
    if (i < 0 || i >= (int64_t)p->ops.size()) return publish(err(QI_ERR_INVALID_INPUT_VALUE, i));
    const Op &op = p->ops[(size_t)i];
    const int64_t idx = op.kind == OP_PHASE_POLY ? op.mat_offset : op.kind == OP_FUSED ? op.poly_idx : -1;
    if (idx < 0 || idx >= (int64_t)p->polys.size())
        return publish(err(QI_ERR_INVALID_INPUT_VALUE, i, op.kind, "no phase polynomial on this op"));
    const PhasePoly &pp = p->polys[(size_t)idx];
    *c0 = pp.c0;
    std::copy(pp.a.begin(), pp.a.end(), a);
    std::copy(pp.b.begin(), pp.b.end(), b);
    return publish(ok_status());
}

qi_status qi_plan_op_pauli_group(const qi_plan *p, int64_t i, int32_t *n_tables, int32_t *rank, uint64_t *basis) {
    if (!p || !n_tables || !rank || !basis) return publish(err(QI_ERR_NULL_ARGUMENT));
    {
        Status have = ensure_ops(p);
        if (!have.ok()) return publish(have);
    }
    if (i < 0 || i >= (int64_t)p->ops.size()) return publish(err(QI_ERR_INVALID_INPUT_VALUE, i));
    const Op &op = p->ops[(size_t)i];
    if (op.kind != OP_PAULI_GROUP) return publish(err(QI_ERR_INVALID_INPUT_VALUE, i, op.kind, "not a Pauli-group op"));
    *n_tables = op.nchunk;
    std::copy(op.rank, op.rank + kGroupChunks, rank);
    std::copy(op.basis, op.basis + kGroupChunks * kGroupRank, basis);
    return publish(ok_status());
}

qi_status qi_plan_op_bitperm(const qi_plan *p, int64_t i, int32_t *source_bit, uint64_t *flip) {
    if (!p || !source_bit || !flip) return publish(err(QI_ERR_NULL_ARGUMENT));
    {
        Status have = ensure_ops(p);
        if (!have.ok()) return publish(have);
    }
    if (i < 0 || i >= (int64_t)p->ops.size()) return publish(err(QI_ERR_INVALID_INPUT_VALUE, i));
    const Op &op = p->ops[(size_t)i];
    if (op.kind != OP_BITPERM) return publish(err(QI_ERR_INVALID_INPUT_VALUE, op.kind, OP_BITPERM));
    for (int k = 0; k < p->n; ++k) source_bit[k] = op.perm[k];
    *flip = op.xmask;
    return publish(ok_status());
}

qi_status qi_plan_op_get(const qi_plan *p, int64_t i, qi_plan_op_info *info, double *matrix_out, int64_t capacity) {
    if (!p || !info) return publish(err(QI_ERR_NULL_ARGUMENT));
    {
        Status have = ensure_ops(p);
        if (!have.ok()) return publish(have);
    }
    if (i < 0 || i >= (int64_t)p->ops.size()) return publish(err(QI_ERR_INVALID_INPUT_VALUE, i));
    const Op &op = p->ops[(size_t)i];
    std::memset(info, 0, sizeof(*info));
    info->kind = op.kind;
    info->k = op.k;
    for (int j = 0; j < 6; ++j) info->targets[j] = op.targets[j];
    info->tensor_cores = (op.kind == OP_FUSED && op.tc_offset >= 0) ? 1 : 0;
    info->phase_poly = (op.kind == OP_FUSED && op.poly_idx >= 0) ? 1 : 0;
    info->control_mask = op.cmask;
    info->xmask = op.xmask;
    info->zmask = op.zmask;
    std::vector<double> m;
    switch (op.kind) {
    case OP_MAT1: m.assign(op.m, op.m + 8); break;
    case OP_MAT2: m.assign(op.m, op.m + 32); break;
    case OP_FUSED:
    case OP_DIAGK: {
        const size_t cnt = op.kind == OP_FUSED ? ((size_t)1 << (2 * op.k)) : ((size_t)1 << op.k);
        for (size_t j = 0; j < cnt; ++j) {
            m.push_back(p->mats[(size_t)op.mat_offset + j].real());
            m.push_back(p->mats[(size_t)op.mat_offset + j].imag());
        }
        break;
    }
    case OP_PAULI_EXP: m = {op.cre, op.cim, op.sre, op.sim}; break;
    case OP_MEASURE:   // k measured qubits (the first six in targets), basis in zmask, seed in xmask
        for (int j = 0; j < 6; ++j) info->targets[j] = j < op.k ? op.perm[j] : 0;
        info->zmask = (uint64_t)op.mode;
        if (op.mode == QI_BASIS_CUSTOM) m.assign(op.m, op.m + 8);
        break;
    case OP_PAULI_GROUP: {
        size_t cnt = 0;
        for (int c = 0; c < op.nchunk; ++c) cnt += (size_t)(op.xmask ? 4 : 1) << op.rank[c];
        for (size_t j = 0; j < cnt; ++j) {
            m.push_back(p->mats[(size_t)op.mat_offset + j].real());
            m.push_back(p->mats[(size_t)op.mat_offset + j].imag());
        }
        break;
    }
    default: break;
    }
    info->n_matrix = (int64_t)(m.size() / 2);
    if (matrix_out) {
        if (capacity < info->n_matrix) return publish(err(QI_ERR_INVALID_INPUT_VALUE, capacity, info->n_matrix));
        std::copy(m.begin(), m.end(), matrix_out);
    }
    return publish(ok_status());
}

qi_status qi_plan_destroy(qi_plan *p) {
    if (!p) return QI_OK;
    if (p->d_mats) cudaFree(p->d_mats);
    if (p->d_tc) cudaFree(p->d_tc);
    release_runs(p);
    delete p;
    return QI_OK;
}

// One-call FP32 circuits that run per gate in FP64 on a scratch copy and are rounded at the end: those of fewer than
// 12 qubits where FP32 gate runs are less exact than blocks (build_runs), which take 0.7-3 ms to compose (5 and 6 qubits,
// 20 layers: runs 0.13 and 0.15 ms, blocks 0.76 and 2.9).  Not with measurements: their outcomes are those of the
// FP32 probabilities.
static bool wide_circuit(int n, const qi_gate *gates, int64_t n_gates) {
    if (n >= 12 || !gates) return false;
    bool exponentials = false;
    for (int64_t i = 0; i < n_gates; ++i) {
        if (gates[i].kind == QI_GATE_MEASUREMENT) return false;
        exponentials = exponentials || gates[i].kind == QI_GATE_PAULI_EVOLUTION || gates[i].kind == QI_GATE_PAULI_STRING;
    }
    return n < 7 || exponentials;
}

qi_status qi_circuit_execute(qi_state *s, const qi_gate *gates, int64_t n_gates, const double *theta, int64_t n_theta,
                             const qi_exec_options *opts) {
    if (!s) return publish(err(QI_ERR_NULL_ARGUMENT));
    if (s->prec == QI_F32 && opts && opts->fusion == QI_FUSION_GREEDY && opts->max_block_qubits == 0 &&
        opts->use_tensor_cores == 0 && wide_circuit(s->n, gates, n_gates)) {
        std::lock_guard<std::recursive_mutex> lk(s->mu);
        qi_state *wide = nullptr;
        if (cudaSetDevice(s->device) == cudaSuccess && scratch_take(s, QI_F64, &wide).ok()) {
            Status st = state_copy_async(wide, s);
            const qi_exec_options per_gate = {QI_FUSION_NONE, 0, 0, 0};
            qi_status run = st.ok() ? qi_circuit_execute(wide, gates, n_gates, theta, n_theta, &per_gate) : publish(st);
            if (run == QI_OK) {
                st = state_copy_async(s, wide);
                const cudaError_t e = cudaStreamSynchronize(s->stream);
                if (st.ok() && e != cudaSuccess) st = cuda_status(e, "execute");
                run = publish(st);
            }
            scratch_give(wide);
            return run;
        }
    }
    qi_plan *p = nullptr;
    qi_status st = plan_create(s->n, s->prec, gates, n_gates, theta, n_theta, opts, true, &p);
    if (st != QI_OK) return st;
    std::lock_guard<std::recursive_mutex> lk(s->mu);   // held until the plan's program is no longer in use
    if (cudaSetDevice(s->device) == cudaSuccess) borrow_runs({p}, s);
    st = qi_plan_execute(p, s);
    const cudaError_t e = cudaStreamSynchronize(s->stream);   // after a failure too: earlier passes may be running
    if (st == QI_OK) {
        if (e != cudaSuccess) {
            st = publish(cuda_status(e, "execute"));
        } else {
            int flag = 0;
            Status fs = state_read_flag(s, &flag);
            if (!fs.ok()) st = publish(fs);
            else if (flag == 2) st = publish(err(QI_ERR_TIMEOUT, -1, -1, "tensor-core kernel wait timed out"));
        }
    }
    qi_plan_destroy(p);
    return st;
}

// `steps` steps as an ordered list of exponentials (time_evolution.rs:45-115).
static std::vector<Elem> step_list(const qi_pauli_term *terms, int64_t n_terms, double dt, int32_t order, int64_t steps) {
    std::vector<Elem> elems;
    for (int64_t r = 0; r < steps; ++r) {
        const double f = order == 1 ? -dt : -dt / 2.0;
        for (int64_t k = 0; k < n_terms; ++k) elems.push_back(pauli_exp_elem(terms[k], 0.0, f, (int)k));
        for (int64_t k = n_terms - 1; order == 2 && k >= 0; --k)
            elems.push_back(pauli_exp_elem(terms[k], 0.0, f, (int)k));
    }
    return elems;
}

static Status trotter_steps(qi_state *s, const qi_pauli_term *terms, int64_t n_terms, double dt, int64_t num_steps,
                            int32_t order, bool unitary, const qi_pauli_term *observable, int64_t n_obs,
                            int64_t observe_every, double *energies_out) {
    // FP32: the step is one fused plan: narrow exponentials compose into dense
    // blocks (FP64 composition) and runs of Z-type exponentials into phase
    // polynomials.  With real coefficients every exponential is unitary, so the
    // plan may use the tensor-core blocks and renormalise once per step; complex
    // coefficients (a non-unitary step) keep the CUDA-core blocks and the norm.
    // FP64: FP64 arithmetic is scarce on this part (dense FP64 blocks would be
    // compute-bound), so the exponentials run as gate runs, two operations per
    // amplitude each; where some cannot (wide X strings), each run of exponentials whose
    // X-masks lie in {0, X} is one pass with a parity-indexed table.
    const bool observing = observable && observe_every > 0;
    // FP64 second-order steps: the terms that end one step begin the next, and equal exponentials with
    // nothing between join (qi_gaterun.cu), so a plan covers several steps: the most up to 6 that divide
    // the steps to take (one plan to build; the joined fraction grows as 1 - 1 / steps), else 4.
    // Below 17 qubits a step takes the device less time than the host needs to schedule it.
    int64_t many = 1;
    if (s->prec == QI_F64 && order == 2 && s->n >= 17) {
        const int64_t span = observing ? std::min(observe_every, num_steps) : num_steps;
        const int64_t cap = std::min<int64_t>({span, 6, std::max<int64_t>(1, 1000 / n_terms)});
        for (int64_t k = 2; k <= cap; ++k)
            if (span % k == 0) many = k;
        if (many == 1) many = std::min<int64_t>(cap, 4);
    }
    qi_plan single, several;
    bool have_single = false, have_several = false;
    auto prepare = [&](qi_plan &plan, int64_t steps) {
        plan.n = s->n;
        plan.prec = s->prec;
        plan.opts.use_tensor_cores = unitary ? 0 : 2;
        plan.device_blocks = true;
        // FP32: gate runs cost by the exponential, blocks by the step (about 10 blocks of a lattice, whether it
        // has 50 terms or 140) and by the plan (composing).  Per call, us, runs / blocks: 20 qubits, 113-term
        // XYZ, 1 step 230 / 359, 5 steps 822 / 733, 51-term TFIM, 20 steps 1413 / 2028; 18 qubits XYZ, 10 and 20
        // steps 851 / 943, 1612 / 1635; 21 qubits, XYZ, 1 and 5 steps 329 / 372, 1329 / 815, TFIM, 20 steps 2229 /
        // 2820; 22 qubits XYZ, 1 step 474 / 406, TFIM, 2 and 10 steps 403 / 554, 1819 / 1580; 24 qubits, XYZ and
        // TFIM, 1 step 1786 / 823, 667 / 712; second order, 20 qubits XYZ, 2 and 5 steps 599 / 662, 1286 / 1103.
        // The constants below are fitted to these: lattices of strings on two neighbouring qubits.  Strings of more
        // than six qubits join no block, and 200 of them are 200 launches a step as blocks, which the rule does
        // not know.
        const double size = std::ldexp(1.0, s->n - 20), halves = (double)(order * num_steps), nt = (double)n_terms;
        const double runs = halves * nt * (0.65 + 0.68 * size);
        const double pass = std::max({55.0, 15.0 * (s->n - 14), 33.0 * size});
        const double blocks = 250.0 * order + halves * std::max(1.0, nt / 140.0) * pass;
        // Nor where blocks are more exact: below 13 qubits, and in one or two passes over the terms (13 to 21
        // qubits: 0.44-1.7 times the blocks' error; in three and more 0.09-0.82).
        plan.run_min = 13;
        plan.run_max = runs <= blocks && order * num_steps >= 3 ? s->n : 0;
        plan.opts.renorm_every = unitary ? 0 : -1;
        plan.opts.max_block_qubits = 0;
        std::vector<Elem> elems = step_list(terms, n_terms, dt, order, steps);
        // FP64: grouped exponentials only where some element cannot join a gate run
        plan.opts.fusion = QI_FUSION_GREEDY;
        if (s->prec == QI_F64) {
            plan.opts.fusion = QI_FUSION_NONE;
            for (const Elem &el : elems)
                if (!run_supported(s->n, s->prec, el)) plan.opts.fusion = QI_FUSION_PAULI_GROUPS;
        }
        return build_plan(&plan, elems);
    };
    // which of the two plans the steps will take
    auto chunk = [&](int64_t step) {
        const int64_t left = observing ? std::min(num_steps - step, observe_every - step % observe_every) : num_steps - step;
        return many > 1 && left >= many ? many : 1;
    };
    for (int64_t step = 0; step < num_steps; step += chunk(step)) {
        have_single = have_single || chunk(step) == 1;
        have_several = have_several || chunk(step) > 1;
        if (have_single && (have_several || many == 1)) break;
    }
    Status st = ok_status();
    if (have_single) st = prepare(single, 1);
    if (st.ok() && have_several) st = prepare(several, many);
    if (st.ok()) borrow_runs({&single, &several}, s);
    int64_t obs_k = 0;
    for (int64_t step = 0; step < num_steps && st.ok();) {
        const bool more = chunk(step) > 1;
        st = plan_execute(more ? &several : &single, s);
        if (!st.ok()) break;
        step += more ? many : 1;
        if (observing && step % observe_every == 0) {
            double ev[2];
            st = sumop_expectation(s, observable, n_obs, ev);
            if (!st.ok()) break;
            energies_out[2 * obs_k] = ev[0];
            energies_out[2 * obs_k + 1] = ev[1];
            ++obs_k;
        }
    }
    for (qi_plan *plan : {&single, &several}) {
        if (plan->d_mats) cudaFree(plan->d_mats);
        if (plan->d_tc) cudaFree(plan->d_tc);
        release_runs(plan);
        plan->d_tc = nullptr;
        plan->d_mats = nullptr;
    }
    const cudaError_t e = cudaStreamSynchronize(s->stream);   // the programs are in use until then
    if (st.ok() && e != cudaSuccess) st = cuda_status(e, "trotter");
    return st;
}

qi_status qi_trotter_evolve(qi_state *s, const qi_pauli_term *terms, int64_t n_terms, double dt, int64_t num_steps,
                            int32_t order, const qi_pauli_term *observable, int64_t n_obs, int64_t observe_every,
                            double *energies_out) {
    if (!s || (!terms && n_terms > 0)) return publish(err(QI_ERR_NULL_ARGUMENT));
    std::lock_guard<std::recursive_mutex> lk(s->mu);
    cudaError_t e = cudaSetDevice(s->device);
    if (e != cudaSuccess) return publish(cuda_status(e, "cudaSetDevice"));
    if (n_terms == 0) return publish(err(QI_ERR_INVALID_NUMBER_OF_QUBITS, 0));   // time_evolution.rs:51-53
    if (order != 1 && order != 2) return publish(err(QI_ERR_INVALID_INPUT_VALUE, order));
    for (int64_t k = 0; k < n_terms; ++k) {
        Status st = validate_pauli(s->n, terms[k]);
        if (!st.ok()) return publish(st);
    }
    if (observable && observe_every > 0 && !energies_out) return publish(err(QI_ERR_NULL_ARGUMENT));
    bool unitary = true;
    for (int64_t k = 0; k < n_terms; ++k) unitary = unitary && terms[k].coeff_im == 0.0;
    // FP32 states of up to 12 qubits evolve in FP64 and are rounded at the end.  A small step's
    // exponentials are near the identity: FP32 gate runs had 1.3-8 times the error of blocks on one to three
    // steps (lattices of 4 to 10 qubits; 12 qubits, TFIM, second order: 2.3), and blocks of these sizes take a plan
    // of 0.4-1 ms to compose (3x4, XYZ, 1 and 10 steps: blocks 0.93 and 1.50 ms).
    qi_state *wide = nullptr;
    if (s->prec == QI_F32 && s->n <= 12 && unitary && num_steps > 0 && scratch_take(s, QI_F64, &wide).ok()) {
        Status st = state_copy_async(wide, s);
        if (st.ok())
            st = trotter_steps(wide, terms, n_terms, dt, num_steps, order, unitary, observable, n_obs, observe_every, energies_out);
        if (st.ok() && s->n == 12) {   // renormalised where tensor-core blocks would have been (build_runs)
            qi_plan probe;
            probe.n = s->n;
            probe.prec = s->prec;
            std::vector<Elem> elems = step_list(terms, n_terms, dt, order, 1);
            fuse_narrow_exponentials(elems, 6);
            if (any_tc_block(s->n, elems, partition_with_permutations(&probe, elems, 6))) st = state_normalise_device_async(wide);
        }
        if (st.ok()) st = state_copy_async(s, wide);
        e = cudaStreamSynchronize(s->stream);
        if (st.ok() && e != cudaSuccess) st = cuda_status(e, "trotter");
        scratch_give(wide);
        return publish(st);
    }
    return publish(trotter_steps(s, terms, n_terms, dt, num_steps, order, unitary, observable, n_obs, observe_every,
                                 energies_out));
}

}  // extern "C"

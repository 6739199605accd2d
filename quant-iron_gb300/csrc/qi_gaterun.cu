// qi_gaterun.cu — runs of per-gate operations, many to one pass over the state.
//
// A per-gate plan applies each gate with the gate's own arithmetic (2x2 updates of amplitude
// pairs, phases, index exchanges), not with composed matrices.  One kernel per gate streams the
// whole state for every gate; here the host cuts the gate list into passes.  A pass holds the
// amplitudes of a tile (up to 2^11 16-byte units) in shared memory and applies every gate whose
// non-diagonal qubits are local to the tile; diagonal factors and controls may sit on any qubit
// (they are conditions on the amplitude index).  Inside a pass the gates are grouped into phases:
// a thread holds the 2^r units that differ in r of the tile's bits and applies all of the phase's
// gates to them in registers, so shared memory is read and written once per phase.
//
// Arithmetic.  FP64 operations issue at 2 per clock per SM on this part, so they bound every FP64
// pass: an uncontrolled rotation or Hadamard is applied as a scaled matrix with two unit entries
// (2 instead of 4 or 8 operations per amplitude), the scales and global phases multiplied together
// on the host and applied once; diagonal gates become factors on the amplitudes whose index has
// all bits of a mask set (2 operations per amplitude and bit, merged over a phase); exchanges,
// signs and factors of +-i take none.
//
// Measured (benchmark family, FP64): 20 qubits, 40 layers + QFT (1400 gates) 8.6 ms in 1400 launches ->
// 2.6 ms in 24, 25 qubits, 12 layers + QFT 106 -> 34 ms in 14; the FP64 pipe is 86-88 % busy.  FP32 runs are bound
// by instruction issue (77 %, mostly register moves, index and sign arithmetic).
//
// Reference: Gate::apply / Circuit::execute (src/components/gate.rs:99-122, src/circuit.rs:160-172),
// operator.rs:279-2285, PauliString::apply_exp_factor (src/components/pauli_string.rs:237-262).
#include "qi_gaterun.hpp"
#include "qi_runops.cuh"
#include "qi_async.cuh"

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <unordered_map>

namespace qi {

struct RunGeom {
    int32_t tbits, low;
    int8_t pos[16];
    int32_t nphase, prog_units, nslot;
    uint16_t slot_at[kRunMaxSlots];   // 16-byte unit of the RC_PHASE operation that owns the slot
};

// Shared memory: tile | offsets of the tile's rows | program.
template <typename T>
__global__ void __launch_bounds__(256, 3) k_gate_run(typename Cx<T>::V2 *amps, const uint4 *prog, const __grid_constant__ RunGeom g) {
    using V2 = typename Cx<T>::V2;
    constexpr int RB = RunShape<T>::kRegBits, NV = 1 << RB, UB0 = RunShape<T>::kUnitBits;
    extern __shared__ uint4 sm[];
    const int ubits = g.tbits - UB0, lowu = g.low - UB0;
    const uint32_t nunit = 1u << ubits, nrow = 1u << (ubits - lowu), nt = blockDim.x, tid = threadIdx.x;
    uint4 *tile = sm;
    uint64_t *rows = reinterpret_cast<uint64_t *>(sm + nunit);
    uint4 *code = sm + nunit + ((nrow + 1) >> 1);
    const uint64_t tbase = insert_zeros(blockIdx.x, g.pos, g.tbits);
    for (uint32_t r = tid; r < nrow; r += nt) {   // first unit of each row (2^low consecutive amplitudes)
        uint64_t off = 0;
        for (int j = g.low; j < g.tbits; ++j) off |= (uint64_t)((r >> (j - g.low)) & 1u) << g.pos[j];
        rows[r] = off >> UB0;
    }
    for (uint32_t i = tid; i < (uint32_t)g.prog_units; i += nt) copy16(code + i, prog + i);
    __syncthreads();
    launch_wait();       // the program was there before the pass before this one began; the amplitudes are its result
    uint4 *a4 = reinterpret_cast<uint4 *>(amps) + (tbase >> UB0);
    const RunCopy mine(rows, tid, lowu);
    for (uint32_t u = 0; u < nunit; u += nt)
        copy16((char *)tile + (mine.at ^ (run_swizzle(u) << 4)), a4 + (mine.first + RunCopy::step(rows, u, lowu)));
    __shared__ V2 slot[kRunMaxSlots];
    copy_wait();
    __syncthreads();
    for (uint32_t i = tid; i < (uint32_t)g.nslot; i += nt) {   // read after the first phase's loads, below
        const RunOpHdr &h = *reinterpret_cast<const RunOpHdr *>(code + g.slot_at[i]);
        V2 f = Cx<T>::make(T(1), T(0));
        const uint4 *t = code + g.slot_at[i] + 2;
        for (int j = 0; j < h.zl; ++j, t += 2)
            if ((tbase & reinterpret_cast<const RunSub *>(t)->cg) == reinterpret_cast<const RunSub *>(t)->cg)
                f = Cx<T>::mul(f, *reinterpret_cast<const V2 *>(t + 1));
        slot[i] = f;
    }
    if (g.nslot) __syncthreads();

    uint32_t pc = 0;
    for (int ph = 0; ph < g.nphase; ++ph) {
        const RunPhaseHdr &hd = *reinterpret_cast<const RunPhaseHdr *>(code + pc);
        const int nops = hd.nops;
        const uint32_t place = run_place(hd, tid, ubits - kRunSelBits, UB0), lbase = place >> 16;
        uint32_t at[1 << kRunSelBits];
        run_units<kRunSelBits>(at, place, hd);
        pc += 2;
        V2 v[NV];
        run_load<T, kRunSelBits>(v, tile, at);
        for (int o = 0; o < nops; ++o) {
            const RunOpHdr &h = *reinterpret_cast<const RunOpHdr *>(code + pc);
            const int op = h.code, xi = h.xi;
            const T *c = reinterpret_cast<const T *>(code + pc + 2);
            const uint4 *next = code + pc + 2;
            const int nsub = h.nsub;
            pc += h.units;
            if (op == RC_PHASE) {
                V2 f = Cx<T>::make(T(1), T(0));
                bool any = false;
                const uint32_t flags = h.act;
                pc += h.sgn - 2;   // h.units is 2
                if (flags & kTileFactor) {
                    f = slot[h.cl];
                    any = true;
                    next += 2 * h.zl;
                }
                for (int j = 0; j < nsub; ++j, next += 2) {
                    const RunSub &sb = *reinterpret_cast<const RunSub *>(next);
                    if ((lbase & sb.cl) == sb.cl && (tbase & sb.cg) == sb.cg) {
                        const V2 w = *reinterpret_cast<const V2 *>(next + 1);
                        f = any ? Cx<T>::mul(f, w) : w;
                        any = true;
                    }
                }
                if (flags & kLaneTable) {
                    const V2 w = reinterpret_cast<const V2 *>(next)[tid & 31u];
                    f = any ? Cx<T>::mul(f, w) : w;
                    any = true;
                    next += 32 * sizeof(V2) / 16;
                }
                if (flags & kWarpTable) {
                    const V2 w = reinterpret_cast<const V2 *>(next)[tid >> 5];
                    f = any ? Cx<T>::mul(f, w) : w;
                    any = true;
                }
                if (any) run_phase_m<T, RC_PHASE>(v, xi, f);
                continue;
            }
            const uint32_t cl = h.cl;
            const uint64_t cg = h.cg;
            if ((lbase & cl) != cl || (tbase & cg) != cg) continue;
            const uint32_t act = h.act;
            const bool odd = (__popc(lbase & h.zl) + __popcll(tbase & h.zg)) & 1;
            const uint32_t sgn = odd ? ~h.sgn : h.sgn;
            const bool sign = h.zl || h.zg || h.sgn || (xi & (xi - 1));
            switch (op) {
            case RC_REAL_A:
                if (sign) run_pair_x<T, RC_REAL_A, true>(v, xi, act, sgn, c);
                else run_pair_x<T, RC_REAL_A, false>(v, xi, act, sgn, c);
                break;
            case RC_REAL_H: run_pair_x<T, RC_REAL_H, false>(v, xi, act, sgn, c); break;
            case RC_REAL_X:
                if (sign) run_pair_x<T, RC_REAL_X, true>(v, xi, act, sgn, c);
                else run_pair_x<T, RC_REAL_X, false>(v, xi, act, sgn, c);
                break;
            case RC_IMAG_A:
                if (sign) run_pair_x<T, RC_IMAG_A, true>(v, xi, act, sgn, c);
                else run_pair_x<T, RC_IMAG_A, false>(v, xi, act, sgn, c);
                break;
            case RC_IMAG_X:
                if (sign) run_pair_x<T, RC_IMAG_X, true>(v, xi, act, sgn, c);
                else run_pair_x<T, RC_IMAG_X, false>(v, xi, act, sgn, c);
                break;
            case RC_REAL_G: run_pair_x<T, RC_REAL_G, false>(v, xi, act, sgn, c); break;
            case RC_GEN: run_pair_x<T, RC_GEN, true>(v, xi, act, sgn, c); break;
            case RC_PERM: run_perm_x<T>(v, xi, 255, act); break;   // one form: less code beats fewer selects
            case RC_LIFT:
                run_phase_m<T, RC_LIFT>(v, xi, Cx<T>::make(c[0], c[1]));
                if (nsub == 1) run_phase_m<T, RC_I>(v, xi, Cx<T>::make(T(0), T(0)));
                else if (nsub == 2) run_phase_m<T, RC_NEG>(v, xi, Cx<T>::make(T(0), T(0)));
                else if (nsub == 3) run_phase_m<T, RC_NI>(v, xi, Cx<T>::make(T(0), T(0)));
                break;
            case RC_NEG: run_phase_m<T, RC_NEG>(v, xi, Cx<T>::make(T(0), T(0))); break;
            case RC_I: run_phase_m<T, RC_I>(v, xi, Cx<T>::make(T(0), T(0))); break;
            case RC_NI: run_phase_m<T, RC_NI>(v, xi, Cx<T>::make(T(0), T(0))); break;
            case RC_PARITY: {
                const V2 fe = Cx<T>::make(c[0], c[1]), fo = Cx<T>::make(c[2], c[3]);
#pragma unroll
                for (int k = 0; k < NV; ++k) v[k] = Cx<T>::mul(((sgn >> k) & 1u) ? fo : fe, v[k]);
                break;
            }
            default: {   // RC_SCALE
                const V2 f = Cx<T>::make(c[0], c[1]);
                if (f.y == T(0)) {
#pragma unroll
                    for (int k = 0; k < NV; ++k) v[k] = Cx<T>::make(v[k].x * f.x, v[k].y * f.x);
                } else {
#pragma unroll
                    for (int k = 0; k < NV; ++k) v[k] = Cx<T>::mul(f, v[k]);
                }
                break;
            }
            }
        }
        run_store<T, kRunSelBits>(v, tile, at);
        __syncthreads();
    }
    // Not earlier: while this pass still computes, the next one's blocks would crowd the SMs that are free
    // (256 tiles, FP32, 20 qubits: 0.50 -> 0.63 ms per 20 layers).
    launch_next();
    for (uint32_t u = 0; u < nunit; u += nt)
        a4[mine.first + RunCopy::step(rows, u, lowu)] = *reinterpret_cast<uint4 *>((char *)tile + (mine.at ^ (run_swizzle(u) << 4)));
}

static size_t run_smem(const RunPass &p, int unit_bit) {
    const int ubits = p.tbits - unit_bit, lowu = p.low - unit_bit;
    return ((size_t)16 << ubits) + (((size_t)8 << (ubits - lowu)) + 15) / 16 * 16 + (size_t)p.prog_bytes;
}

Status launch_run_pass(qi_state *s, const RunPass &p, const void *d_prog) {
    const bool f32 = s->prec == QI_F32;
    const int ub0 = f32 ? 1 : 0, ubits = p.tbits - ub0;
    RunGeom g;
    g.tbits = p.tbits;
    g.low = p.low;
    std::copy(p.pos, p.pos + 16, g.pos);
    g.nphase = p.nphase;
    g.prog_units = p.prog_bytes / 16;
    g.nslot = (int32_t)p.slot_at.size();
    std::copy(p.slot_at.begin(), p.slot_at.end(), g.slot_at);
    const size_t sm = run_smem(p, ub0);
    const unsigned threads = 1u << (ubits - kRunSelBits), blocks = (unsigned)(s->dim() >> p.tbits);
    const uint4 *prog = reinterpret_cast<const uint4 *>((const char *)d_prog + p.prog_off);
    // The default limit of 48 KB counts the kernel's static block (the slots) too.
    if (sm + kRunMaxSlots * sizeof(double2) > 48 * 1024) {
        constexpr int cap = (16 << kRunTileBits) + (8 << kRunTileBits) + kRunMaxProg;   // every pass's bound
        if (f32) QI_CUDA(cudaFuncSetAttribute(k_gate_run<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
        else QI_CUDA(cudaFuncSetAttribute(k_gate_run<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
    }
    // A pass's setup (row table, program) overlaps the end of the pass before it: 20 layers of FP64, 12 / 16 /
    // 20 qubits 0.255 / 0.351 / 1.503 -> 0.239 / 0.328 / 1.458 ms; FP32, 17 qubits 0.255 -> 0.229 ms.
    // From 4096 tiles on there is nothing left to gain, and other streams' kernels find SMs between passes.
    ChainedLaunch at(blocks, threads, sm, s->stream, blocks <= 4096);
    if (f32) QI_CUDA(cudaLaunchKernelEx(&at.cfg, k_gate_run<float>, (float2 *)s->amps, prog, g));
    else QI_CUDA(cudaLaunchKernelEx(&at.cfg, k_gate_run<double>, (double2 *)s->amps, prog, g));
    count_launch();
    return check_launch("k_gate_run");
}

// ------------------------------------------------------------ lowering --
using cd = std::complex<double>;

// Double-double complex numbers for the products the host forms (global factors, merged phases, their
// tables): a plan's coefficients are applied again and again (Trotter steps), where roundings of a
// product of many factors would add up coherently.
struct DD {
    double h = 0.0, l = 0.0;
    DD() {}
    DD(double x) : h(x) {}
    DD(double hi, double lo) : h(hi), l(lo) {}
};
static inline DD dd_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return DD(s, (a - (s - t)) + (b - t));
}
static inline DD operator+(const DD &a, const DD &b) {
    DD s = dd_sum(a.h, b.h);
    return dd_sum(s.h, s.l + (a.l + b.l));
}
static inline DD operator-(const DD &a) { return DD(-a.h, -a.l); }
static inline DD operator*(const DD &a, const DD &b) {
    const double p = a.h * b.h;
    return dd_sum(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
static inline DD dd_div(const DD &a, const DD &b) {
    const double q = a.h / b.h;
    const DD r = a + -(b * DD(q));
    return dd_sum(q, r.h / b.h);
}
struct CDD {
    DD re, im;
    CDD(double r = 1.0, double i = 0.0) : re(r), im(i) {}
    CDD(const DD &r, const DD &i) : re(r), im(i) {}
    CDD(const cd &z) : re(z.real()), im(z.imag()) {}
    cd value() const { return cd(re.h, im.h); }
    bool one() const { return re.h == 1.0 && re.l == 0.0 && im.h == 0.0; }
};
static inline CDD operator*(const CDD &a, const CDD &b) {
    return CDD(a.re * b.re + -(a.im * b.im), a.re * b.im + a.im * b.re);
}
static inline CDD cdd_div(const CDD &a, const CDD &b) {
    const DD n = b.re * b.re + b.im * b.im;
    const CDD p = a * CDD(b.re, -b.im);
    return CDD(dd_div(p.re, n), dd_div(p.im, n));
}

struct RunElem {
    int code = RC_PERM;
    uint64_t xs = 0, zs = 0;         // qubits acted on non-diagonally / diagonally
    uint64_t cmask = 0;              // controls, or the AND mask of a phase
    uint64_t xmask = 0, zmask = 0;   // pair partner, sign parity
    double c[8] = {0};
    CDD f;                           // RC_PHASE: the factor
    CDD scale;                       // left to the run's global factor
    int der = 0, slot = -1;          // SweepDer of a parametric gate of a reverse sweep, and its slot
    bool rot = false;                // rc + rs P' with P' P' = -1: exp(i angle P), P = (xmask, zmask)
    DD rc, rs;
    bool diag() const { return xs == 0; }
};

static constexpr int max_x_weight(int prec) { return prec == QI_F32 ? 2 : 3; }

static bool finite_all(const double *m, int k) {
    for (int i = 0; i < k; ++i)
        if (!std::isfinite(m[i])) return false;
    return true;
}

bool run_supported(int n, int prec, const Elem &e) {
    if (n < kRunSelBits + (prec == QI_F32 ? 1 : 0)) return false;
    const GateMatrix &g = e.gm;
    if (g.measure || g.normalise_after) return false;
    if (g.pauli) {
        if (!std::isfinite(g.alpha_re) || !std::isfinite(g.alpha_im)) return false;
        return __builtin_popcountll(g.xmask) <= max_x_weight(prec);
    }
    if (g.nt == 0) return true;
    if (g.nt == 2) return g.kind == QI_GATE_SWAP;
    return finite_all(g.m, 8);
}

namespace {

struct Lowering {
    int prec;
    std::vector<RunElem> out;
    CDD scalar;                     // product of the diagonal gates' global factors
    std::vector<uint64_t> last_x;   // per qubit: number of elements up to the last non-diagonal one
    std::vector<uint64_t> last_any;
    std::unordered_map<uint64_t, uint64_t> phase_at;   // the same for the latest phase of each mask
    explicit Lowering(int p) : prec(p), last_x(64, 0), last_any(64, 0) {}

    void touch(uint64_t xs, uint64_t zs, uint64_t at) {
        for (uint64_t m = xs; m; m &= m - 1) last_x[__builtin_ctzll(m)] = at;
        for (uint64_t m = xs | zs; m; m &= m - 1) last_any[__builtin_ctzll(m)] = at;
    }
    void push(const RunElem &e) {
        out.push_back(e);
        touch(e.xs, e.zs, out.size());
    }
    // factor f on the amplitudes whose index has all bits of m set; joins an earlier phase of the
    // same mask when nothing non-diagonal on those qubits lies between
    void phase(uint64_t m, const CDD &f) {
        if (f.one()) return;
        if (m == 0) {
            scalar = scalar * f;
            return;
        }
        uint64_t since = 0;
        for (uint64_t b = m; b; b &= b - 1) since = std::max(since, last_x[__builtin_ctzll(b)]);
        const auto at = phase_at.find(m);
        if (at != phase_at.end() && at->second > since) {
            out[at->second - 1].f = out[at->second - 1].f * f;
            return;
        }
        RunElem e;
        e.code = RC_PHASE;
        e.zs = e.cmask = m;
        e.f = f;
        push(e);
        phase_at[m] = out.size();
    }
    void diagonal(uint64_t ctl, int t, cd d0, cd d1) {
        phase(ctl, d0);
        phase(ctl | (1ull << t), cdd_div(d1, d0));
    }
    void pair(int code, uint64_t x, uint64_t z, uint64_t ctl, std::initializer_list<double> c, CDD scale = CDD()) {
        RunElem e;
        e.scale = scale;
        e.code = code;
        e.xmask = x;
        e.zmask = z;
        e.cmask = ctl;
        e.xs = x;
        e.zs = (ctl | z) & ~x;
        std::copy(c.begin(), c.end(), e.c);
        push(e);
    }
    static bool near_unit(cd z) { return std::abs(z) > 0.5 && std::abs(z) < 2.0; }

    void matrix1(const GateMatrix &g) {
        const double *m = g.m;
        const int t = g.t[0];
        uint64_t ctl = 0;
        for (int32_t c : g.controls) ctl |= 1ull << c;
        const uint64_t x = 1ull << t;
        const cd m00(m[0], m[1]), m01(m[2], m[3]), m10(m[4], m[5]), m11(m[6], m[7]);
        const cd zero(0.0, 0.0);
        if (m01 == zero && m10 == zero && near_unit(m00) && near_unit(m11)) return diagonal(ctl, t, m00, m11);
        if (m00 == zero && m11 == zero && near_unit(m01) && near_unit(m10)) {   // exchange after a diagonal
            diagonal(ctl, t, m10, m01);
            return pair(RC_PERM, x, 0, ctl, {});
        }
        const bool real = m[1] == 0 && m[3] == 0 && m[5] == 0 && m[7] == 0;
        if (real) {
            const double r00 = m[0], r01 = m[2], r10 = m[4], r11 = m[6];
            const bool unit = std::fabs(r00 * r00 + r01 * r01 - 1.0) < 1e-6;
            if (ctl == 0 && unit) {
                if (std::fabs(r00) >= std::fabs(r01) && std::fabs(r11) == std::fabs(r00)) {
                    return pair(r11 == r00 ? RC_REAL_A : RC_REAL_H, x, 0, 0, {r01 / r00, r10 / r00}, r00);
                }
                if (std::fabs(r00) < std::fabs(r01) && r10 == -r01) {
                    return pair(RC_REAL_X, x, 0, 0, {r00 / r01, r11 / r01}, r01);
                }
            }
            return pair(RC_REAL_G, x, 0, ctl, {r00, r01, r10, r11});
        }
        // c and i s: RX
        if (ctl == 0 && m[1] == 0 && m[7] == 0 && m[2] == 0 && m[4] == 0 && m[0] == m[6] && m[3] == m[5] &&
            std::fabs(m[0] * m[0] + m[3] * m[3] - 1.0) < 1e-6)
            return rotation(x, 0, false, m[0], m[3]);
        pair(RC_GEN, x, 0, ctl, {m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7]});
    }
    // The ratio t of a scaled rotation's entries and its scale (first: the entry that becomes 1).  FP32
    // states: the scale of the rounded t, so that what is applied is a multiple of a unitary exactly.
    double ratio(const DD &other, const DD &first, DD &scale) const {
        const double t = dd_div(other, first).h;
        scale = first;
        if (prec != QI_F32) return t;
        const double r = (double)(float)t;
        scale = DD(std::copysign(1.0 / std::sqrt(1.0 + r * r), first.h));
        return r;
    }
    // odd = false: a' = c a + i s sigma b, b' = c b + i s sigma a; odd = true: a' = c a + s sigma b,
    // b' = c b - s sigma a.  The larger entry becomes the scale.
    void rotation(uint64_t x, uint64_t z, bool odd, const DD &c, const DD &s) {
        DD f;
        if (std::fabs(c.h) >= std::fabs(s.h)) {
            const double t = ratio(s, c, f);
            pair(odd ? RC_REAL_A : RC_IMAG_A, x, z, 0, {t, odd ? -t : t}, CDD(f, DD()));
        } else {
            const double t = ratio(c, s, f);
            if (odd) pair(RC_REAL_X, x, z, 0, {t, t}, CDD(f, DD()));
            else pair(RC_IMAG_X, x, z, 0, {-t, -t}, CDD(DD(), f));
        }
    }
    // diag(c + i s, c - i s) on qubit q
    void rotation_z(int q, const DD &c, const DD &s) {
        RunElem e;
        DD f;
        e.zs = e.zmask = 1ull << q;
        if (std::fabs(c.h) >= std::fabs(s.h)) {
            e.code = RC_ROTZ_A;
            e.c[0] = ratio(s, c, f);
            e.scale = CDD(f, DD());
        } else {
            e.code = RC_ROTZ_X;
            e.c[0] = ratio(c, s, f);
            e.scale = CDD(f, DD());
        }
        push(e);
    }
    // The inverse of an uncontrolled parametric gate; its derivative term goes to `slot`.
    void unapply(const GateMatrix &g, int slot) {
        const uint64_t x = 1ull << g.t[0];
        switch (g.kind) {
        case QI_GATE_RX: rotation(x, 0, false, g.m[0], -g.m[3]); break;
        case QI_GATE_RY: rotation(x, 0, true, g.m[0], g.m[4]); break;
        case QI_GATE_RZ: rotation_z(g.t[0], g.m[6], g.m[7]); break;
        default: {   // P: half the angle each way, up to a phase psi and lambda share
            const double h = 0.5 * std::atan2(g.m[7], g.m[6]);
            rotation_z(g.t[0], std::cos(h), std::sin(h));
        }
        }
        out.back().der = g.kind == QI_GATE_RX ? kDerX : g.kind == QI_GATE_RY ? kDerY : g.kind == QI_GATE_RZ ? kDerZ : kDerP;
        out.back().slot = slot;
    }
    void pauli(const GateMatrix &g) {   // exp(alpha P)
        const double ar = g.alpha_re, ai = g.alpha_im;
        const cd ch(std::cosh(ar) * std::cos(ai), std::sinh(ar) * std::sin(ai));
        const cd sh(std::sinh(ar) * std::cos(ai), std::cosh(ar) * std::sin(ai));
        if (g.xmask == 0) {
            const cd even = ch + sh, odd = ch - sh;
            const int w = __builtin_popcountll(g.zmask);
            if (w == 0) return phase(0, even);
            if (w <= 2 && near_unit(even) && near_unit(odd)) {   // even * (odd / even)^parity
                phase(0, even);
                const CDD r = cdd_div(odd, even), back = cdd_div(even, odd);
                for (uint64_t b = g.zmask; b; b &= b - 1) phase(b & -b, r);
                if (w == 2) phase(g.zmask, back * back);
                return;
            }
            RunElem e;
            e.code = RC_PARITY;
            e.zs = e.zmask = g.zmask;
            e.c[0] = even.real();
            e.c[1] = even.imag();
            e.c[2] = odd.real();
            e.c[3] = odd.imag();
            return push(e);
        }
        if (ar == 0.0) return exponential(g.xmask, g.zmask, ai);
        const int ny = __builtin_popcountll(g.xmask & g.zmask);
        const cd s = sh * minus_i_to(ny);
        const cd back = (ny & 1) ? -s : s;
        pair(RC_GEN, g.xmask, g.zmask, 0, {ch.real(), ch.imag(), s.real(), s.imag(), back.real(), back.imag(), ch.real(), ch.imag()});
    }
    static cd minus_i_to(int k) {
        static const cd mi_pow[4] = {cd(1, 0), cd(0, -1), cd(-1, 0), cd(0, 1)};
        return mi_pow[k & 3];
    }
    // exp(i angle P): cos + (real or imaginary) sin.  Joins an earlier exponential of the same string when
    // no element between touches its qubits (the middle and the ends of second-order Trotter steps);
    // the two rotations are multiplied, in double-double, so the result is that of applying both.
    void exponential(uint64_t x, uint64_t z, double angle) {
        const int ny = __builtin_popcountll(x & z);
        const bool odd = ny & 1;
        const cd si = cd(0.0, std::sin(angle)) * minus_i_to(ny);
        DD c = std::cos(angle), s = odd ? si.real() : si.imag();
        uint64_t last = 0;
        for (uint64_t b = x | z; b; b &= b - 1) last = std::max(last, last_any[__builtin_ctzll(b)]);
        const bool join = last && out[last - 1].rot && out[last - 1].xmask == x && out[last - 1].zmask == z;
        if (join) {
            const DD c1 = out[last - 1].rc, s1 = out[last - 1].rs, cc = c1 * c + -(s1 * s);
            s = c1 * s + s1 * c;
            c = cc;
        }
        rotation(x, z, odd, c, s);
        out.back().rot = true;
        out.back().rc = c;
        out.back().rs = s;
        if (join) {   // in the earlier one's place
            out[last - 1] = out.back();
            out.pop_back();
            touch(x, z & ~x, last);
        }
    }
    void add(const Elem &el) {
        const GateMatrix &g = el.gm;
        if (g.pauli) return pauli(g);
        if (g.nt == 0) return;
        if (g.nt == 1) return matrix1(g);
        uint64_t ctl = 0;   // SWAP: three controlled exchanges
        for (int32_t c : g.controls) ctl |= 1ull << c;
        const uint64_t a = 1ull << g.t[0], b = 1ull << g.t[1];
        pair(RC_PERM, b, 0, ctl | a, {});
        pair(RC_PERM, a, 0, ctl | b, {});
        pair(RC_PERM, b, 0, ctl | a, {});
    }
};

// ----------------------------------------------------------- scheduling --
// Greedy absorption: scan `rem` in order and take every element that may act on the chosen bits W
// and commutes with every element passed over (elements commute when each shared qubit is diagonal
// in both).  grow > 0: W may grow up to `grow` bits (within `pool`).  Diagonal elements need one
// of their qubits in W (their factor then costs half of an all-amplitude factor or less).
struct Masks {   // the remaining elements' qubits, side by side
    uint64_t xs, zs;
};
int absorb(const std::vector<Masks> &rem, uint64_t &W, uint64_t pool, int grow, std::vector<int> *take) {
    uint64_t bx = 0, bz = 0;
    if (take) take->clear();
    int score = 0;
    const size_t count = rem.size();
    for (size_t i = 0; i < count; ++i) {
        const uint64_t xs = rem[i].xs, zs = rem[i].zs;
        bool can = !((xs & (bx | bz)) | (zs & bx));
        if (can) {
            if (xs == 0) {
                if (!(zs & W)) {
                    const uint64_t lo = zs & pool;
                    can = grow && lo && i == 0 && __builtin_popcountll(W) < grow;
                    if (can) W |= lo & -lo;
                }
            } else if (xs & ~W) {
                can = grow && !(xs & ~pool) && __builtin_popcountll(W | xs) <= grow;
                if (can) W |= xs;
            }
        }
        if (can) {
            if (take) take->push_back((int)i);
            score += xs ? 2 : 1;
        } else {
            bx |= xs;
            bz |= zs;
            if ((W & ~bx) == 0 && (!grow || __builtin_popcountll(W) >= grow)) break;
        }
    }
    return score;
}

// The best of the first element's own cone and the windows; W in: the bits that are always in.
uint64_t best_bits(const std::vector<Masks> &rem, uint64_t W0, const std::vector<int> &pool, int bits, std::vector<int> &take) {
    const int have = __builtin_popcountll(W0), width = bits - have;
    uint64_t all = W0;
    for (int q : pool) all |= 1ull << q;
    uint64_t W = W0;
    int score = absorb(rem, W, all, bits, nullptr);
    bool grown = true;
    uint64_t win = 0;
    for (size_t a = 0; a < pool.size(); ++a) {
        win |= 1ull << pool[a];
        if ((int)a >= width) win &= ~(1ull << pool[a - (size_t)width]);
        if ((int)a + 1 < width) continue;
        uint64_t w = W0 | win;
        const int s = absorb(rem, w, 0, 0, nullptr);
        if (s > score) {
            score = s;
            W = w;
            grown = false;
        }
    }
    if (grown) {
        W = W0;
        absorb(rem, W, all, bits, &take);
    } else {
        absorb(rem, W, 0, 0, &take);
    }
    for (size_t a = 0; a < pool.size() && __builtin_popcountll(W) < bits; ++a) W |= 1ull << pool[a];   // unused slots
    return W;
}

struct Encoder {
    int n, prec, ub0;
    RunPass *pass;
    std::vector<int32_t> *der = nullptr;   // slots of the pass's derivative terms, in program order
    std::vector<uint8_t> &prog;
    uint64_t localmask = 0;
    int lbit[64];   // qubit -> local bit or -1

    Encoder(int n_, int prec_, std::vector<uint8_t> &out)
        : n(n_), prec(prec_), ub0(prec_ == QI_F32 ? 1 : 0), pass(nullptr), prog(out) {}
    void begin(RunPass *p) {
        pass = p;
        localmask = 0;
        for (int &b : lbit) b = -1;
        for (int j = 0; j < p->tbits; ++j) {
            lbit[(int)p->pos[j]] = j;
            localmask |= 1ull << p->pos[j];
        }
    }
    void coef(const double *c, int k) {
        const size_t at = prog.size(), sz = prec == QI_F32 ? 4 : 8;
        prog.resize(at + ((size_t)k * sz + 15) / 16 * 16, 0);
        for (int i = 0; i < k; ++i) {
            if (sz == 4) {
                const float f = (float)c[i];
                std::memcpy(&prog[at + 4 * (size_t)i], &f, 4);
            } else {
                std::memcpy(&prog[at + 8 * (size_t)i], &c[i], 8);
            }
        }
    }
    // split a qubit mask into register bits (by rmap), other local bits and tile bits
    void split(uint64_t m, const int8_t *rmap, uint32_t &reg, uint32_t &loc, uint64_t &out) const {
        reg = loc = 0;
        out = m & ~localmask;
        for (uint64_t b = m & localmask; b; b &= b - 1) {
            const int l = lbit[__builtin_ctzll(b)];
            if (rmap[l] >= 0) reg |= 1u << rmap[l];
            else loc |= 1u << l;
        }
    }

    // A term of a phase factor: conditions on the tile's qubits and on local bits.
    struct PhaseTerm {
        int op;
        uint64_t cg;
        uint32_t cl;
        CDD f;
    };
    struct Out {
        RunOpHdr h;
        uint64_t xs;
        int nterm, nc;
        double c[8];
    };
    std::vector<Out> list;           // the phase's operations
    std::vector<PhaseTerm> terms;    // of all its RC_PHASE operations
    std::vector<const PhaseTerm *> mine, tile, lane, warp, rest;

    template <typename S> void raw(const S &x) {
        const uint8_t *p = reinterpret_cast<const uint8_t *>(&x);
        prog.insert(prog.end(), p, p + sizeof(S));
    }
    void sub_term(const PhaseTerm &t) {
        raw(RunSub{t.cg, t.cl, 0});
        const double c[2] = {t.f.re.h, t.f.im.h};
        coef(c, 2);
    }
    // A factor whose value does not depend on the thread or the tile beyond one condition: a sign, a
    // factor of +-i, or (unit modulus) a rotation by three shears after taking out the nearest power of i.
    static bool single_factor(Out &o, const PhaseTerm &t) {
        const cd f = t.f.value();
        o.h.cl = (uint16_t)t.cl;
        o.h.cg = t.cg;
        const int exact = f == cd(-1, 0) ? RC_NEG : f == cd(0, 1) ? RC_I : f == cd(0, -1) ? RC_NI : 0;
        if (exact) {
            o.h.code = (uint8_t)exact;
            return true;
        }
        if (std::fabs(std::norm(f) - 1.0) > 0x1p-50) return false;
        const double pi = 3.14159265358979323846;
        const int turn = ((int)std::lround(std::arg(f) / (pi / 2)) + 4) & 3;
        static const cd back[4] = {cd(1, 0), cd(0, -1), cd(-1, 0), cd(0, 1)};
        const cd r = f * back[turn];   // exact: a power of i
        o.h.code = RC_LIFT;
        o.h.nsub = (uint8_t)turn;
        o.c[0] = r.imag() / (1.0 + r.real());
        o.c[1] = r.imag();
        o.nc = 2;
        return true;
    }
    // The parts of an RC_PHASE factor: terms on tile qubits alone become a tile factor; two or more on
    // thread bits alone become tables (one multiplication each instead of one per term).
    void write_phase(Out &o, int index, const RunPhaseHdr &hd) {
        mine.clear();
        for (const PhaseTerm &t : terms)
            if (t.op == index) mine.push_back(&t);
        const int nthread = pass->tbits - ub0 - kRunSelBits, nwarp = std::min(4, std::max(0, nthread - 5));
        uint32_t lanes = 0, warps = 0;
        for (int j = 0; j < nthread; ++j) (j < 5 ? lanes : warps) |= 1u << (hd.tb[j] + ub0);
        tile.clear();
        lane.clear();
        warp.clear();
        rest.clear();
        for (const PhaseTerm *t : mine) {
            if (t->cl == 0 && t->cg != 0) tile.push_back(t);
            else if (t->cg == 0 && t->cl && !(t->cl & ~lanes)) lane.push_back(t);
            else if (t->cg == 0 && t->cl && !(t->cl & ~warps)) warp.push_back(t);
            else rest.push_back(t);
        }
        auto back = [&](std::vector<const PhaseTerm *> &v, size_t least) {
            if (v.size() >= least) return;
            rest.insert(rest.end(), v.begin(), v.end());
            v.clear();
        };
        back(tile, pass->slot_at.size() < (size_t)kRunMaxSlots ? 2 : SIZE_MAX);
        back(lane, 2);
        back(warp, 2);
        const size_t at = prog.size();
        o.h.units = 2;
        o.h.nsub = (uint8_t)rest.size();
        if (!tile.empty()) {
            o.h.act |= kTileFactor;
            o.h.zl = (uint16_t)tile.size();
            o.h.cl = (uint16_t)pass->slot_at.size();
            pass->slot_at.push_back((uint16_t)((at - (size_t)pass->prog_off) / 16));
        }
        if (!lane.empty()) o.h.act |= kLaneTable;
        if (!warp.empty()) o.h.act |= kWarpTable;
        raw(o.h);
        for (const PhaseTerm *t : tile) sub_term(*t);
        for (const PhaseTerm *t : rest) sub_term(*t);
        auto table = [&](const std::vector<const PhaseTerm *> &v, int first, int bits) {
            double c[64];
            for (uint32_t i = 0; i < (1u << bits); ++i) {
                uint32_t l = 0;
                for (int j = 0; j < bits && first + j < nthread; ++j) l |= ((i >> j) & 1u) << (hd.tb[first + j] + ub0);
                CDD f;
                for (const PhaseTerm *t : v)
                    if ((l & t->cl) == t->cl) f = f * t->f;
                c[2 * i] = f.re.h;
                c[2 * i + 1] = f.im.h;
            }
            coef(c, 2 << bits);
        };
        if (!lane.empty()) table(lane, 0, 5);
        if (!warp.empty()) table(warp, 5, nwarp);
        const uint32_t units = (uint32_t)((prog.size() - at) / 16);
        std::memcpy(&prog[at + offsetof(RunOpHdr, sgn)], &units, sizeof(units));
    }

    // One phase: R = register qubits; ops = elements in order; scale: applied after them.
    void phase(const std::vector<RunElem> &E, const std::vector<int> &ops, uint64_t R, const cd *scale) {
        RunPhaseHdr hd;
        std::memset(&hd, 0, sizeof(hd));
        const int ubits = pass->tbits - ub0;
        int8_t rmap[16];
        std::fill(rmap, rmap + 16, (int8_t)-1);
        if (ub0) rmap[0] = 0;
        uint32_t regu = 0;
        int nr = 0;
        for (int u = 0; u < ubits; ++u)
            if ((R >> pass->pos[u + ub0]) & 1ull) {
                rmap[u + ub0] = (int8_t)(nr++ + ub0);
                regu |= 1u << u;
            }
        run_phase_bits(hd, regu, ubits);

        list.clear();
        terms.clear();
        const int nv = 1 << (kRunSelBits + ub0);
        for (int idx : ops) {
            const RunElem &e = E[(size_t)idx];
            uint32_t reg, loc;
            uint64_t out;
            split(e.cmask, rmap, reg, loc, out);
            if (e.code == RC_PHASE) {
                bool joined = false;
                for (size_t i = list.size(); i-- > 0 && !joined;) {
                    if (list[i].nterm && list[i].h.xi == reg) {
                        ++list[i].nterm;
                        terms.push_back(PhaseTerm{(int)i, out, loc, e.f});
                        joined = true;
                    } else if (list[i].xs & e.zs) {
                        break;
                    }
                }
                if (joined) continue;
            }
            list.emplace_back();
            Out &o = list.back();
            std::memset(&o.h, 0, sizeof(o.h));
            o.xs = e.xs;
            o.nterm = o.nc = 0;
            o.h.code = (uint8_t)e.code;
            if (e.code == RC_PHASE) {
                o.h.xi = (uint8_t)reg;
                o.nterm = 1;
                terms.push_back(PhaseTerm{(int)list.size() - 1, out, loc, e.f});
                continue;
            }
            o.h.cl = (uint16_t)loc;
            o.h.cg = out;
            for (int k = 0; k < nv; ++k)
                if (((uint32_t)k & reg) == reg) o.h.act |= 1u << k;
            if (e.code == RC_PERM) o.h.nsub = (uint8_t)((reg & (reg - 1)) ? 255u : reg);
            split(e.xmask, rmap, reg, loc, out);
            o.h.xi = (uint8_t)reg;
            // sign parity is taken on the partner with the highest qubit of xmask clear: the register
            // bits ascend with the qubits, so that is the partner with the top bit of xi clear
            split(e.zmask, rmap, reg, loc, out);
            o.h.zl = (uint16_t)loc;
            o.h.zg = out;
            for (int k = 0; k < nv; ++k)
                if (__builtin_popcount((uint32_t)k & reg) & 1) o.h.sgn |= 1u << k;
            if (e.code == RC_ROTZ_A || e.code == RC_ROTZ_X) o.h.xi = (uint8_t)reg;
            switch (e.code) {
            case RC_REAL_A: case RC_REAL_H: case RC_REAL_X: case RC_IMAG_A: case RC_IMAG_X: o.nc = 2; break;
            case RC_REAL_G: case RC_PARITY: o.nc = 4; break;
            case RC_GEN: o.nc = 8; break;
            case RC_ROTZ_A: case RC_ROTZ_X: o.nc = 1; break;
            default: break;
            }
            if (e.der) {   // uncontrolled: cg holds the term's place
                o.h.nsub = (uint8_t)e.der;
                o.h.cg = der->size();
                der->push_back(e.slot);
            }
            std::copy(e.c, e.c + 8, o.c);
        }
        if (scale) {
            list.emplace_back();
            Out &o = list.back();
            std::memset(&o.h, 0, sizeof(o.h));
            o.h.code = RC_SCALE;
            o.nterm = 0;
            o.nc = 2;
            o.c[0] = scale->real();
            o.c[1] = scale->imag();
        }
        hd.nops = (uint16_t)list.size();
        raw(hd);
        for (size_t i = 0; i < list.size(); ++i) {
            Out &o = list[i];
            if (o.nterm) {
                bool whole = o.nterm == 1;
                if (whole) {
                    for (const PhaseTerm &t : terms)
                        if (t.op == (int)i) whole = single_factor(o, t);
                }
                if (!whole) {
                    write_phase(o, (int)i, hd);
                    continue;
                }
            }
            o.h.units = (uint8_t)(2 + (o.nc * (prec == QI_F32 ? 4 : 8) + 15) / 16);
            raw(o.h);
            coef(o.c, o.nc);
        }
        ++pass->nphase;
    }
};

}  // namespace

// Tile size in 16-byte units, measured on 20 layers + QFT (before phases were applied as shears), ms for
// 2^9 / 2^10 / 2^11 / 2^12 units.
// FP64: 16 qubits 0.403 / 0.383 / 0.504 / 0.786, 20 qubits 1.73 / 1.64 / 1.83 / 1.98, 25 qubits
// 58.2 / 56.6 / 57.1 / 67.9: six small tiles keep an SM's FP64 pipe busier through barriers and tile
// loads than two large ones, which outweighs the extra passes.  FP32 is bound by instruction issue:
// 16 qubits 0.273 / 0.270 / 0.286 / 0.362, 22 qubits 1.79 / 1.59 / 1.49 / 1.66.
static int run_tile_units(int n, int ub0) {
    const int u = n - ub0;
    return std::min(u, ub0 && n >= 20 ? 11 : 10);
}

// The greedy schedule of E into passes.  sweep: reverse-sweep passes (each pass's derivative terms, with
// the squared size of the scales left out when they are taken); no global factor at the end.
static void schedule_elems(int n, int prec, const std::vector<RunElem> &E, CDD scalar, int tbits, std::vector<RunPass> *passes,
                           std::vector<SweepPass> *sweep, std::vector<uint8_t> &prog) {
    const int ub0 = prec == QI_F32 ? 1 : 0;
    const int low = tbits >= n ? n : 3 + ub0;   // rows of 128 bytes (rows of 512: up to 10 % slower, more passes)
    const uint64_t lowmask = (1ull << low) - 1, always = ub0 ? 1ull : 0ull;
    // The product of the scales left out so far; it is applied at the end of the run, or at the end of a phase when
    // it has become small.  The amplitudes grow as its reciprocal, and a phase of 48 rotations adds 2^24 at most:
    // FP32 states of amplitudes above 2^73 may overflow inside a run (no normalised state comes near).
    const double small = prec == QI_F32 ? 0x1p-30 : 0x1p-300;
    if (E.empty() && (sweep || scalar.one())) return;
    std::vector<int> rem(E.size()), take, ptake, inner, group, rest, free_q, sel_q;
    std::vector<Masks> masks(E.size()), imasks;
    for (size_t i = 0; i < E.size(); ++i) {
        rem[i] = (int)i;
        masks[i] = Masks{E[i].xs, E[i].zs};
    }
    for (int q = low; q < n; ++q) free_q.push_back(q);
    std::vector<char> gone(E.size(), 0);
    const int rbits = kRunSelBits + ub0;
    Encoder enc(n, prec, prog);
    do {
        uint64_t W = n >= 64 ? ~0ull : (1ull << n) - 1;
        inner.clear();
        if (tbits < n) {
            W = best_bits(masks, lowmask, free_q, tbits, take);
            for (int i : take) inner.push_back(rem[(size_t)i]);
        } else {
            inner = rem;
        }
        RunPass pass;
        SweepPass terms;
        enc.der = &terms.slot;
        pass.tbits = tbits;
        int np = 0;
        sel_q.clear();
        for (int q = 0; q < n; ++q)
            if ((W >> q) & 1ull) {
                pass.pos[np++] = (int8_t)q;
                if (!((always >> q) & 1ull)) sel_q.push_back(q);
            }
        while (pass.low < tbits && pass.pos[pass.low] == pass.low) ++pass.low;
        if (tbits < n) pass.low = std::min(pass.low, 5 + ub0);   // a shared table of row offsets
        pass.prog_off = (int32_t)prog.size();
        enc.begin(&pass);
        size_t ndone = 0;
        imasks.clear();
        for (int i : inner) imasks.push_back(Masks{E[(size_t)i].xs, E[(size_t)i].zs});
        do {
            const uint64_t R = best_bits(imasks, always, sel_q, rbits, ptake);
            group.clear();
            if (ptake.size() > kRunMaxPhase) ptake.resize(kRunMaxPhase);
            for (int i : ptake) group.push_back(inner[(size_t)i]);
            CDD after = scalar;
            for (int i : group) {
                if (E[(size_t)i].der) terms.size2.push_back(std::norm(after.value()));
                if (!E[(size_t)i].scale.one()) after = after * E[(size_t)i].scale;
            }
            const bool last = !sweep && ndone + group.size() == rem.size();
            const cd now = after.value();
            const bool apply = (last && !after.one()) || std::abs(now) < small;
            const size_t used = prog.size(), slots = pass.slot_at.size(), nder = terms.slot.size();
            enc.phase(E, group, R, apply ? &now : nullptr);
            if (prog.size() - (size_t)pass.prog_off > (size_t)kRunMaxProg || (sweep && terms.slot.size() > (size_t)kSweepTerms) ||
                (sweep && pass.nphase > kSweepPhases)) {   // left to the next pass
                prog.resize(used);
                pass.slot_at.resize(slots);
                terms.slot.resize(nder);
                terms.size2.resize(nder);
                --pass.nphase;
                break;
            }
            scalar = apply ? CDD() : after;
            ndone += group.size();
            for (int i : group) gone[(size_t)i] = 1;
            size_t k = 0;
            for (size_t i = 0; i < inner.size(); ++i)
                if (!gone[(size_t)inner[i]]) {
                    inner[k] = inner[i];
                    imasks[k++] = imasks[i];
                }
            inner.resize(k);
            imasks.resize(k);
        } while (!inner.empty());
        pass.prog_bytes = (int32_t)(prog.size() - (size_t)pass.prog_off);
        if (sweep) {
            terms.run = std::move(pass);
            sweep->push_back(std::move(terms));
        } else {
            passes->push_back(std::move(pass));
        }
        size_t k = 0;
        for (size_t i = 0; i < rem.size(); ++i)
            if (!gone[(size_t)rem[i]]) {
                rem[k] = rem[i];
                masks[k++] = masks[i];
            }
        rem.resize(k);
        masks.resize(k);
    } while (!rem.empty());
}

void schedule_run(int n, int prec, const std::vector<const Elem *> &elems, RunSegment &seg, std::vector<uint8_t> &prog) {
    Lowering lw(prec);
    const int ub0 = prec == QI_F32 ? 1 : 0;
    for (const Elem *e : elems) lw.add(*e);
    schedule_elems(n, prec, lw.out, lw.scalar, run_tile_units(n, ub0) + ub0, &seg.passes, nullptr, prog);
}

bool sweep_supported(int n, int prec, const GateMatrix &g, int nparams) {
    if (n < kRunSelBits + (prec == QI_F32 ? 1 : 0) || g.pauli || g.measure || g.normalise_after) return false;
    if (nparams) {
        const bool kind = g.kind == QI_GATE_RX || g.kind == QI_GATE_RY || g.kind == QI_GATE_RZ || g.kind == QI_GATE_P;
        return nparams == 1 && kind && g.nt == 1 && g.controls.empty() && finite_all(g.m, 8);
    }
    if (g.nt == 0) return true;
    if (g.nt == 2) return g.kind == QI_GATE_SWAP;
    return finite_all(g.m, 8);
}

void schedule_sweep(int n, int prec, const std::vector<SweepGate> &gates, std::vector<SweepPass> &passes,
                    std::vector<uint8_t> &prog) {
    Lowering lw(prec);
    const int ub0 = prec == QI_F32 ? 1 : 0;
    for (const SweepGate &sg : gates) {
        const GateMatrix &g = *sg.g;
        if (sg.slot >= 0) {
            lw.unapply(g, sg.slot);
            continue;
        }
        if (g.nt == 0) continue;
        if (prec == QI_F32 && g.nt == 1 && g.controls.empty() && g.diagonal) {
            // a fixed phase as the same exact multiple of a unitary (up to a phase both states share);
            // quarter turns stay exact factors
            const cd r = std::conj(cdd_div(CDD(cd(g.m[6], g.m[7])), CDD(cd(g.m[0], g.m[1]))).value());
            const bool quarter = r == cd(1, 0) || r == cd(-1, 0) || r == cd(0, 1) || r == cd(0, -1);
            if (!quarter && std::fabs(std::norm(r) - 1.0) < 1e-12) {
                const double h = -0.5 * std::arg(r);
                lw.rotation_z(g.t[0], std::cos(h), std::sin(h));
                continue;
            }
        }
        Elem e;
        e.gm = g;
        if (g.nt == 1)
            for (int i = 0; i < 2; ++i)
                for (int j = 0; j < 2; ++j) {
                    e.gm.m[2 * (2 * i + j)] = g.m[2 * (2 * j + i)];
                    e.gm.m[2 * (2 * i + j) + 1] = -g.m[2 * (2 * j + i) + 1];
                }
        lw.add(e);
    }
    // 12-layer ansatz, ms with tiles of 2^9 / 2^10 / 2^11 units: FP32 20 qubits 5.1 / 4.3 / 4.2, 22 qubits
    // 9.2 / 7.8 / 7.2 (larger blocks share the instruction stream); FP64 16 qubits, 8 layers 4.1 / 3.9 / 4.2
    const int units = std::min(n - ub0, prec == QI_F32 && n >= 20 ? 11 : 10);
    schedule_elems(n, prec, lw.out, CDD(), units + ub0, nullptr, &passes, prog);
}

// -------------------------------------------------------------- replay --
void replay_run_pass(int n, const RunPass &p, const uint8_t *prog0, cd *amps) {
    const uint8_t *prog = prog0 + p.prog_off;
    const uint64_t ntile = 1ull << (n - p.tbits);
    const uint32_t nl = 1u << p.tbits;
    std::vector<uint64_t> off(nl);
    for (uint32_t l = 0; l < nl; ++l) {
        off[l] = 0;
        for (int j = 0; j < p.tbits; ++j) off[l] |= (uint64_t)((l >> j) & 1u) << p.pos[j];
    }
    std::vector<cd> tile(nl);
    for (uint64_t t = 0; t < ntile; ++t) {
        uint64_t tb = t;
        for (int j = 0; j < p.tbits; ++j) {
            const uint64_t lo = tb & ((1ull << p.pos[j]) - 1);
            tb = ((tb >> p.pos[j]) << (p.pos[j] + 1)) | lo;
        }
        for (uint32_t l = 0; l < nl; ++l) tile[l] = amps[tb | off[l]];
        size_t pc = 0;
        for (int ph = 0; ph < p.nphase; ++ph) {
            RunPhaseHdr hd;
            std::memcpy(&hd, prog + pc, sizeof(hd));
            pc += sizeof(hd);
            size_t end = pc;
            for (uint32_t th = 0; th < (nl >> kRunSelBits); ++th) {
                uint32_t base = 0;
                for (int j = 0; j < p.tbits - kRunSelBits; ++j) base |= ((th >> j) & 1u) << hd.tb[j];
                uint32_t at[1 << kRunSelBits];
                cd v[1 << kRunSelBits];
                for (uint32_t k = 0; k < (1u << kRunSelBits); ++k) {
                    at[k] = base;
                    for (int j = 0; j < kRunSelBits; ++j) at[k] |= ((k >> j) & 1u) << hd.rb[j];
                    v[k] = tile[at[k]];
                }
                size_t q = pc;
                for (int o = 0; o < hd.nops; ++o) {
                    RunOpHdr h;
                    std::memcpy(&h, prog + q, sizeof(h));
                    const uint8_t *body = prog + q + sizeof(h);
                    q += (size_t)(h.code == RC_PHASE ? h.sgn : h.units) * 16;
                    double c[8] = {0};
                    if (h.code != RC_PHASE) std::memcpy(c, body, std::min<size_t>(sizeof(c), (size_t)(h.units - 2) * 16));
                    if (h.code == RC_PHASE) {
                        cd f(1, 0);
                        const int terms = h.nsub + ((h.act & kTileFactor) ? h.zl : 0);
                        for (int j = 0; j < terms; ++j, body += 32) {
                            RunSub sb;
                            std::memcpy(&sb, body, sizeof(sb));
                            double w[2];
                            std::memcpy(w, body + 16, 16);
                            if ((base & sb.cl) == sb.cl && (tb & sb.cg) == sb.cg) f *= cd(w[0], w[1]);
                        }
                        double w[2];
                        if (h.act & kLaneTable) {
                            std::memcpy(w, body + 16 * (th & 31u), 16);
                            f *= cd(w[0], w[1]);
                            body += 512;
                        }
                        if (h.act & kWarpTable) {
                            std::memcpy(w, body + 16 * (th >> 5), 16);
                            f *= cd(w[0], w[1]);
                        }
                        for (uint32_t k = 0; k < (1u << kRunSelBits); ++k)
                            if ((k & h.xi) == h.xi) v[k] *= f;
                        continue;
                    }
                    if ((base & h.cl) != h.cl || (tb & h.cg) != h.cg) continue;
                    const bool odd = (__builtin_popcount(base & h.zl) + __builtin_popcountll(tb & h.zg)) & 1;
                    const uint32_t sgn = odd ? ~h.sgn : h.sgn;
                    for (uint32_t k = 0; k < (1u << kRunSelBits); ++k) {
                        const double s = ((sgn >> k) & 1u) ? -1.0 : 1.0;
                        if (h.code >= RC_NEG && h.code <= RC_NI) {
                            if ((k & h.xi) == h.xi) v[k] *= h.code == RC_NEG ? cd(-1, 0) : h.code == RC_I ? cd(0, 1) : cd(0, -1);
                            continue;
                        }
                        if (h.code == RC_LIFT) {
                            static const cd turn[4] = {cd(1, 0), cd(0, 1), cd(-1, 0), cd(0, -1)};
                            if ((k & h.xi) != h.xi) continue;
                            const double x = v[k].real() - c[0] * v[k].imag(), y = v[k].imag() + c[1] * x;
                            v[k] = cd(x - c[0] * y, y) * turn[h.nsub];
                            continue;
                        }
                        if (h.code == RC_PARITY) {
                            v[k] *= s < 0 ? cd(c[2], c[3]) : cd(c[0], c[1]);
                            continue;
                        }
                        if (h.code == RC_SCALE) {
                            v[k] *= cd(c[0], c[1]);
                            continue;
                        }
                        int top = 1;
                        while (2 * top <= h.xi) top *= 2;
                        if ((int)k & top || !((h.act >> k) & 1u)) continue;
                        const cd a = v[k], b = v[k ^ h.xi];
                        cd na = b, nb = a;
                        switch (h.code) {
                        case RC_REAL_A: na = a + s * c[0] * b; nb = b + s * c[1] * a; break;
                        case RC_REAL_H: na = a + c[0] * b; nb = c[1] * a - b; break;
                        case RC_REAL_X: na = s * b + c[0] * a; nb = c[1] * b - s * a; break;
                        case RC_IMAG_A: na = a + cd(0, s * c[0]) * b; nb = b + cd(0, s * c[1]) * a; break;
                        case RC_IMAG_X: na = s * b + cd(0, c[0]) * a; nb = s * a + cd(0, c[1]) * b; break;
                        case RC_REAL_G: na = c[0] * a + c[1] * b; nb = c[2] * a + c[3] * b; break;
                        case RC_GEN:
                            na = cd(c[0], c[1]) * a + s * cd(c[2], c[3]) * b;
                            nb = s * cd(c[4], c[5]) * a + cd(c[6], c[7]) * b;
                            break;
                        default: break;
                        }
                        v[k] = na;
                        v[k ^ h.xi] = nb;
                    }
                }
                end = q;
                for (uint32_t k = 0; k < (1u << kRunSelBits); ++k) tile[at[k]] = v[k];
            }
            pc = end;
        }
        for (uint32_t l = 0; l < nl; ++l) amps[tb | off[l]] = tile[l];
    }
}

}  // namespace qi

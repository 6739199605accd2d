// qi_sumrun.cu — <psi|H|psi> and H|psi> of a sum of Pauli strings, many X-mask groups to a pass.
//
// Terms that share an X mask x act on the same amplitude pairs (i, i ^ x):
//   (H psi)_i = sum_g f_g(i) psi_{i ^ x_g},  f_g(i) = sum_k c_k (-i)^ny (-1)^popc(i & z_k),
//   <psi|H|psi> = sum_g sum_pairs f_g(i) conj(psi_i) psi_j + f_g(j) conj(psi_j) psi_i.
// A pass holds a tile of the state in shared memory, as the gate runs do (qi_runtile.cuh), and handles
// every group whose x lies within the tile's qubits: in each phase a thread has the amplitudes of
// three (FP32: four) index bits in registers, so a pair group costs no further loads.  The
// 25-qubit open chain's 25 groups take 3 passes over the state instead of 25.
//
// f_g(i) is one of at most four values, chosen by up to two parities of i: a table the host makes,
// selected per pair.  FP64 arithmetic bounds the FP64 passes (2 operations per clock per SM):
// an expectation pair costs 3 operations, an applied pair 8, where evaluating f_g by additions
// and multiplying complex numbers took 20 and more.  The diagonal group (x = 0) sums its terms by
// local Z mask once per tile (the signs on the tile's fixed qubits are then part of the
// coefficients), a thread adds them per register Z mask, and a Walsh-Hadamard transform over the
// register bits gives f of all its amplitudes.
//
// Measured, open Heisenberg chain, host call to result, one pass per group before -> now (ms): <H> FP64
// 25 qubits 22.9 -> 3.2, 20 qubits 1.11 -> 0.19; FP32 27 qubits 4.98 -> 1.68, 20 qubits 0.55 -> 0.10,
// 10 qubits 0.33 -> 0.06.  H|psi> FP64 25 qubits 16.2 -> 3.65; FP32 27 qubits 3.76 -> 3.48, 20 qubits
// 0.23 -> 0.09.  FP64 passes keep the FP64 pipe 86 % busy; FP32 passes are bound by instruction issue
// (a pass over 2^25 FP32 amplitudes 0.10 ms, 0.04 at the copy rate).
//
// Reference: SumOp::apply / expectation_value (src/components/pauli_string.rs:453-507).
#include "qi_sumrun.hpp"
#include "qi_runtile.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>

namespace qi {

// ------------------------------------------------------------- program --
// Per phase a RunPhaseHdr, then its groups.  A pair group: header and, for each value e = b0 + 2 b1 of
// the parities over the bits outside the registers, the weights of the 2^(S + unit bits - 1) register
// pairs in ascending order (the parities over register bits are worked into them: no test per pair).
// The diagonal group: header (zg0 = register masks that occur), offsets by register Z mask and one uint16 local Z mask per distinct mask,
// sorted by the mask's register bits.
struct SumHdr {        // 32 bytes
    uint8_t kind;      // kPair* / kDiag*
    uint8_t xi;        // register partner mask
    uint8_t r;         // parities the weights depend on
    uint8_t pad;
    uint32_t units;    // 16-byte size
    uint32_t stride;   // values per e
    uint16_t zl0, zl1;
    uint64_t zg0, zg1;
};
static_assert(sizeof(SumHdr) == 32, "program layout");
// Weights of a pair, c = conj(psi_i) psi_j.  Expectation: kPairFirst re += w Re c; kPairSecond
// re += w Im c; kPairGeneral (p, q, s, t) re += p Re c + q Im c, im += s Re c + t Im c.
// Apply, f(i) and f(j): kPairFirst real (f, g); kPairSecond imaginary; kPairGeneral (f, g) complex.
// kDiagSplit (FP32, real coefficients): every coefficient as a multiple of 2^-23 of their sum's size, whose sums are
// exact in FP32, and the rest; both are summed and transformed.  Sums of rounded coefficients err alike in all
// amplitudes that share them: <H> of fields and bonds on 10 to 19 qubits 1.2-2.2 times the error of a factor per
// amplitude (0.5-0.8 from 20 on), split 0.04-0.35.
enum SumKind : int { kPairFirst = 0, kPairSecond = 1, kPairGeneral = 2, kDiagReal = 3, kDiagComplex = 4, kDiagSplit = 5 };
constexpr int kMaxPhases = 24;  // phases of a pass (their thread tables: 1 KB each at most)
constexpr int kMaxDiag = 96;   // distinct local Z masks of a pass's diagonal group
constexpr int kMaxDiagTerms = 256;
constexpr int kSplitExpect = 19, kSplitApply = 11;   // kDiagSplit up to this many qubits
// Register bits of a phase: FP64 3 (its arithmetic is the bound), FP32 4 (a phase's set-up and an
// operation's decoding are shared by 32 amplitudes instead of 16)
// of an expectation; an applied phase holds the sums too and keeps to 3
template <typename T, bool APPLY> struct SumShape {
    static constexpr int S = sizeof(T) == 8 || APPLY ? 3 : 4, kRegBits = S + RunShape<T>::kUnitBits;
};

struct DiagEntry {     // table of the diagonal group: terms [first, first + count) have this local mask
    uint32_t first, count;
};
template <typename T> struct alignas(16) DiagTerm {
    uint64_t zg;       // Z bits on the tile's fixed qubits
    T re, im;
};

struct SumGeom {
    int32_t tbits, low;
    int8_t pos[16];
    int32_t nphase, prog_units, ndiag, diag_at;
    int32_t cplx, diag_cplx, nterm;
};

// -------------------------------------------------------------- kernel --
__device__ __forceinline__ void keep(float2 &v) { asm volatile("" : "+f"(v.x), "+f"(v.y)); }
__device__ __forceinline__ void keep(double2 &v) { asm volatile("" : "+d"(v.x), "+d"(v.y)); }

template <typename T, int N>
__device__ __forceinline__ void load_weights(T (&w)[N], const T *c) {   // c 16-byte aligned
    static_assert(N * sizeof(T) % 16 == 0, "whole units");
#pragma unroll
    for (int i = 0; i < N; i += 16 / (int)sizeof(T)) {
        if constexpr (sizeof(T) == 4) {
            const float4 q = *reinterpret_cast<const float4 *>(c + i);
            w[i] = q.x, w[i + 1] = q.y, w[i + 2] = q.z, w[i + 3] = q.w;
        } else {
            const double2 q = *reinterpret_cast<const double2 *>(c + i);
            w[i] = q.x, w[i + 1] = q.y;
        }
    }
}

// A thread's sum.  FP64: of a tile.  FP32: of all its tiles (PairSum): FP64 operations would bound the pass, and
// FP32 sums of a tile's groups lost up to eight times the bits of sums of single pairs.
template <typename T> struct SumAcc {
    T v = T(0);
};
template <> struct SumAcc<float> : PairSum {};

// FINE (FP32 expectations): every pair on its own enters the sum, else chains of eight do.
template <typename T, int X, int KIND, bool APPLY, bool FINE>
__device__ __forceinline__ void sum_pair(const typename Cx<T>::V2 (&v)[1 << SumShape<T, APPLY>::kRegBits],
                                         typename Cx<T>::V2 (&o)[APPLY ? 1 << SumShape<T, APPLY>::kRegBits : 1], const T *c,
                                         SumAcc<T> &re, SumAcc<T> &im) {
    using V2 = typename Cx<T>::V2;
    constexpr int NV = 1 << SumShape<T, APPLY>::kRegBits, NP = NV / 2, NW = KIND == kPairGeneral ? 4 : APPLY ? 2 : 1;
    constexpr int STEP = 4 / NW;   // pairs whose weights are loaded together
    [[maybe_unused]] T part = T(0);
    [[maybe_unused]] T t[2] = {T(0), T(0)}, u[2] = {T(0), T(0)};   // FP32: two chains of each component
#pragma unroll
    for (int p0 = 0; p0 < NP; p0 += STEP) {
        T w[STEP * NW];
        load_weights<T, STEP * NW>(w, c + p0 * NW);
#pragma unroll
        for (int j = 0; j < STEP; ++j) {
            const int p = p0 + j, k = (p & (top_bit(X) - 1)) | ((p & ~(top_bit(X) - 1)) << 1);
            const V2 a = v[k], b = v[k ^ X];
            const T *f = w + j * NW;
            if constexpr (APPLY) {
                if constexpr (KIND == kPairFirst) {
                    o[k] = Cx<T>::make(::fma(f[0], b.x, o[k].x), ::fma(f[0], b.y, o[k].y));
                    o[k ^ X] = Cx<T>::make(::fma(f[1], a.x, o[k ^ X].x), ::fma(f[1], a.y, o[k ^ X].y));
                } else if constexpr (KIND == kPairSecond) {
                    o[k] = Cx<T>::make(::fma(-f[0], b.y, o[k].x), ::fma(f[0], b.x, o[k].y));
                    o[k ^ X] = Cx<T>::make(::fma(-f[1], a.y, o[k ^ X].x), ::fma(f[1], a.x, o[k ^ X].y));
                } else {
                    o[k] = Cx<T>::fma(Cx<T>::make(f[0], f[1]), b, o[k]);
                    o[k ^ X] = Cx<T>::fma(Cx<T>::make(f[2], f[3]), a, o[k ^ X]);
                }
            } else if constexpr (sizeof(T) == 4) {
                T &acc = t[p & 1], &acc_im = u[p & 1];
                if (FINE) acc = acc_im = T(0);
                if constexpr (KIND == kPairGeneral) {
                    const T cr = ::fma(a.x, b.x, a.y * b.y), ci = ::fma(a.x, b.y, -a.y * b.x);
                    acc = ::fma(f[0], cr, ::fma(f[1], ci, acc));
                    acc_im = ::fma(f[2], cr, ::fma(f[3], ci, acc_im));
                } else {
                    const T x = KIND == kPairFirst ? ::fma(a.x, b.x, a.y * b.y) : ::fma(a.x, b.y, -a.y * b.x);
                    acc = ::fma(f[0], x, acc);
                }
                if ((p & 1) && (FINE || p == NP - 1)) {
                    re.add(t[0], t[1]);
                    if constexpr (KIND == kPairGeneral) im.add(u[0], u[1]);
                }
            } else {
                T &acc = (p & 1) ? part : re.v;   // two chains
                if constexpr (KIND == kPairFirst) {
                    acc = ::fma(f[0], ::fma(a.x, b.x, a.y * b.y), acc);
                } else if constexpr (KIND == kPairSecond) {
                    acc = ::fma(f[0], ::fma(a.x, b.y, -a.y * b.x), acc);
                } else {
                    const T cr = ::fma(a.x, b.x, a.y * b.y), ci = ::fma(a.x, b.y, -a.y * b.x);
                    acc = ::fma(f[0], cr, ::fma(f[1], ci, acc));
                    im.v = ::fma(f[2], cr, ::fma(f[3], ci, im.v));
                }
            }
        }
    }
    if constexpr (!APPLY && sizeof(T) == 8) re.v += part;
}

// Dispatch on the partner mask; MASKS of three bits only for the one-component kinds.
template <typename T, int KIND, bool APPLY, bool FINE>
__device__ __forceinline__ void sum_pair_x(int xi, const typename Cx<T>::V2 (&v)[1 << SumShape<T, APPLY>::kRegBits],
                                           typename Cx<T>::V2 (&o)[APPLY ? 1 << SumShape<T, APPLY>::kRegBits : 1], const T *c,
                                           SumAcc<T> &re, SumAcc<T> &im) {
#define QI_X(M) case M: sum_pair<T, M, KIND, APPLY, FINE>(v, o, c, re, im); break;
    switch (xi) {
        QI_X(1) QI_X(2) QI_X(3) QI_X(4) QI_X(5) QI_X(6)
    default: break;
    }
    if constexpr (KIND != kPairGeneral || sizeof(T) == 8) {
        if (xi == 7) sum_pair<T, 7, KIND, APPLY, FINE>(v, o, c, re, im);
    }
    if constexpr (sizeof(T) == 4) {
        switch (xi) {
            QI_X(8) QI_X(9) QI_X(10) QI_X(12) QI_X(16) QI_X(17) QI_X(18) QI_X(20) QI_X(24)
        default: break;
        }
        if constexpr (KIND != kPairGeneral) {
            switch (xi) {
                QI_X(11) QI_X(13) QI_X(14) QI_X(19) QI_X(21) QI_X(22) QI_X(25) QI_X(26) QI_X(28)
            default: break;
            }
        }
    }
#undef QI_X
}

template <typename T, bool APPLY, bool FINE>
__global__ void __launch_bounds__(1 << (kRunTileBits - SumShape<T, APPLY>::S), 512 >> (kRunTileBits - SumShape<T, APPLY>::S))
    k_sum_run(const typename Cx<T>::V2 *in, typename Cx<T>::V2 *out, int add,
                                                 uint64_t ntiles, const uint4 *prog, const __grid_constant__ SumGeom g,
                                                 double *partials) {
    using V2 = typename Cx<T>::V2;
    constexpr int S = SumShape<T, APPLY>::S, NV = 1 << SumShape<T, APPLY>::kRegBits, UB0 = RunShape<T>::kUnitBits;
    extern __shared__ uint4 sm[];
    __shared__ V2 dcoef[kMaxDiag], dterm[kMaxDiagTerms];
    __shared__ uint64_t next_base;
    const int ubits = g.tbits - UB0, lowu = g.low - UB0;
    const uint32_t nunit = 1u << ubits, nrow = 1u << (ubits - lowu), nt = blockDim.x, tid = threadIdx.x;
    uint4 *tile = sm, *otile = sm + nunit;   // otile: APPLY only
    uint64_t *rows = reinterpret_cast<uint64_t *>(sm + (APPLY ? 2 : 1) * nunit);
    uint4 *code = sm + (APPLY ? 2 : 1) * nunit + ((nrow + 1) >> 1);
    uint32_t *places = reinterpret_cast<uint32_t *>(code + g.prog_units);   // [phase][thread]
    for (uint32_t r = tid; r < nrow; r += nt) {   // row offsets within the tile
        uint64_t off = 0;
        for (int j = g.low; j < g.tbits; ++j) off |= (uint64_t)((r >> (j - g.low)) & 1u) << g.pos[j];
        rows[r] = off >> UB0;
    }
    for (uint32_t i = tid; i < (uint32_t)g.prog_units; i += nt) copy16(code + i, prog + i);
    const uint4 *in4 = reinterpret_cast<const uint4 *>(in);
    uint4 *out4 = reinterpret_cast<uint4 *>(out);
    double dre = 0.0, dim = 0.0;
    SumAcc<T> re, im;
    copy_wait();
    __syncthreads();
    uint32_t pc0 = 0;
    for (int ph = 0; ph < g.nphase; ++ph) {   // the threads' places are the same for every tile
        const RunPhaseHdr &hd = *reinterpret_cast<const RunPhaseHdr *>(code + pc0);
        places[ph * nt + tid] = run_place(hd, tid, ubits - S, UB0);
        pc0 += 2;
        for (int q = 0; q < hd.nops; ++q) pc0 += reinterpret_cast<const SumHdr *>(code + pc0)->units;
    }
    const RunCopy mine(rows, tid, lowu);
    uint64_t tbase = insert_zeros(blockIdx.x, g.pos, g.tbits);
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        if (tid == 0) next_base = insert_zeros(t + gridDim.x, g.pos, g.tbits);   // read after the barriers below
        const uint64_t first = (tbase >> UB0) + mine.first;
        for (uint32_t u = 0; u < nunit; u += nt)
            copy16((char *)tile + (mine.at ^ (run_swizzle(u) << 4)), in4 + (first + RunCopy::step(rows, u, lowu)));
        if (APPLY && add)
            for (uint32_t u = 0; u < nunit; u += nt)
                copy16((char *)otile + (mine.at ^ (run_swizzle(u) << 4)), out4 + (first + RunCopy::step(rows, u, lowu)));
        copy_wait();
        __syncthreads();
        if (g.ndiag) {   // the diagonal terms' coefficients by local Z mask, with this tile's signs
            const DiagEntry *ent = reinterpret_cast<const DiagEntry *>(code + g.diag_at);
            const DiagTerm<T> *term = reinterpret_cast<const DiagTerm<T> *>(code + g.diag_at + (g.ndiag + 1) / 2);
            for (uint32_t k = tid; k < (uint32_t)g.nterm; k += nt) {   // one term a thread, then the sums in term order
                const uint32_t s = (uint32_t)__popcll(tbase & term[k].zg) & 1u;
                dterm[k] = Cx<T>::make(flip_sign(term[k].re, s), flip_sign(term[k].im, s));
            }
            __syncthreads();
            for (uint32_t i = tid; i < (uint32_t)g.ndiag; i += nt) {
                T re = T(0), im = T(0);
                const uint32_t end = ent[i].first + ent[i].count;
                for (uint32_t k = ent[i].first; k < end; ++k) re += dterm[k].x;
                for (uint32_t k = ent[i].first; g.diag_cplx && k < end; ++k) im += dterm[k].y;
                dcoef[i] = Cx<T>::make(re, im);
            }
            __syncthreads();
        }
        if constexpr (sizeof(T) == 8) re.v = im.v = T(0);
        uint32_t pc = 0;
        for (int ph = 0; ph < g.nphase; ++ph) {
            const RunPhaseHdr &hd = *reinterpret_cast<const RunPhaseHdr *>(code + pc);
            const int nops = hd.nops;
            const uint32_t place = places[ph * nt + tid], lbase = place >> 16;
            uint32_t at[1 << S];
            run_units<S>(at, place, hd);
            pc += 2;
            V2 v[NV], o[APPLY ? NV : 1];
            run_load<T, S>(v, tile, at);
            if constexpr (APPLY) {
                if (add || ph) {
                    run_load<T, S>(o, otile, at);
                } else {
#pragma unroll
                    for (int k = 0; k < NV; ++k) o[k] = Cx<T>::make(T(0), T(0));
                }
            }
            for (int q = 0; q < nops; ++q) {
                if constexpr (!APPLY) {
                    // the amplitudes do not change in this loop: without this the compiler computes the
                    // products of every pair of every mask before it (52 FP64 operations per amplitude
                    // in place of 11, and 255 registers)
#pragma unroll
                    for (int k = 0; k < NV; ++k) keep(v[k]);
                }
                const SumHdr &h = *reinterpret_cast<const SumHdr *>(code + pc);
                const int kind = h.kind;
                if (kind >= kDiagReal) {
                    const uint16_t *range = reinterpret_cast<const uint16_t *>(code + pc + 2), *mask = range + NV + 1;
                    for (int part = 0; part < (kind == kDiagReal ? 1 : 2); ++part) {
                        T A[NV];
#pragma unroll
                        for (int m = 0; m < NV; ++m) {
                            T a = T(0);
                            if (!((h.zg0 >> m) & 1u)) {   // no terms with these register bits
                                A[m] = a;
                                continue;
                            }
                            for (int k = range[m]; k < range[m + 1]; ++k) {
                                const T cf = part ? dcoef[k].y : dcoef[k].x;
                                a += flip_sign(cf, (uint32_t)__popc(lbase & mask[k]) & 1u);
                            }
                            A[m] = a;
                        }
#pragma unroll
                        for (int b = 1; b < NV; b <<= 1)   // f[k] = sum_m A[m] (-1)^popc(k & m)
#pragma unroll
                            for (int m = 0; m < NV; ++m)
                                if (!(m & b)) {
                                    const T x = A[m], y = A[m | b];
                                    A[m] = x + y;
                                    A[m | b] = x - y;
                                }
                        [[maybe_unused]] T t[2] = {T(0), T(0)};   // FP32: two chains, FINE: two values
#pragma unroll
                        for (int k = 0; k < NV; ++k) {
                            if constexpr (APPLY) {
                                if (part == 0 || kind == kDiagSplit) o[k] = Cx<T>::make(::fma(A[k], v[k].x, o[k].x), ::fma(A[k], v[k].y, o[k].y));
                                else o[k] = Cx<T>::make(::fma(-A[k], v[k].y, o[k].x), ::fma(A[k], v[k].x, o[k].y));
                            } else {
                                const T p = ::fma(v[k].x, v[k].x, v[k].y * v[k].y);
                                if constexpr (sizeof(T) == 4) {
                                    t[k & 1] = ::fma(A[k], p, FINE ? T(0) : t[k & 1]);
                                    if ((k & 1) && (FINE || k == NV - 1)) {
                                        if (part && kind == kDiagComplex) im.add(t[0], t[1]);
                                        else re.add(t[0], t[1]);
                                    }
                                } else {
                                    if (part == 0) re.v = ::fma(A[k], p, re.v);
                                    else im.v = ::fma(A[k], p, im.v);
                                }
                            }
                        }
                    }
                    pc += h.units;
                    continue;
                }
                const T *c = reinterpret_cast<const T *>(code + pc + 2);
                if (h.r >= 1 && ((__popc(lbase & h.zl0) + __popcll(tbase & h.zg0)) & 1)) c += h.stride;
                if (h.r == 2 && ((__popc(lbase & h.zl1) + __popcll(tbase & h.zg1)) & 1)) c += 2 * h.stride;
                const int xi = h.xi;
                pc += h.units;
                if (kind == kPairFirst) sum_pair_x<T, kPairFirst, APPLY, FINE>(xi, v, o, c, re, im);
                else if (kind == kPairSecond) sum_pair_x<T, kPairSecond, APPLY, FINE>(xi, v, o, c, re, im);
                else sum_pair_x<T, kPairGeneral, APPLY, FINE>(xi, v, o, c, re, im);
            }
            if constexpr (APPLY) {
                run_store<T, S>(o, otile, at);
                __syncthreads();
            }
        }
        if constexpr (APPLY) {
            for (uint32_t u = 0; u < nunit; u += nt)
                out4[first + RunCopy::step(rows, u, lowu)] =
                    *reinterpret_cast<uint4 *>((char *)otile + (mine.at ^ (run_swizzle(u) << 4)));
        } else if constexpr (sizeof(T) == 8) {
            dre += re.v;
            if (g.cplx) dim += im.v;
        }
        tbase = next_base;
        __syncthreads();   // the tile is read to the end before the next one lands
    }
    if constexpr (!APPLY) {
        if constexpr (sizeof(T) == 4) {
            dre = re.total();
            if (g.cplx) dim = im.total();
        }
        const double r0 = block_sum(dre), r1 = block_sum(dim);
        if (tid == 0) {
            partials[blockIdx.x * 4 + 0] = r0;
            partials[blockIdx.x * 4 + 1] = r1;
        }
    }
}

static SumGeom sum_geom(const SumPass &p) {
    SumGeom g;
    g.tbits = p.tile.tbits;
    g.low = p.tile.low;
    std::copy(p.tile.pos, p.tile.pos + 16, g.pos);
    g.nphase = p.tile.nphase;
    g.prog_units = p.tile.prog_bytes / 16;
    g.ndiag = p.ndiag;
    g.diag_at = p.diag_at;
    g.cplx = p.complex_out ? 1 : 0;
    g.diag_cplx = p.diag_complex ? 1 : 0;
    g.nterm = p.nterm;
    return g;
}
static size_t sum_smem(const SumPass &p, int ub0, int tiles, int sel) {
    const int ubits = p.tile.tbits - ub0, lowu = p.tile.low - ub0;
    return ((size_t)tiles * 16 << ubits) + (((size_t)8 << (ubits - lowu)) + 15) / 16 * 16 + (size_t)p.tile.prog_bytes +
           ((size_t)p.tile.nphase * 4 << (ubits - sel));
}
constexpr int kSumSmemCap = 160 * 1024;   // tiles 64 KB, rows 16 KB, program 24 KB, places 24 KB at most

template <typename T, bool APPLY, bool FINE = false>
static Status launch_sum(cudaStream_t st, uint64_t dim, const void *in, void *out, bool add, const SumPass &p,
                         const void *d_prog, double *partials, unsigned cap, unsigned *blocks) {
    const int ub0 = RunShape<T>::kUnitBits;
    const size_t sm = sum_smem(p, ub0, APPLY ? 2 : 1, SumShape<T, APPLY>::S);
    const uint64_t ntiles = dim >> p.tile.tbits;
    const unsigned threads = 1u << (p.tile.tbits - ub0 - SumShape<T, APPLY>::S);
    const unsigned nb = (unsigned)std::min<uint64_t>(ntiles, cap);
    if (sm > (size_t)kSumSmemCap) return err(QI_ERR_UNKNOWN, (int64_t)sm, kSumSmemCap, "SumOp pass too large");
    if (sm > 36 * 1024)   // beside the static block
        QI_CUDA(cudaFuncSetAttribute(k_sum_run<T, APPLY, FINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSumSmemCap));
    k_sum_run<T, APPLY, FINE><<<nb, threads, sm, st>>>((const typename Cx<T>::V2 *)in, (typename Cx<T>::V2 *)out, add ? 1 : 0, ntiles,
                                                 (const uint4 *)((const char *)d_prog + p.tile.prog_off), sum_geom(p), partials);
    count_launch();
    if (blocks) *blocks = nb;
    return check_launch("k_sum_run");
}

Status launch_sum_expect(qi_state *s, const SumPass &p, const void *d_prog, unsigned *nblocks) {
    const unsigned cap = kReduceBlocks;   // 8 blocks per SM; one row of partials each
    // FP32 up to 22 qubits: every pair on its own, as one launch per group summed them (a thread had 1 pair of a
    // group up to 19 qubits, 7 at 22, 32 from 24 on; here a chain of eight).
    if (s->prec == QI_F32 && s->n <= 22)
        return launch_sum<float, false, true>(s->stream, s->dim(), s->amps, nullptr, false, p, d_prog, s->d_partials, cap, nblocks);
    if (s->prec == QI_F32)
        return launch_sum<float, false>(s->stream, s->dim(), s->amps, nullptr, false, p, d_prog, s->d_partials, cap, nblocks);
    return launch_sum<double, false>(s->stream, s->dim(), s->amps, nullptr, false, p, d_prog, s->d_partials, cap, nblocks);
}

Status launch_sum_apply(qi_state *out, const qi_state *in, const SumPass &p, const void *d_prog, bool add) {
    const unsigned cap = 152 * 12;
    if (out->prec == QI_F32)
        return launch_sum<float, true>(out->stream, out->dim(), in->amps, out->amps, add, p, d_prog, nullptr, cap, nullptr);
    return launch_sum<double, true>(out->stream, out->dim(), in->amps, out->amps, add, p, d_prog, nullptr, cap, nullptr);
}

// ---------------------------------------------------------- scheduling --
namespace {

// Up to two basis parities of a group's Z masks (on the partner with x's highest bit clear).
struct TwoParities {
    uint64_t w[2] = {0, 0};
    int r = 0;
    // subset of the basis whose XOR is z; false when a third would be needed
    bool place(uint64_t z, uint32_t *sub) {
        for (uint32_t s = 0; s < (1u << r); ++s)
            if ((((s & 1u) ? w[0] : 0) ^ ((s & 2u) ? w[1] : 0)) == z) {
                *sub = s;
                return true;
            }
        if (r == 2) return false;
        w[r] = z;
        *sub = 1u << r++;
        return true;
    }
};

// f(i) and f(j) for each value of the parities (entries past 2^r repeat those that exist).
bool pair_table(const SumGroup &g, TwoParities &par, double f[4][4]) {
    const uint64_t hb = 1ull << (63 - __builtin_clzll(g.x));
    std::vector<uint32_t> sub(g.terms.size());
    for (size_t k = 0; k < g.terms.size(); ++k)
        if (!par.place(g.terms[k].z & ~hb, &sub[k])) return false;
    std::memset(f, 0, sizeof(double) * 16);
    for (int e = 0; e < 4; ++e)
        for (size_t k = 0; k < g.terms.size(); ++k) {
            const SumTerm &t = g.terms[k];
            const double si = (__builtin_popcount((uint32_t)e & sub[k]) & 1) ? -1.0 : 1.0;
            const double sj = (__builtin_popcountll(g.x & t.z) & 1) ? -si : si;
            f[e][0] += si * t.re;
            f[e][1] += si * t.im;
            f[e][2] += sj * t.re;
            f[e][3] += sj * t.im;
        }
    return true;
}

bool any_imaginary(const SumGroup &g) {
    for (const SumTerm &t : g.terms)
        if (t.im != 0) return true;
    return false;
}

// Weights of the parities' values and which of them are needed (SumKind).
int pair_weights(const double f[4][4], bool apply, double w[4][4], bool *cplx) {
    bool v[4] = {false, false, false, false};
    for (int e = 0; e < 4; ++e) {
        if (apply) {
            std::copy(f[e], f[e] + 4, w[e]);
        } else {
            w[e][0] = f[e][0] + f[e][2];
            w[e][1] = f[e][3] - f[e][1];
            w[e][2] = f[e][1] + f[e][3];
            w[e][3] = f[e][0] - f[e][2];
        }
        for (int i = 0; i < 4; ++i) v[i] = v[i] || w[e][i] != 0;
    }
    *cplx = !apply && (v[2] || v[3]);
    if (apply) return !v[1] && !v[3] ? kPairFirst : !v[0] && !v[2] ? kPairSecond : kPairGeneral;
    return *cplx ? kPairGeneral : !v[1] ? kPairFirst : !v[0] ? kPairSecond : kPairGeneral;
}

}  // namespace

bool schedule_sum(int n, int prec, bool apply, const std::vector<SumGroup> &groups, std::vector<SumPass> &passes,
                  std::vector<uint8_t> &prog, std::vector<int> *left) {
    const int ub0 = prec == QI_F32 ? 1 : 0;
    const uint64_t always = ub0 ? 1ull : 0ull;
    const int S = prec == QI_F32 && !apply ? SumShape<float, false>::S : SumShape<double, false>::S, rbits = S + ub0;
    std::vector<int> rem;
    int diag = -1;
    bool all = true;
    auto leave = [&](size_t i) {
        all = false;
        if (left) left->push_back((int)i);
    };
    for (size_t i = 0; i < groups.size(); ++i) {
        const SumGroup &g = groups[i];
        TwoParities par;
        double f[4][4], w[4][4];
        bool cplx;
        if (n < rbits) leave(i);
        else if (g.x == 0 && ub0 && !apply && (n >= 25 || any_imaginary(g))) leave(i);   // k_diag_expect_f32 streams at the copy rate
        else if (g.x == 0 && g.terms.size() <= (size_t)kMaxDiagTerms) diag = (int)i;
        else if (g.x == 0 || __builtin_popcountll(g.x) > 3 || !pair_table(g, par, f)) leave(i);
        else if (ub0 && __builtin_popcountll(g.x) == 3 && pair_weights(f, apply, w, &cplx) == kPairGeneral) leave(i);
        else rem.push_back((int)i);
    }
    if (!all && !left) return false;
    // Tiles of 2^10 units (2^11 within 4 % either way, 2^9 up to 70 % slower), rows of 128 bytes.
    const int tbits = std::min(n - ub0, 10) + ub0, low = tbits >= n ? n : 3 + ub0;
    // the bits (W0, then a window of the pool or the first groups' own qubits) that most groups lie in
    auto choose = [&](const std::vector<int> &list, uint64_t W0, const std::vector<int> &pool, int bits) {
        auto score = [&](uint64_t W) {
            int c = 0;
            for (int i : list) c += !(groups[(size_t)i].x & ~W);
            return c;
        };
        uint64_t best = W0;
        for (int i : list)
            if (__builtin_popcountll(best | groups[(size_t)i].x) <= bits) best |= groups[(size_t)i].x;
        int top = score(best);
        const int width = bits - __builtin_popcountll(W0);
        uint64_t win = 0;
        for (size_t a = 0; a < pool.size(); ++a) {
            win |= 1ull << pool[a];
            if ((int)a >= width) win &= ~(1ull << pool[a - (size_t)width]);
            const int s = score(W0 | win);
            if (s > top) {
                top = s;
                best = W0 | win;
            }
        }
        for (size_t a = 0; a < pool.size() && __builtin_popcountll(best) < bits; ++a) best |= 1ull << pool[a];
        return best;
    };
    const size_t op_bytes = sizeof(SumHdr) + (size_t)4 * (ub0 ? 4 : 8) * (4u << (rbits - 1));   // at most
    std::vector<int> pool, sel;
    for (int q = low; q < n; ++q) pool.push_back(q);
    while (!rem.empty() || diag >= 0) {
        const uint64_t W = tbits >= n ? (n >= 64 ? ~0ull : (1ull << n) - 1) : choose(rem, (1ull << low) - 1, pool, tbits);
        SumPass p;
        RunPass &tile = p.tile;
        tile.tbits = tbits;
        int np = 0;
        int lbit[64];
        std::fill(lbit, lbit + 64, -1);
        sel.clear();
        for (int q = 0; q < n; ++q)
            if ((W >> q) & 1ull) {
                lbit[q] = np;
                tile.pos[np++] = (int8_t)q;
                if (!((always >> q) & 1ull)) sel.push_back(q);
            }
        while (tile.low < tbits && tile.pos[tile.low] == tile.low) ++tile.low;
        if (tbits < n) tile.low = std::min(tile.low, 5 + ub0);
        tile.prog_off = (int32_t)prog.size();
        auto bytes = [&]() { return prog.size() - (size_t)tile.prog_off; };
        auto raw = [&](const void *x, size_t k) {
            const uint8_t *b = static_cast<const uint8_t *>(x);
            prog.insert(prog.end(), b, b + k);
            prog.resize(prog.size() + (16 - prog.size() % 16) % 16);
        };
        auto number = [&](const double *c, int k) {
            if (ub0) {
                std::vector<float> x(c, c + k);
                raw(x.data(), (size_t)k * 4);
            } else {
                raw(c, (size_t)k * 8);
            }
        };
        double grid = 0.0;   // of the coefficients' larger parts (kDiagSplit), 0: not split
        if (diag >= 0 && ub0 && n <= (apply ? kSplitApply : kSplitExpect) && !any_imaginary(groups[(size_t)diag])) {
            double size = 0.0;
            for (const SumTerm &t : groups[(size_t)diag].terms) size += std::fabs(t.re);
            int e = 0;
            std::frexp(size, &e);
            const double unit = std::ldexp(1.0, e - 23);   // multiples up to 2^23: their sums fit 24 bits
            for (const SumTerm &t : groups[(size_t)diag].terms)
                if (std::isfinite(size) && std::nearbyint(t.re / unit) * unit != t.re) grid = unit;
        }
        const bool in_two = grid > 0.0;
        // diagonal terms by local mask (first pass that has room for them: the first)
        std::map<uint32_t, std::vector<SumTerm>> dterms;   // key: local Z mask
        bool with_diag = false;
        if (diag >= 0) {
            for (const SumTerm &t : groups[(size_t)diag].terms) {
                uint32_t l = 0;
                for (uint64_t b = t.z & W; b; b &= b - 1) l |= 1u << lbit[__builtin_ctzll(b)];
                dterms[l].push_back(t);
            }
            with_diag = dterms.size() <= (size_t)kMaxDiag;
            if (!with_diag) {
                if (!left) return false;
                left->push_back(diag);
                all = false;
                diag = -1;
                if (rem.empty()) break;
            }
        }
        std::vector<uint32_t> dorder;   // local masks in table order
        std::vector<int> inner;
        for (int i : rem)
            if (!(groups[(size_t)i].x & ~W)) inner.push_back(i);
        std::vector<int> done;
        const size_t reserve = with_diag ? groups[(size_t)diag].terms.size() * 32 + dterms.size() * 10 + 256 : 0;
        while ((!inner.empty() && tile.nphase < kMaxPhases) || (with_diag && dorder.empty())) {
            const uint64_t R = choose(inner, always, sel, rbits);
            std::vector<int> take;
            for (int i : inner)
                if (!(groups[(size_t)i].x & ~R)) take.push_back(i);
            while (!take.empty() && bytes() + reserve + 32 + take.size() * op_bytes > (size_t)kRunMaxProg) take.pop_back();
            if (take.empty() && !(with_diag && dorder.empty())) break;
            RunPhaseHdr hd;
            std::memset(&hd, 0, sizeof(hd));
            int8_t rmap[16];
            std::fill(rmap, rmap + 16, (int8_t)-1);
            if (ub0) rmap[0] = 0;
            uint32_t regu = 0;
            int nr = 0;
            for (int u = 0; u < tbits - ub0 && nr < S; ++u)
                if ((R >> tile.pos[u + ub0]) & 1ull) {
                    rmap[u + ub0] = (int8_t)(nr++ + ub0);
                    regu |= 1u << u;
                }
            run_phase_bits(hd, regu, tbits - ub0);
            auto split = [&](uint64_t m, uint32_t &reg, uint32_t &loc, uint64_t &out) {
                reg = loc = 0;
                out = m & ~W;
                for (uint64_t b = m & W; b; b &= b - 1) {
                    const int l = lbit[__builtin_ctzll(b)];
                    if (rmap[l] >= 0) reg |= 1u << rmap[l];
                    else loc |= 1u << l;
                }
            };
            const bool diag_here = with_diag && dorder.empty();
            hd.nops = (uint16_t)(take.size() + (diag_here ? 1 : 0));
            raw(&hd, sizeof(hd));
            const int nv = 1 << rbits;
            for (int i : take) {
                const SumGroup &g = groups[(size_t)i];
                TwoParities par;
                double f[4][4], w[4][4];
                bool cplx;
                pair_table(g, par, f);
                SumHdr h;
                std::memset(&h, 0, sizeof(h));
                h.kind = (uint8_t)pair_weights(f, apply, w, &cplx);
                p.complex_out |= cplx;
                h.r = (uint8_t)par.r;
                uint32_t reg, loc, regz[2] = {0, 0};
                uint64_t out;
                split(g.x, reg, loc, out);
                h.xi = (uint8_t)reg;
                for (int j = 0; j < par.r; ++j) {
                    split(par.w[j], regz[j], loc, out);
                    (j ? h.zl1 : h.zl0) = (uint16_t)loc;
                    (j ? h.zg1 : h.zg0) = out;
                }
                const uint32_t top = 31u - (uint32_t)__builtin_clz(reg);
                std::vector<double> c;
                for (uint32_t e = 0; e < (1u << par.r); ++e)
                    for (uint32_t q = 0; q < (uint32_t)nv / 2; ++q) {
                        const uint32_t k = (q & ((1u << top) - 1)) | ((q >> top) << (top + 1));
                        const double *x = w[e ^ (uint32_t)(__builtin_popcount(k & regz[0]) & 1) ^
                                            ((uint32_t)(__builtin_popcount(k & regz[1]) & 1) << 1)];
                        if (h.kind == kPairGeneral) c.insert(c.end(), x, x + 4);
                        else if (apply) c.insert(c.end(), {x[h.kind], x[2 + h.kind]});
                        else c.push_back(x[h.kind]);
                    }
                h.stride = (uint32_t)(c.size() >> par.r);
                h.units = (uint32_t)(2 + (c.size() * (ub0 ? 4 : 8) + 15) / 16);
                raw(&h, sizeof(h));
                number(c.data(), (int)c.size());
            }
            if (diag_here) {
                std::vector<std::pair<uint32_t, uint32_t>> by_reg;   // (register bits, local mask)
                bool cplx = false;
                for (const auto &kv : dterms) {
                    uint32_t reg = 0;
                    for (int l = 0; l < tbits; ++l)
                        if (((kv.first >> l) & 1u) && rmap[l] >= 0) reg |= 1u << rmap[l];
                    by_reg.emplace_back(reg, kv.first);
                    for (const SumTerm &t : kv.second) cplx |= t.im != 0;
                }
                std::sort(by_reg.begin(), by_reg.end());
                std::vector<uint16_t> body((size_t)nv + 1, 0);
                uint64_t present = 0;   // register masks that occur
                for (const auto &e : by_reg) {
                    dorder.push_back(e.second);
                    for (uint32_t m = e.first + 1; m <= (uint32_t)nv; ++m) ++body[m];
                    uint32_t loc = 0;   // bits outside the registers
                    for (int l = 0; l < tbits; ++l)
                        if (((e.second >> l) & 1u) && rmap[l] < 0) loc |= 1u << l;
                    body.push_back((uint16_t)loc);
                    present |= 1ull << e.first;
                }
                SumHdr h;
                std::memset(&h, 0, sizeof(h));
                h.kind = in_two ? kDiagSplit : cplx ? kDiagComplex : kDiagReal;
                h.zg0 = present;
                h.units = (uint32_t)(2 + (body.size() * 2 + 15) / 16);
                p.diag_complex = cplx || in_two;
                p.complex_out |= cplx;
                raw(&h, sizeof(h));
                raw(body.data(), body.size() * 2);
            }
            ++tile.nphase;
            done.insert(done.end(), take.begin(), take.end());
            inner.erase(std::remove_if(inner.begin(), inner.end(),
                                       [&](int i) { return std::find(take.begin(), take.end(), i) != take.end(); }),
                        inner.end());
        }
        if (with_diag) {
            p.ndiag = (int32_t)dorder.size();
            p.nterm = (int32_t)groups[(size_t)diag].terms.size();
            p.diag_at = (int32_t)(bytes() / 16);
            std::vector<DiagEntry> ent;
            uint32_t first = 0;
            for (uint32_t l : dorder) {
                ent.push_back(DiagEntry{first, (uint32_t)dterms[l].size()});
                first += (uint32_t)dterms[l].size();
            }
            raw(ent.data(), ent.size() * sizeof(DiagEntry));
            for (uint32_t l : dorder)
                for (const SumTerm &t : dterms[l]) {
                    if (ub0) {
                        const double whole = in_two ? std::nearbyint(t.re / grid) * grid : t.re;
                        const DiagTerm<float> d{t.z & ~W, (float)whole, in_two ? (float)(t.re - whole) : (float)t.im};
                        raw(&d, sizeof(d));
                    } else {
                        const DiagTerm<double> d{t.z & ~W, t.re, t.im};
                        raw(&d, sizeof(d));
                    }
                }
            diag = -1;
        }
        tile.prog_bytes = (int32_t)bytes();
        passes.push_back(std::move(p));
        rem.erase(std::remove_if(rem.begin(), rem.end(),
                                 [&](int i) { return std::find(done.begin(), done.end(), i) != done.end(); }),
                  rem.end());
    }
    return all;
}

}  // namespace qi

// qi_adjrun.cu — the reverse sweep of an adjoint gradient, many gates to a pass.
//
// Un-applying gate after gate to psi and lambda while Re <lambda| dU U^dagger |psi> accumulates touches
// both states once per group of four qubits in k_adjoint_multi, and once more per run of CNOTs.  Here a
// pass holds a tile of both states in shared memory and runs through every gate whose non-diagonal
// qubits lie in the tile, as a gate run does (qi_gaterun.cu: same schedule, same program).
//
// Measured, gradients of the RY / RZ / CNOT ansatz (with the forward pass and H psi as gate runs and SumOp
// passes): FP64 12 qubits, 4 layers 3.4 -> 0.70 ms, 16 qubits, 8 layers 6.8 -> 1.7; FP32 8 qubits 1.75 ->
// 0.37, 20 qubits, 12 layers 5.9 -> 2.6.  FP64 passes are bound by FP64 arithmetic (6 operations per
// amplitude and rotation instead of 28), FP32 passes by instruction issue and fetch (issue 42 %, the
// operations' straight-line code for both states passes through the instruction cache; 128 registers for two blocks
// an SM leave 0.9 KB of spills a thread).
//
// A parametric gate is U = exp(-i theta P / 2) (or a phase), so its term is Im <lambda| P |psi> / 2, two
// operations per amplitude instead of a general 2x2 derivative, and both states take the same scaled
// inverse with unit entries; the size of the scales left out multiplies the term on the host.
// A thread's part of a term is summed in the state's precision, everything above it in FP64 or as finely: over
// the warp in FP64, or (FP32) as integers of 2^-26 of the largest part or less, then over the block's warps and
// the tiles in FP64 by one thread per term.  (Terms whose products have one sign, 12 qubits: 0.44 * 2^-24 off with
// FP32 sums over the block, 0.05 as integers; FP32 gradients of 8 to 22 qubits take 1-3 % less time, as two integer
// reductions take the place of five shuffles.)
#include "qi_gaterun.hpp"
#include "qi_runops.cuh"

#include <algorithm>

namespace qi {

struct SweepGeom {
    int32_t tbits, low;
    int8_t pos[16];
    int32_t nphase, prog_units, nslot, nterm;
    uint16_t slot_at[kRunMaxSlots];
};

// The thread's part of a term on the register amplitudes.
template <typename T, int X, bool Y>
__device__ __forceinline__ T der_pair(const typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits],
                                      const typename Cx<T>::V2 (&l)[1 << RunShape<T>::kRegBits]) {
    constexpr int NV = 1 << RunShape<T>::kRegBits;
    T p = T(0), q = T(0);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if (k & X) continue;
        const typename Cx<T>::V2 a = v[k], b = v[k ^ X], c = l[k], d = l[k ^ X];
        if constexpr (Y) {   // Re conj(d) a - Re conj(c) b
            p = ::fma(d.x, a.x, ::fma(d.y, a.y, p));
            q = ::fma(c.x, b.x, ::fma(c.y, b.y, q));
        } else {             // Im conj(c) b + Im conj(d) a
            p = ::fma(c.x, b.y, ::fma(d.x, a.y, p));
            q = ::fma(c.y, b.x, ::fma(d.y, a.x, q));
        }
    }
    return p - q;
}
template <typename T, bool Y>
__device__ __forceinline__ T der_pair_x(int xi, const typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits],
                                        const typename Cx<T>::V2 (&l)[1 << RunShape<T>::kRegBits]) {
    switch (xi) {
    case 1: return der_pair<T, 1, Y>(v, l);
    case 2: return der_pair<T, 2, Y>(v, l);
    case 4: return der_pair<T, 4, Y>(v, l);
    default:
        if constexpr (sizeof(T) == 4) return der_pair<T, 8, Y>(v, l);
        return T(0);
    }
}
// kDerZ: sum of sigma Im conj(l) v; kDerP: of Im conj(l) v where the qubit's bit is set.  M, odd as in
// run_rotz.
template <typename T, int M>
__device__ __forceinline__ T der_diag(const typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits],
                                      const typename Cx<T>::V2 (&l)[1 << RunShape<T>::kRegBits], bool odd, bool z) {
    constexpr int NV = 1 << RunShape<T>::kRegBits;
    T p = T(0), q = T(0);   // M: bit clear, bit set; M == 0: both all
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        T &acc = (k & M) ? q : p;
        acc = ::fma(l[k].x, v[k].y, ::fma(-l[k].y, v[k].x, acc));
    }
    if (M == 0) return odd ? (z ? -p : p) : (z ? p : T(0));
    return z ? p - q : q;
}
template <typename T>
__device__ __forceinline__ T der_diag_m(int m, const typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits],
                                        const typename Cx<T>::V2 (&l)[1 << RunShape<T>::kRegBits], bool odd, bool z) {
    switch (m) {
    case 0: return der_diag<T, 0>(v, l, odd, z);
    case 1: return der_diag<T, 1>(v, l, odd, z);
    case 2: return der_diag<T, 2>(v, l, odd, z);
    case 4: return der_diag<T, 4>(v, l, odd, z);
    default:
        if constexpr (sizeof(T) == 4) return der_diag<T, 8>(v, l, odd, z);
        return T(0);
    }
}

// Sum over the warp's lanes as a multiple of a power of two that holds the largest |p| in 26 bits (32 of them
// in 31): every p is rounded to at most 2^-26 of that.  e: its biased exponent, 255 when some p is not finite.
__device__ __forceinline__ int warp_sum_fixed(unsigned lanes, float p, uint8_t &e) {
    const uint32_t big = __reduce_max_sync(lanes, __float_as_uint(p) & 0x7fffffffu) >> 23;
    e = (uint8_t)max(big, 25u);   // the scale stays a normal number
    return __reduce_add_sync(lanes, __float2int_rn(p * __uint_as_float((279u - e) << 23)));
}
__device__ __forceinline__ double fixed_value(int sum, uint8_t e) {
    return (double)sum * __hiloint2double(e == 255 ? 0x7ff80000 : ((int)e + 871) << 20, 0);
}

template <typename T>
__global__ void __launch_bounds__(sizeof(T) == 8 ? 128 : 256, sizeof(T) == 8 ? 3 : 2) k_sweep_run(typename Cx<T>::V2 *psi, typename Cx<T>::V2 *lam, uint64_t ntiles,
                                                   const uint4 *prog, const __grid_constant__ SweepGeom g, double *partials) {
    using V2 = typename Cx<T>::V2;
    constexpr int S = kRunSelBits, NV = 1 << RunShape<T>::kRegBits, UB0 = RunShape<T>::kUnitBits;
    extern __shared__ uint4 sm[];
    __shared__ V2 slot[kRunMaxSlots];
    constexpr int kParts = kSweepTerms * (sizeof(T) == 8 ? 4 : 8);
    __shared__ T part[kParts];                                  // of each term and warp; FP32: integer bits
    __shared__ uint8_t part_exp[sizeof(T) == 8 ? 1 : kParts];
    __shared__ double total[kSweepTerms];
    __shared__ uint64_t next_base;
    const int ubits = g.tbits - UB0, lowu = g.low - UB0;
    const uint32_t nunit = 1u << ubits, nrow = 1u << (ubits - lowu), nt = blockDim.x, tid = threadIdx.x;
    const uint32_t nwarp = (nt + 31) >> 5, lane = tid & 31u, warp = tid >> 5;
    const unsigned lanes = nt >= 32 ? 0xffffffffu : (1u << nt) - 1u;
    uint4 *tile = sm, *ltile = sm + nunit;
    uint64_t *rows = reinterpret_cast<uint64_t *>(sm + 2 * nunit);
    uint4 *code = sm + 2 * nunit + ((nrow + 1) >> 1);
    uint32_t *places = reinterpret_cast<uint32_t *>(code + g.prog_units);   // [phase][thread]
    for (uint32_t r = tid; r < nrow; r += nt) {
        uint64_t off = 0;
        for (int j = g.low; j < g.tbits; ++j) off |= (uint64_t)((r >> (j - g.low)) & 1u) << g.pos[j];
        rows[r] = off >> UB0;
    }
    for (uint32_t i = tid; i < (uint32_t)g.prog_units; i += nt) copy16(code + i, prog + i);
    for (uint32_t i = tid; i < (uint32_t)g.nterm; i += nt) total[i] = 0.0;
    copy_wait();
    __syncthreads();
    uint32_t pc = 0;
    for (int ph = 0; ph < g.nphase; ++ph) {   // the threads' places are the same for every tile
        const RunPhaseHdr &hd = *reinterpret_cast<const RunPhaseHdr *>(code + pc);
        places[ph * nt + tid] = run_place(hd, tid, ubits - S, UB0);
        pc += 2;
        for (int q = 0; q < hd.nops; ++q) {
            const RunOpHdr &h = *reinterpret_cast<const RunOpHdr *>(code + pc);
            pc += h.code == RC_PHASE ? h.sgn : h.units;
        }
    }
    const RunCopy mine(rows, tid, lowu);
    uint64_t tbase = insert_zeros(blockIdx.x, g.pos, g.tbits);
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        if (tid == 0) next_base = insert_zeros(t + gridDim.x, g.pos, g.tbits);   // read after the barriers below
        uint4 *a4 = reinterpret_cast<uint4 *>(psi) + ((tbase >> UB0) + mine.first);
        uint4 *l4 = reinterpret_cast<uint4 *>(lam) + ((tbase >> UB0) + mine.first);
        for (uint32_t u = 0; u < nunit; u += nt) {
            const uint32_t at = mine.at ^ (run_swizzle(u) << 4);
            const uint64_t o = RunCopy::step(rows, u, lowu);
            copy16((char *)tile + at, a4 + o);
            copy16((char *)ltile + at, l4 + o);
        }
        for (uint32_t i = tid; i < (uint32_t)g.nslot; i += nt) {   // phase factors of this tile's fixed qubits
            const RunOpHdr &h = *reinterpret_cast<const RunOpHdr *>(code + g.slot_at[i]);
            V2 f = Cx<T>::make(T(1), T(0));
            const uint4 *s = code + g.slot_at[i] + 2;
            for (int j = 0; j < h.zl; ++j, s += 2) {
                const RunSub &sb = *reinterpret_cast<const RunSub *>(s);
                if ((tbase & sb.cg) == sb.cg) f = Cx<T>::mul(f, *reinterpret_cast<const V2 *>(s + 1));
            }
            slot[i] = f;
        }
        copy_wait();
        __syncthreads();
        pc = 0;
        for (int ph = 0; ph < g.nphase; ++ph) {
            const RunPhaseHdr &hd = *reinterpret_cast<const RunPhaseHdr *>(code + pc);
            const int nops = hd.nops;
            const uint32_t place = places[ph * nt + tid], lbase = place >> 16;
            uint32_t at[1 << S];
            run_units<S>(at, place, hd);
            pc += 2;
            V2 v[NV], l[NV];
            run_load<T, S>(v, tile, at);
            run_load<T, S>(l, ltile, at);
            for (int o = 0; o < nops; ++o) {
                const RunOpHdr &h = *reinterpret_cast<const RunOpHdr *>(code + pc);
                const int op = h.code, xi = h.xi, nsub = h.nsub;
                const T *c = reinterpret_cast<const T *>(code + pc + 2);
                if (op == RC_PHASE) {
                    const uint4 *next = code + pc + 2;
                    const uint32_t flags = h.act;
                    V2 f = Cx<T>::make(T(1), T(0));
                    pc += h.sgn;
                    if (flags & kTileFactor) {
                        f = slot[h.cl];
                        next += 2 * h.zl;
                    }
                    for (int j = 0; j < nsub; ++j, next += 2) {
                        const RunSub &sb = *reinterpret_cast<const RunSub *>(next);
                        if ((lbase & sb.cl) == sb.cl && (tbase & sb.cg) == sb.cg)
                            f = Cx<T>::mul(f, *reinterpret_cast<const V2 *>(next + 1));
                    }
                    if (flags & kLaneTable) {
                        f = Cx<T>::mul(f, reinterpret_cast<const V2 *>(next)[tid & 31u]);
                        next += 32 * sizeof(V2) / 16;
                    }
                    if (flags & kWarpTable) f = Cx<T>::mul(f, reinterpret_cast<const V2 *>(next)[tid >> 5]);
                    run_phase_m<T, RC_PHASE>(v, xi, f);
                    run_phase_m<T, RC_PHASE>(l, xi, f);
                    continue;
                }
                pc += h.units;
                const bool odd = (__popc(lbase & h.zl) + __popcll(tbase & h.zg)) & 1;
                const bool rotation = op == RC_ROTZ_A || op == RC_ROTZ_X;
                if (nsub && op != RC_LIFT && op != RC_PERM) {   // derivative term (uncontrolled: every thread is here)
                    T p;
                    if (nsub == kDerX) p = der_pair_x<T, false>(xi, v, l);
                    else if (nsub == kDerY) p = der_pair_x<T, true>(xi, v, l);
                    else p = der_diag_m<T>(xi, v, l, odd, nsub == kDerZ);
                    const uint32_t at_part = (uint32_t)h.cg * nwarp + warp;
                    if constexpr (sizeof(T) == 4) {
                        uint8_t e;
                        const int sum = warp_sum_fixed(lanes, p, e);
                        if (lane == 0) {
                            part[at_part] = __int_as_float(sum);
                            part_exp[at_part] = e;
                        }
                    } else {
                        for (uint32_t w = min(nt, 32u) >> 1; w; w >>= 1) p += __shfl_xor_sync(lanes, p, w);
                        if (lane == 0) part[at_part] = p;
                    }
                } else if (!rotation) {
                    const uint64_t cg = h.cg;
                    if ((lbase & h.cl) != h.cl || (tbase & cg) != cg) continue;
                }
                const uint32_t act = h.act;
#define QI_BOTH(CODE) run_pair_x<T, CODE, false>(v, xi, act, 0u, c); run_pair_x<T, CODE, false>(l, xi, act, 0u, c); break
#define QI_PHASE_BOTH(CODE, F) { run_phase_m<T, CODE>(v, xi, F); run_phase_m<T, CODE>(l, xi, F); }
                const V2 none = Cx<T>::make(T(0), T(0));
                switch (op) {
                case RC_REAL_A: QI_BOTH(RC_REAL_A);
                case RC_REAL_H: QI_BOTH(RC_REAL_H);
                case RC_REAL_X: QI_BOTH(RC_REAL_X);
                case RC_IMAG_A: QI_BOTH(RC_IMAG_A);
                case RC_IMAG_X: QI_BOTH(RC_IMAG_X);
                case RC_REAL_G: QI_BOTH(RC_REAL_G);
                case RC_GEN: QI_BOTH(RC_GEN);
                case RC_PERM:
                    run_perm_x<T>(v, xi, nsub, act);
                    run_perm_x<T>(l, xi, nsub, act);
                    break;
                case RC_ROTZ_A:
                    run_rotz_m<T, false>(v, xi, c[0], odd);
                    run_rotz_m<T, false>(l, xi, c[0], odd);
                    break;
                case RC_ROTZ_X:
                    run_rotz_m<T, true>(v, xi, c[0], odd);
                    run_rotz_m<T, true>(l, xi, c[0], odd);
                    break;
                case RC_LIFT:
                    QI_PHASE_BOTH(RC_LIFT, Cx<T>::make(c[0], c[1]))
                    if (nsub == 1) QI_PHASE_BOTH(RC_I, none)
                    else if (nsub == 2) QI_PHASE_BOTH(RC_NEG, none)
                    else if (nsub == 3) QI_PHASE_BOTH(RC_NI, none)
                    break;
                case RC_NEG: QI_PHASE_BOTH(RC_NEG, none) break;
                case RC_I: QI_PHASE_BOTH(RC_I, none) break;
                case RC_NI: QI_PHASE_BOTH(RC_NI, none) break;
                default: {   // RC_SCALE
                    const V2 f = Cx<T>::make(c[0], c[1]);
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        v[k] = Cx<T>::mul(f, v[k]);
                        l[k] = Cx<T>::mul(f, l[k]);
                    }
                    break;
                }
                }
#undef QI_BOTH
#undef QI_PHASE_BOTH
            }
            run_store<T, S>(v, tile, at);
            run_store<T, S>(l, ltile, at);
            __syncthreads();
        }
        for (uint32_t i = tid; i < (uint32_t)g.nterm; i += nt) {
            double s = 0.0;
            for (uint32_t w = 0; w < nwarp; ++w) {
                if constexpr (sizeof(T) == 4) s += fixed_value(__float_as_int(part[i * nwarp + w]), part_exp[i * nwarp + w]);
                else s += part[i * nwarp + w];
            }
            total[i] += s;
        }
        for (uint32_t u = 0; u < nunit; u += nt) {
            const uint32_t at = mine.at ^ (run_swizzle(u) << 4);
            const uint64_t o = RunCopy::step(rows, u, lowu);
            a4[o] = *reinterpret_cast<const uint4 *>((const char *)tile + at);
            l4[o] = *reinterpret_cast<const uint4 *>((const char *)ltile + at);
        }
        tbase = next_base;
        __syncthreads();   // tile and terms are read to the end before the next ones land
    }
    for (uint32_t i = tid; i < (uint32_t)g.nterm; i += nt) partials[(uint64_t)blockIdx.x * g.nterm + i] = total[i];
}

// out[i] = fixed-order sum of partials[b * nterm + i] over the blocks.
__global__ void k_sweep_finalize(const double *partials, int nb, int nterm, double *out) {
    double v = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) v += partials[(size_t)b * nterm + blockIdx.x];
    const double r = block_sum(v);
    if (threadIdx.x == 0) out[blockIdx.x] = r;
}

template <typename T>
static Status launch_sweep(cudaStream_t st, uint64_t dim, void *psi, void *lam, const SweepPass &p, const void *d_prog,
                           double *partials, double *out) {
    constexpr int ub0 = RunShape<T>::kUnitBits;
    SweepGeom g;
    g.tbits = p.run.tbits;
    g.low = p.run.low;
    std::copy(p.run.pos, p.run.pos + 16, g.pos);
    g.nphase = p.run.nphase;
    g.prog_units = p.run.prog_bytes / 16;
    g.nslot = (int32_t)p.run.slot_at.size();
    g.nterm = (int32_t)p.slot.size();
    std::copy(p.run.slot_at.begin(), p.run.slot_at.end(), g.slot_at);
    const int ubits = g.tbits - ub0, lowu = g.low - ub0;
    const unsigned threads = 1u << (ubits - kRunSelBits);
    const size_t sm = ((size_t)32 << ubits) + (((size_t)8 << (ubits - lowu)) + 15) / 16 * 16 + (size_t)p.run.prog_bytes +
                      (size_t)g.nphase * 4 * threads;
    // at most: tiles of 2^11 units of two states 64 KB, 2^8 rows 2 KB (16 KB should a tile have no rows),
    // program 24 KB, places of 24 phases 24 KB
    constexpr int cap = 128 * 1024;
    static_assert((32 << kRunTileBits) + (8 << kRunTileBits) + kRunMaxProg + kSweepPhases * 4 * (1 << (kRunTileBits - kRunSelBits)) <= cap,
                  "every pass fits");
    if (sm > (size_t)cap) return err(QI_ERR_UNKNOWN, (int64_t)sm, cap, "sweep pass too large");
    if (sm > 36 * 1024) QI_CUDA(cudaFuncSetAttribute(k_sweep_run<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
    const uint64_t ntiles = dim >> g.tbits;
    const unsigned nb = (unsigned)std::min<uint64_t>(ntiles, kSweepBlocks);
    k_sweep_run<T><<<nb, threads, sm, st>>>((typename Cx<T>::V2 *)psi, (typename Cx<T>::V2 *)lam, ntiles,
                                            (const uint4 *)((const char *)d_prog + p.run.prog_off), g, partials);
    count_launch();
    Status s = check_launch("k_sweep_run");
    if (!s.ok() || g.nterm == 0) return s;
    k_sweep_finalize<<<(unsigned)g.nterm, nb >= 256 ? 256 : 32, 0, st>>>(partials, (int)nb, g.nterm, out);
    count_launch();
    return check_launch("k_sweep_finalize");
}

Status launch_sweep_pass(qi_state *psi, void *lam, const SweepPass &p, const void *d_prog, double *partials, double *out) {
    if (psi->prec == QI_F32) return launch_sweep<float>(psi->stream, psi->dim(), psi->amps, lam, p, d_prog, partials, out);
    return launch_sweep<double>(psi->stream, psi->dim(), psi->amps, lam, p, d_prog, partials, out);
}

}  // namespace qi

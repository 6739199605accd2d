// qi_runops.cuh — the program of a gate run's pass and the register arithmetic of its operations
// (qi_gaterun.cu applies it to a state, qi_adjrun.cu to psi and lambda of a reverse sweep).
#pragma once
#include "qi_runtile.cuh"

namespace qi {

// ------------------------------------------------------------- program --
// A pass's program: per phase one 32-byte header, then its operations.  An operation is a 32-byte
// header and its coefficients; all sizes are multiples of 16 bytes.
enum RunCode : int {
    RC_REAL_A = 0,   // a' = a + s u b,      b' = b + s v a
    RC_REAL_H = 1,   // a' = a + u b,        b' = v a - b
    RC_REAL_X = 2,   // a' = s b + u a,      b' = v b - s a
    RC_IMAG_A = 3,   // a' = a + i s u b,    b' = b + i s v a
    RC_IMAG_X = 4,   // a' = s b + i u a,    b' = s a + i v b
    RC_REAL_G = 5,   // real 2x2
    RC_GEN = 6,      // complex 2x2, off-diagonal entries times s
    RC_PERM = 7,     // exchange (nsub: register control bit, 0: none, 255: as act says)
    RC_PHASE = 8,    // factor = product of what holds: tile factor, thread tables, sub-terms
    RC_NEG = 9, RC_I = 10, RC_NI = 11,   // factor -1, i, -i
    RC_PARITY = 12,  // factor c0 (even parity) or c1 (odd)
    RC_LIFT = 13,    // factor exp(i phi) i^nsub by three shears (c0 = tan(phi/2), c1 = sin(phi))
    RC_SCALE = 14,   // all amplitudes times a real or complex number
    RC_ROTZ_A = 15,  // a' = a + i s t a      (s = +1 where the qubit's bit is clear; xi: its register bit
    RC_ROTZ_X = 16   // a' = t a + i s a       or 0)
};

struct RunOpHdr {      // 32 bytes
    uint8_t code, xi, nsub, units;   // xi: register partner mask / AND mask; units: 16-byte size, of the
                                     // header alone for RC_PHASE (its parts give their own)
    uint32_t act;      // pairs (bit = index with xi's top bit clear) whose register controls hold
    uint32_t sgn;      // pairs with a negative sign (before the thread's parity)
    uint16_t cl, zl;   // local index bits outside the registers: controls, sign parity
    uint64_t cg, zg;   // the same on the tile's fixed qubits
};
struct RunSub {        // 16 bytes, followed by a complex factor padded to 16
    uint64_t cg;
    uint32_t cl, pad;
};
// RC_PHASE (act, sgn, cl hold other things): act = flags, sgn = 16-byte units of the whole operation,
// cl = tile slot, zl = number of its tile terms.  Its factor is the product of
//   kTileFactor: the terms on the tile's fixed qubits, multiplied together once per tile into slot cl,
//   kLaneTable / kWarpTable: 32 factors by lane / 16 by warp (terms on thread bits, tabulated on the host),
//   nsub sub-terms with conditions on both (or too few to tabulate).
// Layout: header, tile terms (RunSub + factor each), sub-terms, lane table, warp table.
enum RunPhaseFlags : uint32_t { kTileFactor = 1, kLaneTable = 2, kWarpTable = 4 };
constexpr size_t kRunMaxPhase = 48;   // elements of a phase: with headers, terms and (one per two terms) tables
                                      // 48 * 96 + 24 * 768 bytes, always less than a pass may hold
constexpr int kRunMaxSlots = 64;   // tile factors a pass may hold
static_assert(sizeof(RunOpHdr) == 32 && sizeof(RunSub) == 16, "program layout");

// ------------------------------------------------------------- kernel ---
// Pair updates on the register pairs (k, k ^ X).  SIGN: off-diagonal terms carry the sign of the
// pair's Z parity.
template <typename T, int CODE, int X, bool SIGN>
__device__ __forceinline__ void run_pair(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], uint32_t act, uint32_t sgn,
                                         const T *c) {
    using V2 = typename Cx<T>::V2;
    constexpr int NV = 1 << RunShape<T>::kRegBits;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if (k & top_bit(X)) continue;
        // the scaled forms and Pauli exponentials are never controlled
        if ((CODE == RC_REAL_G || CODE == RC_GEN) && !((act >> k) & 1u)) continue;
        V2 &a = v[k], &b = v[k ^ X];
        const uint32_t s = SIGN ? (sgn >> k) & 1u : 0u;
        V2 na, nb;
        if constexpr (CODE == RC_REAL_A) {
            const T u = SIGN ? flip_sign(c[0], s) : c[0], w = SIGN ? flip_sign(c[1], s) : c[1];
            na = Cx<T>::make(::fma(u, b.x, a.x), ::fma(u, b.y, a.y));
            nb = Cx<T>::make(::fma(w, a.x, b.x), ::fma(w, a.y, b.y));
        } else if constexpr (CODE == RC_REAL_H) {
            na = Cx<T>::make(::fma(c[0], b.x, a.x), ::fma(c[0], b.y, a.y));
            nb = Cx<T>::make(::fma(c[1], a.x, -b.x), ::fma(c[1], a.y, -b.y));
        } else if constexpr (CODE == RC_REAL_X) {
            const V2 sb = SIGN ? Cx<T>::make(flip_sign(b.x, s), flip_sign(b.y, s)) : b;
            const V2 sa = SIGN ? Cx<T>::make(flip_sign(a.x, s), flip_sign(a.y, s)) : a;
            na = Cx<T>::make(::fma(c[0], a.x, sb.x), ::fma(c[0], a.y, sb.y));
            nb = Cx<T>::make(::fma(c[1], b.x, -sa.x), ::fma(c[1], b.y, -sa.y));
        } else if constexpr (CODE == RC_IMAG_A) {
            const T u = SIGN ? flip_sign(c[0], s) : c[0], w = SIGN ? flip_sign(c[1], s) : c[1];
            na = Cx<T>::make(::fma(-u, b.y, a.x), ::fma(u, b.x, a.y));
            nb = Cx<T>::make(::fma(-w, a.y, b.x), ::fma(w, a.x, b.y));
        } else if constexpr (CODE == RC_IMAG_X) {
            const V2 sb = SIGN ? Cx<T>::make(flip_sign(b.x, s), flip_sign(b.y, s)) : b;
            const V2 sa = SIGN ? Cx<T>::make(flip_sign(a.x, s), flip_sign(a.y, s)) : a;
            na = Cx<T>::make(::fma(-c[0], a.y, sb.x), ::fma(c[0], a.x, sb.y));
            nb = Cx<T>::make(::fma(-c[1], b.y, sa.x), ::fma(c[1], b.x, sa.y));
        } else if constexpr (CODE == RC_REAL_G) {
            na = Cx<T>::make(::fma(c[1], b.x, c[0] * a.x), ::fma(c[1], b.y, c[0] * a.y));
            nb = Cx<T>::make(::fma(c[3], b.x, c[2] * a.x), ::fma(c[3], b.y, c[2] * a.y));
        } else {   // RC_GEN
            const V2 m01 = SIGN ? Cx<T>::make(flip_sign(c[2], s), flip_sign(c[3], s)) : Cx<T>::make(c[2], c[3]);
            const V2 m10 = SIGN ? Cx<T>::make(flip_sign(c[4], s), flip_sign(c[5], s)) : Cx<T>::make(c[4], c[5]);
            na = Cx<T>::fma(m01, b, Cx<T>::mul(Cx<T>::make(c[0], c[1]), a));
            nb = Cx<T>::fma(Cx<T>::make(c[6], c[7]), b, Cx<T>::mul(m10, a));
        }
        a = na;
        b = nb;
    }
}

// Dispatch on the partner mask: single bits, and with MULTI every mask of two bits (FP64: also
// all three), the X masks of Pauli exponentials.
template <typename T, int CODE, bool SIGN>
__device__ __forceinline__ void run_pair_x(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], int xi, uint32_t act,
                                           uint32_t sgn, const T *c) {
#define QI_X(M) case M: run_pair<T, CODE, M, SIGN>(v, act, sgn, c); break;
    constexpr bool f32 = sizeof(T) == 4;
    switch (xi) {
        QI_X(1) QI_X(2) QI_X(4)
    default: break;
    }
    if constexpr (f32) {
        if (xi == 8) run_pair<T, CODE, (f32 ? 8 : 1), SIGN>(v, act, sgn, c);
    }
    if constexpr (SIGN) {
        switch (xi) {
            QI_X(3) QI_X(5) QI_X(6)
        default: break;
        }
        if constexpr (f32) {
            if (xi == 9) run_pair<T, CODE, (f32 ? 9 : 1), SIGN>(v, act, sgn, c);
            if (xi == 10) run_pair<T, CODE, (f32 ? 10 : 1), SIGN>(v, act, sgn, c);
            if (xi == 12) run_pair<T, CODE, (f32 ? 12 : 1), SIGN>(v, act, sgn, c);
        } else {
            if (xi == 7) run_pair<T, CODE, 7, SIGN>(v, act, sgn, c);
        }
    }
#undef QI_X
}

// Exchange of the register pairs whose index contains the control bit C (0: all); a control known at
// compile time costs register moves only, an act mask a select per register.
template <typename T, int X, int C>
__device__ __forceinline__ void run_perm(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], uint32_t act) {
    constexpr int NV = 1 << RunShape<T>::kRegBits;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if ((k & X) || (C < 255 && (k & C) != C)) continue;
        if (C == 255 && !((act >> k) & 1u)) continue;
        const typename Cx<T>::V2 a = v[k];
        v[k] = v[k ^ X];
        v[k ^ X] = a;
    }
}
template <typename T, int X>
__device__ __forceinline__ void run_perm_c(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], int ctl, uint32_t act) {
    if (sizeof(T) == 8 || ctl == 255) run_perm<T, X, 255>(v, act);   // FP64 arithmetic covers the selects
    else if (ctl == 0) run_perm<T, X, 0>(v, act);
    else if (X != 1 && ctl == 1) run_perm<T, X, X == 1 ? 0 : 1>(v, act);
    else if (X != 2 && ctl == 2) run_perm<T, X, X == 2 ? 0 : 2>(v, act);
    else if (X != 4 && ctl == 4) run_perm<T, X, X == 4 ? 0 : 4>(v, act);
    else if (X != 8 && ctl == 8 && sizeof(T) == 4) run_perm<T, X, X == 8 || sizeof(T) == 8 ? 0 : 8>(v, act);
}
template <typename T>
__device__ __forceinline__ void run_perm_x(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], int xi, int ctl,
                                           uint32_t act) {
    switch (xi) {
    case 1: run_perm_c<T, 1>(v, ctl, act); break;
    case 2: run_perm_c<T, 2>(v, ctl, act); break;
    case 4: run_perm_c<T, 4>(v, ctl, act); break;
    default:
        if constexpr (sizeof(T) == 4) run_perm_c<T, 8>(v, ctl, act);
        break;
    }
}

// Multiples of diag(e^{i phi}, e^{-i phi}) on one qubit with unit entries, both halves scaled alike.  M: the
// qubit's register bit; 0: the qubit is not in the registers and odd says whether its bit is set.
template <typename T, bool SWAPPED, int M>
__device__ __forceinline__ void run_rotz(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], T t, bool odd) {
    constexpr int NV = 1 << RunShape<T>::kRegBits;
    const T s = odd ? T(-1) : T(1), u = odd ? -t : t;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const typename Cx<T>::V2 a = v[k];
        if constexpr (SWAPPED) {
            if constexpr (M == 0) v[k] = Cx<T>::make(::fma(t, a.x, -s * a.y), ::fma(t, a.y, s * a.x));
            else if (k & M) v[k] = Cx<T>::make(::fma(t, a.x, a.y), ::fma(t, a.y, -a.x));
            else v[k] = Cx<T>::make(::fma(t, a.x, -a.y), ::fma(t, a.y, a.x));
        } else {
            if (k & M) v[k] = Cx<T>::make(::fma(u, a.y, a.x), ::fma(-u, a.x, a.y));
            else v[k] = Cx<T>::make(::fma(-u, a.y, a.x), ::fma(u, a.x, a.y));
        }
    }
}
template <typename T, bool SWAPPED>
__device__ __forceinline__ void run_rotz_m(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], int m, T t, bool odd) {
    switch (m) {
    case 0: run_rotz<T, SWAPPED, 0>(v, t, odd); break;
    case 1: run_rotz<T, SWAPPED, 1>(v, t, odd); break;
    case 2: run_rotz<T, SWAPPED, 2>(v, t, odd); break;
    case 4: run_rotz<T, SWAPPED, 4>(v, t, odd); break;
    default:
        if constexpr (sizeof(T) == 4) run_rotz<T, SWAPPED, 8>(v, t, odd);
        break;
    }
}

// Factor on the register amplitudes whose index contains all bits of M.  RC_LIFT: f = (tan(phi/2),
// sin(phi)); the rotation is three shears, one operation less than a complex product.
template <typename T, int CODE, int M>
__device__ __forceinline__ void run_phase(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], typename Cx<T>::V2 f) {
    constexpr int NV = 1 << RunShape<T>::kRegBits;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if ((k & M) != M) continue;
        if constexpr (CODE == RC_PHASE) v[k] = Cx<T>::mul(f, v[k]);
        else if constexpr (CODE == RC_LIFT) {
            const T x = ::fma(-f.x, v[k].y, v[k].x), y = ::fma(f.y, x, v[k].y);
            v[k] = Cx<T>::make(::fma(-f.x, y, x), y);
        }
        else if constexpr (CODE == RC_NEG) v[k] = Cx<T>::make(-v[k].x, -v[k].y);
        else if constexpr (CODE == RC_I) v[k] = Cx<T>::make(-v[k].y, v[k].x);
        else v[k] = Cx<T>::make(v[k].y, -v[k].x);
    }
}
template <typename T, int CODE>
__device__ __forceinline__ void run_phase_m(typename Cx<T>::V2 (&v)[1 << RunShape<T>::kRegBits], int m,
                                            typename Cx<T>::V2 f) {
#define QI_M(M) case M: run_phase<T, CODE, M>(v, f); break;
    switch (m) {
        QI_M(0) QI_M(1) QI_M(2) QI_M(3) QI_M(4) QI_M(5) QI_M(6) QI_M(7)
    default: break;
    }
    if constexpr (sizeof(T) == 4) {
        switch (m) {
            QI_M(8) QI_M(9) QI_M(10) QI_M(11) QI_M(12) QI_M(13) QI_M(14) QI_M(15)
        default: break;
        }
    }
#undef QI_M
}

}  // namespace qi

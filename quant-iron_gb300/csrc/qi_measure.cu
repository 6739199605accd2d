// qi_measure.cu — State::measure / measure_n on the device.
//
// Reference: src/components/state.rs:525-784.  Probabilities of the measured
// qubits are summed in FP64 on the device in a fixed order (FP32 states: a
// thread's |a|^2 as two floats), copied to the host,
// normalised and sampled exactly as the reference does (sequential CDF in
// outcome order, `r < cumulative`, last outcome on fall-through).  The
// reference draws r from an unseeded rand::rng() (state.rs:601); here r comes
// from splitmix64 of a caller seed, so outcomes are reproducible and
// bit-identical to the oracle for the same r.  The outcome index arithmetic
// (bit k of the outcome = qubit qubits[k]) is integer and exact.
#include "qi_internal.hpp"
#include "qi_device.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace qi {

// P[d] = sum of |a_i|^2 over the indices whose measured bits spell d, as a streaming pass.  A thread's
// index fixes the lowest qubits (a warp reads 32 consecutive amplitudes), the measured qubits and as
// many others as spread the state over the chip; it loops over the qubits left, all of them
// unmeasured, so its outcome never changes and its sum stays in a register.  Lanes that differ in
// unmeasured qubits are then added by shuffles, and the sums of threads that differ in the other
// unmeasured thread bits (chunks) by k_meas_reduce, always in the same order.
// Measured (measure_n, 4096 shots, host call to result; before: one block per outcome and chunk gathering
// its amplitudes): FP64 22 qubits, 10 measured 463 -> 72 us, all 22 measured 153 -> 15 ms; FP32 24 qubits, 16
// measured 2.4 -> 0.33 ms.  The FP64 sums are bound by the FP64 pipe: two fused operations per amplitude (as
// three the 22-qubit measurement with its collapse took 80 us, now 66).
struct MeasGeom {
    int32_t nthread;         // thread-index bits
    int32_t nlane;           // of them within a warp
    int32_t nmeas, nchunk;   // measured qubits; chunk bits
    uint32_t lane_free;      // lane bits whose qubit is not measured
    int8_t qubit[44];        // qubit of thread-index bit j
    int8_t place[44];        // its bit in the outcome (measured) or 64 + its bit in the chunk index, -1: lane, unmeasured
    uint64_t loop;           // mask of the loop's qubits
    uint64_t off[8];         // offsets of its first three bits (unroll)
    int32_t unroll;          // how many of the eight
};

template <typename T>
__global__ void __launch_bounds__(256) k_meas_sum(const typename Cx<T>::V2 *a, const __grid_constant__ MeasGeom g,
                                                  double *partials) {
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint64_t base = 0, out = 0, chunk = 0;
    for (int j = 0; j < g.nthread; ++j) {
        const uint64_t bit = (t >> j) & 1ull;
        base |= bit << g.qubit[j];
        const int p = g.place[j];
        if (p >= 64) chunk |= bit << (p - 64);
        else if (p >= 0) out |= bit << p;
    }
    double acc = 0.0, acc2 = 0.0;
    PairSum sum;   // FP32: every |a|^2 on its own (FP64 additions would bound this pass)
    uint64_t off = 0;
    do {   // subsets of the loop mask, ascending
        if constexpr (sizeof(T) == 4) {
            float p[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                p[u] = 0.0f;
                if (u < g.unroll) {
                    const float2 v = a[base | off | g.off[u]];
                    p[u] = fmaf(v.x, v.x, v.y * v.y);
                }
            }
#pragma unroll
            for (int u = 0; u < 8; u += 2)
                if (u < g.unroll) sum.add(p[u], p[u + 1]);
        } else {
            double2 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < g.unroll) v[u] = a[base | off | g.off[u]];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < g.unroll) {   // two FP64 operations an amplitude: they bound this pass
                    acc = ::fma(v[u].x, v[u].x, acc);
                    acc2 = ::fma(v[u].y, v[u].y, acc2);
                }
        }
        off = ((off | ~g.loop) + 1) & g.loop;
    } while (off);
    acc += acc2;
    if constexpr (sizeof(T) == 4) acc = sum.total();
    const unsigned lanes = g.nlane >= 5 ? 0xffffffffu : (1u << (1 << g.nlane)) - 1u;
    for (int j = 0; j < g.nlane; ++j)
        if ((g.lane_free >> j) & 1u) acc += __shfl_xor_sync(lanes, acc, 1 << j);
    if ((threadIdx.x & g.lane_free) == 0) partials[(chunk << g.nmeas) | out] = acc;
}

// P[d] = sum over the chunks: a block per outcome (few outcomes), or a thread.
__global__ void k_meas_reduce(const double *partials, uint64_t chunks, uint64_t outcomes, double *P, int by_block) {
    if (by_block) {
        double acc = 0.0;
        for (uint64_t c = threadIdx.x; c < chunks; c += blockDim.x) acc += partials[c * outcomes + blockIdx.x];
        const double r = block_sum(acc);
        if (threadIdx.x == 0) P[blockIdx.x] = r;
        return;
    }
    const uint64_t d = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (d >= outcomes) return;
    double acc = 0.0;
    for (uint64_t c = 0; c < chunks; ++c) acc += partials[c * outcomes + d];
    P[d] = acc;
}

// Collapse and renormalisation (state.rs:622-660) in one pass: amplitudes whose measured bits differ from
// `want` become zero (not read), the others are divided by the collapsed state's norm, which is the root
// of the outcome's summed probability.
template <typename T>
__global__ void __launch_bounds__(256) k_collapse(typename Cx<T>::V2 *a, uint64_t dim, uint64_t dmask, uint64_t want, T inv) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < dim; i += (uint64_t)gridDim.x * blockDim.x) {
        typename Cx<T>::V2 v = Cx<T>::make(0, 0);
        if ((i & dmask) == want) {
            v = a[i];
            v = Cx<T>::make(v.x * inv, v.y * inv);
        }
        a[i] = v;
    }
}

uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
static double uniform01(uint64_t seed) { return (double)(splitmix64(seed) >> 11) * 0x1.0p-53; }

static Status apply_named(qi_state *s, int kind, int q, const double *m8) {
    qi_gate g;
    std::memset(&g, 0, sizeof(g));
    g.kind = kind;
    g.n_targets = 1;
    g.targets[0] = q;
    g.param_ids[0] = g.param_ids[1] = g.param_ids[2] = -1;
    if (m8) for (int j = 0; j < 8; ++j) g.params[j] = m8[j];
    GateMatrix gm;
    Status st = gate_to_matrix(s->n, g, &gm);
    if (!st.ok()) return st;
    return launch_op(s, lower_gate(s->n, gm), nullptr);
}

// Basis change before (dir = 0) or after (dir = 1) the computational measurement.
static Status basis_change(qi_state *s, int basis, const double *u, const int32_t *q, int m, int dir) {
    Status st = ok_status();
    double ud[8];
    if (basis == QI_BASIS_CUSTOM) {   // calculate_adjoint (state.rs:17-22)
        ud[0] = u[0]; ud[1] = -u[1]; ud[2] = u[4]; ud[3] = -u[5];
        ud[4] = u[2]; ud[5] = -u[3]; ud[6] = u[6]; ud[7] = -u[7];
    }
    auto each = [&](int kind, const double *mm) {
        for (int k = 0; k < m && st.ok(); ++k) st = apply_named(s, kind, q[k], mm);
    };
    if (basis == QI_BASIS_X) each(QI_GATE_H, nullptr);
    else if (basis == QI_BASIS_Y) {
        if (dir == 0) { each(QI_GATE_SDAG, nullptr); each(QI_GATE_H, nullptr); }
        else { each(QI_GATE_H, nullptr); each(QI_GATE_S, nullptr); }
    } else if (basis == QI_BASIS_CUSTOM) {
        each(QI_GATE_U2, dir == 0 ? u : ud);
    }
    return st;
}

constexpr size_t kKeptSums = 2u << 20;

// Outcome probabilities (host, unnormalised, outcome order) for the caller's qubit list.
static Status outcome_probs(qi_state *s, const int32_t *q, int m, std::vector<double> &prob, double *total_out) {
    const int n = s->n;
    uint64_t dmask = 0;
    for (int k = 0; k < m; ++k) dmask |= 1ull << q[k];
    MeasGeom g;
    std::memset(&g, 0, sizeof(g));
    int rank[64], nd = 0;   // bit of a measured qubit in the sorted outcome
    for (int b = 0; b < n; ++b)
        if ((dmask >> b) & 1ull) rank[b] = nd++;
    g.nmeas = nd;
    uint64_t in_thread = 0;
    auto add = [&](int qb, int place) {
        g.qubit[g.nthread] = (int8_t)qb;
        g.place[g.nthread++] = (int8_t)place;
        in_thread |= 1ull << qb;
    };
    g.nlane = std::min(n, 5);
    for (int b = 0; b < g.nlane; ++b) {
        if ((dmask >> b) & 1ull) {
            add(b, rank[b]);
        } else {
            g.lane_free |= 1u << b;
            add(b, -1);
        }
    }
    for (int b = g.nlane; b < n; ++b)
        if ((dmask >> b) & 1ull) add(b, rank[b]);
    // others until 2^17 threads, leaving three for the unrolled loop
    for (int b = n - 1, left = n - g.nthread; b >= g.nlane && left > 3 && g.nthread < 17; --b)
        if (!((in_thread >> b) & 1ull)) {
            add(b, 64 + g.nchunk++);
            --left;
        }
    uint64_t loop = (n >= 64 ? ~0ull : (1ull << n) - 1) & ~in_thread;
    g.unroll = 1;
    for (int k = 0; k < 3 && loop; ++k) {
        const uint64_t low = loop & (~loop + 1);
        for (int u = 0; u < g.unroll; ++u) g.off[g.unroll + u] = g.off[u] | low;
        g.unroll *= 2;
        loop &= loop - 1;
    }
    g.loop = loop;
    const uint64_t outcomes = 1ull << nd, chunks = 1ull << g.nchunk;
    // The workspace stays with the state, so only sums of the size that the thread split makes (2^17) lie
    // there; many measured qubits take memory for this call alone.
    const size_t sum_bytes = (chunks > 1 ? outcomes * chunks + outcomes : outcomes) * sizeof(double);
    const bool keep = sum_bytes <= kKeptSums;
    void *ws = nullptr;
    Status st = ok_status();
    if (keep) st = state_workspace(s, sum_bytes, &ws);
    else QI_CUDA(device_malloc_async(&ws, sum_bytes, s->stream));
    if (!st.ok()) return st;
    double *d_part = static_cast<double *>(ws), *d_P = d_part + outcomes * chunks;
    const unsigned tpb = 1u << std::min(8, (int)g.nthread), nb = 1u << (g.nthread - std::min(8, (int)g.nthread));
    if (s->prec == QI_F32) k_meas_sum<float><<<nb, tpb, 0, s->stream>>>((const float2 *)s->amps, g, d_part);
    else k_meas_sum<double><<<nb, tpb, 0, s->stream>>>((const double2 *)s->amps, g, d_part);
    count_launch();
    if (chunks > 1) {
        const bool by_block = outcomes <= 4096;
        k_meas_reduce<<<by_block ? (unsigned)outcomes : (unsigned)((outcomes + 255) / 256), by_block ? 128 : 256, 0, s->stream>>>(
            d_part, chunks, outcomes, d_P, by_block ? 1 : 0);
        count_launch();
    } else {
        d_P = d_part;
    }
    st = check_launch("k_meas_sum");
    std::vector<double> P(st.ok() ? outcomes : 0);
    cudaError_t e = cudaSuccess;
    if (st.ok()) e = cudaMemcpyAsync(P.data(), d_P, outcomes * sizeof(double), cudaMemcpyDeviceToHost, s->stream);
    if (!keep) cudaFreeAsync(ws, s->stream);
    const cudaError_t done = cudaStreamSynchronize(s->stream);   // after a failure too: the workspace is in use until then
    if (!st.ok()) return st;
    if (e == cudaSuccess) e = done;
    if (e != cudaSuccess) return cuda_status(e, "measure");
    // map to the caller's outcome integers (bit k = qubit q[k]); duplicated qubits must agree
    const uint64_t no = 1ull << m;
    bool sorted = nd == m;
    for (int k = 0; sorted && k < m; ++k) sorted = rank[q[k]] == k;
    if (sorted) {
        prob.swap(P);
    } else if (nd == m) {   // a permutation of the bits: each outcome from that without its lowest set bit
        prob.assign(no, 0.0);
        std::vector<uint32_t> d(no, 0);
        for (uint64_t o = 0; o < no; ++o) {
            if (o) d[o] = d[o & (o - 1)] | (1u << rank[q[__builtin_ctzll(o)]]);
            prob[o] = P[d[o]];
        }
    } else {
        prob.assign(no, 0.0);
        for (uint64_t o = 0; o < no; ++o) {
            uint64_t d = 0, seen = 0, val = 0;
            bool ok = true;
            for (int k = 0; k < m; ++k) {
                const uint64_t bit = (o >> k) & 1ull, qb = 1ull << q[k];
                if (seen & qb) { if (((val & qb) != 0) != (bit != 0)) { ok = false; break; } }
                seen |= qb;
                if (bit) {
                    val |= qb;
                    d |= 1ull << rank[q[k]];
                }
            }
            if (ok) prob[o] = P[d];
        }
    }
    double total = 0.0;
    for (double x : prob) total += x;   // probabilities.iter().sum()
    *total_out = total;
    return ok_status();
}

static Status check_measured(int n, const int32_t *q, int m) {
    if (m > n) return err(QI_ERR_INVALID_NUMBER_OF_QUBITS, n);
    for (int k = 0; k < m; ++k)
        if (q[k] < 0 || q[k] >= n) return err(QI_ERR_INVALID_QUBIT_INDEX, q[k], n);
    if (m > 24) return err(QI_ERR_UNSUPPORTED, m, 24, "measuring more than 24 qubits");
    return ok_status();
}

static uint64_t sample(const std::vector<double> &prob, double r) {   // state.rs:604-619
    double cum = 0.0;
    for (size_t i = 0; i < prob.size(); ++i) {
        cum += prob[i];
        if (r < cum) return i;
    }
    return prob.size() - 1;
}

Status measure_state(qi_state *s, int basis, const double *custom_u, const int32_t *qubits, int n_qubits,
                     uint64_t seed, uint64_t *outcome_out, double *probs_out) {
    std::vector<int32_t> all;
    if (n_qubits == 0) { for (int q = 0; q < s->n; ++q) all.push_back(q); qubits = all.data(); n_qubits = s->n; }
    Status st = check_measured(s->n, qubits, n_qubits);
    if (!st.ok()) return st;
    st = basis_change(s, basis, custom_u, qubits, n_qubits, 0);
    std::vector<double> prob;
    double total = 0.0;
    if (st.ok()) st = outcome_probs(s, qubits, n_qubits, prob, &total);
    if (st.ok() && total < 2.220446049250313e-16) st = err(QI_ERR_UNKNOWN, -1, -1, "total probability below f64::EPSILON");
    if (!st.ok()) {
        basis_change(s, basis, custom_u, qubits, n_qubits, 1);   // leave the state as it was
        return st;
    }
    const std::vector<double> sums = prob;
    for (double &x : prob) x = x / total;
    const uint64_t o = sample(prob, uniform01(seed));
    if (prob[o] * total <= 2.220446049250313e-16) {   // the collapsed state would not be normalisable
        basis_change(s, basis, custom_u, qubits, n_qubits, 1);
        return err(QI_ERR_STATE_NOT_NORMALISED);
    }
    // required measured bits for outcome o
    uint64_t dmask = 0, want = 0;
    for (int k = 0; k < n_qubits; ++k) {
        dmask |= 1ull << qubits[k];
        if ((o >> k) & 1ull) want |= 1ull << qubits[k];
    }
    uint64_t gsz = std::min<uint64_t>((s->dim() + 255) / 256, 152 * 16);
    const double inv = 1.0 / std::sqrt(sums[o]);
    if (s->prec == QI_F32)
        k_collapse<float><<<(unsigned)gsz, 256, 0, s->stream>>>((float2 *)s->amps, s->dim(), dmask, want, (float)inv);
    else k_collapse<double><<<(unsigned)gsz, 256, 0, s->stream>>>((double2 *)s->amps, s->dim(), dmask, want, inv);
    count_launch();
    st = check_launch("k_collapse");
    if (st.ok()) st = basis_change(s, basis, custom_u, qubits, n_qubits, 1);
    if (!st.ok()) return st;
    *outcome_out = o;
    if (probs_out) std::copy(prob.begin(), prob.end(), probs_out);
    QI_CUDA(cudaStreamSynchronize(s->stream));   // the collapsed state is there for whichever stream reads it next
    return ok_status();
}

}  // namespace qi

using namespace qi;

extern "C" {

qi_status qi_measure(qi_state *s, int32_t basis, const double *custom_u, const int32_t *qubits, int32_t n_qubits,
                     uint64_t seed, uint64_t *outcome_out, double *probs_out) {
    if (!s || !outcome_out || (n_qubits > 0 && !qubits)) return publish(err(QI_ERR_NULL_ARGUMENT));
    if (basis < 0 || basis > 3 || (basis == QI_BASIS_CUSTOM && !custom_u))
        return publish(err(QI_ERR_INVALID_INPUT_VALUE, basis));
    std::lock_guard<std::recursive_mutex> lk(s->mu);
    cudaError_t e = cudaSetDevice(s->device);
    if (e != cudaSuccess) return publish(cuda_status(e, "cudaSetDevice"));
    return publish(measure_state(s, basis, custom_u, qubits, n_qubits, seed, outcome_out, probs_out));
}

qi_status qi_measure_n(qi_state *s, int32_t basis, const double *custom_u, const int32_t *qubits, int32_t n_qubits,
                       int64_t n_shots, uint64_t seed, uint64_t *outcomes_out) {
    if (!s || (n_shots > 0 && !outcomes_out) || (n_qubits > 0 && !qubits)) return publish(err(QI_ERR_NULL_ARGUMENT));
    if (n_shots <= 0) return publish(err(QI_ERR_INVALID_NUMBER_OF_MEASUREMENTS, 0));   // state.rs:756-758
    if (basis < 0 || basis > 3 || (basis == QI_BASIS_CUSTOM && !custom_u))
        return publish(err(QI_ERR_INVALID_INPUT_VALUE, basis));
    std::lock_guard<std::recursive_mutex> lk(s->mu);
    cudaError_t e = cudaSetDevice(s->device);
    if (e != cudaSuccess) return publish(cuda_status(e, "cudaSetDevice"));
    std::vector<int32_t> all;
    if (n_qubits == 0) { for (int q = 0; q < s->n; ++q) all.push_back(q); qubits = all.data(); n_qubits = s->n; }
    Status st = check_measured(s->n, qubits, n_qubits);
    if (!st.ok()) return publish(st);
    st = basis_change(s, basis, custom_u, qubits, n_qubits, 0);
    std::vector<double> prob;
    double total = 0.0;
    if (st.ok()) st = outcome_probs(s, qubits, n_qubits, prob, &total);
    // undo the basis change: the state is left as it was
    Status st2 = basis_change(s, basis, custom_u, qubits, n_qubits, 1);
    if (!st.ok()) return publish(st);
    if (!st2.ok()) return publish(st2);
    if (total < 2.220446049250313e-16) return publish(err(QI_ERR_UNKNOWN, -1, -1, "total probability below f64::EPSILON"));
    for (double &x : prob) x = x / total;
    // CDF once, binary search per shot (same result as the sequential scan)
    std::vector<double> cdf(prob.size());
    double cum = 0.0;
    for (size_t i = 0; i < prob.size(); ++i) { cum += prob[i]; cdf[i] = cum; }
    // first outcome whose cumulative probability exceeds r; the search starts at the first that exceeds
    // the lower end of r's interval of width 1 / 2^m (exact: a power of two)
    const size_t no = cdf.size();
    std::vector<uint32_t> from(no);
    for (size_t b = 0, i = 0; b < no; ++b) {
        const double lo = (double)b / (double)no;
        while (i < no && !(lo < cdf[i])) ++i;
        from[b] = (uint32_t)i;
    }
    for (int64_t j = 0; j < n_shots; ++j) {
        const double r = uniform01(seed + (uint64_t)j);
        size_t i = from[(size_t)(r * (double)no)];
        while (i < no && !(r < cdf[i])) ++i;
        outcomes_out[j] = i < no ? i : no - 1;
    }
    return publish(ok_status());
}

}  // extern "C"

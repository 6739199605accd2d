// qi_compose.cu — operand blocks of tensor-core blocks composed on the device.
//
// A plan that is made for one call pays for its block matrices in that call: composing ten 6-qubit blocks
// of a 24-qubit Trotter step on the host's threads and splitting them into TF32 operands took 1.0 ms beside
// 2.5 ms of blocks (5 steps: 4.15 -> 2.84 ms a call).  Here one thread holds one element of a block's matrix: a CUDA block has 4 columns
// (columns are independent) of one matrix in shared memory and multiplies the members on from the left, in
// FP64 and in the host's order of summation, then writes the operands in the layout of tc_blocks.  Bound by
// the FP64 pipe: 4 * 2^m multiply-adds per element and member of m qubits (2.1 us of an SM for 512 elements,
// m = 2), so four columns a block spread ten blocks over all SMs.
#include "qi_internal.hpp"
#include "qi_plan.hpp"

#include <algorithm>
#include <cstring>

namespace qi {

constexpr int kComposeCols = 4;
constexpr int kComposeThreads = 64 * kComposeCols;

__device__ __forceinline__ float tf32_nearest(double x) {   // as tc_blocks rounds
    uint32_t u = __float_as_uint((float)x);
    if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;
    return __uint_as_float(u);
}

__global__ void __launch_bounds__(kComposeThreads) k_compose_blocks(const ComposeBlock *blocks, const ComposeMember *members,
                                                                    const double2 *data, float *tc) {
    __shared__ double2 B[2][kComposeThreads];
    const ComposeBlock b = blocks[blockIdx.x];
    const int R = 1 << b.k, r = threadIdx.x / kComposeCols, cc = threadIdx.x % kComposeCols;
    const int col = (int)blockIdx.y * kComposeCols + cc;
    if (col >= R) return;   // whole block: kComposeCols divides R
    const bool on = r < R;
    double2 mine = make_double2(r == col ? 1.0 : 0.0, 0.0);
    int cur = 0;
    if (on) B[0][threadIdx.x] = mine;
    __syncthreads();
    for (uint32_t i = 0; i < b.count; ++i) {
        const ComposeMember &g = members[b.first + i];
        const int m = g.m, gd = 1 << m;
        if (on) {
            int local = 0, base = r;
            for (int j = 0; j < m; ++j) {
                local |= ((r >> g.pos[j]) & 1) << j;
                base &= ~(1 << g.pos[j]);
            }
            const double2 *row = data + g.off + (size_t)local * gd;
            double2 acc = make_double2(0.0, 0.0);
            for (int c = 0; c < gd; ++c) {
                int from = base;
                for (int j = 0; j < m; ++j) from |= ((c >> j) & 1) << g.pos[j];
                const double2 d = row[c], x = B[cur][from * kComposeCols + cc];
                acc.x += d.x * x.x - d.y * x.y;
                acc.y += d.x * x.y + d.y * x.x;
            }
            mine = acc;
            B[cur ^ 1][threadIdx.x] = acc;
        }
        cur ^= 1;
        __syncthreads();
    }
    if (!on) return;
    // blocks along N: -Im U, Re U, Im U, high parts then low parts; core matrices of 8 rows x 16 bytes
    const size_t off = (size_t)(r / 8) * (R / 4) * 32 + (size_t)(col / 4) * 32 + (size_t)(r % 8) * 4 + (size_t)(col % 4);
    float *out = tc + b.tc + off;
    const size_t blk = (size_t)R * R;
    const float rh = tf32_nearest(mine.x), ih = tf32_nearest(mine.y);
    const float rl = tf32_nearest(mine.x - (double)rh), il = tf32_nearest(mine.y - (double)ih);
    out[0] = -ih;
    out[blk] = rh;
    out[2 * blk] = ih;
    out[3 * blk] = -il;
    out[4 * blk] = rl;
    out[5 * blk] = il;
}

// Appends the jobs to the plan's words (one copy to the device with them) and places the composed blocks
// behind; the offsets of the blocks' ops follow.
void finish_compose(qi_plan *p) {
    ComposeJobs &c = p->compose;
    if (c.blocks.empty()) return;
    auto append = [&](const void *src, size_t bytes) {
        while (p->tc.size() % 4) p->tc.push_back(0.0f);
        const size_t at = p->tc.size();
        p->tc.resize(at + (bytes + 15) / 16 * 4, 0.0f);
        std::memcpy(p->tc.data() + at, src, bytes);
        return at;
    };
    const size_t nb = c.blocks.size();
    c.at_members = append(c.members.data(), c.members.size() * sizeof(ComposeMember));
    c.at_data = append(c.data.data(), c.data.size() * sizeof(std::complex<double>));
    const size_t base = p->tc.size() + (nb * sizeof(ComposeBlock) + 15) / 16 * 4;   // after the block list, too
    for (ComposeBlock &b : c.blocks) b.tc += base;
    for (size_t i : c.ops) p->ops[i].tc_offset += (int64_t)base;
    c.at_blocks = append(c.blocks.data(), nb * sizeof(ComposeBlock));
}

Status launch_compose(qi_plan *p, qi_state *s) {
    const ComposeJobs &c = p->compose;
    int kmax = 0;
    for (const ComposeBlock &b : c.blocks) kmax = std::max(kmax, (int)b.k);
    float *tc = (float *)p->d_tc;
    const dim3 grid((unsigned)c.blocks.size(), (unsigned)(1 << kmax) / kComposeCols);
    k_compose_blocks<<<grid, kComposeThreads, 0, s->stream>>>((const ComposeBlock *)(tc + c.at_blocks),
                                                              (const ComposeMember *)(tc + c.at_members),
                                                              (const double2 *)(tc + c.at_data), tc);
    count_launch();
    return check_launch("k_compose_blocks");
}

}  // namespace qi

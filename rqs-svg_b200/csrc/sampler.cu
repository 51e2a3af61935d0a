// Shot sampler: draws full bitstrings from the current state without
// modifying it, with the outcome rule of measure_qubit (reference
// src/qcs.cu:2609-2626) applied qubit by qubit in measurement order.
//
// Measuring steps j = 0, 1, ..., n-1 (physical qubit order[j] at step j)
// sequentially is a walk down a binary tree: the node reached after steps
// 0..d-1 holds the squared norm of the amplitudes consistent with those
// outcomes, and step d compares P0 = child(bit = 0) with r = u * (P0 + P1).
//
// Data layout:
//   L[r], r < 2^s:  sum of |a|^2 over amplitudes whose step-0..s-1 bits equal
//                   r (one pass over the register in physical order);
//   tree level d:   2^d doubles at offset 2^d, T_d[p] = T_{d+1}[p] +
//                   T_{d+1}[p + 2^d]; level s is L itself;
//   steps >= s:     per shot, the 2^(n-s) amplitudes below the chosen leaf
//                   are loaded into shared memory and reduced to a local tree.
// s = max(min(n, 20), n - 11), so the per-shot subtree is at most 2048
// doubles (its tree: 32 KB of shared memory).

#include "qcs_internal.h"

namespace qcsb
{
namespace
{

constexpr int kThreads = 256;
constexpr int kMaxLocalBits = 11;

constexpr int kTopBits = 10;       // levels of the tree one block reduces
constexpr int kColumns = 4;        // nodes of level 10 per block below them: 32-byte rows
constexpr int kMaxColumnRows = 1 << 10;
constexpr int kLeafLoads = 8;      // amplitudes in flight per thread

struct OrderParams
{
    int n;
    int s;
    int identity;         // order[j] == j
    int order[kMaxQubits];
};

__device__ __forceinline__ uint64_t deposit_steps(uint64_t v, const OrderParams &op, int first, int count)
{
    uint64_t idx = 0;
    for (int k = 0; k < count; ++k)
        idx |= ((v >> k) & 1ull) << op.order[first + k];
    return idx;
}

template <typename V>
__device__ __forceinline__ double norm2(V a)
{
    const double x = a.x, y = a.y;
    return fma(x, x, y * y);
}

// Leaf sums in physical order, so that the register is read in full lines
// whatever the measurement order (a register in reversed order, as a QFT's
// swaps leave it, would read a 16-byte amplitude per 4 KiB: 6.29 -> 0.71 ms at
// 28 qubits, 6.1 TB/s). Lane l of a warp
// holds physical bits 0..4; `rest` are the physical bits of the steps below
// the leaves. A thread adds up the amplitudes that differ in the rest bits
// above the lane's (the subsets h of rest_hi, kLeafLoads loads in flight),
// the warp adds the lanes that differ in the rest bits among the lane's, and
// the lanes with those bits clear write their leaf.
template <typename V>
__global__ void __launch_bounds__(kThreads) leaf_sums_kernel(const V *state, const __grid_constant__ OrderParams op,
                                                             uint64_t rest, double *leaves)
{
    const uint64_t rest_hi = rest & ~31ull;
    const uint32_t rest_lo = static_cast<uint32_t>(rest) & 31u;
    const uint64_t nh = 1ull << __popcll(rest_hi);
    const uint64_t items = 1ull << (op.n - __popcll(rest_hi));
    for (uint64_t g = (uint64_t)blockIdx.x * kThreads + threadIdx.x; (g & ~31ull) < items; g += (uint64_t)gridDim.x * kThreads)
    {
        // zero bits at the rest positions above the lane's
        uint64_t base = g;
        for (uint64_t m = rest_hi; m; m &= m - 1)
        {
            const uint64_t lo = base & ((m & (0 - m)) - 1);
            base = lo | ((base ^ lo) << 1);
        }
        double acc = 0.0;
        if (g < items)
        {
            uint64_t h = 0;
            if (nh >= kLeafLoads)
            {
                for (uint64_t i = 0; i < nh; i += kLeafLoads)
                {
                    V a[kLeafLoads];
#pragma unroll
                    for (int u = 0; u < kLeafLoads; ++u)
                    {
                        a[u] = __ldcs(state + (base | h));
                        h = (h - rest_hi) & rest_hi;
                    }
#pragma unroll
                    for (int u = 0; u < kLeafLoads; ++u)
                        acc += norm2(a[u]);
                }
            }
            else
            {
                for (uint64_t i = 0; i < nh; ++i)
                {
                    acc += norm2(__ldcs(state + (base | h)));
                    h = (h - rest_hi) & rest_hi;
                }
            }
        }
#pragma unroll
        for (int b = 0; b < 5; ++b)
            if ((rest_lo >> b) & 1)
                acc += __shfl_xor_sync(0xffffffffu, acc, 1 << b);
        if (g < items && (g & rest_lo) == 0)
        {
            uint64_t r = base;
            if (!op.identity)
            {
                r = 0;
                for (int j = 0; j < op.s; ++j)
                    r |= ((base >> op.order[j]) & 1ull) << j;
            }
            leaves[r] = acc;
        }
    }
}

// Level d (2^d nodes at tree + 2^d) from level d + 1 (levels above 20 of the
// largest registers).
__global__ void tree_level_kernel(double *tree, int d)
{
    const uint64_t size = 1ull << d;
    const double *child = tree + 2 * size;
    double *parent = tree + size;
    for (uint64_t p = (uint64_t)blockIdx.x * kThreads + threadIdx.x; p < size; p += (uint64_t)gridDim.x * kThreads)
        parent[p] = child[p] + child[p + size];
}

// Levels top - 1 .. 10 from level `top` (11 .. 20). A node's children differ
// in their highest bit, so the nodes below node p of level 10 are those with
// p as their low ten bits: a block takes kColumns adjacent p and reduces
// their columns in shared memory. One launch of 10 us instead of one per level
// (each 2.5-5 us).
__global__ void __launch_bounds__(kThreads) tree_columns_kernel(double *tree, int top)
{
    __shared__ double col[kMaxColumnRows][kColumns];
    const int c = threadIdx.x % kColumns;
    const int r0 = threadIdx.x / kColumns;
    constexpr int kRowStep = kThreads / kColumns;
    const uint32_t p = blockIdx.x * kColumns + c;
    const int rows = 1 << (top - kTopBits);
    for (int r = r0; r < rows; r += kRowStep)
        col[r][c] = tree[(1ull << top) + p + ((uint64_t)r << kTopBits)];
    __syncthreads();
    for (int d = top - 1; d >= kTopBits; --d)
    {
        const int half = 1 << (d - kTopBits);
        for (int r = r0; r < half; r += kRowStep)
        {
            const double v = col[r][c] + col[r + half][c];
            col[r][c] = v;
            tree[(1ull << d) + p + ((uint64_t)r << kTopBits)] = v;
        }
        __syncthreads();
    }
}

// Levels top - 1 .. 0 from level top <= 10, in one block.
__global__ void __launch_bounds__(512) tree_top_kernel(double *tree, int top)
{
    __shared__ double v[1 << kTopBits];
    for (int p = threadIdx.x; p < (1 << top); p += 512)
        v[p] = tree[(1 << top) + p];
    __syncthreads();
    for (int d = top - 1; d >= 0; --d)
    {
        const int half = 1 << d;
        if ((int)threadIdx.x < half)
        {
            const double t = v[threadIdx.x] + v[threadIdx.x + half];
            v[threadIdx.x] = t;
            tree[half + threadIdx.x] = t;
        }
        __syncthreads();
    }
}

// The walk down the tree, a thread per shot: step d compares P0 = child(0)
// with r = u (P0 + P1). The first ten levels are read from shared memory; the
// others are dependent L2 reads, which the shots of an SM overlap.
__global__ void __launch_bounds__(kThreads) walk_kernel(const double *tree, int s, int n, uint32_t num_shots,
                                                        const double *uniforms, uint64_t *out_bits)
{
    __shared__ double top[2 << kTopBits];
    const int ts = s < kTopBits ? s : kTopBits;
    for (int i = threadIdx.x; i < (2 << ts); i += kThreads)
        top[i] = tree[i];
    __syncthreads();
    const uint32_t shot = blockIdx.x * kThreads + threadIdx.x;
    if (shot >= num_shots)
        return;
    const double *u = uniforms + (size_t)shot * n;
    uint64_t p = 0;
    for (int d = 0; d < s; ++d)
    {
        const double *child = d < ts ? top + (2 << d) : tree + (2ull << d);
        const double p0 = child[p];
        const double p1 = child[p | (1ull << d)];
        const double r = u[d] * (p0 + p1);
        if (p0 < r)
            p |= 1ull << d;
    }
    out_bits[shot] = p;
}

// Steps s .. n - 1 of registers deeper than the tree: a block per shot loads
// the 2^(n - s) amplitudes below the shot's leaf into a local tree.
template <typename V>
__global__ void __launch_bounds__(kThreads) shots_kernel(const V *state, const __grid_constant__ OrderParams op,
                                                         uint32_t num_shots, const double *uniforms, uint64_t *out_bits)
{
    __shared__ double local[2 << kMaxLocalBits];
    const int m_bits = op.n - op.s;
    const int m = 1 << m_bits;
    for (uint32_t shot = blockIdx.x; shot < num_shots; shot += gridDim.x)
    {
        const double *u = uniforms + (size_t)shot * op.n;
        const uint64_t p = out_bits[shot];
        const uint64_t base = op.identity ? p : deposit_steps(p, op, 0, op.s);
        // leaves of the local tree at offset m
        for (int h = threadIdx.x; h < m; h += kThreads)
        {
            const uint64_t idx = op.identity ? (base | ((uint64_t)h << op.s))
                                             : (base | deposit_steps((uint64_t)h, op, op.s, m_bits));
            local[m + h] = norm2(state[idx]);
        }
        __syncthreads();
        for (int e = m_bits - 1; e >= 0; --e)
        {
            const int size = 1 << e;
            for (int q = threadIdx.x; q < size; q += kThreads)
                local[size + q] = local[2 * size + q] + local[2 * size + q + size];
            __syncthreads();
        }
        if (threadIdx.x == 0)
        {
            uint64_t q = 0;
            for (int e = 0; e < m_bits; ++e)
            {
                const double *child = local + (2 << e);
                const double p0 = child[q];
                const double p1 = child[q | (1ull << e)];
                const double r = u[op.s + e] * (p0 + p1);
                if (p0 < r)
                    q |= 1ull << e;
            }
            out_bits[shot] = p | (q << op.s);
        }
        __syncthreads();
    }
}

int split_for(int n)
{
    int s = n < 20 ? n : 20;
    if (n - s > kMaxLocalBits)
        s = n - kMaxLocalBits;
    return s;
}

} // namespace

size_t sampler_tree_bytes(int n, int *split_out)
{
    const int s = split_for(n);
    if (split_out)
        *split_out = s;
    return sizeof(double) * (2ull << s);
}

namespace
{

OrderParams make_order(int n, const int *order, int split)
{
    OrderParams op;
    op.n = n;
    op.s = split;
    op.identity = 1;
    for (int j = 0; j < n; ++j)
    {
        op.order[j] = order[j];
        op.identity = op.identity && order[j] == j;
    }
    return op;
}

unsigned capped_grid(uint64_t items, unsigned cap)
{
    const uint64_t g = (items + kThreads - 1) / kThreads;
    return static_cast<unsigned>(g < cap ? g : cap);
}

} // namespace

template <typename R>
int launch_sampler_tree(const typename Cx<R>::T *state, int n, const int *order, double *tree, int split,
                        cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    const OrderParams op = make_order(n, order, split);
    uint64_t rest = 0;
    for (int j = split; j < n; ++j)
        rest |= 1ull << order[j];
    int launches = 0;
    const uint64_t items = 1ull << (n - __builtin_popcountll(rest & ~31ull));
    leaf_sums_kernel<V><<<capped_grid(items, 148 * 8), kThreads, 0, stream>>>(state, op, rest, tree + (1ull << split));
    QCSB_CUDA(cudaGetLastError());
    ++launches;
    int top = split;
    for (; top > 20; --top)
    {
        tree_level_kernel<<<capped_grid(1ull << (top - 1), 148 * 16), kThreads, 0, stream>>>(tree, top - 1);
        QCSB_CUDA(cudaGetLastError());
        ++launches;
    }
    if (top > kTopBits)
    {
        tree_columns_kernel<<<(1 << kTopBits) / kColumns, kThreads, 0, stream>>>(tree, top);
        QCSB_CUDA(cudaGetLastError());
        ++launches;
        top = kTopBits;
    }
    tree_top_kernel<<<1, 512, 0, stream>>>(tree, top);
    QCSB_CUDA(cudaGetLastError());
    return launches + 1;
}

template <typename R>
int launch_sampler_shots(const typename Cx<R>::T *state, int n, const int *order, uint32_t num_shots,
                         const double *uniforms, uint64_t *out_bits, const double *tree, int split,
                         cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    if (num_shots == 0)
        return 0;
    walk_kernel<<<(num_shots + kThreads - 1) / kThreads, kThreads, 0, stream>>>(tree, split, n, num_shots, uniforms,
                                                                                out_bits);
    QCSB_CUDA(cudaGetLastError());
    if (split == n)
        return 1;
    const OrderParams op = make_order(n, order, split);
    shots_kernel<V><<<num_shots < 148u * 7u ? num_shots : 148u * 7u, kThreads, 0, stream>>>(state, op, num_shots, uniforms,
                                                                                         out_bits);
    QCSB_CUDA(cudaGetLastError());
    return 2;
}

#define QCSB_INSTANTIATE(R)                                                                                      \
    template int launch_sampler_tree<R>(const Cx<R>::T *, int, const int *, double *, int, cudaStream_t);       \
    template int launch_sampler_shots<R>(const Cx<R>::T *, int, const int *, uint32_t, const double *,          \
                                         uint64_t *, const double *, int, cudaStream_t);
QCSB_INSTANTIATE(double)
QCSB_INSTANTIATE(float)

} // namespace qcsb

// Plain-path kernels: one launch per gate, state preparation, measurement
// reductions, collapse, <Z> sums and logical-order transfers.
//
// Layout: the register is one contiguous array of complex amplitudes
// (double2 for complex128, float2 for complex64); physical qubit q is bit q
// of the index. A gate on targets T with controls C visits "groups": the
// 2^(n - |T u C|) indices whose T and C bits are zero, enumerated by
// inserting zero bits at the sorted operand positions (the role of
// thread_num_to_state_index_q*, reference src/qcs.cu:156-376), then ORs in
// the control values and each active target offset.
//
// Consecutive threads take consecutive groups, so every warp reads and writes
// contiguous amplitudes wherever the operand bits are >= 5; loads and stores
// use evict-first hints (each amplitude is touched once per pass over a
// register far larger than L2). Gate arithmetic runs in the amplitude's
// precision; every reduction accumulates in FP64.

#include "qcs_internal.h"

#include <cuda_runtime.h>

#include <cstdlib>

namespace qcsb
{
namespace
{

constexpr int kThreads = 256;
constexpr int kSMs = 148;
constexpr int kMaxOps = kMaxQubits;

template <typename V>
__device__ __forceinline__ V cfma(V m, V v, V acc)
{
    acc.x = fma(m.x, v.x, acc.x);
    acc.x = fma(-m.y, v.y, acc.x);
    acc.y = fma(m.x, v.y, acc.y);
    acc.y = fma(m.y, v.x, acc.y);
    return acc;
}

template <typename V>
__device__ __forceinline__ V cmul(V m, V v)
{
    V r;
    r.x = fma(m.x, v.x, -m.y * v.y);
    r.y = fma(m.x, v.y, m.y * v.x);
    return r;
}

template <typename V>
__device__ __forceinline__ double norm2(V a)
{
    const double x = a.x, y = a.y;
    return fma(x, x, y * y);
}

template <typename V>
__host__ __device__ __forceinline__ V make_cx(double re, double im);
template <>
__host__ __device__ __forceinline__ double2 make_cx<double2>(double re, double im) { return make_double2(re, im); }
template <>
__host__ __device__ __forceinline__ float2 make_cx<float2>(double re, double im)
{
    return make_float2(static_cast<float>(re), static_cast<float>(im));
}

// Insert a zero bit below each mask boundary: masks[i] = (1 << pos_i) - 1
// for operand positions sorted ascending.
template <int MAXOPS>
__device__ __forceinline__ uint64_t insert_zero_bits(uint64_t g, const uint64_t *masks, int nops)
{
#pragma unroll
    for (int i = 0; i < MAXOPS; ++i)
    {
        if (i >= nops)
            break;
        const uint64_t lo = g & masks[i];
        g = lo | ((g ^ lo) << 1);
    }
    return g;
}

template <typename R, int NA, bool DIAG>
struct PlainParams
{
    typedef typename Cx<R>::T V;
    V *state;
    uint64_t ngroups;
    uint64_t cval;
    int nops;
    uint64_t masks[kMaxOps];
    uint64_t off[NA];
    V m[DIAG ? NA : NA * NA];
};

template <bool STREAM, typename V>
__device__ __forceinline__ V ld_amp(const V *p) { return STREAM ? __ldcs(p) : *p; }
template <bool STREAM, typename V>
__device__ __forceinline__ void st_amp(V *p, V v)
{
    if (STREAM)
        __stcs(p, v);
    else
        *p = v;
}

// STREAM selects evict-first cache hints; U groups per thread per iteration.
template <typename R, int NA, bool DIAG, int U, bool STREAM>
__global__ void __launch_bounds__(kThreads) gate_plain_kernel(const __grid_constant__ PlainParams<R, NA, DIAG> p)
{
    typedef typename Cx<R>::T V;
    const uint64_t step = (uint64_t)gridDim.x * kThreads * U;
    for (uint64_t g0 = (uint64_t)blockIdx.x * kThreads * U + threadIdx.x; g0 < p.ngroups; g0 += step)
    {
        uint64_t base[U];
        V v[U][NA];
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const uint64_t g = g0 + (uint64_t)u * kThreads;
            base[u] = insert_zero_bits<kMaxOps>(g, p.masks, p.nops) | p.cval;
            if (g < p.ngroups)
            {
#pragma unroll
                for (int a = 0; a < NA; ++a)
                    v[u][a] = ld_amp<STREAM>(p.state + (base[u] | p.off[a]));
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const uint64_t g = g0 + (uint64_t)u * kThreads;
            if (g >= p.ngroups)
                continue;
            if (DIAG)
            {
#pragma unroll
                for (int a = 0; a < NA; ++a)
                    st_amp<STREAM>(p.state + (base[u] | p.off[a]), cmul(p.m[a], v[u][a]));
            }
            else
            {
#pragma unroll
                for (int a = 0; a < NA; ++a)
                {
                    V acc = make_cx<V>(0.0, 0.0);
#pragma unroll
                    for (int b = 0; b < NA; ++b)
                        acc = cfma(p.m[a * NA + b], v[u][b], acc);
                    st_amp<STREAM>(p.state + (base[u] | p.off[a]), acc);
                }
            }
        }
    }
}

// Sorted operand positions (targets and controls) as insertion masks.
int fill_masks(const GateOp &op, uint64_t *masks)
{
    uint64_t bits = op.cmask;
    for (int i = 0; i < op.nt; ++i)
        bits |= 1ull << op.tq[i];
    int nops = 0;
    while (bits)
    {
        const int pos = __builtin_ctzll(bits);
        masks[nops++] = (1ull << pos) - 1;
        bits &= bits - 1;
    }
    return nops;
}

unsigned grid_for(uint64_t work_items, int per_block, uint64_t cap = (uint64_t)kSMs * 16)
{
    uint64_t blocks = (work_items + per_block - 1) / per_block;
    if (blocks > cap)
        blocks = cap;
    if (blocks == 0)
        blocks = 1;
    return static_cast<unsigned>(blocks);
}

// Launch shape of the plain gate kernel (tuning knob QCS_PLAIN_VARIANT):
//   0  grid-stride over 148 x 16 blocks, U groups per thread, evict-first hints
//   1  one thread per group over the whole grid, default cache policy
//   2  one thread per group over the whole grid, evict-first hints (default:
//      measured fastest on B200, 103% of the copy bandwidth at 30 qubits)
//   3  grid-stride, U groups per thread, default cache policy
int plain_variant()
{
    static int v = [] {
        const char *e = std::getenv("QCS_PLAIN_VARIANT");
        const int x = (e && e[0]) ? std::atoi(e) : 2;
        return (x >= 0 && x <= 3) ? x : 2;
    }();
    return v;
}

template <typename R, int NA, bool DIAG>
int launch_plain_na(typename Cx<R>::T *state, int n, const GateOp &op, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    constexpr int U = NA == 1 ? 4 : (NA == 2 ? 2 : 1);
    PlainParams<R, NA, DIAG> p;
    std::memset(&p, 0, sizeof(p));
    p.state = state;
    p.nops = fill_masks(op, p.masks);
    p.ngroups = 1ull << (n - p.nops);
    p.cval = op.cval;
    for (int a = 0; a < NA; ++a)
    {
        uint64_t off = 0;
        for (int i = 0; i < op.nt; ++i)
            if ((op.act[a] >> i) & 1)
                off |= 1ull << op.tq[i];
        p.off[a] = off;
    }
    const int nm = DIAG ? NA : NA * NA;
    for (int k = 0; k < nm; ++k)
        p.m[k] = make_cx<V>(op.mat[k].re, op.mat[k].im);
    const uint64_t one_shot_cap = 1ull << 31;
    switch (plain_variant())
    {
    case 0:
        gate_plain_kernel<R, NA, DIAG, U, true><<<grid_for(p.ngroups, kThreads * U), kThreads, 0, stream>>>(p);
        break;
    case 2:
        gate_plain_kernel<R, NA, DIAG, 1, true><<<grid_for(p.ngroups, kThreads, one_shot_cap), kThreads, 0, stream>>>(p);
        break;
    case 3:
        gate_plain_kernel<R, NA, DIAG, U, false><<<grid_for(p.ngroups, kThreads * U), kThreads, 0, stream>>>(p);
        break;
    default:
        gate_plain_kernel<R, NA, DIAG, 1, false><<<grid_for(p.ngroups, kThreads, one_shot_cap), kThreads, 0, stream>>>(p);
        break;
    }
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R, bool DIAG>
int launch_plain_dispatch(typename Cx<R>::T *state, int n, const GateOp &op, cudaStream_t stream)
{
    switch (op.na)
    {
    case 1: return launch_plain_na<R, 1, DIAG>(state, n, op, stream);
    case 2: return launch_plain_na<R, 2, DIAG>(state, n, op, stream);
    case 3: return launch_plain_na<R, 3, DIAG>(state, n, op, stream);
    case 4: return launch_plain_na<R, 4, DIAG>(state, n, op, stream);
    default: throw std::runtime_error(strformat("internal: %d active sub-indices", op.na));
    }
}

// ---------------------------------------------------------- small registers

// A run of gates on a register of at most kSmallQubits qubits: one block holds
// it in shared memory and applies the gates one after another, each with the
// plain kernel's formula (bit-identical to it). A kernel per gate cost a
// launch (3.7 us of host time) for a few hundred bytes of work.
constexpr int kSmallQubits = 8;
constexpr int kSmallThreads = 128;
constexpr int kSmallOps = 32;        // per launch: parameters of 3 KiB (larger blocks launch slower)
constexpr int kSmallEntries = 128;

struct SmallOp
{
    uint8_t nops, na, diag, pad;
    uint16_t entry, cval;
    uint16_t off[4];
    uint8_t masks[kSmallQubits];   // insertion masks below each operand position, ascending
};

template <typename R>
struct SmallParams
{
    typedef typename Cx<R>::T V;
    V *state;
    int n, count;
    SmallOp ops[kSmallOps];
    V entries[kSmallEntries];
};

template <typename R>
__global__ void __launch_bounds__(kSmallThreads) small_register_kernel(const __grid_constant__ SmallParams<R> p)
{
    typedef typename Cx<R>::T V;
    __shared__ V amp[1 << kSmallQubits];
    for (int i = threadIdx.x; i < (1 << p.n); i += kSmallThreads)
        amp[i] = p.state[i];
    __syncthreads();
    for (int k = 0; k < p.count; ++k)
    {
        const SmallOp &op = p.ops[k];
        const int na = op.na;
        for (int g = threadIdx.x; g < (1 << (p.n - op.nops)); g += kSmallThreads)
        {
            uint32_t base = static_cast<uint32_t>(g);
            for (int i = 0; i < op.nops; ++i)
            {
                const uint32_t lo = base & op.masks[i];
                base = lo | ((base ^ lo) << 1);
            }
            base |= op.cval;
            V v[4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
                if (a < na)
                    v[a] = amp[base | op.off[a]];
            for (int a = 0; a < na; ++a)
            {
                V acc = make_cx<V>(0.0, 0.0);
                if (op.diag)
                    acc = cmul(p.entries[op.entry + a], amp[base | op.off[a]]);
                else
                {
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (b < na)
                            acc = cfma(p.entries[op.entry + a * na + b], v[b], acc);
                }
                amp[base | op.off[a]] = acc;
            }
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < (1 << p.n); i += kSmallThreads)
        p.state[i] = amp[i];
}

// ------------------------------------------------------------ preparation

template <typename V>
__global__ void fill_kernel(V *state, uint64_t count, V value)
{
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < count; i += (uint64_t)gridDim.x * kThreads)
        __stcs(state + i, value);
}

template <typename V>
__global__ void sequential_kernel(V *state, uint64_t count)
{
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < count; i += (uint64_t)gridDim.x * kThreads)
        __stcs(state + i, make_cx<V>(static_cast<double>(i), 0.0));
}

template <typename V>
__global__ void set_one_kernel(V *state, uint64_t index, V value) { state[index] = value; }

// a *= sqrt(target / norm), the factor formed in FP64 from the squared norm
// the reduction left in device memory (no host round trip); a zero norm
// leaves the state as it is.
template <typename V>
__global__ void rescale_kernel(V *state, uint64_t count, double target, const double *norm)
{
    const double nrm = *norm;
    if (!(nrm > 0.0))
        return;
    const double f = sqrt(target / nrm);
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < count; i += (uint64_t)gridDim.x * kThreads)
    {
        const V a = state[i];
        __stcs(state + i, make_cx<V>(a.x * f, a.y * f));
    }
}

// ------------------------------------------------------------ reductions

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Insertion of zero bits by runs of adjacent operand positions: run i starts
// above masks[i] = (1 << pos_i) - 1 and is shifts[i] bits long. A chain of
// measurements that takes the qubits in order has one run, where a loop over
// its positions would grow with every measured qubit.
struct ZeroRuns
{
    int count;
    uint8_t shifts[kMaxOps];
    uint64_t masks[kMaxOps];
};

__device__ __forceinline__ uint64_t insert_zero_runs(uint64_t g, const ZeroRuns &z)
{
    for (int i = 0; i < z.count; ++i)
    {
        const uint64_t lo = g & z.masks[i];
        g = lo | ((g ^ lo) << z.shifts[i]);
    }
    return g;
}

// operand positions: the set bits of `bits`; returns how many
int fill_runs(uint64_t bits, ZeroRuns &z)
{
    const int n = __builtin_popcountll(bits);
    z.count = 0;
    while (bits)
    {
        const int pos = __builtin_ctzll(bits);
        const int len = __builtin_ctzll(~(bits >> pos));
        z.masks[z.count] = (1ull << pos) - 1;
        z.shifts[z.count++] = static_cast<uint8_t>(len);
        bits &= ~(((1ull << len) - 1) << pos);
    }
    return n;
}

template <typename R>
struct ProbParams
{
    const typename Cx<R>::T *state;
    uint64_t ngroups;
    uint64_t cval;
    uint64_t tbit;
    ZeroRuns runs;
    double2 *partials;
    double2 *result;      // final (P0, P1); may be mapped host memory
    unsigned *ticket;     // zero between calls
    volatile unsigned *done;   // host-mapped: set to seq once result is written (or null)
    unsigned seq;
};

// Fixed-order sum of count double2 partials by one block of kThreads threads
// (the same order in every call, so repeated measurements agree bit for bit).
__device__ __forceinline__ double2 block_sum_partials(const double2 *partials, int count)
{
    double s0 = 0.0, s1 = 0.0;
    for (int i = threadIdx.x; i < count; i += kThreads)
    {
        const double2 v = __ldcg(partials + i);
        s0 += v.x;
        s1 += v.y;
    }
    __shared__ double sh[2][kThreads / 32];
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    const int w = threadIdx.x / 32, l = threadIdx.x % 32;
    if (l == 0)
    {
        sh[0][w] = s0;
        sh[1][w] = s1;
    }
    __syncthreads();
    double t0 = 0.0, t1 = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < kThreads / 32; ++k)
        {
            t0 += sh[0][k];
            t1 += sh[1][k];
        }
    return make_double2(t0, t1);
}

// Per-block (sum |a0|^2, sum |a1|^2) over the groups; the grid depends on the
// group count alone and the reduction order is fixed, so repeated calls give
// identical sums. The last block to finish adds the per-block partials and
// writes (P0, P1) to p.result. A chain of measurements halves the groups at
// every step, and most of its reductions are bound by latency: a block per
// 2048 groups (eight per thread, four of them in flight), and with one block
// no partials and no ticket (9.0 -> 6.8 us for the last ones of a 20-qubit
// chain under the profiler).
constexpr int kProbGroups = 4;   // groups in flight per thread

template <typename R>
__global__ void __launch_bounds__(kThreads) measure_probs_kernel(const __grid_constant__ ProbParams<R> p)
{
    double s0 = 0.0, s1 = 0.0;
    const uint64_t step = (uint64_t)gridDim.x * kThreads;
    for (uint64_t g = (uint64_t)blockIdx.x * kThreads + threadIdx.x; g < p.ngroups; g += kProbGroups * step)
    {
        typename Cx<R>::T a0[kProbGroups], a1[kProbGroups];
#pragma unroll
        for (int u = 0; u < kProbGroups; ++u)
        {
            a0[u] = a1[u] = make_cx<typename Cx<R>::T>(0.0, 0.0);
            if (g + u * step < p.ngroups)
            {
                const uint64_t i0 = insert_zero_runs(g + u * step, p.runs) | p.cval;
                a0[u] = __ldcs(p.state + i0);
                a1[u] = __ldcs(p.state + (i0 | p.tbit));
            }
        }
#pragma unroll
        for (int u = 0; u < kProbGroups; ++u)
        {
            s0 += norm2(a0[u]);
            s1 += norm2(a1[u]);
        }
    }
    __shared__ double sh[2][kThreads / 32];
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    const int w = threadIdx.x / 32, l = threadIdx.x % 32;
    if (l == 0)
    {
        sh[0][w] = s0;
        sh[1][w] = s1;
    }
    __syncthreads();
    double2 total = make_double2(0.0, 0.0);
    if (threadIdx.x == 0)
        for (int k = 0; k < kThreads / 32; ++k)
        {
            total.x += sh[0][k];
            total.y += sh[1][k];
        }
    if (gridDim.x > 1)
    {
        __shared__ bool last;
        if (threadIdx.x == 0)
        {
            p.partials[blockIdx.x] = total;
            __threadfence();
            last = atomicAdd(p.ticket, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!last)
            return;
        __threadfence();
        total = block_sum_partials(p.partials, gridDim.x);
        if (threadIdx.x == 0)
            *p.ticket = 0;
    }
    if (threadIdx.x == 0)
    {
        *p.result = total;
        if (p.done != nullptr)
        {
            // the result reaches host memory before the flag does
            __threadfence_system();
            *p.done = p.seq;
        }
    }
}

template <typename V>
__global__ void collapse_kernel(V *state, uint64_t ngroups, uint64_t lowmask, uint64_t zero_bit)
{
    for (uint64_t g = (uint64_t)blockIdx.x * kThreads + threadIdx.x; g < ngroups; g += (uint64_t)gridDim.x * kThreads)
    {
        const uint64_t lo = g & lowmask;
        const uint64_t i = lo | ((g ^ lo) << 1) | zero_bit;
        __stcs(state + i, make_cx<V>(0.0, 0.0));
    }
}

// Kept amplitudes are not touched (no reads at all).
template <typename V>
__global__ void collapse_mask_kernel(V *state, uint64_t count, uint64_t cmask, uint64_t cval)
{
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < count; i += (uint64_t)gridDim.x * kThreads)
        if ((i & cmask) != cval)
            __stcs(state + i, make_cx<V>(0.0, 0.0));
}

// <Z> sums: [0] the squared norm, [1 + q] the part with bit q set. A block
// takes a contiguous range of tiles; in a tile thread t reads kZLoads 16-byte
// words, word u * 256 + t, all in flight together (one complex128 or two
// complex64 amplitudes each). Bits of the index inside a word and of u split
// a thread's own sums, bits of t split the block's sums of thread totals, and
// bits of the tile number add a tile's total to the sum of each set bit.
// A large register is bound by HBM reads: 296 blocks of eight 16-byte loads
// per thread keep 64 KiB per SM in flight, and contiguous tile ranges keep
// the blocks within one tile of one another (a grid of 512 blocks left the
// last of its 3.5 blocks per SM alone). Small registers are bound by
// latency: up to one tile (11 or 12 qubits) one block writes the sums
// itself; otherwise the second kernel adds the blocks' partials, a warp per
// sum. Under the profiler: 800 -> 9 us at 11 qubits (one thread did it all),
// 18 + 59 -> 5.5 + 9 at 17, 36 + 60 -> 17 + 9 at 22; complex128 at 27
// qubits reads at 6.6 TB/s.
constexpr int kZThreads = 256;
constexpr int kZLoads = 8;
constexpr int kZMaxBlocks = 296;                // two per SM
constexpr int kZMaxHi = kMaxQubits - 11;        // bits of the tile number

template <typename V>
struct ZTile
{
    static constexpr int kBits = 11 + (sizeof(V) == 16 ? 0 : 1);   // amplitudes of a tile
};

// The sums as the host receives them: result in device memory and, when host
// is not null, in pinned host memory followed by done = seq (as for a
// measurement).
struct ZResult
{
    double *sums;
    double *host;
    volatile unsigned *done;
    unsigned seq;
};

__device__ __forceinline__ void zsums_write(const ZResult &r, int j, double v)
{
    r.sums[j] = v;
    if (r.host != nullptr)
    {
        r.host[j] = v;
        __threadfence_system();
    }
}

// after a block-wide barrier behind every zsums_write of the block
__device__ __forceinline__ void zsums_signal(const ZResult &r)
{
    if (threadIdx.x == 0 && r.host != nullptr)
    {
        __threadfence_system();
        *r.done = r.seq;
    }
}

__device__ __forceinline__ double2 ld_word(const double2 *p) { return __ldcs(p); }
__device__ __forceinline__ float4 ld_word(const float2 *p) { return __ldcs(reinterpret_cast<const float4 *>(p)); }
// squared norms of a word's amplitudes: the word's sum, and the part of its
// odd amplitude (complex64)
__device__ __forceinline__ void word_norms(double2 a, double &sum, double &odd)
{
    sum = norm2(a);
    odd = 0.0;
}
__device__ __forceinline__ void word_norms(float4 a, double &sum, double &odd)
{
    odd = norm2(make_float2(a.z, a.w));
    sum = norm2(make_float2(a.x, a.y)) + odd;
}

// partials: [sum][block]; with one block the sums go to r
template <typename V>
__global__ void __launch_bounds__(kZThreads, 2) zsums_kernel(const V *state, int n, double *partials, ZResult r)
{
    constexpr int kTileBits = ZTile<V>::kBits;
    constexpr int kWordBits = kTileBits - 11;           // 0 or 1
    constexpr int kThreadBit = kWordBits;               // thread bits of the index start here
    constexpr int kLoadBit = kWordBits + 8;             // then the bits of u
    const int tid = threadIdx.x, w = tid / 32, l = tid % 32;
    const int nhi = n > kTileBits ? n - kTileBits : 0;
    const uint64_t tiles = 1ull << nhi;
    const uint64_t first = tiles * blockIdx.x / gridDim.x, last = tiles * (blockIdx.x + 1) / gridDim.x;
    // words of the register below one tile
    const uint32_t words = n >= kTileBits ? kZLoads * kZThreads : (1u << n) >> kWordBits;
    double total = 0.0, odd = 0.0, ub[3] = {0.0, 0.0, 0.0}, hi[kZMaxHi];
#pragma unroll
    for (int q = 0; q < kZMaxHi; ++q)
        hi[q] = 0.0;
    for (uint64_t tile = first; tile < last; ++tile)
    {
        const V *base = state + (tile << kTileBits);
        decltype(ld_word(base)) a[kZLoads];
        if (words == kZLoads * kZThreads)
        {
#pragma unroll
            for (int u = 0; u < kZLoads; ++u)
                a[u] = ld_word(base + ((u * kZThreads + tid) << kWordBits));
        }
        else
        {
#pragma unroll
            for (int u = 0; u < kZLoads; ++u)
                if (u * kZThreads + tid < words)
                    a[u] = ld_word(base + ((u * kZThreads + tid) << kWordBits));
                else
                    a[u] = decltype(ld_word(base)){};
        }
        double pr[kZLoads], t = 0.0;
#pragma unroll
        for (int u = 0; u < kZLoads; ++u)
        {
            double o;
            word_norms(a[u], pr[u], o);
            odd += o;
        }
#pragma unroll
        for (int b = 0; b < 3; ++b)
        {
            double s = 0.0;
#pragma unroll
            for (int u = 0; u < kZLoads; ++u)
                if ((u >> b) & 1)
                    s += pr[u];
            ub[b] += s;
        }
#pragma unroll
        for (int u = 0; u < kZLoads; ++u)
            t += pr[u];
        total += t;
#pragma unroll
        for (int q = 0; q < kZMaxHi; ++q)
            if (q < nhi && ((tile >> q) & 1))
                hi[q] += t;
    }
    // per warp: the total, its five lane-bit sums, the thread's own splits
    constexpr int kFixed = 6 + 3 + 1;
    __shared__ double sh[kFixed + kZMaxHi][kZThreads / 32];
    auto put = [&](int row, double v) {
        const double s = warp_sum(v);
        if (l == 0)
            sh[row][w] = s;
    };
    put(0, total);
#pragma unroll
    for (int b = 0; b < 5; ++b)
        put(1 + b, ((l >> b) & 1) ? total : 0.0);
#pragma unroll
    for (int b = 0; b < 3; ++b)
        put(6 + b, ub[b]);
    if (kWordBits)
        put(9, odd);
#pragma unroll
    for (int q = 0; q < kZMaxHi; ++q)
        if (q < nhi)
            put(kFixed + q, hi[q]);
    __syncthreads();
    if (tid <= n)
    {
        // sum tid: the total, then bit tid - 1 of the index
        const int q = tid - 1;
        int row = 0;
        unsigned warps = 0xffu;
        if (q >= 0)
        {
            if (q < kThreadBit)
                row = 9;
            else if (q < kThreadBit + 5)
                row = 1 + q - kThreadBit;
            else if (q < kLoadBit)
                warps = q - kThreadBit == 5 ? 0xaau : q - kThreadBit == 6 ? 0xccu : 0xf0u;
            else if (q < kTileBits)
                row = 6 + q - kLoadBit;
            else
                row = kFixed + q - kTileBits;
        }
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < kZThreads / 32; ++k)
            if ((warps >> k) & 1)
                s += sh[row][k];
        if (gridDim.x == 1)
            zsums_write(r, tid, s);
        else
            partials[(size_t)tid * gridDim.x + blockIdx.x] = s;
    }
    if (gridDim.x == 1)
    {
        __syncthreads();
        zsums_signal(r);
    }
}

__global__ void __launch_bounds__(1024) zsums_final_kernel(const double *partials, int nblocks, int nsums, ZResult r)
{
    const int w = threadIdx.x / 32, l = threadIdx.x % 32;
    for (int j = w; j < nsums; j += 32)
    {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < (kZMaxBlocks + 31) / 32; ++i)
            if (l + 32 * i < nblocks)
                s += __ldcg(partials + (size_t)j * nblocks + l + 32 * i);
        s = warp_sum(s);
        if (l == 0)
            zsums_write(r, j, s);
    }
    __syncthreads();
    zsums_signal(r);
}

// ------------------------------------------------------------ transfers

struct PermParams
{
    int n;
    int l2p[kMaxQubits];
};

__device__ __forceinline__ uint64_t logical_to_physical(uint64_t l, const PermParams &pp)
{
    uint64_t ph = 0;
    for (int j = 0; j < pp.n; ++j)
        ph |= ((l >> j) & 1ull) << pp.l2p[j];
    return ph;
}

template <typename V>
__global__ void gather_logical_kernel(const V *state, PermParams pp, uint64_t begin, uint64_t count, double2 *out)
{
    for (uint64_t k = (uint64_t)blockIdx.x * kThreads + threadIdx.x; k < count; k += (uint64_t)gridDim.x * kThreads)
    {
        const V a = state[logical_to_physical(begin + k, pp)];
        out[k] = make_double2(a.x, a.y);
    }
}

template <typename V>
__global__ void scatter_logical_kernel(V *state, PermParams pp, uint64_t begin, uint64_t count, const double2 *in)
{
    for (uint64_t k = (uint64_t)blockIdx.x * kThreads + threadIdx.x; k < count; k += (uint64_t)gridDim.x * kThreads)
        state[logical_to_physical(begin + k, pp)] = make_cx<V>(in[k].x, in[k].y);
}

template <typename V>
__global__ void widen_kernel(const V *in, uint64_t count, double2 *out)
{
    for (uint64_t k = (uint64_t)blockIdx.x * kThreads + threadIdx.x; k < count; k += (uint64_t)gridDim.x * kThreads)
        out[k] = make_double2(in[k].x, in[k].y);
}

template <typename V>
__global__ void narrow_kernel(const double2 *in, uint64_t count, V *out)
{
    for (uint64_t k = (uint64_t)blockIdx.x * kThreads + threadIdx.x; k < count; k += (uint64_t)gridDim.x * kThreads)
        out[k] = make_cx<V>(in[k].x, in[k].y);
}

template <typename V>
__global__ void gather_indices_kernel(const V *state, const uint64_t *physical, uint64_t count, double2 *out)
{
    for (uint64_t k = (uint64_t)blockIdx.x * kThreads + threadIdx.x; k < count; k += (uint64_t)gridDim.x * kThreads)
    {
        const V a = state[physical[k]];
        out[k] = make_double2(a.x, a.y);
    }
}

// Per block: sum of conj(x_i) * y_i (re, im), max |x_i - y_i|, sum |x_i|^2
// and sum |y_i|^2, written as five doubles; a fixed grid and order make
// repeated calls identical.
__global__ void __launch_bounds__(kThreads) compare_kernel(const double2 *x, const double2 *y, uint64_t count,
                                                           double *partials)
{
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (uint64_t k = (uint64_t)blockIdx.x * kThreads + threadIdx.x; k < count; k += (uint64_t)gridDim.x * kThreads)
    {
        const double2 a = __ldcs(x + k), b = __ldcs(y + k);
        v[0] += a.x * b.x + a.y * b.y;
        v[1] += a.x * b.y - a.y * b.x;
        const double dx = a.x - b.x, dy = a.y - b.y;
        v[2] = fmax(v[2], sqrt(dx * dx + dy * dy));
        v[3] += a.x * a.x + a.y * a.y;
        v[4] += b.x * b.x + b.y * b.y;
    }
    __shared__ double sh[5][kThreads / 32];
    const int w = threadIdx.x / 32, l = threadIdx.x % 32;
#pragma unroll
    for (int i = 0; i < 5; ++i)
    {
        double t = v[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            const double u = __shfl_xor_sync(0xffffffffu, t, o);
            t = i == 2 ? fmax(t, u) : t + u;
        }
        if (l == 0)
            sh[i][w] = t;
    }
    __syncthreads();
    if (threadIdx.x < 5)
    {
        const int i = threadIdx.x;
        double t = 0.0;
        for (int k = 0; k < kThreads / 32; ++k)
            t = i == 2 ? fmax(t, sh[i][k]) : t + sh[i][k];
        partials[5 * blockIdx.x + i] = t;
    }
}

PermParams make_perm(int n, const int *l2p)
{
    PermParams pp;
    pp.n = n;
    for (int j = 0; j < n; ++j)
        pp.l2p[j] = l2p[j];
    return pp;
}

} // namespace

template <typename R>
int launch_gate_plain(typename Cx<R>::T *state, int n, const GateOp &op, cudaStream_t stream)
{
    if (op.na == 0)
        return 0;
    return op.diag ? launch_plain_dispatch<R, true>(state, n, op, stream)
                   : launch_plain_dispatch<R, false>(state, n, op, stream);
}

template <typename R>
int launch_gates_small(typename Cx<R>::T *state, int n, const GateOp *ops, size_t count, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    if (n > kSmallQubits)
        throw std::runtime_error("internal: register too large for the small-register kernel");
    int launches = 0;
    SmallParams<R> p;
    std::memset(&p, 0, sizeof(p));
    p.state = state;
    p.n = n;
    int entries = 0;
    auto flush = [&]() {
        if (p.count == 0)
            return;
        small_register_kernel<R><<<1, kSmallThreads, 0, stream>>>(p);
        QCSB_CUDA(cudaGetLastError());
        ++launches;
        p.count = entries = 0;
    };
    for (size_t k = 0; k < count; ++k)
    {
        const GateOp &op = ops[k];
        if (op.na == 0)
            continue;
        const int ne = op.diag ? op.na : op.na * op.na;
        if (p.count == kSmallOps || entries + ne > kSmallEntries)
            flush();
        SmallOp &o = p.ops[p.count++];
        uint64_t masks[kMaxOps];
        o.nops = static_cast<uint8_t>(fill_masks(op, masks));
        for (int i = 0; i < o.nops; ++i)
            o.masks[i] = static_cast<uint8_t>(masks[i]);
        o.na = static_cast<uint8_t>(op.na);
        o.diag = op.diag;
        o.entry = static_cast<uint16_t>(entries);
        o.cval = static_cast<uint16_t>(op.cval);
        for (int a = 0; a < op.na; ++a)
        {
            o.off[a] = 0;
            for (int i = 0; i < op.nt; ++i)
                if ((op.act[a] >> i) & 1)
                    o.off[a] |= static_cast<uint16_t>(1u << op.tq[i]);
        }
        for (int e = 0; e < ne; ++e)
            p.entries[entries++] = make_cx<V>(op.mat[e].re, op.mat[e].im);
    }
    flush();
    return launches;
}

template <typename R>
int launch_init_zero(typename Cx<R>::T *state, int n, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    QCSB_CUDA(cudaMemsetAsync(state, 0, sizeof(V) << n, stream));
    set_one_kernel<V><<<1, 1, 0, stream>>>(state, 0, make_cx<V>(1.0, 0.0));
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_init_flat(typename Cx<R>::T *state, int n, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    const uint64_t count = 1ull << n;
    fill_kernel<V><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(state, count, make_cx<V>(1.0, 0.0));
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_init_sequential(typename Cx<R>::T *state, int n, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    const uint64_t count = 1ull << n;
    sequential_kernel<V><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(state, count);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_rescale(typename Cx<R>::T *state, int n, double target, const double *norm_dev, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    const uint64_t count = 1ull << n;
    rescale_kernel<V><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(state, count, target, norm_dev);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_set_amplitude(typename Cx<R>::T *state, uint64_t index, double re, double im, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    set_one_kernel<V><<<1, 1, 0, stream>>>(state, index, make_cx<V>(re, im));
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_measure_probs(const typename Cx<R>::T *state, int n, int t, uint64_t cmask, uint64_t cval,
                         double2 *partials, double2 *result, unsigned *ticket, unsigned *done, unsigned seq,
                         cudaStream_t stream)
{
    ProbParams<R> p;
    std::memset(&p, 0, sizeof(p));
    p.state = state;
    p.ngroups = 1ull << (n - fill_runs(cmask | (1ull << t), p.runs));
    p.cval = cval;
    p.tbit = 1ull << t;
    p.partials = partials;
    p.result = result;
    p.ticket = ticket;
    p.done = done;
    p.seq = seq;
    measure_probs_kernel<R><<<grid_for(p.ngroups, kThreads * 2 * kProbGroups, kReduceBlocks), kThreads, 0, stream>>>(p);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_collapse(typename Cx<R>::T *state, int n, int t, int keep_value, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    const uint64_t ngroups = 1ull << (n - 1);
    const uint64_t zero_bit = keep_value ? 0ull : (1ull << t);
    collapse_kernel<V><<<grid_for(ngroups, kThreads * 4), kThreads, 0, stream>>>(state, ngroups, (1ull << t) - 1, zero_bit);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_collapse_mask(typename Cx<R>::T *state, int n, uint64_t cmask, uint64_t cval, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    const uint64_t count = 1ull << n;
    collapse_mask_kernel<V><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(state, count, cmask, cval);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_zsums(const typename Cx<R>::T *state, int n, double *partials, double *sums, cudaStream_t stream,
                 double *host, unsigned *done, unsigned seq)
{
    typedef typename Cx<R>::T V;
    const ZResult r{sums, host, done, seq};
    const int tile_bits = ZTile<V>::kBits;
    const uint64_t tiles = n > tile_bits ? 1ull << (n - tile_bits) : 1;
    const unsigned blocks = static_cast<unsigned>(tiles < kZMaxBlocks ? tiles : kZMaxBlocks);
    zsums_kernel<V><<<blocks, kZThreads, 0, stream>>>(state, n, partials, r);
    QCSB_CUDA(cudaGetLastError());
    if (blocks == 1)
        return 1;
    zsums_final_kernel<<<1, 1024, 0, stream>>>(partials, static_cast<int>(blocks), n + 1, r);
    QCSB_CUDA(cudaGetLastError());
    return 2;
}

template <typename R>
int launch_gather_indices(const typename Cx<R>::T *state, const uint64_t *physical, uint64_t count, double2 *out,
                          cudaStream_t stream)
{
    gather_indices_kernel<typename Cx<R>::T><<<grid_for(count, kThreads), kThreads, 0, stream>>>(state, physical, count, out);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

int launch_compare(const double2 *x, const double2 *y, uint64_t count, double *partials, cudaStream_t stream)
{
    compare_kernel<<<kReduceBlocks, kThreads, 0, stream>>>(x, y, count, partials);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_gather_logical(const typename Cx<R>::T *state, int n, const int *l2p, uint64_t begin,
                          uint64_t count, double2 *out, cudaStream_t stream)
{
    gather_logical_kernel<typename Cx<R>::T><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(state, make_perm(n, l2p), begin, count, out);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_scatter_logical(typename Cx<R>::T *state, int n, const int *l2p, uint64_t begin,
                           uint64_t count, const double2 *in, cudaStream_t stream)
{
    scatter_logical_kernel<typename Cx<R>::T><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(state, make_perm(n, l2p), begin, count, in);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_widen(const typename Cx<R>::T *in, uint64_t count, double2 *out, cudaStream_t stream)
{
    widen_kernel<typename Cx<R>::T><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(in, count, out);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template <typename R>
int launch_narrow(const double2 *in, uint64_t count, typename Cx<R>::T *out, cudaStream_t stream)
{
    narrow_kernel<typename Cx<R>::T><<<grid_for(count, kThreads * 4), kThreads, 0, stream>>>(in, count, out);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

#define QCSB_INSTANTIATE(R)                                                                                         \
    template int launch_gate_plain<R>(Cx<R>::T *, int, const GateOp &, cudaStream_t);                               \
    template int launch_gates_small<R>(Cx<R>::T *, int, const GateOp *, size_t, cudaStream_t);                      \
    template int launch_init_zero<R>(Cx<R>::T *, int, cudaStream_t);                                                \
    template int launch_init_flat<R>(Cx<R>::T *, int, cudaStream_t);                                                \
    template int launch_init_sequential<R>(Cx<R>::T *, int, cudaStream_t);                                          \
    template int launch_set_amplitude<R>(Cx<R>::T *, uint64_t, double, double, cudaStream_t);                      \
    template int launch_rescale<R>(Cx<R>::T *, int, double, const double *, cudaStream_t);                          \
    template int launch_measure_probs<R>(const Cx<R>::T *, int, int, uint64_t, uint64_t, double2 *, double2 *,      \
                                         unsigned *, unsigned *, unsigned, cudaStream_t);                           \
    template int launch_collapse<R>(Cx<R>::T *, int, int, int, cudaStream_t);                                       \
    template int launch_collapse_mask<R>(Cx<R>::T *, int, uint64_t, uint64_t, cudaStream_t);                        \
    template int launch_zsums<R>(const Cx<R>::T *, int, double *, double *, cudaStream_t, double *, unsigned *,     \
                                 unsigned);                                                                         \
    template int launch_gather_logical<R>(const Cx<R>::T *, int, const int *, uint64_t, uint64_t, double2 *,        \
                                          cudaStream_t);                                                            \
    template int launch_scatter_logical<R>(Cx<R>::T *, int, const int *, uint64_t, uint64_t, const double2 *,       \
                                           cudaStream_t);                                                           \
    template int launch_widen<R>(const Cx<R>::T *, uint64_t, double2 *, cudaStream_t);                              \
    template int launch_narrow<R>(const double2 *, uint64_t, Cx<R>::T *, cudaStream_t);                           \
    template int launch_gather_indices<R>(const Cx<R>::T *, const uint64_t *, uint64_t, double2 *, cudaStream_t);

QCSB_INSTANTIATE(double)
QCSB_INSTANTIATE(float)

} // namespace qcsb

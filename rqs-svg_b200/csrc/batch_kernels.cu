// <Z> of every register of a batch in one pass over the arena, and the
// |0..0> preparation of registers that no fused pass initialises.
//
// Work item = a slice of up to 2^16 amplitudes of one register; one CTA of
// 256 threads per item. Thread t reads amplitudes t + 256 j: bits 0..7 of the
// index are t's bits (constant per thread), bits 8.. come from j (at most 8
// bits), bits above the slice from the item. So a thread only needs its total
// and one sum per loop bit; the thread-bit sums and the slice-bit sums follow
// from the totals. Everything accumulates in FP64.

#include "batch.h"

namespace qcsb
{
namespace
{

constexpr int kZThreads = 256;

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// partials[item * kBatchZPartials + ...] = total, sums over bits 0..7 (thread
// bits), sums over bits 8..15 (loop bits) of this slice
template <typename V>
__global__ void __launch_bounds__(kZThreads) batch_zsums_kernel(const V *arena, const BatchZItem *items,
                                                                double *partials)
{
    const BatchZItem it = items[blockIdx.x];
    const int sb = it.n < kBatchZSliceBits ? it.n : kBatchZSliceBits;
    const int jbits = sb - 8;
    const V *base = arena + it.amp_off + ((uint64_t)it.slice << sb);
    const int t = threadIdx.x;
    double tot = 0.0, hi[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int nj = 1 << jbits;
    for (int j = 0; j < nj; ++j)
    {
        const V a = __ldcs(base + t + (j << 8));
        const double p = (double)a.x * (double)a.x + (double)a.y * (double)a.y;
        tot += p;
#pragma unroll
        for (int b = 0; b < 8; ++b)
            if (b < jbits && ((j >> b) & 1))
                hi[b] += p;
    }
    double v[kBatchZPartials];
    v[0] = tot;
#pragma unroll
    for (int b = 0; b < 8; ++b)
        v[1 + b] = ((t >> b) & 1) ? tot : 0.0;
#pragma unroll
    for (int b = 0; b < 8; ++b)
        v[9 + b] = hi[b];
    __shared__ double sh[kBatchZPartials][kZThreads / 32];
    const int w = t / 32, l = t % 32;
#pragma unroll
    for (int i = 0; i < kBatchZPartials; ++i)
    {
        const double s = warp_sum(v[i]);
        if (l == 0)
            sh[i][w] = s;
    }
    __syncthreads();
    if (t < kBatchZPartials)
    {
        double s = 0.0;
        for (int k = 0; k < kZThreads / 32; ++k)
            s += sh[t][k];
        partials[(uint64_t)blockIdx.x * kBatchZPartials + t] = s;
    }
}

// One thread per register: <Z_q> = (total - 2 sum_q) / total.
__global__ void batch_zfinal_kernel(const double *partials, const BatchZItem *items, const BatchZReg *regs,
                                    uint32_t num_regs, double *out)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= num_regs)
        return;
    const BatchZReg g = regs[r];
    const int n = g.n;
    const int sb = n < kBatchZSliceBits ? n : kBatchZSliceBits;
    double tot = 0.0, s[kMaxQubits];
    for (int q = 0; q < n; ++q)
        s[q] = 0.0;
    for (uint32_t i = 0; i < g.count; ++i)
    {
        const double *p = partials + (uint64_t)(g.first + i) * kBatchZPartials;
        const uint32_t slice = items[g.first + i].slice;
        tot += p[0];
        for (int q = 0; q < 8 && q < n; ++q)
            s[q] += p[1 + q];
        for (int q = 8; q < sb; ++q)
            s[q] += p[9 + (q - 8)];
        for (int q = sb; q < n; ++q)
            if ((slice >> (q - sb)) & 1)
                s[q] += p[0];
    }
    for (int q = 0; q < n; ++q)
        out[g.out_off + q] = tot > 0.0 ? (tot - 2.0 * s[q]) / tot : 0.0;
}

// Element (r, c) of a parametrised gate, the formulas of gate_matrix
// (gate_table.cpp).
//
// e^{ix} with both parts within 0.66 ulp (root mean square 0.29, what the
// host's sin and cos give), where CUDA's sincos may be 2 ulp off: with it the
// states of ansatz circuits were 1.04-1.24 times as far from 80-bit results as
// with entries from the host. x - k pi/2 with pi/2 in three parts
// (Cody-Waite; the products' errors by FMA, Knuth's two-sum), Taylor series to
// x^17 and x^18 on +-pi/4, the leading terms in two parts. Beyond 2^40, where
// the three parts would not do, sincos.
__device__ __forceinline__ double two_sum(double a, double b, double &err)
{
    const double s = __dadd_rn(a, b), z = __dsub_rn(s, a);
    err = __dadd_rn(__dsub_rn(a, __dsub_rn(s, z)), __dsub_rn(b, z));
    return s;
}

__device__ __noinline__ double2 expi(double x)
{
    if (!(fabs(x) <= 1099511627776.0))
    {
        double s, c;
        sincos(x, &s, &c);
        return make_double2(c, s);
    }
    constexpr double kHalfPi[3] = {1.5707963267948966, 6.123233995736766e-17, -1.4973849048591698e-33};
    const double k = rint(x * 0.6366197723675814);
    const double p = __dmul_rn(k, kHalfPi[0]), q = __dmul_rn(k, kHalfPi[1]);
    double e0, e1, e2;
    double r = two_sum(x, -p, e0);
    r = two_sum(r, -__fma_rn(k, kHalfPi[0], -p), e1);
    r = two_sum(r, -q, e2);
    const double lo = __dsub_rn(__dsub_rn(__dadd_rn(__dadd_rn(e0, e1), e2), __fma_rn(k, kHalfPi[1], -q)), k * kHalfPi[2]);
    const double h = __dadd_rn(r, lo), l = __dsub_rn(lo, __dsub_rn(h, r));
    const double z = __dmul_rn(h, h), zl = __fma_rn(h, h, -z);
    // (-1)^j / (2j + 1)!, j = 8 .. 1, and (-1)^j / (2j)!, j = 9 .. 2
    constexpr double kSin[8] = {1.0 / 355687428096000.0, -1.0 / 1307674368000.0, 1.0 / 6227020800.0, -1.0 / 39916800.0,
                                1.0 / 362880.0, -1.0 / 5040.0, 1.0 / 120.0, -1.0 / 6.0};
    constexpr double kCos[8] = {-1.0 / 6402373705728000.0, 1.0 / 20922789888000.0, -1.0 / 87178291200.0, 1.0 / 479001600.0,
                                -1.0 / 3628800.0, 1.0 / 40320.0, -1.0 / 720.0, 1.0 / 24.0};
    double ps = kSin[0], pc = kCos[0];
#pragma unroll
    for (int i = 1; i < 8; ++i)
    {
        ps = __fma_rn(ps, z, kSin[i]);
        pc = __fma_rn(pc, z, kCos[i]);
    }
    const double s = __dadd_rn(h, __fma_rn(__dmul_rn(h, z), ps, l * (1.0 - 0.5 * z)));
    const double half = 0.5 * z, w = __dsub_rn(1.0, half);
    const double tail = __fma_rn(__dmul_rn(z, z), pc, -0.5 * zl) - h * l;
    const double c = __dadd_rn(w, __dadd_rn(__dsub_rn(__dsub_rn(1.0, w), half), tail));
    switch (static_cast<long long>(k) & 3)
    {
    case 0: return make_double2(c, s);
    case 1: return make_double2(-s, c);
    case 2: return make_double2(-c, -s);
    default: return make_double2(s, -c);
    }
}
__device__ __forceinline__ double2 scaled(double f, double2 a) { return make_double2(f * a.x, f * a.y); }
__device__ __forceinline__ double2 times(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ double2 gate_element(uint8_t formula, int r, int c, const double *p)
{
    constexpr double kRsqrt2 = 0.70710678118654752440;
    const double2 same = make_double2(r == c ? 1.0 : 0.0, 0.0);
    switch (formula)
    {
    case B_GLOBAL_PHASE: return expi(p[0]);
    case B_P: return r == 1 && c == 1 ? expi(p[0]) : same;
    case B_U2:
        if (r == 0)
            return c == 0 ? make_double2(kRsqrt2, 0.0) : scaled(-kRsqrt2, expi(p[1]));
        return scaled(kRsqrt2, expi(c == 0 ? p[0] : p[0] + p[1]));
    default: break;
    }
    // the others turn by half of their first parameter
    const double2 h = expi(0.5 * p[0]);
    const double cs = h.x, sn = h.y;
    switch (formula)
    {
    case B_RX: return r == c ? make_double2(cs, 0.0) : make_double2(0.0, -sn);
    case B_RY: return make_double2(r == c ? cs : r == 0 ? -sn : sn, 0.0);
    case B_RZ: return r != c ? same : make_double2(cs, r == 0 ? -sn : sn);
    case B_U3:
        if (r == 0)
            return c == 0 ? make_double2(cs, 0.0) : scaled(-sn, expi(p[2]));
        return c == 0 ? scaled(sn, expi(p[1])) : scaled(cs, expi(p[1] + p[2]));
    case B_U4:
    {
        const double2 eg = expi(p[3]);
        if (r == 0)
            return c == 0 ? scaled(cs, eg) : times(eg, scaled(-sn, expi(p[2])));
        return c == 0 ? times(eg, scaled(sn, expi(p[1]))) : times(eg, times(expi(p[1]), scaled(cs, expi(p[2]))));
    }
    case B_RXX:
    case B_RYY:
        if (r == c)
            return make_double2(cs, 0.0);
        return r + c != 3 ? same : make_double2(0.0, formula == B_RYY && (r == 0 || r == 3) ? sn : -sn);
    case B_RZZ: return r != c ? same : make_double2(cs, r == 0 || r == 3 ? -sn : sn);
    case B_RZX:
        if (r == c)
            return make_double2(cs, 0.0);
        return (r ^ c) != 2 ? same : make_double2(0.0, (r & 1) ? sn : -sn);
    default: break;
    }
    // B_R, B_XX_PLUS_YY, B_XX_MINUS_YY: [[c, -i s e^{-i b}], [-i s e^{i b}, c]]
    // on sub-indices lo and hi
    const int lo = formula == B_XX_PLUS_YY ? 1 : 0;
    const int hi = formula == B_R ? 1 : formula == B_XX_PLUS_YY ? 2 : 3;
    if ((r != lo && r != hi) || (c != lo && c != hi))
        return same;
    if (r == c)
        return make_double2(cs, 0.0);
    const double2 b = expi(p[1]);
    return make_double2(r == lo ? -sn * b.y : sn * b.y, -sn * b.x);
}

// A block per register: thread by thread the entries of its block, each one
// matrix element. A batch's entries take a few microseconds (on the host,
// gate by gate, 17 us per 20-qubit circuit of 480 gates on one core, more
// than the GPU's time for its passes).
template <typename Real>
__global__ void __launch_bounds__(kZThreads) batch_fill_kernel(const BatchFillReg *regs, const BatchEntry *recipes,
                                                               const double2 *consts, const double *params,
                                                               double2 *entries)
{
    const BatchFillReg g = regs[blockIdx.x];
    for (uint32_t i = threadIdx.x; i < g.count; i += kZThreads)
    {
        const BatchEntry e = recipes[g.recipe + i];
        const double2 v = e.formula == B_CONST
                              ? consts[g.consts + e.index]
                              : gate_element(e.formula, e.element >> 2, e.element & 3, params + g.params + e.index);
        if (sizeof(Real) == 4)
            reinterpret_cast<float2 *>(entries + g.block)[i] = make_float2(static_cast<float>(v.x), static_cast<float>(v.y));
        else
            entries[g.block + i] = v;
    }
}

template <typename V>
__global__ void batch_set_ones_kernel(V *base, uint64_t stride, uint32_t count)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < count)
    {
        V one;
        one.x = 1;
        one.y = 0;
        base[(uint64_t)r * stride] = one;
    }
}

} // namespace

template <typename R>
int launch_batch_zsums(const void *arena, const BatchZItem *items, uint32_t num_items, const BatchZReg *regs,
                       uint32_t num_regs, double *partials, double *out, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    if (num_items == 0)
        return 0;
    batch_zsums_kernel<V><<<num_items, kZThreads, 0, stream>>>(static_cast<const V *>(arena), items, partials);
    QCSB_CUDA(cudaGetLastError());
    batch_zfinal_kernel<<<(num_regs + 127) / 128, 128, 0, stream>>>(partials, items, regs, num_regs, out);
    QCSB_CUDA(cudaGetLastError());
    return 2;
}

template <typename R>
int launch_batch_fill(const BatchFillReg *regs, uint32_t num_regs, const BatchEntry *recipes, const double2 *consts,
                      const double *params, double2 *entries, cudaStream_t stream)
{
    if (num_regs == 0)
        return 0;
    batch_fill_kernel<R><<<num_regs, kZThreads, 0, stream>>>(regs, recipes, consts, params, entries);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}
template int launch_batch_fill<double>(const BatchFillReg *, uint32_t, const BatchEntry *, const double2 *,
                                       const double *, double2 *, cudaStream_t);
template int launch_batch_fill<float>(const BatchFillReg *, uint32_t, const BatchEntry *, const double2 *,
                                      const double *, double2 *, cudaStream_t);

template <typename R>
int launch_batch_set_ones(void *base, uint64_t stride, uint32_t count, cudaStream_t stream)
{
    typedef typename Cx<R>::T V;
    if (count == 0)
        return 0;
    batch_set_ones_kernel<V><<<(count + 127) / 128, 128, 0, stream>>>(static_cast<V *>(base), stride, count);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}

template int launch_batch_zsums<double>(const void *, const BatchZItem *, uint32_t, const BatchZReg *, uint32_t,
                                        double *, double *, cudaStream_t);
template int launch_batch_zsums<float>(const void *, const BatchZItem *, uint32_t, const BatchZReg *, uint32_t,
                                       double *, double *, cudaStream_t);
template int launch_batch_set_ones<double>(void *, uint64_t, uint32_t, cudaStream_t);
template int launch_batch_set_ones<float>(void *, uint64_t, uint32_t, cudaStream_t);

} // namespace qcsb

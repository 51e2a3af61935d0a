// Butterfly passes: register passes whose stages are Hadamard gates and
// diagonal runs only (a quantum Fourier transform's), as radix-2 butterflies.
//
// The general register pass (fused_pass.cu) interprets such a stage op by op:
// H as a real 2x2 (four FP64 operations per output pair and component where
// two do), a factor for all 16 slots after it (where half of them are 1), and
// the register moves between the ops' fixed register assignments: the
// 28-qubit QFT's passes issued 39% of their instructions as moves and took
// 3.86 ms against 1.31 ms of HBM time. Here a stage is straight-line code
// over its four bits, highest first: a bit's H as a + b and a - b, its phases
// to the other stage bits as one factor per difference, its phases to the
// thread's and the chunk's bits as one table-fed factor. The sqrt(1/2) of the
// Hs, m in a pass, is one factor 2^(-m/2) at its end.
//
// Memory: thread t holds 16 amplitudes that differ in the stage's bits. When
// the first (last) stage leaves local bits 0..2 alone, eight threads hold
// whole 128- (64-) byte runs: each loads straight to its own slots (stores
// straight from registers), and a two-stage pass has two barriers per chunk.
// For complex128 the next chunk streams into the buffer during this one's
// last stage (28-qubit flush 9.85 -> 9.35 ms); complex64 loads to registers
// (with it 7.11 -> 7.38 ms). The 28-qubit QFT with 1024 shots
// went from 16.9 to 11.3 ms (four passes of about 2.5 ms), its error against
// 64 bits from 4.1e-15 to 2.2e-15.
// One chunk buffer per CTA, four (complex64: eight) CTAs per SM.

#include "fused_pass.h"
#include "fused_device.cuh"

#include <cmath>
#include <cstring>

namespace qcsb
{
namespace
{

using namespace fdev;

constexpr int kThreads = 1 << (kTensorLocal - kStageBits);
constexpr double kRsqrt2 = 0.70710678118654752440;   // the entries of gate_matrix's H

// One run's table-fed factors: E[0] on every slot, E[1 + b] on the slots with
// stage bit b (layout as for F_PRUN). The chunk's part of factor e is the
// same for the whole CTA: lane e of each warp multiplies it together (its
// loads in flight with the other lanes') and hands it round, instead of every
// thread reading up to four tables per factor.
template <typename V>
__device__ __forceinline__ V from_lane(V v, int lane)
{
    return V{__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane)};
}

template <typename V>
__device__ __forceinline__ void apply_run(V (&a)[R], const BRun &run, const double2 *tables, uint64_t chunk, int tid)
{
    const uint32_t lm = static_cast<uint32_t>(run.packed) & 31u;
    V part = V{1, 0};
    const int lane = tid & 31;
    if (lane <= kStageBits)
        for (int g = 0; g < run.groups; ++g)
            if ((run.packed >> (kChunkGroupBits * (g + 1) + lane)) & 1)
            {
                const uint32_t idx = static_cast<uint32_t>(chunk >> (kChunkGroupBits * g)) & ((1u << kChunkGroupBits) - 1);
                part = cmul(cvt<V>(__ldg(tables + run.group_table[g][lane] + idx)), part);
            }
#pragma unroll
    for (int e = 0; e <= kStageBits; ++e)
    {
        if (!((run.used >> e) & 1))
            continue;
        V f = from_lane(part, e);
        if ((lm >> e) & 1)
            f = cmul(cvt<V>(__ldg(tables + run.thread_table[e] + tid)), f);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (e == 0 || ((r >> (e > 0 ? e - 1 : 0)) & 1))
                a[r] = cmul(f, a[r]);
    }
}

template <typename Real>
__global__ void __launch_bounds__(kThreads, sizeof(Real) == 8 ? 4 : 8)
    butterfly_pass_kernel(const __grid_constant__ BPassParams p)
{
    typedef typename Cx<Real>::T V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *const sb = reinterpret_cast<V *>(smem_raw);
    V *const state = static_cast<V *>(p.state);
    const V *const entries = reinterpret_cast<const V *>(p.entries);
    const int tid = threadIdx.x;

    // local index of the thread's slot 0 in a stage: zeros at the stage bits
    auto slot0 = [&](const BStage &S) {
        uint32_t j = static_cast<uint32_t>(tid);
#pragma unroll
        for (int b = 0; b < kStageBits; ++b)
        {
            const uint32_t lo = j & ((1u << S.sbits[b]) - 1u);
            j = lo | ((j ^ lo) << 1);
        }
        return j;
    };
    // a local index's amplitude offset
    auto offset_of = [&](uint32_t j) {
        uint64_t off = 0;
#pragma unroll
        for (int i = 0; i < kTensorLocal; ++i)
            if ((j >> i) & 1)
                off |= p.qbit[i];
        return off;
    };
    const int last = p.nstages - 1;
    const uint64_t in_off = offset_of(p.direct_in ? slot0(p.stages[0]) : static_cast<uint32_t>(tid));
    const uint64_t out_off = offset_of(p.direct_out ? slot0(p.stages[last]) : static_cast<uint32_t>(tid));
    // amplitude offset of slot (or, staged, of element tid + 128 m) r of a
    // thread: bits b of r at local positions pos(b)
    auto slot_offset = [&](int r, bool direct, const BStage &S) {
        uint64_t off = 0;
#pragma unroll
        for (int b = 0; b < kStageBits; ++b)
            if ((r >> b) & 1)
                off |= p.qbit[direct ? S.sbits[b] : kTensorLocal - kStageBits + b];
        return off;
    };
    // shared-memory position of a stage's slot r
    struct Slots
    {
        uint32_t p0, bit[kStageBits];
        __device__ __forceinline__ uint32_t operator()(int r) const
        {
            uint32_t q = p0;
#pragma unroll
            for (int b = 0; b < kStageBits; ++b)
                if ((r >> b) & 1)
                    q ^= bit[b];
            return q;
        }
    };
    auto slots_of = [&](const BStage &S) {
        Slots w;
        w.p0 = static_cast<uint32_t>(swz<V>(static_cast<int>(slot0(S))));
#pragma unroll
        for (int b = 0; b < kStageBits; ++b)
            w.bit[b] = static_cast<uint32_t>(swz<V>(1 << S.sbits[b]));
        return w;
    };
    auto chunk_base = [&](uint64_t c) {
        for (int i = 0; i < kTensorLocal; ++i)
        {
            const uint64_t lo = c & p.qmasks[i];
            c = lo | ((c ^ lo) << 1);
        }
        return c;
    };
    // the chunk's amplitudes on their way to shared memory: directly to the
    // first stage's slots of the same thread, or in order
    auto issue_load = [&](uint64_t base) {
        const V *src = state + (base | in_off);
        const Slots w = slots_of(p.stages[0]);
#pragma unroll
        for (int r = 0; r < R; ++r)
            cp_async_amp<V>(sb + (p.direct_in ? w(r) : swz<V>(tid + r * kThreads)),
                            src + slot_offset(r, p.direct_in, p.stages[0]));
        cp_async_commit();
    };

    const Real scale = static_cast<Real>(p.scale);
    uint64_t c = blockIdx.x;
    if (c >= p.chunks)
        return;
    uint64_t cbase = chunk_base(c);
    // straight to registers where nothing is left to stream behind, and for
    // complex64 (whose eight CTAs per SM overlap loads and stages as they are)
    const bool to_registers = p.direct_in && (sizeof(Real) == 4 || p.chunks <= gridDim.x);
    if (!to_registers)
        issue_load(cbase);
    for (; c < p.chunks; c += gridDim.x)
    {
        const uint64_t next = c + gridDim.x;
        const uint64_t cbase_next = next < p.chunks ? chunk_base(next) : cbase;
        V a[R];
        if (to_registers)
        {
            const V *src = state + (cbase | in_off);
#pragma unroll
            for (int r = 0; r < R; ++r)
                a[r] = __ldcg(src + slot_offset(r, true, p.stages[0]));
        }
        else
        {
            cp_async_wait<0>();
            if (!p.direct_in)
                __syncthreads();
        }
        for (int st = 0; st <= last; ++st)
        {
            const BStage &S = p.stages[st];
            const Slots w = slots_of(S);
            if (st > 0 || !to_registers)
            {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    a[r] = sb[w(r)];
            }
            if (st == last && p.direct_out && next < p.chunks)
            {
                // the buffer is free: the next chunk streams in during this
                // chunk's last stage
                __syncthreads();
                if (!to_registers)
                    issue_load(cbase_next);
            }
            // steps: the diagonals before the first H, then bits 3 .. 0
#pragma unroll
            for (int s = kStageBits; s >= 0; --s)
            {
                const BStep &step = S.steps[s];
                if (s < kStageBits && step.h)
                {
                    const int bit = 1 << (s < kStageBits ? s : 0);
#pragma unroll
                    for (int r = 0; r < R; ++r)
                    {
                        if (r & bit)
                            continue;
                        const V x = a[r], y = a[r | bit];
                        a[r] = V{x.x + y.x, x.y + y.y};
                        a[r | bit] = V{x.x - y.x, x.y - y.y};
                    }
                }
                if (step.factors == 1)
                {
                    // one factor per slot with bit s
                    int f = 0;
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (s < kStageBits && ((r >> (s < kStageBits ? s : 0)) & 1))
                            a[r] = cmul(entries[step.entry + f++], a[r]);
                }
                else if (step.factors == 2)
                {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        a[r] = cmul(entries[step.entry + r], a[r]);
                }
                if (step.run.used)
                    apply_run<V>(a, step.run, p.tables, c, tid);
            }
            if (st < last || !p.direct_out)
            {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    sb[w(r)] = a[r];
                __syncthreads();
            }
        }
        if (!p.direct_out)
        {
#pragma unroll
            for (int r = 0; r < R; ++r)
                a[r] = sb[swz<V>(tid + r * kThreads)];
            if (next < p.chunks)
            {
                __syncthreads();
                if (!to_registers)
                    issue_load(cbase_next);
            }
        }
        V *dst = state + (cbase | out_off);
#pragma unroll
        for (int r = 0; r < R; ++r)
            __stcs(dst + slot_offset(r, p.direct_out, p.stages[last]), V{a[r].x * scale, a[r].y * scale});
        cbase = cbase_next;
    }
}

bool identity2(const double2 *m)
{
    return m[0].x == 1.0 && m[0].y == 0.0 && m[1].x == 0.0 && m[1].y == 0.0 && m[2].x == 0.0 && m[2].y == 0.0 &&
           m[3].x == 1.0 && m[3].y == 0.0;
}

// 0: neither, 1: H, 2: H with its columns exchanged (an X before it)
int hadamard(const double2 *m)
{
    for (int i = 0; i < 4; ++i)
        if (m[i].y != 0.0 || std::fabs(m[i].x) != kRsqrt2)
            return 0;
    if (m[0].x < 0.0 || m[1].x < 0.0 || (m[2].x < 0.0) == (m[3].x < 0.0))
        return 0;
    return m[3].x < 0.0 ? 1 : 2;
}

double2 cmul_host(double2 x, double2 y) { return make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x); }

} // namespace

bool make_butterfly_params(const FPassParams &prm, int amp_bytes, BPassParams &bp)
{
    if (prm.k != kTensorLocal || prm.from_zero || prm.nstages <= 0 || prm.nstages > kButterflyStages)
        return false;
    std::memset(&bp, 0, sizeof(bp));
    bp.chunks = prm.chunks;
    std::memcpy(bp.qmasks, prm.qmasks, sizeof(bp.qmasks));
    std::memcpy(bp.qbit, prm.qbit, sizeof(bp.qbit));
    bp.nstages = prm.nstages;
    int entries = 0, hs = 0;
    for (int s = 0; s < prm.nstages; ++s)
    {
        const FStage &FS = prm.stages[s];
        BStage &S = bp.stages[s];
        std::memcpy(S.sbits, FS.sbits, sizeof(S.sbits));
        double2 f[kStageBits + 1][16];
        bool has[kStageBits + 1] = {};
        auto factor = [&](int step, int r, double2 v) {
            if (!has[step])
                for (int i = 0; i < 16; ++i)
                    f[step][i] = make_double2(1.0, 0.0);
            has[step] = true;
            f[step][r] = cmul_host(v, f[step][r]);
        };
        auto add_h = [&](int b, int form) {
            S.steps[b].h = 1;
            ++hs;
            if (form == 2)
                for (int r = 0; r < 16; ++r)
                    if ((r >> b) & 1)
                        factor(b, r, make_double2(-1.0, 0.0));
        };
        int at = kStageBits;   // the step being filled: bits come highest first
        for (int oi = FS.op_begin; oi < FS.op_end; ++oi)
        {
            const FOp &op = prm.ops[oi];
            const double2 *m = prm.entries + op.moff;
            if (op.kind == F_PRUN)
            {
                BStep &step = S.steps[at];
                if (op.lcmask != 0)
                    return false;   // explicit terms
                if (op.b1)
                    for (int r = 0; r < 16; ++r)
                        factor(at, r, m[r]);
                if (op.b0)
                {
                    if (step.run.used)
                        return false;
                    // the tables as an F_PRUN stores them: the thread tables,
                    // then each chunk group's, factors ascending
                    BRun &run = step.run;
                    run.packed = op.gcmask;
                    run.used = op.b0;
                    uint32_t off = op.lcval;
                    for (int e = 0; e <= kStageBits; ++e)
                        if ((run.packed >> e) & 1)
                        {
                            run.thread_table[e] = off;
                            off += kThreads;
                        }
                    for (int g = 0; g < kMaxChunkGroups; ++g)
                        for (int e = 0; e <= kStageBits; ++e)
                            if ((run.packed >> (kChunkGroupBits * (g + 1) + e)) & 1)
                            {
                                run.group_table[g][e] = off;
                                off += 1u << kChunkGroupBits;
                                run.groups = g + 1;
                            }
                }
                continue;
            }
            if (op.lcmask != 0 || op.gcmask != 0)
                return false;
            if (op.kind == F_PHASE || op.kind == F_MULI)
            {
                const double2 e = op.kind == F_PHASE ? m[0] : make_double2(0.0, op.b1 ? -1.0 : 1.0);
                for (int r = 0; r < 16; ++r)
                    if ((r & op.smask) == op.sval)
                        factor(at, r, e);
                continue;
            }
            if (op.kind == F_DENSE1R && op.smask == 0)
            {
                const int form = hadamard(m);
                if (form == 0 || op.b0 >= at)
                    return false;
                at = op.b0;
                add_h(at, form);
                continue;
            }
            if (op.kind == F_DENSE1RX4 && at == kStageBits)
            {
                for (int b = kStageBits - 1; b >= 0; --b)
                {
                    if (identity2(m + 4 * b))
                        continue;
                    const int form = hadamard(m + 4 * b);
                    if (form == 0)
                        return false;
                    at = b;
                    add_h(b, form);
                }
                continue;
            }
            return false;
        }
        for (int step = 0; step <= kStageBits; ++step)
        {
            if (!has[step])
                continue;
            bool half = step < kStageBits;
            for (int r = 0; r < 16 && half; ++r)
                half = ((r >> step) & 1) || (f[step][r].x == 1.0 && f[step][r].y == 0.0);
            if (entries + (half ? 8 : 16) > kButterflyEntries)
                return false;
            S.steps[step].factors = half ? 1 : 2;
            S.steps[step].entry = static_cast<uint16_t>(entries);
            for (int r = 0; r < 16; ++r)
                if (!half || ((r >> step) & 1))
                    bp.entries[entries++] = f[step][r];
        }
    }
    if (hs == 0)
        return false;
    bp.scale = std::ldexp(hs % 2 ? kRsqrt2 : 1.0, -(hs / 2));
    auto low_free = [](const BStage &S) {
        return S.sbits[0] >= kLowBits && S.sbits[1] >= kLowBits && S.sbits[2] >= kLowBits && S.sbits[3] >= kLowBits;
    };
    bp.direct_in = low_free(bp.stages[0]);
    bp.direct_out = low_free(bp.stages[bp.nstages - 1]);
    if (amp_bytes == (int)sizeof(float2))
        entries_to_float(bp.entries, entries);
    return true;
}

bool is_hadamard(const GateOp &op)
{
    if (op.diag || op.nt != 1 || op.na != 2 || op.cmask != 0)
        return false;
    double2 m[4];
    for (int i = 0; i < 4; ++i)
        m[i] = make_double2(op.mat[i].re, op.mat[i].im);
    return hadamard(m) != 0;
}

// Fitted on B200 to 48 passes at 25 and 27 qubits: H layers alone 5.9-7.2 ps
// per amplitude, the passes of a QFT 8.7-11.2 (as interpreted register passes
// they are priced at 14.7-18.4); rms difference 0.5.
double butterfly_pass_cost(const BPassParams &bp)
{
    double ps = 4.9 + 0.7 * bp.nstages;
    for (int s = 0; s < bp.nstages; ++s)
        for (const BStep &step : bp.stages[s].steps)
            ps += (step.factors ? 0.25 : 0.0) + 0.22 * __builtin_popcount(step.run.used);
    return ps;
}

template <typename R>
int launch_butterfly_pass(const BPassParams &bp, cudaStream_t stream)
{
    const size_t smem = sizeof(typename Cx<R>::T) << kTensorLocal;
    int dev = 0, sms = 0, per_sm = 0;
    QCSB_CUDA(cudaGetDevice(&dev));
    QCSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    QCSB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, butterfly_pass_kernel<R>, kThreads, smem));
    const uint64_t cap = static_cast<uint64_t>(sms) * (per_sm > 0 ? per_sm : 1);
    const uint64_t grid = bp.chunks < cap ? bp.chunks : cap;
    butterfly_pass_kernel<R><<<static_cast<unsigned>(grid), kThreads, smem, stream>>>(bp);
    QCSB_CUDA(cudaGetLastError());
    return 1;
}
template int launch_butterfly_pass<double>(const BPassParams &, cudaStream_t);
template int launch_butterfly_pass<float>(const BPassParams &, cudaStream_t);

} // namespace qcsb

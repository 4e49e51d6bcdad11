// tile_dev.cuh -- device side of the tile-program interpreter, shared by the
// per-pass kernel (tile.cu) and the batched persistent kernel (batch.cu).
//
// A thread holds R = 2^RB amplitudes of each of NS states in registers: the RB
// "register" tile bits of the current layout select the register, the other
// tile bits are the thread index.  run_ops() executes one pass program (the
// KOp list of planner.h) on them; K_TRANSPOSE exchanges the tile through
// shared memory with an XOR-swizzled slot map.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "planner.h"

namespace qse {
namespace tile {
namespace dev {

using plan::KOp;

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// Im(conj(l) * s)
__device__ __forceinline__ double im_ls(double2 l, double2 s) { return l.x * s.y - l.y * s.x; }

template <int R, int P, class F>
__device__ __forceinline__ void pairs_at(double2 (&a)[R], F& f)
{
#pragma unroll
    for (int j = 0; j < R; ++j)
        if (!(j & (1 << P))) f(a[j], a[j | (1 << P)], j);
}

template <int RB, class F>
__device__ __forceinline__ void pairs(int p, double2 (&a)[1 << RB], F& f)
{
    constexpr int R = 1 << RB;
    switch (p) {
    case 0: pairs_at<R, 0>(a, f); break;
    case 1: pairs_at<R, 1>(a, f); break;
    case 2: pairs_at<R, 2>(a, f); break;
    default:
        if constexpr (RB > 3) pairs_at<R, 3>(a, f);
        break;
    }
}

template <int R, int P, class F>
__device__ __forceinline__ void pairs2_at(const double2 (&s)[R], const double2 (&l)[R], F& f)
{
#pragma unroll
    for (int j = 0; j < R; ++j)
        if (!(j & (1 << P))) f(s[j], s[j | (1 << P)], l[j], l[j | (1 << P)]);
}

template <int RB, class F>
__device__ __forceinline__ void pairs2(int p, const double2 (&s)[1 << RB], const double2 (&l)[1 << RB], F& f)
{
    constexpr int R = 1 << RB;
    switch (p) {
    case 0: pairs2_at<R, 0>(s, l, f); break;
    case 1: pairs2_at<R, 1>(s, l, f); break;
    case 2: pairs2_at<R, 2>(s, l, f); break;
    default:
        if constexpr (RB > 3) pairs2_at<R, 3>(s, l, f);
        break;
    }
}

struct OpH {
    __device__ void operator()(double2& v0, double2& v1, int) const
    {
        double2 a = v0, b = v1;
        v0 = make_double2(a.x + b.x, a.y + b.y);
        v1 = make_double2(a.x - b.x, a.y - b.y);
    }
};
struct OpX {
    int f;
    __device__ void operator()(double2& v0, double2& v1, int j) const
    {
        if ((j & f) == f) { double2 t = v0; v0 = v1; v1 = t; }
    }
};
struct OpY {
    int f;
    __device__ void operator()(double2& v0, double2& v1, int j) const
    {
        if ((j & f) == f) {
            double2 a = v0, b = v1;
            v0 = make_double2(b.y, -b.x);
            v1 = make_double2(-a.y, a.x);
        }
    }
};
struct OpRX {
    double c, s;
    __device__ void operator()(double2& v0, double2& v1, int) const
    {
        double2 a = v0, b = v1;
        v0 = make_double2(c * a.x + s * b.y, c * a.y - s * b.x);
        v1 = make_double2(s * a.y + c * b.x, c * b.y - s * a.x);
    }
};
struct OpRY {
    double c, s;
    __device__ void operator()(double2& v0, double2& v1, int) const
    {
        double2 a = v0, b = v1;
        v0 = make_double2(c * a.x - s * b.x, c * a.y - s * b.y);
        v1 = make_double2(s * a.x + c * b.x, s * a.y + c * b.y);
    }
};
struct OpU {
    double2 g00, g01, g10, g11;
    int f;
    __device__ void operator()(double2& v0, double2& v1, int j) const
    {
        if ((j & f) == f) {
            double2 a = v0, b = v1;
            double2 x = cmul(g00, a), y = cmul(g01, b), z = cmul(g10, a), w = cmul(g11, b);
            v0 = make_double2(x.x + y.x, x.y + y.y);
            v1 = make_double2(z.x + w.x, z.y + w.y);
        }
    }
};
// multiply the bit-p-set half by e
struct OpPhase1 {
    double2 e;
    __device__ void operator()(double2&, double2& v1, int) const { v1 = cmul(v1, e); }
};

template <int R, int F>
__device__ __forceinline__ void phase_pattern(double2 (&a)[R], double2 e)
{
#pragma unroll
    for (int j = 0; j < R; ++j)
        if ((j & F) == F) a[j] = cmul(a[j], e);
}

template <int RB>
__device__ __forceinline__ void phase_masked(int f, double2 (&a)[1 << RB], double2 e)
{
    constexpr int R = 1 << RB;
    switch (f) {
    case 1: phase_pattern<R, 1>(a, e); break;
    case 2: phase_pattern<R, 2>(a, e); break;
    case 4: phase_pattern<R, 4>(a, e); break;
    case 3: phase_pattern<R, 3>(a, e); break;
    case 5: phase_pattern<R, 5>(a, e); break;
    case 6: phase_pattern<R, 6>(a, e); break;
    case 7: phase_pattern<R, 7>(a, e); break;
    default:
        if constexpr (RB > 3) {
            switch (f) {
            case 8: phase_pattern<R, 8>(a, e); break;
            case 9: phase_pattern<R, 9>(a, e); break;
            case 10: phase_pattern<R, 10>(a, e); break;
            case 11: phase_pattern<R, 11>(a, e); break;
            case 12: phase_pattern<R, 12>(a, e); break;
            case 13: phase_pattern<R, 13>(a, e); break;
            case 14: phase_pattern<R, 14>(a, e); break;
            case 15: phase_pattern<R, 15>(a, e); break;
            default:
#pragma unroll
                for (int j = 0; j < R; ++j)
                    if ((j & f) == f) a[j] = cmul(a[j], e);
            }
        } else {
#pragma unroll
            for (int j = 0; j < R; ++j)
                if ((j & f) == f) a[j] = cmul(a[j], e);
        }
    }
}

// sum over the lanes of a warp; blocks smaller than a warp (tiny states) use
// only their own lanes in the mask and only partner offsets inside the block
__device__ __forceinline__ double warp_sum(double v)
{
    const uint32_t nb = blockDim.x;
    const unsigned mask = nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        if (uint32_t(o) < nb) v += __shfl_xor_sync(mask, v, o);
    return v;
}

// XOR of the 16-bit images img[t] over the set bits t < kThrBits of tid, two
// per word (img 16-byte aligned).
__device__ __forceinline__ uint32_t slot_of(const uint16_t* img, uint32_t tid)
{
    const uint4 w = *reinterpret_cast<const uint4*>(img);
    const uint32_t v[5] = {w.x, w.y, w.z, w.w, *reinterpret_cast<const uint32_t*>(img + 8)};
    static_assert(plan::kThrBits == 10, "five words of two images");
    uint32_t s = 0;
#pragma unroll
    for (int p = 0; p < 5; ++p)
        s ^= v[p] & (((tid >> (2 * p)) & 1u) * 0xffffu | ((tid >> (2 * p + 1)) & 1u) * 0xffff0000u);
    return (s ^ (s >> 16)) & 0xffffu;
}

// index of register 0 of thread tid in layout r: the outer bits and its thread bits
template <class I>
__device__ __forceinline__ I thread_base(const plan::LayoutRec* r, I obase, uint32_t tid)
{
    I g = obase;
#pragma unroll
    for (uint32_t t = 0; t < plan::kThrBits; ++t) g |= I((tid >> t) & 1u) << r->pthr[t];
    return g;
}

template <int RB, class I>
__device__ __forceinline__ I reg_index(I base, const I (&rg)[RB], int j)
{
#pragma unroll
    for (int i = 0; i < RB; ++i)
        if ((j >> i) & 1) base |= rg[i];
    return base;
}

template <int RB>
__device__ __forceinline__ uint32_t sidx(uint32_t sb, const uint32_t (&sreg)[RB], int j)
{
    uint32_t s = sb;
#pragma unroll
    for (int i = 0; i < RB; ++i)
        if ((j >> i) & 1) s ^= sreg[i];
    return s;
}

__device__ __forceinline__ bool is_one(double2 e) { return e.x == 1.0 && e.y == 0.0; }

// acc: the thread's accumulated phase of register bit p (shared memory)
template <int RB, int NS>
__device__ __forceinline__ void flush_reg(int p, double2* acc, double2 (&a)[NS][1 << RB], int nact)
{
    const double2 v = *acc;
    if (!is_one(v)) {
        *acc = make_double2(1.0, 0.0);
        OpPhase1 ph{v};
#pragma unroll
        for (int st = 0; st < NS; ++st)
            if (st < nact) pairs<RB>(p, a[st], ph);
    }
}

// Outer bits of tile `c` (the bits of c spread over the set bits of outer_mask).
__device__ __forceinline__ uint64_t tile_base(uint64_t c, uint64_t outer_mask)
{
    uint64_t obase = 0, m = outer_mask;
    while (m && c) {
        uint32_t b = __ffsll((long long)m) - 1;
        m &= m - 1;
        if (c & 1) obase |= uint64_t(1) << b;
        c >>= 1;
    }
    return obase;
}

// Per-CTA value of every diagonal group of a pass: (cos, sin) of the sum of the
// angles of its terms whose outer condition holds for this tile, in term order.
__device__ __forceinline__ void group_values(const plan::GroupRec* __restrict__ groups, uint32_t ngroups,
                                             const plan::TermRec* __restrict__ terms, uint64_t obase, double2* gval)
{
    for (uint32_t g = threadIdx.x; g < ngroups; g += blockDim.x) {
        const plan::GroupRec gr = groups[g];
        double th = 0.0;
        for (uint32_t i = 0; i < gr.count; ++i) {
            const plan::TermRec t = terms[gr.first + i];
            if ((obase & t.ocond) == t.ocond) th += t.theta;
        }
        double s, c;
        sincos(th, &s, &c);
        gval[g] = make_double2(c, s);
    }
}

// Everything run_ops needs besides the registers.
struct OpsEnv {
    const KOp* ops;
    uint32_t nops;
    const plan::LayoutRec* layouts;   // layout indices of the program are relative to this
    const double* mats;               // K_U matrix indices are relative to this
    uint64_t obase;
    double2* xbuf;                    // 2^k slots
    const double2* gval;              // group values of this CTA: unit phases
    double* wpart;                    // gradient partials (NS == 2), wpart_stride(nwarps, WL) per slot
    uint32_t nwarps;
    double2* acc;                     // phase accumulators of register bit p at acc[p * acc_stride] (1 on entry and exit)
    uint32_t acc_stride;
};

// Gradient partials of a slot: WL (8 or 1) per warp (add_partial), and, with 8, a
// double of padding so that the threads that sum a slot each (slot_sum) hit distinct
// banks.  The launch takes 8 where they leave room for its CTAs in shared memory, else
// 1; a compile-time choice, since a runtime one costs the batched kernel 2 %.
__host__ __device__ constexpr uint32_t wpart_stride(uint32_t nwarps, uint32_t wl)
{
    return wl * nwarps + (wl > 1 ? 1 : 0);
}

// Adds a gate's per-thread sums to its slot: with WL 8, two exchange steps leave
// eight sums a warp, and the rest waits for the end of the tile, where all slots are
// summed at once (five dependent steps per gate were a tenth of a reverse tile's
// latency).
template <uint32_t WL>
__device__ __forceinline__ void add_partial(double v, double* slot)
{
    const uint32_t nb = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    const unsigned mask = nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u);
#pragma unroll
    for (uint32_t o = 16; o >= WL; o >>= 1)
        if (o < nb) v += __shfl_xor_sync(mask, v, o);
    if (lane < WL) slot[(tid >> 5) * WL + lane] += v;
}
template <uint32_t WL>
__device__ __forceinline__ double slot_sum(const double* slot, uint32_t nwarps)
{
    double v = 0.0;
    for (uint32_t i = 0; i < WL * nwarps; ++i) v += slot[i];
    return v;
}

// A program record as two 16-byte words, its fields taken out where they are used
// (loaded field by field, a record is eight loads).
struct OpWords {
    uint4 h, v;
    __device__ __forceinline__ void load(const KOp* op)
    {
        const uint4* p = reinterpret_cast<const uint4*>(op);
        h = __ldg(p);
        v = __ldg(p + 1);
    }
    __device__ __forceinline__ uint32_t kind() const { return h.x & 0xffu; }
    __device__ __forceinline__ int p() const { return int((h.x >> 8) & 0xffu); }
    __device__ __forceinline__ int f() const { return int(h.x >> 24); }
    __device__ __forceinline__ uint32_t tcond() const { return h.y & 0xffffu; }
    __device__ __forceinline__ uint32_t g() const { return h.y >> 16; }
    __device__ __forceinline__ uint64_t ocond() const { return uint64_t(h.z) | uint64_t(h.w) << 32; }
    __device__ __forceinline__ double a() const { return __hiloint2double(int(v.y), int(v.x)); }
    __device__ __forceinline__ double b() const { return __hiloint2double(int(v.w), int(v.z)); }
};
static_assert(offsetof(KOp, kind) == 0 && offsetof(KOp, p) == 1 && offsetof(KOp, f) == 3 && offsetof(KOp, tcond) == 4 &&
                  offsetof(KOp, g) == 6 && offsetof(KOp, ocond) == 8 && offsetof(KOp, a) == 16 && alignof(KOp) == 16,
              "OpWords reads KOp");

// Executes a pass program on the registers a[NS][R], which hold layout `lay` and
// leave in the layout returned.  nact states take part
// (1: only |psi>, forward; NS: the adjoint sweep on |psi> and |lambda>).
// Threads with active == false hold zeros, never touch the exchange buffer
// and add nothing to the gradient partials; they only join the barriers
// (a CTA wider than the tile of a small state).
template <int RB, int NS, uint32_t WL>
__device__ __forceinline__ const plan::LayoutRec* run_ops(const OpsEnv& E, const plan::LayoutRec* lay,
                                                         double2 (&a)[NS][1 << RB], int nact, bool active)
{
    constexpr int R = 1 << RB;
    const uint32_t tid = threadIdx.x;
    double2 acc_thr = make_double2(1.0, 0.0);
    double2* const acc = E.acc;

    OpWords nxt;
    if (E.nops) nxt.load(E.ops);
    for (uint32_t i = 0; i < E.nops; ++i) {
        const OpWords op = nxt;
        nxt.load(E.ops + min(i + 1, E.nops - 1));  // in flight while this op executes
        const bool tc = (tid & op.tcond()) == op.tcond();
        switch (op.kind()) {
        case plan::K_H: {
            OpH f;
#pragma unroll
            for (int st = 0; st < NS; ++st)
                if (st < nact) pairs<RB>(op.p(), a[st], f);
            break;
        }
        case plan::K_X: {
            if (tc && (E.obase & op.ocond()) == op.ocond()) {
                OpX f{op.f()};
#pragma unroll
                for (int st = 0; st < NS; ++st)
                    if (st < nact) pairs<RB>(op.p(), a[st], f);
            }
            break;
        }
        case plan::K_Y: {
            if (tc && (E.obase & op.ocond()) == op.ocond()) {
                OpY f{op.f()};
#pragma unroll
                for (int st = 0; st < NS; ++st)
                    if (st < nact) pairs<RB>(op.p(), a[st], f);
            }
            break;
        }
        case plan::K_RX: {
            OpRX f{op.a(), op.b()};
#pragma unroll
            for (int st = 0; st < NS; ++st)
                if (st < nact) pairs<RB>(op.p(), a[st], f);
            break;
        }
        case plan::K_RY: {
            OpRY f{op.a(), op.b()};
#pragma unroll
            for (int st = 0; st < NS; ++st)
                if (st < nact) pairs<RB>(op.p(), a[st], f);
            break;
        }
        case plan::K_U: {
            if (tc && (E.obase & op.ocond()) == op.ocond()) {
                const double* m = E.mats + 8 * op.g();
                OpU f{make_double2(m[0], m[1]), make_double2(m[2], m[3]), make_double2(m[4], m[5]),
                      make_double2(m[6], m[7]), op.f()};
#pragma unroll
                for (int st = 0; st < NS; ++st)
                    if (st < nact) pairs<RB>(op.p(), a[st], f);
            }
            break;
        }
        case plan::K_ACC_THR:
            if (tc) acc_thr = cmul(acc_thr, E.gval[op.g()]);
            break;
        case plan::K_ACC_REG: {
            if (tc) acc[op.p() * E.acc_stride] = cmul(acc[op.p() * E.acc_stride], E.gval[op.g()]);
            break;
        }
        case plan::K_PHD: {
            if (tc) {
                double2 e = E.gval[op.g()];
#pragma unroll
                for (int st = 0; st < NS; ++st)
                    if (st < nact) phase_masked<RB>(op.f(), a[st], e);
            }
            break;
        }
        case plan::K_FLUSH_REG:
            flush_reg<RB, NS>(op.p(), acc + op.p() * E.acc_stride, a, nact);
            break;
        case plan::K_FLUSH_ALL: {
#pragma unroll
            for (int r = 0; r < RB; ++r)
                if ((op.f() >> r) & 1) flush_reg<RB, NS>(r, acc + r * E.acc_stride, a, nact);
            const double2 e = cmul(make_double2(op.a(), op.b()), acc_thr);
            acc_thr = make_double2(1.0, 0.0);
            if (!is_one(e)) {
#pragma unroll
                for (int st = 0; st < NS; ++st)
                    if (st < nact)
#pragma unroll
                        for (int j = 0; j < R; ++j) a[st][j] = cmul(a[st][j], e);
            }
            break;
        }
        case plan::K_TRANSPOSE: {
            lay = E.layouts + op.g();
            const uint32_t sbw = slot_of(lay->wthr, tid), sbr = slot_of(lay->rthr, tid);
            uint32_t sreg_w[RB], sreg_r[RB];
#pragma unroll
            for (int i = 0; i < RB; ++i) {
                sreg_w[i] = lay->wreg[i];
                sreg_r[i] = lay->rreg[i];
            }
#pragma unroll
            for (int st = 0; st < NS; ++st) {
                if (st < nact) {
                    __syncthreads();
                    if (active)
#pragma unroll
                        for (int j = 0; j < R; ++j) E.xbuf[sidx<RB>(sbw, sreg_w, j)] = a[st][j];
                    __syncthreads();
                    if (active)
#pragma unroll
                        for (int j = 0; j < R; ++j) a[st][j] = E.xbuf[sidx<RB>(sbr, sreg_r, j)];
                }
            }
            break;
        }
        case plan::K_GRAD_X:
        case plan::K_GRAD_Y:
        case plan::K_GRAD_Z:
        case plan::K_GRAD_P: {
            if constexpr (NS == 2) {
                // each a branch of its own with four chains of FMAs: a kind or a
                // register sign decided per amplitude took three times the
                // instructions of the sums
                double part = 0.0, c0 = 0.0, c1 = 0.0, c2 = 0.0, c3 = 0.0;
                if (op.kind() == plan::K_GRAD_X) {
                    auto f = [&](const double2& s0, const double2& s1, const double2& l0, const double2& l1) {
                        c0 = fma(l0.x, s1.y, c0);
                        c1 = fma(-l0.y, s1.x, c1);
                        c2 = fma(l1.x, s0.y, c2);
                        c3 = fma(-l1.y, s0.x, c3);
                    };
                    pairs2<RB>(op.p(), a[0], a[NS - 1], f);
                    part = (c0 + c1) + (c2 + c3);
                } else if (op.kind() == plan::K_GRAD_Y) {
                    auto f = [&](const double2& s0, const double2& s1, const double2& l0, const double2& l1) {
                        c0 = fma(l1.x, s0.x, c0);
                        c1 = fma(l1.y, s0.y, c1);
                        c2 = fma(-l0.x, s1.x, c2);
                        c3 = fma(-l0.y, s1.y, c3);
                    };
                    pairs2<RB>(op.p(), a[0], a[NS - 1], f);
                    part = (c0 + c1) + (c2 + c3);
                } else if (op.kind() == plan::K_GRAD_Z) {
                    const bool reg = op.p() < RB;   // else the sign is the thread's or the CTA's
                    auto f = [&](const double2& s0, const double2& s1, const double2& l0, const double2& l1) {
                        c0 = fma(l0.x, s0.y, c0);
                        c1 = fma(-l0.y, s0.x, c1);
                        c2 = fma(l1.x, s1.y, c2);
                        c3 = fma(-l1.y, s1.x, c3);
                    };
                    pairs2<RB>(reg ? op.p() : 0, a[0], a[NS - 1], f);
                    part = reg ? (c0 + c1) - (c2 + c3) : (c0 + c1) + (c2 + c3);
                    if (((tid & op.tcond()) != 0) != ((E.obase & op.ocond()) != 0)) part = -part;
                } else {
                    if (tc && (E.obase & op.ocond()) == op.ocond()) {
#pragma unroll
                        for (int j = 0; j < R; ++j)
                            if ((j & op.f()) == op.f()) part += im_ls(a[1][j], a[0][j]);
                    }
                }
                add_partial<WL>(part * op.a(), E.wpart + op.g() * wpart_stride(E.nwarps, WL));
            }
            break;
        }
        default:
            break;
        }
    }
    return lay;
}

}  // namespace dev
}  // namespace tile
}  // namespace qse

// CTA-level negacyclic NTT of length 4096 on one residue channel, operating on
// a shared-memory array, so every kernel fuses its transforms with their
// producers and consumers.
//
// Order and root follow HEXL as the reference uses it: the forward transform
// maps natural order to bit-reversed order, slot j holding
// sum_k x_k psi^((2 bitrev(j) + 1) k)  (reference utils.cpp:1473-1478), and the
// inverse includes N^-1.
//
// What bounds a transform on this chip, and what follows from it (measured
// per SM sub-partition: mad.lo issues every 2 cycles, mul.hi and mad.wide every 4,
// additions every cycle):
//
// * The multiply pipe: a butterfly's modular product is a mul.hi and two
//   mad.lo, 8 cycles.
// * Instruction issue.  Words are signed and twiddles centred in (-q/2, q/2):
//   a product lands within (-0.25, 1.25) q and a layer widens the range by
//   little more than q, so words stay below 8 q < 2^31 (q < 2^28) for four layers
//   at a time with one fold of the eight summands per pass in between,
//   instead of a conditional subtraction per butterfly.  A butterfly is four
//   instructions: the quotient, x + y w, its multiple, and 2x - (x + t).
// * Shared-memory wavefronts and barriers.  256 threads hold one radix-16 unit
//   each (16 elements, four butterfly layers): three passes and four
//   barriers per transform, one shared-memory round trip per four layers.  The first pass takes its
//   15 twiddles (the same for every thread) from constant memory; the others
//   read them as eight 16-byte vectors per unit through L1 (twiddle_table).
//
// The inverse decimates in time as well: its input is in bit-reversed order,
// which is what a cyclic decimation-in-time transform starts from (a
// decimation in frequency doubles its sums with every layer and would pay
// reductions).  Its first and last passes are plain 16-point transforms whose
// twiddles every thread shares; the last one first multiplies its inputs by the
// thread's sixteen twiddles with psi^-u N^-1 in them (u the thread), and its
// outputs u + 256 t by psi^-256 t, so that the negacyclic twist needs no table of its
// own.
//
// 4096-point forward and inverse transforms of a batch of 64 (r = 16), giant
// steps included: see the figures at k_giant_fused and k_baby.cuh.
//
// Shared-memory layout.  A polynomial occupies kPadN words: coefficient (or
// slot) i sits at pidx(i) = i + 4 (i / 32) + 16 (i / 256).  With that padding
// every pass (strides 256 and 16 words, then sixteen contiguous words as four
// 16-byte vectors) hits 32 distinct banks per warp access, and the position of
// element t of a thread's unit is the unit's base plus a compile-time offset.
//
// Device table of a channel: uint2 {w, round(w 2^32 / q)}, w centred, signed:
//   forward  [unit pass 1: 8 x 16 uint4][unit pass 2: 8 x 256 uint4]
//   inverse  [pass 1: 8 x 16 uint4][pass 2: 8 x 256 uint4]
// vector v of a unit holds entries 2v and 2v + 1 of its sixteen: (unused, one
// twiddle of the first layer), two of the second, four of the third, eight of
// the fourth; in the inverse's pass 2 entry t belongs to input t.  The host
// builds it (build_twiddles in kspir.cu).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace kspir {

constexpr int kNttThreads = 512;        // threads of a kernel that runs transforms: two groups
constexpr int kNttGroup = 256;          // threads of one transform
constexpr int kPadN = kN + kN / 8 + kN / 16;   // padded length of a polynomial in shared memory
constexpr int kPadStep = 608;           // pidx(i + 512) - pidx(i), i < 512
constexpr int kPadGroupStep = 304;      // pidx(i + 256) - pidx(i), i < 256

__host__ __device__ __forceinline__ int pidx(int i) { return i + ((i >> 5) << 2) + ((i >> 8) << 4); }

// device table of a channel, in uint2 entries
constexpr int kTwPass1 = 16 * 16;             // entries of pass 1 (16 units of 16)
constexpr int kTwPass2 = 256 * 16;
constexpr int kTwFwd = kTwPass1 + kTwPass2;
constexpr int kTwChannel = 2 * kTwFwd;

struct NttTables {
    const uint2* tw[CH_COUNT];   // [kTwChannel] per channel
};

// Barrier of the threads that run a transform.  A stand-alone kernel
// synchronises its whole CTA; the fused answer kernel (k_answer.cuh) runs its
// transforms in a 512-thread warp group beside the scan warps and uses a named
// barrier (KsSync there).
struct CtaSync {
    __device__ __forceinline__ static void sync() { __syncthreads(); }
};

// Lane order: coefficient k = u + 256 (4 v + w) of a polynomial read by 256
// threads u sits at 4 (256 v + u) + w, so that a thread's sixteen coefficients
// u + 256 t arrive as four coalesced 16-byte vectors while scalar accesses of
// the same coefficients stay coalesced too.  The resident keys and slot
// permutations are kept in it.
__host__ __device__ __forceinline__ int lane_pos(int k) { return ((((k >> 10) << 8) + (k & 255)) << 2) + ((k >> 8) & 3); }

// the 256-thread group of this thread (0 or 1), as a value the compiler knows to
// be the same for the whole warp: constants indexed by it stay uniform loads
__device__ __forceinline__ int thread_group() { return __shfl_sync(0xffffffffu, (int)threadIdx.x / kNttGroup, 0); }

// The barrier of one 256-thread group (named barriers 2 and 3): the groups of a
// CTA work on different polynomials between the points where they exchange
// them, and drift apart, so that one's butterflies cover the other's loads.
struct GroupSync {
    __device__ __forceinline__ static void sync() {
        asm volatile("bar.sync %0, 256;" ::"r"(2 + (int)threadIdx.x / kNttGroup) : "memory");
    }
};

enum NttDir : int { NTT_FWD = 0, NTT_INV = 1 };

// The device table of (ch, dir), read through L1.
__device__ __forceinline__ const uint4* twiddle_table(const NttTables& tabs, int ch, int dir) {
    // a select chain, not tabs.tw[ch]: a run-time index into a kernel
    // parameter array makes the compiler copy the array to local memory
    const uint2* t = ch == 0 ? tabs.tw[0] : ch == 1 ? tabs.tw[1] : ch == 2 ? tabs.tw[2] : ch == 3 ? tabs.tw[3]
                   : ch == 4 ? tabs.tw[4] : ch == 5 ? tabs.tw[5] : tabs.tw[6];
    return reinterpret_cast<const uint4*>(t + (dir ? kTwFwd : 0));
}

// Brings a table's lines into L1 ahead of the transform (a kernel with one CTA
// per SM would otherwise wait for L2 in every pass).
__device__ __forceinline__ void warm_twiddles(const NttTables& tabs, int ch, int dir, int tid, int threads) {
    const char* t = reinterpret_cast<const char*>(twiddle_table(tabs, ch, dir));
    constexpr int lines = kTwFwd * 8 / 128;
    for (int i = tid; i < lines; i += threads) asm volatile("prefetch.global.L1 [%0];" ::"l"(t + (size_t)i * 128));
}

// offset of element t of a radix-16 unit from its base, pass P (strides 256, 16, 1)
template <int P>
__device__ __forceinline__ constexpr int unit_off(int t) {
    return P == 0 ? 304 * t : P == 1 ? 16 * t + 4 * (t >> 1) : t;
}

// base of thread u's unit in pass P
template <int P>
__device__ __forceinline__ int unit_base(int u) {
    return P == 0 ? pidx(u) : P == 1 ? 304 * (u >> 4) + (u & 15) : pidx(16 * u);
}

template <int P>
__device__ __forceinline__ void unit_load(const uint32_t* s, uint32_t* x) {
    if (P == 2) {
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const uint4 a = *reinterpret_cast<const uint4*>(s + 4 * v);
            x[4 * v] = a.x; x[4 * v + 1] = a.y; x[4 * v + 2] = a.z; x[4 * v + 3] = a.w;
        }
    } else {
#pragma unroll
        for (int t = 0; t < 16; t++) x[t] = s[unit_off<P>(t)];
    }
}

template <int P>
__device__ __forceinline__ void unit_store(uint32_t* s, const uint32_t* x) {
    if (P == 2) {
#pragma unroll
        for (int v = 0; v < 4; v++)
            *reinterpret_cast<uint4*>(s + 4 * v) = make_uint4(x[4 * v], x[4 * v + 1], x[4 * v + 2], x[4 * v + 3]);
    } else {
#pragma unroll
        for (int t = 0; t < 16; t++) s[unit_off<P>(t)] = x[t];
    }
}

// the sixteen entries of unit i of a pass with `units` units (entry 0 unused)
__device__ __forceinline__ void unit_twiddles(const uint4* __restrict__ tab, int units, int i, uint2* w) {
#pragma unroll
    for (int v = 0; v < 8; v++) {
        const uint4 a = __ldg(tab + v * units + i);
        w[2 * v] = make_uint2(a.x, a.y);
        w[2 * v + 1] = make_uint2(a.z, a.w);
    }
}

// four decimation-in-time layers of one unit: FWD pairs the largest distance
// first (natural to bit-reversed order), otherwise the smallest first
// (bit-reversed to natural); w[1], w[2..3], w[4..7], w[8..15] are the twiddles
// of the four layers in that order.
template <bool FWD>
__device__ __forceinline__ void unit_layers(uint32_t* x, const uint2* w, uint32_t nq) {
#pragma unroll
    for (int l = 0; l < 4; l++) {
        const int d = FWD ? 8 >> l : 1 << l;
#pragma unroll
        for (int t = 0; t < 16; t++) {
            if (t & d) continue;
            // FWD: one twiddle per block of the layer; else per position in a block
            const int k = FWD ? t / (2 * d) : t & (d - 1);
            bfly(x[t], x[t + d], w[(1 << l) + k], nq);
        }
    }
}

// Plain 16-point transform from bit-reversed to natural order (twiddles: powers
// of the 16th root).  FIRST: the inverse's first pass, inputs in [0, q); places 0
// and 8 reach 8 q (no twiddle intervened) and are folded to +-4 q, the others
// stay below 5.2 q.  Otherwise inputs in (-0.25, 1.25) q (just multiplied), and
// the sums without twiddles are folded before the last layer; all below 6.1 q.
template <bool FIRST>
__device__ __forceinline__ void unit_dft16(uint32_t* x, const ChanConst& cc) {
    const uint32_t q = cc.q, nq = cc.nq;
#pragma unroll
    for (int t = 0; t < 16; t += 2) {
        const uint32_t X = x[t], Y = x[t + 1];
        x[t] = X + Y - q;   // centred sum
        x[t + 1] = X - Y;
    }
#pragma unroll
    for (int l = 1; l < 4; l++) {
        const int d = 1 << l;
        if (l == 3 && !FIRST) {
#pragma unroll
            for (int t = 0; t < 16; t += 4) x[t] = fold6(x[t], q);
        }
#pragma unroll
        for (int t = 0; t < 16; t++) {
            if (t & d) continue;
            const int k = (t & (d - 1)) * (8 >> l);   // exponent of the 16th root
            if (k == 0) {
                const uint32_t X = x[t], Y = x[t + d];
                x[t] = X + Y;
                x[t + d] = X - Y;
            } else {
                bfly(x[t], x[t + d], cc.iw[k], nq);
            }
        }
    }
    if (FIRST) {
#pragma unroll
        for (int t = 0; t < 16; t += 8) x[t] = umin(x[t], x[t] + 8 * q) - 4 * q;
    }
}

// the twiddles thread u needs in pass P (forward: of pass 0, shared by all)
template <int P>
__device__ __forceinline__ void fwd_twiddles(const uint4* __restrict__ tab, int ch, int u, uint2* w) {
    if (P == 0) {
        const ChanConst& cc = c_dev.ch[ch];
#pragma unroll
        for (int k = 1; k < 16; k++) w[k] = cc.fw[k];
    } else {
        unit_twiddles(P == 1 ? tab : tab + kTwPass1 / 2, P == 1 ? 16 : 256, P == 1 ? u >> 4 : u, w);
    }
}
template <int P>
__device__ __forceinline__ void inv_twiddles(const uint4* __restrict__ tab, int u, uint2* w) {
    unit_twiddles(P == 1 ? tab : tab + kTwPass1 / 2, P == 1 ? 16 : 256, P == 1 ? u & 15 : u, w);
}

// One forward pass over M polynomials (s + m * stride) by group thread u; inputs
// within +-q (signed words).  Ranges, in q, with B' = 1.03125 B + 1 per layer: 5.3 after
// pass 0; the summands folded to 3: 7.7 after pass 1; folded to 2: 6.7 after
// pass 2.  LAZY: the last pass leaves those signed words instead of canonical.
// The first pass takes its inputs from `in(m, x)` if there is one.
struct NoSource {};
template <int P, int M, bool LAZY, class In = NoSource>
__device__ __forceinline__ void fwd_pass(uint32_t* s, int stride, const uint2* w, int ch, int u, const In& in = In()) {
    const ChanConst& cc = c_dev.ch[ch];
    uint32_t* b = s + unit_base<P>(u);
#pragma unroll
    for (int m = 0; m < M; m++) {
        uint32_t x[16];
        if constexpr (P == 0 && !std::is_same<In, NoSource>::value) in(m, x);
        else unit_load<P>(b + m * stride, x);
        if (P > 0) {
#pragma unroll
            for (int t = 0; t < 8; t++) x[t] = P == 1 ? fold6(x[t], cc.q) : fold8(x[t], cc.q);
        }
        unit_layers<true>(x, w, cc.nq);
        if (P == 2 && !LAZY) {
#pragma unroll
            for (int t = 0; t < 16; t++) x[t] = canon_lazy(x[t], cc);
        }
        unit_store<P>(b + m * stride, x);
    }
}

// One inverse pass, in the order P = 0 (contiguous), 1 (stride 16: inputs below
// 5.2 q, the summands folded to 3, 7.7 q after it), 2 (stride 256; canonical
// outputs, handed to `out(m, t, value)` if there is one, else stored in place).
// The first pass takes its inputs, places 16 u .. 16 u + 15, from `in(m, x)` if there
// is one.
struct NoSink {};
template <int P, int M, class Out = NoSink, class In = NoSource>
__device__ __forceinline__ void inv_pass(uint32_t* s, int stride, const uint2* w, int ch, int u, const Out& out = Out(),
                                         const In& in = In()) {
    const ChanConst& cc = c_dev.ch[ch];
    const uint32_t q = cc.q, nq = cc.nq;
    constexpr int F = 2 - P;   // the forward pass of the same strides
    uint32_t* b = s + unit_base<F>(u);
#pragma unroll
    for (int m = 0; m < M; m++) {
        uint32_t x[16];
        if constexpr (P == 0 && !std::is_same<In, NoSource>::value) in(m, x);
        else unit_load<F>(b + m * stride, x);
        if (P == 0) {
            unit_dft16<true>(x, cc);
        } else if (P == 1) {
#pragma unroll
            for (int t = 0; t < 16; t += 2) x[t] = fold6(x[t], q);
            unit_layers<false>(x, w, nq);
        } else {
#pragma unroll
            for (int t = 0; t < 16; t++) x[t] = mul_lazy(x[t], w[t], nq);
            unit_dft16<false>(x, cc);
            x[0] = canon_lazy(x[0], cc);
#pragma unroll
            for (int t = 1; t < 16; t++) x[t] = canon_m1p2(mul_lazy(x[t], cc.ic[t], nq), q);
        }
        if constexpr (P == 2 && !std::is_same<Out, NoSink>::value) {
#pragma unroll
            for (int t = 0; t < 16; t++) out(m, t, x[t]);
        } else {
            unit_store<F>(b + m * stride, x);
        }
    }
}

// Forward transforms by one 256-thread group (thread u) of M padded polynomials
// s + m * stride of channel ch.  The caller has synchronised their inputs; ends
// with a barrier.  Each pass's twiddle loads are issued before the barrier
// that precedes it.
template <int M, class Sync, bool LAZY, class In = NoSource>
__device__ __forceinline__ void group_ntt_forward(uint32_t* s, int stride, const NttTables& tabs, int ch, int u,
                                                  const In& in = In()) {
    const uint4* tab = twiddle_table(tabs, ch, NTT_FWD);
    uint2 w[16];
    fwd_twiddles<0>(tab, ch, u, w);
    if (M) fwd_pass<0, M, LAZY>(s, stride, w, ch, u, in);
    if (M) fwd_twiddles<1>(tab, ch, u, w);
    Sync::sync();
    if (M) fwd_pass<1, M, LAZY>(s, stride, w, ch, u);
    if (M) fwd_twiddles<2>(tab, ch, u, w);
    Sync::sync();
    if (M) fwd_pass<2, M, LAZY>(s, stride, w, ch, u);
    Sync::sync();
}

// Inverse transforms by one group; canonical inputs (synchronised by the
// caller) and outputs; ends with a barrier unless the outputs go to `out`.
template <int M, class Sync, class Out = NoSink, class In = NoSource>
__device__ __forceinline__ void group_ntt_inverse(uint32_t* s, int stride, const NttTables& tabs, int ch, int u,
                                                  const Out& out = Out(), const In& in = In()) {
    const uint4* tab = twiddle_table(tabs, ch, NTT_INV);
    uint2 w[16];
    if (M) inv_pass<0, M>(s, stride, w, ch, u, NoSink(), in);
    if (M) inv_twiddles<1>(tab, u, w);
    Sync::sync();
    if (M) inv_pass<1, M>(s, stride, w, ch, u);
    if (M) inv_twiddles<2>(tab, u, w);
    Sync::sync();
    if (M) inv_pass<2, M>(s, stride, w, ch, u, out);
    if (std::is_same<Out, NoSink>::value) Sync::sync();
}

// The same by a 512-thread CTA: its two groups share the M polynomials (group
// g takes g, g + 2, ...).  Starts and ends with a barrier.
template <int M, class Sync = CtaSync, bool LAZY = false>
__device__ __forceinline__ void cta_ntt_forward_m(uint32_t* s, int stride, const NttTables& tabs, int ch) {
    const int u = threadIdx.x & (kNttGroup - 1), g = thread_group();
    Sync::sync();
    if (M % 2 == 0 || g == 0) group_ntt_forward<(M + 1) / 2, GroupSync, LAZY>(s + g * stride, 2 * stride, tabs, ch, u);
    else if (M > 1) group_ntt_forward<M / 2, GroupSync, LAZY>(s + stride, 2 * stride, tabs, ch, u);
    Sync::sync();
}

template <int M, class Sync = CtaSync>
__device__ __forceinline__ void cta_ntt_inverse_m(uint32_t* s, int stride, const NttTables& tabs, int ch) {
    const int u = threadIdx.x & (kNttGroup - 1), g = thread_group();
    Sync::sync();
    if (M % 2 == 0 || g == 0) group_ntt_inverse<(M + 1) / 2, GroupSync>(s + g * stride, 2 * stride, tabs, ch, u);
    else if (M > 1) group_ntt_inverse<M / 2, GroupSync>(s + stride, 2 * stride, tabs, ch, u);
    Sync::sync();
}

// Copies of whole polynomials between global memory (natural order) and a
// padded shared-memory polynomial; 16-byte vectors.  The loads bypass L1
// (ld.global.cg): the source is usually the previous kernel's output, and a
// kernel started early by programmatic dependent launch must not hit lines
// an overlapping kernel left in L1.
template <int T = kNttThreads>
__device__ __forceinline__ void poly_to_smem(uint32_t* s, const uint32_t* __restrict__ g) {
    const uint4* g4 = reinterpret_cast<const uint4*>(g);
#pragma unroll
    for (int k = threadIdx.x % T; k < kN / 4; k += T) *reinterpret_cast<uint4*>(s + pidx(4 * k)) = __ldcg(g4 + k);
}
template <int T = kNttThreads>
__device__ __forceinline__ void poly_from_smem(uint32_t* __restrict__ g, const uint32_t* s) {
    uint4* g4 = reinterpret_cast<uint4*>(g);
#pragma unroll
    for (int k = threadIdx.x % T; k < kN / 4; k += T) g4[k] = *reinterpret_cast<const uint4*>(s + pidx(4 * k));
}

}  // namespace kspir

// Giant steps (reference evalAutoRNSCRT, twosteps.cpp:599-677), the external
// product (externalProduct, lwe.cpp:761-808) and the RLWE packing tree
// (packingRLWEs / convertTwoRLWEs / evalAuto, answer.cpp:576-835).
//
// All three are key switches of the same shape: bring `a` to coefficient form,
// apply an automorphism, gadget-decompose, transform the digits, multiply by
// the key and accumulate.  Each runs as one fused kernel whose intermediates
// stay in shared memory (k_giant_fused, k_ext_fused, k_pack_fused).  The
// unfused element-wise decomposition and multiply-accumulate kernels of the
// external product remain for the allocation-free entry point.
#pragma once

#include "k_baby.cuh"
#include "ntt.cuh"
#include "pipeline.cuh"
#include "ptx.cuh"

namespace kspir {

// The key products of a thread's coefficients u + 256 (4 v + w), w = 0..3, on prime
// ch: ra, rb = sum over the ROWS polynomials d (in shared memory at stride
// `dstride`, lazy signed words below 6.7 q) times the keys of components a
// and b, reduced to within +-q (ROWS = 2) or +-1.4 q (ROWS = 4).  The keys (lane
// order, centred, times +-2^32: k_keys_from_words) come as one 16-byte vector per
// row and component, at `krow` vectors between rows and `kcomp` between components.
// |sum| <= ROWS 6.7 q q / 2 < 2^60; / 2^32 it is 0.21 ROWS q at most, and the
// Montgomery term adds q / 2: within +-q for ROWS = 2, +-1.4 q for ROWS = 4.
template <int ROWS>
__device__ __forceinline__ void key_mac4(const uint32_t* d, int dstride, const uint4* __restrict__ key, int krow,
                                         int kcomp, int ch, uint32_t* ra, uint32_t* rb) {
    uint64_t sa[4] = {0, 0, 0, 0}, sb[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < ROWS; j++) {
        const uint4 ka = __ldg(key + j * krow), kb = __ldg(key + j * krow + kcomp);
        const uint32_t kaw[4] = {ka.x, ka.y, ka.z, ka.w}, kbw[4] = {kb.x, kb.y, kb.z, kb.w};
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const uint32_t dv = d[j * dstride + w * kPadGroupStep];
            mad_wide_s(sa[w], dv, kaw[w]);
            mad_wide_s(sb[w], dv, kbw[w]);
        }
    }
    const ChanConst& cc = c_dev.ch[ch];
#pragma unroll
    for (int w = 0; w < 4; w++) {
        ra[w] = mont_redc(sa[w], cc);
        rb[w] = mont_redc(sb[w], cc);
    }
}

// ---------------------------------------------------------------------------
// external product, unfused (the allocation-free entry point)

// Signed digits of decompose_rlwe(a, b) (utils.cpp:974-1044) of the
// coefficient-form first-dimension result: edig[r][row][ch][k], rows 0..ell-1
// from a and ell..2ell-1 from b.
__global__ void k_ext_decomp(const uint32_t* __restrict__ ecoef, uint32_t* __restrict__ edig, int R, GadgetS g) {
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)R * kN) return;
    const int k = (int)(idx % kN);
    const long r = idx / kN;
    const uint32_t* e = ecoef + (size_t)r * 4 * kN;
    uint32_t* o = edig + (size_t)r * 2 * g.ell * 2 * kN;
    for (int comp = 0; comp < 2; comp++) {
        const uint64_t v = crt_compose_res(e[(comp * 2 + 0) * kN + k], e[(comp * 2 + 1) * kN + k]);
        int32_t dig[kMaxEll];
        decompose_signed(v, kCrtMod, g, dig);
        for (int j = 0; j < g.ell; j++) {
            const int row = comp * g.ell + j;
            o[(row * 2 + 0) * kN + k] = signed_to_res(dig[j], kQ1);
            o[(row * 2 + 1) * kN + k] = signed_to_res(dig[j], kQ2);
        }
    }
}

// dynamic shared memory of the fused multiply-accumulate + inverse-transform kernels
constexpr int kMacSmem = kPadN * 4;

// One CTA per (r, comp, ch): ext = INTT( init + sum_row digit_row * rgsw[row].comp ),
// init being the caller's NTT-domain accumulator (zero on the answer path,
// test-pir.cpp:102-104) or null.
__global__ void __launch_bounds__(kNttThreads) k_ext_mac_intt(const uint32_t* __restrict__ edig,
                                                              const uint32_t* __restrict__ rgsw,
                                                              const uint32_t* __restrict__ init,
                                                              uint32_t* __restrict__ ext, int rows, NttTables tabs) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint32_t* s = reinterpret_cast<uint32_t*>(smem_raw);
    constexpr int T = kNttThreads;
    const int ch = blockIdx.x % 2, comp = (blockIdx.x / 2) % 2, r = blockIdx.x / 4;
    const ChanConst cc = c_dev.ch[ch];
    const uint32_t* d = edig + (size_t)r * rows * 2 * kN;
#pragma unroll
    for (int k = threadIdx.x; k < kN; k += T) {
        uint64_t acc = 0;
        for (int row = 0; row < rows; row++)
            acc += (uint64_t)d[(row * 2 + ch) * kN + k] * rgsw[((row * 2 + comp) * 2 + ch) * kN + k];
        const uint32_t m = reduce64(acc, cc.q, cc.barrett);
        s[pidx(k)] = init ? addmod(init[((size_t)r * 4 + comp * 2 + ch) * kN + k], m, cc.q) : m;
    }
    cta_ntt_inverse_m<1>(s, kPadN, tabs, ch);
    uint32_t* o = ext + ((size_t)r * 4 + comp * 2 + ch) * kN;
#pragma unroll
    for (int k = threadIdx.x; k < kN; k += T) o[k] = s[pidx(k)];
}

// ---------------------------------------------------------------------------
// fused giant step: one CTA per (r, c >= 1) (blockIdx.y = query of the batch) runs the whole key switch of
// evalAutoRNSCRT for output[c] (twosteps.cpp:612-672) in shared memory:
//   INTT(a) per prime -> compose -> X -> X^g -> decompose (ell digits)
//   -> digit transforms -> -sum_j d_j * key[j]  and  b[sigma_g] - sum_j d_j * key[j]
// and adds both, canonical, into the sub-database's accumulator (u32 words
// in L2; the scan output is only read).  k_giant_finish, or the external product
// itself, then adds output[0] and reduces (giant_sum4).  A u32 word holds at most kGiantTermsPerAcc terms below
// q1 (16 (q1 - 1) < 2^32); with more giant steps per sub-database (N1 = 64:
// 31) rows c odd go to acc0 and rows c even to acc1.
constexpr int kGiantTermsPerAcc = 16;
static_assert((uint64_t)kGiantTermsPerAcc * (kQ1 - 1) < (1ull << 32) && kQ2 < kQ1, "giant accumulator width");

constexpr int kGiantPolys = 4;   // two primes x two digits (ell = 2)
constexpr int kPerThreadG = kN / kNttThreads;
constexpr int kGiantSmem = kGiantPolys * kPadN * 4;

// The key switch of output row `row` (= r N2 + c) into acc ([comp][prime][N] of
// sub-database r), by 512 threads.  Each 256-thread group runs one prime: its
// inverse transform of a (read from global memory by the first pass), and, after
// both have met for the decomposition, the transforms of the two digits (one
// set of twiddle loads for both) and the key products.  X -> X^g keeps
// coefficients u + 256 t in column u, the column that a thread's last inverse and
// first forward pass hold, so the digits reach the transform in registers and only
// the other prime's half crosses shared memory.  Bounded by issue, load and store
// wavefronts and the multiply pipe together (57, 55 and 46 % busy at 2 CTAs per SM;
// without the decomposition, the b gather and the accumulation 0.99 ms remain of
// 1.16).  Batch of 64 at r = 16: 1.56 ms with conditional-subtraction radix-8
// transforms and 64-bit Barrett reductions, 1.18 ms with the digits written
// twice to shared memory and read back, 1.16 ms; batch of 32 at r = 64: 2.37 -> 2.31.
template <int ELL, class Sync>
__device__ __forceinline__ void giant_body(uint32_t* P, const uint32_t* __restrict__ sout, uint32_t* acc,
                                           const uint32_t* __restrict__ gkeys, const uint16_t* __restrict__ gsigma,
                                           int N1, const NttTables& tabs, const GadgetB& g, int row, int c, int rows) {
    static_assert(ELL == 2 && 2 * ELL <= kGiantPolys, "shared-memory polynomials");
    const int ch = thread_group(), u = threadIdx.x & (kNttGroup - 1);

    // a of output[c] on this group's prime, to coefficient form
    auto load_a = [&](int, uint32_t* x) {
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const uint32_t* src = sout + sout_idx(row, 0 * 2 + ch, 16 * u + 8 * v, rows);
            if constexpr (std::is_same<Sync, CtaSync>::value) {
                ldg_256(src, x + 8 * v);
            } else {   // written by other CTAs of this launch: through L2
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    const uint4 t = __ldcg(reinterpret_cast<const uint4*>(src + i));
                    x[8 * v + i] = t.x; x[8 * v + i + 1] = t.y; x[8 * v + i + 2] = t.z; x[8 * v + i + 3] = t.w;
                }
            }
        }
    };
    uint32_t* D = P + ch * ELL * kPadN;              // this group's polynomials
    uint32_t* O = P + (1 - ch) * ELL * kPadN;        // the other's
    auto keep = [&](int, int t, uint32_t v) { D[kPadN + pidx(u) + t * kPadGroupStep] = v; };
    group_ntt_inverse<1, GroupSync>(D, kPadN, tabs, ch, u, keep, load_a);
    Sync::sync();
    // X -> X^g, g = 5^(N1 c), then the digits of half of the coefficients in each group.
    // g = 1 mod 256 (N1 >= 64), so coefficient u + 256 t comes from u + 256 h with
    // h = (u g^-1 >> 8) + t g^-1 mod 32, negated when h >= 16.
    const uint32_t e = (uint32_t)(N1 * c) & 2047u;
    uint32_t ginv = 1, b5 = 5, x = (2048u - e) & 2047u;
    while (x) { if (x & 1) ginv = (ginv * b5) & (2 * kN - 1); b5 = (b5 * b5) & (2 * kN - 1); x >>= 1; }
    int32_t dres[kPerThreadG][ELL];
    uint32_t h = ((u * ginv) >> 8) + 8 * ch * ginv;
    const uint32_t* Pu = P + kPadN + pidx(u);
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {   // coefficient u + 256 (8 ch + it)
        const uint32_t* src = Pu + (h & 15) * kPadGroupStep;
        decompose_b_res<ELL>(src[0], src[ELL * kPadN], h & 16, g, dres[it]);
        h += ginv;
    }
    // A digit is a small signed word, the same for both primes: each group hands its half
    // to the other, column u to the thread that transforms column u, through the
    // other's first polynomial (free since its inverse transform; this group's half of
    // the second digit takes the places of the other's half of the first).  Only
    // the two threads of column u touch it until the first pass has stored it.
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        O[pidx(u) + (8 * ch + it) * kPadGroupStep] = (uint32_t)dres[it][0];
        O[pidx(u) + (8 * (1 - ch) + it) * kPadGroupStep] = (uint32_t)dres[it][1];
    }
    Sync::sync();
    uint32_t ex[ELL][kPerThreadG];
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        ex[0][it] = D[pidx(u) + (8 * (1 - ch) + it) * kPadGroupStep];
        ex[1][it] = D[pidx(u) + (8 * ch + it) * kPadGroupStep];
    }
    auto digits = [&](int m, uint32_t* x) {
#pragma unroll
        for (int it = 0; it < kPerThreadG; it++) {
            x[it] = ch ? ex[m][it] : (uint32_t)dres[it][m];
            x[8 + it] = ch ? (uint32_t)dres[it][m] : ex[m][it];
        }
    };
    group_ntt_forward<ELL, GroupSync, true>(D, kPadN, tabs, ch, u, digits);   // signed, below 6.7 q
    const uint32_t q = c_dev.ch[ch].q;
    const uint4* key = reinterpret_cast<const uint4*>(gkeys + (size_t)(c - 1) * ELL * 4 * kN + (size_t)ch * kN);
    const uint16_t* sig = gsigma + (size_t)(c - 1) * kN;
    uint32_t* acc_a = acc + (size_t)ch * kN + u;
    uint32_t* acc_b = acc_a + 2 * kN;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int i = v * kNttGroup + u;
        uint32_t sl[4], ra[4], rb[4];
        perm4(sig, i, sl);
        uint32_t bv[4];
#pragma unroll
        for (int w = 0; w < 4; w++) bv[w] = __ldcg(sout + sout_idx(row, 1 * 2 + ch, sl[w], rows));
        key_mac4<ELL>(D + pidx(u) + 4 * v * kPadGroupStep, kPadN, key + i, 4 * kN / 4, 2 * kN / 4, ch, ra, rb);
#pragma unroll
        for (int w = 0; w < 4; w++) {
            atomicAdd(acc_a + kNttGroup * (4 * v + w), canon_pm1(ra[w], q));
            atomicAdd(acc_b + kNttGroup * (4 * v + w), canon_m1p2(rb[w] + bv[w], q));
        }
    }
}

template <int ELL>
__global__ void __launch_bounds__(kNttThreads, 2)
    k_giant_fused(const uint32_t* __restrict__ sout, uint32_t* acc0, uint32_t* acc1,
                  const uint32_t* __restrict__ gkeys, const uint16_t* __restrict__ gsigma, int N1, NttTables tabs,
                  GadgetB g, int R, Batch bt) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int N2 = kN / 2 / N1;
    const int rc = blockIdx.x;
    const int r = rc / (N2 - 1), c = rc % (N2 - 1) + 1;
    pdl_launch_dependents();
    pdl_wait();   // the scan output comes from the previous kernel
    giant_body<ELL, CtaSync>(reinterpret_cast<uint32_t*>(smem_raw), shifted(sout, ws_off(bt)),
                             shifted((acc1 && !(c & 1)) ? acc1 : acc0, ws_off(bt)) + (size_t)r * 4 * kN,
                             shifted(gkeys, key_off(bt)), gsigma, N1, tabs, g, r * N2 + c, c, R * N2);
}

// Where the external product finds output[0] and the second accumulator of its
// first-dimension results (slot-0 addresses).  sout null: the residues given are
// final.
struct GiantSums {
    const uint32_t* sout;
    const uint32_t* acc1;   // or null
    int N2, rows;           // rows = R N2
};

// (output[0] + the giant-step accumulators) mod q of slots z .. z + 3, polynomial cv =
// comp * 2 + prime of sub-database r; fd points at the polynomial of the accumulator
// acc0, wo is the query's workspace offset
__device__ __forceinline__ uint4 giant_sum4(const GiantSums& g, size_t wo, const uint32_t* fd, int r, int cv, int z) {
    const ChanConst& q = c_dev.ch[cv & 1];
    const uint4 a = __ldcg(reinterpret_cast<const uint4*>(fd + z));
    const uint4 w = __ldcg(reinterpret_cast<const uint4*>(shifted(g.sout, wo) + sout_idx(r * g.N2, cv, z, g.rows)));
    uint64_t v0 = (uint64_t)a.x + w.x, v1 = (uint64_t)a.y + w.y, v2 = (uint64_t)a.z + w.z, v3 = (uint64_t)a.w + w.w;
    if (g.acc1) {
        const uint4 b = __ldcg(reinterpret_cast<const uint4*>(shifted(g.acc1, wo) + ((size_t)r * 4 + cv) * kN + z));
        v0 += b.x; v1 += b.y; v2 += b.z; v3 += b.w;
    }
    return make_uint4(reduce64(v0, q.q, q.barrett), reduce64(v1, q.q, q.barrett), reduce64(v2, q.q, q.barrett),
                      reduce64(v3, q.q, q.barrett));
}

// The first-dimension results [r][comp][ch][k] from their accumulators acc0, in place
// or (one query) into out, for the external products that do not add it up themselves
// (first_dim_to_smem), the staged calls and diagnostics.  One thread per four
// consecutive slots.
__global__ void k_giant_finish(GiantSums g, uint32_t* acc0, uint32_t* out, int R, Batch bt) {
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)R * 4 * (kN / 4)) return;
    const size_t wo = ws_off(bt);
    const int z = (int)(idx % (kN / 4)) * 4;
    const int cv = (int)((idx / (kN / 4)) % 4);
    const int r = (int)(idx / (4 * (kN / 4)));
    const size_t at = ((size_t)r * 4 + cv) * kN;
    acc0 = shifted(acc0, wo);
    *reinterpret_cast<uint4*>((out ? out : acc0) + at + z) = giant_sum4(g, wo, acc0 + at, r, cv, z);
}

// Polynomial cv of first-dimension result r (at fd) into shared memory, by T threads.
// With the sums here instead of in k_giant_finish, which writes every result once
// more to be read back: batch of 64 at r = 16 3.484 -> 3.447 ms, of 32 at r = 64
// 5.648 -> 5.582 ms.  Where a CTA per prime reads all of first_dim (k_ext_fused) the
// longer load costs what the launch did (r = 1: 168.9 -> 170.2 us, r = 16: 383.9 ->
// 383.0), so that one keeps the kernel.
template <int T = kNttThreads>
__device__ __forceinline__ void first_dim_to_smem(uint32_t* s, const uint32_t* fd, const GiantSums& g, size_t wo, int r,
                                                  int cv) {
    if (!g.sout) {
        poly_to_smem<T>(s, fd);
        return;
    }
#pragma unroll
    for (int k = threadIdx.x % T; k < kN / 4; k += T)
        *reinterpret_cast<uint4*>(s + pidx(4 * k)) = giant_sum4(g, wo, fd, r, cv, 4 * k);
}

// ---------------------------------------------------------------------------
// fused packing level: one CTA per (pair j, prime ch) runs convertTwoRLWEs
// (answer.cpp:720-739) with its evalAuto key switch (answer.cpp:576-648) in
// shared memory.  It reads level input `in` and writes level output `out`
// (two buffers: both primes of in[j] are read while the other CTA of the pair
// writes its prime of out[j]).
//   c' = X^I c,  r1 = r0 - c',  c2 = c' + r0,  temp = auto_g(r1), g = N/I + 1
//   a' = -sum_d dig_d * key[d].a,  b' = NTT(temp.b) - sum_d dig_d * key[d].b
//   out[j] = INTT(a', b') + c2
constexpr int kPackPolys = 5;    // ell = 4 digits + temp.b
constexpr int kPackSmem = kPackPolys * kPadN * 4;

template <int ELL>
__global__ void __launch_bounds__(kNttThreads, 2) k_pack_fused(const uint32_t* __restrict__ in,
                                                            uint32_t* __restrict__ out,
                                                            const uint32_t* __restrict__ key, int I, uint32_t ginv,
                                                            NttTables tabs, GadgetB g, Batch bt) {
    static_assert(ELL + 1 <= kPackPolys, "shared-memory polynomials");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    in = shifted(in, ws_off(bt));
    out = shifted(out, ws_off(bt));
    key = shifted(key, key_off(bt));
    uint32_t* P = reinterpret_cast<uint32_t*>(smem_raw);   // [kPackPolys][N]
    const int j = blockIdx.x >> 1, ch = blockIdx.x & 1;
    const int tid = threadIdx.x;
    const uint32_t* r0 = in + (size_t)j * 4 * kN;
    const uint32_t* cc = in + (size_t)(I + j) * 4 * kN;
    const uint32_t q = c_dev.ch[ch].q;
    pdl_launch_dependents();
    pdl_wait();   // the level input comes from the previous kernel
    // launched after that kernel completes (no early launch), and no CTA writes
    // the level input: its gathers below read through L1
    // X^I c at position p of polynomial (comp, prime)
    auto cshift = [&](int comp, int pch, int p) -> uint32_t {
        const int s = p - I;
        const uint32_t qq = pch ? kQ2 : kQ1;
        return s >= 0 ? __ldg(cc + (comp * 2 + pch) * kN + s) : negmod(__ldg(cc + (comp * 2 + pch) * kN + s + kN), qq);
    };
    uint32_t c2v[kPerThreadG][2];
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        const int k = tid + it * kNttThreads;
#pragma unroll
        for (int comp = 0; comp < 2; comp++)
            c2v[it][comp] = addmod(cshift(comp, ch, k), __ldg(r0 + (comp * 2 + ch) * kN + k), q);
        bool neg;
        const int src = auto_src(k, ginv, &neg);
        uint32_t ra[2];
#pragma unroll
        for (int pch = 0; pch < 2; pch++) {
            const uint32_t qq = pch ? kQ2 : kQ1;
            const uint32_t v = submod(__ldg(r0 + (0 * 2 + pch) * kN + src), cshift(0, pch, src), qq);
            ra[pch] = neg ? negmod(v, qq) : v;
        }
        int32_t dig[kMaxEll];
        decompose_b(crt_compose_res(ra[0], ra[1]), kCrtMod, g, dig);
        const int pk = pidx(tid) + it * kPadStep;
#pragma unroll
        for (int d = 0; d < ELL; d++) P[d * kPadN + pk] = (uint32_t)dig[d];
        const uint32_t vb = submod(__ldg(r0 + (1 * 2 + ch) * kN + src), cshift(1, ch, src), q);
        P[ELL * kPadN + pk] = neg ? 0u - vb : vb;
    }
    cta_ntt_forward_m<ELL + 1, CtaSync, true>(P, kPadN, tabs, ch);   // signed, below 6.7 q
    const int g2 = thread_group(), u = tid & (kNttGroup - 1);
#pragma unroll
    for (int vv = 0; vv < 2; vv++) {
        const int v = 2 * g2 + vv;
        uint32_t* p = P + pidx(u) + 4 * v * kPadGroupStep;
        uint32_t ra[4], rb[4];
        key_mac4<ELL>(p, kPadN, reinterpret_cast<const uint4*>(key + ch * kN) + v * kNttGroup + u, 4 * kN / 4, 2 * kN / 4,
                      ch, ra, rb);
#pragma unroll
        for (int w = 0; w < 4; w++) {   // only this thread reads these coefficients of the rows
            const uint32_t b = reduce_lazy(p[ELL * kPadN + w * kPadGroupStep], c_dev.ch[ch].rq, c_dev.ch[ch].nq);
            p[w * kPadGroupStep] = canon_pm2(ra[w], q);
            p[kPadN + w * kPadGroupStep] = canon_pm4(rb[w] + b, q);
        }
    }
    cta_ntt_inverse_m<2>(P, kPadN, tabs, ch);
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        const int k = tid + it * kNttThreads;
#pragma unroll
        for (int comp = 0; comp < 2; comp++)
            out[((size_t)j * 4 + comp * 2 + ch) * kN + k] = addmod(P[comp * kPadN + pidx(tid) + it * kPadStep], c2v[it][comp], q);
    }
}

// ---------------------------------------------------------------------------
// packing level split over more CTAs, for single queries and small batches:
// the fused kernel's CTA runs ELL + 1 forward and 2 inverse transforms in a
// row, and the last levels have only 2 * I CTAs, so a level's latency is
// those seven transforms.  Split, each CTA runs one:
//   k_pack_split_fwd  (pair j, prime ch, d <= ELL): digit d (or temp.b for
//                     d = ELL) -> transform -> its terms dig_d * key[d].a/.b
//                     into part[j][ch][d][comp]
//   k_pack_split_inv  (pair j, prime ch, comp): the sum of the terms ->
//                     inverse transform -> + c2 into out[j]
// Same residues as k_pack_fused (sums mod q in another order).
constexpr int kPackPartPolys = 2 * 5 * 2;   // per pair: [prime][ELL + 1][comp]
constexpr int kPackSplitSmem = kPadN * 4;

// One split forward task, pair j, prime ch, digit d (d = ELL: temp.b); in,
// part and key already point at the query's workspace and key slot.  Shared
// with the fused answer kernel (Sync = its named barrier).
template <int ELL, class Sync>
__device__ __forceinline__ void pack_split_fwd_body(const uint32_t* __restrict__ in, uint32_t* __restrict__ part,
                                                    const uint32_t* __restrict__ key, int I, uint32_t ginv,
                                                    const NttTables& tabs, const GadgetB& g, int j, int ch, int d,
                                                    uint8_t* smem_raw) {
    static_assert(2 * (ELL + 1) * 2 <= kPackPartPolys, "term buffer");
    uint32_t* S = reinterpret_cast<uint32_t*>(smem_raw);
    const int tid = threadIdx.x;
    const uint32_t* r0 = in + (size_t)j * 4 * kN;
    const uint32_t* cc = in + (size_t)(I + j) * 4 * kN;
    const uint32_t q = c_dev.ch[ch].q;
    pdl_launch_dependents();
    warm_twiddles(tabs, ch, NTT_FWD, tid, kNttThreads);
    // the key words of this digit, loaded while the previous kernel finishes
    // (keys are never written by the answer), used after the transform
    const int g2 = thread_group(), u = tid & (kNttGroup - 1);
    uint4 ka[2], kb[2];
    if (d < ELL) {
        const uint4* k4 = reinterpret_cast<const uint4*>(key + (size_t)(d * 4 + ch) * kN) + 2 * g2 * kNttGroup + u;
#pragma unroll
        for (int vv = 0; vv < 2; vv++) {
            ka[vv] = __ldg(k4 + vv * kNttGroup);
            kb[vv] = __ldg(k4 + 2 * kN / 4 + vv * kNttGroup);
        }
    }
    pdl_wait();   // the level input comes from the previous kernel
    auto cshift = [&](int comp, int pch, int p) -> uint32_t {   // (X^I c)[p]
        const int s = p - I;
        const uint32_t qq = pch ? kQ2 : kQ1;
        return s >= 0 ? __ldcg(cc + (comp * 2 + pch) * kN + s) : negmod(__ldcg(cc + (comp * 2 + pch) * kN + s + kN), qq);
    };
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        const int k = tid + it * kNttThreads;
        bool neg;
        const int src = auto_src(k, ginv, &neg);
        uint32_t v;
        if (d < ELL) {
            uint32_t ra[2];
#pragma unroll
            for (int pch = 0; pch < 2; pch++) {
                const uint32_t qq = pch ? kQ2 : kQ1;
                const uint32_t x = submod(__ldcg(r0 + (0 * 2 + pch) * kN + src), cshift(0, pch, src), qq);
                ra[pch] = neg ? negmod(x, qq) : x;
            }
            int32_t dig[kMaxEll];
            decompose_b(crt_compose_res(ra[0], ra[1]), kCrtMod, g, dig);
            v = (uint32_t)dig[d];
        } else {
            const uint32_t vb = submod(__ldcg(r0 + (1 * 2 + ch) * kN + src), cshift(1, ch, src), q);
            v = neg ? 0u - vb : vb;
        }
        S[pidx(tid) + it * kPadStep] = v;
    }
    cta_ntt_forward_m<1, Sync, true>(S, kPadN, tabs, ch);   // signed, below 6.7 q
    uint32_t* pa = part + (((size_t)j * 2 + ch) * (ELL + 1) + d) * 2 * kN;
    const ChanConst& cc2 = c_dev.ch[ch];
#pragma unroll
    for (int vv = 0; vv < 2; vv++) {
        const uint32_t kaw[4] = {ka[vv].x, ka[vv].y, ka[vv].z, ka[vv].w}, kbw[4] = {kb[vv].x, kb[vv].y, kb[vv].z, kb[vv].w};
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const int t = 4 * (2 * g2 + vv) + w, k = u + kNttGroup * t;
            const uint32_t dv = S[pidx(u) + t * kPadGroupStep];
            if (d < ELL) {   // within +-0.71 q
                uint64_t sa = 0, sb = 0;
                mad_wide_s(sa, dv, kaw[w]);
                mad_wide_s(sb, dv, kbw[w]);
                pa[k] = canon_pm1(mont_redc(sa, cc2), q);
                pa[kN + k] = canon_pm1(mont_redc(sb, cc2), q);
            } else {
                pa[k] = canon_lazy(dv, cc2);   // NTT(temp.b)
            }
        }
    }
}

template <int ELL>
__global__ void __launch_bounds__(kNttThreads) k_pack_split_fwd(const uint32_t* __restrict__ in,
                                                                uint32_t* __restrict__ part,
                                                                const uint32_t* __restrict__ key, int I,
                                                                uint32_t ginv, NttTables tabs, GadgetB g, Batch bt) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int d = blockIdx.x % (ELL + 1), ch = (blockIdx.x / (ELL + 1)) & 1, j = blockIdx.x / (ELL + 1) / 2;
    pack_split_fwd_body<ELL, CtaSync>(shifted(in, ws_off(bt)), shifted(part, ws_off(bt)), shifted(key, key_off(bt)), I,
                                      ginv, tabs, g, j, ch, d, smem_raw);
}

// c2out (or null): the reference's packingRLWEs leaves c2 = X^I c + r of the
// merge of (j, I + j) in rlwes[I + j] (answer.cpp:727-731, 821-828); the
// staged entry point returns it there, as [r][comp][ch][N] residues.
template <int ELL, class Sync>
__device__ __forceinline__ void pack_split_inv_body(const uint32_t* __restrict__ in, const uint32_t* __restrict__ part,
                                                    uint32_t* __restrict__ out, int I, const NttTables& tabs, int j,
                                                    int ch, int comp, uint32_t* __restrict__ c2out,
                                                    uint8_t* smem_raw) {
    uint32_t* S = reinterpret_cast<uint32_t*>(smem_raw);
    const int tid = threadIdx.x;
    const uint32_t q = c_dev.ch[ch].q;
    pdl_launch_dependents();
    warm_twiddles(tabs, ch, NTT_INV, tid, kNttThreads);
    pdl_wait();   // the terms come from the previous kernel
    const uint32_t* pj = part + ((size_t)j * 2 + ch) * (ELL + 1) * 2 * kN;
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        const int k = tid + it * kNttThreads;
        uint32_t sum = 0;
#pragma unroll
        for (int d = 0; d < ELL; d++) sum = addmod(sum, __ldcg(pj + ((size_t)d * 2 + comp) * kN + k), q);
        // a' = sum_d dig_d (-key[d].a) ;  b' = NTT(temp.b) + sum_d dig_d (-key[d].b)
        S[pidx(tid) + it * kPadStep] = comp == 0 ? sum : addmod(__ldcg(pj + (size_t)ELL * 2 * kN + k), sum, q);
    }
    // c2 = X^I c + r of the level input, loaded ahead of the transform
    const uint32_t* r0 = in + (size_t)j * 4 * kN;
    const uint32_t* cc = in + (size_t)(I + j) * 4 * kN + (comp * 2 + ch) * kN;
    uint32_t c2[kPerThreadG];
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        const int k = tid + it * kNttThreads;
        const int s = k - I;
        const uint32_t sh = s >= 0 ? __ldcg(cc + s) : negmod(__ldcg(cc + s + kN), q);
        c2[it] = addmod(sh, __ldcg(r0 + (comp * 2 + ch) * kN + k), q);
        if (c2out) c2out[((size_t)(I + j) * 4 + comp * 2 + ch) * kN + k] = c2[it];
    }
    cta_ntt_inverse_m<1, Sync>(S, kPadN, tabs, ch);
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        const int k = tid + it * kNttThreads;
        out[((size_t)j * 4 + comp * 2 + ch) * kN + k] = addmod(S[pidx(tid) + it * kPadStep], c2[it], q);
    }
}

template <int ELL>
__global__ void __launch_bounds__(kNttThreads) k_pack_split_inv(const uint32_t* __restrict__ in,
                                                                const uint32_t* __restrict__ part,
                                                                uint32_t* __restrict__ out, int I, NttTables tabs,
                                                                Batch bt, uint32_t* __restrict__ c2out) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int comp = blockIdx.x & 1, ch = (blockIdx.x >> 1) & 1, j = blockIdx.x >> 2;
    pack_split_inv_body<ELL, CtaSync>(shifted(in, ws_off(bt)), shifted(part, ws_off(bt)), shifted(out, ws_off(bt)), I,
                                      tabs, j, ch, comp, shifted(c2out, ws_off(bt)), smem_raw);
}

// The external product after first_dim is in coefficient form in P[comp * 2 +
// prime] (both primes, as the decomposition needs the composed word): signed
// digits of a and b, their transforms on prime ch, init (or 0) + sum_row
// row * rgsw[row], inverse transform, into ext [comp][ch][N].  rgsw, init and
// ext point at the query's key slot and its polynomial r.
template <int ELL, class Sync>
__device__ __forceinline__ void ext_tail(uint32_t* P, const uint32_t* __restrict__ rgsw,
                                         const uint32_t* __restrict__ init, uint32_t* __restrict__ ext,
                                         const NttTables& tabs, const GadgetS& g, int ch) {
    const int tid = threadIdx.x;
    // signed digits of a and b (rows comp * ELL + t), residues of this prime
    uint32_t dres[kPerThreadG][2 * ELL];
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
#pragma unroll
        for (int comp = 0; comp < 2; comp++) {
            int32_t dig[kMaxEll];
            const int pk = pidx(tid) + it * kPadStep;
            decompose_signed(crt_compose_res(P[(comp * 2 + 0) * kPadN + pk], P[(comp * 2 + 1) * kPadN + pk]), kCrtMod, g,
                             dig);
#pragma unroll
            for (int t = 0; t < ELL; t++) dres[it][comp * ELL + t] = (uint32_t)dig[t];
        }
    }
    Sync::sync();
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++)
#pragma unroll
        for (int row = 0; row < 2 * ELL; row++) P[row * kPadN + pidx(tid) + it * kPadStep] = dres[it][row];
    cta_ntt_forward_m<2 * ELL, Sync, true>(P, kPadN, tabs, ch);   // signed, below 6.7 q
    const uint32_t q = c_dev.ch[ch].q;
    const int g2 = thread_group(), u = tid & (kNttGroup - 1);
#pragma unroll
    for (int vv = 0; vv < 2; vv++) {
        const int v = 2 * g2 + vv;
        uint32_t* p = P + pidx(u) + 4 * v * kPadGroupStep;
        uint32_t ra[4], rb[4];
        key_mac4<2 * ELL>(p, kPadN, reinterpret_cast<const uint4*>(rgsw + ch * kN) + v * kNttGroup + u, 4 * kN / 4,
                          2 * kN / 4, ch, ra, rb);
#pragma unroll
        for (int w = 0; w < 4; w++) {   // only this thread reads these coefficients of the rows
            const int k = u + kNttGroup * (4 * v + w);
            uint32_t oa = canon_pm2(ra[w], q), ob = canon_pm2(rb[w], q);
            if (init) {
                oa = addmod(__ldcg(init + (size_t)ch * kN + k), oa, q);
                ob = addmod(__ldcg(init + (size_t)(2 + ch) * kN + k), ob, q);
            }
            p[w * kPadGroupStep] = oa;
            p[kPadN + w * kPadGroupStep] = ob;
        }
    }
    cta_ntt_inverse_m<2, Sync>(P, kPadN, tabs, ch);
#pragma unroll
    for (int it = 0; it < kPerThreadG; it++) {
        const int k = tid + it * kNttThreads;
#pragma unroll
        for (int comp = 0; comp < 2; comp++)
            ext[(size_t)(comp * 2 + ch) * kN + k] = P[comp * kPadN + pidx(tid) + it * kPadStep];
    }
}

// ---------------------------------------------------------------------------
// fused external product: one CTA per (r, prime ch) runs externalProduct
// (lwe.cpp:761-808) in shared memory:
//   INTT(first_dim) (both primes, to compose) -> decompose_rlwe (2 ell rows)
//   -> row transforms -> init + sum_row row * rgsw[row] -> INTT
constexpr int kExtPolys = 4;
constexpr int kExtSmem = kExtPolys * kPadN * 4;

template <int ELL>
__global__ void __launch_bounds__(kNttThreads, 2) k_ext_fused(const uint32_t* __restrict__ first_dim,
                                                           const uint32_t* __restrict__ rgsw,
                                                           const uint32_t* __restrict__ init,
                                                           uint32_t* __restrict__ ext,
                                                           uint32_t* __restrict__ coef_out, NttTables tabs,
                                                           GadgetS g, Batch bt) {
    static_assert(2 * ELL <= kExtPolys, "shared-memory polynomials");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    first_dim = shifted(first_dim, ws_off(bt));
    init = shifted(init, ws_off(bt));
    ext = shifted(ext, ws_off(bt));
    coef_out = shifted(coef_out, ws_off(bt));
    rgsw = shifted(rgsw, key_off(bt));
    uint32_t* P = reinterpret_cast<uint32_t*>(smem_raw);   // [4][N]
    const int r = blockIdx.x >> 1, ch = blockIdx.x & 1;
    const uint32_t* fd = first_dim + (size_t)r * 4 * kN;          // [comp][prime][N]
    pdl_launch_dependents();
    // first_dim to coefficient form, all four polynomials (P[comp * 2 + prime])
#pragma unroll
    for (int pch = 0; pch < 2; pch++) {
        pdl_wait();   // the first-dimension results come from the previous kernel
#pragma unroll
        for (int comp = 0; comp < 2; comp++) {
            poly_to_smem(P + (comp * 2 + pch) * kPadN, fd + (comp * 2 + pch) * kN);
        }
        cta_ntt_inverse_m<2>(P + pch * kPadN, 2 * kPadN, tabs, pch);   // a and b of this prime
    }
    if (coef_out && ch == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) poly_from_smem(coef_out + ((size_t)r * 4 + i) * kN, P + i * kPadN);
    }
    ext_tail<ELL, CtaSync>(P, rgsw, init ? init + (size_t)r * 4 * kN : nullptr, ext + (size_t)r * 4 * kN, tabs, g,
                           ch);
}

// ---------------------------------------------------------------------------
// external product of many ciphertexts: one CTA per r on four thread groups, 16
// transforms where k_ext_fused's CTA per prime runs 2 x 12 (both bring all of
// first_dim to coefficient form): batch of 64 at r = 16 0.223 -> 0.185 ms.  With
// few ciphertexts (one per SM or less) the CTA per prime is faster, two SMs
// sharing the work: one query at r = 16 0.025 against 0.031 ms.
//   INTT(first_dim), one polynomial per group -> decompose_rlwe (2 ell digits,
//   small signed words for both primes) -> two digit transforms per group (prime
//   grp / 2) -> init + sum_row row * rgsw[row] -> INTT, one polynomial per group
constexpr int kExtWideThreads = 4 * kNttGroup;
constexpr int kExtWideSmem = 8 * kPadN * 4;   // two primes x four digits

template <int ELL>
__global__ void __launch_bounds__(kExtWideThreads, 1)
    k_ext_wide(const uint32_t* __restrict__ first_dim, GiantSums sums, const uint32_t* __restrict__ rgsw,
               const uint32_t* __restrict__ init, uint32_t* __restrict__ ext, uint32_t* __restrict__ coef_out, NttTables tabs, GadgetS g, Batch bt) {
    static_assert(ELL == 2, "four digits, two per group and prime");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint32_t* P = reinterpret_cast<uint32_t*>(smem_raw);
    const int r = blockIdx.x, grp = thread_group(), u = threadIdx.x & (kNttGroup - 1);
    const size_t wo = ws_off(bt);
    const uint32_t* fd = shifted(first_dim, wo) + (size_t)r * 4 * kN;          // [comp][prime][N]
    rgsw = shifted(rgsw, key_off(bt));
    pdl_launch_dependents();
    pdl_wait();   // the first-dimension results come from the previous kernel
    {
        uint32_t* S = P + grp * kPadN;   // polynomial grp = comp * 2 + prime
        first_dim_to_smem<kNttGroup>(S, fd + (size_t)grp * kN, sums, wo, r, grp);
        GroupSync::sync();
        uint32_t* co = coef_out ? shifted(coef_out, wo) + ((size_t)r * 4 + grp) * kN + u : nullptr;
        auto keep = [&](int, int t, uint32_t x) {
            S[pidx(u) + t * kPadGroupStep] = x;
            if (co) co[kNttGroup * t] = x;
        };
        group_ntt_inverse<1, GroupSync>(S, kPadN, tabs, grp & 1, u, keep);
    }
    __syncthreads();
    uint32_t dres[4][2 * ELL];   // coefficients u + 256 (4 grp + w): digits of a, then of b
#pragma unroll
    for (int w = 0; w < 4; w++) {
        const uint32_t* p = P + pidx(u) + (4 * grp + w) * kPadGroupStep;
#pragma unroll
        for (int comp = 0; comp < 2; comp++) {
            int32_t dig[kMaxEll];
            decompose_signed(crt_compose_res(p[comp * 2 * kPadN], p[(comp * 2 + 1) * kPadN]), kCrtMod, g, dig);
#pragma unroll
            for (int t = 0; t < ELL; t++) dres[w][comp * ELL + t] = (uint32_t)dig[t];
        }
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 4; w++)
#pragma unroll
        for (int row = 0; row < 2 * ELL; row++)
#pragma unroll
            for (int p = 0; p < 2; p++)
                P[(p * 2 * ELL + row) * kPadN + pidx(u) + (4 * grp + w) * kPadGroupStep] = dres[w][row];
    __syncthreads();
    const int ch = grp >> 1, half = grp & 1;
    uint32_t* D = P + ch * 2 * ELL * kPadN;
    group_ntt_forward<ELL, GroupSync, true>(D + half * ELL * kPadN, kPadN, tabs, ch, u);   // signed, below 6.7 q
    __syncthreads();
    const uint32_t q = c_dev.ch[ch].q;
#pragma unroll
    for (int vv = 0; vv < 2; vv++) {
        const int v = 2 * half + vv;
        uint32_t* p = D + pidx(u) + 4 * v * kPadGroupStep;
        uint32_t ra[4], rb[4];
        key_mac4<2 * ELL>(p, kPadN, reinterpret_cast<const uint4*>(rgsw + ch * kN) + v * kNttGroup + u, 4 * kN / 4,
                          2 * kN / 4, ch, ra, rb);
#pragma unroll
        for (int w = 0; w < 4; w++) {   // only this thread reads these coefficients of the rows
            uint32_t oa = canon_pm2(ra[w], q), ob = canon_pm2(rb[w], q);
            if (init) {
                const uint32_t* i0 = shifted(init, wo) + ((size_t)r * 4 + ch) * kN + u + kNttGroup * (4 * v + w);
                oa = addmod(__ldcg(i0), oa, q);
                ob = addmod(__ldcg(i0 + 2 * kN), ob, q);
            }
            p[w * kPadGroupStep] = oa;
            p[kPadN + w * kPadGroupStep] = ob;
        }
    }
    __syncthreads();
    uint32_t* o = shifted(ext, wo) + ((size_t)r * 4 + half * 2 + ch) * kN + u;   // component `half` of prime ch
    auto store = [&](int, int t, uint32_t x) { o[kNttGroup * t] = x; };
    group_ntt_inverse<1, GroupSync>(D + half * kPadN, kPadN, tabs, ch, u, store);
}

}  // namespace kspir

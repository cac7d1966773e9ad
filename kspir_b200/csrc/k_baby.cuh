// The hoisted baby steps (reference evalAutoSRNSFirst / evalAutoSRNSSecond,
// twosteps.cpp:937-1204) fused with the RNS modswitch and reorientCipher
// (twosteps.cpp:1386-1403): one CTA produces one rotation of the query and
// writes it, as residue pairs, straight into its cipherbuf column.
//
// Per rotation g = 5^(i+1) (key index i), with digits d_j of the source a in
// NTT form (hoisted: decomposed once, reference :960-979 / :1109-1127):
//   A_c = -sum_j d_j[perm[k]] * key_j.a     (crtMod channels c and bsMod)
//   B_c = -sum_j d_j[perm[k]] * key_j.b
// The reference then leaves the NTT domain for the modswitch:
//   out.a = NTT((INTT(A_crt) - x2a) * bsMod^-1),  x2a = INTT_bs(A_bs)
//   out.b = NTT((INTT(B_crt) + auto_g(b) - x2b) * bsMod^-1),
//           x2b = INTT_bs(B_bs) + auto_g(b mod bsMod)
// (twosteps.cpp:1034-1071).  All of it is exact arithmetic mod crtMod and
// bsMod with canonical values, so by linearity of the transform the same words are
//   out.a = A_crt * bsMod^-1 - NTT(x2a) * bsMod^-1
//   out.b = B_crt * bsMod^-1 + (NTT(b) * bsMod^-1)[sigma_g] - NTT(x2b) * bsMod^-1
//   x2b   = INTT_bs(B_bs + NTT_bs(b)[sigma_g])
// where sigma_g is the slot permutation of X -> X^g in the NTT domain.  Only
// the bsMod channel is brought to coefficient form (x2 must be the canonical
// integer < bsMod); the crt channels stay in the NTT domain throughout.
//
// The resident keys carry the signs, bsMod^-1 and 2^32 (k_keys_from_words), so a
// slot is the Montgomery reduction of one 64-bit sum of four products: the
// three digits' and NTT(x2) times a constant.  The query side keeps the three
// digits of a slot and its b side by side (16 bytes), one gather per slot for
// the three digits of both components.
//
// What bounds it: load and store wavefronts (65 % busy, the digit gathers above all),
// issue (51 %) and the multiply pipe (41 %; ntt.cuh) together, with the keys (22 MiB
// per client) streaming from L2 or HBM beside it.  Batch of 64:
// 1.20 ms with one component per CTA, conditional-subtraction transforms and
// 64-bit Barrett reductions, 0.77 ms in this form.
#pragma once

#include <type_traits>

#include "ntt.cuh"
#include "pipeline.cuh"
#include "ptx.cuh"

namespace kspir {

struct BabyArgs {
    const uint32_t* dig;     // [3 ch][N][4]: the three digits and b of a slot, NTT form (crt channels: b * bsMod^-1)
    const uint16_t* perms;   // caller permutations [N1][N] (reference test-pir.cpp:92-93), lane order
    const uint16_t* sigma;   // [N1/2][N] slot permutation of X -> X^(5^(i+1)), lane order
    uint64_t* cipherbuf;     // [N][N1][2]
    uint32_t* interA;        // outputs of the intermediate rotation: a before the modswitch [2 ch][N], NTT form
    uint32_t* inter_dig;     // its b as the fourth word of the second half's dig
    uint32_t* inter_bs;      // its a mod bsMod [N], coefficient form
    int32_t N1;
    int32_t col_base;        // cipherbuf column of key index 0
    int32_t inter_idx;       // key index whose pre-modswitch state is exported, or -1
    int32_t cb_rm;           // 1: write cipherbuf rotation-major (see cipherbuf_rm_idx)
};

// Rotation-major cipherbuf, the layout the tensor-core scan's operand split
// reads: u32 [N1 columns][2 comp][2 primes][N slots], so that a rotation's
// CTA writes whole contiguous polynomials.  The reference layout
// ([N][N1][2] words, primes packed in one word) scatters every 4-byte store
// across a 16 * N1-byte stride; the CUDA-core scan streams it per slot.
__host__ __device__ __forceinline__ size_t cipherbuf_rm_idx(int col, int comp, int ch, int z) {
    return ((size_t)(col * 2 + comp) * 2 + ch) * kN + z;
}

// Rotation-major columns into the reference layout ([z][col] of four words: a q1,
// a q2, b q1, b q2), for the CUDA-core scan.  One CTA per 32 slots and 64 columns
// (grid.z: query): 128-byte rows in, 1 KiB pieces out, through 32 KiB of shared
// memory where slot z of column col sits at z ^ (col mod 32), so that both sides
// touch 32 distinct banks.
constexpr int kCbRowsZ = 32, kCbRowsCols = 64;
__global__ void __launch_bounds__(256) k_cipherbuf_rows(const uint32_t* __restrict__ rm, uint64_t* __restrict__ cbuf,
                                                        int N1, Batch bt) {
    __shared__ uint32_t V[kCbRowsCols * 4 * kCbRowsZ];
    const size_t wo = (size_t)(bt.slot0 + (int)blockIdx.z) * bt.ws_bytes;
    rm = shifted(rm, wo);
    uint4* out = reinterpret_cast<uint4*>(shifted(cbuf, wo));
    const int z0 = blockIdx.x * kCbRowsZ, c0 = blockIdx.y * kCbRowsCols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < kCbRowsCols * 4 / 8; i++) {
        const int row = warp + 8 * i;   // col * 4 + comp * 2 + ch
        V[row * kCbRowsZ + (lane ^ ((row >> 2) & 31))] = __ldcg(rm + ((size_t)c0 * 4 + row) * kN + z0 + lane);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kCbRowsZ * kCbRowsCols / 256; i++) {
        const int t = threadIdx.x + 256 * i, col = t % kCbRowsCols, z = t / kCbRowsCols;
        const uint32_t* v = V + col * 4 * kCbRowsZ + (z ^ (col & 31));
        out[(size_t)(z0 + z) * N1 + c0 + col] = make_uint4(v[0], v[kCbRowsZ], v[2 * kCbRowsZ], v[3 * kCbRowsZ]);
    }
}

constexpr int kBabyEll = 3;
constexpr int kBabyPolys1 = 2, kBabyPolys2 = 4;   // padded polynomials: x2 of one or two components, per prime

// Loads of the query-side inputs (digits, b): written by earlier kernels, so a
// stand-alone launch (CtaSync) reads them through L1 (their gathers reuse
// lines across the rotations on an SM); inside the fused answer kernel other
// CTAs write them during the launch, so those loads bypass L1.
template <class Sync, class T>
__device__ __forceinline__ T ld_query(const T* p) {
    if constexpr (std::is_same<Sync, CtaSync>::value) return __ldg(p);
    else return __ldcg(p);
}

// the permutation entries of a thread's coefficients u + 256 (4 v + w), w = 0..3
__device__ __forceinline__ void perm4(const uint16_t* __restrict__ p, int i, uint32_t* o) {
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(p) + i);
    o[0] = a.x & 0xffff; o[1] = a.x >> 16; o[2] = a.y & 0xffff; o[3] = a.y >> 16;
}

// sum_j d_j[perm] key_j of four coefficients: the vector of component `comp`
// added to acc; d: the gathered slots, key: [j][comp][...] at stride `jstride`
// vectors between digits
__device__ __forceinline__ void baby_mac4(uint64_t* acc, const uint4* d, const uint4* __restrict__ key, int jstride) {
#pragma unroll
    for (int j = 0; j < kBabyEll; j++) {
        const uint4 k = __ldg(key + (size_t)j * jstride);
        const uint32_t kw[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
        for (int w = 0; w < 4; w++) mad_wide_s(acc[w], j == 0 ? d[w].x : j == 1 ? d[w].y : d[w].z, kw[w]);
    }
}

// Rotation ki of one query by 512 threads, COMPS components: both (COMPS = 2),
// or the one given (1).  P: 2 COMPS padded polynomials.
//
//  1. bsMod part in the NTT domain, eight slots per thread;
//  2. x2 by the inverse transform mod bsMod, one component per thread group
//     (COMPS = 1: the second group waits), stored twice;
//  3. NTT_ch(x2), one prime per group: with COMPS = 2 both components of the
//     prime share one set of twiddle loads;
//  4. the crt products, the modswitch and the cipherbuf store, one prime per
//     group, sixteen slots per thread, one digit gather for both components.
template <int COMPS, class Sync>
__device__ __forceinline__ void baby_rotation(uint32_t* P, const BabyArgs& a, const ClientKeysDev& keys,
                                              const NttTables& tabs, const Batch& bt, int ki, int comp0) {
    const int g = thread_group(), u = threadIdx.x & (kNttGroup - 1);
    const bool inter = ki == a.inter_idx;
    // slot-0 workspace pointers: each use adds the query's offset
    const size_t wo = ws_off(bt), ko = key_off(bt);
    const uint16_t* perm = a.perms + (size_t)(ki + 1) * kN;
    const uint16_t* sig = a.sigma + (size_t)ki * kN;
    const uint4* dig = reinterpret_cast<const uint4*>(shifted(a.dig, wo));

    // 1. sum_j d_j key_j (+ NTT_bs(b)[sigma] for component b) mod bsMod
    {
        const ChanConst& cb = c_dev.ch[CH_BS];
        const uint4* kbs = reinterpret_cast<const uint4*>(shifted(keys.baby_bs, ko) + (size_t)ki * kBabyEll * 2 * kN);
#pragma unroll
        for (int vv = 0; vv < 2; vv++) {
            const int v = 2 * g + vv, i = v * kNttGroup + u;
            uint32_t pk[4];
            uint4 d[4];
            perm4(perm, i, pk);
#pragma unroll
            for (int w = 0; w < 4; w++) d[w] = ld_query<Sync>(dig + CH_BS * kN + pk[w]);
#pragma unroll
            for (int c = 0; c < COMPS; c++) {
                const int comp = COMPS == 2 ? c : comp0;
                uint64_t acc[4] = {0, 0, 0, 0};
                baby_mac4(acc, d, kbs + comp * (kN / 4) + i, 2 * kN / 4);
                uint32_t r[4];
#pragma unroll
                for (int w = 0; w < 4; w++) r[w] = mont_redc(acc[w], cb);
                if (comp == 1) {
                    perm4(sig, i, pk);
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        r[w] = canon_m1p2(r[w] + ld_query<Sync>(reinterpret_cast<const uint32_t*>(dig + CH_BS * kN + pk[w]) + 3), cb.q);
                        // the second half's b mod bsMod is this sum
                        if (inter) shifted(a.inter_dig, wo)[(size_t)(CH_BS * kN + u + kNttGroup * (4 * v + w)) * 4 + 3] = r[w];
                    }
                } else {
#pragma unroll
                    for (int w = 0; w < 4; w++) r[w] = canon_pm1(r[w], cb.q);
                }
#pragma unroll
                for (int w = 0; w < 4; w++) P[2 * c * kPadN + pidx(u) + (4 * v + w) * kPadGroupStep] = r[w];
            }
        }
    }

    // 2. x2, once for each prime
    {
        const int comp = COMPS == 2 ? g : comp0;
        uint32_t* S = P + (COMPS == 2 ? 2 * g : 0) * kPadN;
        uint32_t* bs_out = inter && comp == 0 ? shifted(a.inter_bs, wo) : nullptr;
        auto out = [&](int, int t, uint32_t x) {
            S[pidx(u) + t * kPadGroupStep] = x;
            S[kPadN + pidx(u) + t * kPadGroupStep] = x;
            if (bs_out) bs_out[u + kNttGroup * t] = x;
        };
        Sync::sync();
        if (COMPS == 2 || g == 0) group_ntt_inverse<1, GroupSync>(S, kPadN, tabs, CH_BS, u, out);
    }

    // 3.
    const int ch = g;
    uint32_t* S = P + ch * kPadN;
    Sync::sync();
    group_ntt_forward<COMPS, GroupSync, true>(S, 2 * kPadN, tabs, ch, u);   // x2 < bsMod < q / 14: signed, lazy

    // 4.
    const ChanConst& cc = c_dev.ch[ch];
    const uint4* kcrt = reinterpret_cast<const uint4*>(shifted(keys.baby_crt, ko) + (size_t)ki * kBabyEll * 4 * kN);
    const int col = a.col_base + ki;
    uint32_t* cb32 = reinterpret_cast<uint32_t*>(shifted(a.cipherbuf, wo));
    auto cb_at = [&](int comp, int k) -> uint32_t* {
        return cb32 + (a.cb_rm ? cipherbuf_rm_idx(col, comp, ch, k) : (((size_t)k * a.N1 + col) * 2 + comp) * 2 + ch);
    };
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int i = v * kNttGroup + u;
        uint32_t pk[4];
        uint4 d[4];
        perm4(perm, i, pk);
#pragma unroll
        for (int w = 0; w < 4; w++) d[w] = ld_query<Sync>(dig + ch * kN + pk[w]);
#pragma unroll
        for (int c = 0; c < COMPS; c++) {
            const int comp = COMPS == 2 ? c : comp0;
            uint64_t acc[4] = {0, 0, 0, 0};
#pragma unroll
            for (int w = 0; w < 4; w++)
                mad_wide_s(acc[w], S[2 * c * kPadN + pidx(u) + (4 * v + w) * kPadGroupStep], cc.xs);
            baby_mac4(acc, d, kcrt + (comp * 2 + ch) * (kN / 4) + i, 4 * kN / 4);
            uint32_t r[4];
            // below (3 q + 6.7 q) q / 2 / 2^32 + q / 2 < 0.9 q in magnitude
#pragma unroll
            for (int w = 0; w < 4; w++) r[w] = mont_redc(acc[w], cc);
            if (comp == 1) {
                perm4(sig, i, pk);
#pragma unroll
                for (int w = 0; w < 4; w++)
                    r[w] = canon_m1p2(r[w] + ld_query<Sync>(reinterpret_cast<const uint32_t*>(dig + ch * kN + pk[w]) + 3), cc.q);
            } else {
#pragma unroll
                for (int w = 0; w < 4; w++) r[w] = canon_pm1(r[w], cc.q);
            }
#pragma unroll
            for (int w = 0; w < 4; w++) *cb_at(comp, u + kNttGroup * (4 * v + w)) = r[w];
        }
    }
    if (inter) {
        // the state before the modswitch: a = out * bsMod + x2, and b * bsMod^-1 =
        // out + x2 * bsMod^-1 as the second half's b
#pragma unroll 1
        for (int t = 0; t < 16; t++) {
            const int k = u + kNttGroup * t;
#pragma unroll
            for (int c = 0; c < COMPS; c++) {
                const int comp = COMPS == 2 ? c : comp0;
                const uint32_t o = *cb_at(comp, k);   // this thread's own store
                const uint32_t x2 = canon_lazy(S[2 * c * kPadN + pidx(u) + t * kPadGroupStep], cc);
                if (comp == 0)
                    shifted(a.interA, wo)[ch * kN + k] = reduce64((uint64_t)o * kBsMod + x2, cc.q, cc.barrett);
                else
                    shifted(a.inter_dig, wo)[(size_t)(ch * kN + k) * 4 + 3] =
                        addmod(o, shoup_mul(x2, cc.bsinv, cc.bsinv_p, cc.q), cc.q);
            }
        }
    }
}

// Both components of a rotation per CTA (batches: one digit gather and one set
// of forward twiddles for both), or one (single queries: 126 CTAs instead of
// 63): blockIdx.x = ki, or 2 ki + comp; blockIdx.y = query of the batch.
template <int COMPS>
__global__ void __launch_bounds__(kNttThreads, 2) k_baby_rot(BabyArgs a, ClientKeysDev keys, NttTables tabs, Batch bt) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    pdl_launch_dependents();
    if (COMPS == 1) {
        warm_twiddles(tabs, CH_BS, NTT_INV, threadIdx.x, kNttThreads);
        warm_twiddles(tabs, thread_group(), NTT_FWD, threadIdx.x & (kNttGroup - 1), kNttGroup);
    }
    pdl_wait();   // the digits come from the previous kernel
    baby_rotation<COMPS, CtaSync>(reinterpret_cast<uint32_t*>(smem_raw), a, keys, tabs, bt,
                                  COMPS == 2 ? blockIdx.x : blockIdx.x >> 1, blockIdx.x & 1);
}

}  // namespace kspir

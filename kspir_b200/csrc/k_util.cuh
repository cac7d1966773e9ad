// Generic building blocks: batched transforms driven by job lists, residue
// composition into 64-bit words, and small element-wise helpers.
#pragma once

#include "common.cuh"
#include "ntt.cuh"
#include "pipeline.cuh"
#include "ptx.cuh"

namespace kspir {

// One transform: read N residues from src (stride 1), transform on channel
// `ch`, write to dst[k * dst_stride] (dst may equal src).
struct NttJob {
    const uint32_t* src;
    uint32_t* dst;
    int32_t ch;
    int32_t dst_stride;
};

// dynamic shared memory: one padded polynomial
constexpr int kNttJobSmem = kPadN * 4;

// The transform of one job by T threads (its first 256 run the transform; the
// caller synchronises nothing: the transform starts with a barrier).
template <bool INVERSE, class Sync, int T>
__device__ __forceinline__ void ntt_job_run(const NttJob& jb, const NttTables& tabs, uint32_t* s) {
    poly_to_smem<T>(s, jb.src);
    if (INVERSE) cta_ntt_inverse_m<1, Sync>(s, kPadN, tabs, jb.ch);
    else cta_ntt_forward_m<1, Sync>(s, kPadN, tabs, jb.ch);
    if (jb.dst_stride == 1) {
        poly_from_smem<T>(jb.dst, s);
    } else {
        for (int k = threadIdx.x; k < kN; k += T) jb.dst[(size_t)k * jb.dst_stride] = s[pidx(k)];
    }
}

template <bool INVERSE>
__global__ void __launch_bounds__(kNttGroup) k_ntt_jobs(const NttJob* __restrict__ jobs, NttTables tabs, Batch bt) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint32_t* s = reinterpret_cast<uint32_t*>(smem_raw);
    pdl_launch_dependents();
    NttJob jb = jobs[blockIdx.x];
    jb.src = shifted(jb.src, ws_off(bt));   // job lists address workspace slot 0
    jb.dst = shifted(jb.dst, ws_off(bt));
    warm_twiddles(tabs, jb.ch, INVERSE ? NTT_INV : NTT_FWD, threadIdx.x, kNttGroup);
    pdl_wait();
    ntt_job_run<INVERSE, CtaSync, kNttGroup>(jb, tabs, s);
}

// words[p][k] = canonical crtMod value of residues (res[p][0][k], res[p][1][k])
// for `polys` consecutive [2][N] residue polynomials.
__global__ void k_compose_words(const uint32_t* __restrict__ res, uint64_t* __restrict__ words, int polys) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= polys * kN) return;
    int p = idx / kN, k = idx % kN;
    const uint32_t* r = res + (size_t)p * 2 * kN;
    words[idx] = crt_compose_res(r[k], r[kN + k]);
}

// words[comp][k] = canonical crtMod value of column 0 of a cipherbuf in the
// reference layout ([N][N1][2] words of two residues): 64 KiB to copy out instead
// of the whole cipherbuf (8 MiB at N1 = 128).
__global__ void k_compose_column(const uint64_t* __restrict__ cipherbuf, uint64_t* __restrict__ words, int N1) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 2 * kN) return;
    const uint64_t v = cipherbuf[(size_t)(idx % kN) * N1 * 2 + idx / kN];
    words[idx] = crt_compose_res((uint32_t)v, (uint32_t)(v >> 32));
}

// Last kernel of an answer: the response words [nq][2][N] of its queries, the
// canonical words of the two residue polynomials `res` (a workspace pointer of
// slot 0), into device memory or the pinned staging of a host-buffer answer;
// err_out (or null) receives the error word of the launch's first slot.
__global__ void k_compose_resp(const uint32_t* __restrict__ res, uint64_t* resp, const int* errs, int* err_out, Batch bt) {
    pdl_wait();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx == 0 && err_out) *err_out = *reinterpret_cast<const volatile int*>(errs + (size_t)bt.slot0 * kErrStride);
    if (idx >= 2 * kN) return;
    const uint32_t* r = shifted(res, ws_off(bt)) + (size_t)(idx / kN) * 2 * kN;
    const int k = idx % kN;
    resp[(size_t)blockIdx.y * 2 * kN + idx] = crt_compose_res(__ldcg(r + k), __ldcg(r + kN + k));
}

// res[p][ch][k] = words[p][k] mod q_ch (ch = q1, q2) for `polys` polynomials.
__global__ void k_split_words(const uint64_t* __restrict__ words, uint32_t* __restrict__ res, int polys) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= polys * kN) return;
    int p = idx / kN, k = idx % kN;
    uint64_t v = words[idx];
    uint32_t* r = res + (size_t)p * 2 * kN;
    r[k] = mod_q1(v);
    r[kN + k] = mod_q2(v);
}

// Client keys from reference words (layouts of include/kspir_b200.h) into a
// key slot: baby rows 0-2 mod crtMod -> baby_crt (both primes), rows 3-5 mod
// bsMod -> baby_bs; giant, packing and RGSW -> both primes.  Each word is
// multiplied by its channel's factor (ChanConst) and centred, so that the
// kernels' signed sums reduce with mont_redc, and sits in lane order.  The
// words were checked canonical before.  One thread per four words of a
// polynomial that share a vector (k = u + 256 (4 v + w)).
__device__ __forceinline__ uint32_t key_word(uint64_t v, uint32_t factor, int ch) {
    const ChanConst& c = c_dev.ch[ch];
    return centre(reduce64((uint64_t)reduce64(v, c.q, c.barrett) * factor, c.q, c.barrett), c.q);
}

__global__ void k_keys_from_words(const uint64_t* __restrict__ baby, const uint64_t* __restrict__ giant,
                                  const uint64_t* __restrict__ packing, const uint64_t* __restrict__ rgsw,
                                  uint32_t* __restrict__ baby_crt, uint32_t* __restrict__ baby_bs,
                                  uint32_t* __restrict__ giant_res, uint32_t* __restrict__ packing_res,
                                  uint32_t* __restrict__ rgsw_res, int nbaby, int ngiant, int npack) {
    // polynomial index over [baby: nbaby * 6 * 2][giant: ngiant][packing: npack][rgsw: 8]
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long nb = (long)nbaby * 12, total = nb + ngiant + npack + 8;
    if (idx >= total * (kN / 4)) return;
    const int i = (int)(idx % (kN / 4)), u = i & (kNttGroup - 1), v = i / kNttGroup;
    long p = idx / (kN / 4);
    const uint64_t* src;
    uint32_t* dst;      // first prime (or bsMod)
    int ch0 = CH_Q1;
    int kind = 0;       // 0: kneg, 1: kbaby, 2: kpos
    if (p < nb) {
        const long bi = p / 12, j = (p / 2) % 6, comp = p % 2;
        src = baby + p * kN;
        if (j < 3) {
            dst = baby_crt + (((bi * 3 + j) * 2 + comp) * 2) * kN;
            kind = 1;
        } else {
            dst = baby_bs + ((bi * 3 + j - 3) * 2 + comp) * kN;
            ch0 = CH_BS;
        }
    } else if ((p -= nb) < ngiant) {
        src = giant + p * kN;
        dst = giant_res + p * 2 * kN;
    } else if ((p -= ngiant) < npack) {
        src = packing + p * kN;
        dst = packing_res + p * 2 * kN;
    } else {
        p -= npack;
        src = rgsw + p * kN;
        dst = rgsw_res + p * 2 * kN;
        kind = 2;
    }
    uint64_t w[4];
#pragma unroll
    for (int t = 0; t < 4; t++) w[t] = src[u + kNttGroup * (4 * v + t)];
    for (int ch = ch0; ch <= (ch0 == CH_BS ? CH_BS : CH_Q2); ch++) {
        const ChanConst& c = c_dev.ch[ch];
        const uint32_t f = kind == 0 ? c.kneg : kind == 1 ? c.kbaby : c.kpos;
        *reinterpret_cast<uint4*>(dst + (ch == CH_Q2 ? kN : 0) + 4 * i) =
            make_uint4(key_word(w[0], f, ch), key_word(w[1], f, ch), key_word(w[2], f, ch), key_word(w[3], f, ch));
    }
}

// Validation of caller words: flags[0] |= 1 when some word is >= its modulus.
__global__ void k_check_canonical(const uint64_t* __restrict__ words, size_t n, uint64_t modulus,
                                  int* __restrict__ flag) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (words[i] >= modulus) atomicOr(flag, 1);
}

}  // namespace kspir

// Database preprocessing on the device: the reference's database_tobsgsntt
// followed by database_tocrt (twosteps.cpp:42-179, crt.cpp:859-885), for every
// sub-database at once.
//
// Reference steps for sub-database `data` ([N][N/2] words < bsgsp = 65537):
//   1. diagonal rearrangement into rows R < N/2 (twosteps.cpp:64-74):
//        D[R][j]       = data[(j - R + N/2) mod N/2][j]          j < N/2
//        D[R][N-1-j]   = data[N-1 - ((j - R + N/2) mod N/2)][j]
//   2. slot permutation of row R = k N1 + i (twosteps.cpp:104-118):
//        temp[query_encode[j]] = D[R][j];  row[j] = temp[perm[i][j]]
//      Both are powers of 5 in the exponent: query_encode[c] is the slot of 5^c
//      (of -5^j for c = N-1-j) and perm[i] the automorphism by 5^i, so entry c of
//      D[R] lands in slot query_encode[c - i] (query_encode[N-1-(j-i)]), indices
//      mod N/2.  With c = rho + R (rho the data row of step 1), c - i =
//      rho + k N1: a data row's entries for consecutive R are consecutive in
//      memory, and go to the same slot.
//   3. inverse NTT mod bsgsp (HEXL, minimal root), lift to signed
//      (v > bsgsp/2: v + crtMod - bsgsp), forward NTT mod crtMod with
//      root_of_unity_crt (twosteps.cpp:156-176);
//   4. datacrt[z * N/2 + R] = (x mod q1) | (x mod q2) << 32 for slot z of row R
//      (crt.cpp:868-880).
// Steps 3-4 run per prime: the NTT mod crtMod reduced mod q1 (q2) is the NTT
// mod q1 (q2) of the signed lift, whose small words serve both primes.
#pragma once

#include "common.cuh"
#include "ntt.cuh"

namespace kspir {

// flag |= 1 when some of the n raw words is not below bsgsp.  Four 16-byte loads in
// flight per thread where the words are aligned.
__global__ void __launch_bounds__(256) k_check_raw(const uint64_t* __restrict__ words, size_t n, int* __restrict__ flag) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x, T = (size_t)gridDim.x * blockDim.x;
    bool bad = false;
    size_t i0 = 0;
    if ((uintptr_t)words % 16 == 0) {
        const uint4* v = reinterpret_cast<const uint4*>(words);
        const size_t full = n / 2 / (4 * T) * (4 * T);
        for (size_t i = t; i < full; i += 4 * T) {
            uint4 a[4];
#pragma unroll
            for (int k = 0; k < 4; k++) a[k] = __ldcs(v + i + k * T);
#pragma unroll
            for (int k = 0; k < 4; k++) bad |= (a[k].y | a[k].w) != 0 || a[k].x >= kP || a[k].z >= kP;
        }
        i0 = 2 * full;
    }
    for (size_t i = i0 + t; i < n; i += T) bad |= words[i] >= kP;
    if (bad) atomicOr(flag, 1);
}

// A CTA transforms two consecutive rows: it takes their words of a data row as
// one 16-byte piece, and writes their words for one slot as one 16-byte piece of
// datacrt (the CTA of the neighbouring pair runs beside it and fills the sector
// in L2).  One 256-thread group per row for the inverse, then per prime for the
// forward transforms of both rows (twiddles shared).  What bounds it is the
// multiply pipe (six transforms) and the load and store of words 16 KiB
// apart, one address each (LSU wavefronts 57 % busy); two CTAs per SM overlap the
// two.  r = 16, with the validation pass: 1.88 ms; 2.02 ms with four rows per CTA
// at one CTA per SM; 2.4 ms with a permutation table and a gather of 8-byte words
// per row.
constexpr int kDbRowsPerCta = 2;
constexpr int kDbRowsThreads = kDbRowsPerCta * kNttGroup;
constexpr int kDbRowsSmem = 2 * kDbRowsPerCta * kPadN * 4;   // the rows mod q1, then mod q2

// grid (N/2 / 2, sub-databases).
//   raw   [sub][N][N/2] words < bsgsp (validated by the caller); VEC: 16-byte aligned
//   qenc  [N] query_encode
//   out   [sub][N][N/2] datacrt words (database_tocrt applied)
//   rows  ROWS: also [sub][N/2][N] rows mod crtMod, database_tobsgsntt's own
//         output (its `result`)
template <bool ROWS, bool VEC>
__global__ void __launch_bounds__(kDbRowsThreads, 2)
k_db_rows(const uint64_t* __restrict__ raw, const uint16_t* __restrict__ qenc, uint64_t* __restrict__ out,
          uint64_t* __restrict__ rows, int N1, NttTables tabs) {
    static_assert(kDbRowsPerCta == 2, "pieces of two words, one group per prime");
    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint32_t* S = reinterpret_cast<uint32_t*>(smem_raw);          // [prime][row][kPadN]
    constexpr int H = kN / 2;
    const int R0 = blockIdx.x * kDbRowsPerCta;
    const size_t sub = (size_t)blockIdx.y * kN * H;
    const int tid = threadIdx.x, g = thread_group(), u = tid & (kNttGroup - 1);
    const int kN1 = R0 / N1 * N1;   // k N1: N1 is even

    // steps 1 and 2: i < H stands for data row rho (entries c), i >= H for row
    // N-1-rho (entries N-1-j).  A warp's rows have one parity, so that the piece of
    // two words starts on a 16-byte boundary for all its lanes or for none.
#pragma unroll
    for (int i = tid; i < kN; i += kDbRowsThreads) {
        const int w = i & (H - 1), rho = (w & ~63) | ((w & 31) << 1) | ((w >> 5) & 1);
        const bool lower = i < H;
        const uint64_t* d = raw + sub + (size_t)(lower ? rho : kN - 1 - rho) * H;
        const int c0 = (rho + R0) & (H - 1), e = (rho + kN1) & (H - 1);
        uint32_t v[2];
        if (VEC && !(rho & 1)) {
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(d + c0));
            v[0] = a.x; v[1] = a.z;
        } else {
            v[0] = (uint32_t)__ldg(d + c0);
            v[1] = (uint32_t)__ldg(d + ((c0 + 1) & (H - 1)));
        }
        const int p = pidx(__ldg(qenc + (lower ? e : kN - 1 - e)));
        S[p] = v[0];
        S[kPadN + p] = v[1];
    }
    __syncthreads();

    // step 3: row g's inverse, lifted to signed, once for each prime
    uint32_t* row = S + g * kPadN;
    auto lift = [&](int, int t, uint32_t v) {
        const uint32_t s = v > kP / 2 ? v - kP : v;
        row[pidx(u) + t * kPadGroupStep] = s;
        row[kDbRowsPerCta * kPadN + pidx(u) + t * kPadGroupStep] = s;
    };
    group_ntt_inverse<1, GroupSync>(row, kPadN, tabs, CH_P, u, lift);
    __syncthreads();
    group_ntt_forward<2, GroupSync, false>(S + g * kDbRowsPerCta * kPadN, kPadN, tabs, g, u);   // prime g
    __syncthreads();

    const uint32_t* s1 = S;
    const uint32_t* s2 = S + kDbRowsPerCta * kPadN;
    if (ROWS) {
        // the canonical value mod crtMod of each slot, row by row (coalesced)
#pragma unroll
        for (int t = 0; t < kDbRowsPerCta; t++) {
            uint64_t* o = rows + sub + (size_t)(R0 + t) * kN;
            for (int z = tid; z < kN; z += kDbRowsThreads)
                o[z] = crt_compose_res(s1[t * kPadN + pidx(z)], s2[t * kPadN + pidx(z)]);
        }
    }
    // step 4: slot z of rows R0, R0 + 1 at datacrt[z * N/2 + R0]
    uint64_t* o = out + sub + R0;
#pragma unroll
    for (int z = tid; z < kN; z += kDbRowsThreads) {
        const int pz = pidx(z);
        *reinterpret_cast<uint4*>(o + (size_t)z * H) = make_uint4(s1[pz], s2[pz], s1[kPadN + pz], s2[kPadN + pz]);
    }
}

// database_tocrt alone (crt.cpp:859-885) on rows mod crtMod of one or more
// sub-databases: datacrt[z][R] = (x mod q1) | (x mod q2) << 32 for
// x = rows[R][z], any 64-bit x (the reference's Barrett reduction is exact
// for every 64-bit input).  32 x 32 tiles through shared memory; grid
// (N / 32, N/2 / 32, sub-databases), 32 x 8 threads.
__global__ void k_db_tocrt(const uint64_t* __restrict__ rows, uint64_t* __restrict__ datacrt) {
    __shared__ uint64_t tile[32][33];
    const size_t sub = (size_t)blockIdx.z * kN * (kN / 2);
    const int z0 = blockIdx.x * 32, R0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
    for (int i = ty; i < 32; i += 8) {
        const uint64_t x = rows[sub + (size_t)(R0 + i) * kN + z0 + tx];
        tile[i][tx] = mod_q1(x) | (uint64_t)mod_q2(x) << 32;
    }
    __syncthreads();
#pragma unroll
    for (int i = ty; i < 32; i += 8) datacrt[sub + (size_t)(z0 + i) * (kN / 2) + R0 + tx] = tile[tx][i];
}

}  // namespace kspir

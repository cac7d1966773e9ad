// Device-side arithmetic shared by every KsPIR kernel.
//
// Representation.  The reference computes modulo crtMod = q1*q2 (56 bits,
// reference src/crt.h:16-18) and bsMod (24 bits, crt.h:32) on 64-bit words
// through HEXL.  Every HEXL operation on the answer path is exact modular
// arithmetic with canonical outputs, so a value mod crtMod is held here as its
// two 28-bit residues (mod q1, mod q2) in 32-bit words, and bsMod is a third
// 32-bit channel.  The NTT with root_of_unity_crt (crt.h:81) is, residue by
// residue, the NTT with psi mod q1 and psi mod q2.  A canonical 56-bit (or
// crtMod*bsMod 80-bit) integer is formed by CRT only where the reference
// leaves modular arithmetic: the gadget decompositions and the response words.
#pragma once

#include <stdint.h>

namespace kspir {

constexpr int kN = 4096;          // ring dimension, reference params.h:16
constexpr int kLogN = 12;
constexpr uint32_t kQ1 = 268369921u;   // crt.h:16
constexpr uint32_t kQ2 = 249561089u;   // crt.h:17
constexpr uint64_t kCrtMod = (uint64_t)kQ1 * kQ2;
constexpr uint32_t kBsMod = 16760833u; // crt.h:32
constexpr uint64_t kBsModInvCrt = 51309461009346113ull;  // bsMod^-1 mod crtMod, crt.h:33
constexpr uint32_t kCrtModInvBs = 3920321u;              // crtMod^-1 mod bsMod, crt.h:34

constexpr uint32_t kP = 65537u;        // plaintext modulus bsgsp, params.h:94
constexpr uint32_t kAuxMod = 268361729u;   // auxiliary modulus of the offline key derivation, crt.h:37

// channels of the RNS representation (p: only for the database preprocessing;
// the last three only for the offline key derivation: crtBaMod = bsMod * auxMod
// transformed with root_of_unity_crt_bamod, crt.h:82, as its two residues, and
// auxMod with HEXL's minimal root)
enum Chan : int { CH_Q1 = 0, CH_Q2 = 1, CH_BS = 2, CH_P = 3, CH_BA_BS = 4, CH_BA_AUX = 5, CH_AUX = 6, CH_COUNT = 7 };

// Per-channel constants, filled on the host (context.cu) and kept in
// __constant__ memory.
struct ChanConst {
    uint32_t q;
    uint32_t nq;           // -q mod 2^32
    uint64_t barrett;      // floor(2^64 / q)
    uint32_t rq;           // round(2^32 / q)
    uint32_t qinv;         // q^-1 mod 2^32 (mont_redc)
    uint32_t bsinv, bsinv_p;  // bsMod^-1 mod crtMod, reduced mod q (crt channels only)
    // factors of the resident keys (k_keys_from_words), canonical: -2^32 (giant,
    // packing; bsMod rows of the baby keys), 2^32 (RGSW), -bsMod^-1 2^32 (baby)
    uint32_t kneg, kpos, kbaby;
    uint32_t xs;           // kbaby, centred
    // transform twiddles every thread shares (ntt.cuh), as {w, round(w 2^32 / q)}
    // with w centred: the first forward pass (entry m + i: psi^brv(m + i), m = 1,
    // 2, 4, 8), the powers 0..7 of psi^(-2N/16) of the inverse's 16-point
    // transforms, and psi^(-256 t) of its outputs
    uint2 fw[16], iw[8], ic[16];
};

struct DevConst {
    ChanConst ch[CH_COUNT];
    uint32_t q1inv_mod_q2;     // q1^-1 mod q2 (Garner)
    uint32_t q1inv_mod_q2_p;
};

// Defined here: the library is one translation unit (kspir.cu includes every
// kernel header), so no relocatable device code is needed.
__constant__ DevConst c_dev;

// ---------------------------------------------------------------------------
// 32-bit residue arithmetic (q < 2^28)

__device__ __forceinline__ uint32_t shoup_lazy(uint32_t x, uint32_t w, uint32_t wp, uint32_t q) {
    // x*w mod q in [0, 2q) for any 32-bit x; wp = floor(w * 2^32 / q)
    uint32_t t = __umulhi(x, wp);
    return x * w - t * q;
}

// Conditional subtractions as an unsigned minimum: for x < 2m, x - m wraps
// above x exactly when x < m.
__device__ __forceinline__ uint32_t shoup_mul(uint32_t x, uint32_t w, uint32_t wp, uint32_t q) {
    const uint32_t r = shoup_lazy(x, w, wp, q);
    return umin(r, r - q);
}

// Exact reduction of any 64-bit p by Barrett with barrett = floor(2^64 / q):
// qh = floor(p * barrett / 2^64) is floor(p / q) or one less (p * barrett
// falls short of p * 2^64 / q by less than p < 2^64), so p - qh q is in
// [0, 2q) and is computed in 32 bits.
__device__ __forceinline__ uint32_t reduce64(uint64_t p, uint32_t q, uint64_t barrett) {
    const uint32_t qh = (uint32_t)__umul64hi(p, barrett);
    const uint32_t r = (uint32_t)p - qh * q;
    return umin(r, r - q);
}

// ---------------------------------------------------------------------------
// signed lazy words of the transforms: any word below 8 q in magnitude
// (q < 2^28) stands for its residue

// y w mod q within (-|y| / 2^33, 1 + |y| / 2^33) q; w = {centred, round(w 2^32 / q)}.
// The quotient is the floor: rounding it would keep products within +-q/2, but the
// rounding addend costs two additions beside the mul.hi (the wide
// multiply-add is split), more than the few reductions that the wider
// range needs.
__device__ __forceinline__ uint32_t mul_lazy(uint32_t y, uint2 w, uint32_t nq) {
    return y * w.x + (uint32_t)__mulhi((int)y, (int)w.y) * nq;
}

// decimation-in-time butterfly: (X + wY, X - wY); widens a range of +-B q to
// +-(1.03125 B + 1) q
__device__ __forceinline__ void bfly(uint32_t& X, uint32_t& Y, uint2 w, uint32_t nq) {
    const uint32_t s = Y * w.x + X + (uint32_t)__mulhi((int)Y, (int)w.y) * nq;
    Y = 2 * X - s;
    X = s;
}

// to within (-0.11, 1.11) q
__device__ __forceinline__ uint32_t reduce_lazy(uint32_t x, uint32_t rq, uint32_t nq) {
    return x + (uint32_t)__mulhi((int)x, (int)rq) * nq;
}

// +-6 q to +-3 q; +-8 q to +-2 q
__device__ __forceinline__ uint32_t fold6(uint32_t x, uint32_t q) { return umin(x, x + 6 * q) - 3 * q; }
__device__ __forceinline__ uint32_t fold8(uint32_t x, uint32_t q) {
    const uint32_t r = umin(x, x + 8 * q);
    return umin(r, r - 4 * q) - 2 * q;
}

// p 2^-32 mod q within +-(|p| / 2^32 + q/2) for a signed 64-bit p (Montgomery: the
// low words of p and m q are equal).  Two multiplies, where an exact 64-bit
// Barrett reduction takes about fourteen instructions; the resident keys
// carry the factor 2^32.
__device__ __forceinline__ uint32_t mont_redc(uint64_t p, const ChanConst& c) {
    const uint32_t m = (uint32_t)p * c.qinv;
    return (uint32_t)(p >> 32) - (uint32_t)__mulhi((int)m, (int)c.q);
}

// a word in (-q, q), (-q, 2q), (-2q, 2q) or (-4q, 4q) to [0, q)
__device__ __forceinline__ uint32_t canon_pm1(uint32_t x, uint32_t q) { return umin(x, x + q); }
__device__ __forceinline__ uint32_t canon_m1p2(uint32_t x, uint32_t q) {
    const uint32_t r = umin(x, x + q);
    return umin(r, r - q);
}

__device__ __forceinline__ uint32_t canon_pm2(uint32_t x, uint32_t q) {
    const uint32_t r = umin(x, x + 2 * q);
    return umin(r, r - q);
}
__device__ __forceinline__ uint32_t canon_pm4(uint32_t x, uint32_t q) {
    uint32_t r = umin(x, x + 4 * q);
    r = umin(r, r - 2 * q);
    return umin(r, r - q);
}

// to [0, q)
__device__ __forceinline__ uint32_t canon_lazy(uint32_t x, const ChanConst& c) {
    return canon_m1p2(reduce_lazy(x, c.rq, c.nq), c.q);
}

// a canonical residue to [-q/2, q/2]
__device__ __forceinline__ uint32_t centre(uint32_t x, uint32_t q) {
    const uint32_t h = q >> 1, u = x + h;
    return umin(u, u - q) - h;
}

__device__ __forceinline__ uint32_t mulmod(uint32_t a, uint32_t b, int ch) {
    return reduce64((uint64_t)a * b, c_dev.ch[ch].q, c_dev.ch[ch].barrett);
}

__device__ __forceinline__ uint32_t addmod(uint32_t a, uint32_t b, uint32_t q) {
    const uint32_t s = a + b;
    return umin(s, s - q);
}

__device__ __forceinline__ uint32_t submod(uint32_t a, uint32_t b, uint32_t q) {
    const uint32_t d = a - b;   // wraps when a < b, and d + q is then the residue
    return umin(d, d + q);
}

// A signed small integer (|v| < q) as a canonical residue.
__device__ __forceinline__ uint32_t signed_to_res(int64_t v, uint32_t q) {
    const uint32_t u = (uint32_t)v;   // above 2^32 - q exactly when v < 0, and u + q then wraps to v + q
    return umin(u, u + q);
}

// ---------------------------------------------------------------------------
// crtMod <-> residues

// canonical value mod crtMod from its residues (Garner)
__device__ __forceinline__ uint64_t crt_compose_res(uint32_t r1, uint32_t r2) {
    const uint32_t r1m = umin(r1, r1 - kQ2);             // r1 mod q2 (q1 < 2 q2)
    const uint32_t d = submod(r2, r1m, kQ2);             // (r2 - r1) mod q2
    uint32_t t = shoup_mul(d, c_dev.q1inv_mod_q2, c_dev.q1inv_mod_q2_p, kQ2);
    return (uint64_t)r1 + (uint64_t)kQ1 * t;
}

// unsigned minimum for code compiled for the host as well
__host__ __device__ __forceinline__ uint32_t min_u32(uint32_t a, uint32_t b) { return a < b ? a : b; }

// x mod q, exact for every 64-bit x = xl + 2^32 xh, q one of the crt primes; c32 =
// 2^32 mod q, mu = floor(2^59 / q).  The high word is brought below 2^29.1 with its
// quotient by 2^28 (q is within 7 % of it), so y = (its residue) 2^32 + xl is below
// 2^57.1; the estimate umulhi(y >> 27, mu) of y / q falls short by less than 1.8
// (0.26 from mu, 0.54 from the shift, 1 from its floor), so one conditional
// subtraction finishes.
__host__ __device__ __forceinline__ uint32_t mod28(uint64_t x, uint32_t q, uint32_t c32, uint32_t mu) {
    const uint32_t xh = (uint32_t)(x >> 32);
    const uint32_t r = xh - (xh >> 28) * q;
    const uint64_t y = (uint64_t)r * c32 + (uint32_t)x;
    const uint32_t qh = (uint32_t)(((uint64_t)(uint32_t)(y >> 27) * mu) >> 32);
    const uint32_t t = (uint32_t)y - qh * q;   // in [0, 1.8 q)
    return min_u32(t, t - q);
}

__device__ __forceinline__ uint32_t mod_q1(uint64_t v) { return reduce64(v, kQ1, c_dev.ch[CH_Q1].barrett); }
__device__ __forceinline__ uint32_t mod_q2(uint64_t v) { return reduce64(v, kQ2, c_dev.ch[CH_Q2].barrett); }
__device__ __forceinline__ uint32_t mod_bs(uint64_t v) { return reduce64(v, kBsMod, c_dev.ch[CH_BS].barrett); }

// ---------------------------------------------------------------------------
// 128-bit helpers (hi:lo pairs)

struct u128 { uint64_t lo, hi; };

__device__ __forceinline__ u128 mul_64x64(uint64_t a, uint64_t b) {
    u128 r; r.lo = a * b; r.hi = __umul64hi(a, b); return r;
}

__device__ __forceinline__ u128 add128(u128 a, u128 b) {
    u128 r; r.lo = a.lo + b.lo; r.hi = a.hi + b.hi + (r.lo < a.lo ? 1 : 0); return r;
}

__device__ __forceinline__ u128 sub128(u128 a, u128 b) {
    u128 r; r.lo = a.lo - b.lo; r.hi = a.hi - b.hi - (a.lo < b.lo ? 1 : 0); return r;
}

__device__ __forceinline__ bool gt128(u128 a, u128 b) {
    return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo);
}

__device__ __forceinline__ u128 shr128(u128 a, int s) {  // 0 < s < 64
    u128 r; r.lo = (a.lo >> s) | (a.hi << (64 - s)); r.hi = a.hi >> s; return r;
}

// ---------------------------------------------------------------------------
// automorphism X -> X^g, coefficient domain, as a gather:
// out[k] = +-in[i] with i*g = k or k+N (mod 2N).  `neg_canonical` selects the
// negation: the reference's automorphic_rns writes 0 for -0 (twosteps.cpp:776-778);
// the inline loops of evalAutoRNSCRT / evalAuto write q (twosteps.cpp:629-630,
// answer.cpp:606-607).  Downstream every consumer treats q exactly like 0, so
// the kernels only need the canonical form.
__device__ __forceinline__ int auto_src(int k, uint32_t ginv, bool* neg) {
    uint32_t i0 = ((uint32_t)k * ginv) & (2 * kN - 1);
    *neg = i0 >= (uint32_t)kN;
    return (int)(i0 & (kN - 1));
}

// q - x, and 0 for x = 0 (0 - x wraps above q - x for every other x)
__device__ __forceinline__ uint32_t negmod(uint32_t x, uint32_t q) { return umin(q - x, 0u - x); }

// acc += a * b, signed
__device__ __forceinline__ void mad_wide_s(uint64_t& acc, uint32_t a, uint32_t b) {
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}

// acc += a * b with a 32x32->64-bit product, as one fused wide multiply-add
__device__ __forceinline__ void mad_wide(uint64_t& acc, uint32_t a, uint32_t b) {
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}

}  // namespace kspir

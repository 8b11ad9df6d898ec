// Montgomery prime-field arithmetic on 32-bit limbs for sm_100a.
//
// One template serves the BN254 base field (8 limbs) and the BLS12-381 base
// field (12 limbs); the constants come from params.cuh.  The hot routine is
// the CIOS Montgomery product (Koc, Acar, Kaliski 1996) written as explicit
// PTX carry chains.  fe_mul_body_eo (the default) splits each row into an
// even-index and an odd-index chain that run independently; fe_mul_body is
// the straight form (four chains of N multiply-adds per row, 4N+3
// instructions, accumulator in N+1 registers).  One out-of-line copy of the
// product per kernel keeps the hot loops within the instruction cache.
// Carry chains are written as asm volatile so the compiler keeps their order
// (the carry flag is invisible to it).
// Bounds: both moduli satisfy 4p < 2^(32N), so for inputs below 2p the
// accumulator stays below 2^(32(N+1)) (no carry is ever dropped) and the
// result before the last conditional subtraction is below 2p.
//
// Role in the reference: the Metal field kernels (Shaders/fields/bn254_fp.metal
// :134-233, Shaders/fields/bls12381_fq.metal:160-264) and the C CIOS kernels
// (NeonFieldOps/bn254_msm.c:38-267); same arithmetic, new implementation.
#pragma once
#include <cstdint>
#include "params.cuh"

namespace zkmsm {

template <class P>
struct Fe {
    uint32_t v[P::N];
};

#define ZK_DEV __device__ __forceinline__

// ---------------------------------------------------------------- helpers

template <class P>
ZK_DEV void fe_set_zero(Fe<P>& r) {
#pragma unroll
    for (int i = 0; i < P::N; i++) r.v[i] = 0;
}

template <class P>
ZK_DEV void fe_set_one(Fe<P>& r) {
#pragma unroll
    for (int i = 0; i < P::N; i++) r.v[i] = P::ONE(i);
}

template <class P>
ZK_DEV bool fe_is_zero(const Fe<P>& a) {
    uint32_t t = 0;
#pragma unroll
    for (int i = 0; i < P::N; i++) t |= a.v[i];
    return t == 0;
}

template <class P>
ZK_DEV bool fe_eq(const Fe<P>& a, const Fe<P>& b) {
    uint32_t t = 0;
#pragma unroll
    for (int i = 0; i < P::N; i++) t |= a.v[i] ^ b.v[i];
    return t == 0;
}

// r = a - p if a >= p else a   (a < 2p)
template <class P>
ZK_DEV void fe_reduce_once(Fe<P>& r, const Fe<P>& a) {
    constexpr int N = P::N;
    uint32_t d[N], borrow;
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(d[0]) : "r"(a.v[0]), "r"(P::P(0)));
#pragma unroll
    for (int i = 1; i < N; i++)
        asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(d[i]) : "r"(a.v[i]), "r"(P::P(i)));
    asm volatile("subc.u32 %0, 0, 0;" : "=r"(borrow));
#pragma unroll
    for (int i = 0; i < N; i++) r.v[i] = borrow ? a.v[i] : d[i];
}

// r = a + b mod p  (a, b < p)
template <class P>
ZK_DEV void fe_add(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
    constexpr int N = P::N;
    Fe<P> s;
    asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(s.v[0]) : "r"(a.v[0]), "r"(b.v[0]));
#pragma unroll
    for (int i = 1; i < N; i++)
        asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(s.v[i]) : "r"(a.v[i]), "r"(b.v[i]));
    // 2p < 2^(32N): no carry out of the top limb
    fe_reduce_once(r, s);
}

// r = a - b mod p  (a, b < p)
template <class P>
ZK_DEV void fe_sub(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
    constexpr int N = P::N;
    uint32_t d[N], mask;
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(d[0]) : "r"(a.v[0]), "r"(b.v[0]));
#pragma unroll
    for (int i = 1; i < N; i++)
        asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(d[i]) : "r"(a.v[i]), "r"(b.v[i]));
    asm volatile("subc.u32 %0, 0, 0;" : "=r"(mask));  // 0 or 0xffffffff
    asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r.v[0]) : "r"(d[0]), "r"(P::P(0) & mask));
#pragma unroll
    for (int i = 1; i < N - 1; i++)
        asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r.v[i]) : "r"(d[i]), "r"(P::P(i) & mask));
    asm volatile("addc.u32 %0, %1, %2;" : "=r"(r.v[N - 1]) : "r"(d[N - 1]), "r"(P::P(N - 1) & mask));
}

template <class P>
ZK_DEV void fe_dbl(Fe<P>& r, const Fe<P>& a) { fe_add(r, a, a); }

// r = -a mod p
template <class P>
ZK_DEV void fe_neg(Fe<P>& r, const Fe<P>& a) {
    Fe<P> z;
    fe_set_zero(z);
    fe_sub(r, z, a);
}

// r = a*b / 2^(32N) mod p, canonical (a, b < p; also correct mod p for a, b < 2p)
template <class P>
ZK_DEV void fe_mul_body(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
    constexpr int N = P::N;
    uint32_t t[N + 1];
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint32_t bi = b.v[i];
        if (i == 0) {
#pragma unroll
            for (int j = 0; j < N; j++) t[j] = a.v[j] * bi;
            asm volatile("mad.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[1]) : "r"(a.v[0]), "r"(bi));
#pragma unroll
            for (int j = 1; j < N - 1; j++)
                asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[j + 1]) : "r"(a.v[j]), "r"(bi));
            asm volatile("madc.hi.u32 %0, %1, %2, 0;" : "=r"(t[N]) : "r"(a.v[N - 1]), "r"(bi));
        } else {
            asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(t[0]) : "r"(a.v[0]), "r"(bi));
#pragma unroll
            for (int j = 1; j < N; j++)
                asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(t[j]) : "r"(a.v[j]), "r"(bi));
            asm volatile("addc.u32 %0, 0, 0;" : "=r"(t[N]));
            asm volatile("mad.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[1]) : "r"(a.v[0]), "r"(bi));
#pragma unroll
            for (int j = 1; j < N - 1; j++)
                asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[j + 1]) : "r"(a.v[j]), "r"(bi));
            asm volatile("madc.hi.u32 %0, %1, %2, %0;" : "+r"(t[N]) : "r"(a.v[N - 1]), "r"(bi));
        }
        const uint32_t m = t[0] * P::N0R();
        asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(t[0]) : "r"(m), "r"(P::P(0)));
#pragma unroll
        for (int j = 1; j < N; j++)
            asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(t[j]) : "r"(m), "r"(P::P(j)));
        asm volatile("addc.u32 %0, %0, 0;" : "+r"(t[N]));
        asm volatile("mad.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[1]) : "r"(m), "r"(P::P(0)));
#pragma unroll
        for (int j = 1; j < N - 1; j++)
            asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[j + 1]) : "r"(m), "r"(P::P(j)));
        asm volatile("madc.hi.u32 %0, %1, %2, %0;" : "+r"(t[N]) : "r"(m), "r"(P::P(N - 1)));
        // divide by 2^32: t[0] is zero now
#pragma unroll
        for (int j = 0; j < N; j++) t[j] = t[j + 1];
    }
    Fe<P> s;
#pragma unroll
    for (int j = 0; j < N; j++) s.v[j] = t[j];
    fe_reduce_once(r, s);
}


// Even/odd-split CIOS: a*b_i = E + 2^32*O where E holds the products a_j*b_i
// of even j (low word at limb j, high word at limb j+1) and O those of odd j
// shifted down one limb, so each is one carry chain without collisions and
// the two chains of a phase are independent.  State t = e + 2^32*o; after the
// reduction step e_0 = 0 and t/2^32 = (e >> 32) + o is re-split as
// e' = o + e_1 (the carry of that one addition enters the next odd chain,
// whose limb 0 has the same weight) and o' = e >> 64 (a register renaming).
// Bounds as for fe_mul_body (validated by emulating this exact schedule).
template <class P>
ZK_DEV void fe_mul_body_eo(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
    constexpr int N = P::N;
    uint32_t e[N + 1], o[N + 1];
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint32_t bi = b.v[i];
        if (i == 0) {
#pragma unroll
            for (int j = 0; j < N; j += 2) {
                e[j] = a.v[j] * bi;
                e[j + 1] = __umulhi(a.v[j], bi);
                o[j] = a.v[j + 1] * bi;
                o[j + 1] = __umulhi(a.v[j + 1], bi);
            }
            e[N] = 0;
            o[N] = 0;
        } else {
            uint32_t x[N + 1], y[N + 1];
            asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(x[0]) : "r"(o[0]), "r"(e[1]));
#pragma unroll
            for (int j = 0; j < N; j += 2) {
                const uint32_t slo = j + 2 < N ? e[j + 2] : e[N];
                const uint32_t shi = j + 3 < N ? e[j + 3] : 0u;
                asm volatile("madc.lo.cc.u32 %0, %1, %2, %3;" : "=r"(y[j]) : "r"(a.v[j + 1]), "r"(bi), "r"(slo));
                if (j + 2 < N)
                    asm volatile("madc.hi.cc.u32 %0, %1, %2, %3;" : "=r"(y[j + 1]) : "r"(a.v[j + 1]), "r"(bi), "r"(shi));
                else
                    asm volatile("madc.hi.u32 %0, %1, %2, %3;" : "=r"(y[j + 1]) : "r"(a.v[j + 1]), "r"(bi), "r"(shi));
            }
            y[N] = 0;
#pragma unroll
            for (int j = 1; j <= N; j++) x[j] = o[j];
            asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(x[0]) : "r"(a.v[0]), "r"(bi));
            asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(x[1]) : "r"(a.v[0]), "r"(bi));
#pragma unroll
            for (int j = 2; j < N; j += 2) {
                asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(x[j]) : "r"(a.v[j]), "r"(bi));
                asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(x[j + 1]) : "r"(a.v[j]), "r"(bi));
            }
            asm volatile("addc.u32 %0, %0, 0;" : "+r"(x[N]));
#pragma unroll
            for (int j = 0; j <= N; j++) {
                e[j] = x[j];
                o[j] = y[j];
            }
        }
        const uint32_t m = e[0] * P::N0R();
        asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(e[0]) : "r"(m), "r"(P::P(0)));
        asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(e[1]) : "r"(m), "r"(P::P(0)));
#pragma unroll
        for (int j = 2; j < N; j += 2) {
            asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(e[j]) : "r"(m), "r"(P::P(j)));
            asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(e[j + 1]) : "r"(m), "r"(P::P(j)));
        }
        asm volatile("addc.u32 %0, %0, 0;" : "+r"(e[N]));
        asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(o[0]) : "r"(m), "r"(P::P(1)));
        asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(o[1]) : "r"(m), "r"(P::P(1)));
#pragma unroll
        for (int j = 2; j < N; j += 2) {
            asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(o[j]) : "r"(m), "r"(P::P(j + 1)));
            asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(o[j + 1]) : "r"(m), "r"(P::P(j + 1)));
        }
        asm volatile("addc.u32 %0, %0, 0;" : "+r"(o[N]));
    }
    // t = (e >> 32) + o, below 2p
    Fe<P> s;
    asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(s.v[0]) : "r"(e[1]), "r"(o[0]));
#pragma unroll
    for (int j = 1; j < N - 1; j++)
        asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(s.v[j]) : "r"(e[j + 1]), "r"(o[j]));
    asm volatile("addc.u32 %0, %1, %2;" : "=r"(s.v[N - 1]) : "r"(e[N]), "r"(o[N - 1]));
    fe_reduce_once(r, s);
}

#ifndef ZKMSM_MUL_OUTLINE
#define ZKMSM_MUL_OUTLINE 1
#endif
#ifndef ZKMSM_MUL_EO
#define ZKMSM_MUL_EO 1
#endif

// One out-of-line copy of the product per kernel keeps the hot loops inside
// the instruction cache (arguments and result travel in registers).
template <class P>
__device__ __noinline__ Fe<P> fe_mul_ool(const Fe<P> a, const Fe<P> b) {
    Fe<P> r;
#if ZKMSM_MUL_EO
    fe_mul_body_eo(r, a, b);
#else
    fe_mul_body(r, a, b);
#endif
    return r;
}

template <class P>
ZK_DEV void fe_mul(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
#if ZKMSM_MUL_OUTLINE
    r = fe_mul_ool(a, b);
#elif ZKMSM_MUL_EO
    fe_mul_body_eo(r, a, b);
#else
    fe_mul_body(r, a, b);
#endif
}

// A square is a product: with 32-bit limbs the CIOS form cannot use the
// symmetry, and separating product and reduction (to use it) breaks the
// register pairing that lets each lo/hi pair issue as one instruction.
template <class P>
ZK_DEV void fe_sqr(Fe<P>& r, const Fe<P>& a) { fe_mul(r, a, a); }

// integer -> Montgomery form (a < p)
template <class P>
ZK_DEV void fe_to_mont(Fe<P>& r, const Fe<P>& a) {
    Fe<P> r2;
#pragma unroll
    for (int i = 0; i < P::N; i++) r2.v[i] = P::R2(i);
    fe_mul(r, a, r2);
}

// Montgomery form -> integer: a * R^-1 mod p by N reduction rounds alone
// (the product with 1 that a Montgomery multiplication would form is
// skipped).  Each round adds m*p with m = t0 * (-p^-1 mod 2^32), clearing the
// low limb, and drops it.  For any a < 2^(32N) and p < 2^(32N-1) the sum
// stays inside N+1 limbs and the result is below 2p, so one conditional
// subtraction leaves it below p.
template <class P>
ZK_DEV void fe_from_mont(Fe<P>& r, const Fe<P>& a) {
    constexpr int N = P::N;
    uint32_t t[N + 1];
#pragma unroll
    for (int i = 0; i < N; i++) t[i] = a.v[i];
    t[N] = 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint32_t m = t[0] * P::N0R();
        asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(t[0]) : "r"(m), "r"(P::P(0)));
#pragma unroll
        for (int j = 1; j < N; j++) asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(t[j]) : "r"(m), "r"(P::P(j)));
        asm volatile("addc.u32 %0, %0, 0;" : "+r"(t[N]));
        asm volatile("mad.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[1]) : "r"(m), "r"(P::P(0)));
#pragma unroll
        for (int j = 1; j < N - 1; j++)
            asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(t[j + 1]) : "r"(m), "r"(P::P(j)));
        asm volatile("madc.hi.u32 %0, %1, %2, %0;" : "+r"(t[N]) : "r"(m), "r"(P::P(N - 1)));
#pragma unroll
        for (int j = 0; j < N; j++) t[j] = t[j + 1];
        t[N] = 0;
    }
    Fe<P> x;
#pragma unroll
    for (int i = 0; i < N; i++) x.v[i] = t[i];
    fe_reduce_once(r, x);
}

template <class P>
ZK_DEV bool fe_geq_int(const Fe<P>& a, const Fe<P>& b) {
    constexpr int N = P::N;
    uint32_t d, borrow;
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a.v[0]), "r"(b.v[0]));
#pragma unroll
    for (int i = 1; i < N; i++) asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a.v[i]), "r"(b.v[i]));
    asm volatile("subc.u32 %0, 0, 0;" : "=r"(borrow));
    return borrow == 0;
}

template <class P>
ZK_DEV void fe_sub_int(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
    constexpr int N = P::N;
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r.v[0]) : "r"(a.v[0]), "r"(b.v[0]));
#pragma unroll
    for (int i = 1; i < N - 1; i++) asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r.v[i]) : "r"(a.v[i]), "r"(b.v[i]));
    asm volatile("subc.u32 %0, %1, %2;" : "=r"(r.v[N - 1]) : "r"(a.v[N - 1]), "r"(b.v[N - 1]));
}

// ------------------------------------------------------------ inversion
// Division steps of Bernstein and Yang ("Fast constant-time gcd computation
// and modular inversion", 2019), delta starting at 1/2 (kept doubled): from
// f = p, g = a, each step halves g after making it even with f, swapping the
// roles when delta > 0 and g is odd; f ends as +-gcd when g = 0.  INV_STEPS
// steps at a time run on the low words alone and give a matrix (u v; q r)
// with (f, g) <- (u f + v g, q f + r g) / 2^INV_STEPS, applied then to the
// whole numbers and, mod p, to the cofactors d, e (d*a = f, e*a = g mod p,
// so d*f = 1/a at the end).  Numbers are signed 30-bit limbs.
// A chain of dependent instructions either way, but every step is the same
// short branch-free sequence: all lanes of a warp invert in lockstep, and a
// lone inversion needs no 12-limb shift or comparison per bit, as a binary
// Euclid does.  Not constant time (the loop ends when g = 0; inputs are
// public).  Zero, and anything not invertible, maps to zero.

constexpr int INV_STEPS = 30;
constexpr uint32_t INV_MASK = (1u << INV_STEPS) - 1;

template <class P>
struct InvLimbs {
    // Steps end at about 2.3 per bit at the latest for an input below p (the
    // bound proven for this delta); a third more, since an input may be any
    // 32N-bit number, and the cap only bounds the loop.
    static constexpr int BATCHES = (3 * P::BITS + 64) / INV_STEPS;
    // |d| and |e| start below p and grow by at most p/2 per batch, so they stay
    // below 32p: BITS + 5 bits and a sign
    static_assert(1 + (BATCHES + 1) / 2 < 32, "d and e stay below 32p");
    static constexpr int L = (P::BITS + 6 + INV_STEPS - 1) / INV_STEPS;
    static_assert(INV_STEPS * L >= 32 * P::N + 1, "limbs hold f and g with a sign");
    // limb i of k-bit-limb p
    __host__ __device__ static constexpr uint32_t p(int i) {
        const int w = 30 * i / 32, s = 30 * i % 32;
        const uint64_t lo = w < P::N ? P::P(w) : 0u, hi = w + 1 < P::N ? P::P(w + 1) : 0u;
        return (uint32_t)((lo | hi << 32) >> s) & INV_MASK;
    }
};

// 32-bit limbs -> 30-bit limbs (the value is below 2^(30 L - 1))
template <class P>
ZK_DEV void inv_split(int32_t (&x)[InvLimbs<P>::L], const Fe<P>& a) {
#pragma unroll
    for (int i = 0; i < InvLimbs<P>::L; i++) {
        const int w = 30 * i / 32, s = 30 * i % 32;
        const uint32_t lo = w < P::N ? a.v[w] : 0u, hi = w + 1 < P::N ? a.v[w + 1] : 0u;
        x[i] = (int32_t)(__funnelshift_r(lo, hi, s) & INV_MASK);
    }
}

template <class P>
__device__ __noinline__ void fe_inv(Fe<P>& r, const Fe<P>& a) {
    using IL = InvLimbs<P>;
    constexpr int L = IL::L;
    int32_t f[L], g[L], d[L], e[L];
    Fe<P> t;
#pragma unroll
    for (int i = 0; i < P::N; i++) t.v[i] = P::R2(i);
    inv_split<P>(g, a);
    inv_split<P>(e, t);  // e starts at R^2: (xR)^-1 * R^2 = x^-1 * R
#pragma unroll
    for (int i = 0; i < L; i++) {
        f[i] = (int32_t)IL::p(i);
        d[i] = 0;
    }
    int32_t delta = 1;  // twice delta
#pragma unroll 1
    for (int batch = 0; batch < IL::BATCHES; batch++) {
        uint32_t nz = 0;
#pragma unroll
        for (int i = 0; i < L; i++) nz |= (uint32_t)g[i];
        if (nz == 0) break;
        int32_t u = 1, v = 0, q = 0, w = 1;
        uint32_t fl = (uint32_t)f[0] | (uint32_t)f[1] << 30, gl = (uint32_t)g[0] | (uint32_t)g[1] << 30;
#pragma unroll 10
        for (int k = 0; k < INV_STEPS; k++) {
            const bool odd = gl & 1u, swap = odd && delta > 0;
            // what an odd g takes: f, or -f when the roles swap
            const uint32_t fa = swap ? 0u - fl : fl;
            const int32_t ua = swap ? -u : u, va = swap ? -v : v;
            fl = swap ? gl : fl;
            u = swap ? q : u;
            v = swap ? w : v;
            gl = (gl + (odd ? fa : 0u)) >> 1;
            q += odd ? ua : 0;
            w += odd ? va : 0;
            u <<= 1;
            v <<= 1;
            delta = (swap ? -delta : delta) + 2;
        }
        // apply the matrix; the low INV_STEPS bits of each f, g sum are zero,
        // and a multiple m*p (|m| <= 2^29) clears those of d and e
        int64_t cf = (int64_t)u * f[0] + (int64_t)v * g[0], cg = (int64_t)q * f[0] + (int64_t)w * g[0];
        int64_t cd = (int64_t)u * d[0] + (int64_t)v * e[0], ce = (int64_t)q * d[0] + (int64_t)w * e[0];
        // sign-extended low 30 bits of sum * (-1/p)
        const int32_t md = (int32_t)(((uint32_t)cd * P::N0R()) << 2) >> 2;
        const int32_t me = (int32_t)(((uint32_t)ce * P::N0R()) << 2) >> 2;
        cd += (int64_t)md * IL::p(0);
        ce += (int64_t)me * IL::p(0);
        cf >>= INV_STEPS;
        cg >>= INV_STEPS;
        cd >>= INV_STEPS;
        ce >>= INV_STEPS;
#pragma unroll
        for (int i = 1; i < L; i++) {
            cf += (int64_t)u * f[i] + (int64_t)v * g[i];
            cg += (int64_t)q * f[i] + (int64_t)w * g[i];
            cd += (int64_t)u * d[i] + (int64_t)v * e[i] + (int64_t)md * IL::p(i);
            ce += (int64_t)q * d[i] + (int64_t)w * e[i] + (int64_t)me * IL::p(i);
            f[i - 1] = (int32_t)((uint32_t)cf & INV_MASK);
            g[i - 1] = (int32_t)((uint32_t)cg & INV_MASK);
            d[i - 1] = (int32_t)((uint32_t)cd & INV_MASK);
            e[i - 1] = (int32_t)((uint32_t)ce & INV_MASK);
            cf >>= INV_STEPS;
            cg >>= INV_STEPS;
            cd >>= INV_STEPS;
            ce >>= INV_STEPS;
        }
        f[L - 1] = (int32_t)cf;
        g[L - 1] = (int32_t)cg;
        d[L - 1] = (int32_t)cd;
        e[L - 1] = (int32_t)ce;
    }
    // f = +-1 (the limbs of -1 are all-ones with a negative top limb)
    uint32_t one = (uint32_t)f[0] ^ 1u, mone = (uint32_t)f[0] ^ INV_MASK, left = 0;
#pragma unroll
    for (int i = 1; i < L; i++) {
        one |= (uint32_t)f[i];
        mone |= (uint32_t)f[i] ^ (i == L - 1 ? 0xffffffffu : INV_MASK);
    }
#pragma unroll
    for (int i = 0; i < L; i++) left |= (uint32_t)g[i];
    if (left || (one && mone)) {
        fe_set_zero(r);
        return;
    }
    // |d| < 32p to [0, p]: add or subtract 16p, 8p, .., p against the sign of
    // d (times f's sign first), then p once more if negative
    const int32_t sg = one ? -1 : 1;
#pragma unroll
    for (int i = 0; i < L; i++) d[i] *= sg;
#pragma unroll 1
    for (int k = 4; k >= -1; k--) {
        // the sign of d is its top limb's once the limbs are carried
        int64_t c = 0;
#pragma unroll
        for (int i = 0; i < L; i++) {
            c += d[i];
            if (i < L - 1) {
                d[i] = (int32_t)((uint32_t)c & INV_MASK);
                c >>= INV_STEPS;
            } else {
                d[i] = (int32_t)c;
            }
        }
        const bool ng = d[L - 1] < 0;
        const int32_t s = k < 0 ? (ng ? 1 : 0) : ng ? 1 << k : -(1 << k);
        c = 0;
#pragma unroll
        for (int i = 0; i < L; i++) {
            c += d[i] + (int64_t)s * IL::p(i);
            if (i < L - 1) {
                d[i] = (int32_t)((uint32_t)c & INV_MASK);
                c >>= INV_STEPS;
            } else {
                d[i] = (int32_t)c;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < P::N; i++) {
        const int w0 = 32 * i / 30, s = 32 * i % 30;  // bit 32i lies in limb w0 at s
        uint64_t x = (uint64_t)(uint32_t)d[w0] >> s;
        if (w0 + 1 < L) x |= (uint64_t)(uint32_t)d[w0 + 1] << (30 - s);
        if (w0 + 2 < L && 60 - s < 32) x |= (uint64_t)(uint32_t)d[w0 + 2] << (60 - s);
        t.v[i] = (uint32_t)x;
    }
    fe_reduce_once(r, t);
}

}  // namespace zkmsm

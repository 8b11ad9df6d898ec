// Point arithmetic by quads: four neighbouring lanes hold one XYZZ point, one
// coordinate each (lane 0: X, 1: Y, 2: ZZ, 3: ZZZ), and share its products.
//
// Bound.  A Montgomery product occupies a lone warp's scheduler for ~830
// cycles at 8 limbs (560 of them heavy-pipe issue), so a chain of XYZZ
// additions in one thread (14 products, at most two overlapping) costs 8.7 us
// per addition on a B200 however few points are in flight.  The products of
// an addition form four layers of at most four independent ones (a doubling:
// three, and two in the projective form below), so a quad runs an addition in
// four product times, with the same number of product slots (16 against 14),
// and a warp keeps eight points.  Values pass between lanes by shuffles.
// Used where points are few and the chain of additions is the time; kernels
// with enough points to fill the multiply pipe keep one point per thread.
//
// Every lane of the warp calls these functions together (full-mask shuffles;
// branches are warp-uniform); a lane without work holds the identity (0).
#pragma once
#include "types.cuh"

namespace zkmsm {

// the value of quad lane `src` (may differ per lane)
template <class P>
ZK_DEV void quad_get(Fe<P>& r, const Fe<P>& a, uint32_t src) {
#pragma unroll
    for (int i = 0; i < P::N; i++) r.v[i] = __shfl_sync(0xffffffffu, a.v[i], src, 4);
}

// the value of the lane two further (X <-> ZZ, Y <-> ZZZ)
template <class P>
ZK_DEV void quad_swap2(Fe<P>& r, const Fe<P>& a) {
#pragma unroll
    for (int i = 0; i < P::N; i++) r.v[i] = __shfl_xor_sync(0xffffffffu, a.v[i], 2);
}

template <class P>
ZK_DEV void fe_select(Fe<P>& r, bool c, const Fe<P>& x, const Fe<P>& y) {
#pragma unroll
    for (int i = 0; i < P::N; i++) r.v[i] = c ? x.v[i] : y.v[i];
}

// quad lane `src`'s flag
ZK_DEV bool quad_flag(bool f, uint32_t src) { return __shfl_sync(0xffffffffu, f ? 1u : 0u, src, 4) != 0; }

// coordinate q of src[...] (16-byte loads)
template <class P>
ZK_DEV void quad_load(Fe<P>& a, const Xyzz<P>* __restrict__ src, uint32_t q) {
    const uint4* s = reinterpret_cast<const uint4*>(src) + q * (P::N / 4);
#pragma unroll
    for (int i = 0; i < P::N / 4; i++) {
        const uint4 v = s[i];
        a.v[4 * i] = v.x; a.v[4 * i + 1] = v.y; a.v[4 * i + 2] = v.z; a.v[4 * i + 3] = v.w;
    }
}

template <class P>
ZK_DEV void quad_store(Xyzz<P>* dst, const Fe<P>& a, uint32_t q) {
    uint4* d = reinterpret_cast<uint4*>(dst) + q * (P::N / 4);
#pragma unroll
    for (int i = 0; i < P::N / 4; i++)
        d[i] = make_uint4(a.v[4 * i], a.v[4 * i + 1], a.v[4 * i + 2], a.v[4 * i + 3]);
}

// a = 2a (dbl-2008-s-1), three layers; the identity and 2-torsion give 0
template <class P>
ZK_DEV void quad_dbl(Fe<P>& a, uint32_t q) {
    const bool z = fe_is_zero(a);
    // ZZ = 0 or Y = 0 (both flags fetched by every lane: no short circuit
    // around a shuffle)
    const bool zz0 = quad_flag(z, 2), y0 = quad_flag(z, 1), zero = zz0 | y0;
    Fe<P> y, u, m1, v, x, w, m2, m3, t;
    quad_get(y, a, 1);
    fe_dbl(u, y);                      // U = 2Y
    fe_select(x, q == 0, a, u);
    fe_mul(m1, x, x);                  // X^2 | V = U^2
    quad_get(v, m1, 1);
    quad_get(t, m1, 0);
    fe_dbl(w, t);
    fe_add(w, w, t);                   // M = 3X^2
    fe_select(x, q == 1, u, a);
    fe_select(x, q == 3, w, x);
    fe_select(t, q == 3, w, v);
    fe_mul(m2, x, t);                  // S = X*V | W = U*V | ZZ3 = ZZ*V | M^2
    Fe<P> s, mm, x3;
    quad_get(s, m2, 0);
    quad_get(mm, m2, 3);
    fe_sub(mm, mm, s);
    fe_sub(x3, mm, s);                 // X3 = M^2 - 2S
    fe_sub(s, s, x3);
    quad_get(t, m2, 1);                // W
    fe_select(x, q == 0, w, a);        // M | Y | - | ZZZ
    fe_select(t, q == 0, s, t);        // S - X3 | W | - | W
    fe_mul(m3, x, t);                  // M(S - X3) | W*Y | - | ZZZ3 = W*ZZZ
    quad_get(t, m3, 0);
    fe_sub(t, t, m3);                  // Y3, lane 1
    fe_select(a, q == 1, t, m3);
    fe_select(a, q == 0, x3, a);
    fe_select(a, q == 2, m2, a);
    if (zero) fe_set_zero(a);
}

// a += b (add-2008-s), four layers; the identity on either side, P + P and
// P + (-P) handled
template <class P>
ZK_DEV void quad_add(Fe<P>& a, const Fe<P>& b, uint32_t q) {
    const bool hi = q & 2u;
    const bool ida = quad_flag(fe_is_zero(a), 2), idb = quad_flag(fe_is_zero(b), 2);
    Fe<P> m1, m2, m3, m4, d, x, y, pp;
    quad_swap2(x, b);
    fe_mul(m1, a, x);                  // U1 = X1*ZZ2 | S1 = Y1*ZZZ2 | U2 = ZZ1*X2 | S2 = ZZZ1*Y2
    quad_swap2(x, m1);
    fe_select(y, hi, m1, x);
    fe_select(x, hi, x, m1);
    fe_sub(d, y, x);                   // P = U2 - U1 | R = S2 - S1 | P | R
    const bool zd = fe_is_zero(d);
    const bool p0 = quad_flag(zd, 0), r0 = quad_flag(zd, 1);
    fe_select(x, hi, a, d);
    fe_select(y, hi, b, d);
    fe_mul(m2, x, y);                  // PP | R^2 | ZZ1*ZZ2 | ZZZ1*ZZZ2
    quad_get(pp, m2, 0);
    quad_get(x, d, 0);
    fe_select(y, q == 0, m1, m2);
    fe_select(x, q & 1u, x, y);
    fe_mul(m3, x, pp);                 // Q = U1*PP | PPP = P*PP | ZZ3 | PPP
    Fe<P> x3, qq, r;
    quad_get(x3, m2, 1);
    quad_get(x, m3, 1);
    quad_get(qq, m3, 0);
    fe_sub(x3, x3, x);
    fe_sub(x3, x3, qq);
    fe_sub(x3, x3, qq);                // X3 = R^2 - PPP - 2Q
    fe_sub(qq, qq, x3);
    quad_get(r, d, 1);
    fe_select(x, q == 1, m1, m2);
    fe_select(x, q == 0, r, x);
    fe_select(y, q == 0, qq, m3);
    fe_mul(m4, x, y);                  // R(Q - X3) | S1*PPP | - | ZZZ3 = ZZZ1*ZZZ2*PPP
    quad_get(x, m4, 0);
    fe_sub(x, x, m4);                  // Y3, lane 1
    fe_select(y, q == 0, x3, m4);
    fe_select(y, q == 1, x, y);
    fe_select(y, q == 2, m3, y);
    const bool same = !ida && !idb && p0 && r0;
    if (__any_sync(0xffffffffu, same)) {  // P + P (rare): the whole warp doubles
        x = a;
        quad_dbl(x, q);
        fe_select(y, same, x, y);
    }
    if (!same && p0 && !ida && !idb) fe_set_zero(y);  // P + (-P)
    fe_select(y, ida, b, y);
    fe_select(a, idb, a, y);
}

// ------------------------------------------------------- chains of doublings
// 2^count * point for long chains, in homogeneous coordinates: X/Z, Y/Z.  The
// doubling for a = 0 of Renes, Costello and Batina ("Complete addition
// formulas for prime order elliptic curves", 2016) is, with B = 3b*Z^2,
//   X3 = 2XY (Y^2 - 3B),  Y3 = (Y^2 - 3B)(Y^2 + B) + 8 Y^2 B,  Z3 = 8 Y^3 Z:
// two layers of four products where XYZZ needs three.  B takes no product by
// b: the chain carries W = c*Z with c^2 = +-3b (DBL_C, DBL_NEG in the curve's
// parameters), so that B = +-W^2.  Quad lanes: X, Y, W, W.
template <class C>
struct QuadChain {
    using P = typename C::Fp;

    // The chain's formulas hold on the curve with this b only; XYZZ doublings
    // and additions never see b, and callers may hand over points that lie on
    // y^2 = x^3 + b' instead.  True for points of the curve and the identity:
    // Y^2 = X^3 + b ZZZ^2.  Two of k_combine's ~250 product times (2^8 points
    // BN254: 312.9 us a call without the check, 312.7 with it).
    static ZK_DEV bool on_curve(const Fe<P>& a, uint32_t q) {
        Fe<P> m, s, t;
        fe_mul(m, a, a);               // X^2 | Y^2 | - | ZZZ^2
        fe_mul(s, m, a);               // X^3
        quad_get(t, m, 3);
#pragma unroll 1
        for (uint32_t i = 0; i < C::Gen::B; i++) fe_add(s, s, t);
        quad_get(t, m, 1);
        return quad_flag(fe_eq(s, t), 0);
    }

    // XYZZ -> (X*ZZZ, Y*ZZ, c*ZZ*ZZZ); the identity becomes all zeros, which
    // doubling keeps
    static ZK_DEV void enter(Fe<P>& a, uint32_t q) {
        Fe<P> t, c;
        quad_get(t, a, q == 1 ? 2 : 3);
        quad_get(a, a, q == 3 ? 2 : q);
        fe_mul(a, a, t);               // X*ZZZ | Y*ZZ | ZZ*ZZZ | ZZ*ZZZ
#pragma unroll
        for (int i = 0; i < P::N; i++) c.v[i] = C::Gen::DBL_C_MONT(i);
        fe_mul(t, a, c);
        fe_select(a, q & 2u, t, a);
    }

    // One product at a time and a dozen sums between them, on the critical
    // path.  So the products are inline (a call costs its moves), and sums that
    // only enter products stay unreduced: a product takes operands whose
    // product is below p*2^(32N), and 5p < 2^(32N) on every curve here.
    // k_combine at 2^8 points (BN254): 266 us with every sum reduced, 200 so;
    // BLS12-377 10^5 487 and 382 us.  (A product whose rows a*b_i run ahead of
    // the reduction in a second accumulator: 215 us, more instructions than
    // the waits it fills.)
    // r = a << k (k <= 2)
    static ZK_DEV void raw_shl(Fe<P>& r, const Fe<P>& a, uint32_t k) {
#pragma unroll
        for (int i = P::N - 1; i >= 0; i--) r.v[i] = __funnelshift_l(i ? a.v[i - 1] : 0u, a.v[i], k);
    }
    static ZK_DEV void raw_add(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
        asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r.v[0]) : "r"(a.v[0]), "r"(b.v[0]));
#pragma unroll
        for (int i = 1; i < P::N - 1; i++)
            asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r.v[i]) : "r"(a.v[i]), "r"(b.v[i]));
        asm volatile("addc.u32 %0, %1, %2;" : "=r"(r.v[P::N - 1]) : "r"(a.v[P::N - 1]), "r"(b.v[P::N - 1]));
    }
    // word i of 3p
    __host__ __device__ static constexpr uint32_t p3(int i) {
        uint64_t c = 0;
        for (int k = 0; k <= i; k++) c = 3ull * P::P(k) + (c >> 32);
        return (uint32_t)c;
    }
    // r = a + 3p - b (b <= 3p)
    static ZK_DEV void raw_3p_minus(Fe<P>& r, const Fe<P>& a, const Fe<P>& b) {
        Fe<P> c;
        asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(c.v[0]) : "r"(p3(0)), "r"(b.v[0]));
#pragma unroll
        for (int i = 1; i < P::N - 1; i++)
            asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(c.v[i]) : "r"(p3(i)), "r"(b.v[i]));
        asm volatile("subc.u32 %0, %1, %2;" : "=r"(c.v[P::N - 1]) : "r"(p3(P::N - 1)), "r"(b.v[P::N - 1]));
        raw_add(r, a, c);
    }

    static ZK_DEV void dbl(Fe<P>& a, uint32_t q) {
        Fe<P> y, m1, A, B, t, s, u, v, x;
        quad_get(y, a, 1);
        raw_shl(y, y, q == 0 || q == 3 ? 1 : 0);
        fe_select(y, q == 2, a, y);
        fe_mul_body_eo(m1, y, a);    // 2YX | A = Y^2 | W^2 | 2YW
        quad_get(A, m1, 1);
        quad_get(B, m1, 2);
        // t = Y^2 - 3B below 4p, s = Y^2 + B below p
        raw_shl(v, B, 1);
        raw_add(v, v, B);
        if (C::Gen::DBL_NEG) {
            raw_add(t, A, v);
            fe_sub(s, A, B);
        } else {
            raw_3p_minus(t, A, v);
            fe_add(s, A, B);
        }
        raw_shl(u, A, q == 2 ? 1 : 2);     // 2A for 4A*|B|, 4A for W3
        raw_shl(v, B, 1);
        fe_select(x, q & 2u, u, t);
        fe_select(y, q == 1, s, m1);
        fe_select(y, q == 2, v, y);
        fe_mul_body_eo(m1, x, y);    // X3 = t*2XY | t*s | 2A*2|B| | W3 = 4A*2YW
        quad_get(x, m1, q == 1 ? 2 : 3);
        fe_dbl(u, x);                  // lane 1: 8A|B|
        if (C::Gen::DBL_NEG) fe_sub(y, m1, u);
        else fe_add(y, m1, u);
        fe_select(a, q == 1, y, m1);
        fe_select(a, q == 2, x, a);
    }

    // back to XYZZ with ZZ = W^2: x = cX / W = (cX*W) / W^2
    static ZK_DEV void leave(Fe<P>& a, uint32_t q) {
        Fe<P> c, t, w, m;
#pragma unroll
        for (int i = 0; i < P::N; i++) c.v[i] = C::Gen::DBL_C_MONT(i);
        fe_select(t, q & 2u, a, c);
        fe_mul(m, a, t);               // cX | cY | W^2 | W^2
        quad_get(w, a, 2);
        quad_get(t, m, 2);
        fe_select(t, q == 1, t, w);
        fe_mul(t, m, t);               // cX*W | cY*W^2 | - | W^3
        fe_select(a, q == 2, m, t);
    }
};

// BN254 G2: 3b = 9 / (9 + u) has no cheap form there; the chain stays XYZZ
template <>
struct QuadChain<Bn254G2> {
    using P = Bn254G2::Fp;
    static ZK_DEV bool on_curve(const Fe<P>&, uint32_t) { return true; }
    static ZK_DEV void enter(Fe<P>&, uint32_t) {}
    static ZK_DEV void dbl(Fe<P>& a, uint32_t q) { quad_dbl(a, q); }
    static ZK_DEV void leave(Fe<P>&, uint32_t) {}
};

}  // namespace zkmsm

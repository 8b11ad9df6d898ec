// Pippenger MSM kernels (sm_100a), templated on the curve.
//
// Pipeline for a batch of MSMs over one base table (a single plain call is a
// batch of one).  Reference counterparts (Shaders/msm/*.metal and the Swift
// engine MSM/MSMEngine.swift) are cited per kernel.
//
//  1. k_radix_digits  scalar -> integer (Montgomery reduce or mod r), GLV
//                     split, signed c-bit digits; entries (bucket id,
//                     point|endo|sign) appended densely, unsorted.
//                     [glv_kernels.metal:172-256, msm_kernels.metal:399-439]
//  2. k_radix_hist /  LSD radix sort of the entries by bucket id, 7-8 bits
//     k_radix_scatter per pass: per-tile digit counts, scan, stable
//                     tile-local ranking staged in shared memory and written
//                     as contiguous runs.  [MSMEngine.swift:595-661 (CPU
//                     counting sort per window)]
//     (k_digit_hist / k_digit_scatter: the earlier one-pass counting sort
//     with global atomics, kept for the allocation-free entry point.)
//  4. k_acc_l1        bucket accumulation: each thread sums a fixed-length
//                     chunk of the sorted list with mixed XYZZ additions;
//                     runs strictly inside a chunk are final buckets, a
//                     chunk's first and last run become partial sums.
//                     [msm_kernels.metal:16-62]
//                     (k_aff_*, affine.cuh: the same by affine pair sums, for
//                     large entry sets on the 12-limb curves and G2.)
//  5. k_acc_fold      the same segmented reduction over the partial sums (in
//                     small calls over the entries too), quads of lanes and a
//                     tree per block, repeated until one block is left
//                     (handles any skew, e.g. 20% of all points in one bucket
//                     for witness scalars).
//  6. k_reduce_level, k_reduce_quads, k_reduce_windows
//                     per window sum_b b*B_b: running sums while there are
//                     many nodes, then bit sums by quads of lanes.
//                     [msm_kernels.metal:152-248]
//  7. k_combine       the windows' bit sums shifted into place (quads of
//                     lanes), normalise to affine.
//                     [MSMEngine.swift:899-904, msm_kernels.metal:251-275]
#pragma once
#include "quad.cuh"
#include "types.cuh"

namespace zkmsm {

// Scalar state after preparation: up to two halves, each a magnitude (up to
// 9 limbs: 256 bits plus a zero guard limb) and a sign.
struct Halves {
    uint32_t k[2][9];
    uint32_t neg[2];
    int count;
};

// ------------------------------------------------------------ scalar prep

// Constants of a curve's GLV split by name (W: 0 = G1, 1 = G2, 2 = A1,
// 3 = A2, 4 = B1, 5 = B2), their nonzero limbs and bit length.
template <class G, int W>
struct GlvK {
    __host__ __device__ static constexpr uint32_t limb(int i) {
        return W == 0 ? G::G1(i) : W == 1 ? G::G2(i) : W == 2 ? G::A1(i) : W == 3 ? G::A2(i) : W == 4 ? G::B1(i)
                                                                                                      : G::B2(i);
    }
    __host__ __device__ static constexpr int limbs() {
        return limb(4) ? 5 : limb(3) ? 4 : limb(2) ? 3 : limb(1) ? 2 : limb(0) ? 1 : 0;
    }
    __host__ __device__ static constexpr int bits() {
        int b = 0;
        for (uint32_t t = limbs() ? limb(limbs() - 1) : 0u; t; t >>= 1) b++;
        return limbs() ? 32 * (limbs() - 1) + b : 0;
    }
};

// Babai rounding c = (s * G + 2^255) >> 256 for an 8-limb s below 2^BITS and
// a constant G of K::limbs() nonzero limbs; c has `LC` limbs.  One row per
// limb of G: the 8 low halves (carry into the row's top limb, still zero),
// then the 8 high halves.
template <class K, int LC>
ZK_DEV void babai_round(uint32_t (&c)[5], const uint32_t (&s)[8]) {
    constexpr int NG = K::limbs();
    uint32_t p[8 + NG];
#pragma unroll
    for (int i = 0; i < 8 + NG; i++) p[i] = 0;
#pragma unroll
    for (int l = 0; l < NG; l++) {
        const uint32_t g = K::limb(l);
        asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(p[l]) : "r"(s[0]), "r"(g));
#pragma unroll
        for (int i = 1; i < 8; i++) asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(p[l + i]) : "r"(s[i]), "r"(g));
        asm volatile("addc.u32 %0, %0, 0;" : "+r"(p[l + 8]));
        asm volatile("mad.hi.cc.u32 %0, %1, %2, %0;" : "+r"(p[l + 1]) : "r"(s[0]), "r"(g));
#pragma unroll
        for (int i = 1; i < 7; i++) asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(p[l + 1 + i]) : "r"(s[i]), "r"(g));
        asm volatile("madc.hi.u32 %0, %1, %2, %0;" : "+r"(p[l + 8]) : "r"(s[7]), "r"(g));
    }
    asm volatile("add.cc.u32 %0, %0, %1;" : "+r"(p[7]) : "r"(0x80000000u));
#pragma unroll
    for (int i = 8; i < 8 + NG - 1; i++) asm volatile("addc.cc.u32 %0, %0, 0;" : "+r"(p[i]));
    asm volatile("addc.u32 %0, %0, 0;" : "+r"(p[8 + NG - 1]));
#pragma unroll
    for (int i = 0; i < 5; i++) c[i] = i < NG && i < LC ? p[8 + i] : 0u;
}

// acc -= c * K (SUB) or acc += c * K, mod 2^160; c has LC limbs, the
// lattice constant K its nonzero limbs.
template <class K, int LC, bool SUB>
ZK_DEV void lattice_mac(uint32_t (&acc)[5], const uint32_t (&c)[5]) {
    constexpr int LK = K::limbs();
    uint32_t p[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < LC && i < 5; i++) {
        uint32_t carry = 0;
#pragma unroll
        for (int l = 0; l < LK && i + l < 5; l++) {
            const uint64_t t = (uint64_t)c[i] * K::limb(l) + p[i + l] + carry;
            p[i + l] = (uint32_t)t;
            carry = (uint32_t)(t >> 32);
        }
        if (i + LK < 5) p[i + LK] = carry;
    }
    if (SUB) {
        asm volatile("sub.cc.u32 %0, %0, %1;" : "+r"(acc[0]) : "r"(p[0]));
#pragma unroll
        for (int i = 1; i < 4; i++) asm volatile("subc.cc.u32 %0, %0, %1;" : "+r"(acc[i]) : "r"(p[i]));
        asm volatile("subc.u32 %0, %0, %1;" : "+r"(acc[4]) : "r"(p[4]));
    } else {
        asm volatile("add.cc.u32 %0, %0, %1;" : "+r"(acc[0]) : "r"(p[0]));
#pragma unroll
        for (int i = 1; i < 4; i++) asm volatile("addc.cc.u32 %0, %0, %1;" : "+r"(acc[i]) : "r"(p[i]));
        asm volatile("addc.u32 %0, %0, %1;" : "+r"(acc[4]) : "r"(p[4]));
    }
}

// Scalar preparation into registers: the integer scalar (Montgomery
// reduction for Fr input, bn254_msm.c:1537-1552; subtractions of r for
// integer input, MSMEngine.swift:182-200), then for GLV the split
// k = k1 + k2*lambda with k1 = s - c1*a1 - c2*a2, k2 = -c1*b1 - c2*b2 and the
// Babai roundings c_j = round(s*G_j / 2^256) (GLV.swift:8-33,
// glv_kernels.metal:172-256).  x[j] holds |k_j| (NL limbs; 5 suffice for
// GLV halves, 9 for a whole 256-bit scalar plus the guard limb of the top
// window's carry), neg[j] its sign; count = 2 with GLV, else 1 (x[0] the
// scalar).  All indexing is static, so everything stays in registers.
template <class C, int NL>
ZK_DEV void prep_scalar(uint32_t (&x)[2][NL], uint32_t (&neg)[2], int& count, const uint32_t* __restrict__ s8,
                        uint32_t fmt, uint32_t glv) {
    using Fr = typename C::Fr;
    using G = typename C::Glv;
    static_assert(NL >= 5, "a GLV half needs five limbs");
    Fe<Fr> s;
    const uint4* p4 = reinterpret_cast<const uint4*>(s8);
    const uint4 a = __ldg(p4), b = __ldg(p4 + 1);
    s.v[0] = a.x; s.v[1] = a.y; s.v[2] = a.z; s.v[3] = a.w;
    s.v[4] = b.x; s.v[5] = b.y; s.v[6] = b.z; s.v[7] = b.w;
    if (fmt == 1) {
        fe_from_mont(s, s);
    } else {
        // integer form may exceed r: subtract r until below;
        // REDUCE_PASSES = floor((2^256 - 1) / r) passes always suffice (5 for
        // BN254, 2 for BLS12-381, 13 for BLS12-377)
        Fe<Fr> r;
#pragma unroll
        for (int i = 0; i < 8; i++) r.v[i] = Fr::P(i);
#pragma unroll 1
        for (int it = 0; it < Fr::REDUCE_PASSES && fe_geq_int(s, r); it++) fe_sub_int(s, s, r);
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
        neg[j] = 0;
#pragma unroll
        for (int i = 0; i < NL; i++) x[j][i] = 0;
    }
    if (!glv) {
        if (NL >= 9) {
#pragma unroll
            for (int i = 0; i < 8 && i < NL; i++) x[0][i] = s.v[i];
        }
        count = NL >= 9 ? 1 : 0;  // a five-limb kernel is never launched without GLV
        return;
    }
    using KG1 = GlvK<G, 0>;
    using KG2 = GlvK<G, 1>;
    // c_j < 2^(BITS + bits(G_j) - 256) + 1/2
    constexpr int LC1 = (Fr::BITS + KG1::bits() - 256 + 1 + 31) / 32 < 5 ? (Fr::BITS + KG1::bits() - 256 + 1 + 31) / 32 : 5;
    constexpr int LC2 = (Fr::BITS + KG2::bits() - 256 + 1 + 31) / 32 < 5 ? (Fr::BITS + KG2::bits() - 256 + 1 + 31) / 32 : 5;
    uint32_t c1[5], c2[5];
    babai_round<KG1, LC1>(c1, s.v);
    babai_round<KG2, LC2>(c2, s.v);
    // k1 = s - c1*a1 - c2*a2, k2 = -c1*b1 - c2*b2   (mod 2^160, signed)
    uint32_t k1[5] = {s.v[0], s.v[1], s.v[2], s.v[3], s.v[4]};
    uint32_t k2[5] = {0, 0, 0, 0, 0};
    lattice_mac<GlvK<G, 2>, LC1, !G::A1_NEG>(k1, c1);
    lattice_mac<GlvK<G, 3>, LC2, !G::A2_NEG>(k1, c2);
    lattice_mac<GlvK<G, 4>, LC1, !G::B1_NEG>(k2, c1);
    lattice_mac<GlvK<G, 5>, LC2, !G::B2_NEG>(k2, c2);
    uint32_t* ks[2] = {k1, k2};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        uint32_t* k = ks[j];
        const uint32_t ng = k[4] >> 31;
        // magnitude = ng ? -k : k  (two's complement under a mask)
        const uint32_t m = 0u - ng;
        asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(x[j][0]) : "r"(k[0] ^ m), "r"(ng));
#pragma unroll
        for (int i = 1; i < 4; i++) asm volatile("addc.cc.u32 %0, %1, 0;" : "=r"(x[j][i]) : "r"(k[i] ^ m));
        asm volatile("addc.u32 %0, %1, 0;" : "=r"(x[j][4]) : "r"(k[4] ^ m));
        neg[j] = ng;
    }
    count = 2;
}

template <class C>
ZK_DEV void prepare_scalar(Halves& h, const uint32_t* __restrict__ s8, uint32_t fmt, uint32_t glv) {
    uint32_t x[2][9], neg[2];
    prep_scalar<C, 9>(x, neg, h.count, s8, fmt, glv);
#pragma unroll
    for (int j = 0; j < 2; j++) {
#pragma unroll
        for (int i = 0; i < 9; i++) h.k[j][i] = x[j][i];
        h.neg[j] = neg[j];
    }
}

// c-bit field of a multi-limb magnitude starting at bit `off` (c <= 31, off + c <= 288)
ZK_DEV uint32_t bit_field(const uint32_t* k, uint32_t off, uint32_t c) {
    uint32_t li = off >> 5, sh = off & 31;
    uint64_t w = k[li];
    if (li + 1 < 9) w |= (uint64_t)k[li + 1] << 32;
    return (uint32_t)(w >> sh) & ((1u << c) - 1);
}

// Binary search: the MSM owning global scalar index gi (descs sorted by scalar_off)
ZK_DEV int find_msm(const MsmDesc* __restrict__ d, int nd, uint64_t gi) {
    int lo = 0, hi = nd - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (d[mid].scalar_off <= gi) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Signed-digit stream of a prepared scalar.  Digits of half j, window w:
// v = field + carry; v > 2^(c-1) gives digit v - 2^c (negative, carry 1),
// otherwise v (carry 0); digits lie in [-2^(c-1), 2^(c-1)].  The stream
// yields only nonzero digits, DBATCH at a time, so a thread can issue a whole
// batch of independent atomics before waiting for any of them.
constexpr int DBATCH = 8;

struct DigitGen {
    uint32_t j, w, carry;
};

ZK_DEV void next_digits(DigitGen& g, const Halves& h, const MsmDesc& d, uint32_t idx, bool (&valid)[DBATCH],
                        uint32_t (&gb)[DBATCH], uint32_t (&val)[DBATCH]) {
#pragma unroll
    for (int s = 0; s < DBATCH; s++) {
        valid[s] = false;
        gb[s] = 0;
        val[s] = 0;
#pragma unroll 1
        while (g.j < (uint32_t)h.count) {
            const uint32_t cw = win_width(d, g.w);
            uint32_t v = bit_field(h.k[g.j], win_bit(d, g.w), cw) + g.carry;
            uint32_t a, dn;
            if (v > (1u << (cw - 1))) {
                a = (1u << cw) - v;
                dn = 1;
                g.carry = 1;
            } else {
                a = v;
                dn = 0;
                g.carry = 0;
            }
            uint32_t w = g.w, j = g.j;
            if (++g.w == d.nwin) {
                g.w = 0;
                g.carry = 0;
                g.j++;
            }
            if (a) {
                valid[s] = true;
                if (d.wstep) {  // shift table: window w's base is 2^(c*w)*P, one bucket set
                    gb[s] = d.bucket_off + (a - 1);
                    val[s] = (idx + w * d.wstep) | ((h.neg[j] ^ dn) << 31);
                } else {
                    gb[s] = d.bucket_off + win_bucket(d, w) + (a - 1);
                    val[s] = idx | (j << 30) | ((h.neg[j] ^ dn) << 31);
                }
                break;
            }
        }
    }
}

// Lanes of `mask` whose key equals the first valid lane's key share one
// atomic (the hot-bucket case, e.g. many scalars equal to 1).
struct AggSlot {
    uint32_t leader, same;
    bool grp;
};

ZK_DEV AggSlot agg_slot(uint32_t mask, bool valid, uint32_t key) {
    AggSlot a;
    uint32_t m = __ballot_sync(mask, valid);
    a.leader = m ? __ffs(m) - 1 : 0;
    uint32_t lk = __shfl_sync(mask, key, a.leader);
    a.grp = valid && m && key == lk;
    a.same = __ballot_sync(mask, a.grp);
    return a;
}

template <class C>
__global__ void __launch_bounds__(256) k_digit_hist(const uint32_t* __restrict__ scalars,
                                                    const MsmDesc* __restrict__ descs, int nd,
                                                    uint64_t total, uint32_t* __restrict__ counts) {
    uint64_t gi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= total) return;
    const uint32_t mask = __activemask();
    const uint32_t lane = threadIdx.x & 31;
    const MsmDesc d = descs[find_msm(descs, nd, gi)];
    Halves h;
    prepare_scalar<C>(h, scalars + gi * 8, d.fmt, d.glv);
    DigitGen g{0, 0, 0};
    if (d.nwin == 0) g.j = (uint32_t)h.count;
    bool valid[DBATCH];
    uint32_t gb[DBATCH], val[DBATCH];
#pragma unroll 1
    while (__any_sync(mask, g.j < (uint32_t)h.count)) {
        next_digits(g, h, d, 0, valid, gb, val);
#pragma unroll
        for (int s = 0; s < DBATCH; s++) {
            AggSlot a = agg_slot(mask, valid[s], gb[s]);
            if (a.grp) {
                if (lane == a.leader) atomicAdd(counts + gb[s], (uint32_t)__popc(a.same));
            } else if (valid[s]) {
                atomicAdd(counts + gb[s], 1u);
            }
        }
    }
}

// Scalar profile: the bit lengths of the prepared halves (after the
// Montgomery reduce or mod-r reduction and the GLV split) of m scalars spread
// evenly over [0, n): hist[b] counts halves of bit length b.  The host turns
// it into the expected number of nonzero digits of a window layout, so that
// skewed scalar sets (many zeros, ones or short scalars) get a layout with
// fewer buckets.  The reference samples a window-0 bucket histogram for the
// same purpose (MSM/MSMEngine.swift:565-593, 768-783).
template <class C>
__global__ void __launch_bounds__(256) k_scalar_profile(const uint32_t* __restrict__ scalars, uint64_t n, uint32_t m,
                                                        uint32_t fmt, uint32_t glv, uint32_t* __restrict__ hist) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    const uint64_t i = (uint64_t)j * n / m;
    Halves h;
    prepare_scalar<C>(h, scalars + i * 8, fmt, glv);
#pragma unroll 1
    for (int k = 0; k < h.count; k++) {
        uint32_t b = 0;
#pragma unroll
        for (int l = 0; l < 9; l++)
            if (h.k[k][l]) b = 32u * l + 32u - __clz(h.k[k][l]);
        atomicAdd(hist + min(b, PROFILE_BINS - 1), 1u);
    }
}

// Counting-sort scatter: entry = (global bucket id, base index | endo << 30 | negate << 31)
template <class C>
__global__ void __launch_bounds__(256) k_digit_scatter(const uint32_t* __restrict__ scalars,
                                                       const MsmDesc* __restrict__ descs, int nd,
                                                       uint64_t total, uint32_t* __restrict__ cursor,
                                                       uint2* __restrict__ ents) {
    uint64_t gi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= total) return;
    const uint32_t mask = __activemask();
    const uint32_t lane = threadIdx.x & 31;
    const MsmDesc d = descs[find_msm(descs, nd, gi)];
    Halves h;
    prepare_scalar<C>(h, scalars + gi * 8, d.fmt, d.glv);
    const uint32_t idx = d.base_off + (uint32_t)(gi - d.scalar_off);
    DigitGen g{0, 0, 0};
    if (d.nwin == 0) g.j = (uint32_t)h.count;
    bool valid[DBATCH];
    uint32_t gb[DBATCH], val[DBATCH], base[DBATCH];
    AggSlot a[DBATCH];
#pragma unroll 1
    while (__any_sync(mask, g.j < (uint32_t)h.count)) {
        next_digits(g, h, d, idx, valid, gb, val);
        // issue every atomic of the batch before consuming any result
#pragma unroll
        for (int s = 0; s < DBATCH; s++) {
            a[s] = agg_slot(mask, valid[s], gb[s]);
            base[s] = 0;
            if (valid[s] && (!a[s].grp || lane == a[s].leader))
                base[s] = atomicAdd(cursor + gb[s], a[s].grp ? (uint32_t)__popc(a[s].same) : 1u);
        }
#pragma unroll
        for (int s = 0; s < DBATCH; s++) {
            uint32_t b = __shfl_sync(mask, base[s], a[s].leader);
            uint32_t pos = a[s].grp ? b + __popc(a[s].same & ((1u << lane) - 1)) : base[s];
            if (valid[s]) ents[pos] = make_uint2(gb[s], val[s]);
        }
    }
}

// ------------------------------------------------------------ radix sort
// Entries (bucket id, point | endo | sign) are sorted by bucket id with an
// LSD radix sort, without global atomics on the data path:
//  k_radix_digits   digits of SORT_DTILE-ish scalars per block, buffered in
//                   shared memory and appended densely to A (one atomic per
//                   block claims the range; the order of blocks is free);
//  per pass (RBITS-bit digit at `shift`), over tiles of SORT_ETILE entries:
//  k_radix_hist     per-tile digit counts, stored digit-major [digit][tile];
//  scan             exclusive, so [digit][tile] holds the tile's first slot;
//  k_radix_scatter  stable rank inside the tile (warp ballots per digit bit,
//                   per-warp counters), staged in shared memory in digit
//                   order, then written out as one contiguous run per digit.
// Passes after the first are stable, so the result is sorted by the whole
// key; the order inside a bucket comes from the first pass and is not
// fixed (bucket sums do not depend on it).

// Lanes of the warp whose BITS-bit digit equals this lane's (valid lanes
// only; `vmask` = ballot of valid): one ballot per digit bit.
template <int BITS>
ZK_DEV uint32_t digit_peers(uint32_t d, uint32_t vmask) {
    uint32_t peers = vmask;
#pragma unroll
    for (int b = 0; b < BITS; b++) {
        const bool bit = (d >> b) & 1u;
        const uint32_t bal = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? bal : ~bal;
    }
    return peers;
}

// Shared-memory counter bump with the hot-key case aggregated: lanes whose
// key equals the first valid lane's key share one atomic (all lanes of a
// warp hitting one bin, e.g. many scalars equal to 1, cost one atomic, not
// 32 serialised ones); other valid lanes add 1 each.  All 32 lanes of the
// warp call it together.
ZK_DEV void warp_count(uint32_t* __restrict__ ctr, bool valid, uint32_t key) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t m = __ballot_sync(0xffffffffu, valid);
    if (!m) return;
    const uint32_t leader = __ffs(m) - 1;
    const uint32_t lk = __shfl_sync(0xffffffffu, key, leader);
    const bool grp = valid && key == lk;
    const uint32_t same = __ballot_sync(0xffffffffu, grp);
    if (lane == leader) atomicAdd(ctr + lk, (uint32_t)__popc(same));
    else if (valid && !grp) atomicAdd(ctr + key, 1u);
}

// Signed digit of the current window of a prepared half held in registers
// (NL limbs, shifted right window by window: the low bits are always the
// current window).  v = field + carry; v > 2^(cw-1) gives digit v - 2^cw
// (negative: dn = 1, carry 1), otherwise v (carry 0); digits lie in
// [-2^(cw-1), 2^(cw-1)].  Returns the digit's magnitude.

template <int NL>
ZK_DEV uint32_t take_window(uint32_t (&x)[NL], uint32_t cw, uint32_t& carry, uint32_t& dn) {
    const uint32_t v = (x[0] & ((1u << cw) - 1u)) + carry;
    const bool hi = v > (1u << (cw - 1));
    dn = hi ? 1u : 0u;
    carry = dn;
#pragma unroll
    for (int i = 0; i < NL - 1; i++) x[i] = __funnelshift_r(x[i], x[i + 1], cw);
    x[NL - 1] >>= cw;
    return hi ? (1u << cw) - v : v;
}

// hist0 (optional, zeroed before the launch): the first radix pass's
// digit-major per-tile counts of the low h0bits bits of the bucket ids, for
// tiles of SORT_ETILE entries of A ([digit][tile], ntiles tiles), added here
// so that the first LSD pass needs no histogram kernel.  D (optional): the
// first MSD pass's digit of each entry, (key >> dshift) & dmask, beside A, so
// that its count kernel reads 2 bytes per entry instead of 8.
//
// Each thread prepares one scalar per round into registers; the warp then
// walks (half, window) in step: each lane takes its digit and a ballot ranks
// the nonzero ones inside the warp's own slice of the block buffer, behind a
// running count the whole warp holds (no atomics, no shuffles).  A slice
// takes SORT_DBUF / 8 entries: with maxd digits per scalar at most, a block
// runs min(32, spb / 8) lanes per warp and rounds of 8 * lanes scalars, so
// that a slice never overflows (spb from the plan: 256 * floor(16 / maxd)
// scalars when maxd <= 16, else 8 * floor(512 / maxd)).  The slices go to A
// in one run claimed by one atomic per block.  NL = 5 when every MSM of the
// launch splits with GLV, else 9.
constexpr uint32_t SORT_DWARPS = SORT_DTHREADS / 32;
constexpr uint32_t SORT_DSLICE = SORT_DBUF / SORT_DWARPS;
static_assert(SORT_DBUF <= SORT_ETILE, "a digit block's range spans at most two sort tiles");
template <class C, int NL>
__global__ void __launch_bounds__(SORT_DTHREADS) k_radix_digits(const uint32_t* __restrict__ scalars,
                                                                const MsmDesc* __restrict__ descs, int nd,
                                                                uint64_t total, uint32_t scalars_per_block,
                                                                uint2* __restrict__ A,
                                                                uint32_t* __restrict__ d_count,
                                                                uint32_t* __restrict__ hist0, uint32_t h0bits,
                                                                uint32_t ntiles, uint16_t* __restrict__ D,
                                                                uint32_t dshift, uint32_t dmask) {
    __shared__ uint2 buf[SORT_DBUF];
    __shared__ uint32_t wpre[SORT_DWARPS + 1];
    __shared__ uint32_t base_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t lanes = scalars_per_block / SORT_DWARPS < 32 ? scalars_per_block / SORT_DWARPS : 32u;
    uint2* slice = buf + wid * SORT_DSLICE;
    uint32_t wc = 0;  // entries in the warp's slice (the same in every lane)
#pragma unroll 1
    for (uint32_t k = 0; k < scalars_per_block; k += SORT_DWARPS * lanes) {
        const uint32_t r = k + wid * lanes + lane;  // scalar of the block
        const uint64_t gi = (uint64_t)blockIdx.x * scalars_per_block + r;
        uint32_t x[2][NL], neg[2] = {0, 0};
        int cnt = 0;
        MsmDesc d{};
        d.c = 2;
        uint32_t idx = 0;
        if (lane < lanes && r < scalars_per_block && gi < total) {
            d = descs[find_msm(descs, nd, gi)];
            prep_scalar<C, NL>(x, neg, cnt, scalars + gi * 8, d.fmt, d.glv);
            idx = d.base_off + (uint32_t)(gi - d.scalar_off);
            if (d.nwin == 0) cnt = 0;
        } else {
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int i = 0; i < NL; i++) x[j][i] = 0;
        }
        // warp-uniform walk: the most halves and windows of any lane
        const uint32_t jm = __reduce_max_sync(0xffffffffu, (uint32_t)cnt);
        const uint32_t wm = __reduce_max_sync(0xffffffffu, cnt ? d.nwin : 0u);
#pragma unroll
        for (uint32_t j = 0; j < 2; j++) {
            if (j >= jm) break;
            uint32_t carry = 0, wb = 0;
#pragma unroll 1
            for (uint32_t w = 0; w < wm; w++) {
                const uint32_t cw = d.c + (w >= d.nlo ? 1u : 0u);
                uint32_t dn;
                const uint32_t a = take_window<NL>(x[j], cw, carry, dn);
                const bool ok = j < (uint32_t)cnt && w < d.nwin && a != 0;
                const uint32_t m = __ballot_sync(0xffffffffu, ok);
                if (ok) {
                    uint2 e;
                    if (d.wstep) {  // shift table: window w's base is 2^(c*w)*P, one bucket set
                        e.x = d.bucket_off + (a - 1);
                        e.y = (idx + w * d.wstep) | ((neg[j] ^ dn) << 31);
                    } else {
                        e.x = d.bucket_off + wb + (a - 1);
                        e.y = idx | (j << 30) | ((neg[j] ^ dn) << 31);
                    }
                    slice[wc + __popc(m & lt)] = e;
                }
                wc += __popc(m);
                wb += 1u << (cw - 1);
            }
        }
    }
    // slices -> one dense run of A
    if (lane == 0) wpre[wid] = wc;
    __syncthreads();
    if (tid == 0) {
        uint32_t run = 0;
        for (uint32_t w = 0; w < SORT_DWARPS; w++) {
            const uint32_t c = wpre[w];
            wpre[w] = run;
            run += c;
        }
        wpre[SORT_DWARPS] = run;
        base_s = run ? atomicAdd(d_count, run) : 0;
    }
    __syncthreads();
    const uint32_t base = base_s, wbase = wpre[wid];
    for (uint32_t i = lane; i < wc; i += 32) {
        const uint2 e = slice[i];
        A[(size_t)base + wbase + i] = e;
        if (D) D[(size_t)base + wbase + i] = (uint16_t)((e.x >> dshift) & dmask);
    }
    if (hist0) {
        // counts of the range [base, base + cnt) per tile (the tile of base,
        // and the next one from entry `split` on) and digit, then one
        // global add per non-zero count
        __shared__ uint32_t hc[2 * SORT_MAX_BINS];
        for (uint32_t i = tid; i < 2 * SORT_MAX_BINS; i += SORT_DTHREADS) hc[i] = 0;
        __syncthreads();
        const uint32_t mask = (1u << h0bits) - 1;
        const uint32_t split = SORT_ETILE - base % SORT_ETILE;
        for (uint32_t i0 = 0; i0 < SORT_DSLICE; i0 += 32) {
            const uint32_t i = i0 + lane;
            const bool v = i < wc;
            const uint32_t key = v ? (wbase + i < split ? 0u : SORT_MAX_BINS) + (slice[i].x & mask) : 0u;
            if (__any_sync(0xffffffffu, v)) warp_count(hc, v, key);
        }
        __syncthreads();
        const uint32_t t0 = base / SORT_ETILE;
        for (uint32_t i = tid; i < 2 * SORT_MAX_BINS; i += SORT_DTHREADS) {
            const uint32_t c = hc[i];
            if (c) atomicAdd(hist0 + (size_t)(i % SORT_MAX_BINS) * ntiles + t0 + i / SORT_MAX_BINS, c);
        }
    }
}

// Per-warp digit counts of the warp's SORT_ETILE / SORT_WARPS entries of a
// tile (blocked: warp w owns entries [w*PER, (w+1)*PER)); also each entry's
// rank among the warp's earlier entries with the same digit.
constexpr uint32_t SORT_WARPS = SORT_ETHREADS / 32;
constexpr uint32_t SORT_PER_WARP = SORT_ETILE / SORT_WARPS;
constexpr uint32_t SORT_ROUNDS = SORT_PER_WARP / 32;

static __global__ void __launch_bounds__(SORT_ETHREADS) k_radix_hist(const uint2* __restrict__ A,
                                                                     const uint32_t* __restrict__ d_total,
                                                                     uint32_t shift, uint32_t bits,
                                                                     uint32_t ntiles, uint32_t* __restrict__ hist) {
    __shared__ uint32_t cnt[SORT_MAX_BINS];
    const uint32_t tid = threadIdx.x;
    const uint32_t nb = 1u << bits, mask = nb - 1;
    for (uint32_t i = tid; i < SORT_MAX_BINS; i += SORT_ETHREADS) cnt[i] = 0;
    __syncthreads();
    const uint64_t total = *d_total;
    const uint64_t tbase = (uint64_t)blockIdx.x * SORT_ETILE;
    constexpr uint32_t R = SORT_ETILE / SORT_ETHREADS;
    uint32_t key[R];
#pragma unroll
    for (uint32_t r = 0; r < R; r++) {
        const uint64_t i = tbase + r * SORT_ETHREADS + tid;
        key[r] = i < total ? (A[i].x >> shift) & mask : 0xffffffffu;
    }
#pragma unroll
    for (uint32_t r = 0; r < R; r++) warp_count(cnt, key[r] != 0xffffffffu, key[r]);
    __syncthreads();
    for (uint32_t dg = tid; dg < nb; dg += SORT_ETHREADS) hist[(size_t)dg * ntiles + blockIdx.x] = cnt[dg];
}

template <int BITS>
__global__ void __launch_bounds__(SORT_ETHREADS, 4) k_radix_scatter(const uint2* __restrict__ A,
                                                                 const uint32_t* __restrict__ d_total,
                                                                 uint32_t shift, uint32_t ntiles,
                                                                 const uint32_t* __restrict__ hoff,
                                                                 uint2* __restrict__ B) {
    constexpr uint32_t NB = 1u << BITS, MASK = NB - 1;
    __shared__ uint32_t wcnt[SORT_WARPS][SORT_MAX_BINS];
    __shared__ uint32_t loff[SORT_MAX_BINS], goff[SORT_MAX_BINS], wtot[SORT_ETHREADS / 32];
    __shared__ uint2 stage[SORT_ETILE];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t i = tid; i < SORT_WARPS * SORT_MAX_BINS; i += SORT_ETHREADS) (&wcnt[0][0])[i] = 0;
    __syncthreads();
    const uint64_t total = *d_total;
    const uint64_t tbase = (uint64_t)blockIdx.x * SORT_ETILE;
    const uint32_t n_tile = tbase >= total ? 0u : total - tbase < SORT_ETILE ? (uint32_t)(total - tbase) : SORT_ETILE;
    const uint64_t t0 = tbase + (uint64_t)warp * SORT_PER_WARP;
    // pass 1: stable rank of each entry among the warp's earlier entries
    // with its digit (warp w owns entries [w*PER, (w+1)*PER) of the tile)
    // kr[r] = digit | rank << 16 (rank < SORT_PER_WARP)
    uint32_t kr[SORT_ROUNDS];
#pragma unroll
    for (uint32_t r = 0; r < SORT_ROUNDS; r++) {
        const uint64_t i = t0 + r * 32 + lane;
        kr[r] = i < total ? (A[i].x >> shift) & MASK : 0;
    }
#pragma unroll
    for (uint32_t r = 0; r < SORT_ROUNDS; r++) {
        const uint64_t i = t0 + r * 32 + lane;
        const bool v = i < total;
        const uint32_t vm = __ballot_sync(0xffffffffu, v);
        if (vm) {
            const uint32_t d = kr[r];
            const uint32_t peers = digit_peers<BITS>(d, vm);
            const uint32_t before = v ? wcnt[warp][d] : 0;
            kr[r] = d | (before + __popc(peers & ((1u << lane) - 1))) << 16;
            __syncwarp();
            if (v && lane == 31 - __clz(peers)) wcnt[warp][d] = before + __popc(peers);
            __syncwarp();
        }
    }
    __syncthreads();
    // per digit: warps' counts -> warp offsets inside the digit; digit totals
    for (uint32_t dg = tid; dg < SORT_MAX_BINS; dg += SORT_ETHREADS) {
        uint32_t run = 0;
#pragma unroll
        for (uint32_t w = 0; w < SORT_WARPS; w++) {
            const uint32_t c = wcnt[w][dg];
            wcnt[w][dg] = run;
            run += c;
        }
        loff[dg] = dg < NB ? run : 0;
        goff[dg] = dg < NB ? hoff[(size_t)dg * ntiles + blockIdx.x] : 0;
    }
    __syncthreads();
    // exclusive scan of the digit totals (SORT_MAX_BINS == SORT_ETHREADS)
    {
        const uint32_t c = loff[tid];
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        if (lane == 31) wtot[warp] = incl;
        __syncthreads();
        uint32_t add = 0;
        for (uint32_t w = 0; w < warp; w++) add += wtot[w];
        __syncthreads();
        loff[tid] = add + incl - c;
    }
    __syncthreads();
    // pass 2: re-read the tile (it is in L2) and stage it in digit order
#pragma unroll
    for (uint32_t r = 0; r < SORT_ROUNDS; r++) {
        const uint64_t i = t0 + r * 32 + lane;
        if (i < total) {
            const uint32_t d = kr[r] & 0xffffu;
            stage[loff[d] + wcnt[warp][d] + (kr[r] >> 16)] = A[i];
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < n_tile; i += SORT_ETHREADS) {
        const uint2 v = stage[i];
        const uint32_t d = (v.x >> shift) & MASK;
        B[(size_t)goff[d] + (i - loff[d])] = v;
    }
}

// ------------------------------------------------------------ loads/stores

template <class P>
ZK_DEV void load_fe(Fe<P>& f, const uint4* __restrict__ s) {
#pragma unroll
    for (int i = 0; i < P::N / 4; i++) {
        uint4 q = __ldg(s + i);
        f.v[4 * i] = q.x; f.v[4 * i + 1] = q.y; f.v[4 * i + 2] = q.z; f.v[4 * i + 3] = q.w;
    }
}

template <class P>
ZK_DEV void store_fe(uint4* d, const Fe<P>& f) {
#pragma unroll
    for (int i = 0; i < P::N / 4; i++) d[i] = make_uint4(f.v[4 * i], f.v[4 * i + 1], f.v[4 * i + 2], f.v[4 * i + 3]);
}

template <class P>
ZK_DEV void load_affine(Affine<P>& a, const uint32_t* __restrict__ table, uint32_t idx) {
    const uint4* s = reinterpret_cast<const uint4*>(table + (size_t)idx * 2 * P::N);
    load_fe(a.x, s);
    load_fe(a.y, s + P::N / 4);
}

template <class P>
ZK_DEV void load_xyzz(Xyzz<P>& a, const Xyzz<P>* __restrict__ src) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    load_fe(a.x, s);
    load_fe(a.y, s + P::N / 4);
    load_fe(a.zz, s + P::N / 2);
    load_fe(a.zzz, s + 3 * P::N / 4);
}

template <class P>
ZK_DEV void store_xyzz(Xyzz<P>* dst, const Xyzz<P>& a) {
    uint4* d = reinterpret_cast<uint4*>(dst);
    store_fe(d, a.x);
    store_fe(d + P::N / 4, a.y);
    store_fe(d + P::N / 2, a.zz);
    store_fe(d + 3 * P::N / 4, a.zzz);
}

// ------------------------------------------------------------ endomorphism

// phi[i] = (beta * x_i, y_i)   [glv_kernels.metal:260-297]; on BN254 G2
// (Glv::PSI) the image is psi(P) = (conj(x) * GAMMA1, conj(y) * GAMMA2), the
// Frobenius endomorphism of the twist, = (p mod r) * P on G2
template <class C>
__global__ void __launch_bounds__(256) k_endo(const uint32_t* __restrict__ bases, uint32_t n,
                                              uint32_t* __restrict__ phi) {
    using P = typename C::Fp;
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Affine<P> a;
    load_affine(a, bases, i);
    if constexpr (C::Glv::PSI) {
        Fe<P> g1, g2;
#pragma unroll
        for (int l = 0; l < P::N; l++) {
            g1.v[l] = C::Glv::GAMMA1_MONT(l);
            g2.v[l] = C::Glv::GAMMA2_MONT(l);
        }
        conj_fp2(a.x);
        conj_fp2(a.y);
        fe_mul(a.x, a.x, g1);
        fe_mul(a.y, a.y, g2);
    } else {
        Fe<P> beta;
#pragma unroll
        for (int l = 0; l < P::N; l++) beta.v[l] = C::Glv::BETA_MONT(l);
        fe_mul(a.x, a.x, beta);
    }
    uint4* d = reinterpret_cast<uint4*>(phi + (size_t)i * 2 * P::N);
    store_fe(d, a.x);
    store_fe(d + P::N / 4, a.y);
}

// ------------------------------------------------------------ shift tables
//
// A resident table of n affine points extended with window shifts: copy k
// (0 <= k < copies) holds 2^(s*k) * P_i at index k*n + i, copy 0 being the
// points themselves.  An MSM over the table with window width c (a multiple
// of s) then takes window w's digit against copy w*c/s, so every window
// adds into one bucket set and the result needs no doublings.  Replaces the
// reference's BGMW precomputation (MSM/MSMPrecomputation.swift:17-274,
// bn254_msm.c:2163-2230), whose tables hold every digit multiple of every
// window shift (2^c - 1 points per window per base); here only the shifts
// are stored and the digit multiples come from the bucket method.

// Step 1, points [i0, i0 + m): the doubling chain of each point in XYZZ,
// copy k >= 1 of point i0 + j to scratch[(k - 1) * m + j].
template <class C>
__global__ void __launch_bounds__(128) k_shift_chain(const uint32_t* __restrict__ pts, uint32_t i0, uint32_t m,
                                                     uint32_t s, uint32_t copies,
                                                     Xyzz<typename C::Fp>* __restrict__ scratch) {
    using P = typename C::Fp;
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    Affine<P> a;
    load_affine(a, pts, i0 + j);
    Xyzz<P> acc;
    xyzz_from_affine(acc, a);
#pragma unroll 1
    for (uint32_t k = 1; k < copies; k++) {
#pragma unroll 1
        for (uint32_t b = 0; b < s; b++) xyzz_dbl_ni(acc, acc);
        store_xyzz(scratch + (size_t)(k - 1) * m + j, acc);
    }
}

// Step 2: scratch element e = (k - 1) * m + j to affine at table index
// k * n + i0 + j, SHIFT_G consecutive elements per thread sharing one
// inversion (simultaneous inversion: prefix products forward, then one
// inverse unwound backwards).  The identity (ZZ = 0) becomes (0, 0) and
// contributes 1 to the products.
constexpr uint32_t SHIFT_G = 16;
template <class C>
__global__ void __launch_bounds__(128) k_shift_affine(const Xyzz<typename C::Fp>* __restrict__ scratch,
                                                      uint64_t total, uint32_t m, uint32_t i0, uint64_t n,
                                                      uint32_t* __restrict__ table) {
    using P = typename C::Fp;
    const uint64_t e0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * SHIFT_G;
    if (e0 >= total) return;
    const uint32_t cnt = (uint32_t)(total - e0 < SHIFT_G ? total - e0 : SHIFT_G);
    Fe<P> pre[SHIFT_G];
    Fe<P> acc, t;
    fe_set_one(acc);
#pragma unroll 1
    for (uint32_t g = 0; g < cnt; g++) {
        Xyzz<P> q;
        load_xyzz(q, scratch + e0 + g);
        pre[g] = acc;
        if (!xyzz_is_id(q)) {
            fe_mul(t, q.zz, q.zzz);
            fe_mul(acc, acc, t);
        }
    }
    Fe<P> inv;
    fe_inv(inv, acc);
#pragma unroll 1
    for (int g = (int)cnt - 1; g >= 0; g--) {
        Xyzz<P> q;
        load_xyzz(q, scratch + e0 + g);
        const uint64_t e = e0 + (uint32_t)g;
        const uint64_t k = e / m + 1, j = e % m;
        uint4* d = reinterpret_cast<uint4*>(table + (size_t)(k * n + i0 + j) * 2 * P::N);
        Affine<P> a;
        if (xyzz_is_id(q)) {
            fe_set_zero(a.x);
            fe_set_zero(a.y);
        } else {
            Fe<P> it, u;
            fe_mul(it, inv, pre[g]);    // 1 / (ZZ * ZZZ)
            fe_mul(t, q.zz, q.zzz);
            fe_mul(inv, inv, t);        // 1 / (product of the earlier elements)
            fe_mul(u, it, q.zzz);       // 1 / ZZ
            fe_mul(a.x, q.x, u);
            fe_mul(u, it, q.zz);        // 1 / ZZZ
            fe_mul(a.y, q.y, u);
        }
        store_fe(d, a.x);
        store_fe(d + P::N / 4, a.y);
    }
}

// ------------------------------------------------------------ segmented sums

// Bucket sums are segmented sums of the sorted entry list, in levels.  A level
// cuts its list into chunks; runs of one key strictly inside a chunk are
// final and go to their buckets, and chunk t hands its first run to slot 2t
// and its last run to slot 2t + 1 of the next level's list (ACC_EMPTY there
// when one run fills the chunk), still sorted by key.  Whether a boundary run
// really goes on in the neighbouring chunk is left to the next level, so no
// level counts or scans slots (two to four launches a level, which were a
// third of a small call's launches), and the list length
// 2 * ceil(length / chunk) needs no host.  The last level is one block, whose
// boundary runs are final too.
constexpr uint32_t ACC_EMPTY = 0xffffffffu;  // above every bucket id

// Level 1: chunks of the sorted entry list, mixed additions of gathered bases.
// Launch shape of k_acc_l1 per curve: BN254 fits two 256-thread blocks per
// SM at its natural 114 registers; BLS12-381 (158 registers unbounded) is
// held to 128 registers for two blocks per SM, 8% faster despite a few
// spilled bytes (measured at 2^22).
template <class C>
struct AccLaunch {
    static constexpr int THREADS = 256, MIN_BLOCKS = 1;
};
template <>
struct AccLaunch<Bls381> {
    static constexpr int THREADS = 256, MIN_BLOCKS = 2;
};
template <>
struct AccLaunch<Bls377> {  // the same 12-limb arithmetic as BLS12-381
    static constexpr int THREADS = 256, MIN_BLOCKS = 2;
};

// Chunk length for M entries where the plan has T chunks of K for the entries
// there may be.  Zero digits leave fewer (a third, witness-like scalars), and
// chunks of K would then fill part of a wave of resident threads (wave; 0: K
// whatever M is).  So the entries go to whole waves, in chunks of at most 9/8 K
// (rather than one wave more) and at most T of them.  BN254, witness-like scalars, K throughout and now: 600001
// points 1630 and 1136 us, 1024 MSMs of 1024 points 7371 and 5633 us.
ZK_DEV uint32_t acc_chunk(uint32_t M, uint32_t K, uint32_t T, uint32_t wave) {
    const uint64_t per = (uint64_t)K * wave;
    if (per == 0 || M == 0) return K;
    const uint64_t parts = min(max((M + per - per / 8 - 1) / per, (uint64_t)1) * wave, (uint64_t)T);
    return max(8u, (uint32_t)((M + parts - 1) / parts));
}

template <class C>
__global__ void __launch_bounds__(AccLaunch<C>::THREADS, AccLaunch<C>::MIN_BLOCKS) k_acc_l1(const uint2* __restrict__ ents,
                                                const uint32_t* __restrict__ d_len, uint32_t K, uint32_t T,
                                                uint32_t wave, uint32_t t0,
                                                const uint32_t* __restrict__ bases,
                                                const uint32_t* __restrict__ phi,
                                                uint32_t* __restrict__ d_next,
                                                Xyzz<typename C::Fp>* __restrict__ buckets,
                                                uint32_t* __restrict__ pkeys,
                                                Xyzz<typename C::Fp>* __restrict__ pvals) {
    using P = typename C::Fp;
    uint32_t t = t0 + blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t M = *d_len;
    K = acc_chunk(M, K, T, wave);
    if (t == 0) *d_next = (uint32_t)(2 * (((uint64_t)M + K - 1) / K));
    uint64_t start64 = (uint64_t)t * K;
    if (start64 >= M) return;
    uint32_t start = (uint32_t)start64;
    uint32_t end = (uint32_t)(start64 + K < (uint64_t)M ? start64 + K : (uint64_t)M);
    uint32_t cur = ents[start].x;
    bool first_run = true;
    Xyzz<P> acc;
    xyzz_set_id(acc);
#pragma unroll 1
    for (uint32_t i = start; i < end; i++) {
        const uint2 e = ents[i];
        const uint32_t k = e.x;
        if (k != cur) {
            if (first_run) pkeys[2 * t] = cur;
            store_xyzz(first_run ? pvals + 2 * t : buckets + cur, acc);
            xyzz_set_id(acc);
            cur = k;
            first_run = false;
        }
        const uint32_t v = e.y;
        Affine<P> q;
        load_affine(q, (v >> 30) & 1 ? phi : bases, v & VAL_IDX_MASK);
        if (!affine_is_id(q)) {
            if (v >> 31) fe_neg(q.y, q.y);
            xyzz_add_affine(acc, q);
        }
    }
    const uint32_t slot = 2 * t + (first_run ? 0 : 1);
    pkeys[slot] = cur;
    store_xyzz(pvals + slot, acc);
    if (first_run) pkeys[2 * t + 1] = ACC_EMPTY;
}

// Stripes of one MSM (same window layout, S bucket arrays of nb buckets one
// after another): bucket i of array 0 becomes the sum of bucket i of all S.
template <class C>
__global__ void __launch_bounds__(128) k_bucket_fold(Xyzz<typename C::Fp>* __restrict__ b, uint32_t nb,
                                                     uint32_t S) {
    using P = typename C::Fp;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    Xyzz<P> acc;
    load_xyzz(acc, b + i);
#pragma unroll 1
    for (uint32_t s = 1; s < S; s++) {
        Xyzz<P> q;
        load_xyzz(q, b + (size_t)s * nb + i);
        xyzz_add_ni(acc, q);
    }
    store_xyzz(b + i, acc);
}

// The levels after the first, and for small calls the first as well: one
// block folds FOLD_QUADS * J leaves.  A leaf is one run: a slot of the previous
// level's list or (ENTS) a sorted entry's point.  Quad i adds up leaves
// [i*J, (i+1)*J) one after another, then the quads' nodes merge in a tree,
// three levels inside each warp and three over the eight warps.  A node is
// the first and last run of its range (one run when `whole`); everything
// between is final and already in its bucket, so a merge is one addition at
// most (the left node's last run and the right node's first, when the keys
// agree).
//
// Latency-bound in small calls: J + 5 additions deep per level of 64 J leaves.
// BN254 at 2^8 points (16k entries, J = 4): two levels, 33 + 20 us, against
// 57 us for chunks of eight in one thread each, then four levels of sixteen
// (201 us) with a count and a scan each (21 us).  2^16 points, after
// k_acc_l1: 84 against 354 us + 45 us of counts and scans.
template <class P>
struct FoldNode {
    Fe<P> l, r;       // this lane's coordinate of the first / last run's sum
    uint32_t kl, kr;  // their keys; kl = ACC_EMPTY: nothing in the range
    bool whole;       // the range is one run: l, kl (r, kr unused)
};

// a = a ++ b for the quads with `on` set (all lanes call)
template <class P>
ZK_DEV void fold_merge(FoldNode<P>& a, const FoldNode<P>& b, bool on, uint32_t q, Xyzz<P>* __restrict__ buckets) {
    on = on && b.kl != ACC_EMPTY;
    const bool take = on && a.kl == ACC_EMPTY;  // nothing on the left yet
    const uint32_t ka = a.whole ? a.kl : a.kr;
    const bool same = on && ka == b.kl;
    Fe<P> s, x;
    fe_select(s, a.whole, a.l, a.r);
    if (__any_sync(0xffffffffu, same)) {
        fe_set_zero(x);
        fe_select(x, same, b.l, x);
        quad_add(s, x, q);
    }
    if (!on) return;
    if (take) {
        a = b;
        return;
    }
    // runs that end inside the merged range
    if (!a.whole && !(same && b.whole)) quad_store(buckets + ka, s, q);
    if (!same && !b.whole) quad_store(buckets + b.kl, b.l, q);
    if (same && a.whole) a.l = s;
    if (same && b.whole) {
        if (!a.whole) a.r = s;
    } else {
        a.r = b.whole ? b.l : b.r;
        a.kr = b.whole ? b.kl : b.kr;
        a.whole = false;
    }
}

// the node of the quad `delta` quads further in the warp
template <class P>
ZK_DEV void fold_shfl(FoldNode<P>& b, const FoldNode<P>& a, uint32_t delta) {
#pragma unroll
    for (int i = 0; i < P::N; i++) {
        b.l.v[i] = __shfl_down_sync(0xffffffffu, a.l.v[i], 4 * delta);
        b.r.v[i] = __shfl_down_sync(0xffffffffu, a.r.v[i], 4 * delta);
    }
    b.kl = __shfl_down_sync(0xffffffffu, a.kl, 4 * delta);
    b.kr = __shfl_down_sync(0xffffffffu, a.kr, 4 * delta);
    b.whole = __shfl_down_sync(0xffffffffu, a.whole ? 1u : 0u, 4 * delta) != 0;
}

template <class C, bool ENTS>
__global__ void __launch_bounds__(FOLD_THREADS) k_acc_fold(const uint2* __restrict__ ents,
                                                           const uint32_t* __restrict__ bases,
                                                           const uint32_t* __restrict__ phi,
                                                           const uint32_t* __restrict__ keys,
                                                           const Xyzz<typename C::Fp>* __restrict__ vals,
                                                           const uint32_t* __restrict__ d_len, uint32_t J,
                                                           bool last, uint32_t* __restrict__ d_next,
                                                           Xyzz<typename C::Fp>* __restrict__ buckets,
                                                           uint32_t* __restrict__ pkeys,
                                                           Xyzz<typename C::Fp>* __restrict__ pvals) {
    using P = typename C::Fp;
    constexpr uint32_t WARPS = FOLD_THREADS / 32;
    static_assert(WARPS == 8, "the warps' nodes fill the quads of one warp");
    __shared__ uint4 sh_raw[WARPS * 2 * sizeof(Xyzz<P>) / sizeof(uint4)];
    __shared__ uint32_t shk[WARPS], shr[WARPS];
    __shared__ bool shw[WARPS];
    Xyzz<P>* sh = reinterpret_cast<Xyzz<P>*>(sh_raw);
    const uint32_t q = threadIdx.x & 3, quad = threadIdx.x >> 2, warp = threadIdx.x >> 5;
    const uint32_t M = *d_len, K = FOLD_QUADS * J;
    if (blockIdx.x == 0 && threadIdx.x == 0) *d_next = (uint32_t)(2 * (((uint64_t)M + K - 1) / K));
    if ((uint64_t)blockIdx.x * K >= M) return;  // block-uniform
    const uint64_t i0 = (uint64_t)blockIdx.x * K + (uint64_t)quad * J;
    FoldNode<P> a, b;
    fe_set_zero(a.l);
    a.r = b.r = a.l;
    a.kl = a.kr = b.kr = ACC_EMPTY;
    a.whole = true;
#pragma unroll 1
    for (uint32_t j = 0; j < J; j++) {
        const uint64_t i = i0 + j;
        b.kl = ACC_EMPTY;
        b.whole = true;
        fe_set_zero(b.l);
        if (i < M) {
            if (ENTS) {
                const uint2 e = ents[i];
                b.kl = e.x;
                // lanes 0 and 1 take x and +-y, lanes 2 and 3 one; the
                // identity (0, 0) stays all zeros
                const uint4* s = reinterpret_cast<const uint4*>(((e.y >> 30) & 1 ? phi : bases) +
                                                                (size_t)(e.y & VAL_IDX_MASK) * 2 * P::N);
                Affine<P> pt;
                load_fe(pt.x, s);
                load_fe(pt.y, s + P::N / 4);
                if (!affine_is_id(pt)) {
                    if (e.y >> 31) fe_neg(pt.y, pt.y);
                    Fe<P> one;
                    fe_set_one(one);
                    fe_select(b.l, q == 0, pt.x, pt.y);
                    fe_select(b.l, q & 2u, one, b.l);
                }
            } else {
                b.kl = keys[i];
                if (b.kl != ACC_EMPTY) quad_load(b.l, vals + i, q);
            }
        }
        fold_merge(a, b, true, q, buckets);
    }
#pragma unroll 1
    for (uint32_t st = 1; st < 8; st <<= 1) {
        fold_shfl(b, a, st);
        fold_merge(a, b, !(quad & (2 * st - 1)), q, buckets);
    }
    if (!(quad & 7)) {
        quad_store(sh + 2 * warp, a.l, q);
        quad_store(sh + 2 * warp + 1, a.r, q);
        if (q == 0) {
            shk[warp] = a.kl;
            shr[warp] = a.kr;
            shw[warp] = a.whole;
        }
    }
    __syncthreads();
    if (warp != 0) return;
    quad_load(a.l, sh + 2 * quad, q);
    quad_load(a.r, sh + 2 * quad + 1, q);
    a.kl = shk[quad];
    a.kr = shr[quad];
    a.whole = shw[quad];
#pragma unroll 1
    for (uint32_t st = 1; st < WARPS; st <<= 1) {
        fold_shfl(b, a, st);
        fold_merge(a, b, !(quad & (2 * st - 1)), q, buckets);
    }
    if (quad != 0) return;
    if (last) {
        quad_store(buckets + a.kl, a.l, q);
        if (!a.whole) quad_store(buckets + a.kr, a.r, q);
    } else {
        const uint64_t o = 2 * (uint64_t)blockIdx.x;
        quad_store(pvals + o, a.l, q);
        if (!a.whole) quad_store(pvals + o + 1, a.r, q);
        if (q == 0) {
            pkeys[o] = a.kl;
            pkeys[o + 1] = a.whole ? ACC_EMPTY : a.kr;
        }
    }
}

// ------------------------------------------------------------ bucket reduction
//
// A window's sum is sum_{b=1..B} b*B_b = sum_i (i+1) A_i with A_i = B_{i+1}.
// A node over a bucket range keeps S = sum A_i and W = sum (i - lo) A_i.
// Merging L children of span `span`: S' = sum S_s and
// W' = sum W_s + span * sum_s s*S_s, the last sum by a running sum.
// k_reduce_level does that with one thread per node while the nodes fill the
// multiply pipe.  With fewer nodes a chain of 2L additions in one thread
// costs 8.7 us an addition (BN254), 180-200 us a level whatever its size (BN254
// 2^20: 907 us for five levels; now 151 us for the first, 70 + 22 us for the
// quads; 2^16: 365 us for three, now 82 + 22), so the rest of the tree goes to
// quads of lanes and to plain sums instead: sum_i i*S_i = sum_j 2^j T_j, T_j
// the sum of the S_i whose index has bit j set, all of them by-products of one
// tree of depth log2(nodes) (k_reduce_quads, k_reduce_windows), and k_combine
// shifts the T_j into place on its chain of doublings, which passes those bits
// anyway.

ZK_DEV int find_task(const RedTask* __restrict__ t, int nt, uint32_t g) {
    int lo = 0, hi = nt - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (t[mid].out_off <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <class C>
__global__ void __launch_bounds__(128) k_reduce_level(const Xyzz<typename C::Fp>* __restrict__ inS,
                                                      const Xyzz<typename C::Fp>* __restrict__ inW,
                                                      const RedTask* __restrict__ tasks, int ntasks,
                                                      uint32_t nout_total, uint32_t L, uint32_t log2span,
                                                      uint32_t step,  // between outputs
                                                      Xyzz<typename C::Fp>* __restrict__ outS,
                                                      Xyzz<typename C::Fp>* __restrict__ outW) {
    using P = typename C::Fp;
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nout_total) return;
    const RedTask tk = tasks[find_task(tasks, ntasks, g)];
    uint32_t local = g - tk.out_off;
    uint32_t c0 = tk.in_off + local * L;
    uint32_t cnt = min(L, tk.n_in - local * L);
    Xyzz<P> run, x, q;
    xyzz_set_id(run);
    xyzz_set_id(x);
#pragma unroll 1
    for (int s = (int)cnt - 1; s >= 1; s--) {
        load_xyzz(q, inS + c0 + s);
        xyzz_add(run, q);
        xyzz_add(x, run);
    }
    load_xyzz(q, inS + c0);
    xyzz_add(run, q);
    store_xyzz(outS + (size_t)g * step, run);
#pragma unroll 1
    for (uint32_t d = 0; d < log2span; d++) xyzz_dbl(x, x);
    if (inW != nullptr) {
#pragma unroll 1
        for (uint32_t s = 0; s < cnt; s++) {
            load_xyzz(q, inW + c0 + s);
            xyzz_add(x, q);
        }
    }
    store_xyzz(outW + (size_t)g * step, x);
}

// One step of the tree over the quads of a warp (st < 8) or a block: quad i
// holds S of the nodes it stands for, and w, a plain sum.  Quad i with bit st
// clear and at most one lower bit set adds the S of quad i + st: no lower bit
// set continues the sum of all S, bit j alone continues T_j (whose terms are
// the S that quads with bit j set held at step j).  The w's travel to the
// quad whose lower bits are all set: quad i with bit st set and all lower
// bits set adds quad i - st's w.  So a quad does one addition at most.
template <class P>
ZK_DEV void reduce_step(Fe<P>& S, Fe<P>& w, uint32_t i, uint32_t st, uint32_t q, const Fe<P>& got) {
    const uint32_t low = i & (st - 1);
    const bool up = i & st;
    const bool on = up ? low == st - 1 : (low & (low - 1)) == 0;
    Fe<P> a, b;
    fe_select(a, up, w, S);
    fe_set_zero(b);
    fe_select(b, on, got, b);
    quad_add(a, b, q);
    fe_select(w, up, a, w);
    fe_select(S, up, S, a);
}

// What the partner of quad i at this step needs: its S from above, w from below.
template <class P>
ZK_DEV void reduce_swap(Fe<P>& got, const Fe<P>& S, const Fe<P>& w, uint32_t i, uint32_t st) {
    Fe<P> send;
    fe_select(send, (i & st) != 0, S, w);
#pragma unroll
    for (int l = 0; l < P::N; l++) got.v[l] = __shfl_xor_sync(0xffffffffu, send.v[l], 4 * st);
}

// The nodes of every window (tasks: one per window, n_out blocks each from
// block out_off) in blocks of RED_QUADS * J, or one block of fewer quads (a
// power of two, 8 at least) when no window fills more; quad i sums nodes
// [i*J, (i+1)*J) by a running sum, x = sum s*S_s shifted by the nodes' span
// (2^log2span) and added to the nodes' W, then log2(quads) tree steps.  Block
// b writes RED_SLOTS1 points: S | T_0 .. T_5 | W (no T_j from the block's
// quads on), with the window's sum = S + W + sum_j 2^(log2span + log2J + j) T_j
// when it is one block.  Warps whose quads no node reaches skip the additions.
// 256 MSMs of 64 points (BN254, 8192 windows of eight nodes): 94 us with one
// warp a window, 667 with eight.  Where the levels before leave one node per
// window, k_reduce_level writes the combine's terms itself: 4096 MSMs of 16
// points 467 us, 6093 with a block of eight warps to copy each node.
template <class C>
__global__ void __launch_bounds__(4 * RED_QUADS) k_reduce_quads(const Xyzz<typename C::Fp>* __restrict__ inS,
                                                                const Xyzz<typename C::Fp>* __restrict__ inW,
                                                                const RedTask* __restrict__ tasks, int ntasks,
                                                                uint32_t J, uint32_t log2span,
                                                                Xyzz<typename C::Fp>* __restrict__ out) {
    using P = typename C::Fp;
    __shared__ uint4 sh_raw[RED_QUADS * sizeof(Xyzz<P>) / sizeof(uint4)];
    Xyzz<P>* sh = reinterpret_cast<Xyzz<P>*>(sh_raw);
    const uint32_t i = threadIdx.x >> 2, q = threadIdx.x & 3;
    const RedTask tk = tasks[find_task(tasks, ntasks, blockIdx.x)];
    const uint32_t n0 = (blockIdx.x - tk.out_off) * RED_QUADS * J;
    const uint32_t cnt = min(RED_QUADS * J, tk.n_in - n0);  // nodes of this block
    const uint32_t base = tk.in_off + n0 + i * J, mine = cnt > i * J ? min(J, cnt - i * J) : 0u;
    const uint32_t used = (cnt + J - 1) / J;       // quads with nodes
    const bool busy = (i & ~7u) < used;            // warp-uniform
    Fe<P> run, x, v;
    fe_set_zero(run);
    fe_set_zero(x);
#pragma unroll 1
    for (uint32_t s = busy ? J : 0; s-- > 0;) {
        fe_set_zero(v);
        if (s < mine) quad_load(v, inS + base + s, q);
        quad_add(run, v, q);
        if (s) quad_add(x, run, q);
    }
    if (busy && inW != nullptr) {
        if (J > 1)
#pragma unroll 1
            for (uint32_t d = 0; d < log2span; d++) quad_dbl(x, q);
#pragma unroll 1
        for (uint32_t s = 0; s < J; s++) {
            fe_set_zero(v);
            if (s < mine) quad_load(v, inW + base + s, q);
            quad_add(x, v, q);
        }
    }
    uint32_t st = 1;
#pragma unroll 1
    for (; st < used; st <<= 1) {
        if (st < 8) {
            if (!busy) continue;
            reduce_swap(v, run, x, i, st);
        } else {
            fe_select(v, (i & st) != 0, run, x);
            quad_store(sh + i, v, q);
            __syncthreads();
            quad_load(v, sh + (i ^ st), q);
            __syncthreads();
        }
        reduce_step(run, x, i, st, q, v);
    }
    // S in quad 0, T_j in quad 2^j below st (none above), W in quad st - 1
    Xyzz<P>* o = out + (size_t)blockIdx.x * RED_SLOTS1;
    if (i == 0) quad_store(o, run, q);
    if (i && !(i & (i - 1))) {
        if (i >= st) fe_set_zero(run);
        quad_store(o + __ffs(i), run, q);
    }
    if (i == st - 1) quad_store(o + RED_SLOTS1 - 1, x, q);
}

// Windows of more than one block: one block per window, warp a sums slot a of
// the window's blocks (quad i: blocks [i*E, (i+1)*E), then three tree steps);
// the S of the blocks give three more bit sums and X = sum over quads of
// their running sums.  Writes RED_SLOTS2 points: S | T_0 .. T_5 | W | X |
// T'_0 .. T'_2, X and T'_j at bits log2block and log2block + log2E + j.
template <class C>
__global__ void __launch_bounds__(32 * RED_SLOTS1) k_reduce_windows(const Xyzz<typename C::Fp>* __restrict__ in,
                                                                    const RedTask* __restrict__ tasks, uint32_t E,
                                                                    Xyzz<typename C::Fp>* __restrict__ out) {
    using P = typename C::Fp;
    const uint32_t a = threadIdx.x >> 5, i = (threadIdx.x >> 2) & 7, q = threadIdx.x & 3;
    const RedTask tk = tasks[blockIdx.x];
    Fe<P> run, x, v;
    fe_set_zero(run);
    fe_set_zero(x);
#pragma unroll 1
    for (uint32_t s = E; s-- > 0;) {
        const uint32_t b = i * E + s;
        fe_set_zero(v);
        if (b < tk.n_out) quad_load(v, in + (size_t)(tk.out_off + b) * RED_SLOTS1 + a, q);
        if (a == 0) {  // warp-uniform
            quad_add(run, v, q);
            if (s) quad_add(x, run, q);
        } else {
            quad_add(x, v, q);
        }
    }
#pragma unroll 1
    for (uint32_t st = 1; st < 8; st <<= 1) {
        reduce_swap(v, run, x, i, st);
        reduce_step(run, x, i, st, q, v);
    }
    Xyzz<P>* o = out + (size_t)blockIdx.x * RED_SLOTS2;
    if (a == 0) {
        if (i == 0) quad_store(o, run, q);
        if (i && !(i & (i - 1))) quad_store(o + RED_SLOTS1 + __ffs(i), run, q);
        if (i == 7) quad_store(o + RED_SLOTS1, x, q);
    } else if (i == 7) {
        quad_store(o + a, x, q);
    }
}

// Window combine, one block per MSM: R = sum over windows w and terms t of
// 2^(bit(w) + bit(t)) * term, the terms being the points k_reduce_quads or
// k_reduce_windows left per window, in order of their bits.  Each window's
// terms go to COMBINE_SPLIT(windows) quads, neighbouring terms together; a
// quad adds its terms up by Horner's rule and doubles the sum down to bit 0,
// a tree through shared memory adds the quads' points, and quad 0 normalises
// to affine and writes the reference-layout Jacobian (X, Y, Z) Montgomery
// with Z = 1 (or the identity (1, 1, 0)).
//
// Latency-bound: one chain of as many doublings as the highest bit (BN254:
// 127), a few additions and one inversion, whatever n is.  A quad (quad.cuh)
// runs a doubling in two product layers, so the chain is about 250 product
// times.  Four warps (32 quads) have a scheduler each; more would queue for
// the multiply pipe, hence the split.  With the bit sums' Horner steps 184 us
// at 2^8 points (BN254, 32 windows) and 195 us at 2^16 (10 windows), BLS12-377
// 10^5 384 us, BN254 G2 2^16 839 us; four warps sharing the layers of XYZZ
// doublings through shared memory, with a binary Euclid and without those
// steps, took 378, 434, 885 and 1034 us.
struct CombineTerms {
    uint32_t slots;     // points per window: RED_SLOTS1, RED_SLOTS2, or 2 (S and W alone)
    uint32_t slot_w;    // of W
    uint32_t used;      // positions (term_slot) that hold points; the rest are zero
    uint32_t bit_t;     // bit of T_0
    uint32_t bit_x;     // RED_SLOTS2: bit of X, and of T'_0
    uint32_t bit_t2;
};

// quads per window
__host__ __device__ inline uint32_t combine_split(uint32_t windows) {
    return windows <= 8 ? 4 : windows <= 16 ? 2 : 1;
}
// threads of k_combine for MSMs of at most `windows` windows (the splits of
// fewer windows need no more quads than 32 or `windows`)
inline uint32_t combine_threads(uint32_t windows) {
    const uint32_t quads = windows * combine_split(windows);
    return windows > 1 && quads < 32 ? 128u : (4 * quads + 31) / 32 * 32;
}

// term at position k in order of bits: its slot and its bit in the window
ZK_DEV uint32_t term_slot(uint32_t k, const CombineTerms& ct) {
    return k == 0 ? 0 : k == 1 ? ct.slot_w : k < RED_SLOTS1 ? k - 1 : k;
}
ZK_DEV uint32_t term_bit(uint32_t k, const CombineTerms& ct) {
    return k < 2 ? 0 : k < RED_SLOTS1 ? ct.bit_t + k - 2 : k == RED_SLOTS1 ? ct.bit_x : ct.bit_t2 + k - RED_SLOTS1 - 1;
}

template <class C>
__global__ void __launch_bounds__(4 * MAX_WINDOWS) k_combine(const Xyzz<typename C::Fp>* __restrict__ terms,
                                                             CombineTerms ct, const MsmDesc* __restrict__ descs,
                                                             int nd, uint32_t* __restrict__ out) {
    using P = typename C::Fp;
    __shared__ uint4 sh_raw[MAX_WINDOWS * sizeof(Xyzz<P>) / sizeof(uint4)];
    Xyzz<P>* sh = reinterpret_cast<Xyzz<P>*>(sh_raw);
    const uint32_t u = threadIdx.x >> 2, q = threadIdx.x & 3, warp = threadIdx.x >> 5;
    const int m = (int)blockIdx.x;
    if (m >= nd) return;  // block-uniform
    const MsmDesc d = descs[m];
    uint32_t* o = out + (size_t)m * 3 * P::N;
    Fe<P> one;
    fe_set_one(one);
    if (d.n == 0) {
        if (threadIdx.x == 0)
            for (int l = 0; l < P::N; l++) { o[l] = one.v[l]; o[P::N + l] = one.v[l]; o[2 * P::N + l] = 0; }
        return;
    }
    const uint32_t split = combine_split(d.nred), nq = d.nred * split;  // quads in use
    const uint32_t w = u / split, per = (ct.used + split - 1) / split;
    const uint32_t lo = (u % split) * per;  // this quad's terms: positions [lo, lo + per)
    // (split divides RED_SLOTS1 and RED_SLOTS2, so positions stay below slots)
    const bool live = u < nq && lo < ct.used;
    const Xyzz<P>* wt = terms + (size_t)(d.win_off + w) * ct.slots;
    Fe<P> a, b;
    fe_set_zero(a);
    if (8 * warp < nq) {  // warp-uniform
        if (live && lo + per <= ct.used) quad_load(a, wt + term_slot(lo + per - 1, ct), q);
#pragma unroll 1
        for (uint32_t k = per - 1; k-- > 0;) {
            const uint32_t cnt = live ? term_bit(lo + k + 1, ct) - term_bit(lo + k, ct) : 0u;
            const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
#pragma unroll 1
            for (uint32_t i = 0; i < most; i++) {
                b = a;
                quad_dbl(b, q);
                fe_select(a, i < cnt, b, a);
            }
            fe_set_zero(b);
            if (live && lo + k < ct.used) quad_load(b, wt + term_slot(lo + k, ct), q);
            quad_add(a, b, q);
        }
        // down to bit 0; a warp runs to the most of its quads
        const uint32_t cnt = live ? win_bit(d, w) + term_bit(lo, ct) : 0u;
        const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
        if (most) {
            const bool chain = QuadChain<C>::on_curve(a, q);
            if (__all_sync(0xffffffffu, chain)) {
                QuadChain<C>::enter(a, q);
#pragma unroll 1
                for (uint32_t i = 0; i < most; i++) {
                    b = a;
                    QuadChain<C>::dbl(b, q);
                    fe_select(a, i < cnt, b, a);
                }
                QuadChain<C>::leave(a, q);
            } else {  // points off the curve in this warp
#pragma unroll 1
                for (uint32_t i = 0; i < most; i++) {
                    b = a;
                    quad_dbl(b, q);
                    fe_select(a, i < cnt, b, a);
                }
            }
        }
    }
    for (uint32_t st = 1; st < nq; st <<= 1) {
        // quads u with bits below st clear hold the sums of [u, u + st)
        if (u & st && !(u & (st - 1))) quad_store(sh + u, a, q);
        __syncthreads();
        if (8 * warp < nq) {  // warp-uniform
            fe_set_zero(b);
            if (!(u & (2 * st - 1)) && u + st < nq) quad_load(b, sh + u + st, q);
            quad_add(a, b, q);
        }
        __syncthreads();
    }
    if (warp != 0) return;
    // x = X / ZZ, y = Y / ZZZ from one inverse of ZZ * ZZZ
    Fe<P> t, zz, zzz;
    quad_get(zz, a, 2);
    quad_get(zzz, a, 3);
    fe_mul(t, zz, zzz);
    const bool id = fe_is_zero(zz);
    fe_inv(t, t);
    fe_select(zz, q == 0, zzz, zz);
    fe_mul(t, t, zz);                 // 1/ZZ | 1/ZZZ
    fe_mul(a, a, t);
    if (threadIdx.x < 3) {
        const bool z = q == 2;        // lanes 0 and 1: the coordinates, lane 2: Z
#pragma unroll
        for (int l = 0; l < P::N; l++) o[q * P::N + l] = z ? (id ? 0u : one.v[l]) : id ? one.v[l] : a.v[l];
    }
}

// ------------------------------------------------------------ scan (u32)

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

ZK_DEV uint32_t block_excl_scan(uint32_t v, uint32_t* sh, uint32_t& total) {
    uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t s = lane < SCAN_THREADS / 32 ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= (uint32_t)o) s += y;
        }
        if (lane < SCAN_THREADS / 32) sh[lane] = s;
    }
    __syncthreads();
    total = sh[SCAN_THREADS / 32 - 1];
    uint32_t pre = wid ? sh[wid - 1] : 0;
    __syncthreads();
    return pre + x - v;
}

// phase 1: per-tile exclusive scan, tile totals
static __global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(const uint32_t* __restrict__ in, uint32_t n,
                                                             uint32_t* __restrict__ out,
                                                             uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t sh[SCAN_THREADS / 32];
    uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS], s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        v[i] = base + i < n ? in[base + i] : 0;
        s += v[i];
    }
    uint32_t total;
    uint32_t pre = block_excl_scan(s, sh, total);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        if (base + i < n) out[base + i] = pre;
        pre += v[i];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// the whole scan in one launch when the array fits one tile (small MSMs run a
// dozen such scans, each otherwise three dependent launches)
static __global__ void __launch_bounds__(SCAN_THREADS) k_scan_single(uint32_t* __restrict__ data, uint32_t n,
                                                              uint32_t* __restrict__ d_total,
                                                              uint32_t* __restrict__ copy) {
    __shared__ uint32_t sh[SCAN_THREADS / 32];
    const uint32_t base = threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS], s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        v[i] = base + i < n ? data[base + i] : 0;
        s += v[i];
    }
    uint32_t total;
    uint32_t pre = block_excl_scan(s, sh, total);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        if (base + i < n) {
            data[base + i] = pre;
            if (copy) copy[base + i] = pre;
        }
        pre += v[i];
    }
    if (threadIdx.x == 0) *d_total = total;
}

// phase 2: one block scans the tile totals in place; writes the grand total
static __global__ void __launch_bounds__(SCAN_THREADS) k_scan_sums(uint32_t* __restrict__ tile_sums, uint32_t ntiles,
                                                            uint32_t* __restrict__ d_total) {
    __shared__ uint32_t sh[SCAN_THREADS / 32];
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < ntiles; b0 += SCAN_THREADS) {
        uint32_t i = b0 + threadIdx.x;
        uint32_t v = i < ntiles ? tile_sums[i] : 0;
        uint32_t total;
        uint32_t pre = block_excl_scan(v, sh, total);
        if (i < ntiles) tile_sums[i] = carry + pre;
        carry += total;
    }
    if (threadIdx.x == 0) *d_total = carry;
}

// phase 3: add tile offsets; optionally duplicate into a second array
static __global__ void __launch_bounds__(SCAN_THREADS) k_scan_add(uint32_t* __restrict__ out, uint32_t n,
                                                           const uint32_t* __restrict__ tile_sums,
                                                           uint32_t* __restrict__ copy) {
    uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    uint32_t add = tile_sums[blockIdx.x];
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        uint64_t j = base + (uint64_t)i * SCAN_THREADS + threadIdx.x;
        if (j < n) {
            uint32_t v = out[j] + add;
            out[j] = v;
            if (copy) copy[j] = v;
        }
    }
}

// ------------------------------------------------------------ MSD radix sort
// Large entry sets are sorted most-significant digit first, in two passes of
// up to 12 bits (one pass for keys of up to 12 bits).  An MSD pass needs no
// stability -- entries of one bucket may come out in any order, since bucket
// sums do not depend on it -- so a tile ranks its entries by digit with
// shared-memory atomics instead of the per-bit ballots a stable LSD pass
// needs.  A pass runs over tiles of at most MSD_TILE entries that never
// straddle a segment (pass 1: the whole array is one segment; pass 2: one
// segment per pass-1 digit), and the tiles come in groups of consecutive
// tiles of one segment (pass 1: the tiles split evenly over `ng` groups,
// about one per SM; pass 2: chunks of at most MSD_CHUNK_TILES tiles of a
// segment).  Output order inside a segment: digit, then group, then tile.
//  k_msd_count      each tile's digit counts as a contiguous row C[tile][digit]
//                   (pass 1 from the 2-byte digit array the digit kernel
//                   writes beside the entries, pass 2 from the entries'
//                   keys), and the group's digit totals straight into the
//                   scan layout S[seg][digit][group of seg], so that an exclusive
//                   scan of S gives each (seg, digit, group) the first output
//                   slot of its run (pass 1 counts each group in `sub` parts,
//                   S[digit][group][part], so that two count blocks share an
//                   SM);
//  scan;
//  k_msd_prefix     per group: the slot rows P[tile][digit], the group's
//                   scanned slot plus the counts of its earlier tiles;
//  k_msd_tiles      (between the passes) the segment starts, read from the
//                   pass-1 scan, and the pass-2 tile and chunk tables;
//  k_msd_scatter    one block per tile: reads its count row (local offsets)
//                   and slot row, places the tile in digit order in shared
//                   memory and writes it out as one run per digit.
// The scan layout holds one word per group and digit (pass 1: at most 4.8 MB
// at any size), not one per tile, so the tile rows never need transposing; the
// scatter keeps one block per tile because blocks placing neighbouring
// tiles at the same time write their runs of a digit side by side (one block
// placing a whole group wrote 148 x 4096 separate fronts at 2^24 points and
// took 2.10 ms against 1.28 ms for pass 1).
// Replaces the reference's CPU counting sort per window (MSMEngine.swift:595-661).

// Group (or, for the count kernel of pass 1, part of a group) u of a pass.
// Pass 1 (seg_chunk == nullptr): the ceil(E / MSD_TILE) tiles of [0, E) are
// split into `ng` groups of K = ceil(tiles / ng) tiles, each counted in
// `sub` parts of ceil(K / sub) tiles; the count kernel runs ng*sub units
// (u = group*sub + part), the slot-row kernel ng (u = group, whole groups,
// part 0's scan slot).  Every unit exists (groups past the last tile are empty and
// count zeros).  Pass 2: chunk u of the chunk table seg_chunk (exclusive
// prefix of chunks per segment, nseg + 1 entries), with the tile table
// seg_tile and segment starts seg_start (nseg + 1 entries each, the last
// start E); false past the last chunk.  lo..hi: the entries; row0: the
// count row of the first tile; S[sidx + digit*sstride]: the unit's slot in
// the scan layout.
struct MsdGroup {
    uint32_t lo, hi, row0, sstride;
    uint64_t sidx;
};

ZK_DEV bool msd_group(uint32_t u, uint32_t E, uint32_t ng, uint32_t sub, bool whole,
                      const uint32_t* __restrict__ seg_start, const uint32_t* __restrict__ seg_tile,
                      const uint32_t* __restrict__ seg_chunk, uint32_t nseg, uint32_t nb, MsdGroup& g) {
    if (!seg_chunk) {
        const uint32_t grp = whole ? u : u / sub, part = whole ? 0 : u % sub;
        if (grp >= ng) return false;
        const uint32_t nt = (uint32_t)(((uint64_t)E + MSD_TILE - 1) / MSD_TILE);
        const uint32_t K = (nt + ng - 1) / ng, Ks = (K + sub - 1) / sub;
        const uint64_t gend = (uint64_t)(grp + 1) * K;
        uint64_t t0 = (uint64_t)grp * K, t1 = gend;
        if (!whole) {
            t0 += (uint64_t)part * Ks;
            t1 = t0 + Ks < gend ? t0 + Ks : gend;
        }
        if (t1 > nt) t1 = nt;
        if (t0 > t1) t0 = t1;
        g.row0 = (uint32_t)t0;
        g.lo = (uint32_t)(t0 * MSD_TILE < E ? t0 * MSD_TILE : E);
        g.hi = (uint32_t)(t1 * MSD_TILE < E ? t1 * MSD_TILE : E);
        g.sidx = (uint64_t)grp * sub + part;
        g.sstride = ng * sub;
        return true;
    }
    if (u >= seg_chunk[nseg]) return false;
    // the last segment whose first chunk is at or below u (empty segments
    // before it share its first-chunk index and are skipped)
    uint32_t a = 0, b = nseg - 1;
    while (a < b) {
        const uint32_t mid = (a + b + 1) >> 1;
        if (seg_chunk[mid] <= u) a = mid;
        else b = mid - 1;
    }
    const uint32_t k = u - seg_chunk[a];
    g.row0 = seg_tile[a] + k * MSD_CHUNK_TILES;
    g.lo = seg_start[a] + k * (MSD_CHUNK_TILES * MSD_TILE);
    const uint32_t end = seg_start[a + 1];
    g.hi = end - g.lo > MSD_CHUNK_TILES * MSD_TILE ? g.lo + MSD_CHUNK_TILES * MSD_TILE : end;
    g.sidx = (uint64_t)seg_chunk[a] * nb + k;
    g.sstride = seg_chunk[a + 1] - seg_chunk[a];
    return true;
}

// Exclusive scan over a block of NW warps (sh: NW words).
template <int NW>
ZK_DEV uint32_t block_excl_scan_w(uint32_t v, uint32_t* sh, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t s = lane < (uint32_t)NW ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= (uint32_t)o) s += y;
        }
        if (lane < (uint32_t)NW) sh[lane] = s;
    }
    __syncthreads();
    total = sh[NW - 1];
    const uint32_t pre = wid ? sh[wid - 1] : 0;
    __syncthreads();
    return pre + x - v;
}

// Shared-memory counter bump / slot claim on ctr[key].  A warp whose valid
// lanes all hold one key (a hot bucket, e.g. many scalars equal to 1) takes
// one atomic; otherwise every valid lane takes its own, and the few lanes
// that share a key are serialised by the hardware.  All 32 lanes call it.
ZK_DEV void msd_count_one(uint32_t* __restrict__ ctr, bool valid, uint32_t key) {
    const uint32_t m = __ballot_sync(0xffffffffu, valid);
    if (!m) return;
    const uint32_t leader = __ffs(m) - 1;
    const uint32_t lk = __shfl_sync(0xffffffffu, key, leader);
    if (__all_sync(0xffffffffu, !valid || key == lk)) {
        if ((threadIdx.x & 31) == leader) atomicAdd(ctr + lk, (uint32_t)__popc(m));
    } else if (valid) {
        atomicAdd(ctr + key, 1u);
    }
}

ZK_DEV uint32_t msd_claim_one(uint32_t* __restrict__ ctr, bool valid, uint32_t key) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t m = __ballot_sync(0xffffffffu, valid);
    if (!m) return 0;
    const uint32_t leader = __ffs(m) - 1;
    const uint32_t lk = __shfl_sync(0xffffffffu, key, leader);
    if (__all_sync(0xffffffffu, !valid || key == lk)) {
        uint32_t b = 0;
        if (lane == leader) b = atomicAdd(ctr + lk, (uint32_t)__popc(m));
        b = __shfl_sync(0xffffffffu, b, leader);
        return b + __popc(m & ((1u << lane) - 1));
    }
    return valid ? atomicAdd(ctr + key, 1u) : 0u;
}

constexpr uint32_t MSD_ROUNDS = (MSD_TILE + MSD_THREADS - 1) / MSD_THREADS;
constexpr uint32_t MSD_BATCH = 8;  // entries loaded before they are used
static_assert(MSD_ROUNDS % MSD_BATCH == 0, "tile rounds come in whole load batches");
constexpr uint32_t MSD_PER = (1u << MSD_MAX_BITS) / MSD_THREADS;  // digits per thread in row scans

static __global__ void __launch_bounds__(MSD_THREADS) k_msd_count(const uint16_t* __restrict__ D,
                                                                 const uint2* __restrict__ A, uint32_t shift,
                                                                 const uint32_t* __restrict__ d_total,
                                                                 uint32_t bits, uint32_t ng,
                                                                 uint32_t sub,
                                                                 const uint32_t* __restrict__ seg_start,
                                                                 const uint32_t* __restrict__ seg_tile,
                                                                 const uint32_t* __restrict__ seg_chunk,
                                                                 uint32_t nseg, uint32_t* __restrict__ C,
                                                                 uint32_t* __restrict__ S) {
    __shared__ uint32_t cnt[1u << MSD_MAX_BITS];
    const uint32_t nb = 1u << bits, mask = nb - 1;
    MsdGroup g;
    if (!msd_group(blockIdx.x, *d_total, ng, sub, false, seg_start, seg_tile, seg_chunk, nseg, nb, g)) return;
    for (uint32_t i = threadIdx.x; i < nb; i += MSD_THREADS) cnt[i] = 0;
    __syncthreads();
    uint32_t tot[MSD_PER];
#pragma unroll
    for (uint32_t q = 0; q < MSD_PER; q++) tot[q] = 0;
    uint32_t row = g.row0;
#pragma unroll 1
    for (uint32_t t0 = g.lo; t0 < g.hi; t0 += MSD_TILE, row++) {
        const uint32_t len = g.hi - t0 < MSD_TILE ? g.hi - t0 : MSD_TILE;
#pragma unroll 1
        for (uint32_t r0 = 0; r0 * MSD_THREADS < len; r0 += MSD_BATCH) {
            uint32_t key[MSD_BATCH];
#pragma unroll
            for (uint32_t q = 0; q < MSD_BATCH; q++) {
                const uint32_t j = (r0 + q) * MSD_THREADS + threadIdx.x;
                key[q] = j >= len ? 0xffffffffu
                         : D      ? (uint32_t)D[(uint64_t)t0 + j]
                                  : (A[(uint64_t)t0 + j].x >> shift) & mask;
            }
#pragma unroll
            for (uint32_t q = 0; q < MSD_BATCH; q++) msd_count_one(cnt, key[q] != 0xffffffffu, key[q]);
        }
        __syncthreads();
        // the tile's row; the counters are cleared for the next tile
        uint32_t* crow = C + (uint64_t)row * nb;
#pragma unroll
        for (uint32_t q = 0; q < MSD_PER; q++) {
            const uint32_t d = threadIdx.x * MSD_PER + q;
            if (d < nb) {
                const uint32_t v = cnt[d];
                crow[d] = v;
                tot[q] += v;
                cnt[d] = 0;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (uint32_t q = 0; q < MSD_PER; q++) {
        const uint32_t d = threadIdx.x * MSD_PER + q;
        if (d < nb) S[g.sidx + (uint64_t)d * g.sstride] = tot[q];
    }
}

// Between the passes (one block): seg_start[s] = first output slot of pass-1
// digit s (the scanned slot of (digit s, group 0, part 0), at s * stride1),
// seg_start[nseg] = E; seg_tile and seg_chunk = exclusive prefixes of the
// segments' tiles (ceil(length / MSD_TILE)) and chunks (ceil(tiles /
// MSD_CHUNK_TILES)), nseg + 1 entries each.
static __global__ void __launch_bounds__(MSD_THREADS) k_msd_tiles(const uint32_t* __restrict__ S1,
                                                                 uint32_t stride1, uint32_t nseg,
                                                                 const uint32_t* __restrict__ d_total,
                                                                 uint32_t* __restrict__ seg_start,
                                                                 uint32_t* __restrict__ seg_tile,
                                                                 uint32_t* __restrict__ seg_chunk) {
    __shared__ uint32_t sh[MSD_THREADS / 32];
    const uint32_t E = *d_total;
    uint32_t st[MSD_PER + 1], nt[MSD_PER], nc[MSD_PER], sum = 0, csum = 0;
#pragma unroll
    for (uint32_t q = 0; q <= MSD_PER; q++) {
        const uint32_t s = threadIdx.x * MSD_PER + q;
        st[q] = s < nseg ? S1[(uint64_t)s * stride1] : E;
    }
#pragma unroll
    for (uint32_t q = 0; q < MSD_PER; q++) {
        const uint32_t s = threadIdx.x * MSD_PER + q;
        const uint32_t len = s < nseg ? st[q + 1] - st[q] : 0;
        nt[q] = (len + MSD_TILE - 1) / MSD_TILE;
        nc[q] = (nt[q] + MSD_CHUNK_TILES - 1) / MSD_CHUNK_TILES;
        sum += nt[q];
        csum += nc[q];
    }
    uint32_t total, ctotal;
    uint32_t pre = block_excl_scan_w<MSD_THREADS / 32>(sum, sh, total);
    uint32_t cpre = block_excl_scan_w<MSD_THREADS / 32>(csum, sh, ctotal);
#pragma unroll
    for (uint32_t q = 0; q < MSD_PER; q++) {
        const uint32_t s = threadIdx.x * MSD_PER + q;
        if (s < nseg) {
            seg_start[s] = st[q];
            seg_tile[s] = pre;
            seg_chunk[s] = cpre;
        }
        pre += nt[q];
        cpre += nc[q];
    }
    if (threadIdx.x == 0) {
        seg_start[nseg] = E;
        seg_tile[nseg] = total;
        seg_chunk[nseg] = ctotal;
    }
}

// The slot rows: P[tile][digit] = the first output slot of the tile's run of
// each digit, from the group's scanned slot (part 0's) plus the counts of
// the group's earlier tiles.  One block per group (pass 1) or chunk (pass 2).
static __global__ void __launch_bounds__(MSD_THREADS) k_msd_prefix(const uint32_t* __restrict__ d_total,
                                                                  uint32_t bits, uint32_t ng, uint32_t sub,
                                                                  const uint32_t* __restrict__ seg_start,
                                                                  const uint32_t* __restrict__ seg_tile,
                                                                  const uint32_t* __restrict__ seg_chunk,
                                                                  uint32_t nseg, const uint32_t* __restrict__ C,
                                                                  const uint32_t* __restrict__ S,
                                                                  uint32_t* __restrict__ P) {
    constexpr uint32_t ROWS = 4;  // count rows loaded before any is used
    const uint32_t nb = 1u << bits;
    MsdGroup g;
    if (!msd_group(blockIdx.x, *d_total, ng, sub, true, seg_start, seg_tile, seg_chunk, nseg, nb, g)) return;
    const uint32_t ntl = (g.hi - g.lo + MSD_TILE - 1) / MSD_TILE;
    // digits threadIdx.x + q * MSD_THREADS: each row access is coalesced
    uint32_t run[MSD_PER];
#pragma unroll
    for (uint32_t q = 0; q < MSD_PER; q++) {
        const uint32_t d = threadIdx.x + q * MSD_THREADS;
        run[q] = d < nb ? S[g.sidx + (uint64_t)d * g.sstride] : 0u;
    }
#pragma unroll 1
    for (uint32_t j = 0; j < ntl; j += ROWS) {
        uint32_t c[ROWS][MSD_PER];
#pragma unroll
        for (uint32_t k = 0; k < ROWS; k++)
#pragma unroll
            for (uint32_t q = 0; q < MSD_PER; q++) {
                const uint32_t d = threadIdx.x + q * MSD_THREADS;
                c[k][q] = j + k < ntl && d < nb ? C[(uint64_t)(g.row0 + j + k) * nb + d] : 0u;
            }
#pragma unroll
        for (uint32_t k = 0; k < ROWS; k++)
#pragma unroll
            for (uint32_t q = 0; q < MSD_PER; q++) {
                const uint32_t d = threadIdx.x + q * MSD_THREADS;
                if (j + k < ntl && d < nb) P[(uint64_t)(g.row0 + j + k) * nb + d] = run[q];
                run[q] += c[k][q];
            }
    }
}

// Tile t of a pass: pass 1 (seg_tile == nullptr): [t*MSD_TILE, ...) of
// [0, E), past E empty; pass 2: tile t of the tile table seg_tile inside its
// segment (false past the last tile).  Its count and slot rows are row t.
ZK_DEV bool msd_tile(uint32_t t, uint32_t E, const uint32_t* __restrict__ seg_start,
                     const uint32_t* __restrict__ seg_tile, uint32_t nseg, uint32_t& lo, uint32_t& hi) {
    if (!seg_tile) {
        const uint64_t l = (uint64_t)t * MSD_TILE;
        lo = (uint32_t)(l < E ? l : E);
        hi = (uint32_t)(l + MSD_TILE < E ? l + MSD_TILE : E);
        return true;
    }
    if (t >= seg_tile[nseg]) return false;
    uint32_t a = 0, b = nseg - 1;
    while (a < b) {
        const uint32_t mid = (a + b + 1) >> 1;
        if (seg_tile[mid] <= t) a = mid;
        else b = mid - 1;
    }
    lo = seg_start[a] + (t - seg_tile[a]) * MSD_TILE;
    const uint32_t end = seg_start[a + 1];
    hi = end - lo > MSD_TILE ? lo + MSD_TILE : end;
    return true;
}

// Dynamic shared memory of k_msd_scatter: the staged tile and one word per
// digit (claim cursors, then each run's output slot less its local offset).
constexpr size_t MSD_SCATTER_SMEM = (size_t)MSD_TILE * sizeof(uint2) + (1u << MSD_MAX_BITS) * sizeof(uint32_t);

// One block per tile: the tiles placed at once are neighbours, so their runs
// of one digit land side by side in the output.  (Writing the next pass's
// digit beside each placed entry, 2 bytes at scattered slots, cost more in
// partial-sector writes than the pass-2 count saved.)
static __global__ void __launch_bounds__(MSD_THREADS) k_msd_scatter(const uint2* __restrict__ A,
                                                                   const uint32_t* __restrict__ d_total,
                                                                   uint32_t shift, uint32_t bits, uint32_t ntiles,
                                                                   const uint32_t* __restrict__ seg_start,
                                                                   const uint32_t* __restrict__ seg_tile,
                                                                   uint32_t nseg, const uint32_t* __restrict__ C,
                                                                   const uint32_t* __restrict__ P,
                                                                   uint2* __restrict__ B) {
    extern __shared__ uint4 msd_smem[];
    uint2* stage = reinterpret_cast<uint2*>(msd_smem);
    uint32_t* cur = reinterpret_cast<uint32_t*>(stage + MSD_TILE);
    __shared__ uint32_t sh[MSD_THREADS / 32];
    const uint32_t nb = 1u << bits, mask = nb - 1;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t t = blockIdx.x;
    if (!seg_tile && t >= ntiles) return;
    uint32_t lo, hi;
    if (!msd_tile(t, *d_total, seg_start, seg_tile, nseg, lo, hi) || lo == hi) return;
    const uint32_t len = hi - lo;
    const uint32_t* crow = C + (uint64_t)t * nb;
    const uint32_t* prow = P + (uint64_t)t * nb;
    // local offsets of the digits: exclusive scan of the tile's counts; the
    // claim cursors start there
    uint32_t loff[MSD_PER], slot0[MSD_PER], sum = 0;
    {
        uint32_t c[MSD_PER];
#pragma unroll
        for (uint32_t q = 0; q < MSD_PER; q++) {
            const uint32_t d = threadIdx.x * MSD_PER + q;
            c[q] = d < nb ? crow[d] : 0;
            slot0[q] = d < nb ? prow[d] : 0;
            sum += c[q];
        }
        uint32_t total;
        uint32_t pre = block_excl_scan_w<MSD_THREADS / 32>(sum, sh, total);
#pragma unroll
        for (uint32_t q = 0; q < MSD_PER; q++) {
            const uint32_t d = threadIdx.x * MSD_PER + q;
            loff[q] = pre;
            if (d < nb) cur[d] = pre;
            pre += c[q];
        }
    }
    __syncthreads();
    // place the tile in digit order
#pragma unroll 1
    for (uint32_t r0 = 0; r0 * MSD_THREADS < len; r0 += MSD_BATCH) {
        uint2 e[MSD_BATCH];
#pragma unroll
        for (uint32_t q = 0; q < MSD_BATCH; q++) {
            const uint32_t j = (r0 + q) * MSD_THREADS + threadIdx.x;
            e[q] = j < len ? A[(uint64_t)lo + j] : make_uint2(0, 0);
        }
        // the batch's claims in three sweeps, so that its eight shared-memory
        // atomics are in flight together rather than one after another:
        // digits and the all-lanes-one-key test, the atomics (a cursor
        // returns the stage slot itself), the slots
        uint32_t d[MSD_BATCH], m[MSD_BATCH], lk[MSD_BATCH], b[MSD_BATCH];
        bool one[MSD_BATCH];
#pragma unroll
        for (uint32_t q = 0; q < MSD_BATCH; q++) {
            const uint32_t j = (r0 + q) * MSD_THREADS + threadIdx.x;
            const bool v = j < len;
            d[q] = v ? (e[q].x >> shift) & mask : 0u;
            m[q] = __ballot_sync(0xffffffffu, v);
            const uint32_t leader = m[q] ? __ffs(m[q]) - 1 : 0;
            lk[q] = __shfl_sync(0xffffffffu, d[q], leader);
            one[q] = __all_sync(0xffffffffu, !v || d[q] == lk[q]);
        }
#pragma unroll
        for (uint32_t q = 0; q < MSD_BATCH; q++) {
            const bool v = (m[q] >> lane) & 1u;
            const uint32_t leader = m[q] ? __ffs(m[q]) - 1 : 0;
            b[q] = 0;
            if (one[q]) {
                if (lane == leader && m[q]) b[q] = atomicAdd(cur + lk[q], (uint32_t)__popc(m[q]));
            } else if (v) {
                b[q] = atomicAdd(cur + d[q], 1u);
            }
        }
#pragma unroll
        for (uint32_t q = 0; q < MSD_BATCH; q++) {
            const bool v = (m[q] >> lane) & 1u;
            uint32_t slot = b[q];
            if (one[q]) {
                const uint32_t leader = m[q] ? __ffs(m[q]) - 1 : 0;
                slot = __shfl_sync(0xffffffffu, b[q], leader) + __popc(m[q] & ((1u << lane) - 1));
            }
            if (v) stage[slot] = e[q];
        }
    }
    __syncthreads();
    // each run's output slot less its local offset
#pragma unroll
    for (uint32_t q = 0; q < MSD_PER; q++) {
        const uint32_t d = threadIdx.x * MSD_PER + q;
        if (d < nb) cur[d] = slot0[q] - loff[q];
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < len; i += MSD_THREADS) {
        const uint2 v = stage[i];
        B[(uint64_t)cur[(v.x >> shift) & mask] + i] = v;
    }
}

// ------------------------------------------------------------ synthetic inputs
// Counter-based generator shared with the Python restatement in the oracle:
// word = splitmix64(splitmix64(seed*FNV ^ stream*golden ^ (index*8 + word)) ^ attempt*C)

ZK_DEV uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    uint64_t z = x;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

ZK_DEV uint64_t draw_word(uint64_t seed, uint64_t stream, uint64_t index, uint64_t attempt, uint64_t word) {
    uint64_t ctr = seed * 0x100000001B3ull + stream * 0x9E3779B1ull;
    ctr = splitmix64(ctr ^ (index * 8 + word));
    return splitmix64(ctr ^ (attempt * 0xD1B54A32D192ED03ull));
}

// uniform in [lo, r) by masked rejection (at most 64 attempts; the chance of
// needing more is below 2^-130 for both curves, then 1 is used)
template <class Fr>
ZK_DEV void uniform_fr(uint32_t out[8], uint64_t seed, uint64_t stream, uint64_t index, uint32_t lo) {
    const int nbits = Fr::BITS;
#pragma unroll 1
    for (uint64_t att = 0; att < 64; att++) {
        Fe<Fr> v;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            uint64_t x = draw_word(seed, stream, index, att, w);
            v.v[2 * w] = (uint32_t)x;
            v.v[2 * w + 1] = (uint32_t)(x >> 32);
        }
        // mask to the bit length of r
        const int top = nbits - 224;  // bits kept in limb 7
        v.v[7] &= top >= 32 ? 0xffffffffu : ((1u << top) - 1);
        Fe<Fr> r;
#pragma unroll
        for (int i = 0; i < 8; i++) r.v[i] = Fr::P(i);
        bool below = !fe_geq_int(v, r);
        bool atleast = true;
        if (lo) atleast = !fe_is_zero(v);
        if (below && atleast) {
#pragma unroll
            for (int i = 0; i < 8; i++) out[i] = v.v[i];
            return;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) out[i] = i == 0 ? 1u : 0u;
}

constexpr uint64_t STREAM_BASE_K = 1, STREAM_SCALAR = 2, STREAM_KIND = 3;

// scalars: dist 0 uniform Fr, 1 witness-like; fmt 0 integer, 1 Montgomery
template <class C>
__global__ void k_gen_scalars(uint32_t* __restrict__ out, uint64_t n, uint64_t seed, uint64_t index0,
                              int dist, int fmt) {
    using Fr = typename C::Fr;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t gi = index0 + i;
    uint32_t s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (dist == 0) {
        uniform_fr<Fr>(s, seed, STREAM_SCALAR, gi, 0);
    } else {
        uint64_t u = draw_word(seed, STREAM_KIND, gi, 0, 0) % 100;
        if (u < 40) {
        } else if (u < 60) {
            s[0] = 1;
        } else if (u < 85) {
            s[0] = (uint32_t)draw_word(seed, STREAM_SCALAR, gi, 0, 0);
        } else {
            uniform_fr<Fr>(s, seed, STREAM_SCALAR, gi, 0);
        }
    }
    if (fmt == 1) {
        Fe<Fr> v;
#pragma unroll
        for (int l = 0; l < 8; l++) v.v[l] = s[l];
        fe_to_mont(v, v);
#pragma unroll
        for (int l = 0; l < 8; l++) s[l] = v.v[l];
    }
    uint4* o = reinterpret_cast<uint4*>(out + i * 8);
    o[0] = make_uint4(s[0], s[1], s[2], s[3]);
    o[1] = make_uint4(s[4], s[5], s[6], s[7]);
}

// Fixed-base comb: table[j*256 + v] = v * 2^(8j) * G (affine), j < 32.
// Built by one thread per entry with double-and-add from G.
template <class C>
__global__ void k_comb_table(uint32_t* __restrict__ table) {
    using P = typename C::Fp;
    uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 32 * 256) return;
    uint32_t j = e >> 8, v = e & 255;
    Affine<P> g;
#pragma unroll
    for (int l = 0; l < P::N; l++) { g.x.v[l] = C::Gen::X_MONT(l); g.y.v[l] = C::Gen::Y_MONT(l); }
    Xyzz<P> acc;
    xyzz_set_id(acc);
    // acc = v * 2^(8j) * G: bits of v from the top, then 8j doublings
#pragma unroll 1
    for (int b = 7; b >= 0; b--) {
        xyzz_dbl_ni(acc, acc);
        if ((v >> b) & 1) xyzz_add_affine_ni(acc, g);
    }
#pragma unroll 1
    for (uint32_t d = 0; d < 8 * j; d++) xyzz_dbl_ni(acc, acc);
    Affine<P> a;
    xyzz_to_affine_ni(a, acc);
    uint4* o = reinterpret_cast<uint4*>(table + (size_t)e * 2 * P::N);
    store_fe(o, a.x);
    store_fe(o + P::N / 4, a.y);
}

// bases[i] = k_i * G with k_i uniform in [1, r): 32 mixed additions from the comb
template <class C>
__global__ void __launch_bounds__(128) k_gen_bases(const uint32_t* __restrict__ table, uint32_t* __restrict__ out,
                                                   uint64_t n, uint64_t seed, uint64_t index0) {
    using P = typename C::Fp;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t k[8];
    uniform_fr<typename C::Fr>(k, seed, STREAM_BASE_K, index0 + i, 1);
    Xyzz<P> acc;
    xyzz_set_id(acc);
#pragma unroll 1
    for (int j = 0; j < 32; j++) {
        uint32_t byte = (k[j >> 2] >> (8 * (j & 3))) & 255;
        if (byte) {
            Affine<P> q;
            load_affine(q, table, j * 256 + byte);
            xyzz_add_affine_ni(acc, q);
        }
    }
    Affine<P> a;
    xyzz_to_affine_ni(a, acc);
    uint4* o = reinterpret_cast<uint4*>(out + i * 2 * P::N);
    store_fe(o, a.x);
    store_fe(o + P::N / 4, a.y);
}

}  // namespace zkmsm

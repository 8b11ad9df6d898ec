// Bucket accumulation by affine additions with shared inversions.
//
// A mixed XYZZ addition takes 10 field products.  An affine addition takes
// one inversion, two products and a square, and when many independent
// additions share one inversion by Montgomery's trick (prefix products
// forward, one inverse, unwound backwards) the inversion costs three products
// each: 6 in all.  The accumulation is bound by the multiply pipe (k_acc_l1
// runs at its rate), so that is where its time goes.
//
// The sorted entries are cut into chunks of K, one thread each, as for
// k_acc_l1.  A level adds the neighbouring elements of each run pairwise,
// which halves the runs; all pairs of a thread and a level share one product
// chain, and AFF_G threads one inversion.  Nothing passes between chunks, so
// a level needs no scan and no list in common.  Levels repeat until the runs
// are short; k_aff_finish adds up what is left in XYZZ and hands over bucket
// sums and boundary runs exactly as k_acc_l1 does.
//
//  k_aff_pair    level: find the pairs, prefix products of their differences
//  k_aff_invert  one inverse per AFF_G threads, unwound to each thread
//  k_aff_add     level: inverses backwards, the sums
//  k_aff_finish  remaining runs
//
// A thread's elements are a list of 16-bit references: a place that holds a
// sum, or the one entry of a run that found no partner on the first level
// (its value is kept with the run's key).  Pair j of the first level takes place j; later
// pairs have a sum on the left (a run has one element without a partner per
// level at most, its last) and write into its place, so no point is ever
// copied and a thread needs K/2 places whatever its runs are.  A slab of
// threads (one wave of k_aff_add) goes through all levels before the next, so
// the buffers hold one slab.  Everything is interleaved by lane in 16-byte
// words, so a warp's accesses are whole lines where its lanes are in step.
//
// The sums need five dependent products per pair and fetch five coordinates
// for them; fetched where they are used, k_aff_add spent 44% of its warps' time
// waiting for memory (SMs at 68% of their issue limit, a BN254 build).  So
// each thread copies its next pair to shared memory (cp.async) while it
// computes this one (75-77%, BLS12-381; what is left is the last warps of a
// wave), and k_aff_pair keeps a few pairs' x on their way (63-69%).
//
// BLS12-381 2^20 (16.8 M entries, five levels): k_aff_add 1906 us for the first
// level and 1939 for the others, k_aff_pair 501 + 909, k_aff_invert 224,
// k_aff_finish 424, against 6177 us in k_acc_l1, and 155 against 423 us of
// partial sums after it.
#pragma once
#include "msm_kernels.cuh"

namespace zkmsm {

// references: a place, or (AFF_ENTRY) the entry its run keeps in the table of
// runs; AFF_LAST: the last of its run
constexpr uint32_t AFF_ENTRY = 0x8000u, AFF_LAST = 0x4000u, AFF_INDEX = 0x3fffu;
static_assert(2 * AFF_MAX_CHUNK <= AFF_INDEX, "places fit a reference");
// in a later level's pair info: the right point is an entry
constexpr uint32_t AFF_RIGHT_ENTRY = 0x80000000u;

// The buffers of one slab of `threads` threads (a multiple of 32).
struct AffSlab {
    uint4* pts;        // [warp][pcap][2N/4][lane]: places
    uint4* pre;        // [warp][pcap][N/4][lane]: product of the differences before pair j
    uint2* info;       // [warp][pcap][lane]: pair j's points (entry values or places)
    uint2* elem;       // [warp][K/4][lane]: four references each
    uint2* runs;       // [warp][K][lane]: a run's key, the value of its entry without a partner
    uint32_t* prod;    // [thread][N]: product of all differences, then its inverse
    uint32_t* cnt;     // [thread]: elements
    uint32_t* npair;   // [thread]: pairs of this level
    uint32_t K, pcap, threads;  // K a multiple of 4, pcap = K / 2
    uint32_t slabs;    // that the expected entries fill, at chunks of K
    uint32_t chunks;   // of K for all the entries there may be
};

// A point in memory: words `step` apart, y negated or not.
struct AffPoint {
    const uint4* p;
    uint32_t step, neg;
};

template <class P>
ZK_DEV AffPoint aff_entry(uint32_t v, const uint32_t* bases, const uint32_t* phi) {
    const uint32_t* tab = (v >> 30) & 1 ? phi : bases;
    return AffPoint{reinterpret_cast<const uint4*>(tab + (size_t)(v & VAL_IDX_MASK) * 2 * P::N), 1u, v >> 31};
}

// place i of the thread whose place 0 is at pts
template <class P>
ZK_DEV AffPoint aff_place(const uint4* pts, uint32_t i) {
    return AffPoint{pts + (size_t)i * (2 * P::N / 4) * 32, 32u, 0u};
}

// coordinate Y (0: x, 1: y before its sign) of a point
template <class P>
ZK_DEV void aff_coord(Fe<P>& f, const AffPoint& a, int Y) {
#pragma unroll
    for (int i = 0; i < P::N / 4; i++) {
        const uint4 v = a.p[(i + Y * (P::N / 4)) * a.step];
        f.v[4 * i] = v.x; f.v[4 * i + 1] = v.y; f.v[4 * i + 2] = v.z; f.v[4 * i + 3] = v.w;
    }
}

template <class P>
ZK_DEV void aff_store(uint4* d, const Fe<P>& f) {  // words 32 lanes apart
#pragma unroll
    for (int i = 0; i < P::N / 4; i++)
        d[32 * i] = make_uint4(f.v[4 * i], f.v[4 * i + 1], f.v[4 * i + 2], f.v[4 * i + 3]);
}

template <class P>
ZK_DEV void aff_load_row(Fe<P>& f, const uint4* s) {  // plain loads (in-place rows)
#pragma unroll
    for (int i = 0; i < P::N / 4; i++) {
        const uint4 v = s[i];
        f.v[4 * i] = v.x; f.v[4 * i + 1] = v.y; f.v[4 * i + 2] = v.z; f.v[4 * i + 3] = v.w;
    }
}

// The denominator shared out for a pair whose points need a look: x equal, or
// an x of zero, which the identity (0, 0) has.  Doubling: 2y; nothing to
// invert (an identity, or P + (-P)): 1; else the difference d.
template <class P>
ZK_DEV void aff_special_d(Fe<P>& d, const Affine<P>& a, const Affine<P>& b) {
    const bool same = fe_eq(a.x, b.x);
    if (affine_is_id(a) || affine_is_id(b) || (same && (fe_is_zero(a.y) || !fe_eq(a.y, b.y)))) {
        fe_set_one(d);
    } else if (same) {
        fe_dbl(d, a.y);
    }
}

// Out of line: rare.  d for points a and b, y fetched here.
template <class P>
__device__ __noinline__ Fe<P> aff_look_d(Fe<P> d, const AffPoint a, const AffPoint b) {
    Affine<P> u, v;
    aff_coord(u.x, a, 0);
    aff_coord(v.x, b, 0);
    aff_coord(u.y, a, 1);
    aff_coord(v.y, b, 1);
    if (a.neg) fe_neg(u.y, u.y);
    if (b.neg) fe_neg(v.y, v.y);
    aff_special_d(d, u, v);
    return d;
}

// Chunk length for M entries: as acc_chunk, whole slabs of at most K; K when the
// slabs hold too few (the chunks after them are k_acc_l1's).
ZK_DEV uint32_t aff_len(const AffSlab& s, uint32_t M) {
    const uint64_t per = (uint64_t)s.K * s.threads;
    if (M == 0 || M > per * s.slabs) return s.K;
    const uint64_t parts = min((M + per - 1) / per * s.threads, (uint64_t)s.chunks);
    return min(s.K, max(16u, (uint32_t)((M + 4 * parts - 1) / (4 * parts)) * 4));
}

// Entries of chunk g: [g*K, ..) of M.
ZK_DEV uint32_t aff_chunk(uint64_t g, uint32_t K, uint32_t M) {
    const uint64_t start = g * K;
    return start >= M ? 0u : (uint32_t)(M - start < K ? M - start : K);
}

// The list of references, read forward four at a time with the next four in
// flight, and written behind the reader in place.
struct AffList {
    uint2* base;  // this thread's word 0
    uint2 cur, next, out;
    uint32_t word, words;

    ZK_DEV void open(uint2* b, uint32_t n) {
        base = b;
        word = 0;
        words = (n + 3) / 4;
        cur = words ? base[0] : make_uint2(0, 0);
        next = words > 1 ? base[32] : make_uint2(0, 0);
        out = make_uint2(0, 0);
    }
    // reference i (i never goes back by more than the word it is in)
    ZK_DEV uint32_t get(uint32_t i) {
        if (i >> 2 != word) {
            word++;
            cur = next;
            if (word + 1 < words) next = base[32 * (word + 1)];
        }
        return ((i & 2u ? cur.y : cur.x) >> 16 * (i & 1u)) & 0xffffu;
    }
    ZK_DEV void put(uint32_t k, uint32_t ref) {
        if (!(k & 1u)) {
            if (k & 2u) out.y = ref;
            else out.x = ref;
        } else if (k & 2u) {
            out.y |= ref << 16;
            base[32 * (k >> 2)] = out;
        } else {
            out.x |= ref << 16;
        }
    }
    ZK_DEV void close(uint32_t k) {  // k references written
        if (k & 3u) base[32 * (k >> 2)] = out;
    }
};

// Launch shapes: a slab is the threads of k_aff_add resident at once (12 limbs:
// four blocks of 128 threads, with three the sums are 5% slower; Fp2: three).
constexpr uint32_t AFF_THREADS = 128;
template <class C>
struct AffLaunch {
    static constexpr int BLOCKS = 4;
};
template <>
struct AffLaunch<Bn254G2> {
    static constexpr int BLOCKS = 3;
};

// The points of a pair from its info.
template <class P, bool FIRST>
ZK_DEV void aff_points(AffPoint& a, AffPoint& b, uint2 r, const uint4* pts, const uint32_t* bases,
                       const uint32_t* phi) {
    if (FIRST) a = aff_entry<P>(r.x, bases, phi);
    else a = aff_place<P>(pts, r.x & AFF_INDEX);
    if (FIRST || r.x & AFF_RIGHT_ENTRY) b = aff_entry<P>(r.y, bases, phi);
    else b = aff_place<P>(pts, r.y & AFF_INDEX);
}

ZK_DEV void cp_async16(uint4* smem, const uint4* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}

// Pairs whose x are on their way to shared memory in k_aff_pair: one product
// covers little of a fetch, so several are in flight (as many as 48 KB hold).
template <class P>
struct AffRing {
    static constexpr int D = P::N == 12 ? 3 : 2;
    static constexpr int SLOT = (D * 2 * (P::N / 4)) | 1;
};

template <class C, bool FIRST>
__global__ void __launch_bounds__(AFF_THREADS, AffLaunch<C>::BLOCKS) k_aff_pair(
        AffSlab s, const uint2* __restrict__ ents, const uint32_t* __restrict__ d_len, uint64_t g0,
        const uint32_t* __restrict__ bases, const uint32_t* __restrict__ phi) {
    using P = typename C::Fp;
    constexpr int V = P::N / 4, D = AffRing<P>::D;
    __shared__ uint4 ring[AFF_THREADS * AffRing<P>::SLOT];
    const uint32_t t = blockIdx.x * AFF_THREADS + threadIdx.x;
    if (t >= s.threads) return;
    uint4* my = ring + threadIdx.x * AffRing<P>::SLOT;
    const size_t warp = t >> 5, lane = t & 31;
    const uint64_t g = g0 + t;
    const uint32_t M = FIRST ? *d_len : 0, K = FIRST ? aff_len(s, M) : 0;
    const uint32_t n = FIRST ? aff_chunk(g, K, M) : s.cnt[t];
    const uint2* en = ents + g * K;
    const uint4* pts = s.pts + warp * s.pcap * (2 * V) * 32 + lane;
    uint4* pre = s.pre + warp * s.pcap * V * 32 + lane;
    uint2* info = s.info + warp * s.pcap * 32 + lane;
    uint2* runs = s.runs + warp * s.K * 32 + lane;
    AffList list;
    list.open(s.elem + warp * (s.K / 4) * 32 + lane, FIRST ? 0 : n);
    uint32_t i = 0, k = 0, found = 0, run = 0;
    // FIRST: entries i, i + 1, i + 2, fetched ahead of their use
    const uint2 none = make_uint2(ACC_EMPTY, 0);
    uint2 e0 = none, e1 = none, e2 = none;
    // later levels: the entry kept with the current run, and the next run's on
    // its way
    uint32_t sval = 0, snext = 0;
    if (FIRST) {
        if (n > 0) e0 = en[0];
        if (n > 1) e1 = en[1];
        if (n > 2) e2 = en[2];
    } else if (n) {
        sval = runs[0].y;
        snext = runs[32].y;  // K >= 16 rows
    }
    // the next pair of neighbours of one run, its x on their way to slot `at`;
    // what has no partner stays listed
    auto next_pair = [&](uint32_t at) {
        AffPoint a, b;
        uint2 r = none;
        bool got = false;
        while (i < n && !got) {
            if (FIRST) {
                if (e1.x != e0.x) {
                    list.put(k++, AFF_ENTRY | AFF_LAST);
                    runs[32 * run++] = e0;
                    e0 = e1;
                    e1 = e2;
                    i++;
                    e2 = i + 2 < n ? en[i + 2] : none;
                } else {
                    const bool end = e2.x != e0.x;
                    list.put(k++, found | (end ? AFF_LAST : 0u));
                    if (end) runs[32 * run++] = make_uint2(e0.x, 0);
                    r = make_uint2(e0.y, e1.y);
                    e0 = e2;
                    i += 2;
                    e1 = i + 1 < n ? en[i + 1] : none;
                    e2 = i + 2 < n ? en[i + 2] : none;
                    got = true;
                }
            } else {
                const uint32_t r0 = list.get(i);
                uint32_t last = r0;
                if (r0 & AFF_LAST) {
                    list.put(k++, r0);
                    i++;
                } else {
                    const uint32_t r1 = list.get(i + 1);  // exists: r0 is not its run's last
                    list.put(k++, r0 | (r1 & AFF_LAST));
                    r = r1 & AFF_ENTRY ? make_uint2(r0 | AFF_RIGHT_ENTRY, sval) : make_uint2(r0, r1);
                    last = r1;
                    i += 2;
                    got = true;
                }
                if (last & AFF_LAST) {
                    sval = snext;
                    if (++run + 1 < s.K) snext = runs[32 * (run + 1)].y;
                }
            }
        }
        if (got) {
            info[32 * found++] = r;
            aff_points<P, FIRST>(a, b, r, pts, bases, phi);
#pragma unroll
            for (int w = 0; w < V; w++) {
                cp_async16(my + at * (2 * V) + w, a.p + w * a.step);
                cp_async16(my + at * (2 * V) + V + w, b.p + w * b.step);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    Fe<P> acc;
    fe_set_one(acc);
#pragma unroll 1
    for (uint32_t q = 0; q < D; q++) next_pair(q);
    uint32_t at = 0;
#pragma unroll 1
    for (uint32_t j = 0; j < found; j++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
        Fe<P> x1, x2, d;
        aff_load_row(x1, my + at * (2 * V));
        aff_load_row(x2, my + at * (2 * V) + V);
        next_pair(at);
        at = at + 1 == D ? 0 : at + 1;
        fe_sub(d, x2, x1);
        if (fe_is_zero(x1) || fe_is_zero(x2) || fe_is_zero(d)) {
            AffPoint a, b;
            aff_points<P, FIRST>(a, b, info[32 * j], pts, bases, phi);
            d = aff_look_d<P>(d, a, b);
        }
        if (j) {
            aff_store(pre + (size_t)32 * V * j, acc);
            fe_mul(acc, acc, d);
        } else {
            acc = d;
        }
    }
    list.close(k);
    s.cnt[t] = k;
    s.npair[t] = found;
    store_fe(reinterpret_cast<uint4*>(s.prod + (size_t)t * P::N), acc);
}

// prod[t] -> 1 / prod[t], AFF_G threads' products per inversion
constexpr uint32_t AFF_G = 4;  // divides AFF_SLAB_UNIT / AFF_THREADS
template <class C>
__global__ void __launch_bounds__(AFF_THREADS) k_aff_invert(uint32_t* __restrict__ prod, uint32_t threads) {
    using P = typename C::Fp;
    const uint32_t t0 = (blockIdx.x * AFF_THREADS + threadIdx.x) * AFF_G;
    if (t0 >= threads) return;  // threads is a multiple of AFF_G
    uint4* p = reinterpret_cast<uint4*>(prod + (size_t)t0 * P::N);
    Fe<P> v[AFF_G], pre[AFF_G], inv;
#pragma unroll
    for (uint32_t k = 0; k < AFF_G; k++) {
        aff_load_row(v[k], p + k * (P::N / 4));
        if (k) fe_mul(pre[k], pre[k - 1], v[k]);
        else pre[0] = v[0];
    }
    fe_inv(inv, pre[AFF_G - 1]);
#pragma unroll
    for (uint32_t k = AFF_G; k-- > 1;) {
        Fe<P> o;
        fe_mul(o, inv, pre[k - 1]);
        fe_mul(inv, inv, v[k]);
        store_fe(p + k * (P::N / 4), o);
    }
    store_fe(p, inv);
}

// Rare pairs of k_aff_add, out of line: points (x1, y1) + (x2, y2) where the
// inverse v belongs to aff_special_d's denominator.
template <class P>
__device__ __noinline__ Affine<P> aff_look_add(const Affine<P> a, const Affine<P> b, const Fe<P> v) {
    Affine<P> r;
    if (affine_is_id(a)) return b;
    if (affine_is_id(b)) return a;
    Fe<P> l, m;
    if (fe_eq(a.x, b.x)) {
        if (fe_is_zero(a.y) || !fe_eq(a.y, b.y)) {
            fe_set_zero(r.x);
            fe_set_zero(r.y);
            return r;
        }
        fe_mul(l, a.x, a.x);
        fe_dbl(m, l);
        fe_add(l, m, l);  // 3x^2
    } else {
        fe_sub(l, b.y, a.y);
    }
    fe_mul(l, l, v);
    fe_mul(m, l, l);
    fe_sub(m, m, a.x);
    fe_sub(r.x, m, b.x);
    fe_sub(m, a.x, r.x);
    fe_mul(m, l, m);
    fe_sub(r.y, m, a.y);
    return r;
}

template <class C, bool FIRST>
__global__ void __launch_bounds__(AFF_THREADS, AffLaunch<C>::BLOCKS) k_aff_add(
        AffSlab s, const uint32_t* __restrict__ bases, const uint32_t* __restrict__ phi) {
    using P = typename C::Fp;
    constexpr int V = P::N / 4;            // 16-byte words per coordinate
    constexpr int SLOT = (5 * V) | 1;      // x1 x2 y1 y2 pre; an odd stride has no bank conflicts
    __shared__ uint4 stage[AFF_THREADS * SLOT];
    const uint32_t t = blockIdx.x * AFF_THREADS + threadIdx.x;
    if (t >= s.threads) return;
    uint4* my = stage + threadIdx.x * SLOT;
    const size_t warp = t >> 5, lane = t & 31;
    uint4* pts = s.pts + warp * s.pcap * (2 * V) * 32 + lane;
    const uint4* pre = s.pre + warp * s.pcap * V * 32 + lane;
    const uint2* info = s.info + warp * s.pcap * 32 + lane;
    const uint32_t np = s.npair[t];
    // the warp goes through pair indices together, so that its lanes' rows of
    // prefix products (and first-level places) are the same ones
    const uint32_t top = __reduce_max_sync(0xffffffffu, np);
    Fe<P> inv;
    aff_load_row(inv, reinterpret_cast<const uint4*>(s.prod + (size_t)t * P::N));
    AffPoint a{nullptr, 0, 0}, b{nullptr, 0, 0};
    uint32_t place = 0;  // of the fetched pair
    auto resolve = [&](uint32_t j) {  // pair j's points
        const uint2 r = info[32 * j];
        aff_points<P, FIRST>(a, b, r, pts, bases, phi);
        return FIRST ? j : r.x & AFF_INDEX;
    };
    auto fetch = [&](uint32_t j) {  // to shared memory
#pragma unroll
        for (int i = 0; i < V; i++) {
            cp_async16(my + i, a.p + i * a.step);
            cp_async16(my + V + i, b.p + i * b.step);
            cp_async16(my + 2 * V + i, a.p + (V + i) * a.step);
            cp_async16(my + 3 * V + i, b.p + (V + i) * b.step);
            if (j) cp_async16(my + 4 * V + i, pre + (size_t)32 * (V * j + i));
        }
    };
    // a, b: the points of the pair in the stage while its signs are needed,
    // then those of the pair after it
    uint32_t nplace = 0, na = 0, nb = 0;
    bool have = false;
#pragma unroll 1
    for (uint32_t j = top; j-- > 0;) {
        if (j >= np) continue;
        if (!have) {  // this lane's first pair
            place = resolve(j);
            na = a.neg;
            nb = b.neg;
            fetch(j);
            if (j) nplace = resolve(j - 1);
            have = true;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        Fe<P> x1, x2, y1, y2, d, v;
        aff_load_row(x1, my);
        aff_load_row(x2, my + V);
        if (j) {
            aff_load_row(v, my + 4 * V);
            fe_mul(v, inv, v);  // 1 / d of this pair
        } else {
            v = inv;
        }
        fe_sub(d, x2, x1);
        const bool look = fe_is_zero(d) || fe_is_zero(x1) || fe_is_zero(x2);
        aff_load_row(y1, my + 2 * V);
        aff_load_row(y2, my + 3 * V);
        if (na) fe_neg(y1, y1);
        if (nb) fe_neg(y2, y2);
        const uint32_t at = place;
        if (j) {  // the stage has been read: fetch the next pair over the rest of this one
            place = nplace;
            na = a.neg;
            nb = b.neg;
            fetch(j - 1);
            if (j > 1) nplace = resolve(j - 2);
        }
        if (look) {
            const Affine<P> u{x1, y1}, w{x2, y2};
            aff_special_d(d, u, w);
            const Affine<P> r = aff_look_add<P>(u, w, v);
            aff_store(pts + (size_t)32 * at * (2 * V), r.x);
            aff_store(pts + (size_t)32 * (at * (2 * V) + V), r.y);
        }
        if (j) fe_mul(inv, inv, d);
        if (!look) {
            fe_sub(d, y2, y1);
            fe_mul(v, v, d);        // slope
            fe_mul(d, v, v);
            fe_sub(d, d, x1);
            fe_sub(d, d, x2);       // x3
            fe_sub(x1, x1, d);
            fe_mul(v, v, x1);
            fe_sub(y1, v, y1);      // y3
            aff_store(pts + (size_t)32 * at * (2 * V), d);
            aff_store(pts + (size_t)32 * (at * (2 * V) + V), y1);
        }
    }
}

// What the levels left of each chunk in XYZZ: bucket sums, and the chunk's
// first and last run for the next level of partial sums, as k_acc_l1.
template <class C>
__global__ void __launch_bounds__(AFF_THREADS) k_aff_finish(
        AffSlab s, const uint32_t* __restrict__ d_len, uint64_t g0, const uint32_t* __restrict__ bases,
        const uint32_t* __restrict__ phi, uint32_t* __restrict__ d_next, Xyzz<typename C::Fp>* __restrict__ buckets,
        uint32_t* __restrict__ pkeys, Xyzz<typename C::Fp>* __restrict__ pvals) {
    using P = typename C::Fp;
    const uint32_t t = blockIdx.x * AFF_THREADS + threadIdx.x;
    if (t >= s.threads) return;
    const size_t warp = t >> 5, lane = t & 31;
    const uint64_t g = g0 + t;
    const uint32_t M = *d_len, K = aff_len(s, M);
    if (g == 0) *d_next = (uint32_t)(2 * (((uint64_t)M + K - 1) / K));
    if (!aff_chunk(g, K, M)) return;
    const uint32_t n = s.cnt[t];
    const uint4* pts = s.pts + warp * s.pcap * (2 * P::N / 4) * 32 + lane;
    const uint2* runs = s.runs + warp * s.K * 32 + lane;
    AffList list;
    list.open(s.elem + warp * (s.K / 4) * 32 + lane, n);
    uint32_t run = 0;
    Xyzz<P> acc;
    xyzz_set_id(acc);
    uint2 rk = runs[0];
    // element i of the run rk, fetched ahead of its addition
    auto load = [&](uint32_t ref, Affine<P>& q) {
        const AffPoint a = ref & AFF_ENTRY ? aff_entry<P>(rk.y, bases, phi) : aff_place<P>(pts, ref & AFF_INDEX);
        aff_coord(q.x, a, 0);
        aff_coord(q.y, a, 1);
        return a.neg;
    };
    Affine<P> q;
    uint32_t ref = list.get(0), neg = load(ref, q);
#pragma unroll 1
    for (uint32_t i = 0; i < n; i++) {
        if (!affine_is_id(q)) {
            if (neg) fe_neg(q.y, q.y);
            xyzz_add_affine(acc, q);
        }
        const bool last = ref & AFF_LAST, tail = i + 1 == n;
        const uint32_t key = rk.x;
        if (!tail) {
            if (last) rk = runs[32 * (run + 1)];
            ref = list.get(i + 1);
            neg = load(ref, q);
        }
        if (last) {
            const bool head = run == 0;
            if (head) pkeys[2 * g] = key;
            else if (tail) pkeys[2 * g + 1] = key;
            if (head && tail) pkeys[2 * g + 1] = ACC_EMPTY;
            store_xyzz(head ? pvals + 2 * g : tail ? pvals + 2 * g + 1 : buckets + key, acc);
            xyzz_set_id(acc);
            run++;
        }
    }
}

}  // namespace zkmsm

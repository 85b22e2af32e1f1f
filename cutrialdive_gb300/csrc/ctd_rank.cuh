// ctd_rank.cuh -- Fibonacci and Lucas hits of a list of primes by the rank
// of apparition, the orders p -+ 1 factored for a whole tile of primes at
// once (included by ctd_residue.cu, which has the push and the table of
// trial primes).
//
// For a prime p other than 2 and 5, p | F(n) iff a(p) | n, and a(p) divides
// D = p - (5/p); p | L(n) iff a(p) is even and n is an odd multiple of
// a(p)/2.  A hit at n < e needs a(p) <= e - 1 (Lucas: 2 (e - 1)) with every
// odd prime factor at most e - 1, so a(p) divides S, the part of D made of 2
// and the primes below e.  run_fibonacci_rank finds S by dividing every D by
// every prime below e; here the primes of a tile lie close together, so a
// prime q meets their D's only at the multiples of q in the tile's span: one
// CTA marks the D's in a bitmap and walks each q's multiples over it, a few
// hundred instructions a prime instead of 25,000 (5133 primes below 50000).
//
// What is left per prime is one modular power.  With F(x) = x^2 - x - 1,
// roots u and v = -1/u, F(n) = 0 iff t^n = 1 for t = u/v; t + 1/t =
// (u^2 + v^2)/(uv) = -3, so W(n) = t^n + t^-n runs from W(0) = 2, W(1) = -3 by
// W(2n) = W(n)^2 - 2 and W(2n+1) = W(n) W(n+1) + 3, and F(n) = 0 iff W(n) = 2
// (t + 1/t = 2 only for t = 1): two products a bit of n, one a factor of 2,
// where the doubling of (F(n), F(n+1)) takes three and more additions.
//
// Mersenne numbers go the same way: p | 2^n - 1 iff the order of 2 divides n,
// and the order divides D = p - 1 (and a hit needs it below e); the power is
// 2^-n, one product a bit (half_power).
#pragma once

namespace ctd {

constexpr uint32_t RANK_TILE = 1024;         // primes a tile at most
constexpr uint32_t RANK_SPAN = 1u << 15;     // even numbers a tile's D's may span
constexpr uint32_t RANK_WORDS = RANK_SPAN / 16 + 2;  // two bits (p = D + 1, p = D - 1) an even number
constexpr uint32_t RANK_BY_PRIME = 17;       // table primes below 64: divided prime by prime
constexpr uint32_t RANK_BY_WARP = 171;       // table primes below 1024: a warp walks their multiples
constexpr int RANK_CTAS = 5;                 // a SM: 42 KiB of shared memory, 48 registers a thread
constexpr uint32_t RANK_HITS = 3 * RANK_TILE / 2;
static_assert(RANK_TILE == 1u << 10 && TRIAL_PRIMES < 1u << 22, "a noted multiple is 32 bits");
// Index ranges below e from which the tiles of ranks are taken instead of the
// walk.  Measured on the primes of a 2^27-wide range at 2^34: 768 terms from
// n = 1 take 1.53 ms either way and 1024 take 1.58 (walk 1.77); from n = 40001
// they cost 2.14 (walk 2.14) and 2.17 (walk 2.40).  The primes below e cost a
// tile about as much as 1/256 of e terms.
constexpr uint64_t RANK_MIN_TERMS = 1024;
constexpr uint64_t rank_min_terms(uint64_t e) { return RANK_MIN_TERMS + (e >> 8); }
// Mersenne, against the block walk: on the primes of a 2^28-wide range at 2^31,
// 2000 terms from n = 1 take 1.53 ms (the walk 1.47) and 3000 take 1.59 (1.82);
// from n = 40001, 3000 take 2.28 (2.03) and 5000 take 2.32 (2.73).  From 8192
// terms on the walk over classes takes 5.7 ms, 13.0 for 100,000 terms, where the
// orders take 1.7 and 3.0.
constexpr uint64_t order_min_terms(uint64_t e) { return 2100 + e / 24; }

// x mod q for x < 2^62, q < 2^20, with z = floor(2^32 / q): the high word,
// then the low word in pieces that keep the running value below 2^32
__device__ __forceinline__ uint32_t rank_mod(uint64_t x, uint32_t q, uint32_t z)
{
    auto red = [&](uint32_t a) {
        const uint32_t r = a - __umulhi(a, z) * q;  // < 2q
        return r >= q ? r - q : r;
    };
    const uint32_t lo = (uint32_t)x;
    uint32_t r = red((uint32_t)(x >> 32));
    r = red(r << 12 | lo >> 20);
    r = red(r << 12 | (lo >> 8 & 0xfffu));
    return red(r << 8 | (lo & 0xffu));
}

// whether D = p + 1 (Fibonacci, Lucas: p = +-2 mod 5), else D = p - 1
template <uint32_t FAM>
__device__ __forceinline__ bool rank_above(uint64_t p)
{
    if (FAM == MERSENNE)
        return false;
    const uint32_t r5 = (uint32_t)(p % 5);
    return r5 == 2 || r5 == 3;
}

// the sequence W modulo p, values in Montgomery form.  Below 2^40 the values
// stay in [0, 2p + 2^20]: the lazy product of two such is below p + 2^20.
template <bool NARROW>
struct RankPowers {
    MontT<NARROW> m;
    uint64_t two, w1;  // 2 and -3

    __device__ __forceinline__ void init(uint64_t p)
    {
        m.init_lite(p);
        two = m.dbl(m.one);
        w1 = m.sub(0, m.add(two, m.one));
    }
    __device__ __forceinline__ uint64_t mul_sub(uint64_t a, uint64_t b, uint64_t c) const
    {
        if (NARROW)
            return m.mul_lazy(a, b) + (m.p - c);
        return m.sub(m.mul(a, b), c);
    }
    // F(n) = 0 mod p, n >= 1
    __device__ __forceinline__ bool zero_at(uint64_t n) const
    {
        const int v = __ffsll((long long)n) - 1;
        const uint64_t odd = n >> v;
        uint64_t a = w1, b = mul_sub(w1, w1, two);  // W(k), W(k + 1)
        for (int bit = 62 - __clzll((long long)odd); bit >= 0; --bit) {
            const bool up = (odd >> bit) & 1;
            const uint64_t s = up ? b : a;
            const uint64_t mid = mul_sub(a, b, w1);  // W(2k + 1)
            const uint64_t end = mul_sub(s, s, two); // W(2k) or W(2k + 2)
            a = up ? mid : end;
            b = up ? end : mid;
        }
        for (int i = 0; i < v; ++i)
            a = mul_sub(a, a, two);
        // (the product's excess over p, 2^20 at most, is 0 below 2^31)
        a = a >= m.p ? a - m.p : a;
        a = a >= m.p ? a - m.p : a;
        return a == two;
    }
};

// 2^n - 1 modulo p
template <bool NARROW>
struct OrderPowers {
    uint64_t p, pinv;

    __device__ __forceinline__ void init(uint64_t modulus)
    {
        p = modulus;
        pinv = Mont::neg_inverse(p);
    }
    __device__ __forceinline__ bool zero_at(uint64_t n) const { return half_power<NARROW>(p, pinv, n) == 1; }
};
template <uint32_t FAM, bool NARROW>
using FamilyPowers = std::conditional_t<FAM == MERSENNE, OrderPowers<NARROW>, RankPowers<NARROW>>;

// q^-1 mod 2^64 for odd q
__device__ __forceinline__ uint64_t rank_inverse(uint32_t q)
{
    uint64_t x = inverse_mod_2_32(q);
    return x * (2 - (uint64_t)q * x);
}

// n without its factors q (odd q)
__device__ __forceinline__ uint64_t rank_without(uint64_t n, uint32_t q)
{
    const uint64_t inv = rank_inverse(q);
    for (uint64_t x = n * inv; __umul64hi(x, q) == 0; x = n * inv)
        n = x;
    return n;
}

// a(p) (Mersenne: the order of 2), which divides S, or 0 when it exceeds amax; q1 > q2 the two largest
// odd primes of S (0: none).  A prime at a time is taken out of S while F
// stays zero; what stays is final, and more than amax of it ends the search.
template <uint32_t FAM, bool NARROW>
__device__ __noinline__ uint64_t rank_of(uint64_t p, uint64_t S, uint32_t q1, uint32_t q2, uint64_t amax)
{
    FamilyPowers<FAM, NARROW> w;
    w.init(p);
    uint64_t a = S, fixed = 1;
    auto reduce = [&](uint64_t q) {
        while (a % q == 0 && w.zero_at(a / q))
            a /= q;
        for (uint64_t r = a; r % q == 0 && fixed <= amax; r /= q)
            fixed *= q;
    };
    uint64_t rest = S >> (__ffsll((long long)S) - 1);
    if (q1) {
        reduce(q1);
        rest = rank_without(rest, q1);
    }
    if (q2 && fixed <= amax) {
        reduce(q2);
        rest = rank_without(rest, q2);
    }
    for (uint32_t i = 0; rest > 1 && fixed <= amax; ++i) {
        const uint4 t = g_trial_div[i];
        uint64_t q = t.w;
        if (q * q > rest) {
            q = rest;  // a prime
        } else {
            const uint64_t x = rest * ((uint64_t)t.y << 32 | t.x);
            if (__umul64hi(x, q) != 0)
                continue;
        }
        reduce(q);
        rest = q == rest ? 1 : rank_without(rest, (uint32_t)q);
    }
    if (fixed <= amax)
        reduce(2);
    return a <= amax ? a : 0;
}

// The primes whose rank is left to take, a few in a hundred, go to a list
// that a second kernel works off: in the tile they kept one warp busy for
// several powers while the CTA waited (0.92 ms for the tiles of a 2^26-wide
// segment at 2^34).  Primes with many hits (small ones: 3 divides every second
// 2^n - 1) go on to a third kernel, which spreads a prime's hits over the grid.
struct RankItem {
    uint64_t p, S;
    unsigned long long top;
};
struct RankHits {
    uint64_t p, first, a;  // n = first, first + a, ...
};
constexpr uint32_t RANK_MANY = 64;         // hits
constexpr uint32_t RANK_HEAVY = 1u << 16;  // room for primes with as many; the others push their own
struct RankList {
    RankItem *items;
    uint32_t *count;  // may exceed cap: the items beyond it were taken in their tiles
    uint32_t cap;
    RankHits *heavy;
    uint32_t *nheavy;  // may exceed heavy_cap
    uint32_t heavy_cap;
};

// The hits of the lanes' primes (those with mine; the whole warp calls):
// n = a, 2a, ... or a/2, 3a/2, ...
template <uint32_t FAM, bool NARROW>
__device__ __noinline__ void rank_push(const JobView &job, const RankList &list, bool mine, uint64_t p, uint64_t S,
                                       unsigned long long top)
{
    const uint64_t s = job.n0, e = job.n1;
    const uint64_t amax = FAM == LUCAS ? 2 * (e - 1) : e - 1;
    uint64_t a = 0;
    if (mine)  // a(5) = 5; no Lucas number is a multiple of 5
        a = FAM != MERSENNE && p == 5 ? 5 : rank_of<FAM, NARROW>(p, S, (uint32_t)(top >> 32), (uint32_t)top, amax);
    if (a > amax || (FAM == LUCAS && (a & 1)))
        a = 0;
    // first hit n = h mod a, and how many
    uint64_t first = 0, hits = 0;
    if (a) {
        const uint64_t h = FAM == LUCAS ? a >> 1 : 0, r = s % a;
        first = s + (h >= r ? h - r : a - r + h);
        hits = first < e ? (e - 1 - first) / a + 1 : 0;
    }
    if (hits > RANK_MANY) {
        const uint32_t at = atomicAdd(list.nheavy, 1u);
        if (at < list.heavy_cap) {
            list.heavy[at] = RankHits{p, first, a};
            hits = 0;
        }
    }
    // every lane pushes its own
    for (uint64_t i = 0; i < hits; ++i)
        push(job.fb, first + i * a - s, p);
    __syncwarp();
}

struct RankShared {
    uint64_t p[RANK_TILE];
    uint64_t S[RANK_TILE];
    unsigned long long top[RANK_TILE];  // the two largest odd primes of S: q1 << 32 | q2
    union {
        uint32_t bits[RANK_WORDS];
        uint64_t E[RANK_TILE];   // exponents, once the bitmap is done with
    };
    uint16_t before[RANK_WORDS]; // marks in the words before
    union {
        uint32_t hits[RANK_HITS];  // noted multiples: table index << 10 | slot
        struct {
            uint16_t order[RANK_TILE], second[RANK_TILE], finish[RANK_TILE];
        };
    };
    uint32_t bins[64], warp_sums[8];
    unsigned long long lo, hi;
    uint32_t tile, nsecond, nfinish, nhits;
    uint32_t flags;              // 1: an even or repeated entry, or one beyond 2^62
};

// whether a tile's primes, all odd or not, fit its bitmap
__device__ __forceinline__ bool rank_fits(bool odd, uint64_t lo, uint64_t hi)
{
    return odd && lo >= 3 && hi < (1ull << 62) && hi - lo <= 2 * (RANK_SPAN - 2);
}

// one tile of n <= RANK_TILE primes of the list; false when it does not fit
// the bitmap (a sparse or unordered list), and nothing was pushed
template <uint32_t FAM, bool NARROW>
__device__ __forceinline__ void rank_tile_powers(const JobView &job, const RankList &list, RankShared &sh, uint32_t n);

template <uint32_t FAM>
__device__ bool rank_tile(const JobView &job, const RankList &list, RankShared &sh, const uint64_t *__restrict__ primes,
                          uint32_t n, uint32_t nq)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    __syncthreads();  // the tile before is done with
    if (tid == 0) {
        sh.lo = ~0ull;
        sh.hi = 0;
        sh.nsecond = sh.nfinish = sh.nhits = 0;
        sh.flags = 0;
    }
    if (tid < 64)
        sh.bins[tid] = 0;
    __syncthreads();
    {
        unsigned long long lo = ~0ull, hi = 0;
        bool odd = true;
        for (uint32_t i = tid; i < n; i += 256) {
            const unsigned long long p = primes[i];
            lo = p < lo ? p : lo;
            hi = p > hi ? p : hi;
            odd &= p & 1;
        }
        for (int o = 16; o; o >>= 1) {
            const unsigned long long l = __shfl_xor_sync(0xffffffffu, lo, o), h = __shfl_xor_sync(0xffffffffu, hi, o);
            lo = l < lo ? l : lo;
            hi = h > hi ? h : hi;
        }
        if (lane == 0) {
            atomicMin(&sh.lo, lo);
            atomicMax(&sh.hi, hi);
        }
        if (!odd)
            sh.flags = 1;
    }
    __syncthreads();
    const uint64_t lo = sh.lo, hi = sh.hi;
    if (!rank_fits(!sh.flags, lo, hi))
        return false;
    const uint64_t m0 = lo - 1;                              // even; D = m0 + 2 i
    const uint32_t span = (uint32_t)((hi - lo) >> 1) + 2;    // i < span <= RANK_SPAN
    const uint32_t words = (2 * span + 31) >> 5;
    for (uint32_t i = tid; i < words; i += 256)
        sh.bits[i] = 0;
    __syncthreads();
    // mark the D's: bit 2i for p = D + 1, bit 2i + 1 for p = D - 1
    for (uint32_t i = tid; i < n; i += 256) {
        const uint64_t p = primes[i];
        const bool up = rank_above<FAM>(p);
        const uint32_t pos = 2 * (uint32_t)(((up ? p + 1 : p - 1) - m0) >> 1) + up;
        if (atomicOr(&sh.bits[pos >> 5], 1u << (pos & 31)) >> (pos & 31) & 1)
            sh.flags = 1;
    }
    __syncthreads();
    if (sh.flags)
        return false;
    {
        // exclusive prefix of the words' mark counts: thread t sums a run of
        // words, the run sums are scanned over the CTA
        const uint32_t per = (words + 255) / 256, w0 = tid * per, w1 = w0 + per < words ? w0 + per : words;
        uint32_t sum = 0;
        for (uint32_t w = w0; w < w1; ++w)
            sum += __popc(sh.bits[w]);
        uint32_t x = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            x += lane >= (uint32_t)o ? y : 0;
        }
        if (lane == 31)
            sh.warp_sums[warp] = x;
        __syncthreads();
        uint32_t at = x - sum;
        for (uint32_t k = 0; k < warp; ++k)
            at += sh.warp_sums[k];
        for (uint32_t w = w0; w < w1; ++w) {
            sh.before[w] = (uint16_t)at;
            at += __popc(sh.bits[w]);
        }
    }
    __syncthreads();
    // the primes in the order of their marks, with the powers of 2 and the
    // smallest primes of their D's
    for (uint32_t i = tid; i < n; i += 256) {
        const uint64_t p = primes[i];
        const bool up = rank_above<FAM>(p);
        const uint64_t D = up ? p + 1 : p - 1;
        const uint32_t pos = 2 * (uint32_t)((D - m0) >> 1) + up;
        const uint32_t slot = sh.before[pos >> 5] + __popc(sh.bits[pos >> 5] & ((1u << (pos & 31)) - 1u));
        uint64_t S = D & (0 - D);
        unsigned long long top = 0;
        const uint32_t few = nq < RANK_BY_PRIME ? nq : RANK_BY_PRIME;
        for (uint32_t k = 0; k < few; ++k) {
            const uint4 t = g_trial_div[k];
            const uint64_t inv = (uint64_t)t.y << 32 | t.x;
            uint64_t x = D * inv;
            if ((uint32_t)(x >> 32) <= t.z && __umul64hi(x, t.w) == 0) {
                do {
                    S *= t.w;
                    x *= inv;
                } while (__umul64hi(x, t.w) == 0);
                top = (unsigned long long)t.w << 32 | top >> 32;
            }
        }
        sh.p[slot] = p;
        sh.S[slot] = S;
        sh.top[slot] = top;
    }
    __syncthreads();
    // every other prime q < e over its multiples in the span.  A multiple that
    // is some prime's D is only noted (about one a prime): dividing it out on
    // the spot kept 8 of 32 lanes active; the notes are then taken by all
    auto divide_out = [&](uint32_t slot, uint32_t k) {
        const uint4 t = g_trial_div[k];
        const uint64_t inv = (uint64_t)t.y << 32 | t.x, p = sh.p[slot];
        unsigned long long power = t.w;
        for (uint64_t x = (rank_above<FAM>(p) ? p + 1 : p - 1) * inv * inv; __umul64hi(x, t.w) == 0; x *= inv)
            power *= t.w;
        unsigned long long *const S = (unsigned long long *)&sh.S[slot], *const top = &sh.top[slot];
        for (unsigned long long old = *S, was; (was = atomicCAS(S, old, old * power)) != old; old = was) {
        }
        for (unsigned long long old = *top, was;; old = was) {
            const uint32_t q1 = (uint32_t)(old >> 32);
            if (t.w <= (uint32_t)old)
                break;
            const unsigned long long neu = t.w > q1 ? (unsigned long long)t.w << 32 | q1
                                                    : (unsigned long long)q1 << 32 | t.w;
            if ((was = atomicCAS(top, old, neu)) == old)
                break;
        }
    };
    auto meet = [&](uint32_t i, uint32_t k) {
        const uint32_t word = sh.bits[i >> 4], at = 2 * (i & 15);
        uint32_t both = word >> at & 3;
        if (!both)
            return;
        uint32_t slot = sh.before[i >> 4] + __popc(word & ((1u << at) - 1u));
        for (both = __popc(both); both; --both, ++slot) {
            const uint32_t h = atomicAdd(&sh.nhits, 1u);
            if (h < RANK_HITS)
                sh.hits[h] = k << 10 | slot;
            else
                divide_out(slot, k);
        }
    };
    const uint64_t h0 = m0 >> 1;
    const uint32_t nwarp = nq < RANK_BY_WARP ? nq : RANK_BY_WARP;
    for (uint32_t k = RANK_BY_PRIME + warp; k < nwarp; k += 8) {
        const uint4 t = g_trial_div[k];
        const uint32_t r = rank_mod(h0, t.w, t.z);
        for (uint32_t i = (r ? t.w - r : 0) + lane * t.w; i < span; i += 32 * t.w)
            meet(i, k);
    }
    for (uint32_t k = RANK_BY_WARP + tid; k < nq; k += 256) {
        const uint4 t = g_trial_div[k];
        const uint32_t r = rank_mod(h0, t.w, t.z);
        for (uint32_t i = r ? t.w - r : 0; i < span; i += t.w)
            meet(i, k);
    }
    __syncthreads();
    const uint32_t nhits = sh.nhits < RANK_HITS ? sh.nhits : RANK_HITS;
    for (uint32_t h = tid; h < nhits; h += 256)
        divide_out(sh.hits[h] & (RANK_TILE - 1), sh.hits[h] >> 10);
    __syncthreads();
    if (hi < MONT_NARROW_LIMIT)
        rank_tile_powers<FAM, true>(job, list, sh, n);
    else
        rank_tile_powers<FAM, false>(job, list, sh, n);
    return true;
}

// The powers of a tile.  A prime with S < D has a(p) | S only by chance
// (about S/D): one power rules most out.  S = D is certain to hold a(p), but
// then its two largest primes q1 > q2 with q1 q2 > amax cannot both divide an
// a(p) that gives a hit: F(S without q1) and F(S without q2) both non-zero
// rule the prime out.  What is left (few) has its rank taken prime by prime.
// The first powers are taken in the order of their exponents' lengths, so
// the lanes of a warp run about as long.
template <uint32_t FAM, bool NARROW>
__device__ __forceinline__ void rank_tile_powers(const JobView &job, const RankList &list, RankShared &sh, uint32_t n)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint64_t amax = FAM == LUCAS ? 2 * (job.n1 - 1) : job.n1 - 1;
    constexpr uint32_t SLOT = 0x7ffu, SMOOTH = 0x800u;
    // exponents, and their lengths counted
    for (uint32_t i = tid; i < n; i += 256) {
        const uint64_t p = sh.p[i], S = sh.S[i];
        const uint32_t q1 = (uint32_t)(sh.top[i] >> 32), q2 = (uint32_t)sh.top[i];
        const bool smooth = S >= p - 1;
        uint64_t E = S;
        if (FAM != MERSENNE && p == 5) {
            E = 0;
            sh.finish[atomicAdd(&sh.nfinish, 1u)] = (uint16_t)i;
        } else if (smooth) {
            if (q2 && (uint64_t)q1 * q2 > amax) {
                E = rank_without(S, q1);
            } else {
                E = 0;
                sh.finish[atomicAdd(&sh.nfinish, 1u)] = (uint16_t)i;
            }
        }
        sh.E[i] = E;
        if (E)
            atomicAdd(&sh.bins[63 - __clzll((long long)E)], 1u);
    }
    __syncthreads();
    if (warp == 0) {  // the longest first
        const uint32_t c1 = sh.bins[63 - 2 * lane], c0 = sh.bins[62 - 2 * lane];
        uint32_t x = c1 + c0;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            x += lane >= (uint32_t)o ? y : 0;
        }
        sh.bins[63 - 2 * lane] = x - c0 - c1;
        sh.bins[62 - 2 * lane] = x - c0;
        if (lane == 31)
            sh.nhits = x;
    }
    __syncthreads();
    const uint32_t npow = sh.nhits;
    for (uint32_t i = tid; i < n; i += 256) {
        const uint64_t E = sh.E[i];
        if (E)
            sh.order[atomicAdd(&sh.bins[63 - __clzll((long long)E)], 1u)] =
                (uint16_t)(i | (sh.S[i] >= sh.p[i] - 1 ? SMOOTH : 0));
    }
    __syncthreads();
    for (uint32_t k = tid; k < npow; k += 256) {
        const uint32_t o = sh.order[k], i = o & SLOT;
        FamilyPowers<FAM, NARROW> w;
        w.init(sh.p[i]);
        if (w.zero_at(sh.E[i]))
            sh.finish[atomicAdd(&sh.nfinish, 1u)] = (uint16_t)i;
        else if (o & SMOOTH)
            sh.second[atomicAdd(&sh.nsecond, 1u)] = (uint16_t)i;
    }
    __syncthreads();
    const uint32_t nsecond = sh.nsecond;
    for (uint32_t k = tid; k < nsecond; k += 256) {
        const uint32_t i = sh.second[k];
        FamilyPowers<FAM, NARROW> w;
        w.init(sh.p[i]);
        if (w.zero_at(rank_without(sh.S[i], (uint32_t)sh.top[i])))
            sh.finish[atomicAdd(&sh.nfinish, 1u)] = (uint16_t)i;
    }
    __syncthreads();
    // hand them on; without room in the list they are taken here
    const uint32_t nfinish = sh.nfinish;
    if (tid == 0)
        sh.nhits = atomicAdd(list.count, nfinish);
    __syncthreads();
    for (uint32_t k = tid; k < ((nfinish + 31) & ~31u); k += 256) {
        const uint32_t i = k < nfinish ? sh.finish[k] : 0, at = sh.nhits + k;
        const bool mine = k < nfinish && at >= list.cap;
        if (k < nfinish && !mine)
            list.items[at] = RankItem{sh.p[i], sh.S[i], sh.top[i]};
        if (__any_sync(0xffffffffu, mine))
            rank_push<FAM, NARROW>(job, list, mine, sh.p[i], sh.S[i], sh.top[i]);
    }
}

// Mersenne: a tile's primes each by itself, p - 1 divided by every prime below e
__device__ __noinline__ void rank_alone(const JobView &job, const RankList &list, const uint64_t *__restrict__ primes,
                                        uint32_t n, uint32_t nq)
{
    for (uint32_t k = threadIdx.x; k < ((n + 31) & ~31u); k += 256) {
        const uint64_t p = k < n ? primes[k] : 3, D = p - 1;
        uint64_t S = D & (0 - D);
        unsigned long long top = 0;
        for (uint32_t i = 0; i < nq; ++i) {
            const uint4 t = g_trial_div[i];
            const uint64_t inv = (uint64_t)t.y << 32 | t.x;
            uint64_t x = D * inv;
            if (__umul64hi(x, t.w) != 0)
                continue;
            do {
                S *= t.w;
                x *= inv;
            } while (__umul64hi(x, t.w) == 0);
            top = (unsigned long long)t.w << 32 | top >> 32;
        }
        OrderPowers<false> w;
        w.init(p);
        rank_push<MERSENNE, false>(job, list, k < n && w.zero_at(S), p, S, top);
    }
}

// A list that may hold any primes is looked over first: sparse counts its tiles
// that do not fit the bitmap.  Such a tile is walked item by item in
// rank_kernel, by two or three times the time that the same items take in a
// grid of their own (one prime in three of a 2^26-wide range at 2^33:
// n = 1..50000, 10.6 ms and 5.0; n = 1..200000, 17.0 and 5.6), while a tile that
// fits takes an eighth of it.  So a list with more than a quarter of sparse
// tiles goes to rank_walk_kernel.  (sparse null: a dense list.)
__device__ __forceinline__ bool rank_sparse(const uint32_t *sparse, uint64_t nprimes, uint32_t tile)
{
    return sparse && 4ull * *sparse > (nprimes + tile - 1) / tile;
}

// a warp a tile; bound by the latency of reading the list once, by few warps: 31 us
// for 5.7 million primes from DRAM, 2 % of rank_kernel's 1.2 ms for them (n = 1..50000;
// reads unrolled by eight take as long)
__global__ void __launch_bounds__(256) rank_fit_kernel(const uint64_t *__restrict__ primes, uint64_t nprimes,
                                                       uint32_t tile, uint32_t *sparse)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t ntiles = (nprimes + tile - 1) / tile;
    uint32_t count = 0;
    for (uint64_t t = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5); t < ntiles; t += (uint64_t)gridDim.x * 8) {
        const uint64_t *const p = primes + t * tile;
        const uint32_t n = (uint32_t)(nprimes - t * tile < tile ? nprimes - t * tile : tile);
        uint64_t lo = ~0ull, hi = 0;
        bool fits = true;
        for (uint32_t i = lane; i < n; i += 32) {
            const uint64_t x = p[i];
            lo = x < lo ? x : lo;
            hi = x > hi ? x : hi;
            fits &= (x & 1) && !(i + 1 < n && p[i + 1] == x);  // a repeat fills its mark twice
        }
        for (int o = 16; o; o >>= 1) {
            const uint64_t l = __shfl_xor_sync(0xffffffffu, lo, o), h = __shfl_xor_sync(0xffffffffu, hi, o);
            lo = l < lo ? l : lo;
            hi = h > hi ? h : hi;
        }
        count += !rank_fits(__all_sync(0xffffffffu, fits), lo, hi);
    }
    if (lane == 0 && count)
        atomicAdd(sparse, count);
}

// the walk, item by item, of a list that is too sparse for tiles
template <uint32_t FAM>
__global__ void __launch_bounds__(256, min_ctas_per_sm(FAM))
rank_walk_kernel(JobView job, const uint64_t *__restrict__ primes, uint64_t nprimes, uint32_t tile,
                 unsigned long long *next, const uint32_t *sparse)
{
    if (rank_sparse(sparse, nprimes, tile))
        residue_items<FAM>(job, primes, nprimes, next);
}

// Bound by integer issue (61 % of the slots, 20 of 32 lanes): the powers, about
// 20 bits of two narrow Montgomery products each, are the largest part, then
// the marks and the primes' multiples.  A tile of 1024 primes shares one walk
// over the 5133 primes below 50000.  The 2.8 million primes of a 2^26-wide
// segment at 2^34, n = 1..50000: 8.35 ms dividing each order by every prime,
// 1.82 ms here with the multiples divided out where they are met, 0.92 with
// them noted first, 0.74 + 0.13 with the last ranks in their own kernel.
template <uint32_t FAM>
__global__ void __launch_bounds__(256, RANK_CTAS)
rank_kernel(JobView job, const uint64_t *__restrict__ primes, uint64_t nprimes, uint32_t tile, unsigned long long *next,
            const uint32_t *sparse, RankList list)
{
    if (rank_sparse(sparse, nprimes, tile))
        return;
    extern __shared__ __align__(16) unsigned char rank_smem[];
    RankShared &sh = *reinterpret_cast<RankShared *>(rank_smem);
    const uint64_t ntiles = (nprimes + tile - 1) / tile;
    const uint32_t nq = trial_count(job.n1 - 1);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0)
            sh.lo = atomicAdd(next, 1ull);
        __syncthreads();
        const uint64_t t = sh.lo;
        if (t >= ntiles)
            break;
        const uint64_t first = t * tile;
        const uint32_t n = (uint32_t)(nprimes - first < tile ? nprimes - first : tile);
        if (!rank_tile<FAM>(job, list, sh, primes + first, n, nq)) {
            // a sparse or unordered stretch of the list: item by item
            if constexpr (FAM == MERSENNE)  // (its walks' filter has no room here)
                rank_alone(job, list, primes + first, n, nq);
            else
                for (uint64_t k = threadIdx.x; k < (uint64_t)n * job.tiles; k += 256)
                    residue_item<FAM>(job, primes + first, n, k);
        }
    }
}

// the listed primes' ranks and hits
template <uint32_t FAM>
__global__ void __launch_bounds__(256) rank_finish_kernel(JobView job, RankList list)
{
    const uint32_t n = *list.count < list.cap ? *list.count : list.cap;
    for (uint32_t k = blockIdx.x * 256 + threadIdx.x; k < ((n + 31) & ~31u); k += gridDim.x * 256) {
        const bool mine = k < n;
        const RankItem it = mine ? list.items[k] : RankItem{0, 0, 0};
        if (__any_sync(0xffffffffu, it.p >= MONT_NARROW_LIMIT))
            rank_push<FAM, false>(job, list, mine, it.p, it.S, it.top);
        else
            rank_push<FAM, true>(job, list, mine, it.p, it.S, it.top);
    }
}

// the hits of the primes that have many, 32 chunks of each prime's over the warps
__global__ void __launch_bounds__(256) rank_heavy_kernel(JobView job, RankList list)
{
    constexpr uint32_t CHUNKS = 32;
    const uint32_t n = *list.nheavy < list.heavy_cap ? *list.nheavy : list.heavy_cap, lane = threadIdx.x & 31u;
    for (uint32_t id = (blockIdx.x * 256 + threadIdx.x) >> 5; id < n * CHUNKS; id += gridDim.x * 8) {
        const RankHits h = list.heavy[id % n];
        for (uint64_t x = h.first + (id / n * 32 + lane) * h.a; x < job.n1; x += CHUNKS * 32 * h.a)
            push(job.fb, x - job.n0, h.p);
    }
}

// whether a job's primes go by tiles of ranks
inline bool takes_ranks(const JobView &v)
{
    const bool mersenne = v.family == MERSENNE && (v.list == LIST_DENSE || v.list == LIST_WIDE);
    const bool ranks = (v.family == FIBONACCI || v.family == LUCAS) && v.list <= LIST_DENSE;
    return (ranks || mersenne) && v.variant == CTD_VARIANT_AUTO && v.n0 >= 1 &&
           v.n1 <= TRIAL_LIMIT && v.n1 - v.n0 >= (mersenne ? order_min_terms(v.n1) : rank_min_terms(v.n1));
}

// room for the list: a few in a hundred primes are listed at 2^34, half of
// them and more below 2^20, where all of a list's primes have room
static uint32_t rank_list_cap(uint64_t nprimes)
{
    const uint64_t most = 1u << 20;
    const uint64_t want = nprimes < most ? nprimes : most + nprimes / 8;
    return (uint32_t)(want < (1u << 30) ? want : 1u << 30);
}

template <uint32_t FAM>
static cudaError_t launch_ranks(const JobView &v, const uint64_t *d_primes, uint64_t n, int sm_count, int walk_grid,
                                int walk_block, cudaStream_t st, ClassCounters *counters, const RankList &list)
{
    cudaError_t e = allow_smem(rank_kernel<FAM>, sizeof(RankShared));
    if (e == cudaSuccess)
        e = cudaMemsetAsync(counters, 0, sizeof(*counters), st);
    if (e != cudaSuccess)
        return e;
    // a short list in small tiles, so that every CTA has one
    const uint64_t grid = (uint64_t)sm_count * RANK_CTAS;
    const uint64_t per = (n + grid - 1) / grid;
    const uint32_t tile = per < RANK_TILE ? (uint32_t)per : RANK_TILE;
    const uint64_t ntiles = (n + tile - 1) / tile;
    const bool any = FAM != MERSENNE && v.list == LIST_ANY;
    // The primes of sparse tiles: each by one rank for the whole index range,
    // where there are threads' worth of them or a long range makes up for its
    // latency (0.65 ms for n = 1..50000, however few the primes).  n = 1..50000,
    // 584,000 primes around 2^34: 4.1 ms in index tiles, 2.0 whole; 29,000 at
    // 2^33: 0.38 and 0.67.
    JobView w = v;
    walk_block = walk_block < 256 ? walk_block : 256;
    const uint64_t threads = (uint64_t)walk_grid * walk_block;
    if (any && fibonacci_rank_pays(v.n0, v.n1) && (n >= threads || (4 * n >= threads && v.n1 >= 1u << 14))) {
        w.tiles = 1;
        w.tile_len = v.n1 - v.n0;
    }
    uint32_t *const sparse = any ? &counters->nlisted[0] : nullptr;
    if (any) {
        const uint64_t blocks = (ntiles + 7) / 8;
        rank_fit_kernel<<<(unsigned)(blocks < grid ? blocks : grid), 256, 0, st>>>(d_primes, n, tile, sparse);
        e = cudaGetLastError();
        if (e != cudaSuccess)
            return e;
        note_kernel_launch();
    }
    rank_kernel<FAM><<<(unsigned)(ntiles < grid ? ntiles : grid), 256, sizeof(RankShared), st>>>(
        w, d_primes, n, tile, &counters->next, sparse, list);
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    if constexpr (FAM != MERSENNE)
        if (any) {
            note_kernel_launch();
            rank_walk_kernel<FAM><<<walk_grid, walk_block, 0, st>>>(w, d_primes, n, tile, &counters->next, sparse);
            e = cudaGetLastError();
            if (e != cudaSuccess)
                return e;
        }
    if (!list.cap)  // no list: the tiles have finished their primes and pushed all hits
        return cudaSuccess;
    note_kernel_launch();
    const uint64_t blocks = ((list.cap < n ? list.cap : n) + 255) / 256;
    rank_finish_kernel<FAM><<<(unsigned)(blocks < grid ? blocks : grid), 256, 0, st>>>(v, list);
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    note_kernel_launch();
    rank_heavy_kernel<<<(unsigned)sm_count * 4, 256, 0, st>>>(v, list);
    return cudaGetLastError();
}

}  // namespace ctd

// ctd_sieve.cu -- device segmented sieve of Eratosthenes.
//
// Replaces the reference's host siever (src/siever.hpp:179-237: primesieve
// on `threads` host workers) and the synchronous host-to-device copy of each
// segment's primes (src/prime_data.hpp:166-196).  Primes are produced on the
// GPU and written straight into an HBM chunk, ascending, as u64.
//
// Layout: odd numbers only, one bit each.  A window is WIN_WORDS 32-bit words
// (2^19 odd numbers, a 2^20-wide range) held in shared memory.
//   pass 0  sieve_starts: every base prime's first multiple in the range;
//   pass 1  sieve_windows: each CTA clears a window, crosses off multiples
//           of every odd base prime p (p^2 below the window end) with
//           shared-memory atomics, writes the prime bitmap to global memory
//           and its popcount a chunk (CHUNK_WORDS);
//   pass 2  scan_counts: exclusive scan of the chunk counts (one CTA);
//   pass 3  compact: each CTA re-reads a chunk's bitmap and writes its
//           primes at the chunk's offset, a warp a run of words.
// Short ranges take quarter windows, so that every SM has some.
// Base primes (all odd p <= sqrt(hi)) come from the same kernels: the odd
// primes below 2^16 from a one-CTA sieve, the rest by sieving [3, sqrt(hi)].
#include "ctd_internal.h"

#include <algorithm>
#include <cmath>
#include <vector>

namespace ctd {

namespace {

constexpr uint32_t WIN_WORDS = 16384;                       // 64 KiB of shared memory
constexpr uint64_t WIN_ODD = 32ull * WIN_WORDS;             // odd numbers per window
constexpr uint32_t CHUNK_WORDS = WIN_WORDS / SIEVE_WIN_CHUNKS;  // unit of the counts and the compaction; a short range's window
constexpr int SIEVE_THREADS = 1024;
constexpr int COMPACT_THREADS = 256;
constexpr uint32_t LEVEL0_LIMIT = 65536;                    // level-0 base primes: odd p < 2^16

#define CUDA_TRY(expr)                                                      \
    do {                                                                    \
        cudaError_t e_ = (expr);                                            \
        if (e_ != cudaSuccess) {                                            \
            err = std::string(#expr ": ") + cudaGetErrorString(e_);         \
            return e_ == cudaErrorMemoryAllocation ? CTD_ERR_OUT_OF_MEMORY  \
                                                   : CTD_ERR_CUDA;          \
        }                                                                   \
    } while (0)

// index (in odd steps from wlo) of the first odd multiple of p at or above wlo
__device__ __forceinline__ uint64_t first_multiple(uint32_t p, uint64_t wlo)
{
    const uint64_t r = wlo % p;
    uint64_t m = r ? wlo + (p - r) : wlo;
    if (!(m & 1))
        m += p;
    return (m - wlo) >> 1;
}

// What a window needs of a base prime to find its first multiple there by
// 32-bit arithmetic: the first multiple's index in the whole range, and
// floor((2^32 - 1) / p).  A 64-bit division per prime and window -- and, for
// the primes that a whole CTA crosses off, per thread -- was most of the
// sieve's instructions.
struct SieveStart {
    uint32_t first, recip;
};
__global__ void __launch_bounds__(256) sieve_starts(uint64_t lo_odd, uint64_t last, const uint32_t *__restrict__ base,
                                                    uint32_t nbase, SieveStart *__restrict__ starts)
{
    for (uint32_t k = blockIdx.x * 256 + threadIdx.x; k < nbase; k += gridDim.x * 256) {
        const uint32_t p = base[k];
        if ((uint64_t)p * p > last)
            break;
        starts[k] = SieveStart{(uint32_t)first_multiple(p, lo_odd), 0xffffffffu / p};
    }
}

// index in the window at wlo = lo_odd + 2 off of the first multiple of p to
// cross off: the first at or above max(p^2, wlo)
template <bool STARTS>
__device__ __forceinline__ uint64_t first_index(uint32_t p, uint64_t wlo, uint32_t off,
                                                const SieveStart *__restrict__ starts, uint32_t k)
{
    const uint64_t pp = (uint64_t)p * p;
    if (pp >= wlo)
        return (pp - wlo) >> 1;
    if (!STARTS)
        return first_multiple(p, wlo);
    const SieveStart s = starts[k];
    // off mod p: the quotient is one short at most (2p fits 32 bits, or p > off)
    uint32_t r = off - __umulhi(off, s.recip) * p;
    r = r >= p ? r - p : r;
    return s.first >= r ? s.first - r : s.first + (p - r);
}

// The wheel: the odd primes 3..31, whose multiples take most of a
// window's crossings (sum of 1/q = 1.06 of about 2.3 for all base primes).
// Their multiples in a word of 32 odd numbers are a fixed bit pattern
// shifted to the word's phase, so each word gets them by shifts and ORs
// written once, not by shared-memory atomics bit by bit.
constexpr int WHEEL = 10;
__host__ __device__ constexpr uint32_t wheel_q(int k)
{
    return k < 5 ? (k < 3 ? 3 + 2 * k : (k == 3 ? 11 : 13)) : (k < 8 ? (k == 5 ? 17 : (k == 6 ? 19 : 23)) : (k == 8 ? 29 : 31));
}

// bits 0, q, 2q, ... of a 32-bit word
__host__ __device__ constexpr uint32_t wheel_pattern(uint32_t q)
{
    uint32_t m = 0;
    for (uint32_t b = 0; b < 32; b += q)
        m |= 1u << b;
    return m;
}

// One CTA a window of win_words words.  Bound by the crossings in shared
// memory: a warp crosses off up to 32 multiples an atomic, their banks at
// random.
template <bool STARTS>
__global__ void __launch_bounds__(SIEVE_THREADS) sieve_windows(uint64_t lo_odd, uint64_t nodd, uint32_t nwin,
                                                               uint32_t win_words, const uint32_t *__restrict__ base,
                                                               uint32_t nbase, const SieveStart *__restrict__ starts,
                                                               uint32_t *__restrict__ bits, uint32_t *__restrict__ ccount)
{
    extern __shared__ uint32_t sm[];
    __shared__ uint32_t chunk_count[WIN_WORDS / CHUNK_WORDS];
    const uint32_t tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = bd >> 5;
    const uint32_t win_odd = 32 * win_words;
    for (uint32_t w = blockIdx.x; w < nwin; w += gridDim.x) {
        const uint64_t off = (uint64_t)w * win_odd;
        const uint64_t wlo = lo_odd + 2 * off;
        const uint32_t len = (uint32_t)((nodd - off) < win_odd ? (nodd - off) : win_odd);
        const uint64_t last = wlo + 2 * (uint64_t)(len - 1);  // (not one past it: that may be 2^64)
        {
            // bit b of word i is the odd number wlo + 2 (32 i + b); it is a
            // multiple of q iff its odd index g = (value - 1) / 2 is
            // (q - 1) / 2 mod q, so in word i the multiples start at bit
            // ph = ((q - 1) / 2 - g(i, 0)) mod q, and moving on by bd words
            // lowers ph by 32 bd mod q
            const uint64_t g0 = (wlo - 1) / 2 + 32ull * tid;
            uint32_t ph[WHEEL], step[WHEEL];
#pragma unroll
            for (int k = 0; k < WHEEL; ++k) {
                const uint32_t q = wheel_q(k);
                const uint32_t gm = (uint32_t)(g0 % q);
                const uint32_t h = (q - 1) / 2;
                ph[k] = h >= gm ? h - gm : h + q - gm;
                step[k] = (32u * bd) % q;
            }
            for (uint32_t i = tid; i < win_words; i += bd) {
                uint32_t v = 0;
#pragma unroll
                for (int k = 0; k < WHEEL; ++k) {
                    const uint32_t q = wheel_q(k);
                    v |= wheel_pattern(q) << ph[k];
                    ph[k] = ph[k] >= step[k] ? ph[k] - step[k] : ph[k] + q - step[k];
                }
                sm[i] = v;
            }
        }
        if (tid < WIN_WORDS / CHUNK_WORDS)
            chunk_count[tid] = 0;
        __syncthreads();
        if (tid == 0 && wlo <= wheel_q(WHEEL - 1)) {
            // the wheel primes themselves are not composite
            for (int k = 0; k < WHEEL; ++k) {
                const uint64_t q = wheel_q(k);
                if (q >= wlo && q <= last) {
                    const uint64_t j = (q - wlo) >> 1;
                    sm[j >> 5] &= ~(1u << (j & 31));
                }
            }
        }
        __syncthreads();
        // primes past the wheel with 32 multiples and more in the window: a
        // warp a prime (base[] starts with the wheel primes 3..31)
        uint32_t k = WHEEL + warp;
        for (; k < nbase; k += nwarps) {
            const uint32_t p = base[k];
            if (p > win_odd / 32 || (uint64_t)p * p > last)
                break;
            const uint64_t j0 = first_index<STARTS>(p, wlo, (uint32_t)off, starts, k);
            if (j0 >= len)
                continue;
            for (uint32_t j = (uint32_t)j0 + lane * p; j < len; j += 32 * p)
                atomicOr(&sm[j >> 5], 1u << (j & 31));
        }
        // the others: a prime a thread.  The warps left the list at different
        // places; the first prime above the bound is where this part starts
        {
            uint32_t a = WHEEL, b = nbase;
            while (a < b) {
                const uint32_t mid = (a + b) >> 1;
                if (base[mid] <= win_odd / 32)
                    a = mid + 1;
                else
                    b = mid;
            }
            k = a + tid;
        }
        // (the next prime is loaded while this one's multiples are crossed off)
        uint32_t p = k < nbase ? base[k] : 0;
        while (k < nbase && (uint64_t)p * p <= last) {
            const uint32_t next = k + bd, pn = next < nbase ? base[next] : 0;
            const uint64_t j0 = first_index<STARTS>(p, wlo, (uint32_t)off, starts, k);
            if (j0 < len) {
                uint32_t j = (uint32_t)j0;
                do {
                    atomicOr(&sm[j >> 5], 1u << (j & 31));
                    j = p < len - j ? j + p : len;
                } while (j < len);
            }
            k = next;
            p = pn;
        }
        __syncthreads();
        uint32_t *out = bits + (uint64_t)w * win_words;
        for (uint32_t c = 0; c < win_words; c += CHUNK_WORDS) {
            uint32_t cnt = 0;
            for (uint32_t i = c + tid; i < c + CHUNK_WORDS; i += bd) {
                uint32_t v = ~sm[i];
                const uint32_t j = i * 32;
                if (j + 32 > len)
                    v = (j >= len) ? 0u : (v & ((1u << (len - j)) - 1u));
                out[i] = v;
                cnt += __popc(v);
            }
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            if (lane == 0)
                atomicAdd(&chunk_count[c / CHUNK_WORDS], cnt);
        }
        __syncthreads();
        if (tid < win_words / CHUNK_WORDS)
            ccount[(uint64_t)w * (win_words / CHUNK_WORDS) + tid] = chunk_count[tid];
        __syncthreads();
    }
}

// exclusive scan of chunk counts into 64-bit offsets; offsets[n] = total
__global__ void __launch_bounds__(1024) scan_counts(const uint32_t *__restrict__ wcount, uint32_t nwin,
                                                    uint64_t *__restrict__ offsets)
{
    __shared__ uint64_t warp_sums[32];
    __shared__ uint64_t carry;
    const uint32_t tid = threadIdx.x;
    if (tid == 0)
        carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < nwin; base += blockDim.x) {
        const uint32_t i = base + tid;
        uint64_t v = i < nwin ? wcount[i] : 0;
        uint64_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((tid & 31) >= (uint32_t)o)
                x += y;
        }
        if ((tid & 31) == 31)
            warp_sums[tid >> 5] = x;
        __syncthreads();
        if (tid < 32) {
            uint64_t s = (tid < blockDim.x / 32) ? warp_sums[tid] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                uint64_t y = __shfl_up_sync(0xffffffffu, s, o);
                if (tid >= (uint32_t)o)
                    s += y;
            }
            warp_sums[tid] = s;  // inclusive scan of warp totals
        }
        __syncthreads();
        const uint64_t warp_prefix = (tid >> 5) ? warp_sums[(tid >> 5) - 1] : 0;
        if (i < nwin)
            offsets[i] = carry + warp_prefix + x - v;
        __syncthreads();
        if (tid == 0)
            carry += warp_sums[blockDim.x / 32 - 1];
        __syncthreads();
    }
    if (tid == 0)
        offsets[nwin] = carry;
}

// A CTA a chunk of the bitmap, each warp a run of its words, 32 words at a
// time: the words' primes are written in one stretch of a few hundred bytes,
// a prime a lane and store.  With one CTA a window and a block scan for each
// of its 32 rounds, the primes of a 2^26-wide range took 54 us to write.
template <class T>
__global__ void __launch_bounds__(COMPACT_THREADS) compact_chunks(uint64_t lo_odd, uint32_t nchunks,
                                                                  const uint32_t *__restrict__ bits,
                                                                  const uint64_t *__restrict__ offsets,
                                                                  T *__restrict__ out, uint64_t capacity,
                                                                  uint64_t out_base)
{
    constexpr int WARPS = COMPACT_THREADS / 32, ROUNDS = CHUNK_WORDS / COMPACT_THREADS;
    __shared__ uint32_t warp_count[WARPS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const uint32_t first = warp * (32 * ROUNDS) + lane;  // word of round 0
        const uint32_t *wb = bits + (uint64_t)c * CHUNK_WORDS + first;
        uint32_t v[ROUNDS], cnt = 0;
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            v[r] = wb[32 * r];
            cnt += __popc(v[r]);
        }
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0)
            warp_count[warp] = cnt;
        __syncthreads();
        uint64_t pos = out_base + offsets[c];
        for (uint32_t k = 0; k < warp; ++k)
            pos += warp_count[k];
        const uint64_t value = lo_odd + 64 * ((uint64_t)c * CHUNK_WORDS + first);
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const uint32_t n = __popc(v[r]);
            uint32_t x = n;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                x += lane >= (uint32_t)o ? y : 0;
            }
            uint64_t at = pos + x - n;
            for (uint32_t m = v[r]; m; m &= m - 1) {
                if (at < capacity)
                    out[at] = (T)(value + 64 * 32 * r + 2 * (__ffs(m) - 1));
                ++at;
            }
            pos += __shfl_sync(0xffffffffu, x, 31);
        }
        __syncthreads();
    }
}

// odd primes below 2^16 by one CTA: cross off multiples of every odd k < 256
__global__ void __launch_bounds__(1024) level0_primes(uint32_t *__restrict__ out, uint32_t *__restrict__ count)
{
    constexpr uint32_t NW = LEVEL0_LIMIT / 64;  // odd numbers 1,3,..,65535 -> 32768 bits
    __shared__ uint32_t sm[NW];
    __shared__ uint32_t warp_sums[32];
    const uint32_t tid = threadIdx.x;
    for (uint32_t i = tid; i < NW; i += blockDim.x)
        sm[i] = 0;
    __syncthreads();
    if (tid == 0)
        atomicOr(&sm[0], 1u);  // 1 is not prime
    // (a warp a k: with a thread a k, the multiples of 3 alone took 176 us)
    for (uint32_t k = 3 + 2 * (tid >> 5); k < 256; k += 2 * (blockDim.x >> 5))
        for (uint32_t m = k * k + 2 * k * (tid & 31); m < LEVEL0_LIMIT; m += 64 * k)
            atomicOr(&sm[(m >> 1) >> 5], 1u << ((m >> 1) & 31));
    __syncthreads();
    // ordered compaction, one word per thread (NW = 1024 = blockDim)
    uint32_t v = tid < NW ? ~sm[tid] : 0u;
    if (tid == 0)
        v &= ~1u;  // drop 1 (already marked) -- keep explicit
    uint32_t c = __popc(v), x = c;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if ((tid & 31) >= (uint32_t)o)
            x += y;
    }
    if ((tid & 31) == 31)
        warp_sums[tid >> 5] = x;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (uint32_t k = 0; k < blockDim.x / 32; ++k) {
        if (k < (tid >> 5))
            before += warp_sums[k];
        total += warp_sums[k];
    }
    uint32_t pos = before + x - c;
    while (v) {
        uint32_t b = __ffs(v) - 1;
        v &= v - 1;
        out[pos++] = 2 * (tid * 32 + b) + 1;
    }
    if (tid == 0)
        *count = total;
}

uint64_t isqrt64(uint64_t x)
{
    uint64_t r = (uint64_t)std::sqrt((long double)x);
    while (r * r > x)
        --r;
    while ((r + 1) <= 0xffffffffull && (r + 1) * (r + 1) <= x)
        ++r;
    return r;
}

}  // namespace

struct SieveWorkspace {
    // base primes (odd, ascending) covering [3, base_limit]
    uint32_t *d_base = nullptr;
    uint32_t nbase = 0;
    uint64_t base_limit = 0;
    size_t base_cap = 0;
    SieveStart *d_starts = nullptr;  // one a base prime, of the last range sieved
    size_t starts_cap = 0;
    // per-range scratch
    uint32_t *d_bits = nullptr;
    size_t bits_cap = 0;  // windows
    uint32_t *d_wcount = nullptr;  // SIEVE_WIN_CHUNKS a window
    uint64_t *d_offsets = nullptr;
    size_t win_cap = 0;
    uint64_t *h_total = nullptr;  // pinned
    int sm_count = 0;
};

SieveWorkspace *sieve_workspace_create()
{
    auto *ws = new SieveWorkspace();
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&ws->sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (ws->sm_count <= 0)
        ws->sm_count = 1;
    return ws;
}

void sieve_workspace_destroy(SieveWorkspace *ws)
{
    if (!ws)
        return;
    cudaFree(ws->d_base);
    cudaFree(ws->d_starts);
    cudaFree(ws->d_bits);
    cudaFree(ws->d_wcount);
    cudaFree(ws->d_offsets);
    cudaFreeHost(ws->h_total);
    delete ws;
}

static int ensure_windows(SieveWorkspace *ws, uint64_t nwin, std::string &err)
{
    if (nwin > ws->win_cap) {
        cudaFree(ws->d_bits);
        cudaFree(ws->d_wcount);
        cudaFree(ws->d_offsets);
        ws->d_bits = nullptr;
        ws->d_wcount = nullptr;
        ws->d_offsets = nullptr;
        ws->win_cap = 0;
        CUDA_TRY(cudaMalloc(&ws->d_bits, nwin * WIN_WORDS * sizeof(uint32_t)));
        CUDA_TRY(cudaMalloc(&ws->d_wcount, nwin * SIEVE_WIN_CHUNKS * sizeof(uint32_t)));
        CUDA_TRY(cudaMalloc(&ws->d_offsets, (nwin * SIEVE_WIN_CHUNKS + 1) * sizeof(uint64_t)));
        ws->win_cap = nwin;
    }
    if (!ws->h_total)
        CUDA_TRY(cudaMallocHost(&ws->h_total, sizeof(uint64_t)));
    return CTD_OK;
}

// room for a start a base prime; without the memory for it (8 bytes each) the
// windows divide for themselves
static void ensure_starts(SieveWorkspace *ws)
{
    if (ws->nbase <= ws->starts_cap)
        return;
    cudaFree(ws->d_starts);
    ws->d_starts = nullptr;
    ws->starts_cap = 0;
    if (cudaMalloc(&ws->d_starts, ws->nbase * sizeof(SieveStart)) == cudaSuccess)
        ws->starts_cap = ws->nbase;
    else
        (void)cudaGetLastError();
}

// Launches the passes over the odd numbers lo_odd .. lo_odd + 2 (nodd - 1),
// nodd > 0, into d_out[out_base ...]; the number of chunks is returned (the
// count of primes is left at offsets[chunks]).  starts: room for one a base
// prime, or null (the windows then divide for themselves).
template <class T>
static int launch_sieve(uint64_t lo_odd, uint64_t nodd, const uint32_t *d_base, uint32_t nbase, SieveStart *starts,
                        uint32_t *bits, uint32_t *ccount, uint64_t *offsets, int sm_count, T *d_out, uint64_t capacity,
                        uint64_t out_base, uint32_t *chunks, cudaStream_t st, std::string &err)
{
    // Whole windows where they give half the SMs one, else chunks as windows;
    // 1024 threads a window while the windows are few.  A 2^27-wide range at
    // 2^40 (82,000 base primes a window): 140 us with its 128 whole windows,
    // 226 with 512 chunks; a 2^26-wide one at 2^33: 80 us with 256 chunks of
    // 512 threads, 84 with 1024 and 105 with 64 whole windows; a 2^20-wide one
    // 57 us with 1024 threads a chunk and 68 with 512; a 2^28-wide one 194 us
    // with 1024 threads a whole window, a 2^29-wide one 355, and 335 with 512.
    const uint64_t full = (nodd + WIN_ODD - 1) / WIN_ODD;
    const uint32_t win_words = 2 * full >= (uint64_t)sm_count ? WIN_WORDS : CHUNK_WORDS;
    const uint64_t nwin = (nodd + 32ull * win_words - 1) / (32ull * win_words);
    const uint32_t nchunks = (uint32_t)(nwin * (win_words / CHUNK_WORDS));
    const int threads = nwin <= (uint64_t)sm_count * (win_words == WIN_WORDS ? 2 : 1) ? SIEVE_THREADS : SIEVE_THREADS / 2;
    const size_t smem = win_words * sizeof(uint32_t);
    if (nodd >> 32)
        starts = nullptr;  // offsets in the range are 32-bit
    // a function attribute belongs to the current device: set it on every
    // call (a host-side call, no stream work), so a context on any device
    // launches with it
    CUDA_TRY(cudaFuncSetAttribute(starts ? sieve_windows<true> : sieve_windows<false>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(WIN_WORDS * sizeof(uint32_t))));
    if (starts) {
        const uint32_t blocks = (nbase + 255) / 256;
        sieve_starts<<<blocks < (uint32_t)sm_count * 4 ? blocks : (uint32_t)sm_count * 4, 256, 0, st>>>(
            lo_odd, lo_odd + 2 * (nodd - 1), d_base, nbase, starts);
        CUDA_TRY(cudaGetLastError());
        note_kernel_launch();
        sieve_windows<true><<<(unsigned)nwin, threads, smem, st>>>(lo_odd, nodd, (uint32_t)nwin, win_words, d_base, nbase,
                                                                   starts, bits, ccount);
    } else {
        sieve_windows<false><<<(unsigned)nwin, threads, smem, st>>>(lo_odd, nodd, (uint32_t)nwin, win_words, d_base,
                                                                    nbase, starts, bits, ccount);
    }
    CUDA_TRY(cudaGetLastError());
    note_kernel_launch();
    scan_counts<<<1, 1024, 0, st>>>(ccount, nchunks, offsets);
    CUDA_TRY(cudaGetLastError());
    note_kernel_launch();
    compact_chunks<T><<<nchunks, COMPACT_THREADS, 0, st>>>(lo_odd, nchunks, bits, offsets, d_out, capacity, out_base);
    CUDA_TRY(cudaGetLastError());
    note_kernel_launch();
    *chunks = nchunks;
    return CTD_OK;
}

// odd primes in [lo_odd, lo_odd + 2*nodd) into out[out_base ...], counts in ws
template <class T>
static int sieve_odd(SieveWorkspace *ws, uint64_t lo_odd, uint64_t nodd, const uint32_t *d_base, uint32_t nbase,
                     T *d_out, uint64_t capacity, uint64_t out_base, uint64_t *count, cudaStream_t st,
                     std::string &err)
{
    *count = 0;
    if (!nodd)
        return CTD_OK;
    const uint64_t nwin = (nodd + WIN_ODD - 1) / WIN_ODD;
    if (nwin * SIEVE_WIN_CHUNKS > 0x7fffffffull) {
        err = "sieve range too large";
        return CTD_ERR_INVALID_ARGUMENT;
    }
    int rc = ensure_windows(ws, nwin, err);
    if (rc)
        return rc;
    ensure_starts(ws);
    uint32_t chunks = 0;
    rc = launch_sieve<T>(lo_odd, nodd, d_base, nbase, nbase <= ws->starts_cap ? ws->d_starts : nullptr, ws->d_bits,
                         ws->d_wcount, ws->d_offsets, ws->sm_count, d_out, capacity, out_base, &chunks, st, err);
    if (rc)
        return rc;
    CUDA_TRY(cudaMemcpyAsync(ws->h_total, ws->d_offsets + chunks, sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    *count = *ws->h_total;
    return CTD_OK;
}

// make sure base primes cover every odd p <= limit
static int ensure_base(SieveWorkspace *ws, uint64_t limit, cudaStream_t st, std::string &err)
{
    if (ws->base_limit >= limit && ws->d_base)
        return CTD_OK;
    if (!ws->d_base) {
        ws->base_cap = 8192;
        CUDA_TRY(cudaMalloc(&ws->d_base, ws->base_cap * sizeof(uint32_t)));
        uint32_t *d_cnt = nullptr;
        CUDA_TRY(cudaMalloc(&d_cnt, sizeof(uint32_t)));
        level0_primes<<<1, 1024, 0, st>>>(ws->d_base, d_cnt);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) {
            note_kernel_launch();
            uint32_t n = 0;
            e = cudaMemcpyAsync(&n, d_cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess)
                e = cudaStreamSynchronize(st);
            ws->nbase = n;
        }
        cudaFree(d_cnt);
        if (e != cudaSuccess) {
            err = std::string("level-0 sieve: ") + cudaGetErrorString(e);
            return CTD_ERR_CUDA;
        }
        ws->base_limit = LEVEL0_LIMIT - 1;
    }
    if (ws->base_limit >= limit)
        return CTD_OK;
    // extend: odd primes in (base_limit, new_limit] sieved with the level-0 primes
    uint64_t new_limit = limit;
    if (new_limit > 0xffffffffull)
        new_limit = 0xffffffffull;
    // round up generously so later ranges rarely need another extension
    uint64_t grow = ws->base_limit * 2;
    if (new_limit < grow)
        new_limit = grow < 0xffffffffull ? grow : 0xffffffffull;
    const uint64_t lo_odd = (ws->base_limit + 1) | 1;
    const uint64_t nodd = new_limit >= lo_odd ? (new_limit - lo_odd) / 2 + 1 : 0;
    const uint64_t need = ws->nbase + prime_count_upper_bound(lo_odd, new_limit + 1) + 64;
    if (need > ws->base_cap) {
        uint32_t *nb = nullptr;
        CUDA_TRY(cudaMalloc(&nb, need * sizeof(uint32_t)));
        CUDA_TRY(cudaMemcpyAsync(nb, ws->d_base, ws->nbase * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
        CUDA_TRY(cudaStreamSynchronize(st));
        cudaFree(ws->d_base);
        ws->d_base = nb;
        ws->base_cap = need;
    }
    // level-0 primes (p < 2^16) suffice for any new_limit < 2^32
    uint32_t nlevel0 = 0;
    {
        // the level-0 prefix: all primes below 2^16 are the first entries
        nlevel0 = ws->nbase;  // base_limit >= 2^16 - 1 holds the level-0 list at the front
        // only primes < 2^16 are needed; they are a prefix of d_base
        // (6541 odd primes below 2^16)
        if (nlevel0 > 6541)
            nlevel0 = 6541;
    }
    uint64_t cnt = 0;
    int rc = sieve_odd<uint32_t>(ws, lo_odd, nodd, ws->d_base, nlevel0, ws->d_base, ws->base_cap, ws->nbase, &cnt,
                                 st, err);
    if (rc)
        return rc;
    ws->nbase += (uint32_t)cnt;
    ws->base_limit = new_limit;
    return CTD_OK;
}

uint64_t prime_count_upper_bound(uint64_t lo, uint64_t hi)
{
    if (hi <= lo)
        return 0;
    const double y = (double)(hi - lo);
    double bound = y;  // trivial
    if (y >= 3) {
        // Montgomery-Vaughan: pi(x + y) - pi(x) <= 2y / ln y for y > 1
        bound = std::min(bound, 2.0 * y / std::log(y));
    }
    if (hi > 17) {
        // Rosser-Schoenfeld / Dusart: x/ln x <= pi(x) (x >= 17), pi(x) < 1.25506 x / ln x (x > 1)
        const double up = 1.25506 * (double)hi / std::log((double)hi);
        const double low = lo >= 17 ? (double)lo / std::log((double)lo) : 0.0;
        bound = std::min(bound, up - low);
    }
    return (uint64_t)bound + 64;
}

// ------------------------------------------------ launch-only variant
// For the batched engine: base primes and window scratch are prepared once,
// then each segment is four kernel launches with the prime count left in
// device memory -- no allocation and no host wait, so a whole schedule of
// segments can be captured in one CUDA graph.
int sieve_prepare_base(SieveWorkspace *ws, uint64_t hi, cudaStream_t st, std::string &err)
{
    if (hi < 3)
        return CTD_OK;
    const int rc = ensure_base(ws, isqrt64(hi - 1), st, err);
    if (!rc)
        ensure_starts(ws);
    return rc;
}

int sieve_prepare_windows(SieveWorkspace *ws, uint64_t max_width, std::string &err)
{
    const uint64_t nwin = (max_width / 2 + 1 + WIN_ODD - 1) / WIN_ODD + 1;
    return ensure_windows(ws, nwin, err);
}

uint64_t sieve_state_key(const SieveWorkspace *ws)
{
    // FNV-1a over what sieve_odd_async's launches take besides the range
    const uint64_t parts[] = {(uint64_t)(uintptr_t)ws->d_base, ws->nbase, (uint64_t)(uintptr_t)ws->d_bits,
                              (uint64_t)(uintptr_t)ws->d_wcount, (uint64_t)(uintptr_t)ws->d_offsets,
                              (uint64_t)(uintptr_t)ws->d_starts, (uint64_t)ws->sm_count};
    uint64_t h = 1469598103934665603ull;
    for (uint64_t x : parts)
        for (int b = 0; b < 8; ++b) {
            h ^= (x >> (8 * b)) & 0xff;
            h *= 1099511628211ull;
        }
    return h;
}

int sieve_odd_async(SieveWorkspace *ws, uint64_t lo, uint64_t hi, uint64_t *d_out, uint64_t capacity,
                    const uint64_t **count_out, cudaStream_t st, std::string &err)
{
    const uint64_t lo_odd = lo < 3 ? 3 : (lo | 1);
    const uint64_t nodd = lo_odd < hi ? (hi - lo_odd + 1) / 2 : 0;
    const uint64_t nwin = nodd ? (nodd + WIN_ODD - 1) / WIN_ODD : 0;
    if (nwin > ws->win_cap || !ws->d_base) {
        err = "sieve scratch not prepared for this segment";
        return CTD_ERR_INVALID_ARGUMENT;
    }
    if (!nwin) {  // empty: a zero count
        *count_out = ws->d_offsets;
        CUDA_TRY(cudaMemsetAsync(ws->d_offsets, 0, sizeof(uint64_t), st));
        return CTD_OK;
    }
    uint32_t chunks = 0;
    const int rc = launch_sieve<uint64_t>(lo_odd, nodd, ws->d_base, ws->nbase,
                                          ws->nbase <= ws->starts_cap ? ws->d_starts : nullptr, ws->d_bits, ws->d_wcount,
                                          ws->d_offsets, ws->sm_count, d_out, capacity, 0, &chunks, st, err);
    *count_out = ws->d_offsets + chunks;
    return rc;
}

// ----------------------------------------------- fixed-scratch variant
// The same sieve, without the pass for the first multiples, over scratch the caller provides (no device
// allocation, no cached state): base primes are recomputed on every call
// into `sc.base`, whose unused tail is filled with 0xffffffff so the kernels'
// "p^2 beyond the window" test stops at the real list.
uint64_t sieve_scratch_windows(uint64_t lo, uint64_t hi)
{
    const uint64_t lo_odd = lo < 3 ? 3 : (lo | 1);
    if (lo_odd >= hi)
        return 0;
    const uint64_t nodd = (hi - lo_odd + 1) / 2;
    return (nodd + WIN_ODD - 1) / WIN_ODD;
}

uint64_t sieve_scratch_base_windows(uint64_t limit)
{
    return limit < LEVEL0_LIMIT ? 0 : (limit - LEVEL0_LIMIT) / (2 * WIN_ODD) + 1;
}

int sieve_range_scratch(const SieveScratch &sc, int sm_count, uint64_t lo, uint64_t hi, uint64_t *d_out,
                        uint64_t capacity, uint64_t *count, cudaStream_t st, std::string &err)
{
    *count = 0;
    if (hi <= lo)
        return CTD_OK;
    uint64_t out_base = 0;
    if (lo <= 2 && hi > 2) {
        if (capacity > 0) {  // the u64 value 2, little-endian
            CUDA_TRY(cudaMemsetAsync(d_out, 0, sizeof(uint64_t), st));
            CUDA_TRY(cudaMemsetAsync(d_out, 2, 1, st));
        }
        out_base = 1;
    }
    const uint64_t lo_odd = lo < 3 ? 3 : (lo | 1);
    if (lo_odd >= hi) {
        *count = out_base;
        return CTD_OK;
    }
    // base primes: level 0 (odd p < 2^16), then (2^16, sqrt(hi)] from them
    const uint64_t limit = isqrt64(hi - 1);
    CUDA_TRY(cudaMemsetAsync(sc.base, 0xff, sc.base_cap * sizeof(uint32_t), st));
    level0_primes<<<1, 1024, 0, st>>>(sc.base, sc.level0_count);
    CUDA_TRY(cudaGetLastError());
    note_kernel_launch();
    const uint32_t nlevel0 = 6541;  // odd primes below 2^16
    const uint64_t bwin = sieve_scratch_base_windows(limit);
    if (bwin) {
        const uint64_t b_lo = LEVEL0_LIMIT + 1;
        const uint64_t b_nodd = (limit - b_lo) / 2 + 1;
        uint32_t chunks = 0;
        const int rc = launch_sieve<uint32_t>(b_lo, b_nodd, sc.base, nlevel0, nullptr, sc.bits, sc.wcount, sc.offsets,
                                              sm_count, sc.base, sc.base_cap - 1, nlevel0, &chunks, st, err);
        if (rc)
            return rc;
    }
    // the range itself, against every base prime (the sentinel tail stops the scan)
    const uint64_t nodd = (hi - lo_odd + 1) / 2;
    uint32_t chunks = 0;
    const int rc = launch_sieve<uint64_t>(lo_odd, nodd, sc.base, (uint32_t)sc.base_cap, nullptr, sc.bits, sc.wcount,
                                          sc.offsets, sm_count, d_out, capacity, out_base, &chunks, st, err);
    if (rc)
        return rc;
    uint64_t total = 0;
    CUDA_TRY(cudaMemcpyAsync(&total, sc.offsets + chunks, sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    *count = out_base + total;
    return CTD_OK;
}

int sieve_range(SieveWorkspace *ws, uint64_t lo, uint64_t hi, uint64_t *d_out, uint64_t capacity, uint64_t *count,
                cudaStream_t st, std::string &err)
{
    *count = 0;
    if (hi <= lo)
        return CTD_OK;
    uint64_t total = 0;
    if (lo <= 2 && hi > 2) {
        if (capacity > 0) {
            const uint64_t two = 2;
            CUDA_TRY(cudaMemcpyAsync(d_out, &two, sizeof(two), cudaMemcpyHostToDevice, st));
            CUDA_TRY(cudaStreamSynchronize(st));
        }
        total = 1;
    }
    const uint64_t lo_odd = lo < 3 ? 3 : (lo | 1);
    if (lo_odd < hi) {
        const uint64_t nodd = (hi - lo_odd + 1) / 2;
        const uint64_t limit = isqrt64(hi - 1);
        int rc = ensure_base(ws, limit, st, err);
        if (rc)
            return rc;
        // base primes p with p <= limit: count them on the host side once
        // (the list is ascending; the kernels stop at p^2 >= window end)
        uint64_t cnt = 0;
        rc = sieve_odd<uint64_t>(ws, lo_odd, nodd, ws->d_base, ws->nbase, d_out, capacity, total, &cnt, st, err);
        if (rc)
            return rc;
        total += cnt;
    }
    *count = total;
    return CTD_OK;
}

}  // namespace ctd

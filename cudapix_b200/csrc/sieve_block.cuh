// sieve_block.cuh -- one CTA sieves 1024 odd numbers a thread in shared memory:
// the prime sieve of the pi tables and prime counts, and the sieve of phi(x, a).
//
// Replaces the reference's external CUDASieve (call sites e.g. src/P2.cu:100,103)
// and its phi sieve kernels (src/phi.cu:14-109).
//
// Three ways of crossing off, by the size of p:
//   3 .. 61      six bit patterns, each of a few primes and as long as their
//                product, in shared memory; a word of the bitmap is six
//                two-word reads and shifts
//   67 .. 2053   a warp per prime, a lane per multiple, by atomicAnd
//   above        a thread per prime, by atomicAnd
// (phi(1e10, 100): 1.52 ms with each warp crossing its own 2^15 bits by plain
// read-modify-write, 1.11 so; primes of 1e10 numbers at 1e12: 5.07 ms when a
// thread first looked whether the bit is still set, 3.88 so.)
// From 67 on the multiples of 3 are left out (the patterns cleared them): the
// steps alternate between p and 2p bits.
#pragma once
#include <mutex>

#include "kern_common.cuh"

namespace cpx {

constexpr uint32_t kPatGroups = 6;
constexpr uint32_t kPatFirst = 18;   // P[18] = 67, the first prime after the patterns
constexpr uint32_t kPatMedium = 310;  // P[310] = 2063, the first prime a thread takes alone
static __constant__ uint32_t c_pat_p[kPatGroups][5] = {{3, 5, 7, 11, 13}, {17, 19, 23, 0, 0}, {29, 31, 37, 0, 0},
                                                      {41, 43, 0, 0, 0},  {47, 53, 0, 0, 0},  {59, 61, 0, 0, 0}};
__host__ __device__ constexpr uint32_t pat_period(uint32_t g)
{
    return g == 0 ? 15015u : g == 1 ? 7429u : g == 2 ? 33263u : g == 3 ? 1763u : g == 4 ? 2491u : 3599u;
}
// words of a pattern (two past its last bit's word can be read), and where they start
__host__ __device__ constexpr uint32_t pat_words(uint32_t g) { return ((pat_period(g) - 1) >> 5) + 2; }
__host__ __device__ constexpr uint32_t pat_off(uint32_t g)
{
    return g == 0 ? 0u : g == 1 ? 471u : g == 2 ? 705u : g == 3 ? 1746u : g == 4 ? 1803u : g == 5 ? 1882u : 1996u;
}
static_assert(pat_off(1) == pat_words(0) && pat_off(2) == pat_off(1) + pat_words(1) &&
                  pat_off(3) == pat_off(2) + pat_words(2) && pat_off(4) == pat_off(3) + pat_words(3) &&
                  pat_off(5) == pat_off(4) + pat_words(4) && pat_off(6) == pat_off(5) + pat_words(5),
              "pattern offsets");
constexpr uint32_t kPatWords = pat_off(kPatGroups);

// dynamic shared memory of a CTA of NT threads: the bitmap, then the patterns
__host__ __device__ constexpr size_t sieve_block_smem(uint32_t nt) { return (size_t(nt) * 32 + kPatWords) * 4; }

// raises a kernel's dynamic shared-memory limit (a property of the function,
// shared by every context and thread of the process; once per device)
template <auto Kernel> static void raise_smem(cpx_ctx *ctx, size_t bytes)
{
    static std::mutex m;
    static int done_dev = -1;
    std::lock_guard<std::mutex> g(m);
    if (done_dev == ctx->device) return;
    CPX_CUDA(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done_dev = ctx->device;
}

// The first multiple p k of p above lo with k odd and prime to 3 (k >= p for the
// prime sieve): its bit (0xFFFFFFFF: none below nbits) and the step to the
// next one, 2p for k = 1 mod 6 and p for k = 5 mod 6.  lod = lo as a double.
template <bool PRIME>
__device__ __forceinline__ uint32_t first_multiple(uint64_t lo, double lod, uint32_t p, uint32_t nbits, uint64_t &step)
{
    // floor(lo / p): lo < 2^53 is exact in double, and the product with the once
    // refined reciprocal is within 1 of the quotient (below 2^44, as p >= 67
    // leaves lo / p < 2^47: the remainder then steps at most a few times)
    uint64_t q;
    if (lo >> 53) {
        q = cpx_udiv_leaf(lo, p);
    } else {
        const double r = (double)__frcp_rn(__uint2float_rn(p));
        const double rd = __fma_rn(r, __fma_rn(-(double)p, r, 1.0), r);
        q = __double2ull_rz(__dmul_rn(lod, rd));
        int64_t rem = (int64_t)(lo - q * p);
        while (rem < 0) {
            q--;
            rem += p;
        }
        while (rem >= (int64_t)p) {
            q++;
            rem -= p;
        }
    }
    uint64_t k = (q + 1) | 1;  // the first odd k > lo / p
    if (PRIME && k < p) k = p;
    uint32_t k3 = (uint32_t)(k >> 32) % 3u + (uint32_t)k % 3u;  // 2^32 = 1 mod 3
    k3 = k3 >= 3 ? k3 - 3 : k3;
    if (k3 == 0) {
        k += 2;
        k3 = 2;
    }
    step = k3 == 1 ? 2ull * p : (uint64_t)p;
    const uint64_t i = (k * p - lo - 1) >> 1;
    return i < nbits ? (uint32_t)i : 0xFFFFFFFFu;
}

// Sieves the odd numbers lo + 2i + 1, i < 1024 NT (lo even), into bm (bit i set:
// not crossed off), with patterns in pat; NT threads call it.  PRIME: bit set iff
// the number is prime (P must reach the square root of the block's end or of
// the last number that counts).  Else: bit set iff no P[1] .. P[np - 1] divides it.
template <bool PRIME, uint32_t NT>
__device__ __forceinline__ void sieve_block(uint32_t *bm, uint32_t *pat, uint64_t lo, const uint32_t *__restrict__ P,
                                            uint32_t np)
{
    constexpr uint32_t NBITS = NT * 1024;
    __shared__ uint32_t s_o[kPatGroups];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t hi = lo + 2ull * NBITS < lo ? ~0ull : lo + 2ull * NBITS;
    const uint32_t plim = np ? P[np - 1] : 0;
    // the patterns: bit t of group g, set iff one of its primes divides 2t + 1
    for (uint32_t t = tid; t < kPatWords; t += NT) {
        uint32_t g = 0;
#pragma unroll
        for (uint32_t h = 1; h < kPatGroups; h++) g += t >= pat_off(h);
        const uint32_t w = t - pat_off(g);
        uint32_t m = 0;
        for (uint32_t j = 0; j < 5; j++) {
            const uint32_t p = c_pat_p[g][j];
            if (!p || p > plim) continue;
            const uint32_t r = (64u * w + 1) % p;
            for (uint32_t k = r == 0 ? 0u : ((r & 1u) ? (p - r) >> 1 : p - (r >> 1)); k < 32; k += p) m |= 1u << k;
        }
        pat[t] = m;
    }
    if (tid < kPatGroups) s_o[tid] = (uint32_t)((lo >> 1) % pat_period(tid));
    __syncthreads();
    // ---- 3 .. 61: this warp's words, one a lane
    uint32_t *bw = bm + warp * 1024;
    {
        uint32_t o[kPatGroups];
#pragma unroll
        for (uint32_t g = 0; g < kPatGroups; g++) o[g] = (s_o[g] + (32u * (warp * 1024 + lane)) % pat_period(g)) % pat_period(g);
        for (uint32_t w = lane; w < 1024; w += 32) {
            uint32_t m = 0;
#pragma unroll
            for (uint32_t g = 0; g < kPatGroups; g++) {
                const uint32_t *pg = pat + pat_off(g) + (o[g] >> 5);
                m |= __funnelshift_r(pg[0], pg[1], o[g] & 31);
                o[g] += 1024u % pat_period(g);
                if (o[g] >= pat_period(g)) o[g] -= pat_period(g);
            }
            bw[w] = ~m;
        }
    }
    __syncwarp();
    __syncthreads();
    // ---- 67 .. 2053: a warp per prime over the whole bitmap, a lane per
    // multiple; 32 primes' starts at a time
    const double lod = (double)lo;
    constexpr uint32_t NWRP = NT / 32;
    const uint32_t nmed = min(np, kPatMedium);
    for (uint32_t k0 = kPatFirst + warp; k0 < nmed; k0 += 32 * NWRP) {
        uint32_t lp = 0, li = 0xFFFFFFFFu;
        uint64_t ls = 0;
        if (k0 + lane * NWRP < nmed) {
            lp = P[k0 + lane * NWRP];
            li = first_multiple<PRIME>(lo, lod, lp, NBITS, ls);
        }
        for (uint32_t j = 0; j < 32 && k0 + j * NWRP < nmed; j++) {
            const uint32_t p = __shfl_sync(FULL, lp, j), i0 = __shfl_sync(FULL, li, j);
            const uint32_t st = __shfl_sync(FULL, (uint32_t)ls, j);
            if (i0 == 0xFFFFFFFFu) continue;
#pragma unroll 4
            for (uint32_t i = i0 + (lane >> 1) * 3 * p + (lane & 1) * st; i < NBITS; i += 48 * p)
                atomicAnd(&bm[i >> 5], ~(1u << (i & 31)));
        }
    }
    // ---- above: a thread per prime
    const bool small = (lo >> 53) == 0;
    for (uint32_t k = kPatMedium + tid; k < np; k += NT) {
        const uint32_t p = P[k];
        if (PRIME ? (uint64_t)p * p >= hi : (uint64_t)p >= hi) break;
        if (small && p > NBITS / 2 && p < (1u << 30)) {
            // two multiples at most: lo mod p by the refined reciprocal (lo / p <
            // 2^43, so the truncated product is within 1 of the quotient)
            const float r0 = cpx_rcp_approx(p);
            const double rd = __fma_rn((double)r0, __fma_rn(-(double)p, (double)r0, 1.0), (double)r0);
            uint64_t q = (uint64_t)__double_as_longlong(__dadd_rz(__dmul_rn(lod, rd), 0x1p52)) & 0xFFFFFFFFFFFFFull;
            int64_t r = (int64_t)(lo - q * p);
            if (r < 0) {
                r += p;
                q--;
            } else if (r >= (int64_t)p) {
                r -= p;
                q++;
            }
            // the first odd multiple is lo + d, d = p - r when q + 1 is odd
            uint32_t d = p - (uint32_t)r + ((q & 1) ? p : 0u);
            if (PRIME && q + 1 < p) {
                const uint64_t d2 = (uint64_t)p * p - lo;
                d = d2 < 2 * NBITS ? (uint32_t)d2 : 2 * NBITS + 1;
            }
            for (uint32_t i = (d - 1) >> 1; i < NBITS; i += p) atomicAnd(&bm[i >> 5], ~(1u << (i & 31)));
            continue;
        }
        uint64_t st;
        const uint32_t i0 = first_multiple<PRIME>(lo, lod, p, NBITS, st);
        if (i0 == 0xFFFFFFFFu) continue;
        if (p < (1u << 29)) {  // i + 2p stays below 2^32
            uint32_t s32 = (uint32_t)st;
            const uint32_t p3 = 3 * p;
            for (uint32_t i = i0; i < NBITS; i += s32, s32 = p3 - s32) atomicAnd(&bm[i >> 5], ~(1u << (i & 31)));
        } else {
            atomicAnd(&bm[i0 >> 5], ~(1u << (i0 & 31)));  // p > NBITS: one at most
        }
    }
    __syncthreads();
    if (PRIME && lo == 0) {
        // 1 is not prime, and the patterns removed 3 .. 61 themselves
        if (tid == 0) bm[0] = 0x64B4CB6Eu;
        __syncthreads();
    }
}

}  // namespace cpx

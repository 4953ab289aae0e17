// levels.cuh -- blocks of consecutive levels crossed off at once (the sieve of
// lone queries, hard.cu).
#pragma once
#include "sieve.cuh"

namespace cpx {

// cleared bits a warp notes before it answers the leaves up to them
constexpr uint32_t kEvCap = 192;

// one level's outputs of one warp's sub-segment
struct LvlSum {
    uint32_t cnt;
    int32_t ms;
};

// leaves a warp gathers before answering them 32 at a time
constexpr uint32_t kLeafCap = 128;

// bytes of a warp's cleared bits, or of the 16-bit prefixes of its chunks
__host__ __device__ __forceinline__ size_t ev_bytes(uint32_t lbits, uint32_t threads)
{
    const size_t chunks = ((size_t(1) << lbits) / 128) / (threads / 32);
    return chunks * 2 > kEvCap * 4 ? chunks * 2 : kEvCap * 4;
}

// shared memory of k_hard
__host__ __device__ __forceinline__ size_t levels_smem(uint32_t lbits, uint32_t threads)
{
    const size_t L = size_t(1) << lbits;
    size_t o = L / 8;                               // bitmap
    o += ((L / 128) + 15) & ~size_t(15);            // chunk counters
    o += threads * 4;                               // lane prefixes
    o += 2 * (threads / 32) * 32 * sizeof(LvlSum);  // per-warp level outputs, double buffered
    o = (o + 15) & ~size_t(15);
    o += 32 * sizeof(i128);                         // reductions
    o += (threads / 32) * kLeafCap * sizeof(uint2);  // per-warp gathered leaves
    o += (threads / 32) * ev_bytes(lbits, threads);  // per-warp cleared bits or chunk prefixes
    return o;
}

// Crosses several consecutive levels off one warp's sub-segment at once: lane
// k holds level gb + k, its prime p and the bit i of its next multiple
// (0xFFFFFFFF: none).  The bits go by in windows of W = the smallest of the
// primes, so a lane has at most one multiple in a window and every multiple of
// one number falls into the same window: a number that several of the primes
// divide is found by its lanes in the same step, and the lowest level takes it,
// as when the levels are crossed off one after another.  The lanes first read
// their bits; those that find theirs set clear it by an atomic and see whether
// they were the first.  A lane that saw its bit set but did not clear it shares
// its number with another (about one step in a hundred), and the lanes of that
// number then find their lowest by a vote.
// Stops before window [w_end - W, w_end) when fewer than 32 of the cap event
// slots are left; ev[0..nev): the cleared bits, level k << 20 | bit (cap 0: none
// noted).  cleared counts the bits this lane's level took.  Returns nev.
// (Bit i lies in word i >> 5 of the sub-segment; the lane that owns its chunk,
// i >> (7 + s), swizzles bits 2..4 of the word's index.)
constexpr uint32_t kEvBit = 20;                      // a sub-segment has at most 2^18 bits
constexpr uint32_t kEvMask = (1u << kEvBit) - 1;
__device__ __forceinline__ uint32_t cross_levels(uint32_t *bm, uint8_t *cnt8, uint32_t p, uint32_t &i, uint32_t W,
                                                 uint32_t &w_end, uint32_t &cleared, int s, uint32_t base_ch,
                                                 uint32_t lane, uint32_t Lw, uint32_t *ev, uint32_t cap)
{
    uint32_t nev = 0;
    uint32_t *bw = bm + (base_ch << 2), *cw = reinterpret_cast<uint32_t *>(cnt8 + base_ch);
    const uint32_t swm = s ? 0x1Cu : 0u, below = (1u << lane) - 1u;
    for (; w_end - W < Lw; w_end += W) {
        if (cap && nev + 32 > cap) break;
        const bool hit = i < min(w_end, Lw);
        const uint32_t bit = 1u << (i & 31);
        uint32_t *pw = bw + ((i >> 5) ^ ((i >> (5 + s)) & swm));
        const bool alive = hit && (*pw & bit) != 0;
        const unsigned seen = __ballot_sync(FULL, alive);
        if (seen) {
            bool won = false;
            if (alive) {
                won = (atomicAnd(pw, ~bit) & bit) != 0;
                // the chunk's counter, a byte of its word (at least one, so nothing is borrowed)
                if (won) atomicSub(cw + (i >> 9), 1u << ((i >> 4) & 24));
            }
            unsigned took = __ballot_sync(FULL, won);
            if (took != seen) {
                for (unsigned lost = seen & ~took; lost; lost &= lost - 1) {
                    const uint32_t n = __shfl_sync(FULL, i, __ffs(lost) - 1);
                    const unsigned same = __ballot_sync(FULL, alive && i == n);
                    if (alive && i == n) won = (uint32_t)__ffs(same) - 1 == lane;
                }
                took = __ballot_sync(FULL, won);
            }
            if (won) {
                cleared++;
                if (cap) ev[nev + __popc(took & below)] = lane << kEvBit | i;
            }
            nev += __popc(took);
        }
        if (hit) i += p;
    }
    __syncwarp();
    return nev;
}

// One item of the candidates of a level that takes any squarefree m with lpf(m)
// > p: eight odd m of the packed mu*lpf table, indices 8o .. 8o + 7, of which
// [i_lo, i_hi] count (indices below 2^30).  Bit k: m = 16o + 2k + 1 is a leaf.
struct Octet {
    int32_t v[8];
    uint32_t valid;
};
__device__ __forceinline__ Octet load_octet(const int32_t *__restrict__ MU, uint32_t o, uint32_t i_lo, uint32_t i_hi,
                                            uint32_t p, bool on)
{
    Octet t;
    t.valid = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) t.v[k] = 0;
    if (on) {
        const int4 *m4 = reinterpret_cast<const int4 *>(MU) + 2 * (size_t)o;
        const int4 a = __ldg(m4), b = __ldg(m4 + 1);
        t.v[0] = a.x, t.v[1] = a.y, t.v[2] = a.z, t.v[3] = a.w;
        t.v[4] = b.x, t.v[5] = b.y, t.v[6] = b.z, t.v[7] = b.w;
#pragma unroll
        for (int k = 0; k < 8; k++) t.valid |= (uint32_t)abs(t.v[k]) > p ? 1u << k : 0u;
        const uint32_t i0 = 8 * o;
        if (i0 < i_lo) t.valid &= 0xFFu << (i_lo - i0);
        if (i0 + 7 > i_hi) t.valid &= 0xFFu >> (i0 + 7 - i_hi);
    }
    return t;
}
// puts the octet's leaves among `now` (bits of valid) at buf[at..]: m | (mu(m) = -1) << 31, level
__device__ __forceinline__ void put_octet(const Octet &t, uint32_t o, uint32_t now, uint32_t key, uint2 *buf, uint32_t at)
{
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if ((now >> k) & 1u) {
            buf[at] = make_uint2((16 * o + 2 * k + 1) | ((uint32_t)t.v[k] & 0x80000000u), key);
            at++;
        }
    }
}

// the last lane j with ex[j] <= f: the owner of flat item f, ex the exclusive
// prefix of the lanes' item counts
__device__ __forceinline__ uint32_t item_owner(uint32_t ex, uint32_t f)
{
    uint32_t j = 0;
#pragma unroll
    for (uint32_t st = 16; st; st >>= 1) {
        const uint32_t c = j + st;
        if (__shfl_sync(FULL, ex, c) <= f) j = c;
    }
    return j;
}

}  // namespace cpx

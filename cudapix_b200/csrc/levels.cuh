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
// slots are left; ev[0..nev): the cleared bits, level k << 20 | bit (REC).
// cleared counts the bits this lane's level took.  Returns nev.
constexpr uint32_t kEvBit = 20;                      // a sub-segment has at most 2^18 bits
constexpr uint32_t kEvMask = (1u << kEvBit) - 1;
template <bool REC>
__device__ __forceinline__ uint32_t cross_levels(uint32_t *bm, uint8_t *cnt8, uint32_t p, uint32_t &i, uint32_t W,
                                                 uint32_t &w_end, uint32_t &cleared, int s, uint32_t base_ch,
                                                 uint32_t lane, uint32_t Lw, uint32_t *ev, uint32_t cap)
{
    uint32_t nev = 0;
    uint32_t *cw = reinterpret_cast<uint32_t *>(cnt8);
    for (; w_end - W < Lw; w_end += W) {
        if (REC && nev + 32 > cap) break;
        const bool hit = i < min(w_end, Lw);
        uint32_t ch = 0, bit = 0;
        uint32_t *pw = bm;
        bool alive = false;
        if (hit) {
            const uint32_t w = i >> 5;
            ch = base_ch + (w >> 2);
            pw = bm + ((swz(ch, s) << 2) | (w & 3));
            bit = 1u << (i & 31);
            alive = (*pw & bit) != 0;
        }
        const unsigned seen = __ballot_sync(FULL, alive);
        if (seen) {
            bool won = false;
            if (alive) {
                won = (atomicAnd(pw, ~bit) & bit) != 0;
                // the chunk's counter, a byte of its word (at least one, so nothing is borrowed)
                if (won) atomicSub(cw + (ch >> 2), 1u << (8 * (ch & 3)));
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
                if (REC) ev[nev + __popc(took & ((1u << lane) - 1u))] = lane << kEvBit | i;
            }
            if (REC) nev += __popc(took);
        }
        if (hit) i += p;
    }
    __syncwarp();
    return nev;
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

// hard.cu -- hard special leaves: the segmented phi sieve.
//
// Restates the reference's hard-leaf sieve (S2hardHost / S2ctl,
// src/sieve/S2_hard_host.cu:49-191, src/sieve/S2_hard_device.cu:12-382) with
// this library's exact leaf split: a leaf (b, m) is hard when
// u = x/(p_b m) >= p_b^2, i.e. p_b <= iroot4(x) and m <= x/p_b^3; it
// contributes -mu(m) phi(u, b-1), which the sieve answers from the bitmap of
// the segment holding u plus the survivors of level b-1 below it.
//
// One CTA owns one unit: a segment of 2^lbits odd numbers n = lo + 2i + 1 and
// all of its leaves, or every nparts-th 32 table entries of their candidates
// where the segment holds more leaves than the rest of its work (the early
// segments: their number falls as 1/u^2; dense_units in driver.cu).  Each warp owns a contiguous
// sub-segment as a bitmap in shared memory with one 8-bit survivor counter per
// 16-byte chunk (128 numbers), and walks the levels b = c+1 .. B(seg) on its
// own, synchronising only inside the warp, 32 levels (a block) at a time: one
// level per lane loads x/p, y/p and min(y, x/p^3) from a table filled once per
// query and computes its candidate range and first multiple.
//
// A block goes through at once when its primes have few multiples in the
// sub-segment and its leaves are not many: cross_levels takes one multiple of
// each level a step, the block's candidates are walked as one sequence, and
// each leaf is counted on the bitmap after the whole block plus the bits up to
// u that its own and higher levels cleared, which cross_levels notes down.
// Else the levels go one by one: the warp (1) records its survivor count at
// level b-1, (2) scans the counters into lane prefixes and answers each leaf
// as lane prefix + earlier counters of the owning lane + popcounts in the
// chunk, (3) crosses off p_b, counting cleared bits and keeping the counters
// current.  After each block the CTA combines its warps: carries between
// sub-segments enter the hard sum and the per-unit (count, Sum(-mu)) pairs go
// to k_hard_combine, which adds the carries between segments.
//
// Integer issue and the latency of a warp's chain of levels bound the kernel
// (73% of the issue slots at pi(1e15)), not memory.  Hard leaves on a B200, ms:
// one level at a time with the heavy leaf sets in a kernel of their own; blocks
// at once; units split by their leaves, and leaves found for a run of levels
// before they are needed; octets, and the segment sizes of the tuning table:
//   pi(1e12)    0.300   0.202   0.205   0.123
//   pi(1e15)    3.05    2.43    1.93    1.58
//   pi(1e17)    36.3    30.2    22.3    16.0
//   pi(1.9e19)  1370    950     628     540
//
// This is the sieve of lone queries and small batches.  Larger batches share
// the sieve between queries (hard_shared.cu).
#include <algorithm>
#include <mutex>

#include "levels.cuh"

namespace cpx {

// The unit `u` of a query's units (relative to its first): its segment
// (relative to seg0), which part of the segment's leaves it takes, of how many.
struct UnitSeg {
    uint64_t seg;
    uint32_t part, nparts;
};
__device__ __forceinline__ UnitSeg unit_seg(const QD &d, const uint32_t *__restrict__ dense, uint64_t u)
{
    const uint32_t K = d.dense_segs;
    if (!K) return {u, 0u, 1u};
    const uint32_t *base = dense + d.dense_off;
    const uint32_t nu = __ldg(base + K);
    if (u >= nu) return {K + (u - nu), 0u, 1u};
    uint32_t lo = 0, hi = K;  // base[lo] <= u < base[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(base + mid) <= u) lo = mid;
        else hi = mid;
    }
    const uint32_t b0 = __ldg(base + lo);
    return {lo, (uint32_t)u - b0, __ldg(base + lo + 1) - b0};
}
// the first unit of a query's segment `seg` (relative to seg0)
__device__ __forceinline__ uint64_t seg_unit(const QD &d, const uint32_t *__restrict__ dense, uint64_t seg)
{
    const uint32_t K = d.dense_segs;
    if (!K) return seg;
    const uint32_t *base = dense + d.dense_off;
    return seg < K ? __ldg(base + seg) : __ldg(base + K) + (seg - K);
}

template <class XT> __device__ __forceinline__ XT shfl_xt(XT v, uint32_t src)
{
    if (sizeof(XT) == 8) return (XT)__shfl_sync(FULL, (unsigned long long)v, src);
    const unsigned long long a0 = __shfl_sync(FULL, (unsigned long long)v, src);
    const unsigned long long a1 = __shfl_sync(FULL, (unsigned long long)((u128)v >> 64), src);
    return (XT)(((u128)a1 << 64) | a0);
}

// A block of levels goes through at once when its smallest prime has at most
// kLevelWindows multiples in a warp's sub-segment, and when its leaves times
// the bits it clears (each leaf is compared with all of them) stay below
// kLevelLeafEvents a level: one by one, a level costs about 250 issue slots
// whatever its leaves, which 2048 comparisons of a warp's lanes take too.
constexpr uint32_t kLevelWindows = 64;
constexpr uint32_t kLevelLeafEvents = 2048;

template <class XT>
__global__ void __launch_bounds__(512, 2) k_hard(const QD *__restrict__ qd, uint32_t Q,
                                              const uint64_t *__restrict__ pre_seg, uint64_t total,
                                              const uint32_t *__restrict__ seg_B,
                                              const uint64_t *__restrict__ seg_off,
                                              const uint32_t *__restrict__ P, const int32_t *__restrict__ MU,
                                              const cpx_pient *__restrict__ Tpi,
                                              const uint64_t *__restrict__ pre_comb, const XT *__restrict__ lvx,
                                              const uint2 *__restrict__ lae, const uint32_t *__restrict__ dense,
                                              uint32_t *__restrict__ out_cnt, int32_t *__restrict__ out_ms,
                                              uint64_t cap, unsigned long long *__restrict__ acc,
                                              uint32_t lbits_max)
{
    extern __shared__ uint4 smem4[];
    const uint64_t unit = blockIdx.x;
    if (unit >= total) return;
    const uint32_t B = seg_B[unit];
    const uint32_t q = find_q(pre_seg, Q, unit);
    const QD &d = qd[q];
    const uint32_t c = d.c;
    if (B <= c) return;  // uniform over the CTA
    const uint32_t T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, NW = T >> 5;
    const uint32_t L = 1u << d.lbits;
    const uint32_t NC = L >> 7;    // chunks of the segment
    const uint32_t CPT = NC / T;   // chunks per lane (>= 1)
    const int s = __ffs(CPT) - 1;  // log2 CPT
    const uint32_t Lw = L / NW;    // bits of a warp's sub-segment
    const UnitSeg us = unit_seg(d, dense, unit - pre_seg[q]);
    const uint64_t lo = (us.seg + d.seg0) * 2 * (uint64_t)L;
    const uint64_t lo_w = lo + 2 * (uint64_t)Lw * warp, hi_w = lo_w + 2 * (uint64_t)Lw;
    const bool q41 = hi_w <= (1ull << 41);  // leaf quotients lie in [lo_w, hi_w)
    const uint64_t off = seg_off[unit];
    if (off + (B - c) > cap) return;  // the host sized the ragged outputs exactly; never write past them
    const uint64_t y = d.y;
    const uint64_t lv0 = pre_comb[q];  // the query's rows of the level table
    const uint32_t step = 32 * us.nparts, first = 32 * us.part;  // this unit's candidate entries

    // carve the shared block (sized for lbits_max)
    unsigned char *sp = reinterpret_cast<unsigned char *>(smem4);
    const size_t Lmax = size_t(1) << lbits_max;
    uint32_t *bm = reinterpret_cast<uint32_t *>(sp);
    size_t o = Lmax / 8;
    uint8_t *cnt8 = reinterpret_cast<uint8_t *>(sp + o);
    o += ((Lmax / 128) + 15) & ~size_t(15);
    uint32_t *loff = reinterpret_cast<uint32_t *>(sp + o);  // [NW][32] lane prefixes
    o += T * 4;
    LvlSum *area = reinterpret_cast<LvlSum *>(sp + o);      // [2][NW][32]
    o += 2 * NW * 32 * sizeof(LvlSum);
    o = (o + 15) & ~size_t(15);
    i128 *s_red = reinterpret_cast<i128 *>(sp + o);
    o += 32 * sizeof(i128);
    uint2 *lbuf = reinterpret_cast<uint2 *>(sp + o) + kLeafCap * warp;        // this warp's gathered leaves
    o += NW * kLeafCap * sizeof(uint2);
    // this warp's cleared bits (levels at once) or the prefixes of its chunks
    // within their lanes (levels one by one)
    uint32_t *ev = reinterpret_cast<uint32_t *>(sp + o + ev_bytes(d.lbits, T) * warp);
    uint16_t *pre16 = reinterpret_cast<uint16_t *>(ev) - CPT * 32 * warp;  // by the segment's chunk
    uint32_t *wl = loff + 32 * warp;  // this warp's lane prefixes

    const uint32_t c0 = CPT * tid;  // first owned chunk (of the segment)
    const uint32_t cw0 = c0 - CPT * 32 * warp;  // first owned chunk of the sub-segment
    // ---- pre-sieve with p_2 .. p_c; chunk counters
    const uint32_t cnt0 = presieve(bm, cnt8, c, lo, c0, CPT, s);
    uint32_t tot = __reduce_add_sync(FULL, cnt0);  // survivors of this warp's sub-segment
    __syncwarp();

    const Recip r_lo{lo_w, lo_w ? 1.0 / (double)lo_w : 0.0}, r_hi{hi_w, 1.0 / (double)hi_w};

    int64_t S = 0;       // this lane's share of the hard sum (survivor counts within sub-segments)
    i128 Sx = 0;         // warp 0: carries between the CTA's sub-segments
    uint32_t grp = 0;
    for (uint32_t gb = c + 1; gb <= B; gb += 32, grp++) {
        const uint32_t nl = min(32u, B - gb + 1);
        // ---- level parameters, one level per lane: p, x/p, the candidates
        // (mlo, mhi] with u = xp/m in the sub-segment, the first multiple
        uint32_t lp = 0, lmlo = 0, lmhi = 0, lr0 = 0, li0 = 0xFFFFFFFFu;
        XT lxp = 0;
        if (lane < nl) {
            const uint64_t li = lv0 + (gb - c - 1) + lane;
            lp = P[gb + lane - 1];
            lxp = lvx[li];
            const uint2 ae = lae[li];
            uint64_t a = ae.x, e = ae.y;
            const XT t1 = div_recip(lxp, r_hi);
            if (t1 > (XT)a) a = (uint64_t)t1;
            if (lo_w) {
                const XT t2 = div_recip(lxp, r_lo);
                if (t2 < (XT)e) e = (uint64_t)t2;
            }
            lmlo = (uint32_t)a;
            lmhi = (uint32_t)(e > a ? e : a);
            cross_params(lp, lo_w, hi_w, lr0, li0);
        }
        // Items of each level's candidates: the primes P[k] of a prime-only level
        // (m = q > max(mlo, p)), each a leaf, or the octets of packed mu*lpf.
        // p^2 > y from some level on, so the octet levels of a block come first.
        const bool prime_j = (uint64_t)lp * lp > y;
        const uint32_t qa_j = lmlo > lp ? lmlo : lp;
        uint32_t nw_j = 0, ng_j = 0, k0_j = 0, lf_j = 0;  // lf_j: its leaves at most
        if (lmhi > lmlo) {
            if (!prime_j) {
                ng_j = ((lmhi - 1) >> 4) - ((lmlo + 1) >> 4) + 1;
                lf_j = ((lmhi - 1) >> 1) - ((lmlo + 1) >> 1) + 1;
            } else if (lmhi > qa_j) {
                k0_j = (uint32_t)cpx_pi_ge2(Tpi, qa_j);
                nw_j = lf_j = (uint32_t)cpx_pi_ge2(Tpi, lmhi) - k0_j;
            }
        }
        LvlSum *ar = area + (grp & 1) * NW * 32;
        ar[warp * 32 + lane].ms = 0;
        lf_j = min(lf_j, 1u << 20);
        // about one bit in seven of a level's multiples is still set
        const uint32_t pmin = __shfl_sync(FULL, lp, 0);
        bool at_once = (uint64_t)pmin * kLevelWindows >= Lw;
        if (at_once) {
            const uint32_t est = __reduce_add_sync(FULL, min(nw_j + 2 * ng_j, 1u << 26)) / us.nparts;
            at_once = (uint64_t)est * (nl * (Lw / pmin + 1) / 7 + 4) <= (uint64_t)nl * kLevelLeafEvents;
        }
        uint32_t mine_cnt = 0;
        // item offsets of the levels (32 bits: a level of 2^26 items or more only goes alone)
        uint32_t ex_w, ex_g;
        const uint32_t tot_w = warp_place(min(nw_j, 1u << 26), lane, ex_w),
                       tot_g = warp_place(min(ng_j, 1u << 26), lane, ex_g);

        // item f of the block's primes: its level (the lane holding it) and prime
        auto prime_item = [&](uint32_t f, uint32_t end, uint32_t &jq) -> uint32_t {
            jq = item_owner(ex_w, f);
            const uint32_t k = __shfl_sync(FULL, k0_j - ex_w, jq) + f;
            return f < end ? __ldg(P + k) : 1u;
        };
        // item f of the block's octets: its level and which octet
        auto octet_item = [&](uint32_t f, uint32_t end, uint32_t &jq, uint32_t &o) -> Octet {
            jq = item_owner(ex_g, f);
            const uint32_t exq = __shfl_sync(FULL, ex_g, jq), pq = __shfl_sync(FULL, lp, jq);
            const uint32_t i_lo = (__shfl_sync(FULL, lmlo, jq) + 1) >> 1, i_hi = (__shfl_sync(FULL, lmhi, jq) - 1) >> 1;
            o = (i_lo >> 3) + (f - exq);
            return load_octet(MU, o, i_lo, i_hi, pq, f < end);
        };
        // Gathers the leaves of the octets item(from + lane), item(from + st + lane), ..
        // below end into the warp's buffer, which flush empties when it cannot hold
        // a round's more, and once at the end.
        uint32_t nbuf = 0;
        auto gather = [&](uint32_t from, uint32_t end, uint32_t st, auto &&item, auto &&flush) {
            for (uint32_t base = from;; base += st) {
                const bool last = base >= end;
                uint32_t jq = 0, o = 0;
                const Octet t = item(last ? end : base + lane, jq, o);
                uint32_t now = t.valid, rest = 0, tot_r = __reduce_add_sync(FULL, (uint32_t)__popc(now));
                if (tot_r > kLeafCap) {  // a dense round goes in two halves of the octets
                    rest = now & 0xF0u;
                    now &= 0xFu;
                    tot_r = __reduce_add_sync(FULL, (uint32_t)__popc(now));
                }
                for (;;) {
                    if (last || nbuf + tot_r > kLeafCap) flush();
                    if (last) return;
                    uint32_t off_l;
                    warp_place((uint32_t)__popc(now), lane, off_l);
                    put_octet(t, o, now, jq, lbuf, nbuf + off_l);
                    nbuf += tot_r;
                    if (!__any_sync(FULL, rest != 0)) break;
                    now = rest;
                    rest = 0;
                    tot_r = __reduce_add_sync(FULL, (uint32_t)__popc(now));
                }
            }
        };
        // bits [0, kk) of the sub-segment are the numbers up to u = xp / m
        auto leaf_bits = [&](XT xp, double xpd, uint32_t m) -> uint32_t {
            return ((uint32_t)leaf_quot(xp, xpd, m, q41) - (uint32_t)lo_w + 1u) >> 1;
        };

        if (at_once) {
            uint32_t i = li0, w_end = pmin, cleared = 0;
            if (!(tot_w | tot_g)) {
                cross_levels(bm, cnt8, lp, i, pmin, w_end, cleared, s, CPT * 32 * warp, lane, Lw, ev, 0);
            } else {
                // Slices of the sub-segment, as many as the bits cleared in it fill
                // the event buffer (nearly always one): a slice's leaves have k_lo <
                // kk <= k_hi.
                uint32_t k_lo = 0;
                for (;;) {
                    // bits of the earlier slices cleared by this lane's level and above
                    uint32_t suf = cleared;
#pragma unroll
                    for (int oo = 1; oo < 32; oo <<= 1) {
                        const uint32_t t = __shfl_down_sync(FULL, suf, oo);
                        if (lane + oo < 32) suf += t;
                    }
                    const uint32_t nev = cross_levels(bm, cnt8, lp, i, pmin, w_end, cleared, s, CPT * 32 * warp, lane, Lw,
                                                      ev, kEvCap);
                    const uint32_t k_hi = min(w_end - pmin, Lw);
                    if (lane < 4 && nev + lane < kEvCap) ev[nev + lane] = kEvMask;  // fills the last four
                    uint32_t off0;
                    warp_place(counter_sum(cnt8 + c0, CPT), lane, off0);
                    wl[lane] = off0;
                    __syncwarp();
                    // One leaf a lane: the survivors of level b - 1 up to u are those
                    // after the whole block and the bits up to u that levels b and
                    // above took.
                    auto answer = [&](bool on, uint32_t m, uint32_t key, bool plus) {
                        const XT xk = shfl_xt(lxp, key);
                        uint32_t cv = __shfl_sync(FULL, suf, key);
                        if (!on) return;
                        const uint32_t kk = leaf_bits(xk, (double)(uint64_t)xk, m);
                        if (kk > k_hi || (kk <= k_lo && k_lo)) return;
                        cv += sub_survivors_bits(kk, wl, cnt8, bm, CPT, s, warp);
                        const uint32_t kmin = key << kEvBit;
                        for (uint32_t t = 0; t < nev; t += 4) {
                            const uint4 v = *reinterpret_cast<const uint4 *>(ev + t);
                            cv += (v.x >= kmin && (v.x & kEvMask) < kk) + (v.y >= kmin && (v.y & kEvMask) < kk) +
                                  (v.z >= kmin && (v.z & kEvMask) < kk) + (v.w >= kmin && (v.w & kEvMask) < kk);
                        }
                        if (plus) S += cv;
                        else S -= cv;
                        atomicAdd(&ar[warp * 32 + key].ms, plus ? 1 : -1);
                    };
                    for (uint32_t base = first; base < tot_w; base += step) {
                        uint32_t jq;
                        const uint32_t m = prime_item(base + lane, tot_w, jq);
                        answer(base + lane < tot_w, m, jq, true);  // mu(q) = -1
                    }
                    if (tot_g) {
                        auto flush = [&] {
                            __syncwarp();
                            for (uint32_t j0 = 0; j0 < nbuf; j0 += 32) {
                                const bool on = j0 + lane < nbuf;
                                const uint2 e = on ? lbuf[j0 + lane] : make_uint2(1, 0);
                                answer(on, e.x & 0x7FFFFFFFu, e.y, (e.x >> 31) != 0);
                            }
                            __syncwarp();
                            nbuf = 0;
                        };
                        gather(first, tot_g, step, [&](uint32_t f, uint32_t &jq, uint32_t &o) { return octet_item(f, tot_g, jq, o); },
                               flush);
                    }
                    if (k_hi == Lw) break;
                    k_lo = k_hi;
                    __syncwarp();
                }
            }
            uint32_t before;
            const uint32_t all = warp_place(cleared, lane, before);
            mine_cnt = tot - before;
            tot -= all;
        } else {
            // Runs of levels [ka, kb) whose leaves fit the warp's buffer: all of
            // them are found first (level by level in order: kk | (mu(m) = -1) << 31
            // and the level), then each level answers its own.  A level with more
            // leaves, or one split over units, answers them as it finds them.
            uint32_t ex_l;
            warp_place(lf_j, lane, ex_l);
            uint32_t kb = 0;   // levels found
            uint32_t st = 0, en = 0;  // this lane's level: its leaves in the buffer
            bool dense = false;
            for (uint32_t k = 0; k < nl; k++) {
                if (k == kb) {
                    const uint32_t e0 = __shfl_sync(FULL, ex_l, k);
                    const unsigned fit = __ballot_sync(FULL, lane < k || ex_l + lf_j - e0 <= kLeafCap);
                    kb = min(fit == FULL ? 32u : (uint32_t)__ffs(~fit) - 1, nl);
                    dense = us.nparts > 1 || kb == k;
                    if (dense) {
                        kb = k + 1;
                    } else {
                        const uint32_t gs = __shfl_sync(FULL, ex_g, k), ws = __shfl_sync(FULL, ex_w, k);
                        const uint32_t ge = __shfl_sync(FULL, ex_g + ng_j, kb - 1),
                                       we = __shfl_sync(FULL, ex_w + nw_j, kb - 1);
                        nbuf = 0;
                        // (a run's leaves fit the buffer)
                        gather(gs, ge, 32, [&](uint32_t f, uint32_t &jq, uint32_t &o) { return octet_item(f, ge, jq, o); },
                               [] {});
                        __syncwarp();
                        for (uint32_t t0 = 0; t0 < nbuf; t0 += 32) {
                            const bool on = t0 + lane < nbuf;
                            const uint2 e = on ? lbuf[t0 + lane] : make_uint2(1, 0);
                            const XT xk = shfl_xt(lxp, e.y);
                            if (on)
                                lbuf[t0 + lane].x = leaf_bits(xk, (double)(uint64_t)xk, e.x & 0x7FFFFFFFu) | (e.x & 0x80000000u);
                        }
                        for (uint32_t base = ws; base < we; base += 32) {
                            uint32_t jq;
                            const uint32_t m = prime_item(base + lane, we, jq);
                            const XT xk = shfl_xt(lxp, jq);
                            if (base + lane < we)
                                lbuf[nbuf + base + lane - ws] =
                                    make_uint2(leaf_bits(xk, (double)(uint64_t)xk, m) | 0x80000000u, jq);
                        }
                        nbuf += we - ws;
                        __syncwarp();
                        // the first buffer entry of this lane's level, and of the next
                        st = 0;
                        for (uint32_t half = kLeafCap / 2; half; half >>= 1)
                            if (st + half <= nbuf && lbuf[st + half - 1].y < lane) st += half;
                        if (st < nbuf && lbuf[st].y < lane) st++;
                        en = __shfl_down_sync(FULL, st, 1);
                        if (lane == 31) en = nbuf;
                    }
                }
                const uint32_t p = __shfl_sync(FULL, lp, k);
                if (lane == k) mine_cnt = tot;
                const uint32_t nw = __shfl_sync(FULL, nw_j, k), ng = __shfl_sync(FULL, ng_j, k);
                const uint32_t lb = __shfl_sync(FULL, st, k), le = __shfl_sync(FULL, en, k);
                if (dense ? (nw > first || ng > first) : le > lb) {
                    // chunk and lane prefixes of the sub-segment from the chunk counters
                    uint32_t off0;
                    warp_place(chunk_prefixes(cnt8, pre16, c0, CPT), lane, off0);
                    wl[lane] = off0;
                    __syncwarp();
                    auto count = [&](uint32_t kk) -> uint32_t {
                        return sub_survivors_pre_bits(kk, wl, pre16, bm, CPT, s, warp);
                    };
                    int32_t msl = 0;
                    if (!dense) {
                        for (uint32_t t = lb + lane; t < le; t += 32) {
                            const uint32_t e = lbuf[t].x, cv = count(e & 0x7FFFFFFFu);
                            S += e >> 31 ? (int64_t)cv : -(int64_t)cv;
                            msl += e >> 31 ? 1 : -1;
                        }
                    } else {
                        const XT xp = shfl_xt(lxp, k);
                        const double xpd = (double)(uint64_t)xp;
                        // primes: two leaves a lane a step
                        const uint32_t *Pk = P + __shfl_sync(FULL, k0_j, k);
                        uint32_t f = first + lane;
                        for (; f + step < nw; f += 2 * step) {
                            const uint32_t m0 = __ldg(Pk + f), m1 = __ldg(Pk + f + step);
                            S += (int64_t)(count(leaf_bits(xp, xpd, m0)) + count(leaf_bits(xp, xpd, m1)));
                            msl += 2;
                        }
                        if (f < nw) {
                            S += (int64_t)count(leaf_bits(xp, xpd, __ldg(Pk + f)));
                            msl += 1;
                        }
                        if (ng > first) {
                            const uint32_t i_lo = (__shfl_sync(FULL, lmlo, k) + 1) >> 1,
                                           i_hi = (__shfl_sync(FULL, lmhi, k) - 1) >> 1;
                            nbuf = 0;
                            auto flush = [&] {
                                __syncwarp();
                                for (uint32_t t = lane; t < nbuf; t += 32) {
                                    const uint32_t e = lbuf[t].x, cv = count(leaf_bits(xp, xpd, e & 0x7FFFFFFFu));
                                    S += e >> 31 ? (int64_t)cv : -(int64_t)cv;
                                    msl += e >> 31 ? 1 : -1;
                                }
                                __syncwarp();
                                nbuf = 0;
                            };
                            gather(first, ng, step,
                                   [&](uint32_t f, uint32_t &, uint32_t &o) {
                                       o = (i_lo >> 3) + f;
                                       return load_octet(MU, o, i_lo, i_hi, p, f < ng);
                                   },
                                   flush);
                        }
                    }
                    const int32_t ms = __reduce_add_sync(FULL, msl);
                    if (lane == k) ar[warp * 32 + k].ms = ms;
                }
                // ---- cross off p_b in the sub-segment
                const uint32_t cleared = cross_off<true>(bm, cnt8, p, __shfl_sync(FULL, lr0, k),
                                                         __shfl_sync(FULL, li0, k), c0, cw0, CPT, s, CPT * 32 * warp,
                                                         lane, Lw);
                tot -= __reduce_add_sync(FULL, cleared);
                __syncwarp();
            }
        }
        // ---- combine the warps of the CTA for these 32 levels
        ar[warp * 32 + lane].cnt = mine_cnt;
        __syncthreads();
        if (warp == 0 && lane < nl) {
            const uint32_t b = gb + lane;
            uint64_t carry = 0;
            int32_t msum = 0;
            for (uint32_t w = 0; w < NW; w++) {
                const LvlSum e = ar[w * 32 + lane];
                Sx += (i128)carry * e.ms;
                carry += e.cnt;
                msum += e.ms;
            }
            // the survivors count once, with the segment's last unit
            out_cnt[off + (b - c - 1)] = us.part + 1 == us.nparts ? (uint32_t)carry : 0u;
            out_ms[off + (b - c - 1)] = msum;
        }
    }
    const i128 Sb = cpx_block_sum_i128((i128)S + Sx, s_red);
    if (tid == 0) acc_add(acc, q, ACC_HARD, Sb);
}

// Leaves of the sets the batch-shared sieve hands over.  A warp takes one unit: 256
// pi-table entries of prime m (prime-only levels) or 256 groups of 4 odd m
// read as packed mu*lpf (other levels).  Each leaf's survivor count is the
// job's carry plus the snapshot's chunk prefix plus popcounts inside the
// 16-byte chunk; the sums go to the query's hard-leaf accumulator.
template <class XT>
__global__ void __launch_bounds__(kThreads) k_hard_leaves(const HardJob *__restrict__ jobs,
                                                          const unsigned int *njobs, uint32_t max_jobs,
                                                          const uint64_t *__restrict__ unit0,
                                                          const unsigned char *__restrict__ snap,
                                                          uint32_t lbits_sub, const int32_t *__restrict__ MU,
                                                          const cpx_pient *__restrict__ Tpi,
                                                          unsigned long long *__restrict__ acc)
{
    const uint32_t n = min(*njobs, max_jobs);
    const uint64_t total = unit0[max_jobs];  // exclusive scan of the units; slots past n hold 0
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const size_t stride = snap_stride(lbits_sub);
    const size_t ncmax = (size_t(1) << lbits_sub) >> 7;
    __shared__ uint32_t s_leaf[kThreads / 32][kLeafBuf];
    uint32_t *lbuf = s_leaf[threadIdx.x >> 5];
    for (uint64_t unit = gw; unit < total; unit += nw) {
        uint32_t lo_j = 0, hi_j = n;  // unit0[lo_j] <= unit < unit0[hi_j]
        while (hi_j - lo_j > 1) {
            const uint32_t mid = (lo_j + hi_j) >> 1;
            if (__ldg(unit0 + mid) <= unit) lo_j = mid;
            else hi_j = mid;
        }
        const HardJob &J = jobs[lo_j];
        const uint64_t lu = unit - __ldg(unit0 + lo_j);
        const uint4 *sb = reinterpret_cast<const uint4 *>(snap + (size_t)J.snap * stride);
        const uint32_t *spre = reinterpret_cast<const uint32_t *>(sb + ncmax);
        const XT xp = (XT)J.xp;
        const double xpd = (double)(uint64_t)xp;
        const uint64_t lo = J.lo;
        const bool q41 = lo + (2ull << lbits_sub) <= (1ull << 41);  // the sub-segment ends below 2^41
        // survivors of the sub-segment with n <= uu (the carry is added per unit)
        auto count = [&](uint64_t uu) -> uint32_t {
            const uint32_t kk = (uint32_t)((uu - lo + 1) >> 1);
            if (!kk) return 0u;  // u = lo: no number of the sub-segment is <= u
            const uint32_t jb = kk - 1, w = jb >> 5, ch = w >> 2;
            return __ldg(spre + ch) + chunk_survivors(__ldg(sb + ch), jb);
        };
        int64_t S = 0;
        int32_t ms = 0;
        // leaves gathered into the warp's buffer (m, bit 31: mu(m) = -1) and
        // answered 32 at a time, as in k_hard
        uint32_t nbuf = 0;
        auto flush = [&] {
            __syncwarp();
            for (uint32_t jj = lane; jj < nbuf; jj += 32) {
                const uint32_t e = lbuf[jj];
                const uint32_t cv = count(leaf_quot(xp, xpd, e & 0x7FFFFFFFu, q41));
                if (e >> 31) {
                    S += cv;
                    ms += 1;
                } else {
                    S -= cv;
                    ms -= 1;
                }
            }
            __syncwarp();
            nbuf = 0;
        };
        auto place = [&](uint32_t cnt, uint32_t &off) -> uint32_t {
            uint32_t inc = cnt;
#pragma unroll
            for (int oo = 1; oo < 32; oo <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, oo);
                if (lane >= (uint32_t)oo) inc += t;
            }
            off = inc - cnt;
            return __shfl_sync(FULL, inc, 31);
        };
        if (J.kind == 1) {
            const uint64_t qa = J.mlo, mhi = J.mhi;
            const uint64_t w0 = (qa >> 7) + lu * kJobWords, wl = (mhi - 1) >> 7;
            for (uint64_t k = 0; k < kJobWords / 32; k++) {
                if (w0 + 32 * k > wl) break;  // uniform
                const uint64_t wq = w0 + 32 * k + lane;
                uint64_t qb = 0;
                if (wq <= wl) qb = __ldg(reinterpret_cast<const ulonglong2 *>(Tpi) + wq).x & range_mask(wq, qa, mhi);
                uint32_t off;
                const uint32_t tot_r = place((uint32_t)__popcll(qb), off);
                if (tot_r > kLeafBuf) {  // a dense round: each lane answers its own word
                    while (qb) {
                        const int j = __ffsll((long long)qb) - 1;
                        qb &= qb - 1;
                        S += count(leaf_quot(xp, xpd, 128 * wq + 2 * j + 1, q41));  // mu(q) = -1
                        ms += 1;
                    }
                    continue;
                }
                if (nbuf + tot_r > kLeafBuf) flush();
                uint32_t kk = nbuf + off;
                while (qb) {
                    const int j = __ffsll((long long)qb) - 1;
                    qb &= qb - 1;
                    lbuf[kk++] = (uint32_t)(128 * wq + 2 * j + 1) | 0x80000000u;
                }
                nbuf += tot_r;
            }
        } else {
            const uint64_t i_lo = (J.mlo + 1) >> 1, i_hi = (J.mhi - 1) >> 1;
            const uint64_t g0 = (i_lo >> 2) + lu * kJobGroups, gl = i_hi >> 2;
            const uint32_t p = J.p;
            for (uint64_t k = 0; k < kJobGroups / 32; k++) {
                if (g0 + 32 * k > gl) break;  // uniform
                const uint64_t g = g0 + 32 * k + lane;
                uint32_t neg = 0, vm = 0;
                if (g <= gl) vm = valid_group(__ldg(reinterpret_cast<const int4 *>(MU) + g), g, i_lo, i_hi, p, &neg);
                uint32_t off;
                const uint32_t tot_r = place((uint32_t)__popc(vm), off);
                if (nbuf + tot_r > kLeafBuf) flush();
                uint32_t kk = nbuf + off;
                while (vm) {
                    const int kq = __ffs(vm) - 1;
                    vm &= vm - 1;
                    lbuf[kk++] = (uint32_t)(2 * (4 * g + kq) + 1) | (((neg >> kq) & 1u) << 31);
                }
                nbuf += tot_r;
            }
        }
        flush();
        const i128 Sw = cpx_warp_sum_i128((i128)S);
#pragma unroll
        for (int dd = 16; dd > 0; dd >>= 1) ms += __shfl_down_sync(FULL, ms, dd);
        if (lane == 0) acc_add(acc, J.q, ACC_HARD, Sw + (i128)J.carry * ms);
    }
}

// B(seg) of every work unit (seg_levels) and its level count max(0, B - c);
// then, one thread per (query, level), the level table of the sieve: x/p, y/p
// and min(y, x/p^3), which do not depend on the segment.
template <class XT>
__global__ void k_hard_plan(const QD *__restrict__ qd, uint32_t Q, const uint64_t *__restrict__ pre_seg,
                            uint64_t total, const uint64_t *__restrict__ pre_comb, uint64_t total_lv,
                            const uint32_t *__restrict__ P, uint32_t np, const uint32_t *__restrict__ dense,
                            uint32_t *__restrict__ seg_B, uint64_t *__restrict__ seg_lv, XT *__restrict__ lvx,
                            uint2 *__restrict__ lae)
{
    uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u < total) {
        const uint32_t q = find_q(pre_seg, Q, u);
        const QD &d = qd[q];
        const uint64_t seg = unit_seg(d, dense, u - pre_seg[q]).seg + d.seg0;
        const uint64_t lo = seg * 2 * (1ull << d.lbits), hi = lo + 2 * (1ull << d.lbits);
        const uint32_t a = seg_levels<XT>(xload<XT>(d), d.r4, lo, hi, P, np);
        seg_B[u] = a;
        seg_lv[u] = a > d.c ? a - d.c : 0;
        return;
    }
    u -= total;
    if (u >= total_lv) return;
    const uint32_t q = find_q(pre_comb, Q, u);
    const QD &d = qd[q];
    const uint64_t p = P[d.c + (u - pre_comb[q])];
    const XT xp = cpx_qdiv(xload<XT>(d), p);
    const XT t3 = cpx_qdiv(xp, p * p);
    lvx[u] = xp;
    lae[u] = make_uint2((uint32_t)cpx_udiv_leaf(d.y, p), (uint32_t)(t3 < (XT)d.y ? (uint64_t)t3 : d.y));
}

// H += sum over segments of carry(seg, b) * msum(seg, b); carry = count of
// survivors of level b-1 below the segment.  Level b is sieved from the first
// segment reaching p_b^2; below p_b^2 the survivors of level b-1 are 1 and the
// primes from p_b on, so the carry starts at 1 + max(0, pi(lo - 1) - (b - 1))
// from the pi table and then adds the sieved segments' counts.  One warp per
// (query, b): its lanes take 32 consecutive units at a time and a warp
// scan of their counts gives each unit its carry.  The units sieving
// level b are contiguous from the first one.
__global__ void k_hard_combine(const QD *__restrict__ qd, uint32_t Q, const uint64_t *__restrict__ pre_comb,
                               uint64_t total, const uint64_t *__restrict__ pre_seg,
                               const uint32_t *__restrict__ seg_B, const uint64_t *__restrict__ seg_off,
                               const uint32_t *__restrict__ cnt, const int32_t *__restrict__ ms, uint64_t cap,
                               const uint32_t *__restrict__ P, const cpx_pient *__restrict__ T,
                               const uint32_t *__restrict__ dense, unsigned long long *__restrict__ acc,
                               HardLevel *__restrict__ lvl_out)
{
    const uint64_t u = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (u >= total) return;  // uniform over the warp
    const uint32_t q = find_q(pre_comb, Q, u);
    const uint64_t lvl = u - pre_comb[q];
    const QD &d = qd[q];
    const uint32_t b = d.c + 1 + (uint32_t)lvl;
    const uint64_t span = 2ull << d.lbits;
    const uint64_t p = P[b - 1];
    const uint64_t first = (p * p) / span;  // first segment with hi > p^2
    // the query's segments here are seg0 .. seg0 + n - 1 (all of them unless
    // the query is split over GPUs); carries below the part come from outside
    const uint64_t g0 = d.seg0, g1 = d.seg0 + d.nseg;
    const uint64_t fl = first > g0 ? first : g0;
    // units of a segment follow one another, the last of them with its count:
    // the others' carry is the segment's too
    const uint64_t s0 = pre_seg[q] + seg_unit(d, dense, fl - g0), s1 = pre_seg[q + 1];
    const bool anchored = first >= g0 && first < g1;
    uint64_t carry = 0;
    if (anchored && first > 0) {
        const uint64_t pl = cpx_pi_dev(T, first * span - 1);
        carry = 1 + (pl > b - 1 ? pl - (b - 1) : 0);
    }
    const uint64_t carry0 = carry;
    int64_t msl = 0;
    i128 H = 0;
    for (uint64_t base = s0; base < s1; base += 32) {
        const uint64_t sg = base + lane;
        uint32_t cv = 0;
        int32_t mv = 0;
        bool act = false;
        if (sg < s1 && __ldg(seg_B + sg) >= b) {
            const uint64_t idx = __ldg(seg_off + sg) + lvl;
            if (idx < cap) {
                cv = __ldg(cnt + idx);
                mv = __ldg(ms + idx);
                act = true;
            }
        }
        const unsigned bal = __ballot_sync(FULL, act);
        const int stop = __ffs(~bal) - 1;  // first segment past the level's range (-1: none here)
        if (stop >= 0 && (int)lane >= stop) {
            cv = 0;
            mv = 0;
        }
        uint64_t inc = cv;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t t = __shfl_up_sync(FULL, inc, o);
            if (lane >= (uint32_t)o) inc += t;
        }
        H += (i128)(carry + inc - cv) * (i128)mv;
        msl += mv;
        carry += __shfl_sync(FULL, inc, 31);
        if (stop >= 0) break;
    }
    H = cpx_warp_sum_i128(H);
    if (lane == 0) acc_add(acc, q, ACC_HARD, H);
    if (lvl_out && q == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) msl += __shfl_down_sync(FULL, msl, o);
        if (lane == 0) lvl_out[lvl] = HardLevel{carry - carry0, msl, carry0, anchored ? 1u : 0u, 0u};
    }
}

// ------------------------------------------------------------------ launchers

size_t hard_snapshot_stride(uint32_t lbits_sub) { return snap_stride(lbits_sub); }

size_t hard_smem_bytes(uint32_t lbits, uint32_t threads, bool wide)
{
    (void)wide;
    return levels_smem(lbits, threads);
}

void launch_hard_leaves(cpx_ctx *ctx, const Plan &pl, uint32_t lbits_sub)
{
    const Tables &tb = ctx->tab;
    scan_u64(ctx, pl.job_units, pl.max_jobs + 1);
    if (pl.wide)
        k_hard_leaves<u128><<<(unsigned)ctx->sm_count * 8, kThreads, 0, ctx->stream>>>(
            pl.jobs, pl.njobs, pl.max_jobs, pl.job_units, pl.snap, lbits_sub, tb.MU, tb.T, pl.acc);
    else
        k_hard_leaves<uint64_t><<<(unsigned)ctx->sm_count * 8, kThreads, 0, ctx->stream>>>(
            pl.jobs, pl.njobs, pl.max_jobs, pl.job_units, pl.snap, lbits_sub, tb.MU, tb.T, pl.acc);
    CPX_LAUNCH("k_hard_leaves");
    note_launch(ctx);
}

template <class XT> static void hard_go(cpx_ctx *ctx, const Plan &pl)
{
    const Tables &tb = ctx->tab;
    XT *lvx = static_cast<XT *>(pl.lvx);
    k_hard_plan<XT><<<(unsigned)((pl.n_seg + pl.n_comb + 255) / 256), 256, 0, ctx->stream>>>(
        pl.qd, pl.Q, pl.pre_seg, pl.n_seg, pl.pre_comb, pl.n_comb, tb.P, (uint32_t)tb.prm_n, pl.dense, pl.seg_B,
        pl.seg_off, lvx, pl.lae);
    CPX_LAUNCH("k_hard_plan");
    note_launch(ctx);
    scan_u64(ctx, pl.seg_off, pl.n_seg);
    const size_t smem = levels_smem(pl.lbits_max, pl.hard_threads);
    if (pl.time_hard) CPX_CUDA(cudaEventRecord(ctx->ev_hard0, ctx->stream));
    if (pl.fork) CPX_CUDA(cudaEventRecord(ctx->ev_fork, ctx->stream));
    {
        KSpan ks(ctx, "k_hard");
        k_hard<XT><<<(unsigned)pl.n_seg, pl.hard_threads, smem, ctx->stream>>>(
            pl.qd, pl.Q, pl.pre_seg, pl.n_seg, pl.seg_B, pl.seg_off, tb.P, tb.MU, tb.T, pl.pre_comb, lvx, pl.lae,
            pl.dense, pl.hard_cnt, pl.hard_ms, pl.hard_entries, pl.acc, pl.lbits_max);
    }
    CPX_LAUNCH("k_hard");
    note_launch(ctx);
    if (pl.time_hard) CPX_CUDA(cudaEventRecord(ctx->ev_hard1, ctx->stream));
    if (pl.n_comb) {
        k_hard_combine<<<(unsigned)((pl.n_comb * 32 + 255) / 256), 256, 0, ctx->stream>>>(
            pl.qd, pl.Q, pl.pre_comb, pl.n_comb, pl.pre_seg, pl.seg_B, pl.seg_off, pl.hard_cnt, pl.hard_ms,
            pl.hard_entries, tb.P, tb.T, pl.dense, pl.acc, pl.hard_levels);
        CPX_LAUNCH("k_hard_combine");
        note_launch(ctx);
    }
}

// The dynamic shared-memory limit of k_hard is a property of the function,
// shared by every context and thread of the process, so it is raised to the
// device's opt-in maximum once (under a lock) instead of per launch: a lane
// lowering it while another lane launches a larger segment would fail.
void prepare_hard(cpx_ctx *ctx, const Plan &pl)
{
    if (!pl.n_seg) return;
    const size_t smem = levels_smem(pl.lbits_max, pl.hard_threads);
    if (smem > ctx->smem_optin) fail(CPX_EINVAL, "hard-leaf segment needs more shared memory than a block can have");
    static std::mutex m;
    static int done_dev[2] = {-1, -1};
    std::lock_guard<std::mutex> g(m);
    const int w = pl.wide ? 1 : 0;
    if (done_dev[w] == ctx->device) return;
    if (pl.wide)
        CPX_CUDA(cudaFuncSetAttribute(k_hard<u128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ctx->smem_optin));
    else
        CPX_CUDA(cudaFuncSetAttribute(k_hard<uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)ctx->smem_optin));
    done_dev[w] = ctx->device;
}

void launch_hard(cpx_ctx *ctx, const Plan &pl)
{
    if (!pl.n_seg) return;
    if (pl.n_seg > 0x7FFFFFFFull) fail(CPX_ERANGE, "too many hard-leaf segments in one launch");
    if (pl.wide) hard_go<u128>(ctx, pl);
    else hard_go<uint64_t>(ctx, pl);
}

}  // namespace cpx

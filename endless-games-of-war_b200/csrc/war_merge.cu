// war_merge.cu — the kernels of war_enumerate with the path memo (war_refill.cuh): deals, each state after their
// first floor(n/2) turns played once (war_merge.cuh), and canonical scans; and their host plans.
//
// The loop is the latched loop of war_refill.cuh for one game per lane: `defer` turns without a branch or a
// vote, then a service that saves Brent's checkpoint, looks the game up in the memo, records it if it is
// decided and gives its lane the next one.  A game starts at turn h, so its tortoise is the state at turn h
// and its checkpoints follow from there.
//
// What bounds it: random reads and writes of the table in HBM, as in the kernel that played every deal, but
// nine times fewer (all 13! deals: 5.8e8 lookups and 1.6e8 stores instead of 6.2e9 and 3.8e8) and, for jobs of
// fewer than about 1e6 games, the longest game.  Measured on a B200 against the one-deal-one-game kernel it
// replaces: all 13! deals 166 -> 20.1 ms, the end of them from a saved progress 168 -> 33.5 ms, a span of
// 4.26e9 of 14 cards with --half 124 -> 17.1 ms and of 15 cards 370 -> 168 ms, 1e8 of 13 cards 10.7 -> 2.9 ms,
// 3e5 of 10 cards 1.71 -> 0.076 ms (there the 720-deal units of one lane each were the time).
#include <algorithm>
#include <cstring>
#include <vector>
#include "war_refill.cuh"
#include "war_host.h"
#include "war_merge.cuh"

namespace war {

// One game slot of the merged kernel.
struct MGame {
    u64 w1, w2, t1, t2, ka, kb;
    u32 q, rounds, next, wt, ta, tb, mv;
    bool done, kcy, active;
};

template <int RULE>
__device__ __forceinline__ void merge_body(const MergeArgs& a, DevAcc* __restrict__ acc, u64* __restrict__ counter,
                                           u32* sh) {
    __shared__ MUnit units[32];
    u32* shh = sh;
    u32* she = sh + a.hbins;
    const int bins = a.hbins + WAR_EBINS;
    for (int b = threadIdx.x; b < bins; b += blockDim.x) sh[b] = 0;
    __syncthreads();

    const u32 n = (u32)a.n, h = n >> 1, W = (u32)a.W, n2 = 2u * n;
    const TurnK K = a.tk;
    const u32 hb1 = a.hbins > 0 ? (u32)(a.hbins - 1) : 0u;
    const int period = a.defer > 4 ? (a.defer + 3) & ~3 : 4;
    u64* const memo = a.memo;
    const u32 mbits = a.memo_bits;
    const u32 vmask = (1u << mbits) - 1u;
    const u64 pat = 0x1111111111111111ull * (u64)(n - 1u);
    const u32 lane = threadIdx.x & 31u;
    MUnit& mu = units[threadIdx.x >> 5];

    MCursor c;
    u32 cyc = 0, turns = 0, maxfin = 0, capped = 0, mlook = 0, mhit = 0, mstore = 0;
    MGame g;
    g.active = false; g.done = true; g.kcy = false; g.w1 = g.w2 = 1ull; g.t1 = g.t2 = 0ull; g.q = 0; g.rounds = 0;
    g.next = 0xFFFFFFFFu; g.ta = g.tb = 0; g.ka = g.kb = 0; g.mv = 0; g.wt = 0;

    auto drain = [&]() {
        __syncwarp();
        for (int b = (int)lane; b < bins; b += 32) {
            const u32 v = atomicExch(&sh[b], 0u);
            if (v) atomicAdd(b < a.hbins ? &acc->hist[b] : &acc->endhist[b - a.hbins], (u64)v);
        }
        const u64 v_cyc = warp_sum((u64)cyc), v_turns = warp_sum((u64)turns);
        if (lane == 0u) {
            if (v_cyc) atomicAdd(&acc->cyc, v_cyc);
            if (v_turns) atomicAdd(&acc->turns, v_turns);
        }
        cyc = 0; turns = 0;
    };
    auto setup = [&](const MBlock& B, u64 outer) {
        MUnit m;
        merge_unit<RULE>(B, outer, n, m);
        __syncwarp();
        if (lane == 0u) mu = m;
        __syncwarp();
    };
    auto over = [&]() -> u32 {
        return mu.s2 + 8u * (c.f - c.pa) == 0u ? 1u : (mu.s1 + 8u * c.pa == 0u ? 2u : 0u);
    };
    auto ended = [&](u32 k) {
        if (lane == 0u) atomicAdd(&she[h], k);
        maxfin = max(maxfin, h);
    };
    auto build = [&](u32 sel) -> bool {
        const u32 a8 = 8u * c.pa;
        const u64 lw = mu.O | ((u64)merge_row(mu.c0, mu.c1, sel) << (8u * (c.f - c.fi)));
        g.w1 = mu.U1 | shl64(lw & ~shl64(~0ull, a8), mu.s1) | shl64(1ull, mu.s1 + a8);
        g.w2 = mu.U2 | shl64(shr64(lw, a8), mu.s2) | shl64(1ull, mu.s2 + 8u * c.f - a8);
        if (c.filter) {   // player 1 must hold card n - 1
            const u64 x = g.w1 ^ pat;
            if (((x - 0x1111111111111111ull) & ~x & 0x8888888888888888ull) == 0ull) return false;
        }
        g.q = mu.s1 + a8 - n2;
        g.t1 = g.w1; g.t2 = g.w2; g.rounds = h; g.next = 2u * h + W;
        g.ta = 0; g.tb = 0; g.mv = 0; g.wt = c.wt;
        g.done = false; g.kcy = false; g.active = true;
        return true;
    };
    auto refill = [&](bool want) {
        if (want) g.active = false;
        merge_deal(c, a, counter, want, setup, over, ended, build, drain);
    };

    refill(true);
    bool running = __any_sync(WAR_FULL_MASK, g.active);
    while (running) {
        for (int k = 0; k < period; k += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                war_turn_fma<RULE>(g.w1, g.w2, g.q, K);
                const bool en = g.q * g.q == K.end2;
                if (!g.done) g.rounds += K.one;
                const bool cy = (g.w1 == g.t1) & (g.w2 == g.t2);
                const bool fin = (cy | en) & !g.done;
                g.kcy = fin ? cy : g.kcy;
                g.done = g.done | fin;
            }
        }
        if (!g.done && g.rounds >= g.next) {   // Brent's checkpoint (war_refill.cuh)
            if (g.next > WAR_TURN_CAP) { capped++; g.done = true; }   // abandoned (never expected): the job fails
            else { g.t1 = g.w1; g.t2 = g.w2; g.next = 2u * g.rounds + W; }
        }
        if (!g.done) {
            const u64 key = memo_key_state(g.w1, g.w2, n);
            const u64 e = __ldcg((const unsigned long long*)memo + memo_slot(key, mbits));
            mlook++;
            const u32 v = (u32)e & vmask;
            if (v != 0u && ((e ^ path_entry(key, mbits, 0ull)) >> mbits) == 0ull) {
                mhit++;
                g.done = true; g.kcy = (v & 1u) == 0u; g.mv = v;
            } else {
                g.kb = g.ka; g.tb = g.ta;
                g.ka = key; g.ta = g.rounds;
            }
        }
        const bool fin = g.done & g.active;
        if (__any_sync(WAR_FULL_MASK, fin)) {
            if (fin) {
                turns += g.rounds - h;
                const u32 mcy = (g.mv & 1u) ? 0u : g.mv >> 1;
                const u32 len = (g.mv & 1u) ? g.rounds + (g.mv >> 1) : g.rounds;
                const u32 lam = mcy ? mcy : g.rounds - ((g.next - W) >> 1);
                if (g.ta) {   // the states it missed, with its outcome
                    const u32 v = g.kcy ? 2u * lam : 2u * (len - g.ta) + 1u;
                    if (v <= vmask) {
                        __stcg((unsigned long long*)memo + memo_slot(g.ka, mbits), path_entry(g.ka, mbits, v));
                        mstore++;
                    }
                }
                if (g.tb) {
                    const u32 v = g.kcy ? 2u * lam : 2u * (len - g.tb) + 1u;
                    if (v <= vmask) {
                        __stcg((unsigned long long*)memo + memo_slot(g.kb, mbits), path_entry(g.kb, mbits, v));
                        mstore++;
                    }
                }
                if (g.kcy) {
                    cyc += g.wt;
                    if (mcy == 0u) {   // found by Brent: store its cycle
                        memo_store_cycle<RULE, MEMO_PATH>(memo, mbits, g.w1, g.w2, g.q + n2, n, lam);
                        mstore += lam;
                    }
                    if (a.hbins) atomicAdd(&shh[lam < hb1 ? lam : hb1], g.wt);
                } else {
                    maxfin = max(maxfin, len);
                    atomicAdd(&she[len < WAR_EBINS - 1 ? len : WAR_EBINS - 1], g.wt);
                }
            }
            refill(fin);
            running = __any_sync(WAR_FULL_MASK, g.active);
        }
    }

    const u64 v_cyc = warp_sum((u64)cyc), v_turns = warp_sum((u64)turns), v_max = warp_max((u64)maxfin);
    const u64 v_cap = warp_sum((u64)capped), v_l = warp_sum((u64)mlook), v_h = warp_sum((u64)mhit);
    const u64 v_s = warp_sum((u64)mstore);
    if (lane == 0u) {
        if (c.done) atomicAdd(&acc->done, c.done);
        if (v_cyc) atomicAdd(&acc->cyc, v_cyc);
        if (v_turns) atomicAdd(&acc->turns, v_turns);
        if (v_max) atomicMax(&acc->maxfin, v_max);
        if (v_cap) atomicAdd(&acc->status, v_cap);
        if (v_l) atomicAdd(&acc->memo_lookups, v_l);
        if (v_h) atomicAdd(&acc->memo_hits, v_h);
        if (v_s) atomicAdd(&acc->memo_stores, v_s);
    }
    __syncthreads();
    flush_hist(shh, acc->hist, a.hbins);
    flush_hist(she, acc->endhist, WAR_EBINS);
}

template <int RULE>
__global__ void __launch_bounds__(1024) merge_kernel(const __grid_constant__ MergeArgs a, DevAcc* __restrict__ acc) {
    extern __shared__ u32 sh[];
    merge_body<RULE>(a, acc, &acc->work_next, sh);
}

// ---- canonical scans ----------------------------------------------------------------------------------
//
// The same loop for canonical positions with the path memo, one game each.  EXTRA: the distinct-cycle outputs and
// the sample (gpu/war_gpu.py:217-235); SHAPE: the loop-shape test, whose code travels in the memo with the cycle
// length (war_refill.cuh).  Whether the start of a game lies on its cycle (distinct) shows within Brent's first
// window, which compares every state up to turn W with the start: a memo hit "cycle of length lam" before turn
// lam <= W is held (pend) until then.
//
// What bounds it: instruction issue and the random reads of the table, about equally; in a small scan the number
// of warps at work, which is why a warp, not a lane, takes a unit (a lane of the kernel it replaces played 120
// orders with all their splits alone).  B200: 2e6 positions of 11 cards 8.9 -> 0.40 ms, 3e9 of 14 cards 164 ->
// 152 ms (defer 16; 12: 156, 8: 176 ms; 256 to 1024 threads alike).
template <bool EXTRA>
struct CGame {
    u64 w1, w2, t1, t2, ka, kb;
    u32 q, rounds, next, ta, tb, mv, pend;
    bool done, kcy, active, sampled;
};

template <int RULE, bool EXTRA, bool SHAPE>
__device__ __forceinline__ void canon_body(const MergeArgs& a, DevAcc* __restrict__ acc, u64* __restrict__ counter,
                                           u64* sh64) {
    __shared__ CUnit units[32];
    ulonglong2* const start = (ulonglong2*)sh64 + threadIdx.x;      // EXTRA: the starting piles
    u32* const shh = (u32*)((ulonglong2*)sh64 + (EXTRA ? blockDim.x : 0u));
    u32* const she = shh + a.hbins;
    const int bins = a.hbins + WAR_EBINS;
    for (int b = threadIdx.x; b < bins; b += blockDim.x) shh[b] = 0;
    __syncthreads();

    const u32 n = (u32)a.n, m = n - 1u, k4m4 = 4u * m, W = (u32)a.W, n2 = 2u * n;
    const TurnK K = a.tk;
    const u32 hb1 = a.hbins > 0 ? (u32)(a.hbins - 1) : 0u;
    const int period = a.defer > 4 ? (a.defer + 3) & ~3 : 4;
    u64* const memo = a.memo;
    const u32 mbits = a.memo_bits, lsh = SHAPE ? 3u : 1u;          // a memo value: 8 lam + 2 code, or 2 lam
    const u32 vmask = (1u << mbits) - 1u;
    const u32 lane = threadIdx.x & 31u;
    CUnit& cu = units[threadIdx.x >> 5];

    MCursor c;
    u32 cyc = 0, turns = 0, maxfin = 0, capped = 0, mlook = 0, mhit = 0, mstore = 0, nonstd = 0, unchk = 0;
    u32 sc = 0, scy = 0, slam = 0, slen = 0, smax = 0, oncyc = 0, dmin = 0;
    CGame<EXTRA> g;
    g.active = false; g.done = true; g.kcy = false; g.sampled = false; g.w1 = g.w2 = 1ull; g.t1 = g.t2 = 0ull;
    g.q = 0; g.rounds = 0; g.next = 0xFFFFFFFFu; g.ta = g.tb = 0; g.ka = g.kb = 0; g.mv = 0; g.pend = 0;

    // (A launch plays fewer than 2^32 positions: no bin and no total of a lane or warp can wrap.)
    auto drain = [&]() {};
    auto setup = [&](const MBlock& B, u64 outer) {
        CUnit u;
        canon_unit(B, outer, m, u);
        __syncwarp();
        if (lane == 0u) cu = u;
        __syncwarp();
    };
    auto over = []() -> u32 { return 0u; };
    auto ended = [](u32) {};
    auto build = [&](u32 sel) -> bool {
        u32 q4;
        canon_position(cu.Q | ((u64)merge_row(cu.c0, cu.c1, sel) << (4u * (m - c.fi))), n, c.pa, g.w1, g.w2, q4);
        g.q = q4 - n2;
        g.t1 = g.w1; g.t2 = g.w2; g.rounds = 0; g.next = W;
        g.ta = 0; g.tb = 0; g.mv = 0; g.pend = 0;
        g.done = false; g.kcy = false; g.active = true;
        if (EXTRA) {
            *start = make_ulonglong2(g.w1, g.w2);
            g.sampled = a.sample && war_pick(a.seed, a.thr, g.w1, g.w2);
        }
        return true;
    };
    auto refill = [&](bool want) {
        if (want) g.active = false;
        merge_deal<true>(c, a, counter, want, setup, over, ended, build, drain);
    };

    refill(true);
    bool running = __any_sync(WAR_FULL_MASK, g.active);
    while (running) {
        for (int k = 0; k < period; k += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                war_turn_fma<RULE>(g.w1, g.w2, g.q, K);
                const bool en = g.q * g.q == K.end2;
                if (!g.done) g.rounds += K.one;
                const bool cy = (g.w1 == g.t1) & (g.w2 == g.t2);
                const bool fin = (cy | en) & !g.done;
                g.kcy = fin ? cy : g.kcy;
                g.done = g.done | fin;
            }
        }
        if (!g.done && g.rounds >= g.next) {   // Brent's checkpoint (war_refill.cuh)
            if (g.next > WAR_TURN_CAP) { capped++; g.done = true; }   // abandoned (never expected): the job fails
            else { g.t1 = g.w1; g.t2 = g.w2; g.next = 2u * g.rounds + W; }
        }
        if (!g.done && g.pend == 0u) {
            const u64 key = memo_key_state(g.w1, g.w2, n);
            const u64 e = __ldcg((const unsigned long long*)memo + memo_slot(key, mbits));
            mlook++;
            const u32 v = (u32)e & vmask;
            if (v != 0u && ((e ^ path_entry(key, mbits, 0ull)) >> mbits) == 0ull) {
                mhit++;
                const bool vcy = (v & 1u) == 0u;
                if (EXTRA && a.distinct && vcy && (v >> lsh) <= W && g.rounds < (v >> lsh)) g.pend = v;
                else { g.done = true; g.kcy = vcy; g.mv = v; }
            } else {
                g.kb = g.ka; g.tb = g.ta;
                g.ka = key; g.ta = g.rounds;
            }
        } else if (EXTRA && !g.done && g.rounds >= (g.pend >> lsh)) {
            // turn lam passed without the start coming back: on the cycle, not through the start
            g.done = true; g.kcy = true; g.mv = g.pend;
        }
        const bool fin = g.done & g.active;
        if (__any_sync(WAR_FULL_MASK, fin)) {
            if (fin) {
                turns += g.rounds;
                const bool cy = g.kcy;
                const u32 mcy = (g.mv & 1u) ? 0u : g.mv >> lsh;
                const u32 len = (g.mv & 1u) ? g.rounds + (g.mv >> 1) : g.rounds;
                const u32 lam = mcy ? mcy : g.rounds - ((g.next - W) >> 1);
                u32 code = 0;
                if (SHAPE && cy) {
                    code = mcy ? (g.mv >> 1) & 3u : (u32)loop_shape_walk<RULE>(g.w1, g.w2, g.q + n2, k4m4, lam, (u32)a.blk);
                    if (code == 1u) nonstd++;
                    if (code == 2u) unchk++;
                }
                const u32 vcyc = SHAPE ? 8u * lam + 2u * code : 2u * lam;
                if (g.ta) {   // the states it missed, with its outcome
                    const u32 v = cy ? vcyc : 2u * (len - g.ta) + 1u;
                    if (v <= vmask) {
                        __stcg((unsigned long long*)memo + memo_slot(g.ka, mbits), path_entry(g.ka, mbits, v));
                        mstore++;
                    }
                }
                if (g.tb) {
                    const u32 v = cy ? vcyc : 2u * (len - g.tb) + 1u;
                    if (v <= vmask) {
                        __stcg((unsigned long long*)memo + memo_slot(g.kb, mbits), path_entry(g.kb, mbits, v));
                        mstore++;
                    }
                }
                if (cy) {
                    cyc++;
                    if (mcy == 0u) {   // found by Brent: store its cycle
                        memo_store_cycle<RULE, MEMO_PATH>(memo, mbits, g.w1, g.w2, g.q + n2, n, lam, vcyc);
                        mstore += lam;
                    }
                    if (a.hbins) atomicAdd(&shh[lam < hb1 ? lam : hb1], 1u);
                    if (EXTRA && a.distinct) {
                        // decided by the memo: the start was not seen again within lam <= W turns, or lam > W: walk
                        const ulonglong2 s = *start;
                        const u32 sq = 4u * pile_len(s.x);
                        const bool on = mcy == 0u && g.next == W ? true
                                      : (lam <= W ? false : on_cycle_walk<RULE>(s.x, s.y, sq, n, lam));
                        if (on) {
                            const CycleWalk cw = cycle_walk<RULE>(s.x, s.y, sq, n, lam);
                            oncyc++;
                            if (cw.is_min) dmin++;
                            if (a.dbins) {
                                const u32 d = cw.sym ? cw.c1 : cw.c1 + cw.c2, db1 = (u32)(a.dbins - 1);
                                atomicAdd(&acc->dhist[d < db1 ? d : db1], 1ull);
                            }
                        }
                    }
                } else {
                    maxfin = max(maxfin, len);
                    atomicAdd(&she[len < WAR_EBINS - 1 ? len : WAR_EBINS - 1], 1u);
                }
                if (EXTRA && g.sampled) {
                    sc++;
                    if (cy) { scy++; slam += lam; }
                    else { slen += len; smax = max(smax, len); }
                }
            }
            refill(fin);
            running = __any_sync(WAR_FULL_MASK, g.active);
        }
    }

    const u64 v_cyc = warp_sum((u64)cyc), v_turns = warp_sum((u64)turns), v_max = warp_max((u64)maxfin);
    const u64 v_cap = warp_sum((u64)capped), v_l = warp_sum((u64)mlook), v_h = warp_sum((u64)mhit);
    const u64 v_s = warp_sum((u64)mstore);
    if (lane == 0u) {
        if (c.done) atomicAdd(&acc->done, c.done);
        if (v_cyc) atomicAdd(&acc->cyc, v_cyc);
        if (v_turns) atomicAdd(&acc->turns, v_turns);
        if (v_max) atomicMax(&acc->maxfin, v_max);
        if (v_cap) atomicAdd(&acc->status, v_cap);
        if (v_l) atomicAdd(&acc->memo_lookups, v_l);
        if (v_h) atomicAdd(&acc->memo_hits, v_h);
        if (v_s) atomicAdd(&acc->memo_stores, v_s);
    }
    if (EXTRA) {
        const u64 v_sc = warp_sum((u64)sc), v_scy = warp_sum((u64)scy), v_slam = warp_sum((u64)slam);
        const u64 v_slen = warp_sum((u64)slen), v_smax = warp_max((u64)smax);
        const u64 v_on = warp_sum((u64)oncyc), v_dmin = warp_sum((u64)dmin);
        if (lane == 0u) {
            if (v_sc) {
                atomicAdd(&acc->s_count, v_sc); atomicAdd(&acc->s_cyc, v_scy); atomicAdd(&acc->s_lamsum, v_slam);
                atomicAdd(&acc->s_lensum, v_slen); atomicMax(&acc->s_maxfin, v_smax);
            }
            if (v_on) atomicAdd(&acc->oncycle, v_on);
            if (v_dmin) atomicAdd(&acc->distinct_min, v_dmin);
        }
    }
    if (SHAPE) {
        const u64 v_ns = warp_sum((u64)nonstd), v_un = warp_sum((u64)unchk);
        if (lane == 0u) {
            if (v_ns) atomicAdd(&acc->shape_nonstd, v_ns);
            if (v_un) atomicAdd(&acc->shape_unchecked, v_un);
        }
    }
    __syncthreads();
    flush_hist(shh, acc->hist, a.hbins);
    flush_hist(she, acc->endhist, WAR_EBINS);
}

template <int RULE, bool EXTRA, bool SHAPE>
__global__ void __launch_bounds__(1024) canon_kernel(const __grid_constant__ MergeArgs a, DevAcc* __restrict__ acc) {
    extern __shared__ u64 sh64[];
    canon_body<RULE, EXTRA, SHAPE>(a, acc, &acc->work_next, sh64);
}

// ---- host -----------------------------------------------------------------------------------------

// The ordered lists of fi pairs of 2 fi cards (ranks 0 .. 2 fi - 1), as byte selectors: nibble 2i of a row is
// the first card of pair i under the winner's pile, nibble 2i + 1 the second.  Unused selectors name a byte
// that holds no card (0).
static void table_rows(u32 fi, int rule, u32* out) {
    u32 k = 0;
    const u32 cards = 2u * fi, none = 7u;
    std::vector<u32> sel(2 * MERGE_INNER, none);
    auto rec = [&](auto&& self, u32 i, u32 free) -> void {
        if (i == fi) {
            u32 v = 0;
            for (u32 p = 0; p < 2u * MERGE_INNER; p++) v |= sel[p] << (4u * p);
            out[k++] = v;
            return;
        }
        for (u32 x = 0; x < cards; x++)
            for (u32 y = 0; y < x; y++)
                if ((free >> x & 1u) && (free >> y & 1u)) {
                    sel[2 * i] = rule ? y : x;
                    sel[2 * i + 1] = rule ? x : y;
                    self(self, i + 1u, free & ~(1u << x) & ~(1u << y));
                }
    };
    rec(rec, 0u, (1u << cards) - 1u);
}

void canon_table(u32* rows) {
    for (u32 i = 0; i <= CANON_INNER; i++) {
        u32 p[CANON_INNER], k = canon_row0(i);
        for (u32 j = 0; j < i; j++) p[j] = j;
        do {
            u32 v = 0;
            for (u32 j = 0; j < 8u; j++) v |= (j < i ? p[j] : 7u) << (4u * j);
            rows[k++] = v;
        } while (std::next_permutation(p, p + i));
    }
}

// The plan of a canonical scan: orders of the n - 1 other cards as aligned blocks, the first and the last order
// with the splits that are in the range.
void canon_plan(const war_job* job, u64 warps, MergePlan& p) {
    const u32 m = (u32)job->n - 1u;
    p.blocks.clear();
    p.games = job->hi - job->lo;
    std::vector<u64> orders;
    u64 rows = 0;
    auto add = [&](u64 r, int j, u32 k0, u32 k1) {
        MBlock B;
        memset(&B, 0, sizeof B);
        u32 mask = (1u << m) - 1u;
        for (u32 i = 0; i < m - (u32)j; i++) {
            const u64 f = fact((int)(m - 1u - i));
            u32 x = mask;
            for (u64 d = r / f; d; d--) x &= x - 1u;
            r %= f;
            B.prefix[i] = (u8)__builtin_ctz(x);
            mask &= ~(1u << B.prefix[i]);
        }
        B.b = (u8)(m - (u32)j);
        B.free_mask = mask;
        B.inner = (u8)std::min<u32>((u32)j, CANON_INNER);
        B.k0 = (u8)k0; B.k1 = (u8)k1;
        p.blocks.push_back(B);
        orders.push_back(fact(j));
        rows += fact(j);
    };
    u64 x = job->lo / m, y = job->hi / m;
    if (x == y) {
        if (job->lo < job->hi) add(x, 0, (u32)(job->lo % m), (u32)(job->hi % m));
    } else {
        if (job->lo % m) add(x++, 0, (u32)(job->lo % m), m);
        while (x < y) {
            int j = (int)m;
            while (j > 0 && (x % fact(j) != 0 || fact(j) > y - x)) j--;
            add(x, j, 0, m);
            x += fact(j);
        }
        if (job->hi % m) add(y, 0, 0, (u32)(job->hi % m));
    }
    // about 24 units for each warp, of at least a warp's worth of games
    u64 lc = rows / std::max<u64>(1, warps * 24);
    lc = std::min<u64>(std::max<u64>(lc, (32 + m - 1) / m), 720);
    const u64 parts = (720 + lc - 1) / lc;
    p.lc = (u32)((720 + parts - 1) / parts);
    u64 u = 0;
    for (size_t i = 0; i < p.blocks.size(); i++) {
        MBlock& B = p.blocks[i];
        const u32 r = canon_rows(B.inner);
        B.u0 = u;
        B.nch = (r + p.lc - 1) / p.lc;
        u += orders[i] / r * B.nch;
    }
    p.units = u;
    MBlock end;
    memset(&end, 0, sizeof end);
    end.u0 = ~0ull;   // no unit lies past the last block
    p.blocks.push_back(end);
}

void merge_table(int rule, u32* rows) {
    for (u32 fi = 0; fi <= MERGE_INNER; fi++) table_rows(fi, rule, rows + merge_row0(fi));
}

// The plan of a deals job: its range as aligned blocks, and their units for about `warps` warps.
void merge_plan(const war_job* job, u64 warps, MergePlan& p) {
    const int n = job->n;
    const u32 h = (u32)n / 2u;
    const bool half = (job->flags & WAR_F_HALF) != 0;
    u64 F[21];
    F[0] = 1;
    for (int i = 1; i <= 20; i++) F[i] = F[i - 1] * (u64)i;
    p.blocks.clear();
    p.games = 0;
    u64 rows4 = 0;   // table rows to play, over all outer choices of the blocks
    std::vector<u64> outer;
    for (u64 x = job->lo; x < job->hi;) {
        int j = n;
        while (j > 0 && (x % F[j] != 0 || F[j] > job->hi - x)) j--;
        MBlock B;
        memset(&B, 0, sizeof B);
        const u32 b = (u32)(n - j);
        u32 mask = (1u << n) - 1u;
        u64 r = x;
        int top_at = -1;
        for (u32 i = 0; i < b; i++) {
            const u64 f = F[n - 1 - (int)i];
            u32 m = mask;
            for (u64 d = r / f; d; d--) m &= m - 1u;
            r %= f;
            const u32 v = (u32)__builtin_ctz(m);
            mask &= ~(1u << v);
            B.prefix[i] = (u8)v;
            if ((int)v == n - 1) top_at = (int)i;
        }
        x += F[j];
        B.b = (u8)b;
        B.free_mask = mask;
        const u32 bb = b + (b & 1u);
        B.f = (u8)(bb < 2u * h ? (2u * h - bb) / 2u : 0u);
        B.twice = !half && b == 0u && !(n & 1);
        B.filter = B.twice || (half && top_at < 0);
        if (half && top_at >= 0 && (top_at & 1)) continue;   // card n-1 dealt to player 2
        const u64 lists = F[j] >> B.f;
        outer.push_back(lists / merge_rows(std::min<u32>(B.f, MERGE_INNER)));
        p.blocks.push_back(B);
        p.games += lists * (B.f + 1u);
        rows4 += lists;
    }
    // About 24 units for each warp, so that the last ones end together, of at least a warp's worth of games.
    u64 lc = rows4 / std::max<u64>(1, warps * 24);
    lc = std::min<u64>(std::max<u64>(lc, 7), 2520);
    const u64 parts = (2520 + lc - 1) / lc;
    p.lc = (u32)((2520 + parts - 1) / parts);
    u64 u = 0;
    for (size_t i = 0; i < p.blocks.size(); i++) {
        MBlock& B = p.blocks[i];
        B.u0 = u;
        B.nch = (merge_rows(std::min<u32>(B.f, MERGE_INNER)) + p.lc - 1) / p.lc;
        u += outer[i] * B.nch;
    }
    p.units = u;
    MBlock end;
    memset(&end, 0, sizeof end);
    end.u0 = ~0ull;   // no unit lies past the last block
    p.blocks.push_back(end);
}

// The arguments of a merged kernel; copies the plan's blocks to the device.
int merge_args(const war_job* job, const MergePlan& p, int hbins, int window, int defer, MergeArgs& a) {
    Ctx& c = ctx();
    cudaError_t e;
    if (p.blocks.size() > MERGE_BLOCK_CAP) return fail(WAR_EINVAL, "plan has %zu blocks", p.blocks.size());
    if ((e = cudaMemcpyAsync(c.d_blocks, p.blocks.data(), sizeof(MBlock) * p.blocks.size(), cudaMemcpyHostToDevice,
                             cur_stream())) != cudaSuccess)
        return cuda_fail(e, "copy blocks");
    memset(&a, 0, sizeof a);
    a.blocks = c.d_blocks;
    a.table = c.d_table + (job->mode == WAR_CANON ? 2 * MERGE_ROWS : job->rule ? MERGE_ROWS : 0);
    a.lc = p.lc;
    a.n = job->n; a.hbins = hbins; a.W = window; a.defer = defer;
    a.tk.k16 = 16u; a.tk.km16 = (u32)-16; a.tk.k2p28 = 1u << 28; a.tk.k4 = 4u; a.tk.one = 1u;
    a.tk.c0 = 2 * job->n - 4; a.tk.end2 = (u32)(4 * job->n * job->n);
    return WAR_OK;
}

static size_t merge_shmem(int hbins) { return sizeof(u32) * (size_t)(hbins + WAR_EBINS); }

cudaError_t launch_merged(const MergeArgs& a, int rule, int threads, int blocks, DevAcc* acc, cudaStream_t st) {
    (rule ? merge_kernel<1> : merge_kernel<0>)<<<blocks, threads, merge_shmem(a.hbins), st>>>(a, acc);
    note_launch();
    return cudaGetLastError();
}

int merged_max_blocks_per_sm(int rule, int threads, int hbins) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rule ? merge_kernel<1> : merge_kernel<0>, threads,
                                                      merge_shmem(hbins)) != cudaSuccess)
        return 0;
    return nb;
}

static size_t canon_shmem(int extra, int threads, int hbins) {
    return sizeof(u32) * (size_t)(hbins + WAR_EBINS) + (extra ? sizeof(ulonglong2) * (size_t)threads : 0);
}

typedef void (*MergeFn)(const MergeArgs, DevAcc*);

template <int RULE>
static MergeFn canon_pick(int shape, int extra) {
    if (shape) return extra ? canon_kernel<RULE, true, true> : canon_kernel<RULE, false, true>;
    return extra ? canon_kernel<RULE, true, false> : canon_kernel<RULE, false, false>;
}

cudaError_t launch_canon(const MergeArgs& a, int rule, int extra, int threads, int blocks, DevAcc* acc, cudaStream_t st) {
    const MergeFn fn = rule ? canon_pick<1>(a.blk, extra) : canon_pick<0>(a.blk, extra);
    fn<<<blocks, threads, canon_shmem(extra, threads, a.hbins), st>>>(a, acc);
    note_launch();
    return cudaGetLastError();
}

int canon_max_blocks_per_sm(int rule, int shape, int extra, int threads, int hbins) {
    const MergeFn fn = rule ? canon_pick<1>(shape, extra) : canon_pick<0>(shape, extra);
    const size_t shmem = canon_shmem(extra, threads, hbins);
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, shmem) != cudaSuccess) return 0;
    return nb;
}

}  // namespace war

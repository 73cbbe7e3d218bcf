// war_merge_body.cuh — the loops of the kernels with the path memo, shared by the persistent kernels (war_merge.cu)
// and the serving kernels (war_server.cu): merged deals and canonical scans.
//
// The loop is the latched loop of war_refill.cuh for one game per lane: `defer` turns without a branch or a
// vote, then a service that saves Brent's checkpoint, looks the game up in the memo, records it if it is
// decided and gives its lane the next one.  A merged game starts at turn h, so its tortoise is the state at turn
// h and its checkpoints follow from there.
//
// Landmarks.  What is looked up and stored is not the state at the service but the last landmark before it: a
// state with card n-1 on top of its holder's pile (every card reaches the top again within a lap of the pile).
// Games that have met look at the same landmarks whatever turn they have got to, where states at services
// meet only in games of one phase; and a cycle is stored by its landmarks, about one state in eight.
//
// What bounds it: random reads and writes of the table in HBM (13 cards: at the rate of the random-gather ceiling),
// instruction issue of the turns (canonical scans: ALU pipe 84%), and for jobs of fewer than about 1e6 games the
// longest game.  Measured on a B200 (states at services -> landmarks -> a found cycle recorded by playing on instead
// of by a walk): a span of 4.26e9 deals of 15 cards 210 -> 132 -> 85 ms (stores 3.4e9 -> 1.0e9), 1e8 deals of 13 cards
// 2.5 -> 2.0 -> 1.6 ms, a resumed a(13) 31.2 -> 30.5 -> 29.9 ms, --half span of 14 cards 13.7 -> 13.6 ms, 3e9
// canonical positions of 14 cards 152 -> 148 ms.  The one-deal-one-game kernel before: 370, 10.7, 168 and 124 ms.
#pragma once
#include "war_refill.cuh"
#include "war_merge.cuh"

namespace war {

// The units of a block's warps.
union UnitStore {
    MUnit m[32];
    CUnit c[32];
};

// One game slot of the merged kernel.
struct MGame {
    u64 w1, w2, t1, t2, m1, m2;   // piles, tortoise, the last landmark
    u32 q, rounds, next, wt, mv, at;
    bool done, kcy, active;
};

// A game's last two landmarks looked up and missed, and their turns + 1 (0: none), kept in shared memory.
struct Missed {
    u64 ka, kb;
    u32 ta, tb;
};
constexpr u32 NO_LANDMARK = 0xFFFFFFFFu;
// A game whose cycle Brent found plays on around it once more, to the tortoise's state again, and its services store
// the cycle's landmarks instead of looking them up: the other lanes go on meanwhile, where a walk of the cycle at
// once holds them up.  (Its checkpoint is this, which is never reached.)
constexpr u32 RECORDING = 0xFFFFFFFFu;

// Stores the landmarks that a decided game missed, with its outcome: the cycle value vcyc, or (vcyc = 0) the turns
// from there to its end after len turns.  Returns the entries stored.
__device__ __forceinline__ u32 store_missed(u64* memo, u32 mbits, const Missed& x, u32 vcyc, u32 len) {
    const u32 vmask = (1u << mbits) - 1u;
    u32 k = 0;
    if (x.ta) {
        const u32 v = vcyc ? vcyc : 2u * (len + 1u - x.ta) + 1u;
        if (v <= vmask) {
            __stcg((unsigned long long*)memo + memo_slot(x.ka, mbits), path_entry(x.ka, mbits, v));
            k++;
        }
    }
    if (x.tb) {
        const u32 v = vcyc ? vcyc : 2u * (len + 1u - x.tb) + 1u;
        if (v <= vmask) {
            __stcg((unsigned long long*)memo + memo_slot(x.kb, mbits), path_entry(x.kb, mbits, v));
            k++;
        }
    }
    return k;
}

template <int RULE>
__device__ __forceinline__ void merge_body(const MergeArgs& a, DevAcc* __restrict__ acc, u64* __restrict__ counter,
                                           UnitStore& store, u64* sh64) {
    MUnit* const units = store.m;
    Missed* const miss = (Missed*)sh64 + threadIdx.x;
    u32* const sh = (u32*)((Missed*)sh64 + blockDim.x);
    u32* const shh = sh;
    u32* const she = sh + a.hbins;
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
    g.next = 0xFFFFFFFFu; g.m1 = g.m2 = 0ull; g.at = NO_LANDMARK; g.mv = 0; g.wt = 0;

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
        g.mv = 0; g.wt = c.wt; g.at = NO_LANDMARK;
        miss->ta = 0; miss->tb = 0;
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
                const u64 v1 = g.w1, v2 = g.w2;
                u32 c1, c2;
                war_turn_fma<RULE>(g.w1, g.w2, g.q, K, c1, c2);
                const bool top = (c1 == n - 1u) | (c2 == n - 1u);
                g.m1 = top ? v1 : g.m1;
                g.m2 = top ? v2 : g.m2;
                g.at = top ? (u32)(k + u) : g.at;
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
        if (memo != nullptr && g.done && g.kcy && g.mv == 0u) {   // found by Brent: record the cycle
            const u32 v = 2u * (g.rounds - ((g.next - W) >> 1));
            if (v <= vmask) { g.mv = v; g.next = RECORDING; g.done = false; }
        } else if (memo != nullptr && !g.done && g.at != NO_LANDMARK) {
            const u64 key = memo_key_state(g.m1, g.m2, n);
            const u32 at = g.rounds - (u32)period + g.at;
            if (g.next == RECORDING) {
                __stcg((unsigned long long*)memo + memo_slot(key, mbits), path_entry(key, mbits, g.mv));
                mstore++;
            } else {
                const u64 e = __ldcg((const unsigned long long*)memo + memo_slot(key, mbits));
                mlook++;
                const u32 v = (u32)e & vmask;
                if (v != 0u && ((e ^ path_entry(key, mbits, 0ull)) >> mbits) == 0ull) {
                    mhit++;
                    g.done = true; g.kcy = (v & 1u) == 0u; g.mv = v;
                    g.next = at + (v >> 1);   // the game's length, if it ends
                } else {
                    miss->kb = miss->ka; miss->tb = miss->ta;
                    miss->ka = key; miss->ta = at + 1u;
                }
            }
        }
        g.at = NO_LANDMARK;
        const bool fin = g.done & g.active;
        if (__any_sync(WAR_FULL_MASK, fin)) {
            if (fin) {
                turns += g.rounds - h;
                const u32 mcy = (g.mv & 1u) ? 0u : g.mv >> 1;
                const u32 len = (g.mv & 1u) ? g.next : g.rounds;
                const u32 lam = mcy ? mcy : g.rounds - ((g.next - W) >> 1);
                mstore += store_missed(memo, mbits, *miss, g.kcy ? 2u * lam : 0u, len);
                if (g.kcy) {
                    cyc += g.wt;
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
    u64 w1, w2, t1, t2, m1, m2;
    u32 q, rounds, next, mv, pend, at;
    bool done, kcy, active, sampled, first;   // first: on the cycle from its start
};

template <int RULE, bool EXTRA, bool SHAPE>
__device__ __forceinline__ void canon_body(const MergeArgs& a, DevAcc* __restrict__ acc, u64* __restrict__ counter,
                                           UnitStore& store, u64* sh64) {
    CUnit* const units = store.c;
    Missed* const miss = (Missed*)sh64 + threadIdx.x;
    u64* const starts = (u64*)((Missed*)sh64 + blockDim.x);             // EXTRA: the starting piles
    u32* const shh = (u32*)(starts + (EXTRA ? 2u * blockDim.x : 0u));
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
    g.active = false; g.done = true; g.kcy = false; g.sampled = g.first = false; g.w1 = g.w2 = 1ull; g.t1 = g.t2 = 0ull;
    g.q = 0; g.rounds = 0; g.next = 0xFFFFFFFFu; g.m1 = g.m2 = 0ull; g.at = NO_LANDMARK; g.mv = 0; g.pend = 0;

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
        g.mv = 0; g.pend = 0; g.at = NO_LANDMARK; g.first = false;
        miss->ta = 0; miss->tb = 0;
        g.done = false; g.kcy = false; g.active = true;
        if (EXTRA) {
            starts[threadIdx.x] = g.w1;
            starts[threadIdx.x + blockDim.x] = g.w2;
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
                const u64 v1 = g.w1, v2 = g.w2;
                u32 c1, c2;
                war_turn_fma<RULE>(g.w1, g.w2, g.q, K, c1, c2);
                const bool top = (c1 == n - 1u) | (c2 == n - 1u);
                g.m1 = top ? v1 : g.m1;
                g.m2 = top ? v2 : g.m2;
                g.at = top ? (u32)(k + u) : g.at;
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
        if (g.done && g.kcy && g.mv == 0u && g.active) {   // found by Brent: record the cycle
            const u32 lam = g.rounds - ((g.next - W) >> 1);
            const u32 code = SHAPE ? (u32)loop_shape_walk<RULE>(g.w1, g.w2, g.q + n2, k4m4, lam, (u32)a.blk) : 0u;
            const u32 v = SHAPE ? 8u * lam + 2u * code : 2u * lam;
            g.first = g.next == W;
            g.mv = v;
            g.pend = 0u;
            if (memo != nullptr && v <= vmask) { g.next = RECORDING; g.done = false; }
        } else if (memo == nullptr) {
        } else if (!g.done && g.pend == 0u && g.at != NO_LANDMARK) {
            const u64 key = memo_key_state(g.m1, g.m2, n);
            const u32 at = g.rounds - (u32)period + g.at;
            if (g.next == RECORDING) {
                __stcg((unsigned long long*)memo + memo_slot(key, mbits), path_entry(key, mbits, g.mv));
                mstore++;
            } else {
                const u64 e = __ldcg((const unsigned long long*)memo + memo_slot(key, mbits));
                mlook++;
                const u32 v = (u32)e & vmask;
                if (v != 0u && ((e ^ path_entry(key, mbits, 0ull)) >> mbits) == 0ull) {
                    mhit++;
                    const bool vcy = (v & 1u) == 0u;
                    if (EXTRA && a.distinct && vcy && (v >> lsh) <= W && g.rounds < (v >> lsh)) g.pend = v;
                    else {
                        g.done = true; g.kcy = vcy; g.mv = v;
                        if (!vcy) g.next = at + (v >> 1);   // the game's length
                    }
                } else {
                    miss->kb = miss->ka; miss->tb = miss->ta;
                    miss->ka = key; miss->ta = at + 1u;
                }
            }
        } else if (EXTRA && !g.done && g.pend != 0u && g.rounds >= (g.pend >> lsh)) {
            // turn lam passed without the start coming back: on the cycle, not through the start
            g.done = true; g.kcy = true; g.mv = g.pend;
        }
        g.at = NO_LANDMARK;
        const bool fin = g.done & g.active;
        if (__any_sync(WAR_FULL_MASK, fin)) {
            if (fin) {
                turns += g.rounds;
                const bool cy = g.kcy;
                const u32 mcy = (g.mv & 1u) ? 0u : g.mv >> lsh;
                const u32 len = (g.mv & 1u) ? g.next : g.rounds;
                const u32 lam = mcy;      // (of a cycle: Brent's are values by now, too)
                if (SHAPE && cy) {
                    const u32 code = (g.mv >> 1) & 3u;
                    if (code == 1u) nonstd++;
                    if (code == 2u) unchk++;
                }
                mstore += store_missed(memo, mbits, *miss, cy ? g.mv : 0u, len);
                if (cy) {
                    cyc++;
                    if (a.hbins) atomicAdd(&shh[lam < hb1 ? lam : hb1], 1u);
                    if (EXTRA && a.distinct) {
                        // decided by the memo: the start was not seen again within lam <= W turns, or lam > W: walk
                        const u64 s1 = starts[threadIdx.x], s2 = starts[threadIdx.x + blockDim.x];
                        const u32 sq = 4u * pile_len(s1);
                        const bool on = g.first || (lam > W && on_cycle_walk<RULE>(s1, s2, sq, n, lam));
                        if (on) {
                            const CycleWalk cw = cycle_walk<RULE>(s1, s2, sq, n, lam);
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

}  // namespace war

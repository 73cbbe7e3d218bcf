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
// The service is as long as the turns of its period, so it is written for few operations and branches: a decided
// game is frozen in the turn (war_turn_tests), its outcome is one word from any source, what is rare (Brent's own
// finds, their recording, checkpoints) is behind one branch, a miss goes to one of two slots in shared memory, both
// histograms are one array, and what a unit's games share is prepared once per (unit, split).
//
// What bounds it: instruction issue (12! deals of 13 cards: ALU pipe 82%, issue 75%, beside random accesses at 0.9 of
// the random-gather ceiling), and for jobs of fewer than about 1e6 games the longest game.  Measured on a B200 (states
// at services -> landmarks -> a found cycle recorded by playing on instead of by a walk -> this service and turn): a
// span of 4.26e9 deals of 15 cards 210 -> 132 -> 85 -> 81 ms (stores 3.4e9 -> 1.0e9), 1e8 deals of 13 cards 2.5 -> 2.0
// -> 1.6 -> 1.5 ms, a resumed a(13) 31.2 -> 30.5 -> 29.9 -> 28.8 ms, --half span of 14 cards 13.7 -> 12.9 ms, 3e9
// canonical positions of 14 cards 152 -> 148 -> 148 -> 143 ms and 125 with the queue of starts; with services every 16
// turns from 15 cards and the later steps of the turn (war_turn_tests) 70.3, 1.42, 27.9, 11.9 and 123.6 ms.  The
// one-deal-one-game kernel before: 370, 10.7, 168, 124 and 164 ms.
#pragma once
#include "war_refill.cuh"
#include "war_merge.cuh"

namespace war {

// The units of a block's warps.
union UnitStore {
    MUnit m[32];
    CUnit c[32];
};

// One game slot of the merged kernel.  next: Brent's next checkpoint, or RECORDING, or IDLE for a lane without a game.
struct MGame {
    u64 w1, w2, t1, t2, m1, m2;   // piles, tortoise, the last landmark
    u32 q, rounds, next, wt, mv, at, missed;
};

// The hashes of a game's last two landmarks looked up and missed, and their turns, kept in shared memory: the k-th
// miss in slot k mod 2.
struct Missed {
    u64 h[2];
    u32 t[2];
};
constexpr u32 NO_LANDMARK = 0xFFFFFFFFu;
// A game whose cycle Brent found plays on around it once more, to the tortoise's state again, and its services store
// the cycle's landmarks instead of looking them up: the other lanes go on meanwhile, where a walk of the cycle at
// once holds them up.  (As checkpoints, these are never reached.)
constexpr u32 RECORDING = 0xFFFFFFFFu, IDLE = 0xFFFFFFFEu;

// The table: its words, log2 of their number, the largest value, and the key's constants (memo_key_state): the cards
// that a key holds, and 4(n-1) as a factor.
struct MemoTable {
    u64* T;
    u32 bits, vmask, lenlo, lenhi;
    u64 cards;
    __device__ __forceinline__ MemoTable(u64* t, u32 b, u32 n) : T(t), bits(b), vmask((1u << b) - 1u) {
        const u32 kb = 4u * (n - 1u);
        cards = (1ull << kb) - 1ull;
        lenlo = (u32)(1ull << kb);
        lenhi = (u32)((1ull << kb) >> 32);
    }
    // The hash of a state: memo_key_state(w1, w2) * MEMO_MUL, with the length field added by multiply-adds.
    __device__ __forceinline__ u64 hash(u64 w1, u64 w2) const {
        const bool sw = w2 < w1;
        const u64 h = sw ? w2 : w1, o = sw ? w1 : w2;
        const u32 len = pile_len(h);
        const u64 k = (h ^ ((o ^ 1ull) << (4u * len))) & cards;      // (the sentinel of h goes with o's lowest bit)
        return (((u64)(len * lenhi + (u32)(k >> 32)) << 32) | (len * lenlo + (u32)k)) * MEMO_MUL;
    }
    __device__ __forceinline__ u64* word(u64 h) const { return T + ((u32)(h >> 32) >> (32u - bits)); }
    __device__ __forceinline__ void store(u64 h, u32 v) const {
        __stcg((unsigned long long*)word(h), (unsigned long long)((h << bits) | v));
    }
    // The missed landmarks of a decided game, with its outcome: 2 lam (and the like) for a cycle, else 2 len + 1, from
    // a landmark 2 (turns left) + 1.  Returns the entries stored.
    __device__ __forceinline__ u32 store_missed(const Missed& x, u32 missed, u32 out) const {
        u32 k = 0;
#pragma unroll
        for (u32 i = 0; i < 2u; i++) {
            const u32 v = out - ((out & 1u) ? 2u * x.t[i] : 0u);
            if (missed > i && v <= vmask) { store(x.h[i], v); k++; }
        }
        return k;
    }
};

template <int RULE>
__device__ __forceinline__ void merge_body(const MergeArgs& a, DevAcc* __restrict__ acc, u64* __restrict__ counter,
                                           UnitStore& store, u64* sh64) {
    Missed* const miss = (Missed*)sh64 + threadIdx.x;
    u32* const sh = (u32*)((Missed*)sh64 + blockDim.x);      // cycle lengths, then ending lengths
    const u32 hbins = (u32)a.hbins;
    const int bins = a.hbins + WAR_EBINS;
    for (int b = threadIdx.x; b < bins; b += blockDim.x) sh[b] = 0;
    __syncthreads();

    const u32 n = (u32)a.n, h = n >> 1, W = (u32)a.W, n2 = 2u * n;
    const TestK K = a.tk;
    const u32 hb1 = hbins ? hbins - 1u : 0u;
    const u32 period = a.defer > 4 ? (u32)((a.defer + 3) & ~3) : 4u;
    const MemoTable memo(a.memo, a.memo_bits, n);
    const bool table = a.memo != nullptr;
    const u64 pat = 0x1111111111111111ull * (u64)(n - 1u);
    const u32 lane = threadIdx.x & 31u;
    MUnit& mu = store.m[threadIdx.x >> 5];

    MCursor c;
    u32 cyc = 0, turns = 0, maxfin = 0, capped = 0, mlook = 0, mhit = 0, mstore = 0;
    MGame g;
    g.w1 = g.w2 = 1ull; g.m1 = g.m2 = 0ull; g.rounds = g.mv = g.wt = g.missed = 0; g.at = NO_LANDMARK;

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
    auto split = [&]() {
        const u32 a8 = 8u * c.pa, q1 = mu.s1 + a8, q2 = mu.s2 + 8u * c.f - a8;
        const u64 A1 = mu.U1 | shl64(1ull, q1), A2 = mu.U2 | shl64(1ull, q2);
        __syncwarp();
        if (lane == 0u) {
            mu.A1 = A1; mu.A2 = A2;
            mu.mask = ~shl64(~0ull, a8);
            mu.at = 8u * (c.f - c.fi);
            mu.a8 = a8;
        }
        __syncwarp();
    };
    auto over = [&]() -> u32 {
        return mu.s2 + 8u * (c.f - c.pa) == 0u ? 1u : (mu.s1 + 8u * c.pa == 0u ? 2u : 0u);
    };
    auto ended = [&](u32 k) {
        if (lane == 0u) atomicAdd(&sh[hbins + h], k);
        maxfin = max(maxfin, h);
    };
    auto build = [&](u32 sel) -> bool {
        const u32 a8 = mu.a8, s1 = mu.s1;
        const u64 lw = mu.O | shl64((u64)merge_row(mu.c0, mu.c1, sel), mu.at);
        const u64 w1 = mu.A1 | shl64(lw & mu.mask, s1), w2 = mu.A2 | shl64(shr64(lw, a8), mu.s2);
        if (c.filter) {   // player 1 must hold card n - 1
            const u64 x = w1 ^ pat;
            if (((x - 0x1111111111111111ull) & ~x & 0x8888888888888888ull) == 0ull) return false;
        }
        g.w1 = g.t1 = w1; g.w2 = g.t2 = w2;
        g.q = s1 + a8 - n2;
        g.rounds = h; g.next = 2u * h + W;
        g.mv = 0; g.wt = c.wt; g.missed = 0;
        return true;
    };
    auto refill = [&](u32 need) {
        if ((need >> lane) & 1u) { g.next = IDLE; g.q = FROZEN; g.t1 = g.t2 = ~0ull; }
        merge_deal(c, a, counter, need, setup, split, over, ended, build, drain);
    };

    refill(WAR_FULL_MASK);
    bool running = __any_sync(WAR_FULL_MASK, g.next != IDLE);
    while (running) {
        u32 ev = NO_EVENT;
        g.at = NO_LANDMARK;
        for (u32 k2 = 0; k2 < 2u * period; k2 += 8u) {
            war_turn_tests<RULE, 0, true>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, n - 1u, K);
            war_turn_tests<RULE, 1, true>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, n - 1u, K);
            war_turn_tests<RULE, 2, true>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, n - 1u, K);
            war_turn_tests<RULE, 3, true>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, n - 1u, K);
        }
        // out: a decided game's outcome, 2 lam for a cycle, 2 len + 1 for an end
        const u32 base = g.rounds;
        const bool open = ev == NO_EVENT;
        g.rounds = base + (open ? period : (ev >> 1) + 1u);
        bool fin = !open;
        u32 out = (ev & 1u) ? 2u * g.rounds + 1u : g.mv;
        const bool mark = open & (g.at != NO_LANDMARK);
        const u32 at = base + (g.at >> 1);
        u64 hash = 0;
        if (table) hash = memo.hash(g.m1, g.m2);
        if (open ? (g.rounds >= g.next || (g.next == RECORDING && mark)) : out == 0u) {
            if (!open) {                         // Brent found the cycle: record it
                out = 2u * (g.rounds - ((g.next - W) >> 1));
                if (table && out <= memo.vmask) {
                    fin = false;
                    g.mv = out; g.next = RECORDING;
                    g.w1 = g.t1; g.w2 = g.t2; g.q = 4u * pile_len(g.t1) - n2;   // (the game stands frozen)
                }
            } else if (g.next == RECORDING) {
                memo.store(hash, g.mv);
                mstore++;
            } else if (g.next > WAR_TURN_CAP) {  // abandoned (never expected): the job fails
                capped++; fin = true; out = 1u;
            } else {                             // Brent's checkpoint (war_refill.cuh)
                g.t1 = g.w1; g.t2 = g.w2; g.next = 2u * g.rounds + W;
            }
        }
        const bool look = table & mark & (g.next < IDLE);
        u64 e = 0;
        if (look) e = __ldcg((const unsigned long long*)memo.word(hash));
        e ^= hash << memo.bits;                  // the value, if the entry is the landmark's
        const u32 v = (u32)e;
        const bool hit = look & ((u32)(e >> 32) == 0u) & (v - 1u < memo.vmask);
        mlook += look ? 1u : 0u;
        mhit += hit ? 1u : 0u;
        if (hit) out = v + ((v & 1u) ? 2u * at : 0u);
        if (look & !hit) {
            miss->h[g.missed & 1u] = hash;
            miss->t[g.missed & 1u] = at;
            g.missed++;
        }
        fin = fin | hit;
        const u32 need = __ballot_sync(WAR_FULL_MASK, fin);
        if (need) {
            if (fin) {
                const bool cy = (out & 1u) == 0u;
                turns += g.rounds - h;
                if (g.missed) mstore += memo.store_missed(*miss, g.missed, out);
                const u32 len = out >> 1, bin = cy ? min(len, hb1) : hbins + min(len, (u32)WAR_EBINS - 1u);
                if (!cy | (hbins != 0u)) atomicAdd(&sh[bin], g.wt);
                cyc += cy ? g.wt : 0u;
                maxfin = max(maxfin, cy ? 0u : len);
            }
            refill(need);
            running = __any_sync(WAR_FULL_MASK, g.next != IDLE);
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
    flush_hist(sh, acc->hist, a.hbins);
    flush_hist(sh + hbins, acc->endhist, WAR_EBINS);
}

// ---- canonical scans ----------------------------------------------------------------------------------
//
// The same loop for canonical positions with the path memo, one game each.  EXTRA: the distinct-cycle outputs and
// the sample (gpu/war_gpu.py:217-235); SHAPE: the loop-shape test, whose code travels in the memo with the cycle
// length (war_refill.cuh).  Whether the start of a game lies on its cycle (distinct): Brent's first window compares
// every state up to turn W with the start; the starts of games that the memo decides are queued and walked around
// 32 at a time, without the tests of the loop (playing such games on to turn lam cost a fifth of the n = 14 scan, where
// 3% of the positions cycle).
//
// What bounds it: instruction issue and the random reads of the table, about equally; in a small scan the number
// of warps at work, which is why a warp, not a lane, takes a unit (a lane of the kernel it replaces played 120
// orders with all their splits alone).  B200: 2e6 positions of 11 cards 8.9 -> 0.40 ms, 3e9 of 14 cards 164 ->
// 152 ms (defer 16; 12: 156, 8: 176 ms; 256 to 1024 threads alike).
struct CGame {
    u64 w1, w2, t1, t2, m1, m2;
    u32 q, rounds, next, mv, at, missed;
    bool sampled, first;          // first: on its cycle from the start
};

// Starts of a warp's games that the memo found to cycle, with their cycle lengths, until 32 of them are walked
// around together to see which lie on their cycle.
struct StartQueue {
    u64 s1[64], s2[64];
    u32 lam[64];
};

template <int RULE, bool EXTRA, bool SHAPE>
__device__ __forceinline__ void canon_body(const MergeArgs& a, DevAcc* __restrict__ acc, u64* __restrict__ counter,
                                           UnitStore& store, u64* sh64) {
    Missed* const miss = (Missed*)sh64 + threadIdx.x;
    u64* const starts = (u64*)((Missed*)sh64 + blockDim.x);             // EXTRA: the starting piles,
    StartQueue* const queues = (StartQueue*)(starts + (EXTRA ? 2u * blockDim.x : 0u));   // and the warps' queues
    StartQueue& queue = queues[threadIdx.x >> 5];
    u32* const sh = (u32*)(queues + (EXTRA ? blockDim.x >> 5 : 0u));     // cycle lengths, then ending lengths
    const u32 hbins = (u32)a.hbins;
    const int bins = a.hbins + WAR_EBINS;
    for (int b = threadIdx.x; b < bins; b += blockDim.x) sh[b] = 0;
    __syncthreads();

    const u32 n = (u32)a.n, m = n - 1u, k4m4 = 4u * m, W = (u32)a.W, n2 = 2u * n;
    const TestK K = a.tk;
    const u32 hb1 = hbins ? hbins - 1u : 0u;
    const u32 period = a.defer > 4 ? (u32)((a.defer + 3) & ~3) : 4u;
    const MemoTable memo(a.memo, a.memo_bits, n);
    const bool table = a.memo != nullptr;
    constexpr u32 lsh = SHAPE ? 3u : 1u;                               // a memo value: 8 lam + 2 code, or 2 lam
    const u32 lane = threadIdx.x & 31u;
    CUnit& cu = store.c[threadIdx.x >> 5];

    MCursor c;
    u32 cyc = 0, turns = 0, maxfin = 0, capped = 0, mlook = 0, mhit = 0, mstore = 0, nonstd = 0, unchk = 0;
    u32 sc = 0, scy = 0, slam = 0, slen = 0, smax = 0, oncyc = 0, dmin = 0;
    CGame g;
    g.w1 = g.w2 = 1ull; g.m1 = g.m2 = 0ull; g.rounds = g.mv = g.missed = 0; g.at = NO_LANDMARK;
    g.sampled = g.first = false;

    // (A launch plays fewer than 2^32 positions: no bin and no total of a lane or warp can wrap.)
    auto drain = [&]() {};
    auto setup = [&](const MBlock& B, u64 outer) {
        CUnit u;
        canon_unit(B, outer, m, u);
        __syncwarp();
        if (lane == 0u) cu = u;
        __syncwarp();
    };
    auto split = [&]() {   // canon_position (war_core.cuh) of split c.pa without the other cards
        __syncwarp();
        if (lane == 0u) {
            cu.A1 = (u64)m | (1ull << (4u * (c.pa + 1u)));
            cu.A2 = 1ull << (4u * (m - c.pa));
            cu.mask = ~shl64(~0ull, 4u * c.pa);
            cu.at = 4u * (m - c.fi);
            cu.k4 = 4u * c.pa;
        }
        __syncwarp();
    };
    // a start on its cycle of length lam: the distinct-cycle counts (gpu/war_gpu.py:217-235)
    auto on_cycle = [&](u64 s1, u64 s2, u32 lam) {
        const CycleWalk cw = cycle_walk<RULE>(s1, s2, 4u * pile_len(s1), n, lam);
        oncyc++;
        if (cw.is_min) dmin++;
        if (a.dbins) {
            const u32 d = cw.sym ? cw.c1 : cw.c1 + cw.c2, db1 = (u32)(a.dbins - 1);
            atomicAdd(&acc->dhist[d < db1 ? d : db1], 1ull);
        }
    };
    // walks up to 32 queued starts around, one per lane
    u32 queued = 0;
    auto walk_queue = [&]() {
        __syncwarp();
        const u32 k = min(queued, 32u);
        queued -= k;
        if (lane < k) {
            const u64 s1 = queue.s1[queued + lane], s2 = queue.s2[queued + lane];
            const u32 lam = queue.lam[queued + lane];
            u64 v1 = s1, v2 = s2;
            u32 q = 4u * pile_len(s1) - n2;
            for (u32 t = 0; t < lam; t++) war_turn_fma<RULE>(v1, v2, q, K);
            if (v1 == s1 && v2 == s2) on_cycle(s1, s2, lam);
        }
        __syncwarp();
    };
    auto over = []() -> u32 { return 0u; };
    auto ended = [](u32) {};
    auto build = [&](u32 sel) -> bool {
        const u64 q = cu.Q | shl64((u64)merge_row(cu.c0, cu.c1, sel), cu.at);
        const u32 k4 = cu.k4;
        g.w1 = g.t1 = cu.A1 | ((q & cu.mask) << 4);
        g.w2 = g.t2 = cu.A2 | shr64(q, k4);
        g.q = k4 + 4u - n2;
        g.rounds = 0; g.next = W;
        g.mv = 0; g.missed = 0; g.first = false;
        if (EXTRA) {
            starts[threadIdx.x] = g.w1;
            starts[threadIdx.x + blockDim.x] = g.w2;
            g.sampled = a.sample && war_pick(a.seed, a.thr, g.w1, g.w2);
        }
        return true;
    };
    auto refill = [&](u32 need) {
        if ((need >> lane) & 1u) { g.next = IDLE; g.q = FROZEN; g.t1 = g.t2 = ~0ull; }
        merge_deal<true>(c, a, counter, need, setup, split, over, ended, build, drain);
    };

    refill(WAR_FULL_MASK);
    bool running = __any_sync(WAR_FULL_MASK, g.next != IDLE);
    while (running) {
        u32 ev = NO_EVENT;
        g.at = NO_LANDMARK;
        for (u32 k2 = 0; k2 < 2u * period; k2 += 8u) {
            war_turn_tests<RULE, 0, false>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, m, K);
            war_turn_tests<RULE, 1, false>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, m, K);
            war_turn_tests<RULE, 2, false>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, m, K);
            war_turn_tests<RULE, 3, false>(g.w1, g.w2, g.q, g.t1, g.t2, g.m1, g.m2, g.at, ev, k2, m, K);
        }
        // out: a decided game's outcome, the memo value of a cycle, 2 len + 1 for an end
        const u32 base = g.rounds;
        const bool open = ev == NO_EVENT;
        g.rounds = base + (open ? period : (ev >> 1) + 1u);
        bool fin = !open;
        u32 out = (ev & 1u) ? 2u * g.rounds + 1u : g.mv;
        const bool mark = open & (g.at != NO_LANDMARK);
        const u32 at = base + (g.at >> 1);
        u64 hash = 0;
        if (table) hash = memo.hash(g.m1, g.m2);
        if (open ? (g.rounds >= g.next || (g.next == RECORDING && mark)) : out == 0u) {
            if (!open) {                         // Brent found the cycle: record it
                const u32 lam = g.rounds - ((g.next - W) >> 1);
                out = 2u * lam;
                if (SHAPE)
                    out = 8u * lam + 2u * (u32)loop_shape_walk<RULE>(g.t1, g.t2, 4u * pile_len(g.t1), k4m4, lam, (u32)a.blk);
                g.first = g.next == W;
                if (table && out <= memo.vmask) {
                    fin = false;
                    g.mv = out; g.next = RECORDING;
                    g.w1 = g.t1; g.w2 = g.t2; g.q = 4u * pile_len(g.t1) - n2;   // (the game stands frozen)
                }
            } else if (g.next == RECORDING) {
                memo.store(hash, g.mv);
                mstore++;
            } else if (g.next > WAR_TURN_CAP) {  // abandoned (never expected): the job fails
                capped++; fin = true; out = 1u;
            } else {                             // Brent's checkpoint (war_refill.cuh)
                g.t1 = g.w1; g.t2 = g.w2; g.next = 2u * g.rounds + W;
            }
        }
        const bool look = table & mark & (g.next < IDLE);
        u64 e = 0;
        if (look) e = __ldcg((const unsigned long long*)memo.word(hash));
        e ^= hash << memo.bits;                  // the value, if the entry is the landmark's
        const u32 v = (u32)e;
        const bool hit = look & ((u32)(e >> 32) == 0u) & (v - 1u < memo.vmask);
        mlook += look ? 1u : 0u;
        mhit += hit ? 1u : 0u;
        if (look & !hit) {
            miss->h[g.missed & 1u] = hash;
            miss->t[g.missed & 1u] = at;
            g.missed++;
        }
        if (hit) out = v + ((v & 1u) ? 2u * at : 0u);
        fin = fin | hit;
        const u32 need = __ballot_sync(WAR_FULL_MASK, fin);
        if (need) {
            bool push = false;
            if (fin) {
                const bool cy = (out & 1u) == 0u;
                const u32 len = cy ? out >> lsh : out >> 1;
                turns += g.rounds;
                if (SHAPE && cy) {
                    const u32 code = (out >> 1) & 3u;
                    if (code == 1u) nonstd++;
                    if (code == 2u) unchk++;
                }
                if (g.missed) mstore += memo.store_missed(*miss, g.missed, out);
                const u32 bin = cy ? min(len, hb1) : hbins + min(len, (u32)WAR_EBINS - 1u);
                if (!cy | (hbins != 0u)) atomicAdd(&sh[bin], 1u);
                cyc += cy ? 1u : 0u;
                maxfin = max(maxfin, cy ? 0u : len);
                if (EXTRA && cy && a.distinct) {
                    if (g.first) on_cycle(starts[threadIdx.x], starts[threadIdx.x + blockDim.x], len);
                    // if Brent's first window saw lam turns pass, it would have seen the start again
                    push = !g.first && (len > W || g.rounds < len);
                }
                if (EXTRA && g.sampled) {
                    sc++;
                    if (cy) { scy++; slam += len; }
                    else { slen += len; smax = max(smax, len); }
                }
            }
            if (EXTRA && a.distinct) {
                const u32 pb = __ballot_sync(WAR_FULL_MASK, push);
                if (push) {
                    const u32 i = queued + (u32)__popc(pb & ((1u << lane) - 1u));
                    queue.s1[i] = starts[threadIdx.x];
                    queue.s2[i] = starts[threadIdx.x + blockDim.x];
                    queue.lam[i] = out >> lsh;
                }
                queued += (u32)__popc(pb);
                if (queued >= 32u) walk_queue();
            }
            refill(need);
            running = __any_sync(WAR_FULL_MASK, g.next != IDLE);
        }
    }

    if (EXTRA) while (queued) walk_queue();

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
    flush_hist(sh, acc->hist, a.hbins);
    flush_hist(sh + hbins, acc->endhist, WAR_EBINS);
}

}  // namespace war

// war_wide.cu — the 5-bit-pile engine: deals of up to 20 cards (gpu/war24.py).
//
// Past 16 cards a pile no longer fits one 64-bit word of 4-bit cards.  gpu/war24.py keeps 5-bit cards in
// two 64-bit words (lo, hi) with explicit lengths and counts every deal of n <= 20 cards (deal ranks are
// 64-bit) with one of two cycle tests under a step cap (gpu/war24.py:31-125).  This engine plays the same
// games with the refill design of the 4-bit engine:
//
// * Sentinel piles of 5-bit cards.  A pile of len cards is a 128-bit value (two u64): card i (0 = top) in
//   bits 5i..5i+4 and a single 1 bit at bit 5*len, so the length is part of the words and two positions are
//   equal exactly when their four words are.  A turn pops both tops (a 128-bit shift right by 5), compares
//   them and XORs (pair ^ 0x401) << pos into the winner's words, where pos is the winner's sentinel after
//   the pop: the pair replaces the sentinel and a new sentinel appears 10 bits higher.  No branches; the
//   variable 128-bit shift is two clamped 64-bit shifts (PTX shl/shr give 0 for amounts of 64 or more).
// * Refill.  A persistent grid of SMs x resident blocks; each lane plays one game at a time and every K
//   turns the warp services its lanes together: a decided game is recorded and the lane takes its next deal.
//   Outcomes are latched, so the turn loop has no branch on them.
// * Enumeration.  Work units of j! consecutive lexicographic ranks (a fixed prefix and every order of the
//   last j positions) come from one atomic counter; a lane unranks the unit's first deal once and walks the
//   unit in Heap's order (one transposition per deal).  The deck is held split: player 1's cards (even
//   deck positions) in one word and player 2's (odd positions) in another, 5 bits per card, so a deal is
//   the two words plus their sentinels.
// * Detectors (template DET), each with the step cap after which a game counts as undetermined:
//   Brent with the tortoise saved at turns W, 3W, 7W, ... (the default; its cycle length feeds the
//   histogram), Floyd's tortoise and hare (gpu/war24.py:85-97), and the streak test for odd n
//   (gpu/war24.py:98-125): anchor where the next winner holds an even number of cards, then expect the
//   players to alternate for lcm(n+1, W, L-1) turns and compare with the anchor.  Every detector gives the
//   same counts whenever nothing reaches the cap; the step count of an ending game is its length.
#include <algorithm>
#include <cstring>
#include <mutex>
#include "war_kernels.cuh"
#include "war_host.h"
#include "war_merge.cuh"

namespace war {

enum { DET_BRENT = 0, DET_FLOYD = 1, DET_STREAK = 2 };
enum { K_NONE = 0, K_END = 1, K_CYC = 2, K_UND = 3 };

// One turn on 128-bit sentinel piles (a0, a1) and (b0, b1); la = player 1's length, n1 = n - 1.  Returns
// true if player 1 won.  Rule 0 puts the winning card, then the losing card, under the winner's pile
// (gpu/war24.py:42-47); rule 1 the losing card first.
template <int RULE>
__device__ __forceinline__ bool turn5(u64& a0, u64& a1, u64& b0, u64& b1, u32& la, u32 n1) {
    const u32 c1 = (u32)a0 & 31u, c2 = (u32)b0 & 31u;
    a0 = (a0 >> 5) | (a1 << 59); a1 >>= 5;
    b0 = (b0 >> 5) | (b1 << 59); b1 >>= 5;
    const bool p1 = c1 > c2;
    const u32 hi = max(c1, c2), lo = min(c1, c2);
    const u32 pair = RULE ? (lo | (hi << 5)) : (hi | (lo << 5));
    const u32 pos = 5u * (p1 ? la - 1u : n1 - la);
    const u64 v = (u64)(pair ^ 0x401u);
    const u64 x0 = shl64(v, pos), x1 = shl64(v, pos - 64u) | shr64(v, 64u - pos);
    const u64 m = p1 ? ~0ull : 0ull;
    a0 ^= x0 & m; a1 ^= x1 & m;
    b0 ^= x0 & ~m; b1 ^= x1 & ~m;
    la = p1 ? la + 1u : la - 1u;
    return p1;
}

// The work units of a launch, as in the 4-bit engine (BatchArgs), with the 5-bit engine's own fields.
struct WideArgs {
    u64 fact[21];
    u64 main_base, main_count, n_units;
    const Unit* units;
    int n, m, rule, hbins, W, defer;
    u32 cap;            // step cap: a game undecided after this many turns is undetermined
    u32 lamtab[32];     // streak: lcm(n+1, ws, n-ws-1) for an even next-winner pile ws with n-ws >= 2, else 0
};

__device__ __forceinline__ u32 wide_heap_full(u32 j) {   // Heap counter value of a unit's last order
    u32 f = 0;
    for (u32 i = 1; i < j; i++) f |= i << (4u * i);
    return f;
}

struct WEnum {
    u64 A, B;           // the current deal: player 1's cards (even positions), player 2's (odd), 5 bits each
    u32 ctr, full, base;
    bool live;
};

// Swaps deck positions x and y of the split deck.
__device__ __forceinline__ void swap5(u64& A, u64& B, u32 x, u32 y) {
    const u32 sx = 5u * (x >> 1), sy = 5u * (y >> 1);
    const bool bx = x & 1u, by = y & 1u;
    const u64 t = (((bx ? B : A) >> sx) ^ ((by ? B : A) >> sy)) & 31ull;
    const u64 tx = t << sx, ty = t << sy;
    A ^= (bx ? 0ull : tx) ^ (by ? 0ull : ty);
    B ^= (bx ? tx : 0ull) ^ (by ? ty : 0ull);
}

__device__ __forceinline__ bool wide_fetch(WEnum& E, const WideArgs& a, u64* counter) {
    const u64 u = atomicAdd(counter, 1ull);
    if (u >= a.n_units) return false;
    u64 r;
    u32 j;
    if (u < a.main_count) {
        j = (u32)a.m; r = (a.main_base + u) * a.fact[a.m];
    } else {
        const Unit U = a.units[u - a.main_count];
        r = U.r; j = U.j;
    }
    // lexicographic unrank (gpu/war24.py:60-74) straight into the split deck
    const int n = a.n;
    u32 avail = (1u << n) - 1u;
    u64 A = 0, B = 0;
    for (int i = 0; i < n; i++) {
        const u64 f = a.fact[n - 1 - i];
        const u32 d = (u32)(r / f);
        r -= (u64)d * f;
        u32 mm = avail;
        for (u32 k = 0; k < d; k++) mm &= mm - 1u;
        const u32 v = (u32)(__ffs((int)mm) - 1);
        avail &= ~(1u << v);
        if (i & 1) B |= (u64)v << (5 * (i >> 1));
        else A |= (u64)v << (5 * (i >> 1));
    }
    E.A = A; E.B = B;
    E.ctr = 0;
    E.full = wide_heap_full(j);
    E.base = (u32)n - j;
    E.live = true;
    return true;
}

// Heap's algorithm, one output (as heap_step of the 4-bit engine); false after the unit's last deal.
__device__ __forceinline__ bool wide_heap_step(WEnum& E) {
    const u32 x = E.ctr ^ E.full;
    if (x == 0u) return false;
    const u32 i = (u32)(__ffs((int)x) - 1) >> 2;
    const u32 ci = (E.ctr >> (4u * i)) & 15u;
    const u32 o = (i & 1u) ? ci : 0u;
    swap5(E.A, E.B, E.base + i, E.base + o);
    E.ctr = ((E.ctr >> (4u * i)) + 1u) << (4u * i);
    return true;
}

// One game per deal: for jobs whose games cannot be merged (wide_merged, below).
// SVC (Brent only): W is a multiple of the service period, so an undecided game (which starts at a service and
// plays `period` turns between services) reaches each tortoise checkpoint W, 3W, 7W, ... exactly at a service,
// and the checkpoint is saved there instead of being tested after every turn (2e7 deals of 19 cards with a window and
// a period of 8: 74 ms, tested 102).
template <int RULE, int DET, bool SVC>
__global__ void __launch_bounds__(1024) wide_kernel(const __grid_constant__ WideArgs a, DevAcc* __restrict__ acc) {
    extern __shared__ u32 sh[];
    u32* shh = sh;                    // cycle-length histogram (Brent)
    u32* she = sh + a.hbins;          // ending-length histogram
    u32* slam = she + WAR_EBINS;      // streak periods by pile size
    for (int b = threadIdx.x; b < a.hbins + WAR_EBINS; b += blockDim.x) sh[b] = 0;
    if (threadIdx.x < 32) slam[threadIdx.x] = a.lamtab[threadIdx.x];
    __syncthreads();

    const u32 n = (u32)a.n, n1 = n - 1u, W = (u32)a.W, cap = a.cap;
    const u32 hb1 = a.hbins > 0 ? (u32)(a.hbins - 1) : 0u;
    const int period = a.defer > 4 ? (a.defer + 3) & ~3 : 4;
    const u32 lenA = (n + 1u) / 2u, lenB = n / 2u;
    const u64 sA = 1ull << (5u * lenA), sB = 1ull << (5u * lenB);
    u64* counter = &acc->work_next;

    WEnum E;
    E.live = false;
    // the game: piles, player 1's length, turns played, outcome
    u64 a0 = 0, a1 = 0, b0 = 0, b1 = 0;
    u32 la = 0, rounds = 0, kind = K_NONE;
    bool active = false;
    // detector state: tortoise (Brent, Floyd) or anchor (streak)
    u64 t0 = 0, t1 = 0, t2 = 0, t3 = 0;
    u32 tla = 0, next = 0, lam = 0, since = 0, prevw = 2u;
    bool anch = false;
    // per-lane totals
    u32 cyc = 0, done = 0, maxfin = 0, und = 0;
    u64 turns = 0;

    auto start = [&]() {
        if (!E.live && !wide_fetch(E, a, counter)) { active = false; kind = K_END; return; }
        a0 = E.A | sA; a1 = 0; b0 = E.B | sB; b1 = 0; la = lenA;
        E.live = wide_heap_step(E);
        active = true;
        done++;
        rounds = 0; kind = K_NONE;
        t0 = a0; t1 = a1; t2 = b0; t3 = b1; tla = la;
        next = W; lam = 0; since = 0; prevw = 2u; anch = false;
    };
    start();
    bool running = __any_sync(WAR_FULL_MASK, active);

    while (running) {
        for (int k = 0; k < period; k++) {
            const bool open = kind == K_NONE;
            if (DET == DET_FLOYD) {
                // two hare turns, one tortoise turn (gpu/war24.py:88-96)
                turn5<RULE>(a0, a1, b0, b1, la, n1);
                const bool e1 = (la == 0u) | (la == n);
                turn5<RULE>(a0, a1, b0, b1, la, n1);
                const bool e2 = (la == 0u) | (la == n);
                turn5<RULE>(t0, t1, t2, t3, tla, n1);
                const bool cy = (a0 == t0) & (a1 == t1) & (b0 == t2) & (b1 == t3);
                const u32 r2 = rounds + (e1 ? 1u : 2u);
                const u32 kk = (e1 | e2) ? (u32)K_END : (cy ? (u32)K_CYC : (r2 > cap ? (u32)K_UND : (u32)K_NONE));
                rounds = open ? r2 : rounds;
                kind = open ? kk : kind;
            } else if (DET == DET_STREAK) {
                // anchor where the next winner holds an even number of cards (gpu/war24.py:104-112)
                if (!anch) {
                    const u32 ws = ((u32)a0 & 31u) > ((u32)b0 & 31u) ? la : n - la;
                    // (a lane whose game is decided keeps stepping it until the service, so its pile
                    // length may leave 0..n: the mask keeps the read inside the 32-entry table)
                    const u32 lt = slam[ws & 31u];
                    if (lt) { anch = true; since = 0; prevw = 2u; lam = lt; t0 = a0; t1 = a1; t2 = b0; t3 = b1; }
                }
                const u32 w = turn5<RULE>(a0, a1, b0, b1, la, n1) ? 1u : 0u;
                bool cy = false;
                if (anch) {   // the players must alternate for lam turns (gpu/war24.py:114-123)
                    if (w == prevw) anch = false;
                    else {
                        prevw = w;
                        if (++since == lam) {
                            cy = (a0 == t0) & (a1 == t1) & (b0 == t2) & (b1 == t3);
                            anch = false;
                        }
                    }
                }
                const u32 r1 = rounds + 1u;
                const bool en = (la == 0u) | (la == n);
                const u32 kk = cy ? (u32)K_CYC : (en ? (u32)K_END : (r1 > cap ? (u32)K_UND : (u32)K_NONE));
                rounds = open ? r1 : rounds;
                kind = open ? kk : kind;
            } else {
                turn5<RULE>(a0, a1, b0, b1, la, n1);
                const u32 r1 = rounds + 1u;
                const bool en = (la == 0u) | (la == n);
                const bool cy = (a0 == t0) & (a1 == t1) & (b0 == t2) & (b1 == t3);
                const u32 kk = en ? (u32)K_END : (cy ? (u32)K_CYC : (r1 > cap ? (u32)K_UND : (u32)K_NONE));
                rounds = open ? r1 : rounds;
                kind = open ? kk : kind;
                if (!SVC && open && kk == K_NONE && r1 == next) {   // Brent: tortoise saved at W, 3W, 7W, ...
                    t0 = a0; t1 = a1; t2 = b0; t3 = b1; next = 2u * next + W;
                }
            }
        }
        if (DET == DET_BRENT && SVC && kind == K_NONE && rounds == next) {   // the checkpoint, at the service
            t0 = a0; t1 = a1; t2 = b0; t3 = b1; next = 2u * next + W;
        }
        // service: record every decided game, refill its lane
        const bool fin = active & (kind != K_NONE);
        if (__any_sync(WAR_FULL_MASK, fin)) {
            if (fin) {
                turns += rounds;
                if (kind == K_CYC) {
                    cyc++;
                    if (DET == DET_BRENT && a.hbins) {
                        const u32 l = rounds - ((next - W) >> 1);
                        atomicAdd(&shh[l < hb1 ? l : hb1], 1u);
                    }
                } else if (kind == K_END) {
                    if (rounds > maxfin) maxfin = rounds;
                    atomicAdd(&she[rounds < WAR_EBINS - 1 ? rounds : WAR_EBINS - 1], 1u);
                } else {
                    und++;
                }
                start();
            }
            running = __any_sync(WAR_FULL_MASK, active);
        }
    }

    const u64 v_cyc = warp_sum(cyc), v_done = warp_sum(done), v_turns = warp_sum(turns), v_max = warp_max(maxfin);
    const u64 v_und = warp_sum(und);
    if ((threadIdx.x & 31) == 0) {
        if (v_cyc) atomicAdd(&acc->cyc, v_cyc);
        if (v_done) atomicAdd(&acc->done, v_done);
        if (v_turns) atomicAdd(&acc->turns, v_turns);
        if (v_max) atomicMax(&acc->maxfin, v_max);
        if (v_und) atomicAdd(&acc->undetermined, v_und);
    }
    __syncthreads();
    flush_hist(shh, acc->hist, a.hbins);
    flush_hist(she, acc->endhist, WAR_EBINS);
}

// ---- merged games (war_merge.cuh) -----------------------------------------------------------------------
//
// wide_kernel plays every deal; this kernel plays each state after the deals' first h = floor(n/2) turns once,
// under any detector, and counts it for all its deals.
//
// `turns` stays what playing every deal gives.  Floyd meets at the first multiple of the cycle length that is no
// earlier than the cycle, the same turn for a deal on its own cycle (a cycle is longer than h turns), so the
// tortoise waits at turn h until the hare is at turn 2h and both go on from there.  Brent's checkpoints W, 3W, ..
// (all at or after turn h) decide all deals of a game at the same turn; a deal on its own cycle of length
// lam <= W is decided at turn lam by the checkpoint at turn 0 instead, and wide_start finds the one that is.
// With the tortoise at the state of turn h until turn W, a game on such a cycle is known at turn h + lam and
// counted as decided at W + lam.
//
// The streak test (odd n, winner's card first) needs no anchor of its own here.  The piles' sizes change parity
// every turn, so "the next winner holds an even number of cards" stays true, or stays false, as long as the
// players alternate, and flips at every turn that the same player wins again (a break).  The test's anchor is
// therefore the first turn of an alternating run in which it is true, and its period lcm(n+1, W, L-1) is the
// same all along the run.  While the players alternate a turn can be undone (the winner is known, and its pair
// is at the bottom of its pile), so a run that reaches its cycle was on it from its first turn, and the test
// succeeds at the first try: at the run's first turn + the period.  The kernel keeps the turn of the last break,
// saves the tortoise at the first service after it, finds the cycle one cycle length later and counts that turn.
// Where there was no break after turn h, the run began before it, for each deal of the game at its own turn:
// wide_streak_head sums those up.  (A cycle with breaks, or one in which the condition is false, is one that the
// test never finds: undetermined.)
//
// The step cap must not fall before the turns that are not played: at least 2W (Brent), 2h + 2 (Floyd), h + the
// longest period (streak).
//
// What bounds it: instruction issue of the turns; the gain over wide_kernel is the deals per game (3.2 in a block of
// 9! deals of 18 cards, 5.3 in one of 11!), in short jobs units that a whole warp plays instead of one lane, and a
// turn of half the operations (turn5_pred).  B200: 5e7 deals of 18 cards under Brent 45 -> 2.4 (turn5) -> 1.6 ms, 2e8
// of 17 under the streak test 125 -> 16.8 -> 10.3 ms (which also plays one cycle length after the last break instead
// of the period), 2e8 of 17 under Floyd 24.4 -> 15.3 ms; 256 or 512 threads alike, defer 16 (8: 1.8 and 11.7 ms, 32:
// 1.6 and 10.2 ms).
//
// Piles here are 96 bits (a u64 and a u32) of cards 1..n in 5 bits each, without a sentinel: no card is 0, so the
// words still tell the length, and 19 cards, the most a player can hold while the game goes on, fit.

// Constants of turn5_pred as operands (war_core.cuh, TurnK).
struct Turn5K {
    u32 one, m1, m32, k32, k2p27, c1, c2;   // 1, -1, -32, 32, 2^27, -5, 5n - 5
};

// One turn.  qa = 5 * player 1's length.  Both tops are popped (two funnel shifts and a multiply-high each, the
// card as lo - 32 lo'), the pair is built, placed and added to the winner's pile by multiply-adds, those of player 1's
// win under a predicate: 9 operations are left to the ALU pipe (turn5: about 35), 17 go to the FMA pipe, which
// balances the two with the loop's tests, which only the ALU pipe has.  Returns 1 if player 1 won.
template <int RULE>
__device__ __forceinline__ u32 turn5_pred(u64& a0, u32& a1, u64& b0, u32& b1, u32& qa, const Turn5K& K) {
    const u32 l1 = (u32)a0, h1 = (u32)(a0 >> 32), l2 = (u32)b0, h2 = (u32)(b0 >> 32);
    const u32 nl1 = __funnelshift_r(l1, h1, 5), nh1 = __funnelshift_r(h1, a1, 5);
    const u32 nl2 = __funnelshift_r(l2, h2, 5), nh2 = __funnelshift_r(h2, b1, 5);
    a1 = __umulhi(a1, K.k2p27);
    b1 = __umulhi(b1, K.k2p27);
    const u32 c1 = l1 + nl1 * K.m32, c2 = l2 + nl2 * K.m32;
    const u32 f = RULE ? c1 : c2, g = RULE ? c2 : c1;   // player 2 won: f first in the pair; player 1: g
    u64 x1 = ((u64)nh1 << 32) | nl1, x2 = ((u64)nh2 << 32) | nl2;
    u32 w;
    asm("{\n\t"
        ".reg .pred p;\n\t"
        ".reg .u32 t, ps, pt, xl, xh, yl, yh, al, ah, q;\n\t"
        ".reg .u64 x, y;\n\t"
        "setp.gt.u32 p, %6, %7;\n\t"
        "mad.lo.u32 t, %9, %10, %8;\n\t"         // f + 32 g
        "@p mad.lo.u32 t, %8, %10, %9;\n\t"      // g + 32 f
        "mad.lo.u32 ps, %4, %12, %14;\n\t"       // the place under the winner's pile after the pop
        "@p mad.lo.u32 ps, %4, %11, %13;\n\t"
        "mad.lo.u32 q, %4, %11, -5;\n\t"
        "@p mad.lo.u32 q, %4, %11, 5;\n\t"
        "mov.u32 %4, q;\n\t"
        "mad.lo.u32 pt, ps, %11, -32;\n\t"
        "cvt.u64.u32 x, t;\n\t"
        "shl.b64 y, x, pt;\n\t"
        "shl.b64 x, x, ps;\n\t"
        "mov.b64 {xl, xh}, x;\n\t"
        "mov.b64 {yl, yh}, y;\n\t"
        "@p mad.wide.u32 %0, xl, %11, %0;\n\t"
        "@!p mad.wide.u32 %2, xl, %11, %2;\n\t"
        "mov.b64 {al, ah}, %0;\n\t"
        "@p mad.lo.u32 ah, xh, %11, ah;\n\t"
        "mov.b64 %0, {al, ah};\n\t"
        "mov.b64 {al, ah}, %2;\n\t"
        "@!p mad.lo.u32 ah, xh, %11, ah;\n\t"
        "mov.b64 %2, {al, ah};\n\t"
        "@p mad.lo.u32 %1, yh, %11, %1;\n\t"
        "@!p mad.lo.u32 %3, yh, %11, %3;\n\t"
        "selp.u32 %5, 1, 0, p;\n\t"
        "}"
        : "+l"(x1), "+r"(a1), "+l"(x2), "+r"(b1), "+r"(qa), "=r"(w)
        : "r"(c1), "r"(c2), "r"(f), "r"(g), "r"(K.k32), "r"(K.one), "r"(K.m1), "r"(K.c1), "r"(K.c2));
    a0 = x1;
    b0 = x2;
    return w;
}

// The outer choice of a unit (MUnit with such cards and piles): the outer pairs have 10 bits each.
struct WUnit {
    u64 U1l, U2l, O;
    u32 U1h, U2h;
    u32 c0, c1, s1, s2;
    u32 wins;          // bit t: player 1 wins turn t (turns of the fixed cards)
};

// Adds v << s to a 96-bit pile; v << s may reach past bit 63 (s < 128).
__device__ __forceinline__ void put96(u64& lo, u32& hi, u64 v, u32 s) {
    lo |= shl64(v, s);
    hi |= (u32)(s < 64u ? shr64(v, 64u - s) : shl64(v, s - 64u));
}

template <int RULE>
__device__ __forceinline__ void wide_unit(const MBlock& B, u64 outer, u32 n, WUnit& m) {
    u32 free = B.free_mask;
    const u32 b = B.b, f = B.f, fo = f > MERGE_INNER ? f - MERGE_INNER : 0u;
    m.U1l = m.U2l = m.O = 0ull;
    m.U1h = m.U2h = 0u;
    u32 s1 = 0, s2 = 0, half = 0, wins = 0;
    if ((b & 1u) && b < n) {
        const u32 k = (u32)__popc(free);
        half = take_card(free, take_digit(outer, k)) + 1u;
    }
    if (n & 1u) {   // player 1's last card, unplayed after h turns, is on top
        if (b == n) m.U1l = B.prefix[n - 1u] + 1u;
        else {
            const u32 k = (u32)__popc(free);
            m.U1l = take_card(free, take_digit(outer, k)) + 1u;
        }
        s1 = 5u;
    }
    for (u32 t = 0; 2u * t < b && 2u * t + 1u < n; t++) {
        const u32 x = B.prefix[2u * t] + 1u, y = 2u * t + 1u < b ? B.prefix[2u * t + 1u] + 1u : half;
        const u32 hi = max(x, y), lo = min(x, y);
        const u64 pair = RULE ? lo | (hi << 5) : hi | (lo << 5);
        if (x > y) { put96(m.U1l, m.U1h, pair, s1); s1 += 10u; wins |= 1u << t; }
        else { put96(m.U2l, m.U2h, pair, s2); s2 += 10u; }
    }
    for (u32 i = 0; i < fo; i++) {
        const u32 k = (u32)__popc(free), np = k * (k - 1u) / 2u;
        u32 d = take_digit(outer, np), x = 1;
        while (d >= x) { d -= x; x++; }
        const u32 hi = take_card(free, x) + 1u, lo = take_card(free, d) + 1u;
        m.O |= (u64)(RULE ? lo | (hi << 5) : hi | (lo << 5)) << (10u * i);
    }
    u64 c = 0;
    for (u32 i = 0; free; i++) c |= (u64)(take_card(free, 0u) + 1u) << (8u * i);
    m.s1 = s1; m.s2 = s2; m.wins = wins;
    m.c0 = (u32)c; m.c1 = (u32)(c >> 32);
}

// The pairs of a table row as 10-bit pairs of 5-bit cards.
__device__ __forceinline__ u64 wide_row(u32 c0, u32 c1, u32 sel) {
    u32 x = __byte_perm(c0, c1, sel), y = __byte_perm(c0, c1, sel >> 16);
    x = (x & 0x001F001Fu) | ((x >> 3) & 0x03E003E0u);   // bits 0..9 and 16..25: a pair each
    y = (y & 0x001F001Fu) | ((y >> 3) & 0x03E003E0u);
    x = (x & 0x3FFu) | ((x >> 6) & 0xFFC00u);
    y = (y & 0x3FFu) | ((y >> 6) & 0xFFC00u);
    return (u64)x | ((u64)y << 20);
}

// The start of a lane's game, kept for wide_start, and its block.
struct WideStart {
    u64 a0, b0;
    u32 a1, b1, qa, blk;
};

// How many deals of the game that is at x at turn h lie on their own cycle of length lam (held_start of
// war_held.cu): 0, or 1 (2 with its mirror image).
template <int RULE>
__device__ __noinline__ u32 wide_start(const WideStart x, const MBlock* __restrict__ blocks, u32 n, u32 lam, const Turn5K K) {
    const u32 h = n >> 1;
    u64 a0 = x.a0, b0 = x.b0, d0 = 0, e0 = 0;
    u32 a1 = x.a1, b1 = x.b1, qa = x.qa, d1 = 0, e1 = 0, dq = 0;
    for (u32 t = 0; t < lam; t++) {
        if (t == lam - h) { d0 = a0; d1 = a1; e0 = b0; e1 = b1; dq = qa; }
        turn5_pred<RULE>(a0, a1, b0, b1, qa, K);
    }
    if (a0 != x.a0 || a1 != x.a1 || b0 != x.b0 || b1 != x.b1) return 0u;   // x is not on the cycle
    if (dq != 5u * ((n + 1u) >> 1)) return 0u;                             // not as dealt
    const MBlock& B = blocks[x.blk];
    for (u32 i = 0; i < B.b; i++) {   // (10 cards a player: the low 60 bits)
        const u64 lo = i & 1u ? e0 : d0;
        if (((u32)(lo >> (5u * (i >> 1))) & 31u) != B.prefix[i] + 1u) return 0u;
    }
    return B.twice ? 2u : 1u;
}

// Turns before turn h that belong to the alternating run at turn h, summed over the deals of a game whose free
// pairs are won `a` times by player 1: the deals in which every turn from r on (r < h) has the winner who holds
// an even number of cards, for each r.  wins: the winners of the first p turns.
__device__ __noinline__ u32 wide_streak_head(u32 n, u32 a, u32 p, u32 wins) {
    const u32 h = n >> 1, lenA = (n + 1u) / 2u;
    u32 sum = 0;
    int r = (int)h - 1;
    for (; r >= (int)p; r--) {
        if (((lenA + (u32)r) & 1u) == 0u) {       // player 1's pile is the even one
            if (a == 0u) return sum;
            a--;
        }
        const u32 rem = (u32)r - p;               // turns of free pairs before r, a of them won by player 1
        if (a > rem) return sum;
        u32 c = 1;
        for (u32 i = 1; i <= a; i++) c = c * (rem - a + i) / i;
        sum += c;
    }
    for (; r >= 0 && a == 0u; r--) {
        if (((wins >> r) & 1u) == ((lenA + (u32)r) & 1u)) return sum;
        sum++;
    }
    return sum;
}

// What the kernel needs besides MergeArgs: the step cap, and the streak periods by the next winner's pile.
struct WideMore {
    u32 cap;
    u32 slack;       // streak: turns past the cap after which an undecided game is undetermined for certain
    Turn5K tk;
    u32 lamtab[32];
};

template <int RULE, int DET>
__global__ void __launch_bounds__(1024) wide_merge_kernel(const __grid_constant__ MergeArgs a,
                                                          const __grid_constant__ WideMore more,
                                                          DevAcc* __restrict__ acc) {
    extern __shared__ u64 sh64[];
    __shared__ WUnit units[32];
    WideStart* const start = (WideStart*)sh64 + threadIdx.x;                     // Brent only
    u32* const head = (u32*)sh64 + threadIdx.x;                                  // streak only: a, p and wins
    u32* const shh = DET == DET_BRENT ? (u32*)((WideStart*)sh64 + blockDim.x)
                                      : (u32*)sh64 + (DET == DET_STREAK ? blockDim.x : 0u);
    u32* const she = shh + a.hbins;
    const int bins = a.hbins + WAR_EBINS;
    for (int b = threadIdx.x; b < bins; b += blockDim.x) shh[b] = 0;
    __syncthreads();

    const u32 n = (u32)a.n, h = n >> 1, W = (u32)a.W;
    const u32 hb1 = a.hbins > 0 ? (u32)(a.hbins - 1) : 0u;
    const u32 period = a.defer > 4 ? (u32)((a.defer + 3) & ~3) : 4u;
    const u32 after = DET == DET_BRENT ? h % period : 0u, before = period - after;   // turns around the checkpoint
    const u32 cap = more.cap + (DET == DET_STREAK ? more.slack : 0u);
    const u32 lane = threadIdx.x & 31u;
    WUnit& mu = units[threadIdx.x >> 5];
    u64* const counter = &acc->work_next;

    const Turn5K K = more.tk;
    const u32 n5 = 5u * n;
    u64 a0 = 1, b0 = 1, t0 = ~0ull, t2 = 0, turns = 0;          // the piles' low words, the tortoise's,
    u32 a1 = 0, b1 = 0, t1 = 0, t3 = 0, qa = 0, tqa = 0;        // their high words, 5 * player 1's cards
    u32 rounds = 0, next = 0xFFFFFFFFu, wt = 0, kind = K_END;
    bool done = true, kcy = false;                              // (Brent, streak: decided, by a cycle)
    u32 run = 0, save = 0, prev = 2u;    // streak: turn of the last break, turn of the tortoise, last winner
    bool active = false;
    u32 cyc = 0, maxfin = 0, und = 0;
    MCursor c;

    auto drain = [&]() {
        __syncwarp();
        for (int b = (int)lane; b < bins; b += 32) {
            const u32 v = atomicExch(&shh[b], 0u);
            if (v) atomicAdd(b < a.hbins ? &acc->hist[b] : &acc->endhist[b - a.hbins], (u64)v);
        }
        const u64 v_cyc = warp_sum((u64)cyc), v_und = warp_sum((u64)und);
        if (lane == 0u) {
            if (v_cyc) atomicAdd(&acc->cyc, v_cyc);
            if (v_und) atomicAdd(&acc->undetermined, v_und);
        }
        cyc = 0; und = 0;
    };
    auto setup = [&](const MBlock& B, u64 outer) {
        WUnit m;
        wide_unit<RULE>(B, outer, n, m);
        __syncwarp();
        if (lane == 0u) mu = m;
        __syncwarp();
    };
    auto over = [&]() -> u32 {
        return mu.s2 + 10u * (c.f - c.pa) == 0u ? 1u : (mu.s1 + 10u * c.pa == 0u ? 2u : 0u);
    };
    auto ended = [&](u32 k) {
        if (lane == 0u) { atomicAdd(&she[h], k); turns += (u64)k * h; }
        maxfin = max(maxfin, h);
    };
    auto build = [&](u32 sel) -> bool {
        const u32 a10 = 10u * c.pa, in_at = 10u * (c.f - c.fi);
        const u64 in = wide_row(mu.c0, mu.c1, sel);
        // the list: outer pairs, then inner ones; player 1's first c.pa pairs and player 2's others
        const u64 xl = mu.O | shl64(in, in_at), xh = in_at ? shr64(in, 64u - in_at) : 0ull;
        u64 yl = xl & ~shl64(~0ull, a10), yh = a10 > 64u ? xh & ~shl64(~0ull, a10 - 64u) : 0ull;
        a0 = mu.U1l; a1 = mu.U1h;
        put96(a0, a1, yl, mu.s1);
        if (yh) a1 |= (u32)shl64(yh, mu.s1);
        yl = shr64(xl, a10) | shl64(xh, 64u - a10) | shr64(xh, a10 - 64u);
        yh = shr64(xh, a10);
        b0 = mu.U2l; b1 = mu.U2h;
        put96(b0, b1, yl, mu.s2);
        if (yh) b1 |= (u32)shl64(yh, mu.s2);
        qa = mu.s1 + a10;
        if (c.filter) {   // player 1 must hold card n - 1
            bool has = false;
            for (u32 i = 0; i < qa; i += 5u) has |= ((u32)(i < 60u ? a0 >> i : ((u64)a1 << 32 | a0 >> 32) >> (i - 32u)) & 31u) == n;
            if (!has) return false;
        }
        rounds = h; kind = K_NONE; wt = c.wt; active = true; done = false; kcy = false;
        t0 = a0; t1 = DET == DET_FLOYD ? a1 : a1 + b1; t2 = b0; t3 = b1; tqa = qa;   // (t1: both high words)
        next = W > h ? W : 3u * W;   // (W = h: the tortoise of turn W)
        if (DET == DET_BRENT) {
            WideStart x;
            x.a0 = a0; x.a1 = a1; x.b0 = b0; x.b1 = b1; x.qa = qa; x.blk = c.blk;
            *start = x;
        } else if (DET == DET_STREAK) {
            run = h; save = h; prev = 2u;
            *head = c.pa | ((h - c.f) << 8) | (mu.wins << 16);
        } else if (h & 1u) {         // the hare's turns come in pairs from turn 0
            turn5_pred<RULE>(a0, a1, b0, b1, qa, K);
            rounds = h + 1u;
            if ((qa == 0u) | (qa == n5)) kind = K_END;
        }
        return true;
    };
    auto refill = [&](bool want) {
        if (want) { active = false; kind = K_END; done = true; }
        merge_deal(c, a, counter, __ballot_sync(WAR_FULL_MASK, want), setup, []() {}, over, ended, build, drain);
    };
    // Brent and the streak test latch `done` (and by what) and look at the cap at the services; what is decided by
    // turn cap + 1 is decided (wide_kernel).
    auto turn = [&]() {
        if (DET == DET_FLOYD) {
            const bool open = kind == K_NONE;
            turn5_pred<RULE>(a0, a1, b0, b1, qa, K);
            const bool e1 = (qa == 0u) | (qa == n5);
            turn5_pred<RULE>(a0, a1, b0, b1, qa, K);
            const bool e2 = (qa == 0u) | (qa == n5);
            const u32 r2 = rounds + (e1 ? 1u : 2u);
            if (r2 > 2u * h) turn5_pred<RULE>(t0, t1, t2, t3, tqa, K);
            const bool cy = (a0 == t0) & (b0 == t2) & (a1 * K.one + b1 == t1 * K.one + t3);
            const u32 kk = (e1 | e2) ? (u32)K_END : (cy ? (u32)K_CYC : (r2 > cap ? (u32)K_UND : (u32)K_NONE));
            rounds = open ? r2 : rounds;
            kind = open ? kk : kind;
        } else {
            const u32 w = turn5_pred<RULE>(a0, a1, b0, b1, qa, K);
            if (DET == DET_STREAK) {
                if (!done & (w == prev)) run = rounds * K.one;
                prev = w;
            }
            if (!done) rounds = rounds * K.one + K.one;
            const bool en = qa * K.one - 5u >= n5 - 5u;          // 0 or 5n
            // (at most one of the piles reaches its high word, and equal low words say which)
            const bool cy = (a0 == t0) & (b0 == t2) & (a1 * K.one + b1 == t1);
            kcy = done ? kcy : (cy & !en);
            done = done | cy | en;
        }
    };

    refill(true);
    bool running = __any_sync(WAR_FULL_MASK, active);
    while (running) {
        for (u32 k = 0; k < before; k++) turn();
        if (DET == DET_BRENT) {
            if (!done && rounds == next) { t0 = a0; t1 = a1 + b1; t2 = b0; next = 2u * next + W; }
            for (u32 k = 0; k < after; k++) turn();
        }
        if (DET == DET_STREAK && !done && run > save) { t0 = a0; t1 = a1 + b1; t2 = b0; tqa = qa; save = rounds; }
        if (DET != DET_FLOYD && active)
            kind = done ? (rounds > cap + 1u ? (u32)K_UND : (kcy ? (u32)K_CYC : (u32)K_END)) : (rounds > cap ? (u32)K_UND : (u32)K_NONE);
        const bool fin = active & (kind != K_NONE);
        if (__any_sync(WAR_FULL_MASK, fin)) {
            if (fin) {
                u32 t = rounds;
                if (DET == DET_STREAK) {
                    if (kind == K_CYC) {
                        // the piles are the tortoise's: the next winner's pile and the period are the run's
                        const u32 ws = ((u32)t0 & 31u) > ((u32)t2 & 31u) ? tqa / 5u : n - tqa / 5u;
                        const u32 lam = more.lamtab[ws & 31u];
                        if (run > save || lam == 0u || lam % (rounds - save) != 0u || run + lam > more.cap + 1u)
                            kind = K_UND;
                        else {
                            t = run + lam;
                            if (run == h) turns -= wide_streak_head(n, *head & 255u, (*head >> 8) & 255u, *head >> 16);
                        }
                    }
                    if (kind == K_END && rounds > more.cap + 1u) kind = K_UND;
                }
                if (kind == K_CYC) {
                    cyc += wt;
                    if (DET == DET_BRENT) {
                        // next = W: found with the tortoise at turn h, else at turn (next - W) / 2
                        const u32 at = next == W ? h : (next - W) >> 1, lam = rounds - at;
                        if (a.hbins) atomicAdd(&shh[lam < hb1 ? lam : hb1], wt);
                        if (next == W) t = W + lam;
                        if (lam <= W && at <= W) turns -= (u64)wide_start<RULE>(*start, a.blocks, n, lam, K) * (t - lam);
                    }
                } else if (kind == K_END) {
                    maxfin = max(maxfin, rounds);
                    atomicAdd(&she[rounds < WAR_EBINS - 1 ? rounds : WAR_EBINS - 1], wt);
                } else {
                    und += wt;
                    if (DET != DET_FLOYD) t = more.cap + 1u;
                }
                turns += (u64)wt * t;
            }
            refill(fin);
            running = __any_sync(WAR_FULL_MASK, active);
        }
    }

    const u64 v_cyc = warp_sum((u64)cyc), v_turns = warp_sum(turns), v_max = warp_max((u64)maxfin);
    const u64 v_und = warp_sum((u64)und);
    if (lane == 0u) {
        if (c.done) atomicAdd(&acc->done, c.done);
        if (v_cyc) atomicAdd(&acc->cyc, v_cyc);
        if (v_turns) atomicAdd(&acc->turns, v_turns);
        if (v_max) atomicMax(&acc->maxfin, v_max);
        if (v_und) atomicAdd(&acc->undetermined, v_und);
    }
    __syncthreads();
    flush_hist(shh, acc->hist, a.hbins);
    flush_hist(she, acc->endhist, WAR_EBINS);
}

typedef void (*WideMergeFn)(const MergeArgs, const WideMore, DevAcc*);

static WideMergeFn wide_merge_pick(int det, int rule) {
    if (det == DET_STREAK) return wide_merge_kernel<0, DET_STREAK>;
    if (det == DET_FLOYD) return rule ? wide_merge_kernel<1, DET_FLOYD> : wide_merge_kernel<0, DET_FLOYD>;
    return rule ? wide_merge_kernel<1, DET_BRENT> : wide_merge_kernel<0, DET_BRENT>;
}

static size_t wide_merge_shmem(int det, int threads, int hbins) {
    return sizeof(u32) * (size_t)(hbins + WAR_EBINS) +
           (det == DET_BRENT ? sizeof(WideStart) : det == DET_STREAK ? sizeof(u32) : 0) * (size_t)threads;
}

static bool wide_svc(int W, int defer) {
    const int period = defer > 4 ? (defer + 3) & ~3 : 4;
    return W % period == 0;
}

// Merged games need every checkpoint after turn 0 at or after turn h and at the service period's multiples (Brent),
// and the cap at or after the turns that are not played (above).
static bool wide_merged(int det, int n, int W, int defer, u32 cap, const u32* lamtab) {
    if (det == DET_STREAK) return cap >= (u32)n / 2u + *std::max_element(lamtab, lamtab + 32);
    if (det == DET_FLOYD) return cap >= (u32)n + 2u;
    return det == DET_BRENT && wide_svc(W, defer) && W >= n / 2 && cap >= 2u * (u32)W;
}

typedef void (*WideFn)(const WideArgs, DevAcc*);

static WideFn wide_pick(int det, int rule, bool svc) {
    if (det == DET_FLOYD) return rule ? wide_kernel<1, DET_FLOYD, false> : wide_kernel<0, DET_FLOYD, false>;
    if (det == DET_STREAK) return wide_kernel<0, DET_STREAK, false>;
    if (svc) return rule ? wide_kernel<1, DET_BRENT, true> : wide_kernel<0, DET_BRENT, true>;
    return rule ? wide_kernel<1, DET_BRENT, false> : wide_kernel<0, DET_BRENT, false>;
}

static size_t wide_shmem(int hbins) { return sizeof(u32) * (size_t)(hbins + WAR_EBINS + 32); }

static int wide_max_blocks(int det, int rule, bool svc, int threads, int hbins) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, wide_pick(det, rule, svc), threads, wide_shmem(hbins)) !=
        cudaSuccess)
        return 0;
    return nb;
}

static int wide_merge_max_blocks(int det, int rule, int threads, int hbins) {
    int nb = 0;
    // 1024 threads with more than about 2,500 bins pass the 48 KB that need no asking.  The limit asked for is the
    // same from every call, so that a thread cannot lower it under another one's launch.
    const size_t most = wide_merge_shmem(det, 1024, WAR_HBINS_MAX);
    if (cudaFuncSetAttribute(wide_merge_pick(det, rule), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, wide_merge_pick(det, rule), threads,
                                                      wide_merge_shmem(det, threads, hbins)) != cudaSuccess)
        return 0;
    return nb;
}

}  // namespace war

using namespace war;

extern "C" int war_enumerate_wide(const war_job* job, const war_wide_cfg* cfg, war_result* out) {
    if (!job) return fail(WAR_EINVAL, "job is NULL");
    if (!out) return fail(WAR_EINVAL, "out is NULL");
    war_wide_cfg c;
    memset(&c, 0, sizeof c);
    if (cfg) c = *cfg;
    if (job->mode != WAR_DEALS || job->n < 2 || job->n > 20)
        return fail(WAR_EINVAL, "the 5-bit engine plays deals of 2..20 cards (n=%d, mode=%d)", job->n, job->mode);
    if (job->rule != 0 && job->rule != 1) return fail(WAR_EINVAL, "rule=%d", job->rule);
    if (job->flags & ~WAR_F_MEMO_KEEP) return fail(WAR_EINVAL, "flags=0x%x: none apply to the 5-bit engine", job->flags);
    if (c.det < 0 || c.det > 2) return fail(WAR_EINVAL, "det=%d (0 Brent, 1 Floyd, 2 streak)", c.det);
    if (c.det == DET_STREAK && (!(job->n & 1) || job->rule))
        return fail(WAR_EINVAL, "the streak test holds for odd n and the winner's card first (n=%d, rule=%d)", job->n,
                    job->rule);
    if (job->hbins < 0 || job->hbins > WAR_HBINS_MAX) return fail(WAR_EINVAL, "hbins=%d", job->hbins);
    u64 fn = 1;
    for (int i = 2; i <= job->n; i++) fn *= (u64)i;
    if (job->lo > job->hi || job->hi > fn)
        return fail(WAR_EINVAL, "range [%llu, %llu) outside the %d! deals", (unsigned long long)job->lo,
                    (unsigned long long)job->hi, job->n);
    const u32 cap = c.cap ? c.cap : (1u << 22);
    if (cap > (1u << 30)) return fail(WAR_EINVAL, "cap=%u (at most 2^30)", cap);
    const int threads = c.threads ? c.threads : 256;
    const int block_m = std::min(job->n, c.block_m ? c.block_m : 6);
    const int W = c.window ? c.window : 32;
    const int defer = c.defer ? c.defer : 16;
    if (threads < 64 || threads > 1024 || (threads & 31)) return fail(WAR_EINVAL, "cfg.threads=%d", threads);
    if (block_m < 1 || block_m > 8) return fail(WAR_EINVAL, "cfg.block_m=%d (1..8)", block_m);
    if (W < 1 || W > (1 << 16) || (W & (W - 1))) return fail(WAR_EINVAL, "cfg.window=%d", W);
    if (defer < 1 || defer > 64) return fail(WAR_EINVAL, "cfg.defer=%d (1..64)", defer);
    const int hbins = c.det == DET_BRENT ? job->hbins : 0;
    memset(out, 0, sizeof *out);
    out->hbins = hbins;
    if (job->lo == job->hi) return WAR_OK;
    int st;
    if ((st = ensure_ready())) return st;
    WideMore more;
    memset(&more, 0, sizeof more);
    more.cap = cap;
    more.tk.one = 1u; more.tk.m1 = (u32)-1; more.tk.m32 = (u32)-32; more.tk.k32 = 32u; more.tk.k2p27 = 1u << 27;
    more.tk.c1 = (u32)-5; more.tk.c2 = 5u * (u32)job->n - 5u;
    for (int ws = 2; ws + 2 <= job->n; ws += 2) {   // gpu/war24.py:109: lcm(n+1, lcm(W, L-1))
        auto gcd = [](u64 x, u64 y) { while (y) { u64 t = x % y; x = y; y = t; } return x; };
        const u64 l1 = (u64)ws / gcd(ws, job->n - ws - 1) * (u64)(job->n - ws - 1);
        more.lamtab[ws] = (u32)((u64)(job->n + 1) / gcd(job->n + 1, l1) * l1);
    }
    more.slack = *std::max_element(more.lamtab, more.lamtab + 32) + 64u;
    const bool merged = wide_merged(c.det, job->n, W, defer, cap, more.lamtab);
    const int maxb = merged ? wide_merge_max_blocks(c.det, job->rule, threads, hbins)
                            : wide_max_blocks(c.det, job->rule, wide_svc(W, defer), threads, hbins);
    if (maxb < 1) return fail(WAR_EINVAL, "launch shape threads=%d does not fit an SM", threads);
    const int bps = c.blocks_per_sm ? std::min(c.blocks_per_sm, maxb) : maxb;
    std::lock_guard<std::mutex> lk(ctx().mu);
    Ctx& cx = ctx();
    if (merged) {
        MergePlan p;
        const int blocks = bps * cx.sm_count;
        merge_plan(job, (u64)blocks * (u64)(threads / 32), p);
        MergeArgs m;
        if ((st = merge_args(job, p, hbins, W, defer, m))) return st;
        return run_merged(p, m, MERGE_LAUNCH_UNITS, hbins, 0, out, [&](cudaStream_t x) {
            wide_merge_pick(c.det, job->rule)<<<blocks, threads, wide_merge_shmem(c.det, threads, hbins), x>>>(m, more, cx.d_acc);
            note_launch();
            return cudaGetLastError();
        });
    }
    Plan p;
    make_plan(job, block_m, p);
    if (p.extra.size() > Ctx::UNIT_CAP) return fail(WAR_EINVAL, "plan has %zu extra units", p.extra.size());
    cudaError_t e;
    if (!p.extra.empty() &&
        (e = cudaMemcpyAsync(cx.d_units, p.extra.data(), sizeof(Unit) * p.extra.size(), cudaMemcpyHostToDevice,
                             cur_stream())) != cudaSuccess)
        return cuda_fail(e, "copy units");
    WideArgs a;
    memset(&a, 0, sizeof a);
    a.fact[0] = 1;
    for (int i = 1; i <= 20; i++) a.fact[i] = a.fact[i - 1] * (u64)i;
    a.n = job->n; a.m = block_m; a.rule = job->rule; a.hbins = hbins; a.W = W; a.defer = defer; a.cap = cap;
    a.units = cx.d_units;
    memcpy(a.lamtab, more.lamtab, sizeof a.lamtab);
    // each launch plays fewer than 2^32 - 2^24 games (32-bit per-lane counters)
    const u64 per_unit = a.fact[block_m];
    const u64 max_units = std::max<u64>(1, ((1ull << 32) - (1ull << 24)) / per_unit);
    const WideFn fnp = wide_pick(c.det, job->rule, wide_svc(W, defer));
    const size_t shmem = wide_shmem(hbins);
    u64 done_main = 0;
    bool extras_done = p.extra.empty();
    while (done_main < p.main_count || !extras_done) {
        const u64 take = std::min<u64>(max_units, p.main_count - done_main);
        const bool last = done_main + take >= p.main_count;
        a.main_base = p.main_base + done_main;
        a.main_count = take;
        a.n_units = take + (last ? p.extra.size() : 0);
        st = run_launch([&](cudaStream_t x) {
            fnp<<<bps * cx.sm_count, threads, shmem, x>>>(a, cx.d_acc);
            note_launch();
            return cudaGetLastError();
        }, &out->kernel_ms);
        if (st) return st;
        merge_acc(*cx.h_acc, out, hbins, 0);
        out->units += a.n_units;
        done_main += take;
        if (last) extras_done = true;
    }
    return WAR_OK;
}

// war_merge.cuh — deals played together: the enumeration of the merged kernels (war_merge.cu).
//
// The first h = floor(n/2) turns of a deal only use the cards as dealt: turn t takes the cards of deck
// positions 2t and 2t+1, and the pair goes under the winner's pile.  The state after those h turns is, for
// each player, the pairs that player won, in the order of the turns (odd n: below the one card of player 1
// not played yet).  How the two players' wins alternated leaves no trace in it, and every alternation is a
// deal of its own: which of the two cards of a pair was dealt to which player decides who wins it and
// nothing else.  So all C(f, a) deals that interleave the same a pairs won by player 1 with the same f - a
// pairs won by player 2 are in one state after h turns, and the rest of their game is one game: a merged
// game, played once from turn h and counted C(f, a) times.  No deal is decided before turn h: player 2 has
// an unplayed card left until then, and a cycle is longer than h turns (a shorter one would bring player
// 1's first card back on top while a later one of its cards is there).
//
// Ranks.  A block of j! consecutive lexicographic ranks (a multiple of j!) fixes the first b = n - j deck
// positions, and its deals are every order of the other j cards.  Its merged games are: a card for position
// b if b is odd (dealt against the fixed card before it), a card for position n - 1 if n is odd, an ordered
// list of f = (the other positions) / 2 unordered pairs, and the number a of them that player 1 wins (the
// first a of the list).  That is j!/2^f lists of f + 1 games for j!/2^f * 2^f deals: 9.1 deals per game for
// all 13! deals, 5.3 in a block of 12! of 13 or 15 cards, 3.2 in one of 9!.  A rank range is cut into the
// fewest aligned blocks.  With no fixed card and even n, a state and its mirror image (the players
// swapped) are both in the block, and only the one in which player 1 holds card n - 1 is played, twice
// counted; with --half that one is all there is to play.
//
// Work units.  The first f - 4 pairs of a list (with the two single cards) are the unit's outer choice, by
// mixed-radix index; the last four (fewer in a small block) run through a table of the 2520 ordered lists of
// four pairs of eight cards, as byte selectors: two byte permutes of the unit's eight cards give a list.
// A unit is a run of `lc` table rows under one outer choice, with every a.  A warp takes a unit and deals
// its games to the lanes that need one, so 32 lanes work through it together.
#pragma once
#include <vector>
#include "war_kernels.cuh"

namespace war {

constexpr u32 MERGE_INNER = 4;                       // pairs of a list that the table enumerates
constexpr u32 MERGE_ROWS = 1 + 1 + 6 + 90 + 2520;    // ordered lists of 0..4 pairs of as many cards

__host__ __device__ __forceinline__ u32 merge_rows(u32 fi) {      // (2 fi)! / 2^fi
    return fi < 2u ? 1u : (fi == 2u ? 6u : (fi == 3u ? 90u : 2520u));
}
__host__ __device__ __forceinline__ u32 merge_row0(u32 fi) {      // first row of the table of fi pairs
    return fi == 0u ? 0u : (fi == 1u ? 1u : (fi == 2u ? 2u : (fi == 3u ? 8u : 98u)));
}

typedef unsigned char u8;

// One aligned block of a job.
struct MBlock {
    u64 u0;           // its first unit (the last block is followed by a sentinel with the unit total)
    u32 free_mask;    // cards of the open positions
    u32 nch;          // units per outer choice: ceil(rows / lc)
    u8 f;             // pairs of open positions
    u8 b;             // fixed positions
    u8 filter;        // play only games in which player 1 holds card n - 1
    u8 twice;         // and count them twice (their mirror images)
    u8 prefix[20];    // the fixed cards
    u8 inner;         // table cards of a canonical unit
    u8 k0, k1;        // canonical splits k0 <= k < k1
};

struct HeldK { u32 m1, m260, m252, k65, n4m8; };   // constants of the held-out engine's turn (war_held.cu)

struct MergeArgs {
    const MBlock* blocks;
    const u32* table;     // MERGE_ROWS byte selectors of the rule (winner's or loser's card first)
    u64 unit_lo, unit_hi; // units of this launch
    u32 nblocks, lc;      // blocks[nblocks]: the sentinel
    int n, hbins, W, defer;
    u64* memo;
    u32 memo_bits;
    TestK tk;
    HeldK held;
    // canonical scans
    u64 seed, thr;
    int dbins, blk, distinct, sample;
};

// The outer choice of a unit and what its games share.  The piles without the list's pairs (U1, U2, s1 and
// s2 bits long), the outer pairs (8 bits each), the cards of the inner ones as bytes, and where card n-1 is:
// MTOP_P1 or MTOP_P2 + its place in that pile, MTOP_PAIR + i in outer pair i, MTOP_INNER among the inner cards
// (of which it is the last).  Cards are the low 4 bits of their values (card 16 of 17 is told by its place).
struct MUnit {
    u64 U1, U2, O;
    u32 c0, c1, s1, s2, top;
    // of the number of pairs in hand that player 1 wins: the piles with their sentinels and without the list, the
    // list's pairs that are player 1's
    u64 A1, A2, mask;
    u32 at;           // where the inner pairs go, in bits
    u32 a8;           // 8 * pairs won by player 1
};
constexpr u32 MTOP_INNER = 0, MTOP_PAIR = 32, MTOP_P1 = 64, MTOP_P2 = 128;

// A job's blocks (with the sentinel), units, merged games and rows of a unit.
struct MergePlan {
    std::vector<MBlock> blocks;
    u64 units = 0, games = 0;
    u32 lc = 0;
};
constexpr size_t MERGE_BLOCK_CAP = 512;   // blocks of a range: at most 2 (1 + .. + 16), and the sentinel
// A launch takes at most this many units: a unit stands for at most 2520 rows x 2^11 deals, and a launch for
// fewer than 2^40 (a lane's 32-bit turn total is drained with the histograms).
constexpr u64 MERGE_LAUNCH_UNITS = (1ull << 40) / (2520ull << 11);

void merge_table(int rule, u32* rows);
void merge_plan(const war_job* job, u64 warps, MergePlan& p);
cudaError_t launch_merged(const MergeArgs& a, int rule, int threads, int blocks, DevAcc* acc, cudaStream_t st);
int merged_max_blocks_per_sm(int rule, int threads, int hbins);
void canon_table(u32* rows);
void canon_plan(const war_job* job, u64 warps, MergePlan& p);
cudaError_t launch_canon(const MergeArgs& a, int rule, int extra, int threads, int blocks, DevAcc* acc, cudaStream_t st);
int canon_max_blocks_per_sm(int rule, int shape, int extra, int threads, int hbins);
cudaError_t launch_held_merged(const MergeArgs& a, int rule, bool run, int threads, int blocks, DevAcc* acc, cudaStream_t st);
int held_merged_max_blocks_per_sm(int n, int rule, bool run, int threads, int hbins);

// Card of rank d among the set bits of m; m loses it.
__host__ __device__ __forceinline__ u32 take_card(u32& m, u32 d) {
    u32 x = m;
    for (u32 k = 0; k < d; k++) x &= x - 1u;
    const u32 bit = x & (0u - x);
    m ^= bit;
#ifdef __CUDA_ARCH__
    return (u32)(__ffs((int)bit) - 1);
#else
    return (u32)__builtin_ctz(bit);
#endif
}

__host__ __device__ __forceinline__ u32 card_count(u32 m) {
#ifdef __CUDA_ARCH__
    return (u32)__popc(m);
#else
    return (u32)__builtin_popcount(m);
#endif
}

// x mod k, and x /= k: in 32 bits where x allows (a 64-bit division is some 100 operations).
__host__ __device__ __forceinline__ u32 take_digit(u64& x, u32 k) {
    if ((x >> 32) == 0ull) {
        const u32 y = (u32)x, q = y / k;
        x = q;
        return y - q * k;
    }
    const u64 q = x / k;
    const u32 r = (u32)(x - q * k);
    x = q;
    return r;
}

__host__ __device__ __forceinline__ u64 merge_shl(u64 x, u32 s) { return s < 64u ? x << s : 0ull; }

// Sets a unit up (every lane of the warp the same): the piles of 4-bit cards after the turns that its fixed and
// chosen cards decide.
template <int RULE>
__host__ __device__ __forceinline__ void merge_unit(const MBlock& B, u64 outer, u32 n, MUnit& m) {
    u32 free = B.free_mask;
    const u32 b = B.b, f = B.f, fo = f > MERGE_INNER ? f - MERGE_INNER : 0u, last = n - 1u;
    u64 U1 = 0, U2 = 0;
    u32 s1 = 0, s2 = 0, half = 0, top = MTOP_INNER;
    if ((b & 1u) && b < n) {
        const u32 k = card_count(free);
        half = take_card(free, take_digit(outer, k));
    }
    if (n & 1u) {   // player 1's last card, unplayed after h turns, is on top
        u32 c;
        if (b == n) c = B.prefix[n - 1u];
        else {
            const u32 k = card_count(free);
            c = take_card(free, take_digit(outer, k));
        }
        U1 = c & 15u;
        s1 = 4u;
        if (c == last) top = MTOP_P1;
    }
    for (u32 t = 0; 2u * t < b && 2u * t + 1u < n; t++) {
        const u32 x = B.prefix[2u * t], y = 2u * t + 1u < b ? B.prefix[2u * t + 1u] : half;
        const u32 hi = x > y ? x : y, lo = x > y ? y : x;
        const u64 pair = RULE ? lo | ((hi & 15u) << 4) : (hi & 15u) | (lo << 4);
        if (hi == last) top = x > y ? MTOP_P1 + s1 / 4u + RULE : MTOP_P2 + s2 / 4u + RULE;
        if (x > y) { U1 |= merge_shl(pair, s1); s1 += 8u; }
        else { U2 |= merge_shl(pair, s2); s2 += 8u; }
    }
    u64 O = 0;
    for (u32 i = 0; i < fo; i++) {
        const u32 k = card_count(free), np = k * (k - 1u) / 2u;
        u32 d = take_digit(outer, np), x = 1;
        while (d >= x) { d -= x; x++; }          // the pair of ranks (x, d), x > d
        const u32 hi = take_card(free, x), lo = take_card(free, d);
        if (hi == last) top = MTOP_PAIR + i;
        O |= (u64)(RULE ? lo | ((hi & 15u) << 4) : (hi & 15u) | (lo << 4)) << (8u * i);
    }
    u64 c = 0;
    for (u32 i = 0; free; i++) c |= (u64)(take_card(free, 0u) & 15u) << (8u * i);
    m.U1 = U1; m.U2 = U2; m.O = O; m.s1 = s1; m.s2 = s2; m.top = top;
    m.c0 = (u32)c; m.c1 = (u32)(c >> 32);
}

// The pairs of a table row as 8-bit pairs of 4-bit cards.
__device__ __forceinline__ u32 merge_row(u32 c0, u32 c1, u32 sel) {
    u32 x = __byte_perm(c0, c1, sel), y = __byte_perm(c0, c1, sel >> 16);
    x |= x >> 4;      // bytes 0 and 2: a card and the next one's nibble
    y |= y >> 4;
    return __byte_perm(x, y, 0x6420);
}

// Canonical positions are dealt out the same way, one game each: a block is j! consecutive orders of the n - 1
// other cards with splits k0 <= k < k1, a unit a run of rows of the table of all orders of the last (at most 6)
// cards under one choice of the others, with every split.
constexpr u32 CANON_INNER = 6;
constexpr u32 CANON_ROWS = 1 + 1 + 2 + 6 + 24 + 120 + 720;
__host__ __device__ __forceinline__ u32 canon_rows(u32 i) {       // i!
    return i < 2u ? 1u : i == 2u ? 2u : i == 3u ? 6u : i == 4u ? 24u : i == 5u ? 120u : 720u;
}
__host__ __device__ __forceinline__ u32 canon_row0(u32 i) {       // first row of the table of i cards
    return i == 0u ? 0u : i == 1u ? 1u : i == 2u ? 2u : i == 3u ? 4u : i == 4u ? 10u : i == 5u ? 34u : 154u;
}
struct CUnit {
    u64 Q;            // the cards before the inner ones, 4 bits each
    u32 c0, c1;       // the inner cards as bytes
    // of the split in hand: the piles without the other cards (player 1's card n-1, sentinels), player 1's cards
    u64 A1, A2, mask;
    u32 at;           // where the inner cards go, in bits
    u32 k4;           // 4 * split
};
__host__ __device__ __forceinline__ void canon_unit(const MBlock& B, u64 outer, u32 m, CUnit& u) {
    u32 free = B.free_mask;
    u64 Q = 0, c = 0;
    for (u32 i = 0; i + B.inner < m; i++) {
        u32 v;
        if (i < B.b) v = B.prefix[i];
        else {
            v = take_card(free, take_digit(outer, card_count(free)));
        }
        Q |= (u64)v << (4u * i);
    }
    for (u32 i = 0; free; i++) c |= (u64)take_card(free, 0u) << (8u * i);
    u.Q = Q;
    u.c0 = (u32)c; u.c1 = (u32)(c >> 32);
}

// A warp's place in its unit: row l of [l0, lend) with pa of the f pairs won by player 1, games that stand for wt
// deals each.  Histogram bins of a block are 32 bits: a warp empties them into the accumulators (drain) before
// it has dealt out games that stand for this many deals since it last did.  A bin holds at most what the block's
// warps dealt out since, so 32 x (2^26 + one unit of at most 2520 rows x 2^11 deals) stays below 2^32.
constexpr u32 DRAIN_DEALS = 1u << 26;

struct MCursor {
    u32 l = 0, l0 = 0, lend = 0, pa = 0, f = 0, fi = 0, wt = 0, blk = 0, row0 = 0;
    u32 given = 0;       // deals dealt out since the last drain
    u64 done = 0;        // deals counted by this warp
    bool filter = false, dry = false;
};

// Deals the warp's next games to the lanes of `need`; called by the whole warp.  CANON: pa is the split, the
// rows are orders and every game counts once.
//   setup(B, outer)   sets the unit up for the warp
//   split()           sets up what depends on c.pa
//   over()            whether one player won every pair of the unit's games with c.pa (1: player 1, 2: player 2)
//   ended(count)      counts `count` deals that are over at turn h
//   build(selectors)  the lane's game from a table row; false if it is not played (filter)
//   drain()           empties the histograms
template <bool CANON = false, class Setup, class Split, class Over, class Ended, class Build, class Drain>
__device__ __forceinline__ void merge_deal(MCursor& c, const MergeArgs& a, u64* counter, u32 need, Setup setup,
                                           Split split, Over over, Ended ended, Build build, Drain drain) {
    const u32 lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    while (need && !c.dry) {
        if (c.l == c.lend) {
            if (c.pa < c.f) {
                c.pa++;
                if (!CANON) c.wt = c.wt * (c.f - c.pa + 1u) / c.pa;
                c.l = c.l0;
            } else {
                u64 u = 0;
                if (lane == 0u) u = atomicAdd(counter, 1ull);
                u = __shfl_sync(WAR_FULL_MASK, u, 0) + a.unit_lo;
                if (u >= a.unit_hi) { c.dry = true; break; }
                // its block: the last one that begins at or before it, 32 at a time from the warp's last block on (a
                // job has up to 380 blocks; the last is followed by a sentinel that begins after every unit)
                for (;;) {
                    const u32 i = min(c.blk + 1u + lane, a.nblocks);
                    const u32 adv = (u32)__popc(__ballot_sync(WAR_FULL_MASK, u >= a.blocks[i].u0));
                    c.blk += adv;
                    if (adv < 32u) break;
                }
                const MBlock& B = a.blocks[c.blk];
                u64 outer = u - B.u0;
                const u32 part = take_digit(outer, B.nch);
                setup(B, outer);
                c.f = CANON ? B.k1 - 1u : B.f;
                c.fi = CANON ? B.inner : min(c.f, MERGE_INNER);
                c.row0 = CANON ? canon_row0(c.fi) : merge_row0(c.fi);
                c.l0 = part * a.lc;
                c.lend = min(CANON ? canon_rows(c.fi) : merge_rows(c.fi), c.l0 + a.lc);
                c.l = c.l0;
                c.pa = CANON ? B.k0 : 0u;
                c.wt = !CANON && B.twice ? 2u : 1u;
                c.filter = !CANON && B.filter != 0;
                if (c.given > DRAIN_DEALS) { drain(); c.given = 0; }
            }
            split();
            const u32 o = CANON ? 0u : over();
            if (o) {
                if (o == 1u || !c.filter) {   // (card n-1 is with the player who won every pair)
                    const u32 k = (c.lend - c.l) * c.wt;
                    ended(k);
                    c.done += k; c.given += k;
                }
                c.l = c.lend;
            }
            continue;
        }
        const u32 r = __popc(need & below), take = min((u32)__popc(need), c.lend - c.l);
        bool mine = ((need >> lane) & 1u) && r < take;
        if (mine) mine = build(__ldg(a.table + c.row0 + c.l + r));
        const u32 got = __ballot_sync(WAR_FULL_MASK, mine);
        need &= ~got;
        const u32 k = (u32)__popc(got) * c.wt;
        c.done += k; c.given += k;
        c.l += take;
    }
}

}  // namespace war

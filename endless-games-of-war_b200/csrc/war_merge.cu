// war_merge.cu — the merged kernel of war_enumerate: deals with the path memo (war_refill.cuh), each state
// after the deals' first floor(n/2) turns played once (war_merge.cuh), and its host plan.
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
    a.table = c.d_table + (job->rule ? MERGE_ROWS : 0);
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

}  // namespace war

// war_merge.cu — the kernels of war_enumerate with the path memo (war_refill.cuh): deals, each state after their
// first floor(n/2) turns played once (war_merge.cuh), and canonical scans; and their host plans.
#include <algorithm>
#include <cstring>
#include <vector>
#include "war_host.h"
#include "war_merge_body.cuh"

namespace war {

template <int RULE>
__global__ void __launch_bounds__(1024) merge_kernel(const __grid_constant__ MergeArgs a, DevAcc* __restrict__ acc) {
    extern __shared__ u64 sh64[];
    __shared__ UnitStore store;
    merge_body<RULE>(a, acc, &acc->work_next, store, sh64);
}

template <int RULE, bool EXTRA, bool SHAPE>
__global__ void __launch_bounds__(1024) canon_kernel(const __grid_constant__ MergeArgs a, DevAcc* __restrict__ acc) {
    extern __shared__ u64 sh64[];
    __shared__ UnitStore store;
    canon_body<RULE, EXTRA, SHAPE>(a, acc, &acc->work_next, store, sh64);
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
    // about 24 units for each warp, so that the last ones end together, of at least 64 to 400 games, as many as give
    // every warp one: setting a unit up costs about what ten games do (2e6 positions of 11 cards: units of 40 games
    // 469 us, 200: 370, 300: 351, 400: 344, 800: 363)
    u64 lc = rows / std::max<u64>(1, warps * 24);
    const u64 least = std::min<u64>(std::max<u64>(rows / std::max<u64>(1, warps), (64 + m - 1) / m), (400 + m - 1) / m);
    lc = std::min<u64>(std::max(lc, least), 720);
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
    // About 24 units for each warp, so that the last ones end together, of at least 14 to 60 rows (five games each in a
    // block of ten cards), as many as give every warp one: kernel times with units of 7, 14, 20, 30, 40 and 60 rows
    // 43.0, 41.0, 41.9, 46.2, 47.1 and 54.0 us for 3e5 deals of 10 cards, 193, 154, 141, 129, 123 and 119 us for 5e6 of
    // 11.  (6 units for each warp: a span of 14 cards 14.4 ms instead of 14.1.)
    u64 lc = rows4 / std::max<u64>(1, warps * 24);
    const u64 least = std::min<u64>(std::max<u64>(rows4 / std::max<u64>(1, warps), 14), 60);
    lc = std::min<u64>(std::max(lc, least), 2520);
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
    a.nblocks = (u32)p.blocks.size() - 1u;
    a.lc = p.lc;
    a.n = job->n; a.hbins = hbins; a.W = window; a.defer = defer;
    set_turn(a.tk, job->n);
    a.held.m1 = (u32)-1; a.held.m260 = (u32)-260; a.held.m252 = (u32)-252; a.held.k65 = 65u;
    a.held.n4m8 = 4u * (u32)job->n - 8u;
    return WAR_OK;
}

static size_t merge_shmem(int threads, int hbins) {
    return sizeof(Missed) * (size_t)threads + sizeof(u32) * (size_t)(hbins + WAR_EBINS);
}

cudaError_t launch_merged(const MergeArgs& a, int rule, int threads, int blocks, DevAcc* acc, cudaStream_t st) {
    (rule ? merge_kernel<1> : merge_kernel<0>)<<<blocks, threads, merge_shmem(threads, a.hbins), st>>>(a, acc);
    note_launch();
    return cudaGetLastError();
}

int merged_max_blocks_per_sm(int rule, int threads, int hbins) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rule ? merge_kernel<1> : merge_kernel<0>, threads,
                                                      merge_shmem(threads, hbins)) != cudaSuccess)
        return 0;
    return nb;
}

static size_t canon_shmem(int extra, int threads, int hbins) {
    return merge_shmem(threads, hbins) + (extra ? 2 * sizeof(u64) * (size_t)threads + sizeof(StartQueue) * (size_t)(threads / 32) : 0);
}

typedef void (*MergeFn)(const MergeArgs, DevAcc*);

template <int RULE>
static MergeFn canon_pick(int shape, int extra) {
    if (shape) return extra ? canon_kernel<RULE, true, true> : canon_kernel<RULE, false, true>;
    return extra ? canon_kernel<RULE, true, false> : canon_kernel<RULE, false, false>;
}

cudaError_t launch_canon(const MergeArgs& a, int rule, int extra, int threads, int blocks, DevAcc* acc, cudaStream_t st) {
    const MergeFn fn = rule ? canon_pick<1>(a.blk, extra) : canon_pick<0>(a.blk, extra);   // (shared memory: set below)
    fn<<<blocks, threads, canon_shmem(extra, threads, a.hbins), st>>>(a, acc);
    note_launch();
    return cudaGetLastError();
}

int canon_max_blocks_per_sm(int rule, int shape, int extra, int threads, int hbins) {
    const MergeFn fn = rule ? canon_pick<1>(shape, extra) : canon_pick<0>(shape, extra);
    const size_t shmem = canon_shmem(extra, threads, hbins);
    int nb = 0;
    // large blocks with starts and queues pass the 48 KB that need no asking; the limit asked for is the same from every
    // call, so that a thread cannot lower it under another one's launch
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)canon_shmem(extra, 1024, WAR_HBINS_MAX)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, shmem) != cudaSuccess) return 0;
    return nb;
}

}  // namespace war

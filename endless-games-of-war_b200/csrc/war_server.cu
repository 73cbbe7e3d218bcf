// war_server.cu — continuous batching of enumeration jobs (war_server_* in include/war.h).  No counterpart
// in the reference, which runs one job per process.
//
// Jobs of any n, mode, rule and rank range are submitted from any thread.  A worker thread admits them,
// in submission order, into resident accumulator slots on the device; the number of slots is what the
// device-memory budget allows, so a job waits in the queue until a slot (its accumulators) is free.
// Every "tick" the worker cuts the admitted jobs' remaining ranges into tasks (each a run of work units of
// one job, about task_ranks ranks), sharing the tick's rank budget round-robin so that a short job is not
// stuck behind a long one, and runs the whole tick as one launch per kernel variant: each block plays one
// task with the loops of war_merge_body.cuh (deals and canonical scans of any n and rule: one variant) or
// war_refill.cuh and adds its results to that task's job slot.  Jobs of different n and mode therefore run
// side by side on the device.  Two ticks are in flight at a time (the next one is queued before the previous
// one is waited for), so the GPU does not wait for the host; the jobs whose last tasks were in a finished tick
// are read back together, their slots freed and their results published.
//
// What bounds a burst of small jobs: the longest task and the jobs whose games find no table to help them.  24 jobs
// of 1e4 to 3e7 ranks (four mixes, repeated): 38, 32, 45 and 45 ms with one launch per n-and-mode variant of
// blocks that played units of 720 deals a lane; 33, 5, 12 and 7 ms with this one (B200).
//
// Jobs of the same n and rule share one cycle memo (war_refill.cuh): its entries are facts about n and the
// rule, so every job of that class, now and later, decides its games from what the earlier ones found.
// The tables come from one arena that war_server_create reserves inside the memory budget (after the
// accumulator slots); a class takes its table from the arena when its first job is admitted, cleared on
// the compute stream, and keeps it until the server ends; a class of merged jobs takes at most half of what is left, so
// that a server of several large classes does not leave the last ones without.  The worker thread never calls cudaMalloc, which
// would synchronise the device in the middle of the tick stream.  A class whose table no longer fits runs
// without the memo.
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "war_host.h"
#include "war_refill.cuh"
#include "war_merge_body.cuh"

namespace war {

// One block's work: a run of units of a merged job, whose arguments are kept on the device by accumulator slot
// while it runs.
struct ServeTask {
    u64 lo, hi;           // its units [lo, hi)
    u64 counter;          // the task's work-unit counter (zero when uploaded)
    u32 slot;             // accumulator slot of the job
    u32 kind;             // rule + 2 canon + 2 (canon and distinct or sample)
};

// The same for the other jobs, whose tasks are few (2^16 ranks each).  The arguments come with the task, units and
// all: put together in the kernel from a job's and a task's, the sampled deals' loop without a table is compiled for 56
// registers instead of 64 (3e7 deals of 13 cards 21.5 ms, so 23.7).
struct RefillTask {
    BatchArgs args;   // the job's parameters and this task's units
    u32 slot;         // accumulator slot of the job
    u32 pad;
    u64 counter;      // the task's work-unit counter (zero when uploaded)
};

template <int RULE, int G, bool CANON, bool SHAPE, bool EXTRA, int V>
__global__ void __launch_bounds__(G == 1 ? 1024 : 512) serve_kernel(RefillTask* __restrict__ tasks,
                                                                   DevAcc* __restrict__ slots) {
    extern __shared__ u32 sh[];
    __shared__ BatchArgs A;
    RefillTask* t = tasks + blockIdx.x;
    const u32* src = (const u32*)&t->args;
    for (int i = threadIdx.x; i < (int)(sizeof(BatchArgs) / 4); i += blockDim.x) ((u32*)&A)[i] = src[i];
    __syncthreads();
    refill_dispatch<RULE, G, CANON, SHAPE, EXTRA, V>(A, slots + t->slot, &t->counter, sh);
}

// The same for the loops of war_merge_body.cuh, merged deals and canonical scans with or without a table, all in
// one launch: the tasks of a tick run side by side whatever their kind.
__global__ void __launch_bounds__(1024) serve_merge_kernel(ServeTask* __restrict__ tasks,
                                                           const MergeArgs* __restrict__ jobs,
                                                           DevAcc* __restrict__ slots) {
    extern __shared__ u64 sh64[];
    __shared__ MergeArgs A;
    __shared__ UnitStore store;
    ServeTask* t = tasks + blockIdx.x;
    const u32* src = (const u32*)&jobs[t->slot];
    for (int i = threadIdx.x; i < (int)(sizeof(MergeArgs) / 4); i += blockDim.x) ((u32*)&A)[i] = src[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        A.unit_lo = t->lo;
        A.unit_hi = t->hi;
    }
    __syncthreads();
    DevAcc* const acc = slots + t->slot;
    switch (t->kind) {
        case 0: merge_body<0>(A, acc, &t->counter, store, sh64); break;
        case 1: merge_body<1>(A, acc, &t->counter, store, sh64); break;
        case 2: canon_body<0, false, false>(A, acc, &t->counter, store, sh64); break;
        case 3: canon_body<1, false, false>(A, acc, &t->counter, store, sh64); break;
        case 4: canon_body<0, true, false>(A, acc, &t->counter, store, sh64); break;
        default: canon_body<1, true, false>(A, acc, &t->counter, store, sh64); break;
    }
}

typedef void (*ServeFn)(RefillTask*, DevAcc*);

template <int RULE, int G, int V>
static ServeFn serve_pick(bool canon, bool shape, bool extra) {
    if (!canon) return extra ? serve_kernel<RULE, G, false, false, true, V> : serve_kernel<RULE, G, false, false, false, V>;
    if (shape) return extra ? serve_kernel<RULE, G, true, true, true, V> : serve_kernel<RULE, G, true, true, false, V>;
    return extra ? serve_kernel<RULE, G, true, false, true, V> : serve_kernel<RULE, G, true, false, false, V>;
}

// Launch shapes of the serving kernels: one game per thread, 256-thread blocks, the multiply-add turn form.
// Merged deals and canonical scans are one kernel, serve_merge_kernel (merged = 1, the other fields 0); sampled deals play deal by deal,
// with the path memo where the class has a table (memo); the loop-shape test has the immediate-record loop, and
// so have canonical scans and deals of fewer than 4 cards the latched one.
struct Variant {
    int merged, canon, rule, shape, extra, memo;
    bool operator<(const Variant& o) const {
        return std::tie(merged, canon, rule, shape, extra, memo) <
               std::tie(o.merged, o.canon, o.rule, o.shape, o.extra, o.memo);
    }
    template <int RULE>
    ServeFn fn_rule() const {
        if (shape) return serve_pick<RULE, 1, 1>(true, true, extra);
        if (memo) return serve_kernel<RULE, 1, false, false, true, 31>;
        return serve_pick<RULE, 1, 3>(canon != 0, false, extra);
    }
    ServeFn fn() const { return rule ? fn_rule<1>() : fn_rule<0>(); }
};

constexpr int SERVE_THREADS = 256;

size_t serve_shmem(int hbins, bool merged) {   // (a merged launch may hold canonical tasks that keep their starts)
    return sizeof(u32) * (size_t)(hbins + WAR_EBINS) +
           (merged ? (sizeof(Missed) + 2 * sizeof(u64) + sizeof(StartQueue) / 32) * (size_t)SERVE_THREADS : 0);
}

struct SJob {
    war_job job;
    int state = 0;       // 0 queued, 1 running, 2 done, 3 failed
    int status = 0;
    double t_submit = 0, t_admit = 0, t_finish = 0;
    int slot = -1;
    Plan plan;
    u64 next_main = 0;
    bool extras_issued = false;
    u64 per_unit = 1;    // ranks per main unit
    MergePlan mplan;     // merged jobs: the plan; next_main counts its units
    BatchArgs base;      // the other jobs: the arguments of their tasks, without units
    Variant var;
    u32 kind = 0;        // of its tasks (ServeTask)
    war_result* result = nullptr;
};

struct Tick {
    ServeTask* h_tasks = nullptr;   // pinned
    RefillTask* h_refill = nullptr; // pinned
    Unit* h_units = nullptr;        // pinned
    ServeTask* d_tasks = nullptr;
    RefillTask* d_refill = nullptr;
    Unit* d_units = nullptr;
    int ntasks = 0, nrefill = 0, nunits = 0;
    std::vector<std::pair<Variant, std::pair<int, int>>> groups;   // kernels of the other jobs -> [first task, count)
    std::vector<std::pair<u64, int>> finishing;      // jobs whose last task is in this tick, and their slots
    std::vector<std::pair<int, size_t>> admitted;    // slots to be set up before this tick, and their blocks
    cudaEvent_t ev = nullptr;
    bool in_flight = false;
};

}  // namespace war

struct war_server {
    war_server_cfg cfg;
    int device = 0, sm_count = 0, nslots = 0, max_tasks = 0, max_units = 0;
    std::thread worker;
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    bool stop = false;
    std::deque<uint64_t> pending;
    std::map<uint64_t, war::SJob> jobs;
    std::vector<int> free_slots;
    std::map<std::pair<int, int>, std::pair<u64*, int>> memos;   // (n, rule) -> (table, log2 words)
    u64* memo_arena = nullptr;      // reserved at create; tables are carved from it in admission order
    u64 arena_words = 0, arena_used = 0;
    u32* d_table = nullptr;         // pair lists and orders (war_merge.cuh)
    war::MBlock* d_blocks = nullptr;     // the resident merged jobs' blocks, SLOT_BLOCKS for each slot
    war::MBlock* h_blocks = nullptr;     // and their mirror: pageable, a slot's few KB are staged by the copy, where
                                         // pinning the 4 MB of 256 slots takes longer than all the copies
    war::MergeArgs* d_jobs = nullptr;   // the resident merged jobs' arguments, by slot
    war::MergeArgs* h_jobs = nullptr;   // and their mirror, pinned
    DevAcc* d_slots = nullptr;
    DevAcc* h_slot = nullptr;   // pinned readback buffer, READBACK slots
    cudaStream_t s_comp = nullptr, s_copy = nullptr;
    war::Tick ticks[2];
    uint64_t next_id = 1, nticks = 0, jobs_done = 0, peak_resident = 0, resident = 0;
    int fatal = 0;
    std::chrono::steady_clock::time_point t0;

    double now_ms() const {
        return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
};

namespace war {
namespace {

// Ranks per task of a merged job: as many as give each SM 16 blocks of the tick's work, so that a small tick spreads
// over the GPU (2^13: the block's own start and end stay small beside its games).  Tasks of the other jobs have the
// most: there a lane, not a warp, plays a unit (720 deals), and a smaller task leaves more of a block's lanes without
// one (1e8 sampled deals of 13 cards 6.8 ms, with tasks by the tick's work 11.2).
constexpr u64 TASK_RANKS_MIN = 1ull << 13, TASK_RANKS_MAX = 1ull << 16;
// Refill tasks of a tick: what a tick's ranks make by default, and two more for the ends of each of 256 jobs (room for
// 16384 took 7 ms to pin when the server is made, a third of all).
constexpr int MAX_REFILL = 2560;
constexpr size_t READBACK = 32;          // finished jobs read back at a time
constexpr size_t SLOT_BLOCKS = 256;      // blocks of a job of at most 16 cards: at most 2 (1 + .. + 15), and the sentinel
constexpr int UNITS_PER_EXTRA_CAP = 512;   // sizing of the per-tick extra-unit pool

void set_args(war_server* s, SJob& J) {
    const war_job& job = J.job;
    const bool canon = job.mode == WAR_CANON;
    BatchArgs a;
    memset(&a, 0, sizeof a);
    fill_fact(a.fact);
    a.n = job.n;
    a.m = J.plan.m;
    a.hbins = job.hbins;
    a.dbins = job.dbins;
    a.blk = (job.flags & WAR_F_SHAPE) && canon ? (job.blk ? job.blk : (job.n & -job.n)) : 0;
    a.W = canon ? 128 : 32;
    a.defer = canon ? (job.n < 13 ? 16 : 12) : job.n < 14 ? 8 : job.n == 14 ? 12 : 16;   // (autotune.py's defaults)
    set_turn(a.tk, job.n);
    a.half = (job.flags & WAR_F_HALF) ? 1 : 0;
    a.sample = (job.flags & WAR_F_SAMPLE) ? 1 : 0;
    a.distinct = (job.flags & WAR_F_DISTINCT) && canon ? 1 : 0;
    a.seed = job.seed;
    a.thr = ((u64)job.sample_ppm << 32) / 1000000u;
    const int extra = (a.distinct || a.sample) ? 1 : 0;
    J.var = Variant();
    J.var.merged = !a.blk && job.n >= 4 && (canon || !a.sample) ? 1 : 0;
    if (J.var.merged) {
        J.kind = (u32)job.rule + (canon ? 2u + 2u * (u32)extra : 0u);
        const u64 warps = (u64)s->sm_count * 32u;
        if (canon) canon_plan(&job, warps, J.mplan);
        else merge_plan(&job, warps, J.mplan);
        J.per_unit = std::max<u64>(1, (job.hi - job.lo) / std::max<u64>(1, J.mplan.units));
    } else {
        J.var.canon = canon ? 1 : 0;
        J.var.rule = job.rule;
        J.var.shape = a.blk ? 1 : 0;
        J.var.extra = extra;
    }
    if (!a.blk && job.n >= 4 && s->cfg.memo_bits >= 0) {
        // the class's table: 2^bits words, grown with n (about a thousandth of the class's rank space)
        const std::pair<int, int> cls(job.n, job.rule);
        auto it = s->memos.find(cls);
        if (it == s->memos.end()) {
            const int cap = s->cfg.memo_bits ? s->cfg.memo_bits : 28;
            int bits = std::max(12, std::min(cap, 4 + (int)std::ceil(std::log2((double)fact(job.n)) * 0.75)));
            // the largest table of at most 2^bits words in half of what the arena still holds, so that later classes
            // have one too (in all of it if the arena is below 2^24 words, or for sampled deals, which look every deal
            // up: 5e7 of 13 cards in an arena of 2^25 words 12.1 ms, with half of it 13.6), at least 2^12 words
            const u64 left = s->arena_words - s->arena_used;
            const u64 most = s->arena_words < (1ull << 24) || !J.var.merged ? left : left / 2;
            while (bits >= 12 && (1ull << bits) > most) bits--;
            u64* t = nullptr;
            if (bits >= 12) {
                t = s->memo_arena + s->arena_used;
                if (cudaMemsetAsync(t, 0, sizeof(u64) << bits, s->s_comp) != cudaSuccess) {
                    t = nullptr;
                    cudaGetLastError();   // not cleared: the class runs without the memo
                } else {
                    s->arena_used += 1ull << bits;
                }
            }
            it = s->memos.emplace(cls, std::make_pair(t, bits)).first;
        }
        if (it->second.first) {
            a.memo = it->second.first;
            a.memo_bits = (u32)it->second.second;
            if (!J.var.merged) J.var.memo = 1;
        }
    }
    J.base = a;
    if (!J.var.merged) return;
    MergeArgs& m = s->h_jobs[J.slot];
    memset(&m, 0, sizeof m);
    MBlock* const h = s->h_blocks + (size_t)J.slot * SLOT_BLOCKS;
    memcpy(h, J.mplan.blocks.data(), sizeof(MBlock) * J.mplan.blocks.size());
    m.blocks = s->d_blocks + (size_t)J.slot * SLOT_BLOCKS;
    m.table = s->d_table + (canon ? 2 * MERGE_ROWS : job.rule ? MERGE_ROWS : 0);
    m.nblocks = (u32)J.mplan.blocks.size() - 1u;
    m.lc = J.mplan.lc;
    m.n = a.n; m.hbins = a.hbins; m.W = a.W; m.defer = a.defer;
    m.memo = a.memo; m.memo_bits = a.memo_bits; set_turn(m.tk, job.n);
    m.seed = a.seed; m.thr = a.thr;
    m.dbins = a.dbins; m.distinct = a.distinct; m.sample = a.sample;
}

u64 main_units(const SJob& J) { return J.var.merged ? J.mplan.units : J.plan.main_count; }
bool extras(const SJob& J) { return !J.var.merged && !J.extras_issued && !J.plan.extra.empty(); }
bool remaining(const SJob& J) { return J.next_main < main_units(J) || extras(J); }

// Finishes jobs whose accumulators are complete: reads their slots back, READBACK at a time, and publishes the
// results.
void finish_jobs(war_server* s, const std::vector<std::pair<u64, int>>& ids) {
    for (size_t i0 = 0; i0 < ids.size(); i0 += READBACK) {
        const size_t k = std::min(READBACK, ids.size() - i0);
        cudaError_t e = cudaSuccess;
        for (size_t i = 0; i < k && e == cudaSuccess; i++)
            e = cudaMemcpyAsync(s->h_slot + i, s->d_slots + ids[i0 + i].second, sizeof(DevAcc),
                                cudaMemcpyDeviceToHost, s->s_copy);
        const cudaError_t e2 = cudaStreamSynchronize(s->s_copy);
        if (e == cudaSuccess) e = e2;
        std::lock_guard<std::mutex> lk(s->mu);
        for (size_t i = 0; i < k; i++) {
            SJob& J = s->jobs[ids[i0 + i].first];
            if (e != cudaSuccess) {
                J.state = 3; J.status = WAR_ECUDA;
            } else if (s->h_slot[i].status) {
                J.state = 3; J.status = WAR_ECAP;
            } else {
                merge_acc(s->h_slot[i], J.result, J.job.hbins, J.job.dbins);
                J.state = 2;
            }
            J.t_finish = s->now_ms();
            s->free_slots.push_back(J.slot);
            s->resident--;
            s->jobs_done++;
        }
        s->cv_done.notify_all();
    }
}

// Admits queued jobs into free slots (caller holds the lock).  Empty jobs finish at once.
void admit(war_server* s, Tick& T) {
    while (!s->pending.empty() && !s->free_slots.empty()) {
        u64 id = s->pending.front();
        s->pending.pop_front();
        SJob& J = s->jobs[id];
        J.t_admit = s->now_ms();
        const war_job& job = J.job;
        const bool canon = job.mode == WAR_CANON;
        if (job.lo == job.hi || (!canon && job.n == 1)) {   // nothing to play on the device
            if (!canon && job.n == 1) {
                J.result->done = 1; J.result->endhist[0] = 1;
                if ((job.flags & WAR_F_SAMPLE) && war_sample_pick(job.seed, job.sample_ppm, 0x10ull, 0x1ull))
                    J.result->s_count = 1;
            }
            J.state = 2; J.t_finish = J.t_admit; s->jobs_done++;
            s->cv_done.notify_all();
            continue;
        }
        const int M = canon ? job.n - 1 : job.n;
        make_plan(&job, std::max(1, std::min(canon ? 4 : 6, M)), J.plan);
        J.per_unit = fact(J.plan.m) * J.plan.games_per_order;
        J.slot = s->free_slots.back();
        set_args(s, J);
        if (J.var.merged && J.mplan.units == 0) {   // --half: no deal of the range gives card n-1 to player 1
            J.state = 2; J.t_finish = s->now_ms(); s->jobs_done++;
            s->cv_done.notify_all();
            continue;
        }
        s->free_slots.pop_back();
        J.state = 1;
        s->resident++;
        s->peak_resident = std::max<u64>(s->peak_resident, s->resident);
        T.admitted.push_back({J.slot, J.var.merged ? J.mplan.blocks.size() : 0});
    }
}

// Cuts the running jobs' remaining work into this tick's tasks (caller holds the lock).
void build_tick(war_server* s, Tick& T) {
    T.ntasks = 0; T.nrefill = 0; T.nunits = 0; T.groups.clear(); T.finishing.clear();
    std::vector<u64> run;
    for (auto& kv : s->jobs)
        if (kv.second.state == 1 && remaining(kv.second)) run.push_back(kv.first);
    if (run.empty()) return;
    const u64 budget = s->cfg.tick_ranks;
    u64 left = 0;
    for (u64 id : run) {
        const SJob& J = s->jobs[id];
        left += (main_units(J) - J.next_main) * J.per_unit;
    }
    const u64 task_ranks = std::min(TASK_RANKS_MAX, std::max(TASK_RANKS_MIN, std::min(left, budget) / (16ull * (u64)s->sm_count)));
    const int unit_cap = s->max_units * 8;
    u64 used = 0;
    std::map<Variant, std::vector<RefillTask>> refill;
    bool progress = true;
    while (progress && used < budget && T.ntasks + T.nrefill < s->max_tasks) {
        progress = false;
        for (u64 id : run) {
            if (used >= budget || T.ntasks + T.nrefill >= s->max_tasks) break;
            SJob& J = s->jobs[id];
            if (!remaining(J) || (!J.var.merged && T.nrefill >= MAX_REFILL)) continue;
            const u64 lo = J.next_main, ranks = J.var.merged ? task_ranks : TASK_RANKS_MAX;
            const u64 k = std::min(std::max<u64>(1, ranks / J.per_unit), main_units(J) - lo);
            J.next_main += k;
            used += k * J.per_unit;
            if (J.var.merged) {
                ServeTask& t = T.h_tasks[T.ntasks++];
                t.lo = lo; t.hi = lo + k; t.counter = 0;
                t.slot = (u32)J.slot; t.kind = J.kind;
            } else {
                RefillTask t;
                memset(&t, 0, sizeof t);
                t.args = J.base;
                t.slot = (u32)J.slot;
                if (k) {
                    t.args.main_base = J.plan.main_base + lo;
                    t.args.main_count = t.args.n_units = k;
                } else {
                    const int x = (int)J.plan.extra.size();
                    if (T.nunits + x > unit_cap) continue;   // next tick
                    memcpy(T.h_units + T.nunits, J.plan.extra.data(), sizeof(Unit) * (size_t)x);
                    t.args.units = T.d_units + T.nunits;
                    t.args.n_units = (u64)x;
                    T.nunits += x;
                    J.extras_issued = true;
                    used += 1;
                }
                refill[J.var].push_back(t);
                T.nrefill++;
            }
            if (!remaining(J)) T.finishing.push_back({id, J.slot});
            progress = true;
        }
    }
    int at = 0;
    for (const auto& kv : refill) {   // one launch per kernel variant
        T.groups.push_back({kv.first, {at, (int)kv.second.size()}});
        memcpy(T.h_refill + at, kv.second.data(), sizeof(RefillTask) * kv.second.size());
        at += (int)kv.second.size();
    }
}

cudaError_t launch_tick(war_server* s, Tick& T) {
    cudaError_t e;
    for (const auto& ad : T.admitted) {
        const int slot = ad.first;
        if ((e = cudaMemsetAsync(s->d_slots + slot, 0, sizeof(DevAcc), s->s_comp)) != cudaSuccess) return e;
        if (!ad.second) continue;   // not merged
        if ((e = cudaMemcpyAsync(s->d_jobs + slot, s->h_jobs + slot, sizeof(MergeArgs), cudaMemcpyHostToDevice,
                                 s->s_comp)) != cudaSuccess)
            return e;
        const size_t at = (size_t)slot * SLOT_BLOCKS;
        if ((e = cudaMemcpyAsync(s->d_blocks + at, s->h_blocks + at, sizeof(MBlock) * ad.second, cudaMemcpyHostToDevice,
                                 s->s_comp)) != cudaSuccess)
            return e;
    }
    T.admitted.clear();
    if (T.ntasks + T.nrefill == 0) return cudaSuccess;
    if (T.ntasks &&
        (e = cudaMemcpyAsync(T.d_tasks, T.h_tasks, sizeof(ServeTask) * T.ntasks, cudaMemcpyHostToDevice, s->s_comp)))
        return e;
    if (T.nrefill &&
        (e = cudaMemcpyAsync(T.d_refill, T.h_refill, sizeof(RefillTask) * T.nrefill, cudaMemcpyHostToDevice, s->s_comp)))
        return e;
    if (T.nunits &&
        (e = cudaMemcpyAsync(T.d_units, T.h_units, sizeof(Unit) * T.nunits, cudaMemcpyHostToDevice, s->s_comp)))
        return e;
    // every task of a launch zeroes and flushes hbins of its own; the launch provides the largest
    for (auto& g : T.groups) {
        int hb = 0;
        for (int i = g.second.first; i < g.second.first + g.second.second; i++) hb = std::max(hb, T.h_refill[i].args.hbins);
        g.first.fn()<<<g.second.second, SERVE_THREADS, serve_shmem(hb, false), s->s_comp>>>(T.d_refill + g.second.first,
                                                                                         s->d_slots);
        note_launch();
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (T.ntasks) {
        int hb = 0;
        for (int i = 0; i < T.ntasks; i++) hb = std::max(hb, s->h_jobs[T.h_tasks[i].slot].hbins);
        serve_merge_kernel<<<T.ntasks, SERVE_THREADS, serve_shmem(hb, true), s->s_comp>>>(T.d_tasks, s->d_jobs, s->d_slots);
        note_launch();
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaEventRecord(T.ev, s->s_comp);
}

void worker_main(war_server* s) {
    cudaSetDevice(s->device);
    int cur = 0;
    for (;;) {
        Tick& T = s->ticks[cur];
        bool built = false;
        {
            std::unique_lock<std::mutex> lk(s->mu);
            bool busy = s->ticks[cur ^ 1].in_flight;
            if (!busy) {
                s->cv_work.wait_for(lk, std::chrono::milliseconds(2), [&] {
                    if (s->stop || !s->pending.empty()) return true;
                    for (auto& kv : s->jobs) if (kv.second.state == 1 && remaining(kv.second)) return true;
                    return false;
                });
            }
            if (s->stop && s->pending.empty() && !busy) {
                bool any = false;
                for (auto& kv : s->jobs) if (kv.second.state == 1) any = true;
                if (!any) break;
            }
            if (!s->fatal) {
                admit(s, T);
                build_tick(s, T);
                built = T.ntasks + T.nrefill > 0 || !T.admitted.empty();
            }
        }
        if (built) {
            cudaError_t e = launch_tick(s, T);
            if (e != cudaSuccess) {
                std::lock_guard<std::mutex> lk(s->mu);
                s->fatal = WAR_ECUDA;
                for (auto& kv : s->jobs)
                    if (kv.second.state <= 1) { kv.second.state = 3; kv.second.status = WAR_ECUDA; }
                s->cv_done.notify_all();
            } else if (T.ntasks + T.nrefill > 0) {
                T.in_flight = true;
                s->nticks++;
            }
        }
        Tick& P = s->ticks[cur ^ 1];
        if (P.in_flight) {
            cudaError_t e = cudaEventSynchronize(P.ev);
            P.in_flight = false;
            if (e != cudaSuccess) {
                std::lock_guard<std::mutex> lk(s->mu);
                s->fatal = WAR_ECUDA;
                for (auto& kv : s->jobs)
                    if (kv.second.state <= 1) { kv.second.state = 3; kv.second.status = WAR_ECUDA; }
                s->cv_done.notify_all();
            } else {
                finish_jobs(s, P.finishing);
            }
            P.finishing.clear();
        }
        cur ^= 1;
    }
}

}  // namespace
}  // namespace war

using namespace war;

extern "C" {

int war_server_create(const war_server_cfg* cfg, war_server** out) {
    if (!out) return fail(WAR_EINVAL, "out is NULL");
    *out = nullptr;
    war_server_cfg c;
    memset(&c, 0, sizeof c);
    if (cfg) c = *cfg;
    if (c.max_jobs < 0 || c.queue_cap < 0) return fail(WAR_EINVAL, "negative max_jobs / queue_cap");
    if (!c.max_jobs) c.max_jobs = 256;
    if (!c.queue_cap) c.queue_cap = 1 << 16;
    if (!c.tick_ranks) c.tick_ranks = 1ull << 27;
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) return fail(WAR_ENODEV, "no CUDA device (%s)", cudaGetErrorString(e));
    war_server* s = new war_server();
    s->cfg = c;
    cudaGetDevice(&s->device);
    cudaDeviceGetAttribute(&s->sm_count, cudaDevAttrMultiProcessorCount, s->device);
    size_t fr = 0, tot = 0;
    cudaMemGetInfo(&fr, &tot);
    u64 budget = c.mem_budget ? c.mem_budget : fr / 2;
    s->nslots = (int)std::min<u64>((u64)c.max_jobs, budget / sizeof(DevAcc));
    if (s->nslots < 1) {
        delete s;
        return fail(WAR_ENOMEM, "memory budget %llu holds no job accumulator (%zu bytes each)", (unsigned long long)budget,
                    sizeof(DevAcc));
    }
    // the memo arena: what the budget leaves after the slots, at most 16 GiB, reserved now so that the
    // worker thread never allocates; a smaller one when the device cannot give that much
    if (c.memo_bits >= 0) {
        const u64 rest = budget - (u64)s->nslots * sizeof(DevAcc);
        u64 words = std::min<u64>(rest / sizeof(u64), 1ull << 31);
        while (words >= (1ull << 12)) {
            if (cudaMalloc(&s->memo_arena, words * sizeof(u64)) == cudaSuccess) break;
            s->memo_arena = nullptr;
            cudaGetLastError();
            words /= 2;
        }
        s->arena_words = s->memo_arena ? words : 0;
    }
    s->max_tasks = 16384;
    s->max_units = s->max_tasks + 4 * UNITS_PER_EXTRA_CAP;
    const size_t nblocks = (size_t)s->nslots * SLOT_BLOCKS;
    bool ok = cudaStreamCreateWithFlags(&s->s_comp, cudaStreamNonBlocking) == cudaSuccess &&
              upload_merge_table(&s->d_table, s->s_comp) == cudaSuccess &&
              cudaMalloc(&s->d_blocks, sizeof(MBlock) * nblocks) == cudaSuccess &&
              (s->h_blocks = (MBlock*)calloc(nblocks, sizeof(MBlock))) != nullptr &&
              cudaMalloc(&s->d_jobs, sizeof(MergeArgs) * (size_t)s->nslots) == cudaSuccess &&
              cudaMallocHost(&s->h_jobs, sizeof(MergeArgs) * (size_t)s->nslots) == cudaSuccess &&
              cudaMalloc(&s->d_slots, sizeof(DevAcc) * (size_t)s->nslots) == cudaSuccess &&
              cudaMallocHost(&s->h_slot, sizeof(DevAcc) * READBACK) == cudaSuccess &&
              cudaStreamCreateWithFlags(&s->s_copy, cudaStreamNonBlocking) == cudaSuccess;
    for (int i = 0; ok && i < 2; i++) {
        Tick& T = s->ticks[i];
        ok = cudaMallocHost(&T.h_tasks, sizeof(ServeTask) * s->max_tasks) == cudaSuccess &&
             cudaMallocHost(&T.h_refill, sizeof(RefillTask) * MAX_REFILL) == cudaSuccess &&
             cudaMallocHost(&T.h_units, sizeof(Unit) * (size_t)s->max_units * 8) == cudaSuccess &&
             cudaMalloc(&T.d_tasks, sizeof(ServeTask) * s->max_tasks) == cudaSuccess &&
             cudaMalloc(&T.d_refill, sizeof(RefillTask) * MAX_REFILL) == cudaSuccess &&
             cudaMalloc(&T.d_units, sizeof(Unit) * (size_t)s->max_units * 8) == cudaSuccess &&
             cudaEventCreateWithFlags(&T.ev, cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
        war_server_destroy(s);
        return fail(WAR_ENOMEM, "server buffers could not be allocated");
    }
    for (int i = s->nslots - 1; i >= 0; i--) s->free_slots.push_back(i);
    s->t0 = std::chrono::steady_clock::now();
    s->worker = std::thread(worker_main, s);
    *out = s;
    return WAR_OK;
}

int war_server_submit(war_server* s, const war_job* job, uint64_t* id) {
    if (!s || !id) return fail(WAR_EINVAL, "NULL server or id");
    int st = check_job(job);
    if (st) return st;
    std::lock_guard<std::mutex> lk(s->mu);
    if (s->fatal) return fail(s->fatal, "server stopped after a CUDA error");
    if ((int)s->pending.size() >= s->cfg.queue_cap) return fail(WAR_EBUSY, "queue full (%d jobs)", s->cfg.queue_cap);
    u64 k = s->next_id++;
    SJob& J = s->jobs[k];
    J.job = *job;
    J.result = new war_result();
    memset(J.result, 0, sizeof(war_result));
    J.result->hbins = job->hbins;
    J.result->dbins = job->dbins;
    J.result->blk = (job->flags & WAR_F_SHAPE) && job->mode == WAR_CANON ? (job->blk ? job->blk : (job->n & -job->n)) : 0;
    J.t_submit = s->now_ms();
    s->pending.push_back(k);
    *id = k;
    s->cv_work.notify_one();
    return WAR_OK;
}

int war_server_poll(war_server* s, uint64_t id, war_result* res, war_job_status* st) {
    if (!s) return fail(WAR_EINVAL, "NULL server");
    std::lock_guard<std::mutex> lk(s->mu);
    auto it = s->jobs.find(id);
    if (it == s->jobs.end()) return fail(WAR_ENOTFOUND, "no job %llu", (unsigned long long)id);
    SJob& J = it->second;
    if (st) {
        st->state = J.state; st->status = J.status;
        st->submit_ms = J.t_submit; st->admit_ms = J.t_admit; st->finish_ms = J.t_finish;
    }
    if (J.state < 2) return WAR_PENDING;
    int status = J.state == 2 ? WAR_OK : (J.status ? J.status : WAR_ECUDA);
    if (res && J.state == 2) *res = *J.result;
    delete J.result;
    s->jobs.erase(it);
    return status == WAR_OK ? WAR_OK : fail(status, "job %llu failed", (unsigned long long)id);
}

int war_server_drain(war_server* s, double timeout_ms) {
    if (!s) return fail(WAR_EINVAL, "NULL server");
    std::unique_lock<std::mutex> lk(s->mu);
    auto until = std::chrono::steady_clock::now() + std::chrono::microseconds((long long)(timeout_ms * 1000));
    bool ok = s->cv_done.wait_until(lk, until, [&] {
        if (!s->pending.empty()) return false;
        for (auto& kv : s->jobs) if (kv.second.state < 2) return false;
        return true;
    });
    return ok ? WAR_OK : fail(WAR_ETIMEOUT, "jobs still running after %.0f ms", timeout_ms);
}

int war_server_stats(war_server* s, uint64_t* ticks, uint64_t* jobs_done, uint64_t* peak_resident) {
    if (!s) return fail(WAR_EINVAL, "NULL server");
    std::lock_guard<std::mutex> lk(s->mu);
    if (ticks) *ticks = s->nticks;
    if (jobs_done) *jobs_done = s->jobs_done;
    if (peak_resident) *peak_resident = s->peak_resident;
    return WAR_OK;
}

int war_server_memo_info(war_server* s, uint64_t* arena_bytes, uint64_t* used_bytes, int32_t* classes) {
    if (!s) return fail(WAR_EINVAL, "NULL server");
    std::lock_guard<std::mutex> lk(s->mu);
    int k = 0;
    for (auto& kv : s->memos)
        if (kv.second.first) k++;
    if (arena_bytes) *arena_bytes = s->arena_words * sizeof(u64);
    if (used_bytes) *used_bytes = s->arena_used * sizeof(u64);
    if (classes) *classes = k;
    return WAR_OK;
}

int war_server_destroy(war_server* s) {
    if (!s) return WAR_OK;
    {
        std::lock_guard<std::mutex> lk(s->mu);
        s->stop = true;
        s->pending.clear();
        for (auto& kv : s->jobs)
            if (kv.second.state == 0) { kv.second.state = 3; kv.second.status = WAR_EINVAL; }
        s->cv_work.notify_all();
    }
    if (s->worker.joinable()) s->worker.join();
    for (auto& kv : s->jobs) delete kv.second.result;
    for (int i = 0; i < 2; i++) {
        Tick& T = s->ticks[i];
        if (T.h_tasks) cudaFreeHost(T.h_tasks);
        if (T.h_refill) cudaFreeHost(T.h_refill);
        if (T.h_units) cudaFreeHost(T.h_units);
        if (T.d_tasks) cudaFree(T.d_tasks);
        if (T.d_refill) cudaFree(T.d_refill);
        if (T.d_units) cudaFree(T.d_units);
        if (T.ev) cudaEventDestroy(T.ev);
    }
    if (s->memo_arena) cudaFree(s->memo_arena);
    if (s->d_table) cudaFree(s->d_table);
    if (s->d_jobs) cudaFree(s->d_jobs);
    if (s->h_jobs) cudaFreeHost(s->h_jobs);
    if (s->d_blocks) cudaFree(s->d_blocks);
    free(s->h_blocks);
    if (s->d_slots) cudaFree(s->d_slots);
    if (s->h_slot) cudaFreeHost(s->h_slot);
    if (s->s_comp) cudaStreamDestroy(s->s_comp);
    if (s->s_copy) cudaStreamDestroy(s->s_copy);
    delete s;
    return WAR_OK;
}

}  // extern "C"

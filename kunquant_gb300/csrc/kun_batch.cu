// Many universes of one module in one run, and the launch-shape autotuner.
//
// kunRunGraphBatch runs `njobs` jobs (universes of their own stock count and
// length) of one batch module.  Stage by stage in the module's order, a
// time-series stage that supports grouped launches runs each of its kernels
// ONCE over the tiles of all jobs (the job of a block is found from a tile
// table passed by value); a Rank stage ranks every job's rows in one launch;
// other stages run job by job.  The jobs' parameter
// blocks go to the device with one copy per stage.  On an executor of several
// streams the kernels of all stages run as one graph of nodes (kun_plan.cu)
// after one copy of all blocks.  This replaces the reference's one runGraph per
// universe (cpp/Kun/Runtime.cpp:311-352).
//
// kunExecutorTune picks, per stage, the time tile of the time-parallel
// kernels and the threads per block by timing candidate shapes on the jobs
// given (CUDA events on the executor's stream), keeping the fastest.  The
// executor then uses those shapes in kunRunGraphBatch and kunRunGraphEx.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "kun_runtime_internal.h"
#include "kun_xsec.cuh"

namespace kungpu {

// jobs per grouped launch (the modules' tile tables hold this many)
static constexpr int KUN_GROUP_MAX = 256;

static bool batch_device_pointer(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

struct BatchJob {
    long long S, total_time, cur_time, length;
    const Plan *plan;
    std::vector<void *> ptrs;
    size_t arena_off, slot_bytes;
};

struct BatchRun {
    Executor *ex;
    const KunGpuModuleDesc *m;
    std::vector<BatchJob> jobs;
    std::vector<int> order;
    const Plan *nodes = nullptr;  // the jobs' common plan in kernels, or null: stage by stage
    size_t host_off = 0;          // parameter blocks staged so far in this run
};

// The plan in kernels that all jobs share on a multi-stream executor: slots
// are numbered alike in every job's part of the arena, and the kernels are
// weighed by the jobs' summed cells.  Null when the module or memory has none.
static const Plan *batch_node_plan(Executor *ex, const KunGpuModuleDesc *m, const std::vector<BatchJob> &jobs) {
    const int ns = node_streams(ex);
    if (ns < 2 || jobs.size() < 2) return nullptr;
    long long cells = 0, rows = 0;
    size_t slot_bytes = 0;
    for (const BatchJob &jb : jobs) {
        cells += jb.S * jb.length;
        rows = std::max(rows, jb.length);
        slot_bytes += jb.slot_bytes;
    }
    auto key = std::make_tuple((const void *)m, -cells, -rows, ns);  // negative: not a single run's
    auto it = ex->plans.find(key);
    if (it == ex->plans.end()) {
        Plan p;
        if (!make_plan(m, jobs[0].S, jobs[0].length, ns, p)) return nullptr;
        p.slot_bytes = slot_bytes;
        make_node_plan(m, (double)cells, (double)rows, ns, node_slots(p), p);
        it = ex->plans.emplace(key, std::move(p)).first;
    }
    return it->second.nodes.empty() ? nullptr : &it->second;
}

static KunStatus batch_setup(Executor *ex, const KunGpuModuleDesc *m, int njobs, const NameMap *const *maps,
                             const size_t *S, const size_t *total_time, const size_t *cur_time,
                             const size_t *length, bool by_kernel, BatchRun &br) {
    if (!ex || !m || njobs <= 0 || !maps || !S || !total_time || !cur_time || !length) {
        set_error("kunRunGraphBatch: bad arguments");
        return KUN_INVALID_ARGUMENT;
    }
    if (m->abi != KUN_GPU_MODULE_ABI) {
        set_error("The required version in the module does not match the runtime version");
        return KUN_INVALID_ARGUMENT;
    }
    if (m->output_layout == KUN_LAYOUT_STREAM) {
        set_error("Cannot run stream mode module via runGraph()");
        return KUN_INVALID_ARGUMENT;
    }
    br.ex = ex;
    br.m = m;
    br.jobs.resize(njobs);
    size_t total = 0;
    for (int j = 0; j < njobs; j++) {
        BatchJob &jb = br.jobs[j];
        jb.S = (long long)S[j];
        jb.total_time = (long long)total_time[j];
        jb.cur_time = (long long)cur_time[j];
        jb.length = (long long)length[j];
        if (jb.S <= 0 || jb.length <= 0 || jb.cur_time + jb.length > jb.total_time || !maps[j]) {
            set_error("kunRunGraphBatch: bad shape of job %d", j);
            return KUN_INVALID_ARGUMENT;
        }
        if (m->aligned && m->input_layout == KUN_LAYOUT_TS && (jb.S % m->blocking_len) != 0) {
            set_error("Bad shape: num_stocks %lld of job %d is not a multiple of %d", jb.S, j, m->blocking_len);
            return KUN_INVALID_ARGUMENT;
        }
        auto key = std::make_tuple((const void *)m, jb.S, jb.length, 1);
        auto it = ex->plans.find(key);
        if (it == ex->plans.end()) {
            Plan p;
            if (!make_plan(m, jb.S, jb.length, 1, p)) return KUN_INVALID_ARGUMENT;
            it = ex->plans.emplace(key, std::move(p)).first;
        }
        jb.plan = &it->second;
        jb.slot_bytes = jb.plan->slot_bytes;
    }
    br.order = br.jobs[0].plan->order;
    if (by_kernel && (br.nodes = batch_node_plan(ex, m, br.jobs)))
        for (BatchJob &jb : br.jobs) jb.plan = br.nodes;
    for (BatchJob &jb : br.jobs) {
        jb.arena_off = total;
        total += (jb.slot_bytes * (size_t)jb.plan->num_slots + 255) / 256 * 256;
    }
    if (!ex->arena.ensure(total) && br.nodes) {  // the plan in stages may need less
        br = BatchRun();
        return batch_setup(ex, m, njobs, maps, S, total_time, cur_time, length, false, br);
    }
    if (ex->arena.bytes < total) {
        set_error("out of device memory for the temporaries of %d jobs (%zu bytes)", njobs, total);
        return KUN_OUT_OF_MEMORY;
    }
    for (int j = 0; j < njobs; j++) {
        BatchJob &jb = br.jobs[j];
        jb.ptrs.assign(m->num_buffers, nullptr);
        for (int b = 0; b < m->num_buffers; b++) {
            const KunGpuBufferDesc &bd = m->buffers[b];
            if (bd.kind == KUN_BUF_TEMP) {
                if (jb.plan->temp_slot[b] >= 0)
                    jb.ptrs[b] = (char *)ex->arena.ptr + jb.arena_off +
                                 jb.slot_bytes * (size_t)jb.plan->temp_slot[b];
                continue;
            }
            auto f = maps[j]->find(bd.name);
            if (f == maps[j]->end() || !f->second) {
                set_error("Buffer name not found: %s (job %d)", bd.name, j);
                return KUN_INVALID_ARGUMENT;
            }
            if (!batch_device_pointer(f->second)) {
                set_error("kunRunGraphBatch: buffer %s of job %d is not device memory", bd.name, j);
                return KUN_INVALID_ARGUMENT;
            }
            jb.ptrs[b] = f->second;
        }
    }
    return KUN_SUCCESS;
}

static bool ensure_group_staging(Executor *ex, size_t need) {
    if (need <= ex->group_host_bytes) return ex->group_dev.ensure(need);
    if (ex->group_host) cudaFreeHost(ex->group_host);
    ex->group_host = nullptr;
    ex->group_host_bytes = 0;
    if (cudaHostAlloc(&ex->group_host, need, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    ex->group_host_bytes = need;
    return ex->group_dev.ensure(need);
}

// One stage's launch arguments for every job, and its parameter blocks (or
// the grouped Rank's job table) in the pinned staging.
struct StageBlocks {
    std::vector<std::vector<void *>> scratch;
    std::vector<KunGpuStageArgs> args;
    std::vector<size_t> off;  // per group of KUN_GROUP_MAX jobs
    // the grouped Rank's launches: jobs of like length, so that a block has the
    // threads and shared memory its rows need.  A class more costs 2 to 5 us a
    // stage, a wide one costs blocks that its short rows leave idle (us a stage,
    // these four classes and one: 48 universes of 37 to 6000 stocks x 250 to 5000
    // days 1613 and 2786; 12 of 37 to 3000 x 250 to 1250 149 and 152; 24 of 400 to
    // 600 x 1000 230 and 228).
    struct RankClass {
        int first, jobs;
        long long rows, longest;
    };
    bool rank = false;
    std::vector<RankClass> classes;
};
static int rank_class(long long S) { return S <= 128 ? 0 : (S <= 512 ? 1 : (S <= 2048 ? 2 : 3)); }

static KunStatus stage_blocks(BatchRun &br, int si, const int32_t *tile, const int32_t *block, StageBlocks &sb) {
    Executor *ex = br.ex;
    const KunGpuModuleDesc *m = br.m;
    const KunGpuStageDesc &d = m->stages[si];
    const int n = (int)br.jobs.size();
    sb.scratch.resize(n);
    sb.args.resize(n);
    auto tn = ex->tuning.find((const void *)m);
    for (int j = 0; j < n; j++) {
        BatchJob &jb = br.jobs[j];
        for (int sl : jb.plan->scratch[si])
            sb.scratch[j].push_back((char *)ex->arena.ptr + jb.arena_off + jb.slot_bytes * (size_t)sl);
        KunGpuStageArgs &a = sb.args[j];
        memset(&a, 0, sizeof a);
        a.buffers = jb.ptrs.data();
        a.scratch = sb.scratch[j].data();
        a.num_stocks = jb.S;
        a.total_time = jb.total_time;
        a.start = jb.cur_time;
        a.length = jb.length;
        a.error_flag = ex->d_error;
        if (tile) {
            a.tune_tile = tile;
            a.tune_block = block;
        } else if (tn != ex->tuning.end() && si < (int)tn->second.size() && !tn->second[si].tile.empty()) {
            a.tune_tile = tn->second[si].tile.data();
            a.tune_block = tn->second[si].block.data();
        }
    }
    auto stage_room = [&](size_t bytes) {
        const size_t off = (br.host_off + 255) / 256 * 256;
        if (off + bytes > ex->group_host_bytes) {
            set_error("grouped launch staging exhausted");
            return false;
        }
        sb.off.push_back(off);
        br.host_off = off + bytes;
        return true;
    };
    // Rank stages in the TS layout: every job's rows in one launch
    sb.rank = d.kind == KUN_STAGE_RANK && n > 1 && d.num_in == 1 && d.num_out == 1 &&
              (m->buffers[d.in_bufs[0]].kind != KUN_BUF_INPUT || m->input_layout == KUN_LAYOUT_TS) &&
              (m->buffers[d.out_bufs[0]].kind != KUN_BUF_OUTPUT || m->output_layout == KUN_LAYOUT_TS);
    if (sb.rank) {
        const int bi = d.in_bufs[0], bo = d.out_bufs[0];
        const size_t esz = m->dtype == 0 ? 4 : 8;
        std::vector<kun::RankRowsJob> jobs;
        for (int j = 0; j < n; j++) {
            const BatchJob &jb = br.jobs[j];
            if (jb.S <= 0 || jb.length <= 0) continue;
            kun::RankRowsJob rj;
            const long long row_off = m->buffers[bi].kind == KUN_BUF_INPUT ? jb.cur_time : 0;
            rj.in = (const char *)jb.ptrs[bi] + (size_t)row_off * (size_t)jb.S * esz;
            rj.out = jb.ptrs[bo];
            rj.S = jb.S;
            rj.length = jb.length;
            jobs.push_back(rj);
        }
        std::stable_sort(jobs.begin(), jobs.end(), [](const kun::RankRowsJob &a, const kun::RankRowsJob &b) {
            return rank_class(a.S) > rank_class(b.S);  // the longest rows first
        });
        for (size_t j = 0; j < jobs.size(); j++) {
            if (j == 0 || rank_class(jobs[j].S) != rank_class(jobs[j - 1].S)) sb.classes.push_back({(int)j, 0, 0, 0});
            StageBlocks::RankClass &c = sb.classes.back();
            jobs[j].row0 = c.rows;
            c.jobs++;
            c.rows += jobs[j].length;
            c.longest = std::max(c.longest, jobs[j].S);
        }
        if (!stage_room(jobs.size() * sizeof(kun::RankRowsJob))) return KUN_OUT_OF_MEMORY;
        memcpy((char *)ex->group_host + sb.off[0], jobs.data(), jobs.size() * sizeof(kun::RankRowsJob));
    } else if (d.launch_group && n > 1) {
        for (int j0 = 0; j0 < n; j0 += KUN_GROUP_MAX) {
            const int nj = std::min(KUN_GROUP_MAX, n - j0);
            if (!stage_room(d.prepare(&sb.args[j0], nj, nullptr))) return KUN_OUT_OF_MEMORY;
            d.prepare(&sb.args[j0], nj, (char *)ex->group_host + sb.off.back());
        }
    }
    return KUN_SUCCESS;
}

// Launches a stage (kernel < 0) or one of its kernels, its blocks on the device
static KunStatus launch_blocks(BatchRun &br, int si, int kernel, StageBlocks &sb, cudaStream_t st, int64_t &launches) {
    const KunGpuModuleDesc *m = br.m;
    const KunGpuStageDesc &d = m->stages[si];
    const int n = (int)br.jobs.size();
    char *dev = (char *)br.ex->group_dev.ptr;
    const int kernels = kernel >= 0 || d.num_kernels <= 0 ? 1 : d.num_kernels;
    auto failed = [&](const char *what, int rc) {
        set_error("stage %d (%s) %s failed: %s", si, d.name, what, cudaGetErrorString((cudaError_t)rc));
        return KUN_CUDA_ERROR;
    };
    if (sb.rank) {
        const auto *jobs = (const kun::RankRowsJob *)(dev + sb.off[0]);
        for (const StageBlocks::RankClass &c : sb.classes) {
            int rc = m->dtype == 0 ? kun::launch_rank_rows_multi<float>(jobs + c.first, c.jobs, c.rows, c.longest, st)
                                   : kun::launch_rank_rows_multi<double>(jobs + c.first, c.jobs, c.rows, c.longest, st);
            if (rc) return failed("grouped Rank", rc);
            launches += 1;
        }
        return KUN_SUCCESS;
    }
    for (KunGpuStageArgs &a : sb.args) a.only_kernel = kernel + 1;
    if (!sb.off.empty()) {
        for (size_t g = 0; g < sb.off.size(); g++) {
            const int j0 = (int)g * KUN_GROUP_MAX;
            if (int rc = d.launch_group(&sb.args[j0], std::min(KUN_GROUP_MAX, n - j0), dev + sb.off[g], (void *)st))
                return failed("grouped launch", rc);
            launches += kernels;
        }
        return KUN_SUCCESS;
    }
    for (int j = 0; j < n; j++) {
        if (int rc = d.launch(&sb.args[j], (void *)st)) {
            set_error("stage %d (%s) launch failed for job %d: %s", si, d.name, j,
                      cudaGetErrorString((cudaError_t)rc));
            return KUN_CUDA_ERROR;
        }
        launches += kernels;
    }
    return KUN_SUCCESS;
}

static void copy_blocks(BatchRun &br, size_t from, cudaStream_t st) {
    if (br.host_off > from)
        cudaMemcpyAsync((char *)br.ex->group_dev.ptr + from, (char *)br.ex->group_host + from, br.host_off - from,
                        cudaMemcpyHostToDevice, st);
}

// Enqueue stage `si` for every job; `tile`/`block` override the tuning table.
static KunStatus batch_stage(BatchRun &br, int si, cudaStream_t st, const int32_t *tile, const int32_t *block,
                             int64_t &launches) {
    StageBlocks sb;
    const size_t from = br.host_off;
    KunStatus rs = stage_blocks(br, si, tile, block, sb);
    if (rs != KUN_SUCCESS) return rs;
    copy_blocks(br, from, st);
    return launch_blocks(br, si, -1, sb, st, launches);
}

// Every kernel of the module on the executor's streams: all parameter blocks
// go to the device in one copy, then each kernel runs once over all jobs as
// soon as what it reads is there.
static KunStatus batch_nodes(BatchRun &br, cudaStream_t st, int64_t &launches) {
    std::vector<StageBlocks> blocks(br.m->num_stages);
    KunStatus rs = KUN_SUCCESS;
    for (int si : br.order)
        if ((rs = stage_blocks(br, si, nullptr, nullptr, blocks[si])) != KUN_SUCCESS) return rs;
    copy_blocks(br, 0, st);
    run_nodes(br.ex, *br.nodes, st, [&](int, const PlanNode &n, cudaStream_t on) {
        return (rs = launch_blocks(br, n.stage, n.kernel, blocks[n.stage], on, launches)) == KUN_SUCCESS;
    });
    return rs;
}

// bytes of the parameter blocks of one pass over all stages
static size_t batch_staging_bytes(const BatchRun &br) {
    size_t need = 0;
    const int n = (int)br.jobs.size();
    for (int si = 0; si < br.m->num_stages; si++) {
        const KunGpuStageDesc &d = br.m->stages[si];
        if (d.kind == KUN_STAGE_RANK && n > 1) {  // the grouped Rank's job table
            need += ((size_t)n * sizeof(kun::RankRowsJob) + 255) / 256 * 256;
            continue;
        }
        if (!d.launch_group || n <= 1) continue;
        std::vector<KunGpuStageArgs> args(n);
        memset(args.data(), 0, sizeof(KunGpuStageArgs) * n);
        for (int j0 = 0; j0 < n; j0 += KUN_GROUP_MAX)
            need += (d.prepare(&args[j0], std::min(KUN_GROUP_MAX, n - j0), nullptr) + 255) / 256 * 256;
    }
    return need + 256;
}

static KunStatus batch_begin(Executor *ex, BatchRun &br, size_t passes) {
    if (!ensure_group_staging(ex, batch_staging_bytes(br) * passes)) {
        set_error("out of memory for grouped launch staging");
        return KUN_OUT_OF_MEMORY;
    }
    br.host_off = 0;
    return KUN_SUCCESS;
}

static KunStatus batch_finish(Executor *ex, cudaStream_t st, bool sync) {
    if (ex->has_user_stream) {
        cudaEventRecord(ex->bridge_out, st);
        cudaStreamWaitEvent(ex->user_stream, ex->bridge_out, 0);
    }
    // the pinned staging is reused by the next run: always wait for the copies
    (void)sync;
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        set_error("CUDA error: %s", cudaGetErrorString(e));
        return KUN_CUDA_ERROR;
    }
    return KUN_SUCCESS;
}

}  // namespace kungpu

using namespace kungpu;

KUN_EXPORT KunStatus kunRunGraphBatch(KunExecutorHandle exec, KunModuleHandle mod, int njobs,
                                      const KunBufferNameMapHandle *buffers, const size_t *num_stocks,
                                      const size_t *total_time, const size_t *cur_time, const size_t *length,
                                      int synchronize) {
    clear_error();
    auto *ex = (Executor *)exec;
    if (!ex) return KUN_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(ex->mu);
    cudaSetDevice(ex->device);
    ex->check_epoch();
    BatchRun br;
    KunStatus rs = batch_setup(ex, (const KunGpuModuleDesc *)mod, njobs, (const NameMap *const *)buffers,
                               num_stocks, total_time, cur_time, length, !ex->profile, br);
    if (rs != KUN_SUCCESS) return rs;
    if ((rs = batch_begin(ex, br, 1)) != KUN_SUCCESS) return rs;
    cudaStream_t st = ex->stream();
    if (ex->has_user_stream) {
        cudaEventRecord(ex->bridge_in, ex->user_stream);
        cudaStreamWaitEvent(st, ex->bridge_in, 0);
    }
    int64_t launches = 0;
    if (br.nodes) rs = batch_nodes(br, st, launches);
    for (int si : br.order)
        if (!br.nodes && rs == KUN_SUCCESS) rs = batch_stage(br, si, st, nullptr, nullptr, launches);
    if (rs != KUN_SUCCESS) {
        drain(ex);
        return rs;
    }
    ex->last_launches = launches;
    return batch_finish(ex, st, synchronize != 0);
}

// Tune the launch shapes of every grouped-capable stage on these jobs (the
// jobs' outputs are computed along the way).  Candidates: time tiles
// {default, 16, 32, 64, 128, 256} x {64, 128} threads per block for all the
// time-parallel kernels of a stage together, {32, 64, 128} threads for its
// scan kernels; then per time-parallel kernel, with the others held: its
// 64-register instance (if it has one) or not x block size, then its tile.  Each candidate
// runs the stage `reps` times after one warm-up; the fastest mean wins.
// Returns the number of stages tuned, or -1 on error.
KUN_EXPORT int kunExecutorTune(KunExecutorHandle exec, KunModuleHandle mod, int njobs,
                               const KunBufferNameMapHandle *buffers, const size_t *num_stocks,
                               const size_t *total_time, const size_t *cur_time, const size_t *length, int reps) {
    clear_error();
    auto *ex = (Executor *)exec;
    if (!ex) return -1;
    std::lock_guard<std::mutex> lk(ex->mu);
    cudaSetDevice(ex->device);
    ex->check_epoch();
    const auto *m = (const KunGpuModuleDesc *)mod;
    BatchRun br;
    if (batch_setup(ex, m, njobs, (const NameMap *const *)buffers, num_stocks, total_time, cur_time, length, false,
                    br) != KUN_SUCCESS)
        return -1;
    struct AtEnd {  // also where a stage's launch fails
        Executor *ex;
        ~AtEnd() { drain(ex); }
    } at_end{ex};
    reps = std::max(1, reps);
    const int tiles[] = {0, 16, 32, 64, 128, 256};
    const int blocks[] = {64, 128};
    const int sblocks[] = {32, 64, 128};
    // each candidate run stages its parameter blocks once per repetition
    const size_t passes = (sizeof(tiles) / sizeof(int)) * (sizeof(blocks) / sizeof(int)) * (size_t)(reps + 1) + 4;
    if (batch_begin(ex, br, passes) != KUN_SUCCESS) return -1;
    cudaStream_t st = ex->stream();
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto &table = ex->tuning[(const void *)m];
    table.assign(m->num_stages, Executor::StageTune());
    int tuned = 0;
    int64_t launches = 0;
    for (int si : br.order) {
        const KunGpuStageDesc &d = m->stages[si];
        if (!d.kernel_info || d.num_kernels <= 0) {
            if (batch_stage(br, si, st, nullptr, nullptr, launches) != KUN_SUCCESS) return -1;
            continue;
        }
        const int nk = d.num_kernels;
        bool has_par = false, has_scan = false;
        for (int k = 0; k < nk; k++) (d.kernel_info[k] & 1 ? has_scan : has_par) = true;
        std::vector<int32_t> best_t(nk, 0), best_b(nk, 0), t(nk), b(nk);
        float best = -1.f;
        // times the stage with shape (t, b); keeps it when fastest so far
        auto run = [&]() -> bool {
            // the staging area is reused from its start: the copies of every
            // earlier launch (this stage's trials, and the untuned stages
            // enqueued before it) must have left it
            if (cudaStreamSynchronize(st) != cudaSuccess) return false;
            br.host_off = 0;
            if (batch_stage(br, si, st, t.data(), b.data(), launches) != KUN_SUCCESS) return false;
            cudaEventRecord(e0, st);
            for (int r = 0; r < reps; r++) {
                if (batch_stage(br, si, st, t.data(), b.data(), launches) != KUN_SUCCESS) return false;
            }
            cudaEventRecord(e1, st);
            if (cudaEventSynchronize(e1) != cudaSuccess) return false;
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            if (best < 0 || ms < best) {
                best = ms;
                best_t = t;
                best_b = b;
            }
            return true;
        };
        auto trial = [&](int tile, int blk, int sblk) -> bool {
            for (int k = 0; k < nk; k++) {
                const bool scan = d.kernel_info[k] & 1;
                t[k] = scan ? 0 : tile;
                b[k] = scan ? sblk : blk;
            }
            return run();
        };
        // one shape for every kernel of the stage first
        for (int tile : tiles) {
            if (!has_par && tile != 0) continue;
            for (int blk : blocks) {
                if (!has_par && blk != 128) continue;
                if (!trial(tile, blk, 128)) return -1;
            }
        }
        if (has_scan) {
            std::vector<int32_t> pt = best_t, pb = best_b;
            for (int sblk : sblocks) {
                int tile = 0, blk = 128;
                for (int k = 0; k < nk; k++)
                    if (!(d.kernel_info[k] & 1)) {
                        tile = pt[k];
                        blk = pb[k];
                    }
                if (!trial(tile, blk, sblk)) return -1;
            }
        }
        // then each time-parallel kernel on its own: the 64-register
        // instance and the block size, then the tile, the others held at
        // their best
        for (int k = 0; k < nk && has_par; k++) {
            if (d.kernel_info[k] & 1) continue;
            for (int cap : {0, (int)KUN_BLOCK_REGCAP}) {
                if (cap && !(d.kernel_info[k] & KUN_KERNEL_CAPPED)) continue;
                for (int blk : blocks) {
                    t = best_t;
                    b = best_b;
                    b[k] = blk | cap;
                    if (b[k] == best_b[k]) continue;
                    if (!run()) return -1;
                }
            }
            for (int tile : tiles) {
                t = best_t;
                b = best_b;
                if (tile == t[k]) continue;
                t[k] = tile;
                if (!run()) return -1;
            }
        }
        table[si].tile = best_t;
        table[si].block = best_b;
        // leave the stage's outputs from the chosen shape
        br.host_off = 0;
        if (batch_stage(br, si, st, best_t.data(), best_b.data(), launches) != KUN_SUCCESS) return -1;
        if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
        tuned++;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    // graphs captured before tuning used the old shapes
    for (auto &g : ex->graphs) cudaGraphExecDestroy(g.exec);
    ex->graphs.clear();
    ex->seen.clear();
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    return tuned;
}

// The tuned shape of one stage: fills up to `cap` kernels' tiles and blocks;
// returns the kernel count, 0 when the stage has no tuned shape.
KUN_EXPORT int kunExecutorTunedShape(KunExecutorHandle exec, KunModuleHandle mod, int stage, int32_t *tile,
                                     int32_t *block, int cap) {
    auto *ex = (Executor *)exec;
    if (!ex) return -1;
    auto it = ex->tuning.find((const void *)mod);
    if (it == ex->tuning.end() || stage < 0 || stage >= (int)it->second.size()) return 0;
    const auto &tn = it->second[stage];
    int n = (int)tn.tile.size();
    for (int k = 0; k < std::min(n, cap); k++) {
        if (tile) tile[k] = tn.tile[k];
        if (block) block[k] = tn.block[k];
    }
    return n;
}

KUN_EXPORT KunStatus kunExecutorClearTuning(KunExecutorHandle exec) {
    auto *ex = (Executor *)exec;
    if (!ex) return KUN_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(ex->mu);
    ex->tuning.clear();
    for (auto &g : ex->graphs) cudaGraphExecDestroy(g.exec);
    ex->graphs.clear();
    ex->seen.clear();
    return KUN_SUCCESS;
}

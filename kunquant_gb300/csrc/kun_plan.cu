// Plans in kernels.
//
// The front end's partition leaves a module's stages in long chains: a stage
// waits for whole stages although each of its kernels reads a few series only
// (Alpha101: the chain of stages is 79% of the kernels' summed time, the chain
// of kernels 6%).  Small and medium runs, whose kernels leave most of the GPU
// idle, took the chain's time.  Here every kernel is a node that follows the
// writers of what it reads; the nodes are laid on the executor's streams by
// list scheduling (longest remaining chain first, with estimated times), and
// the arena's slots are handed out along that schedule: a slot whose last
// readers have finished by then is reused, with the order made explicit, so
// that reuse costs the schedule nothing and the arena stays near the live set.
#include <algorithm>
#include <cstring>
#include <queue>

#include "kun_runtime_internal.h"

namespace kungpu {

namespace {

struct Node {
    int stage, kernel;
    double us;
    std::vector<int> reads, writes;  // values: buffer id, or num_buffers + the module's scratch number
    std::vector<int> preds, succs;
};

// Rough times at full occupancy (40e6 instructions a microsecond, half of them
// issued) and of the shortest launches; a scan walks its rows one by one
// whatever the number of stocks.
double par_us(double cells, double inst) { return 4 + cells * inst / 20e6; }
double scan_us(double cells, double inst, double rows) { return 6 + std::max(rows * 0.035, cells * inst / 20e6); }

bool collect(const KunGpuModuleDesc *m, const std::vector<int> &order, double cells, double rows,
             std::vector<Node> &nodes) {
    const int nb = m->num_buffers;
    std::vector<int> first_scratch(m->num_stages + 1, nb);
    for (int i = 0; i < m->num_stages; i++) first_scratch[i + 1] = first_scratch[i] + m->stages[i].num_scratch;
    std::vector<int> writer(first_scratch[m->num_stages], -1);
    for (int si : order) {
        const KunGpuStageDesc &s = m->stages[si];
        if (!s.kernel_info) {
            Node n{si, -1, 0, {}, {}, {}, {}};
            n.reads.assign(s.in_bufs, s.in_bufs + s.num_in);
            n.writes.assign(s.out_bufs, s.out_bufs + s.num_out);
            for (int k = 0; k < s.num_scratch; k++) n.writes.push_back(first_scratch[si] + k);
            n.us = s.kind == KUN_STAGE_SCALE ? 10 + rows * 0.01 : par_us(cells, 250);
            nodes.push_back(n);
            continue;
        }
        const int32_t *q = s.kernel_info + s.num_kernels;
        for (int k = 0; k < s.num_kernels; k++) {
            Node n{si, k, 0, {}, {}, {}, {}};
            const double inst = *q++;
            for (auto *list : {&n.reads, &n.writes})
                for (int c = *q++; c > 0; c--, q++) list->push_back(*q >= 0 ? *q : first_scratch[si] - 1 - *q);
            n.us = (s.kernel_info[k] & 1) ? scan_us(cells, inst, rows) : par_us(cells, inst);
            nodes.push_back(n);
        }
    }
    for (int i = 0; i < (int)nodes.size(); i++)
        for (int v : nodes[i].writes) {
            if (writer[v] >= 0) return false;  // each value has one writer
            writer[v] = i;
        }
    for (int i = 0; i < (int)nodes.size(); i++) {
        Node &n = nodes[i];
        for (int v : n.reads) {
            const bool input = v < nb && m->buffers[v].kind == KUN_BUF_INPUT;
            if (input) continue;
            const int w = writer[v];
            if (w < 0 || w >= i) return false;  // written earlier in the stages' order
            if (std::find(n.preds.begin(), n.preds.end(), w) == n.preds.end()) {
                n.preds.push_back(w);
                nodes[w].succs.push_back(i);
            }
        }
    }
    return true;
}

}  // namespace

bool make_node_plan(const KunGpuModuleDesc *m, double cells, double rows, int nstreams, int max_slots, Plan &p) {
    const int nb = m->num_buffers;
    std::vector<Node> nodes;
    if (nstreams < 2 || !collect(m, p.order, cells, rows, nodes)) return false;
    const int N = (int)nodes.size();
    std::vector<double> chain(N);
    for (int i = N - 1; i >= 0; i--) {
        chain[i] = 0;
        for (int s : nodes[i].succs) chain[i] = std::max(chain[i], chain[s]);
        chain[i] += nodes[i].us;
    }
    // slots are for temporaries and scratch; a value is free after its last
    // reader, or its writer when nobody reads it
    int values = nb;
    for (int i = 0; i < m->num_stages; i++) values += m->stages[i].num_scratch;
    std::vector<int> slot(values, -1), readers(values, 0);
    auto in_arena = [&](int v) { return v >= nb || m->buffers[v].kind == KUN_BUF_TEMP; };
    for (const Node &n : nodes)
        for (int v : n.reads) readers[v]++;
    std::vector<std::vector<int>> touched(values);
    struct Free {
        int slot;
        std::vector<int> after;
    };
    std::vector<Free> free_slots;  // longest free first
    int num_slots = 0;

    auto less_chain = [&](int a, int b) { return chain[a] != chain[b] ? chain[a] < chain[b] : a > b; };
    std::priority_queue<int, std::vector<int>, decltype(less_chain)> ready(less_chain);
    std::vector<int> pending(N);
    for (int i = 0; i < N; i++)
        if ((pending[i] = (int)nodes[i].preds.size()) == 0) ready.push(i);
    using Run = std::pair<double, int>;
    std::priority_queue<Run, std::vector<Run>, std::greater<Run>> running;
    std::vector<int> idle, tail(nstreams, -1);
    for (int k = nstreams - 1; k >= 0; k--) idle.push_back(k);
    std::vector<int> at(N, -1);  // node -> its place in the launch order
    std::vector<PlanNode> out;
    std::vector<std::vector<int>> follows;  // by place: places of the nodes it follows
    double now = 0;
    while (!ready.empty() || !running.empty()) {
        while (!ready.empty() && !idle.empty()) {
            const int i = ready.top();
            ready.pop();
            // a stream whose last node this one follows needs no event
            size_t pick = idle.size() - 1;
            for (size_t k = 0; k < idle.size(); k++)
                if (tail[idle[k]] >= 0 &&
                    std::find(nodes[i].preds.begin(), nodes[i].preds.end(), tail[idle[k]]) != nodes[i].preds.end())
                    pick = k;
            const int stream = idle[pick];
            idle.erase(idle.begin() + pick);
            std::vector<int> after;
            for (int q : nodes[i].preds) after.push_back(at[q]);
            for (int v : nodes[i].writes) {
                if (!in_arena(v)) continue;
                if (free_slots.empty()) {
                    if (num_slots >= max_slots) return false;
                    slot[v] = num_slots++;
                } else {
                    slot[v] = free_slots.front().slot;
                    for (int q : free_slots.front().after) after.push_back(at[q]);
                    free_slots.erase(free_slots.begin());
                }
            }
            at[i] = (int)out.size();
            PlanNode pn{nodes[i].stage, nodes[i].kernel, stream, false, {}, {}};
            for (int v : nodes[i].writes)
                if (v < nb && m->buffers[v].kind == KUN_BUF_OUTPUT) pn.outs.push_back(v);
            out.push_back(pn);
            follows.push_back(after);
            tail[stream] = i;
            running.push({now + nodes[i].us, i});
        }
        now = running.top().first;
        const int i = running.top().second;
        running.pop();
        idle.push_back(out[at[i]].stream);
        auto release = [&](int v) { free_slots.push_back({slot[v], touched[v]}); };
        for (int v : nodes[i].reads) {
            if (slot[v] < 0) continue;
            touched[v].push_back(i);
            if (--readers[v] == 0) release(v);
        }
        for (int v : nodes[i].writes)
            if (slot[v] >= 0 && readers[v] == 0 && touched[v].empty()) {
                touched[v].push_back(i);
                release(v);
            }
        for (int s : nodes[i].succs)
            if (--pending[s] == 0) ready.push(s);
    }
    if ((int)out.size() != N) return false;
    // events: per node the last node of each other stream that it follows,
    // unless an earlier node of its stream has waited for that one or a later
    std::vector<std::vector<int>> seen(nstreams, std::vector<int>(nstreams, -1));
    for (int i = 0; i < N; i++) {
        std::vector<int> last(nstreams, -1);
        for (int q : follows[i]) last[out[q].stream] = std::max(last[out[q].stream], q);
        for (int k = 0; k < nstreams; k++) {
            int &s = seen[out[i].stream][k];
            if (k == out[i].stream || last[k] <= s) continue;
            s = last[k];
            out[i].waits.push_back(last[k]);
            out[last[k]].signal = true;
        }
    }
    p.nodes = std::move(out);
    p.num_streams = nstreams;
    p.num_slots = num_slots;
    p.temp_slot.assign(slot.begin(), slot.begin() + nb);
    for (int si = 0, v = nb; si < m->num_stages; si++) {
        p.scratch[si].clear();
        for (int k = 0; k < m->stages[si].num_scratch; k++, v++) p.scratch[si].push_back(slot[v]);
    }
    return true;
}

}  // namespace kungpu

// executor.cu -- persistent tile-DAG executor of the Cholesky factor/solve.
//
// Host side (device side: executor_kernel.cuh): record the sub-tile task DAG of chameleon_pdpotrf (compute/
// pzpotrf.c:84-194) and of the two chameleon_pdtrsm solves of dpotrs
// (compute/zpotrs.c:302-304 -> compute/pztrsm.c:58-200), order it by a
// list-scheduling simulation with critical-path priorities (the reference's
// task priorities `2*mt - 2*k - n - m`, compute/pzpotrf.c:90-124, play the same
// role for StarPU), cache it per shape, and launch one persistent kernel.
// Device side: dispatch by atomic cursor, bounded waits on per-tile counters,
// tile operations from core.cuh, release by red.release.
#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <memory>
#include <queue>
#include <unordered_map>
#include <cstring>

#include "core.cuh"
#include "internal.h"
#include "rec.cuh"
#include "tc05.cuh"

namespace chb {

// ---------------------------------------------------------------------------
// Host: DAG recording and list-scheduling order
// ---------------------------------------------------------------------------
namespace {

// Cost profile of the task kinds, per execution path: list-scheduling order
// depends on the relative durations, which differ a lot between the FP64 DMMA
// path and the tcgen05 path (where updates are ~6x cheaper relative to the
// panel tasks).  Multipliers of the flop model, calibrated from per-task
// device traces at NB = 512 (POTRF, TRSM, UPD, FWD/BWD TRSM, FWD/BWD UPD).
enum CostProfile : int { PROF_FP64 = 0, PROF_F32_MMA = 1, PROF_F32_TC05 = 2 };
// upd_fix: the fixed cost of one update task (C read and write, dispatch) in
// units of one panel's product, so that a group of cnt panels costs
// upd * (cnt + upd_fix) / (1 + upd_fix).
struct Calib {
    double potrf, trsm, upd, strsm, supd, upd_fix;
};
static const Calib kCalib[3] = {
    {4.9, 4.7, 5.8, 3.9, 7.1, 0.05},   // FP64 DMMA
    {4.0, 4.7, 2.1, 2.4, 3.3, 0.2},    // FP32, split products on mma.sync
    {4.2, 2.7, 0.92, 1.9, 4.0, 0.6},   // FP32, tcgen05 updates, full-inverse substitutions (row-block sub-tasks)
};

// Single-panel update groups at the end of each tile column, per cost profile
// (CHAMELEON_B200_UPD_TAIL_F64 for the FP64 path).
int upd_tail(int prof) { return prof == PROF_FP64 ? ctx().utail_f64 : UPD_TAIL; }

struct Shape {
    int mode, N, NB, nrhs, NBB, P, prof, G;   // G: update group size (upd_group_of)
    int h2d_gbs;                              // MODE_CAST: host-to-device bandwidth of the model (GB/s)
    int tail = UPD_TAIL;                      // single-panel groups at the end of each column
    bool operator==(const Shape &o) const {
        return mode == o.mode && N == o.N && NB == o.NB && nrhs == o.nrhs && NBB == o.NBB && P == o.P &&
               prof == o.prof && G == o.G && h2d_gbs == o.h2d_gbs && tail == o.tail;
    }
};
struct ShapeHash {
    size_t operator()(const Shape &s) const {
        size_t h = 1469598103934665603ull;
        for (int v : {s.mode, s.N, s.NB, s.nrhs, s.NBB, s.P, s.prof, s.G, s.h2d_gbs, s.tail})
            h = (h ^ (size_t)v) * 1099511628211ull;
        return h;
    }
};

constexpr int TK_COPY = 100;   // model only: the host-to-device copy of one tile column (not emitted)

struct Coarse {
    int16_t kind, m, n, k, bn;   // TK_UPD: k = first panel of the group, bn = panel count
    int grp;                     // TK_UPD: index of the group in tile column n
    bool virt = false;           // model-only task: runs on the copy engine, not on a CTA
    int nsub;
    double dur;               // duration of one sub-task (model units)
    int head = -1, tail = -1; // successors: first and last entry of Graph::e
    int npred = 0;
    double blevel = 0;
};

// A coarse DAG.  The successor lists are chains in one array: a vector in every
// task made building the list of an order of 32768 half as long again.
struct Graph {
    std::vector<Coarse> t;
    std::vector<std::pair<int, int>> e;   // successor, next entry
    size_t size() const { return t.size(); }
    Coarse &operator[](int i) { return t[i]; }
    int add(int kind, int m, int n, int k, int bn, int nsub, double dur) {
        Coarse c;
        c.kind = kind; c.m = m; c.n = n; c.k = k; c.bn = bn; c.grp = 0; c.nsub = nsub; c.dur = dur;
        t.push_back(c);
        return (int)t.size() - 1;
    }
    void edge(int a, int b) {
        if (a < 0 || b < 0 || a == b) return;
        const int i = (int)e.size();
        e.push_back({b, -1});
        (t[a].tail < 0 ? t[a].head : e[t[a].tail].second) = i;
        t[a].tail = i;
        t[b].npred++;
    }
    template <class F>
    void succ(int i, F &&f) const {
        for (int j = t[i].head; j >= 0; j = e[j].second) f(e[j].first);
    }
};

struct Schedule {
    std::vector<Task> tasks;
    Task *d_tasks = nullptr;
    int npotrf = 0;              // POTRF tasks (for the dedicated CTA), their indices after the tasks
    const int *d_potrf = nullptr;
};

template <class NBU>
std::vector<Task> list_schedule(Graph &ct, int P, NBU nbu);

std::vector<Task> build_order(const Shape &s) {
    const int NT = (s.N + s.NB - 1) / s.NB;
    const int NTB = s.nrhs > 0 ? (s.nrhs + s.NBB - 1) / s.NBB : 0;
    auto tm = [&](int m) { return (m == NT - 1) ? s.N - m * s.NB : s.NB; };
    const int cb = count_blk(s.mode);
    const int pb = panel_blk(s.mode);
    auto nbp = [&](int m) { return (tm(m) + pb - 1) / pb; };                 // panel-solve row blocks
    auto nbu = [&](int m, int cnt) {                                         // update blocks, cnt panels
        const int e = upd_blk(s.mode, cnt);
        return (tm(m) + e - 1) / e;
    };
    auto wB = [&](int bn) { return (bn == NTB - 1) ? s.nrhs - bn * s.NBB : s.NBB; };
    const bool fact = s.mode & MODE_FACT, solve = s.mode & MODE_SOLVE;

    // the updates are all but all of a factorization's tasks
    size_t count = (size_t)2 * NT * NT + (size_t)NTB * NT * (NT + 1);
    for (int n = 0; fact && n < NT; ++n) count += (size_t)upd_ngroups(n, s.G, s.tail) * (NT - n);
    Graph ct;
    ct.t.reserve(count);
    ct.e.reserve(4 * count);
    auto add = [&](int kind, int m, int n, int k, int bn, int nsub, double dur) {
        return ct.add(kind, m, n, k, bn, nsub, dur);
    };
    auto edge = [&](int a, int b) { ct.edge(a, b); };
    // ids: potrf[k], trsm[m,k], upd[m,n,k] (last update of tile (m,n) so far)
    std::vector<int> P(NT, -1), XI(NT, -1), Tr((size_t)NT * NT, -1), lastU((size_t)NT * NT, -1);
    std::vector<int> Cst((size_t)NT * NT, -1);   // MODE_CAST: cast task of tile (m, n)
    const bool cast = fact && (s.mode & MODE_CAST);
    const bool xinv = s.mode & MODE_XINV;
    const double nb = s.NB;
    const Calib &cal = kCalib[(s.prof >= 0 && s.prof < 3) ? s.prof : 0];
    // tcgen05 path: task durations in microseconds from per-task device traces
    // at NB = 256 and 512 (N = 32768; the diagonal factorization measured
    // alone, 1.05 t: under the full load it runs ~20% longer, but the lower
    // figure ordered the list best -- 1.25 t and 0.8 t both lengthened the
    // launch by 5-8%).  The diagonal and panel tasks there are
    // latency-bound and grow linearly with the tile order, not with its flops,
    // so a flop model misorders the list (tasks whose inputs are not ready are
    // claimed first and their CTAs wait).
    const bool lat = (s.prof == PROF_F32_TC05), f64 = (s.prof == PROF_FP64);
    // FP64 path, likewise in microseconds: a latency term plus the products at
    // the rate of one of an SM's two CTAs
    const double sub = std::min<double>(nb, cb), us = 2.0 / 0.11e6;   // us per multiply-add
    auto ub = [&](int cnt) { return std::min<double>(nb, upd_blk(s.mode, cnt)); };
    auto c_potrf = [&](double t) {
        return f64 ? 0.24 * t + us * t * t * t / 3.0 : lat ? 1.05 * t : cal.potrf * 6.0 * t * t * t / 3.0;
    };
    auto c_xinv = [&](double t) { return lat ? 1.5 * t : cal.potrf * 6.0 * t * t * t / 3.0; };
    auto c_trsm = [&]() {
        return f64 ? 4.0 + us * sub * nb * (nb + IB) / 2 : lat ? (pb < SUBB ? 0.15 : 0.27) * nb : cal.trsm * 2.0 * SUBB * nb * nb;
    };
    auto c_upd = [&](int cnt) {
        return f64 ? 4.0 + us * ub(cnt) * ub(cnt) * nb * cnt
                   : lat ? 5.0 + 0.011 * nb * cnt
                         : cal.upd * SUBB * SUBB * nb * 2.0 * (cnt + cal.upd_fix) / (1.0 + cal.upd_fix);
    };
    auto c_strsm = [&](double t, double w, int parts) {
        return f64 ? (xinv ? 5.0 + us * SOLB * 0.75 * t * std::min(w, 64.0)
                           : 8.0 * t / IB + us * t * (t + IB) / 2 * std::min(w, 64.0))
                   : lat ? 13.0 + 0.01 * t : cal.strsm * 3.0 * t * t * w / parts;
    };
    auto c_supd = [&](double t, double w) {
        return f64 ? 4.0 + us * sub * t * std::min(w, 64.0)
                   : lat ? 8.0 + 0.04 * t : cal.supd * 2.0 * solve_rows(s.mode) * t * w;
    };
    if (cast) {
        // the copy engine delivers the stored triangle one tile column after
        // the other (model-only tasks, in order); each tile's cast waits for
        // its column
        const double gbs = std::max(1, s.h2d_gbs);
        int prev = -1;
        for (int q = 0; q < NT; ++q) {
            const double rows = (s.mode & MODE_CAST) ? (double)(s.N - q * s.NB) : 0.0;
            const double us = lat ? rows * tm(q) * 8.0 / (gbs * 1e3) : 0.0;
            const int cp = add(TK_COPY, q, q, q, 0, 1, us);
            ct[cp].virt = true;
            edge(prev, cp);
            prev = cp;
            // a column's copy covers tile column q of the lower triangle, or
            // tile row q's stored tiles of the upper one: the same tiles by symmetry
            for (int m = q; m < NT; ++m) {
                Cst[m + (size_t)NT * q] = add(TK_CAST, m, q, q, 0, 1, lat ? 8.0 * tm(m) * tm(q) / 65536.0 : 1.0);
                edge(cp, Cst[m + (size_t)NT * q]);
            }
        }
    }
    if (fact) {
        for (int k = 0; k < NT; ++k) {
            const double tk = tm(k);
            P[k] = add(TK_POTRF, k, k, k, 0, 1, c_potrf(tk));
            edge(lastU[k + (size_t)NT * k], P[k]);
            if (k == 0) edge(Cst[0], P[k]);
            if (xinv && solve) {
                XI[k] = add(TK_XINV, k, k, k, 0, 1, c_xinv(tk));
                edge(P[k], XI[k]);
            }
            for (int m = k + 1; m < NT; ++m) {
                const int id = add(TK_TRSM, m, k, k, 0, nbp(m), c_trsm());
                edge(P[k], id);
                edge(lastU[m + (size_t)NT * k], id);
                if (k == 0) edge(Cst[m], id);
                Tr[m + (size_t)NT * k] = id;
            }
            // the update groups of each later tile column whose last panel is k
            // (upd_group_of): they become ready with this step's panel solves
            for (int n = k + 1; n < NT; ++n) {
                int k0, cnt, gi;
                upd_group_of(n, k, s.G, s.tail, &k0, &cnt, &gi);
                if (k0 + cnt - 1 != k) continue;
                for (int m = n; m < NT; ++m) {
                    const int bm = nbu(m, cnt), nsub = (m == n) ? bm * (bm + 1) / 2 : bm * nbu(n, cnt);
                    const double dur = c_upd(cnt);
                    const int id = add(TK_UPD, m, n, k0, cnt, nsub, dur);
                    ct[id].grp = gi;
                    if (gi == 0) edge(Cst[m + (size_t)NT * n], id);
                    edge(Tr[m + (size_t)NT * k], id);
                    if (m != n) edge(Tr[n + (size_t)NT * k], id);
                    edge(lastU[m + (size_t)NT * n], id);
                    lastU[m + (size_t)NT * n] = id;
                }
            }
        }
    } else if (solve && !(s.mode & MODE_NOINV)) {
        for (int k = 0; k < NT; ++k) {
            if (xinv) XI[k] = add(TK_XINV, k, k, k, 0, 1, c_xinv(tm(k)));
            else P[k] = add(TK_INV, k, k, k, 0, 1, 1.0 * tm(k) * IB * IB);
        }
    }
    if (solve) {
        // substitution row blocks (SOLB rows with full tile inverses)
        const int srb = solve_rows(s.mode);
        auto nsb = [&](int m) { return (tm(m) + srb - 1) / srb; };
        std::vector<int> F((size_t)NT * NTB, -1), lastFU((size_t)NT * NTB, -1);
        std::vector<int> Bk((size_t)NT * NTB, -1), lastBU((size_t)NT * NTB, -1);
        for (int bn = 0; bn < NTB; ++bn) {
            const double w = wB(bn);
            for (int k = 0; k < NT; ++k) {
                // MODE_XINV: one sub-task per row block (each applies its rows of the inverse)
                const int f = add(TK_FWD_TRSM, k, k, k, bn, xinv ? nsb(k) : 1,
                                  c_strsm(tm(k), w, xinv ? nsb(k) : 1));
                edge(xinv ? XI[k] : P[k], f);
                edge(lastFU[k + (size_t)NT * bn], f);
                F[k + (size_t)NT * bn] = f;
                for (int m = k + 1; m < NT; ++m) {
                    const int u = add(TK_FWD_UPD, m, k, k, bn, nsb(m), c_supd(tm(k), w));
                    edge(f, u);
                    if (fact) edge(Tr[m + (size_t)NT * k], u);
                    edge(lastFU[m + (size_t)NT * bn], u);
                    lastFU[m + (size_t)NT * bn] = u;
                }
            }
            for (int k = NT - 1; k >= 0; --k) {
                const int b = add(TK_BWD_TRSM, k, k, k, bn, xinv ? nsb(k) : 1,
                                  c_strsm(tm(k), w, xinv ? nsb(k) : 1));
                edge(F[k + (size_t)NT * bn], b);
                edge(lastBU[k + (size_t)NT * bn], b);
                Bk[k + (size_t)NT * bn] = b;
                for (int m = k - 1; m >= 0; --m) {
                    const int u = add(TK_BWD_UPD, m, k, k, bn, nsb(m), c_supd(tm(k), w));
                    edge(b, u);
                    edge(lastBU[m + (size_t)NT * bn], u);
                    lastBU[m + (size_t)NT * bn] = u;
                }
            }
        }
    }
    return list_schedule(ct, s.P, nbu);
}

// List scheduling of a coarse DAG (generation order topological) on P
// workers with critical-path priorities; emits the sub-tasks in start order.
// nbu(m, cnt): row blocks of tile m in an update of cnt panels.
template <class NBU>
std::vector<Task> list_schedule(Graph &ct, int P, NBU nbu) {
    // bottom levels (generation order is topological)
    for (int i = (int)ct.size() - 1; i >= 0; --i) {
        double b = 0;
        ct.succ(i, [&](int j) { b = std::max(b, ct[j].blevel); });
        ct[i].blevel = b + ct[i].dur;
    }
    // list scheduling on s.P workers
    struct Ready {
        double prio; int id;
        bool operator<(const Ready &o) const { return prio < o.prio || (prio == o.prio && id > o.id); }
    };
    struct Fin {
        double t; int id;
        bool operator<(const Fin &o) const { return t > o.t; }
    };
    std::priority_queue<Ready> ready;
    std::priority_queue<Fin> running;
    std::vector<int> started(ct.size(), 0), finished(ct.size(), 0);
    double now = 0;
    // model-only tasks start as soon as they are ready, without a worker
    auto make_ready = [&](int i) {
        if (ct[i].virt) running.push({now + ct[i].dur, i});
        else ready.push({ct[i].blevel, i});
    };
    for (int i = 0; i < (int)ct.size(); ++i)
        if (ct[i].npred == 0) make_ready(i);
    std::vector<Task> out;
    size_t total = 0;
    for (auto &c : ct.t)
        if (!c.virt) total += c.nsub;
    out.reserve(total);
    int free_w = P;
    auto emit = [&](const Coarse &c, int j) {
        Task t{};
        t.kind = c.kind; t.m = c.m; t.n = c.n; t.k = c.k; t.bn = c.bn; t.sub = 0; t.grp = c.grp;
        if (c.kind == TK_UPD) {
            int bi = 0, bj = 0;
            if (c.m == c.n) {   // j-th lower sub-block (row-major over bi >= bj)
                int rem = j;
                bi = 0;
                while (rem > bi) { rem -= bi + 1; ++bi; }
                bj = rem;
            } else {
                bi = j / nbu(c.n, c.bn);
                bj = j % nbu(c.n, c.bn);
            }
            t.sub = (int16_t)(bi | (bj << 8));
        } else if (c.kind == TK_TRSM || c.kind == TK_FWD_UPD || c.kind == TK_BWD_UPD || c.kind == TK_FWD_TRSM ||
                   c.kind == TK_BWD_TRSM) {
            t.sub = (int16_t)j;   // row block (the substitutions have one unless MODE_XINV)
        }
        out.push_back(t);
    };
    while (out.size() < total) {
        while (free_w > 0 && !ready.empty()) {
            const int id = ready.top().id;
            Coarse &c = ct[id];
            emit(c, started[id]);
            started[id]++;
            if (started[id] == c.nsub) ready.pop();
            running.push({now + c.dur, id});
            --free_w;
        }
        if (running.empty()) break;   // cannot happen for a well-formed DAG
        const Fin f = running.top();
        running.pop();
        now = f.t;
        if (!ct[f.id].virt) ++free_w;
        if (++finished[f.id] == ct[f.id].nsub)
            ct.succ(f.id, [&](int j) {
                if (--ct[j].npred == 0) make_ready(j);
            });
    }
    return out;
}

std::mutex g_sched_mu;
std::unordered_map<Shape, std::unique_ptr<Schedule>, ShapeHash> g_sched;

// Device copy of a task list (and of its POTRF indices).
int upload_schedule(Schedule *sch) {
    if (!sch->tasks.empty()) {
        std::vector<int> pidx;
        for (size_t i = 0; i < sch->tasks.size(); ++i)
            if (sch->tasks[i].kind == TK_POTRF) pidx.push_back((int)i);
        const size_t tbytes = sch->tasks.size() * sizeof(Task);
        const size_t bytes = tbytes + pidx.size() * sizeof(int);
        if (!(sch->d_tasks = (Task *)dev_alloc(bytes))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
        sch->npotrf = (int)pidx.size();
        sch->d_potrf = reinterpret_cast<const int *>(reinterpret_cast<const uint8_t *>(sch->d_tasks) + tbytes);
        cudaStream_t ms = meta_stream();
        if (cudaMemcpyAsync(sch->d_tasks, sch->tasks.data(), tbytes, cudaMemcpyHostToDevice, ms) != cudaSuccess ||
            (!pidx.empty() && cudaMemcpyAsync((void *)sch->d_potrf, pidx.data(), pidx.size() * sizeof(int),
                                              cudaMemcpyHostToDevice, ms) != cudaSuccess) ||
            cudaStreamSynchronize(ms) != cudaSuccess)
            return CHAMELEON_ERR_UNEXPECTED;
    }
    return 0;
}

Schedule *get_schedule(const Shape &s) {
    std::lock_guard<std::mutex> lk(g_sched_mu);
    auto it = g_sched.find(s);
    if (it != g_sched.end()) return it->second.get();
    auto sch = std::make_unique<Schedule>();
    sch->tasks = build_order(s);
    if (upload_schedule(sch.get())) return nullptr;
    Schedule *raw = sch.get();
    g_sched[s] = std::move(sch);
    return raw;
}

ExecWs g_ws;   // workspace of the synchronous API entry points

// Bytes of every buffer of a workspace.
struct WsBytes {
    size_t ctr = 0, inv = 0, split = 0, xinv = 0, y = 0;
    void cover(const WsBytes &o) {
        ctr = std::max(ctr, o.ctr);
        inv = std::max(inv, o.inv);
        split = std::max(split, o.split);
        xinv = std::max(xinv, o.xinv);
        y = std::max(y, o.y);
    }
};

// Grow-only workspace buffers.  A buffer that grows is freed first, and the
// pool may hand its memory out again at once, so nothing enqueued may still use
// the workspace: a call reserves what all its launches need before the first.
int ensure_ws(ExecWs &w, const WsBytes &need) {
    if (!w.st) {
        if (!(w.st = (ExecState *)dev_alloc(2 * sizeof(ExecState)))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
        CHB_CUDA(cudaEventCreate(&w.e0));
        CHB_CUDA(cudaEventCreate(&w.e1));
    }
    auto grow = [](auto *&buf, size_t &have, size_t bytes) {
        if (bytes <= have) return true;
        dev_free(buf);
        have = 0;
        buf = static_cast<std::remove_reference_t<decltype(buf)>>(dev_alloc(bytes));
        if (buf) have = bytes;
        return buf != nullptr;
    };
    if (need.xinv > w.xinv_bytes) w.xinv_owner = nullptr;
    if (!grow(w.ctr, w.ctr_bytes, need.ctr) || !grow(w.inv, w.inv_bytes, need.inv) ||
        !grow(w.split, w.split_bytes, need.split) || !grow(w.xinv, w.xinv_bytes, need.xinv) ||
        !grow(w.y, w.y_bytes, need.y))
        return CHAMELEON_ERR_OUT_OF_RESOURCES;
    return 0;
}

}  // namespace

TraceRec *g_trace_buf = nullptr;   // set by the tracing entry point (host-owned device buffer)
int g_trace_cap = 0;

// Kernel variants, one translation unit each (exec_*.cu).
int launch_dag_f64(const ExecParams &p, int grid, cudaStream_t s);
int launch_dag_f32(const ExecParams &p, int grid, cudaStream_t s);
int launch_dag_f32tc(const ExecParams &p, int grid, cudaStream_t s);
int launch_dag_tf32(const ExecParams &p, int grid, cudaStream_t s);

void free_exec_ws(ExecWs &w) {
    dev_free(w.xinv);
    dev_free(w.y);
    dev_free(w.split);
    dev_free(w.ctr);
    dev_free(w.inv);
    dev_free(w.st);
    if (w.e0) cudaEventDestroy(w.e0);
    if (w.e1) cudaEventDestroy(w.e1);
    w = ExecWs();
}

// A task list recorded by a caller (CHAM_B200_Dag_*), already checked and on
// the device; its update groups are single panels.
static thread_local const Schedule *t_given = nullptr;

// A descriptor whose rows are one column-major array: any row tiling of it has
// the same addressing.
static bool one_tile(const CHAM_desc_t *d) { return priv(d)->cm_view || d->mt == 1; }

// The storage of a matrix as the tile rules see it: rows (columns) in one
// column-major array, tile sizes, tile columns.
struct Tiling {
    bool rows1, cols1;
    int mb, nb, nt;
};
static Tiling tiling(const CHAM_desc_t *d) {
    return Tiling{one_tile(d), priv(d)->cm_view || d->nt == 1, d->mb, d->nb, d->nt};
}

// Tile size of the FP64 executor.  The diagonal-tile factorizations are a
// serial chain on one CTA each, so tiles of the caller's size (512, say) leave
// the chip waiting for them: the executor uses tiles of EXEC_NB wherever the
// storage allows it -- any size when it is column-major, else the largest
// divisor of the storage tile up to EXEC_NB (multiples of 64 first; 48 at
// least, below that the tasks are all overhead).  dpotrf of order 8192:
// storage tile 512 24.9 ms, executor tile 256 12.8 ms, 128 9.8 ms, 64 14.9 ms.
// Storage tiles that 128 does not divide still gain, though 64-tiles (NB = 320) and
// odd ones (250 gives 125: 8-byte copies) are not the fastest: dposv of order 2000
// 4.44 -> 1.93 and 4.17 -> 1.82 ms against the storage tile.
constexpr int EXEC_NB = 128;
static int exec_tile(const Tiling &A, const Tiling *B) {
    const bool free_b = !B || B->rows1;
    if (A.rows1 && free_b) return EXEC_NB;
    const int nb = A.rows1 ? B->mb : A.nb;   // A and B have the same row tile size
    for (int d = EXEC_NB; d >= 64; d -= 64)
        if (nb % d == 0) return d;
    for (int d = std::min(EXEC_NB, nb); d >= 48; --d)
        if (nb % d == 0) return d;
    return nb;
}

// Panels per trailing update of the FP64 executor: a depth of n / 16 (n / 8 from
// order 20480 on), at least 512 and at most the configured group (given in tiles
// of 512).  A deeper group amortizes the C round trip, but a tile's last group only
// becomes ready a few steps before the tile is factored, and a 128 x 128 x 4096
// update takes 0.8 ms on a CTA: order 8192 with depth 4096 21.0 ms, 1024 10.0, 512
// 9.8, 256 10.4; order 24576 with 1536 178.3, 3072 176.1; 32768 with 2048 410.2,
// 4096 406.2.
constexpr int GROUP_NB = 512;
static int group_f64(int N, int NB, int kgroup) {
    const int depth = std::min(kgroup * GROUP_NB, std::max(512, N / (N < 20480 ? 16 : 8)));
    return std::max(1, depth / NB);
}

// FP64 substitutions.  The forward and backward sweeps are a chain of 2 N / NB
// dependent steps of a few microseconds each, so they run on tiles as large as
// the storage and the inverses allow (SOLVE_NB), each step one product per
// 64-row block with the tile's full inverse, and on column blocks of SOLVE_NBB
// whose chains run side by side.  The inverses come from products over all
// tiles at once (xinv_launch) before the chain starts, on the whole chip.
// A product with an explicit inverse has a backward error that grows with the
// condition of what was inverted, and nothing refines it here, so a tile whose
// norm times its inverse's is above XINV_COND is solved with its inverted 64 x
// 64 blocks instead (solve_strips).
// Order 8192, 64 right-hand sides: 6.7 ms on the factor's tiles of 512 with
// inverted 64-blocks, 5.0 ms on tiles of 128, 2.0 ms this way.
constexpr int SOLVE_NBB = 32;

// Tile size of the substitutions, 0 when the storage allows none from 64 on.
static int solve_tile(int N, const Tiling &A, const Tiling &B) {
    if (A.rows1 && B.rows1) return std::min(SOLVE_NB, (N + IB - 1) / IB * IB);
    const int nb = A.rows1 ? B.mb : A.nb;
    for (int d = std::min(SOLVE_NB, nb); d >= IB; --d)
        if (nb % d == 0) return d;
    return 0;
}

// Right-hand sides so many that 128-row tasks fill the chip are solved with
// them, on the storage's tiles (384 in a column-major array) with inverted 64 x
// 64 blocks: they read the factor half as often as 64-row ones and need no array
// for the forward results.  The line lies at 2e5 elements of B per row of a tile
// (ms with tile inverses / this way: column-major order 8192 with 6000 columns
// 35.1 / 48.8, 10000 58.4 / 57.9, 16384 95.1 / 85.1; 4096 with 12000 17.9 / 24.4,
// 30000 44.3 / 40.3; tiles of 512, 8192 with 10000 58.3 / 75.7, 16384 94.9 / 89.2;
// tiles of 250, 8192 with 3000 21.0 / 29.0, 6000 40.2 / 39.7).
constexpr size_t WIDE_ELEMS = 200000;
static int wide_tile(const Tiling &A, const Tiling &B) {
    return A.rows1 && B.rows1 ? 384 : A.rows1 ? B.mb : A.nb;
}

// The diagonal tiles (order <= NB, NT of them) of a factor, as lower views.
struct DiagTiles {
    double *A;
    const int64_t *off;
    const int *ld;
    int nt, r, NB, N, upper;
    __device__ int order(int k) const { return min(NB, N - k * NB); }
    __device__ View L(int k) const {
        const int K = k / r, i = k - K * r;
        const int64_t l = ld[K];
        double *q = A + off[K + nt * K] + (int64_t)i * NB * (1 + l);
        return upper ? View{q, l, 1} : View{q, 1, l};
    }
};

// X(k) (ld NB, NB^2 apart) gets the inverted 64 x 64 diagonal blocks of tile k.
__global__ void __launch_bounds__(NT_CTA, 2) xinv_diag_kernel(DiagTiles d, double *X) {
    extern __shared__ __align__(128) double smem[];
    const int k = blockIdx.y, j0 = blockIdx.x * IB, n = min(IB, d.order(k) - j0);
    if (n <= 0) return;
    double *sX = smem + IB * LEAF_LD;
    rec::leaf64_load(d.L(k).sub(j0, j0), n, smem);
    rec::leaf64_core<double, false>(smem, sX, n);
    double *q = X + (int64_t)k * d.NB * d.NB + (int64_t)j0 * (d.NB + 1);
#pragma unroll 4
    for (int idx = threadIdx.x; idx < n * IB; idx += NT_CTA) {
        const int r = idx & (IB - 1), c = idx / IB;
        if (r < n) q[r + (int64_t)c * d.NB] = sX[r + c * LEAF_LD];
    }
}
// One doubling half-step on every tile: the pairs of h-blocks of the tile get
// W21 = L21 X11 (first) or X21 = -X22 W21; 64 x 64 output blocks.
__global__ void __launch_bounds__(NT_CTA, 2) xinv_pair_kernel(DiagTiles d, int h, int pairs, double *X, double *W,
                                                              int first) {
    extern __shared__ __align__(128) double smem[];
    const int k = blockIdx.z / pairs, q = blockIdx.z % pairs, n = d.order(k);
    const int r = h * (2 * q + 1), c = r - h, h2 = min(h, n - r);
    const int i0 = blockIdx.x * IB, j0 = blockIdx.y * IB;
    if (i0 >= h2) return;
    const int rows = min(IB, h2 - i0);
    const int64_t base = (int64_t)k * d.NB * d.NB;
    const View Xv{X + base, 1, d.NB}, Wv{W + base, 1, d.NB};
    Acc<GemmCfg<double, 64, 64, 2, 4, SPLIT_BF16X3, 3>> acc;
    acc.zero();
    if (first) {
        cta_gemm(acc, d.L(k).sub(r + i0, c + j0), Xv.sub(c + j0, c + j0).t(), rows, IB, h - j0, smem);
        acc.store_to(Wv.sub(r + i0, c + j0), rows, IB);
    } else {
        cta_gemm(acc, Xv.sub(r + i0, r), Wv.sub(r, c + j0).t(), rows, IB, i0 + rows, smem);
        acc.for_each([&](int i, int j, double v) {
            if (i < rows) *Xv.at(r + i0 + i, c + j0 + j) = -v;
        });
    }
}

// cond[2 k], cond[2 k + 1] = the infinity norms of diagonal tile k and of its
// inverse (zeroed before): 16 rows of one tile per CTA, 16 threads each, since a
// row is a chain of loads (64 rows and 4 threads: 30 us at order 512).
constexpr int NORM_ROWS = 16;
__global__ void __launch_bounds__(NT_CTA, 4) xinv_norm_kernel(DiagTiles d, double *X, double *cond) {
    const int k = blockIdx.y, r0 = blockIdx.x * NORM_ROWS;
    rec::lower_norms<NORM_ROWS>(d.L(k), View{X + (int64_t)k * d.NB * d.NB, 1, d.NB}, r0,
                                min(NORM_ROWS, d.order(k) - r0), false, cond + 2 * k);
}

// The full inverses of all diagonal tiles into X (W: scratch of the same size),
// and their norms into cond (zeroed).
static int xinv_launch(const DiagTiles &d, int NT, double *X, double *W, double *cond, cudaStream_t s) {
    constexpr size_t inv_smem = sizeof(double) * 2 * IB * LEAF_LD;
    constexpr size_t pair_smem = GemmCfg<double, 64, 64, 2, 4, SPLIT_BF16X3, 3>::SMEM_BYTES;
    static bool attr = false;
    if (!attr) {
        CHB_CUDA(cudaFuncSetAttribute(xinv_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)inv_smem));
        CHB_CUDA(cudaFuncSetAttribute(xinv_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pair_smem));
        attr = true;
    }
    xinv_diag_kernel<<<dim3((d.NB + IB - 1) / IB, NT), NT_CTA, inv_smem, s>>>(d, X);
    CHB_LAUNCHED(1);
    for (int h = IB; h < d.NB; h *= 2) {
        const int pairs = (d.NB + h - 1) / (2 * h), nb = h / IB;
        for (int first = 1; first >= 0; --first)
            xinv_pair_kernel<<<dim3(nb, nb, NT * pairs), NT_CTA, pair_smem, s>>>(d, h, pairs, X, W, first);
        CHB_LAUNCHED(2);
    }
    xinv_norm_kernel<<<dim3((d.NB + NORM_ROWS - 1) / NORM_ROWS, NT), NT_CTA, 0, s>>>(d, X, cond);
    CHB_LAUNCHED(1);
    CHB_CUDA(cudaGetLastError());
    return 0;
}

constexpr int TC_DEEP_GROUP = 12;   // panels per update beyond the chain-bound orders, unless the caller set a number
constexpr size_t OWN_ELEMS = (size_t)1 << 25;

// One launch of the executor: its mode, tiles, task list and workspace.  Made
// on the host alone (plan_launch).
struct Plan {
    int mode, N, NB, NT, nrhs, NBB, NTB, b_c, xnb, grid;
    bool f32, tc, full_inv, xinv;
    Shape sh;
    int G, NIB;
    size_t nctr, xelems;
    WsBytes ws;
};

// mode: factorization, substitutions or both.  xnb > 0 (FP64 substitutions):
// tiles of xnb with their full inverses; xnb < 0: tiles of -xnb with 128-row
// tasks.  B, b_elems: storage of B and its
// elements (nrhs > 0).  reuse: the workspace holds the FP32 tile inverses of
// this factor.
static Plan plan_launch(int mode, int N, bool f32, const Tiling &A, const Tiling *B, int nrhs, size_t b_elems,
                        int split, int grid_req, const CastIn *cin, int xnb, bool reuse) {
    Context &c = ctx();
    Plan q{};
    if (!(mode & MODE_SOLVE)) nrhs = 0;
    q.N = N;
    q.f32 = f32;
    q.xnb = xnb;
    q.nrhs = nrhs;
    const int NB = q.NB = xnb ? std::abs(xnb)
                              : (t_given || f32) ? A.nb : exec_tile(A, (mode & MODE_SOLVE) ? B : nullptr);
    const int NT = q.NT = (N + NB - 1) / NB;
    q.NBB = B ? B->nb : NB;
    q.NTB = nrhs ? B->nt : 0;
    q.b_c = 1;
    if (xnb > 0) {
        // column blocks twice as wide read the factor half as often, from about
        // 1024 columns on, where the blocks alone fill the chip (us at order 3000
        // and 8192, 32 or 64 wide: 512 columns 934 or 1194, 4244 or 3764; 1024
        // columns 1342 or 1353, 8005 or 6447; 4096 columns 4508 or 3517, 31066
        // or 23950)
        const int want = nrhs <= 1024 ? SOLVE_NBB : 2 * SOLVE_NBB;
        if (B->cols1 || B->nb % want == 0) {
            q.b_c = B->cols1 ? (nrhs + want - 1) / want : B->nb / want;
            q.NBB = want;
            q.NTB = (nrhs + want - 1) / want;
        }
    }
    const int NBB = q.NBB, NTB = q.NTB;
    if (cin) mode |= MODE_CAST;
    // tcgen05 trailing updates: FP32 factorization with BF16x3 products and
    // 64-aligned tiles (the split chunks are 64 wide in k).
    const bool tc = q.tc = f32 && split == SPLIT_BF16X3 && (mode & MODE_FACT) && (NB % tc05::BK == 0) && NT > 1 &&
                           c.use_tcgen05;
    // grid_req counts SMs; FP64 places two executor CTAs on each
    const int cps = f32 ? 1 : 2;
    q.grid = cps * ((grid_req > 0) ? std::min(grid_req, c.num_sms) : c.num_sms);
    const bool full_inv = q.full_inv = f32 && c.rec_tile && NB <= (64 << rec::MAX_LVL);
    // (a task names its block by two 8-bit indices: a storage tile too large for
    // 64-blocks, and with no divisor to use instead, keeps 128-blocks)
    if (!f32 && !t_given && xnb >= 0 && NB <= 255 * FINEB) mode |= MODE_FINE;
    // The tcgen05 path is bound by the chain of diagonal tiles at smaller orders
    // and by its updates (L2 operand traffic) at larger ones: there the chain's
    // panel solves are split in two and the update groups kept short (tiles of
    // 256, order 16384: 16.9 -> 15.4 ms, 4096: 3.5 -> 3.05), while a chain that
    // runs further ahead only costs the updates locality beyond (32768: 61 -> 65
    // ms), where deeper groups save C round trips instead (8 panels 61.0 ms, 12
    // panels 59.3).  The line moves with the tile size (short / deep, ms): 128
    // 14000 12.6 / 13.1, 20480 24.9 / 23.8; 384 26880 36.5 / 36.7, 32768 58.1 /
    // 55.9; 512 30000 45.4 / 46.4, 32768 55.2 / 54.2.
    const bool chain_bound = N <= (NB < 384 ? 20480 : 30720);
    if (tc && !full_inv && chain_bound) mode |= MODE_HALF;
    const int prof = !f32 ? PROF_FP64 : (tc ? PROF_F32_TC05 : PROF_F32_MMA);
    // FP32 substitutions with full diagonal-tile inverses: computed off the
    // critical path in a factor+solve launch, reused by later solve-only
    // launches on the same factor and workspace (flags & EXEC_REUSE_INV).
    q.xinv = xnb > 0 || (f32 && !full_inv && c.xinv_solve && (mode & MODE_SOLVE) && nrhs > 0 &&
                         NB <= (64 << rec::MAX_LVL));
    if (xnb > 0) mode |= MODE_XINV | MODE_NOINV;
    else if (q.xinv) {
        mode |= MODE_XINV;
        if (!(mode & MODE_FACT) && reuse) mode |= MODE_NOINV;
    }
    q.mode = mode;
    // The task list depends on N only through NT and the number of SUBB-row
    // blocks of the last tile row, and on nrhs only through NTB (the kernel
    // takes the exact sizes from the parameters): key the cache on that
    // canonical shape so that callers with many distinct N share schedules.
    // (the finer of the update and substitution row blocks decides)
    const int gran = std::min(panel_blk(mode), solve_rows(mode));
    const int last_sub = ((N - (NT - 1) * NB) + gran - 1) / gran;
    const int canonN = (NT - 1) * NB + std::min(NB, last_sub * gran);
    // nrhs enters the cost model (not the task list): keep it, with the last
    // block's width rounded up to 16, so that the costs stay close and the
    // number of distinct schedules stays small
    const int canonR = nrhs ? (NTB - 1) * NBB + std::min(NBB, ((nrhs - (NTB - 1) * NBB + 15) / 16) * 16) : 0;
    // update group size: fused k steps amortize the C round trip and the
    // dispatch of an update over G panels (CHAMELEON_B200_UPD_GROUP per path)
    const int G = q.G = t_given ? 1
                                : prof == PROF_FP64 ? group_f64(N, NB, c.kgroup_f64)
                                                    : !tc ? c.kgroup_f32
                                                          : chain_bound || c.kgroup_tc_set ? c.kgroup_tc : TC_DEEP_GROUP;
    q.sh = Shape{mode, canonN, NB, canonR, NBB, q.grid, prof, G, cin ? std::max(1, cin->h2d_gbs) : 0, upd_tail(prof)};
    q.NIB = (NB + IB - 1) / IB;
    q.nctr = (size_t)(cin ? 3 : 2) * NT * NT + (size_t)4 * NT * std::max(NTB, 1) + NT;
    if (xnb > 0) q.nctr = (q.nctr + 1) / 2 * 2 + 4 * NT;   // the tiles' norms (2 doubles each) at the end
    const size_t esz = f32 ? sizeof(float) : sizeof(double);
    q.ws.ctr = q.nctr * sizeof(int);
    if (xnb <= 0) q.ws.inv = (full_inv ? (size_t)NT * NB * NB : (size_t)NT * q.NIB * IB * IB) * esz;
    if (q.xinv) {
        q.xelems = (size_t)NT * NB * NB;
        q.ws.xinv = q.xelems * (f32 ? sizeof(float) : 2 * sizeof(double));
        q.ws.y = b_elems * esz;   // forward-substitution results, same tile layout as B
    }
    if (tc) {
        const size_t tile_bytes = (size_t)((NB + SUBB - 1) / SUBB) * (NB / tc05::BK) * 2 * tc05::CHUNK_BYTES;
        q.ws.split = (size_t)NT * (NT - 1) / 2 * tile_bytes;
    }
    return q;
}

// The launches of one call (1 or 2); ws: what they need together.  small: the
// form with the least workspace (no array of B's size, no tile inverses in FP64).
static int plan_call(Plan (&q)[2], WsBytes &ws, int mode, int N, bool f32, const Tiling &A, const Tiling *B, int nrhs,
                     size_t b_elems, int split, int grid_req, const CastIn *cin, bool reuse, bool small) {
    // FP64 substitutions above one executor tile: a launch of their own, after
    // the factorization's (which it checks on the device).  With a
    // factorization of a small matrix they stay in its launch, where the
    // forward sweep runs beside it (1 to 17 right-hand sides, dposv 203: 232 us in
    // one launch, 256 in two; 2048: 1.70 and 1.73 ms; 5003: 6.16 and 5.95 ms),
    // unless B outweighs the factorization (2048 with 16384 columns 9.4 and 8.0
    // ms; the line could lie lower: 3000 with 512 takes 8.4 in one, 3200 3.2 in two)
    // and there are more than two tiles (100 with 4e5 columns 1.20 and 1.47 ms).
    const bool own = (mode & MODE_FACT) ? N > 3072 || (N > 2 * EXEC_NB && b_elems > OWN_ELEMS) : N > EXEC_NB;
    int xnb = (!f32 && !t_given && nrhs > 0 && own && !small) ? solve_tile(N, A, *B) : 0;
    if (xnb > 0) {
        const int wide = wide_tile(A, *B);
        if (b_elems / WIDE_ELEMS > (size_t)std::min(wide, 512)) xnb = -wide;
    }
    int n = 0;
    if (xnb != 0) {
        if (mode & MODE_FACT)
            q[n++] = plan_launch(MODE_FACT, N, f32, A, nullptr, 0, 0, split, grid_req, nullptr, 0, false);
        q[n++] = plan_launch(MODE_SOLVE, N, f32, A, B, nrhs, b_elems, split, grid_req, nullptr, xnb, false);
    } else {
        q[n++] = plan_launch(mode, N, f32, A, B, nrhs, b_elems, split, grid_req, cin, 0, reuse);
    }
    ws = WsBytes{};
    for (int i = 0; i < n; ++i) ws.cover(q[i].ws);
    return n;
}

// step(0), step(1), .. up to the first that fails, then drain() whatever
// happened: a call never returns with its own launches still running on the
// caller's arrays, the workspace and the descriptors' tables.
template <class Step, class Drain>
static int enqueue_all(int n, Step step, Drain drain) {
    int rc = 0;
    for (int i = 0; i < n && !rc; ++i) rc = step(i);
    const int rd = drain();
    return rc ? rc : rd;
}

// Enqueue one launch of the executor; the workspace holds what the plan needs
// and the descriptors are uploaded.  st: its state, initialized by the caller;
// after: state of an earlier launch that must not have failed; trace_at: where its
// trace records start, after those of an earlier launch.
static int enqueue_dag(const Plan &q, const Schedule *sch, cham_uplo_t uplo, CHAM_desc_t *A, CHAM_desc_t *B,
                       cudaStream_t s, int split, ExecWs &w, const CastIn *cin, ExecState *st,
                       const ExecState *after, int trace_at) {
    Context &c = ctx();
    const int N = q.N, NB = q.NB, NT = q.NT, nrhs = q.nrhs, NTB = q.NTB;
    int rc = 0;
    ExecParams p{};
    p.tasks = sch->d_tasks;
    p.ntasks = (int)sch->tasks.size();
    // one CTA runs the diagonal-tile factorizations (its instruction cache stays
    // warm for their long unrolled leaves); the others skip them
    const bool dedicate = c.potrf_cta && q.grid > 1 && sch->npotrf > 1;
    p.npotrf = dedicate ? sch->npotrf : 0;
    p.potrf_idx = sch->d_potrf;
    p.mode = q.mode;
    p.upper = (uplo == ChamUpper);
    p.NT = NT; p.N = N; p.NB = NB;
    p.A = A->mat;
    p.a_off = priv(A)->dev.off;
    p.a_ld = priv(A)->dev.ld;
    p.a_nt = A->mt;
    p.a_r = one_tile(A) ? NT : std::max(1, A->nb / NB);
    p.NTB = NTB; p.nrhs = nrhs; p.NBB = q.NBB;
    p.B = nrhs ? B->mat : nullptr;
    p.b_off = nrhs ? priv(B)->dev.off : nullptr;
    p.b_ld = nrhs ? priv(B)->dev.ld : nullptr;
    p.b_nt = nrhs ? B->mt : 1;
    p.b_r = nrhs ? (one_tile(B) ? NT : std::max(1, B->mb / NB)) : 1;
    p.b_c = q.b_c;
    int *ctr = (int *)w.ctr;
    CHB_CUDA(cudaMemsetAsync(ctr, 0, q.nctr * sizeof(int), s));
    p.updA = ctr;
    p.panA = ctr + (size_t)NT * NT;
    const size_t nb4 = (size_t)NT * std::max(NTB, 1);
    p.fwdB = ctr + (size_t)2 * NT * NT;
    p.fwdDone = p.fwdB + nb4;
    p.bwdB = p.fwdDone + nb4;
    p.bwdDone = p.bwdB + nb4;
    p.invd = w.inv;
    p.NIB = q.NIB;
    p.full_inv = q.full_inv ? 1 : 0;
    p.xinvDone = p.bwdDone + nb4;
    if (cin) {
        p.castDone = p.xinvDone + NT;
        p.csrc = cin->src;
        p.csrc_ld = cin->ld;
        p.carrive = cin->arrive;
        p.cepoch = cin->epoch;
        p.colsum = cin->colsum;
        p.covf = cin->ovf;
    }
    p.xinv = nullptr;
    if (q.xinv) {
        p.xinv = w.xinv;
        if (q.xnb > 0 || !(q.mode & MODE_NOINV)) w.xinv_owner = nullptr;   // rewritten by this call
        if (q.xnb > 0) {
            const DiagTiles d{(double *)A->mat, priv(A)->dev.off, priv(A)->dev.ld, p.a_nt, p.a_r, NB, N, p.upper};
            double *cond = reinterpret_cast<double *>(ctr + q.nctr - 4 * NT);
            p.cond = cond;
            if ((rc = xinv_launch(d, NT, (double *)w.xinv, (double *)w.xinv + q.xelems, cond, s))) return rc;
        }
        p.Y = w.y;
    }
    p.st = st;
    p.after = after;
    p.trace = (g_trace_buf && g_trace_cap - trace_at >= p.ntasks) ? g_trace_buf + trace_at : nullptr;
    p.wait_budget_ns = (unsigned long long)c.wait_budget_us * 1000ull;
    p.kgroup = q.G;
    p.utail = q.sh.tail;
    if (q.tc) {
        p.split_nrb = (NB + SUBB - 1) / SUBB;
        p.split_nkc = NB / tc05::BK;
        p.split = w.split;
    }
    if (p.ntasks > 0) {
        CHB_LAUNCHED(1);
        if (!q.f32) rc = launch_dag_f64(p, q.grid, s);
        else if (split == SPLIT_TF32X3) rc = launch_dag_tf32(p, q.grid, s);
        else if (q.tc) rc = launch_dag_f32tc(p, q.grid, s);
        else rc = launch_dag_f32(p, q.grid, s);
        if (rc) return rc;
    }
    return 0;
}

int run_cholesky_dag(int mode, cham_uplo_t uplo, CHAM_desc_t *A, CHAM_desc_t *B, cudaStream_t s,
                     ExecResult *res, int split, ExecWs *wsp, int grid_req, int flags, const CastIn *cin) {
    ExecWs &w = wsp ? *wsp : g_ws;
    const int N = A->n;
    const bool f32 = (A->dtyp == ChamRealFloat);
    const int nrhs = (B && (mode & MODE_SOLVE)) ? B->n : 0;
    res->info = 0; res->error = 0; res->ms = 0.f;
    if (N == 0) return 0;
    if (nrhs && B->dtyp != A->dtyp) return CHAMELEON_ERR_ILLEGAL_VALUE;
    if (cin && (!f32 || !(mode & MODE_FACT))) return CHAMELEON_ERR_ILLEGAL_VALUE;
    const bool reuse = (flags & EXEC_REUSE_INV) && w.xinv_owner == A->mat && w.xinv_nt == A->nt &&
                       w.xinv_nb == A->nb && w.xinv_n == N;
    const Tiling tA = tiling(A), tB = B ? tiling(B) : Tiling{};
    const size_t b_elems = nrhs ? (size_t)(priv(B)->cm_view ? B->lda : B->lm) * B->ln : 0;
    // task lists, memory and tables of every launch before the first one
    // starts: none of them may be replaced while a launch still uses it
    Plan q[2];
    const Schedule *sch[2] = {};
    int nq = 0;
    auto prepare = [&](bool small) -> int {
        WsBytes need;
        nq = plan_call(q, need, mode, N, f32, tA, B ? &tB : nullptr, nrhs, b_elems, split, grid_req, cin, reuse, small);
        for (int i = 0; i < nq; ++i)
            if (!(sch[i] = t_given ? t_given : get_schedule(q[i].sh))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
        return ensure_ws(w, need);
    };
    int rc = prepare(false);
    if (rc == CHAMELEON_ERR_OUT_OF_RESOURCES && q[nq - 1].xnb > 0) {
        // without the workspace of the FP64 tile inverses, and with its memory
        dev_free(w.xinv);
        dev_free(w.y);
        w.xinv = w.y = nullptr;
        w.xinv_bytes = w.y_bytes = 0;
        w.xinv_owner = nullptr;
        rc = prepare(true);
    }
    if (!rc) rc = desc_upload(A);
    if (!rc && nrhs) rc = desc_upload(B);
    if (rc) return rc;
    ExecState init[2] = {};
    init[0].info = init[1].info = INT_MAX;
    init[0].stuck_task = init[1].stuck_task = -1;
    ExecState out[2] = {};
    rc = enqueue_all(
        nq + 2,
        [&](int i) -> int {
            if (i == 0) {
                CHB_CUDA(cudaMemcpyAsync(w.st, init, sizeof(init), cudaMemcpyHostToDevice, s));
                CHB_CUDA(cudaEventRecord(w.e0, s));
                return 0;
            }
            if (i <= nq)
                return enqueue_dag(q[i - 1], sch[i - 1], uplo, A, B, s, split, w, cin, w.st + i - 1,
                                   i > 1 ? w.st : nullptr, i > 1 ? (int)sch[0]->tasks.size() : 0);
            CHB_CUDA(cudaEventRecord(w.e1, s));
            CHB_CUDA(cudaMemcpyAsync(out, w.st, sizeof(out), cudaMemcpyDeviceToHost, s));
            return 0;
        },
        [&]() -> int {
            CHB_CUDA(cudaStreamSynchronize(s));
            return 0;
        });
    if (rc) return rc;
    CHB_CUDA(cudaEventElapsedTime(&res->ms, w.e0, w.e1));
    res->info = (out[0].info == INT_MAX) ? 0 : out[0].info;
    res->error = out[0].error ? out[0].error : out[1].error;
    if (f32 && q[0].xinv && !(q[0].mode & MODE_NOINV) && res->info == 0 && res->error == 0) {
        w.xinv_owner = A->mat;   // the inverses now match this factor
        w.xinv_n = N;
        w.xinv_nt = A->nt;
        w.xinv_nb = A->nb;
    }
    for (int i = 0; i < nq; ++i)
        if (out[i].error) {
            char msg[160];
            snprintf(msg, sizeof msg, "device wait budget exhausted at task %d (%d of %d done)", out[i].stuck_task,
                     out[i].done, (int)sch[i]->tasks.size());
            warning("run_cholesky_dag", msg);
        }
    return 0;
}

// Counters, state and the one-entry tile table of dag_potrf_async.
struct OneTile {
    int64_t off;
    int ld, pad;
};
__global__ void dag_init_kernel(OneTile *tab, int lda, int *ctr, int nctr, ExecState *st) {
    for (int i = threadIdx.x; i < nctr; i += blockDim.x) ctr[i] = 0;
    if (threadIdx.x == 0) {
        *tab = OneTile{0, lda, 0};
        *st = ExecState{};
        st->info = INT_MAX;
        st->stuck_task = -1;
    }
}
__global__ void dag_info_kernel(const ExecState *st, int *info) {
    *info = st->error ? st->error : (st->info == INT_MAX ? 0 : st->info);
}

int dag_potrf_async(cham_uplo_t uplo, int n, double *A, int lda, int *d_info, cudaStream_t s, ExecWs &w, bool *ran) {
    *ran = false;
    const int NB = EXEC_NB, NT = (n + NB - 1) / NB, mode = MODE_FACT | MODE_FINE;
    int dev = 0, sms = 0;
    CHB_CUDA(cudaGetDevice(&dev));
    if (!dag_potrf_usable(n, dev, pool_device())) return 0;
    CHB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // as many CTAs as the first step has panel-solve and update blocks
    const int grid = std::min(2 * sms, 2 * NT * NT);
    const int canon = (NT - 1) * NB + (n - (NT - 1) * NB + FINEB - 1) / FINEB * FINEB;
    const int G = group_f64(n, NB, ctx().kgroup_f64);
    const Shape sh{mode, canon, NB, 0, NB, grid, PROF_FP64, G, 0, upd_tail(PROF_FP64)};
    const size_t nctr = (size_t)2 * NT * NT + (size_t)5 * NT;
    const size_t ctr_bytes = sizeof(OneTile) + nctr * sizeof(int);
    const size_t inv_bytes = (size_t)NT * (NB / IB) * IB * IB * sizeof(double);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CHB_CUDA(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) {
        std::lock_guard<std::mutex> lk(g_sched_mu);
        if (g_sched.find(sh) == g_sched.end() || !w.st || ctr_bytes > w.ctr_bytes || inv_bytes > w.inv_bytes) return 0;
    } else if (w.st && (ctr_bytes > w.ctr_bytes || inv_bytes > w.inv_bytes)) {
        CHB_CUDA(cudaStreamSynchronize(s));   // queued calls still use the buffers that are replaced
    }
    const Schedule *sch = get_schedule(sh);
    if (!sch) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    WsBytes need;
    need.ctr = ctr_bytes;
    need.inv = inv_bytes;
    if (int rc = ensure_ws(w, need)) return rc;
    OneTile *tab = (OneTile *)w.ctr;
    int *ctr = (int *)(tab + 1);
    dag_init_kernel<<<1, 256, 0, s>>>(tab, lda, ctr, (int)nctr, w.st);
    ExecParams p{};
    p.tasks = sch->d_tasks;
    p.ntasks = (int)sch->tasks.size();
    p.mode = mode;
    p.upper = (uplo == ChamUpper);
    p.NT = NT; p.N = n; p.NB = NB;
    p.A = A;
    p.a_off = &tab->off;
    p.a_ld = &tab->ld;
    p.a_nt = 1;
    p.a_r = NT;
    p.NBB = NB;
    p.b_r = p.b_nt = 1;
    p.updA = ctr;
    p.panA = ctr + (size_t)NT * NT;
    p.invd = w.inv;
    p.NIB = NB / IB;
    p.st = w.st;
    p.wait_budget_ns = (unsigned long long)ctx().wait_budget_us * 1000ull;
    p.kgroup = G;
    p.utail = sh.tail;
    if (int rc = launch_dag_f64(p, grid, s)) return rc;
    if (d_info) dag_info_kernel<<<1, 1, 0, s>>>(w.st, d_info);
    CHB_LAUNCHED(d_info ? 3 : 2);
    CHB_CUDA(cudaGetLastError());
    *ran = true;
    return 0;
}

}  // namespace chb

// Trace hooks (tracing subsystem): size the per-task trace buffer, read it back.
extern "C" int CHAM_B200_Trace_Enable(int capacity) {
    using namespace chb;
    if (g_trace_buf) { cudaFree(g_trace_buf); g_trace_buf = nullptr; g_trace_cap = 0; }
    if (capacity <= 0) return 0;
    if (cudaMalloc(&g_trace_buf, (size_t)capacity * sizeof(TraceRec)) != cudaSuccess) {
        g_trace_buf = nullptr;
        return CHAMELEON_ERR_OUT_OF_RESOURCES;
    }
    cudaMemset(g_trace_buf, 0, (size_t)capacity * sizeof(TraceRec));
    g_trace_cap = capacity;
    return 0;
}
extern "C" int CHAM_B200_Trace_Read(void *host_out, int count) {
    using namespace chb;
    if (!g_trace_buf || count > g_trace_cap) return CHAMELEON_ERR_ILLEGAL_VALUE;
    return cudaMemcpy(host_out, g_trace_buf, (size_t)count * sizeof(TraceRec), cudaMemcpyDeviceToHost) ==
                   cudaSuccess
               ? 0
               : CHAMELEON_ERR_UNEXPECTED;
}
// Copy the schedule of a shape into `out` (host only; used by the CPU tests of
// the DAG logic and by the trace tooling).  Returns the task count written.
extern "C" int CHAM_B200_Schedule_Build(int mode, int N, int NB, int nrhs, int NBB, int workers, int prof, int kgroup,
                                        void *out, int cap) {
    using namespace chb;
    const std::vector<Task> t =
        build_order(Shape{mode, N, NB, nrhs, NBB, workers, prof, std::max(1, kgroup), (mode & MODE_CAST) ? 50 : 0,
                          upd_tail(prof)});
    const int n = std::min<int>((int)t.size(), cap);
    memcpy(out, t.data(), sizeof(Task) * (size_t)n);
    return n;
}
// Number of tasks of the schedule of a given shape (for tests and tracing).
extern "C" int CHAM_B200_Schedule_Size(int mode, int N, int NB, int nrhs, int NBB, int workers, int prof, int kgroup) {
    using namespace chb;
    return (int)build_order(Shape{mode, N, NB, nrhs, NBB, workers, prof, std::max(1, kgroup),
                                  (mode & MODE_CAST) ? 50 : 0, upd_tail(prof)})
        .size();
}

// The launches of one call (mode MODE_FACT | MODE_SOLVE; A of order N in nb x nb
// tiles, B in nb x nbb, or both column-major arrays; fp32: the BF16x3 path) and
// their workspace, host only: per launch {tile size, column block, bytes of
// counters, inverted blocks, tile inverses, forward results, mode, update
// group}, and in reserved[4] the bytes
// that the call reserves.  Returns the number of launches (at most 2).
extern "C" int CHAM_B200_Exec_Plan(int mode, int N, int nb, int array, int nrhs, int nbb, int fp32, int64_t *launch,
                                   int64_t *reserved) {
    using namespace chb;
    auto tl = [&](int n, int t) { return Tiling{array || N <= nb, array || n <= t, nb, t, (n + t - 1) / t}; };
    const Tiling A = tl(N, nb), B = tl(std::max(nrhs, 1), nbb);
    Plan q[2];
    WsBytes r;
    const int n = plan_call(q, r, mode, N, fp32 != 0, A, nrhs > 0 ? &B : nullptr, nrhs, (size_t)N * std::max(nrhs, 0),
                            SPLIT_BF16X3, 0, nullptr, false, false);
    for (int i = 0; i < n; ++i) {
        const int64_t v[8] = {q[i].NB, q[i].NBB, (int64_t)q[i].ws.ctr, (int64_t)q[i].ws.inv, (int64_t)q[i].ws.xinv,
                              (int64_t)q[i].ws.y, q[i].mode, q[i].G};
        std::copy(v, v + 8, launch + 8 * i);
    }
    const int64_t v[4] = {(int64_t)r.ctr, (int64_t)r.inv, (int64_t)r.xinv, (int64_t)r.y};
    std::copy(v, v + 4, reserved);
    return n;
}

// Whether CUDA_dpotrf of order n takes the tile DAG on a stream of `device`
// when the library's memory is on pool_device.
extern "C" int CHAM_B200_Test_Potrf_On_Dag(int n, int device, int pool_device) {
    return chb::dag_potrf_usable(n, device, pool_device);
}
// enqueue_all with n steps of which step `bad` fails with rc (none: bad < 0):
// writes the steps in the order of their calls, -1 for the drain, and returns
// its result; *len receives the count (at most n + 1).
extern "C" int CHAM_B200_Test_Enqueue_All(int n, int bad, int rc, int *calls, int *len) {
    *len = 0;
    return chb::enqueue_all(
        n,
        [&](int i) {
            calls[(*len)++] = i;
            return i == bad ? rc : 0;
        },
        [&] {
            calls[(*len)++] = -1;
            return 0;
        });
}

// ---------------------------------------------------------------------------
// Recorded DAGs: tile tasks submitted by a caller (a Chameleon runtime plugin
// whose INSERT_TASK_* calls append here; chameleon_pzpotrf / chameleon_pztrsm
// run unchanged above it) and run by the persistent executor.
// ---------------------------------------------------------------------------
struct cham_b200_dag_s {
    std::vector<std::array<int, 5>> rec;   // kind, m, n, k, bn in submission order
};

namespace chb {
namespace {

// The executor's counter predicates (executor_kernel.cuh task_deps, update
// groups of one panel), replayed on a task list: true when every task's
// inputs are complete once every task before it has run, i.e. the list is
// deadlock-free for any number of CTAs.
bool replay_ok(const std::vector<Task> &tl, int mode, int N, int NB, int NTB) {
    const int NT = (N + NB - 1) / NB;
    auto tm = [&](int m) { return (m == NT - 1) ? N - m * NB : NB; };
    auto nbi = [&](int m) { return (tm(m) + SUBB - 1) / SUBB; };
    auto S = [&](int m, int n) { return m == n ? nbi(m) * (nbi(m) + 1) / 2 : nbi(m) * nbi(n); };
    const bool fact = mode & MODE_FACT;
    const size_t nb4 = (size_t)NT * std::max(NTB, 1);
    std::vector<int> upd((size_t)NT * NT, 0), pan((size_t)NT * NT, 0), fB(nb4, 0), fD(nb4, 0), bB(nb4, 0), bD(nb4, 0);
    for (const Task &t : tl) {
        bool ok = true;
        const size_t kb = t.k + (size_t)NT * t.bn, mb = t.m + (size_t)NT * t.bn;
        switch (t.kind) {
        case TK_POTRF: ok = upd[t.k + (size_t)NT * t.k] >= t.k * S(t.k, t.k); pan[t.k + (size_t)NT * t.k]++; break;
        case TK_INV: pan[t.k + (size_t)NT * t.k]++; break;
        case TK_TRSM:
            ok = pan[t.k + (size_t)NT * t.k] >= 1 && upd[t.m + (size_t)NT * t.k] >= t.k * S(t.m, t.k);
            pan[t.m + (size_t)NT * t.k]++;
            break;
        case TK_UPD:
            ok = t.bn == 1 && pan[t.m + (size_t)NT * t.k] >= nbi(t.m) && pan[t.n + (size_t)NT * t.k] >= nbi(t.n) &&
                 upd[t.m + (size_t)NT * t.n] >= t.k * S(t.m, t.n);
            upd[t.m + (size_t)NT * t.n]++;
            break;
        case TK_FWD_TRSM: ok = pan[t.k + (size_t)NT * t.k] >= 1 && fB[kb] >= t.k; fD[kb]++; break;
        case TK_FWD_UPD: ok = fD[kb] >= 1 && (!fact || pan[t.m + (size_t)NT * t.k] >= nbi(t.m)) && fB[mb] >= t.k; fB[mb]++; break;
        case TK_BWD_TRSM: ok = fD[kb] >= 1 && bB[kb] >= NT - 1 - t.k; bD[kb]++; break;
        case TK_BWD_UPD: ok = bD[kb] >= 1 && bB[mb] >= NT - 1 - t.k; bB[mb]++; break;
        default: ok = false;
        }
        if (!ok) return false;
    }
    return true;
}

}  // namespace
}  // namespace chb

extern "C" {

int CHAM_B200_Dag_Create(CHAM_b200_dag_t *dag) {
    if (!dag) return CHAMELEON_ERR_ILLEGAL_VALUE;
    *dag = new cham_b200_dag_s();
    return 0;
}
int CHAM_B200_Dag_Destroy(CHAM_b200_dag_t dag) {
    delete dag;
    return 0;
}
int CHAM_B200_Dag_Clear(CHAM_b200_dag_t dag) {
    if (!dag) return CHAMELEON_ERR_ILLEGAL_VALUE;
    dag->rec.clear();
    return 0;
}
int CHAM_B200_Dag_Record(CHAM_b200_dag_t dag, int kind, int m, int n, int k, int bn) {
    using namespace chb;
    if (!dag || kind < CHAM_B200_DAG_POTRF || kind > CHAM_B200_DAG_BWD_UPDATE || m < 0 || n < 0 || k < 0 || bn < 0)
        return CHAMELEON_ERR_ILLEGAL_VALUE;
    dag->rec.push_back({kind, m, n, k, bn});
    return 0;
}
int CHAM_B200_Dag_Size(CHAM_b200_dag_t dag) { return dag ? (int)dag->rec.size() : CHAMELEON_ERR_ILLEGAL_VALUE; }
int CHAM_B200_Dag_Get(CHAM_b200_dag_t dag, int *out, int cap) {
    if (!dag || !out) return CHAMELEON_ERR_ILLEGAL_VALUE;
    const int n = std::min<int>(cap, (int)dag->rec.size());
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < 5; ++j) out[5 * i + j] = dag->rec[i][j];
    return n;
}

// The recorded tasks as the executor's coarse DAG: every record's tiles (A's
// lower triangle, B's tile column bn) with read-after-write, write-after-read
// and write-after-write edges in submission order, then the same list
// scheduling as the built-in DAGs, and a replay of the device's wait
// predicates on the result.  Returns the sub-task list (empty + error code on
// a record the executor cannot run in that order).
static int dag_to_tasks(const cham_b200_dag_s &dag, int N, int NB, int nrhs, int NBB, int workers,
                        std::vector<chb::Task> *out, int *mode_out) {
    using namespace chb;
    const int NT = (N + NB - 1) / NB;
    const int NTB = nrhs > 0 ? (nrhs + NBB - 1) / NBB : 0;
    auto tm = [&](int m) { return (m == NT - 1) ? N - m * NB : NB; };
    auto nbi = [&](int m) { return (tm(m) + SUBB - 1) / SUBB; };
    int mode = 0;
    for (auto &r : dag.rec) mode |= (r[0] <= TK_UPD) ? MODE_FACT : MODE_SOLVE;
    Graph ct;
    // tile ids: A (m, n) -> m + NT n; B (m, bn) -> NT NT + m + NT bn
    const size_t ntile = (size_t)NT * NT + (size_t)NT * std::max(NTB, 1);
    std::vector<int> last_w(ntile, -1);
    std::vector<std::vector<int>> readers(ntile);
    auto add = [&](int kind, int m, int n, int k, int bn, int nsub, double dur) {
        return ct.add(kind, m, n, k, bn, nsub, dur);
    };
    auto edge = [&](int a, int b) { ct.edge(a, b); };
    auto rd = [&](size_t tile, int id) {
        edge(last_w[tile], id);
        readers[tile].push_back(id);
    };
    auto wr = [&](size_t tile, int id) {
        edge(last_w[tile], id);
        for (int r : readers[tile]) edge(r, id);
        readers[tile].clear();
        last_w[tile] = id;
    };
    auto At = [&](int m, int n) { return (size_t)m + (size_t)NT * n; };
    auto Bt = [&](int m, int bn) { return (size_t)NT * NT + m + (size_t)NT * bn; };
    const double nb = NB;
    // FP64 path costs (flop model), as in build_order
    const Calib &cal = kCalib[PROF_FP64];
    std::vector<int> inv_id(NT, -1);
    if (!(mode & MODE_FACT)) {   // solve only: the executor inverts the diagonal blocks first
        for (int k = 0; k < NT; ++k) {
            inv_id[k] = add(TK_INV, k, k, k, 0, 1, 1.0 * tm(k) * IB * IB);
            rd(At(k, k), inv_id[k]);
        }
    }
    for (auto &r : dag.rec) {
        const int kind = r[0], m = r[1], n = r[2], k = r[3], bn = r[4];
        const bool inA = m < NT && n < NT && k < NT;
        const bool inB = bn < std::max(NTB, 1);
        if (!inA || !inB) return CHAMELEON_ERR_ILLEGAL_VALUE;
        int id = -1;
        const double w = NTB ? ((bn == NTB - 1) ? nrhs - bn * NBB : NBB) : 0;
        switch (kind) {
        case TK_POTRF:
            if (m != k || n != k) return CHAMELEON_ERR_ILLEGAL_VALUE;
            id = add(TK_POTRF, k, k, k, 0, 1, cal.potrf * 2.0 * tm(k) * tm(k) * tm(k));
            wr(At(k, k), id);
            break;
        case TK_TRSM:
            if (n != k || m <= k) return CHAMELEON_ERR_ILLEGAL_VALUE;
            id = add(TK_TRSM, m, k, k, 0, nbi(m), cal.trsm * 2.0 * SUBB * nb * nb);
            rd(At(k, k), id);
            wr(At(m, k), id);
            break;
        case TK_UPD:
            if (m < n || n <= k) return CHAMELEON_ERR_ILLEGAL_VALUE;
            id = add(TK_UPD, m, n, k, 1, m == n ? nbi(m) * (nbi(m) + 1) / 2 : nbi(m) * nbi(n),
                     cal.upd * SUBB * SUBB * nb * 2.0);
            ct[id].grp = k;
            rd(At(m, k), id);
            if (m != n) rd(At(n, k), id);
            wr(At(m, n), id);
            break;
        case TK_FWD_TRSM:
        case TK_BWD_TRSM:
            if (m != k || n != k || !NTB) return CHAMELEON_ERR_ILLEGAL_VALUE;
            id = add(kind, k, k, k, bn, 1, cal.strsm * 3.0 * tm(k) * tm(k) * w);
            rd(At(k, k), id);
            if (inv_id[k] >= 0) edge(inv_id[k], id);
            wr(Bt(k, bn), id);
            break;
        case TK_FWD_UPD:
        case TK_BWD_UPD:
            // forward: B(m) -= L(m,k) B(k), m > k; backward: B(m) -= L(k,m)^T B(k), m < k
            if (!NTB || (kind == TK_FWD_UPD ? m <= k : m >= k)) return CHAMELEON_ERR_ILLEGAL_VALUE;
            id = add(kind, m, k, k, bn, nbi(m), cal.supd * 2.0 * SUBB * tm(k) * w);
            rd(kind == TK_FWD_UPD ? At(m, k) : At(k, m), id);
            rd(Bt(k, bn), id);
            wr(Bt(m, bn), id);
            break;
        default:
            return CHAMELEON_ERR_ILLEGAL_VALUE;
        }
    }
    *out = list_schedule(ct, workers, [&](int m, int) { return nbi(m); });
    *mode_out = mode;
    if (!replay_ok(*out, mode, N, NB, NTB)) {
        out->clear();
        return CHAMELEON_ERR_NOT_SUPPORTED;
    }
    return 0;
}

int CHAM_B200_Dag_Schedule(CHAM_b200_dag_t dag, int N, int NB, int nrhs, int NBB, int workers, void *out, int cap) {
    using namespace chb;
    if (!dag || N <= 0 || NB <= 0 || nrhs < 0 || (nrhs > 0 && NBB <= 0) || workers <= 0)
        return CHAMELEON_ERR_ILLEGAL_VALUE;
    std::vector<Task> tl;
    int mode = 0;
    if (int rc = dag_to_tasks(*dag, N, NB, nrhs, NBB, workers, &tl, &mode)) return rc;
    const int n = std::min<int>((int)tl.size(), cap);
    if (out) memcpy(out, tl.data(), sizeof(Task) * (size_t)std::max(0, n));
    return (int)tl.size();
}

int CHAM_B200_Dag_Run(CHAM_b200_dag_t dag, cham_uplo_t uplo, int N, int NB, double *A, const int64_t *a_off,
                      const int *a_ld, int nrhs, int NBB, double *B, const int64_t *b_off, const int *b_ld,
                      int *info) {
    using namespace chb;
    int rc = ensure_init();
    if (rc) return rc;
    if (!dag || !A || !a_off || !a_ld || N <= 0 || NB <= 0 || (uplo != ChamUpper && uplo != ChamLower) ||
        (nrhs > 0 && (!B || !b_off || !b_ld || NBB <= 0)))
        return CHAMELEON_ERR_ILLEGAL_VALUE;
    if (info) *info = 0;
    if (dag->rec.empty()) return 0;
    Context &c = ctx();
    const int NT = (N + NB - 1) / NB, NTB = nrhs > 0 ? (nrhs + NBB - 1) / NBB : 0;
    auto sch = std::make_unique<Schedule>();
    int mode = 0;
    if ((rc = dag_to_tasks(*dag, N, NB, nrhs, NBB, c.num_sms, &sch->tasks, &mode))) return rc;
    if ((rc = upload_schedule(sch.get()))) return rc;
    CHAM_desc_t *dA = nullptr, *dB = nullptr;
    rc = desc_create_from_tables(&dA, A, NB, N, N, a_off, a_ld);
    if (!rc && NTB) rc = desc_create_from_tables(&dB, B, NB, N, nrhs, b_off, b_ld, NBB);
    ExecResult res;
    if (!rc) {
        t_given = sch.get();
        rc = run_cholesky_dag(mode, uplo, dA, dB, c.stream, &res, 0, nullptr, 0, 0, nullptr);
        t_given = nullptr;
    }
    if (dA) CHAMELEON_Desc_Destroy(&dA);
    if (dB) CHAMELEON_Desc_Destroy(&dB);
    dev_free(sch->d_tasks);
    if (rc) return rc;
    if (res.error) return res.error;
    if (info) *info = res.info;
    (void)NT;
    return 0;
}

}  // extern "C"

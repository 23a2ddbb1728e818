// fwi_exec.cuh -- continuous batching: several independent runs advanced by the same step
// launches.  Included at the end of fwi_engine.cu (it drives the engine's internals).
//
// A run (one context: its model, shots and, for a gradient, observed data) joins the
// executor's batch at a launch boundary: from then on every step launch -- k_fold_groups launches
// on the executor's stream, and the step kernel's own for large one-shot windows -- advances each shot group of every run in the batch by the
// next item of that group's own program (forward steps, or replay + adjoint steps), whatever
// its grid size, record length or progress.  Between the passes of a run the executor issues
// that run's own work (gathers, adjoint sources, finalisation, stacking) on the same stream, and
// a run whose last work is issued leaves the batch and is handed back to its context's stream.
// Runs therefore overlap on the GPU step by step, and one that arrives while others are in
// flight starts at the next launch, not when they finish.
//
// Every run's arithmetic is the single-run engine's (same kernel body, same programs, same
// per-shot state), so its results are bit-identical alone and in any mix.
//
// The host keeps at most 128 launches in flight ahead of the device (an event every 32
// launches).  A step kernel that gave up waiting for a tile copy sets the executor's error
// word; every run in flight at that point fails with FWI_ERR_CUDA.

struct ExecGroup {
    int shot_base = 0, nshot = 0;
    // on plain fields (fold_wanted): launches of its own, large enough to fill the GPU, in the shape the
    // tuner picks for one shot; else its table entry.  One and three runs of 3.33 million cells, us a
    // forward step: 43.9 and 125 in a table, 27.5 and 83.4 on their own
    bool plain = false;
    FoldGroup G, G2;  // one column per thread; a group of one shot, two
    ShotDesc d;   // its first shot's descriptor
    const Program *prog = nullptr;
    long long L0 = 0;  // launch index of the program's item 0
};

struct ExecRun {
    fwi_ctx *c = nullptr;
    int problem = 0, filter = 2, precondition = 1;
    float freq = 0.f;
    int phase = 0;  // 0 forward pass, 1 adjoint pass, 2 handed back
    std::vector<ExecGroup> groups;
    cudaStream_t own = nullptr;  // the context's stream while it is out of the batch
    cudaEvent_t done = nullptr;
    long long end_launch = 0;  // launch index at which the current pass ends
    int status = FWI_OK;
    double cells = 0.0;
};

struct fwi_exec {
    int device = 0;
    int math = 0;  // arithmetic of the step kernel (FWI_MATH when the executor was created)
    cudaStream_t stream = nullptr;
    std::mutex mu;
    std::vector<ExecRun *> runs;      // in the batch
    std::vector<ExecRun *> finished;  // handed back, not yet polled
    // the groups of the runs in the batch, FOLD_GROUPS to a table, and where each comes from
    std::vector<std::unique_ptr<FoldTable>> tabs;
    std::vector<const ExecGroup *> order;
    bool dirty = true;
    long long L = 0;  // step launches issued
    int *d_err = nullptr, *h_err = nullptr;
    std::deque<cudaEvent_t> inflight, spare;
    long long launches_total = 0;
};

// Groups of one shot, whose blocks load their coefficients for that shot only, take two columns per thread,
// in tables of their own, where the batch has more one-column tiles (times shots and item halves) than
// this: half the blocks, each with more loads in flight, against more of them at once.  One column against
// two, 1 / 3 / 6 / 12 runs of one shot, us a forward step: 0.21 million cells (207 tiles) 4.4 / 7.8 / 12.6 / 28.8
// against 4.8 / 8.0 / 13.0 / 27.4, 0.30 million (356) 4.6 / 11.2 / 20.7 / 48.6 against 5.1 / 10.0 / 19.7 / 44.6,
// 0.67 million (693) 7.6 / 20.4 / 47.6 / 92.8 against 7.5 / 18.8 / 43.7 / 84.3.  (Several shots a group: 3 runs of
// 4 of 0.37 million 24.2 against 30.5.)
static constexpr long long FOLD_TWO_COLS = 1000;

// the batched path's set-up of a run without waves: per-shot runs, groups of consecutive shots
// sharing a model window, their frame pools and descriptors; initial frames zeroed
static int exec_setup(fwi_ctx *c, ExecRun *er)
{
    const bool gradient = er->problem == 1;
    const int ns = (int)c->shots.size();
    if ((int)c->runs.size() != ns) {
        free_runs(c);
        for (int i = 0; i < ns; i++) c->runs.emplace_back(new ShotRun());
    }
    c->direct = false;
    for (int i = 0; i < ns; i++) {
        c->in_batch = true;
        const int rc = prepare_run(c, c->runs[i].get(), i, gradient);
        c->in_batch = false;
        if (rc != FWI_OK) return rc;
        c->runs[i]->d.hessian = gradient && er->precondition == 1;
    }
    std::vector<std::pair<int, int>> gs;
    for (int i = 0; i < ns; i++) {
        if (gs.empty() || !same_group(c->runs[gs.back().first].get(), c->runs[i].get())) gs.push_back({i, 1});
        else gs.back().second++;
    }
    std::vector<ShotDesc> descs(ns);
    for (auto &g : gs) {
        std::vector<ShotRun *> rs;
        for (int i = g.first; i < g.first + g.second; i++) rs.push_back(c->runs[i].get());
        TRY(assign_pool(c, g.first, rs));
    }
    for (int i = 0; i < ns; i++) descs[i] = c->runs[i]->d;
    TRY(upload_descs(c, descs));
    TRY(ensure_red(c));
    void *scr;
    TRY(scratch(c, 64 * 1024, &scr));
    TRY(zero_initial(c, 0, ns, gradient ? 1 : 0));
    Program *pf, *pa;
    TRY(get_program(c, gradient ? "fwd1" : "fwd0", program_forward(c->nt, gradient ? K_FWD1 : K_FWD0), &pf));
    if (gradient) TRY(get_program(c, "adj/overlap", program_adjoint(c->nt, true), &pa));
    er->groups.clear();
    for (auto &g : gs) {
        ExecGroup eg;
        eg.shot_base = g.first;
        eg.nshot = g.second;
        const ShotDesc &d = c->runs[g.first]->d;
        eg.plain = d.W == 0;
        if (!eg.plain) TRY(fold_group_entry(d, c->d_desc, g.first, g.second, 1, &eg.G));
        if (!eg.plain && g.second == 1) TRY(fold_group_entry(d, c->d_desc, g.first, 1, 2, &eg.G2));
        eg.d = c->runs[g.first]->d;
        eg.prog = pf;
        er->groups.push_back(eg);
    }
    // cell updates of the run, as fwi_ctx_run counts them
    er->cells = 0.0;
    for (int i = 0; i < ns; i++) {
        const fwi_shot &s = c->shots[i].s;
        const double cellsz = (double)(c->nz + 2 * c->pml) * (s.ix_max - s.ix_min + 1 + 2 * c->pml);
        er->cells += cellsz * (gradient ? (double)c->nt * 2 + (c->nt - fwi_ck_count(c->nt)) : (double)c->nt);
    }
    return FWI_OK;
}

// the work of a run between its passes, issued on the executor's stream (the context's stream
// is the executor's while the run is in the batch)
static int exec_forward_done(fwi_exec *ex, ExecRun *er)
{
    fwi_ctx *c = er->c;
    for (auto &g : er->groups) {
        std::vector<ShotRun *> rs;
        for (int i = g.shot_base; i < g.shot_base + g.nshot; i++) rs.push_back(c->runs[i].get());
        if (er->problem == 0) {
            TRY(gather(c, rs, 0, false));
        } else if (er->problem == 2) {
            for (ShotRun *r : rs) TRY(prepare_taper(c, r, er->freq));
            if (er->filter == 0 || er->filter == 1) TRY(adjoint_source_filtered(c, rs, er->filter, false));
            else TRY(gather(c, rs, 1, false));
        } else {
            if (er->precondition == 1) TRY(finalize(c, rs, 0));
            for (ShotRun *r : rs) TRY(prepare_taper(c, r, er->freq));
            bool interp = false;
            for (ShotRun *r : rs) interp = interp || c->shots[r->shot].s.sampleRate > 1;
            if (er->filter == 2 && !interp) TRY(gather(c, rs, 1, true));
            else TRY(adjoint_source_filtered(c, rs, er->filter, true));
            TRY(dump_shot_traces(c, rs));
            TRY(adj_init(c, rs, g.shot_base));
            g.prog = &c->progs.at("adj/overlap");
            g.L0 = ex->L;
        }
    }
    return FWI_OK;
}

static int exec_adjoint_done(ExecRun *er)
{
    fwi_ctx *c = er->c;
    std::vector<ShotRun *> all;
    for (auto &g : er->groups) {
        std::vector<ShotRun *> rs;
        for (int i = g.shot_base; i < g.shot_base + g.nshot; i++) rs.push_back(c->runs[i].get());
        TRY(finalize(c, rs, 1));
        TRY(dump_shot_gradients(c, rs));
        if (er->precondition == 1) TRY(shot_precondition(c, rs));
        all.insert(all.end(), rs.begin(), rs.end());
    }
    return stack_and_precondition(c, all, er->precondition);
}

// the run leaves the batch: its context gets its own stream back, ordered after the run's work
static int exec_hand_back(fwi_exec *ex, ExecRun *er)
{
    fwi_ctx *c = er->c;
    CK(cudaEventRecord(er->done, ex->stream));
    c->stream = er->own;
    CK(cudaStreamWaitEvent(er->own, er->done, 0));
    c->stats.cell_updates = er->cells;
    er->phase = 2;
    return FWI_OK;
}

static long long exec_pass_end(const ExecRun *er)
{
    long long e = 0;
    for (const auto &g : er->groups) e = std::max(e, g.L0 + (long long)g.prog->items.size());
    return e;
}

extern "C" int fwi_exec_create(fwi_exec **out, int device)
{
    if (!out) return fail(FWI_ERR_ARG, "NULL output");
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n)
        return fail(FWI_ERR_NODEVICE, "no CUDA device %d: this engine runs on the GPU only", device);
    CK(cudaSetDevice(device));
    fwi_exec *ex = new fwi_exec();
    ex->device = device;
    if (const char *e = getenv("FWI_MATH")) ex->math = atoi(e) ? 1 : 0;
    CK(cudaStreamCreateWithFlags(&ex->stream, cudaStreamNonBlocking));
    CK(cudaMalloc(&ex->d_err, sizeof(int)));
    CK(cudaMemset(ex->d_err, 0, sizeof(int)));
    CK(cudaMallocHost(&ex->h_err, sizeof(int)));
    *ex->h_err = 0;
    *out = ex;
    return FWI_OK;
}

extern "C" int fwi_exec_add(fwi_exec *ex, fwi_ctx *c, int problem, float freq, int filter, int precondition)
{
    if (!ex || !c) return fail(FWI_ERR_ARG, "NULL executor or context");
    if (problem < 0 || problem > 2) return fail(FWI_ERR_ARG, "problem must be 0, 1 or 2 (got %d)", problem);
    if (filter < 0 || filter > 2) return fail(FWI_ERR_ARG, "residual filter %d (0 lowpass, 1 bandpass, 2 none)", filter);
    if (c->shots.empty()) return fail(FWI_ERR_STATE, "no shots");
    if (c->device != ex->device) return fail(FWI_ERR_ARG, "context and executor on different devices");
    if (c->dump.verbose > 1) return fail(FWI_ERR_UNSUPPORTED, "snapshots (verbose > 1) need fwi_ctx_run");
    if (c->math != ex->math) return fail(FWI_ERR_ARG, "context and executor differ in arithmetic (FWI_MATH)");
    CK(cudaSetDevice(c->device));
    ExecRun *er = new ExecRun();
    er->c = c;
    er->problem = problem;
    er->freq = freq;
    er->filter = filter;
    er->precondition = precondition;
    // set-up on the context's own stream (allocations synchronise that stream only)
    int rc = exec_setup(c, er);
    if (rc == FWI_OK && cudaEventCreateWithFlags(&er->done, cudaEventDisableTiming) != cudaSuccess)
        rc = fail(FWI_ERR_CUDA, "cudaEventCreate failed");
    if (rc != FWI_OK) {
        delete er;
        return rc;
    }
    er->own = c->stream;
    std::lock_guard<std::mutex> lk(ex->mu);
    CK(cudaEventRecord(er->done, er->own));
    CK(cudaStreamWaitEvent(ex->stream, er->done, 0));  // the batch waits for the set-up
    c->stream = ex->stream;
    for (auto &g : er->groups) g.L0 = ex->L;
    er->end_launch = exec_pass_end(er);
    ex->runs.push_back(er);
    ex->dirty = true;
    return FWI_OK;
}

// the launch tables: every group of every run in the batch, and the shots per block for all of them
static void exec_tables(fwi_exec *ex)
{
    ex->tabs.clear();
    ex->order.clear();
    long long items = 0;
    for (ExecRun *er : ex->runs)
        for (auto &g : er->groups)
            if (!g.plain) items += (long long)g.G.ntx * g.G.ts.zt * g.nshot * (er->phase == 1 ? 2 : 1);
    const bool two_cols = items > FOLD_TWO_COLS;
    for (int cols : {1, 2})
        for (ExecRun *er : ex->runs)
            for (auto &g : er->groups) {
                if (g.plain || (two_cols && g.nshot == 1 ? 2 : 1) != cols) continue;
                if (ex->tabs.empty() || ex->tabs.back()->ngroups == FOLD_GROUPS || ex->tabs.back()->g[0].T.ncol != cols) {
                    ex->tabs.emplace_back(new FoldTable);
                    ex->tabs.back()->ngroups = 0;
                }
                ex->tabs.back()->g[ex->tabs.back()->ngroups++] = cols == 2 ? g.G2 : g.G;
                ex->order.push_back(&g);
            }
    const int chunk = fold_group_chunk(items);
    for (auto &tb : ex->tabs)
        for (int i = 0; i < tb->ngroups; i++) tb->g[i].chunk = std::min(chunk, tb->g[i].nshot);
    ex->dirty = false;
}

// one step: item L - L0 of every group's program, a launch per table and per group on plain fields
static int exec_launch(fwi_exec *ex)
{
    if (ex->dirty) exec_tables(ex);
    size_t k = 0;
    for (auto &tb : ex->tabs) {
        int nb = 0;
        for (int i = 0; i < tb->ngroups; i++, k++) {
            FoldGroup &G = tb->g[i];
            const ExecGroup &eg = *ex->order[k];
            const Program *p = eg.prog;
            const long long Lg = ex->L - eg.L0;
            tb->b0[i] = nb;
            if (Lg < 0 || Lg >= (long long)p->items.size()) continue;  // no blocks in this launch
            // the adjoint program pairs replay and adjoint items; a half that is empty has no blocks
            const int4 &pw = p->items[(size_t)Lg];
            nb += fold_group_item(&G, eg.d, pw, (int)Lg, pw.z != K_NONE);
        }
        if (nb > 0) TRY(launch_fold_table(*tb, nb, ex->math, true, ex->stream, ex->d_err));
    }
    TileCfg cfg;
    cfg.nst = 2;
    cfg.minb = 3;
    for (ExecRun *er : ex->runs)
        for (const ExecGroup &g : er->groups) {
            const long long Lg = ex->L - g.L0;
            if (!g.plain || Lg < 0 || Lg >= (long long)g.prog->items.size()) continue;
            // the context's stream is the executor's
            TRY(launch_tiles(er->c, g.prog, (int)Lg, (int)Lg + 1, g.shot_base, g.nshot, er->c->runs[g.shot_base].get(), cfg,
                             ex->d_err));
        }
    return FWI_OK;
}

static int exec_fail_all(fwi_exec *ex, int code, const char *why)
{
    cudaStreamSynchronize(ex->stream);  // nothing of the failed runs may still be in flight
    for (ExecRun *er : ex->runs) {
        er->status = code;
        er->c->stream = er->own;
        er->phase = 2;
        ex->finished.push_back(er);
    }
    ex->runs.clear();
    ex->dirty = true;
    return fail(code, "%s", why);
}

// keep at most 128 launches in flight; read the error word as the device catches up.  The copy
// and the event between two launches end the programmatic overlap of that pair, so they come
// once per 32 launches.
static int exec_throttle(fwi_exec *ex)
{
    if (ex->L % 32 != 0) return FWI_OK;
    cudaEvent_t e;
    if (!ex->spare.empty()) {
        e = ex->spare.back();
        ex->spare.pop_back();
    } else {
        CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    CK(cudaMemcpyAsync(ex->h_err, ex->d_err, sizeof(int), cudaMemcpyDeviceToHost, ex->stream));
    CK(cudaEventRecord(e, ex->stream));
    ex->inflight.push_back(e);
    while (ex->inflight.size() > 4) {
        CK(cudaEventSynchronize(ex->inflight.front()));
        ex->spare.push_back(ex->inflight.front());
        ex->inflight.pop_front();
    }
    if (*ex->h_err) return exec_fail_all(ex, FWI_ERR_CUDA, "step kernel: a tile copy did not complete within 2 s");
    return FWI_OK;
}

extern "C" int fwi_exec_step(fwi_exec *ex, int launches, int *active)
{
    if (!ex) return fail(FWI_ERR_ARG, "NULL executor");
    std::lock_guard<std::mutex> lk(ex->mu);
    CK(cudaSetDevice(ex->device));
    for (int k = 0; (launches <= 0 || k < launches) && !ex->runs.empty(); k++) {
        TRY(exec_launch(ex));
        ex->L++;
        ex->launches_total++;
        // runs whose pass ended with this launch: their work between passes, or hand-back
        for (size_t i = 0; i < ex->runs.size();) {
            ExecRun *er = ex->runs[i];
            if (ex->L < er->end_launch) {
                i++;
                continue;
            }
            int rc = FWI_OK;
            if (er->phase == 0 && er->problem == 1) {
                rc = exec_forward_done(ex, er);
                if (rc == FWI_OK) {
                    er->phase = 1;
                    er->end_launch = exec_pass_end(er);
                    ex->dirty = true;
                    i++;
                    continue;
                }
            } else if (er->phase == 0) {
                rc = exec_forward_done(ex, er);
            } else {
                rc = exec_adjoint_done(er);
            }
            if (rc == FWI_OK) rc = exec_hand_back(ex, er);
            if (rc != FWI_OK) {
                er->status = rc;
                er->c->stream = er->own;
                er->phase = 2;
            }
            ex->finished.push_back(er);
            ex->runs.erase(ex->runs.begin() + i);
            ex->dirty = true;
        }
        TRY(exec_throttle(ex));
    }
    if (active) *active = (int)ex->runs.size();
    return FWI_OK;
}

extern "C" int fwi_exec_poll(fwi_exec *ex, fwi_ctx *c, int *done, int *status)
{
    if (!ex || !c || !done) return fail(FWI_ERR_ARG, "NULL argument");
    std::lock_guard<std::mutex> lk(ex->mu);
    *done = 0;
    for (size_t i = 0; i < ex->finished.size(); i++)
        if (ex->finished[i]->c == c) {
            ExecRun *er = ex->finished[i];
            *done = 1;
            if (status) *status = er->status;
            if (er->done) cudaEventDestroy(er->done);
            delete er;
            ex->finished.erase(ex->finished.begin() + i);
            return FWI_OK;
        }
    return FWI_OK;
}

extern "C" int fwi_exec_launches(fwi_exec *ex, long long *launches)
{
    if (!ex || !launches) return fail(FWI_ERR_ARG, "NULL argument");
    *launches = ex->launches_total;
    return FWI_OK;
}

extern "C" int fwi_exec_destroy(fwi_exec *ex)
{
    if (!ex) return FWI_OK;
    cudaSetDevice(ex->device);
    cudaStreamSynchronize(ex->stream);
    for (ExecRun *er : ex->runs) {  // runs never finished: hand their contexts back
        er->c->stream = er->own;
        if (er->done) cudaEventDestroy(er->done);
        delete er;
    }
    for (ExecRun *er : ex->finished) {
        if (er->done) cudaEventDestroy(er->done);
        delete er;
    }
    for (cudaEvent_t e : ex->inflight) cudaEventDestroy(e);
    for (cudaEvent_t e : ex->spare) cudaEventDestroy(e);
    cudaFree(ex->d_err);
    cudaFreeHost(ex->h_err);
    cudaStreamDestroy(ex->stream);
    delete ex;
    return FWI_OK;
}

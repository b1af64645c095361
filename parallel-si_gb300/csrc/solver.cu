// solver.cu -- host orchestration of one solver: device memory, the
// evaluation pipeline, the switch step and the solve_si loop.
#include <algorithm>
#include <cstring>
#include <string>

#include "device_common.cuh"
#include "kernels.h"
#include "psi_internal.h"
#include "solver.h"

namespace psi {

namespace {

int ceil_log2(int64_t x)
{
    int r = 0;
    while (((int64_t)1 << r) < x) r++;
    return r;
}

}  // namespace

int Solver::set_device()
{
    PSI_CUDA_TRY(cudaSetDevice(device_));
    return PSI_OK;
}

namespace {

int check_options(const psi_options &opt)
{
    if (opt.valuation_mode != PSI_VAL_PATH) return fail(PSI_ERR_INVALID, "unknown valuation_mode");
    if (opt.sublist_len < 2) return fail(PSI_ERR_INVALID, "sublist_len must be >= 2");
    if (opt.incremental < PSI_INCR_OFF || opt.incremental > PSI_INCR_ALWAYS)
        return fail(PSI_ERR_INVALID, "unknown incremental mode");
    if (opt.patch_limit < 0) return fail(PSI_ERR_INVALID, "patch_limit must be >= 0");
    if (opt.walk_block != 0 && (opt.walk_block < 32 || opt.walk_block > 1024 || opt.walk_block % 32 != 0))
        return fail(PSI_ERR_INVALID, "walk_block must be 0 or a multiple of 32 in [32, 1024]");
    if (opt.switch_kernel != PSI_SWITCH_THREAD && opt.switch_kernel != PSI_SWITCH_WARP)
        return fail(PSI_ERR_INVALID, "unknown switch_kernel");
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) return fail(PSI_ERR_NO_DEVICE, "no CUDA device available");
    if (opt.device < 0 || opt.device >= ndev) return fail(PSI_ERR_INVALID, "device ordinal out of range");
    return PSI_OK;
}

}  // namespace

int Solver::create(const CsrView &g, const psi_options &opt, Solver **out, bool validate)
{
    *out = nullptr;
    if (g.n < 0) return fail(PSI_ERR_INVALID, "negative vertex count");   // n = 0: the empty game
    if (2 * (int64_t)g.n + 2 > INT32_MAX) return fail(PSI_ERR_TOO_LARGE, "n too large for int32 tour ids");
    int rc = check_options(opt);
    if (rc) return rc;
    Solver *s = new Solver();
    s->device_ = opt.device;
    s->timing_ = opt.timing != 0;
    s->use_graph_ = opt.graph != 0;
    s->incremental_ = opt.incremental;
    s->patch_limit_ = opt.patch_limit;
    s->switch_warp_ = opt.switch_kernel == PSI_SWITCH_WARP;
    rc = s->alloc_arrays(g.n, g.m);
    if (!rc) rc = s->upload_game(g, validate);
    if (rc) {
        delete s;
        return rc;
    }
    *out = s;
    return PSI_OK;
}

int Solver::create_arena(int64_t max_vertices, int64_t max_edges, int32_t slots, const psi_options &opt,
                         Solver **out)
{
    *out = nullptr;
    if (max_vertices < 2 || max_edges < 1 || slots < 1) return fail(PSI_ERR_INVALID, "empty arena");
    if (2 * max_vertices + 2 > INT32_MAX || max_edges > INT32_MAX)
        return fail(PSI_ERR_TOO_LARGE, "arena too large for int32 ids");
    int rc = check_options(opt);
    if (rc) return rc;
    Solver *s = new Solver();
    s->device_ = opt.device;
    s->timing_ = opt.timing != 0;
    // admissions list their new vertices as changed ones: a patch evaluates them
    s->incremental_ = opt.incremental;
    s->patch_limit_ = opt.patch_limit;
    s->switch_warp_ = opt.switch_kernel == PSI_SWITCH_WARP;
    rc = s->alloc_arrays(max_vertices, max_edges, true);
    if (!rc) rc = s->init_arena(slots);
    if (rc) {
        delete s;
        return rc;
    }
    *out = s;
    return PSI_OK;
}

// Many games as one disjoint union (a batch): each game's arrays are copied
// as they are to their place in the device union and shifted there (no host
// packing); base receives the first vertex of every game (K+1 entries).
int Solver::create_union(const std::vector<const HostGame *> &gs, const psi_options &opt, Solver **out,
                         std::vector<int64_t> *base)
{
    *out = nullptr;
    const int32_t K = (int32_t)gs.size();
    if (K < 1) return fail(PSI_ERR_INVALID, "empty batch");
    std::vector<int32_t> table(2 * (size_t)K + 2);
    int32_t *ub = table.data(), *ue = ub + K + 1;
    int64_t n = 0, m = 0;
    int32_t top = 0;
    base->assign(1, 0);
    for (int32_t k = 0; k < K; k++) {
        const HostGame *g = gs[k];
        if (!g || g->n <= 0) return fail(PSI_ERR_INVALID, "empty game in batch");
        ub[k] = (int32_t)n;
        ue[k] = (int32_t)m;
        n += g->n;
        m += g->m;
        top = g->max_pri > top ? g->max_pri : top;
        base->push_back(n);
        if (2 * n + 2 > INT32_MAX) return fail(PSI_ERR_TOO_LARGE, "batch has too many vertices for int32 tour ids");
        if (m > INT32_MAX) return fail(PSI_ERR_TOO_LARGE, "batch has more than 2^31-1 edges");
    }
    ub[K] = (int32_t)n;
    ue[K] = (int32_t)m;
    int rc = check_options(opt);
    if (rc) return rc;
    Solver *s = new Solver();
    s->device_ = opt.device;
    s->timing_ = opt.timing != 0;
    s->use_graph_ = opt.graph != 0;
    s->incremental_ = opt.incremental;
    s->patch_limit_ = opt.patch_limit;
    s->switch_warp_ = opt.switch_kernel == PSI_SWITCH_WARP;
    rc = s->alloc_arrays(n, m, true);
    if (!rc) rc = s->upload_union(gs, table, base->back());
    if (rc) {
        delete s;
        return rc;
    }
    s->max_pri_ = top;
    *out = s;
    return PSI_OK;
}

int Solver::upload_union(const std::vector<const HostGame *> &gs, const std::vector<int32_t> &table, int64_t n)
{
    const int32_t K = (int32_t)gs.size();
    const int32_t *ub = table.data(), *ue = ub + K + 1;
    n_ = (int32_t)n;
    m_ = ue[K];
    np_ = n_;
    const struct {
        void **ptr;
        size_t bytes;
    } arrays[] = {{(void **)&game_of_, 4 * (size_t)n_}, {(void **)&gstate_, sizeof(int4) * (size_t)K},
                  {(void **)&gcount_, sizeof(unsigned long long) * (size_t)K}};
    for (const auto &a : arrays) {
        cudaError_t e = device_alloc(a.ptr, a.bytes, stream_);
        if (e != cudaSuccess) return fail(PSI_ERR_NOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
        allocs_.push_back(*a.ptr);
    }
    int32_t *d_tab = nullptr;
    PSI_CUDA_TRY(device_alloc((void **)&d_tab, 4 * table.size(), stream_));
    PSI_CUDA_TRY(cudaMemcpyAsync(d_tab, table.data(), 4 * table.size(), cudaMemcpyHostToDevice, stream_));
    for (int32_t k = 0; k < K; k++) {
        const HostGame &g = *gs[k];
        const size_t nb = 4 * (size_t)g.n;
        PSI_CUDA_TRY(cudaMemcpyAsync(st_ + ub[k], g.owner.data(), nb, cudaMemcpyHostToDevice, stream_));
        PSI_CUDA_TRY(cudaMemcpyAsync(pri_ + ub[k], g.priority.data(), nb, cudaMemcpyHostToDevice, stream_));
        PSI_CUDA_TRY(cudaMemcpyAsync(off_ + ub[k], g.offsets.data(), nb, cudaMemcpyHostToDevice, stream_));
        if (g.m)
            PSI_CUDA_TRY(cudaMemcpyAsync(tgt_ + ue[k], g.targets.data(), 4 * (size_t)g.m, cudaMemcpyHostToDevice,
                                         stream_));
    }
    launch_union_fixup(stream_, n_, m_, K, d_tab, d_tab + K + 1, off_, tgt_, game_of_);
    PSI_CUDA_TRY(cudaMemsetAsync(gcount_, 0, 8 * (size_t)K, stream_));
    cudaFreeAsync(d_tab, stream_);
    games_ = K;
    return finish_upload();
}

// A patch after few changes runs in one block and, unless patches are always
// wanted, gives up for the full evaluation past this many vertices, so that one
// block's search stays well below a full evaluation.  No game of 12 measured
// (random 1.2*10^6 to 2^24 vertices, few priorities, long paths) comes to it: the
// same patches and times with 65,536 and without it; 4,096 costs one 2 of its 54
// patches (2^24: 28.9 -> 29.9 ms).
constexpr int32_t kSoloMost = 16384;

// Device arrays for games of up to cap_n vertices and cap_m edges.
int Solver::alloc_arrays(int64_t cap_n, int64_t cap_m, bool many)
{
    int rc = set_device();
    if (rc) return rc;
    cap_n_ = cap_n;
    cap_m_ = cap_m;
    // Incremental evaluation: change-list capacity (larger lists mean a full
    // evaluation), re-evaluated set capacity, level cap of its search.  A full
    // evaluation takes about 50 us per 2^20 vertices, a patch 10 us and 1.5 us
    // per level and block, more where levels are wide: n/128 changes, n/16
    // vertices and n/20,000 levels.  Against n/64, n/8, 256, ms per solve: 2^20
    // vertices 5.5 -> 4.9, 2*10^6 8.5 -> 7.8, 2^24 37.0 -> 35.1, long-path 2^23
    // 17.8 -> 17.6, the 256-game batch 16.8 -> 17.2.
    if (incremental_ != PSI_INCR_OFF) {
        const bool always = incremental_ == PSI_INCR_ALWAYS;
        const int64_t cc = always ? cap_n : patch_limit_ > 0 ? patch_limit_ : std::max<int64_t>(1024, cap_n >> 7);
        const int64_t ac = always ? cap_n : std::max<int64_t>(4096, cap_n >> 4);
        ccap_ = (int32_t)std::max<int64_t>(1, std::min(cc, cap_n));
        acap_ = (int32_t)std::max<int64_t>(1, std::min(ac, cap_n));
        max_levels_ = always ? INT32_MAX : (int32_t)std::max<int64_t>(32, std::min<int64_t>(256, cap_n / 20000));
        solo_most_ = always ? INT32_MAX : kSoloMost;
    }
    ucap_ = cap_n + acap_;
    PSI_CUDA_TRY(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    for (auto &p : ph_) {
        PSI_CUDA_TRY(cudaEventCreate(&p.a));
        PSI_CUDA_TRY(cudaEventCreate(&p.b));
    }
    PSI_CUDA_TRY(cudaEventCreate(&region_a_));
    PSI_CUDA_TRY(cudaEventCreate(&region_b_));
    const struct {
        void **ptr;
        size_t bytes;
    } arrays[] = {
        {(void **)&owner_, (size_t)cap_n},
        {(void **)&pri_, 4 * (size_t)cap_n},
        {(void **)&off_, 4 * ((size_t)cap_n + 1)},
        {(void **)&tgt_, 4 * (size_t)cap_m},
        {(void **)&rev_off_, 4 * ((size_t)cap_n + 1)},
        {(void **)&rev_src_, 4 * (size_t)cap_m},
        {(void **)&plist_, 4 * (size_t)cap_n},
        {(void **)&strat_, 4 * (size_t)cap_n},
        {(void **)&st_, 4 * (size_t)cap_n},
        {(void **)&solved_, (size_t)cap_n},
        {(void **)&node_, sizeof(PathNode) * (size_t)cap_n},
        {(void **)&skip_, sizeof(int4) * (size_t)cap_n},
        {(void **)&key_, 4 * (size_t)cap_n},
        {(void **)&rdeep_, 4 * (size_t)cap_n},
        {(void **)&need_, (size_t)cap_n},
        {(void **)&tie_, (size_t)cap_n},
        {(void **)&watch_, (size_t)cap_n},
        {(void **)&ulist_, 4 * (size_t)ucap_},
        {(void **)&paths_, 2 * sizeof(int2) * (size_t)cap_n},
        {(void **)&jA_, sizeof(int4) * (size_t)cap_n},
        {(void **)&jB_, sizeof(int4) * (size_t)cap_n},
        {(void **)&dw_, sizeof(AllWords)},
        {(void **)&sync_, sizeof(SolveSync)},
    };
    for (const auto &a : arrays) {
        cudaError_t e = device_alloc(a.ptr, a.bytes, stream_);
        if (e != cudaSuccess) return fail(PSI_ERR_NOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
        allocs_.push_back(*a.ptr);
    }
    if (incremental_ != PSI_INCR_OFF) {
        const struct {
            void **ptr;
            size_t bytes;
        } patch[] = {
            {(void **)&clist_, 4 * (size_t)ccap_},
            {(void **)&alist_, 4 * (size_t)acap_},
            {(void **)&apos_, 4 * (size_t)std::max<int64_t>(1, cap_n)},
            {(void **)&pj_, (3 * sizeof(int4) + sizeof(int2)) * (size_t)acap_ + 4 * (size_t)kPatchSizes},
        };
        for (const auto &a : patch) {
            cudaError_t e = device_alloc(a.ptr, a.bytes, stream_);
            if (e != cudaSuccess)
                return fail(PSI_ERR_NOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
            allocs_.push_back(*a.ptr);
        }
        PSI_CUDA_TRY(cudaMemsetAsync(apos_, 0xff, 4 * (size_t)std::max<int64_t>(1, cap_n), stream_));   // -1: in no patch
    }
    ctl_ = &reinterpret_cast<AllWords *>(dw_)->ctl;
    // the small winning set; of a batch's or arena's games two words per vertex
    stage_bytes_ = std::max(kStagedCopy, 4 * (size_t)(std::min<int64_t>(cap_n, kSelectSmall) + 1));
    if (many) stage_bytes_ = std::max(stage_bytes_, std::min(kStageMost, 8 * (size_t)cap_n));
    PSI_CUDA_TRY(cudaMallocHost((void **)&hw_, sizeof(AllWords) + stage_bytes_));
    hctl_ = &reinterpret_cast<AllWords *>(hw_)->ctl;
    PSI_CUDA_TRY(cudaMemsetAsync(dw_, 0, sizeof(Words), stream_));
    PSI_CUDA_TRY(cudaMemsetAsync(sync_, 0, sizeof(SolveSync), stream_));
    PSI_CUDA_TRY(cudaMemsetAsync(skip_, 0, sizeof(int4) * (size_t)cap_n, stream_));   // of no evaluation (number 0)
    const GraphCtl fresh;
    // pageable source: staged before the call returns
    PSI_CUDA_TRY(cudaMemcpyAsync(ctl_, &fresh, sizeof fresh, cudaMemcpyHostToDevice, stream_));
    return PSI_OK;
}

// One game filling the arrays: upload, player lists, reverse CSR.  The
// owner array goes up as the caller's int32 (into st_, free until the first
// evaluation) and is narrowed on the device; the player lists are an ordered
// partition on the device.
int Solver::upload_game(const CsrView &g, bool validate)
{
    n_ = g.n;
    m_ = g.m;
    max_pri_ = g.max_pri;
    np_ = n_;
    PSI_CUDA_TRY(cudaMemcpyAsync(st_, g.owner, 4 * (size_t)n_, cudaMemcpyHostToDevice, stream_));
    PSI_CUDA_TRY(cudaMemcpyAsync(pri_, g.priority, 4 * (size_t)n_, cudaMemcpyHostToDevice, stream_));
    PSI_CUDA_TRY(cudaMemcpyAsync(off_, g.offsets, 4 * ((size_t)n_ + 1), cudaMemcpyHostToDevice, stream_));
    if (m_) PSI_CUDA_TRY(cudaMemcpyAsync(tgt_, g.targets, 4 * (size_t)m_, cudaMemcpyHostToDevice, stream_));
    if (validate) {
        int64_t bad_v = -1;
        int32_t check = 0, bad_e = 0, top = 0;
        int ve = validate_game(stream_, n_, m_, st_, pri_, off_, tgt_, &bad_v, &check, &bad_e, &top);
        if (ve) return fail(PSI_ERR_CUDA, std::string("validation: ") + cudaGetErrorString((cudaError_t)ve));
        if (bad_v >= 0) {
            std::string v = std::to_string(bad_v);
            if (check == 1) return fail(PSI_ERR_INVALID, "invalid player at vertex " + v);
            if (check == 2) return fail(PSI_ERR_INVALID, "negative priority at vertex " + v);
            return fail(PSI_ERR_INVALID, "vertex " + v + " has no successor");
        }
        if (bad_e) return fail(PSI_ERR_INVALID, "successor out of range");
        max_pri_ = top;
    }
    return finish_upload();
}

// Common tail of an upload: the owner array (uploaded as int32 into st_)
// narrowed, the player lists, fresh SI state and the reverse CSR.
int Solver::finish_upload()
{
    launch_narrow_owner(stream_, n_, st_, owner_);
    int ce = partition_players(stream_, n_, owner_, plist_, &dw_->selcount);
    if (ce) return fail(PSI_ERR_CUDA, std::string("player lists: ") + cudaGetErrorString((cudaError_t)ce));
    PSI_CUDA_TRY(cudaMemsetAsync(solved_, 0, n_, stream_));
    PSI_CUDA_TRY(cudaMemsetAsync(st_, 0, 4 * (size_t)n_, stream_));
    reset_tracking();
    // reverse CSR on the device (distinct in-neighbours, increasing order)
    int64_t rev_m = 0;
    ce = build_reverse_csr(stream_, n_, m_, off_, tgt_, rev_off_, rev_src_, &rev_m);
    if (ce) return fail(PSI_ERR_CUDA, std::string("reverse CSR: ") + cudaGetErrorString((cudaError_t)ce));
    int rc = sync_and_check("upload");
    if (rc) return rc;
    np0_ = hw_->selcount;
    return PSI_OK;
}

Solver::~Solver()
{
    cudaSetDevice(device_);
    if (stream_) cudaStreamSynchronize(stream_);
    if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
    if (graph_) cudaGraphDestroy(graph_);
    for (void *p : allocs_) cudaFreeAsync(p, stream_);   // back to the library's pool
    if (stream_) cudaStreamSynchronize(stream_);
    if (hw_) cudaFreeHost(hw_);
    for (auto &p : ph_) {
        if (p.a) cudaEventDestroy(p.a);
        if (p.b) cudaEventDestroy(p.b);
    }
    if (region_a_) cudaEventDestroy(region_a_);
    if (region_b_) cudaEventDestroy(region_b_);
    if (stream_) cudaStreamDestroy(stream_);
}

int Solver::timer_begin()
{
    int rc = set_device();
    if (rc) return rc;
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    PSI_CUDA_TRY(cudaEventRecord(region_a_, stream_));
    return PSI_OK;
}

int Solver::timer_end(double *ms)
{
    int rc = set_device();
    if (rc) return rc;
    PSI_CUDA_TRY(cudaEventRecord(region_b_, stream_));
    PSI_CUDA_TRY(cudaEventSynchronize(region_b_));
    float f = 0;
    PSI_CUDA_TRY(cudaEventElapsedTime(&f, region_a_, region_b_));
    *ms = f;
    return PSI_OK;
}

void Solver::phase_begin(Phase p)
{
    if (timing_) cudaEventRecord(ph_[p].a, stream_);
}

void Solver::phase_end(Phase p)
{
    if (!timing_) return;
    cudaEventRecord(ph_[p].b, stream_);
    ph_[p].pending = true;
}

// Called after a stream synchronisation: adds the elapsed time of every phase
// recorded since the last collection.
int Solver::collect_phases()
{
    for (int i = 0; i < PH_COUNT; i++) {
        if (!ph_[i].pending) continue;
        float ms = 0;
        PSI_CUDA_TRY(cudaEventElapsedTime(&ms, ph_[i].a, ph_[i].b));
        times_.ms[i] += ms;
        times_.calls[i]++;
        ph_[i].pending = false;
    }
    return PSI_OK;
}

int Solver::sync_and_check(const char *what)
{
    PSI_CUDA_TRY(cudaGetLastError());
    PSI_CUDA_TRY(cudaMemcpyAsync(hw_, dw_, sizeof(AllWords), cudaMemcpyDeviceToHost, stream_));
    cudaError_t e = cudaStreamSynchronize(stream_);
    if (e != cudaSuccess) return fail(PSI_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    int rc = collect_phases();
    if (rc) return rc;
    times_.patches = (int64_t)hw_->patch[0];
    times_.patched = (int64_t)hw_->patch[1];
    if (hw_->err) {
        uint32_t bits = hw_->err;
        cudaMemsetAsync(dw_, 0, sizeof(Words), stream_);
        cudaStreamSynchronize(stream_);
        return fail(PSI_ERR_LIMIT, std::string(what) + ": device step cap reached (bits " + std::to_string(bits) + ")");
    }
    return PSI_OK;
}

void Solver::reset_times()
{
    times_ = SolverTimes();
    cudaMemsetAsync(dw_->patch, 0, sizeof(dw_->patch), stream_);
    if (hw_) hw_->patch[0] = hw_->patch[1] = 0;
}

void Solver::reset_tracking()
{
    static const int32_t two = 2;   // patch_begin counts it down: nonzero in the next evaluation alone
    stale_ = false;
    fresh_ = true;
    cudaMemsetAsync(need_, 1, (size_t)n_, stream_);
    cudaMemsetAsync(tie_, 0, (size_t)n_, stream_);
    cudaMemsetAsync(watch_, 0, (size_t)n_, stream_);
    cudaMemcpyAsync(&ctl_->quiet, &two, sizeof two, cudaMemcpyHostToDevice, stream_);
}

void Solver::refresh_tracking(bool switching)
{
    if (stale_) reset_tracking();
    // a switch step before the next evaluation takes flags away: the
    // evaluation then has to flag what it changes
    if (fresh_ && switching) cudaMemsetAsync(&ctl_->quiet, 0, sizeof(int32_t), stream_);
    fresh_ = false;
}

int Solver::init_strat()
{
    int rc = set_device();
    if (rc) return rc;
    launch_init_strat(stream_, n_, owner_, off_, tgt_, strat_, st_);
    PSI_CUDA_TRY(cudaMemsetAsync(solved_, 0, n_, stream_));
    reset_tracking();
    rc = sync_and_check("init_strat");
    if (rc) return rc;
    strat_ready_ = true;
    val_ready_ = false;
    tracked_ = false;
    return PSI_OK;
}

int Solver::reset_opponent_strategy()
{
    if (!strat_ready_) return fail(PSI_ERR_STATE, "reset_opponent_strategy before init_strat");
    int rc = set_device();
    if (rc) return rc;
    launch_reset_odd(stream_, n_, owner_, off_, tgt_, strat_);
    reset_tracking();   // Odd's choices start over
    tracked_ = false;
    return sync_and_check("reset_opponent_strategy");
}

PatchArgs Solver::patch_args()
{
    PatchArgs a;
    a.g = ctl_;
    a.ucount = &dw_->ucount;
    a.clist = clist_;
    a.strat = strat_;
    a.pri = pri_;
    a.rev_off = rev_off_;
    a.rev_src = rev_src_;
    a.solved = solved_;
    a.alist = alist_;
    a.apos = apos_;
    a.rel = pj_;
    a.sja = pj_ ? pj_ + acap_ : nullptr;
    if (pj_) {
        a.spill = reinterpret_cast<int32_t *>(pj_ + 2 * (size_t)acap_);
        a.spill2 = a.spill + 2 * (size_t)acap_;
        a.arev = reinterpret_cast<int2 *>(pj_ + 3 * (size_t)acap_);
        a.sizes = reinterpret_cast<int32_t *>(a.arev + acap_);
    }
    a.sync = sync_;
    a.err = &dw_->err;
    a.n = n_;
    a.acap = acap_;
    a.ccap = ccap_;
    a.max_levels = max_levels_;
    a.solo_most = solo_most_;
    a.ucap = ucap_;
    a.st = st_;
    a.node = node_;
    a.rdeep = rdeep_;
    a.key = key_;
    a.ulist = ulist_;
    a.stats = dw_->patch;
    a.track = track();
    a.skip = skip_;
    a.sw = dw_->sw;
    a.epoch = &sync_->epoch;
    a.quiet = &ctl_->quiet;
    return a;
}

// Games up to this size are evaluated in full every time by one launch in the
// host-driven calls: a patch takes three launches and a level of its search
// longer than all the jumps.  Evaluation, mark_solved and switch step by step,
// us per evaluation with patches and walks -> so: 118 -> 85 (n = 1,537), 117 -> 90
// (10^4 and 10^5), 128 -> 100 (3*10^5), 153 -> 144 (10^6), 151 -> 140 (2^20 - 1); 24
// served games 11.9 -> 11.4 ms.
constexpr int32_t kJumpVertices = (1 << 20) - 1;

int Solver::enqueue_eval(bool timed, int32_t try_patch)
{
    if (n_ <= kJumpVertices && incremental_ != PSI_INCR_ALWAYS) {
        if (timed) phase_begin(PH_BROADCAST);
        int ce = launch_eval_jump(stream_, eval_args(), ctl_, &ctl_->quiet);
        if (ce) return fail(PSI_ERR_CUDA, std::string("evaluation kernel: ") + cudaGetErrorString((cudaError_t)ce));
        if (timed) phase_end(PH_BROADCAST);
        return PSI_OK;
    }
    int rc = enqueue_patch(timed, try_patch);
    if (!rc) rc = enqueue_full(timed);
    return rc;
}

// 0. a patch, when the gates allow it and it succeeds; otherwise its
//    kernels return at once and the full evaluation's gates are open
int Solver::enqueue_patch(bool timed, int32_t try_patch, const cudaGraphConditionalHandle *full)
{
    if (timed) phase_begin(PH_PATCH);
    const PatchArgs pa = patch_args();
    if (timed) launch_patch_begin(stream_, pa, try_patch);   // (the graph loop's control has done so)
    if (incremental_ != PSI_INCR_OFF) {
        int pe = launch_patch(stream_, pa, full);
        if (pe) return fail(PSI_ERR_CUDA, std::string("patch kernel: ") + cudaGetErrorString((cudaError_t)pe));
    }
    if (timed) phase_end(PH_PATCH);
    return PSI_OK;
}

EvalArgs Solver::eval_args()
{
    EvalArgs a;
    a.n = n_;
    a.strat = strat_;
    a.pri = pri_;
    a.solved = solved_;
    a.st = st_;
    a.node = node_;
    a.rdeep = rdeep_;
    a.skip = skip_;
    a.cap = cap_n_;
    a.g = ctl_;
    a.sw = dw_->sw;
    a.epoch = &sync_->epoch;
    a.key = key_;
    a.ulist = ulist_;
    a.ucount = &dw_->ucount;
    a.la = reinterpret_cast<int32_t *>(paths_);
    a.lcount = &dw_->lcount;
    a.ja = jA_;
    a.sync = sync_;
    a.err = &dw_->err;
    a.track = track();
    a.gate = &ctl_->eval;
    return a;
}

// The full evaluation (root_kernels.cu), every kernel gated (ctl_->eval).
int Solver::enqueue_full(bool timed)
{
    EvalArgs a = eval_args();
    if (!timed) a.gate = nullptr;   // in the graph's conditional node: it runs only when it has to
    if (timed) phase_begin(PH_BROADCAST);
    launch_root_init(stream_, a);
    launch_root_walk(stream_, a);
    if (timed) phase_end(PH_BROADCAST);
    if (timed) phase_begin(PH_CYCLES);
    int ce = launch_root_settle(stream_, a);
    if (ce) return fail(PSI_ERR_CUDA, std::string("settling kernel: ") + cudaGetErrorString((cudaError_t)ce));
    if (timed) phase_end(PH_CYCLES);
    return PSI_OK;
}

int Solver::compute_valuation()
{
    if (!strat_ready_) return fail(PSI_ERR_STATE, "compute_valuation before init_strat");
    int rc = set_device();
    if (rc) return rc;
    refresh_tracking(false);
    // the last evaluation's state and the switch steps' change list since are
    // usable only if no strategy changed outside a switch step
    const int32_t try_patch = (tracked_ && incremental_ != PSI_INCR_OFF) ? 1 : 0;
    const unsigned long long patches_before = hw_->patch[0];
    phase_begin(PH_EVAL);
    rc = enqueue_eval(true, try_patch);
    if (rc) return rc;
    phase_end(PH_EVAL);
    rc = sync_and_check("compute_valuation");
    if (rc) return rc;
    if (hw_->patch[0] == patches_before) {   // a full evaluation: ucount is its unreached count
        int32_t nu = hw_->ucount;
        last_unreached_ = nu;
        times_.unreached += nu;
        if (nu > 0) times_.jump_rounds += ceil_log2(nu) + 1;
    }
    times_.evals++;
    val_ready_ = true;
    tracked_ = true;
    return PSI_OK;
}

int Solver::mark_solved(int32_t player)
{
    if (player != 0 && player != 1) return fail(PSI_ERR_INVALID, "player must be 0 or 1");
    if (!val_ready_) return fail(PSI_ERR_STATE, "mark_solved before compute_valuation");
    int rc = set_device();
    if (rc) return rc;
    launch_mark_solved(stream_, mark_args(player));
    PSI_CUDA_TRY(cudaGetLastError());
    return PSI_OK;   // ordered on the stream before the next call
}

MarkArgs Solver::mark_args(int32_t player)
{
    MarkArgs m;
    m.ucount = &dw_->ucount;
    m.ulist = ulist_;
    m.player = player;
    m.st = st_;
    m.solved = solved_;
    if (gmask_) {   // a masked step (served games) scans the whole list
        m.game_of = game_of_;
        m.gmask = gmask_;
    } else {
        m.from = &ctl_->mfrom[player];
        m.done = &ctl_->mdone;
    }
    return m;
}

int Solver::switch_strategy(int32_t player, int64_t *switched, bool count, bool mark)
{
    if (player != 0 && player != 1) return fail(PSI_ERR_INVALID, "player must be 0 or 1");
    if (!val_ready_) return fail(PSI_ERR_STATE, "switch_strategy before compute_valuation");
    int rc = set_device();
    if (rc) return rc;
    refresh_tracking(true);
    const MarkArgs m = mark ? mark_args(player) : MarkArgs();
    phase_begin(PH_SWITCH);
    const int32_t np = (player == 0) ? np0_ : np_ - np0_;
    const int32_t *pl = plist_ + (player == 0 ? 0 : np0_);
    // jB_ is free until the next full evaluation: it holds the list of vertices to examine
    launch_switch(stream_, np, pl, player, off_, tgt_, strat_, st_, key_, node_, rdeep_, dw_->sw, game_of_, gcount_,
                  gmask_, &dw_->err, nullptr, need_, reinterpret_cast<int32_t *>(jB_), &dw_->listcount, changes(), tie_,
                  watch_, landmarks(), switch_warp_, &dw_->claim, arena_ ? nullptr : owner_, n_, count,
                  &dw_->listdone, mark ? &m : nullptr);
    phase_end(PH_SWITCH);
    rc = sync_and_check("switch_strategy");
    if (rc) return rc;
    times_.switches++;
    times_.sw_edges += (int64_t)hw_->sw[0];
    times_.sw_loads += (int64_t)hw_->sw[1];
    times_.sw_changed += (int64_t)hw_->sw[2];
    if (switched) *switched = (int64_t)hw_->sw[3];
    return PSI_OK;
}

int Solver::get_infinite(int32_t *out)
{
    int rc = set_device();
    if (rc) return rc;
    std::vector<int32_t> st(n_);
    PSI_CUDA_TRY(cudaMemcpyAsync(st.data(), st_, 4 * (size_t)n_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    for (int32_t v = 0; v < n_; v++) out[v] = st_infinite(st[v]);
    return PSI_OK;
}

int Solver::get_depth(int32_t *out)
{
    int rc = set_device();
    if (rc) return rc;
    PSI_CUDA_TRY(cudaMemcpyAsync(out, st_, 4 * (size_t)n_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    return PSI_OK;
}

int Solver::stage_in(const void *src, size_t bytes)
{
    PSI_CUDA_TRY(cudaMemcpyAsync(stage(), src, bytes, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    return PSI_OK;
}

int Solver::copy_out(void *dst, const void *src, size_t bytes)
{
    if (!bytes) {
        PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
        return PSI_OK;
    }
    cudaPointerAttributes at = {};
    const bool staged = bytes <= kStagedCopy && cudaPointerGetAttributes(&at, dst) == cudaSuccess &&
                        at.type == cudaMemoryTypeUnregistered;
    if (staged) {
        int rc = stage_in(src, bytes);
        if (!rc) std::memcpy(dst, stage(), bytes);
        return rc;
    }
    PSI_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    return PSI_OK;
}

int Solver::get_winning(int32_t player, int32_t *out, int64_t cap, int64_t *count)
{
    if (player != 0 && player != 1) return fail(PSI_ERR_INVALID, "player must be 0 or 1");
    int rc = set_device();
    if (rc) return rc;
    int32_t *sel = reinterpret_cast<int32_t *>(paths_);   // free between evaluations
    if (n_ <= kSelectSmall) {   // one block, size and ids in one copy
        launch_select_small(stream_, n_, player, st_, sel + 1, sel);
        PSI_CUDA_TRY(cudaGetLastError());
        rc = stage_in(sel, 4 * ((size_t)n_ + 1));
        if (rc) return rc;
        const int32_t *h = static_cast<const int32_t *>(stage());
        *count = h[0];
        if (out && cap > 0) std::memcpy(out, h + 1, 4 * (size_t)std::min<int64_t>(cap, h[0]));
        return PSI_OK;
    }
    if (!select_tmp_) {
        int ce = select_winning(stream_, n_, player, st_, sel, &dw_->selcount, nullptr, &select_bytes_);
        if (ce) return fail(PSI_ERR_CUDA, std::string("winning set: ") + cudaGetErrorString((cudaError_t)ce));
        PSI_CUDA_TRY(device_alloc(&select_tmp_, select_bytes_, stream_));
        allocs_.push_back(select_tmp_);
    }
    int ce = select_winning(stream_, n_, player, st_, sel, &dw_->selcount, select_tmp_, &select_bytes_);
    if (ce) return fail(PSI_ERR_CUDA, std::string("winning set: ") + cudaGetErrorString((cudaError_t)ce));
    rc = sync_and_check("get_winning");
    if (rc) return rc;
    *count = hw_->selcount;
    return out && cap > 0 ? copy_out(out, sel, 4 * (size_t)std::min<int64_t>(cap, *count)) : PSI_OK;
}

int Solver::get_winning_range(int64_t v0, int64_t n, int32_t player, int32_t *out, int64_t cap, int64_t *count)
{
    if (v0 < 0 || n < 0 || v0 + n > n_) return fail(PSI_ERR_INVALID, "vertex range out of bounds");
    int rc = set_device();
    if (rc) return rc;
    // half of the staging memory for status words, half for the ids found in them
    const int64_t part = std::min(n, (int64_t)(stage_bytes_ / 8));
    int32_t *st = static_cast<int32_t *>(stage()), *ids = st + part;
    int64_t k = 0;
    for (int64_t at = 0; at < n; at += part) {
        const int64_t len = std::min(n - at, part);
        PSI_CUDA_TRY(cudaMemcpyAsync(st, st_ + v0 + at, 4 * (size_t)len, cudaMemcpyDeviceToHost, stream_));
        PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
        int64_t found = 0;
        for (int64_t i = 0; i < len; i++) {   // no branches
            ids[found] = (int32_t)(at + i);
            found += (st[i] == ST_POS_INF) == (player == 0);
        }
        if (out && k < cap) std::memcpy(out + k, ids, 4 * (size_t)std::min(found, cap - k));
        k += found;
    }
    *count = k;
    return PSI_OK;
}

int Solver::get_range(const int32_t *src, int64_t v0, int64_t count, int32_t *out)
{
    if (v0 < 0 || count < 0 || v0 + count > n_) return fail(PSI_ERR_INVALID, "vertex range out of bounds");
    int rc = set_device();
    if (rc) return rc;
    return copy_out(out, src + v0, 4 * (size_t)count);
}

int Solver::get_strategy_range(int64_t v0, int64_t count, int32_t *out) { return get_range(strat_, v0, count, out); }

int Solver::get_strategy(int32_t *out)
{
    int rc = set_device();
    if (rc) return rc;
    return copy_out(out, strat_, 4 * (size_t)n_);
}

int Solver::get_solved(int32_t *out)
{
    int rc = set_device();
    if (rc) return rc;
    std::vector<uint8_t> s(n_);
    PSI_CUDA_TRY(cudaMemcpyAsync(s.data(), solved_, n_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    for (int32_t v = 0; v < n_; v++) out[v] = s[v];
    return PSI_OK;
}

int Solver::get_path_summary(int32_t *depth, int32_t *top, int32_t *count)
{
    if (!val_ready_) return fail(PSI_ERR_STATE, "get_path_summary before compute_valuation");
    int rc = set_device();
    if (rc) return rc;
    std::vector<int32_t> st(n_), deep(n_);
    std::vector<PathNode> nd(n_);
    PSI_CUDA_TRY(cudaMemcpyAsync(st.data(), st_, 4 * (size_t)n_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaMemcpyAsync(nd.data(), node_, sizeof(PathNode) * (size_t)n_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaMemcpyAsync(deep.data(), rdeep_, 4 * (size_t)n_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    for (int32_t v = 0; v < n_; v++) {
        const bool fin = st[v] >= 1;
        if (depth) depth[v] = fin ? st[v] : 0;
        if (top) top[v] = fin ? nd[v].rmax : -1;
        if (count) count[v] = !fin ? 0 : (st[v] < kDeepPath ? path_word_count(nd[v].word) : deep[v]);
    }
    return PSI_OK;
}

int Solver::set_strategy(const int32_t *in)
{
    int rc = set_device();
    if (rc) return rc;
    // every entry must be one of the vertex's successors, or the sink for Even
    std::vector<int32_t> own(n_), off(n_ + 1), tgt(m_);
    std::vector<int8_t> own8(n_);
    PSI_CUDA_TRY(cudaMemcpyAsync(own8.data(), owner_, n_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaMemcpyAsync(off.data(), off_, 4 * ((size_t)n_ + 1), cudaMemcpyDeviceToHost, stream_));
    if (m_) PSI_CUDA_TRY(cudaMemcpyAsync(tgt.data(), tgt_, 4 * (size_t)m_, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    for (int32_t v = 0; v < n_; v++) {
        int32_t t = in[v];
        bool ok = (t == -1 && own8[v] == 0);
        for (int32_t e = off[v]; !ok && e < off[v + 1]; e++) ok = (tgt[e] == t);
        if (!ok) return fail(PSI_ERR_INVALID, "strategy entry of vertex " + std::to_string(v) + " is not a successor");
    }
    PSI_CUDA_TRY(cudaMemcpyAsync(strat_, in, 4 * (size_t)n_, cudaMemcpyHostToDevice, stream_));
    reset_tracking();
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    strat_ready_ = true;
    tracked_ = false;
    return PSI_OK;
}

int Solver::get_valuation(int32_t v0, int32_t count, int32_t *out)
{
    if (!val_ready_) return fail(PSI_ERR_STATE, "get_valuation before compute_valuation");
    if (v0 < 0 || count < 0 || (int64_t)v0 + count > n_) return fail(PSI_ERR_INVALID, "vertex range out of bounds");
    int64_t d = (int64_t)max_pri_ + 1;
    int64_t bytes = 4 * d * count;
    if (count == 0) return PSI_OK;
    int rc = set_device();
    if (rc) return rc;
    int32_t *rows = nullptr;
    cudaError_t e = device_alloc((void **)&rows, (size_t)bytes, stream_);
    if (e != cudaSuccess) return fail(PSI_ERR_NOMEM, "valuation export buffer");
    launch_materialize(stream_, v0, count, (int32_t)d, st_, node_, rows, &dw_->err);
    PSI_CUDA_TRY(cudaMemcpyAsync(out, rows, (size_t)bytes, cudaMemcpyDeviceToHost, stream_));
    PSI_CUDA_TRY(cudaFreeAsync(rows, stream_));
    return sync_and_check("get_valuation");
}

int Solver::solve(int32_t reset, int32_t *iters, int32_t *brs, int64_t max_evals)
{
    int32_t it = 0, br = 0;
    bool first = true;
    int rc = init_strat();
    if (rc) return rc;
    for (;;) {
        if (!first && reset) {
            rc = reset_opponent_strategy();
            if (rc) return rc;
        }
        for (;;) {
            rc = first ? compute_first_val() : compute_valuation();
            if (rc) return rc;
            br++;
            int64_t sw = 0;
            rc = switch_strategy(1, &sw, false, true);
            if (rc) return rc;
            if (sw == 0) break;
            if (max_evals > 0 && br >= max_evals) {
                *iters = it;
                *brs = br;
                return fail(PSI_ERR_LIMIT, "evaluation cap reached");
            }
        }
        first = false;
        it++;
        int64_t sw = 0;
        rc = switch_strategy(0, &sw, false, true);
        if (rc) return rc;
        if (sw == 0) break;
        if (max_evals > 0 && br >= max_evals) {
            *iters = it;
            *brs = br;
            return fail(PSI_ERR_LIMIT, "evaluation cap reached");
        }
    }
    *iters = it;
    *brs = br;
    return PSI_OK;
}

// solve_si (main.cpp:20-55) over the union with per-game accounting
// (launch_batch_account): the union's loops end when no game switches.
int Solver::solve_batch(int32_t *iters, int32_t *brs)
{
    if (!games_ || arena_) return fail(PSI_ERR_STATE, "not a batch");
    if (use_graph_) {   // the default: the whole loop as one graph launch
        std::vector<int4> st;
        int rc = solve_batch_graph(st);
        if (rc) return rc;
        for (int32_t k = 0; k < games_; k++) {
            brs[k] = st[k].x;
            iters[k] = st[k].y;
            if (!st[k].w) return fail(PSI_ERR_STATE, "batch loop ended with an unfinished game");
        }
        return PSI_OK;
    }
    int rc = init_strat();
    if (rc) return rc;
    PSI_CUDA_TRY(cudaMemsetAsync(gstate_, 0, 16 * (size_t)games_, stream_));
    PSI_CUDA_TRY(cudaMemsetAsync(gcount_, 0, 8 * (size_t)games_, stream_));
    for (;;) {
        for (;;) {
            rc = compute_valuation();
            if (rc) return rc;
            launch_batch_account(stream_, games_, 0, gstate_, gcount_);
            int64_t sw = 0;
            rc = switch_strategy(1, &sw, false, true);
            if (rc) return rc;
            launch_batch_account(stream_, games_, 1, gstate_, gcount_);
            if (sw == 0) break;
        }
        launch_batch_account(stream_, games_, 2, gstate_, gcount_);
        int64_t sw = 0;
        rc = switch_strategy(0, &sw, false, true);
        if (rc) return rc;
        launch_batch_account(stream_, games_, 3, gstate_, gcount_);
        if (sw == 0) break;
    }
    std::vector<int4> st((size_t)games_);
    PSI_CUDA_TRY(cudaMemcpyAsync(st.data(), gstate_, 16 * (size_t)games_, cudaMemcpyDeviceToHost, stream_));
    rc = sync_and_check("solve_batch");
    if (rc) return rc;
    for (int32_t k = 0; k < games_; k++) {
        brs[k] = st[k].x;
        iters[k] = st[k].y;
        if (!st[k].w) return fail(PSI_ERR_STATE, "batch loop ended with an unfinished game");
    }
    return PSI_OK;
}

// ---- serving arena ------------------------------------------------------

int Solver::init_arena(int32_t slots)
{
    n_ = 0;
    m_ = 0;
    max_pri_ = 0;
    np0_ = np_ = 0;
    const struct {
        void **ptr;
        size_t bytes;
    } arrays[] = {{(void **)&game_of_, 4 * (size_t)cap_n_},
                  {(void **)&gstate_, sizeof(int4) * (size_t)slots},
                  {(void **)&gcount_, sizeof(unsigned long long) * (size_t)slots},
                  {(void **)&gmask_, 4 * (size_t)slots}};
    for (const auto &a : arrays) {
        cudaError_t e = device_alloc(a.ptr, a.bytes, stream_);
        if (e != cudaSuccess) return fail(PSI_ERR_NOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
        allocs_.push_back(*a.ptr);
    }
    games_ = slots;
    arena_ = true;
    PSI_CUDA_TRY(cudaMemsetAsync(solved_, 1, (size_t)cap_n_, stream_));          // every slot inert
    PSI_CUDA_TRY(cudaMemsetAsync(game_of_, 0xff, 4 * (size_t)cap_n_, stream_));   // -1: in no game
    PSI_CUDA_TRY(cudaMemsetAsync(st_, 0, 4 * (size_t)cap_n_, stream_));            // no finite depths
    PSI_CUDA_TRY(cudaMemsetAsync(gstate_, 0, sizeof(int4) * (size_t)slots, stream_));
    PSI_CUDA_TRY(cudaMemsetAsync(gcount_, 0, sizeof(unsigned long long) * (size_t)slots, stream_));
    PSI_CUDA_TRY(cudaMemsetAsync(gmask_, 0, 4 * (size_t)slots, stream_));
    PSI_CUDA_TRY(cudaStreamSynchronize(stream_));
    strat_ready_ = true;
    return PSI_OK;
}

// Places the games admitted in one step: each game's arrays are copied as
// they are into a device staging union (no host packing), shifted to union
// numbering on the device, given one reverse-CSR build and placed by one
// launch.  They are listed as changed vertices, so the next evaluation may
// be a patch.
int Solver::arena_add(const std::vector<const HostGame *> &gs, const std::vector<int32_t> &vb,
                      const std::vector<int32_t> &eb, const std::vector<int32_t> &slot, int32_t extent)
{
    if (!arena_) return fail(PSI_ERR_STATE, "not an arena");
    const int32_t K = (int32_t)gs.size();
    if (K == 0) return PSI_OK;
    if ((int32_t)vb.size() != K || (int32_t)eb.size() != K || (int32_t)slot.size() != K || extent > cap_n_)
        return fail(PSI_ERR_INVALID, "arena placement lists disagree");
    int64_t n = 0, m = 0;
    int32_t top = 0;
    // per-game table: ub[K+1], ue[K+1], vb[K], eb[K], slot[K]
    std::vector<int32_t> table(5 * (size_t)K + 2);
    int32_t *ub = table.data(), *ue = ub + K + 1;
    for (int32_t k = 0; k < K; k++) {
        const HostGame &g = *gs[k];
        if (g.n <= 0 || slot[k] < 0 || slot[k] >= games_ || vb[k] < 0 || eb[k] < 0 ||
            (int64_t)vb[k] + g.n + 1 > extent || (int64_t)eb[k] + g.m > cap_m_)
            return fail(PSI_ERR_INVALID, "arena placement out of range");
        ub[k] = (int32_t)n;
        ue[k] = (int32_t)m;
        n += g.n;
        m += g.m;
        top = g.max_pri > top ? g.max_pri : top;
        table[2 * (size_t)K + 2 + k] = vb[k];
        table[3 * (size_t)K + 2 + k] = eb[k];
        table[4 * (size_t)K + 2 + k] = slot[k];
    }
    if (2 * n + 2 > INT32_MAX || m > INT32_MAX) return fail(PSI_ERR_TOO_LARGE, "admission too large for int32 ids");
    ub[K] = (int32_t)n;
    ue[K] = (int32_t)m;
    int rc = set_device();
    if (rc) return rc;
    int32_t *d_tab = nullptr, *u_owner = nullptr, *u_pri = nullptr, *u_off = nullptr, *u_tgt = nullptr,
            *u_roff = nullptr, *u_rsrc = nullptr;
    int32_t **bufs[] = {&d_tab, &u_owner, &u_pri, &u_off, &u_tgt, &u_roff, &u_rsrc};
    const size_t sizes[] = {4 * table.size(),   4 * (size_t)n,       4 * (size_t)n,      4 * ((size_t)n + 1),
                            4 * (size_t)m,      4 * ((size_t)n + 1), 4 * (size_t)m};
    cudaError_t e = cudaSuccess;
    int64_t mr = 0;
    int ce = 0;
    for (int i = 0; i < 7 && e == cudaSuccess; i++) e = device_alloc((void **)bufs[i], sizes[i], stream_);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_tab, table.data(), sizes[0], cudaMemcpyHostToDevice, stream_);
    for (int32_t k = 0; k < K && e == cudaSuccess; k++) {
        const HostGame &g = *gs[k];
        const size_t nb = 4 * (size_t)g.n;
        e = cudaMemcpyAsync(u_owner + ub[k], g.owner.data(), nb, cudaMemcpyHostToDevice, stream_);
        if (e == cudaSuccess) e = cudaMemcpyAsync(u_pri + ub[k], g.priority.data(), nb, cudaMemcpyHostToDevice, stream_);
        if (e == cudaSuccess) e = cudaMemcpyAsync(u_off + ub[k], g.offsets.data(), nb, cudaMemcpyHostToDevice, stream_);
        if (e == cudaSuccess && g.m)
            e = cudaMemcpyAsync(u_tgt + ue[k], g.targets.data(), 4 * (size_t)g.m, cudaMemcpyHostToDevice, stream_);
    }
    if (e == cudaSuccess) {
        launch_union_fixup(stream_, (int32_t)n, m, K, d_tab, d_tab + K + 1, u_off, u_tgt);
        ce = build_reverse_csr(stream_, (int32_t)n, m, u_off, u_tgt, u_roff, u_rsrc, &mr);
    }
    if (e == cudaSuccess && !ce) {
        // with full evaluations only, the unreached list is rebuilt before its next use; after a
        // patch mark_solved reads it (the new vertices are appended by the patch)
        if (incremental_ == PSI_INCR_OFF) e = cudaMemsetAsync(&dw_->ucount, 0, sizeof(int32_t), stream_);
        const int32_t *vbd = d_tab + 2 * K + 2, *ebd = d_tab + 3 * K + 2, *sld = d_tab + 4 * K + 2;
        launch_arena_place(stream_, (int32_t)n, K, d_tab, vbd, ebd, sld, u_owner, u_pri, u_off, u_tgt, u_roff, u_rsrc,
                           owner_, pri_, off_, tgt_, rev_off_, rev_src_, strat_, st_, solved_, game_of_, gstate_,
                           gcount_, need_, changes());
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    for (int i = 0; i < 7; i++)
        if (*bufs[i]) cudaFreeAsync(*bufs[i], stream_);
    if (ce) return fail(PSI_ERR_CUDA, std::string("reverse CSR: ") + cudaGetErrorString((cudaError_t)ce));
    if (e != cudaSuccess) return fail(PSI_ERR_CUDA, std::string("arena_add: ") + cudaGetErrorString(e));
    if (top > max_pri_) max_pri_ = top;
    n_ = extent;
    return sync_and_check("arena_add");
}

// Retires games: their ranges become inert (one
// synchronisation for all of them).
int Solver::arena_remove(const std::vector<int32_t> &vb, const std::vector<int32_t> &count,
                         const std::vector<int32_t> &slot, int32_t extent)
{
    if (!arena_) return fail(PSI_ERR_STATE, "not an arena");
    const size_t K = vb.size();
    if (count.size() != K || slot.size() != K || extent > cap_n_) return fail(PSI_ERR_INVALID, "arena lists disagree");
    for (size_t k = 0; k < K; k++)
        if (slot[k] < 0 || slot[k] >= games_ || vb[k] < 0 || count[k] < 0 || (int64_t)vb[k] + count[k] > cap_n_)
            return fail(PSI_ERR_INVALID, "arena range out of range");
    int rc = set_device();
    if (rc) return rc;
    for (size_t k = 0; k < K; k++) {
        launch_arena_clear(stream_, vb[k], count[k], solved_, game_of_, st_);
        PSI_CUDA_TRY(cudaMemsetAsync(gstate_ + slot[k], 0, sizeof(int4), stream_));
    }
    // the retired vertices left in the unreached list are solved: mark_solved passes them by
    if (incremental_ == PSI_INCR_OFF) PSI_CUDA_TRY(cudaMemsetAsync(&dw_->ucount, 0, sizeof(int32_t), stream_));
    n_ = extent;
    return sync_and_check("arena_remove");
}

int Solver::arena_export(int32_t vb, int32_t count, int32_t *strategy, int32_t *infinite)
{
    if (vb < 0 || count < 0 || (int64_t)vb + count > n_) return fail(PSI_ERR_INVALID, "arena range out of range");
    if (count == 0) return PSI_OK;
    int32_t *out = nullptr;
    cudaError_t e = device_alloc((void **)&out, 8 * (size_t)count, stream_);
    if (e != cudaSuccess) return fail(PSI_ERR_NOMEM, "arena export buffer");
    launch_arena_export(stream_, vb, count, strat_, st_, out);
    // the caller's arrays are new memory: by way of the staging memory where they fit
    auto get = [&](int32_t *dst, const int32_t *src) {
        if (4 * (size_t)count > stage_bytes_) return copy_out(dst, src, 4 * (size_t)count);
        int rc = stage_in(src, 4 * (size_t)count);
        if (!rc) std::memcpy(dst, stage(), 4 * (size_t)count);
        return rc;
    };
    int rc = get(strategy, out);
    if (!rc) rc = get(infinite, out + count);
    cudaFreeAsync(out, stream_);
    return rc ? rc : sync_and_check("arena_export");
}

// Player lists of the vertices that belong to games (Even's first).
int Solver::arena_rebuild_lists()
{
    int rc = set_device();
    if (rc) return rc;
    PSI_CUDA_TRY(cudaMemsetAsync(&dw_->selcount, 0, sizeof(int32_t), stream_));
    launch_build_plist(stream_, n_, 0, owner_, game_of_, plist_, &dw_->selcount);
    rc = sync_and_check("arena_rebuild_lists");
    if (rc) return rc;
    np0_ = hw_->selcount;
    launch_build_plist(stream_, n_, 1, owner_, game_of_, plist_, &dw_->selcount);   // appends after Even's
    rc = sync_and_check("arena_rebuild_lists");
    if (rc) return rc;
    np_ = hw_->selcount;
    return PSI_OK;
}

// One solve_si step (main.cpp:20-55) of every resident game, each by its own
// state machine (launch_serve_account): evaluate all, switch Odd in all, then
// mark_solved(Even) and switch Even only in the games whose Odd made no
// strict improvement in this step.
int Solver::arena_step(bool reset, std::vector<int32_t> &done, std::vector<int32_t> &iters,
                       std::vector<int32_t> &brs)
{
    done.clear();
    iters.clear();
    brs.clear();
    if (!arena_) return fail(PSI_ERR_STATE, "not an arena");
    if (n_ == 0 || np_ == 0) return PSI_OK;
    int rc = compute_valuation();
    if (rc) return rc;
    int32_t *mask = gmask_;
    gmask_ = nullptr;                       // Odd's step: every resident game
    int64_t sw = 0;
    rc = switch_strategy(1, &sw, false, true);
    gmask_ = mask;
    if (rc) return rc;
    launch_serve_account(stream_, games_, 1, gstate_, gcount_, gmask_);
    rc = switch_strategy(0, &sw, false, true);   // Even's step: games with gmask set
    if (rc) return rc;
    if (reset)
        launch_serve_reset_odd(stream_, np_ - np0_, plist_ + np0_, game_of_, gmask_, gcount_, off_, tgt_, strat_,
                               need_, changes());
    launch_serve_account(stream_, games_, 2, gstate_, gcount_, gmask_);
    std::vector<int4> big;
    int4 *st = nullptr;
    if (sizeof(int4) * (size_t)games_ <= stage_bytes_) {
        st = static_cast<int4 *>(stage());
    } else {
        big.resize((size_t)games_);
        st = big.data();
    }
    PSI_CUDA_TRY(cudaMemcpyAsync(st, gstate_, sizeof(int4) * (size_t)games_, cudaMemcpyDeviceToHost, stream_));
    rc = sync_and_check("arena_step");
    if (rc) return rc;
    for (int32_t k = 0; k < games_; k++)
        if ((st[k].z & 1) && (st[k].z & 2)) {
            done.push_back(k);
            iters.push_back(st[k].y);
            brs.push_back(st[k].x);
        }
    return PSI_OK;
}

}  // namespace psi

// mixed_host.cu -- host driver of the mixed-precision solves (see mixed.cu).
#include <algorithm>
#include <cstring>

#include "mixed.h"
#include "runtime.h"
#include "tuner.h"

namespace ns3d {

void DevSys::allocate_f32(cudaStream_t st) {
    if (coef32.n) return;
    invdiag32.alloc_zero(npad, st);
    for (DBuf<float> *b : {&fx, &fr, &fr0, &fp, &fv, &fy, &fs, &fz, &ft, &fp2, &fv2}) b->alloc_zero(npad, st);
    coef32.alloc_zero((size_t)7 * npad, st);  // last: it stands for all of them
}

template <int CAP>
void MixedSetT<CAP>::configure(const std::vector<SolveItem> &items, cudaStream_t st) {
    std::vector<const double *> key;
    for (const SolveItem &it : items) {
        key.push_back(it.sys->coef.p);
        key.push_back(it.x);
        key.push_back(it.b);
    }
    // a merged set's members come and go (a new solve may reuse a finished
    // one's addresses): it is set up afresh every run
    if (CAP <= KMAX && key == key_) return;
    const int ns = (int)items.size();
    if (ns > CAP) throw ApiError(NS3D_ERR_ARG, "too many systems in one solve set");
    std::vector<MSys> ms(ns);
    int chunk = 0;
    key_.clear();  // set_ may name freed buffers until the end of this set-up, should an allocation fail
    bar_.reserve(ns, state_bytes(ns), st);
    if ((int)out_st_.n < ns) out_st_.alloc_zero(ns, st);
    if ((int)h_out_.n < ns) h_out_.alloc(ns);
    for (int i = 0; i < ns; ++i) {
        DevSys &S = *items[i].sys;
        S.allocate_f32(st);
        MSys &m = ms[i];
        std::memset(&m, 0, sizeof m);
        m.n = S.n;
        m.npad = S.npad;
        m.nchunks = S.nchunks;
        m.chunk_begin = chunk;
        chunk += S.nchunks;
        m.nbr = S.nbr.p;
        m.coef64 = S.coef.p;
        m.b64 = items[i].b;
        m.x64 = items[i].x;
        m.r64 = S.r.p;
        m.d64 = S.y.p;
        m.wy = reinterpret_cast<unsigned long long *>(S.p.p);
        m.wz = reinterpret_cast<unsigned long long *>(S.v.p);
        m.coef32 = S.coef32.p;
        m.invdiag32 = S.invdiag32.p;
        m.x = S.fx.p; m.r = S.fr.p; m.r0 = S.fr0.p; m.p = S.fp.p; m.v = S.fv.p;
        m.p2 = S.fp2.p; m.v2 = S.fv2.p;
        m.y = S.fy.p; m.s = S.fs.p; m.z = S.fz.p; m.t = S.ft.p;
        m.part = S.part.p;
        m.st = st_of(bar_.dev.p) + i;
        m.dc = dc_of(bar_.dev.p) + i;
        // a solver instance's own set: the multilevel preconditioner for a
        // single system; a merged set: what each system's own set chose
        const bool mg = CAP > KMAX ? (items[i].mg && S.mg)
                                   : (use_mg && ns == 1 && S.n > kMGCoarsest && S.cell_ny > 0);
        if (mg) {
            if (!S.mg) build_hierarchy(S, st);
            m.mg.nlev = S.mg->nlev;
            m.mg.pack = S.mg->pack.p;
            m.mg.sweeps = 30;
            m.mg.omega = 0.6f;
            for (int k = 1; k <= S.mg->nlev; ++k) {
                MGHostLevel &H = S.mg->lev[k];
                MGLevel &G = m.mg.lev[k];
                G.n = H.n;
                G.npad = H.npad;
                G.nbr = H.nbr.p;
                G.coef = H.coef.p;
                G.invdiag = H.invdiag.p;
                G.pos = H.pos.p;
                G.mstart = H.mstart.p;
                G.members = H.members.p;
                G.x = H.x.p;
                G.b = H.b.p;
                G.t = H.t.p;
                G.xo = H.xo.p;
                G.t8 = H.t8.p;
            }
            // the tail: the levels that fit in a block's shared memory (a
            // merged set has no shared memory of its own per system)
            m.mg.tail = m.mg.nlev + 1;
            if (CAP <= KMAX)
                for (int rows = 0; m.mg.tail > 1; --m.mg.tail) {
                    rows += m.mg.lev[m.mg.tail - 1].n;
                    if (rows > MG_TAIL_ROWS) break;
                }
        }
    }
    std::memset(&set_, 0, sizeof set_);
    set_.nsys = ns;
    set_.total_chunks = chunk;
    for (int i = 0; i < ns; ++i) set_.sys[i] = ms[i];
    key_ = key;
    nsys_ = ns;
    total_chunks_ = chunk;
}

template <int CAP>
int MixedSetT<CAP>::variant() const {
    long rows = 0;
    bool mg = false;
    for (int i = 0; i < nsys_; ++i) {
        rows += set_.sys[i].n;
        mg = mg || set_.sys[i].mg.nlev > 0;
    }
    return m32_fused(rows, mg) ? 1 : 0;
}

template <int CAP>
void MixedSetT<CAP>::run(const std::vector<SolveItem> &items, cudaStream_t st, std::vector<SolveOutcome> &out,
                         int variant) {
    configure(items, st);
    const int ns = nsys_;
    int maxit = 0;
    DCState *const h_dc = dc_of(bar_.host.p);
    KState *const h_st = st_of(bar_.host.p);
    std::memset(bar_.host.p, 0, state_bytes(bar_.cap));
    for (int i = 0; i < ns; ++i) {
        DevSys &S = *items[i].sys;
        launch_to_f32(S.coef.p, S.invdiag.p, S.npad, S.coef32.p, S.invdiag32.p, st);
        if (set_.sys[i].mg.nlev > 0) launch_mg_galerkin(set_.sys[i], st);
        DCState d;
        std::memset(&d, 0, sizeof d);
        d.tol = items[i].tol;
        d.maxit = items[i].maxit;
        d.tin_min = inner_rel_tol;
        d.inner_cap = inner_cap;
        if (S.n == 0) {
            d.done = 1;
            d.zero_rhs = 1;
            d.total_iter = d.maxit;
            d.error = d.tol;
        }
        h_dc[i] = d;
        maxit = std::max(maxit, items[i].maxit);
    }
    NS3D_CUDA_CHECK(cudaMemcpyAsync(bar_.dev.p, bar_.host.p, state_bytes(bar_.cap), cudaMemcpyHostToDevice, st));
    plan_mixed(set_, share);
    launch_dc_resid(set_, 1, st);
    // Every round runs at least one inner iteration per unfinished system, so
    // maxit + 2 rounds bound the loop; each round's inner loop is bounded by
    // the remaining iteration budget.
    long rounds = 0;
    // merged sets: the grid of each FP32 loop launch comes from the
    // autotuner, told the launch's time per inner row-iteration
    const bool tune = CAP > KMAX;
    int cand = 0, kind = 0;
    if (tune) {
        bool mg = false;
        for (int i = 0; i < ns; ++i) mg = mg || set_.sys[i].mg.nlev > 0;
        kind = mg ? 3 : set_.resident ? 4 : (variant == 1 ? 2 : 1);
        if (!ev_[0])
            for (cudaEvent_t &e : ev_) NS3D_CUDA_CHECK(cudaEventCreate(&e));
    }
    const uint64_t tkey = tuner_key(kind, (long)total_chunks_ * MSUB, share);
    std::vector<int> iters_before(ns, 0);
    // One round = FP32 init, the FP32 loop kernel (it ends when every inner
    // solve of the round is done: each is capped by the remaining iteration
    // budget), the FP64 update and residual; the host reads barrier and states
    // once per round.  The first round follows the first residual unseen: its
    // kernels skip the systems that are done already.
    while (true) {
        if (rounds > 0) {
            NS3D_CUDA_CHECK(cudaMemcpyAsync(bar_.host.p, bar_.dev.p, state_bytes(bar_.cap), cudaMemcpyDeviceToHost, st));
            NS3D_CUDA_CHECK(cudaStreamSynchronize(st));
            if (total_chunks_ > 0 && bar_.host.p->err)
                throw ApiError(NS3D_ERR_TIMEOUT, "FP32 BiCGSTAB loop kernel: a grid barrier timed out");
            if (tune) {  // inner iterations of the round, from the FP64 states
                double rows = 0;
                for (int i = 0; i < ns; ++i)
                    if (!h_dc[i].zero_rhs) rows += (double)set_.sys[i].n * (h_dc[i].total_iter - iters_before[i]);
                float ms = 0;
                NS3D_CUDA_CHECK(cudaEventElapsedTime(&ms, ev_[0], ev_[1]));
                grid_tuner().report(tkey, cand, ms, rows);
            }
            for (int i = 0; i < ns; ++i) iters_before[i] = h_dc[i].total_iter;
            bool all_done = true;
            for (int i = 0; i < ns; ++i) all_done = all_done && h_dc[i].done;
            if (all_done) break;
        }
        if (++rounds > maxit + 2L) throw ApiError(NS3D_ERR_TIMEOUT, "defect correction exceeded its round bound");
        launch_m32_init(set_, st);
        if (tune) {
            cand = grid_tuner().choose(tkey);
            NS3D_CUDA_CHECK(cudaEventRecord(ev_[0], st));
        }
        NS3D_CUDA_CHECK(launch_m32_loop(set_, bar_.dev.p, maxit + 64, st, variant, share << cand));
        if (tune) NS3D_CUDA_CHECK(cudaEventRecord(ev_[1], st));
        launch_dc_update(set_, st);
        launch_dc_resid(set_, 0, st);
    }
    out.assign(ns, SolveOutcome());
    for (int i = 0; i < ns; ++i) {
        const DCState &d = h_dc[i];
        out[i].iters = d.total_iter;
        out[i].info = d.info;
        out[i].error = d.error;
        out[i].work = h_st[i].work;
        out[i].valid = true;
        KState k;
        std::memset(&k, 0, sizeof k);
        k.iter = d.total_iter;
        k.info = d.info;
        k.done = 1;
        h_out_.p[i] = k;
    }
    NS3D_CUDA_CHECK(cudaMemcpyAsync(out_st_.p, h_out_.p, ns * sizeof(KState), cudaMemcpyHostToDevice, st));
}

template <int CAP>
MixedSetT<CAP>::~MixedSetT() {
    for (cudaEvent_t e : ev_)
        if (e) cudaEventDestroy(e);
}

template class MixedSetT<KMAX>;
template class MixedSetT<KMAX_MERGED_M>;

}  // namespace ns3d

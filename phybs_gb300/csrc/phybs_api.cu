// Host side of the C ABI (include/phybs.h): mesh packing, device memory,
// the graph-captured pass loop and parity/debug entry points.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <numeric>
#include <vector>

#include "../../include/phybs.h"
#include "phybs_internal.cuh"

using namespace pbs;

namespace {

constexpr int CHUNK_PASSES = 16;  // passes per body of the step graph
constexpr int CG_SOLVES = 64;     // solves of a step between two reads of their states

// TEST_FAIL_ALLOC: the allocation of this thread that is to fail, from 1 (0: none)
thread_local int test_fail_alloc = 0;

// Device memory of n elements; p is null and n 0 without it, so that a call
// whose allocation failed finds nothing to use and allocates again.
template <typename T> struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaError_t alloc(size_t count) {
        release();
        cudaError_t e = cudaErrorMemoryAllocation;
        if (test_fail_alloc == 0 || --test_fail_alloc != 0)
            e = cudaMalloc((void **)&p, std::max<size_t>(count, 1) * sizeof(T));
        if (e != cudaSuccess) {
            (void)cudaGetLastError();  // (the next launch's check is not to find it)
            p = nullptr;
            return e;
        }
        n = count;
        return cudaSuccess;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

int round_up(int x, int a) { return (x + a - 1) / a * a; }

// Default steps now running on a device whose frame kernel takes more than half
// of its SMs, over all handles and threads of the process.  Such kernels run
// one after the other, while the pass kernels of several handles overlap.  From
// the third on a step therefore runs the pass kernels, which give the same
// bits.  Steps of 1 / 2 / 4 / 8 threads, one handle each, us a step of all:
//   24,000 tets    frame 536 / 464 / 466 / 464   pass kernels 1097 / 623 / 340 / 248
//   60,000         653 / 574 / 574 / 572         1207 / 722 / 391 / 290
//   125,000        889 / 800 / 798 / 804         1406 / 861 / 506 / 458
// Smaller ones share the device as frame kernels too (16,000 tets 518 / 275 /
// 231 / 232, pass kernels 1087 / 590 / 325 / 228; 8,000 at eight threads 121 and
// 204).
std::atomic<int> large_steps[64];

// The same for backward-Euler and projective-dynamics steps whose solve has a
// CTA on more than half of the SMs: from the third on the solves take a part of
// a SM each, so that two or three of them run side by side, with the same bits.
std::atomic<int> large_solves[64];

class LargeCount {
  public:
    // Counts this call in; the others that run.
    int enter(std::atomic<int> *counts, int device) {
        count_ = &counts[device & 63];
        return count_->fetch_add(1);
    }
    ~LargeCount() {
        if (count_) count_->fetch_sub(1);
    }

  private:
    std::atomic<int> *count_ = nullptr;
};

}  // namespace

struct pbs_handle {
    int device = 0;
    cudaStream_t stream = nullptr;
    int N = 0, T = 0, B = 0, Np = 0, Tp = 0, n_tblk = 0, n_nblk = 0;
    int material = PBS_MATERIAL_NEOHOOKEAN;
    float density = 1000.f, gravity = 9.8f;
    pbs_step_params params{};
    DevParams dparams{};
    std::vector<int> user2pad, h_pad2user, h_tet_user, h_node_state;
    std::vector<float> h_rest;  // user layout, for reset

    // device mesh
    DevBuf<int4> tets, tslot;
    DevBuf<float4> row0, row1, row2, info, rest4;
    DevBuf<int> inc_ptr, inc, tblk_inst, nblk_inst, pad2user, tet_user, node_state, bad, staging_ids;
    // pass layout (chunks of tets) and the host copies it is rebuilt from
    int n_chunks = 0, chunk_tets = 0, chunk_nodes = 0, chunk_slots = 0, chunk_threads = 0;
    int chunk_stage = 0;
    int node_npt = NODE_NPT_DEFAULT;
    std::vector<int4> h_tets_pad;
    std::vector<double> h_rest_pad;
    DevBuf<int4> chunk;
    DevBuf<int2> piece;
    DevBuf<int> chunk_inst, cpiece, qperm, pptr;
    uint4 *qcor = nullptr;  // in qrows, after the three row arrays
    DevBuf<int4> lmeta;
    // the pass tets' rows and corner records, one allocation (4 x 16 B a tet):
    // the L2 access-policy window of the per-tet kernel covers it
    DevBuf<float4> qrows, part, parth;
    float4 *qrow0 = nullptr, *qrow1 = nullptr, *qrow2 = nullptr;
    // L2 residency of the pass rows: persisting set-aside taken, window bytes,
    // hit ratio, and whether the launches use it (pbs_set_l2_residency)
    bool l2_setaside = false, l2_use = true;
    size_t l2_window = 0;
    float l2_hit = 0.f;
    DevBuf<double2> cpart;
    DevBuf<double> rslot;
    // device state
    DevBuf<float4> uh, ul, dd, oh, ol, u0h, u0l, th, tl, v, vold, ext, diag, hist1, hist2, bh, bl, ub, ch, cl;
    // learned warm start
    DevBuf<float> ws_theta, ws_stats;  // NPARAM; feat mean 24, feat std 24, out std 3
    bool ws_enabled = false;
    int ws_base = 0;  // 0: corrections to the plain guess, 1: to the extrapolation u0 + 2 d1 - d2
    bool guess_pending = false;  // parity 1 holds a caller guess for the next step
    int sms = 148;      // the device's: what layouts are chosen by
    int ctx_sms = 148;  // the context's: what cooperative launches may fill
    DevBuf<float> tf, hd, staging, staging2;
    int last_fp64_svd = 0;  // tets of the last pbs_eval_tets whose stretch stress took the FP64 SVD
    // boundary surface for picking and drag forces: faces and rings in padded
    // node ids on the device, rings in caller ids on the host
    int n_faces = 0;
    std::vector<int> h_ring_ptr, h_ring;
    DevBuf<int4> faces_pad;
    DevBuf<int> ring_pad, pick_id;
    DevBuf<float> pick_d2;
    DevBuf<float4> drag_ext;
    // backward-Euler and projective-dynamics steps: block-CSR pattern and the
    // solve's plan (built on first use), values, block-Jacobi inverses, CG
    // vectors and exchanged words
    bool bsr_ready = false;
    DevBuf<int> bsr_ptr, bsr_col;
    DevBuf<float> bsr_val, cg_dinv, cg_val;
    DevBuf<float4> cg_b, cg_x, cg_xp, cg_red, cg_ws;
    DevBuf<int> cg_plan;
    DevBuf<unsigned char> cg_col;
    CgPlanView cgp[2][2]{};     // of the two matrix kinds (nine values a block, one), for a SM and for a part of one
    bool solve_light = false;   // the running step's solves take a part of a SM (LargeCount)
    size_t cg_entries = 0, cg_rows_pad = 0, cg_halo = 0;
    DevBuf<CgState> cg_state;   // of the solves of a step
    DevBuf<unsigned> cg_ctl;    // [0] the last tag of the exchanged words, [1] a wait gave up
    CgState *h_cg = nullptr;    // pinned, CG_SOLVES of them, and the two control words
    int test_solve_smem = -1;        // TEST_SOLVE_SMEM
    bool test_solve_col32 = false;   // TEST_SOLVE_COL32
    bool test_refuse_frame = false;  // TEST_REFUSE_FRAME
    bool test_wait_error = false;  // TEST_WAIT_ERROR: the next solve or step finds its wait flag set
    DevBuf<double2> tpart;
    DevBuf<double> npart;
    DevBuf<float> npartf;
    DevBuf<InstCtl> ctl, ctl2;  // ctl2: the pass graph's second control-block copy
    DevBuf<unsigned int> tcount;
    int *active = nullptr;  // DevState::active, behind the control blocks: one copy brings both to the host
    // strain-based PBD (levels built on first use) and projective dynamics
    // (its matrix built per (dt_matrix, stiffness)); dyn_* are their per-step
    // positions, start positions and right-hand-side base
    std::vector<int> h_inst_tets;  // per instance: first, end padded tet
    std::vector<int> h_inst_nodes;  // per instance: first, end padded node
    bool pbd_ready = false;
    int pbd_groups = 0;
    DevBuf<int> pbd_grp, pbd_lvl, pbd_delay;
    DevBuf<int4> pbd_tet;
    DevBuf<float4> pbd_d0, pbd_d1, pbd_d2;
    DevBuf<float2> pbd_node;  // {1 / mass, gravity_y} of the PBD rest data
    // distributed-shared-memory variant: per-corner codes and per-group ranges
    int pbd_smem = 0;  // 0: positions stay in global memory
    DevBuf<int4> pbd_codes, pbd_gnode;
    bool pd_ready = false;
    float pd_dtm = 0.f, pd_k = 0.f;
    DevBuf<float> pd_val, pd_dinv, pd_cgval;
    DevBuf<float4> dyn_px, dyn_x0, dyn_s;
    // host pinned
    int *h_active = nullptr;   // 2 slots: running counts of the host loop, or the bodies the loop ran
    InstCtl *h_ctl = nullptr;
    cudaEvent_t ev_start = nullptr, ev_end = nullptr, ev_chunk[2] = {nullptr, nullptr};
    cudaGraphExec_t graph = nullptr;
    bool graph_valid = false;
    bool teams = false;       // DevMesh::teams
    bool joined = false;      // chunks of several pieces: for the pass kernels only
    bool share_sums = true;   // every instance's |g|^2 is summed by share (InstCtl::by_share)
    bool shape_auto = true;   // no caller set the chunk shape (pbs_set_chunk_shape, pbs_autotune)
    bool engine_auto = true;  // nor the pass engine (pbs_set_pass_engine)
    bool plan_valid = false;  // fplan describes the current layout, material and stress
    FramePlan fplan;
    bool graph_loop = false;  // graph is the WHILE node over the pass body (else the body alone)
    // persistent frame kernel: its exchanged words
    int engine = PBS_ENGINE_GRAPH;
    int step_engine = PBS_ENGINE_GRAPH;  // what ran the last pbs_step's passes
    DevBuf<float4> fxh, fxl, fce;
    DevBuf<uint2> fcr;
    unsigned frame_tag = 0;     // the last tag any word may hold
    bool frame_clean = false;   // false: the words are cleared before the next launch
    double last_ms = 0.0;
    pbs_stats stats{};

    DevMesh mesh() const {
        DevMesh m;
        m.Np = Np; m.Tp = Tp; m.n_inst = B; m.n_tblk = n_tblk; m.n_nblk = n_nblk;
        m.tets = tets.p; m.row0 = row0.p; m.row1 = row1.p; m.row2 = row2.p;
        m.inc_ptr = inc_ptr.p; m.inc = inc.p; m.tslot = tslot.p; m.info = info.p; m.rest = rest4.p;
        m.tblk_inst = tblk_inst.p; m.nblk_inst = nblk_inst.p;
        m.n_chunks = n_chunks; m.chunk = chunk.p; m.chunk_inst = chunk_inst.p;
        m.piece = piece.p; m.cpiece = cpiece.p;
        m.chunk_tets = chunk_tets; m.chunk_nodes = chunk_nodes; m.chunk_threads = chunk_threads;
        m.chunk_slots = chunk_slots;
        m.teams = teams;
        m.noise_tets = shape_auto ? CHUNK_NOISE_TETS : 0;
        m.chunk_stage = chunk_stage;
        m.node_npt = node_npt;
        m.qrow0 = qrow0; m.qrow1 = qrow1; m.qrow2 = qrow2; m.qcor = qcor; m.lmeta = lmeta.p;
        m.l2_base = l2_use && l2_window ? (const void *)qrows.p : nullptr;
        m.l2_bytes = l2_window;
        m.l2_hit = l2_hit;
        m.pptr = pptr.p;
        m.stream_grid = stream_grid(m, material, dparams.incremental != 0, ctx_sms);
        return m;
    }
    DevState state() const {
        DevState s;
        s.uh = uh.p; s.ul = ul.p; s.dd = dd.p; s.oh = oh.p; s.ol = ol.p; s.u0h = u0h.p; s.u0l = u0l.p;
        s.th = th.p; s.tl = tl.p; s.v = v.p; s.vold = vold.p; s.ext = ext.p; s.diag = diag.p;
        s.hist1 = hist1.p; s.hist2 = hist2.p; s.bh = bh.p; s.bl = bl.p; s.ub = ub.p; s.ch = ch.p; s.cl = cl.p;
        s.tf = tf.p; s.hd = hd.p; s.tpart = tpart.p; s.npart = npart.p; s.npartf = npartf.p; s.ctl = ctl.p; s.active = active;
        s.ctl2 = ctl2.p; s.tcount = tcount.p;
        s.cpart = cpart.p; s.part = part.p; s.parth = parth.p; s.rslot = rslot.p;
        return s;
    }
    void release() {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        DevBuf<int4> *i4[] = {&tets, &tslot};
        for (auto b : i4) b->release();
        DevBuf<float4> *f4[] = {&row0, &row1, &row2, &info, &rest4, &uh, &ul, &dd, &oh, &ol, &u0h, &u0l, &th, &tl,
                                &v, &vold, &ext, &diag, &hist1, &hist2, &bh, &bl, &ub, &ch, &cl};
        for (auto b : f4) b->release();
        DevBuf<int> *ii[] = {&inc_ptr, &inc, &tblk_inst, &nblk_inst, &pad2user, &tet_user, &node_state, &bad,
                             &staging_ids};
        for (auto b : ii) b->release();
        ws_theta.release(); ws_stats.release();
        chunk.release(); piece.release(); lmeta.release(); cpart.release(); rslot.release();
        DevBuf<int> *ci[] = {&chunk_inst, &cpiece, &qperm, &pptr};
        for (auto b : ci) b->release();
        DevBuf<float4> *cf[] = {&qrows, &part, &parth};
        for (auto b : cf) b->release();
        tf.release(); hd.release(); staging.release(); staging2.release(); tpart.release(); npart.release(); npartf.release(); ctl.release(); ctl2.release(); tcount.release();
        fxh.release(); fxl.release(); fce.release(); fcr.release();
        faces_pad.release(); ring_pad.release(); pick_id.release(); pick_d2.release(); drag_ext.release();
        bsr_ptr.release(); bsr_col.release(); bsr_val.release(); cg_dinv.release(); cg_state.release();
        cg_val.release(); cg_plan.release(); cg_col.release(); cg_ctl.release();
        pbd_grp.release(); pbd_lvl.release(); pbd_delay.release(); pbd_tet.release(); pbd_d0.release(); pbd_d1.release(); pbd_d2.release();
        pbd_node.release(); pbd_codes.release(); pbd_gnode.release();
        pd_val.release(); pd_dinv.release(); pd_cgval.release(); dyn_px.release(); dyn_x0.release(); dyn_s.release();
        pbd_ready = pd_ready = false;
        DevBuf<float4> *cv[] = {&cg_b, &cg_x, &cg_xp, &cg_red, &cg_ws};
        for (auto b : cv) b->release();
        if (h_cg) cudaFreeHost(h_cg);
        h_cg = nullptr;
        bsr_ready = false;
        if (h_active) cudaFreeHost(h_active);
        if (h_ctl) cudaFreeHost(h_ctl);
        h_active = nullptr; h_ctl = nullptr;
        cudaEvent_t evs[] = {ev_start, ev_end, ev_chunk[0], ev_chunk[1]};
        for (auto e : evs) if (e) cudaEventDestroy(e);
        if (stream) cudaStreamDestroy(stream);
        stream = nullptr;
    }
};

#define CK(x)                                                   \
    do {                                                        \
        cudaError_t e__ = (x);                                  \
        if (e__ != cudaSuccess) {                               \
            return e__ == cudaErrorMemoryAllocation ? PBS_E_OUT_OF_MEMORY : PBS_E_CUDA; \
        }                                                       \
    } while (0)

// (Re)builds the pass layout: host chunking of the padded mesh, the device
// arrays, the chunk-ordered copy of the per-tet rows (when they exist) and the
// instances' chunk ranges.  threads > 0: that chunk shape for every instance;
// threads = 0: each instance's automatic limits.  host_ctl: the control
// blocks still on the host (creation), else those on the device are updated.
static int set_pass_layout(pbs_handle *h, int threads, int ct, int cn, int stage, std::vector<InstCtl> *host_ctl) {
    std::vector<InstCtl> ctl;
    if (host_ctl) {
        ctl = *host_ctl;
    } else {
        ctl.resize(h->B);
        CK(cudaMemcpy(ctl.data(), h->ctl.p, sizeof(InstCtl) * h->B, cudaMemcpyDeviceToHost));
    }
    std::vector<ChunkLimits> limits(h->B, ChunkLimits{ct, cn});
    const bool automatic = threads == 0;
    int max_team = 0;
    for (InstCtl &c : ctl) c.team = threads;
    if (automatic) {
        ct = cn = 0;
        for (int b = 0; b < h->B; ++b) {
            const int nt = ctl[b].tet_end - ctl[b].tet_begin;
            limits[b] = auto_chunk_limits(nt, h->sms);
            ctl[b].team = auto_team(nt, h->sms);
            max_team = std::max(max_team, ctl[b].team);
            ct = std::max(ct, limits[b].tets);
            cn = std::max(cn, limits[b].nodes);
        }
    }
    const bool grouped = automatic;  // (a caller's own shape keeps a reference node a chunk)
    // The pass kernels run chunks of more than 256 tets with two tets a thread
    // (a packed batch's with 256 threads, which its smaller instances can use);
    // the frame kernel, where every chunk has its place, with up to four
    // (auto_chunk_limits has both sides).  In a batch that 256 threads run and
    // that is too large to be resident, the smaller instances' pieces are joined
    // up to the largest one's chunk: every CTA takes the shared memory of that,
    // and alone in it a piece of 128 tets kept half of its threads idle (96
    // passes, full / incremental stress, us: a body of 300,000 tets and 100 of
    // 2,000 2925 / 3312 joined, 3516 / 3889 in pieces; 120,000 and 60 of 2,000-10,000
    // 2874 / 3255 and 3329 / 3698; 90,000 and 100 of 2,000-4,000 2135 / 2418 and
    // 2541 / 2844).
    size_t est = 0;  // pieces at least
    for (int b = 0; automatic && b < h->B; ++b)
        est += (ctl[b].tet_end - ctl[b].tet_begin + limits[b].tets - 1) / limits[b].tets;
    const bool wide = ct == CHUNK_GROUP_TETS || (ct > 256 && est > 2 * (size_t)h->sms);
    int join = automatic && h->B > 1 && wide && est > 2 * (size_t)h->sms ? ct : 0;
    ChunkLayout cl;
    const std::vector<InstCtl> ctl0 = ctl;
    auto build = [&](bool pad) {
        ctl = ctl0;
        build_chunks(h->Np, h->h_tets_pad, h->h_rest_pad, ctl, limits, grouped, join, pad, cl);
        const int nodes = join ? std::max(cn, cl.max_local) : cn;
        return chunk_smem(ct, nodes, cl.max_slots, true, stage) <= (size_t)CHUNK_MAX_SMEM;
    };
    // (no room to pad slot runs, nor for the joined ones)
    if (!build(true) && !build(false) && join) {
        join = 0;
        if (!build(true)) build(false);
    }
    if (join) cn = std::max(cn, cl.max_local);
    const int nc = (int)cl.chunk.size();
    if (automatic) {
        if (ct == CHUNK_GROUP_TETS) threads = max_team == 512 && h->B == 1 ? 512 : 256;
        else threads = wide || (ct > 256 && nc > 2 * h->sms) ? 256 : 128;
        if (h->B == 1) threads = std::max(threads, max_team);
        else if (threads < max_team) threads = 256;  // (teams of 512 take two rounds)
    }
    bool share_sums = true, teams = join > 0;
    for (InstCtl &c : ctl) {
        const int nodes = c.node_end - c.node_begin, pieces = c.pblk_end - c.pblk_begin;
        c.share = node_share(nodes, pieces);
        c.by_share = c.tet_end - c.tet_begin <= CHUNK_GROUP_TETS * h->sms && pieces <= SUM_PIECES &&
                     c.share <= 32 * SUM_GROUPS;
        share_sums = share_sums && c.by_share;
        teams = teams || c.team != threads;
    }
    const size_t L = cl.lmeta.size(), T = (size_t)h->T;
    // all of the new layout's memory before the old one's is given up: a
    // handle that runs out of it keeps the layout it had
    DevBuf<int4> chunk, lmeta;
    DevBuf<int2> piece;
    DevBuf<int> chunk_inst, cpiece, qperm, pptr;
    DevBuf<double2> cpart;
    DevBuf<float4> part, parth;
    cudaError_t ea = chunk.alloc(nc);
    if (ea == cudaSuccess) ea = chunk_inst.alloc(nc);
    if (ea == cudaSuccess) ea = piece.alloc(cl.piece.size());
    if (ea == cudaSuccess) ea = cpiece.alloc(cl.cpiece.size());
    if (ea == cudaSuccess) ea = cpart.alloc(cl.piece.size());
    if (ea == cudaSuccess) ea = qperm.alloc(T);
    if (ea == cudaSuccess) ea = lmeta.alloc(L);
    if (ea == cudaSuccess) ea = pptr.alloc(h->Np + 1);
    if (ea == cudaSuccess) ea = part.alloc(L);
    if (ea == cudaSuccess) ea = parth.alloc(L);
    if (ea == cudaSuccess) {
        std::swap(h->chunk, chunk); std::swap(h->lmeta, lmeta);
        std::swap(h->chunk_inst, chunk_inst); std::swap(h->qperm, qperm); std::swap(h->pptr, pptr);
        std::swap(h->cpart, cpart); std::swap(h->piece, piece); std::swap(h->cpiece, cpiece);
        std::swap(h->part, part); std::swap(h->parth, parth);
    }
    chunk.release(); lmeta.release(); chunk_inst.release(); qperm.release(); pptr.release(); cpart.release();
    piece.release(); cpiece.release();
    part.release(); parth.release();
    CK(ea);
    h->shape_auto = automatic;
    h->graph_valid = h->plan_valid = false;
    cudaStream_t s = h->stream;
    CK(cudaMemcpyAsync(h->chunk.p, cl.chunk.data(), sizeof(int4) * nc, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->piece.p, cl.piece.data(), sizeof(int2) * cl.piece.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->cpiece.p, cl.cpiece.data(), sizeof(int) * cl.cpiece.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->chunk_inst.p, cl.chunk_inst.data(), sizeof(int) * nc, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->qperm.p, cl.qperm.data(), sizeof(int) * T, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->qcor, cl.qcor.data(), sizeof(uint4) * T, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->lmeta.p, cl.lmeta.data(), sizeof(int4) * L, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->pptr.p, cl.pptr.data(), sizeof(int) * (h->Np + 1), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(h->part.p, 0, sizeof(float4) * std::max<size_t>(L, 1), s));
    CK(cudaMemsetAsync(h->parth.p, 0, sizeof(float4) * std::max<size_t>(L, 1), s));
    h->n_chunks = nc;
    h->chunk_threads = threads;
    h->chunk_tets = ct;
    h->chunk_slots = cl.max_slots;
    h->chunk_nodes = cn;
    h->chunk_stage = stage;
    h->share_sums = share_sums;
    h->joined = join > 0;
    h->teams = teams;
    if (host_ctl) {
        *host_ctl = ctl;
    } else {
        CK(cudaMemcpyAsync(h->ctl.p, ctl.data(), sizeof(InstCtl) * h->B, cudaMemcpyHostToDevice, s));
        CK(launch_pass_rows(s, h->T, h->qperm.p, h->row0.p, h->row1.p, h->row2.p, h->qrow0, h->qrow1,
                            h->qrow2));
    }
    CK(cudaStreamSynchronize(s));
    return PBS_OK;
}

int pbs::context_sms(const cudaDeviceProp &prop) {
    // (through the runtime: the library does not link the driver's)
    void *get = nullptr, *current = nullptr;
    cudaDriverEntryPointQueryResult st;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetDevResource", &get, 12040, cudaEnableDefault, &st) != cudaSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &current, 4000, cudaEnableDefault, &st) != cudaSuccess) {
        (void)cudaGetLastError();
        return prop.multiProcessorCount;
    }
    CUcontext ctx = nullptr;
    CUdevResource res = {};
    if (!get || !current || reinterpret_cast<decltype(&cuCtxGetCurrent)>(current)(&ctx) != CUDA_SUCCESS || !ctx ||
        reinterpret_cast<decltype(&cuCtxGetDevResource)>(get)(ctx, &res, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS ||
        res.sm.smCount == 0)
        return prop.multiProcessorCount;
    return std::min((int)res.sm.smCount, prop.multiProcessorCount);
}

static void to_dev_params(const pbs_step_params &p, DevParams &d) {
    d.h = p.h;
    d.h2inv = 1.0f / (p.h * p.h);
    d.max_iters = p.max_iters;
    d.tol = p.tol;
    d.control = p.control;
    d.alpha0 = p.alpha0; d.alpha_min = p.alpha_min; d.alpha_shrink = p.alpha_shrink;
    d.ls_every = p.line_search_every; d.hd_every = p.hessian_every;
    d.n_profile = p.n_profile;
    for (int i = 0; i < 4; ++i) { d.profile_k[i] = p.profile_k[i]; d.profile_rho[i] = p.profile_rho[i]; }
    d.damping = p.damping; d.warm_start = p.warm_start; d.body_scale = p.body_force_scale;
    d.clamp_cpu = p.energy_clamp == PBS_CLAMP_CPU ? 1 : 0;
    d.pass_cap = p.pass_cap > 0 ? p.pass_cap : p.max_iters + 16;
    d.energy_slack = p.energy_slack;
    d.alpha_grow = p.alpha_grow;
    d.incremental = 0;  // set from the material and incremental_stress by the handle
}

extern "C" {

void pbs_default_params(pbs_step_params *p) {
    if (!p) return;
    std::memset(p, 0, sizeof(*p));
    p->h = 0.03f;
    p->max_iters = 96;
    p->tol = 0.0f;
    p->control = PBS_CONTROL_REFERENCE;
    p->alpha0 = 0.1f; p->alpha_min = 0.01f; p->alpha_shrink = 0.7f;
    p->line_search_every = 8;
    p->hessian_every = 32;
    p->n_profile = 3;
    p->profile_k[0] = 1; p->profile_k[1] = 7; p->profile_k[2] = 10;
    p->profile_rho[0] = 0.96f; p->profile_rho[1] = 0.991f; p->profile_rho[2] = 0.999f;
    p->damping = 0.99f;
    p->warm_start = 0.2f;
    p->body_force_scale = 2.0f;
    p->energy_clamp = PBS_CLAMP_CPU;
    p->pass_cap = 0;
    p->energy_slack = 0.0f;
    p->alpha_grow = 1.0f;
    p->incremental_stress = 1;
}

const char *pbs_error_string(int code) {
    switch (code) {
        case PBS_OK: return "ok";
        case PBS_E_INVALID_ARG: return "invalid argument";
        case PBS_E_CUDA: return "CUDA error";
        case PBS_E_NONFINITE: return "non-finite energy or residual";
        case PBS_E_ITER_CAP: return "pass cap reached";
        case PBS_E_BAD_MESH: return "bad mesh (index out of range, or non-positive rest volume)";
        case PBS_E_NO_DEVICE: return "no compute capability 10.3 CUDA device";
        case PBS_E_OUT_OF_MEMORY: return "out of device memory";
        case PBS_E_CAPACITY: return "size beyond the fixed maximum";
        case PBS_E_DEVICE_TIMEOUT: return "a kernel's bounded wait (its own copies, another CTA's words) ran out";
        default: return "unknown error";
    }
}

void pbs_lame(float young, float poisson, int reference_formula, float *mu, float *lambda) {
    float m = 0.5f * young / (1.0f + poisson);
    float l = m * 2.0f / (1.0f - 2.0f * poisson);
    if (!reference_formula) l *= poisson;
    if (mu) *mu = m;
    if (lambda) *lambda = l;
}

static int validate_params(const pbs_step_params *p) {
    if (!p) return PBS_E_INVALID_ARG;
    if (!(p->h > 0.f) || p->max_iters < 0 || p->line_search_every <= 0 || p->hessian_every <= 0 ||
        p->n_profile < 0 || p->n_profile > 4 || !(p->alpha0 > 0.f) || !(p->alpha_shrink > 0.f) ||
        p->alpha_shrink >= 1.f || (p->control != PBS_CONTROL_REFERENCE && p->control != PBS_CONTROL_RESTART) ||
        p->tol < 0.f || p->pass_cap < 0 || !(p->energy_slack >= 0.f) ||
        (p->incremental_stress != 0 && p->incremental_stress != 1) || !(p->alpha_grow >= 1.0f) ||
        !std::isfinite(p->alpha_grow))
        return PBS_E_INVALID_ARG;
    return PBS_OK;
}

// L2 residency of the pass rows (the per-tet kernels' 64 B a tet, read every
// pass): without it they stream from HBM on every pass although the step's
// working set is near L2's size.  Takes the persisting-L2 set-aside of this
// process's context (at most the rows' size, at most what the device allows)
// and sizes the window and its hit ratio to it; the limit belongs to the
// context, and pbs_destroy gives it back.  Devices without persisting L2 run
// without a window.
static void setup_l2_residency(pbs_handle *h, const cudaDeviceProp &prop) {
    const size_t bytes = h->qrows.n * sizeof(float4);
    if (prop.persistingL2CacheMaxSize <= 0 || prop.accessPolicyMaxWindowSize <= 0 || bytes == 0) return;
    const size_t aside = std::min<size_t>((size_t)prop.persistingL2CacheMaxSize, bytes);
    if (cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, aside) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    h->l2_setaside = true;
    h->l2_window = std::min<size_t>(bytes, (size_t)prop.accessPolicyMaxWindowSize);
    h->l2_hit = (float)std::min(1.0, (double)aside / (double)h->l2_window);
}

// Every tet's corners are four different nodes of its own instance.  Checked
// before anything is built from them: the pass layout sorts a chunk's nodes by
// their corner count, which a tet that repeats a node could raise past the
// chunk's tets.
static int check_tets(const int *tets, const std::vector<int> &nptr, const std::vector<int> &tptr) {
    for (size_t b = 0; b + 1 < nptr.size(); ++b)
        for (int t = tptr[b]; t < tptr[b + 1]; ++t) {
            const int *q = tets + 4 * (size_t)t;
            for (int c = 0; c < 4; ++c) {
                if (q[c] < nptr[b] || q[c] >= nptr[b + 1]) return PBS_E_BAD_MESH;
                for (int e = 0; e < c; ++e)
                    if (q[c] == q[e]) return PBS_E_BAD_MESH;
            }
        }
    return PBS_OK;
}

int pbs_create(const pbs_mesh_desc *d, pbs_handle **out) {
    if (!d || !out || d->n_nodes <= 0 || d->n_tets <= 0 || !d->rest || !d->tets || d->n_instances < 1 ||
        !(d->density > 0.f))
        return PBS_E_INVALID_ARG;
    if (d->n_instances > 1 && (!d->instance_node_ptr || !d->instance_tet_ptr)) return PBS_E_INVALID_ARG;
    *out = nullptr;
    const int N = d->n_nodes, T = d->n_tets, B = d->n_instances;
    std::vector<int> nptr(B + 1), tptr(B + 1);
    if (B == 1) { nptr = {0, N}; tptr = {0, T}; }
    else {
        std::memcpy(nptr.data(), d->instance_node_ptr, sizeof(int) * (B + 1));
        std::memcpy(tptr.data(), d->instance_tet_ptr, sizeof(int) * (B + 1));
    }
    if (nptr[0] != 0 || tptr[0] != 0 || nptr[B] != N || tptr[B] != T) return PBS_E_INVALID_ARG;
    for (int b = 0; b < B; ++b)
        if (nptr[b + 1] < nptr[b] || tptr[b + 1] < tptr[b]) return PBS_E_INVALID_ARG;
    int rc = check_tets(d->tets, nptr, tptr);
    if (rc != PBS_OK) return rc;

    int dev = 0, ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return PBS_E_NO_DEVICE;
    if (cudaGetDevice(&dev) != cudaSuccess) return PBS_E_NO_DEVICE;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return PBS_E_NO_DEVICE;
    if (prop.major != 10 || prop.minor != 3) return PBS_E_NO_DEVICE;

    pbs_handle *h = new (std::nothrow) pbs_handle();
    if (!h) return PBS_E_OUT_OF_MEMORY;
    h->device = dev;
    h->sms = prop.multiProcessorCount;
    h->ctx_sms = context_sms(prop);
    h->N = N; h->T = T; h->B = B;
    h->density = d->density; h->gravity = d->gravity;
    pbs_default_params(&h->params);
    to_dev_params(h->params, h->dparams);

    // ---- packing: each instance starts on a PAD boundary
    std::vector<InstCtl> ctl(B);
    int pn = 0, pt = 0;
    h->user2pad.assign(N, -1);
    std::vector<int> node_off(B), tet_off(B);
    for (int b = 0; b < B; ++b) {
        node_off[b] = pn; tet_off[b] = pt;
        int nn = nptr[b + 1] - nptr[b], nt = tptr[b + 1] - tptr[b];
        std::memset(&ctl[b], 0, sizeof(InstCtl));
        ctl[b].node_begin = pn; ctl[b].node_end = pn + nn;
        ctl[b].tet_begin = pt; ctl[b].tet_end = pt + nt;
        ctl[b].nblk_begin = pn / BLOCK; ctl[b].tblk_begin = pt / BLOCK;
        pn += round_up(std::max(nn, 1), PAD);
        pt += round_up(std::max(nt, 1), PAD);
        ctl[b].nblk_end = pn / BLOCK; ctl[b].tblk_end = pt / BLOCK;
        ctl[b].rho = 0.f; ctl[b].omega = 1.f; ctl[b].alpha = h->params.alpha0;
        for (int i = nptr[b]; i < nptr[b + 1]; ++i) h->user2pad[i] = node_off[b] + (i - nptr[b]);
        h->h_inst_tets.push_back(ctl[b].tet_begin);
        h->h_inst_tets.push_back(ctl[b].tet_end);
        h->h_inst_nodes.push_back(ctl[b].node_begin);
        h->h_inst_nodes.push_back(ctl[b].node_end);
    }
    const int Np = pn, Tp = pt;
    for (int b = 0; b < B; ++b) {  // mean edge length: cbrt(6 * mean |vol|)
        double vs = 0.0;
        for (int t = tptr[b]; t < tptr[b + 1]; ++t) {
            const int *q = d->tets + 4 * (size_t)t;
            double e[3][3];
            for (int c = 0; c < 3; ++c)
                for (int k = 0; k < 3; ++k) {
                    const int a = q[c + 1], o = q[0];
                    e[c][k] = (double)d->rest[3 * (size_t)a + k] - d->rest[3 * (size_t)o + k];
                }
            vs += std::fabs(e[0][0] * (e[1][1] * e[2][2] - e[1][2] * e[2][1]) - e[0][1] * (e[1][0] * e[2][2] - e[1][2] * e[2][0]) +
                            e[0][2] * (e[1][0] * e[2][1] - e[1][1] * e[2][0])) / 6.0;
        }
        const int nt = tptr[b + 1] - tptr[b];
        ctl[b].ell = nt > 0 ? (float)std::cbrt(6.0 * vs / nt) : 1.0f;
    }
    h->Np = Np; h->Tp = Tp; h->n_tblk = Tp / BLOCK; h->n_nblk = Np / BLOCK;
    h->h_pad2user.assign(Np, -1);
    for (int i = 0; i < N; ++i) h->h_pad2user[h->user2pad[i]] = i;
    h->h_tet_user.assign(Tp, -1);
    std::vector<int4> tets_pad(Tp, make_int4(-1, -1, -1, -1));
    std::vector<int> tblk(h->n_tblk), nblk(h->n_nblk);
    for (int b = 0; b < B; ++b) {
        for (int j = ctl[b].tblk_begin; j < ctl[b].tblk_end; ++j) tblk[j] = b;
        for (int j = ctl[b].nblk_begin; j < ctl[b].nblk_end; ++j) nblk[j] = b;
        for (int t = tptr[b]; t < tptr[b + 1]; ++t) {
            int tp = tet_off[b] + (t - tptr[b]);
            h->h_tet_user[tp] = t;
            int id[4];
            for (int c = 0; c < 4; ++c) id[c] = h->user2pad[d->tets[4 * (size_t)t + c]];
            tets_pad[tp] = make_int4(id[0], id[1], id[2], id[3]);
        }
    }
    // ---- canonical node -> (tet, corner) gather (ascending tet, then corner)
    std::vector<int> iptr(Np + 1, 0), ient(4 * (size_t)T);
    for (int tp = 0; tp < Tp; ++tp) {
        if (tets_pad[tp].x < 0) continue;
        const int *q = &tets_pad[tp].x;
        for (int c = 0; c < 4; ++c) iptr[q[c] + 1]++;
    }
    for (int i = 0; i < Np; ++i) iptr[i + 1] += iptr[i];
    {
        std::vector<int> fill(iptr.begin(), iptr.end() - 1);
        for (int tp = 0; tp < Tp; ++tp) {
            if (tets_pad[tp].x < 0) continue;
            const int *q = &tets_pad[tp].x;
            for (int c = 0; c < 4; ++c) ient[fill[q[c]]++] = 4 * tp + c;
        }
    }
    std::vector<int4> tslot(Tp, make_int4(-1, -1, -1, -1));
    for (size_t j = 0; j < ient.size(); ++j) (&tslot[ient[j] >> 2].x)[ient[j] & 3] = (int)j;
    h->h_node_state.assign(Np, 2);
    for (int i = 0; i < N; ++i) h->h_node_state[h->user2pad[i]] = (d->pin_mask && d->pin_mask[i] > 0) ? 1 : 0;
    std::vector<double> rest_pad(3 * (size_t)Np, 0.0);
    std::vector<float4> rest4(Np, make_float4(0.f, 0.f, 0.f, 0.f));
    const float *p0 = d->positions ? d->positions : d->rest;
    for (int i = 0; i < N; ++i) {
        int ip = h->user2pad[i];
        for (int k = 0; k < 3; ++k) {
            float r = d->rest[3 * (size_t)i + k];
            if (!std::isfinite(r) || !std::isfinite(p0[3 * (size_t)i + k])) { delete h; return PBS_E_INVALID_ARG; }
            rest_pad[3 * (size_t)ip + k] = r;
        }
        rest4[ip] = make_float4(d->rest[3 * (size_t)i], d->rest[3 * (size_t)i + 1], d->rest[3 * (size_t)i + 2], 0.f);
    }
    h->h_rest.assign(d->rest, d->rest + 3 * (size_t)N);
    h->h_tets_pad = tets_pad;
    h->h_rest_pad = rest_pad;

    auto fail = [&](int code) { h->release(); delete h; return code; };
#define CKC(x) do { cudaError_t e__ = (x); if (e__ != cudaSuccess) return fail(e__ == cudaErrorMemoryAllocation ? PBS_E_OUT_OF_MEMORY : PBS_E_CUDA); } while (0)
    CKC(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    CKC(cudaEventCreate(&h->ev_start));
    CKC(cudaEventCreate(&h->ev_end));
    CKC(cudaEventCreateWithFlags(&h->ev_chunk[0], cudaEventDisableTiming));
    CKC(cudaEventCreateWithFlags(&h->ev_chunk[1], cudaEventDisableTiming));
    CKC(cudaMallocHost((void **)&h->h_active, 2 * sizeof(int)));
    CKC(cudaMallocHost((void **)&h->h_ctl, (B + 1) * sizeof(InstCtl)));
    std::memset(h->h_ctl, 0, (B + 1) * sizeof(InstCtl));
    CKC(h->tets.alloc(Tp)); CKC(h->tslot.alloc(Tp)); CKC(h->row0.alloc(Tp)); CKC(h->row1.alloc(Tp)); CKC(h->row2.alloc(Tp));
    CKC(h->info.alloc(Np)); CKC(h->inc_ptr.alloc(Np + 1)); CKC(h->inc.alloc(4 * (size_t)T));
    CKC(h->tblk_inst.alloc(h->n_tblk)); CKC(h->nblk_inst.alloc(h->n_nblk));
    CKC(h->pad2user.alloc(Np)); CKC(h->tet_user.alloc(Tp)); CKC(h->node_state.alloc(Np)); CKC(h->bad.alloc(1));
    CKC(h->uh.alloc(2 * (size_t)Np)); CKC(h->ul.alloc(2 * (size_t)Np)); CKC(h->dd.alloc(2 * (size_t)Np));
    CKC(h->oh.alloc(Np)); CKC(h->ol.alloc(Np)); CKC(h->u0h.alloc(Np)); CKC(h->u0l.alloc(Np));
    CKC(h->th.alloc(Np)); CKC(h->tl.alloc(Np)); CKC(h->v.alloc(Np)); CKC(h->vold.alloc(Np));
    CKC(h->ext.alloc(Np)); CKC(h->diag.alloc(Np)); CKC(h->rest4.alloc(Np));
    CKC(h->hist1.alloc(Np)); CKC(h->hist2.alloc(Np)); CKC(h->bh.alloc(Np)); CKC(h->bl.alloc(Np));
    CKC(h->ch.alloc(Np)); CKC(h->cl.alloc(Np));
    CKC(h->ub.alloc(Np));
    // slot-ordered hot-loop buffers (3 * 4T) also serve the per-tet probes (12 * Tp)
    CKC(h->tf.alloc(std::max(12 * (size_t)Tp, 16 * (size_t)T))); CKC(h->hd.alloc(std::max(12 * (size_t)Tp, 16 * (size_t)T)));
    CKC(h->staging.alloc(3 * (size_t)N)); CKC(h->staging2.alloc(12 * (size_t)Tp)); CKC(h->staging_ids.alloc(N));
    CKC(h->tpart.alloc(h->n_tblk)); CKC(h->npart.alloc(h->n_nblk)); CKC(h->npartf.alloc(8 * (size_t)h->n_nblk));
    CKC(h->ctl.alloc(B + 1)); CKC(h->ctl2.alloc(B)); CKC(h->tcount.alloc(B));
    h->active = reinterpret_cast<int *>(h->ctl.p + B);
    CKC(cudaMemsetAsync(h->ctl2.p, 0, sizeof(InstCtl) * B, h->stream));
    CKC(cudaMemsetAsync(h->tcount.p, 0, sizeof(unsigned int) * B, h->stream));
    CKC(cudaMemsetAsync(h->active, 0, 4 * sizeof(int), h->stream));
    CKC(h->qrows.alloc(4 * (size_t)T)); CKC(h->rslot.alloc(12 * (size_t)T));
    h->qrow0 = h->qrows.p;
    h->qrow1 = h->qrows.p + (size_t)T;
    h->qrow2 = h->qrows.p + 2 * (size_t)T;
    h->qcor = reinterpret_cast<uint4 *>(h->qrows.p + 3 * (size_t)T);
    setup_l2_residency(h, prop);
    CKC(prepare_chunk_kernels());
    cudaStream_t s = h->stream;
    rc = set_pass_layout(h, 0, 0, 0, 0, &ctl);
    if (rc != PBS_OK) return fail(rc);
    CKC(cudaMemcpyAsync(h->tets.p, tets_pad.data(), sizeof(int4) * Tp, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->tslot.p, tslot.data(), sizeof(int4) * Tp, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->inc_ptr.p, iptr.data(), sizeof(int) * (Np + 1), cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->inc.p, ient.data(), sizeof(int) * 4 * (size_t)T, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->tblk_inst.p, tblk.data(), sizeof(int) * h->n_tblk, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->nblk_inst.p, nblk.data(), sizeof(int) * h->n_nblk, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->pad2user.p, h->h_pad2user.data(), sizeof(int) * Np, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->tet_user.p, h->h_tet_user.data(), sizeof(int) * Tp, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->node_state.p, h->h_node_state.data(), sizeof(int) * Np, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->ctl.p, ctl.data(), sizeof(InstCtl) * B, cudaMemcpyHostToDevice, s));
    CKC(cudaMemcpyAsync(h->rest4.p, rest4.data(), sizeof(float4) * Np, cudaMemcpyHostToDevice, s));
    CKC(cudaMemsetAsync(h->v.p, 0, sizeof(float4) * Np, s));
    CKC(cudaMemsetAsync(h->vold.p, 0, sizeof(float4) * Np, s));
    CKC(cudaMemsetAsync(h->diag.p, 0, sizeof(float4) * Np, s));
    CKC(cudaMemsetAsync(h->ext.p, 0, sizeof(float4) * Np, s));
    CKC(cudaMemsetAsync(h->tf.p, 0, sizeof(float) * std::max(12 * (size_t)Tp, 16 * (size_t)T), s));
    CKC(cudaMemsetAsync(h->hd.p, 0, sizeof(float) * std::max(12 * (size_t)Tp, 16 * (size_t)T), s));
    {
        DevBuf<float4> *zero[] = {&h->uh, &h->ul, &h->dd};
        for (auto b : zero) CKC(cudaMemsetAsync(b->p, 0, sizeof(float4) * 2 * (size_t)Np, s));
        DevBuf<float4> *zero1[] = {&h->oh, &h->ol, &h->u0h, &h->u0l, &h->th, &h->tl, &h->hist1, &h->hist2, &h->bh,
                                   &h->bl, &h->ub};
        for (auto b : zero1) CKC(cudaMemsetAsync(b->p, 0, sizeof(float4) * (size_t)Np, s));
    }
    CKC(cudaMemsetAsync(h->bad.p, 0, sizeof(int), s));
    {
        // FP64 rest state on the device
        DevBuf<double> rest_d, tmass;
        CKC(rest_d.alloc(3 * (size_t)Np));
        if (tmass.alloc(Tp) != cudaSuccess) { rest_d.release(); return fail(PBS_E_OUT_OF_MEMORY); }
        cudaError_t e = cudaMemcpyAsync(rest_d.p, rest_pad.data(), sizeof(double) * 3 * (size_t)Np, cudaMemcpyHostToDevice, s);
        DevMesh m = h->mesh();
        if (e == cudaSuccess) e = launch_rest(s, m, rest_d.p, h->density, h->row0.p, h->row1.p, h->row2.p, tmass.p, h->bad.p);
        if (e == cudaSuccess) e = launch_mass(s, m, tmass.p, h->node_state.p, h->gravity, h->info.p);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        rest_d.release();
        tmass.release();
        CKC(e);
    }
    int bad = 0;
    CKC(cudaMemcpy(&bad, h->bad.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (bad) return fail(PBS_E_BAD_MESH);
    if (d->positions) {
        CKC(cudaMemcpyAsync(h->staging.p, d->positions, sizeof(float) * 3 * (size_t)N, cudaMemcpyHostToDevice, s));
        CKC(launch_unpack_positions(s, h->mesh(), h->staging.p, h->pad2user.p, h->u0h.p, h->u0l.p));
        CKC(cudaStreamSynchronize(s));
    }
    // default material: TetMesh.cpp:185 (E = 5e5, nu = 0.45), the reference's Lame formula
    float mu, lam;
    pbs_lame(5e5f, 0.45f, 1, &mu, &lam);
    rc = pbs_set_material(h, PBS_MATERIAL_NEOHOOKEAN, &mu, &lam, 1);
    if (rc != PBS_OK) return fail(rc);
    CKC(cudaStreamSynchronize(s));
    *out = h;
    return PBS_OK;
#undef CKC
}

void pbs_destroy(pbs_handle *h) {
    if (!h) return;
    DeviceScope scope(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->l2_setaside) {  // the persisting lines back to normal, the set-aside returned
        cudaCtxResetPersistingL2Cache();
        cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, 0);
    }
    h->release();
    delete h;
}

int pbs_set_l2_residency(pbs_handle *h, int enable) {
    if (!h || (enable != 0 && enable != 1)) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    if (enable && !h->l2_setaside) return PBS_E_INVALID_ARG;  // the device offers no persisting L2
    if ((enable != 0) != h->l2_use) {
        h->l2_use = enable != 0;
        h->graph_valid = h->plan_valid = false;  // the captured launches carry the window
        if (!enable) cudaCtxResetPersistingL2Cache();
    }
    return PBS_OK;
}

int pbs_set_material(pbs_handle *h, int model, const float *mu, const float *lambda, int count) {
    if (!h || !mu || !lambda || (count != 1 && count != h->T)) return PBS_E_INVALID_ARG;
    if (model != PBS_MATERIAL_NEOHOOKEAN && model != PBS_MATERIAL_STRETCH) return PBS_E_INVALID_ARG;
    for (int i = 0; i < count; ++i)
        if (!std::isfinite(mu[i]) || !std::isfinite(lambda[i])) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    // stage mu and lambda through the (3N-float) staging buffer's neighbour
    DevBuf<float> buf;
    CK(buf.alloc(2 * (size_t)count));
    cudaError_t e = cudaMemcpyAsync(buf.p, mu, sizeof(float) * count, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(buf.p + count, lambda, sizeof(float) * count, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = launch_set_lame(h->stream, h->Tp, h->tets.p, buf.p, buf.p + count, count, h->row1.p, h->row2.p, h->tet_user.p);
    if (e == cudaSuccess)  // the pass kernel's copy of the rows, in chunk order
        e = launch_pass_rows(h->stream, h->T, h->qperm.p, h->row0.p, h->row1.p, h->row2.p, h->qrow0, h->qrow1,
                             h->qrow2);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    buf.release();
    CK(e);
    if (h->material != model) h->graph_valid = h->plan_valid = false;
    h->material = model;
    h->dparams.incremental = model == PBS_MATERIAL_NEOHOOKEAN && h->params.incremental_stress ? 1 : 0;
    return PBS_OK;
}

int pbs_set_params(pbs_handle *h, const pbs_step_params *p) {
    if (!h) return PBS_E_INVALID_ARG;
    int rc = validate_params(p);
    if (rc != PBS_OK) return rc;
    h->params = *p;
    to_dev_params(h->params, h->dparams);
    h->dparams.incremental = h->material == PBS_MATERIAL_NEOHOOKEAN && h->params.incremental_stress ? 1 : 0;
    h->graph_valid = h->plan_valid = false;
    return PBS_OK;
}

int pbs_get_params(pbs_handle *h, pbs_step_params *p) {
    if (!h || !p) return PBS_E_INVALID_ARG;
    *p = h->params;
    return PBS_OK;
}

// CHUNK_PASSES passes and the closing settle, captured from h->stream.
static cudaError_t capture_body(pbs_handle *h, const LoopCtl *loop) {
    DevMesh m = h->mesh();
    DevState st = h->state();
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < CHUNK_PASSES && e == cudaSuccess; ++i)
        e = launch_pass(h->stream, m, h->dparams, st, h->material, i & 1);
    // the last pass's decision, so that the next run, the host and the
    // epilogue see settled control blocks
    if (e == cudaSuccess) e = launch_settle(h->stream, m, h->dparams, st, CHUNK_PASSES & 1, true, loop);
    return e;
}

// Bodies of CHUNK_PASSES passes a step needs at most (its pass cap).
static int max_runs(const pbs_handle *h) { return (h->dparams.pass_cap + CHUNK_PASSES - 1) / CHUNK_PASSES; }

// The step graph as a WHILE node over the body: k_settle's last CTA ends the
// loop when no instance runs or max_runs bodies ran, so a step is one graph
// launch and neither the host nor an extra body waits on the outcome.
static cudaError_t build_loop_graph(pbs_handle *h, cudaGraphExec_t *out) {
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) return e;
    LoopCtl lc{};
    lc.max_runs = max_runs(h);
    e = cudaGraphConditionalHandleCreate(&lc.cond, g, 1, cudaGraphCondAssignDefault);
    cudaGraphNodeParams np = {};
    if (e == cudaSuccess) {
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = lc.cond;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        cudaGraphNode_t node = nullptr;
        e = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &np);
    }
    if (e == cudaSuccess)
        e = cudaStreamBeginCaptureToGraph(h->stream, np.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                          cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        const cudaError_t ec = capture_body(h, &lc);
        cudaGraph_t body = nullptr;
        e = cudaStreamEndCapture(h->stream, &body);
        if (ec != cudaSuccess) e = ec;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    return e;
}

static int ensure_graph(pbs_handle *h) {
    if (h->graph_valid) return PBS_OK;
    if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    h->graph_loop = build_loop_graph(h, &h->graph) == cudaSuccess;
    if (!h->graph_loop) {
        // without conditional nodes: the body alone, launched by the host
        (void)cudaGetLastError();
        h->graph = nullptr;
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
        const cudaError_t e = capture_body(h, nullptr);
        const cudaError_t e2 = cudaStreamEndCapture(h->stream, &g);
        if (e != cudaSuccess || e2 != cudaSuccess) { if (g) cudaGraphDestroy(g); return PBS_E_CUDA; }
        const cudaError_t e3 = cudaGraphInstantiate(&h->graph, g, 0);
        cudaGraphDestroy(g);
        CK(e3);
    }
    h->graph_valid = true;
    return PBS_OK;
}

// The mesh as the frame kernel takes it: automatic chunks that the pass kernels
// run with 512 threads, which it has no variant for, with 256.
static DevMesh frame_mesh(pbs_handle *h) {
    DevMesh m = h->mesh();
    if (h->shape_auto && m.chunk_threads == 512) m.chunk_threads = 256;
    return m;
}

// How the frame kernel runs the handle's current layout.
static const FramePlan &handle_frame_plan(pbs_handle *h) {
    if (!h->plan_valid) {
        h->fplan = frame_plan(frame_mesh(h), h->material,
                              h->material == PBS_MATERIAL_NEOHOOKEAN && h->dparams.incremental, h->ctx_sms);
        h->plan_valid = true;
    }
    return h->fplan;
}

// A handle whose caller chose neither an engine nor a shape, and whose chunks
// all have resident CTAs.
static bool auto_frame_applies(pbs_handle *h) {
    return h->engine_auto && h->shape_auto && h->share_sums && !h->joined && handle_frame_plan(h).resident;
}

// The frame engine as the caller selects it: one instance.
static bool frame_applies(pbs_handle *h) { return h->B == 1 && handle_frame_plan(h).grid > 0; }

// Enqueues one frame-kernel launch of at most max_passes passes with params p;
// frame_done must follow once the launch has ended.  PBS_E_INVALID_ARG when
// the frame kernel does not apply to the handle's layout.  *refused: the launch
// was refused because its CTAs cannot be resident together; nothing ran.
static int launch_frame_step(pbs_handle *h, const DevParams &p, int max_passes, bool count_void, bool *refused) {
    *refused = false;
    const FramePlan &plan = handle_frame_plan(h);
    if (plan.grid <= 0) return PBS_E_INVALID_ARG;
    cudaStream_t s = h->stream;
    // (each group is known by its last member)
    if (!h->fxl.p) {
        h->frame_clean = false;
        CK(h->fxh.alloc(h->Np));
        CK(h->fxl.alloc(h->Np));
    }
    if (h->fcr.n < 2 * (size_t)plan.grid) {
        h->frame_clean = false;
        CK(h->fce.alloc(plan.grid));
        CK(h->fcr.alloc(2 * (size_t)plan.grid));
    }
    // tags only grow, so the words of earlier launches need no clearing; they
    // are cleared after a launch whose passes are not known, and long before
    // the tags would wrap
    if (!h->frame_clean || h->frame_tag > 0x40000000u) {
        CK(cudaMemsetAsync(h->fxh.p, 0, sizeof(float4) * h->fxh.n, s));
        CK(cudaMemsetAsync(h->fxl.p, 0, sizeof(float4) * h->fxl.n, s));
        CK(cudaMemsetAsync(h->fce.p, 0, sizeof(float4) * h->fce.n, s));
        CK(cudaMemsetAsync(h->fcr.p, 0, sizeof(uint2) * h->fcr.n, s));
        CK(cudaMemsetAsync(h->part.p, 0, sizeof(float4) * h->part.n, s));
        CK(cudaMemsetAsync(h->parth.p, 0, sizeof(float4) * h->parth.n, s));
        h->frame_tag = 0;
    }
    FrameAux fx;
    fx.xh = h->fxh.p;
    fx.xl = h->fxl.p;
    fx.ce = h->fce.p;
    fx.cr = h->fcr.p;
    fx.tag0 = h->frame_tag;
    fx.max_passes = max_passes;
    fx.count_void = count_void;
    h->frame_clean = false;
    const cudaError_t e = h->test_refuse_frame ? cudaErrorCooperativeLaunchTooLarge
                                               : launch_frame(s, frame_mesh(h), p, h->state(), h->material, fx, plan);
    *refused = e == cudaErrorCooperativeLaunchTooLarge;
    if (*refused) (void)cudaGetLastError();
    CK(e);
    return PBS_OK;
}

// After a frame launch that ended with at most `passes` passes of any
// instance; gave_up: the device's flag of a wait that ran out (st.active[1]).
// Without it the tags the launch used are spent.  With it a CTA may have gone
// further than the one that reports, so the words are not clean and every
// instance's results are invalid, whatever its control block says.
static int frame_done(pbs_handle *h, int passes, int gave_up) {
    if (gave_up) return PBS_E_DEVICE_TIMEOUT;
    h->frame_tag += (unsigned)passes + 2u;
    h->frame_clean = true;
    return PBS_OK;
}

int pbs_step(pbs_handle *h, const float *ext, int *iters_out) {
    if (!h) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    bool frame = h->engine == PBS_ENGINE_FRAME;
    if (frame && !frame_applies(h)) return PBS_E_INVALID_ARG;
    // the caller chose neither an engine nor a shape: the frame kernel where
    // every chunk has a resident CTA of its own (auto_chunk_limits), which
    // spares a pass its two launches and its trips to memory
    bool auto_frame = !frame && auto_frame_applies(h);
    LargeCount large;
    if (auto_frame) {
        const FramePlan &plan = handle_frame_plan(h);
        if ((plan.per_sm > 1 || 2 * plan.grid > h->ctx_sms) && large.enter(large_steps, h->device) >= 2)
            auto_frame = false;
    }
    frame |= auto_frame;
    int rc = frame ? PBS_OK : ensure_graph(h);
    if (rc != PBS_OK) return rc;
    cudaStream_t s = h->stream;
    DevMesh m = h->mesh();
    DevState st = h->state();
    CK(cudaEventRecord(h->ev_start, s));
    if (ext) CK(cudaMemcpyAsync(h->staging.p, ext, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(h->active, 0, 4 * sizeof(int), s));
    if (h->test_wait_error) {
        h->test_wait_error = false;
        CK(cudaMemsetAsync(h->active + 1, 1, sizeof(int), s));
    }
    CK(launch_init_ctl(s, h->B, h->dparams, st));
    CK(launch_prologue(s, m, h->dparams, st, ext ? h->staging.p : nullptr, h->pad2user.p));
    CK(launch_guess_check(s, m, h->dparams, st));
    CK(launch_ref_force(s, m, h->dparams, st));
    if (h->ws_enabled || h->guess_pending) {
        CK(launch_ws_gref(s, m, h->dparams, st, h->material));
        if (h->guess_pending)
            CK(launch_ws_choose(s, m, h->dparams, st));
        else
            CK(launch_ws_predict(s, m, h->dparams, st, h->ws_theta.p, h->ws_stats.p, h->ws_stats.p + 24,
                                 h->ws_stats.p + 48, h->hd.p, h->sms, h->ws_base, h->material));
        h->guess_pending = false;
    }
    CK(launch_to_increment(s, m, h->dparams, st));
    // The graph's WHILE node runs bodies of CHUNK_PASSES passes until no
    // instance runs; without it the host launches the body and reads the
    // active-instance count of body j-1 while body j runs, so the device never
    // idles on the poll (body j may then find every instance done).  The frame
    // engine: one launch runs every pass of the step (its pass cap ends it at
    // the latest).
    if (frame) {
        bool refused = false;
        rc = launch_frame_step(h, h->dparams, h->dparams.pass_cap, auto_frame, &refused);
        if (refused && auto_frame) {  // this step's own choice: the pass kernels run it as well
            frame = auto_frame = false;
            rc = ensure_graph(h);
        }
        if (rc != PBS_OK) return rc;
    }
    const int max_chunks = frame || h->graph_loop ? 0 : max_runs(h);
    int launched = 0;
    if (frame) {
        // (enqueued)
    } else if (h->graph_loop) {
        CK(cudaGraphLaunch(h->graph, s));
        CK(cudaMemcpyAsync(h->h_active, h->active + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    }
    for (int j = 0; j < max_chunks; ++j) {
        ++launched;
        CK(cudaGraphLaunch(h->graph, s));
        CK(cudaMemcpyAsync(h->h_active + (j & 1), h->active, sizeof(int), cudaMemcpyDeviceToHost, s));
        CK(cudaEventRecord(h->ev_chunk[j & 1], s));
        if (j >= 1) {
            CK(cudaEventSynchronize(h->ev_chunk[(j - 1) & 1]));
            if (h->h_active[(j - 1) & 1] == 0) break;
        }
    }
    CK(launch_from_increment(s, m, h->dparams, st));
    CK(launch_epilogue(s, m, h->dparams, st, h->pad2user.p));
    CK(cudaMemcpyAsync(h->h_ctl, h->ctl.p, sizeof(InstCtl) * h->B + 4 * sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaEventRecord(h->ev_end, s));
    CK(cudaMemsetAsync(h->ext.p, 0, sizeof(float4) * h->Np, s));  // fvm.cpp:188 resetExternalForce
    CK(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, h->ev_start, h->ev_end);
    h->last_ms = ms;
    if (!frame && h->graph_loop) launched = h->h_active[0];
    const bool gave_up = frame && reinterpret_cast<const int *>(h->h_ctl + h->B)[1] != 0;
    pbs_stats S{};
    S.status = PBS_OK;
    for (int b = 0; b < h->B; ++b) {
        InstCtl &c = h->h_ctl[b];
        if (gave_up) c.status = PBS_E_DEVICE_TIMEOUT;
        S.passes = std::max(S.passes, c.passes);
        S.iterations = std::max(S.iterations, c.k);
        S.rejections += c.rejections;
        S.converged += c.converged;
        S.warm_start_used += c.ws_used;
        S.guess_fallbacks += c.guess_bad;
        if (c.status != PBS_OK && S.status == PBS_OK) S.status = c.status;
        if (c.status == PBS_E_NONFINITE) S.status = PBS_E_NONFINITE;
    }
    S.alpha = h->h_ctl[0].alpha;
    S.rho = h->h_ctl[0].rho;
    S.omega = h->h_ctl[0].omega;
    S.energy = h->h_ctl[0].energy;
    S.residual_ratio = residual_ratio(h->h_ctl[0]);
    S.device_ms = ms;
    // the default engine counts in bodies whichever kernel ran its passes
    S.graph_launches = auto_frame ? std::max(1, (S.passes + CHUNK_PASSES - 1) / CHUNK_PASSES) : launched;
    h->stats = S;
    h->step_engine = frame ? PBS_ENGINE_FRAME : PBS_ENGINE_GRAPH;
    if (frame) frame_done(h, S.passes, gave_up);
    if (iters_out) *iters_out = S.iterations;
    return S.status;
}

int pbs_read_positions(pbs_handle *h, float *out) {
    if (!h || !out) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    CK(launch_pack_positions(h->stream, h->mesh(), h->u0h.p, h->u0l.p, h->pad2user.p, h->staging.p));
    CK(cudaMemcpyAsync(out, h->staging.p, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return PBS_OK;
}

static int upload_user(pbs_handle *h, const float *src, float4 *dst) {
    for (size_t i = 0; i < 3 * (size_t)h->N; ++i)
        if (!std::isfinite(src[i])) return PBS_E_INVALID_ARG;
    CK(cudaMemcpyAsync(h->staging.p, src, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyHostToDevice, h->stream));
    CK(launch_unpack(h->stream, h->Np, h->staging.p, h->pad2user.p, dst));
    CK(cudaStreamSynchronize(h->stream));
    return PBS_OK;
}

static int download_user(pbs_handle *h, const float4 *src, float *dst) {
    CK(launch_pack(h->stream, h->Np, src, h->pad2user.p, h->staging.p));
    CK(cudaMemcpyAsync(dst, h->staging.p, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return PBS_OK;
}

static int upload_positions(pbs_handle *h, const float *positions, float4 *hi, float4 *lo) {
    for (size_t i = 0; i < 3 * (size_t)h->N; ++i)
        if (!std::isfinite(positions[i])) return PBS_E_INVALID_ARG;
    CK(cudaMemcpyAsync(h->staging.p, positions, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyHostToDevice, h->stream));
    CK(launch_unpack_positions(h->stream, h->mesh(), h->staging.p, h->pad2user.p, hi, lo));
    CK(cudaStreamSynchronize(h->stream));
    return PBS_OK;
}

int pbs_update_positions(pbs_handle *h, const float *positions) {
    if (!h || !positions) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    return upload_positions(h, positions, h->u0h.p, h->u0l.p);
}

int pbs_set_node_positions(pbs_handle *h, int count, const int *ids, const float *xyz) {
    if (!h || count < 0 || count > h->N || (count > 0 && (!ids || !xyz))) return PBS_E_INVALID_ARG;
    if (count == 0) return PBS_OK;
    PBS_DEVICE_SCOPE(h->device);
    std::vector<int> pad(count);
    for (int i = 0; i < count; ++i) {
        if (ids[i] < 0 || ids[i] >= h->N) return PBS_E_INVALID_ARG;
        for (int k = 0; k < 3; ++k)
            if (!std::isfinite(xyz[3 * (size_t)i + k])) return PBS_E_INVALID_ARG;
        pad[i] = h->user2pad[ids[i]];
    }
    CK(cudaMemcpyAsync(h->staging_ids.p, pad.data(), sizeof(int) * count, cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(h->staging.p, xyz, sizeof(float) * 3 * (size_t)count, cudaMemcpyHostToDevice, h->stream));
    CK(launch_scatter_positions(h->stream, h->mesh(), count, h->staging_ids.p, h->staging.p, h->u0h.p, h->u0l.p));
    CK(cudaStreamSynchronize(h->stream));
    return PBS_OK;
}

int pbs_set_warm_start(pbs_handle *h, const float *theta, const float *feat_mean, const float *feat_std,
                       const float *out_std, int enabled) {
    if (!h) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    if (!enabled) {
        h->ws_enabled = false;
        return PBS_OK;
    }
    if (enabled != 1 && enabled != 2) return PBS_E_INVALID_ARG;
    const int np = pbs_mlp_param_count();
    if (!theta || !feat_mean || !feat_std || !out_std) return PBS_E_INVALID_ARG;
    for (int i = 0; i < np; ++i)
        if (!std::isfinite(theta[i])) return PBS_E_INVALID_ARG;
    for (int i = 0; i < 24; ++i)
        if (!std::isfinite(feat_mean[i]) || !(feat_std[i] > 0.f)) return PBS_E_INVALID_ARG;
    for (int i = 0; i < 3; ++i)
        if (!(out_std[i] > 0.f)) return PBS_E_INVALID_ARG;
    if (!h->ws_theta.p) CK(h->ws_theta.alloc(np));
    if (!h->ws_stats.p) CK(h->ws_stats.alloc(51));
    std::vector<float> st(51);
    std::memcpy(st.data(), feat_mean, 24 * sizeof(float));
    std::memcpy(st.data() + 24, feat_std, 24 * sizeof(float));
    std::memcpy(st.data() + 48, out_std, 3 * sizeof(float));
    CK(cudaMemcpy(h->ws_theta.p, theta, sizeof(float) * np, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->ws_stats.p, st.data(), sizeof(float) * 51, cudaMemcpyHostToDevice));
    h->ws_enabled = true;
    h->ws_base = enabled == 2 ? 1 : 0;
    return PBS_OK;
}

int pbs_warm_start_features(pbs_handle *h, const float *ext, float *features, float *x_init, float *scale) {
    if (!h || !features) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    cudaStream_t s = h->stream;
    DevMesh m = h->mesh();
    DevState st = h->state();
    if (ext) CK(cudaMemcpyAsync(h->staging.p, ext, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(h->active, 0, 4 * sizeof(int), s));
    CK(launch_init_ctl(s, h->B, h->dparams, st));
    CK(launch_prologue(s, m, h->dparams, st, ext ? h->staging.p : nullptr, h->pad2user.p));
    DevBuf<float> out;
    CK(out.alloc(25 * (size_t)h->N));
    float *sc = out.p + 24 * (size_t)h->N;
    cudaError_t e = launch_ws_features(s, m, h->dparams, st, h->hd.p, h->pad2user.p, out.p, sc);
    if (e == cudaSuccess) e = cudaMemcpyAsync(features, out.p, sizeof(float) * 24 * (size_t)h->N, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && scale) e = cudaMemcpyAsync(scale, sc, sizeof(float) * h->N, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && x_init) e = launch_pack_positions(s, m, h->uh.p, h->ul.p, h->pad2user.p, h->staging.p);
    if (e == cudaSuccess && x_init)
        e = cudaMemcpyAsync(x_init, h->staging.p, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    out.release();
    CK(e);
    return PBS_OK;
}

int pbs_set_guess(pbs_handle *h, const float *positions) {
    if (!h || !positions) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    int rc = upload_positions(h, positions, h->uh.p + h->Np, h->ul.p + h->Np);
    if (rc != PBS_OK) return rc;
    h->guess_pending = true;
    return PBS_OK;
}

// For the tests only (not in phybs.h).
int pbs_test_hook(pbs_handle *h, int what, int value) {
    if (!h) return PBS_E_INVALID_ARG;
    switch (what) {
        case TEST_WAIT_ERROR: h->test_wait_error = value != 0; return PBS_OK;
        case TEST_FAIL_ALLOC: test_fail_alloc = value; return PBS_OK;
        case TEST_SOLVE_SMEM: h->test_solve_smem = value; return PBS_OK;
        case TEST_SOLVE_COL32: h->test_solve_col32 = value != 0; return PBS_OK;
        case TEST_REFUSE_FRAME: h->test_refuse_frame = value != 0; return PBS_OK;
        case TEST_LARGE_STEPS:
            large_steps[h->device & 63] += value;
            large_solves[h->device & 63] += value;
            return PBS_OK;
        default: return PBS_E_INVALID_ARG;
    }
}

int pbs_get_stream(pbs_handle *h, void **stream) {
    if (!h || !stream) return PBS_E_INVALID_ARG;
    *stream = (void *)h->stream;
    return PBS_OK;
}

}  // extern "C"

// Times `passes` passes from the current state (CUDA events around each
// kernel on the handle's stream); the state the next step starts from (u0,
// velocities) is untouched.  Fails when an instance stopped before the last
// pass, leaving its counters in h->stats.
static int time_passes(pbs_handle *h, int passes, double *tet_ms, double *node_ms) {
    cudaStream_t s = h->stream;
    DevParams p = h->dparams;
    // a line-search rejection adds a pass and, under the reference control,
    // shortens the iteration budget (iterations -= k - 8): neither may end the
    // timed passes early
    p.max_iters = 4 * passes + 64;
    p.tol = 0.f;
    p.pass_cap = 4 * passes + 64;
    DevMesh m = h->mesh();
    DevState st = h->state();
    std::vector<cudaEvent_t> ev(2 * passes + 1, nullptr);
    for (auto &e : ev) CK(cudaEventCreate(&e));
    cudaError_t e = cudaMemsetAsync(h->active, 0, 4 * sizeof(int), s);
    if (e == cudaSuccess) e = launch_init_ctl(s, h->B, p, st);
    if (e == cudaSuccess) e = launch_prologue(s, m, p, st, nullptr, h->pad2user.p);
    if (e == cudaSuccess) e = launch_guess_check(s, m, p, st);
    if (e == cudaSuccess) e = launch_ref_force(s, m, p, st);
    if (e == cudaSuccess) e = launch_to_increment(s, m, p, st);
    if (e == cudaSuccess) e = cudaEventRecord(ev[0], s);
    for (int i = 0; i < passes && e == cudaSuccess; ++i) {
        e = launch_tet_only(s, m, p, st, h->material, i & 1);
        if (e == cudaSuccess) e = cudaEventRecord(ev[2 * i + 1], s);
        if (e == cudaSuccess) e = launch_node_only(s, m, p, st, i & 1);
        if (e == cudaSuccess) e = cudaEventRecord(ev[2 * i + 2], s);
    }
    if (e == cudaSuccess) e = launch_settle(s, m, p, st, passes & 1);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    double tt = 0.0, tn = 0.0;
    for (int i = 0; i < passes && e == cudaSuccess; ++i) {
        float a = 0.f, b = 0.f;
        cudaEventElapsedTime(&a, ev[2 * i], ev[2 * i + 1]);
        cudaEventElapsedTime(&b, ev[2 * i + 1], ev[2 * i + 2]);
        tt += a;
        tn += b;
    }
    for (auto &x : ev) cudaEventDestroy(x);
    CK(e);
    // every pass must have done real work: an instance that finished early
    // (non-finite state, line-search stop) would leave no-op launches behind
    std::vector<InstCtl> c(h->B);
    CK(cudaMemcpy(c.data(), h->ctl.p, sizeof(InstCtl) * h->B, cudaMemcpyDeviceToHost));
    for (const InstCtl &x : c) {
        if (x.tet_end == x.tet_begin) continue;
        if (x.status != PBS_OK || x.passes < passes) {  // pbs_get_stats then describes the stopped instance
            pbs_stats S{};
            S.passes = x.passes; S.iterations = x.k; S.rejections = x.rejections; S.converged = x.converged;
            S.status = x.status; S.alpha = x.alpha; S.rho = x.rho; S.omega = x.omega; S.energy = x.energy;
            S.residual_ratio = residual_ratio(x);
            h->stats = S;
            return x.status != PBS_OK ? x.status : PBS_E_ITER_CAP;
        }
    }
    *tet_ms = tt / passes;
    *node_ms = tn / passes;
    return PBS_OK;
}

// The frame engine's counterpart of time_passes: one launch of exactly
// `passes` passes from the step's start state, timed with CUDA events.
static int time_frame(pbs_handle *h, int passes, double *pass_ms) {
    cudaStream_t s = h->stream;
    DevParams p = h->dparams;
    p.max_iters = 4 * passes + 64;
    p.tol = 0.f;
    p.pass_cap = 4 * passes + 64;
    DevMesh m = h->mesh();
    DevState st = h->state();
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (auto &e : ev) CK(cudaEventCreate(&e));
    cudaError_t e = cudaMemsetAsync(h->active, 0, 4 * sizeof(int), s);
    if (e == cudaSuccess) e = launch_init_ctl(s, h->B, p, st);
    if (e == cudaSuccess) e = launch_prologue(s, m, p, st, nullptr, h->pad2user.p);
    if (e == cudaSuccess) e = launch_guess_check(s, m, p, st);
    if (e == cudaSuccess) e = launch_ref_force(s, m, p, st);
    if (e == cudaSuccess) e = launch_to_increment(s, m, p, st);
    if (e == cudaSuccess) e = cudaEventRecord(ev[0], s);
    int rc = PBS_OK;
    bool refused = false;
    if (e == cudaSuccess) rc = launch_frame_step(h, p, passes, false, &refused);
    if (e == cudaSuccess && rc == PBS_OK) e = cudaEventRecord(ev[1], s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    float ms = 0.f;
    if (e == cudaSuccess && rc == PBS_OK) cudaEventElapsedTime(&ms, ev[0], ev[1]);
    for (auto &x : ev) cudaEventDestroy(x);
    CK(e);
    if (rc != PBS_OK) return rc;
    std::vector<InstCtl> ctl(h->B);
    int gave_up = 0;
    CK(cudaMemcpy(ctl.data(), h->ctl.p, sizeof(InstCtl) * h->B, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(&gave_up, h->active + 1, sizeof(int), cudaMemcpyDeviceToHost));
    const bool ok = frame_done(h, passes, gave_up) == PBS_OK;
    for (InstCtl &c : ctl) {
        if (c.tet_end == c.tet_begin) continue;
        if (!ok) c.status = PBS_E_DEVICE_TIMEOUT;
        if (c.status == PBS_OK && c.passes >= passes) continue;
        pbs_stats S{};
        S.passes = c.passes; S.iterations = c.k; S.rejections = c.rejections; S.converged = c.converged;
        S.status = c.status; S.alpha = c.alpha; S.rho = c.rho; S.omega = c.omega; S.energy = c.energy;
        S.residual_ratio = residual_ratio(c);
        h->stats = S;
        return c.status != PBS_OK ? c.status : PBS_E_ITER_CAP;
    }
    *pass_ms = ms / passes;
    return PBS_OK;
}

extern "C" {

int pbs_set_pass_engine(pbs_handle *h, int engine) {
    if (!h || (engine != PBS_ENGINE_GRAPH && engine != PBS_ENGINE_FRAME)) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    if (engine == PBS_ENGINE_FRAME && !frame_applies(h)) return PBS_E_INVALID_ARG;
    h->engine = engine;
    h->engine_auto = false;
    return PBS_OK;
}

int pbs_get_pass_engine(pbs_handle *h, int *engine) {
    if (!h || !engine) return PBS_E_INVALID_ARG;
    *engine = h->engine;
    return PBS_OK;
}

int pbs_get_step_engine(pbs_handle *h, int *engine) {
    if (!h || !engine) return PBS_E_INVALID_ARG;
    *engine = h->step_engine;
    return PBS_OK;
}

int pbs_profile_frame(pbs_handle *h, int passes, double *pass_ms) {
    if (!h || passes <= 0 || !pass_ms) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    return time_frame(h, passes, pass_ms);
}

int pbs_profile_kernels(pbs_handle *h, int passes, double *tet_ms, double *node_ms) {
    if (!h || passes <= 0 || !tet_ms || !node_ms) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    return time_passes(h, passes, tet_ms, node_ms);
}

int pbs_set_chunk_shape(pbs_handle *h, int threads, int chunk_tets, int chunk_nodes, int staged, int node_npt) {
    if (!h || (threads != 128 && threads != 256 && threads != 512) || chunk_tets < 1 || chunk_nodes < 4 ||
        (node_npt != 1 && node_npt != 2) ||
        4 * (size_t)chunk_tets > 65536 || chunk_nodes > 65536 || staged < 0 || staged > 2 ||
        (staged && threads == 512) ||
        // (48 B a node without staging too: the packed words' 24 leave room to pad every run of slots)
        chunk_smem(chunk_tets, chunk_nodes, 4 * chunk_tets, true, staged) + (staged ? 0 : 24 * (size_t)chunk_nodes) >
            (size_t)CHUNK_MAX_SMEM)
        return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    const int rc = set_pass_layout(h, threads, chunk_tets, chunk_nodes, staged, nullptr);
    if (rc == PBS_OK) h->node_npt = node_npt;
    return rc;
}

int pbs_autotune(pbs_handle *h, int passes, pbs_tune_result *out) {
    if (!h || passes <= 0) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    // chunk shapes: CTA threads, tets per chunk, nodes a chunk may touch,
    // staging (neo-Hookean only: 1 = rows staged in shared memory, 2 = the
    // persistent double-buffered kernel)
    static const int shapes[][4] = {{256, 1024, 448, 0}, {256, 768, 352, 0}, {256, 512, 256, 0},
                                    {128, 512, 256, 0},  {128, 256, 160, 0}, {512, 1024, 448, 0},
                                    {512, 2048, 832, 0}, {256, 640, 320, 0}, {256, 512, 256, 1},
                                    {256, 384, 208, 1},  {128, 256, 160, 1}, {128, 384, 208, 1},
                                    {256, 256, 160, 2},  {128, 256, 160, 2}, {256, 512, 256, 2},
                                    {128, 128, 96, 2},   {128, 384, 208, 0}, {256, 384, 208, 0},
                                    {128, 192, 128, 0},  {256, 256, 160, 0}};
    const int n = (int)(sizeof(shapes) / sizeof(shapes[0]));
    const bool can_stage = h->material == PBS_MATERIAL_NEOHOOKEAN;
    // threads 0: the automatic shape
    const int t0 = h->shape_auto ? 0 : h->chunk_threads, c0 = h->chunk_tets, n0 = h->chunk_nodes, s0 = h->chunk_stage;
    double best = 1e300, first = -1.0;
    int bi = -1, tried = 0;
    for (int i = 0; i < n; ++i) {
        if (shapes[i][3] && !can_stage) continue;
        int rc = set_pass_layout(h, shapes[i][0], shapes[i][1], shapes[i][2], shapes[i][3], nullptr);
        if (rc != PBS_OK) return rc;
        double a = 0.0, b = 0.0;
        rc = time_passes(h, passes, &a, &b);  // warm-up run, then the timed one
        if (rc == PBS_OK) rc = time_passes(h, passes, &a, &b);
        if (rc != PBS_OK) {
            // the state cannot be timed: restore the shape the handle had
            const int rc2 = set_pass_layout(h, t0, c0, n0, s0, nullptr);
            return rc2 != PBS_OK ? rc2 : rc;
        }
        const double t = a + b;
        ++tried;
        if (i == 0) first = t;
        if (t < best) {
            best = t;
            bi = i;
        }
    }
    // the frame kernel on the automatic layout, where a default step would run
    // it: kept when it beats every shape of the pass kernels
    int rc = PBS_OK;
    bool keep_frame = false;
    if (h->engine_auto) {
        rc = set_pass_layout(h, 0, 0, 0, 0, nullptr);
        if (rc != PBS_OK) return rc;
        double f = 0.0;
        keep_frame = auto_frame_applies(h) && time_frame(h, passes, &f) == PBS_OK &&
                     time_frame(h, passes, &f) == PBS_OK && f <= best;
    }
    rc = set_pass_layout(h, shapes[bi][0], shapes[bi][1], shapes[bi][2], shapes[bi][3], nullptr);
    if (rc != PBS_OK) return rc;
    // the node kernel: 1 or 2 nodes per thread (independent of the chunk shape)
    double node_ms[2] = {0.0, 0.0};
    const int npt0 = h->node_npt;
    for (int npt = 1; npt <= 2; ++npt) {
        h->node_npt = npt;
        double a = 0.0, b = 0.0;
        rc = time_passes(h, passes, &a, &b);
        if (rc == PBS_OK) rc = time_passes(h, passes, &a, &b);
        if (rc != PBS_OK) {
            h->node_npt = npt0;
            return rc;
        }
        node_ms[npt - 1] = b;
    }
    h->node_npt = node_ms[1] < node_ms[0] ? 2 : 1;
    h->graph_valid = h->plan_valid = false;
    if (out) {
        out->node_npt = h->node_npt;
        out->chunk_threads = shapes[bi][0];
        out->chunk_tets = shapes[bi][1];
        out->chunk_nodes = shapes[bi][2];
        out->chunk_staged = shapes[bi][3];
        out->n_tried = tried;
        out->pass_ms = best;
        out->default_pass_ms = first;
    }
    return keep_frame ? set_pass_layout(h, 0, 0, 0, 0, nullptr) : PBS_OK;
}

int pbs_read_velocities(pbs_handle *h, float *v, float *v_old) {
    if (!h || (!v && !v_old)) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    int rc = PBS_OK;
    if (v) rc = download_user(h, h->v.p, v);
    if (rc == PBS_OK && v_old) rc = download_user(h, h->vold.p, v_old);
    return rc;
}

int pbs_write_velocities(pbs_handle *h, const float *v, const float *v_old) {
    if (!h || (!v && !v_old)) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    int rc = PBS_OK;
    if (v) rc = upload_user(h, v, h->v.p);
    if (rc == PBS_OK && v_old) rc = upload_user(h, v_old, h->vold.p);
    return rc;
}

int pbs_reset(pbs_handle *h) {
    if (!h) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    CK(cudaMemsetAsync(h->u0h.p, 0, sizeof(float4) * h->Np, h->stream));
    CK(cudaMemsetAsync(h->u0l.p, 0, sizeof(float4) * h->Np, h->stream));
    CK(cudaMemsetAsync(h->v.p, 0, sizeof(float4) * h->Np, h->stream));
    CK(cudaMemsetAsync(h->vold.p, 0, sizeof(float4) * h->Np, h->stream));
    // the warm start's displacement history starts over with the motion
    CK(cudaMemsetAsync(h->hist1.p, 0, sizeof(float4) * h->Np, h->stream));
    CK(cudaMemsetAsync(h->hist2.p, 0, sizeof(float4) * h->Np, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return PBS_OK;
}

int pbs_get_stats(pbs_handle *h, pbs_stats *s) {
    if (!h || !s) return PBS_E_INVALID_ARG;
    *s = h->stats;
    return PBS_OK;
}

int pbs_get_instance_stats(pbs_handle *h, int instance, pbs_stats *s) {
    if (!h || !s || instance < 0 || instance >= h->B) return PBS_E_INVALID_ARG;
    const InstCtl &c = h->h_ctl[instance];  // copied back at the end of every pbs_step
    pbs_stats S{};
    S.passes = c.passes; S.iterations = c.k; S.rejections = c.rejections; S.converged = c.converged;
    S.status = c.status; S.alpha = c.alpha; S.rho = c.rho; S.omega = c.omega; S.energy = c.energy;
    S.residual_ratio = residual_ratio(c); S.device_ms = h->stats.device_ms; S.graph_launches = h->stats.graph_launches;
    S.warm_start_used = c.ws_used;
    S.guess_fallbacks = c.guess_bad;
    *s = S;
    return PBS_OK;
}

int pbs_get_sizes(pbs_handle *h, int *n_nodes, int *n_tets, int *n_instances) {
    if (!h) return PBS_E_INVALID_ARG;
    if (n_nodes) *n_nodes = h->N;
    if (n_tets) *n_tets = h->T;
    if (n_instances) *n_instances = h->B;
    return PBS_OK;
}

int pbs_set_surface(pbs_handle *h, const int *faces, int n_faces) {
    if (!h || n_faces < 0 || (n_faces > 0 && !faces)) return PBS_E_INVALID_ARG;
    for (size_t i = 0; i < 3 * (size_t)n_faces; ++i)
        if (faces[i] < 0 || faces[i] >= h->N) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    h->faces_pad.release(); h->ring_pad.release(); h->pick_id.release(); h->pick_d2.release();
    h->n_faces = 0;
    h->h_ring_ptr.assign(1, 0);
    h->h_ring.clear();
    if (n_faces == 0) return PBS_OK;
    // TetMesh::computeBoundfaceRingIndices (TetMesh.cpp:229-277): each node's
    // neighbours through surface edges; a face's ring = its three nodes, then
    // the union of their neighbours without them, ascending
    std::vector<std::vector<int>> nbr(h->N);
    for (int f = 0; f < n_faces; ++f) {
        const int *q = faces + 3 * (size_t)f;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b)
                if (a != b) nbr[q[a]].push_back(q[b]);
    }
    for (auto &v : nbr) {
        std::sort(v.begin(), v.end());
        v.erase(std::unique(v.begin(), v.end()), v.end());
    }
    std::vector<int4> fpad(n_faces);
    std::vector<int> tmp;
    for (int f = 0; f < n_faces; ++f) {
        const int *q = faces + 3 * (size_t)f;
        fpad[f] = make_int4(h->user2pad[q[0]], h->user2pad[q[1]], h->user2pad[q[2]], 0);
        tmp.clear();
        for (int a = 0; a < 3; ++a) tmp.insert(tmp.end(), nbr[q[a]].begin(), nbr[q[a]].end());
        std::sort(tmp.begin(), tmp.end());
        tmp.erase(std::unique(tmp.begin(), tmp.end()), tmp.end());
        h->h_ring.insert(h->h_ring.end(), q, q + 3);
        for (int v : tmp)
            if (v != q[0] && v != q[1] && v != q[2]) h->h_ring.push_back(v);
        h->h_ring_ptr.push_back((int)h->h_ring.size());
    }
    std::vector<int> rpad(h->h_ring.size());
    for (size_t j = 0; j < rpad.size(); ++j) rpad[j] = h->user2pad[h->h_ring[j]];
    const int nb = pick_blocks(n_faces, h->sms);
    CK(h->faces_pad.alloc(n_faces)); CK(h->ring_pad.alloc(rpad.size()));
    CK(h->pick_id.alloc(nb + 1)); CK(h->pick_d2.alloc(nb));
    if (!h->drag_ext.p) CK(h->drag_ext.alloc(h->Np));
    CK(cudaMemcpyAsync(h->faces_pad.p, fpad.data(), sizeof(int4) * n_faces, cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(h->ring_pad.p, rpad.data(), sizeof(int) * rpad.size(), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->n_faces = n_faces;
    return PBS_OK;
}

int pbs_get_face_ring(pbs_handle *h, int face, int *ring, int capacity, int *size) {
    if (!h || !size || face < 0 || face >= h->n_faces || (ring && capacity < 0)) return PBS_E_INVALID_ARG;
    const int b = h->h_ring_ptr[face], e = h->h_ring_ptr[face + 1];
    *size = e - b;
    if (ring)
        for (int j = 0; j < std::min(e - b, capacity); ++j) ring[j] = h->h_ring[b + j];
    return PBS_OK;
}

static bool finite3(const float *v) { return std::isfinite(v[0]) && std::isfinite(v[1]) && std::isfinite(v[2]); }

int pbs_pick_face(pbs_handle *h, const float *orig, const float *dir, int *face) {
    if (!h || !orig || !dir || !face || h->n_faces == 0 || !finite3(orig) || !finite3(dir)) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    const int nb = pick_blocks(h->n_faces, h->sms);
    CK(launch_pick_face(h->stream, h->mesh(), h->state(), h->n_faces, h->faces_pad.p,
                        make_float3(orig[0], orig[1], orig[2]), make_float3(dir[0], dir[1], dir[2]), nb, h->pick_d2.p,
                        h->pick_id.p, h->pick_id.p + nb));
    int out = -1;
    CK(cudaMemcpyAsync(&out, h->pick_id.p + nb, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    *face = out;
    return PBS_OK;
}

int pbs_drag_face_ring(pbs_handle *h, int face, const float *drag, float *ext) {
    if (!h || !drag || !ext || face < 0 || face >= h->n_faces || !finite3(drag)) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    const int b = h->h_ring_ptr[face], len = h->h_ring_ptr[face + 1] - b;
    CK(launch_drag_ring(h->stream, h->mesh(), h->state(), h->faces_pad.p, h->ring_pad.p, b, len,
                        make_float3(drag[0], drag[1], drag[2]), h->drag_ext.p));
    return download_user(h, h->drag_ext.p, ext);
}

// Block-CSR pattern of the padded mesh (per padded node, itself and every node
// sharing a tet with it, ascending) and the conjugate-gradient solve's plan:
// real nodes in the Morton order of their rest positions, instance by
// instance, split evenly over the CTAs; each CTA's halo (the other CTAs' nodes
// that its rows multiply) and the rows of its own that are in others' halos.
static int ensure_bsr(pbs_handle *h) {
    if (h->bsr_ready) return PBS_OK;
    CK(prepare_cg_kernels());
    cudaStream_t s = h->stream;
    const size_t np = (size_t)h->Np;
    std::vector<int> ptr(np + 1, 0);
    CK(h->bsr_ptr.alloc(np + 1));
    CK(launch_bsr_count(s, h->mesh(), h->bsr_ptr.p + 1));
    CK(cudaMemcpyAsync(ptr.data() + 1, h->bsr_ptr.p + 1, sizeof(int) * np, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    // the rows of nodes with many tets, which the kernels leave out (-1)
    std::vector<std::vector<int>> hub;  // a node, then its row's columns
    std::vector<int> hub_of;
    for (size_t i = 0; i < np; ++i)
        if (ptr[i + 1] < 0) {
            hub_of.resize(np, -1);
            hub_of[i] = (int)hub.size();
            hub.push_back({(int)i});
        }
    if (!hub.empty())
        for (const int4 &q : h->h_tets_pad)
            for (int c = 0; c < 4 && q.x >= 0; ++c) {
                const int r = hub_of[(&q.x)[c]];
                if (r >= 0) hub[r].insert(hub[r].end(), &q.x, &q.x + 4);
            }
    for (auto &r : hub) {
        std::sort(r.begin() + 1, r.end());
        r.erase(std::unique(r.begin() + 1, r.end()), r.end());
    }
    for (const auto &r : hub) ptr[r[0] + 1] = (int)r.size() - 1;
    for (size_t i = 0; i < np; ++i) ptr[i + 1] += ptr[i];
    const size_t nnzb = (size_t)ptr[np];
    std::vector<int> col(nnzb);
    CK(h->bsr_col.alloc(nnzb));
    CK(cudaMemcpyAsync(h->bsr_ptr.p, ptr.data(), sizeof(int) * (np + 1), cudaMemcpyHostToDevice, s));
    CK(launch_bsr_fill(s, h->mesh(), h->bsr_ptr.p, h->bsr_col.p));
    for (const auto &r : hub)
        CK(cudaMemcpyAsync(h->bsr_col.p + ptr[r[0]], r.data() + 1, sizeof(int) * (r.size() - 1), cudaMemcpyHostToDevice,
                           s));
    CK(cudaMemcpyAsync(col.data(), h->bsr_col.p, sizeof(int) * nnzb, cudaMemcpyDeviceToHost, s));
    // rows: (instance, Morton code) order, on the host meanwhile
    std::vector<std::pair<uint64_t, int>> order;
    order.reserve(h->N);
    for (int b = 0; b < h->B; ++b) {
        const int n0 = h->h_inst_nodes[2 * b], n1 = h->h_inst_nodes[2 * b + 1];
        double lo[3], inv[3];
        for (int d = 0; d < 3; ++d) {
            double mn = 1e300, mx = -1e300;
            for (int i = n0; i < n1; ++i) {
                mn = std::min(mn, h->h_rest_pad[3 * (size_t)i + d]);
                mx = std::max(mx, h->h_rest_pad[3 * (size_t)i + d]);
            }
            lo[d] = mn;
            inv[d] = mx > mn ? 1023.0 / (mx - mn) : 0.0;
        }
        for (int i = n0; i < n1; ++i) {
            uint32_t code = 0;
            for (int d = 0; d < 3; ++d)
                code |= spread10((uint32_t)((h->h_rest_pad[3 * (size_t)i + d] - lo[d]) * inv[d])) << d;
            order.emplace_back(((uint64_t)b << 32) | code, i);
        }
    }
    std::sort(order.begin(), order.end());
    CK(cudaStreamSynchronize(s));
    const int n = (int)order.size();
    // one CTA a SM, but no fewer than CG_MIN_ROWS rows each: more CTAs shorten
    // the row loops, fewer the sums every CTA waits for
    const int G = std::max(1, std::min(h->ctx_sms, (n + CG_MIN_ROWS - 1) / CG_MIN_ROWS));
    std::vector<int> cta_slice(G + 1, 0), cta_rows(G), cta_halo(G + 1, 0), cta_send(G + 1, 0);
    std::vector<int> srow, rlen, soff(1, 0), soff_local, halo, send;
    std::vector<int> place_of(np, -1), owner(np, -1), stamp(np, -1), lidx(np, 0), key;
    std::vector<char> sent(np, 0);
    auto row_len = [&](int i) { return ptr[i + 1] - ptr[i]; };
    // each CTA's rows, longest first, then by node: a slice's rows end together,
    // and on a mesh with rows of a few lengths in turn (a 5-tet box) a warp's
    // rows multiply runs of neighbouring words
    for (int c = 0; c < G; ++c) {
        const int a = (int)((int64_t)n * c / G), e = (int)((int64_t)n * (c + 1) / G), nr = e - a;
        std::sort(order.begin() + a, order.begin() + e, [&](const auto &x, const auto &y) {
            const int lx = row_len(x.second), ly = row_len(y.second);
            return lx != ly ? lx > ly : x.second < y.second;
        });
        for (int r0 = 0; r0 < nr; r0 += 32)
            for (int l = 0; l < 32; ++l) {
                const int i = r0 + l < nr ? order[a + r0 + l].second : -1;
                if (i >= 0) {
                    place_of[i] = (int)srow.size();
                    owner[i] = c;
                }
                srow.push_back(i);
                rlen.push_back(i < 0 ? 0 : row_len(i));
            }
        cta_rows[c] = nr;
        cta_slice[c + 1] = (int)srow.size() / 32;
    }
    // the halos, in the order of the words (the places of their rows)
    std::vector<int> lcol;  // by entry and lane
    int max_rows = 0, max_local = 0, max_halo = 0, max_entries = 0;
    for (int c = 0; c < G; ++c) {
        const int s0 = cta_slice[c], s1 = cta_slice[c + 1], nr = cta_rows[c], entry0 = soff.back();
        key.clear();
        for (int lr = 0; lr < nr; ++lr) {
            const int i = srow[32 * (size_t)s0 + lr];
            lidx[i] = lr;
            for (int k = ptr[i]; k < ptr[i + 1]; ++k) {
                const int j = col[k];
                if (owner[j] == c || stamp[j] == c) continue;
                stamp[j] = c;
                sent[j] = 1;
                key.push_back(place_of[j]);
            }
        }
        std::sort(key.begin(), key.end());
        const int nh = (int)key.size();
        for (int j = 0; j < nh; ++j) lidx[srow[key[j]]] = nr + j;
        halo.insert(halo.end(), key.begin(), key.end());
        for (int sl = s0; sl < s1; ++sl) {
            const int e0 = soff.back(), len = rlen[32 * (size_t)sl];
            soff_local.push_back(e0 - entry0);
            soff.push_back(e0 + len);
            lcol.resize((size_t)(e0 + len) * 32, 0);
            for (int l = 0; l < 32; ++l) {
                const int i = srow[32 * (size_t)sl + l], m = rlen[32 * (size_t)sl + l];
                for (int k = 0; k < m; ++k) lcol[(size_t)(e0 + k) * 32 + l] = lidx[col[ptr[i] + k]];
            }
        }
        cta_halo[c + 1] = cta_halo[c] + nh;
        max_rows = std::max(max_rows, nr);
        max_local = std::max(max_local, nr + nh);
        max_halo = std::max(max_halo, nh);
        max_entries = std::max(max_entries, soff.back() - entry0);
    }
    // the local rows whose words other CTAs read
    int max_send = 0;
    for (int c = 0; c < G; ++c) {
        const size_t base = 32 * (size_t)cta_slice[c];
        for (int lr = 0; lr < cta_rows[c]; ++lr)
            if (sent[srow[base + lr]]) send.push_back(lr);
        cta_send[c + 1] = (int)send.size();
        max_send = std::max(max_send, cta_send[c + 1] - cta_send[c]);
    }
    const int ns = (int)soff.size() - 1;
    // one allocation for the plan's index arrays
    struct Part {
        const std::vector<int> *v;
        size_t at;
    } part[] = {{&cta_slice, 0}, {&cta_rows, 0}, {&cta_halo, 0}, {&srow, 0}, {&rlen, 0}, {&soff, 0}, {&soff_local, 0},
                {&halo, 0}, {&cta_send, 0}, {&send, 0}};
    size_t total = 0;
    for (auto &p : part) {
        p.at = total;
        total += (p.v->size() + 31) / 32 * 32;  // (16-byte copies of srow and rlen)
    }
    CK(h->cg_plan.alloc(total));
    for (auto &p : part)
        CK(cudaMemcpyAsync(h->cg_plan.p + p.at, p.v->data(), sizeof(int) * p.v->size(), cudaMemcpyHostToDevice, s));
    const bool col32 = max_local > 0xffff || h->test_solve_col32;
    std::vector<uint16_t> lcol16;
    if (!col32) lcol16.assign(lcol.begin(), lcol.end());
    const void *src = col32 ? (const void *)lcol.data() : (const void *)lcol16.data();
    const size_t cbytes = lcol.size() * (col32 ? 4 : 2);
    CK(h->cg_col.alloc(cbytes));
    CK(cudaMemcpyAsync(h->cg_col.p, src, cbytes, cudaMemcpyHostToDevice, s));
    CgPlanView v{};
    v.grid = G;
    v.threads = max_rows > 256 ? 512 : 256;
    v.n_slices = ns;
    const int *base = h->cg_plan.p;
    v.cta_slice = base + part[0].at; v.cta_rows = base + part[1].at; v.cta_halo = base + part[2].at;
    v.srow = base + part[3].at; v.rlen = base + part[4].at; v.soff = base + part[5].at;
    v.soff_local = base + part[6].at; v.halo = base + part[7].at;
    v.cta_send = base + part[8].at; v.send = base + part[9].at;
    v.scol = h->cg_col.p;
    v.col32 = col32;
    for (int kind = 0; kind < 2; ++kind)
    for (int light = 0; light < 2; ++light) {
        // what fits shared memory, the most often read first
        const size_t budget = h->test_solve_smem >= 0 ? h->test_solve_smem : light ? CG_LIGHT_SMEM[kind] : CG_MAX_SMEM;
        CgPlanView &w = h->cgp[kind][light];
        w = v;
        w.light = light != 0;
        w.smem = 0;
        auto place = [&](size_t bytes) {
            bytes = (bytes + 127) / 128 * 128;
            if (w.smem + bytes > budget) return -1;
            const int at = w.smem;
            w.smem += (int)bytes;
            return at;
        };
        const size_t pad = 128 * (size_t)((max_rows + 31) / 32), nv = kind == 0 ? 9 : 1;  // 4 B a row, padded
        w.off_node = place(pad);
        w.off_rlen = place(pad);
        w.off_small = place(sizeof(int) * ((max_rows + 31) / 32 + (size_t)max_halo + max_send));
        w.off_p = place(sizeof(float4) * max_local);
        w.off_q = place(sizeof(float4) * max_rows);
        w.off_r = place(sizeof(float4) * max_rows);
        w.off_val = w.off_col = -1;
        const size_t vb = (size_t)max_entries * 128 * nv, cb = (size_t)max_entries * 32 * (col32 ? 4 : 2);
        if (w.smem + vb + cb + 256 <= budget) {
            w.off_val = place(vb);
            w.off_col = place(cb);
        }
        w.off_dinv = place(pad * nv);
        w.off_x = place(sizeof(float4) * max_rows);
    }
    h->cg_entries = (size_t)soff.back();
    h->cg_rows_pad = 32 * (size_t)ns;
    h->cg_halo = (size_t)cta_halo[G];
    CK(h->bsr_val.alloc(9 * nnzb)); CK(h->cg_dinv.alloc(9 * np));
    CK(h->cg_b.alloc(np)); CK(h->cg_x.alloc(np)); CK(h->cg_xp.alloc(h->cg_rows_pad));
    CK(h->cg_red.alloc(2 * 3 * (size_t)CG_COPIES * G));
    CK(h->cg_ws.alloc(4 * h->cg_rows_pad + h->cg_halo));
    CK(h->cg_state.alloc(CG_SOLVES)); CK(h->cg_ctl.alloc(2));
    CK(cudaMemsetAsync(h->cg_xp.p, 0, sizeof(float4) * h->cg_xp.n, s));
    CK(cudaMemsetAsync(h->cg_red.p, 0, sizeof(float4) * h->cg_red.n, s));
    CK(cudaMemsetAsync(h->cg_ctl.p, 0, 2 * sizeof(unsigned), s));
    if (!h->h_cg) CK(cudaMallocHost(&h->h_cg, sizeof(CgState) * CG_SOLVES + 2 * sizeof(unsigned)));
    CK(cudaStreamSynchronize(s));
    h->bsr_ready = true;
    return PBS_OK;
}

// Before a step's solves: how much of a SM they take.
static void enter_solves(pbs_handle *h, LargeCount &large) {
    h->solve_light = 2 * h->cgp[0][0].grid > h->ctx_sms && large.enter(large_solves, h->device) >= 2;
}

// Enqueues one solve A x = b (slot: where its state goes).
static cudaError_t enqueue_solve(pbs_handle *h, bool scalar, const float *val, const float *dinv, double tol2,
                                 int max_iters, int pnorm, int slot) {
    if (h->test_wait_error) {
        h->test_wait_error = false;
        const cudaError_t e = cudaMemsetAsync(h->cg_ctl.p + 1, 1, sizeof(unsigned), h->stream);
        if (e != cudaSuccess) return e;
    }
    CgArgs a{};
    a.val = val;
    a.dinv = dinv;
    a.b = h->cg_b.p; a.x = h->cg_x.p; a.xp = h->cg_xp.p; a.red = h->cg_red.p;
    a.ws_p = h->cg_ws.p;
    a.ws_r = a.ws_p + h->cg_rows_pad + h->cg_halo;
    a.ws_q = a.ws_r + h->cg_rows_pad;
    a.ws_x = a.ws_q + h->cg_rows_pad;
    a.cs = h->cg_state.p + slot;
    a.tag = h->cg_ctl.p;
    a.err = (int *)(h->cg_ctl.p + 1);
    a.tol2 = tol2;
    a.max_iters = max_iters;
    a.pnorm = pnorm;
    return launch_cg_solve(h->stream, h->cgp[scalar ? 1 : 0][h->solve_light], a, scalar);
}

// The states of the last `count` solves on the host, and the exchanged words'
// tags kept from wrapping.  A solve takes its state from its first CTA, which
// may have every word when another CTA's wait gave up (and wrote no rows), so
// the flag of such a wait makes every one of these solves a timeout; the words
// are then made clean again.
static int read_solves(pbs_handle *h, int count) {
    cudaStream_t s = h->stream;
    unsigned *ctl = (unsigned *)(h->h_cg + CG_SOLVES);
    CK(cudaMemcpyAsync(h->h_cg, h->cg_state.p, sizeof(CgState) * count, cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(ctl, h->cg_ctl.p, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (ctl[1])
        for (int k = 0; k < count; ++k) h->h_cg[k].status = PBS_E_DEVICE_TIMEOUT;
    if (ctl[0] > 0x40000000u || ctl[1]) {
        CK(cudaMemsetAsync(h->cg_xp.p, 0, sizeof(float4) * h->cg_xp.n, s));
        CK(cudaMemsetAsync(h->cg_red.p, 0, sizeof(float4) * h->cg_red.n, s));
        CK(cudaMemsetAsync(h->cg_ctl.p, 0, 2 * sizeof(unsigned), s));
    }
    return PBS_OK;
}

int pbs_backward_euler_step(pbs_handle *h, float dt, float alpha, float beta, const float *ext, float tol,
                            int max_iters, int *iters_out, double *residual_out) {
    if (!h || !(dt > 0.f) || !(alpha >= 0.f) || !(beta >= 0.f) || !(tol > 0.f) || max_iters <= 0)
        return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    int rc = ensure_bsr(h);
    if (rc != PBS_OK) return rc;
    if (ext) {
        rc = upload_user(h, ext, h->ext.p);
        if (rc != PBS_OK) return rc;
    }
    LargeCount large;
    enter_solves(h, large);
    cudaStream_t s = h->stream;
    const DevMesh m = h->mesh();
    const DevState st = h->state();
    BsrView A;
    A.ptr = h->bsr_ptr.p;
    A.col = h->bsr_col.p;
    A.val = h->bsr_val.p;
    const double tol2 = (double)tol * (double)tol;
    if (!h->cg_val.p) CK(h->cg_val.alloc(9 * (32 * h->cg_entries + h->cg_rows_pad)));
    float *cgd = h->cg_val.p + 9 * 32 * h->cg_entries;  // the inverses by row
    CK(launch_be_assemble(s, m, st, h->material, A, dt, alpha, beta, ext ? h->ext.p : nullptr, h->cg_b.p, h->cg_x.p,
                          h->cg_dinv.p));
    CK(launch_cg_pack(s, h->cgp[0][0], A, h->cg_dinv.p, h->cg_val.p, cgd));
    CK(enqueue_solve(h, false, h->cg_val.p, cgd, tol2, max_iters, 0, 0));
    rc = read_solves(h, 1);
    if (rc != PBS_OK) return rc;
    const CgState c = h->h_cg[0];
    if (iters_out) *iters_out = c.iters;
    if (residual_out) *residual_out = c.bb > 0.0 ? std::sqrt(c.rr / c.bb) : 0.0;
    // the state is left as it was
    if (c.status == PBS_E_NONFINITE || c.status == PBS_E_DEVICE_TIMEOUT) return c.status;
    CK(launch_be_finish(s, m, st, h->cg_x.p, dt));
    CK(cudaStreamSynchronize(s));
    h->guess_pending = false;
    return c.status;
}

// ---- strain-based PBD and projective dynamics


// Levels of the caller's tet order per instance (a tet above the last earlier
// tet touching any of its nodes), the level-ordered tets, and the step's rest
// data formed as the reference forms it (launch_pbd_rest).
static int ensure_pbd(pbs_handle *h) {
    if (h->pbd_ready) return PBS_OK;
    const int B = h->B, Tp = h->Tp;
    std::vector<int> level(Tp, -1), second(Tp, -1), last(h->Np, -1), grp(B + 1, 0), delay(B, 1);
    for (int b = 0; b < B; ++b) {
        // levels of the instance's tets after the levels in `last`, from 0:
        // {their number, the delay between sweeps}
        auto levels = [&](std::vector<int> &lv) {
            int lo = INT_MAX, top = -1, D = 1;
            for (int tp = h->h_inst_tets[2 * b]; tp < h->h_inst_tets[2 * b + 1]; ++tp) {
                const int4 q = h->h_tets_pad[tp];
                if (q.x < 0) continue;
                const int l = 1 + std::max(std::max(last[q.x], last[q.y]), std::max(last[q.z], last[q.w]));
                lv[tp] = l;
                last[q.x] = last[q.y] = last[q.z] = last[q.w] = l;
                lo = std::min(lo, l);
                top = std::max(top, l);
            }
            // (last: the highest level at each node)
            for (int tp = h->h_inst_tets[2 * b]; tp < h->h_inst_tets[2 * b + 1]; ++tp) {
                const int4 q = h->h_tets_pad[tp];
                if (q.x < 0) continue;
                const int up = std::max(std::max(last[q.x], last[q.y]), std::max(last[q.z], last[q.w]));
                D = std::max(D, up - lv[tp] + 1);
                lv[tp] -= lo;
            }
            return std::make_pair(top < 0 ? 0 : top - lo + 1, D);
        };
        // the earliest levels, or those that the tets have in a second sweep
        // behind the first, where nothing is earlier than the next sweep needs
        // it: about as many, and a smaller delay (the 24,000-tet bar 348 and 72
        // against 348 and 34, the 1M-tet box 2,320 and 44 against 2,325 and 39).
        // Whichever gives the reference's five sweeps fewer steps
        const auto p1 = levels(level), p2 = levels(second);
        auto best = p1;
        if (p2.first + 4 * p2.second < p1.first + 4 * p1.second) {
            best = p2;
            for (int tp = h->h_inst_tets[2 * b]; tp < h->h_inst_tets[2 * b + 1]; ++tp) level[tp] = second[tp];
        }
        delay[b] = best.second;
        grp[b + 1] = grp[b] + best.first;
    }
    const int L = grp[B];
    std::vector<int> lvl(L + 1, 0);
    for (int b = 0; b < B; ++b)
        for (int tp = h->h_inst_tets[2 * b]; tp < h->h_inst_tets[2 * b + 1]; ++tp)
            if (level[tp] >= 0) lvl[grp[b] + level[tp] + 1]++;
    for (int l = 0; l < L; ++l) lvl[l + 1] += lvl[l];
    const int n = lvl[L];
    std::vector<int> fill(lvl.begin(), lvl.end() - 1), order(std::max(n, 1));
    for (int b = 0; b < B; ++b)
        for (int tp = h->h_inst_tets[2 * b]; tp < h->h_inst_tets[2 * b + 1]; ++tp)
            if (level[tp] >= 0) order[fill[grp[b] + level[tp]]++] = tp;
    std::vector<int4> tet(std::max(n, 1));
    for (int j = 0; j < n; ++j) tet[j] = h->h_tets_pad[order[j]];
    const size_t nn = (size_t)std::max(n, 1);
    CK(h->pbd_grp.alloc(B + 1)); CK(h->pbd_delay.alloc(B)); CK(h->pbd_lvl.alloc(L + 1)); CK(h->pbd_tet.alloc(nn));
    CK(h->pbd_d0.alloc(nn)); CK(h->pbd_d1.alloc(nn)); CK(h->pbd_d2.alloc(nn)); CK(h->pbd_node.alloc(h->Np));
    CK(cudaMemcpy(h->pbd_grp.p, grp.data(), sizeof(int) * (B + 1), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->pbd_delay.p, delay.data(), sizeof(int) * B, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->pbd_lvl.p, lvl.data(), sizeof(int) * (L + 1), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->pbd_tet.p, tet.data(), sizeof(int4) * n, cudaMemcpyHostToDevice));
    DevBuf<int> ord;  // level order -> padded tet, needed only here
    CK(ord.alloc(nn));
    cudaError_t e = cudaMemcpy(ord.p, order.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = launch_pbd_rest(h->stream, h->mesh(), ord.p, n, h->density, h->gravity, h->pbd_d0.p, h->pbd_d1.p,
                            h->pbd_d2.p, h->staging2.p, h->pbd_node.p);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    ord.release();
    CK(e);
    h->pbd_groups = B;
    // positions in the cluster's distributed shared memory when every
    // instance's nodes fit 16 slices (a few instances; batches of many small
    // instances keep the global-memory sweep)
    h->pbd_smem = 0;
    if (B <= 4) {
        int slice = 0;
        for (int b = 0; b < B; ++b)
            slice = std::max(slice, (h->h_inst_nodes[2 * b + 1] - h->h_inst_nodes[2 * b] + 15) / 16);
        const int smem = std::max(slice, 1) * (int)sizeof(float4);
        if (slice <= 0xffff && pbd_dsmem_fits(smem)) {
            std::vector<int4> gn(B), codes(std::max(n, 1));
            for (int b = 0; b < B; ++b) {
                const int nb = h->h_inst_nodes[2 * b], cnt = h->h_inst_nodes[2 * b + 1] - nb;
                gn[b] = make_int4(nb, std::max((cnt + 15) / 16, 1), cnt, 0);
            }
            for (int b = 0; b < B; ++b)
                for (int j = lvl[grp[b]]; j < lvl[grp[b + 1]]; ++j) {
                    const int *q = &tet[j].x;
                    int c[4];
                    for (int k = 0; k < 4; ++k) {
                        const int loc = q[k] - gn[b].x;
                        c[k] = ((loc % 16) << 16) | (loc / 16);
                    }
                    codes[j] = make_int4(c[0], c[1], c[2], c[3]);
                }
            CK(h->pbd_codes.alloc(codes.size())); CK(h->pbd_gnode.alloc(B));
            CK(cudaMemcpy(h->pbd_codes.p, codes.data(), sizeof(int4) * codes.size(), cudaMemcpyHostToDevice));
            CK(cudaMemcpy(h->pbd_gnode.p, gn.data(), sizeof(int4) * B, cudaMemcpyHostToDevice));
            h->pbd_smem = smem;
        }
    }
    h->pbd_ready = true;
    return PBS_OK;
}

static int ensure_dyn_buffers(pbs_handle *h) {
    if (h->dyn_s.p) return PBS_OK;  // (the last of the three)
    CK(h->dyn_px.alloc(h->Np)); CK(h->dyn_x0.alloc(h->Np)); CK(h->dyn_s.alloc(h->Np));
    return PBS_OK;
}

static bool finite_n(const float *v, int n) {
    for (int i = 0; i < n; ++i)
        if (!std::isfinite(v[i])) return false;
    return true;
}

int pbs_pbd_step(pbs_handle *h, float dt, int iterations, const float *stretch, const float *shear,
                 const float *ext) {
    if (!h || !(dt > 0.f) || !std::isfinite(dt) || iterations < 0 || (stretch && !finite_n(stretch, 3)) ||
        (shear && !finite_n(shear, 3)))
        return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    int rc = ensure_pbd(h);
    if (rc == PBS_OK) rc = ensure_dyn_buffers(h);
    if (rc == PBS_OK && ext) rc = upload_user(h, ext, h->ext.p);
    if (rc != PBS_OK) return rc;
    const float st_def[3] = {1.f, 1.f, 1.f}, sh_def[3] = {0.8f, 0.8f, 0.8f};
    cudaStream_t s = h->stream;
    const DevMesh m = h->mesh();
    const DevState st = h->state();
    CK(launch_pbd_begin(s, m, st, h->pbd_node.p, ext ? h->ext.p : nullptr, dt, h->dyn_px.p, h->dyn_x0.p));
    if (iterations > 0) {
        PbdView v;
        v.grp = h->pbd_grp.p; v.lvl = h->pbd_lvl.p; v.delay = h->pbd_delay.p; v.tet = h->pbd_tet.p;
        v.d0 = h->pbd_d0.p; v.d1 = h->pbd_d1.p; v.d2 = h->pbd_d2.p; v.px = h->dyn_px.p;
        if (h->pbd_smem > 0)
            CK(launch_pbd_sweeps_dsmem(s, v, h->pbd_codes.p, h->pbd_gnode.p, h->pbd_groups, h->pbd_smem, iterations,
                                       stretch ? stretch : st_def, shear ? shear : sh_def));
        else
            CK(launch_pbd_sweeps(s, v, h->pbd_groups, iterations, stretch ? stretch : st_def, shear ? shear : sh_def));
    }
    CK(launch_dyn_end(s, m, st, h->dyn_px.p, h->dyn_x0.p, dt, 0));
    CK(cudaStreamSynchronize(s));
    h->guess_pending = false;
    return PBS_OK;
}

int pbs_pd_step(pbs_handle *h, float dt, float dt_matrix, float stiffness, int iterations, const float *ext,
                float tol, int max_cg, int *cg_iters_out) {
    if (!h || !(dt > 0.f) || !std::isfinite(dt) || !(dt_matrix >= 0.f) || !std::isfinite(dt_matrix) ||
        !(stiffness > 0.f) || !std::isfinite(stiffness) || iterations < 0 || !(tol > 0.f) || max_cg <= 0)
        return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    const float dtm = dt_matrix > 0.f ? dt_matrix : dt;
    int rc = ensure_bsr(h);
    if (rc == PBS_OK) rc = ensure_dyn_buffers(h);
    if (rc == PBS_OK && ext) rc = upload_user(h, ext, h->ext.p);
    if (rc != PBS_OK) return rc;
    LargeCount large;
    enter_solves(h, large);
    cudaStream_t s = h->stream;
    const DevMesh m = h->mesh();
    const DevState st = h->state();
    BsrView A;
    A.ptr = h->bsr_ptr.p;
    A.col = h->bsr_col.p;
    A.scalar = 1;
    if (!h->pd_dinv.p) {  // (the last of the three)
        int nnzb = 0;
        CK(cudaMemcpy(&nnzb, h->bsr_ptr.p + h->Np, sizeof(int), cudaMemcpyDeviceToHost));
        CK(h->pd_val.alloc((size_t)nnzb));
        CK(h->pd_cgval.alloc(32 * h->cg_entries + h->cg_rows_pad));
        CK(h->pd_dinv.alloc(9 * (size_t)h->Np));
    }
    A.val = h->pd_val.p;
    if (!h->pd_ready || h->pd_dtm != dtm || h->pd_k != stiffness) {
        CK(launch_pd_assemble(s, m, A, dtm, stiffness, h->pd_dinv.p));
        CK(launch_cg_pack(s, h->cgp[1][0], A, h->pd_dinv.p, h->pd_cgval.p, h->pd_cgval.p + 32 * h->cg_entries));
        h->pd_ready = true;
        h->pd_dtm = dtm;
        h->pd_k = stiffness;
    }
    CK(launch_pd_begin(s, m, st, ext ? h->ext.p : nullptr, dt, h->dyn_s.p, h->dyn_px.p, h->dyn_x0.p));
    const double tol2 = (double)tol * (double)tol;
    int total = 0, status = PBS_OK;
    // the solves follow one another on the stream; their states are read once
    // (a solve that ends non-finite leaves the rest nothing to do, and the
    // handle's state is only written after the last)
    for (int it = 0; it < iterations; it += CG_SOLVES) {
        const int count = std::min(CG_SOLVES, iterations - it);
        for (int k = 0; k < count; ++k) {
            CK(launch_pd_residual(s, m, h->dyn_px.p, stiffness, dt, dtm, reinterpret_cast<float4 *>(h->tf.p),
                                  h->dyn_s.p, h->dyn_x0.p, h->cg_b.p, h->cg_x.p));
            CK(enqueue_solve(h, true, h->pd_cgval.p, h->pd_cgval.p + 32 * h->cg_entries, tol2, max_cg, 1, k));
            CK(launch_pd_apply(s, h->Np, h->dyn_px.p, h->cg_x.p));
        }
        rc = read_solves(h, count);
        if (rc != PBS_OK) return rc;
        for (int k = 0; k < count; ++k) {
            const CgState &c = h->h_cg[k];
            total += c.iters;
            if (c.status == PBS_E_NONFINITE || c.status == PBS_E_DEVICE_TIMEOUT) {
                if (cg_iters_out) *cg_iters_out = total;
                return c.status;  // the state is left as it was
            }
            if (c.status == PBS_E_ITER_CAP) status = PBS_E_ITER_CAP;
        }
    }
    CK(launch_dyn_end(s, m, st, h->dyn_px.p, h->dyn_x0.p, dt, 1));
    CK(cudaStreamSynchronize(s));
    h->guess_pending = false;
    if (cg_iters_out) *cg_iters_out = total;
    return status;
}

int pbs_get_incidence(pbs_handle *h, int *row_ptr, int *entries) {
    if (!h || !row_ptr || !entries) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    std::vector<int> iptr(h->Np + 1), ient(4 * (size_t)h->T);
    CK(cudaMemcpy(iptr.data(), h->inc_ptr.p, sizeof(int) * (h->Np + 1), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(ient.data(), h->inc.p, sizeof(int) * 4 * (size_t)h->T, cudaMemcpyDeviceToHost));
    // translate padded ids back to the caller's numbering
    row_ptr[0] = 0;
    size_t w = 0;
    for (int u = 0; u < h->N; ++u) {
        int ip = h->user2pad[u];
        for (int j = iptr[ip]; j < iptr[ip + 1]; ++j) {
            int tp = ient[j] >> 2, c = ient[j] & 3;
            entries[w++] = 4 * h->h_tet_user[tp] + c;
        }
        row_ptr[u + 1] = (int)w;
    }
    return PBS_OK;
}

int pbs_get_rest_data(pbs_handle *h, float *dm_inv9, float *signed_vol, float *mass, float *grav_y) {
    if (!h) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    std::vector<float4> r0(h->Tp), r1(h->Tp), r2(h->Tp), inf(h->Np);
    CK(cudaMemcpy(r0.data(), h->row0.p, sizeof(float4) * h->Tp, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(r1.data(), h->row1.p, sizeof(float4) * h->Tp, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(r2.data(), h->row2.p, sizeof(float4) * h->Tp, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(inf.data(), h->info.p, sizeof(float4) * h->Np, cudaMemcpyDeviceToHost));
    for (int tp = 0; tp < h->Tp; ++tp) {
        int t = h->h_tet_user[tp];
        if (t < 0) continue;
        if (dm_inv9) {
            float *o = dm_inv9 + 9 * (size_t)t;
            o[0] = r0[tp].x; o[1] = r0[tp].y; o[2] = r0[tp].z;
            o[3] = r1[tp].x; o[4] = r1[tp].y; o[5] = r1[tp].z;
            o[6] = r2[tp].x; o[7] = r2[tp].y; o[8] = r2[tp].z;
        }
        if (signed_vol) signed_vol[t] = r0[tp].w;
    }
    for (int u = 0; u < h->N; ++u) {
        int ip = h->user2pad[u];
        if (mass) mass[u] = inf[ip].x;
        if (grav_y) grav_y[u] = inf[ip].y;
    }
    return PBS_OK;
}

// The saved-state buffers are rewritten at iteration 0 of every step, so
// between steps they serve as scratch for evaluating given positions.
// The displacement pair (hi, lo) the probes evaluate: the uploaded positions,
// or the current state.
static int eval_common(pbs_handle *h, const float *positions, const float4 **xsrc, const float4 **xlo = nullptr) {
    if (positions) {
        int rc = upload_positions(h, positions, h->oh.p, h->ol.p);
        if (rc != PBS_OK) return rc;
        *xsrc = h->oh.p;
        if (xlo) *xlo = h->ol.p;
    } else {
        *xsrc = h->u0h.p;
        if (xlo) *xlo = h->u0l.p;
    }
    return PBS_OK;
}

int pbs_eval_tets(pbs_handle *h, const float *positions, float *corner_forces, float *energy, float *hess_diag) {
    if (!h) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    const float4 *x, *xl;
    int rc = eval_common(h, positions, &x, &xl);
    if (rc != PBS_OK) return rc;
    // per-tet outputs land in tf / hd / staging2 (padded order), then are
    // compacted into the caller's tet order on the host
    struct Counter {  // freed on every return path
        DevBuf<unsigned int> b;
        ~Counter() { b.release(); }
    } n64_buf;
    DevBuf<unsigned int> &n64 = n64_buf.b;
    CK(n64.alloc(1));
    CK(cudaMemsetAsync(n64.p, 0, sizeof(unsigned int), h->stream));
    CK(launch_eval_tets(h->stream, h->mesh(), x, h->material, h->dparams.clamp_cpu, h->tf.p, h->staging2.p, h->hd.p,
                        n64.p, xl));
    std::vector<float> tf(12 * (size_t)h->Tp), hd(12 * (size_t)h->Tp), en(h->Tp);
    unsigned int n64_host = 0;
    CK(cudaMemcpyAsync(tf.data(), h->tf.p, sizeof(float) * tf.size(), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(hd.data(), h->hd.p, sizeof(float) * hd.size(), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(en.data(), h->staging2.p, sizeof(float) * en.size(), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(&n64_host, n64.p, sizeof(unsigned int), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->last_fp64_svd = (int)n64_host;
    for (int tp = 0; tp < h->Tp; ++tp) {
        int t = h->h_tet_user[tp];
        if (t < 0) continue;
        if (corner_forces) std::memcpy(corner_forces + 12 * (size_t)t, &tf[12 * (size_t)tp], 12 * sizeof(float));
        if (hess_diag) std::memcpy(hess_diag + 12 * (size_t)t, &hd[12 * (size_t)tp], 12 * sizeof(float));
        if (energy) energy[t] = en[tp];
    }
    return PBS_OK;
}

int pbs_eval_fp64_svd_count(pbs_handle *h, int *count) {
    if (!h || !count) return PBS_E_INVALID_ARG;
    *count = h->last_fp64_svd;
    return PBS_OK;
}

int pbs_eval_base_force(pbs_handle *h, const float *positions, double *forces) {
    if (!h || !positions || !forces) return PBS_E_INVALID_ARG;
    if (h->material != PBS_MATERIAL_NEOHOOKEAN) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    const float4 *x;
    int rc = eval_common(h, positions, &x);
    if (rc != PBS_OK) return rc;
    struct Scratch {  // freed on every return path
        DevBuf<float4> b;
        ~Scratch() { b.release(); }
    } sb;
    CK(sb.b.alloc(4 * (size_t)h->Np));
    // the step's base-force kernels on the displacement's hi words, with the
    // body forces off and the sums landing in the scratch pair
    DevParams p = h->dparams;
    p.incremental = 1;
    p.body_scale = 0.f;
    DevState st = h->state();
    st.ub = const_cast<float4 *>(x);
    st.bh = sb.b.p;
    st.bl = sb.b.p + h->Np;
    st.ch = sb.b.p + 2 * (size_t)h->Np;  // the gather's gradient constant: scratch too
    st.cl = sb.b.p + 3 * (size_t)h->Np;
    CK(launch_ref_force(h->stream, h->mesh(), p, st));
    std::vector<float4> b(2 * (size_t)h->Np);
    CK(cudaMemcpyAsync(b.data(), sb.b.p, sizeof(float4) * b.size(), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (int i = 0; i < h->Np; ++i) {
        const int u = h->h_pad2user[i];
        if (u < 0) continue;
        const float4 hi = b[i], lo = b[h->Np + i];
        forces[3 * (size_t)u] = (double)hi.x + (double)lo.x;
        forces[3 * (size_t)u + 1] = (double)hi.y + (double)lo.y;
        forces[3 * (size_t)u + 2] = (double)hi.z + (double)lo.z;
    }
    return PBS_OK;
}

int pbs_eval_nodes(pbs_handle *h, const float *positions, float *forces, float *hess_diag) {
    if (!h) return PBS_E_INVALID_ARG;
    PBS_DEVICE_SCOPE(h->device);
    const float4 *x, *xl;
    int rc = eval_common(h, positions, &x, &xl);
    if (rc != PBS_OK) return rc;
    DevBuf<float> out;
    CK(out.alloc(6 * (size_t)h->N));
    cudaError_t e = launch_eval_tets(h->stream, h->mesh(), x, h->material, h->dparams.clamp_cpu, h->tf.p, nullptr,
                                     h->hd.p, nullptr, xl);
    if (e == cudaSuccess) e = launch_gather(h->stream, h->mesh(), h->tf.p, h->hd.p, h->pad2user.p, out.p, out.p + 3 * (size_t)h->N);
    if (e == cudaSuccess && forces) e = cudaMemcpyAsync(forces, out.p, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess && hess_diag) e = cudaMemcpyAsync(hess_diag, out.p + 3 * (size_t)h->N, sizeof(float) * 3 * (size_t)h->N, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    out.release();
    CK(e);
    return PBS_OK;
}

// IsotropicMaterial::allocateGlobalStiffnessMatrix (IsotropicMaterial.cpp:554-644):
// rows 3n+d hold the sorted columns 3m+e of every node m sharing a tet with n.
int pbs_stiffness_pattern(int n_nodes, int n_tets, const int *tets, int *nnz, int *row_ptr, int *col, int *diag_idx,
                          int *kid48) {
    if (n_nodes <= 0 || n_tets < 0 || !tets || !nnz) return PBS_E_INVALID_ARG;
    std::vector<int64_t> pairs;
    pairs.reserve(16 * (size_t)n_tets);
    for (int t = 0; t < n_tets; ++t)
        for (int a = 0; a < 4; ++a)
            for (int b = 0; b < 4; ++b) {
                int na = tets[4 * (size_t)t + a], nb = tets[4 * (size_t)t + b];
                if (na < 0 || na >= n_nodes || nb < 0 || nb >= n_nodes) return PBS_E_BAD_MESH;
                pairs.push_back(((int64_t)na << 32) | (uint32_t)nb);
            }
    std::sort(pairs.begin(), pairs.end());
    pairs.erase(std::unique(pairs.begin(), pairs.end()), pairs.end());
    std::vector<int> nptr(n_nodes + 1, 0);
    for (int64_t pr : pairs) nptr[(pr >> 32) + 1]++;
    for (int i = 0; i < n_nodes; ++i) nptr[i + 1] += nptr[i];
    const int64_t total = 9 * (int64_t)pairs.size();
    if (total > INT32_MAX) return PBS_E_CAPACITY;
    *nnz = (int)total;
    if (!col) return PBS_OK;
    if (!row_ptr) return PBS_E_INVALID_ARG;
    row_ptr[0] = 0;
    for (int n = 0; n < n_nodes; ++n) {
        int deg = nptr[n + 1] - nptr[n];
        for (int d = 0; d < 3; ++d) {
            int r = 3 * n + d;
            int start = 9 * nptr[n] + d * 3 * deg;
            row_ptr[r + 1] = start + 3 * deg;
            for (int j = 0; j < deg; ++j) {
                int m = (int)(pairs[nptr[n] + j] & 0xffffffff);
                for (int e = 0; e < 3; ++e) col[start + 3 * j + e] = 3 * m + e;
            }
        }
    }
    auto slot = [&](int r, int c) {
        const int *b = col + row_ptr[r], *e = col + row_ptr[r + 1];
        return (int)(std::lower_bound(b, e, c) - col);
    };
    if (diag_idx)
        for (int r = 0; r < 3 * n_nodes; ++r) diag_idx[r] = slot(r, r);
    if (kid48)
        for (int t = 0; t < n_tets; ++t)
            for (int fi = 0; fi < 4; ++fi)
                for (int fj = 0; fj < 3; ++fj) {
                    int gki = 3 * tets[4 * (size_t)t + fi] + fj;
                    for (int ni = 0; ni < 4; ++ni) kid48[48 * (size_t)t + (fi * 3 + fj) * 4 + ni] = slot(gki, 3 * tets[4 * (size_t)t + ni]);
                }
    return PBS_OK;
}

}  // extern "C"

void pbs::handle_view(const pbs_handle *h, HandleView *v) {
    v->device = h->device;
    v->stream = h->stream;
    v->material = h->material;
    v->mesh = h->mesh();
    v->pad2user = h->pad2user.p;
}

// The per-tet kernel of a descent pass, on chunks of tets.
//
// A chunk is a run of at most chunk_tets tets of one instance, consecutive in
// the Morton order of their centroids, that touches at most chunk_nodes nodes
// (the instance's automatic limits, auto_chunk_limits, or the chunk shape that
// the caller or pbs_autotune set).  One CTA per chunk:
//   1. stages the chunk's nodes (displacements hi and lo, or increments and
//      force base) in shared memory: each node is read once per chunk instead
//      of once per corner;
//   2. evaluates its tets (one thread per tet, chunk tets / CTA threads tets
//      a thread), streaming the per-tet rows in chunk order, and writes the 12
//      corner forces to shared-memory slots, where a node's slots are
//      contiguous in (tet, corner) order;
//   3. sums each node's slots in that order into one partial per (node,
//      chunk), written to part[] at the node's place for this chunk.
// The node kernel adds a node's partials in chunk order.  No atomics touch a
// force, so results are bit-reproducible run to run, and instances are
// chunked on their own, so a packed batch gives each instance the bits it gets
// alone (the order of the energy and |g|^2 sums: phybs_internal.cuh).  Against one thread per tet writing 4 global slots, this moves the
// corner forces through shared memory instead of HBM (64 B written and read
// back per tet per pass) and replaces 4 gathers of 3 node words per tet with
// one staged read per touched node.
//
// On line-search passes the CTA also adds the clamped tet energies and its
// share of the instance's node energy terms (FP64, fixed order); the
// instance's last chunk to finish decides accept / reject
// (DescentOptimize.cpp:107-128) before any node moves.
//
// The pass decision of the previous node update (residual test, Chebyshev
// state, caps) is taken by the instance's first chunk CTA (settle_pass) from
// one control-block copy into the other, while every CTA runs on its
// foreseen outcome (pass_view): the next k, or work that goes unused when the
// instance stopped.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <limits>
#include <utility>
#include <vector>

#include "../../include/phybs.h"
#include "chunk_tets.cuh"
#include "exchange.cuh"
#include "pass_ctl.cuh"
#include "pass_math.cuh"
#include "phybs_internal.cuh"
#include "tet_math.cuh"

namespace pbs {

// ------------------------------------------------------------ host: layout
// Sorts (30-bit Morton code, tet) pairs, given by ascending tet, by both: a
// stable radix sort, ten bits at a time (chunking 1M tets takes 120 ms, and 145
// with std::sort).
static void sort_by_code(std::vector<std::pair<uint32_t, int>> &v, std::vector<std::pair<uint32_t, int>> &tmp) {
    tmp.resize(v.size());
    for (int shift = 0; shift < 30; shift += 10) {
        size_t at[1025] = {};
        for (const auto &x : v) at[((x.first >> shift) & 1023u) + 1]++;
        for (int k = 0; k < 1024; ++k) at[k + 1] += at[k];
        for (const auto &x : v) tmp[at[(x.first >> shift) & 1023u]++] = x;
        v.swap(tmp);
    }
}

void build_chunks(int Np, const std::vector<int4> &tets, const std::vector<double> &rest, std::vector<InstCtl> &ctl,
                  const std::vector<ChunkLimits> &limits, bool grouped, int join_tets, bool pad_slots,
                  ChunkLayout &out) {
    out = ChunkLayout();
    std::vector<int> stamp(Np, -1), lidx(Np, 0), n_part(Np, 0);
    int mark = -1;
    std::vector<std::pair<uint32_t, int>> order, sorted;
    std::vector<int> ctets, lnodes, scount, first, by_count, run_of, lnode_all, lrun_all, lsptr_all, lsend_all;
    int tq = 0;
    for (size_t b = 0; b < ctl.size(); ++b) {
        InstCtl &C = ctl[b];
        const int chunk_tets = limits[b].tets, chunk_nodes = limits[b].nodes;
        const int group_tets = grouped ? CHUNK_GROUP_TETS : 0, group_nodes = CHUNK_GROUP_NODES;
        C.cblk_begin = (int)out.chunk.size();
        C.pblk_begin = (int)out.piece.size();
        double lo[3], hi[3];
        for (int d = 0; d < 3; ++d) {
            lo[d] = std::numeric_limits<double>::max();
            hi[d] = -std::numeric_limits<double>::max();
        }
        auto centroid = [&](int t, double c[3]) {
            const int *q = &tets[t].x;
            for (int d = 0; d < 3; ++d)
                c[d] = 0.25 * (rest[3 * (size_t)q[0] + d] + rest[3 * (size_t)q[1] + d] + rest[3 * (size_t)q[2] + d] +
                               rest[3 * (size_t)q[3] + d]);
        };
        for (int t = C.tet_begin; t < C.tet_end; ++t) {
            double c[3];
            centroid(t, c);
            for (int d = 0; d < 3; ++d) {
                lo[d] = std::min(lo[d], c[d]);
                hi[d] = std::max(hi[d], c[d]);
            }
        }
        order.clear();
        for (int t = C.tet_begin; t < C.tet_end; ++t) {
            double c[3];
            centroid(t, c);
            uint32_t code = 0;
            for (int d = 0; d < 3; ++d) {
                const double ext = hi[d] - lo[d];
                const double f = ext > 0.0 ? (c[d] - lo[d]) / ext : 0.0;
                const uint32_t v = (uint32_t)std::min(1023.0, std::max(0.0, std::floor(f * 1024.0)));
                code |= spread10(v) << d;
            }
            order.emplace_back(code, t);
        }
        sort_by_code(order, sorted);
        if (order.empty()) {  // an instance without tets still needs a CTA for its line-search decisions
            out.cpiece.push_back((int)out.piece.size());
            out.chunk.push_back(make_int4(tq, 0, (int)lnode_all.size(), 0));
            out.piece.push_back(make_int2(tq, 0));
            out.chunk_inst.push_back((int)b);
        }
        // the tets from pos on, up to end, that fit the limits -> ctets; their
        // nodes -> lnodes
        auto take = [&](size_t pos, size_t end, int max_tets, int max_nodes, int ref) {
            ctets.clear();
            lnodes.clear();
            ++mark;
            if (ref >= 0) {
                stamp[ref] = mark;
                lnodes.push_back(ref);
            }
            for (; pos < end && (int)ctets.size() < max_tets; ++pos) {
                const int t = order[pos].second;
                const int *q = &tets[t].x;
                // (a tet's corners are four different nodes: pbs_create)
                int add = 0;
                for (int c = 0; c < 4; ++c) add += stamp[q[c]] != mark;
                if ((int)lnodes.size() + add > max_nodes) break;
                for (int c = 0; c < 4; ++c)
                    if (stamp[q[c]] != mark) {
                        stamp[q[c]] = mark;
                        lnodes.push_back(q[c]);
                    }
                ctets.push_back(t);
            }
        };
        size_t pos = 0, group_end = 0;
        int ref = -1, piece = chunk_tets, slot = 0;  // slot: of the chunk so far
        while (pos < order.size()) {
            bool join = join_tets > 0, taken = false;
            if (group_tets && pos == group_end) {
                join = false;
                // a new group, cut into pieces of even size
                take(pos, order.size(), group_tets, group_nodes, -1);
                group_end = pos + ctets.size();
                ref = *std::min_element(lnodes.begin(), lnodes.end());
                const int n = (int)ctets.size(), k = (n + chunk_tets - 1) / chunk_tets;
                piece = (n + k - 1) / k;
                taken = k == 1 && (int)lnodes.size() <= chunk_nodes;  // the group is its one piece
            }
            if (!taken) take(pos, group_tets ? group_end : order.size(), piece, chunk_nodes, ref);
            pos += ctets.size();
            // local nodes in ascending id order: a warp's node gathers then
            // share sectors
            std::sort(lnodes.begin(), lnodes.end());
            const int nl = (int)lnodes.size(), nt = (int)ctets.size();
            if (!(join && out.chunk.back().y + nt <= join_tets)) {
                out.cpiece.push_back((int)out.piece.size());
                out.chunk.push_back(make_int4(tq, 0, (int)lnode_all.size(), 0));
                out.chunk_inst.push_back((int)b);
                slot = 0;
            }
            int4 &cd = out.chunk.back();
            const int l0 = cd.w;  // the chunk's local nodes so far
            for (int j = 0; j < nl; ++j) lidx[lnodes[j]] = j;
            scount.assign(nl + 1, 0);
            first.resize(nl);
            for (int t : ctets)
                for (int c = 0; c < 4; ++c) scount[lidx[(&tets[t].x)[c]] + 1]++;
            // slot runs: the nodes with the most corners first (a counting sort),
            // so that a warp's partial-sum loops end together; runs of even
            // length padded to odd, so that eight neighbouring lanes read eight
            // different bank groups (1M-tet box, full / incremental stress: 39.6
            // / 44.3 us a pass with the runs in node order, 36.6 / 42.0 so; with
            // the packed node words 35.3 / 41.1)
            by_count.assign(nt + 2, 0);
            for (int j = 0; j < nl; ++j) by_count[nt - scount[j + 1] + 1]++;
            for (int k = 0; k <= nt; ++k) by_count[k + 1] += by_count[k];
            run_of.resize(nl);
            for (int j = 0; j < nl; ++j) run_of[by_count[nt - scount[j + 1]]++] = j;
            for (int r = 0; r < nl; ++r) {
                const int j = run_of[r], cnt = scount[j + 1];
                first[j] = slot;
                slot += pad_slots ? cnt | 1 : cnt;
                lnode_all.push_back(lnodes[r]);
                lrun_all.push_back(lnodes[j]);
                lsptr_all.push_back(first[j]);
                lsend_all.push_back(first[j] + cnt);
                n_part[lnodes[r]]++;
            }
            for (int lt = 0; lt < nt; ++lt) {
                const int *q = &tets[ctets[lt]].x;
                unsigned loc[4], sl[4];
                for (int c = 0; c < 4; ++c) {
                    const int j = lidx[q[c]];
                    loc[c] = (unsigned)(l0 + j);
                    sl[c] = (unsigned)first[j]++;
                }
                out.qcor.push_back(make_uint4(loc[0] | loc[1] << 16, loc[2] | loc[3] << 16, sl[0] | sl[1] << 16,
                                              sl[2] | sl[3] << 16));
                out.qperm.push_back(ctets[lt]);
            }
            out.piece.push_back(make_int2(tq, nt));
            cd.y += nt;
            cd.w += nl;
            out.max_local = std::max(out.max_local, cd.w);
            out.max_slots = std::max(out.max_slots, slot);
            tq += nt;
        }
        C.cblk_end = (int)out.chunk.size();
        C.pblk_end = (int)out.piece.size();
    }
    out.cpiece.push_back((int)out.piece.size());
    // node -> partials, in piece order
    out.pptr.assign(Np + 1, 0);
    for (int i = 0; i < Np; ++i) out.pptr[i + 1] = out.pptr[i] + n_part[i];
    std::vector<int> fill(out.pptr.begin(), out.pptr.end() - 1);
    out.lmeta.resize(lnode_all.size());
    // (a piece's runs are of its own nodes: each node's places go up by piece)
    for (size_t j = 0; j < lnode_all.size(); ++j)
        out.lmeta[j] = make_int4(lnode_all[j], lsptr_all[j], lsend_all[j], fill[lrun_all[j]]++);
}

// Where the lines lie (96 passes of a 5-tet box, full / incremental stress, us;
// "graph" the pass kernels at their best shape, "frame" the frame kernel, with
// 128 threads a CTA):
//   up to 4,096 tets: 128 a chunk (2,340 tets: 409 / 444, 256 a chunk 473 /
//     507, graph 1003 / 1050; up to 8,192 a single instance gained 7% and the
//     batch below lost 4%);
//   up to 2 * sms * 256 (77,824): 256, up to two CTAs a SM of the frame kernel
//     (24,500 tets: 491 / 534, 192 a chunk 497 / 539; 59,940: 616 / 655, 512 a
//     chunk 649 / 712, graph 1114 / 1200).  Finer chunks cost a large batch,
//     whose instances are of these sizes and which the pass kernels run, more
//     partials than they save a single instance: 256 boxes of 1K-41K tets take
//     12.4 ms at 256 a chunk, 14.5 at 128;
//   up to 2 * sms * 342 (103,968): 384, which a group makes 342 (78,000: 694 /
//     748, 256 a chunk 799 / 747; 100,800: 744 / 799, 256 a chunk and three
//     CTAs a SM 917 / 838, 512 a chunk 839 / 879, graph 1226 / 1329);
//   up to sms * 1,024 (155,648): whole groups, one CTA of 256 threads a SM
//     (125,000: 855 / 924, 512 a chunk, 128 threads and two CTAs a SM 849 /
//     894, the same with 256 threads, which spill, 1120 / 1160; 154,980: 879 /
//     950, graph 1240 / 1360).  Where they cost so little, whole groups are
//     worth their sums: a node's partials are then the ones of every other
//     machine width, and iterations to a tolerance stop at the same pass
//     (pieces move one pull in 40 to a residual of 1e-4 by more than 2e-5 of
//     its velocities);
//   beyond, the pass kernels: 384 with 256 threads up to 1,600 a SM (243,200),
//     else whole groups with 512 (384 / groups, full, then incremental stress:
//     160,720 tets 1331 / 1403, 1453 / 1568; 203,205 1309 / 1505, 1444 / 1675;
//     221,030 1429 / 1482, 1607 / 1670; 234,135 1476 / 1493, 1651 / 1686;
//     248,540 1514 / 1490, 1690 / 1685; 298,080 and 400,000 equal within 0.5%;
//     the frame kernel with 704 a chunk took 1291 / 1314 at 203,205, but a group
//     has no pieces of that size).  1M tets, us a pass of both kernels: 48.6 /
//     54.9, 512 a chunk on 256 threads 47.5 / 51.6: the groups' one path to a
//     residual is worth that.
// The node limit leaves room for meshes with more nodes a tet than a box.
ChunkLimits auto_chunk_limits(int tets, int sms) {
    int n;
    if (tets <= 4096) n = 128;
    else if (tets <= 2 * 256 * sms) n = 256;
    else if (tets <= 2 * 342 * sms || (tets > CHUNK_GROUP_TETS * sms && tets <= 1600 * sms)) n = 384;
    else return ChunkLimits{CHUNK_GROUP_TETS, CHUNK_GROUP_NODES};
    return ChunkLimits{n, 32 + n / 2 + n / 16};
}

int auto_team(int tets, int sms) { return tets <= 2 * 342 * sms ? 128 : tets <= 1600 * sms ? 256 : 512; }

// ------------------------------------------------------------ device
__global__ void k_pass_rows(int T, const int *qperm, const float4 *row0, const float4 *row1, const float4 *row2,
                            float4 *q0, float4 *q1, float4 *q2) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= T) return;
    const int t = qperm[j];
    q0[j] = row0[t];
    q1[j] = row1[t];
    q2[j] = row2[t];
}

// Line-search pass: the {sum e, sum e^2} of each of the chunk's pieces, of its
// tets and of its share of the instance's nodes -> st.cpart.  ec: the thread's
// tet energies, where the chunk is one piece and the team is the CTA's threads.
// Double-float (e) and FP32 (e^2, a noise scale), in the order that
// phybs_internal.cuh gives.  Called by every thread, before anything else goes
// into the slots.  (Its values are formed here, not carried through the tet
// loop: registers are short.)
template <int THREADS>
__device__ __forceinline__ void chunk_energy(const DevMesh &m, const DevParams &p, const DevState &st, int c, int inst,
                                             int par, size_t cur, int nt, DFloat ec) {
    __shared__ float2 s_e[THREADS / 32];
    __shared__ float s_e2[THREADS / 32];
    const InstCtl *src = ctl_buf(st, par) + inst;
    const int q = src->pblk_begin + c - src->cblk_begin, a = src->node_begin + (c - src->cblk_begin) * src->share;
    float noise;
    if (THREADS == 512 && m.noise_tets != 0 && nt > THREADS) {
        // two tets a thread: with those of the thread half a CTA away
        __shared__ float s_x[THREADS / 2];
        if (threadIdx.x >= THREADS / 2) s_x[threadIdx.x - THREADS / 2] = ec.hi;
        __syncthreads();
        const float x = threadIdx.x < THREADS / 2 ? ec.hi + s_x[threadIdx.x] : 0.f;
        noise = x * x;
    } else {
        noise = noise_square(m, THREADS, nt, ec.hi);
    }
    DFloat e{0.f, 0.f};
    float e2 = 0.f;
    share_energy(m, p, st, cur, a + threadIdx.x, min(a + src->share, src->node_end), THREADS,
                 p.incremental ? st.ub : nullptr, e, e2);
    e = warp_sum_df(df_add(e, ec));
    e2 = warp_sum_f(e2 + noise);
    if ((threadIdx.x & 31) == 0) {
        s_e[threadIdx.x >> 5] = make_float2(e.hi, e.lo);
        s_e2[threadIdx.x >> 5] = e2;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    double d;
    join_warps(s_e, s_e2, THREADS, d, e2);
    if (threadIdx.x == 0) st.cpart[q] = make_double2(d, (double)e2);
}

// The same where the layout has chunks of several pieces or teams that are not
// the CTA's threads (a packed batch's), from the energies in the slots: teams
// of fewer threads take a piece each at a time, one of 512 takes two rounds.
// In kernels of their own, so that the others keep their registers (two bodies
// of 150,000 tets, 96 passes without a line search: 1460 us, and 1470 when one
// kernel held both).
template <int THREADS>
__device__ __forceinline__ void chunk_energy_teams(const DevMesh &m, const DevParams &p, const DevState &st, int c,
                                                   int inst, int par, size_t cur, const ChunkView &v,
                                                   const float4 *sf) {
    constexpr int MAX_TEAM = 512;
    __shared__ float2 s_e[MAX_TEAM / 32];
    __shared__ float s_e2[MAX_TEAM / 32];
    const InstCtl *src = ctl_buf(st, par) + inst;
    const int pb = src->pblk_begin, per = src->share, p0 = m.cpiece[c], p1 = m.cpiece[c + 1], t0 = m.piece[p0].x;
    const int team = src->team, width = min(team, THREADS), sides = THREADS / width;
    const int tid = threadIdx.x & (width - 1), side = threadIdx.x / width;
    for (int q0 = p0; q0 < p1; q0 += sides) {
        const int q = q0 + side;
        if (q < p1) {
            const int2 pc = m.piece[q];
            const int a = src->node_begin + (q - pb) * per, n1 = min(a + per, src->node_end);
            const uint4 *cor = v.cor + (pc.x - t0);
            float x = 0.f;  // (a team of 512 with two tets a thread: those of the threads t and t + 256)
            for (int r = team - width; r >= 0; r -= width) {
                const DFloat ec = team_energy(cor, pc.y, r + tid, team, sf);
                float noise;
                if (team == MAX_TEAM && m.noise_tets != 0 && pc.y > team) {
                    x = r > 0 ? ec.hi : ec.hi + x;
                    noise = r > 0 ? 0.f : x * x;
                } else {
                    noise = noise_square(m, team, pc.y, ec.hi);
                }
                DFloat e{0.f, 0.f};
                float e2 = 0.f;
                share_energy(m, p, st, cur, a + r + tid, n1, team, p.incremental ? st.ub : nullptr, e, e2);
                e = warp_sum_df(df_add(e, ec));
                e2 = warp_sum_f(e2 + noise);
                if ((tid & 31) == 0) {
                    const int w = side * (width >> 5) + ((r + tid) >> 5);
                    s_e[w] = make_float2(e.hi, e.lo);
                    s_e2[w] = e2;
                }
            }
        }
        __syncthreads();
        if (q < p1 && tid < 32) {
            double d;
            float e2;
            join_warps(s_e + side * (width >> 5), s_e2 + side * (width >> 5), team, d, e2);
            if (tid == 0) {
                st.cpart[q] = make_double2(d, (double)e2);
                __threadfence();  // (thread 0 counts the chunk in for every team)
            }
        }
        __syncthreads();
    }
}

// Then counts the chunk in, and in the instance's last one sums the chunks and
// decides accept / reject (DescentOptimize.cpp:107-128) on dst, the
// control-block copy the pass's node kernel reads (its first chunk settled the
// last pass into it before counting itself in).  The sum runs in FP64.  Called
// by every thread of the CTA; *is_last is a shared word.
template <int THREADS>
__device__ __forceinline__ void chunk_line_search(const DevParams &p, const DevState &st, int inst, int par, int k,
                                                  double *sh, int *is_last) {
    const InstCtl *src = ctl_buf(st, par) + inst;
    InstCtl *dst = ctl_buf(st, par ^ 1) + inst;
    unsigned int *cnt = st.tcount + inst;
    const int pb = src->pblk_begin, pe = src->pblk_end;
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned int prev = atomicAdd(cnt, 1u);
        *is_last = (prev == (unsigned int)(src->cblk_end - src->cblk_begin - 1));
    }
    __syncthreads();
    if (!*is_last) return;
    __threadfence();
    // the instance's last chunk: fixed-order sums, then accept / reject.  The
    // partials are loaded eight at a time ahead of their additions: this tail
    // runs on one CTA while the rest of the GPU waits, and one load round trip
    // per partial made it several microseconds
    constexpr int U = 8;
    const int lanes = src->by_share ? 32 : min(src->team, 256);
    double ea = 0.0, eb = 0.0;
    if (threadIdx.x < lanes)
        for (int j0 = pb + threadIdx.x; j0 < pe; j0 += U * lanes) {
            double2 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + u * lanes;
                v[u] = j < pe ? __ldcg(st.cpart + j) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ea += v[u].x;
                eb += v[u].y;
            }
        }
    const double E = block_sum(ea, sh);
    const double E2 = block_sum(eb, sh);
    if (threadIdx.x != 0) return;
    *cnt = 0;
    // one load, updates in registers, one store; an instance the settled
    // decision stopped keeps its control block (this pass ran on speculation)
    InstCtl ci = load_ctl_cg(dst);
    if (ci.done) return;
    decide_line_search(ci, p, k, E, E2);
    *dst = ci;
    if (ci.done) atomicSub(st.active, 1);
}

// The whole of one chunk once its node words (and, with STAGE, its rows and
// records) are in shared memory: forces, partials, the Jacobi diagonal every
// hd_every passes, and the line-search tail.
template <int MATERIAL, int THREADS, bool INC, bool PACK, bool PRE, bool TEAMS>
__device__ __forceinline__ void chunk_body(const DevMesh &m, const DevParams &p, const DevState &st, int c,
                                           int inst, int par, const PassView &pv, size_t cur, const ChunkView &v,
                                           const int4 *meta, int nt, int nl, float4 *sf, double *sh,
                                           int *is_last, const TetRows &first = TetRows()) {
    const DFloat e = chunk_forces_all<MATERIAL, THREADS, INC, PACK, PRE>(p, v, nt, pv.check, sf, first);
    chunk_partials<THREADS>(meta, nl, sf, st.part);
    if (pv.check) {
        if (TEAMS) chunk_energy_teams<THREADS>(m, p, st, c, inst, par, cur, v, sf);
        else chunk_energy<THREADS>(m, p, st, c, inst, par, cur, nt, e);
    }
    if (pv.do_h) {
        __syncthreads();
        chunk_hdiag<MATERIAL, THREADS, INC, PACK>(v, nt, sf);
        __syncthreads();
        chunk_partials<THREADS>(meta, nl, sf, st.parth);
    }
    // the instance's first chunk takes the last pass's pending decision after
    // its own tets (the other chunks run on its foreseen outcome without
    // waiting), and before it counts itself into a line search
    const InstCtl *src = ctl_buf(st, par) + inst;
    if (c == src->cblk_begin) settle_pass<THREADS>(p, st, src, ctl_buf(st, par ^ 1) + inst, true);
    if (pv.check) chunk_line_search<THREADS>(p, st, inst, par, pv.k, sh, is_last);
}

// One CTA per chunk.  What bounds it: with four CTAs of 256 threads a SM, each
// of them two waits for memory and two barriers, the latency of its loads (the
// shared-memory wavefronts take 39% of the active cycles at 512,000 tets).  The
// constants of a thread's first node and first tet are therefore read before
// the grid-dependency wait, and the first node's words beside the control block
// instead of after it: 1M tets, full / incremental stress, 35.3 / 41.7 -> 34.1
// / 38.1 us a pass; 256 boxes of 1K-41K tets 93.4 / 107 -> 90.2 / 99.6.  (Rows
// of the second tet prefetched into L1 or L2 as well: no change.)
// STAGE: every thread first issues asynchronous copies of
// its tets' rows and corner records and of the chunk's local-node records into
// shared memory -- before the grid-dependency wait, since they are constant --
// and of the chunk's node words after it; one wait then covers all of them,
// instead of one global round trip per tet inside the loop.
#ifndef PBS_INC_THREADS_PER_SM
#define PBS_INC_THREADS_PER_SM 1024
#endif
// Register budget: 64 a thread (1024 threads a SM; with the incremental stress
// a few registers spill, and the extra resident warps pay for them: 44.9
// against 49.7 us a pass on the 1M-tet box at 85 registers).  The full stress
// of either material needs 64 on its tet loop; the bound keeps the out-of-line
// calls of near-inverted tets, after the loop, from raising it.
template <int MATERIAL, int THREADS, bool INC, bool STAGE, bool TEAMS>
__global__ void __launch_bounds__(THREADS, PBS_INC_THREADS_PER_SM / THREADS)
    k_tchunk(DevMesh m, DevParams p, DevState st, int par) {
    extern __shared__ float4 smem4[];
    const int CN = m.chunk_nodes, CT = m.chunk_tets;
    // node words: 24 bytes a node, or with STAGE u hi, u lo (without INC) or the
    // increment (with INC), base (INC only); corner slots; with STAGE the rows
    // and records
    float4 *s_uh = smem4, *s_ul = smem4 + CN, *s_ub = smem4 + 2 * CN;
    float4 *s_wa = smem4;
    float2 *s_wb = reinterpret_cast<float2 *>(smem4 + CN);
    float4 *s_f = smem4 + node_words(CN, INC, STAGE ? 1 : 0);  // corner slots
    float4 *s_r0 = s_f + m.chunk_slots, *s_r1 = s_r0 + CT, *s_r2 = s_r1 + CT;  // STAGE only
    uint4 *s_cor = reinterpret_cast<uint4 *>(s_r2 + CT);
    int4 *s_meta = reinterpret_cast<int4 *>(s_cor + CT);
    __shared__ double sh[THREADS / 32];
    __shared__ int is_last;
    const int c = blockIdx.x;
    // the chunk table and the per-tet rows are constant: read them before
    // waiting for the node kernel
    const int4 cd = m.chunk[c];
    const int inst = m.chunk_inst[c];
    const int tq0 = cd.x, nt = cd.y, l0 = cd.z, nl = cd.w;
    // the chunk's reference node for the increments (incremental form; the
    // chunk of an instance without tets has no local node: its first record
    // may lie past the table), this thread's first node and its first tet's
    // constants
    const int g_ref = INC && !STAGE && nl > 0 ? m.lmeta[l0].x : 0;
    int g_first = 0;
    TetRows first;
    if (!STAGE) {
        if (threadIdx.x < nl) g_first = m.lmeta[l0 + threadIdx.x].x;
        if (threadIdx.x < nt) {
            const int q = tq0 + threadIdx.x;
            first = TetRows{m.qrow0[q], m.qrow1[q], m.qrow2[q], m.qcor[q]};
        }
    }
    if (STAGE) {
        for (int lt = threadIdx.x; lt < nt; lt += THREADS) {
            const int q = tq0 + lt;
            cp_async16(s_r0 + lt, m.qrow0 + q);
            cp_async16(s_r1 + lt, m.qrow1 + q);
            cp_async16(s_r2 + lt, m.qrow2 + q);
            cp_async16(s_cor + lt, m.qcor + q);
        }
        for (int j = threadIdx.x; j < nl; j += THREADS) cp_async16(s_meta + j, m.lmeta + l0 + j);
        cp_async_commit();
    }
    const size_t cur = (size_t)par * m.Np;
    pdl_launch_dependents();
    pdl_wait();
    const InstCtl *src = ctl_buf(st, par) + inst;
    InstCtl *dst = ctl_buf(st, par ^ 1) + inst;
    const int4 *meta = STAGE ? s_meta : m.lmeta + l0;
    if (STAGE) {
        // each thread stages the node words of the records it copied itself;
        // the gathers need no control word (the pass's parity is known at
        // launch) and run while it is read
        cp_async_wait_all();
        for (int j = threadIdx.x; j < nl; j += THREADS) {
            const int g = s_meta[j].x;
            cp_async16(s_uh + j, st.uh + cur + g);
            cp_async16(s_ul + j, st.ul + cur + g);
            if (INC) cp_async16(s_ub + j, st.ub + g);
        }
        cp_async_commit();
    }
    // the first node's words, read while the control block is (a stopped
    // instance's go unused)
    float4 uh0, ul0, ub0, r_ref;
    if (!STAGE && threadIdx.x < nl) {
        uh0 = st.uh[cur + g_first];
        ul0 = st.ul[cur + g_first];
        if (INC) ub0 = st.ub[g_first];
    }
    if (!STAGE && INC && nl > 0) r_ref = st.uh[cur + g_ref];
    const PassView pv = pass_view(src, p);
    if (pv.skip) {
        // an instance that stopped: its first chunk carries the control block
        // over to the copy the node kernel reads
        if (c == src->cblk_begin) settle_pass<THREADS>(p, st, src, dst, true);
        if (STAGE) cp_async_wait_all();
        return;
    }
    if (STAGE) {
        cp_async_wait_all();
        if (INC) {
            // the increments of the nodes this thread staged, relative to the
            // chunk's local node 0 (staged by thread 0)
            __syncthreads();
            const float4 r = s_uh[0];
            __syncthreads();
            for (int j = threadIdx.x; j < nl; j += THREADS) s_ul[j] = increment_rel(s_uh[j], s_ul[j], r);
        }
    } else {
        // (the increments relative to the chunk's local node 0)
        for (int j = threadIdx.x; j < nl; j += THREADS) {
            if (j != threadIdx.x) {
                const int g = meta[j].x;
                uh0 = st.uh[cur + g];
                ul0 = st.ul[cur + g];
                if (INC) ub0 = st.ub[g];
            }
            if (INC) pack_words(s_wa, s_wb, j, increment_rel(uh0, ul0, r_ref), ub0);
            else pack_words(s_wa, s_wb, j, uh0, ul0);
        }
    }
    __syncthreads();
    ChunkView v;
    v.wa = s_wa;
    v.wb = s_wb;
    v.uh = s_uh;
    v.ul = s_ul;
    v.ub = s_ub;
    v.r0 = STAGE ? s_r0 : m.qrow0 + tq0;
    v.r1 = STAGE ? s_r1 : m.qrow1 + tq0;
    v.r2 = STAGE ? s_r2 : m.qrow2 + tq0;
    v.cor = STAGE ? s_cor : m.qcor + tq0;
    v.meta = meta;
    v.rest = m.rest;
    chunk_body<MATERIAL, THREADS, INC, !STAGE, !STAGE, TEAMS>(m, p, st, c, inst, par, pv, cur, v, meta, nt, nl, s_f, sh,
                                                              &is_last, first);
}

// ------------------------------------------------------------ persistent, TMA-fed variant
// mbarrier and bulk-copy (TMA) primitives.  A bulk copy moves a contiguous
// global range into shared memory and reports its bytes to an mbarrier; the
// phase completes when the expected byte count has arrived.
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// dst, src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for phase `parity` of *bar for at most limit_ns; false when it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity, unsigned long long limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = globaltimer_ns();
    while (!mbar_try_wait(bar, parity))
        if (globaltimer_ns() - t0 > limit_ns) return false;
    return true;
}

// A wait on a bulk copy that has not completed in a second means the copy
// engine or the pipeline bookkeeping is broken: the kernel records
// PBS_E_DEVICE_TIMEOUT in the instance and returns instead of spinning on.
constexpr unsigned long long STREAM_WAIT_NS = 1000000000ull;

// One staging buffer of the persistent kernel.
struct StageBuf {
    float4 *r0, *r1, *r2;
    uint4 *cor;
    int4 *meta;
    float4 *uh, *ul, *ub;
};

// Buffer b of the persistent kernel's shared memory: [buffer 0][buffer 1]
// [slots]; a buffer holds rows 0..2 and corner records (16 B a tet each),
// then local-node records and node words (16 B a node each).
__device__ __forceinline__ StageBuf stage_buf(float4 *smem4, int b, int CT, int CN, int stride) {
    float4 *q = smem4 + b * stride;
    StageBuf s;
    s.r0 = q;
    s.r1 = q + CT;
    s.r2 = q + 2 * CT;
    s.cor = reinterpret_cast<uint4 *>(q + 3 * CT);
    s.meta = reinterpret_cast<int4 *>(q + 4 * CT);
    s.uh = q + 4 * CT + CN;
    s.ul = q + 4 * CT + 2 * CN;
    s.ub = q + 4 * CT + 3 * CN;  // with incremental stress only
    return s;
}

// Thread 0: the chunk's rows, corner records and local-node records by bulk
// copies, completing on *bar.
__device__ __forceinline__ void stage_chunk_bulk(const DevMesh &m, int c, const StageBuf &b, uint64_t *bar) {
    const int4 cd = m.chunk[c];
    const unsigned nt = (unsigned)cd.y, nl = (unsigned)cd.w;
    mbar_expect_tx(bar, 64u * nt + 16u * nl);
    if (nt) {
        bulk_g2s(b.r0, m.qrow0 + cd.x, 16u * nt, bar);
        bulk_g2s(b.r1, m.qrow1 + cd.x, 16u * nt, bar);
        bulk_g2s(b.r2, m.qrow2 + cd.x, 16u * nt, bar);
        bulk_g2s(b.cor, m.qcor + cd.x, 16u * nt, bar);
    }
    if (nl) bulk_g2s(b.meta, m.lmeta + cd.z, 16u * nl, bar);
}

// What a chunk's pass needs from its instance's control blocks.
struct StreamCtx {
    const InstCtl *src;
    InstCtl *dst;
    int inst, nt, nl;
    bool first, skip;
    PassView pv;
    size_t cur;
};

__device__ __forceinline__ StreamCtx stream_ctx(const DevMesh &m, const DevParams &p, const DevState &st, int c,
                                                int par, size_t cur) {
    StreamCtx x;
    const int4 cd = m.chunk[c];
    x.nt = cd.y;
    x.nl = cd.w;
    x.inst = m.chunk_inst[c];
    x.src = ctl_buf(st, par) + x.inst;
    x.dst = ctl_buf(st, par ^ 1) + x.inst;
    x.first = c == x.src->cblk_begin;
    x.pv = pass_view(x.src, p);
    x.skip = x.pv.skip;
    x.cur = cur;
    return x;
}

// Node words of a chunk (local-node records already in b.meta) by cp.async.
template <int THREADS, bool INC>
__device__ __forceinline__ void stage_nodes(const DevState &st, const StageBuf &b, int nl, size_t cur) {
    for (int j = threadIdx.x; j < nl; j += THREADS) {
        const int g = b.meta[j].x;
        cp_async16(b.uh + j, st.uh + cur + g);
        cp_async16(b.ul + j, st.ul + cur + g);
        if (INC) cp_async16(b.ub + j, st.ub + g);
    }
}

// Persistent chunk kernel: CTA b walks chunks b, b + G, b + 2G, ... (G =
// gridDim.x, a whole number of resident CTAs per SM) through two staging
// buffers.  While chunk j computes, chunk j+1's node words are in flight by
// cp.async and chunk j+2's rows and records by bulk copies, so the global
// round trips of the one-CTA-per-chunk kernel (control block, records, node
// gather) leave the critical path.  Chunk for chunk, the arithmetic and its
// order are those of k_tchunk with the same shape: results are bit-identical.
template <int MATERIAL, int THREADS, bool INC>
__global__ void __launch_bounds__(THREADS, 768 / THREADS) k_tstream(DevMesh m, DevParams p, DevState st, int par) {
    extern __shared__ float4 smem4[];
    const int CN = m.chunk_nodes, CT = m.chunk_tets;
    const int stride = 4 * CT + (INC ? 4 : 3) * CN;  // float4 words of one staging buffer
    float4 *s_f = smem4 + 2 * stride;  // corner slots, 4 a tet
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ double sh[THREADS / 32];
    __shared__ int is_last;
    const int G = gridDim.x, c0 = blockIdx.x;
    const int nj = c0 < m.n_chunks ? (m.n_chunks - c0 + G - 1) / G : 0;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init_fence();
    }
    __syncthreads();
    // the first two chunks' rows and records are constant: they go out before
    // the grid-dependency wait
    if (threadIdx.x == 0) {
        if (nj > 0) stage_chunk_bulk(m, c0, stage_buf(smem4, 0, CT, CN, stride), &bar[0]);
        if (nj > 1) stage_chunk_bulk(m, c0 + G, stage_buf(smem4, 1, CT, CN, stride), &bar[1]);
    }
    pdl_launch_dependents();
    pdl_wait();
    if (nj == 0) return;
    StreamCtx cur, nxt;
    nxt.skip = true;
    // chunk 0: its records, then its node words
    bool ok = mbar_wait_bounded(&bar[0], 0u, STREAM_WAIT_NS);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) atomicExch(st.active + 1, 1);  // the instances stop with PBS_E_DEVICE_TIMEOUT
        if (nj > 1) mbar_wait_bounded(&bar[1], 0u, STREAM_WAIT_NS);
        return;
    }
    const size_t pcur = (size_t)par * m.Np;
    cur = stream_ctx(m, p, st, c0, par, pcur);
    if (!cur.skip) stage_nodes<THREADS, INC>(st, stage_buf(smem4, 0, CT, CN, stride), cur.nl, cur.cur);
    cp_async_commit();
    for (int j = 0; j < nj; ++j) {
        const int b = j & 1, c = c0 + j * G;
        if (j + 1 < nj) {
            // chunk j+1: wait for its records, start its node words
            ok = mbar_wait_bounded(&bar[b ^ 1], (unsigned)((j + 1) >> 1) & 1u, STREAM_WAIT_NS);
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0) atomicExch(st.active + 1, 1);
                cp_async_wait_all();
                mbar_wait_bounded(&bar[b ^ 1], (unsigned)((j + 1) >> 1) & 1u, STREAM_WAIT_NS);
                return;
            }
            nxt = stream_ctx(m, p, st, c + G, par, pcur);
            if (!nxt.skip) stage_nodes<THREADS, INC>(st, stage_buf(smem4, b ^ 1, CT, CN, stride), nxt.nl, nxt.cur);
            cp_async_commit();
            asm volatile("cp.async.wait_group 1;" ::: "memory");  // chunk j's node words (this thread's)
        } else {
            cp_async_wait_all();
        }
        const StageBuf sb = stage_buf(smem4, b, CT, CN, stride);
        if (INC && !cur.skip) {
            // the increments of the nodes this thread staged, relative to the
            // chunk's local node 0 (staged by thread 0)
            __syncthreads();
            const float4 r = sb.uh[0];
            __syncthreads();
            for (int i = threadIdx.x; i < cur.nl; i += THREADS) sb.ul[i] = increment_rel(sb.uh[i], sb.ul[i], r);
        }
        __syncthreads();
        if (cur.first && cur.skip) settle_pass<THREADS>(p, st, cur.src, cur.dst, true);
        if (!cur.skip) {
            ChunkView v;
            v.uh = sb.uh;
            v.ul = sb.ul;
            v.ub = sb.ub;
            v.r0 = sb.r0;
            v.r1 = sb.r1;
            v.r2 = sb.r2;
            v.cor = sb.cor;
            v.meta = sb.meta;
            v.rest = m.rest;
            chunk_body<MATERIAL, THREADS, INC, false, false, false>(m, p, st, c, cur.inst, par, cur.pv, cur.cur, v, sb.meta,
                                                                    cur.nt, cur.nl, s_f, sh, &is_last);
        }
        __syncthreads();  // buffer b and the slots are free again
        if (threadIdx.x == 0 && j + 2 < nj) stage_chunk_bulk(m, c + 2 * G, sb, &bar[b]);
        cur = nxt;
    }
}

// ------------------------------------------------------------ launchers
template <int MATERIAL, int THREADS, bool INC, bool STAGE, bool TEAMS = false> static cudaError_t allow_smem() {
    return cudaFuncSetAttribute(k_tchunk<MATERIAL, THREADS, INC, STAGE, TEAMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                CHUNK_MAX_SMEM);
}

template <int MATERIAL, int THREADS, bool INC> static cudaError_t allow_smem_stream() {
    return cudaFuncSetAttribute(k_tstream<MATERIAL, THREADS, INC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                CHUNK_MAX_SMEM);
}

template <int MATERIAL, bool INC> static cudaError_t allow_smem_all() {
    const cudaError_t e[] = {allow_smem<MATERIAL, 128, INC, false>(), allow_smem<MATERIAL, 256, INC, false>(),
                             allow_smem<MATERIAL, 512, INC, false>(), allow_smem<MATERIAL, 256, INC, false, true>()};
    for (cudaError_t x : e)
        if (x != cudaSuccess) return x;
    return cudaSuccess;
}

cudaError_t prepare_chunk_kernels() {
    const cudaError_t e[] = {allow_smem_all<PBS_MATERIAL_NEOHOOKEAN, true>(),
                             allow_smem_all<PBS_MATERIAL_NEOHOOKEAN, false>(),
                             allow_smem_all<PBS_MATERIAL_STRETCH, false>(),
                             allow_smem<PBS_MATERIAL_NEOHOOKEAN, 128, false, true>(),
                             allow_smem<PBS_MATERIAL_NEOHOOKEAN, 256, false, true>(),
                             allow_smem<PBS_MATERIAL_NEOHOOKEAN, 128, true, true>(),
                             allow_smem<PBS_MATERIAL_NEOHOOKEAN, 256, true, true>(),
                             allow_smem_stream<PBS_MATERIAL_NEOHOOKEAN, 128, false>(),
                             allow_smem_stream<PBS_MATERIAL_NEOHOOKEAN, 256, false>(),
                             allow_smem_stream<PBS_MATERIAL_NEOHOOKEAN, 128, true>(),
                             allow_smem_stream<PBS_MATERIAL_NEOHOOKEAN, 256, true>()};
    for (cudaError_t x : e)
        if (x != cudaSuccess) return x;
    return cudaSuccess;
}

cudaError_t launch_pass_rows(cudaStream_t s, int T, const int *qperm, const float4 *row0, const float4 *row1,
                             const float4 *row2, float4 *q0, float4 *q1, float4 *q2) {
    if (T <= 0) return cudaSuccess;
    k_pass_rows<<<(T + 255) / 256, 256, 0, s>>>(T, qperm, row0, row1, row2, q0, q1, q2);
    return cudaGetLastError();
}

// Launch of a per-tet pass kernel: programmatic dependent launch (pdl), and
// the mesh's L2 access-policy window over the pass rows when it has one.  at:
// room for two attributes.
static cudaLaunchConfig_t chunk_config(cudaStream_t s, int grid, int threads, size_t smem, bool pdl,
                                       cudaLaunchAttribute *at, const DevMesh &m) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    int n = 0;
    if (pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    if (m.l2_base) {
        at[n].id = cudaLaunchAttributeAccessPolicyWindow;
        at[n].val.accessPolicyWindow.base_ptr = const_cast<void *>(m.l2_base);
        at[n].val.accessPolicyWindow.num_bytes = m.l2_bytes;
        at[n].val.accessPolicyWindow.hitRatio = m.l2_hit;
        at[n].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        at[n].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cfg;
}

template <int MATERIAL, int THREADS, bool INC, bool STAGE, bool TEAMS = false>
static cudaError_t launch_tchunk_t(cudaStream_t s, const DevMesh &m, const DevParams &p, const DevState &st, int par,
                                   bool pdl) {
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = chunk_config(s, m.n_chunks, THREADS,
                                          chunk_smem(m.chunk_tets, m.chunk_nodes, m.chunk_slots, INC, STAGE ? 1 : 0), pdl, at, m);
    return cudaLaunchKernelEx(&cfg, k_tchunk<MATERIAL, THREADS, INC, STAGE, TEAMS>, m, p, st, par);
}

template <int MATERIAL, int THREADS, bool INC>
static cudaError_t launch_tstream_t(cudaStream_t s, const DevMesh &m, const DevParams &p, const DevState &st, int par,
                                    bool pdl) {
    if (m.stream_grid <= 0) return cudaErrorInvalidConfiguration;
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg =
        chunk_config(s, m.stream_grid, THREADS, chunk_smem(m.chunk_tets, m.chunk_nodes, m.chunk_slots, INC, 2), pdl, at, m);
    return cudaLaunchKernelEx(&cfg, k_tstream<MATERIAL, THREADS, INC>, m, p, st, par);
}

template <int MATERIAL, bool INC>
static cudaError_t launch_tchunk(cudaStream_t s, const DevMesh &m, const DevParams &p, const DevState &st, int par,
                                 bool pdl) {
    if (m.chunk_threads == 128) return launch_tchunk_t<MATERIAL, 128, INC, false>(s, m, p, st, par, pdl);
    if (m.teams)  // (packed automatic layouts, with 256 threads)
        return m.chunk_threads == 256 ? launch_tchunk_t<MATERIAL, 256, INC, false, true>(s, m, p, st, par, pdl)
                                      : cudaErrorInvalidConfiguration;
    if (m.chunk_threads == 512) return launch_tchunk_t<MATERIAL, 512, INC, false>(s, m, p, st, par, pdl);
    return launch_tchunk_t<MATERIAL, 256, INC, false>(s, m, p, st, par, pdl);
}

cudaError_t launch_tet_only(cudaStream_t s, const DevMesh &m, const DevParams &p, DevState st, int material, int par,
                            bool pdl) {
    if (m.n_chunks <= 0) return cudaSuccess;
    if (material == PBS_MATERIAL_STRETCH) return launch_tchunk<PBS_MATERIAL_STRETCH, false>(s, m, p, st, par, pdl);
    // staged shapes: neo-Hookean, 128 or 256 threads
    const bool t128 = m.chunk_threads == 128, t256 = m.chunk_threads == 256;
    if (m.chunk_stage == 2) {
        if (p.incremental) {
            if (t128) return launch_tstream_t<PBS_MATERIAL_NEOHOOKEAN, 128, true>(s, m, p, st, par, pdl);
            if (t256) return launch_tstream_t<PBS_MATERIAL_NEOHOOKEAN, 256, true>(s, m, p, st, par, pdl);
        } else {
            if (t128) return launch_tstream_t<PBS_MATERIAL_NEOHOOKEAN, 128, false>(s, m, p, st, par, pdl);
            if (t256) return launch_tstream_t<PBS_MATERIAL_NEOHOOKEAN, 256, false>(s, m, p, st, par, pdl);
        }
    }
    const bool st128 = m.chunk_stage == 1 && t128, st256 = m.chunk_stage == 1 && t256;
    if (p.incremental) {
        if (st128) return launch_tchunk_t<PBS_MATERIAL_NEOHOOKEAN, 128, true, true>(s, m, p, st, par, pdl);
        if (st256) return launch_tchunk_t<PBS_MATERIAL_NEOHOOKEAN, 256, true, true>(s, m, p, st, par, pdl);
        return launch_tchunk<PBS_MATERIAL_NEOHOOKEAN, true>(s, m, p, st, par, pdl);
    }
    if (st128) return launch_tchunk_t<PBS_MATERIAL_NEOHOOKEAN, 128, false, true>(s, m, p, st, par, pdl);
    if (st256) return launch_tchunk_t<PBS_MATERIAL_NEOHOOKEAN, 256, false, true>(s, m, p, st, par, pdl);
    return launch_tchunk<PBS_MATERIAL_NEOHOOKEAN, false>(s, m, p, st, par, pdl);
}

// CTAs of the persistent chunk kernel for the mesh's shape: as many as fit on
// the device at once, at most one per chunk.  0 when the shape has no
// persistent variant.
template <int MATERIAL, int THREADS, bool INC> static int stream_fit(const DevMesh &m, int sms) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tstream<MATERIAL, THREADS, INC>, THREADS,
                                                      chunk_smem(m.chunk_tets, m.chunk_nodes, m.chunk_slots, INC, 2)) != cudaSuccess)
        return 0;
    return std::min(m.n_chunks, per_sm * sms);
}

int stream_grid(const DevMesh &m, int material, bool inc, int sms) {
    if (m.chunk_stage != 2 || material != PBS_MATERIAL_NEOHOOKEAN || m.n_chunks <= 0) return 0;
    if (m.chunk_threads == 128)
        return inc ? stream_fit<PBS_MATERIAL_NEOHOOKEAN, 128, true>(m, sms)
                   : stream_fit<PBS_MATERIAL_NEOHOOKEAN, 128, false>(m, sms);
    if (m.chunk_threads == 256)
        return inc ? stream_fit<PBS_MATERIAL_NEOHOOKEAN, 256, true>(m, sms)
                   : stream_fit<PBS_MATERIAL_NEOHOOKEAN, 256, false>(m, sms);
    return 0;
}

}  // namespace pbs
